// The radix sort with a poll limit of 0 in its look-back: a tile whose predecessor has not published yet counts that
// tile's keys itself (test_gpu_sort_forms.py).
#define YS_SORT_LOOK_POLLS 0
#include "ys_sort.cu"

namespace ys {
ys_status fail(ys_status code, const std::string&) { return code; }
}  // namespace ys

extern "C" int sort_pairs(uint32_t* keys, uint32_t* vals, uint32_t n) {
    void* scratch = nullptr;
    cudaError_t e = cudaMalloc(&scratch, ys::sort_scratch_bytes(n));
    if (e == cudaSuccess) e = ys::radix_sort_pairs(keys, vals, n, scratch, 0, 32, nullptr);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    cudaFree(scratch);
    return (int)e;
}
