// Sweeps of the branch-free unit vector against sqrtf and the IEEE division (test_gpu_unit_vector.py).
#include "ys_collide.cuh"

using namespace ys;

__device__ u32 rnd(u64 i) {  // splitmix64
    i += 0x9E3779B97F4A7C15ull;
    i = (i ^ (i >> 30)) * 0xBF58476D1CE4E5B9ull;
    i = (i ^ (i >> 27)) * 0x94D049BB133111EBull;
    return (u32)((i ^ (i >> 31)) >> 32);
}

__device__ bool all_ones(float len) { return (~__float_as_uint(len) & 0x7FFFFFu) == 0u; }

// s in [1, 4): every significand at both parities; bad[0] roots, bad[1] reciprocals that are off.
__global__ void k_roots(unsigned long long* bad) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 1u << 24) return;
    const float s = __uint_as_float(0x3F800000u + i);
    float len, inv;
    unit_root(s, len, inv);
    if (len != sqrtf(s)) atomicAdd(&bad[0], 1ull);
    if (!all_ones(len) && inv != 1.f / len) atomicAdd(&bad[1], 1ull);
}

// Every significand of the length against n numerators: at random, and beside the midpoints between two quotients.
__global__ void k_quotients(u32 n, unsigned long long* bad) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (1u << 23) - 1u) return;  // not all ones
    const float len = __uint_as_float(0x3F800000u + i), inv = 1.f / len;
    u32 off = 0;
    for (u32 k = 0; k < n; ++k) {
        const u32 r = rnd((u64)i * n + k);
        float a;
        if (k & 1u) {
            const double mid = (double)__uint_as_float(0x3F000000u | (r & 0x7FFFFFu)) + 0x1p-25;  // between two in [1/2, 1)
            a = __uint_as_float(__float_as_uint((float)(mid * (double)len)) + ((r >> 23) % 3u) - 1u);
        } else {
            a = __uint_as_float(((127u - (r >> 23) % 50u) << 23) | (r & 0x7FFFFFu));
            a = (r >> 31) ? -a : a;
        }
        if (unit_quotient(a, len, inv) != a / len) ++off;
    }
    if (off) atomicAdd(bad, (unsigned long long)off);
}

// Vectors from far below the bounds to far above them, components down to and through 2^-80 of the largest, zeros of both
// signs; bad[0]: taken and off in a bit; bad[1]: how many were taken.
__global__ void k_vectors(u32 n, unsigned long long* bad) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float c[3];
    const int e0 = (int)(rnd(4ull * i) % 80u) - 40;
    for (int k = 0; k < 3; ++k) {
        const u32 r = rnd(4ull * i + 1 + k), m = rnd(~(4ull * i + 1 + k));
        const int drop = (m >> 28) < 8 ? 0 : (m >> 28) < 12 ? (int)(r >> 8) % 12 : (int)(r >> 8) % 70;
        const float v = ldexpf(1.f + (float)(r & 0x7FFFFFu) * 0x1p-23f, e0 - drop);
        c[k] = (m >> 24 & 15u) == 0 ? 0.f : v;
        if (m & 1u) c[k] = -c[k];
    }
    float len;
    f3 u;
    const f3 d = mk(c[0], c[1], c[2]);
    if (!unit_vector(d, len, u)) return;
    atomicAdd(&bad[1], 1ull);
    const float want = sqrtf(dot(d, d));
    const f3 w = d / want;
    if (__float_as_uint(len) != __float_as_uint(want) || __float_as_uint(u.x) != __float_as_uint(w.x) ||
        __float_as_uint(u.y) != __float_as_uint(w.y) || __float_as_uint(u.z) != __float_as_uint(w.z))
        atomicAdd(&bad[0], 1ull);
}

// out: wrong roots, wrong reciprocals, wrong quotients, wrong vectors, vectors taken
extern "C" int sweep(unsigned long long out[5], u32 numerators, u32 vectors) {
    unsigned long long* bad = nullptr;
    cudaError_t e = cudaMalloc((void**)&bad, 40);
    if (e == cudaSuccess) e = cudaMemset(bad, 0, 40);
    if (e != cudaSuccess) return (int)e;
    k_roots<<<(1u << 24) / 256, 256>>>(bad);
    k_quotients<<<(1u << 23) / 256, 256>>>(numerators, bad + 2);
    k_vectors<<<(vectors + 255) / 256, 256>>>(vectors, bad + 3);
    e = cudaMemcpy(out, bad, 40, cudaMemcpyDeviceToHost);
    cudaFree(bad);
    return (int)e;
}
