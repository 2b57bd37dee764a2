// ys_groups.cuh -- one block of the sorted-leaf groups' refit (GroupJob): for k_refit_groups, and for the kernel of small
// scenes that has the spring forces in its other blocks.
#pragma once
#include "ys_collide.cuh"
#include "ys_lbvh.cuh"

namespace ys {

static constexpr u32 GROUP_THREADS = 512;  // two leaves per thread: all of a 512k-leaf tree's blocks are resident

// One block's 32 warp-runs of one box set: each run's box to l1 (written by
// the caller's warps through group_run), then the block's to l2 and the top.
__device__ __forceinline__ void group_run(float4* __restrict__ l0, float4* __restrict__ l1, u32 first, u32 i, bool has,
                                          f3 lo, f3 hi, u32 (*sh)[6], u32 run) {
    if (has) {
        l0[2 * (size_t)(first + i)] = make_float4(lo.x, lo.y, lo.z, 0.f);
        l0[2 * (size_t)(first + i) + 1] = make_float4(hi.x, hi.y, hi.z, 0.f);
    }
    const u32 POS = ford(__int_as_float(0x7F800000)), NEG = ford(-__int_as_float(0x7F800000));
    const float v[6] = {lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
    u32 r[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {  // NaN takes no part, as in fminf / fmaxf
        const bool on = has && v[k] == v[k];
        r[k] = k < 3 ? __reduce_min_sync(0xFFFFFFFFu, on ? ford(v[k]) : POS)
                     : __reduce_max_sync(0xFFFFFFFFu, on ? ford(v[k]) : NEG);
    }
    if ((threadIdx.x & 31u) == 0) {
        const u32 j = (first + i) >> 5;
        l1[2 * (size_t)j] = make_float4(funord(r[0]), funord(r[1]), funord(r[2]), 0.f);
        l1[2 * (size_t)j + 1] = make_float4(funord(r[3]), funord(r[4]), funord(r[5]), 0.f);
#pragma unroll
        for (int k = 0; k < 6; ++k) sh[run][k] = r[k];
    }
}

// The box of the block's 32 runs (warp 0) to l2, the top and the root.
__device__ __forceinline__ void group_block(float4* __restrict__ l2, u32* __restrict__ top, u32* __restrict__ root,
                                            u32 first, u32 b, u32 (*sh)[6]) {
    u32 r[6];
#pragma unroll
    for (int k = 0; k < 6; ++k)
        r[k] = k < 3 ? __reduce_min_sync(0xFFFFFFFFu, sh[threadIdx.x][k]) : __reduce_max_sync(0xFFFFFFFFu, sh[threadIdx.x][k]);
    if (threadIdx.x == 0) {
        if (l2) {
            const size_t j = first / GROUP_BLOCK + b;
            l2[2 * j] = make_float4(funord(r[0]), funord(r[1]), funord(r[2]), 0.f);
            l2[2 * j + 1] = make_float4(funord(r[3]), funord(r[4]), funord(r[5]), 0.f);
        }
        const u32 POS = ford(__int_as_float(0x7F800000));
        if (r[0] != POS || r[1] != POS || r[2] != POS)  // not a block of empty boxes
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const u32 a = k < 3 ? ~r[k] : r[k];
                if (top) atomicMax(&top[8 * (size_t)(b / (GROUP_TOP / GROUP_BLOCK)) + k], a);
                if (root) atomicMax(&root[k], a);
            }
    }
}

// Every box set, record, grid extent and root box of a substep in one launch:
// the gathers of x (and v) are the dependent loads, every write is a
// coalesced stream.  It replaces the 4-wide tree's refit in the fused
// substep (leaf pass + range pass, 48.8 + 10.9 us under ncu on the 522,242-face
// cloth, bound by its scattered slot writes; 25.3 us here).
__device__ __forceinline__ void refit_groups_block(const GroupJob* __restrict__ jobs, const u32* __restrict__ blkJob,
                                                   const float4* __restrict__ x, const float4* __restrict__ v,
                                                   const GroupBufs& B) {
    __shared__ u32 shk[32][6], shb[32][6], sh_ext[GROUP_THREADS / 32];
    const GroupJob& J = jobs[blkJob[blockIdx.x]];
    const u32 b = blockIdx.x - J.block0, w = threadIdx.x >> 5, flags = J.flags, n = J.n;
    if (blockIdx.x == 0 && threadIdx.x < B.nctr) B.ctr[threadIdx.x] = 0ull;
    if (flags & GJ_VERTS) {
        u32 r[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
#pragma unroll
        for (u32 h = 0; h < GROUP_BLOCK / GROUP_THREADS; ++h) {
            const u32 i = b * GROUP_BLOCK + h * GROUP_THREADS + threadIdx.x;
            if (i >= n) continue;
            const f3 p = ld(x, J.voff + i);
            f3 lo = p, hi = p;
            if (flags & GJ_SWEPT) {
                const f3 sp = p + ld(v, J.voff + i) * J.dt;  // the swept leaf's x + v dt
                lo = vmin(p, sp);
                hi = vmax(p, sp);
            }
            r[0] = min(r[0], ford(lo.x)); r[1] = min(r[1], ford(lo.y)); r[2] = min(r[2], ford(lo.z));
            r[3] = max(r[3], ford(hi.x)); r[4] = max(r[4], ford(hi.y)); r[5] = max(r[5], ford(hi.z));
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            r[k] = k < 3 ? __reduce_min_sync(0xFFFFFFFFu, r[k]) : __reduce_max_sync(0xFFFFFFFFu, r[k]);
            if ((threadIdx.x & 31u) == 0) shk[w][k] = r[k];
        }
        if (threadIdx.x < 6) {  // the runs no warp fills
            for (u32 q = GROUP_THREADS / 32; q < 32; ++q) shk[q][threadIdx.x] = threadIdx.x < 3 ? 0xFFFFFFFFu : 0u;
        }
        __syncthreads();
        if (w == 0) group_block(nullptr, nullptr, B.root + 8 * (size_t)J.root, 0u, b, shk);
        return;
    }
    float ext = 0.f;
#pragma unroll
    for (u32 h = 0; h < GROUP_BLOCK / GROUP_THREADS; ++h) {
        const u32 i = b * GROUP_BLOCK + h * GROUP_THREADS + threadIdx.x;
        const u32 run = h * (GROUP_THREADS / 32) + w;
        const bool has = i < n;
        const u32 li = has ? i : n - 1;
        uint4 q;
        if (J.lvid) q = J.lvid[li];
        else q = make_uint4(J.facets[3 * li], J.facets[3 * li + 1], J.facets[3 * li + 2], li);
        const u32 vid[3] = {J.voff + q.x, J.voff + q.y, J.voff + q.z};
        const f3 P[3] = {ld(x, vid[0]), ld(x, vid[1]), ld(x, vid[2])};
        if (flags & GJ_KEY) {
            // key box and H1 grid extent (collectFaceBoxes, spatial_hash.hpp:1613-1655)
            float4 lo, hi;
            const bool ok = h1_key_box(P[0], P[1], P[2], J.margin, lo, hi);
            if (ok && has) ext = fmaxf(fmaxf(ext, hi.x - lo.x), fmaxf(hi.y - lo.y, hi.z - lo.z));
            const float inf = __int_as_float(0x7F800000);
            const f3 klo = ok ? mk(lo.x, lo.y, lo.z) : mk(inf, inf, inf);
            const f3 khi = ok ? mk(hi.x, hi.y, hi.z) : mk(-inf, -inf, -inf);
            group_run(B.l0, B.l1, J.keyL0, i, has, klo, khi, shk, run);
        }
        if (flags & (GJ_BOX | GJ_ROOT)) {
            f3 lo, hi;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const f3 p = P[k];
                f3 a = p, c = p;
                if (flags & GJ_SWEPT) {
                    const f3 sp = p + ld(v, vid[k]) * J.dt;
                    a = vmin(p, sp);
                    c = vmax(p, sp);
                }
                if (k == 0) { lo = a; hi = c; } else { lo = vmin(lo, a); hi = vmax(hi, c); }
            }
            if (flags & GJ_BOX) {
                group_run(B.l0, B.l1, J.boxL0, i, has, lo, hi, shb, run);
            } else {
                const float u[6] = {lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    const bool on = has && u[k] == u[k];
                    const u32 r = k < 3 ? __reduce_min_sync(0xFFFFFFFFu, on ? ford(u[k]) : ford(__int_as_float(0x7F800000)))
                                        : __reduce_max_sync(0xFFFFFFFFu, on ? ford(u[k]) : ford(-__int_as_float(0x7F800000)));
                    if ((threadIdx.x & 31u) == 0) shb[run][k] = r;
                }
            }
        }
        if ((flags & GJ_REC) && has) {
            const f3 nr = cross(P[1] - P[0], P[2] - P[0]);
            const float nl2 = dot(nr, nr);
            const bool flat = nl2 < 1e-12f;
            const f3 u = flat ? nr : nr * (1.0f / sqrtf(nl2));
            float4* o = B.rec + 4 * (size_t)(J.rec + i);
            o[0] = make_float4(P[0].x, P[0].y, P[0].z, __uint_as_float(q.w));
            o[1] = make_float4(P[1].x, P[1].y, P[1].z, 0.f);
            o[2] = make_float4(P[2].x, P[2].y, P[2].z, 0.f);
            o[3] = make_float4(u.x, u.y, u.z, flat ? 0.f : 1.f);
        }
    }
    if (flags & GJ_KEY) {
        const u32 e = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(ext));  // positive floats order as ints
        if ((threadIdx.x & 31u) == 0) sh_ext[w] = e;
    }
    __syncthreads();
    if (w == 0) {
        if (flags & GJ_KEY) {
            group_block(B.l2, B.top + 8 * (size_t)J.keyTop, nullptr, J.keyL0, b, shk);
            const u32 e = __reduce_max_sync(0xFFFFFFFFu, threadIdx.x < GROUP_THREADS / 32 ? sh_ext[threadIdx.x] : 0u);
            if (threadIdx.x == 0) atomicMax(J.maxExt, e);
        }
        if (flags & (GJ_BOX | GJ_ROOT))
            group_block((flags & GJ_BOX) ? B.l2 : nullptr, (flags & GJ_BOX) ? B.top + 8 * (size_t)J.boxTop : nullptr,
                        (flags & GJ_ROOT) ? B.root + 8 * (size_t)J.root : nullptr, J.boxL0, b, shb);
    }
}

}  // namespace ys
