// ys_adj64.cuh -- FP64 rollout of one FastGridCloth over static triangle
// obstacles, and its reverse pass (the adjoint's 64-bit mode).
//
// The single-precision adjoint differentiates the substep exactly as the
// fused kernel computes it, so its gradients carry FP32 round-off amplified
// by the rollout's conditioning (stiff springs over hundreds of steps).  This
// mode runs the same step in binary64, operation for operation as the FP64
// reference rollout states it, so that the gradient differs from FP64 finite
// differences only by the differencing error:
//
//   f_i = (ext_i or g m_i) + kair v_i + sum_s (k_s (l - L_s) + kd (dv . n)) n,
//         n = dx (1 / l), springs in the stencil order of
//         compute_cloth_grid_forces_fast (physics.metal:197-218), l < 1e-7 skipped
//   v'  = v + f ((subh / m) mask)
//   for each contact (n_c, d_c) in (object, triangle) order with d_c < thickness:
//         { if v'.n_c < 0: v' -= (v'.n_c) n_c;  x += (thickness - d_c) n_c }
//   x'  = x + v' (subh mask)
//
// Contacts: the cloth's swept box (x and x + v subh over its vertices) culls
// each obstacle by its root box; the point query box x +- margin selects
// every face whose exact AABB it overlaps (queryPoints, bvh.metal:1322-1412),
// and narrow_pt_tri (bruteforce.metal:41-178) runs in double on each.  The
// candidates come from the obstacle's sorted-leaf groups (float boxes), queried
// with the double box rounded outward to float: a float box that contains the
// double one overlaps every leaf whose face AABB the double box overlaps, so
// the exact double test then sees the same faces as a search over all faces.
// The contacts of a vertex are kept sorted by face, so the order of the
// descent does not reach the result.
//
// Every operation is a single IEEE binary64 add, multiply, divide or square
// root (the library is built without contraction), in the order of the
// expressions above, so the rollout is the FP64 reference's bit for bit.
#pragma once

namespace ys {

struct dd3 { double x, y, z; };
__device__ __forceinline__ dd3 dm(double a, double b, double c) { return dd3{a, b, c}; }
__device__ __forceinline__ dd3 operator+(dd3 a, dd3 b) { return dm(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ dd3 operator-(dd3 a, dd3 b) { return dm(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ dd3 operator*(dd3 a, double s) { return dm(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ double ddot(dd3 a, dd3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ dd3 dcross(dd3 a, dd3 b) {
    return dm(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// One vertex's position / velocity / adjoint in binary64 (32-byte aligned:
// two 16-byte loads).
struct __align__(32) D4 { double x, y, z, w; };
__device__ __forceinline__ dd3 ldd(const D4* p, u32 i) { const D4 q = p[i]; return dm(q.x, q.y, q.z); }
__device__ __forceinline__ void std4(D4* p, u32 i, dd3 a) { p[i] = D4{a.x, a.y, a.z, 0.0}; }
__device__ __forceinline__ dd3 ldf(const float4* p, u32 i) {
    const float4 q = p[i];
    return dm((double)q.x, (double)q.y, (double)q.z);
}

// A contact of one step: normal and signed distance.
struct __align__(32) DContact { double nx, ny, nz, d; };

static constexpr u32 D64_CAP = 16;    // contacts kept per vertex and step
// Bound on one warp's search in one obstacle, per vertex: candidates tested
// and runs of 32 leaves opened; past it the search stops and the rollout fails.
static constexpr u32 D64_STEPS = 1u << 24;
// Block size of the search, step and reverse kernels.
static constexpr u32 D64_BLOCK = 128;

// Order-preserving map of binary64 onto u64 (larger double, larger key), so
// that min / max are integer atomics; NaN is left out by the callers.
__device__ __forceinline__ unsigned long long dord(double d) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double dunord(unsigned long long o) {
    const unsigned long long b = (o >> 63) ? (o & 0x7FFFFFFFFFFFFFFFull) : ~o;
    return __longlong_as_double((long long)b);
}

struct A64 {
    // the scene: obstacle positions (the current buffer; obstacles are
    // static), faces, trees, meshes, the cloth's target list
    const float4* sx;
    const uint4* F;
    GroupBufs grp;
    const uint4* lvid;
    const MeshDev* meshes;
    const u32* targets;
    const float4* ext;  // external forces or null (then g m)
    const float* mass;
    const float* mask;
    u32 tgt_begin, tgt_end, cloth, voff, nV, N;
    double gx, gy, gz, kair, kd, subh, thickness, margin, radius;
    const double* k;  // per-spring stiffness / rest length (canonical order)
    const double* L;
    // state of step t and the step's outputs (cloth vertices, local index)
    const D4* x;
    const D4* xp;
    const D4* v;
    D4* xn;
    D4* vn;
    DContact* cs;  // D64_CAP slots per vertex, sorted by (object, face)
    u32* cf;       // their face ids
    u32* cn;       // contacts per vertex
    // the contact search's output, per vertex: up to D64_CAP contacts in
    // search order, their face ids and target ordinals, the count
    DContact* ls;
    u32* lf;
    u32* lk;
    u32* ln;
    u32 vpw;  // vertices per warp of the contact search
    unsigned long long* box;  // cloth swept box: ~dord(min) x3 then dord(max) x3, all by atomicMax
    u32* status;
};

__device__ __forceinline__ double grid_k64(const A64& A, u32 sid) { return A.k[sid]; }

// narrow_pt_tri in double (the FP64 reference's restatement): the face's
// plane normal oriented by the previous position (the current one when the
// previous lies on the plane), a crossing or a distance below radius +
// margin, the barycentric test at the crossing point (or the current point).
__device__ __forceinline__ bool narrow64(dd3 qc, dd3 qp, dd3 t0, dd3 t1, dd3 t2, double radius, double margin,
                                         dd3& nout, double& dout) {
    const dd3 e0 = t1 - t0, e1 = t2 - t0;
    dd3 n = dcross(e0, e1);
    const double nl2 = ddot(n, n);
    if (nl2 < 1e-12) return false;
    n = n * (1.0 / sqrt(nl2));
    double dp = ddot(n, qp - t0), dc = ddot(n, qc - t0);
    const double dref = (dp != 0.0) ? dp : dc;
    if (dref < 0.0) {
        n = n * -1.0;
        dp = -dp;
        dc = -dc;
    }
    const bool crossed = dc < 0.0, inm = dc < radius + margin;
    if (!crossed && !inm) return false;
    const dd3 cp = (crossed && dp > 0.0) ? qp + (qc - qp) * (dp / (dp - dc)) : qc;
    const dd3 pc = cp - t0;
    const dd3 inplane = pc - n * ddot(n, pc);
    const double d00 = ddot(e0, e0), d01 = ddot(e0, e1), d11 = ddot(e1, e1), d20 = ddot(inplane, e0),
                 d21 = ddot(inplane, e1);
    const double den = d00 * d11 - d01 * d01;
    if (fabs(den) < 1e-12) return false;
    const double b = (d11 * d20 - d01 * d21) / den, c = (d00 * d21 - d01 * d20) / den, a = 1.0 - b - c;
    if (!(a >= 0.0 && b >= 0.0 && c >= 0.0)) return false;
    nout = n;
    dout = dc;
    return true;
}

// Spring q (0 .. 11, in grid_stencil's order) of grid vertex (row, col): its
// other end and id; false when the cloth ends before it.
__device__ __forceinline__ bool grid_spring(int N, int row, int col, int q, u32& j, u32& sid) {
    // per spring: row and column offset, family, and the first end's offset
    // from the vertex (the id counts first ends, row-major in the family)
    static constexpr signed char DR[12] = {0, 0, -1, 1, -1, -1, 1, 1, 0, 0, -2, 2};
    static constexpr signed char DC[12] = {-1, 1, 0, 0, -1, 1, -1, 1, -2, 2, 0, 0};
    if (q >= 12) return false;
    int dr = 0, dc = 0;
#pragma unroll
    for (int k = 0; k < 12; ++k)
        if (q == k) { dr = DR[k]; dc = DC[k]; }
    const int r = row + dr, c = col + dc;
    if (r < 0 || r >= N || c < 0 || c >= N) return false;
    j = (u32)(r * N + c);
    const u32 n = (u32)N, top = (u32)min(row, r), left = (u32)min(col, c);
    const u32 bSY = n * (n - 1), bHA = bSY + (n - 1) * n, bHB = bHA + (n - 1) * (n - 1), bBX = bHB + (n - 1) * (n - 1),
              bBY = bBX + n * (n - 2);
    if (dr == 0) sid = dc * dc == 1 ? top * (n - 1) + left : bBX + top * (n - 2) + left;
    else if (dc == 0) sid = dr * dr == 1 ? bSY + top * n + left : bBY + top * n + left;
    else sid = (dr == dc ? bHA : bHB) + top * (n - 1) + left;
    return true;
}

// LPV lanes per vertex: 1 (a thread runs its vertex's 12 springs) or 16 (a
// lane per spring, then every lane adds the forces in the stencil's order).
// With a thread per vertex a small cloth is a hundred warps of twelve
// dependent square roots and divisions each; a lane per spring issues three
// times the instructions (a step, a vertex and a springs pass of the 65 x 65
// cloth: 8.1 / 7.8 / 12.0 us by thread, 4.2 / 4.3 / 5.0 us by lane).
static constexpr u32 D64_SPREAD = 65536;  // vertices up to which a lane per spring is used
__device__ __forceinline__ double d64_from(double v, int q) { return __shfl_sync(0xFFFFFFFFu, v, q, 16); }

// Force on cloth vertex i (local) from the state (x, v); q: this lane's
// spring (LPV 16; every lane of the warp calls).
template <int LPV>
__device__ __forceinline__ dd3 force64(const A64& A, const D4* x, const D4* v, u32 i, int q) {
    const u32 g = A.voff + i;
    const dd3 p = ldd(x, i), w = ldd(v, i);
    const double m = (double)A.mass[g];
    const dd3 f0 = A.ext ? ldf(A.ext, g) : dm(A.gx * m, A.gy * m, A.gz * m);
    dd3 f = f0 + w * A.kair;
    const int N = (int)A.N, row = (int)(i / A.N), col = (int)(i % A.N);
    auto one = [&](u32 j, u32 sid, dd3& s) {
        const dd3 dx = ldd(x, j) - p, dv = ldd(v, j) - w;
        const double l = sqrt(ddot(dx, dx));
        if (l < 1e-7) return false;
        const dd3 nd = dx * (1.0 / l);
        s = nd * (A.k[sid] * (l - A.L[sid]) + A.kd * ddot(dv, nd));
        return true;
    };
    if constexpr (LPV == 1) {
        grid_stencil(N, row, col, [&](int r, int c, int, u32 sid) {
            dd3 s;
            if (one((u32)(r * N + c), sid, s)) f = f + s;
        });
    } else {
        u32 j = 0, sid = 0;
        dd3 s = dm(0.0, 0.0, 0.0);
        const bool on = grid_spring(N, row, col, q, j, sid) && one(j, sid, s);
        const unsigned have = __ballot_sync(0xFFFFFFFFu, on) >> (threadIdx.x & 16u);
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            const dd3 t = dm(d64_from(s.x, k), d64_from(s.y, k), d64_from(s.z, k));
            if ((have >> k) & 1u) f = f + t;
        }
    }
    return f;
}

// Cloth swept box of step t: x and x + v subh over the cloth's vertices.
__global__ void __launch_bounds__(256) k_d64_box(A64 A) {
    unsigned long long r[6] = {0, 0, 0, 0, 0, 0};
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < A.nV; i += gridDim.x * blockDim.x) {
        const dd3 p = ldd(A.x, i), s = p + ldd(A.v, i) * A.subh;
        const double c[6] = {p.x, p.y, p.z, s.x, s.y, s.z};
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            if (c[q] != c[q]) continue;  // NaN: fmin / fmax skip it
            const int a = q % 3;
            const unsigned long long o = dord(c[q]);
            r[a] = max(r[a], ~o);
            r[3 + a] = max(r[3 + a], o);
        }
    }
    __shared__ unsigned long long sh[6][8];
    const u32 lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        unsigned long long v = r[q];
        for (int o = 16; o; o >>= 1) v = max(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
        if (lane == 0) sh[q][wid] = v;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        unsigned long long v = 0;
        for (u32 w = 0; w < (blockDim.x >> 5); ++w) v = max(v, sh[threadIdx.x][w]);
        if (v) atomicMax(A.box + threadIdx.x, v);
    }
}

// Contact search of one step: a warp descends each obstacle's groups once for
// its vpw vertices, as the fused substep does (one lane per child, then one
// per leaf), and tests the candidates 32 at a time in double.  (Sixteen
// one-thread subtree descents per vertex: 41 us on the 65 x 65 cloth.)
struct D64Work {
    u32 qf[64], qk[64];       // candidates: sorted leaf, target ordinal << 5 | owner lane
    float4 vlo[32], vhi[32];  // the vertices' query boxes, rounded outward
    u32 n[32];                // contacts found per vertex
};
__global__ void __launch_bounds__(D64_BLOCK) k_d64_cand(A64 A) {
    __shared__ D64Work work[D64_BLOCK / 32];
    D64Work& Q = work[threadIdx.x >> 5];
    const u32 lane = threadIdx.x & 31u;
    const u32 first = (blockIdx.x * (D64_BLOCK / 32) + (threadIdx.x >> 5)) * A.vpw;
    const bool in = lane < A.vpw && first + lane < A.nV;
    const u32 i = in ? first + lane : 0u;
    const dd3 p = ldd(A.x, i);
    u32 st = 0, qn = 0;
    const f3 blo = mk(__double2float_rd(p.x - A.margin), __double2float_rd(p.y - A.margin), __double2float_rd(p.z - A.margin));
    const f3 bhi = mk(__double2float_ru(p.x + A.margin), __double2float_ru(p.y + A.margin), __double2float_ru(p.z + A.margin));
    Q.vlo[lane] = make_float4(blo.x, blo.y, blo.z, 0.f);
    Q.vhi[lane] = make_float4(bhi.x, bhi.y, bhi.z, 0.f);
    Q.n[lane] = 0;
    __syncwarp();
    const LaneBox LB = lane_box(blo, bhi);
    f3 alo, ahi;
    lane_union(LB, in, alo, ahi);
    const dd3 slo = dm(dunord(~A.box[0]), dunord(~A.box[1]), dunord(~A.box[2]));
    const dd3 shi = dm(dunord(A.box[3]), dunord(A.box[4]), dunord(A.box[5]));
    auto drain = [&](u32 base, u32 cnt) {
        __syncwarp();
        if (lane < cnt) {
            const u32 key = Q.qk[base + lane], v = key & 31u, k = key >> 5;
            const MeshDev& T = A.meshes[A.targets[A.tgt_begin + k]];
            const u32 f = A.lvid[T.foff + Q.qf[base + lane]].w;
            const uint4 tri = A.F[T.foff + f];
            const dd3 t0 = ldf(A.sx, T.voff + tri.x), t1 = ldf(A.sx, T.voff + tri.y), t2 = ldf(A.sx, T.voff + tri.z);
            const dd3 x = ldd(A.x, first + v);
            const dd3 qmn = x - dm(A.margin, A.margin, A.margin), qmx = x + dm(A.margin, A.margin, A.margin);
            const double mnx = fmin(t0.x, fmin(t1.x, t2.x)), mxx = fmax(t0.x, fmax(t1.x, t2.x));
            const double mny = fmin(t0.y, fmin(t1.y, t2.y)), mxy = fmax(t0.y, fmax(t1.y, t2.y));
            const double mnz = fmin(t0.z, fmin(t1.z, t2.z)), mxz = fmax(t0.z, fmax(t1.z, t2.z));
            dd3 cn;
            double cd;
            if (!(qmx.x < mnx || qmn.x > mxx || qmx.y < mny || qmn.y > mxy || qmx.z < mnz || qmn.z > mxz) &&
                narrow64(x, ldd(A.xp, first + v), t0, t1, t2, A.radius, A.margin, cn, cd)) {
                const u32 slot = atomicAdd(&Q.n[v], 1u);
                const size_t o = (size_t)(first + v) * D64_CAP + slot;
                if (slot >= D64_CAP) st |= YS_FLAG_CONTACT_OVF;
                else {
                    A.ls[o] = DContact{cn.x, cn.y, cn.z, cd};
                    A.lf[o] = f;
                    A.lk[o] = k;
                }
            }
        }
        __syncwarp();
    };
    for (u32 k = A.tgt_begin; k < A.tgt_end; ++k) {
        const u32 t = A.targets[k];
        const MeshDev& T = A.meshes[t];
        if (t == A.cloth || T.nF == 0 || (T.flags & MF_ANALYTIC)) continue;
        float rl[3], rh[3];
        group_acc_box(A.grp.root + 8 * (size_t)T.root, rl, rh);
        if (shi.x < (double)rl[0] || slo.x > (double)rh[0] || shi.y < (double)rl[1] || slo.y > (double)rh[1] ||
            shi.z < (double)rl[2] || slo.z > (double)rh[2])
            continue;
        const u32 n = T.nF, n1 = (n + 31u) / 32u, n2 = (n + 1023u) / 1024u;
        u32 steps = 0;
        const float4* __restrict__ L0 = A.grp.l0 + 2 * (size_t)T.boxL0;
        const float4* __restrict__ L1 = A.grp.l1 + 2 * (size_t)(T.boxL0 / 32u);
        const float4* __restrict__ L2 = A.grp.l2 + 2 * (size_t)(T.boxL0 / 1024u);
        for (u32 q2 = 0; q2 < n2; q2 += 32u) {
            // the children of a run of 32768 at once
            const u32 k2 = min(q2 + lane, n2 - 1u);
            unsigned m2 = __ballot_sync(FULL_MASK, q2 + lane < n2 && meets(alo, ahi, __ldg(L2 + 2 * (size_t)k2), __ldg(L2 + 2 * (size_t)k2 + 1)));
            while (m2) {
                const u32 c2 = q2 + (u32)__ffs(m2) - 1u;
                m2 &= m2 - 1u;
                const bool in2 = in && meets(blo, bhi, __ldg(L2 + 2 * (size_t)c2), __ldg(L2 + 2 * (size_t)c2 + 1));
                if (!__ballot_sync(FULL_MASK, in2)) continue;
                f3 ulo, uhi;
                lane_union(LB, in2, ulo, uhi);
                const u32 k1 = min(c2 * 32u + lane, n1 - 1u);
                unsigned m1 = __ballot_sync(FULL_MASK, c2 * 32u + lane < n1 && meets(ulo, uhi, __ldg(L1 + 2 * (size_t)k1), __ldg(L1 + 2 * (size_t)k1 + 1)));
                while (m1) {
                    const u32 c1 = c2 * 32u + (u32)__ffs(m1) - 1u;
                    m1 &= m1 - 1u;
                    unsigned vm = __ballot_sync(FULL_MASK, in2 && meets(blo, bhi, __ldg(L1 + 2 * (size_t)c1), __ldg(L1 + 2 * (size_t)c1 + 1)));
                    if (!vm) continue;
                    const u32 leaf = c1 * 32u + lane, li = min(leaf, n - 1u);
                    const float4 lo = __ldg(L0 + 2 * (size_t)li), hi = __ldg(L0 + 2 * (size_t)li + 1);
                    do {
                        const u32 v = (u32)__ffs(vm) - 1u;
                        vm &= vm - 1u;
                        const float4 a = Q.vlo[v], b = Q.vhi[v];
                        const bool hit = leaf < n && meets(mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), lo, hi);
                        const unsigned hm = __ballot_sync(FULL_MASK, hit);
                        if (hit) {
                            const u32 slot = qn + (u32)__popc(hm & ((1u << lane) - 1u));
                            Q.qf[slot] = leaf;
                            Q.qk[slot] = ((k - A.tgt_begin) << 5) | v;
                        }
                        qn += (u32)__popc(hm);
                        if (qn >= 32u) {
                            qn -= 32u;
                            steps += 32u;
                            drain(qn, 32);
                        }
                    } while (vm);
                }
                if ((steps += 32u) > D64_STEPS * A.vpw) {  // at most 2^29
                    st |= YS_FLAG_STACK_OVF;
                    m2 = 0;
                    q2 = n2;
                }
            }
        }
    }
    if (qn) drain(0, qn);
    if (in) A.ln[i] = Q.n[lane];
    if (st) atomicOr(A.status, st);
}

// One step of the FP64 rollout for each vertex: its contacts sorted by
// (object, face) (recorded in cs / cf / cn), then forces, integration and the
// contact response.
template <int LPV>
__global__ void __launch_bounds__(D64_BLOCK) k_d64_step(A64 A) {
    const u32 t = blockIdx.x * blockDim.x + threadIdx.x, lane = t % LPV;
    const bool in = t / LPV < A.nV;
    const u32 i = in ? t / LPV : A.nV - 1;  // threads past the end help with the last vertex's sums and drop them
    const dd3 f = force64<LPV>(A, A.x, A.v, i, (int)lane);
    if (!in || lane != 0) return;
    const u32 g = A.voff + i;
    const dd3 p = ldd(A.x, i);
    DContact* cs = A.cs + (size_t)i * D64_CAP;
    u32* cf = A.cf + (size_t)i * D64_CAP;
    unsigned long long key[D64_CAP];
    u32 n = 0, st = 0;
    const u32 m0 = min(A.ln[i], D64_CAP);
    for (u32 c = 0; c < m0; ++c) {
        const size_t o = (size_t)i * D64_CAP + c;
        const unsigned long long kc = ((unsigned long long)A.lk[o] << 32) | A.lf[o];
        u32 s2 = n++;
        while (s2 > 0 && key[s2 - 1] > kc) {
            key[s2] = key[s2 - 1];
            cs[s2] = cs[s2 - 1];
            cf[s2] = cf[s2 - 1];
            --s2;
        }
        key[s2] = kc;
        cs[s2] = A.ls[o];
        cf[s2] = A.lf[o];
    }
    A.cn[i] = n;
    const double m = (double)A.mass[g], mk_ = (double)A.mask[g];
    dd3 vel = ldd(A.v, i) + f * (A.subh / m * mk_);
    dd3 pos = p;
    for (u32 c = 0; c < n; ++c) {
        const DContact C = cs[c];
        const dd3 nc = dm(C.nx, C.ny, C.nz);
        if (C.d < A.thickness) {
            const double vn = ddot(vel, nc);
            if (vn < 0.0) vel = vel - nc * vn;
            pos = pos + nc * (A.thickness - C.d);
        }
    }
    pos = pos + vel * (A.subh * mk_);
    std4(A.xn, i, pos);
    std4(A.vn, i, vel);
    if (!isfinite(pos.x) || !isfinite(pos.y) || !isfinite(pos.z) || !isfinite(vel.x) || !isfinite(vel.y) ||
        !isfinite(vel.z))
        st |= YS_FLAG_NONFINITE;
    if (st) atomicOr(A.status, st);
}

struct J64 {
    const D4* ax;  // dL/dx_{t+1}, dL/dv_{t+1}
    const D4* av;
    D4* xbar;
    D4* vbar;
    D4* fbar;
    D4* ax_out;
    D4* av_out;
    double* gk;  // per-spring accumulators
    double* gL;
};

// Reverse of the integration and the contact response of step t (the
// forward's active set replayed from the recorded contacts).
template <int LPV>
__global__ void __launch_bounds__(D64_BLOCK) k_d64_adj_vertex(A64 A, J64 J) {
    const u32 t = blockIdx.x * blockDim.x + threadIdx.x, lane = t % LPV;
    const bool in = t / LPV < A.nV;
    const u32 i = in ? t / LPV : A.nV - 1;
    const dd3 f = force64<LPV>(A, A.x, A.v, i, (int)lane);
    if (!in || lane != 0) return;
    const u32 g = A.voff + i;
    const DContact* cs = A.cs + (size_t)i * D64_CAP;
    const u32 n = A.cn[i] < D64_CAP ? A.cn[i] : D64_CAP;
    const double m = (double)A.mass[g], mk_ = (double)A.mask[g];
    const double s = A.subh / m * mk_;
    dd3 vel = ldd(A.v, i) + f * s;
    u32 proj = 0;
    for (u32 c = 0; c < n; ++c) {
        const DContact C = cs[c];
        if (C.d < A.thickness) {
            const dd3 nc = dm(C.nx, C.ny, C.nz);
            const double vn = ddot(vel, nc);
            if (vn < 0.0) {
                vel = vel - nc * vn;
                proj |= 1u << c;
            }
        }
    }
    const dd3 axi = ldd(J.ax, i);
    dd3 vb = ldd(J.av, i) + axi * (A.subh * mk_);
    for (int c = (int)n - 1; c >= 0; --c)
        if (proj >> c & 1u) {
            const DContact C = cs[c];
            const dd3 nc = dm(C.nx, C.ny, C.nz);
            vb = vb - nc * ddot(nc, vb);
        }
    dd3 xb = axi;
    for (u32 c = 0; c < n; ++c) {
        const DContact C = cs[c];
        if (C.d < A.thickness) {
            const dd3 nc = dm(C.nx, C.ny, C.nz);
            xb = xb - nc * ddot(nc, axi);
        }
    }
    std4(J.xbar, i, xb);
    std4(J.vbar, i, vb);
    std4(J.fbar, i, vb * s);
}

// Reverse of the spring and drag forces of step t: gathered per vertex, the
// spring parameters' gradients accumulated by the lower-index end.
template <int LPV>
__global__ void __launch_bounds__(D64_BLOCK) k_d64_adj_springs(A64 A, J64 J) {
    const u32 t = blockIdx.x * blockDim.x + threadIdx.x, lane = t % LPV;
    const bool in = t / LPV < A.nV;
    const u32 i = in ? t / LPV : A.nV - 1;
    const int N = (int)A.N, row = (int)(i / A.N), col = (int)(i % A.N);
    const dd3 p = ldd(A.x, i), w = ldd(A.v, i), fi = ldd(J.fbar, i);
    const double kd = A.kd;
    dd3 dxb = dm(0.0, 0.0, 0.0), dvb = dm(0.0, 0.0, 0.0);
    auto one = [&](u32 j, u32 sid, dd3& ddx, dd3& ddv) {
        const dd3 dx = ldd(A.x, j) - p, dv = ldd(A.v, j) - w;
        const double l = sqrt(ddot(dx, dx));
        if (l < 1e-7) return false;
        const double k = A.k[sid], rest = A.L[sid];
        const dd3 nd = dx * (1.0 / l);
        const double a = k * (l - rest) + kd * ddot(dv, nd);
        const dd3 gdir = fi - ldd(J.fbar, j);
        const double ng = ddot(nd, gdir);
        const dd3 dvp = dv - nd * ddot(nd, dv), gp = gdir - nd * ng;
        ddx = nd * (k * ng) + dvp * (kd * ng / l) + gp * (a / l);
        ddv = nd * (kd * ng);
        if (in && i < j) {  // one owner per spring: no race on the accumulators
            J.gk[sid] += (l - rest) * ng;
            J.gL[sid] += -k * ng;
        }
        return true;
    };
    dd3 ddx = dm(0.0, 0.0, 0.0), ddv = dm(0.0, 0.0, 0.0);
    if constexpr (LPV == 1) {
        grid_stencil(N, row, col, [&](int r, int c, int, u32 sid) {
            if (!one((u32)(r * N + c), sid, ddx, ddv)) return;
            dxb = dxb - ddx;
            dvb = dvb - ddv;
        });
    } else {
        u32 j = 0, sid = 0;
        const bool on = grid_spring(N, row, col, (int)lane, j, sid) && one(j, sid, ddx, ddv);
        const unsigned have = __ballot_sync(0xFFFFFFFFu, on) >> (threadIdx.x & 16u);
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            const dd3 a = dm(d64_from(ddx.x, k), d64_from(ddx.y, k), d64_from(ddx.z, k));
            const dd3 c = dm(d64_from(ddv.x, k), d64_from(ddv.y, k), d64_from(ddv.z, k));
            if ((have >> k) & 1u) {
                dxb = dxb - a;
                dvb = dvb - c;
            }
        }
    }
    if (!in || lane != 0) return;
    std4(J.ax_out, i, ldd(J.xbar, i) + dxb);
    std4(J.av_out, i, ldd(J.vbar, i) + (dvb + fi * A.kair));
}

// The per-vertex kernels with a lane per spring or a thread per vertex.
inline void launch_d64_step(const A64& A, cudaStream_t st) {
    if (A.nV <= D64_SPREAD) k_d64_step<16><<<ceil_div((long long)A.nV * 16, D64_BLOCK), D64_BLOCK, 0, st>>>(A);
    else k_d64_step<1><<<ceil_div(A.nV, D64_BLOCK), D64_BLOCK, 0, st>>>(A);
}
inline void launch_d64_adjoint(const A64& A, const J64& J, cudaStream_t st) {
    if (A.nV <= D64_SPREAD) {
        const int g = ceil_div((long long)A.nV * 16, D64_BLOCK);
        k_d64_adj_vertex<16><<<g, D64_BLOCK, 0, st>>>(A, J);
        k_d64_adj_springs<16><<<g, D64_BLOCK, 0, st>>>(A, J);
    } else {
        const int g = ceil_div(A.nV, D64_BLOCK);
        k_d64_adj_vertex<1><<<g, D64_BLOCK, 0, st>>>(A, J);
        k_d64_adj_springs<1><<<g, D64_BLOCK, 0, st>>>(A, J);
    }
}

__global__ void k_d64_from_f4(const float4* __restrict__ in, D4* __restrict__ out, u32 voff, u32 n) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { const float4 q = in[voff + i]; out[i] = D4{(double)q.x, (double)q.y, (double)q.z, 0.0}; }
}
__global__ void k_d64_from_f3(const float* __restrict__ in, D4* __restrict__ out, u32 n) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = D4{(double)in[3 * i], (double)in[3 * i + 1], (double)in[3 * i + 2], 0.0};
}
__global__ void k_d64_from_d3(const double* __restrict__ in, D4* __restrict__ out, u32 n) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = D4{in[3 * i], in[3 * i + 1], in[3 * i + 2], 0.0};
}
__global__ void k_d64_to_f3(const D4* __restrict__ in, float* __restrict__ out, u32 n) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { const D4 q = in[i]; out[3 * i] = (float)q.x; out[3 * i + 1] = (float)q.y; out[3 * i + 2] = (float)q.z; }
}
__global__ void k_d64_to_d3(const D4* __restrict__ in, double* __restrict__ out, u32 n) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { const D4 q = in[i]; out[3 * i] = q.x; out[3 * i + 1] = q.y; out[3 * i + 2] = q.z; }
}
__global__ void k_d64_widen(const float* __restrict__ in, double* __restrict__ out, u32 n) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (double)in[i];
}
__global__ void k_d64_narrow(const double* __restrict__ in, float* __restrict__ out, u32 n) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)in[i];
}

}  // namespace ys
