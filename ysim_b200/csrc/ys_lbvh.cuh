// ys_lbvh.cuh -- linear BVH over triangles: Morton codes, Karras topology,
// swept refit.  Node layout and slot numbering follow the reference
// (bvh.hpp:148-177, bvh.metal:260-393): internal nodes [0, N-2] with the root
// at slot 0, leaves at [N-1, 2N-2].
#pragma once
#include <cstring>

#include "ys_common.cuh"
#include "ys_scan.cuh"

namespace ys {

// Order-preserving float <-> uint map so atomicMin/atomicMax on uints give
// float min/max (the min/max of a set does not depend on order).
__device__ __forceinline__ u32 ford(float f) {
    u32 u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ __forceinline__ float funord(u32 u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
#else
    u32 r = (u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u;
    float f; memcpy(&f, &r, 4); return f;
#endif
}

// expandBits (bvh.metal:26-32): the 10 low bits of v spread to every third bit.
__device__ __forceinline__ u32 expand_bits(u32 v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

// One tree to refit: leaves are recomputed from positions (optionally swept by
// v*dt) and combined bottom-up.  Positions/velocities are float4 (padded) or
// packed float3 (reference layout) depending on which pointer is set.
struct RefitJob {
    Node* nodes;            // 2N-1 nodes
    const i32* parent;      // 2N-1: largest internal node claiming the node as a child (-1: none)
    const u32* claimOff;    // claimant lists: node c's are claims[claimOff[c-1] (0 for c = 0) .. claimOff[c])
    const i32* claims;      // 2N-2 internal node ids
    u32* visits;            // N-1 per-internal-node arrival counters
    const u32* facets;      // 3 local vertex ids per face (packed)
    const float4* x4;       // positions (float4) or nullptr
    const float4* v4;
    const float* x3;        // positions (packed xyz) or nullptr
    const float* v3;
    u32 voff;               // vertex offset of this mesh in x4/v4
    u32 n;                  // leaves
    u32 leafBase;           // prefix of leaves over jobs
    float dt;
    u32 swept;
    float selfMargin;       // > 0: also reduce the H1 grid extent into *maxExt
    u32* maxExt;            // float bits, atomicMax (positive floats order as ints)
    // 4-wide form (cube layout): when set the refit fills the wide nodes'
    // child slots and the binary root box instead of the binary nodes
    Wide4* w4;
    const int2* leafW;      // per leaf: (wide node, slot)
    u32* warrive;           // per wide node: arrivals this refit (self-resetting)
    // root only: no query descends this tree, only its root box is used (the
    // inter-object cull); the leaves (face i for thread i, the tree need not
    // be built) are reduced straight into rootAcc (3 ordered-int minima, then
    // 3 maxima) and launch_refit_roots writes the root node and resets
    // rootAcc to (~0, ~0, ~0, 0, 0, 0) for the next refit.
    u32 rootOnly;
    u32* rootAcc;
    u32 nVert;              // vertices of the mesh (vertex form of the root box)
    // level-synchronous 4-wide refit: the leaf kernel (face order) only
    // writes each leaf box into its slot (leafWf); launch_refit_levels then
    // combines the wide nodes height by height
    u32 levels;
    const int2* leafWf;     // per face: (wide node, slot)
    const u32* wcount;      // number of wide nodes of this tree
    u32* hacc;              // per wide node: height (1 = leaf children only)
    // face positions (or null): per face its three vertices' current
    // positions, each float4 carrying the mesh-local vertex id in w, written
    // by the leaf pass for the queries that test the face
    float4* fpos;
    // range refit of the 4-wide form (with levels; leafBase a multiple of
    // 256): the leaf pass runs in sorted-leaf order (idx: the face of each
    // sorted leaf), writes each leaf box into its binary leaf node and its
    // wide slot (leafW) and the boxes of every 16- and 256-leaf block (bb16 /
    // bb256, indexed by (leafBase + leaf) / 16 and / 256);
    // launch_refit_ranges then gives every internal wide child its slot box,
    // and the tree its root box, as the union of the leaves of a sorted-leaf
    // range (wrange), from the block boxes.
    u32 ranges;
    const u32* idx;
    // range mode, optional: per sorted leaf its face's three vertex ids and
    // the face id (w), written at the build (one coalesced load in place of
    // the face index and the facet)
    const uint4* lvid;
    Node* bb16;
    Node* bb256;
    uint2* wrange;          // per wide node: (first, last) sorted leaf under it
    // the wide nodes whose range lies in one 256-leaf block, per block (index
    // (leafBase + leaf) / 256): (parent, slot, first, last) records
    // blkEnt[blkOff[b] .. blkOff[b + 1]); the leaf pass's block fills their
    // slots from its leaf boxes in shared memory
    const uint4* blkEnt;
    const u32* blkOff;
};

// Scene box of a mesh (min/max over all its vertices) into box[6] (float
// bits stored via ordered-int atomics; call box_init first).
void launch_box_init(u32* box, cudaStream_t s);
void launch_box(const float4* x4, const float* x3, u32 voff, u32 nV, u32* box, cudaStream_t s);
// Morton code per face from the scene box (fillMortons_Tri, bvh.metal:42-63);
// cube = one scale for all axes (the box's largest width) instead of per axis.
void launch_morton(const float4* x4, const float* x3, u32 voff, const u32* facets, u32 nF, const u32* box, u32* codes,
                   u32* idx, cudaStream_t s, bool cube = false);
// Karras topology (buildTree_Tri, bvh.metal:352-393); zeroes visit counters.
// Runs of three or more equal Morton codes make the reference's topology
// inconsistent (findSplit splits them at the midpoint, bvh.metal:204, while
// determineRange orders them by index): a node can then be claimed as a child
// by several internal nodes, or by none.  Child arrays stay exactly the
// reference's; parent keeps the largest claimant (what a serial build loop
// leaves behind) and the claimant lists (claimOff, 2N entries; claims, 2N - 2)
// hold every claimant, so the refit reaches all of them.
// consistent = true splits runs of equal codes by the (code, index) key that
// determineRange already orders them by, so every node has one parent (the
// cube layout); false keeps the reference's midpoint split.
size_t karras_scratch_bytes(u32 n);
// Optional outputs of a Karras build for the range refit: per internal node
// its sorted-leaf range, and the nodes whose range leaves the 256-leaf block of
// their own index, in big (ranges under BIN_RANGE_HUGE leaves, count[0]) or
// huge (count[1]); both lists need n entries.  range = null: none, and the
// claimant lists are built instead (with ranges they are not: nothing climbs).
//
// With the midpoint split, a node over one run of three or more equal codes
// reaches only some leaves of its range, some of them twice.  Every other
// node splits as in the consistent tree, so its box is the union of its range
// over the leaves that the topmost node of each run reaches.  runs gets the nodes
// inside such runs (n entries, count[2]); their boxes are followed through
// their children.  count[3] is the longest run; count has 4 words.
// launch_run_reach then clears the bits of the other leaves in reach (all
// ones before, n bits; null: no run).
static constexpr u32 BIN_RANGE_HUGE = 16384;
// Runs up to this length are followed node by node; with a longer one the
// tree is climbed (a node's thread visits its part of the run).
static constexpr u32 BIN_RUN_MAX = 64;
struct BinRanges {
    uint2* range = nullptr;
    u32* big = nullptr;
    u32* huge = nullptr;
    u32* runs = nullptr;
    u32* count = nullptr;
};
void launch_run_reach(const Node* nodes, u32 n, const uint2* range, const u32* codes, const u32* runs, u32 nruns,
                      u32* reach, cudaStream_t s);
// The child words of the leaves (launch_karras leaves them out with ranges).
void launch_leaf_nodes(const u32* idx, u32 n, Node* nodes, cudaStream_t s);
// Claimant lists of a built tree (for the climb).
cudaError_t launch_claims(const Node* nodes, u32 n, u32* claimOff, i32* claims, void* scratch, cudaStream_t s);
cudaError_t launch_karras(const u32* codes, const u32* idx, u32 n, Node* nodes, i32* parent, u32* claimOff,
                          i32* claims, u32* visits, void* scratch, cudaStream_t s, bool consistent = false,
                          BinRanges R = BinRanges());
// Range refit of a binary tree built with BinRanges (J: nodes,
// facets, positions (and velocities when swept), n; bb16 / bb256 with
// n / 16 + 1 and n / 256 + 1 boxes): leaf pass, then the big and huge nodes.
// With rank (each face's sorted-leaf position) and lbox (2 float4 per leaf) a
// face-order pass computes the leaf boxes first, so the leaf pass reads them
// in order instead of gathering facets and vertices; *nan becomes nonzero when
// a leaf box has a NaN (the unions leave NaN out, a climb's tinym::min keeps
// it or not by operand order).  A minimum of zeros of both signs is -0 in a
// union and the first operand's in a climb, a maximum +0; the values are equal.
void launch_refit_bin(const RefitJob& J, const uint2* range, const u32* big, u32 nbig, const u32* huge, u32 nhuge,
                      const u32* rank, float4* lbox, cudaStream_t s, const u32* runs = nullptr, u32 nruns = 0,
                      const u32* reach = nullptr, u32* nan = nullptr);
// lvid[i] = (facet of idx[i], idx[i]) for the sorted faces of a build.
void launch_leaf_vids(const u32* idx, const u32* facets, u32 n, uint4* lvid, cudaStream_t s);
// rank[idx[i]] = i for the sorted face indices of a build.
void launch_leaf_rank(const u32* idx, u32 n, u32* rank, cudaStream_t s);
// Apetrei build (agglomerativeBuild_Tri + agglomerativeSwapRoot,
// bvh.metal:884-1199) of sorted (code, index) pairs: topology, leaf boxes
// from the current positions and every internal box in one pass, the root
// moved to slot 0, claimant lists filled as launch_karras does, visit
// counters left even.  Its tree is consistent for any input (runs of equal
// codes split by index).  aggScratch holds apetrei_scratch_bytes(n).
size_t apetrei_scratch_bytes(u32 n);
cudaError_t launch_apetrei(const float4* x4, const float* x3, u32 voff, const u32* facets, const u32* codes,
                           const u32* idx, u32 n, Node* nodes, i32* parent, u32* claimOff, i32* claims, u32* visits,
                           void* scanScratch, void* aggScratch, u32* status, cudaStream_t s);
// 4-wide form of a consistent binary tree of n leaves: internal nodes at even
// depth become wide nodes (numbered by an exclusive scan), their children and
// grandchildren their slots.  w4 and warrive need max(n - 1, 1) entries,
// leafW n, scratch wide_build_scratch_bytes(n).  Boxes are filled by a refit.
size_t wide_build_scratch_bytes(u32 n);
cudaError_t launch_wide_build(const Node* nodes, const i32* parent, u32 n, Wide4* w4, int2* leafW, int2* leafWf,
                              u32* warrive, u32* wcount, void* scratch, cudaStream_t s);

// Level lists of the 4-wide trees of a job table (jobs with w4 and levels):
// heights by a climb, then every wide node into the list of its height as
// (node, job).  hcount / hoff: MAX_LEVELS + 1 entries; the host reads hcount
// to size the level launches.
static constexpr u32 MAX_LEVELS = 64;
void launch_wide_heights(const RefitJob* jobsDev, u32 numJobs, u32 totalLeaves, u32* status, cudaStream_t s);
void launch_level_count(const RefitJob* jobsDev, u32 numJobs, u32 totalLeaves, u32* hcount, u32* status,
                        cudaStream_t s);
void launch_level_fill(const RefitJob* jobsDev, u32 numJobs, u32 totalLeaves, const u32* hoff, u32* hcursor,
                       uint2* list, cudaStream_t s);
// Per substep, after launch_refit wrote the leaf slots: levels 1 .. split-1
// one launch each (hostOff[h] .. hostOff[h+1] of list), then levels split ..
// top in one block, level by level.
// Query points in Morton order (over their own box): idx[k] is the point of
// sorted slot k.  The standalone point queries run one thread per sorted
// slot, so neighbouring threads query neighbouring points and share the tree
// nodes / hash buckets they read.  Buffers grow on demand.
struct QueryOrder {
    u32* codes = nullptr;
    u32* idx = nullptr;
    void* scratch = nullptr;
    u32* box = nullptr;
    u32 cap = 0;
};
// From these sizes on the order pays for its sort (measured on uniform
// points: LBVH query at 4M 1.64 -> 1.38 ms and 16M 18.3 -> 11.4 ms, at 1M
// 0.32 -> 0.37 ms; hash query at 16M 44.0 -> 40.2 ms, at 4M 3.48 -> 3.60 ms)
static constexpr u32 QUERY_ORDER_MIN_LBVH = 1u << 21;
static constexpr u32 QUERY_ORDER_MIN_HASH = 1u << 23;
cudaError_t query_order(QueryOrder& o, const float* qx, u32 n, cudaStream_t s);
void query_order_free(QueryOrder& o);

// The range refit's second pass (after launch_refit) over the records
// (parent, slot | job << 2, first, last) of the wide nodes whose range spans
// more than one 256-leaf block: nmed at the front of big (8 lanes each), nhuge
// at its back (ranges over 16384 leaves, a block each), then a block per job
// for its root box.
void launch_refit_ranges(const RefitJob* jobsDev, u32 numJobs, const uint4* big, u32 bigCap, u32 nmed, u32 nhuge,
                         cudaStream_t s);
// The range refit's node records after launch_wide_heights: each non-root
// wide node of the range jobs goes to the list of the 256-leaf block holding
// its range, or to big (bigCap records: medium ones from the front, huge
// ones from the back).  blkCnt (numBlocks + 1 entries) is used as scratch;
// blkOff gets the per-block offsets; bigCnt[0] / [1] the medium and huge
// counts.  Scratch of scan_scratch_bytes(numBlocks + 1).
cudaError_t launch_range_lists(const RefitJob* jobsDev, u32 numJobs, u32 totalLeaves, u32* blkCnt, u32* blkOff,
                               uint4* blkEnt, uint4* big, u32 bigCap, u32* bigCnt, void* scanScratch,
                               cudaStream_t s);
// Allow the top-levels refit kernel its staging shared memory (once, before
// the first launch_refit_levels; not during a stream capture).
cudaError_t refit_levels_prepare();
void launch_refit_levels(const RefitJob* jobsDev, const uint2* list, const u32* hoffDev, const u32* hostOff,
                         u32 top, cudaStream_t s);
// ---- sorted-leaf groups: what the fused substep descends in the cube layout.
// The leaves of a tree in sorted (Morton) order, and the boxes of every run
// of 32, 1024 and 32768 of them: a 32-wide tree without child pointers, in
// which a warp tests the 32 children of a node with one coalesced load.  A
// box is two float4 (minimum, maximum); the runs of 32768 ("tops") and the
// whole-mesh boxes ("roots") are 8 words each, six of them order-preserving
// integers that only ever grow (~ford(min), ford(max); 0 = empty), so that
// blocks reduce into them by atomicMax after one clear.
//
// A job is one mesh: GJ_KEY writes the key boxes of the CPU-hash self rows
// (AABB +- margin, an empty box for a face with a non-finite corner), GJ_BOX
// the boxes of the point queries (swept by v dt with GJ_SWEPT), each with its
// own runs; GJ_REC the records of the candidate tests, per leaf {corner 0,
// face}, {corner 1, -}, {corner 2, -}, {unit normal, 0 if the face is
// degenerate}; GJ_ROOT the root box by faces; GJ_VERTS (alone) the root box
// by vertices, for a mesh whose every vertex is on a face (the same set of
// points then).
enum : u32 { GJ_KEY = 1, GJ_BOX = 2, GJ_SWEPT = 4, GJ_REC = 8, GJ_ROOT = 16, GJ_VERTS = 32 };
struct GroupJob {
    const uint4* lvid;     // per sorted leaf (vertex ids, face), or null: leaf i is face i of facets
    const u32* facets;
    u32* maxExt;           // GJ_KEY: the H1 grid extent
    u32 flags, voff, n;    // n leaves (GJ_VERTS: vertices)
    u32 block0;            // first block of the launch working on this job
    u32 keyL0, keyTop, boxL0, boxTop, rec, root;
    float dt, margin;
};
struct GroupBufs {
    float4 *l0, *l1, *l2;  // boxes of leaves, runs of 32 and of 1024 (pairs; a tree's first leaf is a multiple of 1024)
    float4* rec;           // 4 per leaf
    u32 *top, *root;       // 8 words per run of 32768 / per mesh
    unsigned long long* ctr;  // the launch sets the first nctr of these to 0
    u32 nctr;
};
static constexpr u32 GROUP_BLOCK = 1024;    // leaves (or vertices) per block
static constexpr u32 GROUP_TOP = 32768;
__device__ __forceinline__ void group_acc_box(const u32* a, float lo[3], float hi[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const u32 l = a[k], h = a[3 + k];
        lo[k] = l ? funord(~l) : __int_as_float(0x7F800000);
        hi[k] = h ? funord(h) : -__int_as_float(0x7F800000);
    }
}
// One launch over the jobs' blocks (blkJob: the job of each block).  The tops
// and roots the jobs write were cleared before.
void launch_refit_groups(const GroupJob* jobs, const u32* blkJob, u32 numBlocks, const float4* x, const float4* v,
                         GroupBufs B, cudaStream_t s);

// Leaves + bottom-up for every job (jobs in device memory, jobsHost mirrors
// them for the launch size).
void launch_refit(const RefitJob* jobsDev, u32 numJobs, u32 totalLeaves, u32* status, cudaStream_t s);
// Root boxes of the root-only jobs from their accumulators (after launch_refit).
void launch_refit_roots(const RefitJob* jobsDev, u32 numJobs, cudaStream_t s);
// Root boxes from vertices, for meshes whose every vertex belongs to a face
// (then the union of the swept leaf boxes is the union of {x, x + v dt} over
// the vertices): one block per chunk (job, first vertex) of ROOT_CHUNK
// vertices, then launch_refit_roots on the same jobs.
static constexpr u32 ROOT_CHUNK = 512;
void launch_root_boxes(const RefitJob* jobsDev, u32 numJobs, const uint2* chunks, u32 numChunks, cudaStream_t s);

}  // namespace ys
