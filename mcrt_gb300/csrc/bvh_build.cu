// bvh_build.cu — GPU binned SAH BVH builder, compact-layout conversion, scan.
//
// The builder is a level-synchronous parallel restatement of the reference's
// recursive CPU builder (src/mesh.rs:82-291 with src/bvh.rs:87-463):
//   * primitive bounds: the triangle AABB padded by 1e-4 on degenerate axes
//     (mesh.rs:282-291, bvh.rs:194-207), centroid = (min+max)*0.5;
//   * a node with <= 4 primitives is a leaf (bvh.rs:32, :302);
//   * otherwise 8 bins per axis over the node's centroid bounds (axes with
//     extent < 1e-8 skipped), left-prefix / right-suffix sweep, half-area SAH
//     cost (Ct = 0, Ci = 1) against a parent area clamped to 1e-8, a split is
//     taken only when strictly cheaper than the leaf (bvh.rs:388-463);
//   * the split sends the primitives of bins 0..s left.  Binning is monotone in
//     the centroid, so this is exactly the set of the l smallest centroids the
//     reference takes after sorting (bvh.rs:303-306);
//   * pre-order layout, left child = i+1, right = right_or_offset, leaves
//     reference consecutive ranges of the ordered triangle list.
// All arithmetic is the same IEEE sequence (compiled with -fmad=false), so the
// output nodes equal the reference builder's bit for bit; only the order of the
// primitives inside a leaf may differ (the partition here is stable, starting
// from the Morton order of the centroids; the reference uses an unstable sort).
#include <algorithm>
#include <utility>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "traverse.cuh"

namespace mcrt {

// ------------------------------------------------------------------ scan
namespace {
constexpr uint32_t kScanBlock = 1024;   // elements per block (256 threads x 4)

__global__ void k_scan_block(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *block_sums) {
    __shared__ uint32_t sh[256];
    uint32_t base = blockIdx.x * kScanBlock + threadIdx.x * 4;
    uint32_t v[4];
    uint32_t local = 0;
    for (int k = 0; k < 4; ++k) {
        uint32_t idx = base + k;
        v[k] = idx < n ? in[idx] : 0u;
        local += v[k];
    }
    sh[threadIdx.x] = local;
    __syncthreads();
    for (uint32_t off = 1; off < 256; off <<= 1) {
        uint32_t t = threadIdx.x >= off ? sh[threadIdx.x - off] : 0u;
        __syncthreads();
        sh[threadIdx.x] += t;
        __syncthreads();
    }
    uint32_t run = sh[threadIdx.x] - local;   // exclusive prefix of this thread
    for (int k = 0; k < 4; ++k) {
        uint32_t idx = base + k;
        if (idx < n) out[idx] = run;
        run += v[k];
    }
    if (threadIdx.x == 255 && block_sums) block_sums[blockIdx.x] = sh[255];
}

__global__ void k_scan_add(uint32_t *out, uint32_t n, const uint32_t *block_offsets) {
    uint32_t idx = blockIdx.x * kScanBlock + threadIdx.x;
    uint32_t add = block_offsets[blockIdx.x];
    for (int k = 0; k < 4; ++k, idx += 256)
        if (idx < n) out[idx] += add;
}
}  // namespace

size_t scan_tmp_words(uint32_t n) {
    size_t words = 0;
    while (n > kScanBlock) {
        n = (n + kScanBlock - 1) / kScanBlock;
        words += 2 * (size_t)n;
    }
    return words + 2;
}

void exclusive_scan_u32(const uint32_t *d_in, uint32_t *d_out, uint32_t n, uint32_t *d_tmp, cudaStream_t st) {
    if (n == 0) return;
    uint32_t nb = (n + kScanBlock - 1) / kScanBlock;
    if (nb == 1) {
        k_scan_block<<<1, 256, 0, st>>>(d_in, d_out, n, nullptr); ::mcrt::note_launch();
        return;
    }
    uint32_t *sums = d_tmp;
    uint32_t *offs = d_tmp + nb;
    k_scan_block<<<nb, 256, 0, st>>>(d_in, d_out, n, sums); ::mcrt::note_launch();
    exclusive_scan_u32(sums, offs, nb, d_tmp + 2 * (size_t)nb, st);
    k_scan_add<<<nb, 256, 0, st>>>(d_out, n, offs); ::mcrt::note_launch();
}

// ------------------------------------------------------------------ float atomics
namespace {
// (decided by the sign bit: -0 is below +0 and must not be compared as the integer INT_MIN)
__device__ __forceinline__ void atomic_min_f(float *a, float v) {
    if (__float_as_int(v) >= 0) atomicMin(reinterpret_cast<int *>(a), __float_as_int(v));
    else atomicMax(reinterpret_cast<unsigned *>(a), __float_as_uint(v));
}
__device__ __forceinline__ void atomic_max_f(float *a, float v) {
    if (__float_as_int(v) >= 0) atomicMax(reinterpret_cast<int *>(a), __float_as_int(v));
    else atomicMin(reinterpret_cast<unsigned *>(a), __float_as_uint(v));
}

// Order-preserving map of floats onto unsigned integers (the order the float
// atomics above use: -0 below +0), so min / max reduce as integers (redux.sync).
__device__ __forceinline__ unsigned f2ord(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
constexpr unsigned kOrdPosInf = 0xff800000u;     // f2ord(+inf): empty minimum
constexpr unsigned kOrdNegInf = 0x007fffffu;     // f2ord(-inf): empty maximum
constexpr unsigned kFull = 0xffffffffu;

constexpr int kBins = 8;
constexpr uint32_t kLeafMax = 4;
constexpr int kBinStride = 7;                    // count, min xyz, max xyz
constexpr int kTaskBinWords = 3 * kBins * kBinStride;

struct Aabb { float mn[3], mx[3]; };
__device__ __forceinline__ Aabb aabb_empty() {
    Aabb a;
    for (int i = 0; i < 3; ++i) { a.mn[i] = __int_as_float(0x7f800000); a.mx[i] = __int_as_float(0xff800000); }
    return a;
}
__device__ __forceinline__ Aabb aabb_union(const Aabb &a, const Aabb &b) {
    Aabb r;
    for (int i = 0; i < 3; ++i) { r.mn[i] = fminf(a.mn[i], b.mn[i]); r.mx[i] = fmaxf(a.mx[i], b.mx[i]); }
    return r;
}
__device__ __forceinline__ float half_area(const Aabb &a) {          // bvh.rs:168-175
    float d0 = a.mx[0] - a.mn[0], d1 = a.mx[1] - a.mn[1], d2 = a.mx[2] - a.mn[2];
    return d0 * d1 + d1 * d2 + d0 * d2;
}

// Build state (device pointers), sized for nt primitives.
struct BuildState {
    uint32_t nt;
    float4 *pmin, *pmax, *pcen;       // per original primitive
    uint32_t *perm[2];                // position -> original id
    int32_t *ptask[2];                // position -> task (-1: in a finished leaf)
    uint32_t *flags, *scan;           // partition flags and their exclusive scan
    // tasks (per level, double-buffered)
    uint32_t *t_start[2], *t_count[2], *t_node[2];
    float *t_bounds[2];               // 6 per task
    float *t_cb;                      // centroid bounds, 6 per task (current level)
    float *t_bins;                    // kTaskBinWords per task (current level)
    int32_t *t_split;                 // per task: axis*16 + bin, or -1 (leaf)
    uint32_t *t_lcount;
    // BFS nodes
    float4 *n_min, *n_max;            // bounds
    uint32_t *n_a, *n_b;              // internal: left bfs, right bfs; leaf: start, count
    uint32_t *n_leaf;                 // 1 = leaf
    uint32_t *n_size, *n_pre;         // subtree size, pre-order index
    // Large tasks (above kSub primitives) are split level by level by the
    // whole-array passes; the tasks their splits leave at kSub primitives and
    // below go to this list and are built whole, one block each.
    uint32_t *sub_start, *sub_count, *sub_node;
    float4 *sub_rec;                  // their nodes: 3 float4 each (min, max, link | count | pre-order index), the
                                      // nodes of a subtree from index 2 * its first position
    uint32_t *counters;               // [0] large tasks of the next level, [1] bfs node count, [4] subtrees,
                                      // [8] large tasks of the current level, [9] error word (a look-back wait
                                      // gave up), [10] levels of the deepest subtree
    uint32_t *level_end;              // bfs node count at the start of each level
    // spatial order: primitives are built in the order of their centroids'
    // Morton codes (radix-sorted), so a warp's positions are neighbours
    uint32_t *rkey[2], *rval[2];      // sort keys / primitive ids (ping-pong)
    uint32_t *rhist, *roffs;          // digit counts per tile and their exclusive scan
    float4 *qmin, *qmax, *qcen;       // second set of primitive bounds: the reordering target
    // single-pass partition scan of a level (k_flag_scan): [0] tile ticket,
    // [2 + t] status of tile t:
    // flag << 32 | value (flag 1: the tile's own sum, 2: inclusive prefix)
    unsigned long long *part;
};
constexpr uint32_t kFlagThreads = 256;                     // k_flag_scan: threads per tile
constexpr uint32_t kMinFlagTile = kFlagThreads * 2;
constexpr uint32_t kLookbackPolls = 1u << 20;              // polls of one predecessor before giving up
// Subtrees up to this size are built by one block in shared memory: the
// primitives' 36 bytes, their order and the nodes take 70 KB at 1024, so three
// blocks share an SM.
constexpr uint32_t kSub = 1024;
constexpr uint32_t kSubThreads = 256, kSubWarps = kSubThreads / 32;
constexpr uint32_t kSubCoop = 256;         // within a subtree: larger tasks by the whole block, others by a warp
constexpr uint32_t kSubTasks = kSub / 5 + 4;   // a level's tasks hold more than 4 primitives each
// Below this many primitives the whole-array passes take 256 positions per block
// instead of 1024, so that there are more blocks than SMs.
constexpr uint32_t kWideBlocks = 1u << 19;
constexpr uint32_t kMaxLevels = 4096;
}  // namespace

struct BvhScratch {
    uint32_t cap = 0;
    void *mem = nullptr;
    BuildState s{};
    uint32_t *scan_tmp = nullptr;
    uint32_t *large = nullptr;  // host memory that the device writes: the large tasks that the first split left
    cudaEvent_t looked = nullptr;
    bool configured = false;   // k_subtrees' 70 KB of dynamic shared memory, set on the context's device
};

void free_bvh_scratch(BvhScratch *s) {
    if (!s) return;
    if (s->mem) cudaFree(s->mem);
    if (s->large) cudaFreeHost(s->large);
    if (s->looked) cudaEventDestroy(s->looked);
    delete s;
}

namespace {

__global__ void k_prim_bounds(const mcrt_gpu_vertex *verts, const mcrt_gpu_triangle *tris, BuildState S) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.nt) return;
    mcrt_gpu_triangle t = tris[i];
    Aabb b = aabb_empty();
    for (int k = 0; k < 3; ++k) {                                   // from_points_3, bvh.rs:113-126
        const float *p = verts[t.v[k]].position;
        for (int a = 0; a < 3; ++a) { b.mn[a] = fminf(b.mn[a], p[a]); b.mx[a] = fmaxf(b.mx[a], p[a]); }
    }
    const float EPS = 1e-4f;                                        // padded, bvh.rs:194-207
    Aabb pb;
    for (int a = 0; a < 3; ++a) { pb.mn[a] = fminf(b.mn[a], b.mx[a] - EPS); pb.mx[a] = fmaxf(b.mx[a], b.mn[a] + EPS); }
    float c[3];
    for (int a = 0; a < 3; ++a) c[a] = (pb.mn[a] + pb.mx[a]) * 0.5f;   // centroid, bvh.rs:179-185
    S.pmin[i] = make_float4(pb.mn[0], pb.mn[1], pb.mn[2], 0.0f);
    S.pmax[i] = make_float4(pb.mx[0], pb.mx[1], pb.mx[2], 0.0f);
    S.pcen[i] = make_float4(c[0], c[1], c[2], 0.0f);
    S.perm[0][i] = i;
    S.ptask[0][i] = 0;
}

// Sphere primitive bounds: Aabb::from_sphere (bvh.rs:133-143), not padded.
__global__ void k_sphere_bounds(const mcrt_gpu_sphere *sph, BuildState S) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.nt) return;
    float4 cr = *reinterpret_cast<const float4 *>(sph + i);
    float mn[3] = {cr.x - cr.w, cr.y - cr.w, cr.z - cr.w};
    float mx[3] = {cr.x + cr.w, cr.y + cr.w, cr.z + cr.w};
    float c[3];
    for (int a = 0; a < 3; ++a) c[a] = (mn[a] + mx[a]) * 0.5f;
    S.pmin[i] = make_float4(mn[0], mn[1], mn[2], 0.0f);
    S.pmax[i] = make_float4(mx[0], mx[1], mx[2], 0.0f);
    S.pcen[i] = make_float4(c[0], c[1], c[2], 0.0f);
    S.perm[0][i] = i;
    S.ptask[0][i] = 0;
}

// root bounds: one task covering everything
__global__ void k_root_init(BuildState S) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        S.t_start[0][0] = 0;
        S.t_count[0][0] = S.nt;
        S.t_node[0][0] = 0;
        for (int a = 0; a < 3; ++a) {
            S.t_bounds[0][a] = __int_as_float(0x7f800000);
            S.t_bounds[0][3 + a] = __int_as_float(0xff800000);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x < 16) S.counters[threadIdx.x] = threadIdx.x <= 1 ? 1u : 0u;   // the root
}

// A build of at most kSub primitives: the root is the one subtree.
__global__ void k_root_subtree(BuildState S) {
    S.sub_start[0] = 0;
    S.sub_count[0] = S.nt;
    S.sub_node[0] = 0;
    S.n_leaf[0] = 2u;
    S.level_end[0] = 1;
}

// Root bounds: per-thread min / max over the block's primitives, warp and block
// reductions on the ordered integers, six global atomics per block.
__global__ void __launch_bounds__(256) k_root_bounds(BuildState S, uint32_t per) {
    __shared__ unsigned sh[6];
    if (threadIdx.x < 6) sh[threadIdx.x] = threadIdx.x < 3 ? kOrdPosInf : kOrdNegInf;
    __syncthreads();
    const uint32_t first = blockIdx.x * per, end = min(first + per, S.nt);
    unsigned o[6] = {kFull, kFull, kFull, 0u, 0u, 0u};
    for (uint32_t i = first + threadIdx.x; i < end; i += 256) {
        const float4 a = S.pmin[i], b = S.pmax[i];
        o[0] = min(o[0], f2ord(a.x)); o[1] = min(o[1], f2ord(a.y)); o[2] = min(o[2], f2ord(a.z));
        o[3] = max(o[3], f2ord(b.x)); o[4] = max(o[4], f2ord(b.y)); o[5] = max(o[5], f2ord(b.z));
    }
    for (int a = 0; a < 3; ++a) {
        o[a] = __reduce_min_sync(kFull, o[a]);
        o[3 + a] = __reduce_max_sync(kFull, o[3 + a]);
    }
    if ((threadIdx.x & 31u) == 0)
        for (int a = 0; a < 3; ++a) { atomicMin(&sh[a], o[a]); atomicMax(&sh[3 + a], o[3 + a]); }
    __syncthreads();
    if (threadIdx.x < 3) atomic_min_f(&S.t_bounds[0][threadIdx.x], ord2f(sh[threadIdx.x]));
    else if (threadIdx.x < 6) atomic_max_f(&S.t_bounds[0][threadIdx.x], ord2f(sh[threadIdx.x]));
}

// ---- spatial order of the primitives
// The tree does not depend on the order the primitives start in (binning and
// the stable partition are decided by centroids alone); only the order inside
// a leaf does.  Starting from Morton order keeps the 32 positions of a warp
// neighbours in space at every level, so their bins mostly agree and the
// warp reductions above take one pass.

__device__ __forceinline__ uint32_t morton_expand10(uint32_t v) {
    v &= 1023u;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

// 30-bit Morton code of each centroid on a 1024^3 grid over the root bounds.
__global__ void k_morton(BuildState S) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.nt) return;
    const float4 c = S.pcen[i];
    const float cc[3] = {c.x, c.y, c.z};
    uint32_t q[3];
    for (int a = 0; a < 3; ++a) {
        const float lo = S.t_bounds[0][a], ext = S.t_bounds[0][3 + a] - lo;
        const float f = ext > 0.0f ? (cc[a] - lo) / ext * 1024.0f : 0.0f;
        q[a] = min(f2u_sat(f), 1023u);
    }
    S.rkey[0][i] = (morton_expand10(q[0]) << 2) | (morton_expand10(q[1]) << 1) | morton_expand10(q[2]);
    S.rval[0][i] = i;
}

constexpr uint32_t kRadixTile = 2048;      // keys per block of a radix pass (256 threads x 8 rounds)

// Digit counts of one tile, stored digit-major (digit * tiles + tile) so that
// their exclusive scan is each tile's output offset per digit.
__global__ void __launch_bounds__(256) k_radix_hist(const uint32_t *keys, uint32_t n, int shift, uint32_t tiles,
                                                    uint32_t *hist) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * kRadixTile;
    for (uint32_t k = threadIdx.x; k < kRadixTile; k += 256) {
        const uint32_t i = base + k;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// Stable scatter of one tile by its digit: rounds of 256 keys in tile order;
// within a round, a key's rank = the tile's running offset of its digit + the
// counts of earlier warps + the lanes before it with the same digit.
__global__ void __launch_bounds__(256) k_radix_scatter(const uint32_t *kin, const uint32_t *vin, uint32_t n, int shift,
                                                       uint32_t tiles, const uint32_t *offs, uint32_t *kout,
                                                       uint32_t *vout) {
    __shared__ uint32_t wcnt[8][256];
    __shared__ uint32_t wpre[8][256];
    __shared__ uint32_t run[256];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    for (int k = 0; k < 8; ++k) wcnt[k][threadIdx.x] = 0;
    run[threadIdx.x] = offs[threadIdx.x * tiles + blockIdx.x];
    __syncthreads();
    const uint32_t base = blockIdx.x * kRadixTile;
    const unsigned lanes_below = (1u << lane) - 1u;
    for (uint32_t r = 0; r < kRadixTile / 256; ++r) {
        const uint32_t i = base + r * 256 + threadIdx.x;
        const bool valid = i < n;
        uint32_t key = 0, val = 0, d = 256;             // 256: no key (its own group)
        if (valid) { key = kin[i]; val = vin[i]; d = (key >> shift) & 255u; }
        const unsigned peers = __match_any_sync(kFull, d);
        const uint32_t prank = __popc(peers & lanes_below);
        if (valid && prank == 0) wcnt[w][d] = __popc(peers);
        __syncthreads();
        {
            const uint32_t dd = threadIdx.x;             // one digit per thread: prefix over the warps
            uint32_t acc = run[dd];
            for (int k = 0; k < 8; ++k) {
                const uint32_t c = wcnt[k][dd];
                wpre[k][dd] = acc;
                acc += c;
                wcnt[k][dd] = 0;
            }
            run[dd] = acc;
        }
        __syncthreads();
        if (valid) {
            const uint32_t pos = wpre[w][d] + prank;
            kout[pos] = key;
            vout[pos] = val;
        }
    }
}

// Primitive bounds into Morton order; positions start as the identity of that order.
__global__ void k_reorder(BuildState S) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= S.nt) return;
    const uint32_t id = S.rval[0][j];
    S.qmin[j] = S.pmin[id];
    S.qmax[j] = S.pmax[id];
    S.qcen[j] = S.pcen[id];
    S.perm[0][j] = j;
    S.ptask[0][j] = 0;
}

// Output order: the primitive ids of the final positions (Morton index -> id).
__global__ void k_final_order(const uint32_t *perm, const uint32_t *sorted_ids, uint32_t n, uint32_t *out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = sorted_ids[perm[i]];
}

// The start of a level: its number of large tasks, a fresh count of their
// large children, and the node count.  One thread.
__device__ __forceinline__ void level_advance(BuildState &S, uint32_t level) {
    S.counters[8] = S.counters[0];
    S.counters[0] = 0;
    S.level_end[level] = S.counters[1];
}

// The start of a level with large tasks, in one launch: level_advance, the
// status words of the level's partition scan zeroed (n_part), and the large
// tasks' centroid bounds and bins set to empty.
// ntasks: at least the number of large tasks, which goes to *large when given.
__global__ void k_task_reset(BuildState S, uint32_t level, uint32_t ntasks, uint32_t n_part, uint32_t *large) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        if (large) *large = S.counters[0];
        level_advance(S, level);
    }
    if (i < n_part) S.part[i] = 0ull;
    if (i >= ntasks * (6 + kTaskBinWords)) return;
    uint32_t t = i / (6 + kTaskBinWords), k = i % (6 + kTaskBinWords);
    if (k < 6) {
        S.t_cb[6 * t + k] = __int_as_float(k < 3 ? 0x7f800000 : 0xff800000);
    } else {
        uint32_t w = k - 6;
        uint32_t f = w % kBinStride;
        float v = f == 0 ? 0.0f : __int_as_float(f < 4 ? 0x7f800000 : 0xff800000);
        S.t_bins[(size_t)t * kTaskBinWords + w] = v;
    }
}

// First and last position of a block; the block's task if every position in
// between belongs to it (tasks are contiguous ranges, so the ends decide), else -1.
__device__ __forceinline__ int block_single_task(const BuildState &S, int cur, uint32_t first, uint32_t end) {
    const int t0 = S.ptask[cur][first], t1 = S.ptask[cur][end - 1];
    return (t0 == t1 && t0 >= 0) ? t0 : -1;
}

// Centroid bounds per task.  Lanes reduce first (one pass per distinct task in
// the warp, redux.sync on the ordered integers); a block inside one task
// combines its warps in shared memory and issues six global atomics.
__global__ void __launch_bounds__(256) k_centroid_bounds(BuildState S, int cur, uint32_t per) {
    __shared__ unsigned sh[6];
    __shared__ int block_task;
    const uint32_t first = blockIdx.x * per;
    const uint32_t end = min(first + per, S.nt);
    const uint32_t lane = threadIdx.x & 31u;
    if (threadIdx.x == 0) block_task = block_single_task(S, cur, first, end);
    if (threadIdx.x < 6) sh[threadIdx.x] = threadIdx.x < 3 ? kOrdPosInf : kOrdNegInf;
    __syncthreads();
    const int bt = block_task;
    if (bt >= 0) {
        unsigned o[6] = {kFull, kFull, kFull, 0u, 0u, 0u};
        for (uint32_t i = first + threadIdx.x; i < end; i += 256) {
            const float4 c = S.pcen[S.perm[cur][i]];
            const unsigned q[3] = {f2ord(c.x), f2ord(c.y), f2ord(c.z)};
            for (int a = 0; a < 3; ++a) { o[a] = min(o[a], q[a]); o[3 + a] = max(o[3 + a], q[a]); }
        }
        for (int a = 0; a < 3; ++a) {
            o[a] = __reduce_min_sync(kFull, o[a]);
            o[3 + a] = __reduce_max_sync(kFull, o[3 + a]);
        }
        if (lane == 0)
            for (int a = 0; a < 3; ++a) { atomicMin(&sh[a], o[a]); atomicMax(&sh[3 + a], o[3 + a]); }
        __syncthreads();
        if (threadIdx.x < 3) atomic_min_f(&S.t_cb[6 * bt + threadIdx.x], ord2f(sh[threadIdx.x]));
        else if (threadIdx.x < 6) atomic_max_f(&S.t_cb[6 * bt + threadIdx.x], ord2f(sh[threadIdx.x]));
        return;
    }
    for (uint32_t base = first + (threadIdx.x & ~31u); base < end; base += 256) {   // warp-uniform
        const uint32_t i = base + lane;
        const int task = i < end ? S.ptask[cur][i] : -1;
        float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (task >= 0) c = S.pcen[S.perm[cur][i]];
        const unsigned q[3] = {f2ord(c.x), f2ord(c.y), f2ord(c.z)};
        unsigned pending = __ballot_sync(kFull, task >= 0);
        while (pending) {
            const int leader = __ffs(pending) - 1;
            const int lt = __shfl_sync(kFull, task, leader);
            const bool mine = task == lt;
            pending &= ~__ballot_sync(kFull, mine);
            unsigned r[6];
            for (int a = 0; a < 3; ++a) {
                r[a] = __reduce_min_sync(kFull, mine ? q[a] : kFull);
                r[3 + a] = __reduce_max_sync(kFull, mine ? q[a] : 0u);
            }
            if ((int)lane == leader)
                for (int a = 0; a < 3; ++a) {
                    atomic_min_f(&S.t_cb[6 * lt + a], ord2f(r[a]));
                    atomic_max_f(&S.t_cb[6 * lt + 3 + a], ord2f(r[3 + a]));
                }
        }
    }
}

__device__ __forceinline__ uint32_t bin_of(float c, float cmin, float len) {
    float t = (c - cmin) / len;                                     // bvh.rs:412-415
    uint32_t b = f2u_sat(t * (float)kBins);
    return b > (uint32_t)(kBins - 1) ? (uint32_t)(kBins - 1) : b;
}

// One warp's contribution to the bins of one axis: lanes with the same
// (task, bin) key form a group (match.any) and reduce within it (redux.sync
// on the group's mask, the ordered integers); the group's first lane adds the
// result — into the shared bins `sh` (ordered-integer form) when given, else
// into the task's global bins.
__device__ __forceinline__ void bin_axis_warp(BuildState &S, unsigned *sh, int axis, bool valid, int task,
                                              uint32_t b, const unsigned mn[3], const unsigned mx[3],
                                              uint32_t lane) {
    const unsigned key = valid ? ((unsigned)task << 3) | b : kFull;
    const unsigned peers = __match_any_sync(kFull, key);
    if (!valid) return;
    unsigned r[6];
    for (int a = 0; a < 3; ++a) {
        r[a] = __reduce_min_sync(peers, mn[a]);
        r[3 + a] = __reduce_max_sync(peers, mx[a]);
    }
    if ((int)lane != __ffs(peers) - 1) return;
    const int o = (axis * kBins + (int)b) * kBinStride;
    if (sh) {
        atomicAdd(sh + o, (unsigned)__popc(peers));
        for (int a = 0; a < 3; ++a) { atomicMin(sh + o + 1 + a, r[a]); atomicMax(sh + o + 4 + a, r[3 + a]); }
    } else {
        float *g = S.t_bins + (size_t)task * kTaskBinWords + o;
        atomicAdd(reinterpret_cast<unsigned *>(g), (unsigned)__popc(peers));
        for (int a = 0; a < 3; ++a) {
            atomic_min_f(g + 1 + a, ord2f(r[a]));
            atomic_max_f(g + 4 + a, ord2f(r[3 + a]));
        }
    }
}

// One warp's contribution to the bins of all three axes (task < 0: lane
// without a primitive).  An axis on which every lane has the same (task, bin)
// adds the warp's union of primitive bounds, reduced once for all such axes;
// the other axes reduce by groups (bin_axis_warp).  b[axis] = the lane's bin
// on each axis with an extent (0 otherwise).
__device__ __forceinline__ void bins_warp(BuildState &S, unsigned *sh, int task, float4 c, const float cb[6],
                                          const unsigned mn[3], const unsigned mx[3], uint32_t lane,
                                          uint32_t b[3]) {
    const float cc[3] = {c.x, c.y, c.z};
    bool valid[3];
    bool uni[3];
    for (int axis = 0; axis < 3; ++axis) {
        const float len = cb[3 + axis] - cb[axis];
        valid[axis] = task >= 0 && !(len < 1e-8f);
        b[axis] = valid[axis] ? bin_of(cc[axis], cb[axis], len) : 0u;
        const unsigned key = valid[axis] ? ((unsigned)task << 3) | b[axis] : kFull;
        const unsigned k0 = __shfl_sync(kFull, key, 0);
        uni[axis] = __all_sync(kFull, key == k0) && k0 != kFull;
    }
    if (uni[0] || uni[1] || uni[2]) {                 // warp-uniform; every lane holds a primitive
        unsigned r[6];
        for (int a = 0; a < 3; ++a) {
            r[a] = __reduce_min_sync(kFull, mn[a]);
            r[3 + a] = __reduce_max_sync(kFull, mx[a]);
        }
        if (lane == 0)
            for (int axis = 0; axis < 3; ++axis) {
                if (!uni[axis]) continue;
                const int o = (axis * kBins + (int)b[axis]) * kBinStride;
                if (sh) {
                    atomicAdd(sh + o, 32u);
                    for (int a = 0; a < 3; ++a) { atomicMin(sh + o + 1 + a, r[a]); atomicMax(sh + o + 4 + a, r[3 + a]); }
                } else {
                    float *g = S.t_bins + (size_t)task * kTaskBinWords + o;
                    atomicAdd(reinterpret_cast<unsigned *>(g), 32u);
                    for (int a = 0; a < 3; ++a) {
                        atomic_min_f(g + 1 + a, ord2f(r[a]));
                        atomic_max_f(g + 4 + a, ord2f(r[3 + a]));
                    }
                }
            }
    }
    for (int axis = 0; axis < 3; ++axis)
        if (!uni[axis]) bin_axis_warp(S, sh, axis, valid[axis], task, b[axis], mn, mx, lane);
}

// Bin accumulation (count and primitive-bounds union per bin and axis).  Warps
// reduce lanes of equal (task, bin) first; a block inside one task collects
// its warps in shared memory and adds the block's bins to the global ones.
__global__ void __launch_bounds__(256) k_bins(BuildState S, int cur, uint32_t per) {
    __shared__ unsigned sh[kTaskBinWords];
    __shared__ int block_task;
    const uint32_t first = blockIdx.x * per;
    const uint32_t end = min(first + per, S.nt);
    const uint32_t lane = threadIdx.x & 31u;
    if (threadIdx.x == 0) block_task = block_single_task(S, cur, first, end);
    for (int k = threadIdx.x; k < kTaskBinWords; k += blockDim.x) {
        const uint32_t f = k % kBinStride;
        sh[k] = f == 0 ? 0u : (f < 4 ? kOrdPosInf : kOrdNegInf);
    }
    __syncthreads();
    const int bt = block_task;
    unsigned *dst = bt >= 0 ? sh : nullptr;
    for (uint32_t base = first + (threadIdx.x & ~31u); base < end; base += 256) {   // warp-uniform
        const uint32_t i = base + lane;
        const int task = i < end ? S.ptask[cur][i] : -1;
        if (__all_sync(kFull, task < 0)) continue;              // leaves and small tasks only
        float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f), bmn = c, bmx = c;
        float cb[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (task >= 0) {
            const uint32_t id = S.perm[cur][i];
            c = S.pcen[id]; bmn = S.pmin[id]; bmx = S.pmax[id];
            for (int k = 0; k < 6; ++k) cb[k] = S.t_cb[6 * task + k];
        }
        const unsigned mn[3] = {f2ord(bmn.x), f2ord(bmn.y), f2ord(bmn.z)};
        const unsigned mx[3] = {f2ord(bmx.x), f2ord(bmx.y), f2ord(bmx.z)};
        uint32_t b[3];
        bins_warp(S, dst, task, c, cb, mn, mx, lane, b);
    }
    if (bt < 0) return;
    __syncthreads();
    float *g = S.t_bins + (size_t)bt * kTaskBinWords;
    for (int k = threadIdx.x; k < kTaskBinWords; k += blockDim.x) {
        const uint32_t f = k % kBinStride;
        if (f == 0) {
            if (sh[k]) atomicAdd(reinterpret_cast<unsigned *>(g + k), sh[k]);
        } else if (f < 4) {
            if (sh[k] != kOrdPosInf) atomic_min_f(g + k, ord2f(sh[k]));
        } else {
            if (sh[k] != kOrdNegInf) atomic_max_f(g + k, ord2f(sh[k]));
        }
    }
}

// ---- SAH split choice (bvh.rs:388-463): per axis, prefix unions of bins 0..s and
// suffix unions of bins 7..s+1, cost (A_l * n_l + A_r * n_r) / A_parent, taken in
// the serial order (axes ascending, s descending) and replaced only on a strictly
// smaller cost, starting from the leaf's cost n.  Evaluated by a warp, or by two or
// four groups of its lanes for small tasks: a lane holds one bin of one axis.
__device__ __forceinline__ float node_half_area(const float *tb) {
    Aabb nb;
    for (int a = 0; a < 3; ++a) { nb.mn[a] = tb[a]; nb.mx[a] = tb[3 + a]; }
    return fmaxf(half_area(nb), 1e-8f);
}

// One lane's bin of one axis: its primitives' number and box.
struct LaneBin { uint32_t n; Aabb b; };

// Adds to a lane's bin (axis, bin) those of cnt staged primitives (two float4
// each: box, then the bins of the three axes in 4 bits each) that fall into it.
__device__ __forceinline__ void bin_add(LaneBin &acc, const float4 *stage, uint32_t cnt, uint32_t axis, uint32_t bin) {
    const float inf = __int_as_float(0x7f800000);
#pragma unroll 4
    for (uint32_t i = 0; i < cnt; ++i) {
        const float4 q0 = stage[2 * i], q1 = stage[2 * i + 1];
        const bool in = ((__float_as_uint(q1.z) >> (4u * axis)) & 15u) == bin;
        const float qn[3] = {q0.x, q0.y, q0.z}, qx[3] = {q0.w, q1.x, q1.y};
        acc.n += in ? 1u : 0u;
        for (int a = 0; a < 3; ++a) {
            acc.b.mn[a] = fminf(acc.b.mn[a], in ? qn[a] : inf);
            acc.b.mx[a] = fmaxf(acc.b.mx[a], in ? qx[a] : -inf);
        }
    }
}

// A candidate split of the serial order: k = axis * 7 + 6 - bin.
struct LaneSplit {
    unsigned cost = kFull;                 // ordered cost, kFull: none
    uint32_t k = 32u, l = 0;
    Aabb lb = aabb_empty(), rb = aabb_empty();
};
// The lane's candidate (left: bins up to its own of its axis), from the bins of
// the eight lanes of the axis by a prefix and a suffix scan; kept in best when it
// is cheaper than the leaf and than best.  Same costs, bit for bit, as the serial
// sweep: the unions are the same sets, and min and max do not depend on order.
__device__ __forceinline__ void bin_candidate(const LaneBin &mine, uint32_t axis, uint32_t bin, bool flat, uint32_t n,
                                              float parent, LaneSplit &best) {
    LaneBin p = mine, q = mine;
#pragma unroll
    for (uint32_t h = 1; h < 8; h <<= 1) {
        LaneBin a, b;
        a.n = __shfl_up_sync(kFull, p.n, h, 8);
        b.n = __shfl_down_sync(kFull, q.n, h, 8);
        for (int c = 0; c < 3; ++c) {
            a.b.mn[c] = __shfl_up_sync(kFull, p.b.mn[c], h, 8); a.b.mx[c] = __shfl_up_sync(kFull, p.b.mx[c], h, 8);
            b.b.mn[c] = __shfl_down_sync(kFull, q.b.mn[c], h, 8); b.b.mx[c] = __shfl_down_sync(kFull, q.b.mx[c], h, 8);
        }
        if (bin >= h) { p.n += a.n; p.b = aabb_union(p.b, a.b); }
        if (bin + h < 8u) { q.n += b.n; q.b = aabb_union(q.b, b.b); }
    }
    Aabb rb;
    const uint32_t rc = __shfl_down_sync(kFull, q.n, 1, 8);
    for (int c = 0; c < 3; ++c) {
        rb.mn[c] = __shfl_down_sync(kFull, q.b.mn[c], 1, 8);
        rb.mx[c] = __shfl_down_sync(kFull, q.b.mx[c], 1, 8);
    }
    const float cost = (half_area(p.b) * (float)p.n + half_area(rb) * (float)rc) / parent;
    const bool ok = axis < 3u && bin < 7u && !flat && p.n != 0u && rc != 0u && cost < (float)n;
    const unsigned oc = ok ? f2ord(cost) : kFull;
    if (oc < best.cost || (oc == best.cost && oc != kFull && axis * 7u + 6u - bin < best.k)) {
        best.cost = oc;
        best.k = axis * 7u + 6u - bin;
        best.l = p.n;
        best.lb = p.b;
        best.rb = rb;
    }
}

// The cheapest candidate of a group of G lanes, ties to the earliest; every
// lane of the group gets it.  Returns whether there is one.
template <uint32_t G>
__device__ __forceinline__ bool best_split(LaneSplit &v, uint32_t lane) {
    unsigned cost = v.cost;
#pragma unroll
    for (uint32_t h = G / 2; h; h >>= 1) cost = min(cost, __shfl_xor_sync(kFull, cost, h));
    uint32_t key = v.cost == cost ? (v.k << 8) | lane : kFull;
#pragma unroll
    for (uint32_t h = G / 2; h; h >>= 1) key = min(key, __shfl_xor_sync(kFull, key, h));
    const int from = (int)(key & 31u);
    v.cost = cost;
    v.k = key >> 8;
    v.l = __shfl_sync(kFull, v.l, from);
    for (int a = 0; a < 3; ++a) {
        v.lb.mn[a] = __shfl_sync(kFull, v.lb.mn[a], from); v.lb.mx[a] = __shfl_sync(kFull, v.lb.mx[a], from);
        v.rb.mn[a] = __shfl_sync(kFull, v.rb.mn[a], from); v.rb.mx[a] = __shfl_sync(kFull, v.rb.mx[a], from);
    }
    return cost != kFull;
}

// Child tasks of a split: large (above kSub primitives) and subtrees (above the
// leaf size).
__device__ __forceinline__ uint32_t child_large(uint32_t n, uint32_t lcount) {
    return (lcount > kSub ? 1u : 0u) + (n - lcount > kSub ? 1u : 0u);
}
__device__ __forceinline__ uint32_t child_sub(uint32_t n, uint32_t lcount) {
    auto sub = [](uint32_t c) { return c > kLeafMax && c <= kSub; };
    return (sub(lcount) ? 1u : 0u) + (sub(n - lcount) ? 1u : 0u);
}
constexpr uint32_t kSubMark = 2u;                // n_leaf of a subtree's root

// Node records of a large task.  A leaf (sp < 0) keeps its range.  A split gets
// the BFS ids child0, child0 + 1 for its children; its large children get the
// task ids large0, large0 + 1 and its subtrees the list entries sub0, sub0 + 1
// (in child order).
__device__ void record_task(BuildState &S, int nxt, uint32_t start, uint32_t n, uint32_t node, int sp,
                            uint32_t lcount, const Aabb &bl, const Aabb &br, uint32_t child0, uint32_t large0,
                            uint32_t sub0) {
    if (sp < 0) {
        S.n_leaf[node] = 1; S.n_a[node] = start; S.n_b[node] = n;
        return;
    }
    S.n_leaf[node] = 0;
    const uint32_t counts[2] = {lcount, n - lcount};
    const uint32_t starts[2] = {start, start + lcount};
    const Aabb *cbx[2] = {&bl, &br};
    for (int c = 0; c < 2; ++c) {
        const uint32_t id = child0 + (uint32_t)c;
        S.n_min[id] = make_float4(cbx[c]->mn[0], cbx[c]->mn[1], cbx[c]->mn[2], 0.0f);
        S.n_max[id] = make_float4(cbx[c]->mx[0], cbx[c]->mx[1], cbx[c]->mx[2], 0.0f);
        if (counts[c] <= kLeafMax) {
            S.n_leaf[id] = 1; S.n_a[id] = starts[c]; S.n_b[id] = counts[c];
            continue;
        }
        if (counts[c] <= kSub) {
            const uint32_t k = sub0++;
            S.sub_start[k] = starts[c];
            S.sub_count[k] = counts[c];
            S.sub_node[k] = id;
            S.n_leaf[id] = kSubMark;
            continue;
        }
        S.n_leaf[id] = 0;
        const uint32_t task = large0++;
        S.t_start[nxt][task] = starts[c];
        S.t_count[nxt][task] = counts[c];
        S.t_node[nxt][task] = id;
        for (int a = 0; a < 3; ++a) {
            S.t_bounds[nxt][6 * task + a] = cbx[c]->mn[a];
            S.t_bounds[nxt][6 * task + 3 + a] = cbx[c]->mx[a];
        }
        S.n_size[id] = task;               // temporary: child node -> task id, for k_scatter
    }
    S.n_a[node] = child0;
    S.n_b[node] = child0 + 1;
}

// One warp per large task: split choice from its 24 bins, then the node records
// and the children's ids by lane 0.  (A thread per task ran the sweep in 10 us a
// level, for one task as for a thousand, and the 80,000-triangle build 0.80 ms
// instead of 0.74.)
__global__ void __launch_bounds__(128) k_split(BuildState S, int cur) {
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    if (t >= S.counters[8]) return;                       // whole warps
    const uint32_t start = S.t_start[cur][t], n = S.t_count[cur][t], node = S.t_node[cur][t];
    const uint32_t axis = lane >> 3, bin = lane & 7u;
    LaneBin mine{0u, aabb_empty()};
    bool flat = true;
    if (axis < 3u) {
        const float *q = S.t_bins + (size_t)t * kTaskBinWords + lane * kBinStride;
        mine.n = __float_as_uint(q[0]);
        for (int a = 0; a < 3; ++a) { mine.b.mn[a] = q[1 + a]; mine.b.mx[a] = q[4 + a]; }
        flat = S.t_cb[6 * t + 3 + axis] - S.t_cb[6 * t + axis] < 1e-8f;
    }
    LaneSplit best;
    bin_candidate(mine, axis, bin, flat, n, node_half_area(S.t_bounds[cur] + 6 * t), best);
    const bool split = best_split<32>(best, lane);
    if (lane != 0) return;
    const int sp = split ? (int)(best.k / 7u) * 16 + (int)(6u - best.k % 7u) : -1;
    const uint32_t large = split ? child_large(n, best.l) : 0u, sub = split ? child_sub(n, best.l) : 0u;
    const uint32_t child0 = split ? atomicAdd(S.counters + 1, 2u) : 0u;
    const uint32_t large0 = large ? atomicAdd(S.counters, large) : 0u;
    const uint32_t sub0 = sub ? atomicAdd(S.counters + 4, sub) : 0u;
    record_task(S, cur ^ 1, start, n, node, sp, best.l, best.lb, best.rb, child0, large0, sub0);
    S.t_split[t] = sp;
    if (split) S.t_lcount[t] = best.l;
}

// ------------------------------------------------------------------ subtrees
// A task of at most kSub primitives is built whole by one block: the same
// level-synchronous algorithm (centroid bounds, 8 bins per axis, the cheapest
// split, a stable partition) on primitives, order and nodes in shared memory.
// Within a level, a task above kSubCoop primitives is split by the whole block,
// one of 33 to kSubCoop by a warp, and two or four of at most 16 or 8 by a warp.
// A lane first holds a primitive and computes its bins, then it holds a bin of
// one axis and runs over the staged primitives, taking those of its bin: 18
// instructions per primitive and warp.  (Groups of lanes of equal bin by
// match.any and redux.sync on their masks, as the whole-array passes have them,
// took 12,000 cycles per 32 primitives here: each mask is its own instruction.)
//
// The smaller levels hold most of a tree's nodes.  As launches over all tasks
// of a level (a warp per task, a thread per task of at most 8) they took 1.64 of
// the 4.2 ms of the 1.3M-triangle build and 0.61 of the 1.9 ms of an 80,000
// triangle build, in 25 launches, and another 46 launches found the subtree sizes
// and pre-order indices.  Now k_subtrees takes 0.70 and 0.14 ms and the builds
// 2.54 and 0.74 ms, in 118 launches (206 before) and 94 (173).  It is bound by
// the instructions of bin_add and by a block's idle warps on a subtree's first
// and last levels; blocks of 512 threads, two to an SM, take the same time.
struct SubShared {
    float c[3][kSub], mn[3][kSub], mx[3][kSub];       // centroids and boxes by local index
    uint16_t perm[2][kSub];                           // position -> local index
    unsigned scratch[kSubWarps][256];                 // per warp: 32 staged primitives of 8 words, or bins
    uint16_t t_start[2][kSubTasks], t_count[2][kSubTasks], t_node[2][kSubTasks];
    float t_area[2][kSubTasks];                       // the tasks' half areas, clamped as the cost wants them
    uint16_t a[2 * kSub], b[2 * kSub];                // node: left child (b = 0), or first position and count
    uint16_t size[2 * kSub], pre[2 * kSub];
    uint16_t level_end[kSub + 2];
    unsigned red[6];
    uint32_t warp_left[kSubWarps];
    uint32_t n_nodes, n_tasks[2], lcount;
    uint32_t n_class[2][3];                           // tasks of at most 8, at most 16, and more primitives
    uint8_t of_class[2][3][kSubTasks];
    int split, leaf_child[2];
};
static_assert(kSubTasks < 256, "task indices are bytes");
static_assert(kTaskBinWords <= 256, "a warp's bins fit its scratch");

__device__ __forceinline__ void sub_box(const BuildState &S, size_t rec, const Aabb &b) {
    S.sub_rec[3 * rec] = make_float4(b.mn[0], b.mn[1], b.mn[2], 0.0f);
    S.sub_rec[3 * rec + 1] = make_float4(b.mx[0], b.mx[1], b.mx[2], 0.0f);
}

// Node records of a subtree's task and its children (one thread); rec0: the
// subtree's first record; *leaf0, *leaf1: whether the children are leaves.
__device__ void sub_record(const BuildState &S, SubShared &sh, int nxt, size_t rec0, uint32_t start, uint32_t n,
                           uint32_t node, int sp, uint32_t lcount, const Aabb &bl, const Aabb &br, int *leaf0,
                           int *leaf1) {
    if (sp < 0) {
        sh.a[node] = (uint16_t)start;
        sh.b[node] = (uint16_t)n;
        return;
    }
    const uint32_t kid = atomicAdd(&sh.n_nodes, 2u);
    sh.a[node] = (uint16_t)kid;
    sh.b[node] = 0;
    sub_box(S, rec0 + kid, bl);
    sub_box(S, rec0 + kid + 1, br);
    const uint32_t counts[2] = {lcount, n - lcount}, starts[2] = {start, start + lcount};
    for (int c = 0; c < 2; ++c) {
        const bool leaf = counts[c] <= kLeafMax;
        *(c ? leaf1 : leaf0) = leaf;
        if (leaf) {
            sh.a[kid + c] = (uint16_t)starts[c];
            sh.b[kid + c] = (uint16_t)counts[c];
        } else {
            const uint32_t t = atomicAdd(&sh.n_tasks[nxt], 1u);
            sh.t_start[nxt][t] = (uint16_t)starts[c];
            sh.t_count[nxt][t] = (uint16_t)counts[c];
            sh.t_node[nxt][t] = (uint16_t)(kid + c);
            sh.t_area[nxt][t] = fmaxf(half_area(c ? br : bl), 1e-8f);
            const uint32_t k = counts[c] <= 8u ? 0u : (counts[c] <= 16u ? 1u : 2u);
            sh.of_class[nxt][k][atomicAdd(&sh.n_class[nxt][k], 1u)] = (uint8_t)t;
        }
    }
}

// A primitive's bins on the three axes, 4 bits each (0 on a flat axis).
__device__ __forceinline__ uint32_t bins_of(const float c[3], const float cb[6]) {
    uint32_t bits = 0;
    for (int a = 0; a < 3; ++a) {
        const float len = cb[3 + a] - cb[a];
        if (!(len < 1e-8f)) bits |= bin_of(c[a], cb[a], len) << (4 * a);
    }
    return bits;
}
constexpr uint32_t kNoBins = 0xfffu;       // staged place without a primitive

// Tasks of at most G primitives, 32 / G of them by one warp, a group of G lanes
// each (have_task: the group has one).  A lane holds a primitive, then a bin:
// with G = 8 the bins of one axis per round, with G = 16 of two.
template <uint32_t G>
__device__ void sub_task_group(BuildState &S, SubShared &sh, int cur, bool have_task, uint32_t t, size_t rec0,
                               uint32_t lane, unsigned *scratch) {
    const uint32_t gl = lane & (G - 1u), g0 = lane & ~(G - 1u);
    const unsigned group = G == 32u ? kFull : ((1u << (G & 31u)) - 1u) << g0;
    const unsigned below = (1u << lane) - 1u;
    uint32_t start = 0, n = 0, node = 0;
    float parent = 1.0f;
    if (have_task) {
        start = sh.t_start[cur][t]; n = sh.t_count[cur][t]; node = sh.t_node[cur][t];
        parent = sh.t_area[cur][t];
    }
    const bool have = gl < n;
    const uint32_t p = have ? sh.perm[cur][start + gl] : 0u;
    float c[3], cb[6];
    for (int a = 0; a < 3; ++a) {
        c[a] = sh.c[a][p];
        const unsigned o = f2ord(c[a]);
        unsigned lo = have ? o : kFull, hi = have ? o : 0u;
#pragma unroll
        for (uint32_t h = G / 2; h; h >>= 1) {
            lo = min(lo, __shfl_xor_sync(kFull, lo, h));
            hi = max(hi, __shfl_xor_sync(kFull, hi, h));
        }
        cb[a] = ord2f(lo);
        cb[3 + a] = ord2f(hi);
    }
    const uint32_t bits = bins_of(c, cb);
    float4 *stage = reinterpret_cast<float4 *>(scratch);
    __syncwarp();
    stage[2 * lane] = make_float4(sh.mn[0][p], sh.mn[1][p], sh.mn[2][p], sh.mx[0][p]);
    stage[2 * lane + 1] = make_float4(sh.mx[1][p], sh.mx[2][p], __uint_as_float(have ? bits : kNoBins), 0.0f);
    __syncwarp();
    LaneSplit best;
    const uint32_t longest = __reduce_max_sync(kFull, n);
#pragma unroll
    for (uint32_t r = 0; r < (G == 8u ? 3u : (G == 16u ? 2u : 1u)); ++r) {
        const uint32_t axis = r * (G / 8u) + (gl >> 3), bin = gl & 7u;
        LaneBin mine{0u, aabb_empty()};
        bin_add(mine, stage + 2 * g0, longest, axis, bin);
        const float lo = axis == 0 ? cb[0] : (axis == 1 ? cb[1] : cb[2]);
        const float hi = axis == 0 ? cb[3] : (axis == 1 ? cb[4] : cb[5]);
        bin_candidate(mine, axis, bin, hi - lo < 1e-8f, n, parent, best);
    }
    const bool split = best_split<G>(best, lane);
    int leaf0 = 0, leaf1 = 0;
    if (gl == 0 && have_task)
        sub_record(S, sh, cur ^ 1, rec0, start, n, node, split ? 0 : -1, best.l, best.lb, best.rb, &leaf0, &leaf1);
    leaf0 = __shfl_sync(kFull, leaf0, (int)g0);
    leaf1 = __shfl_sync(kFull, leaf1, (int)g0);
    // stable partition; positions in a leaf are final in both orders
    uint16_t *out0 = sh.perm[cur ^ 1], *out1 = sh.perm[cur];
    const bool left = have && split && ((bits >> (4u * (best.k / 7u))) & 15u) <= 6u - best.k % 7u;
    const unsigned lm = __ballot_sync(kFull, left) & group, rm = __ballot_sync(kFull, have && !left) & group;
    if (have) {
        const uint32_t pos = !split ? start + gl : left ? start + __popc(lm & below) : start + best.l + __popc(rm & below);
        out0[pos] = (uint16_t)p;
        if (split && (left ? leaf0 : leaf1)) out1[pos] = (uint16_t)p;
    }
}

// Stages the primitive of position i (none: i >= end) in the warp's scratch.
__device__ __forceinline__ void stage_position(const SubShared &sh, const uint16_t *in, uint32_t i, uint32_t end,
                                               const float cb[6], uint32_t lane, float4 *stage) {
    const bool have = i < end;
    const uint32_t p = have ? in[i] : 0u;
    const float c[3] = {sh.c[0][p], sh.c[1][p], sh.c[2][p]};
    const uint32_t bits = bins_of(c, cb);
    __syncwarp();
    stage[2 * lane] = make_float4(sh.mn[0][p], sh.mn[1][p], sh.mn[2][p], sh.mx[0][p]);
    stage[2 * lane + 1] = make_float4(sh.mx[1][p], sh.mx[2][p], __uint_as_float(have ? bits : kNoBins), 0.0f);
    __syncwarp();
}
__device__ __forceinline__ bool axis_flat(const float cb[6], uint32_t axis) {
    const float lo = axis == 0 ? cb[0] : (axis == 1 ? cb[1] : cb[2]);
    const float hi = axis == 0 ? cb[3] : (axis == 1 ? cb[4] : cb[5]);
    return hi - lo < 1e-8f;
}

// A task of 33 to kSubCoop primitives, by one warp.
__device__ void sub_task_warp(BuildState &S, SubShared &sh, int cur, uint32_t t, size_t rec0, uint32_t lane,
                              unsigned *scratch) {
    const uint32_t start = sh.t_start[cur][t], n = sh.t_count[cur][t], node = sh.t_node[cur][t];
    const uint16_t *in = sh.perm[cur];
    uint16_t *out0 = sh.perm[cur ^ 1], *out1 = sh.perm[cur];
    const unsigned below = (1u << lane) - 1u;
    unsigned co[6] = {kFull, kFull, kFull, 0u, 0u, 0u};
    for (uint32_t i = start + lane; i < start + n; i += 32u) {
        const uint32_t p = in[i];
        for (int a = 0; a < 3; ++a) {
            const unsigned o = f2ord(sh.c[a][p]);
            co[a] = min(co[a], o);
            co[3 + a] = max(co[3 + a], o);
        }
    }
    float cb[6];
    for (int a = 0; a < 3; ++a) {
        cb[a] = ord2f(__reduce_min_sync(kFull, co[a]));
        cb[3 + a] = ord2f(__reduce_max_sync(kFull, co[3 + a]));
    }
    float4 *stage = reinterpret_cast<float4 *>(scratch);
    LaneBin mine{0u, aabb_empty()};
    for (uint32_t base = start; base < start + n; base += 32u) {
        stage_position(sh, in, base + lane, start + n, cb, lane, stage);
        bin_add(mine, stage, 32u, lane >> 3, lane & 7u);
    }
    LaneSplit best;
    bin_candidate(mine, lane >> 3, lane & 7u, axis_flat(cb, lane >> 3), n, sh.t_area[cur][t], best);
    const bool split = best_split<32>(best, lane);
    int leaf0 = 0, leaf1 = 0;
    if (lane == 0) sub_record(S, sh, cur ^ 1, rec0, start, n, node, split ? 0 : -1, best.l, best.lb, best.rb, &leaf0, &leaf1);
    leaf0 = __shfl_sync(kFull, leaf0, 0);
    leaf1 = __shfl_sync(kFull, leaf1, 0);
    if (!split) {
        for (uint32_t i = start + lane; i < start + n; i += 32u) out0[i] = in[i];
        return;
    }
    const uint32_t axis = best.k / 7u, bin = 6u - best.k % 7u, lcount = best.l;
    const float lo = axis == 0 ? cb[0] : (axis == 1 ? cb[1] : cb[2]);
    const float len = (axis == 0 ? cb[3] : (axis == 1 ? cb[4] : cb[5])) - lo;
    uint32_t lbase = start, rbase = start + lcount;
    for (uint32_t base = start; base < start + n; base += 32u) {
        const uint32_t i = base + lane;
        const bool have = i < start + n;
        const uint32_t p = have ? in[i] : 0u;
        const bool left = have && bin_of(sh.c[axis][p], lo, len) <= bin;
        const unsigned lm = __ballot_sync(kFull, left), rm = __ballot_sync(kFull, have && !left);
        if (have) out0[left ? lbase + __popc(lm & below) : rbase + __popc(rm & below)] = (uint16_t)p;
        lbase += __popc(lm);
        rbase += __popc(rm);
    }
    __syncwarp();                                              // every read of this order is done
    if (leaf0)
        for (uint32_t i = start + lane; i < start + lcount; i += 32u) out1[i] = out0[i];
    if (leaf1)
        for (uint32_t i = start + lcount + lane; i < start + n; i += 32u) out1[i] = out0[i];
}

// A task above kSubCoop primitives, by the whole block.
__device__ void sub_task_block(BuildState &S, SubShared &sh, int cur, uint32_t t, size_t rec0) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    const uint32_t start = sh.t_start[cur][t], n = sh.t_count[cur][t], node = sh.t_node[cur][t];
    const uint16_t *in = sh.perm[cur];
    if (tid < 6u) sh.red[tid] = tid < 3u ? kOrdPosInf : kOrdNegInf;
    __syncthreads();
    unsigned co[6] = {kFull, kFull, kFull, 0u, 0u, 0u};
    for (uint32_t i = start + tid; i < start + n; i += kSubThreads) {
        const uint32_t p = in[i];
        for (int a = 0; a < 3; ++a) {
            const unsigned o = f2ord(sh.c[a][p]);
            co[a] = min(co[a], o);
            co[3 + a] = max(co[3 + a], o);
        }
    }
    for (int a = 0; a < 3; ++a) {
        co[a] = __reduce_min_sync(kFull, co[a]);
        co[3 + a] = __reduce_max_sync(kFull, co[3 + a]);
    }
    if (lane == 0)
        for (int a = 0; a < 3; ++a) { atomicMin(&sh.red[a], co[a]); atomicMax(&sh.red[3 + a], co[3 + a]); }
    __syncthreads();
    float cb[6];
    for (int a = 0; a < 6; ++a) cb[a] = ord2f(sh.red[a]);
    float4 *stage = reinterpret_cast<float4 *>(sh.scratch[w]);
    LaneBin mine{0u, aabb_empty()};
    for (uint32_t base = start + 32u * w; base < start + n; base += kSubThreads) {
        stage_position(sh, in, base + lane, start + n, cb, lane, stage);
        bin_add(mine, stage, 32u, lane >> 3, lane & 7u);
    }
    __syncwarp();
    if (lane < 24u) {                                          // the warp's bins over its staged primitives
        unsigned *q = sh.scratch[w] + lane * kBinStride;
        q[0] = mine.n;
        for (int a = 0; a < 3; ++a) {
            q[1 + a] = __float_as_uint(mine.b.mn[a]);
            q[4 + a] = __float_as_uint(mine.b.mx[a]);
        }
    }
    __syncthreads();
    if (w == 0) {
        mine = LaneBin{0u, aabb_empty()};
        if (lane < 24u)
            for (uint32_t k = 0; k < kSubWarps; ++k) {
                const unsigned *q = sh.scratch[k] + lane * kBinStride;
                mine.n += q[0];
                for (int a = 0; a < 3; ++a) {
                    mine.b.mn[a] = fminf(mine.b.mn[a], __uint_as_float(q[1 + a]));
                    mine.b.mx[a] = fmaxf(mine.b.mx[a], __uint_as_float(q[4 + a]));
                }
            }
        LaneSplit best;
        bin_candidate(mine, lane >> 3, lane & 7u, axis_flat(cb, lane >> 3), n, sh.t_area[cur][t], best);
        const bool split = best_split<32>(best, lane);
        if (lane == 0) {
            sh.split = split ? (int)best.k : -1;
            sh.lcount = best.l;
            sub_record(S, sh, cur ^ 1, rec0, start, n, node, split ? 0 : -1, best.l, best.lb, best.rb,
                       &sh.leaf_child[0], &sh.leaf_child[1]);
        }
    }
    __syncthreads();
    const int k = sh.split;
    uint16_t *out0 = sh.perm[cur ^ 1], *out1 = sh.perm[cur];
    if (k < 0) {
        for (uint32_t i = start + tid; i < start + n; i += kSubThreads) out0[i] = in[i];
        __syncthreads();
        return;
    }
    // stable partition: a contiguous share of the positions per warp
    const int axis = k / 7;
    const uint32_t bin = (uint32_t)(6 - k % 7), lcount = sh.lcount;
    const float lo = ord2f(sh.red[axis]), len = ord2f(sh.red[3 + axis]) - lo;
    const uint32_t share = (n + kSubThreads - 1u) / kSubThreads * 32u;
    const uint32_t first = start + min(w * share, n), last = start + min((w + 1u) * share, n);
    const unsigned below = (1u << lane) - 1u;
    uint32_t lefts = 0;
    for (uint32_t base = first; base < last; base += 32u) {
        const uint32_t i = base + lane;
        const bool left = i < last && bin_of(sh.c[axis][in[i]], lo, len) <= bin;
        lefts += __popc(__ballot_sync(kFull, left));
    }
    if (lane == 0) sh.warp_left[w] = lefts;
    __syncthreads();
    uint32_t lbase = start;
    for (uint32_t j = 0; j < w; ++j) lbase += sh.warp_left[j];
    uint32_t rbase = start + lcount + (first - start) - (lbase - start);
    for (uint32_t base = first; base < last; base += 32u) {
        const uint32_t i = base + lane;
        const bool have = i < last;
        const uint32_t p = have ? in[i] : 0u;
        const bool left = have && bin_of(sh.c[axis][p], lo, len) <= bin;
        const unsigned lm = __ballot_sync(kFull, left), rm = __ballot_sync(kFull, have && !left);
        if (have) out0[left ? lbase + __popc(lm & below) : rbase + __popc(rm & below)] = (uint16_t)p;
        lbase += __popc(lm);
        rbase += __popc(rm);
    }
    __syncthreads();
    if (sh.leaf_child[0])
        for (uint32_t i = start + tid; i < start + lcount; i += kSubThreads) out1[i] = out0[i];
    if (sh.leaf_child[1])
        for (uint32_t i = start + lcount + tid; i < start + n; i += kSubThreads) out1[i] = out0[i];
    __syncthreads();
}

// One block per subtree: its nodes into sub_rec (links and pre-order indices
// local to the subtree), the final order of its positions into perm[buf], its
// size into n_size of its root.
__global__ void __launch_bounds__(kSubThreads, 3) k_subtrees(BuildState S, int buf) {
    extern __shared__ __align__(16) unsigned char sub_smem[];
    SubShared &sh = *reinterpret_cast<SubShared *>(sub_smem);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    const uint32_t start = S.sub_start[blockIdx.x], n = S.sub_count[blockIdx.x], node = S.sub_node[blockIdx.x];
    const size_t rec0 = 2 * (size_t)start;
    for (uint32_t i = tid; i < n; i += kSubThreads) {
        const uint32_t id = S.perm[buf][start + i];
        const float4 c = S.pcen[id], mn = S.pmin[id], mx = S.pmax[id];
        sh.c[0][i] = c.x; sh.c[1][i] = c.y; sh.c[2][i] = c.z;
        sh.mn[0][i] = mn.x; sh.mn[1][i] = mn.y; sh.mn[2][i] = mn.z;
        sh.mx[0][i] = mx.x; sh.mx[1][i] = mx.y; sh.mx[2][i] = mx.z;
        sh.perm[0][i] = (uint16_t)i;
    }
    if (tid == 0) {
        const float4 mn = S.n_min[node], mx = S.n_max[node];
        Aabb b;
        b.mn[0] = mn.x; b.mn[1] = mn.y; b.mn[2] = mn.z;
        b.mx[0] = mx.x; b.mx[1] = mx.y; b.mx[2] = mx.z;
        sub_box(S, rec0, b);
        sh.t_start[0][0] = 0; sh.t_count[0][0] = (uint16_t)n; sh.t_node[0][0] = 0;
        sh.t_area[0][0] = fmaxf(half_area(b), 1e-8f);
        sh.n_nodes = 1;
        sh.n_tasks[0] = 1; sh.n_tasks[1] = 0;
        for (int k = 0; k < 3; ++k) sh.n_class[0][k] = sh.n_class[1][k] = 0;
        const uint32_t k = n <= 8u ? 0u : (n <= 16u ? 1u : 2u);
        sh.n_class[0][k] = 1;
        sh.of_class[0][k][0] = 0;
        sh.level_end[0] = 1;
    }
    int cur = 0;
    uint32_t levels = 0;
    for (;;) {
        __syncthreads();
        const uint32_t tasks = sh.n_tasks[cur];
        if (tasks == 0) break;
        bool wide = false;                                     // uniform: every thread reads the same counts
        if (tasks <= kSub / kSubCoop)
            for (uint32_t t = 0; t < tasks; ++t)
                if (sh.t_count[cur][t] > kSubCoop) { sub_task_block(S, sh, cur, t, rec0); wide = true; }
        if (wide) __syncthreads();
        // the level's remaining tasks: the larger ones first, then two and four of the smaller ones per warp
        const uint32_t n2 = sh.n_class[cur][2], n1 = sh.n_class[cur][1], n0 = sh.n_class[cur][0];
        const uint32_t items = n2 + (n1 + 1u) / 2u + (n0 + 3u) / 4u;
        for (uint32_t k = w; k < items; k += kSubWarps) {
            if (k < n2) {
                const uint32_t t = sh.of_class[cur][2][k], cnt = sh.t_count[cur][t];
                if (cnt <= 32u) sub_task_group<32>(S, sh, cur, true, t, rec0, lane, sh.scratch[w]);
                else if (cnt <= kSubCoop || tasks > kSub / kSubCoop) sub_task_warp(S, sh, cur, t, rec0, lane, sh.scratch[w]);
            } else if (k < n2 + (n1 + 1u) / 2u) {
                const uint32_t j = 2u * (k - n2) + (lane >> 4);
                sub_task_group<16>(S, sh, cur, j < n1, j < n1 ? sh.of_class[cur][1][j] : 0u, rec0, lane, sh.scratch[w]);
            } else {
                const uint32_t j = 4u * (k - n2 - (n1 + 1u) / 2u) + (lane >> 3);
                sub_task_group<8>(S, sh, cur, j < n0, j < n0 ? sh.of_class[cur][0][j] : 0u, rec0, lane, sh.scratch[w]);
            }
        }
        __syncthreads();
        ++levels;
        if (tid == 0) {
            sh.n_tasks[cur] = 0;
            for (int k = 0; k < 3; ++k) sh.n_class[cur][k] = 0;
            sh.level_end[levels] = (uint16_t)sh.n_nodes;
        }
        cur ^= 1;
    }
    // subtree sizes bottom-up, pre-order indices top-down: level k holds the nodes [level_end[k - 1], level_end[k])
    for (uint32_t k = levels + 1; k-- > 0;) {
        for (uint32_t i = (k ? sh.level_end[k - 1] : 0u) + tid; i < sh.level_end[k]; i += kSubThreads)
            sh.size[i] = sh.b[i] ? 1u : (uint16_t)(1u + sh.size[sh.a[i]] + sh.size[sh.a[i] + 1u]);
        __syncthreads();
    }
    if (tid == 0) sh.pre[0] = 0;
    __syncthreads();
    for (uint32_t k = 0; k <= levels; ++k) {
        for (uint32_t i = (k ? sh.level_end[k - 1] : 0u) + tid; i < sh.level_end[k]; i += kSubThreads)
            if (!sh.b[i]) {
                const uint32_t l = sh.a[i];
                sh.pre[l] = (uint16_t)(sh.pre[i] + 1u);
                sh.pre[l + 1u] = (uint16_t)(sh.pre[i] + 1u + sh.size[l]);
            }
        __syncthreads();
    }
    for (uint32_t i = tid; i < sh.n_nodes; i += kSubThreads) {
        const uint32_t count = sh.b[i], link = count ? start + sh.a[i] : (uint32_t)sh.pre[sh.a[i] + 1u];
        S.sub_rec[3 * (rec0 + i) + 2] = make_float4(__uint_as_float(link), __uint_as_float(count),
                                                    __uint_as_float((uint32_t)sh.pre[i]), 0.0f);
    }
    uint32_t id[kSub / kSubThreads];
    for (uint32_t k = 0; k < kSub / kSubThreads; ++k) {
        const uint32_t i = k * kSubThreads + tid;
        if (i < n) id[k] = S.perm[buf][start + sh.perm[cur][i]];
    }
    __syncthreads();
    for (uint32_t k = 0; k < kSub / kSubThreads; ++k) {
        const uint32_t i = k * kSubThreads + tid;
        if (i < n) S.perm[buf][start + i] = id[k];
    }
    if (tid == 0) {
        S.n_size[node] = sh.n_nodes;
        S.n_a[node] = start;
        atomicMax(S.counters + 10, levels);
    }
}

// The subtrees' nodes into their places, one block per subtree.
__global__ void __launch_bounds__(256) k_emit_subtrees(BuildState S, mcrt_gpu_bvh_node *out) {
    const uint32_t start = S.sub_start[blockIdx.x], node = S.sub_node[blockIdx.x];
    const uint32_t base = S.n_pre[node], size = S.n_size[node];
    const float4 *rec = S.sub_rec + 6 * (size_t)start;
    for (uint32_t i = threadIdx.x; i < size; i += 256u) {
        const float4 mn = rec[3 * (size_t)i], mx = rec[3 * (size_t)i + 1];
        float4 link = rec[3 * (size_t)i + 2];
        const uint32_t pre = __float_as_uint(link.z);
        if (__float_as_uint(link.y) == 0u) link.x = __uint_as_float(__float_as_uint(link.x) + base);
        link.z = 0.0f;
        float4 *o = reinterpret_cast<float4 *>(out + base + pre);
        o[0] = mn;
        o[1] = mx;
        o[2] = link;
    }
}

// Partition flag of position i: 1 when its primitive goes to the left child of
// its large task's split, else 0.
__device__ __forceinline__ uint32_t partition_flag(const BuildState &S, int cur, uint32_t i) {
    const int task = S.ptask[cur][i];
    if (task < 0) return 0u;
    const int sp = S.t_split[task];
    if (sp < 0) return 0u;
    const int axis = sp >> 4, bin = sp & 15;
    const float *cb = S.t_cb + 6 * task;
    const float4 c = S.pcen[S.perm[cur][i]];
    const float cc = axis == 0 ? c.x : (axis == 1 ? c.y : c.z);
    const float len = cb[3 + axis] - cb[axis];
    return bin_of(cc, cb[axis], len) <= (uint32_t)bin ? 1u : 0u;
}

// The partition flags of every position and their exclusive scan in one pass
// (decoupled look-back, Merrill and Garland 2016): a block takes the next tile
// from a ticket (tiles start in order, so every predecessor of a tile is
// running or done), scans its kFlagTile flags, publishes its sum, adds its
// predecessors' published sums walking back to the first inclusive prefix,
// and publishes its own.  The walk reads 32 predecessors per step, one per lane
// of the first warp: the nearest inclusive prefix among them (ballot) ends it,
// else their sums are added and the window moves back.  Every wait is bounded:
// after kLookbackPolls polls of a predecessor the tile records the error word
// and goes on (the host fails the build).
template <uint32_t kFlagItems>
__global__ void __launch_bounds__(kFlagThreads) k_flag_scan(BuildState S, int cur) {
    constexpr uint32_t kFlagTile = kFlagThreads * kFlagItems;
    __shared__ uint32_t s_tile, s_excl, s_warp[kFlagThreads / 32];
    const uint32_t t = threadIdx.x, lane = t & 31u, w = t >> 5;
    unsigned long long *status = S.part + 2;
    if (t == 0) s_tile = atomicAdd(reinterpret_cast<unsigned int *>(S.part), 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t i0 = tile * kFlagTile + t * kFlagItems;
    uint32_t f[kFlagItems], sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < kFlagItems; ++k) {
        f[k] = i0 + k < S.nt ? partition_flag(S, cur, i0 + k) : 0u;
        sum += f[k];
    }
    uint32_t x = sum;                                          // inclusive scan over the warp
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    if (w == 0) {                                              // inclusive scan of the warp totals
        uint32_t v = lane < kFlagThreads / 32 ? s_warp[lane] : 0u;
#pragma unroll
        for (uint32_t d = 1; d < kFlagThreads / 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, v, d);
            if (lane >= d) v += y;
        }
        if (lane < kFlagThreads / 32) s_warp[lane] = v;
    }
    __syncthreads();
    const uint32_t block_total = s_warp[kFlagThreads / 32 - 1];
    const uint32_t thread_excl = (w ? s_warp[w - 1] : 0u) + x - sum;
    if (w == 0) {
        uint32_t excl = 0;
        if (tile == 0) {
            if (lane == 0) {
                __threadfence();
                atomicExch(status, (2ull << 32) | block_total);
            }
        } else {
            if (lane == 0) atomicExch(status + tile, (1ull << 32) | block_total);
            bool gave_up = false;
            for (int j = (int)tile - 1; !gave_up;) {            // window: predecessors j, j - 1, ..., j - 31
                const int idx = j - (int)lane;
                unsigned long long v = 2ull << 32;              // before tile 0: an inclusive prefix of 0
                if (idx >= 0) {
                    uint32_t polls = 0;
                    for (;;) {
                        v = *reinterpret_cast<volatile unsigned long long *>(status + idx);
                        if ((uint32_t)(v >> 32) != 0u) break;
                        if (++polls > kLookbackPolls) { v = 2ull << 32; gave_up = true; break; }
                    }
                }
                gave_up = __any_sync(kFull, gave_up);
                const unsigned incl = __ballot_sync(kFull, (uint32_t)(v >> 32) == 2u);
                const uint32_t last = incl ? (uint32_t)__ffs(incl) - 1u : 31u;   // nearest inclusive lane
                excl += __reduce_add_sync(kFull, lane <= last ? (uint32_t)v : 0u);
                if (incl) break;
                j -= 32;
            }
            if (lane == 0) {
                if (gave_up) atomicExch(S.counters + 9, 1u);
                __threadfence();
                atomicExch(status + tile, (2ull << 32) | (excl + block_total));
            }
        }
        if (lane == 0) s_excl = excl;
    }
    __syncthreads();
    uint32_t run = s_excl + thread_excl;
#pragma unroll
    for (uint32_t k = 0; k < kFlagItems; ++k) {
        if (i0 + k < S.nt) {
            S.flags[i0 + k] = f[k];
            S.scan[i0 + k] = run;
        }
        run += f[k];
    }
}

__global__ void k_scatter(BuildState S, int cur) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.nt) return;
    int task = S.ptask[cur][i];
    uint32_t id = S.perm[cur][i];
    if (task < 0) { S.perm[cur ^ 1][i] = id; S.ptask[cur ^ 1][i] = -1; return; }
    int sp = S.t_split[task];
    uint32_t start = S.t_start[cur][task], node = S.t_node[cur][task];
    if (sp < 0) { S.perm[cur ^ 1][i] = id; S.ptask[cur ^ 1][i] = -1; return; }
    uint32_t lcount = S.t_lcount[task];
    uint32_t left_rank = S.scan[i] - S.scan[start];
    uint32_t pos;
    uint32_t child;
    if (S.flags[i]) { pos = start + left_rank; child = S.n_a[node]; }
    else { pos = start + lcount + ((i - start) - left_rank); child = S.n_b[node]; }
    S.perm[cur ^ 1][pos] = id;
    S.ptask[cur ^ 1][pos] = S.n_leaf[child] ? -1 : (int)S.n_size[child];   // -1: in a leaf or a subtree
}

// Subtree sizes (bottom-up) and pre-order indices (top-down) of the nodes above
// the subtrees, one block: a level is a few hundred to a few thousand nodes, and
// a launch per level and direction cost 3.6 us each.
__global__ void __launch_bounds__(1024) k_upper_order(BuildState S, uint32_t levels) {
    const uint32_t tid = threadIdx.x;
    auto begin = [&](uint32_t k) { return k ? S.level_end[k - 1] : 0u; };
    for (uint32_t k = levels + 1; k-- > 0;) {
        const uint32_t end = k < levels ? S.level_end[k] : S.counters[1];
        for (uint32_t i = begin(k) + tid; i < end; i += 1024u) {
            const uint32_t kind = S.n_leaf[i];
            if (kind == 1u) S.n_size[i] = 1u;
            else if (kind == 0u) S.n_size[i] = 1u + S.n_size[S.n_a[i]] + S.n_size[S.n_b[i]];
        }
        __syncthreads();
    }
    if (tid == 0) {
        S.n_pre[0] = 0;
        S.counters[11] = S.n_size[0];
    }
    __syncthreads();
    for (uint32_t k = 0; k <= levels; ++k) {
        const uint32_t end = k < levels ? S.level_end[k] : S.counters[1];
        for (uint32_t i = begin(k) + tid; i < end; i += 1024u) {
            if (S.n_leaf[i] != 0u) continue;
            const uint32_t p = S.n_pre[i], l = S.n_a[i];
            S.n_pre[l] = p + 1;
            S.n_pre[S.n_b[i]] = p + 1 + S.n_size[l];
        }
        __syncthreads();
    }
}
__global__ void k_emit(BuildState S, uint32_t n_bfs, mcrt_gpu_bvh_node *out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_bfs || S.n_leaf[i] == kSubMark) return;        // a subtree's root: k_emit_subtrees
    mcrt_gpu_bvh_node nd;
    float4 mn = S.n_min[i], mx = S.n_max[i];
    nd.aabb_min[0] = mn.x; nd.aabb_min[1] = mn.y; nd.aabb_min[2] = mn.z; nd.aabb_min[3] = 0.0f;
    nd.aabb_max[0] = mx.x; nd.aabb_max[1] = mx.y; nd.aabb_max[2] = mx.z; nd.aabb_max[3] = 0.0f;
    if (S.n_leaf[i]) { nd.right_or_offset = S.n_a[i]; nd.prim_count = S.n_b[i]; }
    else { nd.right_or_offset = S.n_pre[S.n_b[i]]; nd.prim_count = 0; }
    nd._pad[0] = 0; nd._pad[1] = 0;
    out[S.n_pre[i]] = nd;
}

template <typename T> T *carve(char *&p, size_t count) {
    T *r = reinterpret_cast<T *>(p);
    size_t bytes = (count * sizeof(T) + 255) & ~(size_t)255;
    p += bytes;
    return r;
}

}  // namespace

static cudaError_t gpu_build(const mcrt_gpu_vertex *d_verts, const mcrt_gpu_triangle *d_tris,
                             const mcrt_gpu_sphere *d_sph, uint32_t nt, mcrt_gpu_bvh_node *d_nodes,
                             uint32_t *d_order, uint32_t *n_nodes_out, BvhScratch **scratch_io, cudaStream_t st,
                             std::string *err) {
    *n_nodes_out = 0;
    if (nt == 0) return cudaSuccess;
    BvhScratch *sc = *scratch_io;
    if (!sc || sc->cap < nt) {
        free_bvh_scratch(sc);
        sc = new BvhScratch();
        *scratch_io = sc;
        size_t n = nt, nn = 2 * (size_t)nt, tc = (size_t)nt / 4 + 1;   // tasks hold > 4 primitives
        size_t bytes = 0;
        auto acc = [&](size_t b) { bytes += (b + 255) & ~(size_t)255; };
        acc(n * 16); acc(n * 16); acc(n * 16);               // pmin, pmax, pcen
        acc(n * 4); acc(n * 4); acc(n * 4); acc(n * 4);      // perm x2, ptask x2
        acc(n * 4); acc(n * 4);                              // flags, scan
        for (int k = 0; k < 2; ++k) { acc(tc * 4); acc(tc * 4); acc(tc * 4); acc(tc * 24); }
        acc(tc * 24); acc(tc * 4 * kTaskBinWords); acc(tc * 4); acc(tc * 4);
        acc(nn * 16); acc(nn * 16); acc(nn * 4); acc(nn * 4); acc(nn * 4); acc(nn * 4); acc(nn * 4);
        acc(64);
        acc(kMaxLevels * 4);
        const size_t tiles = (n + kRadixTile - 1) / kRadixTile;
        const size_t scan_words = std::max(scan_tmp_words(nt), scan_tmp_words((uint32_t)(256 * tiles)));
        acc(scan_words * 4);
        acc(n * 4); acc(n * 4); acc(n * 4); acc(n * 4);      // sort keys, ids (ping-pong)
        acc(256 * tiles * 4); acc(256 * tiles * 4);          // digit counts, offsets
        acc(n * 16); acc(n * 16); acc(n * 16);               // reordered bounds
        acc(tc * 4); acc(tc * 4); acc(tc * 4); acc(nn * 48);  // subtrees and their nodes
        acc((2 + (n + kMinFlagTile - 1) / kMinFlagTile) * 8);   // partition scan state
        cudaError_t e = cudaMalloc(&sc->mem, bytes);
        if (e != cudaSuccess) { if (err) *err = "BVH scratch allocation failed"; return e; }
        sc->cap = nt;
        char *p = static_cast<char *>(sc->mem);
        BuildState &S = sc->s;
        S.pmin = carve<float4>(p, n); S.pmax = carve<float4>(p, n); S.pcen = carve<float4>(p, n);
        S.perm[0] = carve<uint32_t>(p, n); S.perm[1] = carve<uint32_t>(p, n);
        S.ptask[0] = carve<int32_t>(p, n); S.ptask[1] = carve<int32_t>(p, n);
        S.flags = carve<uint32_t>(p, n); S.scan = carve<uint32_t>(p, n);
        for (int k = 0; k < 2; ++k) {
            S.t_start[k] = carve<uint32_t>(p, tc); S.t_count[k] = carve<uint32_t>(p, tc);
            S.t_node[k] = carve<uint32_t>(p, tc); S.t_bounds[k] = carve<float>(p, 6 * tc);
        }
        S.t_cb = carve<float>(p, 6 * tc); S.t_bins = carve<float>(p, tc * kTaskBinWords);
        S.t_split = carve<int32_t>(p, tc); S.t_lcount = carve<uint32_t>(p, tc);
        S.n_min = carve<float4>(p, nn); S.n_max = carve<float4>(p, nn);
        S.n_a = carve<uint32_t>(p, nn); S.n_b = carve<uint32_t>(p, nn); S.n_leaf = carve<uint32_t>(p, nn);
        S.n_size = carve<uint32_t>(p, nn); S.n_pre = carve<uint32_t>(p, nn);
        S.counters = carve<uint32_t>(p, 16);
        S.level_end = carve<uint32_t>(p, kMaxLevels);
        sc->scan_tmp = carve<uint32_t>(p, scan_words);
        S.rkey[0] = carve<uint32_t>(p, n); S.rkey[1] = carve<uint32_t>(p, n);
        S.rval[0] = carve<uint32_t>(p, n); S.rval[1] = carve<uint32_t>(p, n);
        S.rhist = carve<uint32_t>(p, 256 * tiles); S.roffs = carve<uint32_t>(p, 256 * tiles);
        S.qmin = carve<float4>(p, n); S.qmax = carve<float4>(p, n); S.qcen = carve<float4>(p, n);
        S.sub_start = carve<uint32_t>(p, tc); S.sub_count = carve<uint32_t>(p, tc); S.sub_node = carve<uint32_t>(p, tc);
        S.sub_rec = carve<float4>(p, 3 * nn);
        S.part = carve<unsigned long long>(p, 2 + (n + kMinFlagTile - 1) / kMinFlagTile);
    }
    BuildState S = sc->s;
    S.nt = nt;
    const uint32_t per = nt < kWideBlocks ? 256u : 1024u;    // positions per block of the whole-array passes
    const uint32_t TB = 256;
    const uint32_t nb = (nt + TB - 1) / TB;
    if (d_sph) k_sphere_bounds<<<nb, TB, 0, st>>>(d_sph, S);
    else k_prim_bounds<<<nb, TB, 0, st>>>(d_verts, d_tris, S);
    ::mcrt::note_launch();
    k_root_init<<<1, 32, 0, st>>>(S); ::mcrt::note_launch();
    k_root_bounds<<<(nt + per - 1) / per, 256, 0, st>>>(S, per); ::mcrt::note_launch();
    if (nt <= kLeafMax) {
        // the root is a single leaf (bvh.rs:301-304)
        std::vector<float> tb(6);
        cudaMemcpyAsync(tb.data(), S.t_bounds[0], 24, cudaMemcpyDeviceToHost, st);
        cudaStreamSynchronize(st);
        mcrt_gpu_bvh_node nd{};
        for (int a = 0; a < 3; ++a) { nd.aabb_min[a] = tb[a]; nd.aabb_max[a] = tb[3 + a]; }
        nd.right_or_offset = 0;
        nd.prim_count = nt;
        cudaMemcpyAsync(d_nodes, &nd, sizeof(nd), cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(d_order, S.perm[0], 4 * (size_t)nt, cudaMemcpyDeviceToDevice, st);
        cudaError_t e = cudaStreamSynchronize(st);
        *n_nodes_out = 1;
        return e;
    }
    // Morton order: 4 stable radix passes of 8 bits over the 30-bit codes
    // (ends in buffer 0), then the bounds are gathered into that order and the
    // build runs on Morton indices; the output order maps them back to ids.
    {
        const uint32_t tiles = (nt + kRadixTile - 1) / kRadixTile;
        k_morton<<<nb, TB, 0, st>>>(S); ::mcrt::note_launch();
        for (int pass = 0; pass < 4; ++pass) {
            const int in = pass & 1;
            k_radix_hist<<<tiles, 256, 0, st>>>(S.rkey[in], nt, 8 * pass, tiles, S.rhist); ::mcrt::note_launch();
            exclusive_scan_u32(S.rhist, S.roffs, 256 * tiles, sc->scan_tmp, st);
            k_radix_scatter<<<tiles, 256, 0, st>>>(S.rkey[in], S.rval[in], nt, 8 * pass, tiles, S.roffs,
                                                  S.rkey[in ^ 1], S.rval[in ^ 1]);
            ::mcrt::note_launch();
        }
        k_reorder<<<nb, TB, 0, st>>>(S); ::mcrt::note_launch();
        std::swap(S.pmin, S.qmin);
        std::swap(S.pmax, S.qmax);
        std::swap(S.pcen, S.qcen);
    }
    // BFS node 0 = root
    cudaMemcpyAsync(S.n_min, S.t_bounds[0], 12, cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(S.n_max, S.t_bounds[0] + 3, 12, cudaMemcpyDeviceToDevice, st);
    // Levels of large tasks, by the whole-array passes; level_end[r] = the BFS
    // node count when level r starts, so level r creates the nodes
    // [level_end[r], level_end[r + 1]).  A level at most halves the largest task,
    // so the first log2(nt / kSub) levels run without a look at the count of
    // large tasks; after those the host reads it once per level.  Where the root
    // itself has no split (all centroids in one place: a leaf of any size), the
    // levels after it would be run for nothing, so the second level's first kernel
    // writes the count to host memory, and the host looks at it once the rest of
    // that level is queued: the device does not wait.  (50,000 triangles in one
    // place: 306 us without a look, 241 with it, 236 with one at every level.)
    const uint32_t nbp = (nt + per - 1) / per;
    const uint32_t flag_tile = nt < kWideBlocks ? kMinFlagTile : 4u * kMinFlagTile;
    const uint32_t n_flag_tiles = (nt + flag_tile - 1) / flag_tile, n_part = 2 + n_flag_tiles;
    uint32_t host_counters[16] = {};
    uint32_t level = 0, n_large = nt > kSub ? 1u : 0u, n_sub = 0, n_bfs = 1;
    uint32_t unseen = 0;                                 // levels to run before the next look
    while ((uint64_t)kSub << (unseen + 1) <= nt) ++unseen;
    int cur = 0;
    while (n_large > 0) {
        if (level + 1 >= kMaxLevels) {
            if (err) *err = "BVH build exceeded 4096 levels";
            return cudaErrorUnknown;
        }
        const uint32_t nw = std::max(n_large * (6 + kTaskBinWords), n_part);
        const bool look = level == 1 && unseen > 1;
        if (look) {
            cudaError_t e = cudaSuccess;
            if (!sc->large) e = cudaHostAlloc(reinterpret_cast<void **>(&sc->large), 4, cudaHostAllocMapped);
            if (e == cudaSuccess && !sc->looked) e = cudaEventCreateWithFlags(&sc->looked, cudaEventDisableTiming);
            if (e != cudaSuccess) { if (err) *err = "BVH level count"; return e; }
        }
        k_task_reset<<<(nw + TB - 1) / TB, TB, 0, st>>>(S, level++, n_large, n_part, look ? sc->large : nullptr);
        ::mcrt::note_launch();
        if (look) cudaEventRecord(sc->looked, st);
        k_centroid_bounds<<<nbp, 256, 0, st>>>(S, cur, per); ::mcrt::note_launch();
        k_bins<<<nbp, 256, 0, st>>>(S, cur, per); ::mcrt::note_launch();
        k_split<<<(n_large + 3) / 4, 128, 0, st>>>(S, cur); ::mcrt::note_launch();
        if (nt < kWideBlocks) k_flag_scan<2><<<n_flag_tiles, kFlagThreads, 0, st>>>(S, cur);
        else k_flag_scan<8><<<n_flag_tiles, kFlagThreads, 0, st>>>(S, cur);
        ::mcrt::note_launch();
        k_scatter<<<nb, TB, 0, st>>>(S, cur); ::mcrt::note_launch();
        cur ^= 1;
        if (unseen > 1) {                                // at most twice as many, each above kSub primitives
            --unseen;
            n_large = std::min(2u * n_large, nt / (kSub + 1u));
            if (look) cudaEventSynchronize(sc->looked);
            if (!look || *sc->large > 0) continue;
        }
        cudaMemcpyAsync(host_counters, S.counters, sizeof(host_counters), cudaMemcpyDeviceToHost, st);
        cudaError_t e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) { if (err) *err = "BVH build level failed"; return e; }
        if (host_counters[9]) { if (err) *err = "BVH build: partition scan look-back gave up"; return cudaErrorUnknown; }
        n_large = host_counters[0];
        n_bfs = host_counters[1];
        n_sub = host_counters[4];
    }
    if (nt <= kSub) {                                    // the root is a subtree itself
        k_root_subtree<<<1, 1, 0, st>>>(S); ::mcrt::note_launch();
        n_sub = 1;
    }
    if (n_sub) {
        if (!sc->configured) {
            cudaError_t e = cudaFuncSetAttribute(k_subtrees, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)sizeof(SubShared));
            if (e != cudaSuccess) { if (err) *err = "BVH subtree kernel"; return e; }
            sc->configured = true;
        }
        k_subtrees<<<n_sub, kSubThreads, sizeof(SubShared), st>>>(S, cur); ::mcrt::note_launch();
    }
    k_upper_order<<<1, 1024, 0, st>>>(S, level); ::mcrt::note_launch();
    k_emit<<<(n_bfs + TB - 1) / TB, TB, 0, st>>>(S, n_bfs, d_nodes); ::mcrt::note_launch();
    if (n_sub) { k_emit_subtrees<<<n_sub, 256, 0, st>>>(S, d_nodes); ::mcrt::note_launch(); }
    k_final_order<<<nb, TB, 0, st>>>(S.perm[cur], S.rval[0], nt, d_order); ::mcrt::note_launch();
    cudaMemcpyAsync(host_counters, S.counters, sizeof(host_counters), cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { if (err) *err = "BVH emit failed"; return e; }
    if (level + host_counters[10] + 1 >= kMaxLevels) {
        if (err) *err = "BVH build exceeded 4096 levels";
        return cudaErrorUnknown;
    }
    *n_nodes_out = host_counters[11];
    return cudaSuccess;
}

cudaError_t gpu_build_mesh_bvh(const mcrt_gpu_vertex *d_verts, const mcrt_gpu_triangle *d_tris, uint32_t nt,
                               mcrt_gpu_bvh_node *d_nodes, uint32_t *d_order, uint32_t *n_nodes_out,
                               BvhScratch **scratch, cudaStream_t st, std::string *err) {
    return gpu_build(d_verts, d_tris, nullptr, nt, d_nodes, d_order, n_nodes_out, scratch, st, err);
}

cudaError_t gpu_build_sphere_bvh(const mcrt_gpu_sphere *d_spheres, uint32_t n, mcrt_gpu_bvh_node *d_nodes,
                                 uint32_t *d_order, uint32_t *n_nodes_out, BvhScratch **scratch, cudaStream_t st,
                                 std::string *err) {
    return gpu_build(nullptr, nullptr, d_spheres, n, d_nodes, d_order, n_nodes_out, scratch, st, err);
}

// ------------------------------------------------------------------ compact layout
namespace {
__global__ void k_internal_flags(const mcrt_gpu_bvh_node *nodes, uint32_t n, uint32_t *flags) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) flags[i] = nodes[i].prim_count == 0 ? 1u : 0u;
}
__device__ __forceinline__ uint32_t child_code(const mcrt_gpu_bvh_node *nodes, const uint32_t *rank, uint32_t c) {
    const mcrt_gpu_bvh_node &nd = nodes[c];
    return nd.prim_count == 0 ? rank[c] : leaf_code(nd.right_or_offset, nd.prim_count);
}
__global__ void k_compact(const mcrt_gpu_bvh_node *nodes, uint32_t n, const uint32_t *rank, float4 *out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || nodes[i].prim_count != 0) return;
    uint32_t l = i + 1, r = nodes[i].right_or_offset;
    const mcrt_gpu_bvh_node &L = nodes[l], &R = nodes[r];
    float4 *o = out + 4ull * rank[i];
    o[0] = make_float4(L.aabb_min[0], L.aabb_max[0], L.aabb_min[1], L.aabb_max[1]);
    o[1] = make_float4(R.aabb_min[0], R.aabb_max[0], R.aabb_min[1], R.aabb_max[1]);
    o[2] = make_float4(L.aabb_min[2], L.aabb_max[2], R.aabb_min[2], R.aabb_max[2]);
    o[3] = make_float4(__uint_as_float(child_code(nodes, rank, l)), __uint_as_float(child_code(nodes, rank, r)),
                       __uint_as_float(kNoChild), 0.0f);
}
// Word 3.z of each compact record: its parent's index (the root keeps
// kNoChild), the up-link of the stackless walk.  Runs after k_compact.
__global__ void k_compact_parents(const mcrt_gpu_bvh_node *nodes, uint32_t n, const uint32_t *rank, float4 *out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || nodes[i].prim_count != 0) return;
    const uint32_t kids[2] = {i + 1, nodes[i].right_or_offset};
    for (int k = 0; k < 2; ++k)
        if (nodes[kids[k]].prim_count == 0)
            reinterpret_cast<uint32_t *>(out + 4ull * rank[kids[k]] + 3)[2] = rank[i];
}
// Shading records in original triangle order: the three vertex normals, the
// first carrying the material word.
__global__ void k_shade_recs(const mcrt_gpu_vertex *verts, const mcrt_gpu_triangle *tris, uint32_t nt, float4 *out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nt) return;
    const mcrt_gpu_triangle t = tris[i];
    float4 *r = out + 3ull * i;
    for (int k = 0; k < 3; ++k) {
        const float *n = verts[t.v[k]].normal;
        r[k] = make_float4(n[0], n[1], n[2], k == 0 ? __uint_as_float(t.mat_idx) : 0.0f);
    }
}

__global__ void k_trirecs(const uint32_t *order, const mcrt_gpu_vertex *verts, const mcrt_gpu_triangle *tris,
                          uint32_t nt, TriRec *out) {
    uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nt) return;
    uint32_t id = order[s];
    mcrt_gpu_triangle t = tris[id];
    f3 v0 = ld3(verts[t.v[0]].position), v1 = ld3(verts[t.v[1]].position), v2 = ld3(verts[t.v[2]].position);
    f3 e1 = v1 - v0, e2 = v2 - v0;                                 // path_trace.wgsl:302-303
    TriRec r;
    r.v0 = make_float4(v0.x, v0.y, v0.z, __uint_as_float(id));
    r.e1 = make_float4(e1.x, e1.y, e1.z, __uint_as_float(t.mat_idx));
    r.e2 = make_float4(e2.x, e2.y, e2.z, 0.0f);
    out[s] = r;
}
__global__ void k_leaf_counts(const mcrt_gpu_bvh_node *nodes, uint32_t n, TriRec *recs) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || nodes[i].prim_count == 0) return;
    recs[nodes[i].right_or_offset].e2.w = __uint_as_float(nodes[i].prim_count);
}
}  // namespace

void launch_shade_recs(const mcrt_gpu_vertex *d_verts, const mcrt_gpu_triangle *d_tris, uint32_t nt, float4 *out,
                       cudaStream_t st) {
    if (nt == 0) return;
    k_shade_recs<<<(nt + 255) / 256, 256, 0, st>>>(d_verts, d_tris, nt, out); ::mcrt::note_launch();
}

cudaError_t gpu_make_compact(const mcrt_gpu_bvh_node *d_nodes, uint32_t n_nodes, const uint32_t *d_order,
                             const mcrt_gpu_vertex *d_verts, const mcrt_gpu_triangle *d_tris, uint32_t nt,
                             float4 **d_cnodes, uint32_t *n_cnodes, void *d_trirecs, uint32_t *d_tmp,
                             size_t tmp_words, cudaStream_t st) {
    // d_tmp: 2*n_nodes + scan_tmp_words(n_nodes) words
    (void)tmp_words;
    const uint32_t TB = 256;
    TriRec *recs = static_cast<TriRec *>(d_trirecs);
    if (nt) k_trirecs<<<(nt + TB - 1) / TB, TB, 0, st>>>(d_order, d_verts, d_tris, nt, recs); ::mcrt::note_launch();
    *n_cnodes = 0;
    if (n_nodes == 0) return cudaGetLastError();
    k_leaf_counts<<<(n_nodes + TB - 1) / TB, TB, 0, st>>>(d_nodes, n_nodes, recs); ::mcrt::note_launch();
    if (n_nodes == 1) return cudaGetLastError();
    uint32_t *flags = d_tmp, *rank = d_tmp + n_nodes, *stmp = d_tmp + 2 * (size_t)n_nodes;
    k_internal_flags<<<(n_nodes + TB - 1) / TB, TB, 0, st>>>(d_nodes, n_nodes, flags); ::mcrt::note_launch();
    exclusive_scan_u32(flags, rank, n_nodes, stmp, st);
    uint32_t last_rank = 0, last_flag = 0;
    cudaMemcpyAsync(&last_rank, rank + n_nodes - 1, 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&last_flag, flags + n_nodes - 1, 4, cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    uint32_t n_int = last_rank + last_flag;
    if (*d_cnodes == nullptr) return cudaErrorInvalidValue;
    k_compact<<<(n_nodes + TB - 1) / TB, TB, 0, st>>>(d_nodes, n_nodes, rank, *d_cnodes); ::mcrt::note_launch();
    k_compact_parents<<<(n_nodes + TB - 1) / TB, TB, 0, st>>>(d_nodes, n_nodes, rank, *d_cnodes);
    ::mcrt::note_launch();
    *n_cnodes = n_int;
    return cudaGetLastError();
}

// The top levels of the compact tree in heap order, for the shared-memory
// top-tree traversal: entry 0 is the root, entry j's children go to 2j+1 and
// 2j+2 while those fit (kTopNodes entries, 7 levels); an internal child that
// gets an entry is recoded kTopBit | entry, every other child keeps its code
// (a deeper internal node's compact index, a leaf, or none).  One block, one
// thread per entry, a level per step.
__global__ void k_top_tree(const float4 *cnodes, uint32_t n_cnodes, float4 *top) {
    __shared__ uint32_t src[kTopNodes];            // compact index held by an entry, or kNoChild
    const uint32_t j = threadIdx.x;
    if (j < kTopNodes) src[j] = (j == 0 && n_cnodes > 0) ? 0u : kNoChild;
    __syncthreads();
    for (uint32_t first = 0, width = 1; first < kTopNodes; first += width, width *= 2) {
        if (j >= first && j < first + width && j < kTopNodes) {
            float4 r[4] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f),
                           make_float4(0.f, 0.f, 0.f, 0.f),
                           make_float4(__uint_as_float(kNoChild), __uint_as_float(kNoChild), 0.f, 0.f)};
            if (src[j] != kNoChild) {
                const float4 *np = cnodes + 4ull * src[j];
                for (int k = 0; k < 4; ++k) r[k] = np[k];
                uint32_t code[2] = {__float_as_uint(r[3].x), __float_as_uint(r[3].y)};
                for (int side = 0; side < 2; ++side) {
                    const uint32_t slot = 2 * j + 1 + side;
                    if (code[side] != kNoChild && !(code[side] & kLeafBit) && slot < kTopNodes) {
                        src[slot] = code[side];
                        code[side] = kTopBit | slot;
                    }
                }
                r[3].x = __uint_as_float(code[0]);
                r[3].y = __uint_as_float(code[1]);
            }
            for (int k = 0; k < 4; ++k) top[4ull * j + k] = r[k];
        }
        __syncthreads();
    }
}

cudaError_t gpu_make_top(const float4 *d_cnodes, uint32_t n_cnodes, float4 *d_top, cudaStream_t st) {
    k_top_tree<<<1, 128, 0, st>>>(d_cnodes, n_cnodes, d_top); ::mcrt::note_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ quantised 4-wide layout
// Collapse of the reference-layout binary BVH into 4-wide nodes (64 bytes):
//   w0: origin.xyz (float, the node box minimum) | exponent bytes ex, ey, ez
//       (grid step 2^(e-127) per axis) and the child count
//   w1: qlo.x[4] | qlo.y[4] | qlo.z[4] | qhi.x[4]   (8-bit grid coordinates)
//   w2: qhi.y[4] | qhi.z[4] | 0 | 0
//   w3: child codes (internal 4-wide node index, leaf code, or kNoChild)
// A node takes the two children of a binary node and repeatedly replaces the
// internal child of largest surface area by its two children until it has
// four.  Leaves are the reference's leaves.  Child boxes are rounded outward:
// the builder checks that every grid plane origin + q * step, as an exact real
// number, lies outside the exact child box (the traversal bounds its plane
// distances from that exact value), so a ray that reaches a leaf of the
// reference tree also reaches it here.
namespace {

__device__ __forceinline__ float step_of(uint32_t e) { return __uint_as_float(e << 23); }

// Smallest exponent byte e with extent / 2^(e-127) <= 250 (a normal power of two).
__device__ __forceinline__ uint32_t grid_exponent(float extent) {
    if (!(extent > 0.0f)) return 1u;
    float s = extent / 250.0f;
    uint32_t e = (__float_as_uint(s) >> 23) & 0xffu;     // 2^(e-127) <= s < 2^(e-126)
    if (e == 0u) e = 1u;
    while (e < 254u && step_of(e) * 250.0f < extent) ++e;
    while (e > 1u && step_of(e - 1u) * 250.0f >= extent) --e;
    return e;
}

// Sign of the exact real origin + qs - v (qs = q * step, exact: step is a
// power of two).  The rounded sum s lies within half an ulp of the exact one,
// so s != v decides; at s == v the error-free residual of the sum (Knuth's
// TwoSum: s + err is exactly origin + qs) does.
__device__ __forceinline__ int grid_plane_vs(float origin, float qs, float v) {
    const float s = origin + qs;
    if (s != v) return s < v ? -1 : 1;
    const float bb = s - origin;
    const float err = (origin - (s - bb)) + (qs - bb);
    return err < 0.0f ? -1 : (err > 0.0f ? 1 : 0);
}
__device__ __forceinline__ uint32_t quant_lo(float origin, float step, float v) {
    float q = floorf((v - origin) / step);
    int qi = q < 0.0f ? 0 : (q > 255.0f ? 255 : (int)q);
    while (qi > 0 && grid_plane_vs(origin, (float)qi * step, v) > 0) --qi;
    return (uint32_t)qi;
}
__device__ __forceinline__ uint32_t quant_hi(float origin, float step, float v, bool *ok) {
    float q = ceilf((v - origin) / step);
    int qi = q < 0.0f ? 0 : (q > 255.0f ? 255 : (int)q);
    while (qi < 255 && grid_plane_vs(origin, (float)qi * step, v) < 0) ++qi;
    if (grid_plane_vs(origin, (float)qi * step, v) < 0) *ok = false;
    return (uint32_t)qi;
}

__global__ void k_widen(const mcrt_gpu_bvh_node *nodes, const uint32_t *front, uint32_t n_front, uint32_t level_base,
                        uint32_t next_base, uint32_t *next_front, uint32_t *counter, uint4 *out, uint32_t *bad) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_front) return;
    const uint32_t i = front[k];
    uint32_t set[4] = {i + 1, nodes[i].right_or_offset, kNoChild, kNoChild};
    uint32_t cnt = 2;
    auto area = [&](uint32_t c) {
        const mcrt_gpu_bvh_node &nd = nodes[c];
        float d0 = nd.aabb_max[0] - nd.aabb_min[0], d1 = nd.aabb_max[1] - nd.aabb_min[1],
              d2 = nd.aabb_max[2] - nd.aabb_min[2];
        return d0 * d1 + d1 * d2 + d0 * d2;
    };
    while (cnt < 4) {
        int pick = -1;
        float best = -1.0f;
        for (uint32_t j = 0; j < cnt; ++j) {
            if (nodes[set[j]].prim_count != 0) continue;
            float a = area(set[j]);
            if (a > best) { best = a; pick = (int)j; }
        }
        if (pick < 0) break;
        uint32_t c = set[pick];
        set[pick] = c + 1;
        set[cnt++] = nodes[c].right_or_offset;
    }
    uint32_t n_int = 0;
    for (uint32_t j = 0; j < cnt; ++j) n_int += nodes[set[j]].prim_count == 0 ? 1u : 0u;
    uint32_t base = n_int ? atomicAdd(counter, n_int) : 0u;
    const mcrt_gpu_bvh_node &nd = nodes[i];
    float org[3], stp[3];
    uint32_t ex[3];
    for (int a = 0; a < 3; ++a) {
        org[a] = nd.aabb_min[a];
        ex[a] = grid_exponent(nd.aabb_max[a] - nd.aabb_min[a]);
        stp[a] = step_of(ex[a]);
    }
    uint32_t qlo[3] = {0, 0, 0}, qhi[3] = {0, 0, 0}, refs[4];
    bool ok = true;
    uint32_t r = 0;
    for (uint32_t j = 0; j < 4; ++j) {
        if (j >= cnt) { refs[j] = kNoChild; continue; }
        const mcrt_gpu_bvh_node &c = nodes[set[j]];
        for (int a = 0; a < 3; ++a) {
            qlo[a] |= quant_lo(org[a], stp[a], c.aabb_min[a]) << (8 * j);
            qhi[a] |= quant_hi(org[a], stp[a], c.aabb_max[a], &ok) << (8 * j);
        }
        if (c.prim_count == 0) {
            refs[j] = next_base + base + r;
            next_front[base + r] = set[j];
            ++r;
        } else {
            refs[j] = leaf_code(c.right_or_offset, c.prim_count);
        }
    }
    if (!ok) atomicOr(bad, 1u);
    uint4 *o = out + 4ull * (level_base + k);
    o[0] = make_uint4(__float_as_uint(org[0]), __float_as_uint(org[1]), __float_as_uint(org[2]),
                      ex[0] | (ex[1] << 8) | (ex[2] << 16) | (cnt << 24));
    o[1] = make_uint4(qlo[0], qlo[1], qlo[2], qhi[0]);
    o[2] = make_uint4(qhi[1], qhi[2], 0u, 0u);
    o[3] = make_uint4(refs[0], refs[1], refs[2], refs[3]);
}

}  // namespace

// d_tmp: 2 * n_nodes + 4 words.  d_wide: capacity (n_nodes / 2 + 1) nodes of 64 bytes.
cudaError_t gpu_make_wide4(const mcrt_gpu_bvh_node *d_nodes, uint32_t n_nodes, uint4 *d_wide, uint32_t *n_wide,
                           uint32_t *d_tmp, cudaStream_t st) {
    *n_wide = 0;
    if (n_nodes <= 1) return cudaSuccess;           // a single leaf: traversed without wide nodes
    uint32_t *front[2] = {d_tmp, d_tmp + n_nodes};
    uint32_t *counter = d_tmp + 2 * (size_t)n_nodes;
    uint32_t *bad = counter + 1;
    uint32_t zero = 0;
    cudaMemcpyAsync(front[0], &zero, 4, cudaMemcpyHostToDevice, st);   // root
    cudaMemsetAsync(bad, 0, 4, st);
    uint32_t n_front = 1, level_base = 0;
    int cur = 0;
    for (int guard = 0; n_front > 0; ++guard) {
        if (guard > 4096) return cudaErrorUnknown;
        cudaMemsetAsync(counter, 0, 4, st);
        const uint32_t next_base = level_base + n_front;
        k_widen<<<(n_front + 127) / 128, 128, 0, st>>>(d_nodes, front[cur], n_front, level_base, next_base,
                                                      front[cur ^ 1], counter, d_wide, bad); ::mcrt::note_launch();
        uint32_t n_next = 0;
        cudaMemcpyAsync(&n_next, counter, 4, cudaMemcpyDeviceToHost, st);
        cudaError_t e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
        level_base = next_base;
        n_front = n_next;
        cur ^= 1;
    }
    uint32_t b = 0;
    cudaMemcpyAsync(&b, bad, 4, cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    if (b) return cudaErrorInvalidValue;            // a child box could not be enclosed on the grid
    *n_wide = level_base;
    return cudaSuccess;
}

}  // namespace mcrt
