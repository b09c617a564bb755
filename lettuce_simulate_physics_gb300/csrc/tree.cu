// Tree build for the Barnes-Hut method: Morton keys, onesweep LSD radix sort, permute, key
// restarts, the octree in the reference CPU backend's exact topology and node order, walk groups,
// and the FP64 bottom-up upsweep of monopole and quadrupole moments.
//
// Parity target: the reference CPU backend (src/cpu_backend.cpp:395-664). After an upload (FP64
// positions equal to the float inputs) the keys, the sort permutation, the node array (lo, hi,
// first, nchild in the same indices), the cell geometry and the groups are bit-identical to the
// reference's; the moments use the reference's FP64 operation order, with the fused multiply-adds
// its compiler forms (GCC's default contraction on x86-64-v3 and aarch64: a product fused into the
// sum or difference that is its only use) written out as __fma_rn, everything else rounded per
// operation. rcrit2 and the walk's opening distance use the same fused float forms.
//
// Construction (no level-by-level loop, no recursion):
//  1. bbox and key frame (FP64), keys (src/cpu_backend.cpp:418-428 formula), identity values.
//  2. Onesweep radix sort (Adinets & Merrill 2022) by the leading key digits the tree's depth needs:
//     histograms of all 8-bit digits with the keys, then one kernel per digit with decoupled
//     look-back across tiles; ties ordered by the whole keys in the gather. Stable, so the
//     permutation equals the reference's.
//  3. Key restarts: runs of > 16 identical keys are re-keyed in their own bounding cube (the
//     reference's rekey, src/cpu_backend.cpp:503-530) and sorted by the new keys inside each run;
//     runs whose composite keys still tie are re-keyed again, up to FRAMES frames (depth 126).
//     Composite keys (frame 0, then the restart frames) order the bodies as the reference's nested
//     rekeys do, and a common-prefix length over them drives steps 4-6.
//  4. Leaves from key windows (k_leaves): body i's leaf depth is 1 + the deepest common octal prefix of
//     any window of LEAF_MAX+1 consecutive sorted keys that contains i (the first depth at which its
//     cell holds <= LEAF_MAX bodies); group depth likewise with windows of group_max+1. The same
//     launch numbers the leaves and their nodes by one decoupled look-back.
//  5. Octree nodes in pre-order (k_nodes): leaf l owns the ancestors at depths c+1 .. depth-1, c =
//     common prefix with the previous leaf (Karras 2012's adjacent-key rule in octree form); body
//     ranges and parents follow from searches over the sorted keys, and every node sets its octant's
//     bit in its parent's child mask.
//  6. Node indices of the reference (children contiguous, child blocks in parent pre-order): first
//     child of v = 1 + exclusive scan of the masks' bit counts over pre-order (k_node_scan), a child's
//     place under its parent the bits below its own (k_nodes_out).
//  7. Upsweep in FP64, children always combined in index order: one launch for the leaves (one
//     thread per leaf, leaves bucketed by body count; eight lanes per leaf in small trees), then the
//     depths from the deepest (eight lanes per node, each sequential sum folded by one lane), the
//     narrow depths at the top, or all of a small tree's, together in one launch. The group boxes are
//     computed on a side stream meanwhile. (A single-launch form in which the last-arriving child of
//     each node combines it was measured slower: its combines run one node per thread in sparse
//     warps, and an FP64 warp instruction costs the same however few lanes are active.)
// Steps 4 to 6 are four launches (they were 22 with their scans, and 13 clears; build phase 238 ->
// 146 us at 8191 bodies, 289 -> 200 at 1e5, 514 -> 385 on the 1e6 disk, 4.16 -> 3.26 ms at 1.6e7).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <vector>

#include "engine.cuh"

namespace lg {

namespace {

constexpr int LEAF_MAX = 16;   // src/cpu_backend.cpp:24
constexpr int MAX_LEVEL = 21;  // :28
constexpr int FRAMES = 6;                     // key frames: frame 0 and up to five key restarts
constexpr int MAX_DEPTH = FRAMES * MAX_LEVEL;  // 126: depths fit the 8-bit depth fields
constexpr int BS = 256;

// Key restart frames, in device memory. Frame f >= 1 re-keys, in its own bounding cube, every run
// of more than LEAF_MAX bodies whose keys in frames 0..f-1 are all equal (the reference's rekey at
// level kMaxLevel of frame f-1, src/cpu_backend.cpp:536-544); its runs are sorted by the new keys.
struct FrameTable {
    const uint64_t* key[FRAMES];  // [f >= 1] frame-f keys by sorted position (0 outside its runs)
    const int* runid[FRAMES];     // [f >= 1] the body's run in frame f, or -1
    const double* cube[FRAMES];   // [f >= 1] per run: origin xyz, side (0: coincident), 2^21 / side
    const uint8_t* nfr;           // per body: frames it has keys in (1 + its non-coincident restarts)
    int nf;                       // frames in use
};

inline int grid_for(long long n, int bs) { return static_cast<int>((n + bs - 1) / bs); }

// Whether a build's kernels overlap their launches. It hides 1 to 2 us a kernel where the kernels are
// that short, and costs where they run in several waves, as the waiting blocks take the place of
// running ones. Sort + build, plain -> overlapped, Plummer: 8191 bodies 198 -> 176 us, 65536 242 ->
// 210, 131072 277 -> 250, 262144 304 -> 337, 4e5 351 -> 412, 1.6e7 5370 -> 6170.
inline bool overlap(int n) { return n <= 160000; }

// ---- sort control --------------------------------------------------------------------------
constexpr int RADIX = 256;
constexpr int PASSES = 8;
#ifndef LG_SORT_IPT
#define LG_SORT_IPT 8
#endif
constexpr int SORT_BS = 256;
constexpr int SORT_IPT = LG_SORT_IPT;  // keys per thread of a sort tile
constexpr int SORT_TILE = SORT_BS * SORT_IPT;
constexpr unsigned FLAG_AGG = 1u << 30, FLAG_INC = 2u << 30, VAL_MASK = (1u << 30) - 1;
#ifndef LG_LB_BATCH
#define LG_LB_BATCH 4
#endif
constexpr int LB_BATCH = LG_LB_BATCH;  // predecessors read per look-back round trip

// Device memory that one kernel zeroes for those after it (16-byte words).
struct ZeroSpan {
    uint4* p;
    size_t words;
};
constexpr int ZSPANS = 5;
struct ZeroList {
    ZeroSpan span[ZSPANS];
};

}  // namespace

struct TreeState {
    // sort
    DevBuf keysA, keysB, valsA, valsB, hist, lookback;
    bool clusters_of_16 = false;  // k_combine_top may be launched as one
    int known_depth = 0;  // the tree's depth at its last exact build, with headroom (0: unknown): digits to sort
    // sorted frame-0 keys, per-body tree data
    DevBuf skey, leafid;
    // frame, key-restart runs and frames (index 0 of the per-frame buffers unused)
    DevBuf frame, runs, counts, key1tmp, nfr, ftab;
    DevBuf fkey[FRAMES], frunid[FRAMES], fcube[FRAMES];
    int nframes = 1;  // key frames of the last restarted build
    // leaves
    DevBuf leaf_first, leaf_depth, leaf_gdepth, leaf_c, leaf_pre, leaf_node, leaf_state;
    // pre-order nodes
    DevBuf pn_lohi, pn_meta, pn_parent, pn_first, node_zero;
    // reference-order nodes
    DevBuf nd_test, nd_cell, nd_geo, nd_parent;
    // groups
    DevBuf grp_node, grp_range, grp_box, grp_order;
    // upsweep order
    DevBuf dep_nodes, leaf_order;
    // scan state (merged walk groups)
    DevBuf scan_state, scan_ctr;
    size_t K = 0, T = 0, ngroups = 0;  // sizes the last build was launched with
    size_t leaves = 0, nodes = 0;      // what the last exact build counted (K and T: with headroom)
    int max_depth = 0;
    bool restarted = false;
    int group_max = 128;
    // Sync-free builds: sizes from the previous build with headroom; verified after the walk.
    bool have_guess = false;
    bool restart_mode = false;  // key restarts were needed last time: check for them on the host
    bool speculative = false;   // the current build used guessed sizes / assumed no restart
    double theta = 0.6;
    // Forest (ensemble) configuration: the tree covers bodies [0, n_tree) of nsys systems whose
    // ranges are sys_off[0..nsys] (device); sys[i] is body i's system (device); per-system inverse
    // opening angles. n_tree < 0 means one system over all bodies.
    int n_tree = -1;
    int nsys = 1;
    const uint32_t* sys = nullptr;
    const uint32_t* sys_off = nullptr;
    const float* inv_theta_sys = nullptr;
    uint64_t generation = 0;  // bumped by every build that may grow (reallocate) tree buffers
    DevBuf mkeys;   // Morton keys in the bodies' order before the sort
    // merged walk groups
    bool merged = false;
    DevBuf mcount, moff, mrange, mbox;
    DevBuf sticky;  // graph mode: sticky word set when a sync-free build misses
};

namespace {

void destroy_tree(TreeState* t) { delete t; }

// ---- device helpers --------------------------------------------------------------------------
__device__ __forceinline__ uint64_t spread21(uint64_t v) {
    v &= 0x1fffffULL;
    v = (v | v << 32) & 0x1f00000000ffffULL;
    v = (v | v << 16) & 0x1f0000ff0000ffULL;
    v = (v | v << 8) & 0x100f00f00f00f00fULL;
    v = (v | v << 4) & 0x10c30c30c30c30c3ULL;
    v = (v | v << 2) & 0x1249249249249249ULL;
    return v;
}

// Quantised coordinate of src/cpu_backend.cpp:423: uint64(clamp((v - o) * s, 0, lim)), FP64,
// round-to-nearest products, truncation. The clamp is taken after the conversion, in integers:
// the truncating conversion saturates (negative values give 0), and lim = 2^21 - 1 is an integer,
// so min(trunc(q), lim) equals trunc(clamp(q, 0, lim)) for every q, with two FP64 operations fewer.
constexpr uint64_t QLIM = (1ull << MAX_LEVEL) - 1;
__device__ __forceinline__ uint64_t quantize(double v, double o, double s) {
    const uint64_t u = __double2ull_rz(__dmul_rn(__dsub_rn(v, o), s));
    return u < QLIM ? u : QLIM;
}

__device__ __forceinline__ uint64_t morton(double x, double y, double z, double ox, double oy, double oz, double s) {
    return spread21(quantize(x, ox, s)) << 2 | spread21(quantize(y, oy, s)) << 1 | spread21(quantize(z, oz, s));
}

// Common octal prefix (0..21) of two 63-bit keys.
__device__ __forceinline__ int cpl21(uint64_t a, uint64_t b) { return (__clzll(a ^ b) - 1) / 3; }

// Forest builds (many independent systems in one pipeline) pass a per-body system index `sys`:
// bodies of different systems share no prefix (-1), so no leaf, node or group spans two systems.
// Single-system builds pass null.

// Common octal prefix over the restart frames 1..nf-1 of bodies whose frame-0 keys are equal:
// 21 per equal frame, 21 nf when every frame is equal.
__device__ __forceinline__ int cpl_frames(const FrameTable* ft, int i, int j) {
    const int nf = ft->nf;
    for (int f = 1; f < nf; ++f) {
        const uint64_t a = ft->key[f][i], b = ft->key[f][j];
        if (a != b) return MAX_LEVEL * f + cpl21(a, b);
    }
    return MAX_LEVEL * nf;
}

// Common octal prefix (0..126) of the composite keys (frame 0, then the restart frames) of bodies
// i and j; -1 across systems. ft is null when no key restart was needed.
__device__ __forceinline__ int cpl_key(const uint32_t* sys, const uint64_t* k0, const FrameTable* ft, int i, int j) {
    if (sys && sys[i] != sys[j]) return -1;
    const uint64_t a = k0[i], b = k0[j];
    if (a != b || !ft) return cpl21(a, b);
    return cpl_frames(ft, i, j);
}

__device__ __forceinline__ uint32_t sys_of(const uint32_t* sys, int i) { return sys ? sys[i] : 0u; }

// Octal digit of the composite key at depth d (1-based): digit d - 21 f of frame f = (d - 1) / 21.
__device__ __forceinline__ int digit_at(const uint64_t* k0, const FrameTable* ft, int i, int d) {
    const int f = (d - 1) / MAX_LEVEL;
    const uint64_t k = f == 0 ? k0[i] : ft->key[f][i];
    return static_cast<int>((k >> (3 * (MAX_LEVEL * (f + 1) - d))) & 7);
}

// ---- frame and keys --------------------------------------------------------------------------
// frame: [0..2] origin, [3] side, [4] scale 2^21/side.
// Bounding-box minima and maxima on the integer pipes: a double's bits mapped to a signed 64-bit
// integer that orders as the values do (-0 below +0), NaN mapped to +inf for minima and to -inf
// for maxima, so that it is ignored as fmin and fmax ignore it. FP64 issue is scarce on this part.
__device__ __forceinline__ long long ord_bits(long long b) { return b ^ ((b >> 63) & 0x7fffffffffffffffLL); }
__device__ __forceinline__ bool nan_bits(long long b) { return (b & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL; }
__device__ __forceinline__ long long ord_lo(double d) {
    const long long b = __double_as_longlong(d);
    return nan_bits(b) ? 0x7ff0000000000000LL : ord_bits(b);
}
__device__ __forceinline__ long long ord_hi(double d) {
    const long long b = __double_as_longlong(d);
    return nan_bits(b) ? ord_bits(static_cast<long long>(0xfff0000000000000ULL)) : ord_bits(b);
}
__device__ __forceinline__ double ord_value(long long k) { return __longlong_as_double(ord_bits(k)); }

// v[0..2] minima, v[3..5] maxima (ordered integers) of the block's bodies, reduced over the block
// into sh (lane 0 of each warp) and returned by thread 0 in v.
__device__ __forceinline__ void box_block_reduce(long long (&v)[6], long long (*sh)[BS / 32]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        for (int o = 16; o > 0; o >>= 1) {
            const long long t = __shfl_down_sync(0xffffffffu, v[c], o);
            v[c] = c < 3 ? min(v[c], t) : max(v[c], t);
        }
        if (lane == 0) sh[c][w] = v[c];
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int c = 0; c < 6; ++c) {
            long long r = sh[c][0];
            for (int u = 1; u < BS / 32; ++u) r = c < 3 ? min(r, sh[c][u]) : max(r, sh[c][u]);
            v[c] = r;
        }
}

__device__ __forceinline__ void box_init(long long (&v)[6]) {
    for (int c = 0; c < 3; ++c) {
        v[c] = ord_bits(0x7ff0000000000000LL);                                   // +inf
        v[3 + c] = ord_bits(static_cast<long long>(0xfff0000000000000ULL));      // -inf
    }
}

__device__ __forceinline__ void box_add(long long (&v)[6], double x, double y, double z) {
    v[0] = min(v[0], ord_lo(x));
    v[1] = min(v[1], ord_lo(y));
    v[2] = min(v[2], ord_lo(z));
    v[3] = max(v[3], ord_hi(x));
    v[4] = max(v[4], ord_hi(y));
    v[5] = max(v[5], ord_hi(z));
}

// src/cpu_backend.cpp:404-406: origin = the minima; side = max extent, widened by 1e-6; 1 if all
// coincide; scale = 2^21 / side.
__device__ __forceinline__ void write_frame(const long long (&v)[6], double* f) {
    double r[6];
    for (int c = 0; c < 6; ++c) r[c] = ord_value(v[c]);
    double side = fmax(fmax(__dsub_rn(r[3], r[0]), __dsub_rn(r[4], r[1])), __dsub_rn(r[5], r[2]));
    side = side > 0 ? __dmul_rn(side, 1 + 1e-6) : 1.0;
    f[0] = r[0];
    f[1] = r[1];
    f[2] = r[2];
    f[3] = side;
    f[4] = __ddiv_rn(static_cast<double>(1u << MAX_LEVEL), side);
}

__device__ __forceinline__ void zero_spans(const ZeroList& z) {
#pragma unroll
    for (int q = 0; q < ZSPANS; ++q)
        for (size_t k = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; k < z.span[q].words;
             k += static_cast<size_t>(gridDim.x) * blockDim.x)
            z.span[q].p[k] = make_uint4(0u, 0u, 0u, 0u);
}

__global__ void k_frame(const BodyArrays b, int n, long long* partial, unsigned* ticket, double* frame, ZeroList z) {
    pdl_wait();
    zero_spans(z);
    __shared__ long long sh[6][BS / 32];
    __shared__ bool last;
    long long v[6];
    box_init(v);
    for (int i = blockIdx.x * BS + threadIdx.x; i < n; i += gridDim.x * BS) box_add(v, b.x[i], b.y[i], b.z[i]);
    box_block_reduce(v, sh);
    if (threadIdx.x == 0) {
        for (int c = 0; c < 6; ++c) partial[blockIdx.x * 6 + c] = v[c];
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    box_init(v);
    for (int blk = threadIdx.x; blk < static_cast<int>(gridDim.x); blk += BS)
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            const long long t = __ldcg(&partial[blk * 6 + c]);
            v[c] = c < 3 ? min(v[c], t) : max(v[c], t);
        }
    __syncthreads();
    box_block_reduce(v, sh);
    if (threadIdx.x == 0) {
        write_frame(v, frame);
        *ticket = 0;
    }
}

// Morton keys, the keys the sort works on (their values, the positions, are left to the first pass),
// and the digit histograms of the sort's passes. The sort key is the leading `levels` octal digits
// of the Morton key, under the system's index with sys_key. One histogram per block in shared
// memory, blocks few enough that adding them up stays cheap.
__global__ void k_keys(const uint32_t* __restrict__ sys, const BodyArrays b, int n, const double* __restrict__ frame,
                       uint64_t* __restrict__ mkeys, uint64_t* __restrict__ keys, int levels, int passes, int sys_key,
                       unsigned* __restrict__ hist) {
    pdl_wait();
    __shared__ unsigned h[PASSES * RADIX];
    for (int k = threadIdx.x; k < passes * RADIX; k += blockDim.x) h[k] = 0;
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t s = sys_of(sys, i);
        const double* f = frame + 5 * s;
        const uint64_t m = morton(b.x[i], b.y[i], b.z[i], f[0], f[1], f[2], f[4]);
        uint64_t k = m >> (3 * (MAX_LEVEL - levels));
        if (sys_key) k |= static_cast<uint64_t>(s) << (3 * levels);
        mkeys[i] = m;
        keys[i] = k;
        for (int p = 0; p < passes; ++p) atomicAdd(&h[p * RADIX + static_cast<int>((k >> (8 * p)) & 255)], 1u);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < passes * RADIX; k += blockDim.x)
        if (h[k]) atomicAdd(&hist[k], h[k]);
}

// Forest: one block per system computes its key frame over its body range [off[s], off[s + 1]).
__global__ void k_frame_sys(const BodyArrays b, const uint32_t* __restrict__ off, double* frame, ZeroList z) {
    pdl_wait();
    zero_spans(z);
    __shared__ long long sh[6][BS / 32];
    const uint32_t lo = off[blockIdx.x], hi = off[blockIdx.x + 1];
    long long v[6];
    box_init(v);
    for (uint32_t i = lo + threadIdx.x; i < hi; i += BS) box_add(v, b.x[i], b.y[i], b.z[i]);
    box_block_reduce(v, sh);
    if (threadIdx.x == 0) write_frame(v, frame + 5 * blockIdx.x);
}

// keys[i] = (system of body vals[i]): the second key of the forest's (system, Morton) sort.
__global__ void k_sys_keys(const uint32_t* __restrict__ sys, const uint32_t* __restrict__ vals,
                           uint64_t* __restrict__ keys, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) keys[i] = sys_of(sys, static_cast<int>(vals[i]));
}

// ---- onesweep radix sort ---------------------------------------------------------------------
// Digit histograms of keys already in memory (the key restarts' sorts).
__global__ void k_sort_hist(const uint64_t* __restrict__ keys, int n, int passes, unsigned* __restrict__ hist) {
    __shared__ unsigned h[PASSES * RADIX];
    for (int k = threadIdx.x; k < passes * RADIX; k += blockDim.x) h[k] = 0;
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint64_t k = keys[i];
        for (int p = 0; p < passes; ++p) atomicAdd(&h[p * RADIX + static_cast<int>((k >> (8 * p)) & 255)], 1u);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < passes * RADIX; k += blockDim.x)
        if (h[k]) atomicAdd(&hist[k], h[k]);
}

// Exclusive sum over the block's 256 threads (sh: one word per warp); begins with a barrier.
__device__ __forceinline__ unsigned block_excl_sum(unsigned v, unsigned* sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    __syncthreads();
    if (lane == 31) sh[w] = incl;
    __syncthreads();
    unsigned before = 0;
#pragma unroll
    for (int u = 0; u < SORT_BS / 32; ++u)
        if (u < w) before += sh[u];
    return before + incl - v;
}

// One pass: (src_k, src_v) to (dst_k, dst_v) by the digit at `shift`; src_v null: values are the
// positions. hist: the digit's counts over all keys; tile_ctr and lookback start at zero.
__global__ void __launch_bounds__(SORT_BS) k_sort_pass(const uint64_t* __restrict__ src_k,
                                                       const uint32_t* __restrict__ src_v,
                                                       uint64_t* __restrict__ dst_k, uint32_t* __restrict__ dst_v, int n,
                                                       int shift, const unsigned* __restrict__ hist,
                                                       unsigned* __restrict__ lookback, unsigned* tile_ctr,
                                                       unsigned* err) {
    pdl_wait();
    __shared__ unsigned warp_hist[SORT_BS / 32][RADIX];
    __shared__ unsigned gbase[RADIX];       // global start of each digit for this tile
    __shared__ unsigned tstart[RADIX];      // start of each digit in the staged tile
    __shared__ uint64_t stage_k[SORT_TILE]; // the tile in digit order
    __shared__ uint32_t stage_v[SORT_TILE];
    __shared__ unsigned tile_s, scan_s[SORT_BS / 32];
    static_assert(SORT_BS == RADIX, "one thread per digit");
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid == 0) tile_s = atomicAdd(tile_ctr, 1u);
    for (int k = tid; k < (SORT_BS / 32) * RADIX; k += SORT_BS) (&warp_hist[0][0])[k] = 0;
    // The digit's start among all keys; the barriers also publish tile_s and the cleared counts.
    const unsigned digit_start = block_excl_sum(hist[tid], scan_s);
    const unsigned tile = tile_s;
    const int tile0 = tile * SORT_TILE;
    const int wbase = tile0 + w * (32 * SORT_IPT);
    const int tile_n = min(SORT_TILE, n - tile0);

    uint64_t key[SORT_IPT];
    uint32_t val[SORT_IPT];
    unsigned rank[SORT_IPT];
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < SORT_IPT; ++r) {
        const int i = wbase + r * 32 + lane;
        key[r] = i < n ? src_k[i] : 0;
        val[r] = i < n ? (src_v ? src_v[i] : static_cast<uint32_t>(i)) : 0;
    }
    // Stable rank inside the tile: keys in index order (warp, round, lane).
#pragma unroll
    for (int r = 0; r < SORT_IPT; ++r) {
        const bool valid = wbase + r * 32 + lane < n;
        const int d = valid ? static_cast<int>((key[r] >> shift) & 255) : -1 - lane;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const unsigned before = __popc(peers & lt);
        unsigned basev = 0;
        if (valid) basev = warp_hist[w][d];
        __syncwarp();
        if (valid && before == 0) warp_hist[w][d] = basev + __popc(peers);
        __syncwarp();
        rank[r] = basev + before;
    }
    __syncthreads();
    {
        // Per digit (thread d): offsets of the warps inside the digit, the tile's count, then the
        // decoupled look-back across tiles for the digit's global start.
        const int d = tid;
        unsigned run = 0;
#pragma unroll
        for (int u = 0; u < SORT_BS / 32; ++u) {
            const unsigned c = warp_hist[u][d];
            warp_hist[u][d] = run;
            run += c;
        }
        const unsigned tile_count = run;
        volatile unsigned* lb = lookback + static_cast<size_t>(tile) * RADIX;
        unsigned prefix = 0;
        if (tile == 0) {
            lb[d] = FLAG_INC | tile_count;
        } else {
            lb[d] = FLAG_AGG | tile_count;
            // Look back LB_BATCH predecessors per round trip: their flags are read together and
            // taken in order (aggregates added until an inclusive prefix; an unpublished tile is
            // waited for, keeping what was added before it).
            int j = static_cast<int>(tile) - 1;
            unsigned spins = 0;
            while (j >= 0) {
                unsigned sv[LB_BATCH];
#pragma unroll
                for (int q = 0; q < LB_BATCH; ++q)
                    sv[q] = j - q >= 0 ? *reinterpret_cast<volatile const unsigned*>(
                                             &lookback[static_cast<size_t>(j - q) * RADIX + d])
                                       : FLAG_INC;
                int taken = 0;
                bool inc = false;
#pragma unroll
                for (int q = 0; q < LB_BATCH; ++q) {
                    if (inc || taken < q) break;
                    if (sv[q] & (FLAG_INC | FLAG_AGG)) {
                        prefix += sv[q] & VAL_MASK;
                        inc = (sv[q] & FLAG_INC) != 0;
                        ++taken;
                    }
                }
                if (inc) break;
                j -= taken;
                if (taken == 0 && ++spins > kSpinCap) {
                    atomicOr(err, kErrWaitTimeout);
                    break;
                }
            }
            lb[d] = FLAG_INC | ((prefix + tile_count) & VAL_MASK);
        }
        gbase[d] = digit_start + prefix;
        tstart[d] = block_excl_sum(tile_count, scan_s);
    }
    __syncthreads();
    // Stage the tile in digit order (tile-local position = digit start + rank within the digit).
#pragma unroll
    for (int r = 0; r < SORT_IPT; ++r) {
        if (wbase + r * 32 + lane < n) {
            const int d = static_cast<int>((key[r] >> shift) & 255);
            const unsigned pos = tstart[d] + warp_hist[w][d] + rank[r];
            stage_k[pos] = key[r];
            stage_v[pos] = val[r];
        }
    }
    __syncthreads();
    // Write out: consecutive staged entries of one digit go to consecutive global addresses.
    for (int p = tid; p < tile_n; p += SORT_BS) {
        const uint64_t k = stage_k[p];
        const int d = static_cast<int>((k >> shift) & 255);
        const unsigned gpos = gbase[d] + (p - tstart[d]);
        if (gpos < static_cast<unsigned>(n)) {  // false only after a wait that ran out
            dst_k[gpos] = k;
            dst_v[gpos] = stage_v[p];
        }
    }
}

// Gathers every body array into the other body set in the sorted order, and the Morton keys with
// them (mkeys: by body before the sort). A sort by the leading digits only (partial) leaves runs of
// bodies with equal sort keys in their former order; each body of such a run finds its place by
// counting the run's bodies with a smaller Morton key (or an equal one, before it), so the order is
// that of a stable sort by the whole keys. A run of more than LEAF_MAX is left as it is and
// flagged: the tree is then deeper than the sorted digits, and the sort is redone with all of them.
// key1_in (optional): a second key carried through the permutation (no partial runs then).
// After a wait of the passes that ran out (*err) the permutation is not one: every body keeps its
// place, and the kernels that follow do nothing (build_ok).
__global__ void k_permute(const BodyArrays src, BodyArrays dst, const uint64_t* __restrict__ keys,
                          const uint32_t* __restrict__ vals, const uint64_t* __restrict__ mkeys,
                          uint64_t* __restrict__ skey, const uint64_t* __restrict__ key1_in,
                          uint64_t* __restrict__ key1_out, int n, int n_total, int partial, unsigned* long_run,
                          const unsigned* err) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_total) return;
    int to = i;
    uint32_t j = static_cast<uint32_t>(i);  // bodies past the tree's range (the forest's direct systems) stay
    const uint32_t from = vals[min(i, n - 1)], ran_out = *err & kErrWaitTimeout;  // one round trip for both
    if (i < n && !ran_out) {
        j = from;
        if (skey) {
            const uint64_t m = mkeys[j];
            if (partial) {
                const uint64_t k = keys[i];
                int a = i, e = i + 1;
                while (a > 0 && i - a <= LEAF_MAX && keys[a - 1] == k) --a;
                while (e < n && e - i <= LEAF_MAX && keys[e] == k) ++e;
                if (e - a > LEAF_MAX) {
                    *long_run = 1u;
                } else if (e - a > 1) {
                    to = a;
                    for (int q = a; q < e; ++q) {
                        const uint64_t mq = mkeys[vals[q]];
                        to += mq < m || (mq == m && q < i) ? 1 : 0;
                    }
                }
            }
            skey[to] = m;
        }
        if (key1_in) key1_out[to] = key1_in[j];
    } else if (i < n) {
        if (skey) skey[i] = mkeys[i];
        if (key1_in) key1_out[i] = key1_in[i];
    }
    dst.x[to] = src.x[j];
    dst.y[to] = src.y[j];
    dst.z[to] = src.z[j];
    dst.hm[to] = src.hm[j];
    dst.lo[to] = src.lo[j];
    dst.vx[to] = src.vx[j];
    dst.vy[to] = src.vy[j];
    dst.vz[to] = src.vz[j];
    dst.m[to] = src.m[j];
    dst.id[to] = src.id[j];
    dst.cost[to] = src.cost[j];
    dst.level[to] = src.level[j];
}

// ---- exclusive scan (decoupled look-back) ----------------------------------------------------
constexpr int SCAN_BS = 256, SCAN_IPT = 8, SCAN_TILE = SCAN_BS * SCAN_IPT;
constexpr unsigned long long SFLAG_AGG = 1ull << 62, SFLAG_INC = 2ull << 62, SVAL = (1ull << 62) - 1;

__global__ void __launch_bounds__(SCAN_BS) k_scan(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int n,
                                                 unsigned long long* state, unsigned* counter, uint32_t* total,
                                                 unsigned* err) {
    __shared__ unsigned tile_s;
    __shared__ unsigned long long warp_tot[SCAN_BS / 32];
    __shared__ unsigned long long prefix_s;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid == 0) tile_s = atomicAdd(counter, 1u);
    __syncthreads();
    const unsigned tile = tile_s;
    const long long base = static_cast<long long>(tile) * SCAN_TILE + static_cast<long long>(tid) * SCAN_IPT;
    uint32_t v[SCAN_IPT];
    unsigned long long tsum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_IPT; ++k) {
        v[k] = base + k < n ? in[base + k] : 0u;
        tsum += v[k];
    }
    // Warp inclusive scan of thread sums.
    unsigned long long incl = tsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    if (tid == 0) {
        unsigned long long run = 0;
        for (int u = 0; u < SCAN_BS / 32; ++u) {
            unsigned long long c = warp_tot[u];
            warp_tot[u] = run;
            run += c;
        }
        const unsigned long long block_total = run;
        volatile unsigned long long* st = state;
        unsigned long long prefix = 0;
        if (tile == 0) {
            st[0] = SFLAG_INC | block_total;
        } else {
            st[tile] = SFLAG_AGG | block_total;
            long long j = static_cast<long long>(tile) - 1;
            unsigned spins = 0;
            while (j >= 0) {  // LB_BATCH predecessors per round trip, taken in order (as in the sort)
                unsigned long long sv[LB_BATCH];
#pragma unroll
                for (int q = 0; q < LB_BATCH; ++q) {
                    const unsigned long long v = j - q >= 0 ? st[j - q] : 0ull;
                    sv[q] = j - q >= 0 ? v : static_cast<unsigned long long>(SFLAG_INC);
                }
                int taken = 0;
                bool inc = false;
#pragma unroll
                for (int q = 0; q < LB_BATCH; ++q) {
                    if (inc || taken < q) break;
                    if (sv[q] & (SFLAG_INC | SFLAG_AGG)) {
                        prefix += sv[q] & SVAL;
                        inc = (sv[q] & SFLAG_INC) != 0;
                        ++taken;
                    }
                }
                if (inc) break;
                j -= taken;
                if (taken == 0 && ++spins > kSpinCap) { atomicOr(err, kErrWaitTimeout); break; }
            }
            st[tile] = SFLAG_INC | ((prefix + block_total) & SVAL);
        }
        prefix_s = prefix;
        const unsigned ntiles = static_cast<unsigned>((n + SCAN_TILE - 1) / SCAN_TILE);
        if (tile == ntiles - 1 && total) *total = static_cast<uint32_t>(prefix + block_total);
    }
    __syncthreads();
    unsigned long long run = prefix_s + warp_tot[w] + (incl - tsum);
#pragma unroll
    for (int k = 0; k < SCAN_IPT; ++k) {
        if (base + k < n) out[base + k] = static_cast<uint32_t>(run);
        run += v[k];
    }
}

// ---- key restarts ----------------------------------------------------------------------------
// The runs of frame f: maximal ranges of more than LEAF_MAX bodies of one system whose keys in
// frames 0..f-1 are all equal, among the bodies re-keyed in every earlier frame (nfr == f; all
// bodies for f = 1, where nfr and ft are null): appended as (start, end). ft holds frames 0..f-1.
__global__ void k_find_runs(const uint32_t* __restrict__ sys, const uint64_t* __restrict__ skey,
                            const FrameTable* ft, const uint8_t* __restrict__ nfr, int f, int n, uint2* runs,
                            unsigned* count, int cap) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i + LEAF_MAX >= n) return;
    if (nfr && nfr[i] != f) return;
    const int full = MAX_LEVEL * f;
    if (i > 0 && cpl_key(sys, skey, ft, i - 1, i) >= full) return;
    if (cpl_key(sys, skey, ft, i, i + LEAF_MAX) < full) return;
    int lo = i + LEAF_MAX, hi = n;  // first index with a different (system, composite key)
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (cpl_key(sys, skey, ft, i, mid) >= full) lo = mid + 1;
        else hi = mid;
    }
    const unsigned r = atomicAdd(count, 1u);
    if (static_cast<int>(r) < cap) runs[r] = make_uint2(static_cast<unsigned>(i), static_cast<unsigned>(lo));
}

// One block per run: FP64 bounding box (src/cpu_backend.cpp:505-512); cube = (mn, side, scale),
// side 0 marks coincident bodies (kept as one leaf).
__global__ void k_run_cube(const BodyArrays b, const uint2* runs, double* cube) {
    __shared__ double sh[6][BS / 32];
    const uint2 r = runs[blockIdx.x];
    double v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    for (unsigned i = r.x + threadIdx.x; i < r.y; i += BS) {
        double p[3] = {b.x[i], b.y[i], b.z[i]};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            v[c] = fmin(v[c], p[c]);
            v[3 + c] = fmax(v[3 + c], p[c]);
        }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        for (int o = 16; o > 0; o >>= 1) {
            double t = __shfl_down_sync(0xffffffffu, v[c], o);
            v[c] = c < 3 ? fmin(v[c], t) : fmax(v[c], t);
        }
        if (lane == 0) sh[c][w] = v[c];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double q[6];
        for (int c = 0; c < 6; ++c) {
            q[c] = sh[c][0];
            for (int u = 1; u < BS / 32; ++u) q[c] = c < 3 ? fmin(q[c], sh[c][u]) : fmax(q[c], sh[c][u]);
        }
        double side = fmax(fmax(__dsub_rn(q[3], q[0]), __dsub_rn(q[4], q[1])), __dsub_rn(q[5], q[2]));
        double* o = cube + 5 * blockIdx.x;
        o[0] = q[0];
        o[1] = q[1];
        o[2] = q[2];
        if (side == 0) {
            o[3] = 0;
            o[4] = 0;
        } else {
            side = __dmul_rn(side, 1 + 1e-6);
            o[3] = side;
            o[4] = __ddiv_rn(static_cast<double>(1u << MAX_LEVEL), side);
        }
    }
}

// Frame-f keys of the bodies of non-coincident runs (0 elsewhere, from a fill); runid = the run's
// index (-1 elsewhere, from a fill); nfr = f + 1 for the re-keyed bodies.
__global__ void k_run_keys(const BodyArrays b, const uint2* runs, const double* cube, uint64_t* key1, int* runid,
                           uint8_t* nfr, int f) {
    const uint2 r = runs[blockIdx.x];
    const double* c = cube + 5 * blockIdx.x;
    const bool rekeyed = c[3] > 0;
    for (unsigned i = r.x + threadIdx.x; i < r.y; i += BS) {
        runid[i] = static_cast<int>(blockIdx.x);
        if (rekeyed) {
            key1[i] = morton(b.x[i], b.y[i], b.z[i], c[0], c[1], c[2], c[4]);
            nfr[i] = static_cast<uint8_t>(f + 1);
        }
    }
}

// Second key of the stable (run, frame key) sort: the run's first position for bodies of a run,
// the body's own position otherwise, so that every body stays inside its run.
__global__ void k_seg_keys(const uint32_t* __restrict__ vals, const int* __restrict__ runid,
                           const uint2* __restrict__ runs, uint64_t* __restrict__ keys, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t j = vals[i];
    const int r = runid[j];
    keys[i] = r >= 0 ? runs[r].x : j;
}

__global__ void k_put_table(FrameTable v, FrameTable* dst) { *dst = v; }

__global__ void k_fill_u64(uint64_t* a, uint64_t v, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = v;
}
__global__ void k_fill_i32(int* a, int v, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = v;
}

// ---- leaves ----------------------------------------------------------------------------------
// One decoupled look-back over the sorted bodies gives the leaves and their nodes: leaf depths, leaf
// starts, every leaf's index, range and first pre-order node, in one launch. (As depth, flag, scan,
// information, index and second-scan launches with their clears it was 13 operations.) Latency
// bound below 1e5 bodies; at 1e6 it reads the keys once and writes 4 bytes a body and 14 a leaf.
//
// Exclusive prefix of the tile from its predecessors' published sums (one warp, 32 predecessors a
// round trip): state words carry a flag (SFLAG_AGG: the tile's own sum, SFLAG_INC: the sum up to and
// including it) over two 31-bit sums.
constexpr unsigned long long TWO31 = (1ull << 31) - 1;
__device__ unsigned long long look_back(volatile unsigned long long* state, int tile, int lane, unsigned* err) {
    unsigned long long prefix = 0;
    unsigned spins = 0;
    for (int j = tile - 1; j >= 0; j -= 32) {
        unsigned long long v;
        unsigned inc, need;
        for (;;) {
            v = j - lane >= 0 ? state[j - lane] : static_cast<unsigned long long>(SFLAG_INC);
            inc = __ballot_sync(0xffffffffu, (v & SFLAG_INC) != 0);
            // The predecessors needed: up to the nearest inclusive one, or all 32.
            need = inc ? (inc & (0u - inc)) * 2u - 1u : 0xffffffffu;
            if (!(~__ballot_sync(0xffffffffu, (v & (SFLAG_INC | SFLAG_AGG)) != 0) & need)) break;
            if (++spins > kSpinCap) {
                if (lane == 0) atomicOr(err, kErrWaitTimeout);
                break;
            }
        }
        unsigned long long add = (need >> lane) & 1u ? v & SVAL : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
        prefix += add;
        if (inc) break;
    }
    return prefix;
}

// Block-wide exclusive prefix of v (two 31-bit sums), the tiles before it included; *total: the sum
// up to and including the tile. warp_sum, tile_prefix: shared scratch. All threads of the block.
template <int THREADS>
__device__ __forceinline__ unsigned long long tile_scan(unsigned long long v, int tile, volatile unsigned long long* state,
                                                        unsigned long long* warp_sum, unsigned long long* tile_prefix,
                                                        unsigned long long* total, unsigned* err) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    unsigned long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sum[w] = incl;
    __syncthreads();
    if (w == 0) {
        unsigned long long sum = 0;
#pragma unroll
        for (int u = 0; u < THREADS / 32; ++u) sum += warp_sum[u];
        if (lane == 0) state[tile] = (tile == 0 ? SFLAG_INC : SFLAG_AGG) | sum;
        const unsigned long long prefix = look_back(state, tile, lane, err);
        if (lane == 0) {
            if (tile) state[tile] = SFLAG_INC | ((prefix + sum) & SVAL);
            *tile_prefix = prefix;
        }
    }
    __syncthreads();
    unsigned long long before = *tile_prefix, sum = 0;
#pragma unroll
    for (int u = 0; u < THREADS / 32; ++u) {
        if (u < w) before += warp_sum[u];
        sum += warp_sum[u];
    }
    *total = *tile_prefix + sum;
    return before + incl - v;
}

constexpr int GMAX_LIMIT = 1024;
constexpr int LEAF_BS = 256, LEAF_IPT = 4, LEAF_TILE = LEAF_BS * LEAF_IPT;
inline int leaf_tiles(int n) { return grid_for(n, LEAF_TILE); }

// counts[1], counts[2]: leaves, nodes; counts[4]: deepest leaf; counts[8]: 1 if they fit Kcap and Tcap
// and the bodies are sorted (no long run flagged): what follows runs only then.
struct LeafOut {
    uint32_t* lid;         // per body: its leaf
    uint32_t* first;       // per leaf: first body (one past the last leaf: n)
    uint32_t* pre;         // per leaf: pre-order index of the first node it owns (one past: node count)
    uint8_t *depth, *gdepth;  // per leaf: its depth, the depth of its walk group
    int8_t* c;             // per leaf: common octal prefix with the body before it (-1: none)
};

// Maximum of `count` consecutive values from every place, by doubling: on return v[t] holds the
// maximum of v[t .. t + 2^p), 2^p the largest power of two up to count.
__device__ __forceinline__ int window_max(int8_t* v, int size, int count) {
    int p = 1;
    for (; 2 * p <= count; p *= 2) {
        constexpr int PER = (LEAF_TILE + 1 + GMAX_LIMIT + LEAF_BS - 1) / LEAF_BS;
        int8_t r[PER];
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int t = threadIdx.x + q * LEAF_BS;
            if (t < size) r[q] = t + p < size ? max(v[t], v[t + p]) : v[t];
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int t = threadIdx.x + q * LEAF_BS;
            if (t < size) v[t] = r[q];
        }
        __syncthreads();
    }
    return p;
}

__global__ void __launch_bounds__(LEAF_BS) k_leaves(const uint32_t* __restrict__ sys, const uint64_t* __restrict__ k0,
                                                    const FrameTable* ft, int n, int gmax, LeafOut out,
                                                    unsigned long long* state, unsigned* tile_ctr, unsigned* counts,
                                                    unsigned Kcap, unsigned Tcap, ZeroList z, unsigned* err) {
    pdl_wait();
    // Common prefixes of every window of LEAF_MAX + 1 and of gmax + 1 sorted keys that holds one of
    // the tile's bodies or the one before them; then their maxima over a body's windows.
    __shared__ int8_t c16[LEAF_TILE + 1 + LEAF_MAX];
    __shared__ int8_t cg[LEAF_TILE + 1 + GMAX_LIMIT];
    __shared__ unsigned long long warp_sum[LEAF_BS / 32], prefix_s;
    __shared__ unsigned tile_s;
    zero_spans(z);
    const int tid = threadIdx.x;
    if (tid == 0) tile_s = atomicAdd(tile_ctr, 1u);
    __syncthreads();
    const int tile = static_cast<int>(tile_s), i0 = tile * LEAF_TILE - 1;  // slot q stands for body i0 + q
    for (int t = tid; t < LEAF_TILE + 1 + LEAF_MAX; t += LEAF_BS) {
        const int j = i0 - LEAF_MAX + t;
        c16[t] = static_cast<int8_t>((j >= 0 && j + LEAF_MAX < n) ? cpl_key(sys, k0, ft, j, j + LEAF_MAX) : -1);
    }
    for (int t = tid; t < LEAF_TILE + 1 + gmax; t += LEAF_BS) {
        const int j = i0 - gmax + t;
        cg[t] = static_cast<int8_t>((j >= 0 && j + gmax < n) ? cpl_key(sys, k0, ft, j, j + gmax) : -1);
    }
    __syncthreads();
    const int p16 = window_max(c16, LEAF_TILE + 1 + LEAF_MAX, LEAF_MAX + 1);
    const int pg = window_max(cg, LEAF_TILE + 1 + gmax, gmax + 1);
    // The windows that hold slot q's body start in slots q .. q + w (w the window's length less one).
    // A body's keys end with the last frame it was re-keyed in: coincident bodies, and bodies of a
    // run past the last frame, stay one leaf there.
    auto leaf_depth = [&](int q, int i) {
        const int best = max(c16[q], c16[q + LEAF_MAX + 1 - p16]);
        return min(best + 1, ft ? MAX_LEVEL * ft->nfr[i] : MAX_LEVEL);
    };
    int depth[LEAF_IPT], c[LEAF_IPT];
    bool flag[LEAF_IPT];
    unsigned long long mine = 0;
    int deepest = 0;
    const int q0 = 1 + tid * LEAF_IPT;
    int before = i0 + q0 > 0 && i0 + q0 <= n ? leaf_depth(q0 - 1, i0 + q0 - 1) : -1;
#pragma unroll
    for (int u = 0; u < LEAF_IPT; ++u) {
        const int q = q0 + u, i = i0 + q;
        flag[u] = false;
        depth[u] = c[u] = -1;
        if (i < n) {
            depth[u] = leaf_depth(q, i);
            c[u] = i > 0 ? cpl_key(sys, k0, ft, i - 1, i) : -1;
            flag[u] = i == 0 || before != depth[u] || c[u] < depth[u];
            before = depth[u];
            if (flag[u]) {
                // The leaf owns its ancestors at depths c + 1 .. depth - 1, and itself.
                mine += 1ull + (static_cast<unsigned long long>(depth[u] - c[u]) << 31);
                deepest = max(deepest, depth[u]);
            }
        }
    }
    deepest = __reduce_max_sync(0xffffffffu, deepest);
    if ((tid & 31) == 0) atomicMax(reinterpret_cast<int*>(counts + 4), deepest);
    unsigned long long total;
    const unsigned long long at = tile_scan<LEAF_BS>(mine, tile, state, warp_sum, &prefix_s, &total, err);
    uint32_t l = static_cast<uint32_t>(at & TWO31), pre = static_cast<uint32_t>(at >> 31);
#pragma unroll
    for (int u = 0; u < LEAF_IPT; ++u) {
        const int q = q0 + u, i = i0 + q;
        if (i >= n) break;
        if (flag[u]) {
            const int gbest = max(cg[q], cg[q + gmax + 1 - pg]);
            out.first[l] = static_cast<uint32_t>(i);
            out.pre[l] = pre;
            out.depth[l] = static_cast<uint8_t>(depth[u]);
            out.gdepth[l] = static_cast<uint8_t>(min(depth[u], gbest + 1));
            out.c[l] = static_cast<int8_t>(c[u]);
            ++l;
            pre += static_cast<uint32_t>(depth[u] - c[u]);
        }
        out.lid[i] = l - 1;
    }
    if (tile == (n + LEAF_TILE - 1) / LEAF_TILE - 1 && tid == 0) {
        const unsigned K = static_cast<unsigned>(total & TWO31), T = static_cast<unsigned>(total >> 31);
        if (K <= static_cast<unsigned>(n)) {
            out.first[K] = static_cast<uint32_t>(n);
            out.pre[K] = T;
        }
        counts[1] = K;
        counts[2] = T;
        counts[8] = K <= Kcap && T <= Tcap && counts[7] == 0 ? 1u : 0u;
    }
}

// ---- nodes -----------------------------------------------------------------------------------
struct NodeCtx {
    const uint32_t* sys;  // per-body system (forest) or null
    const uint64_t* k0;          // sorted frame-0 keys
    const FrameTable* ft;        // key restart frames, or null
    LeafOut leaf;
    int n;
    const unsigned* counts;
    unsigned nroots;       // systems in the forest (1 for one system); roots take node indices 0..nroots-1
};

// Whether the leaves are there and fit what the build was launched for, and no wait before this kernel
// ran out: what a kernel left after one is not to be used as an index. (In a forest only the tree's own
// kernels, one after another, set that bit; the direct systems' have a word of their own.)
__device__ __forceinline__ bool build_ok(const unsigned* counts, const unsigned* err) {
    const unsigned fit = counts[8], ran_out = *err & kErrWaitTimeout;  // one round trip for both
    return (fit != 0) & (ran_out == 0);
}

// Pre-order nodes as k_nodes leaves them. meta: depth | leaf << 8 | group << 9 | octal digit under
// the parent << 10; mask (zero before): which of a node's eight octants have a child; first: its
// first child in the reference's numbering (k_node_scan).
struct PreNodes {
    uint2* lohi;
    uint16_t* meta;
    uint32_t* parent;  // pre-order index, 0xffffffff for a root
    uint32_t* mask;
    uint32_t* first;
};

// The last index in [a, end) for which share(index) holds, known to hold at a and to hold on a
// leading part of the range: probes at growing powers of eight, then seven probes a round, all
// loads of a round in flight together. A search costs two or three rounds for a small node and
// about fourteen for the root of 1e6 bodies (forty dependent loads by bisection).
template <class F>
__device__ __forceinline__ int last_sharing(int a, int end, F&& share) {
    long long step = 1;
    int hi = end;  // first index known not to share (or the end)
    for (;; step *= 8) {
        const long long probe = a + step;
        if (probe >= end) break;
        if (!share(static_cast<int>(probe))) {
            hi = static_cast<int>(probe);
            break;
        }
        a = static_cast<int>(probe);
    }
    while (hi - a > 1) {
        const int gap = max(1, (hi - a + 7) / 8);
        int na = a, nhi = hi;
        bool ok[7];
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const int m = a + (q + 1) * gap;
            ok[q] = m < hi && share(m);
        }
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const int m = a + (q + 1) * gap;
            if (m < hi) {
                if (ok[q]) na = m;
                else nhi = min(nhi, m);
            }
        }
        a = na;
        hi = nhi;
    }
    return a;
}

// Ranges, flags and parents of the pre-order nodes (one thread per node), and the parents' child
// masks. Leaf l owns nodes pre[l] .. pre[l + 1) - 1, at depths c[l] + 1 .. depth[l]; the parent of a
// node that is not its leaf's first is the node before it, that of a first node the node at depth
// c[l] that also holds the body before the leaf.
constexpr int NODE_BS = 256;
__global__ void __launch_bounds__(NODE_BS) k_nodes(NodeCtx x, PreNodes pn, const unsigned* err) {
    pdl_wait();
    __shared__ int l_first;
    if (!build_ok(x.counts, err)) return;
    const uint32_t T = x.counts[2];
    const int K = static_cast<int>(x.counts[1]);
    const uint32_t v0 = blockIdx.x * NODE_BS;
    if (v0 >= T) return;
    if (threadIdx.x < 32) {  // the leaf that owns the block's first node: 32 probes a round
        int a = 0, b = K;    // pre[a] <= v0 < pre[b]
        while (b - a > 1) {
            const int gap = max(1, (b - a + 32) / 33);
            const int m = a + (static_cast<int>(threadIdx.x) + 1) * gap;
            const unsigned le = __ballot_sync(0xffffffffu, m < b && x.leaf.pre[m] <= v0);
            const int k = __popc(le);  // the probes that hold are the first ones
            b = min(b, a + (k + 1) * gap);
            a += k * gap;
        }
        if (threadIdx.x == 0) l_first = a;
    }
    __syncthreads();
    const uint32_t v = v0 + threadIdx.x;
    if (v >= T) return;
    // A block's nodes belong to at most NODE_BS leaves from the first.
    int a = l_first, b = min(K, l_first + NODE_BS);
    while (b - a > 1) {
        const int m = (a + b) >> 1;
        if (x.leaf.pre[m] <= v) a = m;
        else b = m;
    }
    const int l = a, c = x.leaf.c[l], d = c + 1 + static_cast<int>(v - x.leaf.pre[l]);
    const bool leaf = d == x.leaf.depth[l];
    const int lo = static_cast<int>(x.leaf.first[l]), lend = static_cast<int>(x.leaf.first[l + 1]);
    int hi = lend;
    if (!leaf) hi = 1 + last_sharing(lend - 1, x.n, [&](int j) { return cpl_key(x.sys, x.k0, x.ft, lo, j) >= d; });
    uint32_t parent = 0xffffffffu;
    int digit = 0;
    if (d > 0) {
        digit = digit_at(x.k0, x.ft, lo, d);
        if (d > c + 1) {
            parent = v - 1;
        } else {
            // Mirrored: the place lo - 1 - j shares c digits with lo for j from 0 to the answer.
            const int back = last_sharing(0, lo, [&](int j) { return cpl_key(x.sys, x.k0, x.ft, lo - 1 - j, lo) >= c; });
            const uint32_t pl = x.leaf.lid[lo - 1 - back];
            parent = x.leaf.pre[pl] + static_cast<uint32_t>(c - x.leaf.c[pl] - 1);
        }
        if (parent < T) atomicOr(&pn.mask[parent], 1u << digit);
    }
    pn.lohi[v] = make_uint2(static_cast<uint32_t>(lo), static_cast<uint32_t>(hi));
    pn.meta[v] = static_cast<uint16_t>(d | (leaf ? 256 : 0) | (d == x.leaf.gdepth[l] ? 512 : 0) | digit << 10);
    pn.parent[v] = parent;
}

// Upsweep bookkeeping: internal nodes bucketed by depth, leaves bucketed by body count.
constexpr int NDEP = MAX_DEPTH + 2;  // depth buckets (depth <= MAX_DEPTH + 1 with headroom)
constexpr int NLSZ = 18;   // leaf-size buckets: 1..16, then larger
constexpr int NBUCKET = NDEP + NLSZ;
struct UpsweepIndex {
    unsigned count[NBUCKET];  // depths, then leaf sizes
    unsigned cur[NBUCKET];
    unsigned off[NBUCKET + 1];  // where a bucket starts in its list (written by k_nodes_out)
};

__device__ __forceinline__ int bucket_of(uint16_t meta, uint2 r) {
    return meta & 256 ? NDEP + static_cast<int>(min(r.y - r.x, 17u)) : meta & 255;
}

// One scan over the pre-order nodes: the first child of every node in the reference's numbering (child
// blocks in parent pre-order, after the roots), the walk groups' nodes in order (counts[3] their
// number), and the bucket counts of the upsweep.
constexpr int NSCAN_BS = 256, NSCAN_IPT = 4, NSCAN_TILE = NSCAN_BS * NSCAN_IPT;
__global__ void __launch_bounds__(NSCAN_BS) k_node_scan(NodeCtx x, PreNodes pn, unsigned long long* state,
                                                        unsigned* tile_ctr, unsigned* counts, UpsweepIndex* ix,
                                                        uint32_t* grp_node, unsigned* err) {
    pdl_wait();
    __shared__ unsigned long long warp_sum[NSCAN_BS / 32], prefix_s;
    __shared__ unsigned tile_s, bucket[NBUCKET];
    if (!build_ok(x.counts, err)) return;
    const uint32_t T = x.counts[2];
    const int tid = threadIdx.x;
    if (tid == 0) tile_s = atomicAdd(tile_ctr, 1u);
    if (tid < NBUCKET) bucket[tid] = 0;
    __syncthreads();
    const int tile = static_cast<int>(tile_s);
    const uint32_t v0 = static_cast<uint32_t>(tile) * NSCAN_TILE + tid * NSCAN_IPT;
    if (static_cast<uint32_t>(tile) * NSCAN_TILE >= T) return;  // past the last tile: nobody waits for it
    unsigned long long mine = 0;
    unsigned nch[NSCAN_IPT];
    bool group[NSCAN_IPT];
#pragma unroll
    for (int u = 0; u < NSCAN_IPT; ++u) {
        const uint32_t v = v0 + u;
        nch[u] = 0;
        group[u] = false;
        if (v < T) {
            const uint16_t meta = pn.meta[v];
            nch[u] = __popc(pn.mask[v]);
            group[u] = (meta & 512) != 0;
            atomicAdd(&bucket[bucket_of(meta, pn.lohi[v])], 1u);
            mine += nch[u] + (group[u] ? 1ull << 31 : 0ull);
        }
    }
    unsigned long long total;
    const unsigned long long at = tile_scan<NSCAN_BS>(mine, tile, state, warp_sum, &prefix_s, &total, err);
    uint32_t first = x.nroots + static_cast<uint32_t>(at & TWO31), g = static_cast<uint32_t>(at >> 31);
#pragma unroll
    for (int u = 0; u < NSCAN_IPT; ++u) {
        const uint32_t v = v0 + u;
        if (v >= T) break;
        pn.first[v] = first;
        first += nch[u];
        if (group[u]) {
            if (g < T) grp_node[g] = v;
            ++g;
        }
    }
    if (tid < NBUCKET && bucket[tid]) atomicAdd(&ix->count[tid], bucket[tid]);
    if (v0 < T && T <= v0 + NSCAN_IPT) counts[3] = min(static_cast<uint32_t>(total >> 31), T);
}

// A pre-order node's index in the reference's numbering.
__device__ __forceinline__ uint32_t ref_index(const NodeCtx& x, const PreNodes& pn, uint32_t v, uint16_t meta, uint32_t lo,
                                              uint32_t parent) {
    if ((meta & 255) == 0) return sys_of(x.sys, static_cast<int>(lo));  // a system's root
    return pn.first[parent] + __popc(pn.mask[parent] & ((1u << (meta >> 10)) - 1u));
}

// Geometric centre (FP64, the reference's iterative halving, src/cpu_backend.cpp:575-582 and
// 585-592) of the node at depth d containing body b; at depth 21 f the node of a run re-keyed in
// frame f takes that run's cube (src/cpu_backend.cpp:536-544).
__device__ void node_geo(const NodeCtx& c, const double* frame, uint32_t b, int d, double& gx, double& gy, double& gz,
                         double& half) {
    frame += 5 * sys_of(c.sys, static_cast<int>(b));
    half = 0.5 * frame[3];
    gx = __dadd_rn(frame[0], half);
    gy = __dadd_rn(frame[1], half);
    gz = __dadd_rn(frame[2], half);
    for (int l = 1; l <= d; ++l) {
        const int o = digit_at(c.k0, c.ft, b, l);
        const double q = 0.5 * half;
        gx = __dadd_rn(gx, (o & 4) ? q : -q);
        gy = __dadd_rn(gy, (o & 2) ? q : -q);
        gz = __dadd_rn(gz, (o & 1) ? q : -q);
        half = q;
        if (c.ft && l % MAX_LEVEL == 0 && l / MAX_LEVEL < c.ft->nfr[b]) {
            const int f = l / MAX_LEVEL;
            const double* cb = c.ft->cube[f] + 5 * c.ft->runid[f][b];
            half = 0.5 * cb[3];
            gx = __dadd_rn(cb[0], half);
            gy = __dadd_rn(cb[1], half);
            gz = __dadd_rn(cb[2], half);
        }
    }
}

// The nodes in the reference's order, and the buckets of the upsweep filled.
__global__ void __launch_bounds__(NODE_BS) k_nodes_out(NodeCtx x, PreNodes pn, const double* frame, NodeTest* nd_test,
                                                       float4* nd_geo, uint32_t* nd_parent, uint32_t* leaf_node,
                                                       UpsweepIndex* ix, uint32_t* dep_nodes, uint32_t* leaf_order,
                                                       unsigned* err) {
    pdl_wait();
    __shared__ unsigned start[NBUCKET], count[NBUCKET];
    if (!build_ok(x.counts, err)) return;
    const uint32_t T = x.counts[2], K = x.counts[1];
    const int tid = threadIdx.x;
    if (blockIdx.x * NODE_BS >= T) return;
    // Where the buckets start: exclusive sums of the counts, depths and leaf sizes apart.
    if (tid < NBUCKET) {
        start[tid] = ix->count[tid];
        count[tid] = 0;
    }
    __syncthreads();
    unsigned before = 0;
    if (tid < NBUCKET)
        for (int k = tid < NDEP ? 0 : NDEP; k < tid; ++k) before += start[k];
    const unsigned own = tid < NBUCKET ? start[tid] : 0u;
    __syncthreads();
    if (tid < NBUCKET) {
        start[tid] = before;
        if (blockIdx.x == 0) {
            ix->off[tid] = before;
            if (tid == NBUCKET - 1) ix->off[NBUCKET] = before + own;
        }
    }
    __syncthreads();
    const uint32_t v = blockIdx.x * NODE_BS + tid;
    uint32_t me = 0xffffffffu;
    int bucket = -1;
    unsigned rank = 0;
    if (v < T) {
        const uint16_t meta = pn.meta[v];
        const int d = meta & 255;
        const bool leaf = meta & 256;
        const uint2 r = pn.lohi[v];
        const uint32_t parent = pn.parent[v];
        const uint32_t nch = __popc(pn.mask[v]);
        const uint32_t first = leaf ? r.x : pn.first[v];
        if (d == 0 || parent < T) me = ref_index(x, pn, v, meta, r.x, parent);
        if (me >= T || (!leaf && (nch == 0 || first + nch > T)) || r.x >= r.y || r.y > static_cast<uint32_t>(x.n)) {
            atomicOr(err, kErrNodeOverflow);
        } else {
            nd_test[me].range = make_uint4(r.x, r.y, first, leaf ? 0u : nch);
            double gx, gy, gz, half;
            node_geo(x, frame, r.x, d, gx, gy, gz, half);
            nd_geo[me] = make_float4(static_cast<float>(gx), static_cast<float>(gy), static_cast<float>(gz),
                                     static_cast<float>(half));
            uint32_t up = 0xffffffffu;
            if (d > 0) {
                const uint32_t pp = pn.parent[parent];
                const uint16_t pmeta = pn.meta[parent];
                if ((pmeta & 255) == 0 || pp < T) up = ref_index(x, pn, parent, pmeta, pn.lohi[parent].x, pp);
            }
            nd_parent[me] = up;
            if (leaf) {
                const uint32_t l = x.leaf.lid[r.x];
                if (l < K) leaf_node[l] = me;
                else atomicOr(err, kErrNodeOverflow);
            }
            bucket = bucket_of(meta, r);
            rank = atomicAdd(&count[bucket], 1u);
        }
    }
    __syncthreads();
    if (tid < NBUCKET && count[tid]) start[tid] += atomicAdd(&ix->cur[tid], count[tid]);
    __syncthreads();
    if (bucket < 0) return;
    const unsigned pos = start[bucket] + rank;
    if (bucket < NDEP) {
        if (pos < T) dep_nodes[pos] = me;
    } else if (pos < K) {
        leaf_order[pos] = me;
    }
}

// Walk order of the groups: classes of body count, largest first. A group's walk costs about its
// size times its list, a few times the average for the largest groups; taken last, they run alone
// at the end of the walk. Up to GFINE groups (about 16 per resident walk block): four bodies to a
// class, 124 and more in the first. Above, the tail is a few per cent and neighbouring groups on
// the GPU at the same time share more of the tree's lines in the caches: only the groups of fewer
// than GSMALL bodies (a few per cent of the work) move to the end. Measured (walk): Plummer 1e5
// (2700 groups) 0.49 ms in the groups' own order, 0.38 by class; 1e6 disk (29 000 groups) 2.23 ms
// in their own order, 2.29 by class, 2.18 with the groups below 8 last (below 16: 2.22, 32: 2.28);
// 1.6e7 collision 47.2, 49.5 and 47.2 ms.
constexpr int GCLASS = 32;
constexpr uint32_t GFINE = 10000, GSMALL = 8;
__device__ __forceinline__ int group_class(uint32_t count, uint32_t ngroups) {
    if (ngroups > GFINE) return count < GSMALL ? 1 : 0;
    return GCLASS - 1 - static_cast<int>(min(count, 127u) >> 2);
}

// Group boxes from the bodies' float positions (src/cpu_backend.cpp:604-616); cls[c] counts the
// groups of class c.
__global__ void k_groups(const uint32_t* grp_node, const uint2* pn_lohi, uint32_t Tcap, const unsigned* counts,
                         const BodyArrays b, uint2* grp_range, float4* grp_box, unsigned* cls) {
    __shared__ unsigned count[GCLASS];
    if (threadIdx.x < GCLASS) count[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t G = min(counts[3], Tcap);  // zero when the build did not run
    if (g < G) {
        const uint32_t v = grp_node[g];
        uint2 r = v < counts[2] ? pn_lohi[v] : make_uint2(0u, 0u);
        if (r.x >= r.y) r = make_uint2(0u, 0u);
        grp_range[g] = r;
        atomicAdd(&count[group_class(r.y - r.x, G)], 1u);
        if (r.x < r.y) {
            float4 p = b.hm[r.x];
            float mnx = p.x, mny = p.y, mnz = p.z, mxx = mnx, mxy = mny, mxz = mnz;
            for (uint32_t i = r.x + 1; i < r.y; ++i) {
                p = b.hm[i];
                mnx = fminf(mnx, p.x); mny = fminf(mny, p.y); mnz = fminf(mnz, p.z);
                mxx = fmaxf(mxx, p.x); mxy = fmaxf(mxy, p.y); mxz = fmaxf(mxz, p.z);
            }
            grp_box[2 * g] = make_float4(__fmul_rn(0.5f, __fadd_rn(mnx, mxx)), __fmul_rn(0.5f, __fadd_rn(mny, mxy)),
                                         __fmul_rn(0.5f, __fadd_rn(mnz, mxz)), 0.f);
            grp_box[2 * g + 1] = make_float4(__fmul_rn(0.5f, __fsub_rn(mxx, mnx)), __fmul_rn(0.5f, __fsub_rn(mxy, mny)),
                                             __fmul_rn(0.5f, __fsub_rn(mxz, mnz)), 0.f);
        }
    }
    __syncthreads();
    if (threadIdx.x < GCLASS && count[threadIdx.x]) atomicAdd(&cls[threadIdx.x], count[threadIdx.x]);
}

// order = the groups by class; cls[0..GCLASS) their counts, cls[GCLASS..) cursors (zero at entry).
// Within a class the order depends on scheduling; a group's forces do not.
__global__ void k_group_order(const uint2* grp_range, uint32_t Tcap, const unsigned* ngroups, unsigned* cls,
                              uint32_t* order) {
    __shared__ unsigned base[GCLASS], count[GCLASS];
    if (threadIdx.x < GCLASS) {
        unsigned before = 0;
        for (int c = 0; c < static_cast<int>(threadIdx.x); ++c) before += cls[c];
        base[threadIdx.x] = before;
        count[threadIdx.x] = 0;
    }
    __syncthreads();
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x, G = min(*ngroups, Tcap);
    int c = 0;
    unsigned rank = 0;
    if (g < G) {
        const uint2 r = grp_range[g];
        c = group_class(r.y - r.x, G);
        rank = atomicAdd(&count[c], 1u);
    }
    __syncthreads();
    if (threadIdx.x < GCLASS && count[threadIdx.x])
        base[threadIdx.x] += atomicAdd(&cls[GCLASS + threadIdx.x], count[threadIdx.x]);
    __syncthreads();
    if (g < G) order[base[c] + rank] = g;
}

// ---- merged walk groups (GB300 grouping; off by default) ------------------------------------
// The reference's groups are the largest subtrees of <= group_max bodies, which the octree's
// eight-way split leaves small (a few dozen bodies). Runs of consecutive sibling groups (same
// parent, contiguous bodies) are packed greedily, in order, into groups of <= group_max bodies:
// fewer, fuller walk groups. Every packed group is still contained in its parent, whose walk
// rule opens it, so the lists stay exact-rule lists for the larger box.
__device__ __forceinline__ uint32_t group_parent(const uint32_t* grp_node, const uint32_t* pn_parent, uint32_t T, uint32_t g) {
    const uint32_t v = grp_node[g];
    return v < T ? pn_parent[v] : 0xffffffffu;
}

template <bool WRITE>
__global__ void k_merge_groups(const uint32_t* grp_node, const uint32_t* pn_parent,
                               const uint2* grp_range, const unsigned* ngroups, uint32_t Tcap, const unsigned* Tdev,
                               int gmax, uint32_t* mcount, const uint32_t* moff, uint2* mrange) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= Tcap) return;
    const uint32_t T = min(*Tdev, Tcap), G = min(*ngroups, Tcap);
    if (g >= G) {
        if (!WRITE) mcount[g] = 0;
        return;
    }
    const uint32_t P = group_parent(grp_node, pn_parent, T, g);
    const bool start = g == 0 || group_parent(grp_node, pn_parent, T, g - 1) != P ||
                       grp_range[g - 1].y != grp_range[g].x;
    if (!start) {
        if (!WRITE) mcount[g] = 0;
        return;
    }
    uint32_t bins = 0, cur = 0, lo = grp_range[g].x, hi = lo;
    for (uint32_t h = g; h < G; ++h) {
        const uint2 r = grp_range[h];
        if (h > g && (group_parent(grp_node, pn_parent, T, h) != P || r.x != hi)) break;
        const uint32_t sz = r.y - r.x;
        if (cur > 0 && cur + sz > static_cast<uint32_t>(gmax)) {
            if (WRITE) mrange[moff[g] + bins] = make_uint2(lo, hi);
            ++bins;
            cur = 0;
            lo = r.x;
        }
        cur += sz;
        hi = r.y;
    }
    if (WRITE) mrange[moff[g] + bins] = make_uint2(lo, hi);
    ++bins;
    if (!WRITE) mcount[g] = bins;
}

__global__ void k_merged_boxes(const uint2* mrange, const unsigned* mcount_total, uint32_t cap, const BodyArrays b,
                               float4* box) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= *mcount_total || g >= cap) return;
    const uint2 r = mrange[g];
    if (r.x >= r.y) return;
    float4 p = b.hm[r.x];
    float mnx = p.x, mny = p.y, mnz = p.z, mxx = mnx, mxy = mny, mxz = mnz;
    for (uint32_t i = r.x + 1; i < r.y; ++i) {
        p = b.hm[i];
        mnx = fminf(mnx, p.x); mny = fminf(mny, p.y); mnz = fminf(mnz, p.z);
        mxx = fmaxf(mxx, p.x); mxy = fmaxf(mxy, p.y); mxz = fmaxf(mxz, p.z);
    }
    box[2 * g] = make_float4(__fmul_rn(0.5f, __fadd_rn(mnx, mxx)), __fmul_rn(0.5f, __fadd_rn(mny, mxy)),
                             __fmul_rn(0.5f, __fadd_rn(mnz, mxz)), 0.f);
    box[2 * g + 1] = make_float4(__fmul_rn(0.5f, __fsub_rn(mxx, mnx)), __fmul_rn(0.5f, __fsub_rn(mxy, mny)),
                                 __fmul_rn(0.5f, __fsub_rn(mxz, mnz)), 0.f);
}

// ---- upsweep ---------------------------------------------------------------------------------
struct Moments {
    NodeTest* test;  // com, rcrit2 (the ranges are there already)
    NodeCell* cell;  // the reference's stored floats; lo: FP64 com minus its float
};

// rcrit2 = (2 half / theta + |com - centre|)^2 capped at FLT_MAX (src/cpu_backend.cpp:595-600), with
// |com - centre|^2 as the reference's compiler forms it: fma(dz, dz, fma(dx, dx, dy*dy)).
__device__ __forceinline__ float rcrit2_of(float cx, float cy, float cz, float4 g, float inv_theta) {
    const float dx = __fsub_rn(cx, g.x), dy = __fsub_rn(cy, g.y), dz = __fsub_rn(cz, g.z);
    const float s = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
    const double r = __dadd_rn(__dmul_rn(static_cast<double>(__fmul_rn(2.f, g.w)), static_cast<double>(inv_theta)),
                               __dsqrt_rn(static_cast<double>(s)));
    const double r2 = __dmul_rn(r, r);
    return static_cast<float>(r2 < static_cast<double>(FLT_MAX) ? r2 : static_cast<double>(FLT_MAX));
}

__device__ void store_moments(Moments mo, uint32_t node, double M, double cx, double cy, double cz, double qxx,
                              double qxy, double qxz, double qyy, double qyz, double qzz, float4 g, float inv_theta) {
    const float fx = static_cast<float>(cx), fy = static_cast<float>(cy), fz = static_cast<float>(cz);
    const float rc2 = rcrit2_of(fx, fy, fz, g, inv_theta);
    NodeCell& c = mo.cell[node];
    mo.test[node].com = make_float4(fx, fy, fz, rc2);
    c.com = make_float4(fx, fy, fz, static_cast<float>(M));
    c.lo = make_float4(static_cast<float>(__dsub_rn(cx, fx)), static_cast<float>(__dsub_rn(cy, fy)),
                                 static_cast<float>(__dsub_rn(cz, fz)), 0.f);
    c.q0 = make_float4(static_cast<float>(qxx), static_cast<float>(qxy), static_cast<float>(qxz),
                              static_cast<float>(qyy));
    c.q1 = make_float4(static_cast<float>(qyz), static_cast<float>(qzz), rc2, 0.f);
}

#define DADD __dadd_rn
#define DMUL __dmul_rn
#define DSUB __dsub_rn
#define DFMA __fma_rn

// Leaf moments about each leaf's centre of mass in FP64 (src/cpu_backend.cpp:619-640), one
// thread per leaf, leaves taken in body-count order so a warp's loops have equal trip counts.
__global__ void k_leaf_moments(const uint32_t* __restrict__ leaf_order, const unsigned* counts,
                               const float4* __restrict__ nd_geo, const BodyArrays b, Moments mo, float inv_theta,
                               const float* __restrict__ inv_theta_sys, const uint32_t* __restrict__ sys, unsigned* err) {
    pdl_wait();
    const uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
    if (!build_ok(counts, err)) return;
    const uint32_t T = counts[2];
    if (l >= counts[1]) return;
    const uint32_t node = leaf_order[l];
    if (node >= T) {
        atomicOr(err, kErrNodeOverflow);
        return;
    }
    const uint4 r = mo.test[node].range;
    const float4 g = nd_geo[node];
    if (inv_theta_sys) inv_theta = inv_theta_sys[sys_of(sys, static_cast<int>(r.x))];
    double M = 0, sx = 0, sy = 0, sz = 0;
    for (uint32_t i = r.x; i < r.y; ++i) {
        const double m = b.m[i];
        M = DADD(M, m);
        sx = DADD(sx, DMUL(m, b.x[i]));
        sy = DADD(sy, DMUL(m, b.y[i]));
        sz = DADD(sz, DMUL(m, b.z[i]));
    }
    const double cx = M > 0 ? __ddiv_rn(sx, M) : g.x, cy = M > 0 ? __ddiv_rn(sy, M) : g.y,
                 cz = M > 0 ? __ddiv_rn(sz, M) : g.z;
    double qxx = 0, qxy = 0, qxz = 0, qyy = 0, qyz = 0, qzz = 0;
    for (uint32_t i = r.x; i < r.y; ++i) {
        const double m = b.m[i], dx = DSUB(b.x[i], cx), dy = DSUB(b.y[i], cy), dz = DSUB(b.z[i], cz);
        const double r2 = DFMA(dz, dz, DFMA(dx, dx, DMUL(dy, dy)));
        const double m3 = DMUL(m, 3.0);
        qxx = DFMA(m, DFMA(DMUL(3.0, dx), dx, -r2), qxx);
        qyy = DFMA(m, DFMA(DMUL(3.0, dy), dy, -r2), qyy);
        qzz = DFMA(m, DFMA(DMUL(3.0, dz), dz, -r2), qzz);
        qxy = DFMA(DMUL(m3, dx), dy, qxy);
        qxz = DFMA(DMUL(m3, dx), dz, qxz);
        qyz = DFMA(DMUL(m3, dy), dz, qyz);
    }
    store_moments(mo, node, M, cx, cy, cz, qxx, qxy, qxz, qyy, qyz, qzz, g, inv_theta);
}

// Eight lanes per node or leaf, four of them per warp: lane j holds child (or body) j's terms, lays
// them out in rows of the warp's shared memory, one row per sum, and folds row j in order. On this
// part an FP64 warp instruction holds a scheduler's FP64 unit for about 64 cycles whatever its active
// lanes, so the chain that counts is that of FP64 warp instructions: the terms are formed once, side
// by side, the sums that must be sequential run beside each other, one per lane, and each lane
// rounds and stores its own results. A row is 10 doubles long: 16-byte reads without conflicts.
constexpr int WIDE = 8, ROW = 10;

__device__ __forceinline__ void load_row(const double* row, double (&v)[WIDE]) {
    const double2* p = reinterpret_cast<const double2*>(row);
#pragma unroll
    for (int q = 0; q < WIDE / 2; ++q) {
        const double2 d = p[q];
        v[2 * q] = d.x;
        v[2 * q + 1] = d.y;
    }
}

__device__ __forceinline__ double shfl_d(double v, int src_lane) { return __shfl_sync(0xffffffffu, v, src_lane); }

// A node's floats from its eight lanes: f1 / M, that is the centre's coordinate j, on lanes 1..3 (lane
// 0: M itself); the quadrupole's sum j on lanes 0..5. The opening radius is stored by store_rcrit.
__device__ __forceinline__ void store_wide(const Moments& mo, uint32_t node, int j, double M, double cj, double q) {
    float* c = reinterpret_cast<float*>(mo.cell + node);  // com.xyz m, lo.xyz 0, q0, q1
    const double v = j == 0 ? M : cj;
    const float f = static_cast<float>(v);
    const float l = static_cast<float>(__dsub_rn(v, static_cast<double>(f)));
    const float fq = static_cast<float>(q);
    if (j < 4) {
        c[(j + 3) & 3] = f;
        c[4 + ((j + 3) & 3)] = j ? l : 0.f;
    }
    if (j != 6) c[8 + j] = j < 6 ? fq : 0.f;  // q1.z is the opening radius
}

__device__ __forceinline__ void store_rcrit(const Moments& mo, uint32_t node, float4 com, float4 g, float inv_theta) {
    const float rc2 = rcrit2_of(com.x, com.y, com.z, g, inv_theta);
    mo.test[node].com = make_float4(com.x, com.y, com.z, rc2);
    mo.cell[node].q1.z = rc2;
}

// k_leaf_moments for the trees whose leaves are too few to fill the FP64 units one to a thread, where
// a leaf's chain of about 40 FP64 instructions per body is the time (8191 bodies: 27 -> 10 us). Bodies
// in rounds of eight. The two folds of a body leave lanes idle, so more FP64 work is issued in all,
// hence the line (build phase with a thread -> eight lanes per leaf, Plummer: 8191 bodies, 1748 leaves,
// 106 -> 90 us, 16 000, 3348, 115 -> 100, 25 000, 5180, 117 -> 115, 30 000, 6173, 121 -> 129).
constexpr int LEAFW_BS = 128;
constexpr size_t LEAFW_MAX = 5120;  // leaves at the last exact build
__global__ void __launch_bounds__(LEAFW_BS) k_leaf_moments_wide(const uint32_t* __restrict__ leaf_order,
                                                                const unsigned* counts,
                                                                const float4* __restrict__ nd_geo,
                                                                const BodyArrays b, Moments mo, float inv_theta,
                                                                const float* __restrict__ inv_theta_sys,
                                                                const uint32_t* __restrict__ sys, unsigned* err) {
    __shared__ __align__(16) double rows[LEAFW_BS / WIDE][8][ROW];
    pdl_wait();
    if (!build_ok(counts, err)) return;
    const uint32_t T = counts[2], K = counts[1];
    const int lane = threadIdx.x & 31, j = lane & 7, base = lane & ~7;
    double(*row)[ROW] = rows[threadIdx.x / WIDE];
    const uint32_t l = (blockIdx.x * LEAFW_BS + threadIdx.x) / WIDE;
    uint32_t node = l < K ? leaf_order[l] : 0u;
    bool valid = l < K;
    if (valid && node >= T) {
        if (j == 0) atomicOr(err, kErrNodeOverflow);
        valid = false;
        node = 0;
    }
    uint4 r = make_uint4(0, 0, 0, 0);
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
    if (valid) {
        r = mo.test[node].range;
        g = nd_geo[node];
    }
    const int nb = static_cast<int>(r.y - r.x);
    const int rounds = __reduce_max_sync(0xffffffffu, (nb + WIDE - 1) / WIDE);
    double f1 = 0;
    double v[WIDE];
    for (int q0 = 0; q0 < rounds; ++q0) {
        const int at = WIDE * q0 + j;
        const uint32_t i = r.x + at;
        const bool on = at < nb;
        const double m = on ? b.m[i] : 0.f, x = on ? b.x[i] : 0.f, y = on ? b.y[i] : 0.f, z = on ? b.z[i] : 0.f;
        row[0][j] = m;
        row[1][j] = DMUL(m, x);
        row[2][j] = DMUL(m, y);
        row[3][j] = DMUL(m, z);
        __syncwarp();
        load_row(row[j & 3], v);
#pragma unroll
        for (int q = 0; q < WIDE; ++q)
            if (WIDE * q0 + q < nb) f1 = DADD(f1, v[q]);
        __syncwarp();
    }
    const double M = shfl_d(f1, base);
    const double cj = M > 0 ? __ddiv_rn(f1, M) : static_cast<double>(j == 1 ? g.x : j == 2 ? g.y : g.z);
    const double cx = shfl_d(cj, base + 1), cy = shfl_d(cj, base + 2), cz = shfl_d(cj, base + 3);
    // Each sum is a chain of fused multiply-adds: its factors are laid out, m or m3 dx or m3 dy, and
    // the axis terms or dy or dz.
    const int ra = j == 1 || j == 2 ? 1 : j == 4 ? 2 : 0;
    const int rb = j == 0 ? 3 : j == 1 ? 6 : j == 3 ? 4 : j == 5 ? 5 : 7;
    double fq = 0;
    for (int q0 = 0; q0 < rounds; ++q0) {
        const int at = WIDE * q0 + j;
        const uint32_t i = r.x + at;
        const bool on = at < nb;
        const double m = on ? b.m[i] : 0.f, dx = DSUB(on ? b.x[i] : 0.f, cx), dy = DSUB(on ? b.y[i] : 0.f, cy),
                     dz = DSUB(on ? b.z[i] : 0.f, cz);
        const double r2 = DFMA(dz, dz, DFMA(dx, dx, DMUL(dy, dy)));
        const double m3 = DMUL(m, 3.0);
        row[0][j] = m;
        row[1][j] = DMUL(m3, dx);
        row[2][j] = DMUL(m3, dy);
        row[3][j] = DFMA(DMUL(3.0, dx), dx, -r2);
        row[4][j] = DFMA(DMUL(3.0, dy), dy, -r2);
        row[5][j] = DFMA(DMUL(3.0, dz), dz, -r2);
        row[6][j] = dy;
        row[7][j] = dz;
        __syncwarp();
        double u[WIDE];
        load_row(row[ra], u);
        load_row(row[rb], v);
#pragma unroll
        for (int q = 0; q < WIDE; ++q)
            if (WIDE * q0 + q < nb) fq = DFMA(u[q], v[q], fq);
        __syncwarp();
    }
    if (!valid) return;
    store_wide(mo, node, j, M, cj, fq);
    if (j == 0) {
        if (inv_theta_sys) inv_theta = inv_theta_sys[sys_of(sys, static_cast<int>(r.x))];
        store_rcrit(mo, node,
                    make_float4(static_cast<float>(cx), static_cast<float>(cy), static_cast<float>(cz), 0.f), g,
                    inv_theta);
    }
}

// Internal nodes of one depth: combine the children (already final) in index order, FP64, the
// parallel-axis theorem for the traceless quadrupole (src/cpu_backend.cpp:642-663). Lane j forms the
// terms of child j; each of the reference's sequential child-order sums is then folded by one lane:
// M, sx, sy, sz by lanes 0..3, which divide by M together, the quadrupole's by lanes 0..5. Every FP64
// operation of the reference, as its compiler forms it (fused multiply-adds included), is done once,
// in its order, so the moments are the reference's bit for bit. The opening radius, which no parent
// reads, costs a square root: it is left to rcrit_range, a lane per node.
constexpr int COMBINE_BS = 128, TOP_BS = 256;
constexpr int COMBINE_NODES = COMBINE_BS / WIDE;  // nodes per block and round

// What a lane needs of its node before the children are final.
struct CombineNode {
    uint32_t p, first;
    int nch;  // 0: nothing to do
    float4 g;
};

__device__ __forceinline__ CombineNode combine_fetch(const uint32_t* __restrict__ dep_nodes, unsigned k, unsigned hi,
                                                     uint32_t T, const float4* __restrict__ nd_geo, const Moments& mo,
                                                     unsigned* err) {
    CombineNode c{0u, 0u, 0, make_float4(0.f, 0.f, 0.f, 0.f)};
    if (k >= hi) return c;
    c.p = dep_nodes[k];
    if (c.p < T) {
        const uint4 r = mo.test[c.p].range;
        c.g = nd_geo[c.p];
        if (r.w != 0 && r.w <= 8 && r.z + r.w <= T) {
            c.first = r.z;
            c.nch = static_cast<int>(r.w);
            return c;
        }
    }
    if ((threadIdx.x & 7) == 0) atomicOr(err, kErrNodeOverflow);
    return c;
}

// One node per eight lanes; row: their ten rows. FAR: the children were written by other SMs in the
// same launch and are read past the L1 cache.
template <bool FAR>
__device__ __forceinline__ void combine_node(const CombineNode& n, double (*row)[ROW], const Moments& mo) {
    const int lane = threadIdx.x & 31, j = lane & 7, base = lane & ~7;
    float4 cm = make_float4(0.f, 0.f, 0.f, 0.f), qa = cm, qb = cm;  // zeros past the last child: never added
    if (j < n.nch) {
        const NodeCell* ch = mo.cell + n.first + j;
        cm = FAR ? __ldcg(&ch->com) : ch->com;
        qa = FAR ? __ldcg(&ch->q0) : ch->q0;
        qb = FAR ? __ldcg(&ch->q1) : ch->q1;
    }
    const double m = cm.w, x = cm.x, y = cm.y, z = cm.z;
    row[0][j] = m;
    row[1][j] = DMUL(m, x);
    row[2][j] = DMUL(m, y);
    row[3][j] = DMUL(m, z);
    __syncwarp();
    double v[WIDE];
    load_row(row[j & 3], v);
    double f1 = 0;
#pragma unroll
    for (int q = 0; q < WIDE; ++q)
        if (q < n.nch) f1 = DADD(f1, v[q]);
    const double M = shfl_d(f1, base);
    const double cj = M > 0 ? __ddiv_rn(f1, M) : static_cast<double>(j == 1 ? n.g.x : j == 2 ? n.g.y : n.g.z);
    const double cx = shfl_d(cj, base + 1), cy = shfl_d(cj, base + 2), cz = shfl_d(cj, base + 3);
    // The child's quadrupole about the new centre.
    const double dx = DSUB(x, cx), dy = DSUB(y, cy), dz = DSUB(z, cz);
    const double r2 = DFMA(dz, dz, DFMA(dx, dx, DMUL(dy, dy)));
    const double m3 = DMUL(m, 3.0);
    row[4][j] = DFMA(m, DFMA(DMUL(3.0, dx), dx, -r2), static_cast<double>(qa.x));
    row[5][j] = DFMA(DMUL(m3, dx), dy, static_cast<double>(qa.y));
    row[6][j] = DFMA(DMUL(m3, dx), dz, static_cast<double>(qa.z));
    row[7][j] = DFMA(m, DFMA(DMUL(3.0, dy), dy, -r2), static_cast<double>(qa.w));
    row[8][j] = DFMA(DMUL(m3, dy), dz, static_cast<double>(qb.x));
    row[9][j] = DFMA(m, DFMA(DMUL(3.0, dz), dz, -r2), static_cast<double>(qb.y));
    __syncwarp();
    load_row(row[4 + min(j, 5)], v);
    double fq = 0;
#pragma unroll
    for (int q = 0; q < WIDE; ++q)
        if (q < n.nch) fq = DADD(fq, v[q]);
    if (n.nch) store_wide(mo, n.p, j, M, cj, fq);
    __syncwarp();  // the rows are free again
}

// Opening radii of the internal nodes dep_nodes[lo, hi), a lane each, once their centres are final.
__device__ __forceinline__ void rcrit_range(const uint32_t* __restrict__ dep_nodes, unsigned lo, unsigned hi, uint32_t T,
                                            const float4* __restrict__ nd_geo, const Moments& mo, float inv_theta,
                                            const float* __restrict__ inv_theta_sys, const uint32_t* __restrict__ sys,
                                            unsigned tid, unsigned threads) {
    for (unsigned k = lo + tid; k < hi; k += threads) {
        const uint32_t p = dep_nodes[k];
        if (p >= T) continue;  // reported by combine_fetch
        const float th = inv_theta_sys ? inv_theta_sys[sys_of(sys, static_cast<int>(mo.test[p].range.x))] : inv_theta;
        store_rcrit(mo, p, __ldcg(&mo.cell[p].com), nd_geo[p], th);
    }
}

__device__ __forceinline__ unsigned dep_begin(const UpsweepIndex* ix, int depth) {  // of a depth's list
    return ix->off[min(max(depth, 0), NDEP - 1)];
}

// One depth, and the opening radii of the depth below it (depth -1: those of the roots alone).
__global__ void __launch_bounds__(COMBINE_BS) k_combine_level(const uint32_t* __restrict__ dep_nodes,
                                                              const UpsweepIndex* ix, int depth, const unsigned* counts,
                                                              const float4* __restrict__ nd_geo, Moments mo,
                                                              float inv_theta, const float* __restrict__ inv_theta_sys,
                                                              const uint32_t* __restrict__ sys, unsigned* err) {
    __shared__ __align__(16) double rows[COMBINE_NODES][ROW][ROW];
    pdl_wait();
    if (!build_ok(counts, err)) return;
    const uint32_t T = counts[2];
    const unsigned lo = dep_begin(ix, depth), hi = dep_begin(ix, depth + 1), end = dep_begin(ix, depth + 2);
    const unsigned sub = threadIdx.x / WIDE, of = gridDim.x * COMBINE_NODES;
    for (unsigned k = lo + blockIdx.x * COMBINE_NODES; k < hi; k += of)
        combine_node<false>(combine_fetch(dep_nodes, k + sub, hi, T, nd_geo, mo, err), rows[sub], mo);
    rcrit_range(dep_nodes, hi, end, T, nd_geo, mo, inv_theta, inv_theta_sys, sys,
                blockIdx.x * COMBINE_BS + threadIdx.x, gridDim.x * COMBINE_BS);
}

// The depths from `depth` up to the root in one launch of one cluster of 16 blocks, a cluster barrier
// between depths: a depth of up to 512 nodes is one round of the FP64 chain whether it has its own
// launch or not, and the barrier costs less than the launch. What is known of a depth's nodes before
// their children are final is read ahead of the barrier, and all opening radii are formed at the end:
// 4.9 us a depth (8.7 with four lanes to a node, the radii inside and all loads after the barrier).
constexpr int TOP_BLOCKS = 16, TOP_NODES = TOP_BLOCKS * (TOP_BS / WIDE);
__global__ void __launch_bounds__(TOP_BS) k_combine_top(const uint32_t* __restrict__ dep_nodes, const UpsweepIndex* ix,
                                                        int depth, const unsigned* counts,
                                                        const float4* __restrict__ nd_geo, Moments mo, float inv_theta,
                                                        const float* __restrict__ inv_theta_sys,
                                                        const uint32_t* __restrict__ sys, unsigned* err) {
    __shared__ __align__(16) double rows[TOP_BS / WIDE][ROW][ROW];
    pdl_wait();
    if (!build_ok(counts, err)) return;  // the same words for all blocks
    const uint32_t T = counts[2];
    const unsigned sub = threadIdx.x / WIDE;
    // Nodes in order go to the blocks' first warps, then to their second: a narrow depth is spread
    // over all FP64 units.
    const unsigned at = (threadIdx.x / 32 * TOP_BLOCKS + blockIdx.x) * (32 / WIDE) + (threadIdx.x % 32) / WIDE;
    const unsigned warp0 = at - (threadIdx.x % 32) / WIDE;
    const unsigned end = dep_begin(ix, depth + 2);
    unsigned lo = dep_begin(ix, depth), hi = dep_begin(ix, depth + 1);
    CombineNode n = combine_fetch(dep_nodes, lo + at, hi, T, nd_geo, mo, err);
    for (; depth >= 0; --depth) {
        for (unsigned k = lo; k + warp0 < hi; k += TOP_NODES) {  // warp-uniform
            if (k != lo) n = combine_fetch(dep_nodes, k + at, hi, T, nd_geo, mo, err);
            combine_node<true>(n, rows[sub], mo);
        }
        if (depth > 0) {
            hi = lo;
            lo = dep_begin(ix, depth - 1);
            n = combine_fetch(dep_nodes, lo + at, hi, T, nd_geo, mo, err);
        }
        __syncwarp();
        // Releases this thread's writes to the cluster and acquires the others'.
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    rcrit_range(dep_nodes, dep_begin(ix, 0), end, T, nd_geo, mo, inv_theta, inv_theta_sys, sys,
                blockIdx.x * TOP_BS + threadIdx.x, TOP_BLOCKS * TOP_BS);
}

#undef DADD
#undef DMUL
#undef DSUB
#undef DFMA


__global__ void k_probe() {}

// ---- host helpers ----------------------------------------------------------------------------
void scan_u32(Engine& e, TreeState& t, const uint32_t* in, uint32_t* out, int n, uint32_t* total) {
    if (n <= 0) return;
    const int tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    t.scan_state.reserve(static_cast<size_t>(tiles) * 8);
    t.scan_ctr.reserve(256);
    LG_CK(cudaMemsetAsync(t.scan_state.as<char>(), 0, static_cast<size_t>(tiles) * 8, e.stream));
    LG_CK(cudaMemsetAsync(t.scan_ctr.as<char>(), 0, 4, e.stream));
    k_scan<<<tiles, SCAN_BS, 0, e.stream>>>(in, out, n, t.scan_state.as<unsigned long long>(), t.scan_ctr.as<unsigned>(),
                                           total, e.err_word());
    LG_LAUNCHED();
    ++e.launches;
}

// k_leaves' look-back words and its tile counter.
size_t leaf_state_words(int n) { return (static_cast<size_t>(leaf_tiles(n)) * 8 + 16 + 15) / 16; }

int sort_tiles(int n) { return (n + SORT_TILE - 1) / SORT_TILE; }

// Histograms and pass counters, then the passes' look-back words: zero before a sort begins.
size_t hist_words(void) { return (PASSES * RADIX + 16) * 4 / 16; }
size_t lookback_words(int n, int passes) { return static_cast<size_t>(passes) * sort_tiles(n) * RADIX * 4 / 16; }

// Sorts the n keys in keysA by their low 8 * passes bits, values starting as the positions (or as
// valsA); histograms already in t.hist. Returns which buffers hold the result (0: A, 1: B).
int sort_passes(Engine& e, TreeState& t, int n, int passes, bool iota, int pass0 = 0, int from = 0) {
    uint64_t* k[2] = {t.keysA.as<uint64_t>(), t.keysB.as<uint64_t>()};
    uint32_t* v[2] = {t.valsA.as<uint32_t>(), t.valsB.as<uint32_t>()};
    const int tiles = sort_tiles(n);
    unsigned* hist = t.hist.as<unsigned>();
    for (int p = pass0; p < passes; ++p, from ^= 1) {
        launch_pdl(overlap(n), k_sort_pass, tiles, SORT_BS, e.stream, k[from],
                   iota && p == 0 ? nullptr : v[from], k[from ^ 1], v[from ^ 1], n, 8 * p, hist + p * RADIX,
                   t.lookback.as<unsigned>() + static_cast<size_t>(p) * tiles * RADIX,
                   hist + PASSES * RADIX + p, e.err_word());
        ++e.launches;
    }
    return from;
}

// The same with the histograms formed and everything zeroed here; result in A (passes is even).
void sort_pairs(Engine& e, TreeState& t, int n, bool iota) {
    cudaStream_t s = e.stream;
    LG_CK(cudaMemsetAsync(t.hist.as<char>(), 0, hist_words() * 16, s));
    LG_CK(cudaMemsetAsync(t.lookback.as<char>(), 0, lookback_words(n, PASSES) * 16, s));
    const int hb = std::min(e.sms * 4, std::max(1, grid_for(n, 1024)));
    k_sort_hist<<<hb, 256, 0, s>>>(t.keysA.as<uint64_t>(), n, PASSES, t.hist.as<unsigned>());
    LG_LAUNCHED();
    ++e.launches;
    sort_passes(e, t, n, PASSES, iota);
}

void reserve_sort(TreeState& t, int n) {
    const size_t cnt = static_cast<size_t>(n) + 1;
    t.keysA.reserve(cnt * 8); t.keysB.reserve(cnt * 8);
    t.valsA.reserve(cnt * 4); t.valsB.reserve(cnt * 4);
    t.skey.reserve(cnt * 8);
    t.mkeys.reserve(cnt * 8);
    t.hist.reserve(hist_words() * 16);
    t.lookback.reserve(lookback_words(n, PASSES) * 16);
    t.counts.reserve(64);
    t.leaf_state.reserve(leaf_state_words(n) * 16);
}

int bits_for(int count) {
    int b = 0;
    while ((1 << b) < count) ++b;
    return b;
}

}  // namespace

std::unique_ptr<TreeState, void (*)(TreeState*)> make_tree_state() {
    return std::unique_ptr<TreeState, void (*)(TreeState*)>(new TreeState, destroy_tree);
}

const void* probe_kernel() { return reinterpret_cast<const void*>(k_probe); }

void tree_sort(Engine& e) {
    TreeState& t = *e.tree;
    const int n = t.n_tree >= 0 ? t.n_tree : e.n;
    const int n_total = e.n;
    const uint32_t* sys = t.sys;
    cudaStream_t s = e.stream;
    if (n >= (1 << 30)) fail(kRuntime, "cuda tree: n >= 2^30 exceeds the sort's look-back counters");
    reserve_sort(t, n);
    t.frame.reserve(static_cast<size_t>(std::max(t.nsys, 1)) * 5 * 8 + 64);
    t.restarted = false;
    t.nframes = 1;
    unsigned* counts = t.counts.as<unsigned>();
    const int sysbits = sys ? bits_for(t.nsys) : 0;
    const int run_cap = std::max(1, n / (LEAF_MAX + 1) + 1);  // runs hold more than LEAF_MAX bodies each
    unsigned R = 0;
    // The leading digits decide the order of all bodies but those of one cell that deep: as many
    // digits are sorted as the tree was deep at its last exact build (with its headroom), in whole
    // 8-bit passes (8e3 bodies: 4 passes, 1e5: 5, 1e6: 5, 1.6e7: 6, of 8 for all 63 bits), and bodies
    // that tie are ordered where they are gathered (k_permute). A tree that turns out deeper is found
    // there; the sort is redone with every digit and the depth measured anew. Nothing is assumed of new
    // bodies: a first sort takes every digit (a guess from n took three passes less on smooth scenes, 131 072
    // bodies 95 us against 131, and a second whole sort where more than 16 bodies tied: with a tenth of
    // the bodies in a core 220 against 132). With the clearing, the histograms and the digits' scans
    // folded into the kernels around the passes: sort phase 142 -> 54 us (8191 bodies), 160 -> 75 (1e5),
    // 302 -> 184 (1e6 disk), 2.76 -> 2.12 ms (1.6e7); below 1e6 it is the latency of 7 or 8 dependent
    // launches, above, the passes' traffic.
    for (bool full = t.known_depth <= 0 || t.restart_mode;; full = true) {
        int levels = MAX_LEVEL, passes = PASSES;
        if (!full) {
            passes = std::max(1, (3 * std::min(t.known_depth, MAX_LEVEL) + sysbits + 7) / 8);
            levels = std::min(MAX_LEVEL, (8 * passes - sysbits) / 3);
            full = passes >= PASSES;
        }
        if (full) {
            levels = MAX_LEVEL;
            passes = PASSES;
        }
        ZeroList z{};
        z.span[0] = {t.counts.as<uint4>(), 4};
        z.span[1] = {t.hist.as<uint4>(), hist_words()};
        z.span[2] = {t.lookback.as<uint4>(), lookback_words(n, passes)};
        z.span[3] = {t.leaf_state.as<uint4>(), leaf_state_words(n)};
        // A forest's runs read the error word once, after all their steps: it is theirs to clear.
        if (!sys) z.span[4] = {reinterpret_cast<uint4*>(e.err_word()), 1};  // (the frame kernel's ticket lies behind it)
        if (sys) {
            launch_pdl(overlap(n), k_frame_sys, t.nsys, BS, s, e.bodies(e.cur), t.sys_off,
                       t.frame.as<double>(), z);
        } else {
            const int fb = std::min(2 * e.sms, grid_for(n, BS));
            e.diag_partial.reserve(static_cast<size_t>(fb) * 12 * 8);
            launch_pdl(overlap(n), k_frame, fb, BS, s, e.bodies(e.cur), n, e.diag_partial.as<long long>(),
                       e.ticket(), t.frame.as<double>(), z);
        }
        LG_LAUNCHED();
        // With every digit sorted the system index does not fit beside them: it is sorted on its own.
        launch_pdl(overlap(n), k_keys, std::min(2 * e.sms, grid_for(n, 512)), 512, s, sys, e.bodies(e.cur),
                   n, t.frame.as<double>(), t.mkeys.as<uint64_t>(), t.keysA.as<uint64_t>(), levels, passes,
                   sys && !full ? 1 : 0, t.hist.as<unsigned>());
        e.launches += 2;
        int at = sort_passes(e, t, n, passes, true);
        if (full && sys) {
            k_sys_keys<<<grid_for(n, BS), BS, 0, s>>>(sys, t.valsA.as<uint32_t>(), t.keysA.as<uint64_t>(), n);
            LG_LAUNCHED();
            ++e.launches;
            sort_pairs(e, t, n, false);
            at = 0;
        }
        const int other = e.cur ^ 1;
        launch_pdl(overlap(n), k_permute, grid_for(n_total, BS), BS, s, e.bodies(e.cur), e.bodies(other),
                   at ? t.keysB.as<uint64_t>() : t.keysA.as<uint64_t>(),
                   at ? t.valsB.as<uint32_t>() : t.valsA.as<uint32_t>(), t.mkeys.as<uint64_t>(),
                   t.skey.as<uint64_t>(), nullptr, nullptr, n, n_total, full ? 0 : 1, counts + 7, e.err_word());
        ++e.launches;
        e.cur = other;
        if (full) {
            // Key restarts (src/cpu_backend.cpp:536-544): runs of identical keys longer than a leaf.
            // (A partial sort flags any run that long.)
            t.runs.reserve(static_cast<size_t>(run_cap) * 8);
            k_find_runs<<<grid_for(n, BS), BS, 0, s>>>(sys, t.skey.as<uint64_t>(), nullptr, nullptr, 1, n,
                                                       t.runs.as<uint2>(), counts, run_cap);
            LG_LAUNCHED();
            ++e.launches;
        }
        // Key restarts are rare: unless the last build needed them, assume none and let the check
        // after the walk (tree_verify) catch a miss; otherwise read the counts now.
        t.speculative = t.have_guess && !t.restart_mode;
        if (t.speculative) return;
        LG_CK(cudaMemcpyAsync(e.pinned_small, counts, 32, cudaMemcpyDeviceToHost, s));
        LG_CK(cudaStreamSynchronize(s));
        R = e.pinned_small[0];
        if (full || !e.pinned_small[7]) break;
        t.known_depth = 0;
    }
    // Runs are disjoint and longer than LEAF_MAX, so there are fewer than run_cap.
    R = std::min(R, static_cast<unsigned>(run_cap));
    t.restart_mode = R > 0;
    if (R == 0) return;
    t.restarted = true;
    ++t.generation;
    t.key1tmp.reserve(static_cast<size_t>(n) * 8 + 8);
    t.nfr.reserve(static_cast<size_t>(n) + 8);
    t.ftab.reserve(sizeof(FrameTable));
    uint64_t* key1 = t.key1tmp.as<uint64_t>();
    uint8_t* nfr = t.nfr.as<uint8_t>();
    LG_CK(cudaMemsetAsync(nfr, 1, static_cast<size_t>(n), s));
    FrameTable ft{};
    ft.key[0] = t.skey.as<uint64_t>();
    ft.nfr = nfr;
    // Frame by frame: re-key the runs in their own cubes, then a stable sort by (run, new key), which
    // keeps every body inside its run. Inside a run the earlier frames' keys, run indices and nfr
    // are all equal, so only the bodies and the new keys move.
    for (int f = 1; f < FRAMES && R > 0; ++f) {
        BodyArrays b = e.bodies(e.cur);
        t.fkey[f].reserve(static_cast<size_t>(n) * 8 + 8);
        t.frunid[f].reserve(static_cast<size_t>(n) * 4 + 4);
        t.fcube[f].reserve(static_cast<size_t>(R) * 5 * 8);
        int* runid = t.frunid[f].as<int>();
        k_fill_i32<<<grid_for(n, BS), BS, 0, s>>>(runid, -1, n);
        LG_LAUNCHED();
        k_fill_u64<<<grid_for(n, BS), BS, 0, s>>>(key1, 0ull, n);
        LG_LAUNCHED();
        k_run_cube<<<R, BS, 0, s>>>(b, t.runs.as<uint2>(), t.fcube[f].as<double>());
        LG_LAUNCHED();
        k_run_keys<<<R, BS, 0, s>>>(b, t.runs.as<uint2>(), t.fcube[f].as<double>(), key1, runid, nfr, f);
        LG_LAUNCHED();
        LG_CK(cudaMemcpyAsync(t.keysA.as<uint64_t>(), key1, static_cast<size_t>(n) * 8, cudaMemcpyDeviceToDevice, s));
        sort_pairs(e, t, n, true);
        k_seg_keys<<<grid_for(n, BS), BS, 0, s>>>(t.valsA.as<uint32_t>(), runid, t.runs.as<uint2>(),
                                                  t.keysA.as<uint64_t>(), n);
        LG_LAUNCHED();
        sort_pairs(e, t, n, false);
        const int other = e.cur ^ 1;
        launch_pdl(overlap(n), k_permute, grid_for(n_total, BS), BS, s, e.bodies(e.cur), e.bodies(other),
                   t.keysA.as<uint64_t>(), t.valsA.as<uint32_t>(), nullptr, nullptr, key1,
                   t.fkey[f].as<uint64_t>(), n, n_total, 0, nullptr, e.err_word());
        e.cur = other;
        ft.key[f] = t.fkey[f].as<uint64_t>();
        ft.runid[f] = runid;
        ft.cube[f] = t.fcube[f].as<double>();
        ft.nf = f + 1;
        t.nframes = f + 1;
        k_put_table<<<1, 1, 0, s>>>(ft, t.ftab.as<FrameTable>());
        LG_LAUNCHED();
        e.launches += 7;
        if (f + 1 == FRAMES) break;  // runs left now stay leaves at depth MAX_DEPTH
        // The next frame's runs: bodies re-keyed in this frame whose composite keys still tie.
        LG_CK(cudaMemsetAsync(counts + 6, 0, 4, s));
        k_find_runs<<<grid_for(n, BS), BS, 0, s>>>(sys, t.skey.as<uint64_t>(), t.ftab.as<FrameTable>(), nfr, f + 1, n,
                                                   t.runs.as<uint2>(), counts + 6, run_cap);
        LG_LAUNCHED();
        ++e.launches;
        LG_CK(cudaMemcpyAsync(e.pinned_small, counts + 6, 4, cudaMemcpyDeviceToHost, s));
        LG_CK(cudaStreamSynchronize(s));
        R = std::min(e.pinned_small[0], static_cast<unsigned>(run_cap));
    }
}

void tree_build(Engine& e, double theta) {
    TreeState& t = *e.tree;
    const int n = t.n_tree >= 0 ? t.n_tree : e.n;
    const uint32_t* sys = t.sys;
    cudaStream_t s = e.stream;
    t.group_max = e.group_max;
    t.theta = theta;
    const uint64_t* k0 = t.skey.as<uint64_t>();
    const FrameTable* ft = t.restarted ? t.ftab.as<FrameTable>() : nullptr;
    unsigned* counts = t.counts.as<unsigned>();
    const size_t n1 = static_cast<size_t>(n) + 1;
    t.leafid.reserve(n1 * 4);
    t.leaf_first.reserve(n1 * 4);
    t.leaf_depth.reserve(n1);
    t.leaf_gdepth.reserve(n1);
    t.leaf_c.reserve(n1);
    t.leaf_pre.reserve(n1 * 4);
    t.leaf_node.reserve(n1 * 4);
    if (t.group_max > GMAX_LIMIT) fail(kRuntime, "cuda tree build: group size above 1024");
    // Sizes: exact (one host read) for the first build and after a miss; otherwise the previous
    // build's with headroom, checked by tree_verify once the force call synchronises. On a miss the
    // kernels after k_leaves do nothing (counts[8]).
    const bool spec = t.have_guess && (t.speculative || t.restarted);
    const LeafOut leaf{t.leafid.as<uint32_t>(), t.leaf_first.as<uint32_t>(), t.leaf_pre.as<uint32_t>(),
                       t.leaf_depth.as<uint8_t>(), t.leaf_gdepth.as<uint8_t>(), t.leaf_c.as<int8_t>()};
    auto leaves = [&](unsigned Kcap, unsigned Tcap, const ZeroList& z) {
        const int tiles = leaf_tiles(n);
        launch_pdl(overlap(n), k_leaves, tiles, LEAF_BS, s, sys, k0, ft, n, t.group_max, leaf,
                   t.leaf_state.as<unsigned long long>(),
                   t.leaf_state.as<unsigned>() + 2 * static_cast<size_t>(tiles), counts, Kcap, Tcap, z,
                   e.err_word());
        ++e.launches;
    };
    if (!spec) {
        leaves(0xffffffffu, 0xffffffffu, ZeroList{});
        LG_CK(cudaMemcpyAsync(e.pinned_small, counts, 32, cudaMemcpyDeviceToHost, s));
        LG_CK(cudaStreamSynchronize(s));
        const size_t Kx = e.pinned_small[1], Tx = e.pinned_small[2];
        const int dx = static_cast<int>(e.pinned_small[4]);
        if (Kx < 1 || Kx > static_cast<size_t>(n) || Tx < Kx || Tx > Kx * (MAX_DEPTH + 1))
            fail(kRuntime, "cuda tree build: bad leaf/node count " + std::to_string(Kx) + "/" + std::to_string(Tx));
        // Headroom for the sync-free builds that follow (LETTUCE_GB300_TREE_HEADROOM percent, default
        // 25, plus a fixed slack unless it is 0): more memory against fewer exact rebuilds.
        size_t pct = 25;
        if (const char* h = std::getenv("LETTUCE_GB300_TREE_HEADROOM")) pct = static_cast<size_t>(std::atoi(h));
        const size_t slack = pct ? 1024 : 0;
        t.K = std::min(static_cast<size_t>(n), Kx + Kx * pct / 100 + slack);
        t.T = Tx + Tx * pct / 100 + slack;
        t.leaves = Kx;
        t.nodes = Tx;
        t.max_depth = std::min(dx + (pct ? 2 : 0), MAX_DEPTH + 1);
        t.known_depth = std::max(1, t.max_depth);
        t.have_guess = true;
        ++t.generation;
    }
    t.speculative = spec;
    const size_t K = t.K, T = t.T;
    const int depth = t.max_depth;
    // What has to be zero before the node kernels, in one buffer: the upsweep's buckets, the group
    // classes, the scan's look-back words and tile counter, the child masks. Cleared by k_leaves when
    // the sizes are known before it.
    const int scan_tiles = grid_for(static_cast<long long>(T), NSCAN_TILE);
    const size_t z_ix = (sizeof(UpsweepIndex) + 15) / 16 * 16, z_cls = 2 * GCLASS * 4,
                 z_state = static_cast<size_t>(scan_tiles) * 8 + 16;
    const size_t z_mask = (z_ix + z_cls + z_state + 15) / 16 * 16, z_all = z_mask + (T * 4 + 15) / 16 * 16;
    t.node_zero.reserve(z_all);
    t.pn_lohi.reserve(T * 8);
    t.pn_meta.reserve(T * 2);
    t.pn_parent.reserve(T * 4);
    t.pn_first.reserve(T * 4);
    t.grp_node.reserve(T * 4);
    t.grp_range.reserve(T * 8);
    t.grp_box.reserve(T * 32);
    t.grp_order.reserve(T * 4);
    t.nd_test.reserve(T * sizeof(NodeTest));
    t.nd_cell.reserve(T * sizeof(NodeCell));
    t.nd_geo.reserve(T * 16);
    t.nd_parent.reserve(T * 4);
    t.dep_nodes.reserve(T * 4);
    t.leaf_order.reserve(K * 4);
    char* zero = t.node_zero.as<char>();
    if (spec) {
        ZeroList z{};
        z.span[0] = {t.node_zero.as<uint4>(), z_all / 16};
        leaves(static_cast<unsigned>(std::min<size_t>(K, 0xffffffffu)), static_cast<unsigned>(std::min<size_t>(T, 0xffffffffu)), z);
    } else {
        LG_CK(cudaMemsetAsync(zero, 0, z_all, s));
    }
    UpsweepIndex* ix = reinterpret_cast<UpsweepIndex*>(zero);
    unsigned* cls = reinterpret_cast<unsigned*>(zero + z_ix);
    unsigned long long* scan_state = reinterpret_cast<unsigned long long*>(zero + z_ix + z_cls);
    const PreNodes pn{t.pn_lohi.as<uint2>(), t.pn_meta.as<uint16_t>(), t.pn_parent.as<uint32_t>(),
                      reinterpret_cast<uint32_t*>(zero + z_mask), t.pn_first.as<uint32_t>()};
    const NodeCtx x{sys, k0, ft, leaf, n, counts, static_cast<unsigned>(sys ? t.nsys : 1)};
    const uint32_t Tc = static_cast<uint32_t>(T);
    const int tb = grid_for(static_cast<long long>(T), NODE_BS);
    launch_pdl(overlap(n), k_nodes, tb, NODE_BS, s, x, pn, e.err_word());
    launch_pdl(overlap(n), k_node_scan, scan_tiles, NSCAN_BS, s, x, pn, scan_state,
               reinterpret_cast<unsigned*>(scan_state + scan_tiles), counts, ix, t.grp_node.as<uint32_t>(),
               e.err_word());
    e.launches += 2;
    // The group boxes depend neither on the nodes' order nor on the moments: with the reference groups
    // they are computed on the side stream from here on, and joined back before the build returns.
    t.merged = e.walk_merge && !sys;
    cudaStream_t gs = s;
    if (!t.merged) {
        LG_CK(cudaEventRecord(e.fork_ev, s));
        LG_CK(cudaStreamWaitEvent(e.side, e.fork_ev, 0));
        gs = e.side;
    }
    const int gb = grid_for(static_cast<long long>(std::min<size_t>(T, K)), BS);  // a group holds at least one leaf
    k_groups<<<gb, BS, 0, gs>>>(t.grp_node.as<uint32_t>(), t.pn_lohi.as<uint2>(), Tc, counts, e.bodies(e.cur),
                                t.grp_range.as<uint2>(), t.grp_box.as<float4>(), cls);
    LG_LAUNCHED();
    ++e.launches;
    if (!t.merged) {
        k_group_order<<<gb, BS, 0, gs>>>(t.grp_range.as<uint2>(), Tc, counts + 3, cls, t.grp_order.as<uint32_t>());
        LG_LAUNCHED();
        ++e.launches;
        LG_CK(cudaEventRecord(e.join_ev, e.side));
    }
    launch_pdl(overlap(n), k_nodes_out, tb, NODE_BS, s, x, pn, t.frame.as<double>(),
               t.nd_test.as<NodeTest>(), t.nd_geo.as<float4>(), t.nd_parent.as<uint32_t>(),
               t.leaf_node.as<uint32_t>(), ix, t.dep_nodes.as<uint32_t>(), t.leaf_order.as<uint32_t>(),
               e.err_word());
    ++e.launches;
    if (t.merged) {
        t.mcount.reserve(T * 4 + 4);
        t.moff.reserve(T * 4 + 4);
        t.mrange.reserve(T * 8 + 8);
        t.mbox.reserve(T * 32 + 32);
        k_merge_groups<false><<<tb, BS, 0, s>>>(t.grp_node.as<uint32_t>(), t.pn_parent.as<uint32_t>(),
                                                t.grp_range.as<uint2>(), counts + 3, Tc, counts + 2, std::min(e.merge_cap, t.group_max), t.mcount.as<uint32_t>(),
                                                nullptr, nullptr);
        LG_LAUNCHED();
        scan_u32(e, t, t.mcount.as<uint32_t>(), t.moff.as<uint32_t>(), static_cast<int>(T), counts + 5);
        k_merge_groups<true><<<tb, BS, 0, s>>>(t.grp_node.as<uint32_t>(), t.pn_parent.as<uint32_t>(),
                                               t.grp_range.as<uint2>(), counts + 3, Tc, counts + 2, std::min(e.merge_cap, t.group_max), nullptr,
                                               t.moff.as<uint32_t>(), t.mrange.as<uint2>());
        LG_LAUNCHED();
        k_merged_boxes<<<tb, BS, 0, s>>>(t.mrange.as<uint2>(), counts + 5, Tc, e.bodies(e.cur), t.mbox.as<float4>());
        LG_LAUNCHED();
        e.launches += 3;
    }
    // Upsweep: leaves (by size), then internal nodes level by level from the deepest; the depths of at
    // most TOP_NODES nodes (by the eight-way branching, or because the whole tree is small) together.
    const float inv_theta = theta > 0 ? static_cast<float>(1.0 / theta) : FLT_MAX;
    Moments mo{t.nd_test.as<NodeTest>(), t.nd_cell.as<NodeCell>()};
    const bool wide = t.leaves <= LEAFW_MAX;
    launch_pdl(overlap(n), wide ? k_leaf_moments_wide : k_leaf_moments,
               grid_for(static_cast<long long>(K), wide ? LEAFW_BS / WIDE : 128), wide ? LEAFW_BS : 128, s,
               t.leaf_order.as<uint32_t>(), counts, t.nd_geo.as<float4>(), e.bodies(e.cur), mo, inv_theta,
               t.inv_theta_sys, sys, e.err_word());
    ++e.launches;
    int top = -1;
    // The whole tree where that is faster than a launch per depth on all SMs: up to about 25 000 nodes at
    // the last exact build (build phase by depths -> all in one: Plummer 60 000 bodies, 14 460 nodes, 166
    // -> 133 us, 110 000, 25 423, 176 -> 165, 180 000, 41 051, 178 -> 193; a uniform cube, which has fewer
    // and wider depths, 60 000, 13 966, 133 -> 123, 80 000, 27 379, 137 -> 145).
    constexpr size_t WHOLE_MAX = 50 * TOP_NODES;
    if (t.nodes <= WHOLE_MAX) top = depth - 1;
    else
        for (size_t width = x.nroots; width <= TOP_NODES && top < depth - 1; width *= 8) ++top;
    const int cb = std::max(1, std::min(4 * e.sms, grid_for(static_cast<long long>(T), COMBINE_NODES)));
    // With more roots than one round of the cluster takes (a wide forest), every depth has its launch, and
    // the roots' radii a last one.
    const int last = top < 0 && depth > 0 ? -1 : top + 1;
    for (int d = depth - 1; d >= last; --d) {
        launch_pdl(overlap(n), k_combine_level, cb, COMBINE_BS, s, t.dep_nodes.as<uint32_t>(), ix, d,
                   counts, t.nd_geo.as<float4>(), mo, inv_theta, t.inv_theta_sys, sys, e.err_word());
        ++e.launches;
    }
    if (top >= 0) {
        // Clusters of 16 blocks are an opt-in size, for the current device.
        if (!t.clusters_of_16) {
            LG_CK(cudaFuncSetAttribute(k_combine_top, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
            t.clusters_of_16 = true;
        }
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at[2] = {};
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = TOP_BLOCKS;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.gridDim = dim3(TOP_BLOCKS);
        cfg.blockDim = dim3(TOP_BS);
        cfg.stream = s;
        cfg.attrs = at;
        cfg.numAttrs = overlap(n) ? 2 : 1;
        LG_CK(cudaLaunchKernelEx(&cfg, k_combine_top, static_cast<const uint32_t*>(t.dep_nodes.as<uint32_t>()),
                                 static_cast<const UpsweepIndex*>(ix), top, static_cast<const unsigned*>(counts),
                                 static_cast<const float4*>(t.nd_geo.as<float4>()), mo, inv_theta, t.inv_theta_sys, sys,
                                 e.err_word()));
        ++e.launches;
    }
    if (!t.merged) LG_CK(cudaStreamWaitEvent(s, e.join_ev, 0));
}

// After a synchronising point: true if the tree built with guessed sizes is valid (no key restart
// was missed, leaves, nodes and depth within what was launched). Otherwise records the exact need
// so that the caller's rebuild takes the exact path.
bool tree_verify(Engine& e, const unsigned* counts_host) {
    TreeState& t = *e.tree;
    if (!t.speculative) return true;
    const unsigned R = counts_host[0], K = counts_host[1], T = counts_host[2];
    const int depth = static_cast<int>(counts_host[4]);
    const bool long_run = counts_host[7] != 0;  // the tree is deeper than the digits sorted
    const bool ok = (t.restarted || R == 0) && K <= t.K && T <= t.T && depth <= t.max_depth && !long_run;
    if (!ok) {
        if (!t.restarted && R > 0) t.restart_mode = true;
        if (long_run) t.known_depth = 0;
        t.have_guess = false;  // next build reads exact sizes
    }
    return ok;
}

const unsigned* tree_counts_device(Engine& e) { return e.tree->counts.as<unsigned>(); }

namespace {
// Sets *sticky when the build just launched exceeded what it was launched for, or a key restart
// was needed: the same test as tree_verify, on the device, for step loops without host reads.
__global__ void k_tree_check(const unsigned* __restrict__ counts, unsigned K, unsigned T, int depth, int restarted,
                             unsigned* sticky) {
    const bool ok = (restarted || counts[0] == 0) && counts[1] <= K && counts[2] <= T &&
                    static_cast<int>(counts[4]) <= depth && counts[7] == 0;
    if (!ok) atomicOr(sticky, 1u);
}
}  // namespace

void tree_set_forest(Engine& e, int n_tree, int nsys, const uint32_t* sys, const uint32_t* sys_off,
                     const float* inv_theta_sys) {
    TreeState& t = *e.tree;
    t.n_tree = n_tree;
    t.nsys = nsys;
    t.sys = sys;
    t.sys_off = sys_off;
    t.inv_theta_sys = inv_theta_sys;
    t.have_guess = false;
    t.restart_mode = false;
    t.known_depth = 0;
}

bool tree_sync_free_ready(const Engine& e) { return e.tree->have_guess && !e.tree->restart_mode; }
uint64_t tree_generation(const Engine& e) { return e.tree->generation; }

void tree_check_async(Engine& e, unsigned* sticky) {
    TreeState& t = *e.tree;
    if (!t.speculative) return;
    k_tree_check<<<1, 1, 0, e.stream>>>(t.counts.as<unsigned>(), static_cast<unsigned>(t.K),
                                        static_cast<unsigned>(t.T), t.max_depth, t.restarted ? 1 : 0, sticky);
    LG_LAUNCHED();
    ++e.launches;
}
void tree_reset_guess(Engine& e) {
    e.tree->have_guess = false;
    e.tree->restart_mode = false;
}
void tree_reset(Engine& e) {
    tree_reset_guess(e);
    e.tree->known_depth = 0;
}
double tree_theta(const Engine& e) { return e.tree->theta; }

TreeView tree_view(Engine& e) {
    TreeState& t = *e.tree;
    TreeView v;
    v.nd_test = t.nd_test.as<NodeTest>();
    v.nd_cell = t.nd_cell.as<NodeCell>();
    v.grp_range = t.merged ? t.mrange.as<uint2>() : t.grp_range.as<uint2>();
    v.grp_box = t.merged ? t.mbox.as<float4>() : t.grp_box.as<float4>();
    v.grp_order = t.merged ? nullptr : t.grp_order.as<uint32_t>();
    v.ngroups = t.counts.as<unsigned>() + (t.merged ? 5 : 3);
    v.T = t.T;  // capacity the build was launched with (>= the node count)
    v.nd_parent = t.nd_parent.as<uint32_t>();
    v.body_leaf = t.leafid.as<uint32_t>();
    v.leaf_node = t.leaf_node.as<uint32_t>();
    v.nleaves = t.counts.as<unsigned>() + 1;
    v.K = t.K;
    return v;
}

void tree_counts(Engine& e, size_t* nodes, size_t* leaves, size_t* groups, int* max_depth) {
    TreeState& t = *e.tree;
    if (!e.tree_ok) fail(kLogic, "tree introspection: call build_tree (tree method) first");
    e.ensure_tree_valid();
    LG_CK(cudaMemcpyAsync(e.pinned_small, t.counts.as<unsigned>(), 32, cudaMemcpyDeviceToHost, e.stream));
    LG_CK(cudaStreamSynchronize(e.stream));
    if (nodes) *nodes = e.pinned_small[2];
    if (leaves) *leaves = e.pinned_small[1];
    if (groups) *groups = e.pinned_small[t.merged ? 5 : 3];
    if (max_depth) *max_depth = static_cast<int>(e.pinned_small[4]);
}

// The reference's key array after a build (src/cpu_backend.cpp:884-906 key_): each body's key in
// the last frame it was re-keyed in (rekey overwrites key_ inside a run; a coincident run keeps
// the keys it had).
void tree_keys(Engine& e, uint64_t* keys, size_t n) {
    TreeState& t = *e.tree;
    if (!e.tree_ok) fail(kLogic, "tree introspection: call build_tree (tree method) first");
    e.ensure_tree_valid();
    if (n < static_cast<size_t>(e.n)) fail(kArg, "tree_keys: output holds fewer than n keys");
    const size_t N = static_cast<size_t>(e.n);
    LG_CK(cudaMemcpyAsync(keys, t.skey.as<uint64_t>(), N * 8, cudaMemcpyDeviceToHost, e.stream));
    if (t.restarted) {
        std::vector<uint8_t> nfr(N);
        std::vector<std::vector<uint64_t>> fk(t.nframes);
        LG_CK(cudaMemcpyAsync(nfr.data(), t.nfr.as<uint8_t>(), N, cudaMemcpyDeviceToHost, e.stream));
        for (int f = 1; f < t.nframes; ++f) {
            fk[f].resize(N);
            LG_CK(cudaMemcpyAsync(fk[f].data(), t.fkey[f].as<uint64_t>(), N * 8, cudaMemcpyDeviceToHost, e.stream));
        }
        LG_CK(cudaStreamSynchronize(e.stream));
        for (size_t i = 0; i < N; ++i)
            if (nfr[i] > 1) keys[i] = fk[nfr[i] - 1][i];
    }
    LG_CK(cudaStreamSynchronize(e.stream));
}

void tree_nodes(Engine& e, uint32_t* range4, float* moments11, float* geo4, size_t nodes) {
    TreeState& t = *e.tree;
    if (!e.tree_ok) fail(kLogic, "tree introspection: call build_tree (tree method) first");
    size_t T = 0;
    tree_counts(e, &T, nullptr, nullptr, nullptr);
    if (nodes < T) fail(kArg, "tree_nodes: output holds fewer than the node count");
    if (range4)
        LG_CK(cudaMemcpy2DAsync(range4, 16, &t.nd_test.as<NodeTest>()->range, sizeof(NodeTest), 16, T,
                                cudaMemcpyDeviceToHost, e.stream));
    if (geo4) LG_CK(cudaMemcpyAsync(geo4, t.nd_geo.as<float4>(), T * 16, cudaMemcpyDeviceToHost, e.stream));
    if (moments11) {
        std::vector<NodeCell> c(T);
        LG_CK(cudaMemcpyAsync(c.data(), t.nd_cell.as<NodeCell>(), T * sizeof(NodeCell), cudaMemcpyDeviceToHost, e.stream));
        LG_CK(cudaStreamSynchronize(e.stream));
        for (size_t k = 0; k < T; ++k) {
            float* o = moments11 + 11 * k;
            o[0] = c[k].com.x; o[1] = c[k].com.y; o[2] = c[k].com.z; o[3] = c[k].com.w;
            o[4] = c[k].q0.x; o[5] = c[k].q0.y; o[6] = c[k].q0.z; o[7] = c[k].q0.w;
            o[8] = c[k].q1.x; o[9] = c[k].q1.y; o[10] = c[k].q1.z;
        }
    }
    LG_CK(cudaStreamSynchronize(e.stream));
}

void tree_groups(Engine& e, float* box6, uint32_t* lohi, size_t groups) {
    TreeState& t = *e.tree;
    if (!e.tree_ok) fail(kLogic, "tree introspection: call build_tree (tree method) first");
    size_t G = 0;
    tree_counts(e, nullptr, nullptr, &G, nullptr);
    if (groups < G) fail(kArg, "tree_groups: output holds fewer than the group count");
    // The walk's groups (merged ones when the engine packs them).
    const uint2* range = t.merged ? t.mrange.as<uint2>() : t.grp_range.as<uint2>();
    const float4* gbox = t.merged ? t.mbox.as<float4>() : t.grp_box.as<float4>();
    if (lohi) LG_CK(cudaMemcpyAsync(lohi, range, G * 8, cudaMemcpyDeviceToHost, e.stream));
    if (box6) {
        std::vector<float4> box(2 * G);
        LG_CK(cudaMemcpyAsync(box.data(), gbox, G * 32, cudaMemcpyDeviceToHost, e.stream));
        LG_CK(cudaStreamSynchronize(e.stream));
        for (size_t g = 0; g < G; ++g) {
            box6[6 * g] = box[2 * g].x; box6[6 * g + 1] = box[2 * g].y; box6[6 * g + 2] = box[2 * g].z;
            box6[6 * g + 3] = box[2 * g + 1].x; box6[6 * g + 4] = box[2 * g + 1].y; box6[6 * g + 5] = box[2 * g + 1].z;
        }
    }
    LG_CK(cudaStreamSynchronize(e.stream));
}

lg_memory_estimate memory_need(uint64_t n, int method) {
    lg_memory_estimate r{};
    // Two body sets (80 B), accelerations (16 B), staging (12 B), plus fixed buffers.
    r.device = 192 * n + (uint64_t(64) << 20);
    if (method == LG_TREE) r.device += 112 * n;  // keys, sort buffers, per-body tree data, ~0.2 n nodes
    r.host = 0;
    return r;
}

size_t tree_held_bytes(const Engine& e) {
    const TreeState& t = *e.tree;
    size_t h = 0;
    for (const DevBuf* d : {&t.keysA, &t.keysB, &t.valsA, &t.valsB, &t.hist, &t.lookback, &t.mkeys, &t.skey, &t.key1tmp,
                            &t.nfr, &t.ftab, &t.leafid, &t.frame, &t.runs, &t.counts, &t.leaf_first, &t.leaf_depth,
                            &t.leaf_gdepth, &t.leaf_c, &t.leaf_pre, &t.leaf_node, &t.leaf_state, &t.pn_lohi,
                            &t.pn_meta, &t.pn_parent, &t.pn_first, &t.node_zero, &t.nd_test, &t.nd_cell, &t.nd_geo,
                            &t.nd_parent, &t.grp_node, &t.dep_nodes, &t.leaf_order, &t.grp_range, &t.grp_box,
                            &t.grp_order, &t.scan_state, &t.scan_ctr})
        h += d->capacity();
    for (int f = 1; f < FRAMES; ++f) h += t.fkey[f].capacity() + t.frunid[f].capacity() + t.fcube[f].capacity();
    return h;
}

}  // namespace lg
