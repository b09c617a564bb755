// Tree walk: the reference CPU backend's group walk (src/cpu_backend.cpp:667-689 walk,
// :816-838 build_list, :841-882 eval_group), GB300 form.
//
// One block per walk group (persistent blocks pull groups from an atomic counter), its warps
// specialised: one warp builds the group's list while four evaluate it.
//  - List build (one warp): a warp-cooperative depth-first traversal. The stack (shared memory, with
//    a global overflow slice per block) holds child blocks, one entry per opened node. A round takes
//    the top eight entries, two per team of eight lanes, two children per lane (an octree node of these
//    trees has 7.5 children on average, so 94% of the lanes hold a node and no prefix sum is
//    needed to deal nodes out), and applies the reference's opening rule against the group's
//    bounding box: a node that contains the group, or whose box distance d satisfies d^2 < rcrit2,
//    is opened; an accepted leaf of <= 4 bodies is taken as bodies, other accepted nodes as cells;
//    opened leaves give bodies, opened internal nodes push their child block. Appends and pushes
//    are compacted with ballots. Full lists go to the evaluating warps as packets of two
//    alternating slots, so the traversal's latency (a third of the time when the same warps did
//    both) overlaps the arithmetic, across groups too.
//  - Evaluation (four warps): a packet's entries are converted once to coordinates relative to the
//    group's box centre o, (x_hi - o) + x_lo in FP32, two entries per thread, into a shared chunk
//    of packed pairs, and every lane evaluates its share: the 128 lanes form P partitions of
//    ceil(np / IPT) lanes, each partition holds all np bodies of the group (IPT per lane) and takes
//    every P-th pair of entries. P is any whole number, so the lanes stay filled whatever the
//    group's size. Quadrupole cell terms (cuda_backend.cu:783-800 / cpu_backend.cpp:858-871 math)
//    and softened body terms; two consecutive entries per packed f32x2 instruction, operands
//    loaded as 128-bit pairs of pairs. Every MERGE pairs, and
//    at a packet's end, a lane's sums are added to running sums in shared memory with Kahan compensation, and the partitions' sums are added in partition order at the end,
//    compensated too.
// What it measured against one warp per group doing both (IPT up to 4, 16 warps per SM; GB300, walk
// phase): 8191 bodies 364 -> 68 us and 100 003 bodies 873 -> 377 us (several warps now share a
// group, and the walk no longer ends on a few large ones: see group_class in tree.cu), 1e6 disk
// 2.63 -> 2.18 ms, 1.6e7 collision 51.6 -> 47.2 ms. Bound on the 1e6 disk by latency on both
// sides: the FMA pipe is 60% busy, the list warp never waits for a packet slot (96 000 cycles a
// group under load, 53 000 with no evaluation beside it), the evaluating warps wait for it a fifth
// of their time. Measured and not taken there: two list warps per block (2.30 ms), four i-bodies
// per lane on two (2.54) or four (2.42) evaluating warps, 256 evaluating threads (2.42), a second
// chunk buffer in place of the second barrier (2.26), one or three nodes per lane (2.34, 2.32).
// The roles meet at named barriers only: FULL (packet written: the list warp arrives, the others
// wait), EMPTY (packet read: the reverse) and one among the evaluating warps. Every packet sent is
// received, an overflowing traversal still sends its group's last packet, and the list warp ends
// with an END packet, so no wait is left unanswered.
// The interaction count per body is the list length minus its own entry; the reference CPU
// backend counts that self entry, so its count exceeds this one by exactly N. The own entry adds
// nothing to the acceleration (d = 0) and is excluded from the potential by index.
#include "engine.cuh"
#include "walk_common.cuh"

namespace lg {

namespace {

using walk::REMOTE;
using walk::SCAP;
using walk::SMALL_LEAF;

constexpr int EVAL = 128;       // evaluating threads
constexpr int WBS = EVAL + 32;  // and the list warp
constexpr int MINB = 4;         // resident blocks per SM: 20 warps at 96 registers (5 at 72 spill)
constexpr int IPT = 2;          // i-bodies per lane
constexpr int BUNROLL = 3;      // body pairs evaluated together
constexpr int PASS = 128;          // i-bodies per pass
constexpr int CCAP = 320;          // cells per packet
constexpr int BCAP = 768;          // bodies per packet
constexpr int RCAP = 256;          // body ranges per packet
constexpr int MERGE = 96;          // pairs a lane sums in plain FP32 before a compensated addition
constexpr int LEAF = 16;           // ranges up to this length are appended one per lane and node
constexpr int NPL = 2;             // nodes per lane and traversal round
constexpr int BWORDS = (BCAP + 31) / 32;
constexpr int BSTK = 256, BREFILL = 128;  // shared stack entries; entries fetched back at a time
static_assert(PASS <= EVAL * IPT && CCAP % 2 == 0 && CCAP >= 32 * NPL, "cells: whole pairs, at least a round's");
static_assert(BCAP % 2 == 0 && RCAP >= 32 * NPL && BCAP <= 1024 && BWORDS <= 32, "bodies: whole pairs, at least a round's");

enum : unsigned { kFirst = 1u, kLast = 2u, kAbort = 4u, kEnd = 8u };  // packet flags
enum { kBarFull = 1, kBarEmpty = 3, kBarEval = 5 };  // named barriers (FULL, EMPTY: one per slot)

struct __align__(16) Packet {
    uint32_t cell[CCAP];  // node indices
    // Bodies as ranges back to back: position p of the packet lies in the range whose number is one
    // less than the set bits of starts up to and including p; its body is base + p.
    uint32_t base[RCAP];      // first body of the range minus the range's start
    uint32_t starts[BWORDS];  // bit p: a range starts at position p
    int before[BWORDS];       // set bits in the words before, minus one
    float4 centre;        // group box centre, squared softening
    uint32_t plo, np;     // the pass's bodies
    int nc, nb;
    uint32_t list_len;    // on the last packet: entries of the whole list
    unsigned flags;
};

struct __align__(16) WalkSmem {
    // Packed pairs: entry 2q in the even float of each two, entry 2q + 1 in the odd one.
    float4 cell[CCAP / 2][5];  // (x x y y)(z z m m)(xx xx xy xy)(xz xz yy yy)(yz yz zz zz), -Q
    float4 body[BCAP / 2][2];  // (x x y y)(z z m m)
    Packet pk[2];
    uint2 stk[BSTK];           // traversal stack: first child, children
    float ks[IPT][8][EVAL];    // per lane and i-body: Kahan sums x y z phi, their compensations
    uint32_t kself[PASS];      // with the potential: packet number << 10 | position of the i-body in the chunk
};

struct WalkArgs {
    TreeView tv;
    const float4* hm;
    const float4* lo;
    float4* acc;
    float* cost;
    uint2* stack;
    unsigned* group_ctr;
    unsigned long long* inter;
    unsigned* err;
    // What the last block to finish hands to the host (see tree_walk), or null.
    unsigned* report;
    unsigned* done;
    const unsigned* counts;
    float G, e2;
    // Forest (ensemble) walk: body -> system (nullptr: one tree rooted at node 0) and the
    // per-system squared softening; system s's tree is rooted at node s.
    const uint32_t* sys;
    const float* e2_sys;
    // Remote trees walked after the local tree (or alone: local == 0, for the direct method's
    // blocks of consecutive bodies); accumulate adds to acc and cost instead of overwriting.
    LetView let;
    int local;
    int accumulate;
    // Block time steps: passes whose bodies all have level < kmin are skipped (level == nullptr: none).
    const uint8_t* level;
    int kmin;
};

// Two packed pairs by one 128-bit shared load.
__device__ __forceinline__ void ld4(const float4* p, f2x& a, f2x& b) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    a = v.x;
    b = v.y;
}

template <bool EPS0>
__device__ __forceinline__ f2x pair_rsqrt(f2x r2) {
    float lo, hi;
    f2_unpack(r2, lo, hi);
    float a = rsqrt_mufu(lo), b = rsqrt_mufu(hi);
    if (EPS0) {
        a = lo > 0.f ? a : 0.f;
        b = hi > 0.f ? b : 0.f;
    }
    return f2_pack(a, b);
}

// A lane's share of the pass: its i-bodies relative to the group's centre and its partition.
struct Lane {
    f2x X[IPT], Y[IPT], Z[IPT];
    int part, P;  // idle lanes: part past every chunk
};

// The lane's sums over one packet, packed halves.
struct Sums {
    f2x x[IPT], y[IPT], z[IPT], p[IPT];
};

// Quadrupole cell terms: d points from the body to the cell,
// a = G [M d/r^3 - Q d/r^5 + 5/2 (dQd) d/r^7], phi = -G [M/r + 1/2 dQd/r^5]. The chunk holds -Q
// (negated when converted), which spares one negation per pair; sign changes are exact. The next
// pair's position and mass are loaded while this pair is evaluated, so the chain from the offset
// through the reciprocal root starts without waiting for shared memory.
template <bool POT, bool EPS0>
__device__ __forceinline__ void eval_cells(const WalkSmem& s, int pairs, const Lane& l, Sums& a, f2x E2) {
    const f2x CN25 = f2_bcast(-2.5f), CN05 = f2_bcast(-0.5f);
    if (l.part >= pairs) return;
    f2x X, Y, Z, M;
    ld4(s.cell[l.part], X, Y);
    ld4(s.cell[l.part] + 1, Z, M);
    for (int k = l.part; k < pairs; k += l.P) {
        f2x QXX, QXY, QXZ, QYY, QYZ, QZZ, NX, NY, NZ, NM;
        const float4* c = s.cell[k];
        const float4* n = s.cell[min(k + l.P, pairs - 1)];
        ld4(c + 2, QXX, QXY);
        ld4(c + 3, QXZ, QYY);
        ld4(c + 4, QYZ, QZZ);
        ld4(n, NX, NY);
        ld4(n + 1, NZ, NM);
        f2x dx[IPT], dy[IPT], dz[IPT], inv[IPT];
#pragma unroll
        for (int u = 0; u < IPT; ++u) {
            dx[u] = f2_sub(X, l.X[u]);
            dy[u] = f2_sub(Y, l.Y[u]);
            dz[u] = f2_sub(Z, l.Z[u]);
            inv[u] = f2_fma(dx[u], dx[u], f2_fma(dy[u], dy[u], f2_fma(dz[u], dz[u], E2)));
        }
#pragma unroll
        for (int u = 0; u < IPT; ++u) inv[u] = pair_rsqrt<EPS0>(inv[u]);
        // qx, qy, qz = -(Q d); sd = -(dQd)
        f2x qx[IPT], qy[IPT], qz[IPT], sd[IPT];
#pragma unroll
        for (int u = 0; u < IPT; ++u) {
            qx[u] = f2_fma(QXX, dx[u], f2_fma(QXY, dy[u], f2_mul(QXZ, dz[u])));
            qy[u] = f2_fma(QXY, dx[u], f2_fma(QYY, dy[u], f2_mul(QYZ, dz[u])));
            qz[u] = f2_fma(QXZ, dx[u], f2_fma(QYZ, dy[u], f2_mul(QZZ, dz[u])));
            sd[u] = f2_fma(dx[u], qx[u], f2_fma(dy[u], qy[u], f2_mul(dz[u], qz[u])));
        }
#pragma unroll
        for (int u = 0; u < IPT; ++u) {
            const f2x inv2 = f2_mul(inv[u], inv[u]), inv3 = f2_mul(inv[u], inv2), inv5 = f2_mul(inv3, inv2);
            const f2x f = f2_fma(f2_mul(f2_mul(CN25, sd[u]), inv2), inv5, f2_mul(M, inv3));
            a.x[u] = f2_fma(qx[u], inv5, f2_fma(f, dx[u], a.x[u]));
            a.y[u] = f2_fma(qy[u], inv5, f2_fma(f, dy[u], a.y[u]));
            a.z[u] = f2_fma(qz[u], inv5, f2_fma(f, dz[u], a.z[u]));
            if (POT) a.p[u] = f2_add(a.p[u], f2_fma(M, inv[u], f2_mul(f2_mul(CN05, sd[u]), inv5)));
        }
        X = NX; Y = NY; Z = NZ; M = NM;
    }
}

// Softened body terms a = G m d / r^3, phi = -G m / r, NK pairs of entries (k, k + P, ...) at a time
// with their operations interleaved. With the potential, the own body's pair is taken out by index
// (its mass half set to zero): kself[u] is the chunk position of the lane's u-th i-body (-2: not
// in this chunk).
template <int NK, bool POT, bool EPS0>
__device__ __forceinline__ void body_pairs(const WalkSmem& s, int k, const Lane& l, Sums& a, const int (&kself)[IPT],
                                           f2x E2) {
    f2x X[NK], Y[NK], Z[NK], M[NK];
#pragma unroll
    for (int q = 0; q < NK; ++q) {
        ld4(s.body[k + q * l.P], X[q], Y[q]);
        ld4(s.body[k + q * l.P] + 1, Z[q], M[q]);
    }
    f2x dx[NK][IPT], dy[NK][IPT], dz[NK][IPT], inv[NK][IPT];
#pragma unroll
    for (int q = 0; q < NK; ++q)
#pragma unroll
        for (int u = 0; u < IPT; ++u) {
            dx[q][u] = f2_sub(X[q], l.X[u]);
            dy[q][u] = f2_sub(Y[q], l.Y[u]);
            dz[q][u] = f2_sub(Z[q], l.Z[u]);
            inv[q][u] = f2_fma(dx[q][u], dx[q][u], f2_fma(dy[q][u], dy[q][u], f2_fma(dz[q][u], dz[q][u], E2)));
        }
#pragma unroll
    for (int q = 0; q < NK; ++q)
#pragma unroll
        for (int u = 0; u < IPT; ++u) inv[q][u] = pair_rsqrt<EPS0>(inv[q][u]);
#pragma unroll
    for (int q = 0; q < NK; ++q)
#pragma unroll
        for (int u = 0; u < IPT; ++u) {
            f2x Mu = M[q];
            if (POT) {
                const unsigned off = static_cast<unsigned>(kself[u] - 2 * (k + q * l.P));
                if (off <= 1u) Mu = f2_mul(Mu, off == 0 ? f2_pack(0.f, 1.f) : f2_pack(1.f, 0.f));
            }
            const f2x mi = f2_mul(Mu, inv[q][u]);  // the self pair (d = 0) adds nothing to a
            const f2x f = f2_mul(mi, f2_mul(inv[q][u], inv[q][u]));
            a.x[u] = f2_fma(f, dx[q][u], a.x[u]);
            a.y[u] = f2_fma(f, dy[q][u], a.y[u]);
            a.z[u] = f2_fma(f, dz[q][u], a.z[u]);
            if (POT) a.p[u] = f2_add(a.p[u], mi);
        }
}

template <bool POT, bool EPS0>
__device__ __forceinline__ void eval_bodies(const WalkSmem& s, int first, int pairs, const Lane& l, Sums& a,
                                            const int (&kself)[IPT], f2x E2) {
    int k = first + l.part;
    for (; k + (BUNROLL - 1) * l.P < pairs; k += BUNROLL * l.P) body_pairs<BUNROLL, POT, EPS0>(s, k, l, a, kself, E2);
    for (; k < pairs; k += l.P) body_pairs<1, POT, EPS0>(s, k, l, a, kself, E2);
}

// A far, massless entry: pads a chunk to an even count and contributes exactly zero.
constexpr float kFar = 1e18f;

// The record of list entry nd; LET: entries of remote trees carry the REMOTE bit.
template <bool LET>
__device__ __forceinline__ NodeCell load_cell(const WalkArgs& w, uint32_t nd) {
    if (!LET || !(nd & REMOTE)) return w.tv.nd_cell[nd];
    const uint32_t k = nd & ~REMOTE;
    NodeCell r;
    r.com = w.let.com[k]; r.q0 = w.let.q0[k]; r.q1 = w.let.q1[k];
    r.lo = make_float4(0.f, 0.f, 0.f, 0.f);
    return r;
}

template <bool LET>
__device__ __forceinline__ void load_body(const WalkArgs& w, uint32_t j, float4& h, float4& l) {
    if (!LET || !(j & REMOTE)) {
        h = w.hm[j];
        l = w.lo[j];
    } else {
        h = w.let.body[j & ~REMOTE];
        l = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

__device__ __forceinline__ void bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// ---- the list warp -------------------------------------------------------------------------------
// Box distance squared, in the reference's fused float form.
__device__ __forceinline__ float box_d2(float4 com, float4 bc, float4 bh) {
    const float dx = fmaxf(__fsub_rn(fabsf(__fsub_rn(com.x, bc.x)), bh.x), 0.f);
    const float dy = fmaxf(__fsub_rn(fabsf(__fsub_rn(com.y, bc.y)), bh.y), 0.f);
    const float dz = fmaxf(__fsub_rn(fabsf(__fsub_rn(com.z, bc.z)), bh.z), 0.f);
    return __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
}

// What a lane's node turned out to be.
enum { kNone, kCell, kBodies, kChildren };

template <bool LET>
__device__ __forceinline__ void build_lists(const WalkArgs& w, WalkSmem& s) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int team = lane >> 3;
    const uint32_t sub = lane & 7;
    uint2* gstk = w.stack + static_cast<size_t>(blockIdx.x) * SCAP;
    const unsigned ngroups = *w.tv.ngroups;
    const uint32_t T = static_cast<uint32_t>(w.tv.T);
    // With the local tree the own body is in the list (its leaf is inside the group, so it is
    // opened): it is not an interaction, adds nothing to a (d = 0) and is excluded from the
    // potential by index. Remote trees never hold the target.
    const uint32_t self = w.local ? 1u : 0u;
    const int ntrees = LET ? w.let.ntrees : 0;
    unsigned long long inter_b = 0, inter_c = 0;
    unsigned sent = 0;  // packets sent; the next one goes to slot sent & 1
    int nc = 0, nr = 0, nb = 0;
    uint32_t list_len = 0, cells_len = 0;
    unsigned first = 0;
    float4 bc = make_float4(0.f, 0.f, 0.f, 0.f);
    float e2 = w.e2;
    uint32_t plo = 0;
    int np = 0;
    if (lane < BWORDS) s.pk[0].starts[lane] = s.pk[1].starts[lane] = 0u;
    __syncwarp();
    auto send = [&](unsigned flags) {
        list_len += static_cast<uint32_t>(nc + nb);
        cells_len += static_cast<uint32_t>(nc);
        Packet& k = s.pk[sent & 1];
        const int ones = lane < BWORDS ? __popc(k.starts[lane]) : 0;
        int incl = ones;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += t;
        }
        if (lane < BWORDS) k.before[lane] = incl - ones - 1;
        if (lane == 0) {
            k.centre = make_float4(bc.x, bc.y, bc.z, e2);
            k.plo = plo;
            k.np = static_cast<uint32_t>(np);
            k.nc = nc;
            k.nb = nb;
            k.list_len = list_len;
            k.flags = flags | first;
        }
        __syncwarp();
        __threadfence_block();
        bar_arrive(kBarFull + (sent & 1), WBS);
        first = 0;
        nc = nr = nb = 0;
        ++sent;
        if (sent >= 2 && !(flags & kEnd)) {
            bar_sync(kBarEmpty + (sent & 1), WBS);
            if (lane < BWORDS) s.pk[sent & 1].starts[lane] = 0u;
            __syncwarp();
        }
    };
    // The first group by block, so that the largest groups, first in grp_order, start on different
    // SMs; the others from the counter, asked for only when a traversal is over: a number taken
    // earlier would keep a group waiting for this block while others are idle.
    unsigned g = blockIdx.x;
    while (g < ngroups) {
        if (w.tv.grp_order) g = w.tv.grp_order[g];
        const uint2 gr = w.tv.grp_range[g];
        bc = w.tv.grp_box[2 * g];
        const float4 bh = w.tv.grp_box[2 * g + 1];
        const uint32_t root = w.sys ? w.sys[gr.x] : 0u;
        if (w.e2_sys) e2 = w.e2_sys[root];
        unsigned g_next = 0xffffffffu;
        for (plo = gr.x; plo < gr.y; plo += PASS) {
            np = static_cast<int>(min(static_cast<uint32_t>(PASS), gr.y - plo));
            if (w.level) {
                bool active = false;
                for (int k = lane; k < np; k += 32) active |= w.level[plo + k] >= w.kmin;
                if (!__any_sync(0xffffffffu, active)) continue;
            }
            first = kFirst;
            list_len = cells_len = 0;
            int src = !LET || w.local ? -1 : 0;  // -1: the local tree, then the remote trees
            int sp = 0, gsp = 0;                 // stack entries in shared memory, in the global part
            unsigned fault = 0;
            // Each node is visited at most once per pass; the cap stops a malformed tree.
            const uint32_t max_iter = T + (LET ? w.let.nnodes + static_cast<uint32_t>(ntrees) : 0u) + 64u;
            uint32_t iter = 0;
            // The round's entries: the lane's child blocks (first child, children), or none. Their
            // node records are fetched before the previous round's entries are appended, so the fetch
            // overlaps the appends.
            uint2 ent[NPL];
            NodeTest nd[NPL];
            auto fetch = [&] {
#pragma unroll
                for (int h = 0; h < NPL; ++h)
                    if ((!LET || src < 0) && sub < ent[h].y && ent[h].x + sub < T) nd[h] = w.tv.nd_test[ent[h].x + sub];
            };
            bool any = !LET || src < ntrees;
#pragma unroll
            for (int h = 0; h < NPL; ++h) {
                ent[h] = make_uint2(0u, 0u);
                nd[h].com = make_float4(0.f, 0.f, 0.f, 0.f);
                nd[h].range = make_uint4(0u, 0u, 0u, 0u);
            }
            if (any && team == 0) ent[0] = make_uint2(!LET || src < 0 ? root : w.let.roots[src], 1u);
            fetch();
            while (any) {
                if (++iter > max_iter) {
                    fault = kErrNodeOverflow;
                    break;
                }
                int kind[NPL];
                uint32_t a0[NPL], a1[NPL];
#pragma unroll
                for (int h = 0; h < NPL; ++h) {
                    // A block of more than eight (remote trees only) keeps its tail on the stack as
                    // one of the round's pushes.
                    const bool have = sub < ent[h].y;
                    const uint32_t node = ent[h].x + sub;
                    kind[h] = kNone;
                    a0[h] = a1[h] = 0;
                    if (!LET || src < 0) {
                        const uint4 rg = nd[h].range;
                        const bool contains = rg.x <= gr.x && gr.y <= rg.y;
                        const bool open = contains || !(box_d2(nd[h].com, bc, bh) >= nd[h].com.w);
                        const bool leaf = rg.w == 0;
                        const uint32_t cnt = rg.y - rg.x;
                        const bool bodies = leaf && (open || cnt <= static_cast<uint32_t>(SMALL_LEAF));
                        const bool ok = node < T && (!open || leaf || (rg.w <= 8u && rg.z + rg.w <= T));
                        if (have) {
                            kind[h] = bodies ? kBodies : open ? kChildren : kCell;
                            a0[h] = bodies ? rg.x : open ? rg.z : node;
                            a1[h] = bodies ? cnt : rg.w;
                            if (!ok) {
                                kind[h] = kNone;
                                atomicOr(w.err, kErrNodeOverflow);
                            }
                        }
                    } else if (have) {
                        // The receiver walk of a remote tree (src/backend.hpp:77-82,
                        // src/cpu_backend.cpp:787-812): a node with no children and no bodies, or
                        // whose box distance d satisfies d^2 >= rcrit2, is accepted (as bodies when
                        // it holds 1..SMALL_LEAF of them, else as a multipole); otherwise its bodies,
                        // or else its children, are taken.
                        if (node >= w.let.nnodes) atomicOr(w.err, kErrNodeOverflow);
                        else {
                            const int4 L = w.let.link[node];
                            bool accept = L.x < 0 && L.w == 0;
                            if (!accept) accept = box_d2(w.let.com[node], bc, bh) >= w.let.q1[node].z;
                            if (L.w > 0 && (!accept || L.w <= SMALL_LEAF)) {
                                kind[h] = kBodies; a0[h] = REMOTE | static_cast<uint32_t>(L.z); a1[h] = L.w;
                            } else if (accept) {
                                kind[h] = kCell; a0[h] = REMOTE | node;
                            } else if (L.y > 0) {
                                kind[h] = kChildren; a0[h] = static_cast<uint32_t>(L.x); a1[h] = L.y;
                            }
                        }
                    }
                }
                // ---- pushes, and the next round's entries
                unsigned pm[NPL], tm[NPL];
                int npush = 0;
#pragma unroll
                for (int h = 0; h < NPL; ++h) {
                    pm[h] = __ballot_sync(0xffffffffu, kind[h] == kChildren);
                    tm[h] = LET ? __ballot_sync(0xffffffffu, ent[h].y > 8u && sub == 7u) : 0u;
                    npush += __popc(pm[h]) + __popc(tm[h]);
                }
                if (sp + npush > BSTK) {  // the shared part moves to the global part
                    if (gsp + sp > SCAP) {
                        fault = kErrStackOverflow;
                        break;
                    }
                    for (int q = lane; q < sp; q += 32) gstk[gsp + q] = s.stk[q];
                    gsp += sp;
                    sp = 0;
                    __syncwarp();
                }
#pragma unroll
                for (int h = 0; h < NPL; ++h) {
                    int op = sp + __popc(tm[h] & lt) + __popc(pm[h] & lt);
                    if (LET && ((tm[h] >> lane) & 1u)) s.stk[op++] = make_uint2(ent[h].x + 8u, ent[h].y - 8u);
                    if (kind[h] == kChildren) s.stk[op] = make_uint2(a0[h], a1[h]);
                    sp += __popc(pm[h]) + __popc(tm[h]);
                }
                __syncwarp();
                if (sp == 0 && gsp > 0) {  // refill from the global part (its top entries)
                    const int k = min(BREFILL, gsp);
                    for (int q = lane; q < k; q += 32) s.stk[q] = gstk[gsp - k + q];
                    gsp -= k;
                    sp = k;
                    __syncwarp();
                }
                any = sp > 0;
#pragma unroll
                for (int h = 0; h < NPL; ++h)
                    ent[h] = team + 4 * h < sp ? s.stk[sp - 1 - team - 4 * h] : make_uint2(0u, 0u);
                sp = max(sp - 4 * NPL, 0);
                if (LET && !any && src + 1 < ntrees) {  // the next remote tree
                    ++src;
                    if (team == 0) ent[0] = make_uint2(w.let.roots[src], 1u);
                    any = true;
                }
                fetch();
                // ---- appends
                unsigned cm[NPL], rm[NPL], sm[NPL];
                int ncell = 0, nrange = 0, len[NPL], off = 0, tot = 0;
#pragma unroll
                for (int h = 0; h < NPL; ++h) {
                    const bool shortr = kind[h] == kBodies && a1[h] - 1u < static_cast<uint32_t>(LEAF);
                    cm[h] = __ballot_sync(0xffffffffu, kind[h] == kCell);
                    rm[h] = __ballot_sync(0xffffffffu, kind[h] == kBodies);
                    sm[h] = __ballot_sync(0xffffffffu, shortr);
                    ncell += __popc(cm[h]);
                    nrange += __popc(rm[h]);
                    len[h] = shortr ? static_cast<int>(a1[h]) : 0;
                    off += len[h];
                }
                if (nrange) {
                    const int mine = off;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const int t = __shfl_up_sync(0xffffffffu, off, d);
                        if (lane >= d) off += t;
                    }
                    tot = __shfl_sync(0xffffffffu, off, 31);
                    off -= mine;
                    if (tot > BCAP) {  // more than a packet in one round: one range at a time
                        tot = 0;
#pragma unroll
                        for (int h = 0; h < NPL; ++h) {
                            sm[h] = 0u;
                            len[h] = 0;
                        }
                    }
                }
                if (nc + ncell > CCAP || nb + tot > BCAP || nr + nrange > RCAP) send(0);
                Packet& k = s.pk[sent & 1];
                int rat = nr;
#pragma unroll
                for (int h = 0; h < NPL; ++h) rat += __popc(sm[h] & lt);
#pragma unroll
                for (int h = 0; h < NPL; ++h) {
                    if (kind[h] == kCell) k.cell[nc + __popc(cm[h] & lt)] = a0[h];
                    nc += __popc(cm[h]);
                    if (len[h]) {  // a lane's ranges follow one another: numbered in order of position
                        const int at = nb + off;
                        k.base[rat++] = a0[h] - static_cast<uint32_t>(at);
                        atomicOr(&k.starts[at >> 5], 1u << (at & 31));
                        off += len[h];
                    }
                    nr += __popc(sm[h]);
                }
                nb += tot;
                // The other ranges (coincident bodies), split where a packet is full.
#pragma unroll
                for (int h = 0; h < NPL; ++h)
                    for (unsigned lm = rm[h] & ~sm[h]; lm; lm &= lm - 1u) {
                        const int sl = __ffs(lm) - 1;
                        const uint32_t lo = __shfl_sync(0xffffffffu, a0[h], sl), cnt = __shfl_sync(0xffffffffu, a1[h], sl);
                        for (uint32_t q = 0; q < cnt;) {
                            if (nb == BCAP || nr == RCAP) send(0);
                            const uint32_t take = min(cnt - q, static_cast<uint32_t>(BCAP - nb));
                            if (lane == 0) {
                                Packet& kk = s.pk[sent & 1];
                                kk.base[nr] = lo + q - static_cast<uint32_t>(nb);
                                atomicOr(&kk.starts[nb >> 5], 1u << (nb & 31));
                            }
                            ++nr;
                            nb += static_cast<int>(take);
                            q += take;
                        }
                    }
                __syncwarp();
            }
            if (fault && lane == 0) atomicOr(w.err, fault);
            if (plo + PASS >= gr.y && lane == 0) g_next = gridDim.x + atomicAdd(w.group_ctr, 1u);
            send(fault ? kLast | kAbort : kLast);
            inter_b += static_cast<unsigned long long>(list_len - cells_len - self) * static_cast<unsigned long long>(np);
            inter_c += static_cast<unsigned long long>(cells_len) * static_cast<unsigned long long>(np);
        }
        g = __shfl_sync(0xffffffffu, g_next, 0);
        if (g == 0xffffffffu) {  // the group's last pass was skipped
            if (lane == 0) g = gridDim.x + atomicAdd(w.group_ctr, 1u);
            g = __shfl_sync(0xffffffffu, g, 0);
        }
    }
    send(kEnd);
    if (sent >= 2) bar_sync(kBarEmpty + (sent & 1), WBS);  // the other slot's last packet
    if (lane == 0) {
        if (inter_b) atomicAdd(w.inter, inter_b);
        if (inter_c) atomicAdd(w.inter + 1, inter_c);
    }
    if (w.report && lane == 0) {
        __threadfence();
        if (atomicAdd(w.done, 1u) == gridDim.x - 1u) {  // every list warp has taken its last group
            unsigned long long* inter = reinterpret_cast<unsigned long long*>(w.report + 16);
            inter[0] = atomicExch(w.inter, 0ull);
            inter[1] = atomicExch(w.inter + 1, 0ull);
            for (int k = 0; k < 8; ++k) w.report[64 + k] = w.counts[k];
            w.report[0] = atomicOr(w.err, 0u);
            *w.group_ctr = 0u;
            *w.done = 0u;
            __threadfence_system();
        }
    }
}

// ---- the evaluating warps --------------------------------------------------------------------------
template <bool POT, bool EPS0, bool LET>
__device__ __forceinline__ void evaluate(const WalkArgs& w, WalkSmem& s) {
    const int tid = threadIdx.x;
    Lane l;
    int Lp = 1, slot = 0;
    if (POT)
        for (int i = tid; i < PASS; i += EVAL) s.kself[i] = 0u;
    for (unsigned seq = 1;; ++seq) {  // packet number; its slot is (seq - 1) & 1
        const int sl = (seq - 1) & 1;
        bar_sync(kBarFull + sl, WBS);
        const Packet& k = s.pk[sl];
        const unsigned flags = k.flags;
        if (flags & kEnd) break;
        const float4 o = k.centre;
        const uint32_t plo = k.plo, list_len = k.list_len;
        const int np = static_cast<int>(k.np), nc = k.nc, nb = k.nb;
        if (flags & kFirst) {
            // Entry partitions: P of Lp lanes each; slot, slot + Lp, ... are the lane's bodies.
            Lp = (np + IPT - 1) / IPT;
            l.P = EVAL / Lp;
            l.part = tid / Lp;
            slot = tid - l.part * Lp;
            if (l.part >= l.P) l.part = CCAP + BCAP;  // idle
#pragma unroll
            for (int u = 0; u < IPT; ++u) {
                const int i = min(slot + Lp * u, np - 1);
                const float4 h = w.hm[plo + i], lo = w.lo[plo + i];
                l.X[u] = f2_bcast((h.x - o.x) + lo.x);
                l.Y[u] = f2_bcast((h.y - o.y) + lo.y);
                l.Z[u] = f2_bcast((h.z - o.z) + lo.z);
#pragma unroll
                for (int f = 0; f < 8; ++f) s.ks[u][f][tid] = 0.f;
            }
        }
        const int cpairs = (nc + 1) >> 1, bpairs = (nb + 1) >> 1;
        for (int q = tid; q < cpairs; q += EVAL) {
            const uint2 id = *reinterpret_cast<const uint2*>(&k.cell[2 * q]);
            const NodeCell a = load_cell<LET>(w, id.x);
            NodeCell b;
            if (2 * q + 1 < nc) b = load_cell<LET>(w, id.y);
            else {
                b.com = make_float4(kFar, kFar, kFar, 0.f);
                b.lo = b.q0 = b.q1 = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            s.cell[q][0] = make_float4((a.com.x - o.x) + a.lo.x, (b.com.x - o.x) + b.lo.x, (a.com.y - o.y) + a.lo.y,
                                       (b.com.y - o.y) + b.lo.y);
            s.cell[q][1] = make_float4((a.com.z - o.z) + a.lo.z, (b.com.z - o.z) + b.lo.z, a.com.w, b.com.w);
            s.cell[q][2] = make_float4(-a.q0.x, -b.q0.x, -a.q0.y, -b.q0.y);
            s.cell[q][3] = make_float4(-a.q0.z, -b.q0.z, -a.q0.w, -b.q0.w);
            s.cell[q][4] = make_float4(-a.q1.x, -b.q1.x, -a.q1.y, -b.q1.y);
        }
        for (int q = tid; q < bpairs; q += EVAL) {
            const int p = 2 * q;
            const uint32_t st = k.starts[p >> 5];
            const int r0 = k.before[p >> 5] + __popc(st & (0xffffffffu >> (31 - (p & 31))));
            const int r1 = r0 + static_cast<int>((st >> ((p + 1) & 31)) & 1u);
            const uint2 id = make_uint2(k.base[r0] + static_cast<uint32_t>(p), k.base[r1] + static_cast<uint32_t>(p + 1));
            float4 h0, l0, h1 = make_float4(kFar, kFar, kFar, 0.f), l1 = make_float4(0.f, 0.f, 0.f, 0.f);
            load_body<LET>(w, id.x, h0, l0);
            if (2 * q + 1 < nb) load_body<LET>(w, id.y, h1, l1);
            if (POT) {
                if (id.x - plo < static_cast<uint32_t>(np)) s.kself[id.x - plo] = seq << 10 | static_cast<uint32_t>(2 * q);
                if (2 * q + 1 < nb && id.y - plo < static_cast<uint32_t>(np))
                    s.kself[id.y - plo] = seq << 10 | static_cast<uint32_t>(2 * q + 1);
            }
            s.body[q][0] = make_float4((h0.x - o.x) + l0.x, (h1.x - o.x) + l1.x, (h0.y - o.y) + l0.y, (h1.y - o.y) + l1.y);
            s.body[q][1] = make_float4((h0.z - o.z) + l0.z, (h1.z - o.z) + l1.z, h0.w, h1.w);
        }
        __syncwarp();
        bar_arrive(kBarEmpty + sl, WBS);  // the packet is read
        bar_sync(kBarEval, EVAL);         // the chunk is written
        Sums a;
        auto clear = [&] {
#pragma unroll
            for (int u = 0; u < IPT; ++u) a.x[u] = a.y[u] = a.z[u] = a.p[u] = 0ull;
        };
        auto merge = [&] {
#pragma unroll
            for (int u = 0; u < IPT; ++u) {
                const float v[4] = {f2_sum(a.x[u]), f2_sum(a.y[u]), f2_sum(a.z[u]), POT ? f2_sum(a.p[u]) : 0.f};
#pragma unroll
                for (int f = 0; f < (POT ? 4 : 3); ++f) kahan_add(s.ks[u][f][tid], s.ks[u][4 + f][tid], v[f]);
            }
        };
        const f2x E2 = f2_bcast(o.w);
        clear();
        eval_cells<POT, EPS0>(s, cpairs, l, a, E2);
        if (bpairs) {
            int kself[IPT];
#pragma unroll
            for (int u = 0; u < IPT; ++u) {
                const int i = slot + Lp * u;
                const uint32_t v = POT && i < np ? s.kself[i] : 0u;
                kself[u] = v >> 10 == (seq & 0x3fffffu) ? static_cast<int>(v & 1023u) : -2;
            }
            const int step = MERGE * l.P;
            int b0 = 0, b1 = max(0, min(bpairs, step - cpairs));  // what the cells leave of the first sum
            for (;;) {
                eval_bodies<POT, EPS0>(s, b0, b1, l, a, kself, E2);
                if (b1 >= bpairs) break;
                merge();
                clear();
                b0 = b1;
                b1 = min(bpairs, b0 + step);
            }
        }
        merge();
        __syncwarp();
        bar_sync(kBarEval, EVAL);  // the chunk is read
        if (!(flags & kLast)) continue;
        // ---- the partitions' sums, in partition order
        float4* red = &s.body[0][0];  // [u][thread]
#pragma unroll
        for (int u = 0; u < IPT; ++u)
            red[u * EVAL + tid] = make_float4(s.ks[u][0][tid] - s.ks[u][4][tid], s.ks[u][1][tid] - s.ks[u][5][tid],
                                              s.ks[u][2][tid] - s.ks[u][6][tid],
                                              POT ? s.ks[u][3][tid] - s.ks[u][7][tid] : 0.f);
        bar_sync(kBarEval, EVAL);
        for (int k = flags & kAbort ? np : tid; k < np; k += EVAL) {
            const int u = k / Lp, sb = k - u * Lp;
            float f[4] = {0.f, 0.f, 0.f, 0.f}, c[4] = {0.f, 0.f, 0.f, 0.f};
            for (int p = 0; p < l.P; ++p) {
                const float4 v = red[u * EVAL + p * Lp + sb];
                kahan_add(f[0], c[0], v.x);
                kahan_add(f[1], c[1], v.y);
                kahan_add(f[2], c[2], v.z);
                if (POT) kahan_add(f[3], c[3], v.w);
            }
            const uint32_t i = plo + k;
            const float4 a = make_float4(w.G * (f[0] - c[0]), w.G * (f[1] - c[1]), w.G * (f[2] - c[2]),
                                         POT ? -w.G * (f[3] - c[3]) : 0.f);
            if (w.accumulate) {
                const float4 v = w.acc[i];
                w.acc[i] = make_float4(v.x + a.x, v.y + a.y, v.z + a.z, v.w + a.w);
                w.cost[i] += static_cast<float>(list_len);
            } else {
                w.acc[i] = a;
                w.cost[i] = static_cast<float>(list_len - (w.local ? 1u : 0u));
            }
        }
        __syncwarp();
        bar_sync(kBarEval, EVAL);
    }
}

template <bool POT, bool EPS0, bool LET>
__global__ void __launch_bounds__(WBS, MINB) k_walk(WalkArgs w) {
    __shared__ WalkSmem s;
    if (threadIdx.x >= EVAL) build_lists<LET>(w, s);
    else evaluate<POT, EPS0, LET>(w, s);
}

template <bool POT, bool EPS0, bool LET>
void launch_walk_as(Engine& e, WalkArgs& w) {
    static int per_sm = 0;
    if (!per_sm) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_walk<POT, EPS0, LET>, WBS, 0) != cudaSuccess) {
            cudaGetLastError();
            per_sm = 1;
        }
        if (per_sm < 1) per_sm = 1;
    }
    const int blocks = per_sm * e.sms;
    e.walk_stack.reserve(static_cast<size_t>(blocks) * SCAP * sizeof(uint2));
    w.stack = e.walk_stack.as<uint2>();
    k_walk<POT, EPS0, LET><<<blocks, WBS, 0, e.stream>>>(w);
    LG_LAUNCHED();
    ++e.launches;
}

void launch_walk(Engine& e, WalkArgs& w, bool potential, bool eps0) {
    const bool let = w.let.ntrees > 0;
    if (potential) {
        if (eps0) let ? launch_walk_as<true, true, true>(e, w) : launch_walk_as<true, true, false>(e, w);
        else let ? launch_walk_as<true, false, true>(e, w) : launch_walk_as<true, false, false>(e, w);
    } else {
        if (eps0) let ? launch_walk_as<false, true, true>(e, w) : launch_walk_as<false, true, false>(e, w);
        else let ? launch_walk_as<false, false, true>(e, w) : launch_walk_as<false, false, false>(e, w);
    }
}

}  // namespace

void tree_walk_remote_blocks(Engine& e, float G, float e2, bool potential, bool eps0, const LetView& let,
                             const TreeView& blocks) {
    WalkArgs w{};
    w.tv = blocks;
    BodyArrays b = e.bodies(e.cur);
    w.hm = b.hm;
    w.lo = b.lo;
    w.acc = e.acc.as<float4>();
    w.cost = b.cost;
    w.group_ctr = reinterpret_cast<unsigned*>(e.small.as<char>() + 36);
    w.inter = e.inter_counter();
    w.err = e.err_word();
    w.G = G;
    w.e2 = e2;
    w.let = let;
    w.local = 0;
    w.accumulate = 1;
    launch_walk(e, w, potential, eps0);
}

void tree_walk(Engine& e, float G, float e2, bool potential, bool eps0, const uint32_t* sys, const float* e2_sys,
               const LetView* let, unsigned* report) {
    WalkArgs w{};
    w.report = report;
    w.done = e.small.as<unsigned>() + 13;
    w.counts = tree_counts_device(e);
    w.sys = sys;
    w.e2_sys = e2_sys;
    if (let) w.let = *let;
    w.local = 1;
    w.accumulate = 0;
    if (e.walk_kmin >= 0) {
        w.level = e.bodies(e.cur).level;
        w.kmin = e.walk_kmin;
    }
    w.tv = tree_view(e);
    BodyArrays b = e.bodies(e.cur);
    w.hm = b.hm;
    w.lo = b.lo;
    w.acc = e.acc.as<float4>();
    w.cost = b.cost;
    w.group_ctr = reinterpret_cast<unsigned*>(e.small.as<char>() + 32);
    w.inter = e.inter_counter();
    w.err = e.err_word();
    w.G = G;
    w.e2 = e2;
    launch_walk(e, w, potential, eps0);
}

}  // namespace lg
