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

using namespace walk;

constexpr int MINB = 4;         // resident blocks per SM: 20 warps at 96 registers (5 at 72 spill)
constexpr int IPT = 2;          // i-bodies per lane
constexpr int BUNROLL = 3;      // body pairs evaluated together
constexpr int MERGE = 96;          // pairs a lane sums in plain FP32 before a compensated addition
static_assert(PASS <= EVAL * IPT, "a lane for every body");

struct __align__(16) WalkSmem {
    // Packed pairs: entry 2q in the even float of each two, entry 2q + 1 in the odd one.
    float4 cell[CCAP / 2][5];  // (x x y y)(z z m m)(xx xx xy xy)(xz xz yy yy)(yz yz zz zz), -Q
    float4 body[BCAP / 2][2];  // (x x y y)(z z m m)
    Packet pk[2];
    uint2 stk[SSTK];           // traversal stack: first child, children
    float ks[IPT][8][EVAL];    // per lane and i-body: Kahan sums x y z phi, their compensations
    uint32_t kself[PASS];      // with the potential: packet number << 10 | position of the i-body in the chunk
};

struct WalkArgs : ListArgs {
    const float4* hm;
    const float4* lo;
    float4* acc;
    float* cost;
    float G;
    int accumulate;  // adds to acc and cost instead of overwriting
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
            const int r0 = range_of(k, p);
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
