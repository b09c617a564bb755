// Vector-Jacobian product of the tree forces (the adjoint's tree step). No counterpart in the
// reference.
//
// The forces of a tree step are a_i = G [sum over the cells c of i's group list A_c(d) + sum over
// the bodies j of its body ranges m_j K(d)], d = (cell centre of mass or x_j) - x_i,
//   A_c(d) = M d / r^3 - Q d / r^5 + 5/2 (d.Q.d) d / r^7,  K(d) = d / r^3,  r^2 = |d|^2 + eps^2,
// with the lists fixed by the tree (walk.cu, the reference's opening rule) and the cell moments
// M = sum m_b, com = sum m_b x_b / M, Q = sum m_b (3 e e^T - |e|^2 I), e = x_b - com, functions of
// the bodies below the cell. With the lists held fixed ("frozen": the backward pass rebuilds the
// same tree from bit-identical positions), this file computes, for weights w_i,
//   g = d(sum_i w_i . a_i / G) / d(x, m).
//
// Per (i, entry) with u = w_i . d, q = d.Q.d, Qd = Q d, Qw = Q w_i:
//   body j:  gd = m_j (w_i / r^3 - 3 u d / r^5);  dm_j += u / r^3
//   cell c:  gd = (M/r^3 + 5/2 q/r^7) w_i + (-3 M u/r^5 + 5 (w_i.Qd)/r^7 - 35/2 q u/r^9) d
//                 - Qw/r^5 + 5 u Qd / r^7
//            dM_c += u / r^3;  dQ_kl += -(w_k d_l + w_l d_k)/r^5 + 5 u d_k d_l / r^7 (k != l),
//            dQ_kk += -w_k d_k / r^5 + 5/2 u d_k^2 / r^7
//   and dx_i -= gd, dX_entry += gd (X = x_j or the cell's centre of mass).
// The self pair (j == i) is skipped: d is identically zero, so it has no derivative.
// The cell adjoints (dM, dcom, dQ) then reach the bodies through the moment definitions
// (k_leaf_field, k_body_field): for every ancestor cell c of body b, with e = x_b - com_c,
//   dx_b += (m_b/M) dcom + m_b [6 dQ_diag e - 2 tr(dQ) e + 3 offdiag terms]
//   dm_b += dM + e . dcom / M + sum_kl dQ_kl (3 e_k e_l - |e|^2 delta_kl)  (stored components)
// (the derivative of Q through com vanishes because sum_b m_b e_b = 0).
//
// Kernel shape: the force walk's (walk.cu): a block takes a group, its list warp builds the list in
// packets (walk_common.cuh), its four other warps evaluate them. A warp takes 32 entries of a packet
// at a time, one per lane, and runs over the group's i-bodies, two per packed f32x2 instruction. What
// a pair gives the entry is summed in registers and goes to FP64 adjoint arrays with atomics; what it
// gives the i-body, the same vector with the other sign, is laid out in shared memory, 32 entries by
// TP pairs of i-bodies, and summed there by lanes that hold i-bodies, with Kahan sums over the tiles.
// Every pair is so evaluated once for both sides: 86 packed instructions for two cell pairs and 27 for
// two body pairs, where an evaluation for each side (lanes over i-bodies, then over entries) took 153
// and 40; the tile costs a tenth of them. One pass over the 200 000-body collision: 2.25 -> 0.91 ms against
// one warp per group (which ended on the few largest groups, with the SMs idle for a third of it). The
// FMA pipe is now 60% busy: three blocks of 126 registers per SM leave it waiting for latencies.
#include "engine.cuh"
#include "walk_common.cuh"

namespace lg {

namespace {

using namespace walk;

constexpr int NADJ = 10;  // per node: dM, dcom (3), dQ (xx, xy, xz, yy, yz, zz)
constexpr int EWARPS = EVAL / 32;
constexpr int TP = 16;    // pairs of i-bodies per tile
constexpr int VMINB = 3;  // resident blocks per SM: shared memory holds three

struct __align__(16) VjpSmem {
    Packet pk[2];
    uint2 stk[SSTK];
    f2x i[PASS / 2][6];                 // pairs of i-bodies: x, y, z and their weights
    f2x tile[EWARPS][3][TP][33];        // per warp: a pair of i-bodies' terms by entry
    f2x ks[EWARPS][3][2][PASS / 2];     // per warp: Kahan sums of the i side and their compensations
};

struct VjpArgs : ListArgs {
    const float4* hm;
    const float4* lo;
    const float4* w;
    double* gx;
    double* gy;
    double* gz;
    double* gm;
    double* nadj;  // NADJ arrays of T doubles
};

template <bool EPS0>
__device__ __forceinline__ f2x inv_r2(f2x r2) {
    float lo, hi;
    f2_unpack(r2, lo, hi);
    float a = rsqrt_mufu(lo), b = rsqrt_mufu(hi);
    if (EPS0) {
        a = lo > 0.f ? a : 0.f;
        b = hi > 0.f ? b : 0.f;
    }
    return f2_pack(a, b);
}

// i-bodies 2q and 2q + 1 of the pass.
struct IPair {
    f2x x, y, z, wx, wy, wz;
};

__device__ __forceinline__ IPair load_pair(const VjpSmem& s, int q) {
    const ulonglong2* p = reinterpret_cast<const ulonglong2*>(s.i[q]);
    const ulonglong2 a = p[0], b = p[1], c = p[2];
    return IPair{a.x, a.y, b.x, b.y, c.x, c.y};
}

// Adds the tile's terms of pairs q0 .. q0 + TP to the warp's Kahan sums: each half of the warp sums 16
// entries of a pair, the halves are added.
__device__ __forceinline__ void sum_tile(VjpSmem& s, int warp, int q0, int pairs) {
    const int lane = threadIdx.x & 31, p = lane & (TP - 1), e0 = lane & 16;
    static_assert(TP == 16, "two halves of a warp");
    __syncwarp();
    f2x t[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const f2x* v = &s.tile[warp][c][p][e0];
        f2x a = v[0], b = v[1];
#pragma unroll
        for (int e = 2; e < 16; e += 2) {
            a = f2_add(a, v[e]);
            b = f2_add(b, v[e + 1]);
        }
        t[c] = f2_add(a, b);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) t[c] = f2_add(t[c], __shfl_xor_sync(0xffffffffu, t[c], 16));
    if (lane < TP && q0 + p < pairs) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            f2x& sum = s.ks[warp][c][0][q0 + p];
            f2x& comp = s.ks[warp][c][1][q0 + p];
            const f2x y = f2_sub(t[c], comp), n = f2_add(sum, y);
            comp = f2_sub(f2_sub(n, sum), y);
            sum = n;
        }
    }
    __syncwarp();
}

// 32 cells of the packet from e0 on against the pass's i-bodies. With u = w.d, per pair
//   A = M / r^3 + 5/2 q / r^7;  B = -3 M u / r^5 + 5 (w.Qd) / r^7 - 35/2 q u / r^9;  D = 5 u / r^7
//   gd = A w + B d + D Qd - Qw / r^5
//   dQ_kk += d_k (D/2 d_k + p_k),  dQ_kl += d_l (D d_k + p_k) + p_l d_k  (k < l),  p = -w / r^5.
// Lanes past the packet's cells hold a copy of the last one with no moments, whose terms are zero.
template <bool EPS0>
__device__ __forceinline__ void vjp_cells(const VjpArgs& a, VjpSmem& s, const Packet& k, int warp, int e0, int pairs) {
    const int lane = threadIdx.x & 31, nc = k.nc;
    const float4 o = k.centre;
    const f2x E2 = f2_bcast(a.e2), C05 = f2_bcast(0.5f), C25 = f2_bcast(2.5f), C5 = f2_bcast(5.f);
    const f2x CN1 = f2_bcast(-1.f), CN3 = f2_bcast(-3.f), CN175 = f2_bcast(-17.5f);
    const bool on = e0 + lane < nc;
    const uint32_t nd = k.cell[min(e0 + lane, nc - 1)];
    const NodeCell r = a.tv.nd_cell[nd];
    const float z = on ? 1.f : 0.f;
    const f2x X = f2_bcast((r.com.x - o.x) + r.lo.x), Y = f2_bcast((r.com.y - o.y) + r.lo.y),
              Z = f2_bcast((r.com.z - o.z) + r.lo.z), M = f2_bcast(z * r.com.w);
    const f2x qxx = f2_bcast(z * r.q0.x), qxy = f2_bcast(z * r.q0.y), qxz = f2_bcast(z * r.q0.z);
    const f2x qyy = f2_bcast(z * r.q0.w), qyz = f2_bcast(z * r.q1.x), qzz = f2_bcast(z * r.q1.y);
    f2x G[NADJ];
#pragma unroll
    for (int f = 0; f < NADJ; ++f) G[f] = f2_bcast(0.f);
    for (int q0 = 0; q0 < pairs; q0 += TP) {
        const int q1 = min(pairs, q0 + TP);
#pragma unroll 1
        for (int q = q0; q < q1; ++q) {
            const IPair i = load_pair(s, q);
            const f2x dx = f2_sub(X, i.x), dy = f2_sub(Y, i.y), dz = f2_sub(Z, i.z);
            const f2x inv = inv_r2<EPS0>(f2_fma(dx, dx, f2_fma(dy, dy, f2_fma(dz, dz, E2))));
            const f2x inv2 = f2_mul(inv, inv), inv3 = f2_mul(inv, inv2), inv5 = f2_mul(inv3, inv2);
            const f2x inv7 = f2_mul(inv5, inv2), inv9 = f2_mul(inv7, inv2);
            const f2x qx = f2_fma(qxx, dx, f2_fma(qxy, dy, f2_mul(qxz, dz)));
            const f2x qy = f2_fma(qxy, dx, f2_fma(qyy, dy, f2_mul(qyz, dz)));
            const f2x qz = f2_fma(qxz, dx, f2_fma(qyz, dy, f2_mul(qzz, dz)));
            const f2x qd = f2_fma(dx, qx, f2_fma(dy, qy, f2_mul(dz, qz)));
            const f2x u = f2_fma(i.wx, dx, f2_fma(i.wy, dy, f2_mul(i.wz, dz)));
            const f2x qwx = f2_fma(qxx, i.wx, f2_fma(qxy, i.wy, f2_mul(qxz, i.wz)));
            const f2x qwy = f2_fma(qxy, i.wx, f2_fma(qyy, i.wy, f2_mul(qyz, i.wz)));
            const f2x qwz = f2_fma(qxz, i.wx, f2_fma(qyz, i.wy, f2_mul(qzz, i.wz)));
            const f2x wqd = f2_fma(i.wx, qx, f2_fma(i.wy, qy, f2_mul(i.wz, qz)));
            const f2x A = f2_fma(M, inv3, f2_mul(f2_mul(C25, qd), inv7));
            const f2x B = f2_fma(f2_mul(CN3, f2_mul(M, u)), inv5,
                                 f2_fma(f2_mul(C5, wqd), inv7, f2_mul(f2_mul(CN175, f2_mul(qd, u)), inv9)));
            const f2x D = f2_mul(f2_mul(C5, u), inv7);
            const f2x n5 = f2_mul(CN1, inv5);
            const f2x gx = f2_fma(A, i.wx, f2_fma(B, dx, f2_fma(D, qx, f2_mul(qwx, n5))));
            const f2x gy = f2_fma(A, i.wy, f2_fma(B, dy, f2_fma(D, qy, f2_mul(qwy, n5))));
            const f2x gz = f2_fma(A, i.wz, f2_fma(B, dz, f2_fma(D, qz, f2_mul(qwz, n5))));
            s.tile[warp][0][q - q0][lane] = gx;
            s.tile[warp][1][q - q0][lane] = gy;
            s.tile[warp][2][q - q0][lane] = gz;
            G[0] = f2_fma(u, inv3, G[0]);
            G[1] = f2_add(G[1], gx);
            G[2] = f2_add(G[2], gy);
            G[3] = f2_add(G[3], gz);
            const f2x E = f2_mul(C05, D);
            const f2x px = f2_mul(i.wx, n5), py = f2_mul(i.wy, n5), pz = f2_mul(i.wz, n5);
            const f2x Dx = f2_fma(D, dx, px), Dy = f2_fma(D, dy, py);
            G[4] = f2_fma(f2_fma(E, dx, px), dx, G[4]);
            G[5] = f2_fma(Dx, dy, f2_fma(py, dx, G[5]));
            G[6] = f2_fma(Dx, dz, f2_fma(pz, dx, G[6]));
            G[7] = f2_fma(f2_fma(E, dy, py), dy, G[7]);
            G[8] = f2_fma(Dy, dz, f2_fma(pz, dy, G[8]));
            G[9] = f2_fma(f2_fma(E, dz, pz), dz, G[9]);
        }
        sum_tile(s, warp, q0, pairs);
    }
    if (!on) return;
    const size_t T = a.tv.T;
#pragma unroll
    for (int f = 0; f < NADJ; ++f) {
        const float g = f2_sum(G[f]);
        if (g != 0.f) atomicAdd(a.nadj + f * T + nd, static_cast<double>(g));
    }
}

// 32 NE bodies of the packet from e0 on, NE per lane: per pair e = w / r^3 - 3 u d / r^5, dx_j += m_j e,
// dm_j += u / r^3 and dx_i -= m_j e. The self pair is taken out by zeroing its half of the weight. Two
// per lane share the loads of the i-bodies and the tile, whose shared-memory traffic (16 cycles a step
// of each of four warps) would otherwise take longer than the 27 packed instructions of a pair.
template <int NE, bool EPS0>
__device__ __forceinline__ void vjp_bodies(const VjpArgs& a, VjpSmem& s, const Packet& k, int warp, int e0, int pairs) {
    const int lane = threadIdx.x & 31, nb = k.nb;
    const float4 o = k.centre;
    const f2x E2 = f2_bcast(a.e2), CN3 = f2_bcast(-3.f);
    uint32_t j[NE];
    int js[NE];
    float mj[NE];
    f2x X[NE], Y[NE], Z[NE], M[NE], GX[NE], GY[NE], GZ[NE], GM[NE];
#pragma unroll
    for (int v = 0; v < NE; ++v) {
        const int p = min(e0 + 32 * v + lane, nb - 1);
        j[v] = k.base[range_of(k, p)] + static_cast<uint32_t>(p);
        const float4 h = a.hm[j[v]], l = a.lo[j[v]];
        js[v] = j[v] - k.plo < k.np ? static_cast<int>(j[v] - k.plo) : -2;
        mj[v] = e0 + 32 * v + lane < nb ? h.w : 0.f;
        X[v] = f2_bcast((h.x - o.x) + l.x);
        Y[v] = f2_bcast((h.y - o.y) + l.y);
        Z[v] = f2_bcast((h.z - o.z) + l.z);
        M[v] = f2_bcast(mj[v]);
        GX[v] = GY[v] = GZ[v] = GM[v] = f2_bcast(0.f);
    }
    for (int q0 = 0; q0 < pairs; q0 += TP) {
        const int q1 = min(pairs, q0 + TP);
#pragma unroll 1
        for (int q = q0; q < q1; ++q) {
            const IPair ip = load_pair(s, q);
            f2x tx = 0ull, ty = 0ull, tz = 0ull;
#pragma unroll
            for (int v = 0; v < NE; ++v) {
                IPair i = ip;
                const unsigned off = static_cast<unsigned>(js[v] - 2 * q);
                if (off <= 1u) {
                    const f2x msk = off == 0 ? f2_pack(0.f, 1.f) : f2_pack(1.f, 0.f);
                    i.wx = f2_mul(i.wx, msk);
                    i.wy = f2_mul(i.wy, msk);
                    i.wz = f2_mul(i.wz, msk);
                }
                const f2x dx = f2_sub(X[v], i.x), dy = f2_sub(Y[v], i.y), dz = f2_sub(Z[v], i.z);
                const f2x inv = inv_r2<EPS0>(f2_fma(dx, dx, f2_fma(dy, dy, f2_fma(dz, dz, E2))));
                const f2x inv2 = f2_mul(inv, inv), inv3 = f2_mul(inv, inv2), inv5 = f2_mul(inv3, inv2);
                const f2x u = f2_fma(i.wx, dx, f2_fma(i.wy, dy, f2_mul(i.wz, dz)));
                const f2x t = f2_mul(f2_mul(CN3, u), inv5);
                const f2x ex = f2_fma(i.wx, inv3, f2_mul(t, dx)), ey = f2_fma(i.wy, inv3, f2_mul(t, dy)),
                          ez = f2_fma(i.wz, inv3, f2_mul(t, dz));
                tx = v ? f2_fma(M[v], ex, tx) : f2_mul(M[v], ex);
                ty = v ? f2_fma(M[v], ey, ty) : f2_mul(M[v], ey);
                tz = v ? f2_fma(M[v], ez, tz) : f2_mul(M[v], ez);
                GX[v] = f2_add(GX[v], ex);
                GY[v] = f2_add(GY[v], ey);
                GZ[v] = f2_add(GZ[v], ez);
                GM[v] = f2_fma(u, inv3, GM[v]);
            }
            s.tile[warp][0][q - q0][lane] = tx;
            s.tile[warp][1][q - q0][lane] = ty;
            s.tile[warp][2][q - q0][lane] = tz;
        }
        sum_tile(s, warp, q0, pairs);
    }
#pragma unroll
    for (int v = 0; v < NE; ++v) {
        if (e0 + 32 * v + lane >= nb) continue;
        atomicAdd(a.gx + j[v], static_cast<double>(mj[v] * f2_sum(GX[v])));
        atomicAdd(a.gy + j[v], static_cast<double>(mj[v] * f2_sum(GY[v])));
        atomicAdd(a.gz + j[v], static_cast<double>(mj[v] * f2_sum(GZ[v])));
        atomicAdd(a.gm + j[v], static_cast<double>(f2_sum(GM[v])));
    }
}

// The evaluating warps. They take a packet's cells 32 at a time in turn, then its bodies, 64 at a time:
// as 32 cells cost what two times 64 bodies do, the warps that had one turn of cells less begin with
// two of bodies.
template <bool EPS0>
__device__ __forceinline__ void vjp_evaluate(const VjpArgs& a, VjpSmem& s) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (unsigned seq = 0;; ++seq) {
        const int sl = seq & 1;
        bar_sync(kBarFull + sl, WBS);
        const Packet& k = s.pk[sl];
        const unsigned flags = k.flags;
        if (flags & kEnd) break;
        const float4 o = k.centre;
        const uint32_t plo = k.plo;
        const int np = static_cast<int>(k.np), pairs = (np + 1) >> 1;
        if (flags & kFirst) {
            bar_sync(kBarEval, EVAL);  // the last group's sums are read
            if (tid < 2 * pairs) {     // an odd count is padded with a body of no weight
                const uint32_t i = plo + static_cast<uint32_t>(min(tid, np - 1));
                const float4 h = a.hm[i], l = a.lo[i], w = a.w[i];
                const float z = tid < np ? 1.f : 0.f;
                float* f = reinterpret_cast<float*>(s.i[tid >> 1]) + (tid & 1);
                f[0] = (h.x - o.x) + l.x;
                f[2] = (h.y - o.y) + l.y;
                f[4] = (h.z - o.z) + l.z;
                f[6] = z * w.x;
                f[8] = z * w.y;
                f[10] = z * w.z;
            }
            for (int q = lane; q < PASS / 2; q += 32)
#pragma unroll
                for (int c = 0; c < 3; ++c) s.ks[warp][c][0][q] = s.ks[warp][c][1][q] = f2_bcast(0.f);
            __syncwarp();
            bar_sync(kBarEval, EVAL);
        }
        const int tc = (k.nc + 31) >> 5, tb = (k.nb + 63) >> 6;
        for (int t = warp; t < tc; t += EWARPS) vjp_cells<EPS0>(a, s, k, warp, 32 * t, pairs);
        const int ahead = tc % EWARPS, behind = EWARPS - ahead;
        const int lead = ahead ? 2 * behind : 0;  // turns of bodies for the warps behind
        for (int t = 0; t < tb; ++t) {
            const int who = t < lead ? ahead + t % behind : (t - lead) % EWARPS;
            if (who != warp) continue;
            if (k.nb - 64 * t > 32) vjp_bodies<2, EPS0>(a, s, k, warp, 64 * t, pairs);
            else vjp_bodies<1, EPS0>(a, s, k, warp, 64 * t, pairs);
        }
        __syncwarp();
        bar_arrive(kBarEmpty + sl, WBS);  // the packet is read
        if (!(flags & kLast)) continue;
        bar_sync(kBarEval, EVAL);  // every warp's sums are complete
        if (tid < np) {
            double g[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double v = 0;
#pragma unroll
                for (int e = 0; e < EWARPS; ++e) {
                    const float* f = reinterpret_cast<const float*>(s.ks[e][c][0]);
                    const float* r = reinterpret_cast<const float*>(s.ks[e][c][1]);
                    v += static_cast<double>(f[tid]) - static_cast<double>(r[tid]);
                }
                g[c] = v;
            }
            atomicAdd(a.gx + plo + tid, -g[0]);
            atomicAdd(a.gy + plo + tid, -g[1]);
            atomicAdd(a.gz + plo + tid, -g[2]);
        }
        __syncwarp();
    }
}

template <bool EPS0>
__global__ void __launch_bounds__(WBS, VMINB) k_walk_vjp(VjpArgs a) {
    extern __shared__ __align__(16) unsigned char raw[];
    VjpSmem& s = *reinterpret_cast<VjpSmem*>(raw);
    if (threadIdx.x >= EVAL) build_lists<false>(a, s);
    else vjp_evaluate<EPS0>(a, s);
}

// Cell adjoints to bodies through the moment definitions. What a cell gives a body at x is, for dm,
//   dM + p.e + 1/2 e.H e,  and for dx m times its gradient p + H e,
// with e = x - com, p = dcom / M, H_kk = 6 dQ_kk - 2 tr dQ, H_kl = 3 dQ_kl: a quadratic, and so is the
// sum over a leaf's ancestors. A thread per leaf sums it about the leaf's centre of mass, and the
// bodies evaluate their leaf's (FP64 both; the chain from every body cost 355 us a pass for the
// 200 000-body collision, the two kernels 60 and 20).
constexpr int NFIELD = 10;  // per leaf: the value, the gradient (3), H (xx, xy, xz, yy, yz, zz)

__device__ __forceinline__ void cell_centre(const NodeCell& c, double& x, double& y, double& z) {
    x = static_cast<double>(c.com.x) + c.lo.x;
    y = static_cast<double>(c.com.y) + c.lo.y;
    z = static_cast<double>(c.com.z) + c.lo.z;
}

__global__ void k_leaf_field(TreeView tv, const double* __restrict__ nadj, double* __restrict__ field, unsigned* err) {
    const size_t l = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x, T = tv.T, K = tv.K;
    if (l >= min(static_cast<size_t>(*tv.nleaves), K)) return;
    uint32_t node = tv.leaf_node[l];
    if (node >= T) {
        atomicOr(err, kErrNodeOverflow);
        return;
    }
    double x0, y0, z0;
    cell_centre(tv.nd_cell[node], x0, y0, z0);
    double A = 0, Bx = 0, By = 0, Bz = 0, Hxx = 0, Hxy = 0, Hxz = 0, Hyy = 0, Hyz = 0, Hzz = 0;
    for (int guard = 0; node < T && guard < 128; ++guard) {
        const double qxx = nadj[4 * T + node], qyy = nadj[7 * T + node], qzz = nadj[9 * T + node];
        const double hxy = 3 * nadj[5 * T + node], hxz = 3 * nadj[6 * T + node], hyz = 3 * nadj[8 * T + node];
        const double t2 = 2 * (qxx + qyy + qzz), hxx = 6 * qxx - t2, hyy = 6 * qyy - t2, hzz = 6 * qzz - t2;
        const NodeCell c = tv.nd_cell[node];
        double ex, ey, ez;
        cell_centre(c, ex, ey, ez);
        ex = x0 - ex;
        ey = y0 - ey;
        ez = z0 - ez;
        const double iM = c.com.w > 0 ? 1.0 / c.com.w : 0.0;
        const double px = nadj[T + node] * iM, py = nadj[2 * T + node] * iM, pz = nadj[3 * T + node] * iM;
        const double vx = hxx * ex + hxy * ey + hxz * ez, vy = hxy * ex + hyy * ey + hyz * ez,
                     vz = hxz * ex + hyz * ey + hzz * ez;
        A += nadj[node] + (px * ex + py * ey + pz * ez) + 0.5 * (vx * ex + vy * ey + vz * ez);
        Bx += px + vx;
        By += py + vy;
        Bz += pz + vz;
        Hxx += hxx;
        Hxy += hxy;
        Hxz += hxz;
        Hyy += hyy;
        Hyz += hyz;
        Hzz += hzz;
        node = tv.nd_parent[node];
    }
    const double f[NFIELD] = {A, Bx, By, Bz, Hxx, Hxy, Hxz, Hyy, Hyz, Hzz};
#pragma unroll
    for (int k = 0; k < NFIELD; ++k) field[k * K + l] = f[k];
}

__global__ void k_body_field(TreeView tv, const BodyArrays b, int n, const double* __restrict__ field, double* gx,
                             double* gy, double* gz, double* gm, unsigned* err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t K = tv.K;
    const uint32_t l = tv.body_leaf[i];
    if (l >= min(static_cast<size_t>(*tv.nleaves), K) || tv.leaf_node[l] >= tv.T) {
        atomicOr(err, kErrNodeOverflow);
        return;
    }
    double ex, ey, ez;
    cell_centre(tv.nd_cell[tv.leaf_node[l]], ex, ey, ez);
    ex = b.x[i] - ex;
    ey = b.y[i] - ey;
    ez = b.z[i] - ez;
    double f[NFIELD];
#pragma unroll
    for (int k = 0; k < NFIELD; ++k) f[k] = field[k * K + l];
    const double vx = f[4] * ex + f[5] * ey + f[6] * ez, vy = f[5] * ex + f[7] * ey + f[8] * ez,
                 vz = f[6] * ex + f[8] * ey + f[9] * ez;
    const double m = b.m[i];
    gx[i] += m * (f[1] + vx);
    gy[i] += m * (f[2] + vy);
    gz[i] += m * (f[3] + vz);
    gm[i] += f[0] + (f[1] * ex + f[2] * ey + f[3] * ez) + 0.5 * (vx * ex + vy * ey + vz * ez);
}

template <bool EPS0>
void launch_vjp(Engine& e, VjpArgs& a) {
    static int per_sm = 0;
    // On each launch: it holds for the current device only.
    LG_CK(cudaFuncSetAttribute(k_walk_vjp<EPS0>, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(VjpSmem)));
    if (!per_sm) {
        int fit = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_walk_vjp<EPS0>, WBS, sizeof(VjpSmem)) != cudaSuccess)
            cudaGetLastError();
        per_sm = std::max(fit, 1);
    }
    const int blocks = per_sm * e.sms;
    e.walk_stack.reserve(static_cast<size_t>(blocks) * SCAP * sizeof(uint2));
    a.stack = e.walk_stack.as<uint2>();
    k_walk_vjp<EPS0><<<blocks, WBS, sizeof(VjpSmem), e.stream>>>(a);
    LG_LAUNCHED();
    ++e.launches;
}

}  // namespace

void tree_walk_vjp(Engine& e, const float4* w, float e2, bool eps0, double* g) {
    const int n = e.n;
    if (n == 0) return;
    TreeView tv = tree_view(e);
    const size_t T = tv.T;
    e.vjp_scratch.reserve((T * NADJ + tv.K * NFIELD) * 8);
    double* nadj = e.vjp_scratch.as<double>();
    LG_CK(cudaMemsetAsync(nadj, 0, T * NADJ * 8, e.stream));
    LG_CK(cudaMemsetAsync(e.small.as<char>() + 40, 0, 4, e.stream));
    BodyArrays b = e.bodies(e.cur);
    VjpArgs a{};
    a.local = 1;
    a.tv = tv;
    a.hm = b.hm;
    a.lo = b.lo;
    a.w = w;
    a.gx = g;
    a.gy = g + n;
    a.gz = g + 2 * static_cast<size_t>(n);
    a.gm = g + 3 * static_cast<size_t>(n);
    a.nadj = nadj;
    a.group_ctr = reinterpret_cast<unsigned*>(e.small.as<char>() + 40);
    a.err = e.err_word();
    a.e2 = e2;
    if (eps0) launch_vjp<true>(e, a);
    else launch_vjp<false>(e, a);
    double* field = nadj + T * NADJ;
    k_leaf_field<<<static_cast<int>((tv.K + 63) / 64), 64, 0, e.stream>>>(tv, nadj, field, e.err_word());
    LG_LAUNCHED();
    k_body_field<<<(n + 255) / 256, 256, 0, e.stream>>>(tv, b, n, field, a.gx, a.gy, a.gz, a.gm, e.err_word());
    LG_LAUNCHED();
    e.launches += 2;
}

}  // namespace lg
