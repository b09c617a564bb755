// List building of the tree walk, shared by the force walk (walk.cu) and its vector-Jacobian product
// (walk_vjp.cu): a block's last warp builds the lists of the groups the block takes, by the reference
// CPU backend's opening rule (src/cpu_backend.cpp:816-838 build_list), and hands them in packets to
// the warps that evaluate them.
#pragma once

#include "engine.cuh"

namespace lg {
namespace walk {

constexpr int SMALL_LEAF = 4;   // src/cpu_backend.cpp:29
constexpr int SCAP = 16384;     // global traversal stack entries per list warp (overflow of the shared stack)
constexpr int SSTK = 256, SREFILL = 128;  // shared stack entries; entries fetched back at a time
constexpr int EVAL = 128;          // evaluating threads
constexpr int WBS = EVAL + 32;     // and the list warp
constexpr int PASS = 128;          // i-bodies per pass
constexpr int CCAP = 320;          // cells per packet
constexpr int BCAP = 768;          // bodies per packet
constexpr int RCAP = 256;          // body ranges per packet
constexpr int LEAF = 16;           // ranges up to this length are appended one per lane and node
constexpr int NPL = 2;             // nodes per lane and traversal round
constexpr int BWORDS = (BCAP + 31) / 32;
static_assert(CCAP % 2 == 0 && CCAP >= 32 * NPL, "cells: whole pairs, at least a round's");
static_assert(BCAP % 2 == 0 && RCAP >= 32 * NPL && BCAP <= 1024 && BWORDS <= 32, "bodies: whole pairs, at least a round's");

// List entries from a remote tree carry this bit (cell: node index; body range: first body).
constexpr uint32_t REMOTE = 0x80000000u;

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

// Number of the range that holds body p of the packet.
__device__ __forceinline__ int range_of(const Packet& k, int p) {
    return k.before[p >> 5] + __popc(k.starts[p >> 5] & (0xffffffffu >> (31 - (p & 31))));
}

struct ListArgs {
    TreeView tv;
    uint2* stack;  // SCAP entries per block
    unsigned* group_ctr;
    unsigned long long* inter;  // interactions with bodies, with cells; or null
    unsigned* err;
    // What the last block to finish hands to the host (see tree_walk), or null.
    unsigned* report;
    unsigned* done;
    const unsigned* counts;
    float e2;
    // Forest (ensemble) walk: body -> system (nullptr: one tree rooted at node 0) and the
    // per-system squared softening; system s's tree is rooted at node s.
    const uint32_t* sys;
    const float* e2_sys;
    // Remote trees walked after the local tree (or alone: local == 0, for the direct method's
    // blocks of consecutive bodies).
    LetView let;
    int local;
    // Block time steps: passes whose bodies all have level < kmin are skipped (level == nullptr: none).
    const uint8_t* level;
    int kmin;
};

__device__ __forceinline__ void bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Box distance squared, in the reference's fused float form.
__device__ __forceinline__ float box_d2(float4 com, float4 bc, float4 bh) {
    const float dx = fmaxf(__fsub_rn(fabsf(__fsub_rn(com.x, bc.x)), bh.x), 0.f);
    const float dy = fmaxf(__fsub_rn(fabsf(__fsub_rn(com.y, bc.y)), bh.y), 0.f);
    const float dz = fmaxf(__fsub_rn(fabsf(__fsub_rn(com.z, bc.z)), bh.z), 0.f);
    return __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
}

// What a lane's node turned out to be.
enum { kNone, kCell, kBodies, kChildren };

template <bool LET, class S>
__device__ __forceinline__ void build_lists(const ListArgs& w, S& s) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int team = lane >> 3;
    const uint32_t sub = lane & 7;
    uint2* gstk = w.stack + static_cast<size_t>(blockIdx.x) * SCAP;
    // No groups after a build in which a wait ran out: its nodes are not all there.
    const unsigned ran_out = *w.err & kErrWaitTimeout, groups = *w.tv.ngroups;
    const unsigned ngroups = ran_out ? 0u : groups;
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
        __syncwarp();  // the lanes' entries and start bits are there
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
                if (sp + npush > SSTK) {  // the shared part moves to the global part
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
                    const int k = min(SREFILL, gsp);
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
    if (w.inter && lane == 0) {
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

}  // namespace walk
}  // namespace lg
