// Channel-task passes of the flow right-hand side (sm_103a): level-synchronous
// adaptive quadrature.
//
// A pass is the set of channel tasks (channel X, kernel, w1, w2, w3) that one
// call of compute_dΓ_{1l,2l,ml}!/compute_Γ!/compute_Σ! fans out
// (src/Flow/compute.jl, SDE.jl).  Each task integrates its bubble over the
// 4*eval subdomains of integrate_log!/integrate_lin! (src/Flow/quadrature.jl:
// 84-139) plus two boundary nodes (src/Flow/flow_s.jl:37-38), and every
// subdomain runs the adaptive Simpson rule with Richardson extrapolation of
// simps! (quadrature.jl:27-81), whose depth varies by orders of magnitude
// between subdomains.  Instead of one CTA per task (whose slowest member sets
// the pass time), the subdomains of all tasks advance level by level:
//
//   wave 0   every subdomain evaluates its first five nodes (the 3-point and
//            the 5-point Simpson sums) and takes the first convergence test;
//   wave k   the 2^(k+1) new nodes of every subdomain still refining are cut
//            into chunks (cut_level); eval_kernel spreads the chunks over the
//            whole GPU and writes one partial node sum per chunk; decide_kernel sums a subdomain's partials in node order,
//            forms the next Simpson sum and the Richardson value, takes the
//            reference's test (||R - S|| < atol or relative < rtol, or
//            n > 2^20) and either stores the result or queues the next level;
//   reduce   sums each task's subdomain results in a fixed order and writes
//            the output slice (flow_s.jl:41-51).
//
// The reweighted nodes of residual! (quadrature.jl:2-24) are the previous
// level's new nodes, so their sum is carried from the last level instead of
// re-evaluating the integrand there.  Results are deterministic (fixed
// summation order) and agree with the reference's arithmetic up to rounding.
//
// Node evaluation: a team of T lanes evaluates a batch of up to BatchOf::NB nodes.
// The lanes first split the batch's scalar work (propagator halves,
// bubbles.jl; 6 or 12 interpolation plans, buffer.jl + channel.jl), then each
// lane gathers and combines the vertex on its sites (flow_su2_{s,t,u}.jl,
// flow_u1_dm_{s,t,u}.jl); the t channel stages both slots in shared memory for
// the overlap sum (flow_su2_t.jl:66-75) whose rows sit packed in shared memory.
// Every kernel is templated on the vertex component count C: 2 for SU(2)
// (spin, density), 6 for U(1)-DM (xx, zz, DM, dd, zd, dz).
#pragma once

#include <algorithm>
#include <type_traits>

#include "pffrg_internal.h"

namespace pffrg {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarps = 4;

template <typename R, int C>
struct NodeScratch {
    double x;      // the node (integration variable v)
    // the node as the setup uses it: converting it costs FP64 operations, once per node instead of at every step
    typename std::conditional<sizeof(R) == 4, FF, double>::type xs;
    __device__ __forceinline__ void set(double v) {
        x = v;
        xs = decltype(xs)(v);
    }
    PropTerm<R> prop[2];
    R p;           // the bubble propagator
    R loc[2 * C];  // t channel: local vertices v3[C], v4[C] at site 1
    NodePlan<R> plan[4][3];
};

// nodes per team batch: 4 per warp in total, 2 for SU(2) when each lane holds more than four sites
// (the SU(2) t-channel staging grows with sites x nodes).  The node scratch and t-channel staging
// of a batch set the shared memory of a block, which limits the blocks per SM: on the pyrochlore
// L = 6 two-loop state 32x2 teams with 4 nodes ran 403 ms against 470 ms with 8 nodes (two blocks
// per SM instead of three), and 16x3 teams were slower with 1 node than with 2.
template <int T, int C, int SPL>
__host__ __device__ constexpr int base_batch() { return (C == 2 ? (SPL <= 4 ? 4 : 2) : 4) * T / 32; }
// The setup runs the propagators of a batch first, then its plans, and a step of the warp that holds both
// costs the sum of the two.  One-site SU(2) teams of 16 lanes, and of 8 in FP64, therefore take twice the
// nodes: FP64 square L = 3 68 -> 58 ms (50/15/10, noise) and 5.2 -> 4.5 ms (11/4/3), a honeycomb L = 4
// parquet solve 33.9 -> 31.0 ms, a mixed cubic L = 4 step 94 -> 90 ms.  Four times the nodes left one block
// per SM (76 ms), FP32 teams of 8 lanes were 2 % slower with twice (8.6 against 8.45 ms), and 32 lanes
// hold a batch's setup in one step already.  The chunks of a level keep base_batch as their least size.
template <typename R, int T, int C, int SPL>
struct BatchOf {
    static constexpr bool twice = C == 2 && SPL == 1 && (T == 16 || (T == 8 && sizeof(R) == 8));
    static constexpr int NB = (twice ? 2 : 1) * base_batch<T, C, SPL>();
};

// SU(2) t-channel staging: per site the NB (spin, density) pairs of a batch, padded by 16 bytes so
// that the 16-byte loads of lanes reading different sites spread over the shared-memory banks
template <typename R, int NB>
__host__ __device__ constexpr int t_site_stride() {
    return NB + (sizeof(R) == 4 ? 2 : 1);  // in pairs of R
}

template <typename R, int T, int C, int SPL>
struct TeamScratch {
    NodeScratch<R, C> node[BatchOf<R, T, C, SPL>::NB];
};

// ---------------------------------------------------------------------------
// U(1)-DM bubbles of two vertices u, w (components xx, zz, DM, dd, zd, dz), the
// reference's term order; the same combination serves the Katanin, left,
// central, BSE and reduced kernels of a channel
// ---------------------------------------------------------------------------
// a0 b0 + a1 b1 + ...: the second product is rounded, the others enter by fused multiply-adds.  Written out
// because a compiler that chooses which products to fuse chooses differently from one kernel to the next.
template <typename R>
__device__ __forceinline__ R terms_from(R acc) {
    return acc;
}
template <typename R, typename... T>
__device__ __forceinline__ R terms_from(R acc, R a, R b, T... rest) {
    return terms_from(fma(a, b, acc), rest...);
}
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
template <typename R, typename... T>
__device__ __forceinline__ R terms(R a0, R b0, R a1, R b1, T... rest) {
    return terms_from(fma(a0, b0, mul_rn(a1, b1)), rest...);
}
// s channel (flow_u1_dm_s.jl:53-58)
template <typename R>
__device__ __forceinline__ void u1dm_s(const R* a, const R* b, R* g) {
    g[0] = terms(a[2], b[5], -a[2], b[4], a[0], b[3], a[3], b[0], -a[0], b[1], -a[5], b[2], a[4], b[2],
                 -a[1], b[0]);
    const R m0 = mul_rn((R)2 * a[0], b[0]);
    g[1] = terms_from(terms(a[1], b[3], a[3], b[1], -a[5], b[4]) - m0, -((R)2 * a[2]), b[2], -a[4], b[5]);
    g[2] = terms(a[3], b[2], a[2], b[3], -a[4], b[0], -a[0], b[5], -a[1], b[2], a[0], b[4], -a[2], b[1],
                 a[5], b[0]);
    g[3] = terms_from(fma(-a[5], b[5], m0), a[3], b[3], (R)2 * a[2], b[2], -a[4], b[4], a[1], b[1]);
    g[4] = terms(a[4], b[3], a[3], b[4], -((R)2 * a[2]), b[0], a[5], b[1], a[1], b[5], (R)2 * a[0], b[2]);
    g[5] = terms(a[4], b[1], a[3], b[5], a[1], b[4], (R)2 * a[2], b[0], a[5], b[3], -((R)2 * a[0]), b[2]);
}
// u channel (flow_u1_dm_u.jl:52-57)
template <typename R>
__device__ __forceinline__ void u1dm_u(const R* a, const R* b, R* g) {
    g[0] = terms(-a[2], b[5], -a[2], b[4], a[0], b[3], a[3], b[0], a[0], b[1], a[5], b[2], a[4], b[2],
                 a[1], b[0]);
    const R m0 = mul_rn((R)2 * a[0], b[0]);
    g[1] = terms_from(terms(a[1], b[3], a[3], b[1], -a[5], b[4]) + m0, (R)2 * a[2], b[2], -a[4], b[5]);
    g[2] = terms(a[3], b[2], a[2], b[3], -a[4], b[0], a[0], b[5], a[1], b[2], a[0], b[4], a[2], b[1],
                 -a[5], b[0]);
    g[3] = terms_from(fma(-a[5], b[5], m0), a[3], b[3], (R)2 * a[2], b[2], -a[4], b[4], a[1], b[1]);
    g[4] = terms(a[4], b[3], a[3], b[4], -((R)2 * a[2]), b[0], a[5], b[1], a[1], b[5], (R)2 * a[0], b[2]);
    g[5] = terms(a[4], b[1], a[3], b[5], a[1], b[4], -((R)2 * a[2]), b[0], a[5], b[3], (R)2 * a[0], b[2]);
}
// t channel, local part: v1, v2 non-local at site i, v3, v4 local at site 1 (flow_u1_dm_t.jl:68-84)
template <typename R>
__device__ __forceinline__ void u1dm_t(const R* v1, const R* v2, const R* v3, const R* v4, R* g) {
    g[0] = terms(v1[2], v4[5], -v1[2], v4[4], v1[0], v4[3], -v1[0], v4[1], v3[3], v2[0], v3[5], v2[2],
                 -v3[4], v2[2], -v3[1], v2[0]);
    g[1] = terms(v1[1], v4[3], (R)2 * v1[4], v4[2], -v1[4], v4[4], v1[1], v4[1], -((R)2 * v1[1]), v4[0],
                 -v1[4], v4[5], -((R)2 * v3[2]), v2[5], -v3[5], v2[5], v3[3], v2[1], -((R)2 * v3[0]), v2[1],
                 v3[1], v2[1], -v3[4], v2[5]);
    g[2] = terms(v1[2], v4[3], -v1[0], v4[5], v1[0], v4[4], -v1[2], v4[1], -v3[5], v2[0], v3[3], v2[2],
                 v3[4], v2[0], -v3[1], v2[2]);
    g[3] = terms((R)2 * v1[3], v4[0], -v1[5], v4[5], v1[3], v4[1], -v1[5], v4[4], -((R)2 * v1[5]), v4[2],
                 v1[3], v4[3], (R)2 * v3[2], v2[4], (R)2 * v3[0], v2[3], v3[1], v2[3], -v3[5], v2[4],
                 v3[3], v2[3], -v3[4], v2[4]);
    g[4] = terms(v1[4], v4[1], v1[4], v4[3], (R)2 * v1[4], v4[0], v1[1], v4[4], (R)2 * v1[1], v4[2],
                 v1[1], v4[5], v3[4], v2[3], (R)2 * v3[2], v2[3], v3[3], v2[4], v3[1], v2[4],
                 -((R)2 * v3[0]), v2[4], v3[5], v2[3]);
    g[5] = terms(v1[3], v4[4], -((R)2 * v1[3]), v4[2], v1[3], v4[5], v1[5], v4[1], v1[5], v4[3],
                 -((R)2 * v1[5]), v4[0], v3[4], v2[1], (R)2 * v3[0], v2[5], v3[3], v2[5], v3[5], v2[1],
                 -((R)2 * v3[2]), v2[1], v3[1], v2[5]);
}

// vertex component c of one slot at one site (single value), for the t-channel local vertices
template <typename R, int C>
__device__ __forceinline__ R gather_one(const PassArgs<R>& A, const NodeScratch<R, C>& ns, int slot, int c, int i,
                                        int exch_i) {
    const R* __restrict__ src = A.src[slot];
    constexpr int CS = sizeof(R) == 4 && C == 2 ? 2 : 1;  // FP32 copies of SU(2) actions hold (spin, density) pairs
    R val = CS == 2 ? ldg(src + c + 2 * (A.L.pbare() + i)) : ldg(src + A.L.bare(c) + i);
#pragma unroll 1
    for (int ch = 0; ch < 3; ++ch) {
        const NodePlan<R>& P = ns.plan[slot][ch];
        const int nc = P.nc;
        if (!nc) continue;
        R sgn;
        const int cs = comp_read(P, C, c, sgn);
        const R* q = CS == 2 ? src + c + 2 * P.base : src + P.base + cs * A.L.comp;
        const int st = P.exch ? exch_i : i;
        R acc;
        if constexpr (sizeof(R) == 4 && C == 6) {
            // the second product of a bosonic pair is rounded first: the FP32 results stay those of the
            // uncompacted plan, in which the compiler chose this order.  Either is as exact, but one chain of
            // multiply-adds moves mixed right-hand sides of kagome L = 2 to 8 by 2e-9 to 5e-9 of their norm.
            int k = 1;
            acc = mul_rn(P.w[0], ldg(q + P.off[0] + st));
            if (P.flags & 8) {
                acc = fma(P.w[0], ldg(q + P.off[0] + st), mul_rn(P.w[1], ldg(q + P.off[1] + st)));
                k = 2;
            }
            for (; k < nc; ++k) acc = fma(P.w[k], ldg(q + P.off[k] + st), acc);
        } else {
            acc = P.w[0] * ldg(q + CS * (P.off[0] + st));
            for (int k = 1; k < nc; ++k) acc += P.w[k] * ldg(q + CS * (P.off[k] + st));
        }
        val += sgn * acc;
    }
    return val;
}

// all components of one slot on this lane's sites, v[c][k] = Γ_c(site tl + k T) (the U(1)-DM passes;
// SU(2) reads its pair-layout copies in Team::gather_su2): bare + Σ_ch sgn Σ_q w_q q_c'[off_q + site]
// with the read component c' and sign of apply_flags_u1_dm, channels and corners in the reference's
// order.  The loop over a channel's corners is not unrolled: one corner's reads of all components
// and sites are in flight together, and the kernel's code stays small enough for the instruction
// cache (unrolled over the eight corners, six components and the lane's sites, the reads of two
// slots made the three-loop U(1)-DM kernels wait on instruction fetch 15 cycles per issue).  Padding
// sites read site 0 and are zeroed at the end.
template <typename R, int T, int SPL, int C>
__device__ __forceinline__ void gather_slot(const PassArgs<R>& A, const NodeScratch<R, C>& ns, int slot, int tl,
                                            const int* site_ex, R v[C][SPL]) {
    const R* __restrict__ src = A.src[slot];
    const int Ns = A.L.Ns;
    int si[SPL];
#pragma unroll
    for (int k = 0; k < SPL; ++k) {
        const int i = tl + k * T;
        si[k] = i < Ns ? i : 0;
    }
#pragma unroll
    for (int k = 0; k < SPL; ++k)
#pragma unroll
        for (int c = 0; c < C; ++c) v[c][k] = ldg(src + A.L.bare(c) + si[k]);
#pragma unroll 1
    for (int ch = 0; ch < 3; ++ch) {
        const NodePlan<R>& P = ns.plan[slot][ch];
        const int nc = P.nc;
        if (!nc) continue;
        int st[SPL];
#pragma unroll
        for (int k = 0; k < SPL; ++k) st[k] = P.exch ? site_ex[k] : si[k];
        const R* q0[C];
        R sg[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int cs = comp_read(P, C, c, sg[c]);
            q0[c] = src + P.base + cs * A.L.comp;
        }
        R a[C][SPL];
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int k = 0; k < SPL; ++k) a[c][k] = (R)0;
#pragma unroll 1
        for (int q = 0; q < nc; ++q) {
            const R w = P.w[q];
            const int off = P.off[q];
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int k = 0; k < SPL; ++k) a[c][k] += w * ldg(q0[c] + off + st[k]);
        }
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int k = 0; k < SPL; ++k) v[c][k] += sg[c] * a[c][k];
    }
#pragma unroll
    for (int k = 0; k < SPL; ++k)
        if (tl + k * T >= Ns)
#pragma unroll
            for (int c = 0; c < C; ++c) v[c][k] = (R)0;
}

template <typename R>
struct Acc {
    R s;
    R c;
};

template <typename R>
__device__ __forceinline__ void acc_add(Acc<R>& a, R x) {
    a.s += x;
}
// Kahan-Babuska (Neumaier) summation for the FP32 node sums
template <>
__device__ __forceinline__ void acc_add<float>(Acc<float>& a, float x) {
    float t = a.s + x;
    if (fabsf(a.s) >= fabsf(x)) a.c += (a.s - t) + x;
    else a.c += (x - t) + a.s;
    a.s = t;
}

template <int T>
__device__ __forceinline__ double in_team_sum(double v) {
#pragma unroll
    for (int o = 1; o < T; o <<= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// Task of a subdomain record and its frequencies (get_kernel_args, mesh.jl:30-83)
struct TaskInfo {
    int X, kernel, w1, w2, w3;
};

template <typename R>
__device__ __forceinline__ TaskInfo task_of(const PassArgs<R>& A, int sub, int jobs) {
    const int ct = sub / jobs;  // channel-task index = y * ntasks + task
    const int y = ct / A.ntasks;
    const int4 t = A.tasks[ct - y * A.ntasks];
    return TaskInfo{A.chan_of_y[y], t.x, t.y, t.z, t.w};
}

// The plan of a mixed-path argument near a buffer switch: the FP64 path's rounding decides the side.
// Not inlined (and given values, not the kernel's arguments, whose address would copy them to local
// memory): few lanes take it, and the kernels' code has to fit the instruction caches.
static __device__ __noinline__ int plan_fp64(NodePlan<float>& P, const double* mesh, int Nsig, int NO, int Nn, int Ns,
                                             int64_t q0, int X, int w1, int wf, int ch, unsigned code,
                                             double x) {
    const MeshD M = mesh_view_d(mesh, Nsig, NO, Nn);
    const double W = M.at(X == 1 ? M.Ot() : M.Os(), w1);
    const double F = wf >= 0 ? M.at(X == 1 ? M.nt() : M.ns(), wf) : INFINITY;
    return build_plan(P, ch, plan_arg(code, W, x, F), plan_arg(code >> 7, W, x, F), plan_arg(code >> 14, W, x, F), M, Ns,
                      q0);
}

template <typename R, int T, int SPL, int C>
struct Team {
    const PassArgs<R>& A;
    // node setup: FP64 on the FP64 path, float-float on the mixed path
    using SetupT = typename std::conditional<sizeof(R) == 4, FF, double>::type;
    using SetupMesh = typename std::conditional<sizeof(R) == 4, MeshFF, MeshD>::type;
    const SetupMesh& M;
    TeamScratch<R, T, C, SPL>& ts;
    R* tmp;                 // t channel: [2 C][Ns] slot values of the current node
    const unsigned* rows;   // packed overlap rows (shared or global)
    const int* row_off;     // [Ns+1]
    int tl;                 // lane in team
    int site_ex[SPL];       // exchange[site] of this lane's sites
    unsigned long long nodes, alg;
    bool odd_first = false;  // FP32 U(1)-DM: see eval_u1dm

    // offset of the first kernel of the s channel in a vertex source
    __device__ __forceinline__ int64_t q0() const {
        return sizeof(R) == 4 && C == 2 ? A.L.pbare() + A.L.Ns : A.L.qbase(0, 0, 0);
    }

    // Evaluate the integrand of channel X at the up to NB nodes ts.node[0..count).x of one task and
    // hand each node's values to sink(j, g) in node order, g[c][k] = Γ_c(site tl + k T; x_j)
    // (zero on the padding sites k T + tl >= Ns).  Team-collective: all lanes of the warp call it
    // together (inactive teams with count = 0).
    template <class Sink>
    __device__ __forceinline__ void eval(const TaskInfo& ti, SetupT W, SetupT V, SetupT VP, int count, Sink& sink) {
        const int X = ti.X;
        const int Ns = A.L.Ns;
        const int nslots = (X == 1) ? 4 : 2;
        const bool kat = A.prop_kind == PROP_KAT;
        const int nplans = 3 * nslots, nitems = 2 + nplans;
        nodes += count;
        // teams of one warp may hold different channels and batch lengths: every lane runs
        // the same sequence of warp syncs, bounded by the warp's longest batch
        int mx = count;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(kFull, mx, o));
        // phase A: scalar work of all nodes of the batch, split over the team's lanes
        unsigned corners = 0;  // corners of this lane's plans times the sites that read them
#pragma unroll 1
        for (int it = tl; it < count * nitems; it += T) {
            // the propagators of all nodes, then the plans
            const int k = it - 2 * count;
            const int j = k < 0 ? it >> 1 : k / nplans;
            NodeScratch<R, C>& ns = ts.node[j];
            const SetupT v = ns.xs;
            if (k < 0) {
                const int item = it & 1;
                if constexpr (sizeof(R) == 4)
                    ns.prop[item] = prop_term(kat, M, A.prop_a, A.prop_da, (float)A.Lam,
                                              prop_freq(X, item, v, FF{0.5f, 0.f} * W));
                else
                    ns.prop[item] = prop_term(kat, M, A.prop_a64, A.prop_da64, A.pc, prop_freq(X, item, v, 0.5 * W));
                continue;
            }
            const int sc = k - j * nplans, slot = sc / 3, ch = sc - 3 * slot;
            NodePlan<R>& P = ns.plan[slot][ch];
            if (!(A.mask[X][slot] & (1 << ch))) {
                P.nc = 0;
                continue;
            }
            const unsigned code = __ldg(&kArgCodes[X][slot][ch]);
            const SetupT F = (slot & 1) ? VP : V;
            const SetupT a0 = plan_arg(code, W, v, F), a1 = plan_arg(code >> 7, W, v, F),
                         a2 = plan_arg(code >> 14, W, v, F);
            int nc;
            if constexpr (sizeof(R) == 4) {
                const float scale = fabsf(v.h) + fabsf(W.h) + (isinf(V.h) ? 0.f : fabsf(V.h)) +
                                    (isinf(VP.h) ? 0.f : fabsf(VP.h));
                if (ff_near_switch(a0, scale, M, A.L.NO, A.L.Nn) || ff_near_switch(a1, scale, M, A.L.NO, A.L.Nn) ||
                    ff_near_switch(a2, scale, M, A.L.NO, A.L.Nn))
                    nc = plan_fp64(P, A.mesh, A.L.Nsig, A.L.NO, A.L.Nn, Ns, q0(), X, ti.w1, (slot & 1) ? ti.w3 : ti.w2, ch,
                                   code, ns.x);
                else
                    nc = build_plan(P, ch, a0, a1, a2, M, Ns, q0());
            } else {
                nc = build_plan(P, ch, a0, a1, a2, M, Ns, q0());
            }
            corners += nc * (slot < 2 ? Ns : 1);
        }
        if (A.node_counter) {
            alg += (unsigned long long)corners * C;
            if (tl == 0) alg += (unsigned long long)count * C * (3ull * Ns + (X == 1 ? 2ull * row_off[Ns] : 0ull));
        }
        __syncwarp();
        if (tl < count) ts.node[tl].p = prop_combine(kat, ts.node[tl].prop);
        if (X == 1) {
            // local vertices at site 1 (flow_su2_t.jl:46-48, flow_u1_dm_t.jl:44-46)
            const int e0 = ldg(A.exch);
            for (int it = tl; it < count * 2 * C; it += T) {
                const int j = it / (2 * C), q = it - j * (2 * C);
                ts.node[j].loc[q] = gather_one<R, C>(A, ts.node[j], 2 + q / C, q % C, 0, e0);
            }
        }
        __syncwarp();
        if constexpr (C == 2) {
            // every team of the warp passes the same two warp barriers, whatever its channel
            eval_su2_nodes(X, count, sink);
            __syncwarp();
            if (X == 1) eval_t_overlap(count, sink);
            __syncwarp();
        } else {
            // phase B of U(1)-DM: gathers and per-site combination, node by node
#pragma unroll 1
            for (int j = 0; j < mx; ++j) {
                const bool act = j < count;
                const NodeScratch<R, C>& ns = ts.node[act ? j : 0];
                R p = (R)0;
                R v1[C][SPL], v2[C][SPL];
                if (act) {
                    p = ns.p;
                    gather_slot<R, T, SPL, C>(A, ns, 0, tl, site_ex, v1);
                    gather_slot<R, T, SPL, C>(A, ns, 1, tl, site_ex, v2);
                }
                eval_u1dm(X, j, act, p, ns, v1, v2, sink);
            }
        }
    }

    // One non-local vertex slot of an SU(2) node on this lane's sites (get_Γ_avx!,
    // action_su2.jl:115-134): bare + Σ_ch sgn Σ_q w_q q[off_q + site], channels in the reference's
    // order.  A channel's corners are walked by a loop (smaller code and fewer live registers than
    // all eight unrolled: 113 instead of 127 for the FP32 32x2 kernel, 155 instead of 229 for the
    // FP64 one; 4-8 % faster), the FP32 loop two corners at a time (the reads of two corners for both
    // components and all of the lane's sites in flight together: a further 3-4 %; four at a time
    // was slower); the loop over the sites has no branch (padding sites read site 0 and are zeroed
    // at the end).
    __device__ __forceinline__ void gather_su2(const NodeScratch<R, C>& ns, int slot, R v[2][SPL]) {
        const int Ns = A.L.Ns;
        const R* __restrict__ src = A.src[slot];
        int si[SPL];
#pragma unroll
        for (int k = 0; k < SPL; ++k) {
            const int i = tl + k * T;
            si[k] = i < Ns ? i : 0;
        }
        if constexpr (sizeof(R) == 4) {
            // FP32 copies hold (spin, density) pairs: one 8-byte read per corner and site
            const float2* __restrict__ src2 = reinterpret_cast<const float2*>(src);
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                const float2 b = ldg(src2 + A.L.pbare() + si[k]);
                v[0][k] = b.x;
                v[1][k] = b.y;
            }
#pragma unroll 1
            for (int ch = 0; ch < 3; ++ch) {
                const NodePlan<R>& P = ns.plan[slot][ch];
                const int nc = P.nc;
                if (!nc) continue;
                const float2* q = src2 + P.base;
                const R sgn_d = P.sgn_d;
                const int ex = P.exch;
                int st[SPL];
                R a0[SPL], a1[SPL];
#pragma unroll
                for (int k = 0; k < SPL; ++k) {
                    st[k] = ex ? site_ex[k] : si[k];
                    a0[k] = a1[k] = (R)0;
                }
#pragma unroll 2
                for (int c = 0; c < nc; ++c) {
                    const R w = P.w[c];
                    const int off = P.off[c];
#pragma unroll
                    for (int k = 0; k < SPL; ++k) {
                        const float2 t = ldg(q + off + st[k]);
                        a0[k] += w * t.x;
                        a1[k] += w * t.y;
                    }
                }
#pragma unroll
                for (int k = 0; k < SPL; ++k) {
                    v[0][k] += a0[k];
                    v[1][k] += sgn_d * a1[k];
                }
            }
#pragma unroll
            for (int k = 0; k < SPL; ++k)
                if (tl + k * T >= Ns) v[0][k] = v[1][k] = (R)0;
            return;
        }
#pragma unroll
        for (int k = 0; k < SPL; ++k) {
            v[0][k] = ldg(src + A.L.bare(0) + si[k]);
            v[1][k] = ldg(src + A.L.bare(1) + si[k]);
        }
#pragma unroll 1
        for (int ch = 0; ch < 3; ++ch) {
            const NodePlan<R>& P = ns.plan[slot][ch];
            const int nc = P.nc;
            if (!nc) continue;
            const R* q0 = src + P.base;
            const R* q1 = q0 + A.L.comp;
            const R sgn_d = P.sgn_d;
            const int ex = P.exch;
            int st[SPL];
            R a0[SPL], a1[SPL];
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                st[k] = ex ? site_ex[k] : si[k];
                a0[k] = a1[k] = (R)0;
            }
#pragma unroll 1
            for (int q = 0; q < nc; ++q) {
                const R w = P.w[q];
                const int off = P.off[q];
#pragma unroll
                for (int k = 0; k < SPL; ++k) {
                    a0[k] += w * ldg(q0 + off + st[k]);
                    a1[k] += w * ldg(q1 + off + st[k]);
                }
            }
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                v[0][k] += a0[k];
                v[1][k] += sgn_d * a1[k];
            }
        }
#pragma unroll
        for (int k = 0; k < SPL; ++k)
            if (tl + k * T >= Ns) v[0][k] = v[1][k] = (R)0;
    }

    // phase B of SU(2), node by node: the s and u bubbles (flow_su2_s.jl, flow_su2_u.jl) per site,
    // handed to the sink, or for the t channel (flow_su2_t.jl:46-81) the local part per site kept in
    // shared memory and both slots staged as [site][node] (spin, density) pairs for the overlap sums
    template <class Sink>
    __device__ __forceinline__ void eval_su2_nodes(int X, int count, Sink& sink) {
        constexpr int NB = BatchOf<R, T, C, SPL>::NB;
        using R2 = typename std::conditional<sizeof(R) == 4, float2, double2>::type;
        const int Ns = A.L.Ns;
        constexpr int SS = t_site_stride<R, NB>();
        R2* tb1 = reinterpret_cast<R2*>(tmp);  // [Ns][SS]
        R2* tb2 = tb1 + (size_t)Ns * SS;
        R2* tloc = tb2 + (size_t)Ns * SS + (size_t)Ns * NB;  // [Ns][NB] local parts (after the overlap sums)
        const R two = (X == 0) ? (R)-2 : (R)2;
        for (int j = 0; j < count; ++j) {
            const NodeScratch<R, C>& ns = ts.node[j];
            const R p = ns.p;
            R v1[2][SPL], v2[2][SPL];
            gather_su2(ns, 0, v1);
            gather_su2(ns, 1, v2);
            if (X != 1) {
                R g[2][SPL];
#pragma unroll
                for (int k = 0; k < SPL; ++k) {
                    g[0][k] = -p * (two * v1[0][k] * v2[0][k] + v1[0][k] * v2[1][k] + v1[1][k] * v2[0][k]);
                    g[1][k] = -p * ((R)3 * v1[0][k] * v2[0][k] + v1[1][k] * v2[1][k]);
                }
                sink(j, g);
                continue;
            }
            const R v3s = ns.loc[0], v3d = ns.loc[1], v4s = ns.loc[2], v4d = ns.loc[3];
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                const int i = tl + k * T;
                const R v1s = v1[0][k], v1d = v1[1][k], v2s = v2[0][k], v2d = v2[1][k];
                if (i < Ns) {
                    const R Gs = -p * ((R)-1 * v1s * v4s + v1s * v4d - (R)1 * v3s * v2s + v3d * v2s);
                    const R Gd = -p * ((R)3 * v1d * v4s + v1d * v4d + (R)3 * v3s * v2d + v3d * v2d);
                    tloc[(size_t)i * NB + j] = R2{Gs, Gd};
                    tb1[(size_t)i * SS + j] = R2{v1s, v1d};
                    tb2[(size_t)i * SS + j] = R2{v2s, v2d};
                }
            }
        }
    }

    // second half: the overlap sums (flow_su2_t.jl:66-75) of the whole batch.  All lanes walk the
    // sites in the same order; a lane takes every T-th row of a site, decodes it once and adds the
    // row's product for every node of the batch (the (spin, density) pairs of a site's nodes are
    // neighbours in shared memory: two 16-byte reads per vertex slot and row); the 2 NB partial sums
    // of the lanes meet by shuffles that halve the values a lane carries at every step, and one
    // lane per value stores its total.  Then the owner of a site adds -p (-2) (2S) times them to
    // its nodes' local parts and hands the nodes to the sink.  (The earlier split, NB lanes per row
    // each adding one node, decoded every row NB times: 376 against 352 ms for the pyrochlore
    // L = 6 two-loop right-hand side at 50/15/10 frequencies.)  Nodes past `count` hold stale
    // values whose sums are never used.
    template <class Sink>
    __device__ __forceinline__ void eval_t_overlap(int count, Sink& sink) {
        constexpr int NB = BatchOf<R, T, C, SPL>::NB;
        using R2 = typename std::conditional<sizeof(R) == 4, float2, double2>::type;
        const int Ns = A.L.Ns;
        constexpr int SS = t_site_stride<R, NB>();
        const R2* tb1 = reinterpret_cast<const R2*>(tmp);
        const R2* tb2 = tb1 + (size_t)Ns * SS;
        R2* ov = const_cast<R2*>(tb2) + (size_t)Ns * SS;  // [Ns][NB] overlap sums
        const R2* tloc = ov + (size_t)Ns * NB;
        const unsigned team_mask = (T == 32) ? kFull : (((1u << T) - 1u) << ((threadIdx.x & 31) / T * T));
        constexpr int V = 2 * NB;  // sums per site: (spin, density) of every node of the batch
        R* ovr = reinterpret_cast<R*>(ov);
        // FP32 teams of a warp fetch the next row while one is worked on, across the end of a site's list too:
        // long lists do not fit in shared memory beside the staging and are read through L1, of which the
        // vertex gathers leave little (pyrochlore L = 6 two loops mixed 249 -> 235 ms; narrower teams, whose
        // short lists are staged in shared memory up to 14 sites, were 1.5 % slower with it).
        constexpr bool kAhead = sizeof(R) == 4 && T == 32;
        int r = tl, j1 = row_off[0], rn = j1 + tl;
        const int last = row_off[Ns] - 1;
        unsigned next = kAhead && last >= 0 ? rows[min(rn, last)] : 0;
        for (int i = 0; i < Ns; ++i) {
            R x[V];
#pragma unroll
            for (int v = 0; v < V; ++v) x[v] = (R)0;
            r = j1 + tl;
            j1 = row_off[i + 1];
            if (kAhead && rn != r && r < j1) next = rows[r];  // the list before had no row for this lane
#pragma unroll 2
            for (; r < j1; r += T) {
                unsigned row;
                if constexpr (kAhead) {
                    row = next;
                    rn = r + T < j1 ? r + T : j1 + tl;
                    next = rows[min(rn, last)];
                } else {
                    row = rows[r];
                }
                const int ia = row & 0xff, ib = (row >> 8) & 0xff;
                const R2* pa = tb1 + (size_t)ia * SS;
                const R2* pb = tb2 + (size_t)ib * SS;
                // most rows have multiplicity one (pyrochlore L = 6: 60 % of the steps of 32 rows have no other),
                // and in FP64 its product with the first slot is half of a row's operations (pyrochlore L = 6
                // FP64 99 -> 79 ms); short FP32 lists multiply without looking
                const bool scaled = (sizeof(R) == 4 && T < 32) || (row >> 16) != 1;
                if constexpr (sizeof(R) == 4 && NB % 2 == 0) {
                    float4 a[NB / 2];
#pragma unroll
                    for (int j2 = 0; j2 < NB / 2; ++j2) a[j2] = reinterpret_cast<const float4*>(pa)[j2];
                    if (scaled) {
                        const R m = (R)(row >> 16);
#pragma unroll
                        for (int j2 = 0; j2 < NB / 2; ++j2)
                            a[j2].x = m * a[j2].x, a[j2].y = m * a[j2].y, a[j2].z = m * a[j2].z, a[j2].w = m * a[j2].w;
                    }
#pragma unroll
                    for (int j2 = 0; j2 < NB / 2; ++j2) {
                        const float4 b = reinterpret_cast<const float4*>(pb)[j2];
                        x[4 * j2 + 0] = fma(a[j2].x, b.x, x[4 * j2 + 0]);
                        x[4 * j2 + 1] = fma(a[j2].y, b.y, x[4 * j2 + 1]);
                        x[4 * j2 + 2] = fma(a[j2].z, b.z, x[4 * j2 + 2]);
                        x[4 * j2 + 3] = fma(a[j2].w, b.w, x[4 * j2 + 3]);
                    }
                } else {
                    R2 a[NB];
#pragma unroll
                    for (int j = 0; j < NB; ++j) a[j] = pa[j];
                    if (scaled) {
                        const R m = (R)(row >> 16);
#pragma unroll
                        for (int j = 0; j < NB; ++j) a[j].x = m * a[j].x, a[j].y = m * a[j].y;
                    }
#pragma unroll
                    for (int j = 0; j < NB; ++j) {
                        const R2 b = pb[j];
                        x[2 * j] = fma(a[j].x, b.x, x[2 * j]);
                        x[2 * j + 1] = fma(a[j].y, b.y, x[2 * j + 1]);
                    }
                }
            }
            // sum over the team's lanes, halving the values each lane carries at every step
            int n = V, idx = 0;
#pragma unroll
            for (int o = T / 2; o >= 1; o >>= 1) {
                if (n > 1) {
                    n >>= 1;
                    const bool up = (tl & o) != 0;
#pragma unroll
                    for (int k = 0; k < V / 2; ++k) {
                        if (k < n) {
                            const R send = up ? x[k] : x[k + n];
                            const R keep = up ? x[k + n] : x[k];
                            x[k] = keep + __shfl_xor_sync(team_mask, send, o);
                        }
                    }
                    if (up) idx += n;
                } else {
                    x[0] += __shfl_xor_sync(team_mask, x[0], o);
                }
            }
            // every lane now holds the total of value idx; one lane per value writes it
            if ((tl & (T / V - 1)) == 0) ovr[((size_t)i * NB) * 2 + idx] = x[0];
        }
        __syncwarp(team_mask);
        const R twoS = (R)A.twoS;
#pragma unroll 1
        for (int jj = 0; jj < count; ++jj) {
            const NodeScratch<R, C>& ns = ts.node[jj];
            const R p = ns.p;
            const R coef = -p * (R)-2 * twoS;
            R g[2][SPL];
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                const int i = tl + k * T;
                g[0][k] = g[1][k] = (R)0;
                if (i < Ns) {
                    const R2 lo = tloc[(size_t)i * NB + jj], s = ov[(size_t)i * NB + jj];
                    g[0][k] = lo.x + coef * s.x;
                    g[1][k] = lo.y + coef * s.y;
                }
            }
            sink(jj, g);
        }
    }

    // add this warp's evaluations and algorithmic values to the context's counters
    __device__ __forceinline__ void count_nodes() {
        if (!A.node_counter) return;
        unsigned long long n = tl == 0 ? nodes : 0, a = alg;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            n += __shfl_xor_sync(kFull, n, o);
            a += __shfl_xor_sync(kFull, a, o);
        }
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(A.node_counter, n);
            atomicAdd(A.node_counter + 1, a);
        }
    }

    // phase B of one node for U(1)-DM (flow_u1_dm_{s,t,u}.jl); team-collective like eval
    template <class Sink>
    __device__ void eval_u1dm(int X, int j, bool act, R p, const NodeScratch<R, C>& ns, const R v1[C][SPL],
                              const R v2[C][SPL], Sink& sink) {
        const int Ns = A.L.Ns;
        if (act && X != 1) {
            R g[C][SPL];
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                R a[C], b[C], h[C];
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    a[c] = v1[c][k];
                    b[c] = v2[c][k];
                }
                if (X == 0) u1dm_s(a, b, h);
                else u1dm_u(a, b, h);
#pragma unroll
                for (int c = 0; c < C; ++c) g[c][k] = -p * h[c];
                if (A.reduced) {
                    // the reduced s bubble of the SDE keeps xx, zz, dd (SDE_u1_dm.jl:38-46)
                    g[2][k] = (R)0;
                    g[4][k] = (R)0;
                    g[5][k] = (R)0;
                }
            }
            sink(j, g);
        }
        const bool tch = act && X == 1;
        // both slots of a site lie in 16-byte pieces (FP32: four and two components, FP64 three pairs), so a
        // row of the overlap sum takes two or three loads per slot instead of six (with the FP64 form below,
        // kagome L = 8 three loops mixed 252 -> 247 ms, kagome L = 3 FP64 25.2 -> 24.8 ms)
        using V4 = typename std::conditional<sizeof(R) == 4, float4, double2>::type;
        using V2 = typename std::conditional<sizeof(R) == 4, float2, double2>::type;
        V4* t1a = reinterpret_cast<V4*>(tmp);
        V4* t2a = t1a + (sizeof(R) == 4 ? Ns : 2 * Ns);
        V2* t1b = reinterpret_cast<V2*>(t2a + (sizeof(R) == 4 ? Ns : 2 * Ns));
        V2* t2b = t1b + Ns;
        if (tch) {
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                const int i = tl + k * T;
                if (i < Ns) {
                    if constexpr (sizeof(R) == 4) {
                        t1a[i] = make_float4(v1[0][k], v1[1][k], v1[2][k], v1[3][k]);
                        t2a[i] = make_float4(v2[0][k], v2[1][k], v2[2][k], v2[3][k]);
                        t1b[i] = make_float2(v1[4][k], v1[5][k]);
                        t2b[i] = make_float2(v2[4][k], v2[5][k]);
                    } else {
                        t1a[i] = make_double2(v1[0][k], v1[1][k]);
                        t1a[Ns + i] = make_double2(v1[2][k], v1[3][k]);
                        t2a[i] = make_double2(v2[0][k], v2[1][k]);
                        t2a[Ns + i] = make_double2(v2[2][k], v2[3][k]);
                        t1b[i] = make_double2(v1[4][k], v1[5][k]);
                        t2b[i] = make_double2(v2[4][k], v2[5][k]);
                    }
                }
            }
        }
        __syncwarp();
        if (tch) {
            const R coef = -p * (R)-2;
            R g[C][SPL];
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                const int i = tl + k * T;
                R a[C], b[C], G[C];
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    a[c] = v1[c][k];
                    b[c] = v2[c][k];
                }
                u1dm_t(a, b, ns.loc, ns.loc + C, G);
                // overlap sum (flow_u1_dm_t.jl:86-110)
                int r = 0, j1 = 0;
                if (i < Ns) r = row_off[i], j1 = row_off[i + 1];
                if constexpr (sizeof(R) == 4) {
                    // one row: the six bilinear terms of its two sites
                    auto row_terms = [&](unsigned row, R* x) {
                        const int ia = row & 0xff, ib = (row >> 8) & 0xff;
                        const float4 p1 = t1a[ia], p2 = t2a[ib];
                        const float2 q1 = t1b[ia], q2 = t2b[ib];
                        x[0] = terms(p1.x, p2.x, -p1.z, p2.z);
                        x[1] = terms(p1.y, p2.y, -q1.x, q2.y);
                        x[2] = terms(p1.z, p2.x, p1.x, p2.z);
                        x[3] = terms(p1.w, p2.w, -q1.y, q2.x);
                        x[4] = terms(q1.x, p2.w, p1.y, q2.x);
                        x[5] = terms(p1.w, q2.y, q1.y, p2.y);
                    };
                    // refining nodes of lattices with three sites per lane: the first of an odd number of rows is
                    // fused with the local part's factor, as a compiler unrolled these loops once, and the first
                    // level and other lane widths are not.  It costs nothing measurable (kagome L = 8, 0.245 s
                    // either way) and has no numerical purpose; without it such right-hand sides move by 3e-10
                    // to 1.2e-9 of their norm, so it stays with the results.
                    const bool odd = odd_first && k < 2 && ((j1 - r) & 1);
                    if (odd) {
                        R x[C];
                        row_terms(rows[r], x);
                        const R mm = coef * (R)(rows[r] >> 16);
#pragma unroll
                        for (int c = 0; c < C; ++c) G[c] = fma(-p, G[c], mul_rn(mm, x[c]));
                        ++r;
                    } else {
#pragma unroll
                        for (int c = 0; c < C; ++c) G[c] = mul_rn(-p, G[c]);
                    }
#pragma unroll 2
                    for (; r < j1; ++r) {
                        const unsigned row = rows[r];
                        R x[C];
                        row_terms(row, x);
                        const R mm = coef * (R)(row >> 16);
#pragma unroll
                        for (int c = 0; c < C; ++c) G[c] = fma(mm, x[c], G[c]);
                    }
                } else {
                    // FP64: twelve multiply-adds a row; the common factor comes last, and the multiplicity,
                    // which is one for nearly all rows, only where it counts (19 FP64 operations with both in
                    // every row)
                    R S[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 1
                    for (; r < j1; ++r) {
                        const unsigned row = rows[r];
                        const int ia = row & 0xff, ib = (row >> 8) & 0xff;
                        double2 x01 = t1a[ia], x23 = t1a[Ns + ia], x45 = t1b[ia];
                        const double2 y01 = t2a[ib], y23 = t2a[Ns + ib], y45 = t2b[ib];
                        if ((row >> 16) != 1) {
                            const R m = (R)(row >> 16);
                            x01.x *= m, x01.y *= m, x23.x *= m, x23.y *= m, x45.x *= m, x45.y *= m;
                        }
                        S[0] = fma(x01.x, y01.x, S[0]);
                        S[1] = fma(x01.y, y01.y, S[1]);
                        S[2] = fma(x23.x, y01.x, S[2]);
                        S[3] = fma(x23.y, y23.y, S[3]);
                        S[4] = fma(x45.x, y23.y, S[4]);
                        S[5] = fma(x23.y, y45.y, S[5]);
                        S[0] = fma(-x23.x, y23.x, S[0]);
                        S[1] = fma(-x45.x, y45.y, S[1]);
                        S[2] = fma(x01.x, y23.x, S[2]);
                        S[3] = fma(-x45.y, y45.x, S[3]);
                        S[4] = fma(x01.y, y45.x, S[4]);
                        S[5] = fma(x45.y, y01.y, S[5]);
                    }
#pragma unroll
                    for (int c = 0; c < C; ++c) G[c] = fma(coef, S[c], -p * G[c]);
                }
#pragma unroll
                for (int c = 0; c < C; ++c) g[c][k] = G[c];
            }
            sink(j, g);
        }
        __syncwarp();
    }
};

// ---------------------------------------------------------------------------
// wave workspace (device scratch of a pass; one block carved into arrays)
// ---------------------------------------------------------------------------
// The coarse cut of a level of n new nodes: chunks of 32 nodes, at most 256 chunks per subdomain (bigger
// levels use bigger chunks).  The chunk queue's capacity is counted in coarse chunks.
constexpr int kChunk = 32;
constexpr int kMaxChunks = 256;

// How the subdomains of a level are cut.  All subdomains refining at one level have the same number n of
// new nodes (4 at the first level, doubled at each), so a chunk index is (subdomain, part) arithmetic and
// no queue of chunk records is written or read.
struct LevelCut {
    int nact;    // subdomains cut (fewer than are active only after an overflow)
    int coarse;  // coarse chunks per subdomain
    int chunks;  // chunks per subdomain (a multiple of coarse)
    int per;     // nodes per chunk
    bool overflow;
};

// Few active subdomains leave most teams without a coarse chunk, and a level then lasts as long as one
// team takes for 32 nodes one after another (square L = 3 FP64: 93, 166, 308 and 570 us for chunks of 4,
// 8, 16 and 32 nodes; kagome L = 8 FP64: 10 ms for every level).  Chunks are therefore halved, down to one
// batch of nodes, while the level still has fewer chunks than `teams`, about twice the teams that the GPU
// holds at once; larger levels keep the coarse cut, whose partial sums cost least.  Right-hand sides and
// steps, coarse cut only against this rule, means over three states (the times of one case differ by up to a
// factor of two between states): square L = 3 11/4/3 FP64 24.4 -> 12.0 ms and 50/15/10 mixed 30.7 -> 17.1 ms,
// kagome L = 8 U(1)-DM three loops mixed 495 -> 304 ms, honeycomb L = 5 two-loop step mixed 222 -> 171 ms,
// pyrochlore L = 6 two loops mixed 332 -> 302 ms.
__host__ __device__ inline LevelCut cut_level(int nact, long long n, int qcap, int batch, int least, int teams) {
    LevelCut k;
    const int per0 = n <= (long long)kChunk * kMaxChunks ? (int)(n < kChunk ? n : kChunk) : (int)(n / kMaxChunks);
    k.coarse = (int)(n / per0);
    k.overflow = (long long)nact * k.coarse > qcap;
    k.nact = k.overflow ? qcap / k.coarse : nact;
    k.per = per0;
    k.chunks = k.coarse;
    // the upper half of the partial sums holds the fine chunks' sums of |node values| (fine_abs)
    const long long most = teams < qcap / 2 ? teams : qcap / 2;
    while (k.per > batch && 2ll * k.nact * k.chunks <= most) {
        k.per >>= 1;
        k.chunks <<= 1;
    }
    // U(1)-DM batches, whose nodes are evaluated one by one (least = 1), are halved further while an SM has
    // less than a block's teams; SU(2) batches share the overlap rows and the setup
    const long long few = most < teams / 8 ? most : teams / 8;
    while (k.per > least && 2ll * k.nact * k.chunks <= few) {
        k.per >>= 1;
        k.chunks <<= 1;
    }
    return k;
}

// Blocks of eval_kernel that work on nchunks chunks (npw teams per warp).  With fewer warps' worth of
// chunks than fill a block on every SM, one block per SM takes them in turn, so that the work spreads over
// the SMs' FP64 pipes and caches; otherwise the warps of a block take neighbouring chunks, which share
// vertex rows.
constexpr int kSMs = 152;
constexpr int kDeepWave = 10;  // levels of more than 2048 new nodes per subdomain
__host__ __device__ inline int eval_blocks(int nchunks, int npw) {
    const int units = (nchunks + npw - 1) / npw;
    const int full = (units + kWarps - 1) / kWarps;
    return full > kSMs ? full : (units < kSMs ? units : kSMs);
}

// per-site sums of |node values| of the fine chunks of a level (FP32 pass of the mixed path): vectors
// behind the at most qcap / 2 partial sums of such a level
__device__ __forceinline__ float* fine_abs(const WaveSpace& Wsp, int CNs) {
    return reinterpret_cast<float*>(Wsp.part + (size_t)(Wsp.qcap - Wsp.qcap / 2) * CNs);
}

// list subdomain sub for the next level, wave parity par
__device__ __forceinline__ void enqueue(WaveSpace& Wsp, int par, int sub) {
    const int a = atomicAdd(&Wsp.counters[2 + par], 1);
    (par ? Wsp.active[1] : Wsp.active[0])[a] = sub;
}

// the meshes of the node setup (shared memory): FP64 for the FP64 path, float-float pairs for the
// mixed path
template <typename R>
__device__ __forceinline__ auto setup_mesh(const PassArgs<R>& A, const unsigned char* smem) {
    if constexpr (sizeof(R) == 4) return mesh_view_ff(reinterpret_cast<const float*>(smem), A.L.Nsig, A.L.NO, A.L.Nn);
    else return mesh_view_d(reinterpret_cast<const double*>(smem), A.L.Nsig, A.L.NO, A.L.Nn);
}

template <typename R>
__device__ __forceinline__ void task_freqs(const PassArgs<R>& A, const MeshFF& M, const TaskInfo& ti, FF& W, FF& V,
                                           FF& VP) {
    const int oO = (ti.X == 1) ? M.Ot() : M.Os();
    const int on = (ti.X == 1) ? M.nt() : M.ns();
    const FF inf{INFINITY, 0.f};
    W = M.at(oO, ti.w1);
    V = (ti.kernel == 2 || ti.kernel == 4) ? M.at(on, ti.w2) : inf;
    VP = (ti.kernel == 3 || ti.kernel == 4) ? M.at(on, ti.w3) : inf;
}

template <typename R>
__device__ __forceinline__ void task_freqs(const PassArgs<R>& A, const MeshD& M, const TaskInfo& ti, double& W,
                                           double& V, double& VP) {
    const double* Om = M.x + (ti.X == 1 ? M.Ot() : M.Os());
    const double* nu = M.x + (ti.X == 1 ? M.nt() : M.ns());
    const double inf = INFINITY;
    W = Om[ti.w1];
    V = (ti.kernel == 2 || ti.kernel == 4) ? nu[ti.w2] : inf;
    VP = (ti.kernel == 3 || ti.kernel == 4) ? nu[ti.w3] : inf;
}

// shared-memory layout common to the wave kernels
template <typename R, int T, int C, int SPL>
struct SmemLayout {
    static constexpr int NPW = 32 / T;
    // t-channel staging per team: SU(2) both slots, the overlap sums and the local parts of the
    // whole batch, U(1)-DM one node
    __host__ __device__ static size_t tmp_per_team(int Ns) {
        return C == 2 ? (size_t)4 * Ns * t_site_stride<R, BatchOf<R, T, C, SPL>::NB>() + (size_t)4 * Ns * BatchOf<R, T, C, SPL>::NB
                      : (size_t)2 * C * Ns;
    }
    // the meshes of the node setup: float-float pairs and inverse spacings (mixed path) or FP64
    // values and inverse spacings, nm = Nsig + 2 NO + 2 Nn entries each (the float block ends with the
    // placement parameters of its meshes)
    __host__ __device__ static size_t mesh_bytes(int nm) {
        return sizeof(R) == 4 ? sizeof(float) * (3 * (size_t)nm + kMeshGuess) : 2 * sizeof(double) * (size_t)nm;
    }
    size_t mesh, teams, tmp, rows, total;
    __host__ __device__ SmemLayout(int Ns, int nm, long long R_rows, bool rows_in_smem) {
        mesh = 0;
        teams = (mesh_bytes(nm) + 15) & ~(size_t)15;
        tmp = (teams + sizeof(TeamScratch<R, T, C, SPL>) * kWarps * NPW + 15) & ~(size_t)15;  // 16-byte loads
        rows = tmp + ((sizeof(R) * (size_t)kWarps * NPW * tmp_per_team(Ns) + 15) & ~(size_t)15);
        total = rows + (rows_in_smem ? sizeof(unsigned) * (size_t)(R_rows + Ns + 1) : 0);
    }
};

template <typename R, int T, int SPL, int C>
__device__ __forceinline__ Team<R, T, SPL, C> make_team(const PassArgs<R>& A, unsigned char* smem,
                                                        const typename Team<R, T, SPL, C>::SetupMesh& M, int warp,
                                                        int team, int tl) {
    constexpr int NPW = 32 / T;
    const int Ns = A.L.Ns;
    SmemLayout<R, T, C, SPL> lay(Ns, A.L.Nsig + 2 * A.L.NO + 2 * A.L.Nn, A.rows_total, A.rows_in_smem);
    TeamScratch<R, T, C, SPL>* teams = reinterpret_cast<TeamScratch<R, T, C, SPL>*>(smem + lay.teams);
    R* tmp = reinterpret_cast<R*>(smem + lay.tmp) + (size_t)(warp * NPW + team) * lay.tmp_per_team(Ns);
    const unsigned* rows;
    const int* roff;
    if (A.rows_in_smem) {
        rows = reinterpret_cast<const unsigned*>(smem + lay.rows);
        roff = reinterpret_cast<const int*>(rows + A.rows_total);
    } else {
        rows = A.ov_rows;
        roff = A.ov_off;
    }
    Team<R, T, SPL, C> t{A, M, teams[warp * NPW + team], tmp, rows, roff, tl, {}, 0, 0};
#pragma unroll
    for (int k = 0; k < SPL; ++k) {
        const int i = tl + k * T;
        t.site_ex[k] = i < Ns ? ldg(A.exch + i) : 0;
    }
    return t;
}

template <typename R, int T, int C, int SPL>
__device__ __forceinline__ void load_common(const PassArgs<R>& A, unsigned char* smem) {
    const int nm = A.L.Nsig + 2 * A.L.NO + 2 * A.L.Nn;
    if constexpr (sizeof(R) == 4) {
        float* m = reinterpret_cast<float*>(smem);
        for (int k = threadIdx.x; k < 3 * nm + kMeshGuess; k += blockDim.x) m[k] = ldg(A.mesh_ff + k);
    } else {
        double* m = reinterpret_cast<double*>(smem);
        for (int k = threadIdx.x; k < 2 * nm; k += blockDim.x) m[k] = ldg(A.mesh + k);
    }
    if (A.rows_in_smem) {
        SmemLayout<R, T, C, SPL> lay(A.L.Ns, nm, A.rows_total, true);
        unsigned* rows = reinterpret_cast<unsigned*>(smem + lay.rows);
        for (long long k = threadIdx.x; k < A.rows_total; k += blockDim.x) rows[k] = ldg(A.ov_rows + k);
        int* roff = reinterpret_cast<int*>(rows + A.rows_total);
        for (int k = threadIdx.x; k <= A.L.Ns; k += blockDim.x) roff[k] = ldg(A.ov_off + k);
    }
    __syncthreads();
}

// subdomain range of job `job` of a task (flow_s.jl:29-36; quadrature.jl:84-139); false if empty
template <typename R>
__device__ __forceinline__ bool sub_range(const PassArgs<R>& A, const TaskInfo& ti, int job, double& lo, double& hi,
                                          double& sgn) {
    const double* mesh = A.mesh;
    const double* Om64 = mesh + A.L.Nsig + (ti.X == 1 ? A.L.NO + A.L.Nn : 0);
    const double* nu64 = Om64 + A.L.NO;
    const double ref = A.Lam + 0.5 * Om64[ti.w1];
    const double val = Om64[A.L.NO - 1] + nu64[A.L.Nn - 1];
    const int eval = A.eval;
    const int range = job / eval, sub = job % eval + 1;
    sgn = 1.0;
    if (range == 0 || range == 3) {
        const double a = 2.0 * ref, b = 1.0 * val;
        if (!(b > a)) return false;
        // ξ^k a with libm's pow, computed on the host: an end point at ±val sits on the jump
        // of the vertex read-out at Ω[end] + ν[end] and must round exactly like the reference
        const double* lb = A.log_bounds + (size_t)((ti.X == 1 ? A.L.NO : 0) + ti.w1) * (eval + 1);
        lo = lb[sub - 1];
        hi = lb[sub];
        sgn = range == 0 ? -1.0 : 1.0;
    } else {
        const double a = range == 1 ? -2.0 * ref : 0.0 * ref;
        const double b = range == 1 ? 0.0 * ref : 2.0 * ref;
        if (!(b > a)) return false;
        const double h = (b - a) / eval;
        lo = __dadd_rn(a, __dmul_rn((double)(sub - 1), h));
        hi = __dadd_rn(a, __dmul_rn((double)sub, h));
    }
    return true;
}

// Norms of a team's per-site values: x[q] is this lane's sum of squares of quantity q, on return the
// norm over the team's sites in every lane.  The lanes halve the quantities they carry at every step of the
// sum (7 to 9 FP64 additions instead of 6 log2 T), so each ends with one total and takes one square root for
// all quantities (an FP64 square root costs a warp as much as some fifteen additions).
constexpr int kNorms = 8;
template <int T>
__device__ __forceinline__ void team_norms(double x[kNorms]) {
    const int tl = threadIdx.x & (T - 1);
    int n = kNorms;
#pragma unroll
    for (int o = T / 2; o >= 1; o >>= 1) {
        if (n > 1) {
            n >>= 1;
            const bool up = (tl & o) != 0;
#pragma unroll
            for (int k = 0; k < kNorms / 2; ++k)
                if (k < n) {
                    const double send = up ? x[k] : x[k + n];
                    const double keep = up ? x[k + n] : x[k];
                    x[k] = keep + __shfl_xor_sync(kFull, send, o);
                }
        } else {
            x[0] += __shfl_xor_sync(kFull, x[0], o);
        }
    }
    // lane tl holds the quantity of its top three bits
    const double r = sqrt(x[0]);
#pragma unroll
    for (int q = 0; q < kNorms; ++q) x[q] = __shfl_sync(kFull, r, q * (T / kNorms), T);
}

// this lane's sums of squares of the convergence test of simps!: x[0] the Richardson value R, x[1] the new
// Simpson sum S, x[2] R - S
template <int SPL, int C>
__device__ __forceinline__ void simps_squares(const double s_old[C][SPL], const double s_new[C][SPL], double* x) {
    x[0] = x[1] = x[2] = 0.0;
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
        for (int k = 0; k < SPL; ++k) {
            const double rich = s_old[c][k] * (-1.0 / 15.0) + (16.0 / 15.0) * s_new[c][k];
            const double dd = rich - s_new[c][k];
            x[0] += rich * rich;
            x[1] += s_new[c][k] * s_new[c][k];
            x[2] += dd * dd;
        }
}

// the reference's convergence test of simps!, from the norms of R, S and R - S; 1 when done
__device__ __forceinline__ int simps_test(double nr, double ns, double adiff, long long n, double atol, double rtol) {
    const double rdiff = adiff / fmax(nr, ns);
    // a non-finite integrand stops refining at once (the reference would refine it to n > 2^20);
    // the result's finite check then reports it
    return (adiff < atol || rdiff < rtol || 2 * n > (1ll << 20) || !isfinite(adiff)) ? 1 : 0;
}

// The same test on the FP32 pass of the mixed path: 1 done, 0 next level, 2 hand the subdomain to
// the FP64 pass.  sa_old / sa_new bound the norms of the Simpson sums taken over |node values|
// with |weights|; with node values rounded by at most eps of their magnitude the FP64 sums lie
// within eps sa of the FP32 ones, so when the test is closer to one of its bounds than that
// margin the FP64 evaluation of the same nodes could decide the other way, and the subdomain is
// evaluated again in FP64 from its first level (all its decisions then are the FP64 path's).
__device__ __forceinline__ int simps_decide(double nr, double ns, double adiff, long long n, double atol, double rtol,
                                            double eps, double sa_old, double sa_new) {
    const double den = fmax(nr, ns);
    if (2 * n > (1ll << 20) || !isfinite(adiff)) return 1;
    const int done = (adiff < atol || adiff / den < rtol) ? 1 : 0;
    const double E = eps * (sa_new + sa_old) / 15.0;          // |Δ64 - Δ32|
    const double Es = eps * (16.0 * sa_new + sa_old) / 15.0;  // change of the norms in the bound
    const bool can_done = adiff - E < atol || adiff - E < rtol * (den + Es);
    const bool can_go = adiff + E >= atol && adiff + E >= rtol * fmax(den - Es, 0.0);
    return (can_done && can_go) ? 2 : done;
}

// norm of a team's per-site values
template <int T, int SPL, int C>
__device__ __forceinline__ double team_norm(const double v[C][SPL]) {
    double ss = 0.0;
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
        for (int k = 0; k < SPL; ++k) ss += v[c][k] * v[c][k];
    return sqrt(in_team_sum<T>(ss));
}

// hand a subdomain from the FP32 pass to the FP64 pass (team lane 0)
__device__ __forceinline__ void hand_off(WaveSpace& Wsp, int sub) {
    Wsp.esc[atomicAdd(&Wsp.counters[5], 1)] = sub;
}

// ---- wave 0: first five nodes of every subdomain, boundary nodes, first test ----
// (blocks per SM that SU(2) kernels with at most two sites per lane are held to: FP32 three, four and five
// blocks 226, 217 and 222 ms summed over two honeycomb L = 5 steps; FP64 with two sites per lane three, four
// blocks 99.0, 100.0 ms on pyrochlore L = 6, with one site 33.8, 33.3 ms on a honeycomb L = 4 parquet solve)
template <typename R, int SPL, int C>
constexpr int wave0_min_blocks() { return C == 2 && SPL <= 2 ? (sizeof(R) == 4 || SPL == 1 ? 4 : 3) : 1; }

template <typename R, int T, int SPL, int C>
__global__ void __launch_bounds__(kWarps * 32, wave0_min_blocks<R, SPL, C>()) wave0_kernel(PassArgs<R> A, WaveSpace Wsp) {
    constexpr int NPW = 32 / T;
    extern __shared__ __align__(16) unsigned char smem[];
    load_common<R, T, C, SPL>(A, smem);
    const auto M = setup_mesh(A, smem);  // staged in shared memory by load_common
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int team = lane / T, tl = lane % T;
    Team<R, T, SPL, C> tm = make_team<R, T, SPL, C>(A, smem, M, warp, team, tl);
    const int Ns = A.L.Ns;
    const int jobs = 4 * A.eval + 1;
    const long long nwarps = (long long)gridDim.x * kWarps;
    constexpr int NB = BatchOf<R, T, C, SPL>::NB;
    // the FP64 pass of the mixed path starts only the subdomains the FP32 pass handed to it
    const int nwork = A.esc_mode == 2 ? Wsp.counters[5] : Wsp.nsub;
    for (long long base = ((long long)blockIdx.x * kWarps + warp) * NPW; base < nwork; base += nwarps * NPW) {
        const bool valid = base + team < nwork;
        const int sub = !valid ? 0 : (A.esc_mode == 2 ? Wsp.esc[base + team] : (int)(base + team));
        TaskInfo ti{0, 1, 0, 0, 0};
        int job = 0, cnt = 0;
        double x[8], lo = 0, hi = 0, sgn = 1;
        double c0 = 0, c1 = 0;
        bool boundary = false;
        if (valid) {
            ti = task_of(A, sub, jobs);
            job = sub % jobs;
            if (job == 4 * A.eval) {
                const double* Om64 = A.mesh + A.L.Nsig + (ti.X == 1 ? A.L.NO + A.L.Nn : 0);
                const double val = Om64[A.L.NO - 1] + Om64[A.L.NO + A.L.Nn - 1];
                x[0] = -val;
                x[1] = val;
                c0 = A.corrs[0 + 2 * (ti.X + 3 * ti.w1)];
                c1 = A.corrs[1 + 2 * (ti.X + 3 * ti.w1)];
                cnt = 2;
                boundary = true;
            } else if (sub_range(A, ti, job, lo, hi, sgn)) {
                const double mid = 0.5 * (lo + hi);
                const double h = 0.5 * (hi - lo) / 2.0;
                x[0] = sgn * lo;
                x[1] = sgn * __dadd_rn(lo, __dmul_rn(1.0, h));
                x[2] = sgn * mid;
                x[3] = sgn * __dadd_rn(lo, __dmul_rn(3.0, h));
                x[4] = sgn * hi;
                cnt = 5;
            }
        }
        typename Team<R, T, SPL, C>::SetupT W(0.0), V(0.0), VP(0.0);
        if (valid) task_freqs(A, M, ti, W, V, VP);
        // simps!: 3-point sum s_old, 5-point sum s_new via residual! with n = 2 from the new nodes' sum f and
        // the middle node, Richardson test; boundary nodes are summed with their corrections into s_old.
        // FP32 kernels add a node's values as they come: kept until the end, five nodes' values sat in local
        // memory (two honeycomb L = 5 steps 235 -> 218 ms with this and one square root per test); the FP64
        // kernels, bound by their FP64 operations, measured the same either way and keep them.
        const bool simpson = valid && !boundary && cnt == 5;
        const double we = 1.0 * (hi - lo) / 6.0, wm = 2.0 * (hi - lo) / 3.0;
        constexpr int CA = sizeof(R) == 4 ? C : 1;  // sums over |node values|: FP32 pass of the mixed path
        double s_old[C][SPL], f_new[C][SPL], a_old[CA][SPL], a_f[CA][SPL];
        R g2[C][SPL], g5[sizeof(R) == 8 ? 5 : 1][C][SPL];
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                s_old[c][k] = f_new[c][k] = 0.0;
                g2[c][k] = (R)0;
                if (c < CA) a_old[c][k] = a_f[c][k] = 0.0;
            }
        // all teams of the warp evaluate together (cnt = 0 for idle teams), NB nodes at a time
#pragma unroll 1
        for (int b = 0; b < 5; b += NB) {
            const int nb = max(0, min(NB, cnt - b));
            for (int j = tl; j < nb; j += T) tm.ts.node[j].set(x[b + j]);
            __syncwarp();
            auto add = [&](int j, const R (&gv)[C][SPL]) {
                const int q = b + j;
                const bool mid = !boundary && (q & 1);
                const double w = boundary ? (q == 0 ? c0 : c1) : (q == 2 ? wm : we);
#pragma unroll
                for (int c = 0; c < C; ++c)
#pragma unroll
                    for (int k = 0; k < SPL; ++k) {
                        if constexpr (sizeof(R) == 4) {
                            const double g = (double)gv[c][k];
                            if (mid) {
                                f_new[c][k] += g;
                                a_f[c][k] += fabs(g);
                            } else {
                                s_old[c][k] += w * g;
                                a_old[c][k] += w * fabs(g);
                            }
                            if (q == 2) g2[c][k] = gv[c][k];
                        } else {
                            g5[q][c][k] = gv[c][k];
                        }
                    }
            };
            tm.eval(ti, W, V, VP, nb, add);
        }
        const double h = 0.5 * (hi - lo) / 2.0;
        const double wn = 4.0 * h / 3.0, wo = -2.0 * h / 3.0;
        double s_new[C][SPL], nx[kNorms];
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                if constexpr (sizeof(R) == 8) {
                    s_old[c][k] = s_new[c][k] = f_new[c][k] = 0.0;
                    if (!simpson) continue;
                    s_old[c][k] = we * g5[0][c][k];
                    s_old[c][k] += wm * g5[2][c][k];
                    s_old[c][k] += we * g5[4][c][k];
                    f_new[c][k] = g5[1][c][k] + g5[3][c][k];
                    s_new[c][k] = 0.5 * s_old[c][k] + wn * f_new[c][k] + wo * g5[2][c][k];
                } else {
                    s_new[c][k] = 0.5 * s_old[c][k] + wn * f_new[c][k] + wo * (double)g2[c][k];
                }
            }
        // every lane takes part in the test's team reductions
        int done;
        double sa_new = 0.0, fab = 0.0;
        simps_squares<SPL, C>(s_old, s_new, nx);
        nx[3] = nx[4] = nx[5] = nx[6] = nx[7] = 0.0;
        if (sizeof(R) == 4 && A.esc_mode == 1) {
#pragma unroll
            for (int c = 0; c < CA; ++c)
#pragma unroll
                for (int k = 0; k < SPL; ++k) {
                    const double a_new = 0.5 * a_old[c][k] + fabs(wn) * a_f[c][k] + fabs(wo) * fabs((double)g2[c][k]);
                    nx[3] += a_old[c][k] * a_old[c][k];
                    nx[4] += a_new * a_new;
                    nx[5] += a_f[c][k] * a_f[c][k];
                }
            team_norms<T>(nx);
            sa_new = nx[4];
            fab = nx[5];
            done = simps_decide(nx[0], nx[1], nx[2], 2, A.atol, A.rtol, A.esc_eps, nx[3], sa_new);
        } else {
            team_norms<T>(nx);
            done = simps_test(nx[0], nx[1], nx[2], 2, A.atol, A.rtol);
        }
        if (!valid) continue;
        if (simpson && done == 2) {
            if (tl == 0) hand_off(Wsp, sub);
            continue;
        }
        double* sA = Wsp.stA + (size_t)sub * C * Ns;
        double* sB = Wsp.stB + (size_t)sub * C * Ns;
        if (!simpson) {
            // boundary corrections (two nodes weighted by corrs) or an empty range
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int k = 0; k < SPL; ++k) {
                    const int i = tl + k * T;
                    if (i >= Ns) continue;
                    if constexpr (sizeof(R) == 4) sA[c * Ns + i] = boundary ? s_old[c][k] : 0.0;
                    else sA[c * Ns + i] = boundary ? c0 * g5[0][c][k] + c1 * g5[1][c][k] : 0.0;
                }
            continue;
        }
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                const int i = tl + k * T;
                if (i >= Ns) continue;
                if (done) {
                    sA[c * Ns + i] = (s_old[c][k] * (-1.0 / 15.0) + (16.0 / 15.0) * s_new[c][k] - s_new[c][k]) + s_new[c][k];
                } else {
                    sA[c * Ns + i] = s_new[c][k];
                    sB[c * Ns + i] = f_new[c][k];
                }
            }
        if (tl == 0) {
            SubRec& S = Wsp.subs[sub];
            S.lo = lo;
            S.hi = hi;
            S.sgn = sgn;
            S.sa = sa_new;
            S.fab = fab;
            if (!done) enqueue(Wsp, 1, sub);
        }
    }
    tm.count_nodes();
}

// ---- wave k >= 1: evaluate queued chunks, one partial node sum per chunk ----
// (FP32 kernels: SU(2) teams of 8 and 32 lanes with one site per lane held to 102 registers, five blocks of 128
// threads per SM (four, five and six blocks 11.0, 10.5 and 10.8 ms summed over two square L = 3 right-hand
// sides, 8 lanes); those of 16 lanes, whose blocks of 48 to 59 KB fit four times at most, and those with two
// sites per lane to 128, four blocks (the latter's gathers spill beyond that); wider lanes and U(1)-DM entries,
// whose gathers spill at 128, to 168, three blocks)
template <typename R, int T, int SPL, int C>
constexpr int eval_min_blocks() {
    return sizeof(R) == 4 ? (C == 2 && SPL <= 2 ? (SPL == 1 && T != 16 ? 5 : 4) : 3) : 1;
}

template <typename R, int T, int SPL, int C>
__global__ void __launch_bounds__(kWarps * 32, eval_min_blocks<R, T, SPL, C>())
    eval_kernel(PassArgs<R> A, WaveSpace Wsp, int par, long long n) {
    constexpr int NPW = 32 / T;
    constexpr int NB = BatchOf<R, T, C, SPL>::NB;
    extern __shared__ __align__(16) unsigned char smem[];
    const int nactive = Wsp.counters[2 + par];
    const LevelCut K = cut_level(nactive, n, Wsp.qcap, base_batch<T, C, SPL>(),
                                 C == 6 ? 1 : base_batch<T, C, SPL>(), Wsp.teams);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // the next level's list starts empty (this wave's decide_kernel fills it)
        Wsp.counters[2 + (par ^ 1)] = 0;
        // a level whose coarse chunks exceed the queue's capacity is reported and cut short
        if (K.overflow) Wsp.counters[4] = 1;
    }
    const int nchunks = K.nact * K.chunks;
    // blocks without a chunk leave before staging the meshes and rows
    const int nblocks = min((int)gridDim.x, eval_blocks(nchunks, NPW));
    if ((int)blockIdx.x >= nblocks) return;
    load_common<R, T, C, SPL>(A, smem);
    const auto M = setup_mesh(A, smem);  // staged in shared memory by load_common
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int team = lane / T, tl = lane % T;
    Team<R, T, SPL, C> tm = make_team<R, T, SPL, C>(A, smem, M, warp, team, tl);
    tm.odd_first = SPL == 3;
    const int Ns = A.L.Ns;
    const int jobs = 4 * A.eval + 1;
    const int* active = par ? Wsp.active[1] : Wsp.active[0];
    const bool spread = nblocks <= kSMs;  // unit of NPW chunks of this warp: in turn, or a block's warps together
    const long long nwarps = (long long)nblocks * kWarps;
    for (long long base = (long long)(spread ? warp * nblocks + blockIdx.x : blockIdx.x * kWarps + warp) * NPW;
         base < nchunks; base += nwarps * NPW) {
        const int chunk = (int)(base + team);
        const bool valid = chunk < nchunks;
        int first = 0;  // first new node of the chunk
        TaskInfo ti{0, 1, 0, 0, 0};
        double lo = 0, h = 0, sgn = 1;
        typename Team<R, T, SPL, C>::SetupT W(0.0), V(0.0), VP(0.0);
        if (valid) {
            const int a = chunk / K.chunks;
            const int sub = active[a];
            first = (chunk - a * K.chunks) * K.per;
            const SubRec S = Wsp.subs[sub];
            ti = task_of(A, sub, jobs);
            task_freqs(A, M, ti, W, V, VP);
            lo = S.lo;
            sgn = S.sgn;
            h = 0.5 * (S.hi - S.lo) / (double)n;
        }
        const int cnt = valid ? K.per : 0;
        Acc<R> acc[C][SPL];
        R aab[C][SPL];  // FP32 pass of the mixed path: sums of |node values|
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                acc[c][k] = Acc<R>{(R)0, (R)0};
                aab[c][k] = (R)0;
            }
        // each node's values go straight into the chunk's compensated sums, in node order
        auto add = [&](int, const R (&gv)[C][SPL]) {
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int k = 0; k < SPL; ++k) {
                    acc_add(acc[c][k], gv[c][k]);
                    if constexpr (sizeof(R) == 4) aab[c][k] += fabsf(gv[c][k]);
                }
        };
#pragma unroll 1
        for (int b = 0; b < K.per; b += NB) {
            const int nb = max(0, min(NB, cnt - b));
            if (tl < nb) {
                const int nd = first + b + tl;  // 0-based new node of the level
                tm.ts.node[tl].set(sgn * __dadd_rn(lo, __dmul_rn(2.0 * (double)(nd + 1) - 1.0, h)));
            }
            __syncwarp();
            tm.eval(ti, W, V, VP, nb, add);
        }
        if constexpr (sizeof(R) == 4) {
            if (A.esc_mode == 1 && K.chunks == K.coarse) {
                double ad[C][SPL];
#pragma unroll
                for (int c = 0; c < C; ++c)
#pragma unroll
                    for (int k = 0; k < SPL; ++k) ad[c][k] = (double)aab[c][k];
                const double nrm = team_norm<T, SPL, C>(ad);  // every lane of the warp takes part
                if (valid && tl == 0) Wsp.part_abs[chunk] = nrm;
            }
        }
        if (!valid) continue;
        double* P = Wsp.part + (size_t)chunk * C * Ns;
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                const int i = tl + k * T;
                if (i < Ns) P[c * Ns + i] = (double)acc[c][k].s + (double)acc[c][k].c;
            }
        if constexpr (sizeof(R) == 4) {
            if (A.esc_mode == 1 && K.chunks != K.coarse) {
                // the coarse chunk's norm is formed from its fine chunks' sums by decide_kernel
                float* Q = fine_abs(Wsp, C * Ns) + (size_t)chunk * C * Ns;
#pragma unroll
                for (int c = 0; c < C; ++c)
#pragma unroll
                    for (int k = 0; k < SPL; ++k) {
                        const int i = tl + k * T;
                        if (i < Ns) Q[c * Ns + i] = aab[c][k];
                    }
            }
        }
    }
    tm.count_nodes();
}

// ---- wave k >= 1: per subdomain, next Simpson sum, test, result or next level ----
// One team per subdomain, or, for subdomains of many chunks, all teams of a block: each sums a part of the
// chunks and the first team forms the total from their sums in order.
constexpr int kDecideSplit = 64;  // chunks per subdomain from which a block's teams share them

template <int T, int SPL, int C>
__global__ void __launch_bounds__(kWarps * 32) decide_kernel(WaveSpace Wsp, int Ns, double atol, double rtol, int par,
                                                             long long n, int esc_mode, double esc_eps) {
    constexpr int NPW = 32 / T;
    constexpr int TPB = kWarps * NPW;  // teams per block
    static_assert(kDecideSplit >= TPB, "every team of a block has a chunk");
    __shared__ double sh_f[TPB - 1][C * SPL * T];  // sums of all teams but the first
    __shared__ double sh_a[TPB - 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int team = lane / T, tl = lane % T;
    const int bteam = warp * NPW + team;
    const LevelCut K = cut_level(Wsp.counters[2 + par], n, Wsp.qcap, base_batch<T, C, SPL>(),
                                 C == 6 ? 1 : base_batch<T, C, SPL>(), Wsp.teams);
    const int* active = par ? Wsp.active[1] : Wsp.active[0];
    const bool split = K.chunks >= kDecideSplit;
    const int G = split ? TPB : 1, g = split ? bteam : 0;
    const int step = split ? gridDim.x : gridDim.x * TPB;
    const int q0 = K.chunks / G * g, q1 = q0 + K.chunks / G;
    // coarse chunks of this team's share of the |node value| norms
    const int ca = (K.coarse + G - 1) / G, c0 = min(K.coarse, g * ca), c1 = min(K.coarse, c0 + ca);
    for (int base = split ? blockIdx.x : blockIdx.x * TPB + warp * NPW; base < K.nact; base += step) {
        const int a = split ? base : base + team;
        const bool valid = a < K.nact;
        const int sub = valid ? active[a] : 0;
        SubRec S;
        if (valid) S = Wsp.subs[sub];
        else S.lo = 0, S.hi = 0, S.sa = 0, S.fab = 0;
        double* sA = Wsp.stA + (size_t)sub * C * Ns;
        double* sB = Wsp.stB + (size_t)sub * C * Ns;
        double s_old[C][SPL], s_new[C][SPL], f_new[C][SPL];
        const double h = 0.5 * (S.hi - S.lo) / (double)n;
        const double wn = 4.0 * h / 3.0, wo = -2.0 * h / 3.0;
        const double* part = Wsp.part + (size_t)(valid ? a : 0) * K.chunks * C * Ns;
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                const int i = tl + k * T;
                f_new[c][k] = 0.0;
                if (!valid || i >= Ns) continue;
                double f = 0.0;
#pragma unroll 4
                for (int q = q0; q < q1; ++q) f += part[(size_t)q * C * Ns + c * Ns + i];
                f_new[c][k] = f;
            }
        double fa_new = 0.0;
        if (esc_mode == 1 && K.chunks == K.coarse) {
            if (valid)
                for (int q = q0; q < q1; ++q) fa_new += Wsp.part_abs[(size_t)a * K.chunks + q];  // triangle bound
        } else if (esc_mode == 1) {
            // the norms of the coarse chunks, from the sums of their fine chunks: up to the FP32 rounding of
            // these sums the bound does not depend on how a level was cut, so a finer cut can hand off another
            // subdomain only where the bound meets the margin within that rounding
            const int r = K.chunks / K.coarse;
            const float* Q = fine_abs(Wsp, C * Ns) + (size_t)(valid ? a : 0) * K.chunks * C * Ns;
            for (int cc = 0; cc < ca; ++cc) {
                const int q = c0 + cc;
                double ad[C][SPL];
#pragma unroll
                for (int c = 0; c < C; ++c)
#pragma unroll
                    for (int k = 0; k < SPL; ++k) {
                        const int i = tl + k * T;
                        float f = 0.f;
                        if (valid && i < Ns && q < c1)
                            for (int e = 0; e < r; ++e) f += Q[(size_t)(q * r + e) * C * Ns + c * Ns + i];
                        ad[c][k] = (double)f;
                    }
                fa_new += team_norm<T, SPL, C>(ad);  // every lane of the warp takes part
            }
        }
        if (split) {
            __syncthreads();  // the sums of the previous subdomain have been read
            if (bteam > 0) {
#pragma unroll
                for (int c = 0; c < C; ++c)
#pragma unroll
                    for (int k = 0; k < SPL; ++k) sh_f[bteam - 1][(c * SPL + k) * T + tl] = f_new[c][k];
                if (tl == 0) sh_a[bteam - 1] = fa_new;
            }
            __syncthreads();
            if (warp > 0) continue;
            // the first team adds them in order (the others of its warp only take part in its shuffles)
#pragma unroll
            for (int e = 0; e < TPB - 1; ++e) {
                fa_new += sh_a[e];
#pragma unroll
                for (int c = 0; c < C; ++c)
#pragma unroll
                    for (int k = 0; k < SPL; ++k) f_new[c][k] += sh_f[e][(c * SPL + k) * T + tl];
            }
        }
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                const int i = tl + k * T;
                s_old[c][k] = s_new[c][k] = 0.0;
                if (!valid || i >= Ns) continue;
                s_old[c][k] = sA[c * Ns + i];
                s_new[c][k] = 0.5 * s_old[c][k] + wn * f_new[c][k] + wo * sB[c * Ns + i];
            }
        int done;
        double sa_new = 0.0, nx[kNorms];
        simps_squares<SPL, C>(s_old, s_new, nx);
        nx[3] = nx[4] = nx[5] = nx[6] = nx[7] = 0.0;
        team_norms<T>(nx);
        if (esc_mode == 1) {
            const double sa_old = S.sa;
            sa_new = 0.5 * sa_old + fabs(wn) * fa_new + fabs(wo) * S.fab;
            done = simps_decide(nx[0], nx[1], nx[2], n, atol, rtol, esc_eps, sa_old, sa_new);
        } else {
            done = simps_test(nx[0], nx[1], nx[2], n, atol, rtol);
        }
        if (!valid || (split && team > 0)) continue;
        if (done == 2) {
            if (tl == 0) hand_off(Wsp, sub);
            continue;
        }
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int k = 0; k < SPL; ++k) {
                const int i = tl + k * T;
                if (i >= Ns) continue;
                if (done) {
                    sA[c * Ns + i] = (s_old[c][k] * (-1.0 / 15.0) + (16.0 / 15.0) * s_new[c][k] - s_new[c][k]) + s_new[c][k];
                } else {
                    sA[c * Ns + i] = s_new[c][k];
                    sB[c * Ns + i] = f_new[c][k];
                }
            }
        if (tl == 0 && !done) {
            Wsp.subs[sub].sa = sa_new;
            Wsp.subs[sub].fab = fa_new;
            enqueue(Wsp, par ^ 1, sub);
        }
    }
}

// ---- sum each task's subdomain results (range order, boundary last) into the output ----
template <typename R, int C>
__global__ void reduce_kernel(PassArgs<R> A, WaveSpace Wsp) {
    const int ct = blockIdx.x;  // channel task
    const int jobs = 4 * A.eval + 1;
    const int Ns = A.L.Ns;
    const TaskInfo ti = task_of(A, ct * jobs, jobs);
    const Layout& L = A.L;
    int64_t off;
    switch (ti.kernel) {
        case 1: off = (int64_t)Ns * ti.w1; break;
        case 2: off = (int64_t)Ns * (ti.w1 + (int64_t)L.NO * ti.w2); break;
        case 3: off = (int64_t)Ns * (ti.w1 + (int64_t)L.NO * ti.w3); break;
        default: off = (int64_t)Ns * (ti.w1 + (int64_t)L.NO * (ti.w2 + (int64_t)L.Nn * ti.w3)); break;
    }
    for (int e = threadIdx.x; e < C * Ns; e += blockDim.x) {
        const int c = e / Ns, i = e % Ns;
        double s = 0.0;
        for (int j = 0; j < jobs; ++j) s += Wsp.stA[((size_t)ct * jobs + j) * C * Ns + c * Ns + i];
        A.out[L.qbase(c, ti.X, ti.kernel - 1) + off + i] = s;
    }
}

// a pass whose chunk queue overflowed reports it in the call's status word (bit 3)
static __global__ void wave_status_kernel(const int* counters, int* status) {
    if (threadIdx.x == 0 && counters[4]) atomicOr(status, 8);
}

// Raise a kernel's dynamic shared-memory limit to the most a block may use, once per process: the
// attribute is process-wide, and contexts of different sizes launch the same kernel from several
// host threads (coupling sweeps), so a per-launch value could be lowered under another thread's
// launch.  Each launch still asks for its own size.
template <auto K>
inline cudaError_t allow_max_dynamic_smem() {
    static const cudaError_t e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    return e;
}

// Whether a block's overlap rows are staged in shared memory (mode 1 never, 2 where they fit at all): by
// default only while the FP32 eval kernel's register-bound number of blocks (three for FP64) still fits on an
// SM, 228 KB less 1 KB per block; a row word is read once per batch of nodes, so from L1 it costs little.
// FP32 teams of 16 lanes, whose batch scratch alone leaves three or four blocks, stage their rows while that
// costs none of them: right-hand sides on 11 to 16 sites run 1 to 3 % faster than with a register cap for
// five blocks and the rows in L1 (honeycomb L = 5 12.68 -> 12.29 ms, square L = 6 17.36 -> 16.96 ms, cubic
// L = 5 19.34 -> 18.88 ms).  Their FP64 blocks of 73 to 91 KB don't: two or three fit either way, and staged
// rows changed 11 to 16 sites by under 1 % and kagome L = 4 (13 sites) from 25.1 to 26.0 ms.
template <typename R, int T, int C, int SPL>
inline bool stage_rows(int Ns, int nm, long long rows, int mode) {
    if (mode == 1) return false;
    const size_t staged = SmemLayout<R, T, C, SPL>(Ns, nm, rows, true).total;
    if (mode == 2) return staged <= (size_t)227 * 1024;
    int blocks = sizeof(R) == 4 ? eval_min_blocks<R, T, SPL, C>() : 3;
    if (sizeof(R) == 4 && BatchOf<R, T, C, SPL>::twice)
        blocks = std::min(blocks, (int)((size_t)228 * 1024 / (SmemLayout<R, T, C, SPL>(Ns, nm, rows, false).total + 1024)));
    return staged <= (size_t)(228 / blocks - 1) * 1024;
}

// team width T = lanes per node batch, SPL = sites per lane
template <typename R, int C>
struct PassLauncher {
    template <int T, int SPL>
    static cudaError_t run(const PassArgs<R>& a0, WaveSpace& Wsp, int* h_counters, cudaStream_t st, int grid_cap) {
        PassArgs<R> a = a0;
        a.pc = prop_const(a.Lam);
        const int nm = a.L.Nsig + 2 * a.L.NO + 2 * a.L.Nn;
        a.rows_in_smem = stage_rows<R, T, C, SPL>(a.L.Ns, nm, a.rows_total, a.rows_mode);
        SmemLayout<R, T, C, SPL> lay(a.L.Ns, nm, a.rows_total, a.rows_in_smem);
        const size_t smem = lay.total;
        if (smem > (size_t)227 * 1024) return cudaErrorInvalidConfiguration;
        cudaError_t e;
        if ((e = allow_max_dynamic_smem<wave0_kernel<R, T, SPL, C>>())) return e;
        if ((e = allow_max_dynamic_smem<eval_kernel<R, T, SPL, C>>())) return e;
        constexpr int NPW = 32 / T;
        const int teams_per_block = kWarps * NPW;
        // the FP64 pass of the mixed path keeps the count of handed subdomains (counters[5])
        if ((e = cudaMemsetAsync(Wsp.counters, 0, sizeof(int) * (a.esc_mode == 2 ? 5 : 6), st))) return e;
        Wsp.teams = 2 * 4 * kSMs * teams_per_block;  // twice the teams of four blocks per SM
        int g0 = (Wsp.nsub + teams_per_block - 1) / teams_per_block;
        // h_counters[7] counts the kernels this pass launches
        wave0_kernel<R, T, SPL, C><<<g0 < grid_cap ? g0 : grid_cap, kWarps * 32, smem, st>>>(a, Wsp);
        ++h_counters[7];
        if ((e = cudaGetLastError())) return e;
        if (a.async_waves) {
            // device-driven levels: every wave reads its chunk and subdomain counts from the device,
            // idle blocks leave at once, and no host round trip separates the waves (the deepest
            // level the reference allows, n > 2^20 new nodes, is reached by wave 20)
            const int gd = std::max(1, std::min(grid_cap, (Wsp.nsub + teams_per_block - 1) / teams_per_block));
            int par = 1;
            for (int wave = 1; wave <= 21; ++wave) {
                // most states end before the deep levels, whose subdomains are few: smaller grids, which come and
                // go in half the time (a block takes several chunks where there are more)
                const bool deep = wave > kDeepWave;
                eval_kernel<R, T, SPL, C><<<deep ? std::min(grid_cap, 8 * kSMs) : grid_cap, kWarps * 32, smem, st>>>(
                    a, Wsp, par, 2ll << wave);
                h_counters[7] += 2;
                if ((e = cudaGetLastError())) return e;
                decide_kernel<T, SPL, C><<<deep ? std::min(gd, 2 * kSMs) : gd, kWarps * 32, 0, st>>>(Wsp, a.L.Ns, a.atol, a.rtol, par, 2ll << wave,
                                                                     a.esc_mode, a.esc_eps);
                if ((e = cudaGetLastError())) return e;
                par ^= 1;
            }
            wave_status_kernel<<<1, 32, 0, st>>>(Wsp.counters, a.status);
            ++h_counters[7];
            if ((e = cudaGetLastError())) return e;
            if (a.esc_mode == 1) return cudaSuccess;  // the FP64 pass finishes and reduces
            reduce_kernel<R, C><<<a.ntasks * a.nchan, 128, 0, st>>>(a, Wsp);
            ++h_counters[7];
            return cudaGetLastError();
        }
        int par = 1;
        for (int wave = 1; wave <= 21; ++wave) {
            if ((e = cudaMemcpyAsync(h_counters, Wsp.counters, sizeof(int) * 5, cudaMemcpyDeviceToHost, st))) return e;
            if ((e = cudaStreamSynchronize(st))) return e;
            const int nact = h_counters[2 + par];
            if (nact == 0) break;
            const LevelCut K = cut_level(nact, 2ll << wave, Wsp.qcap, base_batch<T, C, SPL>(),
                                 C == 6 ? 1 : base_batch<T, C, SPL>(), Wsp.teams);
            if (K.overflow) {  // chunk queue overflow
                h_counters[4] = 1;
                return cudaErrorLaunchOutOfResources;
            }
            const int ge = eval_blocks(K.nact * K.chunks, NPW);
            eval_kernel<R, T, SPL, C><<<ge < grid_cap ? ge : grid_cap, kWarps * 32, smem, st>>>(a, Wsp, par, 2ll << wave);
            h_counters[7] += 2;
            if ((e = cudaGetLastError())) return e;
            int gd = (nact + teams_per_block - 1) / teams_per_block;
            decide_kernel<T, SPL, C><<<gd < grid_cap ? gd : grid_cap, kWarps * 32, 0, st>>>(Wsp, a.L.Ns, a.atol, a.rtol,
                                                                                           par, 2ll << wave, a.esc_mode,
                                                                                           a.esc_eps);
            if ((e = cudaGetLastError())) return e;
            par ^= 1;
        }
        if (a.esc_mode == 1) return cudaSuccess;  // the FP64 pass finishes and reduces
        reduce_kernel<R, C><<<a.ntasks * a.nchan, 128, 0, st>>>(a, Wsp);
        ++h_counters[7];
        return cudaGetLastError();
    }
};

// one team shape of one precision and component count; instantiated explicitly in
// pffrg_shapes.cu (one object per group of shapes, so the kernels compile in parallel)
template <typename R, int C, int T, int SPL>
cudaError_t run_shape(const PassArgs<R>& a, WaveSpace& Wsp, int* h_counters, cudaStream_t st, int grid_cap) {
    return PassLauncher<R, C>::template run<T, SPL>(a, Wsp, h_counters, st, grid_cap);
}

// the team shapes built: lanes per node batch x sites per lane
#define PFFRG_TEAM_SHAPES(X) X(8, 1) X(16, 1) X(32, 1) X(16, 3) X(16, 4) X(32, 2) X(32, 3) X(32, 4) X(32, 8)

// the default shape for Ns sites: the narrowest team whose lanes hold at most two sites (up to 64
// sites; measured on the pyrochlore L = 6 two-loop state, 48 sites: 32x2 403 ms, 16x3 460 ms,
// 16x4 511 ms), beyond that 32-lane teams with the fewest sites per lane that cover them (32x3 against
// 32x4: kagome L = 8 U(1)-DM three-loop state, 82 sites, mixed 1445 vs 1823 ms, FP64 4935 vs 5506 ms;
// pyrochlore L = 7 one-loop, 70 sites, mixed 455 vs 502 ms, FP64 2312 vs 2432 ms)
__host__ __device__ inline void default_team_shape(int Ns, int& T, int& SPL) {
    if (Ns <= 8) T = 8, SPL = 1;
    else if (Ns <= 16) T = 16, SPL = 1;
    else if (Ns <= 32) T = 32, SPL = 1;
    else if (Ns <= 64) T = 32, SPL = 2;
    else if (Ns <= 96) T = 32, SPL = 3;
    else if (Ns <= 128) T = 32, SPL = 4;
    else T = 32, SPL = 8;
}

template <typename R, int C>
cudaError_t launch_pass_impl(const PassArgs<R>& a, WaveSpace& Wsp, int* h_counters, cudaStream_t st) {
    const int Ns = a.L.Ns;
    if (a.ntasks == 0) return cudaSuccess;
    if (Ns > 256) return cudaErrorInvalidValue;
    const int cap = 152 * 32;
    int T, S;
    default_team_shape(Ns, T, S);
    if (a.team_T > 0 && a.team_T * a.team_SPL >= Ns) T = a.team_T, S = a.team_SPL;  // a requested shape
#define PFFRG_DISPATCH(t, s) \
    if (T == t && S == s) return run_shape<R, C, t, s>(a, Wsp, h_counters, st, cap);
    PFFRG_TEAM_SHAPES(PFFRG_DISPATCH)
#undef PFFRG_DISPATCH
    return cudaErrorInvalidValue;
}

}  // namespace pffrg
