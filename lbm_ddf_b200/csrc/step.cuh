// step.cuh — the fused LBM-DDF time step: moments, BGK collision of f with the
// Boussinesq force, BGK collision of g, and streaming with halfway bounce-back
// and anti-bounce-back plates, for one node per thread, in place (AA pattern).
//
// What one step computes is the reference's six-launch step
// (Summer536/LBM_DDF src/main.cu:27-46):
//   forcing     F_y = g*beta*(phi^{n-1} - t0)                    src/macrovar.cu:36-47
//   collide f   BGK to feq(rho, u) + (1 - 1/(2 tau)) F_y 3(c_y - u_y) feq(1, u)
//                                                               src/collision.cu:3-33
//   collide g   BGK to geq = w phi (1 + 3c.u + 4.5(c.u)^2 - 1.5u^2)  src/collision.cu:52-64
//   stream f/g  with the wall rules of src/streaming.cu:59-124, 183-250
//   macrovar    rho = sum f, u = sum c f + F/2, phi = sum g      src/macrovar.cu:3-34
// fused into a single pass.  The moments of step n are recomputed from the
// populations at the start of step n+1; the only extra per-node state is the
// previous-step temperature phi^{n-1} ("phip"), because the stored velocity of
// the reference carries the force of the previous step (u^n = sum c f^n +
// g*beta*(phi^{n-1} - t0)/2) and the anti-bounce-back uses rho^{n-1}.
//
// AA pattern (Bailey et al., ICPP 2009).  One array per distribution holds
// the populations in one of two layouts:
//   natural : slot k of node x holds f_k(x) after streaming;
//   swapped : slot k of node x holds the post-collision f*_{opp k}(x), not
//             yet streamed.
// From natural, a step reads slot k of x and writes f*_i to slot opp(i) of x
// (all accesses local).  From swapped, a step reads population k of x from
// slot opp(k) of x - c_k, and writes f*_i to slot i of x + c_i (the set of
// locations a node reads is the set it writes, so no two threads touch the
// same word).  Walls: a population that would leave the box through a wall
// is kept at the node, in the slot its reflection is read from next step,
// with the anti-bounce-back transform applied when it is written; the
// rho^{n-1} this needs is the pre-collision density of the same node.
//
// Wall precedence (reference "last write wins", src/streaming.cu:59-124,
// 183-250, faces applied x-, x+, y-, y+, z-, z+): for g a population that
// crosses a z face is bounced back plainly even if it also crosses a y face;
// otherwise crossing a y face gives anti-bounce-back.  For f every rule is the
// same plain bounce-back.
#pragma once

#include "../../include/lbm_ddf.h"
#include "lattice.cuh"

namespace lbm {

template <class S> struct StepArgs {
    using R = typename Codec<S>::R;
    using P = typename Codec<S>::P;
    // Base address of each population row (row k of f at fl[k]; for 16-bit
    // storage the rows hold (f, g) pairs and gl[k] = fl[k] + 1 element, see
    // elem_stride).  Kernel parameters live in the constant bank, so an
    // access costs one multiply-add of a 32-bit node index onto a constant,
    // whatever the case's size.
    S *fl[Q];
    S *gl[Q];
    // The same addresses again, used only for the stores.  In the
    // natural-layout step every store address equals a load address; forming
    // it from separate bases keeps the compiler from holding all 54 load
    // addresses live across the collision (which costs ~110 registers).
    S *fs[Q];
    S *gs[Q];
    P *phip;           // previous-step temperature, one per node
    int32_t lx, ly, lz;
    uint32_t nodes;
    FastDiv div_lx, div_ly;
    R tau, tauc;       // relaxation times (the FP64 path divides by them)
    R rcp_tau, rcp_tauc, rcp_rt;   // their correctly rounded reciprocals, and that of 1/3
    R omega_f;         // 1/tau
    R omega_g;         // 1/tauc
    R force_fac;       // 1 - 1/(2 tau)
    R gb;              // gravity*beta
    R t0, t_hot, t_cold;
    // 16-bit storage shifts g/w by the conduction profile at the node a value
    // is stored at, T_c(iy) = t_top - iy * t_dy (see stored_shift)
    R t_top, t_dy;
    // The reference's rest state (src/initial.cu:218-240) stores phi = 0.5
    // while its populations w_i * 0.5 sum to 0.5 - 2^-54; its first step
    // collides with the stored 0.5.  When set, the moments use phi_fix
    // instead of sum(g) (one step after lbm_init_rest).
    int32_t use_phi_fix;
    R phi_fix;

    // population rows: loads (f, g) and stores (f, g)
    __device__ __forceinline__ S *ld_row(int which, int k) const { return which ? gl[k] : fl[k]; }
    __device__ __forceinline__ S *st_row(int which, int k) const { return which ? gs[k] : fs[k]; }
    // population k of node j (the accessor interface update_node uses); the
    // index keeps its type (unsigned node, signed displaced node), which
    // the register allocation of the update is sensitive to
    template <class I> __device__ __forceinline__ const S *ldp(int which, int k, I j) const {
        if constexpr (elem_stride<S>() == 1) return ld_row(which, k) + j;
        else return ld_row(which, k) + 2u * (uint32_t)j;
    }
    template <class I> __device__ __forceinline__ S ld(int which, int k, I j) const { return *ldp(which, k, j); }
    template <class I> __device__ __forceinline__ S &st(int which, int k, I j) const {
        if constexpr (elem_stride<S>() == 1) return st_row(which, k)[j];
        else return st_row(which, k)[2u * (uint32_t)j];
    }
    // 16-bit storage: address of the (f_k, g_k) pair of node j, one 32-bit
    // word, for the loads (ld2) and the stores (st2).  The pair array is
    // addressed in three blocks of nine rows, pair (k mod 9) * pair_row + j
    // of block k / 9, with a 32-bit index (one multiply-add and one wide add
    // per access).  The index stays below 9 pair_row < 2^32 for every case
    // the C ABI accepts in 16-bit storage.
    template <class I, class SS = S> __device__ __forceinline__ const typename Pack16<SS>::T *ld2(int k, I j) const {
        return reinterpret_cast<const typename Pack16<SS>::T *>(pairs[k / 9]) +
               ((uint32_t)(k % 9) * pair_row + (uint32_t)j);
    }
    template <class I, class SS = S> __device__ __forceinline__ typename Pack16<SS>::T *st2(int k, I j) const {
        return reinterpret_cast<typename Pack16<SS>::T *>(pairs_st[k / 9]) +
               ((uint32_t)(k % 9) * pair_row_st + (uint32_t)j);
    }
    double *obs_rows;  // fused observables: one row of kObsRow sums per warp (else unused)
    double *obs_planes;    // and kObsPlanes plane sums, where a warp needs them
    S *pairs[3];       // 16-bit storage: rows 0, 9 and 18 of the (f, g) pair array
    S *pairs_st[3];    // the same, for the stores (see fs)
    uint32_t pair_row; // pairs per row (the padded node count)
    uint32_t pair_row_st;  // the same, for the stores
    uint32_t zero;         // 0 (see again())
};

// Geometry of one node: coordinates, and node-index displacements to the
// neighbours along each axis (periodic wrap folded in), with validity flags.
struct Node {
    uint32_t n;
    int32_t ix, iy, iz;
    int32_t dxm, dxp, dym, dyp, dzm, dzp;
    bool vxm, vxp, vym, vyp, vzm, vzp;
};

template <bool PERIODIC, class A>
__device__ __forceinline__ Node make_node(const A &a, uint32_t n) {
    Node g;
    g.n = n;
    uint32_t q = a.div_lx.div(n);
    g.ix = (int32_t)(n - q * (uint32_t)a.lx);
    uint32_t z = a.div_ly.div(q);
    g.iy = (int32_t)(q - z * (uint32_t)a.ly);
    g.iz = (int32_t)z;
    const int32_t plane = a.lx * a.ly;
    g.dym = -a.lx;
    g.dyp = a.lx;
    g.vym = g.iy > 0;
    g.vyp = g.iy < a.ly - 1;
    if (PERIODIC) {
        g.dxm = g.ix > 0 ? -1 : a.lx - 1;
        g.dxp = g.ix < a.lx - 1 ? 1 : 1 - a.lx;
        g.dzm = g.iz > 0 ? -plane : (a.lz - 1) * plane;
        g.dzp = g.iz < a.lz - 1 ? plane : (1 - a.lz) * plane;
        g.vxm = g.vxp = g.vzm = g.vzp = true;
    } else {
        g.dxm = -1;
        g.dxp = 1;
        g.dzm = -plane;
        g.dzp = plane;
        g.vxm = g.ix > 0;
        g.vxp = g.ix < a.lx - 1;
        g.vzm = g.iz > 0;
        g.vzp = g.iz < a.lz - 1;
    }
    return g;
}

// displacement (in nodes) and validity of the neighbour x + (DX, DY, DZ)
template <int DX, int DY, int DZ>
__device__ __forceinline__ int32_t disp(const Node &g) {
    return (DX < 0 ? g.dxm : DX > 0 ? g.dxp : 0) + (DY < 0 ? g.dym : DY > 0 ? g.dyp : 0) +
           (DZ < 0 ? g.dzm : DZ > 0 ? g.dzp : 0);
}
template <int DX, int DY, int DZ>
__device__ __forceinline__ bool inside(const Node &g) {
    return (DX < 0 ? g.vxm : DX > 0 ? g.vxp : true) && (DY < 0 ? g.vym : DY > 0 ? g.vyp : true) &&
           (DZ < 0 ? g.vzm : DZ > 0 ? g.vzp : true);
}
// Which neighbours a node update may take as inside the box without a test
// (the INTERIOR template argument of the gathers and scatters):
//   kNoneInside: none, every neighbour is tested;
//   kRowInside:  those along y and z (0 < iy < LY-1, and periodic sides or
//                0 < iz < LZ-1): only the x neighbour is tested, which is a
//                compile-time true with periodic sides and a per-lane select
//                at the x walls of a closed box;
//   kAllInside:  all of them (a closed box's rows whose warp holds no x-wall
//                node: with LX a multiple of 32, all but the first and last
//                warp of a row).
constexpr int kNoneInside = 0, kRowInside = 1, kAllInside = 2;
template <int INTERIOR, int DX, int DY, int DZ>
__device__ __forceinline__ bool inside_t(const Node &g) {
    if constexpr (INTERIOR == kAllInside) return true;
    else if constexpr (INTERIOR == kRowInside) return DX < 0 ? g.vxm : DX > 0 ? g.vxp : true;
    else return inside<DX, DY, DZ>(g);
}
// whether every neighbour of a node taking this path is inside (so the
// swapped layout reads every population from, and writes it to, the
// neighbouring planes: the 16-bit update's plane-shift fold applies)
template <int INTERIOR, bool PERIODIC> constexpr bool all_inside() {
    return INTERIOR == kAllInside || (INTERIOR == kRowInside && PERIODIC);
}

// Whether node g's neighbours along y and z are all inside the box (the
// INTERIOR case of inside_t); uniform over a warp whenever LX is a multiple
// of 32.
template <bool PERIODIC> __device__ __forceinline__ bool yz_interior(const Node &g) {
    return g.vym && g.vyp && (PERIODIC || (g.vzm && g.vzp));
}

// The lanes of the calling warp that hold a node: its nodes are consecutive
// and start at a multiple of 32 in every kernel that updates nodes or forms
// their moments.
template <class A> __device__ __forceinline__ unsigned node_lanes(const A &a, const Node &g) {
    const uint32_t left = a.nodes - (g.n & ~31u);
    return left >= 32u ? 0xffffffffu : (1u << left) - 1u;
}

// Whether rows are whole warps, so that a warp's nodes share an x-row.
template <class A> __device__ __forceinline__ bool whole_warps(const A &a) { return (a.lx & 31) == 0; }

// Whether all nodes of the warp are `inner` (in rows of whole warps, whether
// this one is: they all are or none).
template <class A> __device__ __forceinline__ bool one_body(const A &a, const Node &g, bool inner) {
    return whole_warps(a) ? inner : __all_sync(node_lanes(a, g), inner);
}

// The path of node g's update (the INTERIOR argument, see inside_t):
// kRowInside for rows whose y and z neighbours are inside, kAllInside for
// those of a closed box when no active lane of the warp lies at an x wall
// (decided over the warp, so a warp takes one path), else kNoneInside.
// In the natural layout every access is at the node itself, so kAllInside
// would compile to kRowInside's code again: with SWAPPED false it is not
// returned, which keeps a third copy of the update out of the kernel.
template <bool PERIODIC, bool SWAPPED = true> __device__ __forceinline__ int node_path(const Node &g) {
    if (!yz_interior<PERIODIC>(g)) return kNoneInside;
    if constexpr (!PERIODIC && SWAPPED) {
        if (__all_sync(__activemask(), g.vxm && g.vxp)) return kAllInside;
    }
    return kRowInside;
}
// Population k (of f when WHICH = 0, of g when 1) of node g at the current
// time, from either layout.  `a` supplies the addresses: a.ldp(which, k,
// node).  In the swapped layout the value sits at the neighbour x - c_K
// (population opp(K)) when that is inside the box, else at the node itself
// (population K, bounce-back); the address is chosen by a select, so a warp
// whose lanes differ (one holding an x-wall node) still issues one load
// rather than two half-masked ones.
template <class S, bool SWAPPED, int K, int INTERIOR = kNoneInside, int WHICH = 0, class A>
__device__ __forceinline__ S load_pop(const A &a, const Node &g) {
    if (!SWAPPED) return a.ld(WHICH, K, g.n);
    constexpr int DX = -cx(K), DY = -cy(K), DZ = -cz(K);
    const bool in = inside_t<INTERIOR, DX, DY, DZ>(g);
    return *(in ? a.ldp(WHICH, opp(K), (int32_t)g.n + disp<DX, DY, DZ>(g)) : a.ldp(WHICH, K, g.n));
}

// Whether population K of a 16-bit node takes its address by a select
// between the neighbour and the node itself: the x-moving populations of a
// closed box's rows (see update_node16).  Elsewhere the test is a constant or
// rare, and a branch.
template <bool SWAPPED, bool PERIODIC, int INTERIOR, int K> constexpr bool selects_address() {
    return SWAPPED && !PERIODIC && INTERIOR == kRowInside && cx(K) != 0;
}

// The (f_k, g_k) pair that node g collides in this step, as load_pop finds
// each value, with one 32-bit load.
template <class S, bool SWAPPED, bool PERIODIC, int K, int INTERIOR, class A>
__device__ __forceinline__ typename Pack16<S>::T load_pair(const A &a, const Node &g) {
    if (!SWAPPED) return *a.ld2(K, g.n);
    constexpr int DX = -cx(K), DY = -cy(K), DZ = -cz(K);
    const bool in = inside_t<INTERIOR, DX, DY, DZ>(g);
    if constexpr (selects_address<SWAPPED, PERIODIC, INTERIOR, K>())
        return *(in ? a.ld2(opp(K), (int32_t)g.n + disp<DX, DY, DZ>(g)) : a.ld2(K, g.n));
    if (in) return *a.ld2(opp(K), (int32_t)g.n + disp<DX, DY, DZ>(g));
    return *a.ld2(K, g.n);
}

// 16-bit storage keeps g_i / w_i - T_c at every location, T_c(iy) =
// T_hot - (T_hot - T_cold) (iy + 1/2) / LY the conduction profile at the
// plane of the node the value is stored at (halfway walls: the plates sit
// half a node outside the first and last planes).  Near the plates, where Nu
// is measured, g/w is then close to the stored shift and 16-bit rounding
// small against the plane-to-plane temperature step; with one constant
// shift it was up to 2^-11 (FP16) and 2^-8 (BF16) there.  Inside a node
// update the g values are kept relative to the node's own T_c (shift0); a
// value read from or written to a neighbour's plane differs from that by
// a multiple of t_dy:
//   read (swapped layout, population K from x - c_K): + c_Ky t_dy
//   write (swapped layout, population I to x + c_I):   + c_Iy t_dy
// and by nothing at the node itself (natural layout, bounce-back).
template <class A> __device__ __forceinline__ float shift0(const A &a, const Node &g) {
    return fmaf(-(float)g.iy, (float)a.t_dy, (float)a.t_top);
}
template <bool SWAPPED, int K, int INTERIOR, class A>
__device__ __forceinline__ float read_shift_delta(const A &a, const Node &g) {
    constexpr int DX = -cx(K), DY = -cy(K), DZ = -cz(K);
    if constexpr (!SWAPPED || DY == 0) return 0.f;
    else return inside_t<INTERIOR, DX, DY, DZ>(g) ? (float)cy(K) * (float)a.t_dy : 0.f;
}
template <class S, bool SWAPPED, int INTERIOR = kNoneInside, class A>
__device__ __forceinline__ void gather(const A &a, const Node &g, typename Codec<S>::R (&fr)[Q],
                                       typename Codec<S>::R (&gr)[Q]) {
    using C = Codec<S>;
    float s0 = 0.f;
    if constexpr (elem_stride<S>() == 2) s0 = shift0(a, g);
    Unroll<0, Q>::run([&](auto kk) {
        constexpr int K = decltype(kk)::value;
        if constexpr (elem_stride<S>() == 2) {   // (f, g) pairs: f_i = w_i fh, g_i = w_i (gh + T_c at the location)
            // explicit rounding: the compiler cannot fuse these products into
            // the moment sums in one kernel and not in another, so every
            // kernel that gathers (the step, the observables) forms the same
            // FP32 moments
            const float2 v = Pack16<S>::unpack(load_pair<S, SWAPPED, false, K, INTERIOR>(a, g));
            fr[K] = __fmul_rn((float)wd(K), v.x);
            gr[K] = __fmul_rn((float)wd(K), __fadd_rn(v.y, __fadd_rn(s0, read_shift_delta<SWAPPED, K, INTERIOR>(a, g))));
        } else {
            fr[K] = C::template f_in<K>(load_pop<S, SWAPPED, K, INTERIOR, 0>(a, g), a.t0);
            gr[K] = C::template g_in<K>(load_pop<S, SWAPPED, K, INTERIOR, 1>(a, g), a.t0);
        }
    });
}

// Moments of the populations at one node.  u carries the previous step's
// half force, as the reference's stored velocity does (src/macrovar.cu:28-30).
template <class R> struct Moments {
    R rho, ux, uy, uz, phi;
};

template <class R>
__device__ __forceinline__ Moments<R> moments(const R (&fr)[Q], const R (&gr)[Q], R phip, R gb, R t0) {
    Moments<R> m;
    R rho = 0, jx = 0, jy = 0, jz = 0, phi = 0;
    Unroll<0, Q>::run([&](auto kk) {
        constexpr int K = decltype(kk)::value;
        rho += fr[K];
        if (cx(K) > 0) jx += fr[K];
        if (cx(K) < 0) jx -= fr[K];
        if (cy(K) > 0) jy += fr[K];
        if (cy(K) < 0) jy -= fr[K];
        if (cz(K) > 0) jz += fr[K];
        if (cz(K) < 0) jz -= fr[K];
        phi += gr[K];
    });
    m.rho = rho;
    m.ux = jx;
    if constexpr (std::is_same<R, float>::value)   // explicit rounding: the same in every kernel
        m.uy = __fadd_rn(jy, __fmul_rn(0.5f, __fmul_rn(gb, __fsub_rn(phip, t0))));
    else   // FP64: as written, the rounding the reference build has (bitwise parity)
        m.uy = jy + R(0.5) * (gb * (phip - t0));
    m.uz = jz;
    m.phi = phi;
    return m;
}

template <class S, class A>
__device__ __forceinline__ Moments<typename Codec<S>::R> node_moments(const A &a,
                                                                     const typename Codec<S>::R (&fr)[Q],
                                                                     const typename Codec<S>::R (&gr)[Q],
                                                                     uint32_t n) {
    using R = typename Codec<S>::R;
    Moments<R> m = moments(fr, gr, (R)a.phip[n], a.gb, a.t0);
    if (a.use_phi_fix) m.phi = a.phi_fix;
    return m;
}

// BGK collision of f (with the buoyancy force) and g, in place on fr/gr,
// in FP32: the same equilibria with the divisions by 1/3 and tau folded into
// multiplications and every multiply-add left to the compiler.
template <class R>
__device__ __forceinline__ void collide_fast(R (&fr)[Q], R (&gr)[Q], const Moments<R> &m, R omega_f, R omega_g,
                                             R force_fac, R gb, R t0) {
    const R uv = R(3) * (m.ux * m.ux + m.uy * m.uy + m.uz * m.uz);
    const R fy = gb * (m.phi - t0);           // force of this step, from phi^{n-1}
    const R kf = R(3) * force_fac * fy;
    Unroll<0, Q>::run([&](auto kk) {
        constexpr int K = decltype(kk)::value;
        constexpr R w = R(wd(K));
        R cu = R(0);
        if (cx(K) > 0) cu += m.ux;
        if (cx(K) < 0) cu -= m.ux;
        if (cy(K) > 0) cu += m.uy;
        if (cy(K) < 0) cu -= m.uy;
        if (cz(K) > 0) cu += m.uz;
        if (cz(K) < 0) cu -= m.uz;
        const R eu = R(3) * cu;
        const R p = eu + R(0.5) * (eu * eu - uv);   // velocity part of the equilibria
        const R feq = w * (m.rho + p);
        const R feq0 = w * (R(1) + p);
        const R fo = fr[K];
        fr[K] = fo - omega_f * (fo - feq) + kf * (R(cy(K)) - m.uy) * feq0;
        const R go = gr[K];
        gr[K] = go - omega_g * (go - m.phi * feq0);
    });
}

// Round-to-nearest operations the compiler never fuses or reorders: code
// written with them rounds identically in every kernel that inlines it.
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// Paired FP32 operations (two lanes in one instruction on sm_100): each lane
// rounds exactly as the scalar operation, so code written with them gives
// the scalar code's bits.
__device__ __forceinline__ float2 splat(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// Regularised BGK (Latt and Chopard, Math. Comput. Simul. 72 (2006)
// 165-168), an option beside the reference's BGK for relaxation times near
// 1/2.  Same equilibria and force term as collide_fast; the non-equilibrium
// part that relaxes is replaced by its projection on the second-order
// Hermite polynomial for f and the first-order one for g:
//   f_i* = feq_i + (1 - 1/tau) 4.5 w_i (c_i c_i : Pi - tr(Pi)/3) + force_i,
//          Pi = sum_i c_i c_i f_i - (rho/3 I + u u)
//   g_i* = geq_i + (1 - 1/tau_c) 3 w_i c_i . j,   j = sum_i c_i g_i - phi u
// (rho/3 I + u u and phi u are the equilibria's own second and first
// moments on D3Q27).  rho, u and phi are unchanged, as in BGK; at tau = 1 the
// two models coincide.  Every operation is an explicit round-to-nearest one,
// so a case gives bitwise the same result in the single-case and the batch
// kernels.  FP64 steps run it; FP32 and 16-bit ones its operations on the
// sums alone (reg_sums, reg_relax).
template <class R>
__device__ __forceinline__ void collide_reg(R (&fr)[Q], R (&gr)[Q], const Moments<R> &m, R omega_f, R omega_g,
                                            R force_fac, R gb, R t0) {
    R sxx = 0, syy = 0, szz = 0, sxy = 0, sxz = 0, syz = 0, jx = 0, jy = 0, jz = 0;
    Unroll<0, Q>::run([&](auto kk) {
        constexpr int K = decltype(kk)::value;
        constexpr int X = cx(K), Y = cy(K), Z = cz(K);
        const R f = fr[K], g = gr[K];
        if (X != 0) sxx = add_rn(sxx, f);
        if (Y != 0) syy = add_rn(syy, f);
        if (Z != 0) szz = add_rn(szz, f);
        if (X * Y > 0) sxy = add_rn(sxy, f);
        if (X * Y < 0) sxy = sub_rn(sxy, f);
        if (X * Z > 0) sxz = add_rn(sxz, f);
        if (X * Z < 0) sxz = sub_rn(sxz, f);
        if (Y * Z > 0) syz = add_rn(syz, f);
        if (Y * Z < 0) syz = sub_rn(syz, f);
        if (X > 0) jx = add_rn(jx, g);
        if (X < 0) jx = sub_rn(jx, g);
        if (Y > 0) jy = add_rn(jy, g);
        if (Y < 0) jy = sub_rn(jy, g);
        if (Z > 0) jz = add_rn(jz, g);
        if (Z < 0) jz = sub_rn(jz, g);
    });
    const R third = R(1) / R(3);
    const R rho3 = mul_rn(m.rho, third);
    const R pxx = fma_rn(-m.ux, m.ux, sub_rn(sxx, rho3));
    const R pyy = fma_rn(-m.uy, m.uy, sub_rn(syy, rho3));
    const R pzz = fma_rn(-m.uz, m.uz, sub_rn(szz, rho3));
    const R pxy2 = mul_rn(R(2), fma_rn(-m.ux, m.uy, sxy));
    const R pxz2 = mul_rn(R(2), fma_rn(-m.ux, m.uz, sxz));
    const R pyz2 = mul_rn(R(2), fma_rn(-m.uy, m.uz, syz));
    const R tr3 = mul_rn(add_rn(add_rn(pxx, pyy), pzz), third);
    jx = fma_rn(-m.phi, m.ux, jx);
    jy = fma_rn(-m.phi, m.uy, jy);
    jz = fma_rn(-m.phi, m.uz, jz);
    const R keep_f = mul_rn(R(4.5), sub_rn(R(1), omega_f)), keep_g = mul_rn(R(3), sub_rn(R(1), omega_g));
    const R uv = mul_rn(R(3), fma_rn(m.uz, m.uz, fma_rn(m.uy, m.uy, mul_rn(m.ux, m.ux))));
    const R kf = mul_rn(mul_rn(R(3), force_fac), mul_rn(gb, sub_rn(m.phi, t0)));
    Unroll<0, Q>::run([&](auto kk) {
        constexpr int K = decltype(kk)::value;
        constexpr int X = cx(K), Y = cy(K), Z = cz(K);
        constexpr R w = R(wd(K));
        R cu = R(0), cj = R(0), qpi = -tr3;
        if (X > 0) { cu = add_rn(cu, m.ux); cj = add_rn(cj, jx); qpi = add_rn(qpi, pxx); }
        if (X < 0) { cu = sub_rn(cu, m.ux); cj = sub_rn(cj, jx); qpi = add_rn(qpi, pxx); }
        if (Y > 0) { cu = add_rn(cu, m.uy); cj = add_rn(cj, jy); qpi = add_rn(qpi, pyy); }
        if (Y < 0) { cu = sub_rn(cu, m.uy); cj = sub_rn(cj, jy); qpi = add_rn(qpi, pyy); }
        if (Z > 0) { cu = add_rn(cu, m.uz); cj = add_rn(cj, jz); qpi = add_rn(qpi, pzz); }
        if (Z < 0) { cu = sub_rn(cu, m.uz); cj = sub_rn(cj, jz); qpi = add_rn(qpi, pzz); }
        if (X * Y > 0) qpi = add_rn(qpi, pxy2);
        if (X * Y < 0) qpi = sub_rn(qpi, pxy2);
        if (X * Z > 0) qpi = add_rn(qpi, pxz2);
        if (X * Z < 0) qpi = sub_rn(qpi, pxz2);
        if (Y * Z > 0) qpi = add_rn(qpi, pyz2);
        if (Y * Z < 0) qpi = sub_rn(qpi, pyz2);
        const R eu = mul_rn(R(3), cu);
        const R p = add_rn(eu, mul_rn(R(0.5), fma_rn(eu, eu, -uv)));
        const R feq0 = mul_rn(w, add_rn(R(1), p));
        const R fneq = mul_rn(mul_rn(keep_f, w), qpi);
        const R force = mul_rn(mul_rn(kf, sub_rn(R(Y), m.uy)), feq0);
        fr[K] = add_rn(add_rn(mul_rn(w, add_rn(m.rho, p)), fneq), force);
        gr[K] = fma_rn(mul_rn(keep_g, w), cj, mul_rn(m.phi, feq0));
    });
}

// Correctly rounded a / b for a divisor b known in advance, from its correctly
// rounded reciprocal y = RN(1/b): q = RN(a y), r = a - b q (exact by FMA),
// result RN(q + r y).  Markstein's theorem (P. Markstein, IBM J. Res. Dev.
// 34(1), 1990; "IA-64 and Elementary Functions", 2000, Thm 8.10): if y is
// within half an ulp of 1/b and q within one ulp of a/b, the corrected
// quotient is the correctly rounded one.  Valid for finite quotients away
// from the subnormal range (all quotients here); the C ABI's
// lbm_selfcheck_division checks it against the hardware division on the GPU.
__device__ __forceinline__ double div_by(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    const double r = __fma_rn(-b, q, a);
    return __fma_rn(r, y, q);
}

// The same collision in FP64 as the reference binary computes it: the
// operations of src/collision.cu:19-33 and :65-72 in their order, correctly
// rounded divisions by RT = 1/3, tau and tauc, and a fused multiply-add
// exactly where the reference build has one (u*u sums, eu*eu - uv, f - w*feq,
// g - w*phi*geq; not the force term).  Written with round-to-nearest
// intrinsics, which the compiler never re-fuses, so the results are bitwise
// the reference's.
__device__ __forceinline__ void collide_exact(double (&fr)[Q], double (&gr)[Q], const Moments<double> &m,
                                              double tau, double tauc, double rcp_tau, double rcp_tauc,
                                              double rcp_rt, double force_fac, double gb, double t0) {
    const double RT = 1.0 / 3.0;
    const double uv = div_by(__fma_rn(m.uz, m.uz, __fma_rn(m.ux, m.ux, __dmul_rn(m.uy, m.uy))), RT, rcp_rt);
    const double fy = __dmul_rn(gb, __dsub_rn(m.phi, t0));
    const double kf = __dmul_rn(force_fac, fy);
    // ((1 - 1/(2 tau)) F_y (c_y - u_y)) / RT takes one of three values
    const double fc_m = div_by(__dmul_rn(kf, __dsub_rn(-1.0, m.uy)), RT, rcp_rt);
    const double fc_0 = div_by(__dmul_rn(kf, __dsub_rn(0.0, m.uy)), RT, rcp_rt);
    const double fc_p = div_by(__dmul_rn(kf, __dsub_rn(1.0, m.uy)), RT, rcp_rt);
    Unroll<0, Q>::run([&](auto kk) {
        constexpr int K = decltype(kk)::value;
        constexpr double w = wd(K);
        double cu = 0.0;   // (c.u), summed x, y, z as the reference does; c*u is exact
        if (cx(K) > 0) cu = __dadd_rn(cu, m.ux);
        if (cx(K) < 0) cu = __dsub_rn(cu, m.ux);
        if (cy(K) > 0) cu = __dadd_rn(cu, m.uy);
        if (cy(K) < 0) cu = __dsub_rn(cu, m.uy);
        if (cz(K) > 0) cu = __dadd_rn(cu, m.uz);
        if (cz(K) < 0) cu = __dsub_rn(cu, m.uz);
        const double eu = div_by(cu, RT, rcp_rt);
        const double hq = __dmul_rn(0.5, __fma_rn(eu, eu, -uv));
        const double feq_in = __dadd_rn(__dadd_rn(m.rho, eu), hq);
        const double inner0 = __dadd_rn(__dadd_rn(1.0, eu), hq);
        const double feq0 = __dmul_rn(w, inner0);
        const double fc = cy(K) < 0 ? fc_m : cy(K) > 0 ? fc_p : fc_0;
        const double fo = fr[K];
        double fch = -div_by(__fma_rn(-w, feq_in, fo), tau, rcp_tau);
        fch = __dadd_rn(fch, __dmul_rn(fc, feq0));
        fr[K] = __dadd_rn(fo, fch);
        const double go = gr[K];
        const double gch = -div_by(__fma_rn(-__dmul_rn(w, m.phi), inner0, go), tauc, rcp_tauc);
        gr[K] = __dadd_rn(go, gch);
    });
}

template <class S, int COLL = LBM_COLLISION_BGK, class A>
__device__ __forceinline__ void collide(typename Codec<S>::R (&fr)[Q], typename Codec<S>::R (&gr)[Q],
                                        const Moments<typename Codec<S>::R> &m, const A &a) {
    if constexpr (COLL == LBM_COLLISION_REGULARIZED)
        collide_reg(fr, gr, m, a.omega_f, a.omega_g, a.force_fac, a.gb, a.t0);
    else if constexpr (std::is_same<typename Codec<S>::R, double>::value)
        collide_exact(fr, gr, m, a.tau, a.tauc, a.rcp_tau, a.rcp_tauc, a.rcp_rt, a.force_fac, a.gb, a.t0);
    else
        collide_fast(fr, gr, m, a.omega_f, a.omega_g, a.force_fac, a.gb, a.t0);
}

// Anti-bounce-back value of an outgoing population gv at a plate of
// temperature tw: -gv + 2 w tw (1 + rho), src/streaming.cu:207-227 (the
// product fused into the sum in FP64, as the reference build does).
template <int I, class R>
__device__ __forceinline__ R abb(R gv, R tw, R rho) {
    if constexpr (std::is_same<R, double>::value)
        return __fma_rn(__dmul_rn(__dmul_rn(2.0, wd(I)), tw), __dadd_rn(1.0, rho), -gv);
    else
        return -gv + R(2) * R(wd(I)) * tw * (R(1) + rho);
}

// Whether population I of node g leaves through a plate with the
// anti-bounce-back rule (and not also through a z wall, see the top).
template <bool PERIODIC, int INTERIOR, int I> __device__ __forceinline__ bool meets_plate(const Node &g) {
    if constexpr (INTERIOR != kNoneInside || cy(I) == 0) return false;
    else
        return (cy(I) < 0 ? !g.vym : !g.vyp) &&
               !(!PERIODIC && ((cz(I) < 0 && !g.vzm) || (cz(I) > 0 && !g.vzp)));
}

// Stores population I (of f when which = 0, of g when 1) of node g where the
// next step reads it: the neighbour x + c_I (swapped layout, inside) or the
// node itself, the address chosen by a select (see load_pop).
template <bool SWAPPED, int INTERIOR, int I, class A, class R>
__device__ __forceinline__ void store_pop(const A &a, const Node &g, int which, R v) {
    constexpr int DX = cx(I), DY = cy(I), DZ = cz(I);
    const bool in = SWAPPED && inside_t<INTERIOR, DX, DY, DZ>(g);
    *(in ? &a.st(which, I, (int32_t)g.n + disp<DX, DY, DZ>(g)) : &a.st(which, opp(I), g.n)) = v;
}

// Writes the post-collision populations of node g to where the next step
// reads them (FP32 and FP64).  rho is the node's pre-collision density (for
// anti-bounce-back).
template <class S, bool SWAPPED, bool PERIODIC, int INTERIOR = kNoneInside, class A>
__device__ __forceinline__ void scatter(const A &a, const Node &g, const typename Codec<S>::R (&fr)[Q],
                                        const typename Codec<S>::R (&gr)[Q], typename Codec<S>::R rho) {
    static_assert(elem_stride<S>() == 1, "16-bit pairs are stored by store_word");
    Unroll<0, Q>::run([&](auto ii) {
        constexpr int I = decltype(ii)::value;
        typename Codec<S>::R gv = gr[I];
        if (meets_plate<PERIODIC, INTERIOR, I>(g)) gv = abb<I>(gv, cy(I) < 0 ? a.t_hot : a.t_cold, rho);
        store_pop<SWAPPED, INTERIOR, I>(a, g, 0, fr[I]);
        store_pop<SWAPPED, INTERIOR, I>(a, g, 1, gv);
    });
}

// Threads per block of step_kernel: FP32 and 16-bit steps in blocks of two
// warps (a block holds its SM slot until its slowest warp is done, and
// two-warp blocks waste less of it: B200, 256^3 FP32, natural layout -1.8%,
// closed-box swapped -3.6%; FP16S BGK closed box -4% over both layouts); FP64
// measured 3% slower so and keeps four.
template <class S> __host__ __device__ constexpr int node_threads() { return sizeof(S) == 8 ? 128 : 64; }
// Resident threads per SM the register allocation is sized for: 384 (<= 168
// registers) for FP64, which holds 54 doubles across the collision (B200,
// 256^3: 6.7, 7.4 and 6.6 GLUPS at 256, 384 and 512 threads, the last
// spilling); 512 (<= 128) for FP32; 768 (80) for 16-bit storage, which holds
// 27 packed words (256^3 FP16S, periodic, both layouts summed: BGK 1207 us at
// 768 threads, 1272 at 640, over 2500 at 896 where the rows' body spills;
// regularised 1390 at 768 and 1440 at 640).
template <class S> __host__ __device__ constexpr int step_threads_per_sm() {
    return sizeof(S) == 8 ? 384 : sizeof(S) == 4 ? 512 : 768;
}
// Grids that the device holds at once at this many threads per SM have a step
// of their own (SMALL below), whose time is the length of one update: 16-bit
// BGK is built for this number, since registers that hide nothing there keep
// the 27 words and their update free of spills (B200, us per step, against
// 768: 16^3 FP16S 2.8 and 3.3, 32^3 3.2 and 3.3, two cases of 16^3 on their own
// kernels in a batch 3.4 and 3.7; regularised steps, with few spills, the
// same), and with periodic sides a warp runs one body (update_node16).
constexpr int kSmallGridThreadsPerSm = 512;
template <class S, bool PERIODIC, int COLL, bool OBS> constexpr bool has_small_step() {
    return !OBS && ((sizeof(S) == 2 && (COLL == LBM_COLLISION_BGK || PERIODIC)) ||
                    (sizeof(S) == 4 && COLL == LBM_COLLISION_REGULARIZED && PERIODIC));
}
template <class S, int COLL, bool SMALL> constexpr int step_budget() {
    return SMALL && sizeof(S) == 2 && COLL == LBM_COLLISION_BGK ? kSmallGridThreadsPerSm : step_threads_per_sm<S>();
}
// The step kernel's launch bounds (FP32's are stated for blocks of 128, the
// same register budget).
template <class S> constexpr int bound_threads() { return sizeof(S) == 2 ? node_threads<S>() : 128; }

// ---- observables of a node's moments --------------------------------------
//
// FP64 sums of
//   0 uy*phi  1 |u|^2  2 ux  3 uy  4 uz  5 phi
//   6..8  phi on the planes iy = 0, 1, 2
//   9..11 phi on the planes iy = LY-1, LY-2, LY-3
//   12 number of nodes with a non-finite moment
// (src/output.cu:199-256 and :24-34 reduce the same fields on the host).
constexpr int kObsTerms = 13;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <class R>
__device__ __forceinline__ void add_obs_terms(double (&acc)[kObsTerms], const Moments<R> &m, int iy, int ly) {
    const double ux = m.ux, uy = m.uy, uz = m.uz, phi = m.phi;
    acc[0] += uy * phi;
    acc[1] += ux * ux + uy * uy + uz * uz;
    acc[2] += ux;
    acc[3] += uy;
    acc[4] += uz;
    acc[5] += phi;
    if (iy == 0) acc[6] += phi;
    if (iy == 1) acc[7] += phi;
    if (iy == 2) acc[8] += phi;
    if (iy == ly - 1) acc[9] += phi;
    if (iy == ly - 2) acc[10] += phi;
    if (iy == ly - 3) acc[11] += phi;
    if (!isfinite(ux) || !isfinite(uy) || !isfinite(uz) || !isfinite(phi) || !isfinite((double)m.rho))
        acc[12] += 1.0;
}

// ---- observables inside the step ----
//
// Each warp of an observed step leaves its nodes' sums as a row of kObsRow
// doubles: the six dense terms (0 to 5) and the non-finite count (6).  The
// plane terms are the row's phi sum when its nodes share an x-row, which
// the reduction knows from the row's number; a warp across x-rows that
// touches one of the six planes also leaves kObsPlanes plane sums.
constexpr int kObsRow = 8, kObsPlanes = 6;

// Lane sums of six values: each exchange halves the values a lane carries,
// 8 shuffles instead of the 30 of six butterflies.  Lane l ends with the
// total of value 3 (l >> 4 & 1) + (l & 4 ? 2 : l >> 3 & 1).
__device__ __forceinline__ double warp_sum6(const double (&d)[6], int lane) {
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    double x[3];
#pragma unroll
    for (int k = 0; k < 3; k++) x[k] = (b4 ? d[k + 3] : d[k]) + __shfl_xor_sync(0xffffffffu, b4 ? d[k] : d[k + 3], 16);
    const double y0 = (b3 ? x[1] : x[0]) + __shfl_xor_sync(0xffffffffu, b3 ? x[0] : x[1], 8);
    const double y1 = x[2] + __shfl_xor_sync(0xffffffffu, x[2], 8);
    double z = (b2 ? y1 : y0) + __shfl_xor_sync(0xffffffffu, b2 ? y0 : y1, 4);
    z += __shfl_xor_sync(0xffffffffu, z, 2);
    return z + __shfl_xor_sync(0xffffffffu, z, 1);
}

// The warp's row (and plane sums, if it needs them); all 32 lanes call it,
// `valid` false for lanes without a node, each with its node's six dense
// terms and plane.  What it costs a step is the time it keeps a warp
// resident: the row leaves in one coalesced store, and a warp that finishes
// early leaves at once, with no block barrier.  B200, FP64 closed box at
// 256^3, both layouts: 2397 us per observed step, BF16S at 192x96x192
// 179; with butterflies and 13 stores by one lane 2415 and 188.
__device__ __forceinline__ void warp_obs_row(const double (&d)[6], int iy, bool valid, bool bad, int ly, size_t r,
                                             double *__restrict__ rows, double *__restrict__ planes) {
    const int lane = threadIdx.x & 31;
    const double z = warp_sum6(d, lane);
    const unsigned count = __popc(__ballot_sync(0xffffffffu, valid && bad));
    if ((lane & 3) == 0) {
        const int at = (lane & 12) == 12 ? (lane & 16 ? 7 : 6) : (lane & 16 ? 3 : 0) + (lane & 4 ? 2 : lane >> 3 & 1);
        rows[r * kObsRow + at] = at == 6 ? (double)count : at == 7 ? 0.0 : z;
    }
    const int iy0 = __shfl_sync(0xffffffffu, iy, 0);   // lane 0 holds a node if any lane does
    if (__all_sync(0xffffffffu, !valid || iy == iy0)) return;
    if (!__any_sync(0xffffffffu, valid && (iy <= 2 || iy >= ly - 3))) return;
    double e[6];
#pragma unroll
    for (int k = 0; k < 6; k++) e[k] = valid && iy == (k < 3 ? k : ly - 1 - (k - 3)) ? d[5] : 0.0;
    const double w = warp_sum6(e, lane);
    if ((lane & 3) == 0 && (lane & 12) != 12)
        planes[r * kObsPlanes + (lane & 16 ? 3 : 0) + (lane & 4 ? 2 : lane >> 3 & 1)] = w;
}

// The moments a node update starts from (the observables of the state the
// step reads) and the node's plane.
template <class R> struct NodeOut {
    Moments<R> m;
    int32_t iy;
};

// ---- 16-bit storage: the collision in the stored, normalised variables ----
//
// FP16S / BF16S rows hold (fh_i, gh_i) pairs, fh_i = f_i / w_i and
// gh_i = g_i / w_i - T_c (T_c the conduction profile at the location, see
// shift0), one 32-bit word per population and node.  The updates below work
// on those directly in FP32, one node per thread.  A thread first loads its
// 27 words, all of them before the first is unpacked, so that they are in
// flight together and held in one register each; it sums the moments, then
// relaxes and stores pair by pair.  What bounds these kernels is memory
// latency, and two things decide how well it is hidden:
//  - nothing should be loaded between the stores.  Reading each pair a second
//    time (from L1) instead of holding it ran at a third of the speed, and
//    builds whose registers spilled there at half to two thirds.  So the
//    register budget is the one at which the rows' body hardly spills, not
//    the smallest;
//  - the registers must go to the 27 words.  The 26 neighbour indices of the
//    loads are the stores' again; again() keeps them from being held.
// Warps are retired in blocks of two (a block holds its SM slot until its
// slowest warp is done).

// Node g for the stores: the same node, formed from a zero that the compiler
// cannot see, so that it forms the stores' addresses anew.
template <class A> __device__ __forceinline__ Node again(const A &a, const Node &g) {
    Node s = g;
    s.n += a.zero;
    s.dxm += a.zero;
    s.dxp += a.zero;
    s.dzm += a.zero;
    s.dzp += a.zero;
    return s;
}

// Receives a node's moments as soon as a node update has formed them, before
// the collision and the scatter.
struct NoMomentSink {
    template <class R> __device__ __forceinline__ void operator()(const Moments<R> &) const {}
};

// Parks a node's moments (ux, uy, uz, phi, rho) in shared memory, STRIDE
// elements apart, so a kernel that reduces them after the update does not
// hold them in registers through the collision and the scatter (in the FP64
// kernel, at its register limit, that cost a third of the swapped-layout
// step in a closed box).  T holds the moments exactly (T = double, or float
// for float moments).  Volatile, so the compiler does not forward the stores
// to the loads.
template <class T, int STRIDE> struct SharedMomentSink {
    volatile T *p;
    template <class R> __device__ __forceinline__ void operator()(const Moments<R> &m) const {
        static_assert(sizeof(T) >= sizeof(R), "the parked moments must hold the update's exactly");
        p[0] = (T)m.ux;
        p[STRIDE] = (T)m.uy;
        p[2 * STRIDE] = (T)m.uz;
        p[3 * STRIDE] = (T)m.phi;
        p[4 * STRIDE] = (T)m.rho;
    }
};

// a - b, both lanes (the product by -1 is exact)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return fma2(b, splat(-1.f), a); }
// a b, both lanes, for a product that is then added: the compiler fuses a
// paired multiplication into a paired addition, but not two scalar ones
__device__ __forceinline__ float2 product(float2 a, float2 b) {
    return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y));
}

// Where the g values of a 16-bit node are re-referenced from plane to plane
// (read_shift_delta, write_shift_delta).  BGK folds it into its relaxation
// where every neighbour is inside: on the rows of a periodic box, and in a
// closed box for warps without an x-wall node (fold = t_dy, per-value
// spacing 0); elsewhere it is added value by value (fold 0, spacing t_dy).
struct Shift {
    float s0;     // the node's own T_c
    float t_dy;   // plane spacing applied value by value
    float fold;   // plane spacing folded into the relaxation
};

// Population K's re-referencing on reading, and I's on writing, for a plane
// spacing t_dy.
template <bool SWAPPED, int K, int INTERIOR> __device__ __forceinline__ float read_shift(const Node &g, float t_dy) {
    if constexpr (!SWAPPED || cy(K) == 0) return 0.f;
    else return inside_t<INTERIOR, -cx(K), -cy(K), -cz(K)>(g) ? (float)cy(K) * t_dy : 0.f;
}
template <bool SWAPPED, int I, int INTERIOR> __device__ __forceinline__ float write_shift(const Node &g, float t_dy) {
    if constexpr (!SWAPPED || cy(I) == 0) return 0.f;
    else return inside_t<INTERIOR, cx(I), cy(I), cz(I)>(g) ? (float)cy(I) * t_dy : 0.f;
}

// Stores the word of population I of node g where the next step reads it.
template <class S, bool SWAPPED, bool PERIODIC, int INTERIOR, int I, class A>
__device__ __forceinline__ void store_word(const A &a, const Node &g, typename Pack16<S>::T w) {
    constexpr int DX = cx(I), DY = cy(I), DZ = cz(I);
    const bool in = SWAPPED && inside_t<INTERIOR, DX, DY, DZ>(g);
    if constexpr (selects_address<SWAPPED, PERIODIC, INTERIOR, I>())
        *(in ? a.st2(I, (int32_t)g.n + disp<DX, DY, DZ>(g)) : a.st2(opp(I), g.n)) = w;
    else if (in)
        *a.st2(I, (int32_t)g.n + disp<DX, DY, DZ>(g)) = w;
    else
        *a.st2(opp(I), g.n) = w;
}

// ---- BGK ----
//
// collide_fast in the normalised variables:
//   fh*_i = fh_i - (fh_i - (rho + p_i)) / tau + 3 (1 - 1/(2 tau)) F_y (c_iy - u_y) (1 + p_i)
//   gh*_i = gh_i - (gh_i + s0 - phi (1 + p_i)) / tau_c,
// p_i = 3 c_i.u + 4.5 (c_i.u)^2 - 1.5 u^2: no weight on load or store.
// B200, 256^3 FP16S, periodic: 582 us per step in the natural layout and 626
// in the swapped one, against 664 and 652 with a node's update split over
// two warps that exchanged their partial moments through shared memory (64
// registers, 770-820 instructions per 32 nodes and a barrier; here ~550, no
// barrier, and 27 loads in flight per warp instead of 13).  Closed box: 588
// and 690 against 674 and 710.

// The half of the opposite pairs that population k is summed in.  The
// moments are two partial sums, added: the rest population and the pairs of
// 1, 2, 5, 7, 19 and 20, and the other seven pairs.
__host__ __device__ constexpr int pair_rep(int k) { return k < opp(k) ? k : opp(k); }
__host__ __device__ constexpr int half_of(int k) {
    return (k == 0 || pair_rep(k) == 1 || pair_rep(k) == 2 || pair_rep(k) == 5 || pair_rep(k) == 7 ||
            pair_rep(k) == 19 || pair_rep(k) == 20)
               ? 0
               : 1;
}

// Half H's share of rho, j_x, j_y, j_z and sum w_i gh_i: sums per weight
// class, then weighted; f and g paired.
template <int H, class Value> __device__ __forceinline__ void half_sums(const Value &value, float (&p)[5]) {
    float2 rt[4] = {};   // (sum fh, sum gh) per weight class
    float x[4] = {0.f, 0.f, 0.f, 0.f}, y[4] = {0.f, 0.f, 0.f, 0.f}, z[4] = {0.f, 0.f, 0.f, 0.f};
    Unroll<0, Q>::run([&](auto kk) {
        constexpr int K = decltype(kk)::value;
        if constexpr (half_of(K) == H) {
            constexpr int C = wclass(K);
            const float2 v = value(kk);
            rt[C] = add2(rt[C], v);
            if (cx(K) > 0) x[C] += v.x;
            if (cx(K) < 0) x[C] -= v.x;
            if (cy(K) > 0) y[C] += v.x;
            if (cy(K) < 0) y[C] -= v.x;
            if (cz(K) > 0) z[C] += v.x;
            if (cz(K) < 0) z[C] -= v.x;
        }
    });
    const float w0 = (float)wd(0), w1 = (float)wd(1), w2 = (float)wd(7), w3 = (float)wd(19);
    const float2 s = fma2(splat(w3), rt[3], fma2(splat(w2), rt[2], fma2(splat(w1), rt[1], mul2(splat(w0), rt[0]))));
    p[0] = s.x;
    p[1] = fmaf(w3, x[3], fmaf(w2, x[2], w1 * x[1]));
    p[2] = fmaf(w3, y[3], fmaf(w2, y[2], w1 * y[1]));
    p[3] = fmaf(w3, z[3], fmaf(w2, z[2], w1 * z[1]));
    p[4] = s.y;
}

template <class A, class Value>
__device__ __forceinline__ Moments<float> bgk_moments(const A &a, const Value &value, float phip, float s0) {
    float p0[5], p1[5];
    half_sums<0>(value, p0);
    half_sums<1>(value, p1);
    Moments<float> m;
    m.rho = p0[0] + p1[0];
    m.ux = p0[1] + p1[1];
    m.uy = __fadd_rn(p0[2] + p1[2], __fmul_rn(0.5f, __fmul_rn(a.gb, __fsub_rn(phip, a.t0))));
    m.uz = p0[3] + p1[3];
    m.phi = (p0[4] + p1[4]) + s0;   // sum w_i (gh_i + s0)
    if (a.use_phi_fix) m.phi = a.phi_fix;
    return m;
}

// Both relaxations are affine maps of the old value, with per-node
// coefficients (k = kf (c_y - u_y) takes three values, one per c_y):
//   fh* = (1 - om_f) fh + (om_f rho + k) + (om_f + k) p
//   gh* = (1 - om_g) gh + om_g (phi - s0) + om_g phi p
// and p_I, p_J = (q +/- 2 eu) / 2 with q = eu^2 - 3 u^2: two paired
// multiply-adds per population and three per pair.  With the folded shift:
// ag (v + c_y fold) + ... + c_y fold = ag v + ... + (ag + 1) c_y fold.
template <class S, bool SWAPPED, bool PERIODIC, int INTERIOR, class A, class Value>
__device__ __forceinline__ void bgk_relax_store(const A &a, const Node &g, const Value &value,
                                                const Moments<float> &m, const Shift &sh) {
    const float om_f = a.omega_f, om_g = a.omega_g, s0 = sh.s0;
    const float ux3 = 3.f * m.ux, uy3 = 3.f * m.uy, uz3 = 3.f * m.uz;
    const float uv = 3.f * (m.ux * m.ux + m.uy * m.uy + m.uz * m.uz);
    const float kf = 3.f * a.force_fac * (a.gb * (m.phi - a.t0));
    const float k_m = kf * (-1.f - m.uy), k_0 = kf * (-m.uy), k_p = kf * (1.f - m.uy);
    const float af = 1.f - om_f, orho = om_f * m.rho;
    const float c0[3] = {orho + k_m, orho + k_0, orho + k_p};   // indexed by c_y + 1
    const float c1[3] = {om_f + k_m, om_f + k_0, om_f + k_p};
    const float ag = 1.f - om_g, d1 = om_g * m.phi, d0 = om_g * (m.phi - s0);
    const float df = (ag + 1.f) * sh.fold;
    const float d0c[3] = {d0 - df, d0, d0 + df};
    const float2 a2 = make_float2(af, ag);
    // (fh, gh) <- (af fh + c1 p + c0, ag gh + d1 p + d0c): both at once
    auto relax = [&](auto kk, float p) {
        constexpr int K = decltype(kk)::value, Y = cy(K) + 1;
        const float2 v = fma2(a2, value(kk), fma2(make_float2(c1[Y], d1), splat(p), make_float2(c0[Y], d0c[Y])));
        float gv = v.y;
        if (meets_plate<PERIODIC, INTERIOR, K>(g))
            gv = 2.f * (cy(K) < 0 ? a.t_hot : a.t_cold) * (1.f + m.rho) - gv - 2.f * s0;
        if constexpr (!(SWAPPED && all_inside<INTERIOR, PERIODIC>())) gv += write_shift<SWAPPED, K, INTERIOR>(g, sh.t_dy);
        store_word<S, SWAPPED, PERIODIC, INTERIOR, K>(a, g, Pack16<S>::pack(v.x, gv));
    };
    relax(std::integral_constant<int, 0>{}, -0.5f * uv);
    // corners, edges, faces: of the orders tried, the one whose registers
    // spill least where it costs (closed box, swapped layout: 0.4% less time at
    // 256^3 FP16S and 11% less at 192x96x192 BF16S than in index order)
    auto pairs = [&](auto cls) {
        Unroll<1, Q>::run([&](auto ii) {
            constexpr int I = decltype(ii)::value;
            constexpr int J = opp(I);
            if constexpr (I < J && wclass(I) == decltype(cls)::value) {
                float eu = 0.f;
                if (cx(I) > 0) eu += ux3;
                if (cx(I) < 0) eu -= ux3;
                if (cy(I) > 0) eu += uy3;
                if (cy(I) < 0) eu -= uy3;
                if (cz(I) > 0) eu += uz3;
                if (cz(I) < 0) eu -= uz3;
                const float q = fmaf(eu, eu, -uv);
                relax(ii, fmaf(0.5f, q, eu));
                relax(std::integral_constant<int, J>{}, fmaf(0.5f, q, -eu));
            }
        });
    };
    pairs(std::integral_constant<int, 3>{});
    pairs(std::integral_constant<int, 2>{});
    pairs(std::integral_constant<int, 1>{});
}

// ---- regularised collision ----
//
// collide_reg, operation for operation (each an explicit round-to-nearest
// one, so the single-case and the batch kernels give bitwise the same
// state).  What leaves the collision depends on the old populations only
// through 18 sums, so a population is dead once it is summed, and opposite
// directions share c.u, c.j and q; the sums of f and g and the two
// directions of a pair go two to an instruction.  B200, 256^3 FP16S, per
// step: 654 us periodic, 719 closed box, against 1157 and 1186 with all 54
// values held unpacked (128 registers, 16 warps per SM, ~1600 instructions).
struct RegSums {
    Moments<float> m;
    float sxx, syy, szz, sxy, sxz, syz;   // second moments of f
    float jx, jy, jz;                     // first moments of g
};

// value(K): (f_K, g_K)
template <class A, class Value>
__device__ __forceinline__ RegSums reg_sums(const A &a, const Value &value, float phip) {
    float2 r = {}, jx = {}, jy = {}, jz = {};   // of (f, g)
    RegSums t = {};
    Unroll<0, Q>::run([&](auto kk) {
        constexpr int K = decltype(kk)::value;
        constexpr int X = cx(K), Y = cy(K), Z = cz(K);
        const float2 v = value(kk);
        r = add2(r, v);
        if (X != 0) jx = X > 0 ? add2(jx, v) : sub2(jx, v);
        if (Y != 0) jy = Y > 0 ? add2(jy, v) : sub2(jy, v);
        if (Z != 0) jz = Z > 0 ? add2(jz, v) : sub2(jz, v);
        if (X != 0) t.sxx = add_rn(t.sxx, v.x);
        if (Y != 0) t.syy = add_rn(t.syy, v.x);
        if (Z != 0) t.szz = add_rn(t.szz, v.x);
        if (X * Y != 0) t.sxy = X * Y > 0 ? add_rn(t.sxy, v.x) : sub_rn(t.sxy, v.x);
        if (X * Z != 0) t.sxz = X * Z > 0 ? add_rn(t.sxz, v.x) : sub_rn(t.sxz, v.x);
        if (Y * Z != 0) t.syz = Y * Z > 0 ? add_rn(t.syz, v.x) : sub_rn(t.syz, v.x);
    });
    t.m.rho = r.x;
    t.m.ux = jx.x;
    t.m.uy = add_rn(jy.x, mul_rn(0.5f, mul_rn(a.gb, sub_rn(phip, a.t0))));
    t.m.uz = jz.x;
    t.m.phi = r.y;
    if (a.use_phi_fix) t.m.phi = a.phi_fix;
    t.jx = jx.y;
    t.jy = jy.y;
    t.jz = jz.y;
    return t;
}

// The collision from the sums; put(K, f*_K, g*_K) takes the populations.
template <class A, class Put> __device__ __forceinline__ void reg_relax(const A &a, const RegSums &t, const Put &put) {
    const Moments<float> &m = t.m;
    const float third = 1.f / 3.f;
    const float rho3 = mul_rn(m.rho, third);
    const float pxx = fma_rn(-m.ux, m.ux, sub_rn(t.sxx, rho3));
    const float pyy = fma_rn(-m.uy, m.uy, sub_rn(t.syy, rho3));
    const float pzz = fma_rn(-m.uz, m.uz, sub_rn(t.szz, rho3));
    const float pxy2 = mul_rn(2.f, fma_rn(-m.ux, m.uy, t.sxy));
    const float pxz2 = mul_rn(2.f, fma_rn(-m.ux, m.uz, t.sxz));
    const float pyz2 = mul_rn(2.f, fma_rn(-m.uy, m.uz, t.syz));
    const float tr3 = mul_rn(add_rn(add_rn(pxx, pyy), pzz), third);
    const float jx = fma_rn(-m.phi, m.ux, t.jx), jy = fma_rn(-m.phi, m.uy, t.jy), jz = fma_rn(-m.phi, m.uz, t.jz);
    const float keep_f = mul_rn(4.5f, sub_rn(1.f, a.omega_f)), keep_g = mul_rn(3.f, sub_rn(1.f, a.omega_g));
    const float uv = mul_rn(3.f, fma_rn(m.uz, m.uz, fma_rn(m.uy, m.uy, mul_rn(m.ux, m.ux))));
    const float kf = mul_rn(mul_rn(3.f, a.force_fac), mul_rn(a.gb, sub_rn(m.phi, a.t0)));
    const float k[3] = {mul_rn(kf, sub_rn(-1.f, m.uy)), mul_rn(kf, sub_rn(0.f, m.uy)), mul_rn(kf, sub_rn(1.f, m.uy))};
    {   // the rest population
        const float w = (float)wd(0);
        const float p = add_rn(0.f, mul_rn(0.5f, -uv));
        const float feq0 = mul_rn(w, add_rn(1.f, p));
        const float fneq = mul_rn(mul_rn(keep_f, w), -tr3);
        const float fv = add_rn(add_rn(mul_rn(w, add_rn(m.rho, p)), fneq), mul_rn(k[1], feq0));
        put(std::integral_constant<int, 0>{}, fv, mul_rn(m.phi, feq0));
    }
    Unroll<1, Q>::run([&](auto ii) {
        constexpr int I = decltype(ii)::value;
        constexpr int J = opp(I);
        constexpr int X = cx(I), Y = cy(I), Z = cz(I);
        if constexpr (I < J) {
            // c.u, c.j in the order x, y, z (of J: the negatives); q of both
            auto dot = [](float x, float y, float z) {
                float d = X > 0 ? x : -x;
                if constexpr (Y != 0) d = X != 0 ? (Y > 0 ? add_rn(d, y) : sub_rn(d, y)) : Y > 0 ? y : -y;
                if constexpr (Z != 0) d = X != 0 || Y != 0 ? (Z > 0 ? add_rn(d, z) : sub_rn(d, z)) : Z > 0 ? z : -z;
                return d;
            };
            const float w = (float)wd(I);
            const float eu = mul_rn(3.f, dot(m.ux, m.uy, m.uz)), cj = dot(jx, jy, jz);
            float q = -tr3;
            if (X != 0) q = add_rn(q, pxx);
            if (Y != 0) q = add_rn(q, pyy);
            if (Z != 0) q = add_rn(q, pzz);
            if (X * Y != 0) q = X * Y > 0 ? add_rn(q, pxy2) : sub_rn(q, pxy2);
            if (X * Z != 0) q = X * Z > 0 ? add_rn(q, pxz2) : sub_rn(q, pxz2);
            if (Y * Z != 0) q = Y * Z > 0 ? add_rn(q, pyz2) : sub_rn(q, pyz2);
            // lanes: I, J
            const float2 p = add2(make_float2(eu, -eu), splat(mul_rn(0.5f, fma_rn(eu, eu, -uv))));
            const float2 feq0 = mul2(splat(w), add2(splat(1.f), p));
            const float2 force = product(make_float2(k[1 + Y], k[1 - Y]), feq0);
            const float2 feq = product(splat(w), add2(splat(m.rho), p));
            const float2 fv = add2(add2(feq, splat(mul_rn(mul_rn(keep_f, w), q))), force);
            const float2 gv = fma2(splat(mul_rn(keep_g, w)), make_float2(cj, -cj), mul2(splat(m.phi), feq0));
            put(ii, fv.x, gv.x);
            put(std::integral_constant<int, J>{}, fv.y, gv.y);
        }
    });
}

// ---- one node ----

// Moments of node g on the path INTERIOR, then (with STORE) its collision and
// its stores.  fold: whether the BGK collision folds the node's shift, all its
// neighbours being inside (see Shift).
template <class S, bool SWAPPED, bool PERIODIC, int COLL, int INTERIOR, bool STORE, class A, class Sink>
__device__ __forceinline__ Moments<float> update_path16(const A &a, const Node &g, bool fold, const Sink &sink) {
    const float phip = a.phip[g.n];
    const bool folded = COLL == LBM_COLLISION_BGK && SWAPPED && (all_inside<INTERIOR, PERIODIC>() || fold);
    const Shift sh = {shift0(a, g), folded ? 0.f : (float)a.t_dy, folded ? (float)a.t_dy : 0.f};
    typename Pack16<S>::T w[Q];
    Unroll<0, Q>::run([&](auto kk) {
        constexpr int K = decltype(kk)::value;
        w[K] = load_pair<S, SWAPPED, PERIODIC, K, INTERIOR>(a, g);
    });
    if constexpr (COLL == LBM_COLLISION_REGULARIZED) {
        auto value = [&](auto kk) {   // w_K (fh, gh + T_c at the location)
            constexpr int K = decltype(kk)::value;
            const float2 v = Pack16<S>::unpack(w[K]);
            const float at = add_rn(sh.s0, read_shift<SWAPPED, K, INTERIOR>(g, sh.t_dy));
            return product(splat((float)wd(K)), make_float2(v.x, add_rn(v.y, at)));
        };
        const RegSums t = reg_sums(a, value, phip);
        if constexpr (STORE) {
            sink(t.m);
            const Node gs = again(a, g);
            a.phip[gs.n] = t.m.phi;
            // normalised and relative to T_c where it goes
            reg_relax(a, t, [&](auto kk, float fv, float gv) {
                constexpr int K = decltype(kk)::value;
                if (meets_plate<PERIODIC, INTERIOR, K>(gs)) gv = abb<K>(gv, cy(K) < 0 ? a.t_hot : a.t_cold, t.m.rho);
                const float sl = sub_rn(sh.s0, write_shift<SWAPPED, K, INTERIOR>(gs, sh.t_dy));
                store_word<S, SWAPPED, PERIODIC, INTERIOR, K>(
                    a, gs, Pack16<S>::pack(mul_rn(fv, (float)winv(K)), fma_rn(gv, (float)winv(K), -sl)));
            });
        }
        return t.m;
    } else {
        auto value = [&](auto kk) {   // gh relative to the node's T_c (folded: as stored)
            constexpr int K = decltype(kk)::value;
            float2 v = Pack16<S>::unpack(w[K]);
            if constexpr (!(SWAPPED && all_inside<INTERIOR, PERIODIC>())) v.y += read_shift<SWAPPED, K, INTERIOR>(g, sh.t_dy);
            return v;
        };
        const Moments<float> m = bgk_moments(a, value, phip, sh.s0);
        if constexpr (STORE) {
            sink(m);
            const Node gs = again(a, g);
            a.phip[gs.n] = m.phi;
            bgk_relax_store<S, SWAPPED, PERIODIC, INTERIOR>(a, gs, value, m, sh);
        }
        return m;
    }
}

// Two bodies only, and nothing but the node crosses the branch.  A closed
// box's rows take one body whether or not a warp holds an x-wall node, with
// the x-moving addresses by a select: a third body for the warps without one
// saves its warps the selects but competes for the instruction cache (B200,
// closed-box swapped step, BGK: 2% more time at 256^3 FP16S with three bodies,
// 6% at 192x96x192 BF16S).
//
// With ONE_BODY (periodic sides) a warp takes one body, the tested one if any
// of its nodes needs it (rows that are not whole warps): a warp that took both
// would wait for two rounds of loads and run twice the instructions, which on
// grids of small members and in small grids is most of the time (B200, two
// cases of 16^3 FP16S on their own kernels: 3.7 us per step, 4.7 with both).
// Large grids have few such warps and do better without the vote's registers
// (ensemble of 32, 0.7%), and a closed box's tested body would have to fold
// too, whose spills cost the whole warps more (85 to 96 us per step at 128^3
// BF16S).  The results are the same, bit for bit.
template <class S, bool SWAPPED, bool PERIODIC, int COLL, bool STORE, bool ONE_BODY, class A, class Sink>
__device__ __forceinline__ Moments<float> update_node16(const A &a, const Node &g, const Sink &sink) {
    if constexpr (PERIODIC && ONE_BODY) {
        const bool inner = yz_interior<PERIODIC>(g);
        if (one_body(a, g, inner))
            return update_path16<S, SWAPPED, PERIODIC, COLL, kRowInside, STORE>(a, g, inner, sink);
        return update_path16<S, SWAPPED, PERIODIC, COLL, kNoneInside, STORE>(a, g, inner, sink);
    } else {
        const int path = node_path<PERIODIC, SWAPPED>(g);
        if (path != kNoneInside)
            return update_path16<S, SWAPPED, PERIODIC, COLL, kRowInside, STORE>(a, g, path == kAllInside, sink);
        return update_path16<S, SWAPPED, PERIODIC, COLL, kNoneInside, STORE>(a, g, false, sink);
    }
}

// The moments of node g as the 16-bit step forms them (a closed box's rows by
// the vote that the step takes over the same nodes), so observables reduced
// from them match those an observed step reduces.
template <class S, bool SWAPPED, bool PERIODIC, int COLL, class A>
__device__ __forceinline__ Moments<float> step_moments16(const A &a, const Node &g) {
    return update_node16<S, SWAPPED, PERIODIC, COLL, false, false>(a, g, NoMomentSink{});
}

// FP32 with the regularised collision, likewise: 54 values loaded, 18 sums
// kept, two bodies.  B200, 256^3: 1112 us per step in the natural layout and
// 1162 in the swapped one (0.99 of the copy rate), against 1636 and 1748 with
// collide_reg, whose ~1100 FP32 operations per node bound it; bitwise its
// results.
template <bool SWAPPED, bool PERIODIC, int INTERIOR, class A, class Sink>
__device__ __forceinline__ Moments<float> update_reg32(const A &a, const Node &g, const Sink &sink) {
    const float phip = a.phip[g.n];
    float fr[Q], gr[Q];
    gather<float, SWAPPED, INTERIOR>(a, g, fr, gr);
    const RegSums t = reg_sums(
        a, [&](auto kk) { return make_float2(fr[decltype(kk)::value], gr[decltype(kk)::value]); }, phip);
    sink(t.m);
    const Node gs = again(a, g);
    a.phip[gs.n] = t.m.phi;
    reg_relax(a, t, [&](auto kk, float fv, float gv) {
        constexpr int K = decltype(kk)::value;
        if (meets_plate<PERIODIC, INTERIOR, K>(gs)) gv = abb<K>(gv, cy(K) < 0 ? a.t_hot : a.t_cold, t.m.rho);
        store_pop<SWAPPED, INTERIOR, K>(a, gs, 0, fv);
        store_pop<SWAPPED, INTERIOR, K>(a, gs, 1, gv);
    });
    return t.m;
}

template <class S, bool SWAPPED, bool PERIODIC, int COLL, bool ONE_BODY, class A, class Sink = NoMomentSink>
__device__ __forceinline__ NodeOut<typename Codec<S>::R> update_node(const A &a, uint32_t n,
                                                                     const Sink &sink = Sink()) {
    if constexpr (sizeof(S) == 2) {
        const Node g = make_node<PERIODIC>(a, n);
        return {update_node16<S, SWAPPED, PERIODIC, COLL, true, ONE_BODY>(a, g, sink), g.iy};
    } else if constexpr (sizeof(S) == 4 && COLL == LBM_COLLISION_REGULARIZED) {
        const Node g = make_node<PERIODIC>(a, n);
        // bodies as in update_node16
        const bool inner = yz_interior<PERIODIC>(g);
        return {(PERIODIC && ONE_BODY ? one_body(a, g, inner) : inner)
                    ? update_reg32<SWAPPED, PERIODIC, kRowInside>(a, g, sink)
                    : update_reg32<SWAPPED, PERIODIC, kNoneInside>(a, g, sink),
                g.iy};
    } else {
    using R = typename Codec<S>::R;
    const Node g = make_node<PERIODIC>(a, n);
    R fr[Q], gr[Q];
    // Rows away from the plates (and, in a closed box, from the z walls)
    // need no y or z boundary tests; the path is uniform over a warp whenever
    // LX is a multiple of 32.  In FP32 a closed box's warps with no x-wall
    // node take a body with no test at all in the swapped layout, the one
    // whose accesses depend on them.  FP64 bodies are the longest, and a
    // third one costs more in instruction fetches than its warps save (B200,
    // 256^3 closed box, swapped step: 2334 us with two, 2370 with three, 2395
    // with a body for each x wall too; FP32 1353, 1324 and 1368).
    constexpr bool kThree = sizeof(S) == 4 && SWAPPED && !PERIODIC;
    const int path = node_path<PERIODIC, kThree>(g);
    if (path == kRowInside)
        gather<S, SWAPPED, kRowInside>(a, g, fr, gr);
    else if (kThree && path == kAllInside)
        gather<S, SWAPPED, kThree ? kAllInside : kRowInside>(a, g, fr, gr);
    else
        gather<S, SWAPPED, kNoneInside>(a, g, fr, gr);
    const Moments<R> m = node_moments<S>(a, fr, gr, n);
    sink(m);
    collide<S, COLL>(fr, gr, m, a);
    const Node gs = again(a, g);
    a.phip[gs.n] = (typename Codec<S>::P)m.phi;
    if (path == kRowInside)
        scatter<S, SWAPPED, PERIODIC, kRowInside>(a, gs, fr, gr, m.rho);
    else if (kThree && path == kAllInside)
        scatter<S, SWAPPED, PERIODIC, kThree ? kAllInside : kRowInside>(a, gs, fr, gr, m.rho);
    else
        scatter<S, SWAPPED, PERIODIC, kNoneInside>(a, gs, fr, gr, m.rho);
    return {m, g.iy};
    }
}

// For a launch that may start before the previous kernel of its stream is
// done (programmatic dependent launch; passes at once without that
// attribute): returns when that kernel has completed and its writes are
// visible, so nothing before it may touch global memory.  The previous
// kernel lets this one start as its blocks exit; letting it start earlier
// puts its blocks into the slots a small grid leaves free, unevenly over the
// SMs (B200, 32^3 FP64: 9.1 us per step against 5.9).
__device__ __forceinline__ void await_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// One time step.  With OBS, the kernel also reduces the observables of the
// state it reads — the moments every node update computes anyway — into one
// row of FP64 sums per warp (row W b + w for warp w of block b, W =
// node_threads / 32: the nodes [32 row, 32 row + 32)), at no extra read of
// the populations.
template <class S, bool SWAPPED, bool PERIODIC, int COLL, bool OBS = false, bool SMALL = false>
__global__ void __launch_bounds__(bound_threads<S>(), step_budget<S, COLL, SMALL>() / bound_threads<S>())
    step_kernel(const StepArgs<S> a) {
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    await_previous();
    if constexpr (!OBS) {
        if (n >= a.nodes) return;
        update_node<S, SWAPPED, PERIODIC, COLL, SMALL>(a, n);
    } else {
        using T = typename Codec<S>::R;
        constexpr int kT = node_threads<S>();
        __shared__ T parked[5][kT];   // ux, uy, uz, phi, rho per thread
        // the terms of add_obs_terms: uy*phi, |u|^2, ux, uy, uz, phi
        double d[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        int iy = 0;
        bool bad = false;
        const bool valid = n < a.nodes;
        if (valid) {
            volatile T *mine = &parked[0][threadIdx.x];
            iy = update_node<S, SWAPPED, PERIODIC, COLL, SMALL>(a, n, SharedMomentSink<T, kT>{mine}).iy;
            const double ux = mine[0], uy = mine[kT], uz = mine[2 * kT], phi = mine[3 * kT], rho = mine[4 * kT];
            d[0] = uy * phi;
            d[1] = ux * ux + uy * uy + uz * uz;
            d[2] = ux;
            d[3] = uy;
            d[4] = uz;
            d[5] = phi;
            bad = !isfinite(ux) || !isfinite(uy) || !isfinite(uz) || !isfinite(phi) || !isfinite(rho);
        }
        const size_t warp_row = (size_t)blockIdx.x * (node_threads<S>() / 32) + (threadIdx.x >> 5);
        warp_obs_row(d, iy, valid, bad, a.ly, warp_row, a.obs_rows, a.obs_planes);
    }
}

}  // namespace lbm
