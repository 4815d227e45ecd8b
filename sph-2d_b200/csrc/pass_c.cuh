// pass_c.cuh -- neighbour pass C: the fused force pass.  One thread per
// particle gathers, for every pair neighbour, the linear-Riemann flux (with
// optional MUSCL reconstruction), continuity, pressure force, Monaghan
// artificial viscosity, Morris laplacian, delta-alpha term, SPS force, XSPH,
// delta-SPH density diffusion and (on the last RHS of a step, FP64 and
// moving-square launches) the shifting sum; the mixed Taylor-Green path forms
// the shifting sum in k_shift_gather after this pass.
//
// Reference loops (all in pair order, scattered to pair_i and pair_j):
//   Solver_Normalized_Modified_Linear_Riemann_Delta_SPS.f90:300-502, 552-583, 627-635
//   Solver_Normalized_MUSCL_Linear_Riemann_Delta_SPS.f90:458-682, 690-721
//   Solver_Normalized_Delta_SPH_SPS.f90:324-512, 610-636 (the plain method)
//   MUSCL_Limiter: function_module.f90:34-80
//   Shift_particle_position.f90:78-103
//   assembly: single_step_compute.f90:152-171
//
// The flux seen by the two particles of a pair comes from the same bits: either in
// the reference's own orientation (pair_i = the particle with the lower id, bit 31
// of the list entry; the moving-square launches and the mixed ones without MUSCL),
// or in the particle's own frame, where negation is exact and only the MUSCL
// limiter looks at the orientation (AB, the other launches).  Each thread keeps the
// contribution that belongs to its particle.  The physical terms are summed per pair and then
// accumulated (the reference sums each term over all pairs first); the two
// orders agree to round-off.
//
// Precision: R = double is the FP64 path.  R = float is the mixed path: FP32
// pair arithmetic with reciprocal/rsqrt instead of divisions, FP64 sums of
// the FP32 terms for the acceleration and the density rate, and the shifting
// sum in FP64 (its terms are O(h/10) each and cancel to a displacement that
// is orders of magnitude smaller, so FP32 rounding there would inject position
// noise every step into the unstable lattice modes the shifting excites).
#pragma once
#include "pass_a.cuh"

namespace sph {

// The MUSCL limiter (function_module.f90:34-80) of one field, for particle a of
// the pair (a, b), written without the pair's orientation.  With A = -1/2 grad
// phi_a.(x_a - x_b) and B = 1/2 grad phi_b.(x_a - x_b) the reference's arguments are
// (di, dj) = (A, B) when a is pair_i and (B, A) when it is pair_j, and
// dij = phi_j - phi_i = -sgn dphi with dphi = phi_a - phi_b, sgn = +-1.  Folding
// its two sign branches (the dj <= 0 branch is the dj > 0 one on (-di, -dj),
// negated) its value is
//   lim = s max(0, max(min(1.3 s di, s dj), min(s di, 1.3 s dj))),  s = sign(dj),
// replaced by dij/2 for one side and 0 for the other when s lim > s dij/2.  lim is
// symmetric in di and dj (it is 0 when their signs differ), so s and both
// products can be taken from (A, B) directly; the side that keeps dij/2 is the
// one with the larger s d, which is a when s A > s B (or >= when a is pair_j).
// Returned: L = sgn (li + lj), the sum in a's frame, and own, a's increment times
// sgn; flip = the sign bit of sgn.
//
// FP32: with the arguments selected by a_is_i (the form without the selects has
// fewer instructions between the neighbour-record loads and measured 1 % slower:
// mixed pass C 2.77 -> 2.80 ms per step at 2048^2).
__device__ __forceinline__ void muscl_limiter(float A, float B, float dphi, bool a_is_i, unsigned, float& L,
                                              float& own) {
    const float sgn = a_is_i ? 1.f : -1.f;
    const float di = a_is_i ? A : B, dj = a_is_i ? B : A, dij = -(sgn * dphi);
    const unsigned sb = __float_as_uint(dj) & 0x80000000u;
    const float sdi = __uint_as_float(__float_as_uint(di) ^ sb), sdj = fabsf(dj);
    const float m = fmaxf(0.f, fmaxf(fminf(1.3f * sdi, sdj), fminf(sdi, 1.3f * sdj)));
    const float half = 0.5f * dij;
    const bool big = m > __uint_as_float(__float_as_uint(half) ^ sb) && m > 0.f;
    const bool first = sdi > sdj;
    const float lim = __uint_as_float(__float_as_uint(m) ^ sb);
    L = sgn * (big ? half : 2.f * lim);
    own = sgn * (big ? (first == a_is_i ? half : 0.f) : lim);
}
// FP64: without the selects (a 64-bit select is two instructions); multiplying by
// s or sgn is a flip of the sign bit in the high word, so the only use of a_is_i
// is the tie, and both members of a pair form the same bits.
__device__ __forceinline__ double flip_sign(double v, int hi_bit) {
    return __hiloint2double(__double2hiint(v) ^ hi_bit, __double2loint(v));
}
__device__ __forceinline__ void muscl_limiter(double A, double B, double dphi, bool a_is_i, unsigned flip, double& L,
                                              double& own) {
    const int sb = __double2hiint(B) & (int)0x80000000u;
    const double x = flip_sign(A, sb), y = fabs(B);
    // max(min(1.3 x, y), min(x, 1.3 y)) = min(1.3 min(x, y), max(x, y)) for x, y >= 0
    // (for x <= 0 both are <= 0 and m = 0)
    const bool gt = x > y;
    const double lo = gt ? y : x, hi = gt ? x : y;
    const double l3 = 1.3 * lo;
    const double m = l3 < hi ? l3 : hi;
    const double hb = -0.5 * dphi;
    const int t = sb ^ (int)flip;
    const bool pos = x > 0.0;                        // with y > 0 too: m > 0
    const bool big = pos && m > flip_sign(hb, t) && m > 0.0;
    const bool mine = gt || (x == y && !a_is_i);
    const double lim = pos ? flip_sign(m, t) : 0.0;
    L = big ? hb : 2.0 * lim;
    own = big ? (mine ? hb : 0.0) : lim;
}

// Reciprocal and quotient in the pair loop.  FP32: correctly rounded, except the
// 1/rho-bar and artificial-viscosity quotient (fast_quot: __fdividef, about 2
// ulp).  Fast forms everywhere made mixed pass C slower (3.46 -> 3.85 ms
// per step at 2048^2: fewer instructions between the neighbour-record loads);
// these two alone took it from 2.80 to 2.75 ms with the velocity L2 against
// FP64 unchanged (2.78e-6 after 100 steps).  FP64: the Newton reciprocal.
__device__ __forceinline__ double rcp(double x) { return rcp64(x); }
__device__ __forceinline__ float rcp(float x) { return __frcp_rn(x); }
template <typename R>
__device__ __forceinline__ R quot(R a, R b) { return a / b; }
__device__ __forceinline__ double fast_quot(double a, double b) { return a * rcp64(b); }
__device__ __forceinline__ float fast_quot(float a, float b) { return __fdividef(a, b); }

// Is a near the free surface (Define_freesurface...f90:418-440: a pair neighbour
// is a surface particle)?  The pair lists are symmetric, so a's own list decides;
// they are only searched at an RHS where pass A found a surface particle.  The
// mark (bit 1) is kept for the shift and for the host; the other threads read
// only bit 0, which this store does not change.
template <typename R>
__device__ __forceinline__ bool near_surface(const Params& P, const Sorted<R>& D, int a, int nn) {
    if (!P.free_surface || *D.surf_gen != P.rhs_gen) return false;
    bool near = false;
    for (int e = 0; e < nn && !near; ++e)
        near = (D.flags[D.pairs[(size_t)e * P.nbr_stride + a] & 0x7fffffffu] & 1) != 0;
    if (near) D.flags[a] = D.flags[a] | 2;
    return near;
}

// Per-particle state a thread needs for one side of a pair.
template <typename R>
struct Side {
    using V4 = typename VT<R>::V4;
    double4 kin;   // u, v, rho, p (FP64)
    float4 kh, kl; // the same, hi + lo (mixed Taylor-Green variants)
    V4 aux;        // m, V, c, smass
    V4 nb1, nb2, nb3;
};

// The pair terms are written with the pair differences du = u_i - u_j,
// dv = v_i - v_j, dp = p_i - p_j, drho = rho_j - rho_i formed in FP64 from the
// kinematic records; in real arithmetic this is the reference's expression,
// e.g. v_i - v* = (v_i - v_j)/2 - (U* - Ubar) e for the modified solver.
// MS: the moving-square solvers (HLLC or modified linear with XSPH in the
// continuity flux, laplacian switch, no SPS); SHIFT: the last RHS of a step with
// shifting on, which also forms the shifting sum.  Both are compile-time so that
// each launch carries only the registers of the terms it evaluates.
#ifndef SPH_PASS_C_SHIFT_BLOCKS
#define SPH_PASS_C_SHIFT_BLOCKS 4
#endif
#ifndef SPH_PASS_C_F32_BLOCKS
#define SPH_PASS_C_F32_BLOCKS 4
#endif
//
// The stage that follows the RHS is applied here (StageArgs), on the particle's
// own sums: a stage pass of its own read back the rates and the whole state and
// ran at HBM speed while this kernel leaves HBM at a tenth of its rate.  2048^2,
// ms per step, pass C + update: mixed 2.77 + 1.18 -> 3.06 + 0.45, FP64
// 5.48 + 0.85 -> 6.24; 401^2 mixed 140 + 81 -> 158 + 27 us.
//
// FP64 at 2048^2 (MUSCL, ms per step of three launches): 7.30 with correctly
// rounded square roots, reciprocals and quotients and the limiter's and frame's
// 64-bit selects; 6.02 with rsqrt64 / rcp64, m_b/rho_b read as V_b, the
// orientation-free limiter and 256-bit record loads; 5.46 with the neighbour's
// records loaded one iteration ahead (kept: 168 registers, 3 blocks per SM; 4
// blocks without the prefetch 5.89).  ncu at 1024^2, 398 -> 270 M warp
// instructions, 654 -> 431 us: FP64 pipe 50 % busy, L1 data stage 67 % (176 B of
// records per neighbour), 58 % issue-active, the rest waits on results (1.9 cycles
// an instruction at 3 warps a scheduler).  So branches inside the pair cost more
// than the work they skip, as they end the stretch the compiler can interleave:
// with the stages in this kernel 6.24 ms, 5.86 with the viscosity and the
// near-surface case as selects, 5.06 with the kernel model fixed at compile time
// (KM; FP64 launches).  In the mixed path it is the other way round (3.06 -> 3.27
// ms): there the branch keeps the neighbour's loads early, and KM is 0.
template <typename R, bool MUSCL, bool MS, bool SHIFT, int L = 1, int KM = 0>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? (SHIFT ? SPH_PASS_C_SHIFT_BLOCKS : SPH_PASS_C_F32_BLOCKS) : 3)
    k_pass_c(const __grid_constant__ Params P, const __grid_constant__ Sorted<R> D, const __grid_constant__ StageArgs G) {
    pdl_begin();
    stamp_phase(P.stamp);
    using V4 = typename VT<R>::V4;
    using A = typename Acc<R>::T;
    constexpr bool F32 = sizeof(R) == 4;
    // hi/lo records: every mixed variant (the moving-square HLLC state is then
    // formed in FP32 from differences, below)
    constexpr bool HL = F32;
    // the shifting sum needs the FP64 position differences: that launch reads the
    // neighbour's FP64 position (and FP64 volume) instead of its hi/lo position
    // and takes the FP32 difference as the rounding of the FP64 one
    constexpr bool X64 = !HL || SHIFT;
    const Lanes<L> ln;
    const int t = Lanes<L>::particle();
    const bool live = t < P.n_tot;
    if (L == 1 && !live) return;
    const int a = live ? t : P.n_tot - 1;        // (every lane takes part in the sums)
    const int ta = D.type[a];
    const int nn = live ? D.npairs[a] : 0;
    const double2 xa = X64 ? D.pos[a] : make_double2(0.0, 0.0);
    float4 xa_hl = make_float4(0.f, 0.f, 0.f, 0.f);
    Side<R> S;
    if (HL) { S.kh = D.kh[a]; S.kl = D.kl[a]; }
    if (!X64) xa_hl = D.xhl[a];
    else S.kin = D.kin[a];
    S.aux = D.aux[a]; S.nb1 = D.nb1[a]; S.nb2 = D.nb2[a];
    if (MUSCL) S.nb3 = D.nb3[a];
    const R rho_a = HL ? (R)S.kh.z : (R)S.kin.z;
    const V4 bi = D.binv[a];
    // Solver_Normalized_Delta_SPH_SPS has no Riemann state: its continuity and
    // pressure terms (:333-374) are the pair-mean (v-bar, P-bar) form the Riemann
    // solvers use near the free surface, so it takes that branch for every pair
    const bool dsph = !MUSCL && !MS && P.dsph;
    const bool near_a = near_surface(P, D, a, nn) || dsph;
    // delta-SPH and the assembly only apply to integrated particles (Solver :627-635,
    // Moving_Square.../Single_step_compute.f90:273-281)
    const bool water = integrated(P, ta);
    typename VT<R>::V2 avg_a = mk2<R>(R(0), R(0));
    if (MS) avg_a = D.avg[a];

    const bool gauss = KM ? KM == SPH_KERNEL_GAUSSIAN : P.kernel_model == SPH_KERNEL_GAUSSIAN;
    const R hbar = (R)P.h;
    const R inv_h = (R)P.inv_h;
    const R gk = (R)P.gk;
    const R inv_sqc0 = (R)P.inv_sqrt_c0;
    const R nu2 = (R)(2.0 * P.nu), alpha = (R)P.alpha, beta = (R)P.beta;
    const R fh2 = (R)((P.fai * P.h) * (P.fai * P.h));
    const R dlt2h = (R)(2.0 * P.delta * P.h);
    const R dla_dh = (R)(P.delta * P.h);
    const R dla_h = (R)(P.delta_alpha * P.h);
    const R eps2 = (R)(2.0 * P.eps);
    // 1/rho: the MUSCL records carry it (nb3.w)
    constexpr bool RREC = MUSCL;
    const R inv_rho_a = RREC ? (R)S.nb3.w : rcp(rho_a);
    const R rho0_over_rho_a = (R)P.rho0 * inv_rho_a;
    const R dla_rho = dla_h * rho0_over_rho_a;

    A cont, accx, accy;
    cont.init(); accx.init(); accy.init();
    R xsx = R(0), xsy = R(0);
    double shx = 0.0, shy = 0.0;   // shifting sum, FP64 in both paths
    const double inv_h64 = P.inv_h, inv_h2_64 = P.inv_h2, inv_wdx = 1.0 / P.w_dx;

    // the pairs pass A found inside the support at this RHS
    unsigned ent_n = nn > ln.lane ? load(&D.pairs[(size_t)ln.lane * P.nbr_stride + a]) : 0u;
    // software pipeline: the pair entry two iterations ahead; the neighbour's
    // position and its records one iteration ahead
    unsigned ent_nn = nn > ln.lane + L ? load(&D.pairs[(size_t)(ln.lane + L) * P.nbr_stride + a]) : 0u;
    double2 xb_n = make_double2(0.0, 0.0);
    float4 xbhl_n = make_float4(0.f, 0.f, 0.f, 0.f);
    double vd_n = 0.0;                 // FP64 volume, mixed SHIFT launch
    constexpr bool VPRE = HL && SHIFT;
    Side<R> T_n;
    auto load_records = [&](int bb, Side<R>& t) {
        if (HL) { t.kh = D.kh[bb]; t.kl = D.kl[bb]; }
        else t.kin = load4(&D.kin[bb]);
        t.aux = load4(&D.aux[bb]); t.nb1 = load4(&D.nb1[bb]); t.nb2 = load4(&D.nb2[bb]);
        if (MUSCL) t.nb3 = load4(&D.nb3[bb]);
    };
    if (nn > ln.lane) {
        const int b0 = (int)(ent_n & 0x7fffffffu);
        if (X64) xb_n = load(&D.pos[b0]);
        else xbhl_n = load(&D.xhl[b0]);
        if (VPRE) vd_n = load(&D.vol64[b0]);
        load_records(b0, T_n);
    }
    for (int e = ln.lane; e < nn; e += L) {
        const unsigned ent = ent_n;
        const int b = (int)(ent & 0x7fffffffu);
        const bool a_is_i = (ent >> 31) != 0;
        const double2 xb = xb_n;
        const float4 xbhl = xbhl_n;
        const double vd_b = vd_n;
        const Side<R> T = T_n;
        if (e + L < nn) {
            ent_n = ent_nn;
            const int b1 = (int)(ent_n & 0x7fffffffu);
            if (X64) xb_n = load(&D.pos[b1]);
            else xbhl_n = load(&D.xhl[b1]);
            if (VPRE) vd_n = load(&D.vol64[b1]);
            load_records(b1, T_n);
            if (e + 2 * L < nn) ent_nn = load(&D.pairs[(size_t)(e + 2 * L) * P.nbr_stride + a]);
        }
        // x_a - x_b: FP64, or hi/lo in FP32 (the mixed SHIFT launch: the FP32
        // rounding of the FP64 difference, which its shifting sum needs)
        double dxd = 0.0, dyd = 0.0;
        if (X64) { dxd = xa.x - xb.x; dyd = xa.y - xb.y; }
        const float dxf = !HL ? 0.f : X64 ? (float)dxd : (xa_hl.x - xbhl.x) + (xa_hl.z - xbhl.z);
        const float dyf = !HL ? 0.f : X64 ? (float)dyd : (xa_hl.y - xbhl.y) + (xa_hl.w - xbhl.w);
        R d, inv_d;
        if (F32) {
            const R s = HL ? (R)(dxf * dxf + dyf * dyf) : (R)(dxd * dxd + dyd * dyd);
            inv_d = rsqrtf(s);
            d = s * inv_d;
        } else {
            const double s = dxd * dxd + dyd * dyd;
            inv_d = (R)rsqrt64(s);
            d = (R)(s * (double)inv_d);
        }
        // the pair's i and j members (only the moving-square HLLC state reads
        // them; everything else is formed from a's and b's records directly)
        const Side<R>& I = a_is_i ? S : T;
        const Side<R>& J = a_is_i ? T : S;
        const R sgn = a_is_i ? R(1) : R(-1);
        // AB (the FP64 and the mixed MUSCL Taylor-Green launches): the pair terms are formed in a's
        // frame, x_a - x_b and phi_a - phi_b, instead of the pair's i/j frame.
        // Negation is exact, so a term odd in the orientation takes the i/j-frame
        // bits times sgn and the sgn of the final sums cancels it; only the MUSCL
        // limiter looks at the orientation.
        constexpr bool AB = !MS && (MUSCL || !F32);
        // position_difference_ij = x_i - x_j (find_particle_pair.f90:79-107) = sgn (x_a - x_b);
        // xij: that, or x_a - x_b in AB
        R xab0, xab1;
        if (HL) { xab0 = (R)dxf; xab1 = (R)dyf; }
        else { xab0 = (R)dxd; xab1 = (R)dyd; }
        const R xij0 = AB ? xab0 : sgn * xab0, xij1 = AB ? xab1 : sgn * xab1;
        const R fsg = AB ? R(1) : sgn;      // the orientation of the frame's sums
        // pair differences, FP64 or hi/lo in FP32, formed as a - b and oriented
        // by sgn: b - a is exactly -(a - b), so both members of the pair get the
        // same bits, and sums such as rho_i + rho_j are a's plus b's
        R du, dv, dp, drho_ji, rho_a_, rho_b;
        if (HL) {
            du = fsg * (R)((S.kh.x - T.kh.x) + (S.kl.x - T.kl.x));
            dv = fsg * (R)((S.kh.y - T.kh.y) + (S.kl.y - T.kl.y));
            dp = fsg * (R)((S.kh.w - T.kh.w) + (S.kl.w - T.kl.w));
            drho_ji = -(fsg * (R)((S.kh.z - T.kh.z) + (S.kl.z - T.kl.z)));
            rho_a_ = (R)S.kh.z; rho_b = (R)T.kh.z;
        } else {
            du = fsg * (R)(S.kin.x - T.kin.x); dv = fsg * (R)(S.kin.y - T.kin.y);
            dp = fsg * (R)(S.kin.w - T.kin.w);
            drho_ji = -(fsg * (R)(S.kin.z - T.kin.z));
            rho_a_ = (R)S.kin.z; rho_b = (R)T.kin.z;
        }
        // compute_kernel: W and dwdx(k) = g (x_i - x_j), g with q/(d h) = 1/h^2
        // folded into a constant (gk)
        R w, g;
        {
            const R q = d * inv_h;
            const R kf = (R)P.kfactor;
            if (gauss) {
                const R ex = exp(-(q * q));
                w = (ex - (R)P.gauss_e9) * kf;
                g = ex * gk;
            } else {
                const R t = R(1) - R(0.5) * q;
                const R t3 = t * t * t;
                w = kf * (R(1) + R(2) * q) * (t3 * t);
                g = t3 * gk;
            }
        }
        const R dw0 = g * xij0, dw1 = g * xij1;
        // Normalized_dwdx of this particle's side: B_a^-1 dwdx(k)
        const R nd0 = bi.x * dw0 + bi.y * dw1;
        const R nd1 = bi.z * dw0 + bi.w * dw1;
        const R cbar = R(0.5) * (S.aux.z + T.aux.z);
        const R rbar = R(0.5) * (rho_a_ + rho_b);
        const R inv_rbar = fast_quot(R(1), rbar);
        const R e0 = -xij0 * inv_d, e1 = -xij1 * inv_d;     // x_j - x_i direction (both solvers)
        // Riemann states.  lp, lu, lv are the sums of the MUSCL reconstruction
        // increments of both sides and ou, ov this side's (muscl_limiter, in a's
        // frame); the other solvers have none.
        R lp = R(0), lu = R(0), lv = R(0), ou = R(0), ov = R(0);
        if (MUSCL) {
            // 1/2 grad phi.(x_a - x_b) of both particles; the products are rounded
            // separately and fused in a fixed order, so both members of the pair form
            // the same bits.  nb2 = (grad rho y, grad p x, grad p y, grad u x),
            // nb3 = (grad u y, grad v x, grad v y, 1/rho); the FP32 records hold
            // 1/2 grad phi, so the halving is already done, exactly.
            auto half_dot = [&](R g0, R g1) { return (F32 ? R(1) : R(0.5)) * fma(g1, xab1, mul_rn(g0, xab0)); };
            const R gpa = half_dot(S.nb2.y, S.nb2.z), gpb = half_dot(T.nb2.y, T.nb2.z);
            const R gua = half_dot(S.nb2.w, S.nb3.x), gub = half_dot(T.nb2.w, T.nb3.x);
            const R gva = half_dot(S.nb3.y, S.nb3.z), gvb = half_dot(T.nb3.y, T.nb3.z);
            const unsigned flip = ~ent & 0x80000000u;
            R own;
            muscl_limiter(-gpa, gpb, dp, a_is_i, flip, lp, own);
            muscl_limiter(-gua, gub, du, a_is_i, flip, lu, ou);
            muscl_limiter(-gva, gvb, dv, a_is_i, flip, lv, ov);
        }
        // U_L - U_R and P_L - P_R from the differences (the frame's e0, e1 and
        // differences; the product is the i/j frame's)
        const R dU = (du + lu) * e0 + (dv + lv) * e1;
        const R Pbar = HL ? R(0.5) * ((R)S.kh.w + (R)T.kh.w) : R(0.5) * ((R)S.kin.w + (R)T.kin.w);
        R PA, wa0, wa1;          // this side's star pressure and velocity minus star velocity
        if (AB) { wa0 = R(0.5) * du + ou; wa1 = R(0.5) * dv + ov; }
        else if (a_is_i) { wa0 = R(0.5) * du; wa1 = R(0.5) * dv; }
        else { wa0 = R(-0.5) * du; wa1 = R(-0.5) * dv; }
        if (!MS || !P.hllc) {
            // dP and U* - Ubar in the frame; sU e is the same product in either
            const R dP = dp + lp;
            const R sU = R(0.5) * dP * (inv_rbar * inv_sqc0);               // U* - Ubar
            const R bR = min(R(3) * (max(dU, R(0))), cbar);
            const R Ps = Pbar + R(0.5) * bR * rbar * dU;
            PA = near_a ? Pbar : Ps;
            if constexpr (F32) {
                if (!near_a) { wa0 -= sU * e0; wa1 -= sU * e1; }
            } else {
                const R sn = near_a ? R(0) : sU;
                wa0 -= sn * e0; wa1 -= sn * e1;
            }
        } else if (near_a) {
            PA = Pbar;
        } else if (HL) {
            // The HLLC state of Moving_Square.../Solver_Normalized_HLLC_Riemann_Delta.f90:207-322
            // written in differences, so that FP32 keeps the accuracy of the hi/lo pair
            // differences (rho* and P* = c0^2 (rho_HLLC - rho0) are otherwise differences of
            // O(1) numbers).  Pair frame e (i to j) and t = (-e1, e0); dV = VR0 - VL0 =
            // -(du, dv).e; C_K = rho_K c_K; the reference's contact speed
            // U* = (VR0 C_L + VL0 C_R + P_L - P_R)/(C_L + C_R) gives
            //   sL = U* - VL0 = (C_L dV + dp)/(C_L + C_R),  sR = U* - VR0 = (dp - C_R dV)/(C_L + C_R),
            //   P* - P_L = -C_L (dp + C_R dV)/(C_L + C_R);
            // the state sampled at V0 = (VL0 + VR0)/2, V0 - VL0 = VR0 - V0 = dV/2, gives
            //   rho_HLLC - rho0 = (rho_K - rho0) [+ rho_K (U* - V_K0)/(S_K - U*) in the star regions]
            // and v_K - v* as components along e and t.
            const R rL = a_is_i ? rho_a_ : rho_b, rR = a_is_i ? rho_b : rho_a_;
            const R cL = a_is_i ? (R)S.aux.z : (R)T.aux.z, cR = a_is_i ? (R)T.aux.z : (R)S.aux.z;
            const R rho0f = (R)P.rho0;
            const R dra = (R)((S.kh.z - (float)rho0f) + S.kl.z), drb = (R)((T.kh.z - (float)rho0f) + T.kl.z);
            const R drL = a_is_i ? dra : drb, drR = a_is_i ? drb : dra;   // rho - rho0
            const R CL = rL * cL, CR = rR * cR;
            const R iC = rcp(CL + CR);
            const R dV = -(e0 * du + e1 * dv);
            const R sL = (CL * dV + dp) * iC;
            const R sR = (dp - CR * dV) * iC;
            const R dPL = -(CL * (dp + CR * dV)) * iC;     // P* - P_L
            const R dPR = dPL + dp;                        // P* - P_R
            // shock factor (:243-275): taken when P* > P_K and rho_K > rho*.  With the linear
            // equation of state rho_K - rho* = -(P* - P_K)/c0^2, so the branch is never taken.
            R QL = R(1), QR = R(1);
            if (P.eos != SPH_EOS_LINEAR) {
                const R ic0 = (R)(1.0 / P.c0sq), pbf = (R)P.pb;
                const R pa_ = (R)(S.kh.w + S.kl.w), pbb = (R)(T.kh.w + T.kl.w);
                const R pL = a_is_i ? pa_ : pbb, pR = a_is_i ? pbb : pa_;
                const R gL = drL - (pL - pbf) * ic0 - dPL * ic0;     // rho_L - rho*
                const R gR = drR - (pR - pbf) * ic0 - dPR * ic0;     // rho_R - rho*
                if (dPL > R(0) && gL > R(0)) QL = sqrt(((rL - gL) / rL) * dPL / gL) / cL;
                if (dPR > R(0) && gR > R(0)) QR = sqrt(((rR - gR) / rR) * dPR / gR) / cR;
            }
            const R sLm = -cL * QL, sRm = cR * QR;         // S_L - VL0, S_R - VR0
            const R hdV = R(0.5) * dV;
            const R tdv = e1 * du - e0 * dv;               // VR1 - VL1
            R dH, aI, bI, aJ, bJ;       // rho_HLLC - rho0; v_i - v* = aI e + bI t, v_j - v* = aJ e + bJ t
            if (sLm > hdV) {                                        // S_L > V0: the left state
                dH = drL; aI = R(0); bI = R(0); aJ = dV; bJ = tdv;
            } else if (sL - hdV >= R(0) && hdV >= sLm) {            // U* >= V0 >= S_L
                dH = drL + rL * quot(sL, sLm - sL);
                aI = -sL; bI = R(0); aJ = -sR; bJ = tdv;
            } else if (sRm >= -hdV && sL - hdV <= R(0)) {           // S_R >= V0 >= U*
                dH = drR + rR * quot(sR, sRm - sR);
                aI = -sL; bI = -tdv; aJ = -sR; bJ = R(0);
            } else {                                                // the right state
                dH = drR; aI = -dV; bI = -tdv; aJ = R(0); bJ = R(0);
            }
            PA = (R)P.c0sq * dH + (R)P.pb;
            const R al = a_is_i ? aI : aJ, be = a_is_i ? bI : bJ;
            wa0 = al * e0 - be * e1;
            wa1 = al * e1 + be * e0;
        } else {
            // HLLC in the pair frame (Moving_Square.../Solver_Normalized_HLLC_Riemann_Delta.f90:207-322),
            // FP64 path: the reference's own operations
            const double ed0 = (double)e0, ed1 = (double)e1;
            const double uI = I.kin.x, vI = I.kin.y, uJ = J.kin.x, vJ = J.kin.y;
            const double VL0 = ed0 * uI + ed1 * vI, VL1 = -ed1 * uI + ed0 * vI;
            const double VR0 = ed0 * uJ + ed1 * vJ, VR1 = -ed1 * uJ + ed0 * vJ;
            const double V0 = ed0 * (0.5 * (uI + uJ)) + ed1 * (0.5 * (vI + vJ));
            const double rL = I.kin.z, rR = J.kin.z, cL = (double)I.aux.z, cR = (double)J.aux.z;
            const double PLd = I.kin.w, PRd = J.kin.w;
            const double den = rL * cL + rR * cR;
            const double Us = (VR0 * cL * rL + VL0 * cR * rR + PLd - PRd) / den;
            const double Pst = (PRd * cL * rL + PLd * cR * rR - cL * rL * cR * rR * (VR0 - VL0)) / den;
            const double rst = (Pst - P.pb) / P.c0sq + P.rho0;
            double QL = 1.0, QR = 1.0;
            if (!(Pst <= PLd) && rL > rst) QL = sqrt((rst / rL) * (Pst - PLd) / (rL - rst)) / cL;
            const double SL = VL0 - cL * QL;
            if (!(Pst <= PRd) && rR > rst) QR = sqrt((rst / rR) * (Pst - PRd) / (rR - rst)) / cR;
            const double SR = VR0 + cR * QR;
            double rH, VH0, VH1;
            if (SL > V0) { rH = rL; VH0 = VL0; VH1 = VL1; }
            else if (Us >= V0 && V0 >= SL) {
                const double q = rL * ((SL - VL0) / (SL - Us));
                rH = q; VH0 = (Us * q) / rH; VH1 = (VL1 * q) / rH;
            } else if (SR >= V0 && V0 >= Us) {
                const double q = rR * ((SR - VR0) / (SR - Us));
                rH = q; VH0 = (Us * q) / rH; VH1 = (VR1 * q) / rH;
            } else { rH = rR; VH0 = VR0; VH1 = VR1; }
            const double vs0 = ed0 * VH0 - ed1 * VH1, vs1 = ed1 * VH0 + ed0 * VH1;
            PA = (R)(P.c0sq * (rH - P.rho0) + P.pb);
            const double4& K = S.kin;
            wa0 = (R)(K.x - vs0);
            wa1 = (R)(K.y - vs1);
        }
        if (MS) {        // XSPH velocities inside the continuity flux (MS solvers :199-202)
            const typename VT<R>::V2 avg_b = D.avg[b];
            wa0 += avg_a.x - avg_b.x;
            wa1 += avg_a.y - avg_b.y;
        }
        const R Vb = T.aux.y, mb = T.aux.x;
        // continuity (:360-369)
        R dr = R(2) * rho_a * Vb * (fsg * (wa0 * nd0 + wa1 * nd1));
        // pressure force (:374-388)
        const R rho_ij = inv_rho_a * (RREC ? (R)T.nb3.w : rcp(rho_b));
        // (FP64: m_b / rho_b is V_b)
        const R fp = F32 ? R(-2) * PA * rho_ij * mb : R(-2) * PA * (inv_rho_a * Vb);
        R tx = fp * nd0, ty = fp * nd1;
        // artificial viscosity (:392-417)
        const R inv_r2 = inv_d * inv_d;
        const R vx = du * xij0 + dv * xij1;
        if constexpr (!F32) {
            const R phi1 = hbar * min(vx, R(0)) * rcp(d * d + fh2);
            const R mp = (Vb * rho_b) * ((beta * phi1 - alpha * cbar) * phi1 * inv_rbar);
            tx -= mp * nd0;
            ty -= mp * nd1;
        } else if (vx < R(0)) {
            const R phi1 = fast_quot(hbar * vx, d * d + fh2);
            const R Pi = (-alpha * cbar * phi1 + beta * (phi1 * phi1)) * inv_rbar;
            tx += mb * (-Pi * nd0);
            ty += mb * (-Pi * nd1);
        }
        // (x_i - x_j).B^-1 dwdx / r^2, shared by the laplacian and delta-SPH
        const R xnd = (xij0 * nd0 + xij1 * nd1) * inv_r2;
        if (!MS || P.laplacian == 1) {
            // Morris laplacian (:432-436)
            const R lf = Vb * nu2 * xnd;
            tx += lf * du;
            ty += lf * dv;
        } else {
            // laplacianTerm 0 (Moving_Square.../Solver_..._Delta.f90:315-318): 2 (dim+2) nu V (v.x)/r^2 grad W
            const R lf = Vb * R(4) * nu2 * vx * inv_r2;
            tx += lf * nd0;
            ty += lf * nd1;
        }
        // delta-alpha artificial internal acceleration (:442-446)
        const R tt = dla_rho * cbar * (vx * inv_r2) * Vb;
        tx += tt * nd0;
        ty += tt * nd1;
        // SPS force, unnormalised dwdx and the neighbour's SPS mass (:450-492);
        // the reference does not reset temp_p between x and y (kept with quirks)
        if (!MS) {
            const R sxx = S.nb1.x + T.nb1.x, sxy = S.nb1.y + T.nb1.y, syy = S.nb1.z + T.nb1.z;
            R tp = (sxx * dw0 + sxy * dw1) * rho_ij;
            const R smb = T.aux.w;
            tx += smb * tp;
            if (!P.quirks) tp = R(0);
            tp = (tp + syy * dw1 + sxy * dw0) * rho_ij;
            ty += smb * tp;
        }
        accx.add(fsg * tx);
        accy.add(fsg * ty);
        // XSPH average velocity (:495-500; modified solver only)
        if (!MUSCL && !MS && P.xsph) {
            const R f = eps2 * mb * rcp(rho_a_ + rho_b) * w;
            xsx -= fsg * (f * du);
            xsy -= fsg * (f * dv);
        }
        // delta-SPH density diffusion (:552-583): psi = (rho_j - rho_i) - 0.5 (grad rho_i + grad rho_j).(x_j - x_i)
        if (water) {
            const R sg0 = S.nb1.w + T.nb1.w, sg1 = S.nb2.x + T.nb2.x;
            if (dsph) {
                // Antuono form (Solver_Normalized_Delta_SPH_SPS.f90:610-636):
                // psi = 2 (rho_j - rho_i) (x_j - x_i)/r^2 - (grad rho_i + grad rho_j), D += delta h c psi.gradW V
                const R f = R(2) * drho_ji * inv_r2;
                const R gsc = F32 ? R(2) : R(1);      // FP32 records: 1/2 grad rho
                const R p0 = -(f * xij0) - gsc * sg0, p1 = -(f * xij1) - gsc * sg1;
                dr += fsg * (dla_dh * cbar * (p0 * nd0 + p1 * nd1) * Vb);
            } else {
                const R psi = drho_ji + (F32 ? R(1) : R(0.5)) * (sg0 * xij0 + sg1 * xij1);
                dr += fsg * (dlt2h * cbar * psi * (-xnd) * Vb);
            }
        }
        cont.add(dr);
        // particle shifting sum (Shift_particle_position.f90:97-100), FP64:
        // shift_a = -beta h^2 B_a^-1 sum_b (1 + R (W/W(dx))^n) grad_a W_ab V_b
        if (SHIFT) {
            double gd, wd, Vd;
            if (F32) {
                // FP64 without divisions: q = d/h, grad factor G = g/(d h) = -5 k t^3/h^2
                // (Wendland) or -2 k e^{-q^2}/h^2 (Gaussian), V_b from the FP64 volume record.
                // The distance: one Newton (Heron) step for sqrt(s) from the FP32
                // distance d0 (relative error ~1e-7), d = d0 + (s - d0^2)/(2 d0),
                // leaves a relative error of order 1e-14
                const double d0 = (double)d;
                const double dd2 = fma(fma(-d0, d0, dxd * dxd + dyd * dyd), 0.5 * (double)inv_d, d0);
                const double q = dd2 * inv_h64;
                if (gauss) {
                    const double ex = exp(-(q * q));
                    wd = (ex - P.gauss_e9) * P.kfactor;
                    gd = -2.0 * P.kfactor * ex * inv_h2_64;
                } else {
                    const double t = 1.0 - 0.5 * q;
                    const double t2 = t * t;
                    wd = P.kfactor * (1.0 + 2.0 * q) * (t2 * t2);
                    gd = -5.0 * P.kfactor * (t2 * t) * inv_h2_64;
                }
                Vd = VPRE ? vd_b : load(&D.vol64[b]);
            } else {
                wd = (double)w; gd = (double)g; Vd = (double)Vb;
            }
            const double r = wd * inv_wdx;
            const double r2 = r * r;
            const double f = (1 + P.shift_R * (r2 * r2)) * Vd * gd;
            shx += f * dxd;
            shy += f * dyd;
        }
    }
    if constexpr (L > 1) {
        ln.sum(cont.s); ln.sum(accx.s); ln.sum(accy.s);
        if (!MUSCL && !MS) { ln.sum(xsx); ln.sum(xsy); }
        if (SHIFT) { ln.sum(shx); ln.sum(shy); }
        if (!live || ln.lane != 0) return;
    }
    // assembly (single_step_compute.f90:152-171, Solver :627-635)
    const R drho_a = (R)cont.val();
    const typename VT<R>::V2 acc_a = water ? mk2<R>((R)accx.val(), (R)accy.val()) : mk2<R>(R(0), R(0));
    double2 sh = make_double2(0.0, 0.0);
    if (SHIFT) {
        const double4 b64 = D.binv64[a];
        const double c = -P.shift_beta * (P.h * P.h);
        sh = make_double2(c * (b64.x * shx + b64.y * shy), c * (b64.z * shx + b64.w * shy));
    }
    const typename VT<R>::V2 avg_o = MS ? avg_a : mk2<R>(xsx, xsy);
    if (G.mode == STAGE_NONE) {
        D.drho[a] = drho_a;
        D.acc[a] = acc_a;
        if (!MS) D.avg[a] = avg_o;
        if (SHIFT) D.shift[a] = sh;
        return;
    }
    // the stage that follows this RHS, on a alone: a middle stage writes the other
    // copy of the records (the neighbours still read this one; particles that are
    // not integrated are copied), the last one the master state
    const double dr = (double)drho_a, ax = (double)acc_a.x, ay = (double)acc_a.y, gx = (double)avg_o.x,
                 gy = (double)avg_o.y;
    if (!water) {
        if (G.mode == STAGE_MID) {
            D.pos_n[a] = D.pos[a]; D.kin_n[a] = D.kin[a]; D.aux_n[a] = D.aux[a];
            if (F32) { D.vol64_n[a] = D.vol64[a]; D.kh_n[a] = D.kh[a]; D.kl_n[a] = D.kl[a]; D.xhl_n[a] = D.xhl[a]; }
        } else if (MS && G.to_staging && ta == SPH_TYPE_FIX_GHOST) {
            // a ghost ends the step with what the ghost assignment gave it
            const int i = D.id[a];
            G.S.vel[i] = D.vel0[a]; G.S.rho[i] = D.rho0[a]; G.S.mass[i] = D.mass[a]; G.S.smass[i] = D.smass[a];
        }
        return;
    }
    const double2 x0 = D.pos0[a], v0 = D.vel0[a];
    const double r0 = D.rho0[a];
    double x, y, u, v, rho;
    stage_update<R>(D, a, G.stage, G.dt, x0, v0, r0, dr, ax, ay, gx, gy, x, y, u, v, rho);
    check_skin(P, x0, x, y, G.status);
    if (G.mode == STAGE_MID) {
        store_records<R>(P, D, a, make_double2(x, y), u, v, rho, D.mass[a], D.smass[a], true);
        return;
    }
    if (SHIFT && ta == SPH_TYPE_WATER && !(D.flags[a] & 2))
        shift_by(P, sh, grad_scale<R>() * S.nb1.w, grad_scale<R>() * S.nb2.x, x, y, rho);
    store_end<R>(P, D, G.S, a, x, y, u, v, rho, dr, ax, ay, gx, gy, G.to_staging, G.status);
}

// The particle shifting sum of the mixed Taylor-Green path as a gather of its
// own, launched after pass C on the last RHS of a step (Shift_particle_position.f90:
// 56-100): shift_a = -beta h^2 B_a^-1 sum_b (1 + R (W/W(dx))^4) grad_a W_ab V_b in
// FP64, over the RHS's pair list, with the FP64 positions and volumes.  The same
// sum inside mixed pass C holds its FP64 values at pass C's register bound and
// stalls on their loads; here it runs at full occupancy.  Particles the shift
// does not move (not water, or near the free surface) get 0.  12 blocks of 128
// per SM (40 registers): 0.32 -> 0.29 ms per step at 2048^2 against 44 registers
// at 11 blocks; at 16 blocks (32 registers) it was slower.  With the step's last
// stage behind the sum (StageArgs; 120 B of spill stores) 0.45
// ms, against 0.29 and 0.30 for two passes; 10 blocks 0.49, 8 blocks without spills
// 0.57.
template <typename R>
__global__ void __launch_bounds__(128, 12) k_shift_gather(const __grid_constant__ Params P, const __grid_constant__ Sorted<R> D,
                                                        const __grid_constant__ StageArgs G) {
    pdl_begin();
    stamp_phase(P.stamp);
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= P.n_tot) return;
    const bool moves = D.type[a] == SPH_TYPE_WATER && !(D.flags[a] & 2);
    if (!moves && G.mode == STAGE_NONE) {
        D.shift[a] = make_double2(0.0, 0.0);
        return;
    }
    const int nn = moves ? D.npairs[a] : 0;
    const double2 xa = D.pos[a];
    const double inv_h64 = P.inv_h, inv_h2_64 = P.inv_h2, inv_wdx = 1.0 / P.w_dx;
    double shx = 0.0, shy = 0.0;
    // the pair entry two iterations ahead, the neighbour's position and volume one ahead
    unsigned ent_n = nn > 0 ? load(&D.pairs[a]) : 0u;
    unsigned ent_nn = nn > 1 ? load(&D.pairs[(size_t)P.nbr_stride + a]) : 0u;
    double2 xb_n = make_double2(0.0, 0.0);
    double vd_n = 0.0;
    if (nn > 0) {
        const int b0 = (int)(ent_n & 0x7fffffffu);
        xb_n = load(&D.pos[b0]);
        vd_n = load(&D.vol64[b0]);
    }
    for (int e = 0; e < nn; ++e) {
        const double2 xb = xb_n;
        const double Vd = vd_n;
        if (e + 1 < nn) {
            ent_n = ent_nn;
            const int b1 = (int)(ent_n & 0x7fffffffu);
            xb_n = load(&D.pos[b1]);
            vd_n = load(&D.vol64[b1]);
            if (e + 2 < nn) ent_nn = load(&D.pairs[(size_t)(e + 2) * P.nbr_stride + a]);
        }
        const double dxd = xa.x - xb.x, dyd = xa.y - xb.y;
        const double s2 = dxd * dxd + dyd * dyd;
        // distance: FP32 estimate, then one Newton (Heron) step for sqrt(s2),
        // d = d0 + (s2 - d0^2)/(2 d0): relative error of order 1e-14
        const float sf = (float)s2;
        const float yf = rsqrtf(sf);
        const double d0 = (double)(sf * yf);
        const double dd = fma(fma(-d0, d0, s2), 0.5 * (double)yf, d0);
        const double q = dd * inv_h64;
        // grad factor G = g/(d h) and W (compute_kernel), FP64 without divisions
        double wd, gd;
        if (P.kernel_model == SPH_KERNEL_GAUSSIAN) {
            const double ex = exp(-(q * q));
            wd = (ex - P.gauss_e9) * P.kfactor;
            gd = -2.0 * P.kfactor * ex * inv_h2_64;
        } else {
            const double t = 1.0 - 0.5 * q;
            const double t2 = t * t;
            wd = P.kfactor * (1.0 + 2.0 * q) * (t2 * t2);
            gd = -5.0 * P.kfactor * (t2 * t) * inv_h2_64;
        }
        const double r = wd * inv_wdx;
        const double r2 = r * r;
        const double f = (1 + P.shift_R * (r2 * r2)) * Vd * gd;
        shx += f * dxd;
        shy += f * dyd;
    }
    const double4 b64 = D.binv64[a];
    const double c = -P.shift_beta * (P.h * P.h);
    const double2 sh = make_double2(c * (b64.x * shx + b64.y * shy), c * (b64.z * shx + b64.w * shy));
    if (G.mode == STAGE_NONE) { D.shift[a] = sh; return; }
    // the step's last stage (STAGE_END): it writes only a's own master state, so the
    // positions the other threads are reading stay as they are
    if (!integrated(P, D.type[a])) return;
    const typename VT<R>::V2 ac = D.acc[a], av = D.avg[a];
    const double dr = (double)D.drho[a], ax = (double)ac.x, ay = (double)ac.y, gx = (double)av.x, gy = (double)av.y;
    const double2 x0 = D.pos0[a];
    double x, y, u, v, rho;
    stage_update<R>(D, a, G.stage, G.dt, x0, D.vel0[a], D.rho0[a], dr, ax, ay, gx, gy, x, y, u, v, rho);
    check_skin(P, x0, x, y, G.status);
    if (moves) shift_by(P, sh, grad_scale<R>() * D.nb1[a].w, grad_scale<R>() * D.nb2[a].x, x, y, rho);
    store_end<R>(P, D, G.S, a, x, y, u, v, rho, dr, ax, ay, gx, gy, G.to_staging, G.status);
}

}  // namespace sph
