// update.cuh -- integrator stages, shifting, diagnostics reductions, pair
// enumeration for the find_particle_pair entry point, and layout conversions.
#pragma once
#include "pass_c.cuh"

namespace sph {

// Shift_particle_position.f90:108-131: the capped displacement of the last RHS's
// shifting sum and the first-order density correction, for water particles
// that are not near the free surface.
template <typename R>
__device__ __forceinline__ void apply_shift(const Params& P, const Sorted<R>& D, int s, double& x, double& y,
                                            double& rho) {
    if (D.type[s] != SPH_TYPE_WATER || (D.flags[s] & 2)) return;
    shift_by(P, D.shift[s], grad_scale<R>() * D.nb1[s].w, grad_scale<R>() * D.nb2[s].x, x, y, rho);
}

// A stage as a pass of its own: where the rates are not carried by the kernel
// before it (the first step, a density re-initialisation, the adjoint's segment
// re-run).  Elsewhere the first stage is applied by k_gather_sorted, the middle
// ones and the last by k_pass_c or k_shift_gather (StageArgs).
template <typename R>
__global__ void k_stage(Params P, Sorted<R> D, int stage, double dt, int use_carried, int do_shift,
                        unsigned* status) {
    pdl_begin();
    stamp_phase(P.stamp);
    using V2 = typename VT<R>::V2;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P.n_tot) return;
    if (!integrated(P, D.type[s])) return;
    const double2 x0 = D.pos0[s];
    const double2 v0 = D.vel0[s];
    const double r0 = D.rho0[s];
    double dr, ax, ay, gx, gy;
    if ((stage == 0 || stage == 10) && use_carried) {   // the first stage of either driver
        dr = (double)D.c_drho[s]; V2 a = D.c_acc[s], g = D.c_avg[s];
        ax = (double)a.x; ay = (double)a.y; gx = (double)g.x; gy = (double)g.y;
    } else {
        dr = (double)D.drho[s]; V2 a = D.acc[s], g = D.avg[s];
        ax = (double)a.x; ay = (double)a.y; gx = (double)g.x; gy = (double)g.y;
    }
    double rho, u, v, x, y;
    stage_update<R>(D, s, stage, dt, x0, v0, r0, dr, ax, ay, gx, gy, x, y, u, v, rho);
    check_skin(P, x0, x, y, status);
    if (stage == 3 || stage == 11) {
        if (do_shift) apply_shift(P, D, s, x, y, rho);
        store_end<R>(P, D, Staging{}, s, x, y, u, v, rho, dr, ax, ay, gx, gy, 0, status);
    }
    store_records<R>(P, D, s, make_double2(x, y), u, v, rho, D.mass[s], D.smass[s], false);
}

// Density re-initialisation by moving least squares (Reinitialize_particle_density:
// Taylor_Green_Vortex/Reinitialize_particle_density.f90:98-181 with
// MLS_Interpolation_In_Subdomain_Domain.f90:96-285; moving-square variant
// Moving_Square.../Reinitialize_particle_density.f90:92-200 with
// SPH_Subroutine_Module.f90:2565-2792), FP64, on the state after the integrator
// update (images keep the step-start state).  For a water particle i and its
// neighbours j within the support, with W_j the kernel value (the moving-square
// variant: W_j V_j, and i itself counts as a neighbour),
//   p_j = (1, dx, dy[, dx^2, dx dy, dy^2]),  (dx, dy) = (x_j - x_i)/h,
//   A   = sum_j W_j p_j p_j^T + alpha^3 I,
//   rho_i = sum_j rho_j W_j (A^-1 e_1).p_j = c.r,  A c = e_1,  r = sum_j rho_j W_j p_j.
// The reference inverts A (BRINV / the 3x3 adjugate) and forms the same weights;
// here A c = e_1 is solved by an FP64 Cholesky factorisation (A is symmetric and
// positive definite away from degenerate neighbourhoods).  A failed factorisation,
// and with order 6 at most 8 neighbours (Taylor-Green variant), fall back to the
// Shepard weights W_j / sum W, as the reference does.  Non-water particles keep
// their density (the Taylor-Green routine zeroes its periodic images, which are
// regenerated at the next step start).
template <int M>
__device__ __forceinline__ bool chol_solve_e1(double (&A)[M * (M + 1) / 2], double (&c)[M]) {
    // packed lower triangle, row-major: A[i(i+1)/2 + j], j <= i
    double L[M * (M + 1) / 2];
#pragma unroll
    for (int i = 0; i < M; ++i) {
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            double sum = A[i * (i + 1) / 2 + j];
#pragma unroll
            for (int k = 0; k < j; ++k) sum -= L[i * (i + 1) / 2 + k] * L[j * (j + 1) / 2 + k];
            if (i == j) {
                if (!(sum > 0.0)) return false;
                L[i * (i + 1) / 2 + i] = sqrt(sum);
            } else {
                L[i * (i + 1) / 2 + j] = sum / L[j * (j + 1) / 2 + j];
            }
        }
    }
    // L y = e_1, L^T c = y
    double y[M];
#pragma unroll
    for (int i = 0; i < M; ++i) {
        double sum = i == 0 ? 1.0 : 0.0;
#pragma unroll
        for (int k = 0; k < i; ++k) sum -= L[i * (i + 1) / 2 + k] * y[k];
        y[i] = sum / L[i * (i + 1) / 2 + i];
    }
#pragma unroll
    for (int i = M - 1; i >= 0; --i) {
        double sum = y[i];
#pragma unroll
        for (int k = i + 1; k < M; ++k) sum -= L[k * (k + 1) / 2 + i] * c[k];
        c[i] = sum / L[i * (i + 1) / 2 + i];
    }
    return true;
}

template <typename R, int M>
__global__ void k_mls(Params P, Sorted<R> D, double* rho_new) {
    pdl_begin();
    stamp_phase(P.stamp);
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= P.n_tot) return;
    const double rho_a = D.kin[a].z;
    if (D.type[a] != SPH_TYPE_WATER || D.id[a] >= P.n_host) { rho_new[a] = rho_a; return; }
    const double2 xa = D.pos[a];
    const double inv_h = 1.0 / P.h;
    double A[M * (M + 1) / 2], r[M];
#pragma unroll
    for (int k = 0; k < M * (M + 1) / 2; ++k) A[k] = 0.0;
#pragma unroll
    for (int k = 0; k < M; ++k) r[k] = 0.0;
    double sw = 0.0, srw = 0.0;
    int cnt = 0;
    const int nn = D.nnbr[a];
    // the moving-square variant includes the particle itself (distance 0)
    for (int e = (P.ms ? -1 : 0); e < nn; ++e) {
        const int b = e < 0 ? a : (int)(D.nbr[(size_t)e * P.nbr_stride + a] & 0x7fffffffu);
        const double2 xb = D.pos[b];
        const double px = xa.x - xb.x, py = xa.y - xb.y;
        double d;
        const bool in = in_support(P, px, py, d);
        if (P.ms ? !(d <= P.r_cut) : !in) continue;
        double w, gx, gy;
        kernel_w_dw<double>(P, d, px, py, w, gx, gy);
        const double rho_b = D.kin[b].z;
        if (P.ms) w *= D.mass[b] / rho_b;
        double p[M];
        const double dx = -px * inv_h, dy = -py * inv_h;
        p[0] = 1.0; p[1] = dx; p[2] = dy;
        if (M == 6) { p[3 % M] = dx * dx; p[4 % M] = dx * dy; p[5 % M] = dy * dy; }
#pragma unroll
        for (int i = 0; i < M; ++i) {
            const double wp = w * p[i];
#pragma unroll
            for (int j = 0; j <= i; ++j) A[i * (i + 1) / 2 + j] += wp * p[j];
            r[i] += rho_b * wp;
        }
        sw += w;
        srw += rho_b * w;
        ++cnt;
    }
#pragma unroll
    for (int i = 0; i < M; ++i) A[i * (i + 1) / 2 + i] += P.mls_alpha3;
    double c[M];
    double out;
    const bool few = !P.ms && M == 6 && cnt <= 8;
    if (!few && chol_solve_e1<M>(A, c)) {
        out = 0.0;
#pragma unroll
        for (int i = 0; i < M; ++i) out += c[i] * r[i];
    } else {
        out = srw / sw;
    }
    if (P.ms && isnan(out)) out = rho_a;
    rho_new[a] = out;
}

// RefreshDensity_MLS_Order = 1 (Taylor_Green_Vortex/Reinitialize_particle_density.f90:71-92,
// Moving_Square.../Reinitialize_particle_density.f90:66-88), evaluated on the
// step's last RHS (its pair list and state, which the reference's pair arrays
// and volumes still hold when it runs): for a water particle a,
//   rho_a = sum_b m_b W_ab / sum_b W_ab V_b
// over the pairs with a neighbour of a's type (sum_w,
// Define_freesurface_and_Normailized_derivates.f90:87-91), in FP64.
template <typename R>
__global__ void k_mls1(Params P, Sorted<R> D, double* rho_new) {
    pdl_begin();
    stamp_phase(P.stamp);
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= P.n_tot) return;
    rho_new[a] = D.kin[a].z;
    const int ta = D.type[a];
    if (ta != SPH_TYPE_WATER || D.id[a] >= P.n_host) return;
    const double2 xa = D.pos[a];
    double sw = 0.0, sm = 0.0;
    const int nn = D.npairs[a];
    for (int e = 0; e < nn; ++e) {
        const int b = (int)(D.pairs[(size_t)e * P.nbr_stride + a] & 0x7fffffffu);
        if (D.type[b] != ta) continue;
        const double2 xb = D.pos[b];
        const double px = xa.x - xb.x, py = xa.y - xb.y;
        const double d = __dsqrt_rn(__dadd_rn(__dmul_rn(px, px), __dmul_rn(py, py)));
        double w, gx, gy;
        kernel_w_dw<double>(P, d, px, py, w, gx, gy);
        const double mb = D.mass[b];
        sw += w * (mb / D.kin[b].z);
        sm += mb * w;
    }
    rho_new[a] = sm / sw;
}

// The re-initialised density replaces the integrated one; then the shift of the
// step (when on) is applied, as the reference's driver calls the two in turn.
template <typename R>
__global__ void k_finish_mls(Params P, Sorted<R> D, const double* rho_new, int do_shift, unsigned* status) {
    pdl_begin();
    stamp_phase(P.stamp);
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P.n_tot) return;
    if (!integrated(P, D.type[s]) || D.id[s] >= P.n_host) return;
    const double2 x0 = D.pos0[s];
    double x = x0.x, y = x0.y;
    double rho = D.type[s] == SPH_TYPE_WATER ? rho_new[s] : D.rho0[s];
    if (do_shift) apply_shift(P, D, s, x, y, rho);
    if (!(isfinite(x) && isfinite(y) && isfinite(rho))) atomicOr(status, ST_NONFINITE);
    D.pos0[s] = make_double2(x, y);
    D.pos[s] = make_double2(x, y);
    D.rho0[s] = rho;
    double p, c;
    eos64(P, rho, p, c);
    const double2 v = D.vel0[s];
    const double m = D.mass[s];
    D.kin[s] = make_double4(v.x, v.y, rho, p);
    D.aux[s] = mk4<R>((R)m, (R)(m / rho), (R)c, (R)D.smass[s]);
    store_split(D, s, make_double2(x, y), make_double4(v.x, v.y, rho, p));
}

// Ghost kernel value at squared distance s2.
__device__ __forceinline__ double ghost_w(const Params& P, double s2) {
    if (P.kernel_model == SPH_KERNEL_GAUSSIAN) return (exp(-(s2 * P.ghost_ih2)) - P.gauss_e9) * P.ghost_kf;
    const double q = sqrt(s2 * P.ghost_ih2);
    const double tq = 1.0 - 0.5 * q, t2 = tq * tq;
    return P.ghost_kf * (1.0 + 2.0 * q) * (t2 * t2);
}
// (dw/dd) / d of it.
__device__ __forceinline__ double ghost_dw_over_d(const Params& P, double s2) {
    if (P.kernel_model == SPH_KERNEL_GAUSSIAN) return -2.0 * exp(-(s2 * P.ghost_ih2)) * P.ghost_kf * P.ghost_ih2;
    const double tq = 1.0 - 0.5 * sqrt(s2 * P.ghost_ih2);
    return -5.0 * (tq * tq * tq) * P.ghost_kf * P.ghost_ih2;
}

// The slots of the ghost assignment's window around the list-build cell of x0: fn(b)
// on the lane that visits b.  Lane k finds the slot range of the window's row k
// (the slots of a row's window cells are contiguous in the cell-sorted order), so
// the ranges are one round of loads; then the 32 lanes split each row.
template <typename R, typename F>
__device__ __forceinline__ void window_visit_warp(const Params& P, const Sorted<R>& D, double2 x0, F&& fn) {
    const int lane = threadIdx.x & 31;
    const int cx = (int)floor((x0.x - P.gx0) / P.cs), cy = (int)floor((x0.y - P.gy0) / P.cs);
    const int gx0 = max(cx - P.ghost_cells, 0), gx1 = min(cx + P.ghost_cells, P.gnx - 1);
    const int gy0 = max(cy - P.ghost_cells, 0), gy1 = min(cy + P.ghost_cells, P.gny - 1);
    for (int r0 = gy0; r0 <= gy1; r0 += 32) {
        int lo = 0, hi = 0;
        if (r0 + lane <= gy1) {
            const int row = (r0 + lane) * P.gnx;
            int first = -1;
            for (int gx = gx0; gx <= gx1; ++gx) {
                const int b0 = D.cell_start[row + gx], b1 = D.cell_end[row + gx];
                if (b0 < 0) continue;
                if (first < 0) first = b0;
                hi = b1;
            }
            lo = max(first, 0);
        }
        const int rows = min(gy1 - r0 + 1, 32);
        for (int k = 0; k < rows; ++k) {
            const int end = __shfl_sync(0xffffffffu, hi, k);
            for (int b = __shfl_sync(0xffffffffu, lo, k) + lane; b < end; b += 32) fn(b);
        }
    }
}

// The neighbours the ghost assignment interpolates from for ghost slot s: the
// non-ghost particles within kernel_scale * 1.2 h, found over the window of s's
// cell (the list-build cells, so the window reaches ghost_r plus half the skin).
// fn(b, dx, dy, s2, w) gets (dx, dy) = x_s - x_b, the squared distance and the
// kernel value with the ghost smoothing length, on the lane that visits b.
template <typename R, typename F>
__device__ __forceinline__ void ghost_visit_warp(const Params& P, const Sorted<R>& D, int s, F&& fn) {
    const double2 x = D.pos[s];
    window_visit_warp(P, D, x, [&](int b) {
        const double2 xb = D.pos[b];
        const int tb = D.type[b];
        const double dx = x.x - xb.x, dy = x.y - xb.y;
        const double s2 = dist2(dx, dy);
        if (tb == SPH_TYPE_FIX_GHOST || !(s2 <= P.ghost_s_cut)) return;
        fn(b, dx, dy, s2, ghost_w(P, s2));
    });
}

// Sum over the warp, lane 0's association order, broadcast to every lane (so
// that all lanes continue with bit-identical values).
__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return __shfl_sync(0xffffffffu, v, 0);
}
__device__ __forceinline__ int warp_sum(int v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return __shfl_sync(0xffffffffu, v, 0);
}

// Fixed-ghost assignment of the moving-square driver (Moving_Square.../
// Assign_boundary_particles.f90:611-941, with MLS_order_Boundary = 1, i.e.
// Shepard weights Fai_j = W_j V_j / sum W V), at the start of every RHS, from the
// current state of the non-ghost particles within kernel_scale * 1.2 h:
//   p = sum Fai (p_j + rho_j g.(x - x_j)),  u = sum Fai u_j,  m = sum Fai m_j
// (g: gravity, plus the body acceleration for body ghosts), at least 3
// neighbours or nothing.  Body ghosts take the body velocity; wall ghosts, during
// 0 < t <= Shock_wave_release_time, go through the characteristic variables for
// labels -6 / -7 (which return the interpolated values) and keep the zero
// pressure they start from for other labels, as the reference's branch does;
// then the wall velocity is mirrored by label and wall condition.  Finally
// rho = (p - pb)/c0^2 + rho0, or the rest state when m = 0.
// One warp per ghost (ghost_ids: the host ghosts in id order, n_ghost of them),
// the lanes splitting the neighbours; the sums are reduced in a fixed order.
template <typename R>
// gint / gsw (may be null): the interpolated (p, u, v, m) and the weight sum
// sum W V of each ghost slot, kept for the reverse (k_adj_ghost_lambda).
__global__ void k_assign_ghosts(Params P, Sorted<R> D, const int* ghost_ids, int n_ghost, double t, double bvx,
                                double bvy, double bax, double bay, double4* gint = nullptr,
                                double* gsw = nullptr) {
    pdl_begin();
    stamp_phase(P.stamp);
    const int wg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (wg >= n_ghost) return;                       // whole warps
    const int s = D.slot_of[ghost_ids[wg]];
    const double2 x = D.pos[s];
    const bool body = D.itype[s] == SPH_TYPE_BODY;
    const double gxe = P.grav[0] + (body ? bax : 0.0), gye = P.grav[1] + (body ? bay : 0.0);
    double sw = 0.0, sp = 0.0, su = 0.0, sv = 0.0, sm = 0.0;
    int cnt = 0;
    ghost_visit_warp(P, D, s, [&](int b, double dx, double dy, double, double w) {
        const double4 kb = load4(&D.kin[b]);
        const double mb = D.mass[b];
        const double W = w * (mb * rcp64(kb.z));
        sw += W;
        sp += kb.w * W + kb.z * W * (gxe * dx + gye * dy);
        su += kb.x * W;
        sv += kb.y * W;
        sm += mb * W;
        ++cnt;
    });
    sw = warp_sum(sw); sp = warp_sum(sp); su = warp_sum(su); sv = warp_sum(sv); sm = warp_sum(sm);
    cnt = warp_sum(cnt);
    if ((threadIdx.x & 31) != 0) return;
    double uint = 0.0, vint = 0.0, pint = 0.0, m = 0.0;
    if (cnt >= 3) {
        const double inv = 1.0 / sw;
        pint = sp * inv; uint = su * inv; vint = sv * inv; m = sm * inv;
    }
    if (gint) {
        gint[s] = make_double4(pint, uint, vint, m);
        gsw[s] = sw;
    }
    double u, v, p = 0.0;
    if (body) {
        u = bvx; v = bvy; p = pint;
    } else {
        const int lab = D.blabel[s];
        if (0.0 < t && t <= P.shock_t) {
            const double ri = (pint - P.pb) / P.c0sq + P.rho0;
            const double r = ri / P.rho0;
            const double c = P.sqrt_c0 * (r * r * r);
            u = uint; v = vint;
            if (lab == -6 || lab == -7) {
                const double vn = lab == -6 ? vint : uint;
                const double J2 = ri * c * vn + pint, J3 = -ri * c * vn + pint;
                const double vs = (J2 - J3) / (2 * ri * c);
                if (lab == -6) v = vs; else u = vs;
                p = 0.5 * (J2 + J3);
            }
        } else {
            u = uint; v = vint; p = pint;
        }
        if (lab == -6) { if (P.wall_bc == 1) v = -v; else { u = -u; v = -v; } }
        else if (lab == -7) { u = -u; v = -v; }
        else if (lab == -8) { if (P.wall_bc == 1) u = -u; else { u = -u; v = -v; } }
    }
    double rho, c;
    if (m != 0.0) {
        rho = (p - P.pb) / P.c0sq + P.rho0;
        const double r = rho / P.rho0;
        c = P.sqrt_c0 * (r * r * r);
    } else {
        u = 0.0; v = 0.0; p = 0.0; rho = P.rho0; m = 0.0; c = P.sqrt_c0;
    }
    D.mass[s] = m;
    D.smass[s] = m;
    D.vel0[s] = make_double2(u, v);
    D.rho0[s] = rho;
    D.kin[s] = make_double4(u, v, rho, p);
    D.aux[s] = mk4<R>((R)m, (R)(m / rho), (R)c, (R)m);
    store_split(D, s, x, make_double4(u, v, rho, p));
}

// The per-particle arrays k_assign_ghosts writes besides the records (mass,
// SPS mass, step-start velocity and density), set again from the records of a
// state that already holds the assigned ghosts (FP64 records: aux.x = m exactly).
template <typename R>
__global__ void k_ghost_refill(Sorted<R> D, const int* ghost_ids, int n_ghost) {
    pdl_begin();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n_ghost) return;
    const int s = D.slot_of[ghost_ids[g]];
    const double4 k = D.kin[s];
    const double m = (double)D.aux[s].x;
    D.mass[s] = m;
    D.smass[s] = m;
    D.vel0[s] = make_double2(k.x, k.y);
    D.rho0[s] = k.z;
}

// The end of a timed stretch of work.
__global__ void k_stamp(unsigned long long* slot) { pdl_begin(); stamp_phase(slot); }

// Kinetic energy and max |v| of the water host particles
// (Sampling_subroutine.f90:346-356) in FP64 and the number of flagged surface
// particles: block partials, then the last block to finish adds them in a fixed
// order and writes the results, the status word and the last body force (bf, or
// null) to the page-locked box the host reads after one wait.
constexpr int kRedThreads = 256;
constexpr int kDiagBlocks = 148 * 4;
template <typename R>
__global__ void __launch_bounds__(kRedThreads) k_diag(Params P, Sorted<R> D, double* part_ke, double* part_max,
                                                      int* part_ns, unsigned* done, const unsigned* status,
                                                      const double* bf, HostBox* box) {
    pdl_begin();
    __shared__ double ske[kRedThreads], smx[kRedThreads];
    __shared__ int sns[kRedThreads];
    __shared__ int flag;
    const int t = threadIdx.x;
    auto reduce = [&](double ke, double mx, int ns) {
        ske[t] = ke; smx[t] = mx; sns[t] = ns;
        __syncthreads();
        for (int w = kRedThreads / 2; w > 0; w >>= 1) {
            if (t < w) { ske[t] += ske[t + w]; smx[t] = fmax(smx[t], smx[t + w]); sns[t] += sns[t + w]; }
            __syncthreads();
        }
    };
    double ke = 0.0, mx = 0.0;
    int ns = 0;
    for (int s = blockIdx.x * blockDim.x + t; s < P.n_tot; s += gridDim.x * blockDim.x) {
        ns += D.flags[s] & 1;
        if (D.type[s] != SPH_TYPE_WATER || D.id[s] >= P.n_host) continue;
        double2 v = D.vel0[s];
        double vv = v.x * v.x + v.y * v.y;
        ke += 0.5 * D.mass[s] * vv;
        mx = fmax(mx, sqrt(vv));
    }
    reduce(ke, mx, ns);
    if (t == 0) { part_ke[blockIdx.x] = ske[0]; part_max[blockIdx.x] = smx[0]; part_ns[blockIdx.x] = sns[0]; }
    if (!last_block(done, &flag)) return;
    ke = mx = 0.0;
    ns = 0;
    for (int i = t; i < (int)gridDim.x; i += kRedThreads) {
        ke += __ldcg(&part_ke[i]); mx = fmax(mx, __ldcg(&part_max[i])); ns += __ldcg(&part_ns[i]);
    }
    reduce(ke, mx, ns);
    if (t == 0) {
        box->diag[0] = ske[0]; box->diag[1] = smx[0];
        box->nsurf = sns[0];
        box->status = *status;
    }
    if (t < 6 && bf) box->diag[2 + t] = bf[t];
}

// Body force of the last RHS (Moving_Square.../Calculate_Body_Force.f90:53-142 and
// Single_step_compute.f90:228-243), FP64: for a particle a with body neighbours b
// (initial type SPH_TYPE_BODY)
//   BFP_a = -sum_b V_b (p_a + p_b) B_a^-1 grad_a W_ab
//   BFV_a =  sum_b rho_a V_b 2 nu ((x_a - x_b).B_a^-1 grad_a W_ab) / r^2 (v_a - v_b)   (Morris)
//       or   sum_b rho_a V_b 2 (dim+2) nu ((v_a-v_b).(x_a-x_b)) / r^2 B_a^-1 grad_a W_ab
// and the forces are sum_a V_a BFP_a, sum_a V_a BFV_a and their sum (no gravity).
// Gathered from the body side: body particle b sums V_a times its terms over its
// pair neighbours a (the pair set is symmetric), one warp per body particle
// (body_ids: the body's host particles) with the lanes on the pairs; the last
// block adds the block partials (part, [4][blocks]) in a fixed order into out.
// A thread per particle of the whole tank left a few warps with chains of up to
// 45 neighbours, and a second launch for the sum: pass C and the force together
// 84 -> 52 us per step at D/30 (FP64), 440 -> 389 us at D/100 (mixed).
template <typename R>
__global__ void __launch_bounds__(kRedThreads) k_body_force(Params P, Sorted<R> D, const int* body_ids, int n_body,
                                                            double* part, double* out, unsigned* done) {
    pdl_begin();
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int g = (blockIdx.x * kRedThreads + t) >> 5;
    double f[4] = {0, 0, 0, 0};
    if (g < n_body) {
        const int b = D.slot_of[body_ids[g]];
        const int nn = D.npairs[b];
        if (nn > 0) {
            const double2 xb = D.pos[b];
            const double4 kb = load4(&D.kin[b]);
            const double Vb = D.mass[b] * rcp64(kb.z);
            for (int e = lane; e < nn; e += 32) {
                const int a = (int)(D.pairs[(size_t)e * P.nbr_stride + b] & 0x7fffffffu);
                const double2 xa = D.pos[a];
                const double4 ka = load4(&D.kin[a]), bi = load4(&D.binv64[a]);
                const double Va = D.mass[a] * rcp64(ka.z);
                const double dx = xa.x - xb.x, dy = xa.y - xb.y;
                const double s2 = dx * dx + dy * dy;
                // grad_a W = G (x_a - x_b)
                double G;
                if (P.kernel_model == SPH_KERNEL_GAUSSIAN) G = exp(-(s2 * P.inv_h2)) * P.gk;
                else { const double tq = 1.0 - s2 * rsqrt64(s2) * P.half_inv_h; G = P.gk * (tq * tq * tq); }
                if (s2 * P.inv_h2 <= P.q_zero * P.q_zero) G = 0.0;      // (compute_kernel)
                const double gx = G * dx, gy = G * dy;
                const double n0 = bi.x * gx + bi.y * gy, n1 = bi.z * gx + bi.w * gy;
                const double fp = -Va * Vb * (ka.w + kb.w);
                f[0] += fp * n0; f[1] += fp * n1;
                const double du = ka.x - kb.x, dv = ka.y - kb.y;
                const double fv = Va * ka.z * Vb * 2 * P.nu * rcp64(s2);
                if (P.laplacian == 1) {
                    const double l = fv * (dx * n0 + dy * n1);
                    f[2] += l * du; f[3] += l * dv;
                } else {
                    const double l = fv * (2 + 2) * (du * dx + dv * dy);
                    f[2] += l * n0; f[3] += l * n1;
                }
            }
        }
    }
    __shared__ double sh[4][kRedThreads / 32];
    __shared__ int flag;
    auto reduce = [&]() {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            for (int o = 16; o > 0; o >>= 1) f[c] += __shfl_down_sync(0xffffffffu, f[c], o);
            if (lane == 0) sh[c][w] = f[c];
        }
        __syncthreads();
        if (t < 4) {
            double v = 0.0;
            for (int k = 0; k < kRedThreads / 32; ++k) v += sh[t][k];
            f[0] = v;                       // thread c: component c
        }
    };
    reduce();
    if (t < 4) part[(size_t)t * gridDim.x + blockIdx.x] = f[0];
    if (!last_block(done, &flag)) return;
    for (int c = 0; c < 4; ++c) {
        f[c] = 0.0;
        for (int i = t; i < (int)gridDim.x; i += kRedThreads) f[c] += __ldcg(&part[(size_t)c * gridDim.x + i]);
    }
    reduce();
    if (t < 4) {
        out[t] = f[0];
        sh[t][0] = f[0];
    }
    __syncthreads();
    if (t < 2) out[4 + t] = sh[t][0] + sh[2 + t][0];
}

// --- find_particle_pair entry point ---------------------------------------
// Pairs are emitted once, by their pair_i (lower id), sorted by (i, j).
template <typename R>
__global__ void k_pair_count(Params P, Sorted<R> D, long long* cnt_id) {
    pdl_begin();
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= P.n_tot) return;
    const int nn = D.nnbr[a];
    const double2 xa = D.pos[a];
    int c = 0;
    for (int e = 0; e < nn; ++e) {
        const unsigned ent = D.nbr[(size_t)e * P.nbr_stride + a];
        if (!(ent >> 31)) continue;
        const double2 xb = D.pos[ent & 0x7fffffffu];
        double d;
        if (in_support(P, xa.x - xb.x, xa.y - xb.y, d)) ++c;
    }
    cnt_id[D.id[a]] = c;
}

template <typename R>
__global__ void k_pair_emit(Params P, Sorted<R> D, const long long* off_id, long long cap, int* pi, int* pj,
                            double* w, double* dwdx) {
    pdl_begin();
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= P.n_tot) return;
    const int nn = D.nnbr[a];
    const double2 xa = D.pos[a];
    const int ida = D.id[a];
    int bid[256];
    int m = 0;
    for (int e = 0; e < nn && m < 256; ++e) {
        const unsigned ent = D.nbr[(size_t)e * P.nbr_stride + a];
        if (!(ent >> 31)) continue;
        const int b = (int)(ent & 0x7fffffffu);
        const double2 xb = D.pos[b];
        double d;
        if (!in_support(P, xa.x - xb.x, xa.y - xb.y, d)) continue;
        // insertion by neighbour id
        const int idb = D.id[b];
        int k = m++;
        while (k > 0 && D.id[bid[k - 1]] > idb) { bid[k] = bid[k - 1]; --k; }
        bid[k] = b;
    }
    long long o = off_id[ida];
    for (int k = 0; k < m; ++k, ++o) {
        if (o >= cap) return;
        const int b = bid[k];
        const double2 xb = D.pos[b];
        double dx = xa.x - xb.x, dy = xa.y - xb.y, d;
        in_support(P, dx, dy, d);
        double ww, gx, gy;
        kernel_w_dw<double>(P, d, dx, dy, ww, gx, gy);
        pi[o] = ida + 1;
        pj[o] = D.id[b] + 1;
        if (w) w[o] = ww;
        if (dwdx) { dwdx[o] = gx; dwdx[cap + o] = gy; }
    }
}

// --- column-major (n,2) <-> interleaved conversions -----------------------
__global__ void k_interleave(int n, const double* colmaj, double2* out) {
    pdl_begin();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = make_double2(colmaj[i], colmaj[n + i]);
}
// pos, vel (column-major) and rho, one after another, into the id-order arrays.
__global__ void k_upload(int n, const double* in, double2* pos, double2* vel, double* rho) {
    pdl_begin();
    const size_t nn = (size_t)n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    pos[i] = make_double2(in[i], in[nn + i]);
    vel[i] = make_double2(in[2 * nn + i], in[3 * nn + i]);
    rho[i] = in[4 * nn + i];
}
__global__ void k_deinterleave(int n, const double2* in, double* colmaj) {
    pdl_begin();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { double2 v = in[i]; colmaj[i] = v.x; colmaj[n + i] = v.y; }
}

// Snapshot of the host particles' state (id order, staging arrays) in the
// column-major layout of sph_get_state: [0, 2n) pos, [2n, 4n) vel, [4n, 5n) rho,
// [5n, 6n) pressure from the equation of state.
__global__ void k_snapshot(Params P, int n, const double2* pos, const double2* vel, const double* rho,
                           double* out) {
    pdl_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double2 x = pos[i], v = vel[i];
    const double r = rho[i];
    double p, c;
    eos64(P, r, p, c);
    out[i] = x.x; out[n + i] = x.y;
    out[2 * (size_t)n + i] = v.x; out[3 * (size_t)n + i] = v.y;
    out[4 * (size_t)n + i] = r;
    out[5 * (size_t)n + i] = p;
}

// What sph_rhs returns, in id order (host particles) and in the layout of its
// arrays: drho [n], acc [2n], avg [2n] as doubles, then fs [n], near [n] as ints.
template <typename R>
__global__ void k_export_rhs(Params P, Sorted<R> D, double* out) {
    pdl_begin();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P.n_tot) return;
    const int i = D.id[s];
    if (i >= P.n_host) return;
    const size_t n = (size_t)P.n_host;
    const auto a = D.acc[s], g = D.avg[s];
    out[i] = (double)D.drho[s];
    out[n + i] = (double)a.x; out[2 * n + i] = (double)a.y;
    out[3 * n + i] = (double)g.x; out[4 * n + i] = (double)g.y;
    int* flag = reinterpret_cast<int*>(out + 5 * n);
    flag[i] = D.flags[s] & 1;
    flag[n + i] = (D.flags[s] >> 1) & 1;
}

// Per-particle outputs of the last RHS in id order (host particles), as doubles.
// Layout: [0] drho, [1,2] acc, [3,4] avg, [5] fs, [6] near, [7] fra_v,
// [8..11] binv, [12..14] tau, [15..22] grads  (each block n long).
constexpr int kExportFields = 23;
template <typename R>
__global__ void k_export(Params P, Sorted<R> D, double* out) {
    pdl_begin();
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P.n_tot) return;
    int i = D.id[s];
    if (i >= P.n_host) return;
    const size_t n = (size_t)P.n_host;
    out[0 * n + i] = (double)D.drho[s];
    out[1 * n + i] = (double)D.acc[s].x; out[2 * n + i] = (double)D.acc[s].y;
    out[3 * n + i] = (double)D.avg[s].x; out[4 * n + i] = (double)D.avg[s].y;
    out[5 * n + i] = (D.flags[s] & 1) ? 1.0 : 0.0;
    out[6 * n + i] = (D.flags[s] & 2) ? 1.0 : 0.0;
    out[7 * n + i] = (double)D.fra_v[s];
    auto bi = D.binv[s]; auto n1 = D.nb1[s]; auto n2 = D.nb2[s]; auto n3 = D.nb3[s];
    const double gs = grad_scale<R>();
    out[8 * n + i] = (double)bi.x; out[9 * n + i] = (double)bi.y; out[10 * n + i] = (double)bi.z; out[11 * n + i] = (double)bi.w;
    out[12 * n + i] = (double)n1.x; out[13 * n + i] = (double)n1.y; out[14 * n + i] = (double)n1.z;
    out[15 * n + i] = gs * n1.w; out[16 * n + i] = gs * n2.x;
    out[17 * n + i] = gs * n2.y; out[18 * n + i] = gs * n2.z;
    out[19 * n + i] = gs * n2.w; out[20 * n + i] = gs * n3.x;
    out[21 * n + i] = gs * n3.y; out[22 * n + i] = gs * n3.z;
}

}  // namespace sph
