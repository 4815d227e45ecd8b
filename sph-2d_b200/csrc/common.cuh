// common.cuh -- parameters, precision traits and small device helpers of libsph_b200.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "../../include/sph_b200.h"

namespace sph {

// Status bits set on the device (atomicOr) and turned into SPH_E_* on the host.
enum : unsigned {
    ST_DOMAIN = 1u << 0,     // particle outside the cell grid
    ST_NBR_OVERFLOW = 1u << 1,   // neighbour list capacity exceeded
    ST_SKIN = 1u << 2,       // moved further than half the list skin
    ST_NONFINITE = 1u << 3,  // NaN / Inf in the state
    ST_PAIR_OVERFLOW = 1u << 4,
};

// Everything a kernel needs, derived once on the host from sph_config.
// The default-real literals of the reference are rounded through float when
// reference_literals is set (the same rounding as ifort's default reals).
struct Params {
    // switches
    int kernel_model, solver, renorm, quirks, pair_rule, shifting, muscl, xsph;
    int dsph;                     // Solver_Normalized_Delta_SPH_SPS (Taylor-Green)
    int ms, hllc, laplacian, free_surface, integrator, has_body;
    int mls_order, mls_every;     // density re-initialisation (0: off)
    double mls_alpha3;            // alpha^3 added to the moment matrix diagonal
    // ghost assignment (moving-square driver)
    int ghost_assign, wall_bc, ghost_cells;
    double ghost_h, ghost_r, ghost_kf, shock_t, grav[2];
    double ghost_s_cut, ghost_ih2;   // the largest s with sqrt(s) <= ghost_r, 1 / ghost_h^2
    // kernel / pair search
    double h, r_cut, cut_min, kfactor, gauss_e9, q_zero;
    double s_cut, s_min;     // the support test on the squared distance: the largest s with
                             // sqrt(s) <= r_cut, the smallest with sqrt(s) >= cut_min
    double inv_h, half_inv_h, inv_h2, gk;   // 1/h, 1/(2h), 1/h^2; grad_a W = gk e^{-q^2} r or gk t^3 r
    double r2_list;          // squared neighbour-list radius (support * (1 + skin))
    float r2_list32;         // the same for the mixed path's FP32 test on the hi positions,
                             // widened to cover their rounding (a superset of the FP64 list)
    // equation of state
    double rho0, c0sq, sqrt_c0, inv_sqrt_c0, eos_b, pb;
    int eos;
    // solver coefficients
    double nu, alpha, beta, fai, delta, delta_alpha, eps;
    double sv;               // support volume PI*(kernel_scale*h)^2
    double fs_thr, c1414, pi;
    double sps_dl, sps_c012, sps_23, sps_blin;
    // shifting
    double shift_beta, shift_R, shift_max, w_dx;
    int shift_n;
    // periodic box
    double box_lo[2], box_hi[2], band;
    // cell grid (row-major, cell edge >= list radius)
    double gx0, gy0, cs;
    int gnx, gny;
    // sizes
    int n_host, n_tot, max_nbr, nbr_stride;
    unsigned long long* stamp;   // where the kernel that begins a timed phase writes its start (or null)
    int rhs_gen;             // number of the RHS being evaluated (see Sorted::surf_gen)
    double skin_half2;       // (skin/2)^2: allowed squared displacement since the list build
};

// Start of a timed phase: the first kernel launched after the host marked the
// phase writes the device clock (nanoseconds, steps of 32) into its slot.  An
// event between every two passes cost 5 us of GPU time each, a third of a small
// step; this costs one thread a load.
__device__ __forceinline__ void stamp_phase(unsigned long long* slot) {
    if (slot == nullptr || blockIdx.x != 0 || blockIdx.y != 0 || threadIdx.x != 0) return;
    if (*slot != 0ull) return;
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    *slot = t;
}

// Programmatic dependent launch: every kernel of the library begins with
// pdl_begin and is launched with `launch`.  The next kernel of the stream may then
// be brought in as soon as this one's blocks have ended, while their writes and
// the launch are still being settled, and waits there for both
// (griddepcontrol.wait), so the order of the work is the stream's as before.  What
// goes is 1 to 2 us between two kernels, where a kernel of a small step takes 5 to
// 8: plain 100^2 1079 -> 795 us per 10 steps, adjoint 256^2 61.9 -> 54.6 ms, 401^2
// mixed 1956 -> 1815 us per 5.
//
// For launches up to kPdlThreads threads: above, the time between kernels no
// longer shows.  Letting the next kernel in early (griddepcontrol.launch_dependents
// at the top) was slower: 893 us in the first case, and pass A of 256^2 rose from
// 5.9 to 7.9 ms: its blocks gather on the SMs that have room while the kernel
// before still fills the others; without the size limit 2048^2 took 57.6 instead
// of 34.4 ms.
//
// No non-coherent loads (__ldg, ld.global.nc) in these kernels: they ask for memory
// that nobody writes while the kernel lives, which begins before the previous one's
// writes are complete, and nothing orders them behind the wait.
constexpr unsigned kPdlThreads = 500000;
__host__ __device__ constexpr bool pdl_small(unsigned blocks, unsigned threads) {
    return (unsigned long long)blocks * threads <= kPdlThreads;
}
__device__ __forceinline__ void pdl_begin() {
    if (pdl_small(gridDim.x * gridDim.y, blockDim.x)) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... Params_, typename... Args>
inline void launch(void (*kernel)(Params_...), dim3 grid, dim3 block, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.stream = st;
    cudaLaunchAttribute a[1];
    a[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = a;
    c.numAttrs = pdl_small(grid.x * grid.y, block.x) ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, static_cast<Params_>(args)...);     // (errors: cudaGetLastError at the callers)
}

template <typename R> struct VT;
template <> struct VT<double> { using V2 = double2; using V4 = double4; };
template <> struct VT<float> { using V2 = float2; using V4 = float4; };

template <typename R> __host__ __device__ inline typename VT<R>::V2 mk2(R a, R b);
template <> __host__ __device__ inline double2 mk2<double>(double a, double b) { return make_double2(a, b); }
template <> __host__ __device__ inline float2 mk2<float>(float a, float b) { return make_float2(a, b); }
template <typename R> __host__ __device__ inline typename VT<R>::V4 mk4(R a, R b, R c, R d);
template <> __host__ __device__ inline double4 mk4<double>(double a, double b, double c, double d) { return make_double4(a, b, c, d); }
template <> __host__ __device__ inline float4 mk4<float>(float a, float b, float c, float d) { return make_float4(a, b, c, d); }

// Particles whose rates are assembled and integrated: water; the moving-square
// driver also integrates inlet/outlet particles (Moving_Square.../Single_step_compute.f90:273,
// SPH_Time_Iteration.f90:316).
__device__ __forceinline__ bool integrated(const Params& P, int t) {
    return t == SPH_TYPE_WATER || (P.ms && t <= SPH_TYPE_INLET);
}

__device__ __forceinline__ double pw3(double x) { return x * x * x; }
__device__ __forceinline__ double pw4(double x) { double x2 = x * x; return x2 * x2; }
__device__ __forceinline__ double pw7(double x) { double x2 = x * x; double x4 = x2 * x2; return x4 * x2 * x; }
__device__ __forceinline__ float pw3(float x) { return x * x * x; }
__device__ __forceinline__ float pw4(float x) { float x2 = x * x; return x2 * x2; }

// status_equation (Taylor_Green_Vortex/status_equation.f90:60-63,
// Moving_Square.../Status_Equation.f90:56-76), always in FP64.
__device__ __forceinline__ void eos64(const Params& P, double rho, double& p, double& c) {
    double r = rho / P.rho0;
    if (P.eos == SPH_EOS_TAIT) p = P.eos_b * (pw7(r) - 1.0) + P.pb;
    else p = P.c0sq * (rho - P.rho0) + P.pb;
    c = P.sqrt_c0 * pw3(r);
}

// A squared distance rounded as the reference rounds it.
__device__ __forceinline__ double dist2(double dx, double dy) { return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)); }

// Exact replica of the reference's support test
//   distance = sqrt(dot(dx,dx));  distance <= kernel_scale*h  .and.  distance >= 1.0E-7
// (find_particle_pair.f90:79-87) with the products and the sum rounded
// separately (no FMA), so the pair set is bit-identical to the CPU's.
__device__ __forceinline__ bool in_support(const Params& P, double dx, double dy, double& d) {
    d = __dsqrt_rn(dist2(dx, dy));
    return d <= P.r_cut && d >= P.cut_min;
}

// The same test without the square root: sqrt is monotonic and correctly rounded
// on both sides, so with s rounded as above d <= r_cut is s <= s_cut and
// d >= cut_min is s >= s_min for the bounds derive_params finds; the pair set is
// the same, bit for bit.  s2: the squared distance.
__device__ __forceinline__ bool in_support_s2(const Params& P, double dx, double dy, double& s2) {
    s2 = dist2(dx, dy);
    return s2 <= P.s_cut && s2 >= P.s_min;
}

// A product rounded on its own (never fused into a following add).
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// FP64 reciprocal and reciprocal square root for the pair loops: the hardware's
// coarse approximation (about 20 bits) corrected by one third-order Newton
// (Householder) step.  With r0 = (1 - e0)/x the first gives r0 (1 + e + e^2),
// e = 1 - x r0, relative error e^3; with y0 = (1 - e0)/sqrt(x) the second gives
// y0 (1 + e/2 + 3 e^2/8), e = 1 - x y0^2, relative error of order e^3: both far
// below the rounding of the last multiply-add, so they are within about one ulp.
// No branch and 3 / 5 FP64 operations, where the quotient and the square root
// followed by a quotient take a multiple of that and a special-case branch
// (tests/test_gpu_fp64_math.py measures them against the correctly rounded
// values).  For the arguments of the pair loops: positive, normal, not huge.
__device__ __forceinline__ double rcp64(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ double rsqrt64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y * y, 1.0);      // y has 21 significant bits: y y is exact
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

// Loads of what an earlier kernel wrote.  (volatile: never moved above pdl_begin;
// otherwise free of the stores around them, which plain loads are not, as the
// arrays may alias for all the compiler knows: with those the lane list build took
// 17.0 instead of 15.5 us at 100^2 and k_shift_gather 483 instead of 448 us at 2048^2.)
#define SPH_LOAD1(T, t, c)                                              \
    __device__ __forceinline__ T load(const T* p) {                     \
        T v;                                                            \
        asm volatile("ld.global." t " %0, [%1];" : "=" c(v) : "l"(p)); \
        return v;                                                       \
    }
SPH_LOAD1(unsigned, "u32", "r")
SPH_LOAD1(int, "s32", "r")
SPH_LOAD1(double, "f64", "d")
#undef SPH_LOAD1
__device__ __forceinline__ double2 load(const double2* p) {
    double2 v;
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 load(const float2* p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 load(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// One 32-byte record: a single 256-bit load for FP64 (arrays of 32-byte elements in
// 256-byte aligned allocations, so every element is 32-byte aligned), 128-bit for FP32.
__device__ __forceinline__ double4 load4(const double4* p) {
    double4 v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 load4(const float4* p) { return *p; }

// Lanes that share one particle in the neighbour loops (L = 1: a thread per
// particle): the group's lanes take the list entries lane, lane + L, ... and add
// their sums in a fixed butterfly order.
template <int L>
struct Lanes {
    int lane;            // this thread's place in its group
    unsigned below;      // the lanes of the group before this one, as a warp mask
    unsigned group;      // the group as a warp mask
    __device__ __forceinline__ Lanes() {
        const int l = threadIdx.x & 31;
        lane = L == 1 ? 0 : l & (L - 1);
        group = L == 32 ? 0xffffffffu : ((1u << (L & 31)) - 1u) << (l & ~(L - 1));
        below = group & ((1u << l) - 1u);
    }
    // the particle of this thread
    static __device__ __forceinline__ int particle() { return (int)((blockIdx.x * blockDim.x + threadIdx.x) / L); }
    template <typename T>
    __device__ __forceinline__ void sum(T& v) const {
#pragma unroll
        for (int o = 1; o < L; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    }
};

// Plain accumulator for the FP64 path.
struct DSum {
    double s;
    __device__ __forceinline__ void init() { s = 0.0; }
    __device__ __forceinline__ void add(double x) { s += x; }
    __device__ __forceinline__ double val() const { return s; }
};

// The mixed path's sums: FP32 terms added in FP64 (one conversion and one FP64
// add per term; a compensated FP32 TwoSum takes seven FP32 operations for a
// sum of about the same accuracy).
struct WSum {
    double s;
    __device__ __forceinline__ void init() { s = 0.0; }
    __device__ __forceinline__ void add(float x) { s += (double)x; }
    __device__ __forceinline__ float val() const { return (float)s; }
};

template <typename R> struct Acc;
template <> struct Acc<double> { using T = DSum; };
template <> struct Acc<float> { using T = WSum; };

// compute_kernel for one pair: W and grad_a W(x_a - x_b) = f(d) (x_a - x_b).
// Improved Gaussian: Taylor_Green_Vortex/compute_kernel.f90:122-134.
// Wendland C2: Moving_Square.../Compute_Kernel.f90:179-193.
template <typename R>
__device__ __forceinline__ void kernel_w_dw(const Params& P, R d, R px, R py, R& w, R& gx, R& gy) {
    const R h = (R)P.h;
    const R factor = (R)P.kfactor;
    R q = d / h;
    if (P.kernel_model == SPH_KERNEL_GAUSSIAN) {
        R e = exp(-(q * q));
        w = (e - (R)P.gauss_e9) * factor;
        R g = (e * (R(-2) * q));
        R dh = d * h;
        gx = g * px / dh * factor;
        gy = g * py / dh * factor;
    } else {
        R t = R(1) - q / R(2);
        w = factor * (R(1) + R(2) * q) * pw4(t);
        R g = factor * (R(-5) * q * pw3(t));
        R dh = d * h;
        gx = g * px / dh;
        gy = g * py / dh;
    }
    if (q <= (R)P.q_zero) { gx = R(0); gy = R(0); }
}

}  // namespace sph
