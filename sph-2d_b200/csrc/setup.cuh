// setup.cuh -- per-step set-up kernels: periodic wrap and images, the
// background-cell sort, cell ranges and the per-particle neighbour lists.
#pragma once
#include "common.cuh"

namespace sph {

// Particle arrays in id order ("staging"): the host particles 0..n_host-1
// followed by the periodic images of this step, numbered as the reference
// appends them (Distribute_Period_Boundary_Particle.f90:95-206).
struct Staging {
    double2* pos;     // x, y
    double2* vel;     // u, v
    double* rho;
    double* mass;
    double* smass;    // mass the SPS force multiplies with (quirk A.6), default = mass
    int* type;
    int* itype;       // initial type (body force), images get SPH_TYPE_PERIODIC
    int* blabel;      // wall label of the ghost assignment (host particles)
    // rates of the last RHS of the previous step (the reused K1), host particles only
    double* r_drho;
    double2* r_acc;
    double2* r_avg;
    // image counts and offsets of this step, kept for routing image adjoints:
    // left/right images of host i sit at n_host + lr_off[i] + k (k < lr_cnt[i]),
    // bottom/top images of source s at n_host + n_lr + tb_off[s] + k (k < tb_cnt[s])
    int* lr_cnt;
    int* lr_off;
    int* tb_cnt;
    int* tb_off;
};

// --- 1. periodic wrap (Distribute_Period_Boundary_Particle.f90:56-90), done by
// the first image count below: a host particle outside the box re-enters on the
// opposite side before its images are counted.
__device__ __forceinline__ double2 wrap_position(const Params& P, double2 x) {
    const double Lx = P.box_hi[0] - P.box_lo[0], Ly = P.box_hi[1] - P.box_lo[1];
    if (x.x > P.box_hi[0]) x.x = x.x - Lx;
    else if (x.x < P.box_lo[0]) x.x = x.x + Lx;
    if (x.y > P.box_hi[1]) x.y = x.y - Ly;
    else if (x.y < P.box_lo[1]) x.y = x.y + Ly;
    return x;
}

// --- 2. images and the counting sort into cells -----------------------------
// The step set-up is six launches with no host wait on its critical path:
//   k_img_count   wraps the host positions and counts each block's images; the
//                 last block to finish scans the block sums and posts the totals
//                 to the host (which reads them while the next kernels run, to
//                 size the launches that follow)
//   k_img_emit    writes the images at their offsets, the cell key of every
//                 particle and its arrival number in its cell
//   k_cell_scan   exclusive scan of the cell counts (last block: of the block sums)
//   k_place       cell ranges (on a grid of mostly empty cells, sparse_grid, only those
//                 that hold particles); particle -> slot, unordered inside a cell
//   k_gather_sorted  orders each cell by id while it copies the arrays: the same
//                 order as a stable sort of the keys
//   k_build_lists
// Bound by launch latency below about 10^5 particles and by HBM above.  Against
// image counts and offsets by two library scans with a host wait each, a library
// radix sort and separate key and range passes (18 launches), same slot order:
// images + sort + lists 166 -> 59 us per step at 100^2 (FP64), 195 -> 85 us at
// 401^2 and 1.11 -> 0.98 ms at 2048^2 (mixed); 29, 62 us and 0.91 ms with the lanes,
// the dependent launches and the shared reads below.
constexpr int kImgThreads = 1024;         // host particles per block
constexpr int kScanThreads = 1024;        // cell scan: kScanCells cells per block
constexpr int kScanShift = 12, kScanCells = 1 << kScanShift;

// What the set-up kernels share (device memory of the handle).
struct SetupBuf {
    int4* blk;            // [image blocks] image sums (x: left/right, y: bottom/top of host
                          // particles, z: bottom/top of left/right images), then exclusive
    int* tot;             // [3] their totals
    unsigned* done;       // [4] blocks finished (image count, cell scan, diagnostics, body force); left at 0
    unsigned* key;        // [cap] cell of particle i (id order), ncells = not binned
    int* rank;            // [cap] its arrival number in the cell
    int* cnt;             // [ncells + 1] particles per cell
    int* pre;             // [ncells + 1] exclusive scan within the scan block
    int* blkoff;          // [scan blocks] offset of the scan block
    unsigned* perm;       // [cap] slot -> id, unordered inside a cell
    int ncells;
};

// Totals the host waits for (page-locked, mapped): written by the device, seq last.
struct HostBox {
    int tot[3];
    volatile unsigned seq;        // (the host reads it with acquire order, then tot)
    unsigned status;
    int nsurf;
    double diag[8];
    long long pair_last[2];       // offset and count of the last particle's pairs
};

__device__ __forceinline__ int band_count(double v, double lo, double hi, double band) {
    return (v <= (lo + band) && v >= lo ? 1 : 0) + (v >= (hi - band) && v <= hi ? 1 : 0);
}

// Exclusive scan over one block of up to 1024 threads; total returned to all.
template <typename T>
__device__ __forceinline__ T block_scan(T v, T* sh, T& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) sh[w] = inc;
    __syncthreads();
    if (w == 0) {
        T x = lane < (int)(blockDim.x >> 5) ? sh[lane] : T(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T u = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += u;
        }
        sh[lane] = x;
    }
    __syncthreads();
    total = sh[(blockDim.x >> 5) - 1];
    const T base = w > 0 ? sh[w - 1] : T(0);
    __syncthreads();
    return base + inc - v;
}

// True in every thread of the last block of the grid to get here (its earlier
// writes to global memory, and every other block's, are then visible).
__device__ __forceinline__ bool last_block(unsigned* done, int* sh_flag) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned t = atomicAdd(done, 1u);
        *sh_flag = t == gridDim.x - 1;
    }
    __syncthreads();
    const bool last = *sh_flag != 0;
    if (last) {
        __threadfence();
        if (threadIdx.x == 0) *done = 0u;
    }
    return last;
}

// axis 0: left/right images of the host particles (Distribute_Period_Boundary_Particle.f90:98-148),
// axis 1: bottom/top images of host particles and of left/right images (:156-206).
// A left/right image has its source's y, so every count is a function of the
// host particle.  Packed sums: 20 bits each (at most 4 per particle).
__device__ __forceinline__ void image_counts(const Params& P, double2 x, bool ill, int& lr, int& tb) {
    lr = tb = 0;
    if (ill) return;
    lr = band_count(x.x, P.box_lo[0], P.box_hi[0], P.band);
    tb = band_count(x.y, P.box_lo[1], P.box_hi[1], P.band);
}

// Body_Motion_Solver (Moving_Square.../Body_Motion_Solver.f90:187-193): the body
// particles (initial type SPH_TYPE_BODY) move by the step's displacement.  Applied
// by the kernel that first reads the positions of a step.
__device__ __forceinline__ double2 move_body(const Staging& S, int i, double2 disp) {
    double2 x = S.pos[i];
    if ((disp.x != 0.0 || disp.y != 0.0) && S.itype[i] == SPH_TYPE_BODY) {
        x = make_double2(x.x + disp.x, x.y + disp.y);
        S.pos[i] = x;
    }
    return x;
}

__global__ void __launch_bounds__(kImgThreads) k_img_count(Params P, Staging S, SetupBuf B, HostBox* box, unsigned seq,
                                                           double2 disp, int clear) {
    pdl_begin();
    stamp_phase(P.stamp);
    __shared__ unsigned long long sh[32];
    __shared__ int flag;
    const int i = blockIdx.x * kImgThreads + threadIdx.x;
    if (clear)
        for (int c = i; c <= B.ncells; c += gridDim.x * kImgThreads) B.cnt[c] = 0;
    int lr = 0, tb = 0;
    if (i < P.n_host) {
        const double2 xy = move_body(S, i, disp);
        const bool ill = S.type[i] == SPH_TYPE_ILL;
        const double2 w = wrap_position(P, xy);
        if (!ill && (w.x != xy.x || w.y != xy.y)) S.pos[i] = w;
        image_counts(P, w, ill, lr, tb);
    }
    unsigned long long total;
    block_scan<unsigned long long>((unsigned long long)lr | ((unsigned long long)tb << 20) |
                                       ((unsigned long long)(lr * tb) << 40), sh, total);
    if (threadIdx.x == 0)
        B.blk[blockIdx.x] = make_int4((int)(total & 0xfffff), (int)((total >> 20) & 0xfffff), (int)(total >> 40), 0);
    if (!last_block(&B.done[0], &flag)) return;
    // the last block: exclusive scan of the block sums, then the totals
    __shared__ int shi[32];
    int run[3] = {0, 0, 0};
    const int nb = gridDim.x;
    for (int b0 = 0; b0 < nb; b0 += kImgThreads) {
        const int b = b0 + threadIdx.x;
        const int4 v = b < nb ? __ldcg(&B.blk[b]) : make_int4(0, 0, 0, 0);
        int t0, t1, t2;
        const int e0 = block_scan<int>(v.x, shi, t0), e1 = block_scan<int>(v.y, shi, t1),
                  e2 = block_scan<int>(v.z, shi, t2);
        if (b < nb) B.blk[b] = make_int4(run[0] + e0, run[1] + e1, run[2] + e2, 0);
        run[0] += t0; run[1] += t1; run[2] += t2;
    }
    if (threadIdx.x == 0) {
        for (int k = 0; k < 3; ++k) { B.tot[k] = run[k]; box->tot[k] = run[k]; }
        __threadfence_system();
        box->seq = seq;
    }
}

// Cell key (row-major cells of edge >= list radius) and arrival number of id o.
// Particles that are not binned (Assign_boundary_particles.f90:82) or off the
// grid go past the last cell; there may be many (a host that marks what has left the
// domain), so with MANY the threads of a warp that are here together take their numbers
// with one atomic: with an atomic each on that one counter the images of 2^20 particles took
// 48 / 375 / 640 us a step with none / half / nine tenths not binned.
template <bool MANY>
__device__ __forceinline__ void cell_key(const Params& P, const SetupBuf& B, int o, double2 x, int t, unsigned* status) {
    unsigned key = (unsigned)B.ncells;
    if (t != SPH_TYPE_ILL && t != 0) {
        const double fx = floor((x.x - P.gx0) / P.cs), fy = floor((x.y - P.gy0) / P.cs);
        const int cx = (int)fx, cy = (int)fy;
        if (fx >= 0.0 && fy >= 0.0 && cx < P.gnx && cy < P.gny) key = (unsigned)(cy * P.gnx + cx);
        else atomicOr(status, ST_DOMAIN);
    }
    B.key[o] = key;
    if (!MANY || key < (unsigned)B.ncells) {
        B.rank[o] = atomicAdd(&B.cnt[key], 1);
    } else {
        const unsigned here = __activemask();
        const int lane = threadIdx.x & 31, first = __ffs(here) - 1;
        int base = 0;
        if (lane == first) base = atomicAdd(&B.cnt[key], __popc(here));
        B.rank[o] = __shfl_sync(here, base, first) + __popc(here & ((1u << lane) - 1u));
    }
}

// What an image takes from its source, read once for all its images (up to eight
// in a thin box) and before their stores: the loads of an image used to wait for
// the previous image's stores.  images 14.4 -> 12.6 us per step at 100^2, 206 ->
// 169 us at 2048^2.
struct ImageSource {
    double2 vel;
    double rho, mass, smass;
};
// One image with id o.
__device__ __forceinline__ void put_image(const Params& P, const Staging& S, const SetupBuf& B, const ImageSource& q, int o,
                                          double2 x, int cap, unsigned* status) {
    if (o >= cap) return;                       // the host sees the total and stops
    S.pos[o] = x;
    S.vel[o] = q.vel;
    S.rho[o] = q.rho;
    S.mass[o] = q.mass;
    S.smass[o] = q.smass;
    S.type[o] = SPH_TYPE_PERIODIC;
    S.itype[o] = SPH_TYPE_PERIODIC;
    cell_key<false>(P, B, o, x, SPH_TYPE_PERIODIC, status);
}

// periodic: emit the images, numbered as the reference appends them (left/right
// images in host order, bottom/top images of the host particles, then of the
// left/right images; the low side first).  route: also keep the counts and
// offsets for the reverse sweep.
__global__ void __launch_bounds__(kImgThreads) k_img_emit(Params P, Staging S, SetupBuf B, int cap, int periodic,
                                                          int route, unsigned* status, double2 disp) {
    pdl_begin();
    stamp_phase(P.stamp);
    __shared__ unsigned long long sh[32];
    const int i = blockIdx.x * kImgThreads + threadIdx.x;
    const bool live = i < P.n_host;
    double2 x = make_double2(0.0, 0.0);
    int t = SPH_TYPE_ILL;
    if (live) { x = move_body(S, i, disp); t = S.type[i]; }
    if (live) cell_key<true>(P, B, i, x, t, status);
    if (!periodic) return;
    int lr, tb;
    image_counts(P, x, t == SPH_TYPE_ILL, lr, tb);
    unsigned long long total;
    const unsigned long long e = block_scan<unsigned long long>(
        (unsigned long long)lr | ((unsigned long long)tb << 20) | ((unsigned long long)(lr * tb) << 40), sh, total);
    if (!live || (lr == 0 && tb == 0 && !route)) return;
    const int4 base = B.blk[blockIdx.x];
    const int n_lr = B.tot[0], tb_host = B.tot[1];
    const int o_lr = base.x + (int)(e & 0xfffff), o_tb = base.y + (int)((e >> 20) & 0xfffff),
              o_lt = tb_host + base.z + (int)(e >> 40);
    const int first_tb = P.n_host + n_lr;
    if (route) {
        S.lr_cnt[i] = lr; S.lr_off[i] = o_lr;
        S.tb_cnt[i] = tb; S.tb_off[i] = o_tb;
        for (int k = 0; k < lr; ++k) {
            const int s = P.n_host + o_lr + k;
            if (s < cap) { S.tb_cnt[s] = tb; S.tb_off[s] = o_lt + k * tb; }
        }
    }
    if (lr == 0 && tb == 0) return;
    const ImageSource src = {S.vel[i], S.rho[i], S.mass[i], S.smass[i]};
    const double Lx = P.box_hi[0] - P.box_lo[0], Ly = P.box_hi[1] - P.box_lo[1];
    // sides of each axis in order: low side (shift +L), high side (-L)
    const bool xlo = x.x <= (P.box_lo[0] + P.band) && x.x >= P.box_lo[0];
    const bool xhi = x.x >= (P.box_hi[0] - P.band) && x.x <= P.box_hi[0];
    const bool ylo = x.y <= (P.box_lo[1] + P.band) && x.y >= P.box_lo[1];
    const bool yhi = x.y >= (P.box_hi[1] - P.band) && x.y <= P.box_hi[1];
    // k = 0: the particle itself, then its left/right images
    int o = P.n_host + o_lr, k = 0;
#pragma unroll 1
    for (int sx = -1; sx < 2; ++sx) {
        if ((sx == 0 && !xlo) || (sx == 1 && !xhi)) continue;
        double2 y = x;
        if (sx >= 0) {
            y.x = x.x + (sx == 0 ? Lx : -Lx);
            put_image(P, S, B, src, o, y, cap, status);
            ++o;
        }
        int q = first_tb + (sx < 0 ? o_tb : o_lt + k * tb);
        if (sx >= 0) ++k;
        if (ylo) { put_image(P, S, B, src, q, make_double2(y.x, y.y + Ly), cap, status); ++q; }
        if (yhi) put_image(P, S, B, src, q, make_double2(y.x, y.y + (-Ly)), cap, status);
    }
}

// Exclusive scan of the cell counts within blocks of kScanCells cells; the last
// block scans the block sums.
__global__ void __launch_bounds__(kScanThreads) k_cell_scan(SetupBuf B, unsigned long long* stamp) {
    pdl_begin();
    stamp_phase(stamp);
    __shared__ int sh[32];
    __shared__ int flag;
    constexpr int per = kScanCells / kScanThreads;
    const int c0 = blockIdx.x * kScanCells + threadIdx.x * per;
    int v[per], s = 0;
#pragma unroll
    for (int k = 0; k < per; ++k) { v[k] = c0 + k <= B.ncells ? B.cnt[c0 + k] : 0; s += v[k]; }
    int total;
    int run = block_scan<int>(s, sh, total);
    if (total != 0) {                // (nobody reads the offsets of empty cells)
#pragma unroll
        for (int k = 0; k < per; ++k)
            if (c0 + k <= B.ncells) { B.pre[c0 + k] = run; run += v[k]; }
    }
    if (gridDim.x == 1) {            // one block's offset is 0: nothing to scan
        if (threadIdx.x == 0) B.blkoff[0] = 0;
        return;
    }
    if (threadIdx.x == 0) B.blkoff[blockIdx.x] = total;
    if (!last_block(&B.done[1], &flag)) return;
    int sum = 0;
    for (int b0 = 0; b0 < (int)gridDim.x; b0 += kScanThreads) {
        const int b = b0 + threadIdx.x;
        const int u = b < (int)gridDim.x ? __ldcg(&B.blkoff[b]) : 0;
        int t;
        const int e = block_scan<int>(u, sh, t);
        if (b < (int)gridDim.x) B.blkoff[b] = sum + e;
        sum += t;
    }
}

// Cell ranges (-1 for an empty cell), and each particle at its arrival place.  SPARSE:
// the ranges were set to -1 before, and the first particle of a cell writes its.
template <bool SPARSE>
__global__ void k_place(int n_tot, SetupBuf B, int* cell_start, int* cell_end) {
    pdl_begin();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (!SPARSE && t < B.ncells) {
        const int n = B.cnt[t], st = B.blkoff[t >> kScanShift] + B.pre[t];
        cell_start[t] = n ? st : -1;
        cell_end[t] = n ? st + n : -1;
    }
    if (t < n_tot) {
        const unsigned k = B.key[t];
        const int st = B.blkoff[k >> kScanShift] + B.pre[k], r = B.rank[t];
        B.perm[st + r] = (unsigned)t;
        if (SPARSE && r == 0 && k < (unsigned)B.ncells) {
            cell_start[k] = st;
            cell_end[k] = st + B.cnt[k];
        }
    }
}

// Device-side arrays in cell-sorted order (templated on the pair precision).
template <typename R>
struct Sorted {
    using V2 = typename VT<R>::V2;
    using V4 = typename VT<R>::V4;
    int* id;          // id-order index (host index, or n_host + image number)
    int* slot_of;     // inverse: the sorted slot of id i
    uint8_t* nflag;   // reverse sweep: bit 0 near a ghost (within its interpolation radius),
                      // bit 1 a pair neighbour of a body particle
    int* type;
    int* itype;       // initial type (SPH_TYPE_BODY marks the body)
    int* blabel;      // wall label of the ghost assignment (0 for images)
    double2* pos;     // current stage position (FP64)
    double2* pos0;    // step-start (master) position, also the list-build position
    double2* vel0;    // step-start velocity (FP64 master)
    double* rho0;     // step-start density (FP64 master)
    double* mass;
    double* smass;
    double4* kin;     // u, v, rho, p (FP64 in both paths: pair differences are  -- neighbour record 1
                      // formed from it in FP64 before the FP32 arithmetic)
    V4* aux;          // m, V = m/rho, c, smass                      -- neighbour record 2
    V4* nb1;          // tau_xx, tau_xy, tau_yy, grad rho x          -- neighbour record 3
    V4* nb2;          // grad rho y, grad p x, grad p y, grad u x     -- neighbour record 4
    V4* nb3;          // grad u y, grad v x, grad v y, 1/rho -- neighbour record 5 (MUSCL)
                      // (the FP32 records hold the gradients halved: grad_scale<R>())
    V4* binv;         // B^-1 (11, 12, 21, 22) in the pair precision
    double4* binv64;  // B^-1 in FP64 (applied to the FP64 shifting sum)
    R* fra_v;
    uint8_t* flags;   // bit0 surface, bit1 near surface, bit2 surface candidate
    // rates of the current RHS
    R* drho;
    V2* acc;
    V2* avg;
    double2* shift;   // shifting displacement (last RHS of a step), FP64
    // Runge-Kutta sums K1 + 2 K2 + 2 K3 (time_iteration.f90:1040-1045)
    R* ks_r;
    V2* ks_a;
    double2* ks_v;    // velocity sums in FP64 (they move the FP64 positions)
    // rates carried to the next step (K1 reuse)
    R* c_drho;
    V2* c_acc;
    V2* c_avg;
    // neighbour lists: slot-major [max_nbr][stride], bit 31 = "this particle has the lower id"
    unsigned* nbr;
    int* nnbr;
    // the pairs of the current RHS (list entries inside the support), same layout,
    // written by pass A and read by the passes that follow it
    unsigned* pairs;
    int* npairs;
    // cell ranges
    int* cell_start;
    int* cell_end;
    // mixed path only: the kinematic record and the position split into float
    // hi + lo parts (v = hi + lo, hi = (float)v), so pass C forms pair
    // differences (hi_i - hi_j) + (lo_i - lo_j) in FP32 with the accuracy of the
    // FP64 difference rounded to FP32, without FP64 arithmetic or conversions
    double* vol64;    // m / rho in FP64 (the mixed path's FP64 shifting sum)
    float4* kh;       // u, v, rho, p  (hi)
    float4* kl;       //               (lo)
    float4* xhl;      // x hi, y hi, x lo, y lo
    float2* xh0;      // (float) of the list-build position
    // the other copy of what a stage writes (position and records): pass C forms
    // the next stage's state there while its neighbours still read this one
    double2* pos_n;
    double4* kin_n;
    V4* aux_n;
    double* vol64_n;
    float4* kh_n;
    float4* kl_n;
    float4* xhl_n;
    int* surf_gen;    // [1] Params::rhs_gen of the last RHS with a surface particle
};

// The sorted arrays with the two copies exchanged.
template <typename R>
inline void swap_stage_state(Sorted<R>& D) {
    auto sw = [](auto& x, auto& y) { auto t = x; x = y; y = t; };
    sw(D.pos, D.pos_n); sw(D.kin, D.kin_n); sw(D.aux, D.aux_n); sw(D.vol64, D.vol64_n);
    sw(D.kh, D.kh_n); sw(D.kl, D.kl_n); sw(D.xhl, D.xhl_n);
}

// Factor from the stored gradient records (nb1.w, nb2, nb3.xyz) to the
// gradients: the FP32 records hold 1/2 grad phi (pass C uses only that).
template <typename R>
__host__ __device__ constexpr double grad_scale() { return sizeof(R) == 4 ? 2.0 : 1.0; }

// Hi/lo split of the records a particle's pass-C neighbours read (mixed path).
__device__ __forceinline__ void split_to(float4* kh, float4* kl, float4* xhl, int s, double2 x, double4 k) {
    const float uh = (float)k.x, vh = (float)k.y, rh = (float)k.z, ph = (float)k.w;
    kh[s] = make_float4(uh, vh, rh, ph);
    kl[s] = make_float4((float)(k.x - (double)uh), (float)(k.y - (double)vh), (float)(k.z - (double)rh),
                        (float)(k.w - (double)ph));
    const float xh = (float)x.x, yh = (float)x.y;
    xhl[s] = make_float4(xh, yh, (float)(x.x - (double)xh), (float)(x.y - (double)yh));
}
template <typename R>
__device__ __forceinline__ void store_split(Sorted<R>& D, int s, double2 x, double4 k) {
    if (sizeof(R) != 4) return;
    D.vol64[s] = D.mass[s] / k.z;
    split_to(D.kh, D.kl, D.xhl, s, x, k);
}

// The records of a state (x, v, rho) with mass m and SPS mass sm; next: into the
// other copy.
template <typename R>
__device__ __forceinline__ void store_records(const Params& P, const Sorted<R>& D, int s, double2 x, double u, double v,
                                              double rho, double m, double sm, bool next) {
    double p, c;
    eos64(P, rho, p, c);
    const double4 k = make_double4(u, v, rho, p);
    (next ? D.pos_n : D.pos)[s] = x;
    (next ? D.kin_n : D.kin)[s] = k;
    (next ? D.aux_n : D.aux)[s] = mk4<R>((R)m, (R)(m / rho), (R)c, (R)sm);
    if (sizeof(R) == 4) {
        (next ? D.vol64_n : D.vol64)[s] = m / rho;
        if (next) split_to(D.kh_n, D.kl_n, D.xhl_n, s, x, k);
        else split_to(D.kh, D.kl, D.xhl, s, x, k);
    }
}

// Runge-Kutta stages of time_iteration.f90 (water particles only; images and
// boundary particles keep their step-start state, as the reference only
// updates type 2 at :944, :978, :1008, :1038):
//   stage 0  rho = rho0 + drhodt*dt/2, v = v0 + 0.5 dt a + avg, x = x0 + 0.5 dt v    K = K1
//   stage 1  same with the second RHS                                          K += 2 K2
//   stage 2  full dt with the third RHS                                        K += 2 K3
//   stage 3  rho = rho0 + (K + drhodt) dt/6, v = v0 + (K_a + a) dt/6 + avg,
//            x = x0 + (K_v + v) dt/6 + 0.5 dt^2 a; then Shift_particle_position.
// Stage 0 uses the rates carried from the previous step (K1 reuse, :940-965)
// unless this is the first step, when a fresh RHS precedes it (:821).
//
// With SPH_INTEGRATOR_EULER_PC (Moving_Square.../SPH_Time_Iteration.f90:304-334) the
// stages are 10 (predictor) and 11 (corrector):
//   predictor  rho = rho0 + drhodt dt, x = x0 + dt (v0 + avg) + 0.5 a dt^2, v = v0 + dt a
//   corrector  rho = rho0 + 0.5 (drhodt + drhodt_p) dt,
//              x = x0 + 0.5 dt (v_p + v0) + avg dt + 0.5 a dt^2, v = v0 + 0.5 dt (a + a_p)
//
// The state a stage takes particle s to from the step-start state (x0, v0, r0)
// with the rates (dr, a, g), and the sums and carried rates it leaves.
template <typename R>
__device__ __forceinline__ void stage_update(const Sorted<R>& D, int s, int stage, double dt, double2 x0, double2 v0,
                                             double r0, double dr, double ax, double ay, double gx, double gy, double& x,
                                             double& y, double& u, double& v, double& rho) {
    using V2 = typename VT<R>::V2;
    if (stage == 10) {
        rho = r0 + dr * dt;
        x = x0.x + dt * (v0.x + gx) + 0.5 * ax * (dt * dt);
        y = x0.y + dt * (v0.y + gy) + 0.5 * ay * (dt * dt);
        u = v0.x + dt * ax;
        v = v0.y + dt * ay;
        D.ks_r[s] = (R)dr;
        D.ks_a[s] = mk2<R>((R)ax, (R)ay);
        D.ks_v[s] = v0;
    } else if (stage == 11) {
        const double4 kp = D.kin[s];          // predicted velocity
        const V2 ka = D.ks_a[s];
        const double2 kv = D.ks_v[s];
        rho = r0 + 0.5 * (dr + (double)D.ks_r[s]) * dt;
        x = x0.x + 0.5 * dt * (kp.x + kv.x) + gx * dt + 0.5 * ax * (dt * dt);
        y = x0.y + 0.5 * dt * (kp.y + kv.y) + gy * dt + 0.5 * ay * (dt * dt);
        u = v0.x + 0.5 * dt * (ax + (double)ka.x);
        v = v0.y + 0.5 * dt * (ay + (double)ka.y);
    } else if (stage < 3) {
        const double f = stage < 2 ? 0.5 * dt : dt;
        rho = stage < 2 ? r0 + dr * dt / 2 : r0 + dr * dt;
        u = v0.x + f * ax + gx;
        x = x0.x + f * u;
        v = v0.y + f * ay + gy;
        y = x0.y + f * v;
        if (stage == 0) {
            D.ks_r[s] = (R)dr;
            D.ks_a[s] = mk2<R>((R)ax, (R)ay);
            D.ks_v[s] = make_double2(u, v);
        } else {
            D.ks_r[s] = D.ks_r[s] + R(2) * (R)dr;
            V2 ka = D.ks_a[s];
            double2 kv = D.ks_v[s];
            D.ks_a[s] = mk2<R>(ka.x + R(2) * (R)ax, ka.y + R(2) * (R)ay);
            D.ks_v[s] = make_double2(kv.x + 2 * u, kv.y + 2 * v);
        }
    } else {
        const V2 ka = D.ks_a[s];
        const double2 kv = D.ks_v[s];
        rho = r0 + ((double)D.ks_r[s] + dr) * dt / 6.0;
        u = v0.x + ((double)ka.x + ax) * dt / 6.0 + gx;
        x = x0.x + ((double)kv.x + u) * dt / 6.0 + 0.5 * dt * dt * ax;
        v = v0.y + ((double)ka.y + ay) * dt / 6.0 + gy;
        y = x0.y + ((double)kv.y + v) * dt / 6.0 + 0.5 * dt * dt * ay;
    }
    if (stage == 3 || stage == 11) {
        // rates of this last RHS become next step's K1
        D.c_drho[s] = (R)dr;
        D.c_acc[s] = mk2<R>((R)ax, (R)ay);
        D.c_avg[s] = mk2<R>((R)gx, (R)gy);
    }
}

// What a kernel needs to apply the stage that follows it to its own particle.
struct StageArgs {
    int mode;             // STAGE_NONE, STAGE_MID (into the other copy), STAGE_END
    int stage;
    double dt;
    int to_staging;       // STAGE_END: also write the id-order state
    unsigned* status;
    Staging S;
};
enum { STAGE_NONE = 0, STAGE_MID = 1, STAGE_END = 2 };

// the neighbour lists stay exact while nobody moved more than half the skin
__device__ __forceinline__ void check_skin(const Params& P, double2 x0, double x, double y, unsigned* status) {
    const double ddx = x - x0.x, ddy = y - x0.y;
    if (ddx * ddx + ddy * ddy > P.skin_half2) atomicOr(status, ST_SKIN);
}

// The end of a step for particle s: the new master state, and (to_staging) the
// new state and carried rates of a host particle in the id-order arrays, exactly
// what k_unsort would copy there, so the next step's set-up and a state read
// need no unsort pass (static fields are unchanged in staging).
template <typename R>
__device__ __forceinline__ void store_end(const Params& P, const Sorted<R>& D, const Staging& S, int s, double x, double y,
                                          double u, double v, double rho, double dr, double ax, double ay, double gx,
                                          double gy, int to_staging, unsigned* status) {
    if (!(isfinite(x) && isfinite(y) && isfinite(u) && isfinite(v) && isfinite(rho))) atomicOr(status, ST_NONFINITE);
    D.pos0[s] = make_double2(x, y);
    D.vel0[s] = make_double2(u, v);
    D.rho0[s] = rho;
    if (to_staging) {
        const int i = D.id[s];
        if (i < P.n_host) {
            S.pos[i] = make_double2(x, y);
            S.vel[i] = make_double2(u, v);
            S.rho[i] = rho;
            // the carried rates as k_unsort reads them back (rounded to R)
            S.r_drho[i] = (double)(R)dr;
            S.r_acc[i] = make_double2((double)(R)ax, (double)(R)ay);
            S.r_avg[i] = make_double2((double)(R)gx, (double)(R)gy);
        }
    }
}

// The capped shift (Shift_particle_position.f90:108-131) of a water particle not
// near the free surface: displacement sh, density gradient (g0, g1).
__device__ __forceinline__ void shift_by(const Params& P, double2 sh, double g0, double g1, double& x, double& y,
                                         double& rho) {
    double s0 = sh.x, s1 = sh.y;
    const double amp = sqrt(s0 * s0 + s1 * s1);
    if (amp > P.shift_max) { s0 = s0 / amp * P.shift_max; s1 = s1 / amp * P.shift_max; }
    x = x + s0;
    y = y + s1;
    rho = rho + g0 * s0;
    rho = rho + g1 * s1;
}

// --- 4. gather the id-ordered arrays into cell order -----------------------
// Thread t holds the particle at place t; its slot is the cell's start plus the
// number of lower ids in the cell (about 8 reads that the warp shares).
template <typename R>
__global__ void k_gather_sorted(Params P, Staging S, Sorted<R> D, SetupBuf B, StageArgs G) {
    pdl_begin();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= P.n_tot) return;
    const int i = (int)B.perm[t];
    const unsigned key = B.key[i];
    int s = t;                         // not binned: any order
    if (key < (unsigned)B.ncells) {
        const int st = D.cell_start[key], en = D.cell_end[key];
        s = st;
        for (int q = st; q < en; ++q) s += B.perm[q] < (unsigned)i ? 1 : 0;
    }
    D.id[s] = i;
    D.slot_of[i] = s;
    const int ty = S.type[i];
    D.type[s] = ty;
    D.itype[s] = S.itype[i];
    D.blabel[s] = i < P.n_host ? S.blabel[i] : 0;
    const double2 x = S.pos[i];
    D.pos0[s] = x;
    if (sizeof(R) == 4) D.xh0[s] = make_float2((float)x.x, (float)x.y);
    const double2 v = S.vel[i];
    const double rho = S.rho[i], m = S.mass[i], sm = S.smass[i];
    D.vel0[s] = v;
    D.rho0[s] = rho;
    D.mass[s] = m;
    D.smass[s] = sm;
    double dr = 0.0;
    double2 a = make_double2(0.0, 0.0), g = a;
    if (i < P.n_host) { dr = (double)(R)S.r_drho[i]; a = S.r_acc[i]; g = S.r_avg[i]; }
    a = make_double2((double)(R)a.x, (double)(R)a.y);
    g = make_double2((double)(R)g.x, (double)(R)g.y);
    if (G.mode == STAGE_MID) {
        // the step's first stage with the carried rates, on the values just read
        // (c_* are next written by the step's end)
        double2 xn = x;
        double u = v.x, w = v.y, r = rho;
        if (integrated(P, ty)) {
            stage_update<R>(D, s, G.stage, G.dt, x, v, rho, dr, a.x, a.y, g.x, g.y, xn.x, xn.y, u, w, r);
            check_skin(P, x, xn.x, xn.y, G.status);
        }
        store_records<R>(P, D, s, xn, u, w, r, m, sm, false);
    } else {
        store_records<R>(P, D, s, x, v.x, v.y, rho, m, sm, false);
    }
    if (G.mode != STAGE_MID || !integrated(P, ty)) {
        D.c_drho[s] = (R)dr;
        D.c_acc[s] = mk2<R>((R)a.x, (R)a.y);
        D.c_avg[s] = mk2<R>((R)g.x, (R)g.y);
    }
}

// sorted master state -> id order (host particles only; images are dropped)
template <typename R>
__global__ void k_unsort(Params P, Staging S, Sorted<R> D) {
    pdl_begin();
    stamp_phase(P.stamp);
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P.n_tot) return;
    int i = D.id[s];
    if (i >= P.n_host) return;
    S.pos[i] = D.pos0[s];
    S.vel[i] = D.vel0[s];
    S.rho[i] = D.rho0[s];
    S.mass[i] = D.mass[s];
    S.smass[i] = D.smass[s];
    S.type[i] = D.type[s];
    S.itype[i] = D.itype[s];
    S.r_drho[i] = (double)D.c_drho[s];
    S.r_acc[i] = make_double2((double)D.c_acc[s].x, (double)D.c_acc[s].y);
    S.r_avg[i] = make_double2((double)D.c_avg[s].x, (double)D.c_avg[s].y);
}

// Pair-rule of find_particle_pair (TGV :76, MS :73-75).
__device__ __forceinline__ bool pair_allowed(int rule, int ti, int tj) {
    if (rule == SPH_PAIRS_ONE_FLUID) return ti == SPH_TYPE_WATER || tj == SPH_TYPE_WATER;
    if (ti == -2 && tj == -2) return false;
    if (ti == -3 && tj == -3) return false;
    if (ti == -201 && tj == -201) return false;
    return true;
}

// Whether pair_allowed can refuse a pair of a particle of type ti: with the
// one-fluid rule not for water, with the other rule only for the boundary types.
// Where it cannot, no candidate's type is read: sort + lists 189 -> 172 us per step
// for the square at D/100, 35 -> 30 us at D/30.
__device__ __forceinline__ bool pair_may_fail(int rule, int ti) {
    return rule == SPH_PAIRS_ONE_FLUID ? ti != SPH_TYPE_WATER : ti == -2 || ti == -3 || ti == -201;
}

// Cell column (row) of coordinate v, for a scan of the columns c - 1 .. c + 1 of n.  A
// particle off the grid (not binned, reported as ST_DOMAIN) still comes here, and a
// coordinate of 1e300 or an infinity saturates the conversion to int, so that c + 1
// would overflow: clamped to [-2, n + 1], where the scan meets no column.
__device__ __forceinline__ int scan_cell(double v, double lo, double cs, int n) {
    return min(max(__double2int_rd((v - lo) / cs), -2), n + 1);
}

// --- 5. neighbour lists ----------------------------------------------------
// Every particle b != a in the 3x3 cells with |x_a - x_b|^2 <= (support*(1+skin))^2
// and an allowed type pair.  The exact support test is repeated at every RHS on
// the current positions, so the list only has to be a superset of the pairs of
// the whole step; every stage checks the displacement bound that guarantees it
// (check_skin).
// The first kListStage entries of each list are staged in shared memory
// ([entry][thread], conflict-free) and written out row by row after the scan, so
// the stores of a warp are coalesced; longer lists write the rest directly.
constexpr int kListStage = 32;
// ONE: the one-fluid rule, known to the compiler (the square's rule in the same code
// cost the Taylor-Green lists 3 %: 748 -> 769 us per step at 2048^2, 737 this way).
template <typename R, bool ONE>
__global__ void __launch_bounds__(128) k_build_lists(Params P, Sorted<R> D, unsigned* status) {
    pdl_begin();
    __shared__ unsigned stage[kListStage][128];
    const int tid = threadIdx.x;
    int a = blockIdx.x * blockDim.x + tid;
    if (a >= P.n_tot) return;
    int ta = D.type[a];
    int cnt = 0;
    // one list entry: staged, or (past the stage) straight to global memory
    auto put = [&](int b, unsigned lower) {
        const unsigned v = (unsigned)b | lower;
        if (cnt < kListStage) stage[cnt][tid] = v;
        else if (cnt < P.max_nbr) D.nbr[(size_t)cnt * P.nbr_stride + a] = v;
        ++cnt;
    };
    // the mixed path tests the positions rounded to FP32 against the widened radius
    // r2_list32 (a superset of the FP64 list, see derive_params)
    constexpr bool F32 = sizeof(R) == 4;
    const float2* xh = D.xh0;
    if (ta != SPH_TYPE_ILL && ta != 0) {
        double2 xa = D.pos0[a];
        const float2 xa_h = F32 ? xh[a] : make_float2(0.f, 0.f);
        int ida = D.id[a];
        const int cx = scan_cell(xa.x, P.gx0, P.cs, P.gnx), cy = scan_cell(xa.y, P.gy0, P.cs, P.gny);
        int x0 = max(cx - 1, 0), x1 = min(cx + 1, P.gnx - 1);
        const int rule = ONE ? (int)SPH_PAIRS_ONE_FLUID : P.pair_rule;
        const bool check_type = pair_may_fail(rule, ta);
        for (int gy = max(cy - 1, 0); gy <= min(cy + 1, P.gny - 1); ++gy) {
            // the cells x0..x1 of a row are consecutive keys, so their particles
            // form one contiguous range of the sorted order
            const int row = gy * P.gnx;
            int b0 = -1, b1 = -1;
            for (int gx = x0; gx <= x1; ++gx) {
                const int st = D.cell_start[row + gx];
                if (st < 0) continue;
                if (b0 < 0) b0 = st;
                b1 = D.cell_end[row + gx];
            }
            // candidates four at a time: their loads are issued together, then
            // tested in order (the list is the same as a one-by-one scan)
            int b = b0;
            for (; b + 4 <= b1; b += 4) {
                double2 xb[4];
                float2 xbh[4];
                int tb[4], ib[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (F32) xbh[k] = load(&xh[b + k]);
                    else xb[k] = load(&D.pos0[b + k]);
                    ib[k] = load(&D.id[b + k]);
                    tb[k] = check_type ? load(&D.type[b + k]) : 0;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (b + k == a) continue;
                    if (check_type && !pair_allowed(rule, ta, tb[k])) continue;
                    if (F32) {
                        const float dx = xa_h.x - xbh[k].x, dy = xa_h.y - xbh[k].y;
                        if (dx * dx + dy * dy > P.r2_list32) continue;
                    } else {
                        const double dx = xa.x - xb[k].x, dy = xa.y - xb[k].y;
                        if (dx * dx + dy * dy > P.r2_list) continue;
                    }
                    put(b + k, ida < ib[k] ? 0x80000000u : 0u);
                }
            }
            for (; b < b1; ++b) {
                if (b == a) continue;
                if (check_type && !pair_allowed(rule, ta, D.type[b])) continue;
                if (F32) {
                    const float2 xbh = xh[b];
                    const float dx = xa_h.x - xbh.x, dy = xa_h.y - xbh.y;
                    if (dx * dx + dy * dy > P.r2_list32) continue;
                } else {
                    const double2 xb = D.pos0[b];
                    const double dx = xa.x - xb.x, dy = xa.y - xb.y;
                    if (dx * dx + dy * dy > P.r2_list) continue;
                }
                put(b, ida < D.id[b] ? 0x80000000u : 0u);
            }
        }
        if (cnt > P.max_nbr) { atomicOr(status, ST_NBR_OVERFLOW); cnt = P.max_nbr; }
    }
    const int ns = min(cnt, kListStage);
    for (int e = 0; e < ns; ++e) D.nbr[(size_t)e * P.nbr_stride + a] = stage[e][tid];
    D.nnbr[a] = cnt;
}

// The same lists with L lanes per particle: the lanes split the candidates of the
// three rows, taken as one range, and a ballot gives each accepted one its place,
// so the entries come in the same order.  For particle counts that leave most of
// the GPU idle with a thread per particle, whose ~74 (Wendland C2) to ~140
// (Gaussian) candidates are then a chain of dependent loads.
template <typename R, int L>
__global__ void __launch_bounds__(128) k_build_lists_lanes(Params P, Sorted<R> D, unsigned* status) {
    pdl_begin();
    constexpr bool F32 = sizeof(R) == 4;
    const Lanes<L> ln;
    const int g = Lanes<L>::particle();
    const bool live = g < P.n_tot;
    const int a = live ? g : P.n_tot - 1;
    const int ta = D.type[a];
    const double2 xa = D.pos0[a];
    const float2 xa_h = F32 ? D.xh0[a] : make_float2(0.f, 0.f);
    const int ida = D.id[a];
    int lo[3] = {0, 0, 0}, len[3] = {0, 0, 0};
    if (live && ta != SPH_TYPE_ILL && ta != 0) {
        const int cx = scan_cell(xa.x, P.gx0, P.cs, P.gnx), cy = scan_cell(xa.y, P.gy0, P.cs, P.gny);
        const int x0 = max(cx - 1, 0), x1 = min(cx + 1, P.gnx - 1);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int gy = cy - 1 + r;
            if (gy < 0 || gy > P.gny - 1) continue;
            int b0 = -1, b1 = -1;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int gx = x0 + k;
                if (gx > x1) continue;
                const int st = D.cell_start[gy * P.gnx + gx], en = D.cell_end[gy * P.gnx + gx];
                if (st < 0) continue;
                if (b0 < 0) b0 = st;
                b1 = en;
            }
            lo[r] = b0;
            len[r] = b1 - b0;
        }
    }
    const bool check_type = pair_may_fail(P.pair_rule, ta);
    const int l01 = len[0] + len[1], total = l01 + len[2];
    const int most = __reduce_max_sync(0xffffffffu, total);
    int cnt = 0;
#pragma unroll 2
    for (int t0 = 0; t0 < most; t0 += L) {
        const int t = t0 + ln.lane;
        bool in = false;
        unsigned v = 0u;
        if (t < total) {
            const int b = t < len[0] ? lo[0] + t : t < l01 ? lo[1] + (t - len[0]) : lo[2] + (t - l01);
            v = (unsigned)b | (ida < load(&D.id[b]) ? 0x80000000u : 0u);
            if (F32) {
                const float2 xb = load(&D.xh0[b]);
                const float dx = xa_h.x - xb.x, dy = xa_h.y - xb.y;
                in = !(dx * dx + dy * dy > P.r2_list32);
            } else {
                const double2 xb = load(&D.pos0[b]);
                const double dx = xa.x - xb.x, dy = xa.y - xb.y;
                in = !(dx * dx + dy * dy > P.r2_list);
            }
            in = in && b != a && (!check_type || pair_allowed(P.pair_rule, ta, D.type[b]));
        }
        const unsigned hit = __ballot_sync(0xffffffffu, in) & ln.group;
        const int e = cnt + __popc(hit & ln.below);
        if (in && e < P.max_nbr) D.nbr[(size_t)e * P.nbr_stride + a] = v;
        cnt += __popc(hit);
    }
    if (!live || ln.lane != 0) return;
    if (cnt > P.max_nbr) { atomicOr(status, ST_NBR_OVERFLOW); cnt = P.max_nbr; }
    D.nnbr[a] = cnt;
}

// Measured, sort + lists in us per step, thread per particle against 8 lanes
// (4, 16 and 32 within 3 us of it or slower): 36 -> 28 at 11,000 particles (100^2
// Taylor-Green with images), 40 -> 37 at 42,000, 59 -> 47 at 49,000 (square D/30,
// Gaussian), but 40 -> 43 at 68,000 and 72 -> 82 at 131,000: the GPU is full there.
constexpr int kListLanes = 8, kListLanesBelow = 60000;
template <typename R>
void launch_lists(const Params& P, const Sorted<R>& D, unsigned* status, cudaStream_t st) {
    if (P.n_tot < kListLanesBelow) {
        const long long t = (long long)P.n_tot * kListLanes;
        launch(k_build_lists_lanes<R, kListLanes>, (unsigned)((t + 127) / 128), 128, st, P, D, status);
    } else {
        launch(P.pair_rule == SPH_PAIRS_ONE_FLUID ? k_build_lists<R, true> : k_build_lists<R, false>,
               (P.n_tot + 127) / 128, 128, st, P, D, status);
    }
}

}  // namespace sph
