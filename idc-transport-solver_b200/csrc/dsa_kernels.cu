// Diffusion synthetic acceleration (DSA) for the Peierls-form GMRES: a 2-D cell-centred finite-volume
// diffusion operator on the cell-average moment and a fixed number of Jacobi-preconditioned conjugate
// gradient steps, all scalars on the device (no host round trip per step).
//
// The reference has DSA only in 1-D (a SIP-DG diffusion solve inside its PETSc Peierls solver,
// linear_solvers/RKDG/ImplicitSolver/PETScPeierlsSolver.cpp:27-376); this is a 2-D design.  The
// preconditioner M r = r + C^{-1} (sigma_s r_00) on the (0,0) moment, with
//     C u = -div(D grad u) + sigma_a u,   D = 1 / (3 sigma_t),   sigma_a = sigma_t - sigma_s,
// is the classic DSA correction: for the flat mode of an infinite medium, (I - P L^{-1} S)^{-1} =
// 1 + sigma_s / sigma_a exactly.  Faces use the harmonic mean of the two cells' D (uniform grid); a
// boundary face is a Marshak vacuum condition, flux = u_b / 2 with D (u - u_b) / (h/2) = u_b / 2.
// The right-hand side and all Jacobi-PCG steps run in one kernel, in the Chronopoulos-Gear form of CG with one
// global reduction per step: a thread-block cluster per problem up to kClusterCells cells, a cooperative kernel
// (every block resident) beyond.  Each block adds the partial sums in the same fixed order, so the step lengths
// are identical on every block and the result is bitwise reproducible.  The cooperative kernel's barrier waits are
// bounded: on expiry the device error word is set and every block leaves.  The cluster's barrier is the hardware's,
// whose blocks run together by construction and wait for nothing else.
#include "device_sync.cuh"
#include "idc_internal.hpp"

#include <vector>

namespace idc {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ double face_coef(double Da, double Db) { return 2.0 * Da * Db / (Da + Db); }

// Diagonal of C (for the Jacobi preconditioner).
__global__ void dsa_diag_kernel(int nx, int ny, double dx, double dy, const double *__restrict__ Dc,
                                const double *__restrict__ sa, double *__restrict__ dinv) {
    const int n = nx * ny;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int i = t / ny, j = t - (t / ny) * ny;
        const double D = Dc[t];
        const double ix2 = 1.0 / (dx * dx), iy2 = 1.0 / (dy * dy);
        double acc = sa[t];
        acc += (i > 0) ? face_coef(D, Dc[t - ny]) * ix2 : D / (2.0 * D + 0.25 * dx) / dx;
        acc += (i < nx - 1) ? face_coef(D, Dc[t + ny]) * ix2 : D / (2.0 * D + 0.25 * dx) / dx;
        acc += (j > 0) ? face_coef(D, Dc[t - 1]) * iy2 : D / (2.0 * D + 0.25 * dy) / dy;
        acc += (j < ny - 1) ? face_coef(D, Dc[t + 1]) * iy2 : D / (2.0 * D + 0.25 * dy) / dy;
        dinv[t] = 1.0 / acc;
    }
}

// D = 1/(3 sigma_t), sigma_a = sigma_t - sigma_s (clamped at 0) on interior cells, from the halo arrays.
__global__ void dsa_coef_kernel(int nx, int ny, const double *__restrict__ st, const double *__restrict__ ss,
                                double *__restrict__ Dc, double *__restrict__ sa) {
    const int n = nx * ny;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int i = t / ny, j = t - (t / ny) * ny;
        const size_t c = (size_t)(i + 1) * (ny + 2) + (j + 1);
        const double sigt = fmax(st[c], 1e-12);
        Dc[t] = 1.0 / (3.0 * sigt);
        sa[t] = fmax(st[c] - ss[c], 0.0);
    }
}


// out = v, out_00 += x (forward) or sigma_s x (transposed, ss non-null) on interior cells (phi layout).
// It also re-arms the PCG kernel's barrier counter (zero at the start of every launch).
__global__ void dsa_correct_kernel(int nx, int ny, int N, const double *v, const double *__restrict__ x,
                                   const double *__restrict__ ss, double *out, unsigned *count) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *count = 0u;
    const size_t total = (size_t)(nx + 2) * (ny + 2) * N;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const size_t c = t / N;
        const int k = (int)(t - c * N);
        const int i = (int)(c / (ny + 2)), j = (int)(c % (ny + 2));
        double val = v[t];
        if (k == 0 && i >= 1 && i <= nx && j >= 1 && j <= ny) {
            const double xc = x[(size_t)(i - 1) * ny + (j - 1)];
            val += ss ? ss[c] * xc : xc;
        }
        out[t] = val;
    }
}

inline int blocks_for(size_t n) {
    size_t b = (n + kThreads - 1) / kThreads;
    if (b > 148 * 4) b = 148 * 4;
    return (int)(b == 0 ? 1 : b);
}

constexpr int kPcgThreads = 512;
constexpr int kMaxPcgBlocks = 1024;   // partial sums per reduction (the grid is at most one block per SM)

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid barrier number e (0, 1, ...) of a cooperative launch on an arrival counter that is zero when the
// kernel starts: each block adds one, then waits until the counter reaches (e + 1) blocks.  Bounded: a block
// that waits longer than `limit` polls records kDevTimeout; a block that sees an error leaves.  Returns false
// (in every thread of the block) when the block must leave.
__device__ bool grid_barrier(unsigned *count, unsigned e, int *error, long long limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        __threadfence();
        atomicAdd(count, 1u);
        const unsigned target = (e + 1u) * gridDim.x;
        for (long long n = 0; (int)(ld_acquire_u32(count) - target) < 0; ++n) {
            if ((n & 63) == 63 && ld_relaxed(error) != kDevOk) {
                ok = 0;
                break;
            }
            if (n > limit) {
                atomicCAS(error, kDevOk, kDevTimeout);
                ok = 0;
                break;
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Fixed-order sums of per-thread values (a, b) into part[blockIdx.x] and part[gridDim.x + blockIdx.x].
__device__ __forceinline__ void block_partial2(double a, double b, double *part) {
    __shared__ double w[2][kPcgThreads / 32];
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_down_sync(kFullMask, a, off);
        b += __shfl_down_sync(kFullMask, b, off);
    }
    if ((threadIdx.x & 31) == 0) {
        w[0][threadIdx.x >> 5] = a;
        w[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double acc = w[threadIdx.x][0];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) acc += w[threadIdx.x][k];
        part[threadIdx.x * gridDim.x + blockIdx.x] = acc;
    }
}

// Sums of part[0 .. gridDim.x) and part[gridDim.x .. 2 gridDim.x) in one fixed order: the same values in
// every block.  The partial sums were written by other blocks before the barrier: read from L2.
__device__ __forceinline__ void grid_totals(const double *part, double &a, double &b) {
    __shared__ double s_tot[2];
    if (threadIdx.x < 64) {
        const int h = threadIdx.x >> 5, l = threadIdx.x & 31;
        double v = 0.0;
        for (int k = l; k < (int)gridDim.x; k += 32) v += __ldcg(part + h * gridDim.x + k);
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(kFullMask, v, off);
        if (l == 0) s_tot[h] = v;
    }
    __syncthreads();
    a = s_tot[0];
    b = s_tot[1];
    __syncthreads();
}

struct PcgArgs {
    int nx, ny, N, scale, cg_steps;
    double dx, dy;
    const double *ss, *v, *Dc, *sa, *dinv;
    double *x, *p, *r[2], *u[2], *w[2], *s[2], *part;
    unsigned *count;
    int *error;
    long long spin_limit;
};

// y = (C u)(t) for cell t = (i, j) given u at t (ut) and at any cell (uv).
template <typename U>
__device__ __forceinline__ double apply_c(const PcgArgs &a, int t, int i, int j, double ut, U uv) {
    const int nx = a.nx, ny = a.ny;
    const double ix2 = 1.0 / (a.dx * a.dx), iy2 = 1.0 / (a.dy * a.dy);
    const double D = a.Dc[t];
    double acc = a.sa[t] * ut;
    acc += (i > 0) ? face_coef(D, a.Dc[t - ny]) * ix2 * (ut - uv(t - ny)) : ut * D / (2.0 * D + 0.25 * a.dx) / a.dx;
    acc += (i < nx - 1) ? face_coef(D, a.Dc[t + ny]) * ix2 * (ut - uv(t + ny)) : ut * D / (2.0 * D + 0.25 * a.dx) / a.dx;
    acc += (j > 0) ? face_coef(D, a.Dc[t - 1]) * iy2 * (ut - uv(t - 1)) : ut * D / (2.0 * D + 0.25 * a.dy) / a.dy;
    acc += (j < ny - 1) ? face_coef(D, a.Dc[t + 1]) * iy2 * (ut - uv(t + 1)) : ut * D / (2.0 * D + 0.25 * a.dy) / a.dy;
    return acc;
}

// x = C^{-1} f by cg_steps Jacobi-preconditioned CG steps from x = 0, f = sigma_s v_00 (scale) or v_00, in
// the Chronopoulos-Gear form (one global reduction per step; the same iterates as standard PCG in exact
// arithmetic).  With u = M r and w = C u:
//   gamma = r.u, delta = w.u, beta = gamma / gamma_old (0 at the first step),
//   alpha = gamma / (delta - beta gamma / alpha_old),
//   p = u + beta p, s = w + beta s, x += alpha p, r -= alpha s, u = M r, w = C u.
// r, u, w, s alternate between two buffers: a block forms its neighbours' new u from their old r, w, s
// (complete at the barrier, never overwritten in the same step) instead of waiting for their owners, so a
// step has one grid barrier.
__global__ void __launch_bounds__(kPcgThreads) dsa_pcg_kernel(const PcgArgs a) {
    const int nx = a.nx, ny = a.ny, n = nx * ny;
    const int stride = gridDim.x * blockDim.x;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    (void)nx;
    auto rhs = [&](int t) {
        const int i = t / ny, j = t - (t / ny) * ny;
        const size_t c = (size_t)(i + 1) * (ny + 2) + (j + 1);
        return a.scale ? a.ss[c] * a.v[c * a.N] : a.v[c * a.N];
    };
    // r = f, u = M f, w = C u, x = p = s = 0; partial r.u and w.u
    double g = 0.0, d = 0.0;
    for (int t = t0; t < n; t += stride) {
        const int i = t / ny, j = t - (t / ny) * ny;
        const double f = rhs(t), ut = a.dinv[t] * f;
        const double wt = apply_c(a, t, i, j, ut, [&](int c) { return a.dinv[c] * rhs(c); });
        a.r[0][t] = f;
        a.u[0][t] = ut;
        a.w[0][t] = wt;
        a.s[0][t] = 0.0;
        a.x[t] = 0.0;
        a.p[t] = 0.0;
        g = fma(f, ut, g);
        d = fma(wt, ut, d);
    }
    block_partial2(g, d, a.part);
    unsigned e = 0;
    if (!grid_barrier(a.count, e++, a.error, a.spin_limit)) return;

    double gamma_old = 0.0, alpha_old = 1.0;
    for (int k = 0; k < a.cg_steps; ++k) {
        const int c0 = k & 1, c1 = c0 ^ 1;
        const double *rc = a.r[c0], *wc = a.w[c0], *sc = a.s[c0], *uc = a.u[c0];
        double *rn = a.r[c1], *wn = a.w[c1], *sn = a.s[c1], *un = a.u[c1];
        double gamma, delta;
        grid_totals(a.part + (size_t)2 * kMaxPcgBlocks * c0, gamma, delta);   // partials alternate halves
        const double beta = k == 0 ? 0.0 : (gamma_old != 0.0 ? gamma / gamma_old : 0.0);
        const double den = delta - (k == 0 ? 0.0 : beta * gamma / alpha_old);
        const double alpha = den != 0.0 ? gamma / den : 0.0;
        gamma_old = gamma;
        alpha_old = alpha != 0.0 ? alpha : 1.0;
        const bool last = k + 1 == a.cg_steps;
        // the new u of any cell from its old r, w, s (read from L2: other blocks wrote them)
        auto unew = [&](int c) {
            const double sv = fma(beta, __ldcg(sc + c), __ldcg(wc + c));
            return a.dinv[c] * fma(-alpha, sv, __ldcg(rc + c));
        };
        g = 0.0;
        d = 0.0;
        for (int t = t0; t < n; t += stride) {
            const double pt = fma(beta, a.p[t], uc[t]);
            const double st = fma(beta, sc[t], wc[t]);
            a.p[t] = pt;
            a.x[t] = fma(alpha, pt, a.x[t]);
            if (last) continue;   // x is final; the kernel's end orders it before the correction
            const double rt = fma(-alpha, st, rc[t]);
            const double ut = a.dinv[t] * rt;
            const int i = t / ny, j = t - (t / ny) * ny;
            const double wt = apply_c(a, t, i, j, ut, unew);
            sn[t] = st;
            rn[t] = rt;
            un[t] = ut;
            wn[t] = wt;
            g = fma(rt, ut, g);
            d = fma(wt, ut, d);
        }
        if (last) break;
        block_partial2(g, d, a.part + (size_t)2 * kMaxPcgBlocks * (c1));
        if (!grid_barrier(a.count, e++, a.error, a.spin_limit)) return;
    }
}

// Workspace: Dc, sa, dinv, x, p, r[2], u[2], w[2], s[2] (n each), partial sums, the barrier counter.
struct DsaWs {
    double *Dc, *sa, *dinv, *x, *p, *r[2], *u[2], *w[2], *s[2], *part;
    unsigned *count;
    DsaWs(double *ws, int n) {
        double *q = ws;
        auto take = [&]() { double *o = q; q += n; return o; };
        Dc = take(), sa = take(), dinv = take(), x = take(), p = take();
        for (int b = 0; b < 2; ++b) r[b] = take(), u[b] = take(), w[b] = take(), s[b] = take();
        part = q;
        count = reinterpret_cast<unsigned *>(part + 4 * kMaxPcgBlocks);
    }
};

// ---- the same PCG in one thread-block cluster -----------------------------------------------------------------
//
// Grids of up to kClusterCells cells: a cluster of up to 16 blocks holds a whole problem in registers and shared
// memory (thread l of a block owns K consecutive cells), reads its neighbours' u from the owners' shared memory, and
// meets in the cluster barrier unit instead of at a counter in L2.  A step is bound by its two cluster barriers and the
// latency of the reductions, not by bandwidth; the cooperative kernel's grid barriers and L2 round trips took 4.6 us a
// step whatever the size.  Every problem of a batch is a cluster of the same launch.  Each warp's partial sums go to
// every block and are added in one fixed order: bitwise reproducible, the same step lengths everywhere.
constexpr int kClusterThreads = 512, kClusterWarps = kClusterThreads / 32, kMaxClusterBlocks = 16, kMaxClusterK = 8;
constexpr int kClusterCells = kClusterThreads * kMaxClusterBlocks * kMaxClusterK;
constexpr int kMaxJobs = 24;

struct PcgJob {
    int nx, ny, N, scale;
    double dx, dy;
    const double *ss, *v, *Dc, *sa, *dinv;
    double *x;
};
struct PcgJobs {
    int cg_steps;
    PcgJob job[kMaxJobs];
};
static_assert(sizeof(PcgJobs) <= 4000, "kernel parameters");

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_blocks() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(const void *p, unsigned rank) {   // the same place in block `rank`
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ double ld_cluster(uint32_t p) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_cluster2(uint32_t p, double a, double b) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(p), "d"(a), "d"(b) : "memory");
}

// Shared memory: u, the face coefficients to the next cell in x, the last in x and the next in y (zero at the domain's
// edges), sigma_a with the edge terms, 1 / diagonal, [K][threads] each; the coefficient below a thread's first cell;
// the partial sums of every warp of the cluster.
template <int K>
constexpr size_t cluster_smem_bytes() {
    return sizeof(double) * ((size_t)6 * K * kClusterThreads + kClusterThreads + 2 * kMaxClusterBlocks * kClusterWarps);
}

template <int K>
__global__ void __launch_bounds__(kClusterThreads, 1) dsa_pcg_cluster_kernel(const __grid_constant__ PcgJobs jobs) {
    extern __shared__ __align__(16) unsigned char cluster_smem[];
    constexpr int T = kClusterThreads, KT = K * T;
    double *su = reinterpret_cast<double *>(cluster_smem);
    double *cxp = su + KT, *cxm = cxp + KT, *cyp = cxm + KT, *sap = cyp + KT, *sdi = sap + KT, *cy0 = sdi + KT;
    double *part = cy0 + T;   // [block * warps + warp][2]
    const int rank = (int)cluster_rank(), C = (int)cluster_blocks();
    const PcgJob &a = jobs.job[blockIdx.x / C];
    const int nx = a.nx, ny = a.ny, n = nx * ny, l = threadIdx.x, warp = l >> 5, lane = l & 31;
    const int first = rank * KT + l * K;   // this thread's cells: first .. first + K - 1
    // where cell c's u is
    auto u_addr = [&](int c) {
        const int owner = c / KT, in = c - owner * KT;
        return cluster_addr(su + (in % K) * T + in / K, (unsigned)owner);
    };
    double r[K], s[K], p[K], x[K], w[K];
    uint32_t up[K], um[K];   // u of the next and the last cell in x
    uint32_t ubelow = u_addr(0), uabove = ubelow;   // u below the first and above the last cell in y
    const double ix2 = 1.0 / (a.dx * a.dx), iy2 = 1.0 / (a.dy * a.dy);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int t = first + k, at = k * T + l;
        r[k] = s[k] = p[k] = x[k] = w[k] = 0.0;
        up[k] = um[k] = cluster_addr(su + at, (unsigned)rank);
        double cp = 0.0, cm = 0.0, ca = 0.0, cb = 0.0, sa = 0.0, di = 0.0;
        if (t < n) {
            const int i = t / ny, j = t - i * ny;
            const double D = a.Dc[t];
            const double ex = D / (2.0 * D + 0.25 * a.dx) / a.dx, ey = D / (2.0 * D + 0.25 * a.dy) / a.dy;
            sa = a.sa[t];
            di = a.dinv[t];
            if (i > 0) cm = face_coef(D, a.Dc[t - ny]) * ix2, um[k] = u_addr(t - ny);
            else sa += ex;
            if (i < nx - 1) cp = face_coef(D, a.Dc[t + ny]) * ix2, up[k] = u_addr(t + ny);
            else sa += ex;
            if (j > 0) cb = face_coef(D, a.Dc[t - 1]) * iy2;
            else sa += ey;
            if (j < ny - 1) ca = face_coef(D, a.Dc[t + 1]) * iy2;
            else sa += ey;
            if (k == 0 && t > 0) ubelow = u_addr(t - 1);
            if (k == K - 1 && t + 1 < n) uabove = u_addr(t + 1);
            const size_t c = (size_t)(i + 1) * (ny + 2) + (j + 1);
            r[k] = a.scale ? a.ss[c] * a.v[c * a.N] : a.v[c * a.N];
        }
        cxp[at] = cp;
        cxm[at] = cm;
        cyp[at] = ca;
        sap[at] = sa;
        sdi[at] = di;
        if (k == 0) cy0[l] = cb;
        su[at] = di * r[k];
    }
    double gamma_old = 0.0, alpha_old = 1.0;
    for (int step = 0;; ++step) {
        // w = C u, the partial sums of r.u and w.u
        cluster_sync();   // every u is there
        double g = 0.0, d = 0.0;
        {
            double below = ld_cluster(ubelow), cb = cy0[l], ut = su[l];
            const double above = ld_cluster(uabove);
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int at = k * T + l;
                const double next = k + 1 < K ? su[at + T] : above, ca = cyp[at];
                double acc = sap[at] * ut;
                acc = fma(cxm[at], ut - ld_cluster(um[k]), acc);
                acc = fma(cxp[at], ut - ld_cluster(up[k]), acc);
                acc = fma(cb, ut - below, acc);
                acc = fma(ca, ut - next, acc);
                w[k] = acc;
                g = fma(r[k], ut, g);
                d = fma(acc, ut, d);
                below = ut;
                ut = next;
                cb = ca;
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            g += __shfl_xor_sync(kFullMask, g, off);
            d += __shfl_xor_sync(kFullMask, d, off);
        }
        if (lane < C) st_cluster2(cluster_addr(part + 2 * (rank * kClusterWarps + warp), (unsigned)lane), g, d);
        cluster_sync();   // every partial sum is there, every u has been read
        double gamma = 0.0, delta = 0.0;
        for (int q = lane; q < C * kClusterWarps; q += 32) {
            const double2 v = reinterpret_cast<const double2 *>(part)[q];
            gamma += v.x;
            delta += v.y;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            gamma += __shfl_xor_sync(kFullMask, gamma, off);
            delta += __shfl_xor_sync(kFullMask, delta, off);
        }
        const double beta = step == 0 ? 0.0 : (gamma_old != 0.0 ? gamma / gamma_old : 0.0);
        const double den = delta - (step == 0 ? 0.0 : beta * gamma / alpha_old);
        const double alpha = den != 0.0 ? gamma / den : 0.0;
        gamma_old = gamma;
        alpha_old = alpha != 0.0 ? alpha : 1.0;
        const bool last = step + 1 >= jobs.cg_steps;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int at = k * T + l;
            p[k] = fma(beta, p[k], su[at]);
            s[k] = fma(beta, s[k], w[k]);
            x[k] = fma(alpha, p[k], x[k]);
            r[k] = fma(-alpha, s[k], r[k]);
            su[at] = sdi[at] * r[k];
        }
        if (last) break;
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (first + k < n) a.x[first + k] = x[k];
}

// out = v, out_00 += x (forward) or sigma_s x (transposed, ss non-null) of several problems, as dsa_correct_kernel.
struct CorrectJob {
    int nx, ny, N;
    const double *v, *x, *ss;
    double *out;
};
struct CorrectJobs {
    CorrectJob job[kMaxJobs];
};
__global__ void dsa_correct_jobs_kernel(const __grid_constant__ CorrectJobs jobs) {
    const CorrectJob &a = jobs.job[blockIdx.y];
    const int cells = (a.nx + 2) * (a.ny + 2);
    const size_t total = (size_t)cells * a.N;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(t / a.N), k = (int)(t - (size_t)c * a.N);
        const int i = c / (a.ny + 2), j = c - i * (a.ny + 2);
        double val = a.v[t];
        if (k == 0 && i >= 1 && i <= a.nx && j >= 1 && j <= a.ny) {
            const double xc = a.x[(size_t)(i - 1) * a.ny + (j - 1)];
            val += a.ss ? a.ss[c] * xc : xc;
        }
        a.out[t] = val;
    }
}

template <int K>
cudaError_t launch_cluster(const PcgJobs &jobs, int count, int blocks, cudaStream_t s) {
    auto kern = dsa_pcg_cluster_kernel<K>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cluster_smem_bytes<K>());
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)blocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(blocks * count));
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = cluster_smem_bytes<K>();
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, jobs);
}

// Blocks per cluster and cells per thread for n cells: one cell per thread while the cluster has room for them (the
// steps are latency bound), then 2, 4, 8.
void cluster_shape(int n, int *blocks, int *k) {
    *k = 1;
    while (n > kClusterThreads * kMaxClusterBlocks * *k) *k *= 2;
    *blocks = 1;
    while (n > kClusterThreads * *k * *blocks) *blocks *= 2;
}

}  // namespace

size_t dsa_workspace_doubles(int nx, int ny) { return (size_t)nx * ny * 13 + 4 * kMaxPcgBlocks + 2; }

// Coefficients and the Jacobi diagonal from the cross sections; the barrier words start at zero (also after
// a barrier that gave up).
cudaError_t dsa_setup(const GridDims &g, const double *sigma_t, const double *sigma_s, double *ws, cudaStream_t s) {
    const int n = g.nx * g.ny;
    const DsaWs w(ws, n);
    dsa_coef_kernel<<<blocks_for(n), kThreads, 0, s>>>(g.nx, g.ny, sigma_t, sigma_s, w.Dc, w.sa);
    dsa_diag_kernel<<<blocks_for(n), kThreads, 0, s>>>(g.nx, g.ny, g.dx, g.dy, w.Dc, w.sa, w.dinv);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemsetAsync(w.count, 0, sizeof(unsigned), s);
    return e;
}

static cudaError_t dsa_precondition_grid(const GridDims &g, const double *sigma_s, const double *v, double *out,
                                         int cg_steps, double *ws, bool transpose, int num_sms, int *error,
                                         long long spin_limit, cudaStream_t s) {
    const int n = g.nx * g.ny;
    const DsaWs w(ws, n);
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dsa_pcg_kernel, kPcgThreads, 0);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorCooperativeLaunchTooLarge;
    int blocks = (n + kPcgThreads - 1) / kPcgThreads;
    blocks = blocks < 1 ? 1 : blocks;
    blocks = blocks < num_sms ? blocks : num_sms;   // one block per SM at most: cheap barriers
    blocks = blocks < kMaxPcgBlocks ? blocks : kMaxPcgBlocks;
    PcgArgs a{};
    a.nx = g.nx;
    a.ny = g.ny;
    a.N = g.P * g.P;
    a.scale = transpose ? 0 : 1;
    a.cg_steps = cg_steps;
    a.dx = g.dx;
    a.dy = g.dy;
    a.ss = sigma_s;
    a.v = v;
    a.Dc = w.Dc;
    a.sa = w.sa;
    a.dinv = w.dinv;
    a.x = w.x;
    a.p = w.p;
    for (int b = 0; b < 2; ++b) a.r[b] = w.r[b], a.u[b] = w.u[b], a.w[b] = w.w[b], a.s[b] = w.s[b];
    a.part = w.part;
    a.count = w.count;
    a.error = error;
    a.spin_limit = spin_limit;
    void *args[] = {&a};
    e = cudaLaunchCooperativeKernel((const void *)dsa_pcg_kernel, dim3(blocks), dim3(kPcgThreads), args, 0, s);
    if (e != cudaSuccess) return e;
    const size_t tot = (size_t)(g.nx + 2) * (g.ny + 2) * g.P * g.P;
    dsa_correct_kernel<<<blocks_for(tot), kThreads, 0, s>>>(g.nx, g.ny, g.P * g.P, v, w.x,
                                                            transpose ? sigma_s : nullptr, out, w.count);
    return cudaGetLastError();
}

// `count` problems with one number of CG steps: those of one cluster shape share a launch; larger grids run on the
// cooperative kernel one by one.
cudaError_t dsa_precondition(const DsaJob *jobs, int count, int cg_steps, bool transpose, int num_sms, cudaStream_t s) {
    auto small = [](const DsaJob &j) { return (int64_t)j.g.nx * j.g.ny <= kClusterCells; };
    std::vector<char> done((size_t)count, 0);
    for (int f = 0; f < count; ++f) {
        if (done[f]) continue;
        if (!small(jobs[f])) {
            const DsaJob &j = jobs[f];
            cudaError_t e = dsa_precondition_grid(j.g, j.sigma_s, j.v, j.out, cg_steps, j.ws, transpose, num_sms, j.error,
                                                  j.spin_limit, s);
            if (e != cudaSuccess) return e;
            continue;
        }
        int blocks = 0, k = 0, m = 0;
        cluster_shape(jobs[f].g.nx * jobs[f].g.ny, &blocks, &k);
        PcgJobs pj{};
        CorrectJobs cj{};
        size_t most = 0;
        for (int q = f; q < count && m < kMaxJobs; ++q) {
            const DsaJob &j = jobs[q];
            int b = 0, kk = 0;
            if (done[q] || !small(j)) continue;
            cluster_shape(j.g.nx * j.g.ny, &b, &kk);
            if (b != blocks || kk != k) continue;
            done[q] = 1;
            const DsaWs w(j.ws, j.g.nx * j.g.ny);
            const int N = j.g.P * j.g.P;
            pj.job[m] = PcgJob{j.g.nx, j.g.ny, N, transpose ? 0 : 1, j.g.dx, j.g.dy, j.sigma_s, j.v, w.Dc, w.sa, w.dinv, w.x};
            cj.job[m] = CorrectJob{j.g.nx, j.g.ny, N, j.v, w.x, transpose ? j.sigma_s : nullptr, j.out};
            const size_t tot = (size_t)(j.g.nx + 2) * (j.g.ny + 2) * N;
            most = most > tot ? most : tot;
            ++m;
        }
        pj.cg_steps = cg_steps;
        cudaError_t e = k == 1   ? launch_cluster<1>(pj, m, blocks, s)
                        : k == 2 ? launch_cluster<2>(pj, m, blocks, s)
                        : k == 4 ? launch_cluster<4>(pj, m, blocks, s)
                                 : launch_cluster<8>(pj, m, blocks, s);
        if (e != cudaSuccess) {   // no such cluster on this device: one by one on the cooperative kernel
            (void)cudaGetLastError();
            for (int q = 0; q < count; ++q) {
                const DsaJob &j = jobs[q];
                int b = 0, kk = 0;
                if (!small(j)) continue;
                cluster_shape(j.g.nx * j.g.ny, &b, &kk);
                if (b != blocks || kk != k) continue;
                done[q] = 1;
                e = dsa_precondition_grid(j.g, j.sigma_s, j.v, j.out, cg_steps, j.ws, transpose, num_sms, j.error,
                                          j.spin_limit, s);
                if (e != cudaSuccess) return e;
            }
            continue;
        }
        dsa_correct_jobs_kernel<<<dim3((unsigned)blocks_for(most), (unsigned)m), kThreads, 0, s>>>(cj);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace idc

