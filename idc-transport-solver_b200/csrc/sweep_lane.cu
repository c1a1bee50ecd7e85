// Lane-pipelined sweep: host-side dispatch over degree, row-segment width, direction and second source,
// and the occupancy query.  The kernel is in sweep_lane_impl.cuh.
#include "sweep_lane_impl.cuh"

#include <cmath>

namespace idc {

namespace {

template <int P, bool ADJ, bool SRC2, bool PHI = false, typename TC = double>
cudaError_t launch_p(const SweepArgs &args, int grid, cudaStream_t stream) {
    switch (args.seg) {
        case 4: return lane::launch<P, 4, ADJ, SRC2, PHI, TC>(args, grid, stream);
        case 8: return lane::launch<P, 8, ADJ, SRC2, PHI, TC>(args, grid, stream);
        case 16: return lane::launch<P, 16, ADJ, SRC2, PHI, TC>(args, grid, stream);
        default: return cudaErrorInvalidValue;
    }
}

template <int P>
cudaError_t launch_dir(const SweepArgs &args, int grid, cudaStream_t stream, bool fp32) {
    if (fp32) {   // FP32 arithmetic: forward sweeps, with or without psi
        if (args.adjoint || args.src2) return cudaErrorInvalidValue;
        if (args.modal_src) {
            if (args.src || args.out || !args.phi_part) return cudaErrorInvalidValue;
            return launch_p<P, false, false, true, float>(args, grid, stream);
        }
        return launch_p<P, false, false, false, float>(args, grid, stream);
    }
    if (args.modal_src) {   // moments-only sweep
        if (args.src2 || args.src || args.out || !args.phi_part) return cudaErrorInvalidValue;
        return args.adjoint ? launch_p<P, true, false, true>(args, grid, stream)
                            : launch_p<P, false, false, true>(args, grid, stream);
    }
    if (args.adjoint) return args.src2 ? cudaErrorInvalidValue : launch_p<P, true, false>(args, grid, stream);
    return args.src2 ? launch_p<P, false, true>(args, grid, stream) : launch_p<P, false, false>(args, grid, stream);
}

// Packed modal source (of the forward or the transposed operator) and sigma_t of every interior (cell, quadrant) for
// the moments-only sweep (see idc_internal.hpp): sigma_s phi / (4 pi) scaled (rounded as scatter_moments_kernel rounds
// it), or phi itself without sigma_s.
template <int P, bool ADJ>
__device__ __forceinline__ void modal_sources(int nx, int ny, const double *__restrict__ sigma_t,
                                              const double *__restrict__ sigma_s, const double *__restrict__ phi,
                                              double scale, double *__restrict__ out) {
    constexpr int N = P * P, RD = cell_record_doubles(P);
    const size_t total = (size_t)nx * ny * 4;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(t % 4);
        const size_t cell = t / 4;
        const int i = 1 + (int)(cell / ny), j = 1 + (int)(cell % ny);
        const size_t cidx = (size_t)i * (ny + 2) + j;
        const double ss = sigma_s ? sigma_s[cidx] : 0.0;
        double v[N], S[N];
#pragma unroll
        for (int m = 0; m < N; ++m) {
            v[m] = phi ? phi[cidx * N + m] : 0.0;
            if (sigma_s) v[m] = (ss * v[m]) / (4.0 * M_PI);
            v[m] *= scale;
        }
        const bool xn = k >= 2, yn = (k & 1) != 0;
#pragma unroll
        for (int m = 0; m < N; ++m) {   // the quadrant's sign flip x(d,e) -> sx^d sy^e x(d,e)
            const int d = m / P, e = m % P;
            if (((d & 1) && xn) != ((e & 1) && yn)) v[m] = -v[m];
        }
        modal_forward<P, false, false, double, ADJ>(S, v);
        double *o = out + (cidx * 4 + k) * RD;
#pragma unroll
        for (int m = 0; m < N; ++m) o[m] = S[m];
        o[N] = sigma_t[cidx];
    }
}

template <int P, bool ADJ>
__global__ void modal_sources_kernel(GridDims g, const double *__restrict__ sigma_t, const double *__restrict__ sigma_s,
                                     const double *__restrict__ phi, double scale, double *__restrict__ out, int *reset) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && reset) *reset = 0;
    modal_sources<P, ADJ>(g.nx, g.ny, sigma_t, sigma_s, phi, scale, out);
}
// every problem of a batch's table (grid.y) that is not left out
template <int P>
__global__ void modal_sources_batched_kernel(const SweepArgs *__restrict__ table) {
    const SweepArgs &a = table[blockIdx.y];
    if (!a.skip)
        modal_sources<P, false>(a.nx, a.ny, a.sigma_t, a.sigma_s, a.phi_scatter, a.scatter_scale,
                                const_cast<double *>(a.modal_src));
}

// The records of every interior cell: sigma_s phi / (4 pi) (or phi itself without sigma_s), sigma_t.
template <int P>
__global__ void cell_records_kernel(GridDims g, const double *__restrict__ sigma_t, const double *__restrict__ sigma_s,
                                    const double *__restrict__ phi, double *__restrict__ out, int *reset) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && reset) *reset = 0;
    constexpr int N = P * P, RD = cell_record_doubles(P);
    const size_t total = (size_t)g.nx * g.ny * RD;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int m = (int)(t % RD);
        const size_t cell = t / RD;
        const int i = 1 + (int)(cell / g.ny), j = 1 + (int)(cell % g.ny);
        const size_t cidx = (size_t)i * (g.ny + 2) + j;
        double v = 0.0;
        if (m < N) {
            v = phi[cidx * N + m];
            if (sigma_s) v = (sigma_s[cidx] * v) / (4.0 * M_PI);
        } else if (m == N) {
            v = sigma_t[cidx];
        }
        out[cidx * RD + m] = v;
    }
}

// phi of the moments-only sweep: per interior cell and quadrant the fixed-order sum of its chunks' packed
// partials, transformed back and flipped, the quadrants added in order; ghost cells zero.
struct SlotBounds {
    int b[5];
};
// Four lanes per cell, one per quadrant: the sums over the slots are chains of loads, and a thread per cell left small
// grids with a few blocks of them (B200, 64x64 Q1 S8 8.9 us).
template <int P, bool ADJ>
__device__ __forceinline__ void reduce_modal_partials(int nx, int ny, const double *__restrict__ part, const SlotBounds &sb,
                                                      size_t stride, const double *__restrict__ minuend,
                                                      const double *__restrict__ sigma_s, double *__restrict__ phi) {
    constexpr int N = P * P;
    const size_t total = (size_t)(nx + 2) * (ny + 2);
    const int k = threadIdx.x & 3, lane = threadIdx.x & 31;
    const bool xn = k >= 2, yn = (k & 1) != 0;
    // whole warps stay together: 8 cells a turn
    for (size_t c0 = (blockIdx.x * (size_t)blockDim.x + threadIdx.x - lane) / 4; c0 < total;
         c0 += (size_t)gridDim.x * blockDim.x / 4) {
        const size_t cidx = c0 + lane / 4;
        const int i = (int)(cidx / (ny + 2)), j = (int)(cidx % (ny + 2));
        const bool interior = i >= 1 && i <= nx && j >= 1 && j <= ny;
        double M[N], x[N];
#pragma unroll
        for (int m = 0; m < N; ++m) M[m] = 0.0;
        if (interior)
            for (int sl = sb.b[k]; sl < sb.b[k + 1]; ++sl)
#pragma unroll
                for (int m = 0; m < N; ++m) M[m] += part[(size_t)sl * stride + cidx * N + m];
        modal_backward<P, false, false, double, ADJ>(x, M);
#pragma unroll
        for (int m = 0; m < N; ++m) {
            const int d = m / P, e = m % P;
            const double own = (((d & 1) && xn) != ((e & 1) && yn)) ? -x[m] : x[m];
            double acc = 0.0;   // the quadrants in order
#pragma unroll
            for (int q = 0; q < 4; ++q) acc += __shfl_sync(kFullMask, own, (lane & ~3) + q);
            if (k == m % 4 && cidx < total) {
                const double v = sigma_s && interior ? sigma_s[cidx] / (4.0 * M_PI) * acc : acc;
                phi[cidx * N + m] = minuend ? minuend[cidx * N + m] - v : v;
            }
        }
    }
}
template <int P, bool ADJ>
__global__ void reduce_modal_partials_kernel(GridDims g, const double *__restrict__ part, SlotBounds sb, size_t stride,
                                             const double *__restrict__ minuend, const double *__restrict__ sigma_s,
                                             double *__restrict__ phi) {
    reduce_modal_partials<P, ADJ>(g.nx, g.ny, part, sb, stride, minuend, sigma_s, phi);
}
template <int P>
__global__ void reduce_modal_batched_kernel(const SweepArgs *__restrict__ table) {
    const SweepArgs &a = table[blockIdx.y];
    if (a.skip) return;
    SlotBounds sb;
    for (int k = 0; k < 5; ++k) sb.b[k] = a.slot_begin[k];
    reduce_modal_partials<P, false>(a.nx, a.ny, a.phi_part, sb, a.phi_slot_stride, a.phi_scatter, nullptr, a.phi);
}

int blocks_for(size_t n) {
    const size_t b = (n + 255) / 256;
    return (int)(b < 148 * 32 ? (b > 0 ? b : 1) : 148 * 32);
}

template <int P>
cudaError_t occ_p(int seg, int warps, bool src2, int *n) {
    switch (seg) {
        case 4: return src2 ? lane::occupancy<P, 4, false, true>(warps, n) : lane::occupancy<P, 4, false, false>(warps, n);
        case 8: return src2 ? lane::occupancy<P, 8, false, true>(warps, n) : lane::occupancy<P, 8, false, false>(warps, n);
        case 16: return src2 ? lane::occupancy<P, 16, false, true>(warps, n) : lane::occupancy<P, 16, false, false>(warps, n);
        default: return cudaErrorInvalidValue;
    }
}

// args of a lane launch: warps per block, the rows they make, traces
bool args_ok(const SweepArgs &a) {
    return a.wn >= 1 && a.wn <= lane::kMaxWarps && a.G <= a.seg && a.R == a.wn * (32 / a.seg);
}

}  // namespace

bool sweep_lane_supports(int P, int precision, int seg) {
    return P >= 1 && P <= 3 && (precision == 0 || precision == 2) && (seg == 4 || seg == 8 || seg == 16);
}

// Compute warps per thread block, for a launch of row_blocks(w) items with w warps.  Small launches are bound by the
// latency of an iteration, and two warps on one SM sub-partition slow each other: 3 warps and the helper (one warp per
// sub-partition) while every block then has an SM of its own, else 4 likewise; large ones by the warps in flight and the
// handoffs through L2 between blocks: 7 and the helper.  At DG degree 2, whose iterations keep a sub-partition busier, 4
// up to 4/3 blocks per SM.  B200, sweep kernel in us with 3 / 4 / 7 warps (in brackets the blocks with 4):
//   degrees 0 and 1: 64x64 Q1 S8 65.6 / 67.6 / 71.7 (24), 256x128 Q1 S12 185 / 191 / 211 (96), 128x128 Q1 S16 150 / 130 / 141
//   (144), 256x256 Q1 S12 295 / 303 / 283 (192), 300x200 Q0 S16 234 / 218 / 204 (252), 512x512 Q1 S12 766 / 692 / 688 (384);
//   degree 2: 131x197 S10 267 / 270 / 322 (100), 192x128 S12 315 / 260 / 315 (128), 192x160 S12 352 / 315 / 345 (160),
//   128x128 S16 260 / 227 / 249 (192), 192x200 S12 404 / 351 / 383 (200), 128x144 S16 281 / 242 / 262 (216), 256x256 S16
//   633 / 633 / 600 (384): 4 warps stay ahead a little beyond the line;
//   moments-only: 64x64 Q1 S8 51.2 / 51.2 / 55.3, 128x128 Q2 S16 154 / 124 / 146, 256x256 Q2 S16 346 / 307 / 297.
int sweep_lane_warps(int P, int seg, bool src2, int num_sms, const std::function<int64_t(int)> &row_blocks) {
    int w = row_blocks(3) <= num_sms                              ? 3
            : row_blocks(4) <= (P == 3 ? num_sms * 4 / 3 : num_sms) ? 4
                                                                    : lane::kMaxWarps;
    while (w > 1 && lane::block_smem_bytes(P, seg, src2, false, w) > (size_t)(224 << 10)) --w;
    return w;
}

cudaError_t launch_sweep_lane(int P, int precision, const SweepArgs &args, int grid, cudaStream_t stream) {
    if (!args.trace || !args_ok(args)) return cudaErrorInvalidValue;
    if (precision != 0 && precision != 2) return cudaErrorInvalidValue;
    const bool fp32 = precision == 2;
    switch (P) {
        case 1: return launch_dir<1>(args, grid, stream, fp32);
        case 2: return launch_dir<2>(args, grid, stream, fp32);
        case 3: return launch_dir<3>(args, grid, stream, fp32);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_modal_sources(const GridDims &g, const double *sigma_t, const double *sigma_s, const double *phi,
                                 double scale, bool adjoint, double *out, int *reset, cudaStream_t s) {
    const int b = blocks_for((size_t)g.nx * g.ny * 4);
    switch (g.P + (adjoint ? 4 : 0)) {
        case 1: modal_sources_kernel<1, false><<<b, 256, 0, s>>>(g, sigma_t, sigma_s, phi, scale, out, reset); break;
        case 2: modal_sources_kernel<2, false><<<b, 256, 0, s>>>(g, sigma_t, sigma_s, phi, scale, out, reset); break;
        case 3: modal_sources_kernel<3, false><<<b, 256, 0, s>>>(g, sigma_t, sigma_s, phi, scale, out, reset); break;
        case 5: modal_sources_kernel<1, true><<<b, 256, 0, s>>>(g, sigma_t, sigma_s, phi, scale, out, reset); break;
        case 6: modal_sources_kernel<2, true><<<b, 256, 0, s>>>(g, sigma_t, sigma_s, phi, scale, out, reset); break;
        case 7: modal_sources_kernel<3, true><<<b, 256, 0, s>>>(g, sigma_t, sigma_s, phi, scale, out, reset); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_cell_records(const GridDims &g, const double *sigma_t, const double *sigma_s, const double *phi,
                                double *out, int *reset, cudaStream_t s) {
    const int b = blocks_for((size_t)g.nx * g.ny * cell_record_doubles(g.P));
    switch (g.P) {
        case 1: cell_records_kernel<1><<<b, 256, 0, s>>>(g, sigma_t, sigma_s, phi, out, reset); break;
        case 2: cell_records_kernel<2><<<b, 256, 0, s>>>(g, sigma_t, sigma_s, phi, out, reset); break;
        case 3: cell_records_kernel<3><<<b, 256, 0, s>>>(g, sigma_t, sigma_s, phi, out, reset); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_reduce_modal_partials(const GridDims &g, const double *part, const int slot_begin[5], size_t stride,
                                         bool adjoint, const double *minuend, const double *sigma_s, double *phi,
                                         cudaStream_t s) {
    SlotBounds sb;
    for (int k = 0; k < 5; ++k) sb.b[k] = slot_begin[k];
    const int b = blocks_for((size_t)(g.nx + 2) * (g.ny + 2) * 4);
    switch (g.P + (adjoint ? 4 : 0)) {
        case 1: reduce_modal_partials_kernel<1, false><<<b, 256, 0, s>>>(g, part, sb, stride, minuend, sigma_s, phi); break;
        case 2: reduce_modal_partials_kernel<2, false><<<b, 256, 0, s>>>(g, part, sb, stride, minuend, sigma_s, phi); break;
        case 3: reduce_modal_partials_kernel<3, false><<<b, 256, 0, s>>>(g, part, sb, stride, minuend, sigma_s, phi); break;
        case 5: reduce_modal_partials_kernel<1, true><<<b, 256, 0, s>>>(g, part, sb, stride, minuend, sigma_s, phi); break;
        case 6: reduce_modal_partials_kernel<2, true><<<b, 256, 0, s>>>(g, part, sb, stride, minuend, sigma_s, phi); break;
        case 7: reduce_modal_partials_kernel<3, true><<<b, 256, 0, s>>>(g, part, sb, stride, minuend, sigma_s, phi); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

namespace {
template <int P, bool PHI>
cudaError_t launch_batched_p(int seg, const SweepArgs &args, const SweepArgs *table, int grid, cudaStream_t stream) {
    switch (seg) {
        case 4: return lane::launch_batched<P, 4, PHI>(args, table, grid, stream);
        case 8: return lane::launch_batched<P, 8, PHI>(args, table, grid, stream);
        case 16: return lane::launch_batched<P, 16, PHI>(args, table, grid, stream);
        default: return cudaErrorInvalidValue;
    }
}
template <int P>
cudaError_t launch_batched_any(const SweepArgs &args, const SweepArgs *table, int members, bool moments_only, int grid,
                               cudaStream_t stream) {
    if (!moments_only) return launch_batched_p<P, false>(args.seg, args, table, grid, stream);
    const dim3 helpers(148, (unsigned)members);   // grid-stride over each problem's cells
    modal_sources_batched_kernel<P><<<helpers, 256, 0, stream>>>(table);
    cudaError_t e = launch_batched_p<P, true>(args.seg, args, table, grid, stream);
    if (e != cudaSuccess) return e;
    reduce_modal_batched_kernel<P><<<helpers, 256, 0, stream>>>(table);
    return cudaGetLastError();
}
template <int P>
cudaError_t occupancy_batched_p(int seg, int warps, int *n) {
    switch (seg) {
        case 4: return lane::occupancy_batched<P, 4>(warps, n);
        case 8: return lane::occupancy_batched<P, 8>(warps, n);
        case 16: return lane::occupancy_batched<P, 16>(warps, n);
        default: return cudaErrorInvalidValue;
    }
}
}  // namespace

cudaError_t launch_sweep_lane_batched(int P, const SweepArgs &args, const SweepArgs *table, int members, bool moments_only,
                                      int grid, cudaStream_t stream) {
    if (!args_ok(args) || !table) return cudaErrorInvalidValue;
    switch (P) {
        case 1: return launch_batched_any<1>(args, table, members, moments_only, grid, stream);
        case 2: return launch_batched_any<2>(args, table, members, moments_only, grid, stream);
        case 3: return launch_batched_any<3>(args, table, members, moments_only, grid, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t sweep_lane_batched_occupancy(int P, int seg, int warps, int *blocks_per_sm) {
    switch (P) {
        case 1: return occupancy_batched_p<1>(seg, warps, blocks_per_sm);
        case 2: return occupancy_batched_p<2>(seg, warps, blocks_per_sm);
        case 3: return occupancy_batched_p<3>(seg, warps, blocks_per_sm);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t sweep_lane_occupancy(int P, int seg, int warps, bool src2, int *blocks_per_sm) {
    switch (P) {
        case 1: return occ_p<1>(seg, warps, src2, blocks_per_sm);
        case 2: return occ_p<2>(seg, warps, src2, blocks_per_sm);
        case 3: return occ_p<3>(seg, warps, src2, blocks_per_sm);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace idc
