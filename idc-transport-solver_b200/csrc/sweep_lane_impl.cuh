// Lane-pipelined persistent wavefront sweep for sm_100a.
//
// Replaces SweepPatternUniCartWavefront::Sweep (linear_solvers/Abstract/SweepPattern/
// SweepPatternUniCartWavefront.cpp:121-332) with the per-cell CalcB / CalcA / GE / StoreResult of
// SweepCellSolveBase::ConstructAndSolve (linear_solvers/RKDG/SweepCellSolve/SweepCellSolve.hpp:312-353),
// in the packed modal basis of modal_cell.cuh (the same cell arithmetic as sweep_modal_impl.cuh).
//
// An item is a group of consecutive row blocks of one quadrant for one chunk of <= SEG ordinates, swept across all
// columns by one thread block: warp w owns row block w of the group, Rw = 32/SEG rows (in sweep order).  Lane (rr, o) =
// (lane / SEG, lane % SEG) owns ordinate q_begin + o on row rr; row rr runs one column behind row rr-1 and takes its y
// trace by __shfl_up, the x trace stays in the lane.  A block's last warp is its helper: it takes the block's items from
// the queue and feeds the traces of the row above the block to the first warp.
//
// Iteration s of a warp is one basic block after the (rarely taken) waits:
//   * the chain of step s: the y trace in, the modal cell step, the traces out (the only dependency from cell to cell,
//     so the only part whose latency sits on the wavefront's critical path); beside it the forward modal transform and
//     the reciprocal denominators of step s + 1's inputs, copied into shared memory by cp.async kStages - 1 iterations
//     earlier;
//   * the finish of step s: the backward transform; psi (degree 2: through a per-warp shared buffer, 16-byte stores of
//     the row segment's chunks; degree 1: a lane's 32-byte block in one store); the row segment's moment sums (a shuffle
//     butterfly for 4- and 8-wide segments, sums over a k-major shared buffer for 16-wide ones), one partial per ordinate
//     chunk, each a fixed tree, added in a fixed order by reduce_phi_partials: bitwise reproducible;
//   * the copies of step s + kStages.
// Every global access is predicated instead of branched around, so the scheduler interleaves the parts.  The quadrant's
// sign flips are applied to the cell values at run time as sign-bit flips (exact): one loop body for every quadrant.
//
// What bounds it: a sweep of nx columns and ny rows is nx + ny iterations long plus the handoffs between row blocks, so
// the time of one iteration of a lone warp (latency, at few warps per sub-partition) and the handoffs set the small
// sizes, issue slots the large ones.  Measured on B200 (sweep kernel, before -> after each):
//   * handoff through shared memory, L2 only between blocks and there by the helper: when every warp read the trace of
//     the row above from L2 itself, no iteration could be shorter than an L2 load (0.56 us at degree 0, where it is 0.2
//     us of work).  With the rest below, 300x200 Q0 S16 349 -> 204 us, 64x64 Q1 S8 85 -> 66 us, 512x512 Q1 S12 932 -> 688
//     us; 256x256 Q2 S16 (684 -> 600 us) is bound by issue and latency: 633 warp instructions per iteration, 217 of them
//     FP64, with 253 registers and so two warps per sub-partition.
//   * psi stores: bulk copies through shared memory (proxy fence, commit, wait) cost 0.25 us an iteration at degree 1;
//     a lane's own 32-byte store 0.001 (2048x4 Q1 S8, one row block: 1342 -> 832 us).  Degree 2: 16-byte chunks.
//   * the moments-only sweeps' inputs (modal source and sigma_t) as one record per cell copied once per row, where every
//     lane had copied its own: 256x256 Q2 S16 566 -> 297 us with the above, 128x128 Q1 S8 117 -> 97 us.
//   * the backward transform in its own iteration instead of beside the next one's chain: 38 fewer live registers, no
//     spills at degree 2 (2048x2 Q2 S16, one row block: 1766 -> 1460 us).
//
// Handoffs.  Traces travel as 8-byte values that are their own flags: a slot holds a NaN-payload sentinel until its value
// is written, and the reader writes the sentinel back.  Between the warps of a block a ring of kRing columns in shared
// memory (the reader publishes how many columns it has read, every fourth column; the writer waits for room); from a
// block's last warp the item's row of the global trace buffer, relaxed 8-byte stores, which the helper of the block below
// reads kFeedAhead columns at a time and passes into its first warp's ring.  The grid's first row takes the ghost row's
// inflow traces (inflow_traces_kernel) the same way.  Items are dequeued in row-group order from an atomic counter, so an
// item's producer is always held by a running block: no deadlock, and no block needs any other to be resident.  Every
// wait is bounded (spin_limit); on expiry the warp records kDevTimeout in the device error word and leaves, and every
// other warp leaves when it sees the word.
//
// Transposed sweep (ADJ): reverse traversal order per quadrant, the transposed cell operator and coupling
// of modal_cell.cuh, zero inflow, the fused source w_q * mu and unweighted moment sums (the transposes of
// Smv's broadcast and of Pmv).  SRC2 adds a second source, fma(src2_scale, src2, src), as the IDC source
// kernel combines them.  PHI: the moments-only sweep of the Krylov iterations (no source array,
// psi not stored): the cell's source is its isotropic scattering source, the same for every ordinate of a
// quadrant, read already in the packed modal basis (launch_modal_sources, once per cell and quadrant), and
// the moments are summed in the packed basis (launch_reduce_modal_partials transforms each quadrant's sum
// back once per cell), so neither modal transform is done per ordinate.  TC is the arithmetic: double (the
// reference's FP64) or float (the unrefined FP32 sweep of IDC_PREC_FP32: FP32 cell arithmetic and moment
// sums, FP64 arrays and traces), forward sweeps only.
#pragma once

#include "device_sync.cuh"
#include "idc_internal.hpp"
#include "modal_cell.cuh"

#include <cstdint>

namespace idc {
namespace lane {

constexpr int kMaxWarps = 7;   // compute warps per thread block; the helper warp is the eighth (two per SM sub-partition)
constexpr int kStages = 6;     // stages in shared memory: a step's inputs are copied this many steps minus one ahead
constexpr int kRing = 16;      // columns of y traces between two warps of a thread block: slack that absorbs the warps' jitter
                               // (B200, sweep kernel with 8 -> 16: 256x256 Q2 S16 630 -> 607 us, 512x512 Q1 S12 716 -> 659)
constexpr int kMomStride = 34; // doubles per moment index k in the moment buffer (32 lanes + 2: conflict-free sums)

// Degrees 1 and 2 copy a row segment's source dofs to shared memory, and degree 2 its psi back, in 16-byte chunks: lane o
// of the row takes chunks o, o + SEG, ... of the segment, whose start is moved down to a 16-byte boundary (copies are
// coalesced whatever the degree, where a lane's own 72-byte block at degree 2 would take nine 8-byte accesses in as many
// sectors).  Chunks per lane, and doubles from one row's block in shared memory to the next (it starts at the parity, in
// 8-byte words, of its global address).
__host__ __device__ constexpr bool chunked(int P) { return P >= 2; }
__host__ __device__ constexpr int lane_chunks(int P, int seg) { return (seg * P * P / 2 + 1 + seg - 1) / seg; }
__host__ __device__ constexpr int row_pitch(int P, int seg) { return chunked(P) ? 2 * seg * lane_chunks(P, seg) + 2 : seg; }

// Shared memory of one warp, in doubles (every part an even number, so each starts on a 16-byte boundary): source
// stages [kStages][Rw][pitch], the second source's, cell records [kStages][Rw][cell_record_doubles] (sigma_t and the
// scattering moments, one copy per row), at degree 2 the psi out buffer [Rw][pitch] and, for 16-wide segments, the
// weighted moment values [N][kMomStride] (k-major: a row segment's values of one k are adjacent).
__host__ __device__ constexpr size_t warp_doubles(int P, int seg, bool src2, bool phi) {
    return (size_t)kStages * (32 / seg) * row_pitch(P, seg) * (phi ? 0 : src2 ? 2 : 1) +
           (size_t)kStages * (32 / seg) * cell_record_doubles(P) +
           (phi || P < 3 ? 0 : (size_t)(32 / seg) * row_pitch(P, seg)) +
           (seg >= 16 ? (size_t)P * P * kMomStride : 0);
}
// Doubles of one warp's trace ring [kRing][seg][P].
__host__ __device__ constexpr size_t ring_doubles(int P, int seg) { return (size_t)kRing * seg * P; }
// Doubles of the block's common part: the zero source of lanes without one and the consumed-column counts of every warp.
__host__ __device__ constexpr size_t common_doubles(int P, int warps) {
    return (size_t)((P * P + 1) / 2 * 2) + (size_t)((warps + 3) / 4 * 2);
}
__host__ __device__ constexpr size_t block_smem_bytes(int P, int seg, bool src2, bool phi, int warps) {
    return sizeof(double) * (warps * (warp_doubles(P, seg, src2, phi) + ring_doubles(P, seg)) + common_doubles(P, warps));
}

// x with its sign bit flipped where `mask` has it (mask: 0 or 0x80000000, the sign bit of a float or of a
// double's high word).
__device__ __forceinline__ double flip_by(double x, unsigned mask) {
    return __hiloint2double(__double2hiint(x) ^ (int)mask, __double2loint(x));
}
__device__ __forceinline__ float flip_by(float x, unsigned mask) { return __int_as_float(__float_as_int(x) ^ (int)mask); }

// Sums of v[0 .. N) over the SEG lanes of a row segment (o = lane % SEG) by recursive halving: at the
// stage of distance h a lane keeps the lower half of its current range if bit h of o is clear, the upper
// half otherwise, and adds its partner's copy of it (the halves always sit in slots 0 .. len-1).  After
// log2(SEG) stages lane o holds the sums of k in [*lo, *hi) in slots 0 .. *hi - *lo.  Every sum is a fixed
// tree over the segment's lanes.
template <int N, int SEG, int LEN = N, int H = SEG / 2, typename T>
__device__ __forceinline__ void segment_sums(T (&v)[N], int o, int *lo, int *hi) {
    if constexpr (H >= 1) {
        constexpr int HALF = (LEN + 1) / 2;
        const bool upper = (o & H) != 0;
#pragma unroll
        for (int i = 0; i < HALF; ++i) {
            const T keep = upper ? (i + HALF < LEN ? v[i + HALF] : T(0)) : v[i];
            const T give = upper ? v[i] : (i + HALF < LEN ? v[i + HALF] : T(0));
            v[i] = keep + __shfl_xor_sync(kFullMask, give, H);
        }
        const int mid = *lo + HALF;
        if (upper)
            *lo = mid < *hi ? mid : *hi;
        else
            *hi = mid < *hi ? mid : *hi;
        segment_sums<N, SEG, HALF, H / 2, T>(v, o, lo, hi);
    }
}

// Global accesses under a predicate instead of a branch, so that the loop body stays one basic block and
// the scheduler can interleave the parts of an iteration.  An access whose predicate is false is not made.
__device__ __forceinline__ void st_f64_if(double *p, double v, bool pred) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q st.global.f64 [%0], %1;\n\t}" ::"l"(p), "d"(v),
                 "r"((int)pred));
}
__device__ __forceinline__ void st_relaxed_f64_if(double *p, double v, bool pred) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q st.relaxed.gpu.global.f64 [%0], %1;\n\t}" ::"l"(p),
                 "d"(v), "r"((int)pred));
}
// 0.0 where the predicate is false
__device__ __forceinline__ double ld_relaxed_f64_if(const double *p, bool pred) {
    double v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
                 "@q ld.relaxed.gpu.global.f64 %0, [%1];\n\t}"
                 : "=d"(v)
                 : "l"(p), "r"((int)pred));
    return v;
}
__device__ __forceinline__ void cp_async8_if(void *dst, const void *src, bool pred) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q cp.async.ca.shared.global [%0], [%1], 8;\n\t}" ::"r"(
                     saddr(dst)),
                 "l"(src), "r"((int)pred));
}

__device__ __forceinline__ void cp_async16_if(void *dst, const void *src, bool pred) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q cp.async.cg.shared.global [%0], [%1], 16;\n\t}" ::"r"(
                     saddr(dst)),
                 "l"(src), "r"((int)pred));
}
// Trace rings in shared memory: 8-byte values that are their own flags (relaxed within the block), and the count of
// columns a ring's consumer has read and re-armed (release / acquire).
__device__ __forceinline__ double ld_ring_if(uint32_t p, bool pred) {   // 0.0 where the predicate is false
    double v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
                 "@q ld.relaxed.cta.shared::cta.f64 %0, [%1];\n\t}"
                 : "=d"(v)
                 : "r"(p), "r"((int)pred));
    return v;
}
__device__ __forceinline__ void st_ring_if(uint32_t p, double v, bool pred) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q st.relaxed.cta.shared::cta.f64 [%0], %1;\n\t}" ::"r"(p),
                 "d"(v), "r"((int)pred));
}
// a trace value out: into the next warp's ring or the trace buffer (a generic address)
__device__ __forceinline__ void st_trace_if(double *p, double v, bool pred) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q st.relaxed.gpu.f64 [%0], %1;\n\t}" ::"l"(p), "d"(v),
                 "r"((int)pred));
}
__device__ __forceinline__ int ld_consumed(uint32_t p) {
    int v;
    asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_consumed_if(uint32_t p, int v, bool pred) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q st.release.cta.shared::cta.s32 [%0], %1;\n\t}" ::"r"(p),
                 "r"(v), "r"((int)pred)
                 : "memory");
}

__device__ __forceinline__ void st_f64x2_if(double *p, double2 v, bool pred) {   // 16-byte aligned
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %3, 0;\n\t@q st.global.v2.f64 [%0], {%1, %2};\n\t}" ::"l"(p), "d"(v.x),
                 "d"(v.y), "r"((int)pred));
}
__device__ __forceinline__ void st_f64x4_if(double *p, double a, double b, double c, double d, bool pred) {   // 32-byte aligned
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t@q st.global.v4.f64 [%0], {%1, %2, %3, %4};\n\t}" ::"l"(p),
                 "d"(a), "d"(b), "d"(c), "d"(d), "r"((int)pred));
}

// Waits of the hot loop, out of line and bounded: a warp whose wait gives up, or that hears of another's failure,
// leaves with the error word set.
constexpr int kReadsPerPoll = 32;     // a poll of the waits on shared memory: this many reads (about 1 us)

// One more poll of a wait: false if it gives up (then the error word is set) or another warp has failed.
__device__ __forceinline__ bool poll_on(long long &polls, int *error, long long spin_limit, int lane) {
    if (++polls > spin_limit) {
        if (lane == 0) atomicCAS(error, kDevOk, kDevTimeout);
        return false;
    }
    int e = 0;
    if ((polls & 15) == 0 && lane == 0) e = ld_relaxed(error);
    return __shfl_sync(kFullMask, e, 0) == kDevOk;
}
// The ring whose consumer has read `*consumed` columns has no room for `column`: wait, and return the first column
// that may not be written yet, or -1.
__device__ __forceinline__ int wait_for_credit(uint32_t consumed, int column, int *error, long long spin_limit, int lane,
                                               unsigned sleep_ns) {
    for (long long polls = 0;;) {
        for (int k = 0; k < kReadsPerPoll; ++k) {
            // (every lane acquires the count itself: its writes are ordered after the reader's re-arming)
            const int c = (int)__reduce_min_sync(kFullMask, (unsigned)ld_consumed(consumed));
            if (column < c + kRing) return c + kRing;
            __nanosleep(sleep_ns);
        }
        if (!poll_on(polls, error, spin_limit, lane)) return -1;
    }
}
// Something step s needs is not there: its column of the ring above (not written yet), or room for column cout in the ring
// below.  Waits for both.
template <int P>
struct StepWait {
    double v[P];   // the column's traces; 0.0 in lanes that do not read
    int credit;    // as wait_for_credit; -1: gave up
};
template <int P>
__device__ __noinline__ StepWait<P> wait_for_step(uint32_t slot, bool reader, uint32_t consumed, int cout, int credit,
                                                  int nx, int *error, long long spin_limit, int lane) {
    StepWait<P> r;
    r.credit = -1;
    for (long long polls = 0;;) {
        bool there = false;
        for (int k = 0; k < kReadsPerPoll && !there; ++k) {
            bool still = false;
#pragma unroll
            for (int m = 0; m < P; ++m) {
                r.v[m] = ld_ring_if(slot + 8u * m, reader);
                still |= reader && is_sentinel(r.v[m]);
            }
            there = !__any_sync(kFullMask, still);
        }
        if (there) break;
        if (!poll_on(polls, error, spin_limit, lane)) return r;
    }
    if (cout >= credit && cout < nx) {
        credit = wait_for_credit(consumed, cout, error, spin_limit, lane, 20);
        if (credit < 0) return r;
    }
    r.credit = credit;
    return r;
}

// The helper warp: column by column, the traces entering the block's first row (the trace buffer of the item above,
// polled until its last row has written them and re-armed behind, or the ghost row's inflow) into the first warp's
// ring.  kFeedAhead columns are loaded at a time, so that the L2 round trip of a load is paid once for as many columns
// as are there.
constexpr int kFeedAhead = 4;
template <int P, int SEG>
__device__ __forceinline__ void feed_ring(const SweepArgs &a, const SweepItem &item, uint32_t ring, uint32_t consumed,
                                          int lane) {
    constexpr int V = SEG * P, NL = (V + 31) / 32;   // values per column, loads per lane and column
    const bool has_dep = item.dep >= 0;
    const int count = item.q_count * P;
    const size_t stride = has_dep ? (size_t)a.G * P : (size_t)a.nq * P;
    double *src = has_dep ? a.trace + (size_t)item.dep * a.trace_stride
                          : const_cast<double *>(a.inflow) + (size_t)item.q_begin * P;
    long long polls = 0;
    int credit = kRing;
    int c = 0;
    while (c < a.nx) {
        double v[kFeedAhead][NL];
#pragma unroll
        for (int k = 0; k < kFeedAhead; ++k)
#pragma unroll
            for (int h = 0; h < NL; ++h)
                v[k][h] = ld_relaxed_f64_if(src + (size_t)(c + k) * stride + lane + 32 * h,
                                            c + k < a.nx && lane + 32 * h < count);
        int done = 0;
        bool go = true;
#pragma unroll
        for (int k = 0; k < kFeedAhead; ++k) {
            if (go && c + k < a.nx) {
                bool still = false;
#pragma unroll
                for (int h = 0; h < NL; ++h) still |= lane + 32 * h < count && is_sentinel(v[k][h]);
                if (has_dep && __any_sync(kFullMask, still)) {
                    go = false;
                } else {
                    if (c + k >= credit) {
                        credit = wait_for_credit(consumed, c + k, a.error, a.spin_limit, lane, 200);   // (awake, its polls would take a compute
                                                                                                         // warp's issue slots)
                        if (credit < 0) return;
                    }
                    const uint32_t slot = ring + 8u * (uint32_t)(((c + k) % kRing) * V + lane);
#pragma unroll
                    for (int h = 0; h < NL; ++h) {
                        const bool p = lane + 32 * h < count;
                        st_ring_if(slot + 256u * h, v[k][h], p);
                        st_relaxed_f64_if(src + (size_t)(c + k) * stride + lane + 32 * h, sentinel_value(), p && has_dep);
                    }
                    ++done;
                }
            }
        }
        c += done;
        if (done == 0) {
            if (!poll_on(polls, a.error, a.spin_limit, lane)) return;
        } else {
            polls = 0;
        }
    }
}

// One warp's part of an item: its Rw rows across all columns.  ring_in: the ring (shared address) that feeds its first
// row if `fed` (else that row's y traces are zero: the grid's first row without inflow); ring_out: the next warp's ring,
// or null (the warp writes the item's trace buffer); consumed: this ring's count of columns read, the next ring's four
// bytes on.
template <int P, int SEG, bool ADJ, bool SRC2, bool PHI, typename TC>
__device__ __forceinline__ void run_rows(const SweepArgs &a, const SweepItem &item, int it_index, int row_w, double *wsm,
                                         const double *zero, uint32_t ring_in, bool fed, double *ring_out, uint32_t consumed,
                                         int lane) {
    constexpr int N = P * P, Rw = 32 / SEG, D = kStages, V = SEG * P, PITCH = row_pitch(P, SEG);
    constexpr int RD = cell_record_doubles(P), CH = RD / 2;
    constexpr int NC = lane_chunks(P, SEG);
    constexpr bool CHUNK = chunked(P) && !PHI, OBUF = P >= 3 && !PHI;
    // quadrant signs: flips of the cell values (exact), traversal directions (reversed for the transpose)
    const bool XN = item.quadrant >= 2, YN = (item.quadrant & 1) != 0;
    const bool TX = XN != ADJ, TY = YN != ADJ;
    const int quadrant = item.quadrant;
    const int rr = lane / SEG, o = lane - rr * SEG;
    const int row = row_w + rr;
    const bool row_valid = row < a.ny;
    const bool act = (o < item.q_count) && row_valid;
    const int q = item.q_begin + (act ? o : 0);
    auto row_j = [&](int r) { return TY ? (a.ny - r) : (1 + r); };   // array y index of a sweep row
    const int j = row_valid ? row_j(row) : 1;
    const int nx = a.nx;
    const size_t plane = (size_t)a.nq * N;
    const size_t cstride = (size_t)(a.ny + 2);
    const bool has_consumer = row_w + Rw < a.ny;
    const bool has_rec = PHI || a.cell_rec != nullptr;
    const bool has_src = !PHI && a.src != nullptr;
    const int T = nx + Rw - 1;
    const int xi0 = TX ? nx : 1, xis = TX ? -1 : 1;   // array x index of sweep column c: xi0 + xis * c
    const unsigned xm = XN ? 0x80000000u : 0u, ym = YN ? 0x80000000u : 0u;
    auto fmask = [&](int k) { return ((k / P) & 1 ? xm : 0u) ^ ((k % P) & 1 ? ym : 0u); };   // k = e + P d

    double *stage = wsm;                                                  // step t at + (t % D) * Rw * PITCH
    double *stage2 = wsm + (PHI ? 0 : (size_t)D * Rw * PITCH);            // (SRC2 launches only)
    double *recs = stage2 + (SRC2 ? (size_t)D * Rw * PITCH : 0);          // + (t % D) * Rw * RD
    double *obuf = recs + (size_t)D * Rw * RD + (size_t)rr * PITCH;       // (its row's block)
    double *mbuf = recs + (size_t)D * Rw * RD + (OBUF ? (size_t)Rw * PITCH : 0);   // [N][kMomStride]

    // an inactive lane runs the cell step of a unit ordinate on a zero source with moment weight zero (finite
    // values), so that the moment sums need no selects
    double axd = 1.0, ayd = 1.0, wq = 0.0;
    if (act) {
        axd = fabs(a.xi[q]) / a.dx;
        ayd = fabs(a.eta[q]) / a.dy;
        wq = a.w[q];
    }
    const ModalOrdinate<P, TC> od = modal_ordinate<P, TC, ADJ>(axd, ayd);
    const TC wv = act ? (ADJ ? TC(1) : TC(wq)) : TC(0);   // moment weight (the transpose sums unweighted)

    // the row's x trace entering its first column (ghost-column inflow; zero for the transposed sweep)
    TC f[P];
#pragma unroll
    for (int m = 0; m < P; ++m) f[m] = TC(0);
    if (act && a.inflow && !ADJ) {
        const double *in = a.inflow + ((size_t)(nx + row) * a.nq + q) * P;
#pragma unroll
        for (int m = 0; m < P; ++m) f[m] = TC(in[m]);
    }

    // row 0's y traces come through the ring; the last row's go to the next warp's ring or the trace buffer
    const bool reader = fed && rr == 0 && o < item.q_count && row_valid;
    const bool writer = has_consumer && rr == Rw - 1 && o < item.q_count;
    const bool feeds = ring_out != nullptr && has_consumer;
    ring_in += 8u * (uint32_t)(o * P);
    // column c's traces go to tout + (c & tmask) * tstride
    double *tout = (feeds ? ring_out : a.trace + (size_t)it_index * a.trace_stride) + o * P;
    const int tmask = feeds ? kRing - 1 : -1, tstride = feeds ? V : a.G * P;
    int credit = feeds ? kRing : nx;   // first column that may not be written yet

    // Column addresses advance by a fixed stride per step: step t of row r reads column t - r, whose cell index is
    // (xi0 + xis (t - r)) cstride + j(r); the offsets are kept running (prefetches come in step order).
    const long long dcol = (long long)xis * (long long)cstride;   // cells between consecutive columns
    const long long dsoff = dcol * (long long)plane;              // psi doubles between them
    const long long cell0 = ((long long)xi0 - (long long)xis * rr) * (long long)cstride + j;   // step 0's column
    const long long seg0 = cell0 * (long long)plane + (long long)item.q_begin * N;             // its row segment
    const double *pf_src = a.src + (seg0 + (CHUNK ? 2 * o : (long long)(q - item.q_begin) * N));   // step t's, in order
    const double *pf_src2 = a.src2 + (seg0 + (CHUNK ? 2 * o : (long long)(q - item.q_begin) * N));
    auto chunk16 = [](const double *p) {   // the 16-byte boundary at or below
        return reinterpret_cast<const double *>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)15);
    };
    // parity of a row segment's address in 8-byte words at step t: par ^ (t & podd), kept running (steps s and s + D
    // share it)
    static_assert(D % 2 == 0, "steps s and s + D have the same parity");
    const unsigned podd = (unsigned)dsoff & 1u;
    unsigned spar = ((unsigned)((size_t)a.src >> 3) + (unsigned)seg0) & 1u;
    unsigned s2par = SRC2 ? ((unsigned)((size_t)a.src2 >> 3) + (unsigned)seg0) & 1u : 0u;
    unsigned opar = ((unsigned)((size_t)a.out >> 3) + (unsigned)seg0) & 1u;
    const int seg_n = item.q_count * N;
    const bool odd_out = OBUF && a.out != nullptr && (podd | opar | ((unsigned)seg_n & 1u)) != 0;
    const int out_align = OBUF ? 0 : (int)((size_t)a.out & 31);   // degree 1: 32-byte stores where psi allows
    // the cell records (or sigma_t alone) of a step's rows are copied once per row: lane l copies chunk l % ch of row
    // l / ch (16 bytes of the record, or 8 of sigma_t)
    constexpr int NI = (Rw * CH + 31) / 32;
    const int ch = has_rec ? CH : 1;
    const double *rec_src = PHI ? a.modal_src + (size_t)quadrant * RD : has_rec ? a.cell_rec : a.sigma_t;
    const long long rec_cell = PHI ? 4 * RD : has_rec ? RD : 1;   // doubles per cell
    int prow[NI], pdst[NI];
    const double *pf_rec[NI];
#pragma unroll
    for (int h = 0; h < NI; ++h) {
        const int idx = lane + 32 * h;
        prow[h] = idx / ch;
        const int k = idx - prow[h] * ch;
        pdst[h] = prow[h] * RD + (has_rec ? 2 * k : N);
        if (prow[h] >= Rw || row_w + prow[h] >= a.ny) prow[h] = -(1 << 28);   // nothing to copy: never in range
        const int r = prow[h] < 0 ? 0 : prow[h];
        pf_rec[h] = rec_src + ((((long long)xi0 - (long long)xis * r) * (long long)cstride + row_j(row_w + r)) * rec_cell +
                               (has_rec ? 2 * k : 0));
    }
    const long long dpoff = dcol * rec_cell;
    // step t's inputs into stage slot = t % D; a cell outside the row is not copied (its results are not used)
    // (par, par2: the sources' parities at step t)
    auto prefetch = [&](int t, int slot, unsigned par, unsigned par2) {
        const bool in = row_valid && (unsigned)(t - rr) < (unsigned)nx;
        if constexpr (CHUNK) {
            const int lim = in && has_src ? seg_n + (int)par - 2 * o : 0;
            double *d = stage + (size_t)(slot * Rw + rr) * PITCH + 2 * o;
            const double *g = chunk16(pf_src);
#pragma unroll
            for (int h = 0; h < NC; ++h) cp_async16_if(d + 2 * SEG * h, g + 2 * SEG * h, lim > 2 * SEG * h);
            if constexpr (SRC2) {
                const int lim2 = in ? seg_n + (int)par2 - 2 * o : 0;
                double *d2 = stage2 + (size_t)(slot * Rw + rr) * PITCH + 2 * o;
                const double *g2 = chunk16(pf_src2);
#pragma unroll
                for (int h = 0; h < NC; ++h) cp_async16_if(d2 + 2 * SEG * h, g2 + 2 * SEG * h, lim2 > 2 * SEG * h);
            }
        } else if constexpr (!PHI) {   // degree 0: a row segment's values are adjacent
            cp_async8_if(stage + (size_t)(slot * Rw + rr) * PITCH + o, pf_src, in && act && has_src);
            if constexpr (SRC2)
                cp_async8_if(stage2 + (size_t)(slot * Rw + rr) * PITCH + o, pf_src2, in && act);
        }
#pragma unroll
        for (int h = 0; h < NI; ++h) {
            const bool pr = (unsigned)(t - prow[h]) < (unsigned)nx;
            double *d = recs + (size_t)slot * Rw * RD + pdst[h];
            if (has_rec)
                cp_async16_if(d, pf_rec[h], pr);
            else
                cp_async8_if(d, pf_rec[h], pr);
            pf_rec[h] += dpoff;
        }
        cp_commit();
        pf_src += dsoff;
        if constexpr (SRC2) pf_src2 += dsoff;
    };
    // step t's raw inputs from its landed stage: the source (with the second source and the fused scattering
    // source) and sigma_t + 1/dt
    auto load_inputs = [&](int slot, unsigned par, unsigned par2, double (&src)[N], double &st) {   // slot = t % D of step t
        const double2 *rv = reinterpret_cast<const double2 *>(recs + (size_t)(slot * Rw + rr) * RD);
        double rp[RD];
        if (has_rec) {
#pragma unroll
            for (int h = 0; h < CH; ++h) {
                const double2 v = rv[h];
                rp[2 * h] = v.x;
                rp[2 * h + 1] = v.y;
            }
        } else {
            rp[N] = recs[(size_t)(slot * Rw + rr) * RD + N];
        }
        if constexpr (PHI) {   // the cell's packed modal source of this quadrant (the transpose's times w_q)
#pragma unroll
            for (int k = 0; k < N; ++k) src[k] = ADJ ? wq * rp[k] : rp[k];
        } else {
            const double *sp = has_src && act ? stage + (size_t)(slot * Rw + rr) * PITCH + (CHUNK ? par : 0u) + o * N : zero;
#pragma unroll
            for (int k = 0; k < N; ++k) src[k] = sp[k];
            if constexpr (SRC2) {
                const double *sp2 = act ? stage2 + (size_t)(slot * Rw + rr) * PITCH + (CHUNK ? par2 : 0u) + o * N : zero;
#pragma unroll
                for (int k = 0; k < N; ++k) src[k] = fma(a.src2_scale, sp2[k], src[k]);
            }
            if (has_rec) {
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    if constexpr (!ADJ)   // fused TransportOperator::Smv(scale, 1, sigma_s, phi -> src)
                        src[k] = fma(a.scatter_scale, rp[k], src[k]);
                    else                  // the transpose of Pmv: w_q * mu
                        src[k] = fma(wq, rp[k], src[k]);
                }
            }
        }
        st = rp[N] + a.inv_dt;
    };
    // the modal source and the reciprocal denominators of the raw inputs (the prologue's step; in the loop the
    // forward transform runs beside the previous step's backward transform)
    auto transform = [&](const double (&src)[N], double st, TC (&S)[N], ModalRecip<P, TC> &r) {
        r = modal_recip<P, TC>(od, TC(st));
        if constexpr (PHI) {
#pragma unroll
            for (int k = 0; k < N; ++k) S[k] = TC(src[k]);
        } else {
            TC sv[N];
#pragma unroll
            for (int k = 0; k < N; ++k) sv[k] = flip_by(TC(src[k]), fmask(k));
            modal_forward<P, false, false, TC, ADJ>(S, sv);
        }
    };

    const int phi_slot = a.phi_slots > 0 ? it_index % a.phi_slots : 0;
    double *phi_base = a.phi_part ? a.phi_part + (size_t)phi_slot * a.phi_slot_stride : nullptr;

    // prologue: stages 0 .. D-1 in flight, step 0 prepared
#pragma unroll
    for (int t = 0; t < D; ++t) prefetch(t, t, spar ^ (t & podd), s2par ^ (t & podd));
    cp_wait<D - 1>();
    __syncwarp();   // the other lanes' copies
    TC S[N];
    ModalRecip<P, TC> r;
    {
        double src0[N], st0;
        load_inputs(0, spar, s2par, src0, st0);
        transform(src0, st0, S, r);
    }
    cp_wait<D - 2>();
    __syncwarp();
    double tnext[P];
#pragma unroll
    for (int m = 0; m < P; ++m) tnext[m] = ld_ring_if(ring_in + 8u * m, reader);
    // per-step running values of the loop: the ring slot of column s, the stage slots of steps s and s + 1, and where
    // column s - rr's psi and partial moments go
    uint32_t ring_slot = ring_in;
    int sl = 0, sl1 = 1;
    double *out_p = a.out + seg0;   // column s - rr's row segment
    const int mk = SEG >= 16 ? (o < N ? o : N - 1) : 0;   // 16-wide segments: the moment this lane sums
    double *phi_p = phi_base + cell0 * N + mk;
    const long long dphi = dcol * N;
    TC gprev[P];
#pragma unroll
    for (int m = 0; m < P; ++m) gprev[m] = TC(0);

    // Iteration s: the y trace in and the waits (rarely taken); then one basic block: the chain of step s, the
    // wavefront's critical path, beside the transform of step s + 1's inputs, then step s's backward transform, psi and
    // moments, and the copies of step s + D.
    for (int s = 0; s < T; ++s) {
        const bool inrow = row_valid && (unsigned)(s - rr) < (unsigned)nx;
        const bool valid = act && inrow;
        const int cout = s - (Rw - 1);   // the last row's column: its traces go out

        // ---- the y trace in: from the row below (previous step); row 0 from the ring ----
        TC g[P];
#pragma unroll
        for (int m = 0; m < P; ++m) g[m] = __shfl_up_sync(kFullMask, gprev[m], SEG);
        {
            const bool p = reader && s < nx;
            bool wait = cout >= credit && cout < nx;
#pragma unroll
            for (int m = 0; m < P; ++m) wait |= p && __double2hiint(tnext[m]) == (int)(kTraceSentinel >> 32);   // (no quiet NaN has it)
            if (__builtin_expect(__any_sync(kFullMask, wait), 0)) {
                const StepWait<P> w = wait_for_step<P>(ring_slot, p, consumed + 4u, cout, credit, nx, a.error,
                                                       a.spin_limit, lane);
                credit = w.credit;
                if (credit < 0) break;
#pragma unroll
                for (int m = 0; m < P; ++m) tnext[m] = w.v[m];
            }
#pragma unroll
            for (int m = 0; m < P; ++m) st_ring_if(ring_slot + 8u * m, sentinel_value(), p);   // re-arm
        }
#pragma unroll
        for (int m = 0; m < P; ++m) g[m] = (rr == 0) ? TC(tnext[m]) : g[m];

        // ---- the chain of step s, step s + 1's inputs ----
        double srcn[N], stn;
        load_inputs(sl1, spar ^ podd, s2par ^ podd, srcn, stn);
        TC Z[N], fn[P], gout[P];
#pragma unroll
        for (int m = 0; m < P; ++m) fn[m] = f[m];
        modal_step<P, TC, ADJ>(Z, S, fn, g, gout, od, r);
#pragma unroll
        for (int m = 0; m < P; ++m) {
            f[m] = valid ? fn[m] : f[m];
            gprev[m] = gout[m];   // the row below uses it for this column: only if the column is one of the row's
        }
        {   // traces out: each value its own flag
            double *slot = tout + (long long)((cout & tmask) * (long long)tstride);
            const bool p = writer && (unsigned)cout < (unsigned)nx;
#pragma unroll
            for (int m = 0; m < P; ++m) st_trace_if(slot + m, double(gout[m]), p);
        }

        transform(srcn, stn, S, r);   // (step s's are used up)

        // ---- the finish of step s: cell dofs, psi, moments (PHI: the packed modal moments) ----
        {
            TC x[N];
            if constexpr (PHI) {
#pragma unroll
                for (int k = 0; k < N; ++k) x[k] = Z[k];
            } else {
                modal_backward<P, false, false, TC, ADJ>(x, Z);
#pragma unroll
                for (int k = 0; k < N; ++k) x[k] = flip_by(x[k], fmask(k));
            }
            if constexpr (OBUF || SEG >= 16) __syncwarp();   // every lane's reads of the buffers before
            if constexpr (OBUF) {
#pragma unroll
                for (int k = 0; k < N; ++k) obuf[opar + o * N + k] = double(x[k]);
            }
            if constexpr (SEG >= 16) {
#pragma unroll
                for (int k = 0; k < N; ++k) mbuf[k * kMomStride + lane] = double(wv * x[k]);
            }
            if constexpr (OBUF || SEG >= 16) __syncwarp();
            const bool pb = a.out != nullptr && inrow;
            if constexpr (OBUF) {   // the 16-byte chunks of the row segment
                const int body = (seg_n - (int)opar) & ~1;
                const int lim = pb ? body - 2 * o : 0;
                double *dst = out_p;
                const double2 *ov = reinterpret_cast<const double2 *>(obuf + 2 * opar + 2 * o);
#pragma unroll
                for (int h = 0; h < NC; ++h) st_f64x2_if(dst + opar + 2 * o + 2 * SEG * h, ov[SEG * h], lim > 2 * SEG * h);
                if (odd_out) {   // and a first or last double outside them
                    st_f64_if(dst, double(x[0]), pb && o == 0 && opar != 0);
                    st_f64_if(dst + seg_n - 1, double(x[N - 1]), pb && o + 1 == item.q_count && (int)opar + body != seg_n);
                }
            } else if constexpr (!PHI) {
                double *dst = out_p + o * N;
                if constexpr (N == 4) {   // a lane's block is 32 bytes
                    if (out_align == 0) {
                        st_f64x4_if(dst, double(x[0]), double(x[1]), double(x[2]), double(x[3]), pb && act);
                    } else {
#pragma unroll
                        for (int k = 0; k < N; ++k) st_f64_if(dst + k, double(x[k]), pb && act);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < N; ++k) st_f64_if(dst + k, double(x[k]), pb && act);
                }
            }
            // the moments of row rr: sums of the SEG weighted values in fixed trees, one partial per ordinate
            // chunk (added in a fixed order by the reduction kernel: bitwise reproducible).  16-wide segments
            // sum moment k = o from the shared buffer in a pairwise tree over ordinate order (the sequential
            // sum's 15 dependent adds cost 4% of the 256x256 Q2 S16 sweep on B200); narrower ones by a shuffle
            // butterfly (measured on B200: each is the faster one at its width).
            const bool pp = inrow && phi_base != nullptr;
            if constexpr (SEG >= 16) {
                const double2 *mv = reinterpret_cast<const double2 *>(mbuf + mk * kMomStride + rr * SEG);
                double part[SEG / 2];   // a pairwise tree in ordinate order: 4 dependent adds, not 15
#pragma unroll
                for (int h = 0; h < SEG / 2; ++h) {
                    const double2 v = mv[h];
                    part[h] = v.x + v.y;
                }
#pragma unroll
                for (int w = SEG / 4; w >= 1; w /= 2)
#pragma unroll
                    for (int h = 0; h < w; ++h) part[h] = part[2 * h] + part[2 * h + 1];
                st_f64_if(phi_p, part[0], pp && o < N);
            } else {
#pragma unroll
                for (int k = 0; k < N; ++k) x[k] = wv * x[k];
                int lo = 0, hi = N;
                segment_sums<N, SEG>(x, o, &lo, &hi);
#pragma unroll
                for (int i = 0; i < (N + SEG - 1) / SEG; ++i) st_f64_if(phi_p + lo + i, double(x[i]), pp && lo + i < hi);
            }
        }
        // ---- the copies of step s + D, into the stage of step s (read in the last iteration); step s + 2's inputs ----
        prefetch(s + D, sl, spar, s2par);
        cp_wait<D - 2>();
        __syncwarp();   // the other lanes' copies
        sl = sl1;
        sl1 = sl1 + 1 == D ? 0 : sl1 + 1;
        spar ^= podd;
        s2par ^= podd;
        // how far this ring has been read, and its next column
        st_consumed_if(consumed, s + 1, lane == 0 && (s & 3) == 3);
        ring_slot = ring_in + 8u * (uint32_t)(((s + 1) & (kRing - 1)) * V);
#pragma unroll
        for (int m = 0; m < P; ++m) tnext[m] = ld_ring_if(ring_slot + 8u * m, reader && s + 1 < nx);
        opar ^= podd;
        phi_p += dphi;
        out_p += dsoff;
    }
    cp_wait<0>();
}

// BATCHED: the items of several problems in one launch (a batch's problems of one DG degree, FP64 forward
// sweeps); each item names its problem in `table` and carries its index within that problem (`local`: its trace
// row and moment slot, `dep` is local too).  A block copies its item's entry into shared memory; a problem left
// out of the launch (`skip`) has its items return at once.
template <int P, int SEG, bool ADJ, bool SRC2, bool PHI, typename TC, bool BATCHED>
__global__ void __launch_bounds__((kMaxWarps + 1) * 32, 1)
    sweep_lane_kernel(const SweepArgs a, const SweepArgs *__restrict__ table) {
    static_assert(sizeof(SweepArgs) % 8 == 0, "SweepArgs is copied in 8-byte words");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) SweepArgs s_args;   // (batched launches)
    __shared__ int s_item;
    constexpr int N = P * P, Rw = 32 / SEG;
    constexpr size_t RING = ring_doubles(P, SEG), WD = warp_doubles(P, SEG, SRC2, PHI);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = (int)(blockDim.x >> 5) - 1;
    double *base = reinterpret_cast<double *>(smem_raw);
    double *rings = base + (size_t)W * WD;
    double *zero = rings + (size_t)W * RING;
    int *consumed = reinterpret_cast<int *>(zero + (N + 1) / 2 * 2);
    for (int t = threadIdx.x; t < (int)(W * RING); t += blockDim.x) rings[t] = sentinel_value();
    for (int t = threadIdx.x; t < N; t += blockDim.x) zero[t] = 0.0;
    __syncthreads();
    // Both loops meet at two barriers per item: one when every warp is done with the last item, one when the helper
    // has taken the next.
    if (warp == W) {
        for (;;) {
            __syncthreads();
            {
                int it = 0;
                if (lane == 0) {
                    it = atomicAdd(a.next_item, 1);
                    if (ld_relaxed(a.error) != kDevOk || it >= a.n_items) it = -1;
                    s_item = it;
                }
                it = __shfl_sync(kFullMask, it, 0);
                for (int t = lane; t < W; t += 32) consumed[t] = 0;
                if (BATCHED && it >= 0) {
                    const unsigned long long *sw =
                        reinterpret_cast<const unsigned long long *>(table + a.items[it].problem);
                    unsigned long long *dw = reinterpret_cast<unsigned long long *>(&s_args);
                    for (int k = lane; k < (int)(sizeof(SweepArgs) / 8); k += 32) dw[k] = sw[k];
                }
            }
            __syncthreads();
            const int it = s_item;
            if (it < 0) return;
            const SweepItem item = a.items[it];
            const SweepArgs &b = *(BATCHED ? &s_args : &a);
            if (BATCHED && b.skip) continue;
            if (b.quad_mask != 0 && ((b.quad_mask >> item.quadrant) & 1) == 0) continue;
            if (item.dep >= 0 || (b.inflow && !ADJ)) feed_ring<P, SEG>(b, item, saddr(rings), saddr(consumed), lane);
        }
    } else {
        for (;;) {
            __syncthreads();
            __syncthreads();
            const int it = s_item;
            if (it < 0) return;
            const SweepItem item = a.items[it];
            const SweepArgs &b = *(BATCHED ? &s_args : &a);
            if (BATCHED && b.skip) continue;
            if (b.quad_mask != 0 && ((b.quad_mask >> item.quadrant) & 1) == 0) continue;   // another quadrant's launch
            const int row_w = (item.row_block * W + warp) * Rw;
            if (row_w >= b.ny) continue;
            const bool fed = warp > 0 || item.dep >= 0 || (b.inflow && !ADJ);
            run_rows<P, SEG, ADJ, SRC2, PHI, TC>(b, item, BATCHED ? item.local : it, row_w, base + (size_t)warp * WD, zero,
                                                 saddr(rings + (size_t)warp * RING), fed,
                                                 warp + 1 < W ? rings + (size_t)(warp + 1) * RING : nullptr,
                                                 saddr(consumed + warp), lane);
        }
    }
}

template <int P, int SEG, bool ADJ, bool SRC2, bool PHI = false, typename TC = double>
cudaError_t launch(const SweepArgs &args, int grid, cudaStream_t stream) {
    constexpr auto kern = sweep_lane_kernel<P, SEG, ADJ, SRC2, PHI, TC, false>;
    const size_t smem = block_smem_bytes(P, SEG, SRC2, PHI, args.wn);
    cudaError_t e = allow_dynamic_smem<kern>();
    if (e != cudaSuccess) return e;
    kern<<<grid, (args.wn + 1) * 32, smem, stream>>>(args, nullptr);
    return cudaGetLastError();
}

// A batch's FP64 forward sweep, full or moments-only (items of several problems; `table` on the device, one entry per
// problem)
template <int P, int SEG, bool PHI>
cudaError_t launch_batched(const SweepArgs &args, const SweepArgs *table, int grid, cudaStream_t stream) {
    constexpr auto kern = sweep_lane_kernel<P, SEG, false, false, PHI, double, true>;
    const size_t smem = block_smem_bytes(P, SEG, false, PHI, args.wn);
    cudaError_t e = allow_dynamic_smem<kern>();
    if (e != cudaSuccess) return e;
    kern<<<grid, (args.wn + 1) * 32, smem, stream>>>(args, table);
    return cudaGetLastError();
}

// (of the full sweep: the moments-only instance needs less)
template <int P, int SEG>
cudaError_t occupancy_batched(int warps, int *blocks_per_sm) {
    constexpr auto kern = sweep_lane_kernel<P, SEG, false, false, false, double, true>;
    const size_t smem = block_smem_bytes(P, SEG, false, false, warps);
    cudaError_t e = allow_dynamic_smem<kern>();
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kern, (warps + 1) * 32, smem);
}

template <int P, int SEG, bool ADJ, bool SRC2>
cudaError_t occupancy(int warps, int *blocks_per_sm) {
    constexpr auto kern = sweep_lane_kernel<P, SEG, ADJ, SRC2, false, double, false>;
    const size_t smem = block_smem_bytes(P, SEG, SRC2, false, warps);
    cudaError_t e = allow_dynamic_smem<kern>();
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kern, (warps + 1) * 32, smem);
}

}  // namespace lane
}  // namespace idc
