// Forward emitter-wavefield direct sum for sm_100a.
//
// Two kernels share one persistent work-queue skeleton:
//
//  * fwd_split_kernel (IDIWF_SPLIT) — the throughput kernel.  The phase of
//    each emitter/pixel pair is formed in FP64 *in turns* with the per-pixel
//    constant part pre-folded into a magic number, so the last DFMA leaves
//    the fractional turn as 32-bit fixed point in the low word of the double
//    (phase mod 2pi for free).  Its top bit selects the half turn (folded
//    into the sign of the amplitude) and the next 23 bits become an FP32
//    angle in [-pi/2, pi/2); the near-field second-order term, sincos (MUFU), the 1/r
//    factor and the field accumulation run in FP32, two pixels per
//    instruction with Blackwell's packed f32x2 FMA.  Field sums are FP32
//    partials over 64-emitter blocks folded into Kahan-compensated totals.
//
//  * fwd_double_kernel (IDIWF_DOUBLE) — all-FP64, and op-for-op the
//    rounding sequence of the reference CPU kernel
//    (idi/simulation/cpu.py:42-107 as numba/LLVM contracts it), so its
//    fields match the reference to the last bits of sin/cos.
//
// Both stage emitter tiles from HBM to shared memory with bulk asynchronous
// copies (cp.async.bulk, mbarrier completion, double-buffered, bounded
// waits) and broadcast them to all warps; each thread owns a run of
// consecutive pixels along a detector row, so loads of the tile are
// broadcasts and the output stores are contiguous per warp.
//
// Work units are (image, pixel tile); a CTA takes units from an atomic
// counter in the workspace, images ordered by descending emitter count, so
// one launch balances a batch of images with uneven emitter counts.

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <map>
#include <tuple>
#include <mutex>
#include <numeric>
#include <vector>

#include "idiwf_internal.cuh"
#include "nodes.cuh"

namespace idiwf {

// ---------------------------------------------------------------------------
// record layouts
// ---------------------------------------------------------------------------
// split:  r64 double4 {x, y, z, Psi}              (32 B)  Psi = magic + 1/4 + psi/2pi mod 1
//         rA  float4  {x, y, z, -w}               (16 B)  w = |r|^2 (nf) or x^2+y^2
//         rC  float   a                           ( 4 B)
//         (the kernel pairs each value with itself for the f32x2 operations;
//         storing the pairs would cost a fifth shared-memory load per emitter)
// double: r64 double4 {x, y, z, psi}, ra double a
constexpr int kSplitRecBytes = 52;
constexpr int kDoubleRecBytes = 40;
constexpr int kFold = 64;  // emitters per FP32 partial before the Kahan fold

struct SplitRecs {
    double4 *r64;
    float4 *rA;
    float *rC;
    uint32_t *rmax2;  // per image of the launch: max |r|^2 (float bits, rounded up), where there is no node plan
};
struct DoubleRecs {
    double4 *r64;
    double *ra;
};

static inline SplitRecs split_recs(void *ws, int64_t nrec) {
    char *base = static_cast<char *>(ws) + kWsDataOffset;
    SplitRecs r;
    r.r64 = reinterpret_cast<double4 *>(base);
    base += align256(nrec * 32);
    r.rA = reinterpret_cast<float4 *>(base);
    base += align256(nrec * 16);
    r.rC = reinterpret_cast<float *>(base);
    base += align256(nrec * 4);
    r.rmax2 = reinterpret_cast<uint32_t *>(base);
    return r;
}
static inline size_t split_recs_bytes(int64_t nrec) {
    return align256(nrec * 32) + align256(nrec * 16) + align256(nrec * 4) + align256(kMaxImagesPerLaunch * 4);
}
static inline DoubleRecs double_recs(void *ws, int64_t nrec) {
    char *base = static_cast<char *>(ws) + kWsDataOffset;
    DoubleRecs r;
    r.r64 = reinterpret_cast<double4 *>(base);
    base += align256(nrec * 32);
    r.ra = reinterpret_cast<double *>(base);
    return r;
}
static inline size_t double_recs_bytes(int64_t nrec) {
    return align256(nrec * 32) + align256(nrec * 8);
}

// ---------------------------------------------------------------------------
// prep kernels: caller layout (N,4) f64 [+ amplitudes] -> padded tile records
// ---------------------------------------------------------------------------
__device__ __forceinline__ float load_amp(const void *__restrict__ amps, int amp_dtype, int64_t s) {
    if (!amps) return 1.0f;
    return amp_dtype == IDIWF_F32 ? static_cast<const float *>(amps)[s]
                                  : (float)static_cast<const double *>(amps)[s];
}
// Record r of emitter a, its FP64 part relative to `centre`.
__device__ __forceinline__ void split_record(const SplitRecs &rec, int64_t r, const double4 &a, float amp, int w_mode,
                                             double max_abs, uint32_t *err, double cx, double cy, double cz) {
    double psi = a.w * kInvTwoPi;
    psi = psi - rint(psi);
    // the DFMA chain of the kernel starts from this value: the magic
    // binade, +1/4 turn (bit 31 of the fixed-point phase then marks
    // the half turn centred on pi) and +2^-25 turn (rounds instead of
    // truncating to the 23 angle bits the kernel keeps)
    psi = (kTurnMagic + 0.25 + 0x1p-25) + psi;
    if (!(fabs(a.x) <= max_abs && fabs(a.y) <= max_abs && fabs(a.z) <= max_abs)) record_error(err, kErrRange);
    const double w = w_mode == 1 ? (a.x * a.x + a.y * a.y) + a.z * a.z : (w_mode == 2 ? a.x * a.x + a.y * a.y : 0.0);
    // w is stored negated: the kernel forms s^2 - w and subtracts h times it
    rec.r64[r] = make_double4(a.x - cx, a.y - cy, a.z - cz, psi);
    rec.rA[r] = make_float4((float)a.x, (float)a.y, (float)a.z, (float)(-w));
    rec.rC[r] = amp;
}
__device__ __forceinline__ void empty_record(const SplitRecs &rec, int64_t r) {
    rec.r64[r] = make_double4(0, 0, 0, 0);
    rec.rA[r] = make_float4(0, 0, 0, 0);
    rec.rC[r] = 0.0f;
}

// Clears the CTAs' busy times (first launch of a call), by all threads of a prep kernel: a
// memset of its own costs 5 us of a small call.
__device__ __forceinline__ void clear_times(uint64_t *__restrict__ cta_ns) {
    if (!cta_ns) return;
    const int threads = gridDim.x * gridDim.y * blockDim.x;
    for (int i = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; i < kMaxCtas; i += threads) cta_ns[i] = 0;
}

// The CTA's busy time joins the call's (an atomic without a result: nothing waits for it).
__device__ __forceinline__ void add_busy(uint64_t *__restrict__ cta_ns, uint64_t ns) {
    atomicAdd(reinterpret_cast<unsigned long long *>(cta_ns) + blockIdx.x, (unsigned long long)ns);
}

// Sort of the emitters by cell (images cut into cells): counts per block of kCellSort
// emitters, their prefix over the blocks, the first record block (64 emitters) of every
// cell, and the cells' totals.
struct CellSort {
    int *counts;   // [block][kCellMax]; an image's blocks start at (its first emitter / kCellSort) + image
    int *first;    // [image][kCellMax + 1] in blocks of kNodeBlock records
    int *total;    // [image][kCellMax]
};
__device__ __forceinline__ int64_t sort_block0(const BatchParams &bp, int img) {
    return (bp.img[img].src - bp.img[0].src) / kCellSort + img;
}

// Extents of every image and the plan.
__global__ void __launch_bounds__(256)
    node_extents_kernel(const __grid_constant__ BatchParams bp, const double *__restrict__ atoms,
                        const void *__restrict__ amps, int amp_dtype, uint32_t *__restrict__ ext,
                        WsHeader *__restrict__ hdr, const GeomParams g, const NodeGeom ng,
                        NodePlan *__restrict__ plan) {
    const int b = blockIdx.y;
    const ImageDesc d = bp.img[b];
    NodeExtents ex;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < d.n; j += (int64_t)gridDim.x * blockDim.x)
        ex.add(ng, reinterpret_cast<const double4 *>(atoms)[d.src + j], load_amp(amps, amp_dtype, d.src + j));
    ex.raise(ext, b);
    if (last_block(hdr)) plan_nodes(bp, g, ng, ext, false, hdr, plan);
}

// Records.  MAKE_PLAN: the launch has no cells, and where there is a plan it is made here
// (extents on the way, by the block that finishes last); else the plan is given, and
// images cut into cells are written in cell order (stable: the order of an emitter's
// records, and with it the rounding of the sums, does not depend on timing).
template <bool MAKE_PLAN>
__global__ void __launch_bounds__(256)
    prep_split_kernel(const __grid_constant__ BatchParams bp, const double *__restrict__ atoms,
                      const void *__restrict__ amps, int amp_dtype, int w_mode, double max_abs, SplitRecs rec,
                      WsHeader *__restrict__ hdr, const GeomParams g, const NodeGeom ng, uint32_t *__restrict__ ext,
                      NodePlan *__restrict__ plan, CellSort cs, uint64_t *__restrict__ cta_ns) {
    const int b = blockIdx.y, tid = threadIdx.x;
    clear_times(cta_ns);
    const ImageDesc d = bp.img[b];
    const int64_t nrec = (int64_t)d.ntiles * bp.te;
    uint32_t *err = &hdr->error;
    NodeExtents ex;
    if (!MAKE_PLAN && plan->img[b].path == kPathNodes && plan->img[b].ncell > 1) {
        __shared__ int s_at[kCellMax];
        const NodeImage ni = plan->img[b];
        const int nb = (d.n + kCellSort - 1) / kCellSort;
        const int *counts = cs.counts + sort_block0(bp, b) * kCellMax;
        const int *first = cs.first + b * (kCellMax + 1);
        for (int blk = blockIdx.x; blk < nb; blk += gridDim.x) {
            for (int c = tid; c < ni.ncell; c += 256)
                s_at[c] = first[c] * kNodeBlock + counts[(int64_t)blk * kCellMax + c];
            __syncthreads();
            for (int j0 = blk * kCellSort; j0 < min((blk + 1) * kCellSort, d.n); j0 += 256) {
                const int j = j0 + tid;
                const bool in = j < d.n;
                double4 a = make_double4(0, 0, 0, 0);
                int c = -1;
                if (in) {
                    a = reinterpret_cast<const double4 *>(atoms)[d.src + j];
                    c = cell_of(ng, ni, a);
                }
                // rank among the block's earlier emitters of the cell, warp after warp
                const uint32_t same = __match_any_sync(0xffffffffu, c);
                const int lane = tid & 31, rank = __popc(same & ((1u << lane) - 1u));
                int at = 0;
                for (int w = 0; w < 8; ++w) {
                    if ((tid >> 5) == w && in) at = s_at[c] + rank;
                    __syncwarp();
                    if ((tid >> 5) == w && in && rank == 0) s_at[c] += __popc(same);
                    __syncthreads();
                }
                if (in) {
                    double ctr[3];
                    cell_centre(ng, ni, c, ctr);
                    split_record(rec, d.rec + at, a, load_amp(amps, amp_dtype, d.src + j), w_mode, max_abs, err, ctr[0],
                                 ctr[1], ctr[2]);
                }
            }
            __syncthreads();
        }
        // the rest of every cell's last record block
        for (int c = blockIdx.x; c < ni.ncell; c += gridDim.x) {
            const int end = first[c + 1] * kNodeBlock, at = first[c] * kNodeBlock + cs.total[b * kCellMax + c] + tid;
            if (at < end) empty_record(rec, d.rec + at);
        }
        return;
    }
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + tid; j < nrec; j += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = d.rec + j;
        if (j < d.n) {
            const double4 a = reinterpret_cast<const double4 *>(atoms)[d.src + j];
            const float amp = load_amp(amps, amp_dtype, d.src + j);
            if (MAKE_PLAN) ex.add(ng, a, amp);
            split_record(rec, r, a, amp, w_mode, max_abs, err, 0.0, 0.0, 0.0);
        } else {
            empty_record(rec, r);
        }
    }
    if (!MAKE_PLAN) return;
    // without a plan: |r|_max for the pixel-run bound (the caller zeroes it before the launch)
    if (!plan) {
        const uint32_t m = __reduce_max_sync(0xffffffffu, ex.v[0]);
        if ((tid & 31) == 0 && m) atomicMax(&rec.rmax2[b], m);
        return;
    }
    ex.raise(ext, b);
    if (last_block(hdr)) plan_nodes(bp, g, ng, ext, false, hdr, plan);
}

__global__ void __launch_bounds__(256)
    prep_double_kernel(const __grid_constant__ BatchParams bp, const double *__restrict__ atoms,
                       const void *__restrict__ amps, int amp_dtype, DoubleRecs rec, WsHeader *__restrict__ hdr,
                       const GeomParams g, const NodeGeom ng, uint32_t *__restrict__ ext,
                       NodePlan *__restrict__ plan, uint64_t *__restrict__ cta_ns) {
    const int b = blockIdx.y;
    clear_times(cta_ns);
    const ImageDesc d = bp.img[b];
    NodeExtents ex;
    const int64_t nrec = (int64_t)d.ntiles * bp.te;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nrec;
         j += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = d.rec + j;
        if (j < d.n) {
            const int64_t s = d.src + j;
            const double4 a = reinterpret_cast<const double4 *>(atoms)[s];
            rec.r64[r] = a;
            double amp = 1.0;
            if (amps) amp = amp_dtype == IDIWF_F32 ? (double)static_cast<const float *>(amps)[s]
                                                  : static_cast<const double *>(amps)[s];
            rec.ra[r] = amp;
            // (a phase that is not finite goes the way of such an amplitude: the fixed-point
            // sums would lose the NaN that the direct kernel returns)
            if (plan) ex.add(ng, a, isfinite(a.w) ? __double2float_ru(fabs(amp)) : NAN);
        } else {
            rec.r64[r] = make_double4(0, 0, 0, 0);
            rec.ra[r] = 0.0;
        }
    }
    if (!plan) return;
    ex.raise(ext, b);
    if (last_block(hdr)) plan_nodes(bp, g, ng, ext, true, hdr, plan);
}

// ---------------------------------------------------------------------------
// output
// ---------------------------------------------------------------------------
__device__ __forceinline__ void store_pixel(void *out, int out_kind, int64_t idx, double re,
                                            double im) {
    switch (out_kind) {
        case IDIWF_OUT_C128:
            reinterpret_cast<double2 *>(out)[idx] = make_double2(re, im);
            break;
        case IDIWF_OUT_C64:
            reinterpret_cast<float2 *>(out)[idx] = make_float2((float)re, (float)im);
            break;
        case IDIWF_OUT_I64:
            reinterpret_cast<double *>(out)[idx] = re * re + im * im;
            break;
        default:
            reinterpret_cast<float *>(out)[idx] = (float)(re * re + im * im);
            break;
    }
}

// Final per-pixel step of the split forward: the far-field 1/|d| factor, the
// near-field constant phase k (|d| - d_z) (left out of the per-pair sum,
// applied here in FP64 for field outputs), then the store.
template <bool NF, bool SCALE>
__device__ __forceinline__ void finish_pixel_at(const GeomParams &g, int ix, int iy, double re, double im, void *out,
                                                int out_kind, int64_t idx) {
    if ((!NF && SCALE) || (NF && out_kind <= IDIWF_OUT_C64)) {
        double dx, dy, dz;
        pixel_cpu(g, ix, iy, dx, dy, dz);
        const double rho2 = dx * dx + dy * dy;
        const double D = sqrt(rho2 + dz * dz);
        if (!NF && SCALE) {
            re /= D;
            im /= D;
        }
        if (NF && out_kind <= IDIWF_OUT_C64) {
            const double c = g.kp * (dz > 0 ? rho2 / (D + dz) : D - dz);
            double sn, cs;
            sincospi(2.0 * (c - rint(c)), &sn, &cs);
            const double r2 = re * cs - im * sn;
            im = re * sn + im * cs;
            re = r2;
        }
    }
    store_pixel(out, out_kind, idx, re, im);
}
template <bool NF, bool SCALE>
__device__ __forceinline__ void finish_pixel(const GeomParams &g, int p, double re, double im, void *out,
                                             int out_kind, int64_t idx) {
    const int ix = p / g.ny;
    finish_pixel_at<NF, SCALE>(g, ix, p - ix * g.ny, re, im, out, out_kind, idx);
}

// Sum of the emitter-chunk partials of every pixel, in chunk order, then the
// final per-pixel step.  partials: [ksplit][n_images][npix] double2.
template <bool NF, bool SCALE>
__global__ void fwd_finish_kernel(const GeomParams g, const double2 *__restrict__ partials, int ksplit,
                                  int n_images, void *__restrict__ out, int out_kind,
                                  const NodePlan *__restrict__ plan) {
    const int npix = g.nx * g.ny;
    const int64_t total = (int64_t)n_images * npix;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        if (plan && plan->img[t / npix].path == kPathNodes) continue;
        double re = 0.0, im = 0.0;
        for (int c = 0; c < ksplit; ++c) {
            const double2 v = partials[(int64_t)c * total + t];
            re += v.x;
            im += v.y;
        }
        finish_pixel<NF, SCALE>(g, (int)(t % npix), re, im, out, out_kind, t);
    }
}

// ---------------------------------------------------------------------------
// split-precision kernel
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// Constants of a run's base angle with the 8 low fixed-point bits, in units
// of pi_f = FP32 pi as in the per-pixel path: C is -pi_f (1.5 + 2^-8 + 2^-24)
// rounded to FP32 and S = pi_f 2^-8 minus C's rounding error, so that C + S
// is exact up to the FP32 rounding of S (< 5e-10 rad).
constexpr double kPiF = (double)3.14159274f;
constexpr double kRunBaseCExact = -kPiF * (1.5 + 1.0 / 256.0 + 1.0 / 16777216.0);
constexpr float kRunBaseC = (float)kRunBaseCExact;
constexpr float kRunBaseS = (float)(kPiF / 256.0 - ((double)kRunBaseC - kRunBaseCExact));

// Base point of run b of the thread whose first pixel is p0: the middle of
// the aligned run (rows hold a whole number of runs when runs are in use).
__device__ __forceinline__ PixelDir run_base(const GeomParams &g, int p0, int b, int npix) {
    const int rs = min((p0 & ~(kRun - 1)) + kRun * b, npix - kRun);
    const int ix = rs / g.ny;
    return pixel_dir(g, (double)ix, (double)(rs - ix * g.ny) + 0.5 * (kRun - 1));
}

// One work unit (image, pixel tile[, emitter chunk]) of the split kernel.
//
// PATH = kPathPixel: every pixel forms its phase with its own FP64 DFMA chain;
//   the near-field term h (|r|^2 - s^2), h = k / (2|d|), is added in FP32.
// PATH = kPathRuns: one FP64 chain per run of kRun pixels forms the phase at the
//   middle of the run (fixed point, half-turn fold as below); pixel i adds the
//   FP32 offset D_i . r with D_i = 2 pi (nq_i - nq_base) = -k (d_hat_i -
//   d_hat_base), exact up to FP32 rounding because |D_i . r| <= kGroupMaxPhase
//   (checked per image by the caller).  The near-field term uses
//   s_i = d_hat_i . r = s_base - D_i.r / k.  The half-turn sign of the base
//   applies to the whole run.
// PATH = kPathExact (near field only): as kPathPixel, but the quadratic term
//   k r_perp^2 / (2|d|) joins the FP64 chain (s = d_hat . r recovered from the
//   chain as z - (t - Psi)/kp, so r_perp^2 = |r|^2 - s^2 in FP64), and the
//   exact remainder R = h N (2s - N), N = r_perp^2 / (|d| + |d - r| - s), is
//   added in FP32 (|d - r| from a reciprocal square root, which also gives the
//   "scale" factor 1/|d - r|).
// Returns true when a bounded wait gave up (the unit is abandoned).
template <int PPT, bool NF, bool SCALE, bool SECOND, bool CHUNKED, int PATH>
__device__ __forceinline__ bool split_unit(const BatchParams &bp, const GeomParams &g, const SplitRecs &rec,
                                           void *__restrict__ out, int out_kind, WsHeader *__restrict__ hdr,
                                           double2 *__restrict__ partials, unsigned char *smem, uint64_t *bar,
                                           int *s_abort, uint32_t &issued, uint32_t &consumed, int img,
                                           int chunk, const ImageDesc &d, int p0, int tbeg, int tend,
                                           float *__restrict__ kahan) {
    constexpr bool GROUP = PATH == kPathRuns;
    constexpr bool EXACT = PATH == kPathExact;
    static_assert(!EXACT || NF, "the exact path is a near-field path");
    constexpr int PH = PPT / 2;
    constexpr int NB = PPT >= kRun ? PPT / kRun : 1;  // runs (base phases) per thread
    constexpr int NQ = GROUP ? NB : PPT;
    const int tid = threadIdx.x;
    const int TE = bp.te;
    const uint32_t stage_bytes = (uint32_t)TE * kSplitRecBytes;
    const int npix = g.nx * g.ny;
    const float2 PI2 = f2(3.14159274f, 3.14159274f);
    const float2 NEG_15PI2 = f2(-4.71238898f, -4.71238898f);

    // ---- per-pixel constants (FP64 geometry) ----
    // cx/cy/cz: d_hat of each pixel, or (GROUP) its offset coefficients D_i
    // (EXACT) hq: the quadratic term's FP64 coefficient kp / (2|d|) in turns,
    // dd: |d| in FP32
    double nqx[NQ], nqy[NQ], nqz[NQ], hq[EXACT ? PPT : 1];
    float2 cx[PH], cy[PH], cz[PH], hh[PH], iD[PH], iD2[PH], dd[EXACT ? PH : 1];
    float dbx[NB], dby[NB], dbz[NB];
    PixelDir base[NB];
    if (GROUP) {
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            base[b] = run_base(g, p0, b, npix);
            nqx[b] = base[b].nqx;
            nqy[b] = base[b].nqy;
            nqz[b] = base[b].nqz;
            dbx[b] = (float)base[b].ux;
            dby[b] = (float)base[b].uy;
            dbz[b] = (float)base[b].uz;
        }
    }
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
        const int p = min(p0 + i, npix - 1);
        const int ix = p / g.ny, iy = p - ix * g.ny;
        const PixelDir q = pixel_dir(g, (double)ix, (double)iy);
        float fx, fy, fz;
        if (GROUP) {
            const PixelDir &bs = base[PPT >= kRun ? i / kRun : 0];
            fx = (float)(kTwoPi * (q.nqx - bs.nqx));
            fy = (float)(kTwoPi * (q.nqy - bs.nqy));
            fz = (float)(kTwoPi * (q.nqz - bs.nqz));
        } else {
            nqx[i] = q.nqx;
            nqy[i] = q.nqy;
            nqz[i] = q.nqz;
            fx = (float)q.ux;
            fy = (float)q.uy;
            fz = (float)q.uz;
        }
        const float fh = (float)(-g.k * 0.5 * q.invD);  // -h, pairs with the negated w
        const float fi = (float)q.invD, fi2 = (float)(q.invD * q.invD);
        float fd = 0.f;
        if (EXACT) {
            hq[i] = 0.5 * g.kp * q.invD;
            fd = (float)(1.0 / q.invD);
        }
        if (i & 1) {
            cx[i / 2].y = fx; cy[i / 2].y = fy; cz[i / 2].y = fz;
            hh[i / 2].y = fh; iD[i / 2].y = fi; iD2[i / 2].y = fi2;
            if (EXACT) dd[i / 2].y = fd;
        } else {
            cx[i / 2].x = fx; cy[i / 2].x = fy; cz[i / 2].x = fz;
            hh[i / 2].x = fh; iD[i / 2].x = fi; iD2[i / 2].x = fi2;
            if (EXACT) dd[i / 2].x = fd;
        }
    }
    const float ninvk = (float)(-1.0 / g.k);
    const float2 NEG_INVK2 = f2(ninvk, ninvk);

    // Kahan-compensated totals per pixel (sum, compensation; re, im).  The run
    // kernel keeps them in shared memory, [4 PPT][threads] (touched once per
    // kFold emitters), to leave its registers to the emitter loop.
    float sre[GROUP ? 1 : PPT], cre[GROUP ? 1 : PPT], sim[GROUP ? 1 : PPT], cim[GROUP ? 1 : PPT];
    const int nthr = blockDim.x;
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
        if (GROUP) {
#pragma unroll
            for (int c = 0; c < 4; ++c) kahan[(c * PPT + i) * nthr + tid] = 0.0f;
        } else {
            sre[i] = cre[i] = sim[i] = cim[i] = 0.0f;
        }
    }

    const int nt = tend - tbeg;
    if (tid == 0) {
        for (int s = 0; s < 2 && s < nt; ++s) {
            const uint32_t slot = issued & 1;
            unsigned char *st = smem + slot * stage_bytes;
            const int64_t r0 = d.rec + (int64_t)(tbeg + s) * TE;
            mbar_arrive_expect_tx(&bar[slot], stage_bytes);
            bulk_g2s(st, rec.r64 + r0, TE * 32, &bar[slot]);
            bulk_g2s(st + TE * 32, rec.rA + r0, TE * 16, &bar[slot]);
            bulk_g2s(st + TE * 48, rec.rC + r0, TE * 4, &bar[slot]);
            ++issued;
        }
    }
    for (int it = 0; it < nt; ++it) {
        const uint32_t slot = consumed & 1;
        if (!mbar_wait_bounded(&bar[slot], (consumed >> 1) & 1)) {
            record_error(&hdr->error, kErrTimeout);
            *s_abort = 1;
        }
        const unsigned char *st = smem + slot * stage_bytes;
        const double4 *s64 = reinterpret_cast<const double4 *>(st);
        const float4 *sA = reinterpret_cast<const float4 *>(st + TE * 32);
        const float *sC = reinterpret_cast<const float *>(st + TE * 48);

        for (int jb = 0; jb < TE; jb += kFold) {
            float2 are[PH], aim[PH];
#pragma unroll
            for (int q = 0; q < PH; ++q) are[q] = aim[q] = f2(0.f, 0.f);
            if (GROUP) {
#pragma unroll(PPT <= 4 ? 4 : 2)
                for (int j = jb; j < jb + kFold; ++j) {
                    const double4 r = s64[j];
                    const float4 A = sA[j];
                    const float a1 = sC[j];
                    const float2 X2 = f2(A.x, A.x), Y2 = f2(A.y, A.y), Z2 = f2(A.z, A.z);
                    float2 XB2[NB], AS2[NB], SB2[NB];
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        double t = __fma_rn(nqx[b], r.x, r.w);
                        t = __fma_rn(nqy[b], r.y, t);
                        t = __fma_rn(nqz[b], r.z, t);
                        const uint32_t lo = (uint32_t)__double2loint(t);
                        // base angle and half-turn sign as in the per-pixel path below,
                        // plus the 8 fixed-point bits below the 23 kept there:
                        // pi u + C + (1 + r 2^-23) S = pi (u - 1.5) + pi r 2^-31 - pi 2^-24
                        // (the last term takes back the record's half-step rounding offset)
                        float xb = __fmaf_rn(__uint_as_float(((lo >> 8) & 0x007FFFFFu) | 0x3F800000u),
                                             PI2.x, kRunBaseC);
                        xb = __fmaf_rn(__uint_as_float((lo & 0xFFu) | 0x3F800000u), kRunBaseS, xb);
                        const float as = __uint_as_float(__float_as_uint(a1) ^ (lo & 0x80000000u));
                        XB2[b] = f2(xb, xb);
                        AS2[b] = f2(as, as);
                        SB2[b] = f2(0.f, 0.f);
                        if (NF) {
                            const float sb = __fmaf_rn(dbz[b], A.z, __fmaf_rn(dby[b], A.y, __fmul_rn(dbx[b], A.x)));
                            SB2[b] = f2(sb, sb);
                        }
                    }
#pragma unroll
                    for (int q = 0; q < PH; ++q) {
                        const int b = PPT >= kRun ? q / (kRun / 2) : 0;
                        float2 dl = __fmul2_rn(cx[q], X2);
                        dl = __ffma2_rn(cy[q], Y2, dl);
                        dl = __ffma2_rn(cz[q], Z2, dl);
                        float2 amp = AS2[b];
                        if (NF) {
                            const float2 s = __ffma2_rn(dl, NEG_INVK2, SB2[b]);
                            const float2 w2 = __ffma2_rn(s, s, f2(A.w, A.w));
                            dl = __ffma2_rn(hh[q], w2, dl);
                            if (SCALE) amp = __fmul2_rn(AS2[b], __ffma2_rn(s, iD2[q], iD[q]));
                        } else if (SECOND) {
                            dl = __ffma2_rn(hh[q], f2(A.w, A.w), dl);  // (-h)(-(x^2+y^2))
                        }
                        const float2 arg = __fadd2_rn(XB2[b], dl);
                        float s0, c0, s1, c1;
                        __sincosf(arg.x, &s0, &c0);
                        __sincosf(arg.y, &s1, &c1);
                        are[q] = __ffma2_rn(amp, f2(c0, c1), are[q]);
                        aim[q] = __ffma2_rn(amp, f2(s0, s1), aim[q]);
                    }
                }
            } else {
#pragma unroll(PPT <= 4 ? 4 : 2)
                for (int j = jb; j < jb + kFold; ++j) {
                    const double4 r = s64[j];
                    const float4 A = sA[j];
                    const float a1 = sC[j];
                    const float2 a2 = f2(a1, a1);
                    double rr = 0.0;  // (EXACT) |r|^2 in FP64
                    if (EXACT) rr = __fma_rn(r.z, r.z, __fma_rn(r.y, r.y, r.x * r.x));
#pragma unroll
                    for (int q = 0; q < PH; ++q) {
                        uint32_t lo[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int i = 2 * q + e;
                            double t = __fma_rn(nqx[i], r.x, r.w);
                            t = __fma_rn(nqy[i], r.y, t);
                            t = __fma_rn(nqz[i], r.z, t);
                            if (EXACT) {
                                // t - Psi = nq . r = kp (z - s) exactly (same binade)
                                const double sd = __fma_rn(-g.ikp, t - r.w, r.z);
                                t = __fma_rn(hq[i], __fma_rn(-sd, sd, rr), t);
                            }
                            lo[e] = (uint32_t)__double2loint(t);
                        }
                        // phase = n*pi + x, x = pi*(u - 1.5) in [-pi/2, pi/2): u from
                        // bits 30..8; odd n (bit 31) negates the term, folded into
                        // the amplitude's sign.  Mapping both halves of the circle
                        // onto one half and flipping the sign makes the mean error
                        // of the hardware cosine cancel over the circle instead of
                        // adding up coherently over emitters.
                        const float2 u = f2(__uint_as_float(((lo[0] >> 8) & 0x007FFFFFu) | 0x3F800000u),
                                            __uint_as_float(((lo[1] >> 8) & 0x007FFFFFu) | 0x3F800000u));
                        float2 arg = __ffma2_rn(u, PI2, NEG_15PI2);
                        float2 amp = a2;
                        if (NF) {
                            float2 s = __fmul2_rn(cx[q], f2(A.x, A.x));
                            s = __ffma2_rn(cy[q], f2(A.y, A.y), s);
                            s = __ffma2_rn(cz[q], f2(A.z, A.z), s);
                            const float2 w2 = __ffma2_rn(s, s, f2(A.w, A.w));  // s^2 - |r|^2
                            if (EXACT) {
                                // L^2 = |d|(|d| - 2s) + |r|^2, N = r_perp^2 / (|d| + L - s),
                                // R = h N (2s - N) = (-h)(-N)(2s - N)
                                const float2 l2 = __ffma2_rn(__ffma2_rn(s, f2(-2.f, -2.f), dd[q]), dd[q],
                                                             f2(-A.w, -A.w));
                                const float2 y = f2(rsqrt_approx(l2.x), rsqrt_approx(l2.y));
                                const float2 den = __ffma2_rn(s, f2(-1.f, -1.f), __ffma2_rn(l2, y, dd[q]));
                                const float2 nN = __fmul2_rn(w2, f2(rcp_approx(den.x), rcp_approx(den.y)));
                                arg = __ffma2_rn(__fmul2_rn(hh[q], nN), __ffma2_rn(s, f2(2.f, 2.f), nN), arg);
                                if (SCALE) amp = __fmul2_rn(a2, y);
                            } else {
                                // -h (s^2 - |r|^2) = h (|r|^2 - s^2)
                                arg = __ffma2_rn(hh[q], w2, arg);
                                if (SCALE) amp = __fmul2_rn(a2, __ffma2_rn(s, iD2[q], iD[q]));
                            }
                        } else if (SECOND) {
                            arg = __ffma2_rn(hh[q], f2(A.w, A.w), arg);  // (-h)(-(x^2+y^2))
                        }
                        amp.x = __uint_as_float(__float_as_uint(amp.x) ^ (lo[0] & 0x80000000u));
                        amp.y = __uint_as_float(__float_as_uint(amp.y) ^ (lo[1] & 0x80000000u));
                        float s0, c0, s1, c1;
                        __sincosf(arg.x, &s0, &c0);
                        __sincosf(arg.y, &s1, &c1);
                        are[q] = __ffma2_rn(amp, f2(c0, c1), are[q]);
                        aim[q] = __ffma2_rn(amp, f2(s0, s1), aim[q]);
                    }
                }
            }
            // Kahan fold of the block partials
#pragma unroll
            for (int q = 0; q < PH; ++q) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int i = 2 * q + e;
                    const float pr = e ? are[q].y : are[q].x;
                    const float pi = e ? aim[q].y : aim[q].x;
                    if (GROUP) {
                        float *k0 = kahan + (0 * PPT + i) * nthr + tid, *k1 = kahan + (1 * PPT + i) * nthr + tid;
                        float *k2 = kahan + (2 * PPT + i) * nthr + tid, *k3 = kahan + (3 * PPT + i) * nthr + tid;
                        const float s0 = *k0, c0 = *k1, s1 = *k2, c1 = *k3;
                        float y = pr - c0;
                        float t = s0 + y;
                        *k1 = (t - s0) - y;
                        *k0 = t;
                        y = pi - c1;
                        t = s1 + y;
                        *k3 = (t - s1) - y;
                        *k2 = t;
                    } else {
                        float y = pr - cre[i];
                        float t = sre[i] + y;
                        cre[i] = (t - sre[i]) - y;
                        sre[i] = t;
                        y = pi - cim[i];
                        t = sim[i] + y;
                        cim[i] = (t - sim[i]) - y;
                        sim[i] = t;
                    }
                }
            }
        }
        ++consumed;
        __syncthreads();
        if (*s_abort) return true;
        if (tid == 0 && it + 2 < nt) {
            const uint32_t slot2 = issued & 1;
            unsigned char *st2 = smem + slot2 * stage_bytes;
            const int64_t r0 = d.rec + (int64_t)(tbeg + it + 2) * TE;
            mbar_arrive_expect_tx(&bar[slot2], stage_bytes);
            bulk_g2s(st2, rec.r64 + r0, TE * 32, &bar[slot2]);
            bulk_g2s(st2 + TE * 32, rec.rA + r0, TE * 16, &bar[slot2]);
            bulk_g2s(st2 + TE * 48, rec.rC + r0, TE * 4, &bar[slot2]);
            ++issued;
        }
    }

    const int64_t obase = (int64_t)img * npix;
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
        const int p = p0 + i;
        if (p < npix) {
            double re, im;
            if (GROUP) {
                re = (double)kahan[(0 * PPT + i) * nthr + tid] - (double)kahan[(1 * PPT + i) * nthr + tid];
                im = (double)kahan[(2 * PPT + i) * nthr + tid] - (double)kahan[(3 * PPT + i) * nthr + tid];
            } else {
                re = (double)sre[i] - (double)cre[i];
                im = (double)sim[i] - (double)cim[i];
            }
            if (CHUNKED)
                partials[((int64_t)chunk * bp.n_images + img) * npix + p] = make_double2(re, im);
            else
                finish_pixel<NF, SCALE>(g, p, re, im, out, out_kind, obase + p);
        }
    }
    return false;
}

// The split forward is up to three kernels launched back to back, one per
// path (split_path: pixel runs, per-pixel FP64 phase, exact near field), each
// taking the units of its own images from its own work counter.  Without the
// per-pixel path's registers the run kernel fits three 256-thread CTAs per SM
// (two for the others).  A kernel whose path no image of the launch takes
// returns at once.  The per-pixel kernel, which every launch runs, reports
// images outside the split kernels' range (kErrGeometry); no kernel takes them.
// Every CTA classifies the images once, into shared memory: a square root or
// the classifier's arithmetic in the persistent loop costs the run kernel
// several percent of its speed.
template <int PPT, bool NF, bool SCALE, bool SECOND, bool CHUNKED, int PATH>
__global__ void __launch_bounds__(256, (PPT <= 4 ? (PATH == kPathRuns ? 3 : 2) : 1))
    fwd_split_kernel(const __grid_constant__ BatchParams bp, const GeomParams g, SplitRecs rec,
                     void *__restrict__ out, int out_kind, WsHeader *__restrict__ hdr,
                     uint64_t *__restrict__ cta_ns, double2 *__restrict__ partials,
                     const NodePlan *__restrict__ plan) {
    static_assert(PPT % 2 == 0, "pixels are processed in f32x2 pairs");
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ int s_unit, s_abort;
    __shared__ uint8_t s_path[kMaxImagesPerLaunch];

    const int tid = threadIdx.x;
    bool mine = false;
    for (int i = tid; i < bp.n_images; i += blockDim.x) {
        const int path = plan ? plan->img[i].path : split_path(g, rec.rmax2[i], bp.groups != 0, false);
        s_path[i] = (uint8_t)path;
        mine |= path == PATH;
        if (PATH == kPathPixel && path == kPathReject && blockIdx.x == 0) record_error(&hdr->error, kErrGeometry);
    }
    if (!__syncthreads_or(mine)) return;
    uint32_t *counter = PATH == kPathRuns ? &hdr->work_counter
                                          : (PATH == kPathPixel ? &hdr->work_counter2 : &hdr->work_counter3);

    const uint64_t t_start = globaltimer_ns();
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        s_abort = 0;
        mbar_fence_init();
        if (blockIdx.x == 0) atomicMax(&hdr->n_ctas, gridDim.x);
    }
    __syncthreads();

    const int tile_px = blockDim.x * PPT;
    uint32_t issued = 0, consumed = 0;
    bool aborted = false;

    const int ks = CHUNKED ? bp.ksplit : 1;
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            // next unit of this kernel's path (units of the other kernel are
            // skipped here, out of the CTA's control flow)
            int u;
            for (;;) {
                u = (int)atomicAdd(counter, 1u);
                if (u >= bp.total_units || s_path[bp.order[u / ks / bp.tiles_per_image]] == PATH) break;
            }
            s_unit = u;
        }
        __syncthreads();
        const int unit = s_unit;
        if (unit >= bp.total_units) break;
        const int chunk = unit % ks;
        const int pu = unit / ks;
        const int img = bp.order[pu / bp.tiles_per_image];
        const int ptile = pu % bp.tiles_per_image;
        const ImageDesc d = bp.img[img];
        const int p0 = ptile * tile_px + tid * PPT;
        // emitter tiles of this unit: the whole image, or one chunk of it
        const int tbeg = CHUNKED ? min(chunk * d.tpc, d.ntiles) : 0;
        const int tend = CHUNKED ? min(tbeg + d.tpc, d.ntiles) : d.ntiles;
        if (split_unit<PPT, NF, SCALE, SECOND, CHUNKED, PATH>(
                bp, g, rec, out, out_kind, hdr, partials, smem, bar, &s_abort, issued, consumed, img, chunk, d, p0,
                tbeg, tend, reinterpret_cast<float *>(smem + 2 * (size_t)bp.te * kSplitRecBytes))) {
            aborted = true;
            break;
        }
    }
    if (aborted) {
        // wait (bounded) for copies still in flight into this CTA's shared memory
        if (tid == 0)
            while (consumed < issued) {
                mbar_wait_bounded(&bar[consumed & 1], (consumed >> 1) & 1);
                ++consumed;
            }
        return;
    }
    if (tid == 0) add_busy(cta_ns, globaltimer_ns() - t_start);
}

// ---------------------------------------------------------------------------
// band-limited evaluation: node sums, weights, interpolation
// ---------------------------------------------------------------------------
// Node sums of the images [img0, img1) on kPathNodes, as the split kernel's
// per-pixel path (FP64 phase per pair, second-order near field) at the nodes'
// fractional pixel positions.
//
// Work is tiles of kNodeTile nodes x blocks of 64 emitters (of each cell in turn); the CTAs
// that fit (six 128-thread CTAs per SM) each take an equal, contiguous share of it, so
// the shares end together and a CTA sets up a tile's geometry once or twice per cell.  The FP32
// sums of 16 emitters are added to fixed-point totals (64-bit integers, the image's
// power of two as the unit's inverse, below 2^-58 of the largest possible sum), which
// go to the node accumulators by atomics: integer sums do not depend on how
// the work was cut, so results stay the same from run to run and from batch to batch.
//
// A node sum stands for many pixels, so it is formed more exactly than the direct
// kernels' pixels: polynomial sine and cosine, and short FP32 partials.
//
// FINE (complex128 fields, which differentiation reads): the residuals of a fit are
// differences of nearly equal intensities, and where the direct kernels' rounding errors
// average out over the pixels, a node's error reaches all of them.  So the sine, cosine
// and sums are FP64 polynomials and FP64 additions (a block of 64 emitters each), and cells
// are turned in FP64 as well: intensities to 1.2e-9 of 64-bit ones instead of 9e-8, and
// gradients of residuals a hundredth of them to 1.9e-7 instead of 1e-6 (7e-6 on the direct
// path).  36 cycles of the FP64 pipe per pair of a warp; 1.5 times the FP32 form's time,
// which the other outputs keep; the fit of 10,000 emitters on 512^2 pixels 0.98 ms either
// way.

// Buffers of one group of images: sums on the target grid and of the cells (fixed point),
// interpolation weights of both axes, from the target grid to the pixels and from the
// cells' grid to the target's, the cells' sums interpolated along y, and the intermediate
// W[j][a] = sum_b L_y[j][b] V[a][b] (pixel columns x nodes along x).
struct NodeBuffers {
    double2 *v, *f, *y;  // [image of the group][entries]
    NodeCaps caps;
    int two_words;       // FP64: f holds the second words of v
    double *lx, *ly;     // [image of the group][nx or ny][n0 or n1]
    double *sx, *sy;     // [image of the group][n0 or n1][g0 or g1]
    double2 *w;          // [image of the group][ny][n0]
    int64_t lx_stride, ly_stride, w_stride, sx_stride, sy_stride;
};

// Work of the images [img0, img0 + nimg), prefixed in s_w0 (nimg + 1 entries), by one block of
// kNodeThreads threads.
__device__ __forceinline__ void image_work(const NodePlan *__restrict__ plan, int img0, int nimg, long long *s_w0) {
    __shared__ long long s_sum[kNodeThreads / 32];
    const int tid = threadIdx.x;
    long long base = 0;
    for (int i0 = 0; i0 < nimg; i0 += kNodeThreads) {
        const int i = i0 + tid;
        long long w = 0;
        if (i < nimg) {
            const NodeImage &ni = plan->img[img0 + i];
            w = (long long)ni.ntiles * ni.nblk;
        }
        long long x = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, x, o);
            if ((tid & 31) >= o) x += y;
        }
        if ((tid & 31) == 31) s_sum[tid >> 5] = x;
        __syncthreads();
        long long before = base;
        for (int k = 0; k < kNodeThreads / 32; ++k) {
            before += k < (tid >> 5) ? s_sum[k] : 0;
            base += s_sum[k];
        }
        if (i < nimg) s_w0[i] = before + x - w;
        __syncthreads();
    }
    if (tid == 0) s_w0[nimg] = base;
    __syncthreads();
}

// sin(pi x) / x and (cos(pi x) - 1) / x^2 in x^2, |x| <= 0.52: interpolated at the
// Chebyshev nodes of the range (errors of the sine and cosine 4.4e-11 and 1.4e-9).
__constant__ double kSinPi[6] = {-0.007001047169005128, 0.08203438769606762, -0.599248953113932,
                                 2.550163054613202,     -5.1677127572353685, 3.141592653504127};
__constant__ double kCosPi[5] = {-0.0245331199113542, 0.23503154851442468, -1.3352339849656298, 4.058711155030214,
                                 -4.934802195292975};
__device__ __forceinline__ void sincospi64(double x, double &sn, double &cs) {
    const double z = x * x;
    double p = kSinPi[0], q = kCosPi[0];
#pragma unroll
    for (int i = 1; i < 6; ++i) p = __fma_rn(p, z, kSinPi[i]);
#pragma unroll
    for (int i = 1; i < 5; ++i) q = __fma_rn(q, z, kCosPi[i]);
    sn = p * x;
    cs = __fma_rn(q, z, 1.0);
}
// The half-turn angle of half_turns2 with all its bits: x = bits 30..0 / 2^31 - 1/2 - 2^-24.
__device__ __forceinline__ double half_turn64(uint32_t w) {
    return __hiloint2double(0x41400000, (int)(w & 0x7FFFFFFFu)) - (0x1p21 + 0.5 + 0x1p-24);
}
__device__ __forceinline__ double flip_sign64(double x, uint32_t w) {
    return __hiloint2double(__double2hiint(x) ^ (int)(w & 0x80000000u), __double2loint(x));
}

constexpr int kNodeFold = 16;
template <bool NF, bool SCALE, bool SECOND, bool FINE>
__global__ void __launch_bounds__(kNodeThreads, 6)
    node_sum_kernel(const __grid_constant__ BatchParams bp, const GeomParams g, SplitRecs rec,
                    const NodePlan *__restrict__ plan, NodeBuffers nb, const int *__restrict__ first,
                    WsHeader *__restrict__ hdr, uint64_t *__restrict__ cta_ns, int img0, int img1) {
    constexpr int PPT = kNodePPT, PH = PPT / 2;
    constexpr uint32_t kStage = kNodeTE * kSplitRecBytes;
    __shared__ __align__(128) unsigned char smem[2 * kStage];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ int s_abort;
    __shared__ long long s_w0[kMaxImagesPerLaunch + 1];
    const int tid = threadIdx.x;
    const uint64_t t_start = globaltimer_ns();
    const int nimg = img1 - img0;
    image_work(plan, img0, nimg, s_w0);
    const int64_t wend = s_w0[nimg];
    if (wend == 0) return;
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        s_abort = 0;
        mbar_fence_init();
        if (blockIdx.x == 0) atomicMax(&hdr->n_ctas, gridDim.x);
    }
    __syncthreads();
    int64_t pos = wend * blockIdx.x / gridDim.x;
    const int64_t end = wend * (blockIdx.x + 1) / gridDim.x;
    uint32_t issued = 0, consumed = 0;
    int img = -1, seg = 0;
    NodeImage ni;
    while (pos < end) {
        if (img < 0 || pos >= s_w0[img - img0 + 1]) {
            int lo = 0, hi = nimg;  // last image with w0 <= pos (those without work share the next one's w0)
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (s_w0[mid] <= pos) lo = mid;
                else hi = mid;
            }
            img = img0 + lo;
            ni = plan->img[img];
            seg = -1;
        }
        const ImageDesc d = bp.img[img];
        const int64_t rel = pos - s_w0[img - img0];
        // the cell: blocks [f0, f1) of the image's records
        int f0 = 0, f1 = ni.nblk;
        if (ni.ncell > 1) {
            const int *fs = first + img * (kCellMax + 1);
            const int at = (int)(rel / ni.ntiles);  // record block of the position
            if (seg < 0 || fs[seg + 1] > at) {
                int lo = 0, hi = ni.ncell;
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (fs[mid] <= at) lo = mid;
                    else hi = mid;
                }
                seg = lo;
            } else {
                while (fs[seg + 1] <= at) ++seg;
            }
            f0 = fs[seg];
            f1 = fs[seg + 1];
        } else {
            seg = 0;
        }
        const int tile = (int)((rel - (int64_t)f0 * ni.ntiles) / (f1 - f0));
        const int b0 = f0 + (int)((rel - (int64_t)f0 * ni.ntiles) % (f1 - f0));
        const int b1 = (int)min((int64_t)f1, b0 + (end - pos));
        pos += b1 - b0;
        const int nodes = ni.g0 * ni.g1;
        const int len = (b1 - b0) * kNodeBlock, nt = (len + kNodeTE - 1) / kNodeTE;
        auto issue = [&](int t) {
            const uint32_t slot = issued & 1;
            unsigned char *st = smem + slot * kStage;
            const int cnt = min(kNodeTE, len - t * kNodeTE);  // a multiple of kNodeBlock
            const int64_t r0 = d.rec + (int64_t)b0 * kNodeBlock + (int64_t)t * kNodeTE;
            mbar_arrive_expect_tx(&bar[slot], cnt * kSplitRecBytes);
            bulk_g2s(st, rec.r64 + r0, cnt * 32, &bar[slot]);
            bulk_g2s(st + kNodeTE * 32, rec.rA + r0, cnt * 16, &bar[slot]);
            bulk_g2s(st + kNodeTE * 48, rec.rC + r0, cnt * 4, &bar[slot]);
            ++issued;
        };
        if (tid == 0)
            for (int t = 0; t < 2 && t < nt; ++t) issue(t);

        const int m0 = tile * kNodeTile + tid * PPT;
        double nqx[PPT], nqy[PPT], nqz[PPT];
        float2 cx[PH], cy[PH], cz[PH], hh[PH], iD[PH], iD2[PH];
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
            const int m = min(m0 + i, nodes - 1);
            const int a = m / ni.g1, b = m - a * ni.g1;
            const PixelDir q = pixel_dir(g, node_index(ni.g0, a, g.nx), node_index(ni.g1, b, g.ny));
            nqx[i] = q.nqx;
            nqy[i] = q.nqy;
            nqz[i] = q.nqz;
            // -h in half turns, pairs with the negated w
            const float fx = (float)q.ux, fy = (float)q.uy, fz = (float)q.uz, fh = (float)(-g.kp * q.invD);
            const float fi = (float)q.invD, fi2 = (float)(q.invD * q.invD);
            if (i & 1) {
                cx[i / 2].y = fx; cy[i / 2].y = fy; cz[i / 2].y = fz; hh[i / 2].y = fh; iD[i / 2].y = fi; iD2[i / 2].y = fi2;
            } else {
                cx[i / 2].x = fx; cy[i / 2].x = fy; cz[i / 2].x = fz; hh[i / 2].x = fh; iD[i / 2].x = fi; iD2[i / 2].x = fi2;
            }
        }
        long long sre[PPT], sim[PPT];
#pragma unroll
        for (int i = 0; i < PPT; ++i) sre[i] = sim[i] = 0;

        for (int t = 0; t < nt; ++t) {
            const uint32_t slot = consumed & 1;
            if (!mbar_wait_bounded(&bar[slot], (consumed >> 1) & 1)) {
                record_error(&hdr->error, kErrTimeout);
                s_abort = 1;
            }
            const unsigned char *st = smem + slot * kStage;
            const double4 *s64 = reinterpret_cast<const double4 *>(st);
            const float4 *sA = reinterpret_cast<const float4 *>(st + kNodeTE * 32);
            const float *sC = reinterpret_cast<const float *>(st + kNodeTE * 48);
            // (a warp whose nodes all lie past the grid's end has nothing to add)
            const int cnt = tile * kNodeTile + (tid & ~31) * PPT < nodes ? min(kNodeTE, len - t * kNodeTE) : 0;
            if constexpr (!FINE) {
                for (int jb = 0; jb < cnt; jb += kNodeFold) {
                    float2 are[PH], aim[PH];
#pragma unroll
                    for (int q = 0; q < PH; ++q) are[q] = aim[q] = f2(0.f, 0.f);
#pragma unroll 8
                    for (int j = jb; j < jb + kNodeFold; ++j) {
                        const double4 r = s64[j];
                        const float4 A = sA[j];
                        const float a1 = sC[j];
                        const float2 a2 = f2(a1, a1);
#pragma unroll
                        for (int q = 0; q < PH; ++q) {
                            uint32_t w[2];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const int i = 2 * q + e;
                                double tt = __fma_rn(nqx[i], r.x, r.w);
                                tt = __fma_rn(nqy[i], r.y, tt);
                                tt = __fma_rn(nqz[i], r.z, tt);
                                w[e] = (uint32_t)__double2loint(tt);
                            }
                            float2 x = half_turns2(w[0], w[1]);
                            float2 amp = a2;
                            if (NF) {
                                float2 s = __fmul2_rn(cx[q], f2(A.x, A.x));
                                s = __ffma2_rn(cy[q], f2(A.y, A.y), s);
                                s = __ffma2_rn(cz[q], f2(A.z, A.z), s);
                                const float2 w2 = __ffma2_rn(s, s, f2(A.w, A.w));  // s^2 - |r|^2
                                x = __ffma2_rn(hh[q], w2, x);                      // h (|r|^2 - s^2)
                                if (SCALE) amp = __fmul2_rn(a2, __ffma2_rn(s, iD2[q], iD[q]));
                            } else if (SECOND) {
                                x = __ffma2_rn(hh[q], f2(A.w, A.w), x);  // (-h)(-(x^2+y^2))
                            }
                            amp.x = flip_sign(amp.x, w[0]);
                            amp.y = flip_sign(amp.y, w[1]);
                            float2 sn, cs;
                            sincospi2(x, sn, cs);
                            are[q] = __ffma2_rn(amp, cs, are[q]);
                            aim[q] = __ffma2_rn(amp, sn, aim[q]);
                        }
                    }
#pragma unroll
                    for (int q = 0; q < PH; ++q) {
                        sre[2 * q] += __float2ll_rn(are[q].x * ni.scale);
                        sre[2 * q + 1] += __float2ll_rn(are[q].y * ni.scale);
                        sim[2 * q] += __float2ll_rn(aim[q].x * ni.scale);
                        sim[2 * q + 1] += __float2ll_rn(aim[q].y * ni.scale);
                    }
                }
            } else {
                for (int jb = 0; jb < cnt; jb += kNodeBlock) {
                    double re[PPT], im[PPT];
#pragma unroll
                    for (int i = 0; i < PPT; ++i) re[i] = im[i] = 0.0;
#pragma unroll 4
                    for (int j = jb; j < jb + kNodeBlock; ++j) {
                        const double4 r = s64[j];
                        const float a1 = sC[j];
                        const double ad = (double)a1;
#pragma unroll
                        for (int q = 0; q < PH; ++q) {
                            double x[2], amp[2] = {ad, ad};
                            uint32_t w[2];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const int i = 2 * q + e;
                                double tt = __fma_rn(nqx[i], r.x, r.w);
                                tt = __fma_rn(nqy[i], r.y, tt);
                                tt = __fma_rn(nqz[i], r.z, tt);
                                w[e] = (uint32_t)__double2loint(tt);
                                x[e] = half_turn64(w[e]);
                            }
                            if (NF || SECOND) {
                                const float4 A = sA[j];
                                float2 x2;
                                if (NF) {
                                    float2 s = __fmul2_rn(cx[q], f2(A.x, A.x));
                                    s = __ffma2_rn(cy[q], f2(A.y, A.y), s);
                                    s = __ffma2_rn(cz[q], f2(A.z, A.z), s);
                                    x2 = __fmul2_rn(hh[q], __ffma2_rn(s, s, f2(A.w, A.w)));  // h (|r|^2 - s^2)
                                    if (SCALE) {
                                        const float2 f = __fmul2_rn(f2(a1, a1), __ffma2_rn(s, iD2[q], iD[q]));
                                        amp[0] = (double)f.x;
                                        amp[1] = (double)f.y;
                                    }
                                } else {
                                    x2 = __fmul2_rn(hh[q], f2(A.w, A.w));  // (-h)(-(x^2+y^2))
                                }
                                x[0] += (double)x2.x;
                                x[1] += (double)x2.y;
                            }
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const int i = 2 * q + e;
                                double sn, cs;
                                sincospi64(x[e], sn, cs);
                                const double a = flip_sign64(amp[e], w[e]);
                                re[i] = __fma_rn(a, cs, re[i]);
                                im[i] = __fma_rn(a, sn, im[i]);
                            }
                        }
                    }
#pragma unroll
                    for (int i = 0; i < PPT; ++i) {
                        sre[i] += __double2ll_rn(re[i] * (double)ni.scale);
                        sim[i] += __double2ll_rn(im[i] * (double)ni.scale);
                    }
                }
            }
            ++consumed;
            __syncthreads();
            if (s_abort) {
                // wait (bounded) for copies still in flight into this CTA's shared memory
                if (tid == 0)
                    while (consumed < issued) {
                        mbar_wait_bounded(&bar[consumed & 1], (consumed >> 1) & 1);
                        ++consumed;
                    }
                return;
            }
            if (tid == 0 && t + 2 < nt) issue(t + 2);
        }
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(
            ni.ncell > 1 ? nb.f + (img - img0) * nb.caps.f + (int64_t)seg * nodes : nb.v + (img - img0) * nb.caps.v);
#pragma unroll
        for (int i = 0; i < PPT; ++i)
            if (m0 + i < nodes) {
                atomicAdd(dst + 2 * (m0 + i), (unsigned long long)sre[i]);
                atomicAdd(dst + 2 * (m0 + i) + 1, (unsigned long long)sim[i]);
            }
    }
    if (tid == 0) add_busy(cta_ns, globaltimer_ns() - t_start);
}

// Node sums in FP64 (IDIWF_DOUBLE in the far field, and in the near field with
// IDIWF_ACCURATE): the direct FP64 kernel's phases at the nodes' positions, without the
// near field's pixel constant; the plain near field keeps the direct kernel, whose
// |d - r| - d_z rounding is no smooth function of the pixel.  Shares, blocks and
// fixed-point totals as in node_sum_kernel; a block's 64 emitters are added in FP64.
// Four images of 2,000 emitters on 256^2 pixels (70^2 nodes): whole call 0.29 ms against
// 2.87 ms, error against extended references 2.7e-15 against 1e-14 (sums without Kahan
// steps, but a thirteenth of the pairs and exact totals); of 20,000 and 50,000 emitters in
// phase 1.7e-15 and 1.4e-15 of the field, where the direct kernel's compensated sums hold
// 1.2e-15 and 1.0e-15, and less in the dark beside the peak.
//
// One 64-bit word counts in 2^-58 to 2^-59 of n max|a|, too coarse for FP64 where n is
// large (1.3e-13 of the field of 1e6 emitters, the direct kernel 6e-15).  A second word takes
// what the first leaves.
__device__ __forceinline__ void add_two_words(double x, long long &hi, long long &lo) {
    const double h = rint(x);
    hi += __double2ll_rn(h);
    lo += __double2ll_rn((x - h) * (1.0 / kLowUnit));
}
template <bool ACC, bool SCALE, bool SECOND>
__global__ void __launch_bounds__(kNodeThreads)
    node_sum64_kernel(const __grid_constant__ BatchParams bp, const GeomParams g, DoubleRecs rec,
                      const NodePlan *__restrict__ plan, NodeBuffers nb,
                      WsHeader *__restrict__ hdr, uint64_t *__restrict__ cta_ns, int img0, int img1) {
    constexpr int PPT = kNodePPT64;
    constexpr uint32_t kStage = kNodeBlock * kDoubleRecBytes;
    __shared__ __align__(128) unsigned char smem[2 * kStage];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ int s_abort;
    __shared__ long long s_w0[kMaxImagesPerLaunch + 1];
    const int tid = threadIdx.x;
    const uint64_t t_start = globaltimer_ns();
    const int nimg = img1 - img0;
    image_work(plan, img0, nimg, s_w0);
    const int64_t wend = s_w0[nimg];
    if (wend == 0) return;
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        s_abort = 0;
        mbar_fence_init();
        if (blockIdx.x == 0) atomicMax(&hdr->n_ctas, gridDim.x);
    }
    __syncthreads();
    int64_t pos = wend * blockIdx.x / gridDim.x;
    const int64_t end = wend * (blockIdx.x + 1) / gridDim.x;
    uint32_t issued = 0, consumed = 0;
    while (pos < end) {
        int lo = 0, hi = nimg;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_w0[mid] <= pos) lo = mid;
            else hi = mid;
        }
        const int img = img0 + lo;
        const NodeImage ni = plan->img[img];
        const ImageDesc d = bp.img[img];
        const int64_t rel = pos - s_w0[lo];
        const int tile = (int)(rel / ni.nblk), b0 = (int)(rel % ni.nblk);
        const int nt = (int)min((int64_t)ni.nblk, b0 + (end - pos)) - b0;
        pos += nt;
        const int nodes = ni.n0 * ni.n1;
        // a block of 64 emitters per stage, as many as the image's records hold
        const int nrec = d.ntiles * bp.te;
        auto count = [&](int t) { return min(kNodeBlock, nrec - (b0 + t) * kNodeBlock); };
        auto issue = [&](int t) {
            const uint32_t slot = issued & 1;
            unsigned char *st = smem + slot * kStage;
            const int cnt = count(t);  // a multiple of 16
            const int64_t r0 = d.rec + (int64_t)(b0 + t) * kNodeBlock;
            mbar_arrive_expect_tx(&bar[slot], cnt * kDoubleRecBytes);
            bulk_g2s(st, rec.r64 + r0, cnt * 32, &bar[slot]);
            bulk_g2s(st + kNodeBlock * 32, rec.ra + r0, cnt * 8, &bar[slot]);
            ++issued;
        };
        if (tid == 0)
            for (int t = 0; t < 2 && t < nt; ++t) issue(t);

        const int m0 = tile * kNodeTile64 + tid;
        double px[PPT], py[PPT], pz[PPT], D[PPT], qx[PPT], qy[PPT], qz[PPT], c2[PPT];
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
            const int m = min(m0 + i * kNodeThreads, nodes - 1);
            const int a = m / ni.n1, b = m - a * ni.n1;
            const double fa = node_index(ni.n0, a, g.nx), fb = node_index(ni.n1, b, g.ny);
            pixel_cpu_at(g, fa, fb, px[i], py[i], pz[i]);
            const PixelDir q = pixel_dir(g, fa, fb);
            D[i] = sqrt(px[i] * px[i] + py[i] * py[i] + pz[i] * pz[i]);
            qx[i] = g.k * q.ux;
            qy[i] = g.k * q.uy;
            qz[i] = -kTwoPi * q.nqz;
            c2[i] = 0.5 * g.k * q.invD;
        }
        long long sre[PPT], sim[PPT], lre[PPT], lim[PPT];
#pragma unroll
        for (int i = 0; i < PPT; ++i) sre[i] = sim[i] = lre[i] = lim[i] = 0;
        for (int t = 0; t < nt; ++t) {
            const uint32_t slot = consumed & 1;
            if (!mbar_wait_bounded(&bar[slot], (consumed >> 1) & 1)) {
                record_error(&hdr->error, kErrTimeout);
                s_abort = 1;
            }
            const unsigned char *st = smem + slot * kStage;
            const double4 *s64 = reinterpret_cast<const double4 *>(st);
            const double *sa = reinterpret_cast<const double *>(st + kNodeBlock * 32);
            const int cnt = min(count(t), d.n - (b0 + t) * kNodeBlock);
            double re[PPT], im[PPT];
#pragma unroll
            for (int i = 0; i < PPT; ++i) re[i] = im[i] = 0.0;
            for (int j = 0; j < cnt; ++j) {
                const double4 r = s64[j];
                const double aj = sa[j];
#pragma unroll
                for (int i = 0; i < PPT; ++i) {
                    double phase, w = aj;
                    if (ACC) {
                        const double a = px[i] - r.x, b = py[i] - r.y, c = pz[i] - r.z;
                        const double dist = sqrt(fma(c, c, fma(a, a, b * b)));
                        const double rr = fma(r.z, r.z, fma(r.x, r.x, r.y * r.y));
                        const double dr = fma(pz[i], r.z, fma(px[i], r.x, py[i] * r.y));
                        phase = fma(g.k, (rr - 2.0 * dr) / (dist + D[i]) + r.z, r.w);
                        if (SCALE) w = aj / dist;
                    } else {
                        phase = r.w - fma(r.z, qz[i], fma(r.x, qx[i], r.y * qy[i]));
                        if (SECOND) phase = fma(c2[i], fma(r.x, r.x, r.y * r.y), phase);
                    }
                    double sn, cs;
                    sincos(phase, &sn, &cs);
                    re[i] = fma(w, cs, re[i]);
                    im[i] = fma(w, sn, im[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < PPT; ++i) {
                add_two_words(re[i] * (double)ni.scale, sre[i], lre[i]);
                add_two_words(im[i] * (double)ni.scale, sim[i], lim[i]);
            }
            ++consumed;
            __syncthreads();
            if (s_abort) {
                if (tid == 0)
                    while (consumed < issued) {
                        mbar_wait_bounded(&bar[consumed & 1], (consumed >> 1) & 1);
                        ++consumed;
                    }
                return;
            }
            if (tid == 0 && t + 2 < nt) issue(t + 2);
        }
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(nb.v + (img - img0) * nb.caps.v);
        unsigned long long *low = reinterpret_cast<unsigned long long *>(nb.f + (img - img0) * nb.caps.f);
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
            const int m = m0 + i * kNodeThreads;
            if (m < nodes) {
                atomicAdd(dst + 2 * m, (unsigned long long)sre[i]);
                atomicAdd(dst + 2 * m + 1, (unsigned long long)sim[i]);
                atomicAdd(low + 2 * m, (unsigned long long)lre[i]);
                atomicAdd(low + 2 * m + 1, (unsigned long long)lim[i]);
            }
        }
    }
    if (tid == 0) add_busy(cta_ns, globaltimer_ns() - t_start);
}

// Emitters per cell of every sort block; an image's last block turns the counts into
// offsets and lays the cells out, each on whole blocks of 64 records.
__device__ __forceinline__ void count_cells(const BatchParams &bp, const double *__restrict__ atoms, const NodeGeom &ng,
                                            NodePlan *__restrict__ plan, const CellSort &cs) {
    __shared__ int s_cnt[kCellMax], s_part[8];
    __shared__ int s_last;
    const int img = blockIdx.y, tid = threadIdx.x;
    const NodeImage &pi = plan->img[img];
    if (pi.path != kPathNodes || pi.ncell == 1) return;
    const NodeImage ni = pi;
    const ImageDesc d = bp.img[img];
    const int nb = (d.n + kCellSort - 1) / kCellSort;
    int *counts = cs.counts + sort_block0(bp, img) * kCellMax;
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
        for (int c = tid; c < ni.ncell; c += 256) s_cnt[c] = 0;
        __syncthreads();
        for (int j = b * kCellSort + tid; j < min((b + 1) * kCellSort, d.n); j += 256)
            atomicAdd(&s_cnt[cell_of(ng, ni, reinterpret_cast<const double4 *>(atoms)[d.src + j])], 1);
        __syncthreads();
        for (int c = tid; c < ni.ncell; c += 256) counts[(int64_t)b * kCellMax + c] = s_cnt[c];
        __syncthreads();
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&plan->img[img].ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    int blocks0 = 0;
    for (int c0 = 0; c0 < ni.ncell; c0 += 256) {
        const int c = c0 + tid;
        int sum = 0;
        if (c < ni.ncell) {
            // 16 loads in flight at a time: the chain is the additions, not the memory
            for (int b0 = 0; b0 < nb; b0 += 16) {
                int v[16];
#pragma unroll
                for (int k = 0; k < 16; ++k)
                    v[k] = b0 + k < nb ? __ldcg(counts + (int64_t)(b0 + k) * kCellMax + c) : 0;
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    if (b0 + k < nb) counts[(int64_t)(b0 + k) * kCellMax + c] = sum;
                    sum += v[k];
                }
            }
            cs.total[img * kCellMax + c] = sum;
        }
        // exclusive scan of the cells' record blocks over the 256 threads
        const int nblk = (sum + kNodeBlock - 1) / kNodeBlock;
        int x = nblk;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if ((tid & 31) >= o) x += y;
        }
        if ((tid & 31) == 31) s_part[tid >> 5] = x;
        __syncthreads();
        int before = 0, all = 0;
        for (int w = 0; w < 8; ++w) {
            before += w < (tid >> 5) ? s_part[w] : 0;
            all += s_part[w];
        }
        if (c < ni.ncell) cs.first[img * (kCellMax + 1) + c] = blocks0 + before + x - nblk;
        blocks0 += all;
        __syncthreads();
    }
    if (tid == 0) {
        cs.first[img * (kCellMax + 1) + ni.ncell] = blocks0;
        plan->img[img].nblk = blocks0;
    }
}

// What a group's images need before their sums: zeros in the sums' buffers, the interpolation
// weights, and (COUNT, with the first group and for all images) the emitters' counts per
// cell.  One kernel: where no image takes nodes, every kernel that returns at once
// costs 1.5 us in a graph and up to 4 us in a stream.
template <bool COUNT>
__global__ void __launch_bounds__(256)
    node_setup_kernel(const __grid_constant__ BatchParams bp, const double *__restrict__ atoms, const GeomParams g,
                      const NodeGeom ng, NodePlan *__restrict__ plan, CellSort cs, NodeBuffers nb, int img0, int nimg) {
    const int at = blockIdx.y, tid = threadIdx.x;
    if (plan->img[img0 + at].path != kPathNodes) return;
    if (COUNT && plan->img[img0 + at].ncell > 1) count_cells(bp, atoms, ng, plan, cs);
    if (at >= nimg) return;
    const NodeImage &ni = plan->img[img0 + at];
    const int n0 = ni.n0, n1 = ni.n1, g0 = ni.g0, g1 = ni.g1, ncell = ni.ncell, pix = ni.pix;
    const int64_t nv = (int64_t)n0 * n1, nf = nb.two_words ? nv : (ncell > 1 ? (int64_t)ncell * g0 * g1 : 0);
    double2 *v = nb.v + at * nb.caps.v, *f = nb.f + at * nb.caps.f;
    for (int64_t i = blockIdx.x * blockDim.x + tid; i < nv + nf; i += gridDim.x * blockDim.x)
        (i < nv ? v[i] : f[i - nv]) = make_double2(0.0, 0.0);
    const int lane = tid & 31;
    double *lx = nb.lx + at * nb.lx_stride, *ly = nb.ly + at * nb.ly_stride;
    double *sx = nb.sx + at * nb.sx_stride, *sy = nb.sy + at * nb.sy_stride;
    const int fine = pix ? 0 : g.nx + g.ny, rows = fine + (ncell > 1 ? n0 + n1 : 0);
    for (int row = blockIdx.x * 8 + (tid >> 5); row < rows; row += gridDim.x * 8) {
        if (row < fine) {
            if (row < g.nx) node_weights_row(lx, n0, pixel_x(g.nx, row), row, lane);
            else node_weights_row(ly, n1, pixel_x(g.ny, row - g.nx), row - g.nx, lane);
        } else {
            const int i = row - fine;
            if (i < n0) node_weights_row(sx, g0, pix ? pixel_x(g.nx, i) : node_x(n0, i), i, lane);
            else node_weights_row(sy, g1, pix ? pixel_x(g.ny, i - n0) : node_x(n1, i - n0), i - n0, lane);
        }
    }
}

// Cells, along y: Y[cell][B][a] = sum_b S_y[B][b] F[cell][a][b].
__global__ void __launch_bounds__(kGemmThreads, 4) cell_interp_kernel(const GeomParams g, const NodePlan *__restrict__ plan,
                                                                      NodeBuffers nb, int img0) {
    extern __shared__ __align__(128) unsigned char smem[];
    const NodeImage ni = plan->img[img0 + blockIdx.y];
    if (ni.path != kPathNodes || ni.ncell == 1) return;
    const double unit = 1.0 / (double)ni.scale;
    const double *S = nb.sy + blockIdx.y * nb.sy_stride;
    const int tm = (ni.n1 + kGemmM - 1) / kGemmM, tn = (ni.g0 + kGemmN - 1) / kGemmN;
    for (int t = blockIdx.x; t < tm * tn * ni.ncell; t += gridDim.x) {
        const int cell = t / (tm * tn), u = t - cell * (tm * tn);
        double2 *Y = nb.y + blockIdx.y * nb.caps.y + (int64_t)cell * ni.n1 * ni.g0;
        interp_tile<1>(*reinterpret_cast<GemmSmem *>(smem), S,
                          nb.f + blockIdx.y * nb.caps.f + (int64_t)cell * ni.g0 * ni.g1, nullptr, ni.n1, ni.g0, ni.g1,
                          u % tm * kGemmM, u / tm * kGemmN, unit,
                          [&](int B, int a, double re, double im) { Y[(size_t)B * ni.g0 + a] = make_double2(re, im); });
    }
}

// Cells, along x, and their sum: V[A][B] += exp(i theta_cell(A, B)) sum_a S_x[A][a] Y[cell][B][a],
// theta = the phase of the cell's centre at the target point.  A CTA takes an equal,
// contiguous share of (image, target tile, cell), 32 x 32 targets each; the cells' tiles
// are FP64 products (mma.m8n8k4, K in blocks of 16 by cp.async), turned by the
// phase and added in registers; a tile's total goes to the fixed-point sums by atomics.
//
// The turn takes FP64 polynomials: every emitter of a cell shares its error, which for emitters
// in phase is far more than their sums' own (dark pixels beside the peak of 50,000 fcc
// sites: 3.1e-7 with FP32 ones, 9e-8 with these, 2.2e-7 by the direct kernels; two such images
// 0.360 and 0.364 ms).  How the shares cut a tile's cells depends on the batch, so every
// cell's value is rounded to a grid (2^-50 of the largest possible sum) on which the FP64
// additions are exact in any order.
constexpr int kExpTile = 32;
struct ExpandSmem {
    double a[2][kExpTile * kGemmLd];
    double2 b[2][kExpTile * kGemmLd];
    double nq[3][kExpTile * (kExpTile + 1)];  // turns per length at the targets
};
__global__ void __launch_bounds__(kGemmThreads, 4) cell_expand_kernel(const GeomParams g, const NodeGeom ng,
                                                                      const NodePlan *__restrict__ plan, NodeBuffers nb,
                                                                      int img0, int img1) {
    extern __shared__ __align__(128) unsigned char smem[];
    ExpandSmem &sm = *reinterpret_cast<ExpandSmem *>(smem);
    __shared__ long long s_w0[kMaxImagesPerLaunch + 1];
    const int tid = threadIdx.x, lane = tid & 31, wr = (tid >> 5) >> 1, wc = (tid >> 5) & 1;
    const int nimg = img1 - img0;
    if (tid == 0) {
        long long w = 0;
        for (int i = 0; i < nimg; ++i) {
            s_w0[i] = w;
            const NodeImage &ni = plan->img[img0 + i];
            if (ni.path == kPathNodes && ni.ncell > 1)
                w += (long long)((ni.n0 + kExpTile - 1) / kExpTile) * ((ni.n1 + kExpTile - 1) / kExpTile) * ni.ncell;
        }
        s_w0[nimg] = w;
    }
    __syncthreads();
    const int64_t wend = s_w0[nimg];
    int64_t pos = wend * blockIdx.x / gridDim.x;
    const int64_t end = wend * (blockIdx.x + 1) / gridDim.x;
    while (pos < end) {
        int lo = 0, hi = nimg;  // last image with w0 <= pos
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_w0[mid] <= pos) lo = mid;
            else hi = mid;
        }
        const NodeImage ni = plan->img[img0 + lo];
        const int64_t rel = pos - s_w0[lo];
        const int tile = (int)(rel / ni.ncell), c0 = (int)(rel % ni.ncell);
        const int c1 = (int)min((int64_t)ni.ncell, c0 + (end - pos));
        pos += c1 - c0;
        const int t0 = (ni.n0 + kExpTile - 1) / kExpTile, A0 = tile % t0 * kExpTile, B0 = tile / t0 * kExpTile;
        const double *S = nb.sx + lo * nb.sx_stride;
        const double2 *Y = nb.y + lo * nb.caps.y;
        const int K = ni.g0, nk = (K + kGemmK - 1) / kGemmK;
        __syncthreads();
        for (int i = tid; i < kExpTile * kExpTile; i += kGemmThreads) {
            const int A = min(A0 + i / kExpTile, ni.n0 - 1), B = min(B0 + i % kExpTile, ni.n1 - 1);
            const PixelDir q = pixel_dir(g, ni.pix ? (double)A : node_index(ni.n0, A, g.nx),
                                         ni.pix ? (double)B : node_index(ni.n1, B, g.ny));
            const int at = i / kExpTile * (kExpTile + 1) + i % kExpTile;
            sm.nq[0][at] = q.nqx;
            sm.nq[1][at] = q.nqy;
            sm.nq[2][at] = q.nqz;
        }
        double tot[2][4][2];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) tot[a][b][0] = tot[a][b][1] = 0.0;
        // adding and taking it back rounds to multiples of 2^9 units (|sum| < 2^60 units)
        const double grid = 0x1.8p61 / (double)ni.scale;
        const int steps = (c1 - c0) * nk;
        auto issue = [&](int st) {
            const int s = st & 1, cell = c0 + st / nk, k0 = st % nk * kGemmK;
#pragma unroll
            for (int q = 0; q < 2; ++q) {  // 32 rows x 16 doubles
                const int c = tid + q * kGemmThreads, r = c >> 3, k = (c & 7) * 2;
                const bool ok = A0 + r < ni.n0 && k0 + k < K;
                cp_async16(&sm.a[s][r * kGemmLd + k], S + (ok ? (size_t)(A0 + r) * K + k0 + k : 0), ok);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {  // 32 rows x 16 complex
                const int c = tid + q * kGemmThreads, r = c >> 4, k = c & 15;
                const bool ok = B0 + r < ni.n1 && k0 + k < K;
                cp_async16(&sm.b[s][r * kGemmLd + k], Y + (ok ? ((size_t)cell * ni.n1 + B0 + r) * K + k0 + k : 0), ok);
            }
            cp_async_commit();
        };
        issue(0);
        int st = 0;
        for (int cell = c0; cell < c1; ++cell) {
            double acc[2][4][2];
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
            for (int kb = 0; kb < nk; ++kb, ++st) {
                if (st + 1 < steps) {
                    issue(st + 1);
                    cp_async_wait<1>();
                } else {
                    cp_async_wait<0>();
                }
                __syncthreads();
                const double *sa = sm.a[st & 1] + (wr * 16 + (lane >> 2)) * kGemmLd + (lane & 3);
                const double *sb = reinterpret_cast<const double *>(sm.b[st & 1] + (wc * 16 + (lane >> 3)) * kGemmLd +
                                                                    (lane & 3)) + ((lane >> 2) & 1);
#pragma unroll
                for (int k = 0; k < kGemmK; k += 4) {
                    double fa[2], fb[4];
#pragma unroll
                    for (int t = 0; t < 2; ++t) fa[t] = sa[t * 8 * kGemmLd + k];
#pragma unroll
                    for (int t = 0; t < 4; ++t) fb[t] = sb[(t * 4 * kGemmLd + k) * 2];
#pragma unroll
                    for (int a = 0; a < 2; ++a)
#pragma unroll
                        for (int b = 0; b < 4; ++b) dmma884(acc[a][b][0], acc[a][b][1], fa[a], fb[b]);
                }
                __syncthreads();
            }
            double ctr[3];
            cell_centre(ng, ni, cell, ctr);
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const int at = (wr * 16 + a * 8 + (lane >> 2)) * (kExpTile + 1) + wc * 16 + b * 4 + (lane & 3);
                    double t = __fma_rn(sm.nq[0][at], ctr[0], kTurnMagic + 0.25 + 0x1p-25);
                    t = __fma_rn(sm.nq[1][at], ctr[1], t);
                    t = __fma_rn(sm.nq[2][at], ctr[2], t);
                    const uint32_t w = (uint32_t)__double2loint(t);
                    double sn, cs;
                    sincospi64(half_turn64(w), sn, cs);
                    const double c = flip_sign64(cs, w), s = flip_sign64(sn, w);
                    const double re = acc[a][b][0], im = acc[a][b][1];
                    tot[a][b][0] += __dsub_rn(__dadd_rn(c * re - s * im, grid), grid);
                    tot[a][b][1] += __dsub_rn(__dadd_rn(c * im + s * re, grid), grid);
                }
        }
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(nb.v + lo * nb.caps.v);
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int A = A0 + wr * 16 + a * 8 + (lane >> 2), B = B0 + wc * 16 + b * 4 + (lane & 3);
                if (A < ni.n0 && B < ni.n1) {
                    unsigned long long *o = dst + 2 * ((int64_t)A * ni.n1 + B);
                    atomicAdd(o, (unsigned long long)__double2ll_rn(tot[a][b][0] * (double)ni.scale));
                    atomicAdd(o + 1, (unsigned long long)__double2ll_rn(tot[a][b][1] * (double)ni.scale));
                }
            }
    }
}

template <int WORDS>
__global__ void __launch_bounds__(kGemmThreads, 4) node_interp_y_kernel(const GeomParams g, const NodePlan *__restrict__ plan,
                                                                     NodeBuffers nb, int img0) {
    extern __shared__ __align__(128) unsigned char smem[];
    const NodeImage ni = plan->img[img0 + blockIdx.y];
    if (ni.path != kPathNodes || ni.pix) return;
    const double unit = 1.0 / (double)ni.scale;
    const double *L = nb.ly + blockIdx.y * nb.ly_stride;
    const double2 *V = nb.v + blockIdx.y * nb.caps.v;
    double2 *W = nb.w + blockIdx.y * nb.w_stride;
    const int tm = (g.ny + kGemmM - 1) / kGemmM, tn = (ni.n0 + kGemmN - 1) / kGemmN;
    for (int t = blockIdx.x; t < tm * tn; t += gridDim.x)
        interp_tile<WORDS>(*reinterpret_cast<GemmSmem *>(smem), L, V, nb.f + blockIdx.y * nb.caps.f, g.ny, ni.n0, ni.n1, t % tm * kGemmM,
                          t / tm * kGemmN, unit,
                          [&](int j, int a, double re, double im) { W[(size_t)j * ni.n0 + a] = make_double2(re, im); });
}

template <bool NF, bool SCALE>
__global__ void __launch_bounds__(kGemmThreads, 4) node_interp_x_kernel(const GeomParams g, const NodePlan *__restrict__ plan,
                                                                     NodeBuffers nb, int img0, void *__restrict__ out,
                                                                     int out_kind) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int img = img0 + blockIdx.y;
    const NodeImage ni = plan->img[img];
    if (ni.path != kPathNodes) return;
    const int64_t obase = (int64_t)img * g.nx * g.ny;
    if (ni.pix) {  // the sums are the pixels'
        const double unit = 1.0 / (double)ni.scale;
        const longlong2 *V = reinterpret_cast<const longlong2 *>(nb.v + blockIdx.y * nb.caps.v);
        for (int p = blockIdx.x * kGemmThreads + threadIdx.x; p < g.nx * g.ny; p += gridDim.x * kGemmThreads)
            finish_pixel<NF, SCALE>(g, p, (double)V[p].x * unit, (double)V[p].y * unit, out, out_kind, obase + p);
        return;
    }
    const double *L = nb.lx + blockIdx.y * nb.lx_stride;
    const double2 *W = nb.w + blockIdx.y * nb.w_stride;
    const int tm = (g.nx + kGemmM - 1) / kGemmM, tn = (g.ny + kGemmN - 1) / kGemmN;
    for (int t = blockIdx.x; t < tm * tn; t += gridDim.x)
        interp_tile<0>(*reinterpret_cast<GemmSmem *>(smem), L, W, nullptr, g.nx, g.ny, ni.n0, t % tm * kGemmM, t / tm * kGemmN,
                           1.0, [&](int i, int j, double re, double im) {
                               finish_pixel_at<NF, SCALE>(g, i, j, re, im, out, out_kind, obase + i * g.ny + j);
                           });
}

// ---------------------------------------------------------------------------
// all-FP64 kernel (reference rounding sequence)
// ---------------------------------------------------------------------------
template <int PPT, bool NF, bool SCALE, bool SECOND, bool ACC = false>
__global__ void __launch_bounds__(256) fwd_double_kernel(const __grid_constant__ BatchParams bp,
                                                         const GeomParams g, DoubleRecs rec,
                                                         void *__restrict__ out, int out_kind,
                                                         WsHeader *__restrict__ hdr,
                                                         uint64_t *__restrict__ cta_ns,
                                                         const NodePlan *__restrict__ plan) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ int s_unit, s_abort;
    __shared__ uint8_t s_skip[kMaxImagesPerLaunch];  // images evaluated on nodes

    const int tid = threadIdx.x;
    bool mine = false;
    for (int i = tid; i < bp.n_images; i += blockDim.x) {
        s_skip[i] = plan && plan->img[i].path == kPathNodes;
        mine |= !s_skip[i];
    }
    if (!__syncthreads_or(mine)) return;
    const int TE = bp.te;
    const uint32_t stage_bytes = (uint32_t)TE * kDoubleRecBytes;
    const uint64_t t_start = globaltimer_ns();
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        s_abort = 0;
        mbar_fence_init();
        if (blockIdx.x == 0) atomicMax(&hdr->n_ctas, gridDim.x);
    }
    __syncthreads();
    const int npix = g.nx * g.ny;
    const int tile_px = blockDim.x * PPT;
    uint32_t issued = 0, consumed = 0;
    bool aborted = false;

    for (;;) {
        __syncthreads();
        if (tid == 0) {
            int u;
            do u = (int)atomicAdd(&hdr->work_counter, 1u);
            while (u < bp.total_units && s_skip[bp.order[u / bp.tiles_per_image]]);
            s_unit = u;
        }
        __syncthreads();
        const int unit = s_unit;
        if (unit >= bp.total_units) break;
        const int img = bp.order[unit / bp.tiles_per_image];
        const int ptile = unit % bp.tiles_per_image;
        const ImageDesc d = bp.img[img];
        const int p0 = ptile * tile_px + tid * PPT;

        double px[PPT], py[PPT], pz[PPT], qx[PPT], qy[PPT], qz[PPT], rdist[PPT], c2[PPT];
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
            const int p = min(p0 + i, npix - 1);
            const int ix = p / g.ny, iy = p - ix * g.ny;
            pixel_cpu(g, ix, iy, px[i], py[i], pz[i]);
            // cpu.py:86-89
            rdist[i] = __drcp_rn(__dsqrt_rn(
                __dadd_rn(__dadd_rn(__dmul_rn(px[i], px[i]), __dmul_rn(py[i], py[i])), __dmul_rn(pz[i], pz[i]))));
            qz[i] = __dmul_rn(g.k, __dsub_rn(__dmul_rn(pz[i], rdist[i]), 1.0));
            qx[i] = __dmul_rn(g.k, __dmul_rn(px[i], rdist[i]));
            qy[i] = __dmul_rn(g.k, __dmul_rn(py[i], rdist[i]));
            c2[i] = __dmul_rn(g.k, rdist[i]) * 0.5;
            if (ACC) {
                // accurate near field: the pixel constant k (|d| - d_z) in
                // turns, without cancellation (reuses the far-field slots)
                const double rho2 = px[i] * px[i] + py[i] * py[i];
                const double D = sqrt(rho2 + pz[i] * pz[i]);
                const double cc = g.kp * (pz[i] > 0 ? rho2 / (D + pz[i]) : D - pz[i]);
                qx[i] = D;
                qy[i] = cc - rint(cc);
            }
        }
        double ax[PPT], ay[PPT], cx[PPT], cy[PPT];
#pragma unroll
        for (int i = 0; i < PPT; ++i) ax[i] = ay[i] = cx[i] = cy[i] = 0.0;

        const int nt = d.ntiles;
        if (tid == 0) {
            for (int s = 0; s < 2 && s < nt; ++s) {
                const uint32_t slot = issued & 1;
                unsigned char *st = smem + slot * stage_bytes;
                const int64_t r0 = d.rec + (int64_t)s * TE;
                mbar_arrive_expect_tx(&bar[slot], stage_bytes);
                bulk_g2s(st, rec.r64 + r0, TE * 32, &bar[slot]);
                bulk_g2s(st + TE * 32, rec.ra + r0, TE * 8, &bar[slot]);
                ++issued;
            }
        }
        for (int it = 0; it < nt; ++it) {
            const uint32_t slot = consumed & 1;
            if (!mbar_wait_bounded(&bar[slot], (consumed >> 1) & 1)) {
                record_error(&hdr->error, kErrTimeout);
                s_abort = 1;
            }
            const unsigned char *st = smem + slot * stage_bytes;
            const double4 *s64 = reinterpret_cast<const double4 *>(st);
            const double *sa = reinterpret_cast<const double *>(st + TE * 32);
            const int jend = min(TE, d.n - it * TE);
            for (int j = 0; j < jend; ++j) {
                const double4 r = s64[j];
                const double aj = sa[j];
#pragma unroll
                for (int i = 0; i < PPT; ++i) {
                    double phase, w = 1.0;
                    if (NF) {
                        // cpu.py:44-47 with numba's contraction
                        const double a = __dsub_rn(px[i], r.x), b = __dsub_rn(py[i], r.y),
                                     c = __dsub_rn(pz[i], r.z);
                        const double dist = __dsqrt_rn(__fma_rn(c, c, __fma_rn(a, a, __dmul_rn(b, b))));
                        if (ACC) {
                            // |d-r| - |d| = (|r|^2 - 2 d.r) / (|d-r| + |d|): no cancellation
                            const double rr = fma(r.z, r.z, fma(r.x, r.x, r.y * r.y));
                            const double dr = fma(pz[i], r.z, fma(px[i], r.x, py[i] * r.y));
                            const double delta = (rr - 2.0 * dr) / (dist + qx[i]);
                            phase = fma(kTwoPi, qy[i], fma(g.k, delta + r.z, r.w));
                        } else {
                            phase = __fma_rn(__dadd_rn(__dsub_rn(dist, pz[i]), r.z), g.k, r.w);
                        }
                        if (SCALE) w = __drcp_rn(dist);
                    } else {
                        // cpu.py:59
                        phase = __dadd_rn(-__fma_rn(r.z, qz[i], __fma_rn(r.x, qx[i], __dmul_rn(r.y, qy[i]))), r.w);
                        if (SECOND)  // sim.cu:88
                            phase = __dadd_rn(phase, __dmul_rn(c2[i], __dadd_rn(__dmul_rn(r.x, r.x), __dmul_rn(r.y, r.y))));
                        if (SCALE) w = rdist[i];
                    }
                    w = __dmul_rn(w, aj);
                    double sn, cs;
                    sincos(phase, &sn, &cs);
                    const double vx = __dmul_rn(w, cs), vy = __dmul_rn(w, sn);
                    // Kahan, cpu.py:97-105
                    const double yx = __dsub_rn(vx, cx[i]), yy = __dsub_rn(vy, cy[i]);
                    const double tx = __dadd_rn(ax[i], yx), ty = __dadd_rn(ay[i], yy);
                    cx[i] = __dsub_rn(__dsub_rn(tx, ax[i]), yx);
                    cy[i] = __dsub_rn(__dsub_rn(ty, ay[i]), yy);
                    ax[i] = tx;
                    ay[i] = ty;
                }
            }
            ++consumed;
            __syncthreads();
            if (s_abort) {
                aborted = true;
                break;
            }
            if (tid == 0 && it + 2 < nt) {
                const uint32_t slot2 = issued & 1;
                unsigned char *st2 = smem + slot2 * stage_bytes;
                const int64_t r0 = d.rec + (int64_t)(it + 2) * TE;
                mbar_arrive_expect_tx(&bar[slot2], stage_bytes);
                bulk_g2s(st2, rec.r64 + r0, TE * 32, &bar[slot2]);
                bulk_g2s(st2 + TE * 32, rec.ra + r0, TE * 8, &bar[slot2]);
                ++issued;
            }
        }
        if (aborted) break;
        const int64_t obase = (int64_t)img * npix;
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
            const int p = p0 + i;
            if (p < npix) store_pixel(out, out_kind, obase + p, ax[i], ay[i]);
        }
    }
    if (aborted) {
        if (tid == 0)
            while (consumed < issued) {
                mbar_wait_bounded(&bar[consumed & 1], (consumed >> 1) & 1);
                ++consumed;
            }
        return;
    }
    if (tid == 0) add_busy(cta_ns, globaltimer_ns() - t_start);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

struct LaunchShape {
    int threads, ppt, te, ctas_per_sm;
    int groups = 1;  // split: pixel runs with a base phase where bounded
    bool direct_only = false;  // (the tuner:) without the images on nodes
};

static int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!cached[dev]) {
        int n = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        cached[dev] = n > 0 ? n : 148;
    }
    return cached[dev];
}

GeomParams make_geom(const idiwf_geom *g) {
    GeomParams p;
    p.nx = g->nx;
    p.ny = g->ny;
    p.flags = g->flags;
    p.has_rot = g->has_rot;
    p.pixelsize = g->pixelsize;
    p.detz = g->detz;
    p.k = g->k;
    p.kp = g->k * kInvTwoPi;
    p.ikp = kTwoPi / g->k;
    p.offx = g->offset[0];
    p.offy = g->offset[1];
    for (int i = 0; i < 9; ++i) p.rot[i] = g->has_rot ? g->rot[i] : (i % 4 == 0 ? 1.0 : 0.0);
    // pixel (px, py) sits at px c0 + py c1 + detz c2 (columns of rot); rows run along c1
    const double *M = p.rot;
    const double c0[3] = {M[0], M[3], M[6]}, c1[3] = {M[1], M[4], M[7]}, c2[3] = {M[2], M[5], M[8]};
    const double n[3] = {c0[1] * c1[2] - c0[2] * c1[1], c0[2] * c1[0] - c0[0] * c1[2], c0[0] * c1[1] - c0[1] * c1[0]};
    const double nn = std::sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    const double h = nn > 0 ? std::fabs(g->detz * (c2[0] * n[0] + c2[1] * n[1] + c2[2] * n[2])) / nn : 0.0;
    const double half = 0.5 * (kRun - 1) * std::fabs(g->pixelsize) * std::sqrt(c1[0] * c1[0] + c1[1] * c1[1] + c1[2] * c1[2]);
    p.run_span = h > 0 ? half / h : INFINITY;
    p.dmin = h;
    p.inv_dmin2 = h > 0 ? 1.0 / (h * h) : INFINITY;
    const double c3 = h > 0 ? kNfBoundC * g->k / (h * h) : INFINITY;
    p.nf_c3 = c3 * c3;
    return p;
}

NodeGeom make_node_geom(const GeomParams &g) {
    NodeGeom n;
    std::memset(&n, 0, sizeof(n));
    const double *M = g.rot;
    const double c[3][3] = {{M[0], M[3], M[6]}, {M[1], M[4], M[7]}, {M[2], M[5], M[8]}};
    const auto dot = [](const double *a, const double *b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; };
    const int size[2] = {g.nx, g.ny};
    const double off[2] = {g.offx, g.offy};
    double len[2], far[2];  // length of a unit step along each axis; largest |pixel coordinate|
    for (int a = 0; a < 2; ++a) {
        len[a] = std::sqrt(dot(c[a], c[a]));
        for (int i = 0; i < 3; ++i) n.e[a][i] = len[a] > 0 ? c[a][i] / len[a] : 0.0;
        far[a] = std::max(std::fabs((0.0 - size[a] * 0.5) * g.pixelsize + off[a]),
                          std::fabs((size[a] - 1 - size[a] * 0.5) * g.pixelsize + off[a]));
    }
    n.e[2][0] = n.e[0][1] * n.e[1][2] - n.e[0][2] * n.e[1][1];
    n.e[2][1] = n.e[0][2] * n.e[1][0] - n.e[0][0] * n.e[1][2];
    n.e[2][2] = n.e[0][0] * n.e[1][1] - n.e[0][1] * n.e[1][0];
    n.ortho = std::fabs(dot(n.e[0], n.e[1])) <= 1e-12;
    if (!(g.dmin > 0) || !std::isfinite(g.dmin)) return n;
    n.ok = 1;
    n.inv_d = 1.0 / g.dmin;
    for (int a = 0; a < 2; ++a) {
        const double half = 0.5 * (size[a] - 1) * std::fabs(g.pixelsize) * len[a];
        n.phi[a] = g.k * half / g.dmin;
        n.t[a] = half / g.dmin;
        n.least[a][0] = n.t[a] > 0 ? 20.0 / std::asinh(1.0 / n.t[a]) : 0.0;
        n.least[a][1] = n.t[a] > 0 ? 1.0 + 35.0 / std::asinh((1.0 - kNodeMaxReach) / n.t[a]) : 0.0;
        // |d . e| over the detector, over a lower bound of |d|
        const double de = far[a] * len[a] + far[1 - a] * std::fabs(dot(c[1 - a], n.e[a])) +
                          std::fabs(g.detz * dot(c[2], n.e[a]));
        n.s[a] = std::min(1.0, de / g.dmin);
        if (!(n.t[a] <= kNodeMaxT)) n.ok = 0;
    }
    return n;
}

static idiwf_status validate_geom(const idiwf_geom *g) {
    if (!g) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "geom is NULL");
    if (g->nx <= 0 || g->ny <= 0)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "detector size must be positive");
    if ((int64_t)g->nx * g->ny >= (int64_t)1 << 31)
        return set_error(IDIWF_ERR_UNSUPPORTED, "detector has 2^31 or more pixels");
    if (!(g->k > 0) || !std::isfinite(g->k))
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "k must be positive and finite");
    if (!std::isfinite(g->pixelsize) || !std::isfinite(g->detz))
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "pixelsize/detz must be finite");
    if (g->flags & ~(IDIWF_NF | IDIWF_SCALE | IDIWF_SECONDORDER | IDIWF_ACCURATE))
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "unknown geometry flag");
    return IDIWF_OK;
}

static idiwf_status validate_batch(const idiwf_batch *b) {
    if (!b) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "batch is NULL");
    if (b->n_images <= 0) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "batch has no images");
    if (!b->offsets) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "batch offsets are NULL");
    if (b->offsets[0] != 0) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "offsets[0] must be 0");
    for (int i = 0; i < b->n_images; ++i) {
        const int64_t n = b->offsets[i + 1] - b->offsets[i];
        if (n < 0) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "offsets must be non-decreasing");
        if (n >= ((int64_t)1 << 30)) return set_error(IDIWF_ERR_UNSUPPORTED, "image with 2^30 or more emitters");
    }
    if (b->offsets[b->n_images] > 0 && !b->atoms)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "atoms pointer is NULL");
    if (b->atoms && (reinterpret_cast<uintptr_t>(b->atoms) & 31))
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "atoms must be 32-byte aligned");
    if (b->amplitudes && b->amp_dtype != IDIWF_F64 && b->amp_dtype != IDIWF_F32)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "amp_dtype must be IDIWF_F64 or IDIWF_F32");
    return IDIWF_OK;
}

// --- tuned shape cache ------------------------------------------------------
struct TuneKey {
    int precision, flags, nx, ny, nbucket;
    bool operator<(const TuneKey &o) const {
        return std::tie(precision, flags, nx, ny, nbucket) < std::tie(o.precision, o.flags, o.nx, o.ny, o.nbucket);
    }
};
static std::mutex g_tune_mu;
static std::map<TuneKey, LaunchShape> g_tune_cache;

static int n_bucket(const idiwf_batch *b) {
    const double mean = (double)b->offsets[b->n_images] / b->n_images;
    return mean <= 0 ? 0 : (int)std::floor(std::log2(mean));
}

static LaunchShape default_shape(int precision) {
    if (precision == IDIWF_SPLIT) return LaunchShape{256, 4, 512, 3};
    return LaunchShape{128, 2, 128, 2};
}

static idiwf_status resolve_shape(const idiwf_geom *g, const idiwf_batch *b, int precision,
                                  const idiwf_config *cfg, LaunchShape &s) {
    s = default_shape(precision);
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tune_cache.find(TuneKey{precision, g->flags, g->nx, g->ny, n_bucket(b)});
        if (it != g_tune_cache.end()) s = it->second;
    }
    if (cfg) {
        if (cfg->threads) s.threads = cfg->threads;
        if (cfg->pixels_per_thread) s.ppt = cfg->pixels_per_thread;
        if (cfg->emitters_per_tile) s.te = cfg->emitters_per_tile;
        if (cfg->ctas_per_sm) s.ctas_per_sm = cfg->ctas_per_sm;
        if (cfg->pixel_groups) s.groups = cfg->pixel_groups > 0;
    }
    if (s.threads != 64 && s.threads != 128 && s.threads != 256)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "threads must be 64, 128 or 256");
    if (precision == IDIWF_SPLIT) {
        if (s.ppt != 2 && s.ppt != 4 && s.ppt != 8)
            return set_error(IDIWF_ERR_INVALID_ARGUMENT, "split pixels_per_thread must be 2, 4 or 8");
        if (s.te < kFold || s.te > kChunkEmitters || (s.te & (s.te - 1)))
            return set_error(IDIWF_ERR_INVALID_ARGUMENT, "split emitters_per_tile must be a power of two in [64,1024]");
    } else {
        if (s.ppt != 1 && s.ppt != 2 && s.ppt != 4)
            return set_error(IDIWF_ERR_INVALID_ARGUMENT, "double pixels_per_thread must be 1, 2 or 4");
        if (s.te < 16 || s.te > 1024 || s.te % 16)
            return set_error(IDIWF_ERR_INVALID_ARGUMENT, "double emitters_per_tile must be a multiple of 16 in [16,1024]");
    }
    if (s.ctas_per_sm < 1 || s.ctas_per_sm > 8)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "ctas_per_sm must be in [1,8]");
    return IDIWF_OK;
}

// Emitter chunks per (image, pixel tile) for the split kernel: 1 when the
// batch has pixel tiles for at least 3/4 of one wave of CTA slots (two per
// SM), else about two waves' worth of units.  Depends only on the problem and
// the SM count (not on the kernel shape), so the summation order is the same
// for every shape.
static int choose_ksplit(const idiwf_geom *g, const idiwf_batch *b) {
    const int npix = g->nx * g->ny;
    const int64_t base = (int64_t)std::min(b->n_images, kMaxImagesPerLaunch) * ((npix + 1023) / 1024);
    const int64_t slots = 2 * (int64_t)sm_count();
    if (4 * base >= 3 * slots) return 1;
    int64_t nmax = 0;
    for (int i = 0; i < b->n_images; ++i) nmax = std::max<int64_t>(nmax, b->offsets[i + 1] - b->offsets[i]);
    int64_t k = (2 * slots + base / 2) / base;
    k = std::min<int64_t>(k, (nmax + kChunkEmitters - 1) / kChunkEmitters);
    return (int)std::max<int64_t>(1, std::min<int64_t>(k, 64));
}

static size_t partials_bytes(const idiwf_geom *g, const idiwf_batch *b, int ksplit) {
    if (ksplit <= 1) return 0;
    return align256((size_t)ksplit * std::min(b->n_images, kMaxImagesPerLaunch) * g->nx * g->ny * 16);
}

// Whether a call may take nodes at all (1), and cells (2): not with pixel_groups = -1, not
// in FP64's plain near field (its rounding is the reference's, and no smooth function of
// the pixel), and only with an image of pairs (emitters) enough.
static double node_min_pairs(int precision, int out_kind) {
    return precision != IDIWF_SPLIT ? kNodeMinPairs64 : (out_kind == IDIWF_OUT_C128 ? kNodeMinPairsDiff : kNodeMinPairs);
}
// Bytes of the node buffers of one image of up to nmax emitters.
struct NodeBytes {
    NodeCaps caps;
    size_t v, f, y, lx, ly, sx, sy, w;
    size_t all() const { return v + f + y + lx + ly + sx + sy + w; }
};
static NodeBytes node_bytes(const idiwf_geom *g, int64_t nmax, int precision, bool cells) {
    NodeBytes b;
    b.caps = node_caps(g->nx, g->ny, nmax, cells);
    if (precision != IDIWF_SPLIT) b.caps.f = b.caps.v;  // the sums' second words
    b.v = (size_t)b.caps.v * 16;
    b.f = (size_t)b.caps.f * 16;
    b.y = (size_t)b.caps.y * 16;
    b.lx = (size_t)g->nx * node_cap(g->nx) * 8;
    b.ly = (size_t)g->ny * node_cap(g->ny) * 8;
    b.sx = cells ? (size_t)std::max(g->nx, node_cap(g->nx)) * kCellNodes * 8 : 0;
    b.sy = cells ? (size_t)std::max(g->ny, node_cap(g->ny)) * kCellNodes * 8 : 0;
    b.w = (size_t)g->ny * node_cap(g->nx) * 16;
    return b;
}
static int nodes_possible(const idiwf_geom *g, const idiwf_batch *b, int precision, int out_kind, const LaunchShape &s) {
    const bool split = precision == IDIWF_SPLIT;
    if (!s.groups || (!split && (g->flags & IDIWF_NF) && !(g->flags & IDIWF_ACCURATE))) return 0;
    int64_t nmax = 0;
    for (int i = 0; i < b->n_images; ++i) nmax = std::max(nmax, b->offsets[i + 1] - b->offsets[i]);
    if ((double)nmax * g->nx * g->ny < node_min_pairs(precision, out_kind)) return 0;
    const NodeGeom ng = make_node_geom(make_geom(g));
    if (!ng.ok || !node_buffers_fit(g->nx, g->ny, node_bytes(g, INT32_MAX, precision, split && ng.ortho).all())) return 0;
    return split && nmax >= kCellMinEmitters && ng.ortho ? 2 : 1;
}

// Records of an image: whole emitter tiles, and for images that may be cut into cells
// up to 63 empty ones per cell.
static int64_t image_records(int64_t n, int te, int nodes) {
    const int64_t r = (n + te - 1) / te * te;
    if (nodes < 2 || n < kCellMinEmitters) return r;
    return r + (std::min<int64_t>(kCellMax, n / 64) * kNodeBlock + te - 1) / te * te;
}
static int64_t total_records(const idiwf_batch *b, int te, int nodes) {
    int64_t t = 0;
    for (int i = 0; i < b->n_images; ++i) t += image_records(b->offsets[i + 1] - b->offsets[i], te, nodes);
    return t;
}

// Node part of the workspace: the plan, the emitters' sort, and buffers for groups of
// images that together stay within kNodeGroupBytes.
struct NodeLayout {
    size_t ext, counts, first, tot, v, f, y, lx, ly, sx, sy, w, total;  // offsets from the region's start (the plan)
    int group, two_words;
    NodeCaps caps;
    NodeBuffers at(char *base, const idiwf_geom *g) const {
        NodeBuffers nb;
        nb.v = reinterpret_cast<double2 *>(base + v);
        nb.f = reinterpret_cast<double2 *>(base + f);
        nb.y = reinterpret_cast<double2 *>(base + y);
        nb.caps = caps;
        nb.two_words = two_words;
        nb.lx = reinterpret_cast<double *>(base + lx);
        nb.ly = reinterpret_cast<double *>(base + ly);
        nb.sx = reinterpret_cast<double *>(base + sx);
        nb.sy = reinterpret_cast<double *>(base + sy);
        nb.w = reinterpret_cast<double2 *>(base + w);
        nb.lx_stride = (int64_t)g->nx * node_cap(g->nx);
        nb.ly_stride = (int64_t)g->ny * node_cap(g->ny);
        nb.sx_stride = (int64_t)std::max(g->nx, node_cap(g->nx)) * kCellNodes;
        nb.sy_stride = (int64_t)std::max(g->ny, node_cap(g->ny)) * kCellNodes;
        nb.w_stride = (int64_t)g->ny * node_cap(g->nx);
        return nb;
    }
    CellSort sort(char *base) const {
        return CellSort{reinterpret_cast<int *>(base + counts), reinterpret_cast<int *>(base + first),
                        reinterpret_cast<int *>(base + tot)};
    }
};
static NodeLayout node_layout(const idiwf_geom *g, const idiwf_batch *b, int precision, int nodes) {
    NodeLayout L;
    L.two_words = precision != IDIWF_SPLIT;
    const bool cells = nodes > 1;
    const int imgs = std::min(b->n_images, kMaxImagesPerLaunch);
    int64_t nmax = 0, nlaunch = 0;  // largest image, largest number of emitters of a launch
    for (int i = 0; i < b->n_images; ++i) {
        nmax = std::max(nmax, b->offsets[i + 1] - b->offsets[i]);
        if (i % kMaxImagesPerLaunch == 0)
            nlaunch = std::max(nlaunch, b->offsets[std::min(i + kMaxImagesPerLaunch, b->n_images)] - b->offsets[i]);
    }
    const NodeBytes nb = node_bytes(g, nmax, precision, cells);
    L.caps = nb.caps;
    L.group = (int)std::max<size_t>(1, std::min<size_t>(imgs, kNodeGroupBytes / nb.all()));
    size_t o = align256(sizeof(NodePlan));
    const auto take = [&](size_t bytes) {
        const size_t at = o;
        o += align256(bytes);
        return at;
    };
    L.ext = take((size_t)kMaxImagesPerLaunch * 4 * kNodeExt);
    L.counts = take(cells ? (size_t)(nlaunch / kCellSort + imgs + 1) * kCellMax * 4 : 0);
    L.first = take(cells ? (size_t)imgs * (kCellMax + 1) * 4 : 0);
    L.tot = take(cells ? (size_t)imgs * kCellMax * 4 : 0);
    L.v = take(L.group * nb.v);
    L.f = take(L.group * nb.f);
    L.y = take(L.group * nb.y);
    L.lx = take(L.group * nb.lx);
    L.ly = take(L.group * nb.ly);
    L.sx = take(L.group * nb.sx);
    L.sy = take(L.group * nb.sy);
    L.w = take(L.group * nb.w);
    L.total = o;
    return L;
}

static size_t node_region_offset(const idiwf_geom *g, const idiwf_batch *b, int precision, int64_t nrec, int ksplit) {
    if (precision != IDIWF_SPLIT) return kWsDataOffset + double_recs_bytes(nrec);
    return kWsDataOffset + split_recs_bytes(nrec) + partials_bytes(g, b, ksplit);
}

static size_t forward_ws_bytes(const idiwf_geom *g, const idiwf_batch *b, int precision, const LaunchShape &s) {
    const int nodes = nodes_possible(g, b, precision, IDIWF_OUT_C64, s);  // the output with the most images on nodes
    const int64_t nrec = std::max<int64_t>(total_records(b, s.te, nodes), 1);
    return node_region_offset(g, b, precision, nrec, choose_ksplit(g, b)) +
           (nodes ? node_layout(g, b, precision, nodes).total : 0);
}

// Dynamic shared memory of a forward kernel: two stages of emitter records,
// plus for the pixel-run kernel the Kahan totals (4 floats per pixel of the CTA).
static size_t fwd_smem(int precision, const LaunchShape &s, int path) {
    if (precision != IDIWF_SPLIT) return 2 * (size_t)s.te * kDoubleRecBytes;
    return 2 * (size_t)s.te * kSplitRecBytes + (path == kPathRuns ? (size_t)16 * s.ppt * s.threads : 0);
}

// kernel table ---------------------------------------------------------------
template <int PPT, bool CH, int PATH>
static void *split_kernel_for3(int flags) {
    const bool nf = flags & IDIWF_NF, sc = flags & IDIWF_SCALE, so = flags & IDIWF_SECONDORDER;
    if (nf) return sc ? (void *)fwd_split_kernel<PPT, true, true, false, CH, PATH>
                      : (void *)fwd_split_kernel<PPT, true, false, false, CH, PATH>;
    if (PATH == kPathExact) return nullptr;  // near field only
    constexpr int P = PATH == kPathExact ? kPathPixel : PATH;
    if (so) return sc ? (void *)fwd_split_kernel<PPT, false, true, true, CH, P>
                      : (void *)fwd_split_kernel<PPT, false, false, true, CH, P>;
    return sc ? (void *)fwd_split_kernel<PPT, false, true, false, CH, P>
              : (void *)fwd_split_kernel<PPT, false, false, false, CH, P>;
}
// path: kPathRuns, kPathPixel or kPathExact (nullptr for the exact path
// without "nf")
template <int PPT, bool CH>
static void *split_kernel_for2(int flags, int path) {
    if (path == kPathRuns) return split_kernel_for3<PPT, CH, kPathRuns>(flags);
    if (path == kPathExact) return split_kernel_for3<PPT, CH, kPathExact>(flags);
    return split_kernel_for3<PPT, CH, kPathPixel>(flags);
}
template <int PPT>
static void *split_kernel_for(int flags, bool chunked, int path) {
    return chunked ? split_kernel_for2<PPT, true>(flags, path) : split_kernel_for2<PPT, false>(flags, path);
}
template <int PPT>
static void *double_kernel_for(int flags) {
    const bool nf = flags & IDIWF_NF, sc = flags & IDIWF_SCALE, so = flags & IDIWF_SECONDORDER;
    if (nf && (flags & IDIWF_ACCURATE))
        return sc ? (void *)fwd_double_kernel<PPT, true, true, false, true>
                  : (void *)fwd_double_kernel<PPT, true, false, false, true>;
    if (nf) return sc ? (void *)fwd_double_kernel<PPT, true, true, false> : (void *)fwd_double_kernel<PPT, true, false, false>;
    if (so) return sc ? (void *)fwd_double_kernel<PPT, false, true, true> : (void *)fwd_double_kernel<PPT, false, false, true>;
    return sc ? (void *)fwd_double_kernel<PPT, false, true, false> : (void *)fwd_double_kernel<PPT, false, false, false>;
}
static void *kernel_for(int precision, int ppt, int flags, bool chunked, int path = kPathRuns) {
    if (precision == IDIWF_SPLIT) {
        if (ppt == 2) return split_kernel_for<2>(flags, chunked, path);
        if (ppt == 4) return split_kernel_for<4>(flags, chunked, path);
        return split_kernel_for<8>(flags, chunked, path);
    }
    if (ppt == 1) return double_kernel_for<1>(flags);
    if (ppt == 2) return double_kernel_for<2>(flags);
    return double_kernel_for<4>(flags);
}

static idiwf_status ensure_smem(void *fn, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<void *, int>, size_t> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    auto key = std::make_pair(fn, dev);
    auto it = done.find(key);
    if (it != done.end() && it->second >= bytes) return IDIWF_OK;
    IDIWF_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    done[key] = bytes;
    return IDIWF_OK;
}

// CTAs of `fn` that fit on one SM at this shape (cached per device).  The
// persistent grid never exceeds SMs x this: a CTA that only starts after the
// queue has drained would do no work and report a zero busy time.
static int resident_ctas(void *fn, int threads, size_t smem) {
    static std::mutex mu;
    static std::map<std::tuple<void *, int, int, size_t>, int> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_tuple(fn, dev, threads, smem);
    auto it = done.find(key);
    if (it != done.end()) return it->second;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        occ = 1;
    }
    occ = std::max(occ, 1);
    done[key] = occ;
    return occ;
}

template <bool FINE>
static void *node_sum_fn(bool nf, bool sc, bool so) {
    return nf ? (sc ? (void *)node_sum_kernel<true, true, false, FINE> : (void *)node_sum_kernel<true, false, false, FINE>)
              : (so ? (void *)node_sum_kernel<false, false, true, FINE> : (void *)node_sum_kernel<false, false, false, FINE>);
}

// Blocks per image of a group of n images: about two per SM in all.
static int group_blocks(int n) { return std::max(1, (2 * sm_count() + n - 1) / n); }
// The setup of images [img0, img0 + n), with the cells' counts of every image where count.
static void launch_setup(const GeomParams &g, const NodeGeom &ng, const BatchParams &bp, const double *atoms, NodePlan *plan,
                         const NodeLayout &nl, const NodeBuffers &nb, char *node_base, int img0, int n, bool count,
                         cudaStream_t stream) {
    const CellSort cs = nl.sort(node_base);
    int blocks = std::max((g.nx + g.ny + 15) / 16, group_blocks(n));
    if (count) {
        int nbig = 0;
        for (int i = 0; i < bp.n_images; ++i) nbig = std::max(nbig, bp.img[i].n);
        blocks = std::max(blocks, (nbig + kCellSort - 1) / kCellSort);
        node_setup_kernel<true><<<dim3(blocks, bp.n_images), 256, 0, stream>>>(bp, atoms, g, ng, plan, cs, nb, 0, n);
    } else {
        node_setup_kernel<false><<<dim3(blocks, n), 256, 0, stream>>>(bp, atoms, g, ng, plan, cs, nb, img0, n);
    }
}

// Node sums and interpolation of the images on kPathNodes (each kernel returns at
// once where there is none).
static idiwf_status launch_nodes(const idiwf_geom *geom, const GeomParams &g, const NodeGeom &ng, const BatchParams &bp,
                                 const SplitRecs *split, const DoubleRecs *dbl, NodePlan *plan,
                                 const NodeLayout &nl, char *node_base, WsHeader *hdr, uint64_t *cta_ns, void *out, int out_kind, cudaStream_t stream) {
    const bool nf = geom->flags & IDIWF_NF, sc = geom->flags & IDIWF_SCALE, so = geom->flags & IDIWF_SECONDORDER;
    const NodeBuffers nb = nl.at(node_base, geom);
    const int *first = nl.sort(node_base).first;
    const bool cells = bp.nodes > 1;
    void *fs = out_kind == IDIWF_OUT_C128 ? node_sum_fn<true>(nf, sc, so) : node_sum_fn<false>(nf, sc, so);
    if (dbl)
        fs = nf ? (sc ? (void *)node_sum64_kernel<true, true, false> : (void *)node_sum64_kernel<true, false, false>)
                : (so ? (void *)node_sum64_kernel<false, false, true> : (void *)node_sum64_kernel<false, false, false>);
    void *fx = nf ? (void *)node_interp_x_kernel<true, false>
                  : (sc ? (void *)node_interp_x_kernel<false, true> : (void *)node_interp_x_kernel<false, false>);
    void *fy = dbl ? (void *)node_interp_y_kernel<2> : (void *)node_interp_y_kernel<1>;
    idiwf_status st = ensure_smem(fy, sizeof(GemmSmem));
    if (st == IDIWF_OK) st = ensure_smem(fx, sizeof(GemmSmem));
    if (st == IDIWF_OK) st = ensure_smem((void *)cell_interp_kernel, sizeof(GemmSmem));
    if (st == IDIWF_OK) st = ensure_smem((void *)cell_expand_kernel, sizeof(ExpandSmem));
    if (st != IDIWF_OK) return st;
    const int grid = std::min(sm_count() * resident_ctas(fs, kNodeThreads, 0), kMaxCtas);
    const int egrid = sm_count() * resident_ctas((void *)cell_expand_kernel, kGemmThreads, sizeof(ExpandSmem));
    const int ty = (g.ny + kGemmM - 1) / kGemmM * ((node_cap(g.nx) + kGemmN - 1) / kGemmN);
    const int tx = (g.nx + kGemmM - 1) / kGemmM * ((g.ny + kGemmN - 1) / kGemmN);
    for (int i0 = 0; i0 < bp.n_images; i0 += nl.group) {
        int i1 = std::min(i0 + nl.group, bp.n_images);
        const int n = i1 - i0;
        // (cells: the first group's setup came with the emitters' counts, before the records)
        if (!cells || i0 > 0) launch_setup(g, ng, bp, nullptr, plan, nl, nb, node_base, i0, n, false, stream);
        void *as[] = {(void *)&bp, (void *)&g, (void *)split, &plan, (void *)&nb, &first, &hdr, &cta_ns, &i0, &i1};
        void *ad[] = {(void *)&bp, (void *)&g, (void *)dbl, &plan, (void *)&nb, &hdr, &cta_ns, &i0, &i1};
        IDIWF_CUDA_CHECK(cudaLaunchKernel(fs, dim3(grid), dim3(kNodeThreads), dbl ? ad : as, 0, stream));
        if (cells) {
            cell_interp_kernel<<<dim3(4 * group_blocks(n), n), kGemmThreads, sizeof(GemmSmem), stream>>>(g, plan, nb, i0);
            cell_expand_kernel<<<egrid, kGemmThreads, sizeof(ExpandSmem), stream>>>(g, ng, plan, nb, i0, i1);
        }
        IDIWF_CUDA_CHECK(cudaGetLastError());
        void *ay[] = {(void *)&g, &plan, (void *)&nb, &i0};
        IDIWF_CUDA_CHECK(cudaLaunchKernel(fy, dim3(std::min(ty, 64), n), dim3(kGemmThreads), ay, sizeof(GemmSmem), stream));
        void *ax[] = {(void *)&g, &plan, (void *)&nb, &i0, &out, &out_kind};
        IDIWF_CUDA_CHECK(cudaLaunchKernel(fx, dim3(std::min(tx, 4096), n), dim3(kGemmThreads), ax, sizeof(GemmSmem), stream));
    }
    return IDIWF_OK;
}

// Launch the forward for images [i0, i1) of the batch (records of the whole
// batch are laid out by `rec_base`).
static idiwf_status launch_chunk(const idiwf_geom *geom, const idiwf_batch *b, int precision,
                                 int out_kind, void *out, void *ws, const LaunchShape &s,
                                 int i0, int i1, const std::vector<int64_t> &rec_base, int64_t nrec,
                                 int ksplit, cudaStream_t stream) {
    const GeomParams g = make_geom(geom);
    const int npix = geom->nx * geom->ny;
    const int tile_px = s.threads * s.ppt;
    static thread_local BatchParams bp;  // ~13 KB: keep off the stack
    std::memset(&bp, 0, sizeof(bp));
    bp.n_images = i1 - i0;
    bp.tiles_per_image = (npix + tile_px - 1) / tile_px;
    bp.te = s.te;
    if (precision != IDIWF_SPLIT) ksplit = 1;
    bp.ksplit = ksplit;
    bp.groups = precision == IDIWF_SPLIT && s.groups && geom->ny % kRun == 0;
    bp.nodes = nodes_possible(geom, b, precision, out_kind, s);
    bp.total_units = bp.n_images * bp.tiles_per_image * ksplit;
    int max_tiles = 0;
    std::vector<int> ord(bp.n_images);
    for (int i = 0; i < bp.n_images; ++i) {
        const int64_t n = b->offsets[i0 + i + 1] - b->offsets[i0 + i];
        bp.img[i].src = b->offsets[i0 + i];
        bp.img[i].rec = rec_base[i0 + i];
        bp.img[i].n = (int32_t)n;
        bp.img[i].ntiles = (int32_t)((n + s.te - 1) / s.te);
        const int64_t nblk = (n + kChunkEmitters - 1) / kChunkEmitters;
        bp.img[i].tpc = (int32_t)((nblk + ksplit - 1) / ksplit * (kChunkEmitters / s.te));
        max_tiles = std::max(max_tiles, bp.img[i].ntiles);
        ord[i] = i;
    }
    std::stable_sort(ord.begin(), ord.end(), [&](int a, int c) { return bp.img[a].n > bp.img[c].n; });
    for (int i = 0; i < bp.n_images; ++i) bp.order[i] = (uint16_t)ord[i];

    WsHeader *hdr = static_cast<WsHeader *>(ws);
    uint64_t *cta_ns = reinterpret_cast<uint64_t *>(static_cast<char *>(ws) + kWsTimingOffset);
    void *out_chunk = static_cast<char *>(out) +
                      (size_t)i0 * npix * (out_kind == IDIWF_OUT_C128 ? 16 : (out_kind == IDIWF_OUT_I32 ? 4 : 8));

    // prep
    const NodeLayout nl = bp.nodes ? node_layout(geom, b, precision, bp.nodes) : NodeLayout{};
    char *node_base = static_cast<char *>(ws) + (bp.nodes ? node_region_offset(geom, b, precision, nrec, ksplit) : 0);
    NodePlan *plan = bp.nodes ? reinterpret_cast<NodePlan *>(node_base) : nullptr;
    NodeGeom ng = make_node_geom(g);
    ng.min_pairs = node_min_pairs(precision, out_kind);
    // the header's counters and ticket; its error word and pair count and the CTAs' busy times
    // add up over a call's kernels, so only the first launch clears all of it
    if (i0 == 0) {
        IDIWF_CUDA_CHECK(cudaMemsetAsync(hdr, 0, offsetof(WsHeader, pad), stream));
    } else {
        IDIWF_CUDA_CHECK(cudaMemsetAsync(&hdr->work_counter, 0, sizeof(uint32_t), stream));
        IDIWF_CUDA_CHECK(cudaMemsetAsync(&hdr->work_counter2, 0, 3 * sizeof(uint32_t), stream));  // to the ticket
    }
    if (precision == IDIWF_SPLIT && !plan)
        IDIWF_CUDA_CHECK(cudaMemsetAsync(split_recs(ws, nrec).rmax2, 0, sizeof(uint32_t) * bp.n_images, stream));
    uint32_t *ext = reinterpret_cast<uint32_t *>(node_base + nl.ext);
    if (plan) IDIWF_CUDA_CHECK(cudaMemsetAsync(ext, 0, (size_t)bp.n_images * 4 * kNodeExt, stream));
    uint64_t *clear_ns = i0 == 0 ? cta_ns : nullptr;
    if (max_tiles == 0 && !plan) {
        if (clear_ns) IDIWF_CUDA_CHECK(cudaMemsetAsync(clear_ns, 0, sizeof(uint64_t) * kMaxCtas, stream));
    } else {  // (the prep kernel also writes the plan)
        dim3 pgrid((unsigned)std::max<int64_t>(std::min<int64_t>(((int64_t)max_tiles * s.te + 255) / 256, 1024), 1),
                   bp.n_images);
        if (precision == IDIWF_SPLIT) {
            const int w_mode = (geom->flags & IDIWF_NF) ? 1 : ((geom->flags & IDIWF_SECONDORDER) ? 2 : 0);
            // emitter coordinates must keep |q.r| inside the magic binade
            const double max_abs = kMaxTurns / (3.0 * 2.0 * geom->k * kInvTwoPi);
            const CellSort cs = nl.sort(node_base);
            if (bp.nodes > 1) {
                // extents and plan, the emitters' sort by cell, then the records
                node_extents_kernel<<<pgrid, 256, 0, stream>>>(bp, b->atoms, b->amplitudes, b->amp_dtype, ext, hdr, g,
                                                               ng, plan);
                launch_setup(g, ng, bp, b->atoms, plan, nl, nl.at(node_base, geom), node_base, 0,
                             std::min(nl.group, bp.n_images), true, stream);
                prep_split_kernel<false><<<pgrid, 256, 0, stream>>>(bp, b->atoms, b->amplitudes, b->amp_dtype, w_mode,
                                                                    max_abs, split_recs(ws, nrec), hdr, g, ng, ext,
                                                                    plan, cs, clear_ns);
            } else {
                prep_split_kernel<true><<<pgrid, 256, 0, stream>>>(bp, b->atoms, b->amplitudes, b->amp_dtype, w_mode,
                                                                   max_abs, split_recs(ws, nrec), hdr, g, ng, ext,
                                                                   plan, cs, clear_ns);
            }
        } else {
            prep_double_kernel<<<pgrid, 256, 0, stream>>>(bp, b->atoms, b->amplitudes, b->amp_dtype,
                                                          double_recs(ws, nrec), hdr, g, ng, ext, plan, clear_ns);
        }
        IDIWF_CUDA_CHECK(cudaGetLastError());
    }

    auto grid_for = [&](void *fn, size_t smem, int &grid) -> idiwf_status {
        idiwf_status st = ensure_smem(fn, smem);
        if (st != IDIWF_OK) return st;
        const int per_sm = std::min(s.ctas_per_sm, resident_ctas(fn, s.threads, smem));
        grid = (int)std::min<int64_t>(std::min<int64_t>(bp.total_units, (int64_t)sm_count() * per_sm), kMaxCtas);
        return IDIWF_OK;
    };
    if (precision == IDIWF_SPLIT) {
        SplitRecs rec = split_recs(ws, nrec);
        double2 *partials = ksplit > 1 ? reinterpret_cast<double2 *>(static_cast<char *>(ws) + kWsDataOffset +
                                                                     split_recs_bytes(nrec))
                                       : nullptr;
        void *args[] = {&bp, (void *)&g, &rec, &out_chunk, &out_kind, &hdr, &cta_ns, &partials, &plan};
        // the pixel-run kernel, the per-pixel kernel for the images beyond the
        // runs' bound, and in the near field the exact kernel (each returns at
        // once when it has no image)
        for (const int path : {kPathRuns, kPathPixel, kPathExact}) {
            if (path == kPathRuns && !bp.groups) continue;
            if (path == kPathExact && !(geom->flags & IDIWF_NF)) continue;
            void *fn = kernel_for(precision, s.ppt, geom->flags, ksplit > 1, path);
            const size_t smem = fwd_smem(precision, s, path);
            int grid = 0;
            idiwf_status st = grid_for(fn, smem, grid);
            if (st != IDIWF_OK) return st;
            IDIWF_CUDA_CHECK(cudaLaunchKernel(fn, dim3(grid), dim3(s.threads), args, smem, stream));
        }
        if (ksplit > 1) {
            const int64_t total = (int64_t)bp.n_images * npix;
            const int blocks = (int)std::min<int64_t>((total + 255) / 256, 8 * (int64_t)sm_count());
            const bool nf = geom->flags & IDIWF_NF, sc = geom->flags & IDIWF_SCALE;
            if (nf)
                fwd_finish_kernel<true, false><<<blocks, 256, 0, stream>>>(g, partials, ksplit, bp.n_images,
                                                                           out_chunk, out_kind, plan);
            else if (sc)
                fwd_finish_kernel<false, true><<<blocks, 256, 0, stream>>>(g, partials, ksplit, bp.n_images,
                                                                           out_chunk, out_kind, plan);
            else
                fwd_finish_kernel<false, false><<<blocks, 256, 0, stream>>>(g, partials, ksplit, bp.n_images,
                                                                            out_chunk, out_kind, plan);
            IDIWF_CUDA_CHECK(cudaGetLastError());
        }
        if (plan && !s.direct_only)
            return launch_nodes(geom, g, ng, bp, &rec, nullptr, plan, nl, node_base, hdr, cta_ns, out_chunk, out_kind, stream);
    } else {
        DoubleRecs rec = double_recs(ws, nrec);
        void *args[] = {&bp, (void *)&g, &rec, &out_chunk, &out_kind, &hdr, &cta_ns, &plan};
        void *fn = kernel_for(precision, s.ppt, geom->flags, false);
        const size_t smem = fwd_smem(precision, s, kPathPixel);
        int grid = 0;
        idiwf_status st = grid_for(fn, smem, grid);
        if (st != IDIWF_OK) return st;
        IDIWF_CUDA_CHECK(cudaLaunchKernel(fn, dim3(grid), dim3(s.threads), args, smem, stream));
        if (plan && !s.direct_only)
            return launch_nodes(geom, g, ng, bp, nullptr, &rec, plan, nl, node_base, hdr, cta_ns, out_chunk, out_kind, stream);
    }
    return IDIWF_OK;
}

static idiwf_status forward_impl(const idiwf_geom *geom, const idiwf_batch *b, int precision,
                                 int out_kind, void *out, void *ws, size_t ws_bytes,
                                 const LaunchShape &s, cudaStream_t stream) {
    const size_t need = forward_ws_bytes(geom, b, precision, s);
    if (!ws || ws_bytes < need)
        return set_error(IDIWF_ERR_WORKSPACE, "workspace smaller than idiwf_forward_workspace_size()");
    if (reinterpret_cast<uintptr_t>(ws) & 255) return set_error(IDIWF_ERR_WORKSPACE, "workspace must be 256-byte aligned");
    std::vector<int64_t> rec_base(b->n_images + 1, 0);
    const int nodes = nodes_possible(geom, b, precision, out_kind, s);
    for (int i = 0; i < b->n_images; ++i)
        rec_base[i + 1] = rec_base[i] + image_records(b->offsets[i + 1] - b->offsets[i], s.te, nodes);
    const int64_t nrec = std::max<int64_t>(rec_base[b->n_images], 1);
    const int ksplit = precision == IDIWF_SPLIT ? choose_ksplit(geom, b) : 1;
    for (int i0 = 0; i0 < b->n_images; i0 += kMaxImagesPerLaunch) {
        const int i1 = std::min(b->n_images, i0 + kMaxImagesPerLaunch);
        idiwf_status st =
            launch_chunk(geom, b, precision, out_kind, out, ws, s, i0, i1, rec_base, nrec, ksplit, stream);
        if (st != IDIWF_OK) return st;
    }
    return IDIWF_OK;
}

}  // namespace idiwf

using namespace idiwf;

extern "C" size_t idiwf_forward_workspace_size(const idiwf_geom *geom, const idiwf_batch *batch,
                                               int32_t precision, const idiwf_config *cfg) {
    if (validate_geom(geom) != IDIWF_OK || validate_batch(batch) != IDIWF_OK) return 0;
    if (precision != IDIWF_SPLIT && precision != IDIWF_DOUBLE) return 0;
    // size for the largest tile any shape may use, so a tuned shape always fits
    LaunchShape s;
    if (resolve_shape(geom, batch, precision, cfg, s) != IDIWF_OK) return 0;
    LaunchShape big = s;
    big.te = 1024;
    return std::max(forward_ws_bytes(geom, batch, precision, s), forward_ws_bytes(geom, batch, precision, big));
}

extern "C" idiwf_status idiwf_forward(const idiwf_geom *geom, const idiwf_batch *batch, int32_t precision,
                                      int32_t out_kind, void *out, void *workspace, size_t workspace_bytes,
                                      const idiwf_config *cfg, cudaStream_t stream) {
    idiwf_status st = validate_geom(geom);
    if (st != IDIWF_OK) return st;
    if ((st = validate_batch(batch)) != IDIWF_OK) return st;
    if (precision != IDIWF_SPLIT && precision != IDIWF_DOUBLE)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "precision must be IDIWF_SPLIT or IDIWF_DOUBLE");
    if (out_kind < IDIWF_OUT_C128 || out_kind > IDIWF_OUT_I32)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "unknown out_kind");
    if (!out) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "out is NULL");
    LaunchShape s;
    if ((st = resolve_shape(geom, batch, precision, cfg, s)) != IDIWF_OK) return st;
    return forward_impl(geom, batch, precision, out_kind, out, workspace, workspace_bytes, s, stream);
}

extern "C" idiwf_status idiwf_forward_cta_times(const void *workspace, uint64_t *host_ns, int32_t cap,
                                                int32_t *n, cudaStream_t stream) {
    if (!workspace || !host_ns || !n || cap <= 0) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "bad arguments");
    WsHeader h;
    IDIWF_CUDA_CHECK(cudaMemcpyAsync(&h, workspace, sizeof(h), cudaMemcpyDeviceToHost, stream));
    IDIWF_CUDA_CHECK(cudaStreamSynchronize(stream));
    const int cnt = std::min<int>((int)h.n_ctas, std::min(cap, kMaxCtas));
    if (cnt > 0)
        IDIWF_CUDA_CHECK(cudaMemcpyAsync(host_ns, static_cast<const char *>(workspace) + kWsTimingOffset,
                                         sizeof(uint64_t) * cnt, cudaMemcpyDeviceToHost, stream));
    IDIWF_CUDA_CHECK(cudaStreamSynchronize(stream));
    *n = cnt;
    return IDIWF_OK;
}

extern "C" idiwf_status idiwf_tune(const idiwf_geom *geom, const idiwf_batch *batch, int32_t precision,
                                   int32_t out_kind, void *out, void *workspace, size_t workspace_bytes,
                                   cudaStream_t stream, idiwf_config *best) {
    idiwf_status st = validate_geom(geom);
    if (st != IDIWF_OK) return st;
    if ((st = validate_batch(batch)) != IDIWF_OK) return st;
    if (precision != IDIWF_SPLIT && precision != IDIWF_DOUBLE)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "precision must be IDIWF_SPLIT or IDIWF_DOUBLE");
    // The shape is the direct kernels': images on nodes do not run them, and their own kernels'
    // time would drown the differences.  So the direct images alone are timed, and a batch
    // without any keeps the default shape and leaves the cache to others' tuning.
    LaunchShape best_s = default_shape(precision);
    bool tune = true;
    if (nodes_possible(geom, batch, precision, out_kind, best_s)) {
        best_s.direct_only = true;
        if ((st = forward_impl(geom, batch, precision, out_kind, out, workspace, workspace_bytes, best_s, stream)) != IDIWF_OK)
            return st;
        WsHeader h;
        IDIWF_CUDA_CHECK(cudaMemcpyAsync(&h, workspace, sizeof(h), cudaMemcpyDeviceToHost, stream));
        IDIWF_CUDA_CHECK(cudaStreamSynchronize(stream));
        tune = h.direct > 0;
    }
    std::vector<LaunchShape> cands;
    if (precision == IDIWF_SPLIT) {
        // CTAs per SM: as many as fit.  The persistent queue balances any grid,
        // and a small tuning batch would favour fewer CTAs only through its
        // own last-wave tail.
        for (int th : {128, 256})
            for (int ppt : {2, 4, 8})
                for (int te : {256, 512}) {
                    LaunchShape c{th, ppt, te, 1};
                    void *fn = kernel_for(precision, ppt, geom->flags, false);
                    const size_t smem = fwd_smem(precision, c, kPathRuns);
                    if (ensure_smem(fn, smem) != IDIWF_OK) continue;
                    c.ctas_per_sm = std::min(8, resident_ctas(fn, th, smem));
                    cands.push_back(c);
                }
    } else {
        for (int th : {128, 256})
            for (int ppt : {1, 2})
                for (int te : {64, 128}) cands.push_back(LaunchShape{th, ppt, te, 2});
    }
    // Time each shape on the whole batch (the caller sizes the batch it tunes
    // on; one warm-up + best of two timed runs per shape).
    cudaEvent_t e0, e1;
    IDIWF_CUDA_CHECK(cudaEventCreate(&e0));
    IDIWF_CUDA_CHECK(cudaEventCreate(&e1));
    float best_ms = 1e30f;
    for (LaunchShape &s : cands) {
        if (!tune) break;
        s.direct_only = true;
        if (forward_ws_bytes(geom, batch, precision, s) > workspace_bytes) continue;
        {  // more CTAs per SM than fit would only repeat a smaller candidate
            void *fn = kernel_for(precision, s.ppt, geom->flags, false);
            const size_t smem = fwd_smem(precision, s, kPathRuns);
            if (ensure_smem(fn, smem) == IDIWF_OK && s.ctas_per_sm > resident_ctas(fn, s.threads, smem)) continue;
        }
        st = forward_impl(geom, batch, precision, out_kind, out, workspace, workspace_bytes, s, stream);
        if (st != IDIWF_OK) break;
        float ms_best = 1e30f;
        for (int rep = 0; rep < 2; ++rep) {
            cudaEventRecord(e0, stream);
            st = forward_impl(geom, batch, precision, out_kind, out, workspace, workspace_bytes, s, stream);
            cudaEventRecord(e1, stream);
            if (st != IDIWF_OK) break;
            cudaEventSynchronize(e1);
            float ms = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            ms_best = std::min(ms_best, ms);
        }
        if (st != IDIWF_OK) break;
        if (ms_best < best_ms) {
            best_ms = ms_best;
            best_s = s;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st != IDIWF_OK) return st;
    IDIWF_CUDA_CHECK(cudaGetLastError());
    best_s.direct_only = false;
    // the batch's result, every image's
    if ((st = forward_impl(geom, batch, precision, out_kind, out, workspace, workspace_bytes, best_s, stream)) != IDIWF_OK)
        return st;
    IDIWF_CUDA_CHECK(cudaStreamSynchronize(stream));
    if (tune) {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_tune_cache[TuneKey{precision, geom->flags, geom->nx, geom->ny, n_bucket(batch)}] = best_s;
    }
    if (best) {
        best->threads = best_s.threads;
        best->pixels_per_thread = best_s.ppt;
        best->emitters_per_tile = best_s.te;
        best->ctas_per_sm = best_s.ctas_per_sm;
        best->pixel_groups = best_s.groups ? 1 : -1;
    }
    return IDIWF_OK;
}

// ---------------------------------------------------------------------------
// Split-precision forward for callers that cannot allocate device memory.
//
// Some hosts of this library cannot call cudaMalloc at all: code that runs
// inside another framework's memory pool or allocator hooks, inside a stream
// capture they do not own, or in plug-ins whose host forbids device
// allocation.  For them this entry point keeps its scratch (work counters,
// error word, per-CTA timing, emitter tile records) in one file-scope device
// array of fixed size, so the caller passes only inputs and outputs and no
// device memory is allocated.  The host side uses no heap either: the launch
// descriptor is a static buffer, used under a mutex for the few microseconds
// it takes to build it and enqueue the launches (kernel arguments are copied
// at launch).
// ---------------------------------------------------------------------------
namespace idiwf {

static __device__ __align__(256) unsigned char g_noalloc_scratch[IDIWF_NOALLOC_SCRATCH_BYTES];

constexpr int kNoAllocMaxDevices = 64;
static std::mutex g_noalloc_mu;
static void *g_noalloc_ptr[kNoAllocMaxDevices];
static BatchParams g_noalloc_bp;  // guarded by g_noalloc_mu

// Device address of the scratch array on the current device.  The name
// g_noalloc_scratch in host code is only a host-side stand-in, so the
// address is looked up once per device (with that device current) and
// cached.  The caller holds g_noalloc_mu.
static idiwf_status noalloc_scratch_locked(void **ptr) {
    int dev = 0;
    IDIWF_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices)
        return set_error(IDIWF_ERR_UNSUPPORTED, "idiwf_forward_noalloc: device ordinal out of range");
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_error(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
        g_noalloc_ptr[dev] = p;
    }
    *ptr = g_noalloc_ptr[dev];
    return IDIWF_OK;
}

}  // namespace idiwf

extern "C" idiwf_status idiwf_forward_noalloc(const idiwf_geom *geom, const idiwf_batch *batch, int32_t out_kind,
                                              void *out, cudaStream_t stream) {
    idiwf_status st = validate_geom(geom);
    if (st != IDIWF_OK) return st;
    if ((st = validate_batch(batch)) != IDIWF_OK) return st;
    if (out_kind < IDIWF_OUT_C128 || out_kind > IDIWF_OUT_I32)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "unknown out_kind");
    if (!out) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "out is NULL");
    if (batch->n_images > kMaxImagesPerLaunch)
        return set_error(IDIWF_ERR_UNSUPPORTED, "idiwf_forward_noalloc: at most 512 images per call");

    const LaunchShape s{256, 4, 256, 2};
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    BatchParams &bp = g_noalloc_bp;
    std::memset(&bp, 0, sizeof(bp));
    const int npix = geom->nx * geom->ny;
    const int tile_px = s.threads * s.ppt;
    bp.n_images = batch->n_images;
    bp.tiles_per_image = (npix + tile_px - 1) / tile_px;
    bp.te = s.te;
    bp.total_units = bp.n_images * bp.tiles_per_image;
    bp.groups = geom->ny % kRun == 0;
    int64_t nrec = 0;
    int max_tiles = 0;
    for (int i = 0; i < bp.n_images; ++i) {
        const int64_t n = batch->offsets[i + 1] - batch->offsets[i];
        bp.img[i].src = batch->offsets[i];
        bp.img[i].rec = nrec;
        bp.img[i].n = (int32_t)n;
        bp.img[i].ntiles = (int32_t)((n + s.te - 1) / s.te);
        nrec += (int64_t)bp.img[i].ntiles * s.te;
        max_tiles = std::max(max_tiles, bp.img[i].ntiles);
    }
    nrec = std::max<int64_t>(nrec, 1);
    if (kWsDataOffset + split_recs_bytes(nrec) > (size_t)IDIWF_NOALLOC_SCRATCH_BYTES)
        return set_error(IDIWF_ERR_UNSUPPORTED,
                         "idiwf_forward_noalloc: batch needs more than the 16 MiB static scratch "
                         "(at most 321792 emitters in total after padding every image to a multiple of 256); "
                         "use idiwf_forward with a caller workspace");
    // images by descending emitter count (stable insertion sort, no heap)
    for (int i = 0; i < bp.n_images; ++i) {
        int j = i;
        while (j > 0 && bp.img[bp.order[j - 1]].n < bp.img[i].n) {
            bp.order[j] = bp.order[j - 1];
            --j;
        }
        bp.order[j] = (uint16_t)i;
    }

    void *ws = nullptr;
    if ((st = noalloc_scratch_locked(&ws)) != IDIWF_OK) return st;
    WsHeader *hdr = static_cast<WsHeader *>(ws);
    uint64_t *cta_ns = reinterpret_cast<uint64_t *>(static_cast<char *>(ws) + kWsTimingOffset);
    SplitRecs rec = split_recs(ws, nrec);
    const GeomParams g = make_geom(geom);

    // every call starts from zero work counters and a zero error word; the
    // records are rewritten in full by the prep kernel
    IDIWF_CUDA_CHECK(cudaMemsetAsync(ws, 0, offsetof(WsHeader, pad), stream));
    IDIWF_CUDA_CHECK(cudaMemsetAsync(rec.rmax2, 0, sizeof(uint32_t) * bp.n_images, stream));
    if (max_tiles > 0) {
        const int w_mode = (geom->flags & IDIWF_NF) ? 1 : ((geom->flags & IDIWF_SECONDORDER) ? 2 : 0);
        const double max_abs = kMaxTurns / (3.0 * 2.0 * geom->k * kInvTwoPi);
        dim3 pgrid((unsigned)std::min<int64_t>(((int64_t)max_tiles * s.te + 255) / 256, 1024), bp.n_images);
        prep_split_kernel<true><<<pgrid, 256, 0, stream>>>(bp, batch->atoms, batch->amplitudes, batch->amp_dtype, w_mode,
                                                           max_abs, rec, hdr, g, NodeGeom{}, nullptr,
                                                           nullptr, CellSort{}, cta_ns);
        IDIWF_CUDA_CHECK(cudaGetLastError());
    } else {
        IDIWF_CUDA_CHECK(cudaMemsetAsync(cta_ns, 0, sizeof(uint64_t) * kMaxCtas, stream));
    }
    double2 *no_partials = nullptr;  // bp.ksplit == 0: the kernels write the outputs themselves
    NodePlan *no_plan = nullptr;         // every image takes its direct path
    void *args[] = {&bp, (void *)&g, &rec, &out, &out_kind, &hdr, &cta_ns, &no_partials, &no_plan};
    // the pixel-run, per-pixel and (near field) exact kernels, each returning
    // at once without images; the persistent grid is clamped to the CTAs that
    // fit at once, as in idiwf_forward
    for (const int path : {kPathRuns, kPathPixel, kPathExact}) {
        if (path == kPathRuns && !bp.groups) continue;
        if (path == kPathExact && !(geom->flags & IDIWF_NF)) continue;
        void *fn = split_kernel_for<4>(geom->flags, false, path);
        const size_t smem = fwd_smem(IDIWF_SPLIT, s, path);
        IDIWF_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int occ = 0;
        IDIWF_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, s.threads, smem));
        const int per_sm = std::max(1, std::min(s.ctas_per_sm, occ));
        const int grid = (int)std::min<int64_t>(std::min<int64_t>(bp.total_units, (int64_t)sm_count() * per_sm),
                                                kMaxCtas);
        IDIWF_CUDA_CHECK(cudaLaunchKernel(fn, dim3(grid), dim3(s.threads), args, smem, stream));
    }
    return IDIWF_OK;
}

// Error word of the most recent idiwf_forward_noalloc call on the current
// device, read from the static scratch into a stack variable (no allocation;
// the read waits for `stream`).  Same bits and statuses as
// idiwf_workspace_error.
extern "C" idiwf_status idiwf_forward_noalloc_error(cudaStream_t stream) {
    void *ws = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        idiwf_status st = noalloc_scratch_locked(&ws);
        if (st != IDIWF_OK) return st;
    }
    return idiwf_workspace_error(ws, stream);
}
