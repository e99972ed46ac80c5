// Time-dependent direct sum for sm_100a (FP64).
//
// Per pixel p (reference: idi/simulation/time.py:48-98, simtime.cu:50-148):
//   t_j   = -s_j / c + t0_j          s_j = (d/|d| - zhat) . r_j   (far field)
//   a_j   = exp(-i (s_j k - psi_j)) [ / |d| ]
//   sort (t_j, a_j) by t_j
//   x_0 = a_0,  x_m = a_m + exp(-(t_m - t_{m-1})/tau) x_{m-1}
//   I_p = sum_{m<n-1} -tau/2 |x_m|^2 expm1(-2 (t_{m+1}-t_m)/tau) + tau/2 |x_{n-1}|^2
//
// One CTA handles one pixel at a time, with 32 to 512 threads by the emitter
// count, so that up to 16 pixels share an SM; CTAs take equal shares of consecutive
// pixels and walk them in serpentine order (row by row, every other row backwards),
// so consecutive pixels of a CTA are detector neighbours.  Arrival times are
// computed in FP64 with the exact rounding sequence of the reference (np.inner as
// fma(q2,z,fma(q1,y,q0*x)), IEEE division by c), so the keys -- and therefore
// the sorted order -- are bit for bit those of the reference.
//
// Sorting.  Between neighbouring pixels the keys move by far less than their
// spacing (the arrival-time spread of the emission times dominates the
// geometric term), so the previous pixel's order is almost the new one.  The
// kernel keeps the order in shared memory as position-ordered 16-bit emitter
// indices and the keys in a table by emitter, and repairs the order while it scans
// it: short windows around the starts of the threads' runs, then every thread
// streams its run through a sorted buffer of four entries (scan_run), with an exact
// check.  Where that is not enough, insertion sorts over windows of one run each,
// alternating between two window grids offset by half a run until every window
// boundary is in order (each window is sorted, so the whole array is sorted exactly
// when every boundary pair is).  After a bounded number of window passes -- and for
// a CTA's first pixel -- the exact full sort runs: 16 buckets per thread by a
// monotone FP64 map of the key (so bucket order is key order), insertion sort inside
// each bucket by (key, emitter index), and an on-chip LSD radix sort (8 passes of 8
// bits, per-warp ranking with __match_any_sync) if a bucket overflows.  Every path
// sorts by (key, emitter index), so the order does not depend on which one ran.
//
// The decaying scan is one pass: each thread keeps its run of up to 40 positions as
// an affine map x -> D x + B plus three sums from which the run's share of the
// interval integral follows once the block scan delivers the entering x.
//
// What bounds it.  20,000 emitters, 256 x 256 pixels (one CTA per SM), cycles per
// pixel: key pass 12k (40 bytes per emitter from L2 at 64 B per cycle and SM), run
// starts 4k, streaming scan 43k, run ends and block scan 6k.  The scan gathers one
// 32-byte row per emitter, every lane from another line, and an SM issues one line
// request to L2 in about two cycles, which is those 43k (measured by taking parts
// out: without sine, cosine and expm1 43k, without the gather 26k).  15.3 ms, against
// 18.2 ms when the order was repaired by a window pass of its own (18k cycles) ahead
// of the scan.  Phases kept in shared memory beside the keys, where they fit (up to
// 11,000 emitters), measured no faster: below 10,000 emitters it is FP64 and issue at
// 16 warps per SM.

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "idiwf_internal.cuh"

namespace idiwf {

constexpr int kTimeThreads = 512;  // most threads of a CTA (time_kernel), all of them (time_kernel_large)
constexpr int kTimeWarps = kTimeThreads / 32;
constexpr int kTimeIPT = 40;                                 // most positions per thread
constexpr int kTimeMaxN = kTimeThreads * kTimeIPT;           // 20480
constexpr int kCoarse = 1024;                                // coarse bins of the large kernel's bucket map

// Shape of one on-chip pixel: `threads` threads of `ipt` positions each (even,
// threads * ipt >= n).  The position-ordered index array has two pad slots after
// every two runs, so that the runs of a warp's threads start in different banks
// when every thread walks its own run, and a pair of positions (even, odd) stays
// one 32-bit word.
struct TimeShape {
    int threads, ipt;
    uint32_t inv_group;  // ceil(2^32 / (2 ipt)): m / (2 ipt) = umulhi(m, inv_group) for m < 2^15
    int smem;            // dynamic shared memory, bytes
};
__device__ __forceinline__ int slot(const TimeShape &sh, int m) { return m + 2 * (int)__umulhi((uint32_t)m, sh.inv_group); }
// Shared memory: key table by emitter, order slots, per-warp digit counters (the
// bucket counters, 16 per thread of 16 bits, share them), digit bases or coarse
// bins (2 per thread), and 8 doubles of scratch per warp.
static TimeShape time_shape(int threads, int n) {
    TimeShape s;
    s.threads = threads;
    s.ipt = 2 * std::max(1, (n + 2 * threads - 1) / (2 * threads));
    s.inv_group = (uint32_t)((((uint64_t)1 << 32) + 2 * s.ipt - 1) / (uint64_t)(2 * s.ipt));
    s.smem = threads * s.ipt * 8 + (threads * s.ipt + threads) * 2 + (threads / 32) * 1024 +
             std::max(256, 2 * threads + 4) * 4 + (threads / 32) * 64;
    return s;
}
// Shared memory of one SM and what each resident CTA takes beside its dynamic part.
constexpr int kSmShared = 228 * 1024, kCtaShared = 1024 + 256;
// The largest shape's (every launch sets this limit, whatever its own size, so that
// calls from several threads do not lower it under one another).
constexpr int kTimeSmemMax = kTimeMaxN * 8 + (kTimeMaxN + kTimeThreads) * 2 + kTimeWarps * 1024 +
                             (2 * kTimeThreads + 4) * 4 + kTimeWarps * 64;
static_assert(kTimeSmemMax + kCtaShared <= kSmShared, "time kernel shared memory above the per-block limit");
// Window passes tried on the previous pixel's order before the full sort.
constexpr int kWarmPasses = 8;
// Failed warm starts in a row after which a CTA stops trying them.
constexpr int kWarmMaxFails = 3;
// Key of the padding positions from n on in a radix sort: the positive NaN
// with the largest payload, whose order-preserving image is the largest of all
// 64-bit patterns, so the radix sort leaves the padding behind every real key
// (NaN keys included) and positions below n always hold real emitters.
constexpr long long kPadKeyBits = 0x7FFFFFFFFFFFFFFFll;

__device__ __forceinline__ uint64_t sortable(double v) {
    const uint64_t b = (uint64_t)__double_as_longlong(v);
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

// Order digest base: H = sum_m (j_m + 1) B^m mod 2^64 over the sorted emitter
// indices j_m.  B = 1 mod 4, so B^d - 1 has at most 2 + log2(d) factors of 2
// and swapping two indices (differing by less than 2^15, at positions less
// than 2^15 apart) always changes H.
constexpr uint64_t kDigestBase = 0x9E3779B97F4A7C15ull;
__device__ __forceinline__ uint64_t digest_pow(int e) {
    uint64_t r = 1, b = kDigestBase;
    while (e) {
        if (e & 1) r *= b;
        b *= b;
        e >>= 1;
    }
    return r;
}

struct Affine {
    double d, br, bi;
};
// apply `first` then `second`
__device__ __forceinline__ Affine compose(const Affine &first, const Affine &second) {
    Affine r;
    r.d = second.d * first.d;
    r.br = fma(second.d, first.br, second.br);
    r.bi = fma(second.d, first.bi, second.bi);
    return r;
}

// Correctly rounded quotient a / c from ic = RN(1 / c): q0 = RN(a ic) is a
// faithful quotient, r = a - c q0 is exact in one FMA, and RN(q0 + r ic) is
// RN(a / c) (Markstein's theorem: P. Markstein, IBM J. Res. Dev. 34(1), 1990;
// Muller et al., Handbook of Floating-Point Arithmetic, the theorem on
// FMA-based correction of a faithful quotient).  The theorem needs normal
// numbers away from underflow and overflow: quotients outside [2^-960, 2^1000]
// in magnitude -- zeros, infinities and NaN included -- take the IEEE division
// (which keeps a zero's sign and an infinity).  Bit-exact against the division
// (the arrival keys must be the reference's bits).
__device__ __forceinline__ double div_rn(double a, double c, double ic) {
    const double q0 = __dmul_rn(a, ic);
    if (!(fabs(q0) >= 0x1p-960 && fabs(q0) <= 0x1p1000)) return __ddiv_rn(a, c);
    const double r = __fma_rn(-c, q0, a);
    return __fma_rn(r, ic, q0);
}

// div_rn's range [2^-960, 2^1000] on the high word of |q0|: from kDivLow, kDivSpan wide.
constexpr uint32_t kDivLow = (1023u - 960u) << 20, kDivSpan = 1960u << 20;

// MK: divide by c with div_rn (the on-chip kernel) or the library division (the
// large-count kernel, whose 64 registers the inlined correction would spill);
// both give the correctly rounded quotient.
// One 32-byte emitter row (x, y, z, phase) in a single 256-bit load; the
// rows are 32-byte aligned (the entry points require it of the emitter array).
__device__ __forceinline__ double4 ld_row(const double4 *p) {
    double4 r;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
    return r;
}

template <bool NF, bool SCALE, bool MK = true>
__device__ __forceinline__ void arrival(const GeomParams &g, double dx, double dy, double dz, double dn,
                                        double q0, double q1, double q2, const double4 &a, double t0,
                                        double c, double ic, double &t, double &s_out, double &dist_out) {
    if (!NF) {
        const double s = __fma_rn(q2, a.z, __fma_rn(q1, a.y, __dmul_rn(q0, a.x)));
        t = __dadd_rn(MK ? div_rn(-s, c, ic) : __ddiv_rn(-s, c), t0);
        s_out = s;
        dist_out = dn;
    } else {
        const double ax = __dsub_rn(dx, a.x), ay = __dsub_rn(dy, a.y), az = __dsub_rn(dz, a.z);
        const double dist = __dsqrt_rn(__fma_rn(az, az, __fma_rn(ax, ax, __dmul_rn(ay, ay))));
        const double s = __dadd_rn(__dsub_rn(dist, dn), a.z);
        t = __dadd_rn(MK ? div_rn(s, c, ic) : __ddiv_rn(s, c), t0);
        s_out = s;
        dist_out = dist;
    }
}

// Path difference s (and the 1/r distance) of one emitter, as arrival() but
// without forming the arrival time (the scan reads times from the key table).
template <bool NF>
__device__ __forceinline__ void path_only(double dx, double dy, double dz, double dn, double q0, double q1,
                                          double q2, const double4 &a, double &s_out, double &dist_out) {
    if (!NF) {
        s_out = __fma_rn(q2, a.z, __fma_rn(q1, a.y, __dmul_rn(q0, a.x)));
        dist_out = dn;
    } else {
        const double ax = __dsub_rn(dx, a.x), ay = __dsub_rn(dy, a.y), az = __dsub_rn(dz, a.z);
        const double dist = __dsqrt_rn(__fma_rn(az, az, __fma_rn(ax, ax, __dmul_rn(ay, ay))));
        s_out = __dadd_rn(__dsub_rn(dist, dn), a.z);
        dist_out = dist;
    }
}

// expm1(-x), x >= 0, for the scan.  The arguments are gaps between
// neighbouring arrival times over tau, almost always far below 1: up to 2^-4
// a Taylor polynomial of degree 10 in Horner form (coefficients 1/k!) is exact
// to FP64 rounding (the first omitted term is below 3e-19 of the result);
// larger arguments use the library function.  (The on-chip kernel uses it; in
// the 64-register large-count kernel the inlined polynomial measured slower
// than the library calls.)  The coefficient tables of this file live in
// constant memory: an FP64 FMA takes a constant-bank operand directly, where a
// 64-bit literal costs two moves into registers (measured: half the
// instructions of the polynomials).
__constant__ double kInvFact[11] = {1.0,       1.0,        1.0 / 2,     1.0 / 6,      1.0 / 24,      1.0 / 120,
                                    1.0 / 720, 1.0 / 5040, 1.0 / 40320, 1.0 / 362880, 1.0 / 3628800};
__device__ __forceinline__ double expm1_near(double x) {
    const double t = -x;
    double q = kInvFact[10];
#pragma unroll
    for (int k = 9; k >= 1; --k) q = __fma_rn(q, t, kInvFact[k]);
    return t * q;  // t (1 + t/2! + ... + t^9/10!)
}
__device__ __forceinline__ double expm1_neg(double x) { return x <= 0.0625 ? expm1_near(x) : expm1(-x); }

// sin and cos of x (FP64), for the time path's amplitudes.  Cody-Waite
// reduction (W. J. Cody and W. Waite, Software Manual for the Elementary
// Functions, 1980): n = rint(x 2/pi), a = (x - n P1) - n P2 with P1 + P2 = pi/2
// to twice the precision (P1 = RN(pi/2), P2 = RN(pi/2 - P1)), |a| <= pi/4 up
// to rounding, good to ~1e-16 rad for |x| far below 2^40; then the Taylor
// series of sin and cos (coefficients (-1)^k / k!) to degrees 17 and 18, whose
// first omitted terms are below 1e-19 on |a| <= pi/4, in Horner form over a^2;
// the quadrant n mod 4 swaps and negates.  Arguments beyond 2^30 take the
// library function.
// Cody-Waite constants {2/pi, P1, P2} and the Taylor coefficients of sin
// (degree 17 down to 3) and cos (degree 18 down to 2), highest first.
__constant__ double kCW[3] = {0.63661977236758134308, 1.5707963267948966192, 6.123233995736766036e-17};
__constant__ double kSinC[8] = {1.0 / 355687428096000.0, -1.0 / 1307674368000.0, 1.0 / 6227020800.0,
                                -1.0 / 39916800.0,       1.0 / 362880.0,         -1.0 / 5040.0,
                                1.0 / 120.0,             -1.0 / 6.0};
__constant__ double kCosC[9] = {1.0 / 6402373705728000.0, -1.0 / 20922789888000.0, 1.0 / 87178291200.0,
                                -1.0 / 479001600.0,       1.0 / 3628800.0,         -1.0 / 40320.0,
                                1.0 / 720.0,              -1.0 / 24.0,             0.5};
__device__ __forceinline__ void sincos_near(double x, double &sn, double &cs) {
    // rint by the 1.5 2^52 addition, whose sum holds n in its low bits (|n| < 2^31)
    const double big = __fma_rn(x, kCW[0], 0x1.8p52);
    const double nd = big - 0x1.8p52;
    double a = __fma_rn(-nd, kCW[1], x);
    a = __fma_rn(-nd, kCW[2], a);
    const double a2 = a * a;
    double ps = kSinC[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) ps = __fma_rn(ps, a2, kSinC[i]);
    const double s = __fma_rn(a * a2, ps, a);
    double pc = kCosC[0];
#pragma unroll
    for (int i = 1; i < 9; ++i) pc = __fma_rn(pc, a2, kCosC[i]);
    const double co = __fma_rn(-a2, pc, 1.0);
    const int q = __double2loint(big) & 3;
    sn = (q & 1) ? co : s;
    cs = (q & 1) ? s : co;
    if (q == 1 || q == 2) cs = -cs;
    if (q >= 2) sn = -sn;
}

// Amplitude by the library's sine and cosine (the 64-register large-count kernel;
// the on-chip one evaluates positions in pairs below).
template <bool NF, bool SCALE>
__device__ __forceinline__ void amplitude(double k, double s, double psi, double dist, double &re, double &im) {
    double th;
    if (!NF) th = -__dsub_rn(__dmul_rn(s, k), psi);  // time.py:94 exp(-1j*(s*k-phases))
    else th = __dadd_rn(__dmul_rn(s, k), psi);       // simtime.cu:71 phase = s*k + w
    double sn, cs;
    sincos(th, &sn, &cs);
    if (SCALE) {
        cs = __ddiv_rn(cs, dist);
        sn = __ddiv_rn(sn, dist);
    }
    re = cs;
    im = sn;
}

// Phase of one emitter (and its distance), the argument of amplitude().
template <bool NF>
__device__ __forceinline__ void phase_of(double k, double dx, double dy, double dz, double dn, double q0, double q1,
                                         double q2, const double4 &a, double &th, double &dist) {
    double s;
    path_only<NF>(dx, dy, dz, dn, q0, q1, q2, a, s, dist);
    th = NF ? __dadd_rn(__dmul_rn(s, k), a.w) : -__dsub_rn(__dmul_rn(s, k), a.w);
}

// sincos_cw of two arguments and expm1_neg of two gaps, with one range check for
// both so that the four (two) polynomials run side by side.
__device__ __forceinline__ void sincos_pair(double x0, double x1, double &s0, double &c0, double &s1, double &c1) {
    if (!(fabs(x0) <= 0x1p30 && fabs(x1) <= 0x1p30)) {
        sincos(x0, &s0, &c0);
        sincos(x1, &s1, &c1);
        return;
    }
    sincos_near(x0, s0, c0);
    sincos_near(x1, s1, c1);
}
__device__ __forceinline__ void expm1_neg_pair(double x0, double x1, double &e0, double &e1) {
    if (!(x0 <= 0.0625 && x1 <= 0.0625)) {
        e0 = expm1_neg(x0);
        e1 = expm1_neg(x1);
        return;
    }
    e0 = expm1_near(x0);
    e1 = expm1_near(x1);
}

// Block-wide min / max of the keys; result broadcast through smem (2 doubles).
__device__ __forceinline__ void block_minmax(double &lo, double &hi, double *sm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    __syncthreads();
    if (lane == 0) {
        sm[2 * warp] = lo;
        sm[2 * warp + 1] = hi;
    }
    __syncthreads();
    lo = sm[0];
    hi = sm[1];
    for (int w = 1; w < (int)blockDim.x / 32; ++w) {
        lo = fmin(lo, sm[2 * w]);
        hi = fmax(hi, sm[2 * w + 1]);
    }
    __syncthreads();
}

// Exact sort of emitter indices by key, by buckets.  The bucket of a key is
// a non-decreasing function of the key in IEEE arithmetic, so bucket order is
// key order; each bucket is then insertion-sorted by (key, emitter index).
// The map has two levels so that buckets hold about the same number of keys
// whatever the keys' distribution (arrival times are near-Gaussian, and a
// linear map crowds the middle buckets, whose insertion sort then holds the
// whole CTA at the next barrier): u = (t - kmin) (coarse bins) / (kmax - kmin) picks
// coarse bin c = floor(u); coarse bin c owns the fine buckets [B_c, B_c+1),
// B_c = c + floor(P_c (buckets - coarse bins) / n) with P_c the keys below bin c
// (at least one bucket per coarse bin), and the key goes to fine bucket
// B_c + floor((u - c) (B_c+1 - B_c)), clamped into the bin's range.  Every step
// is monotone in t.  Returns false (perm undefined) when a bucket holds more
// than kMaxBucket keys; the caller then runs the radix sort.  16 buckets and 2
// coarse bins per thread; cnt: 8 words of packed 16-bit counters per thread.
constexpr int kMaxBucket = 128;
constexpr int kBucketsPerThread = 16;
constexpr int kCoarsePerThread = 2;

__device__ __forceinline__ int coarse_of(double u, int ncoarse) { return min(max(__double2int_rz(u), 0), ncoarse - 1); }

__device__ __forceinline__ uint32_t fine_bucket(double t, double kmin, double scale, const uint32_t *coarse,
                                                int ncoarse) {
    const double u = __dmul_rn(__dsub_rn(t, kmin), scale);
    const int c = coarse_of(u, ncoarse);
    const uint32_t b0 = coarse[c], nb = coarse[c + 1] - b0;
    const int f = __double2int_rz(__dmul_rn(__dsub_rn(u, (double)c), (double)nb));
    return b0 + (uint32_t)min(max(f, 0), (int)nb - 1);
}
__device__ __forceinline__ uint32_t cnt_get(const uint32_t *cnt, uint32_t b) {
    const uint32_t w = cnt[b >> 1];
    return (b & 1) ? (w >> 16) : (w & 0xFFFFu);
}

__device__ bool bucket_sort(const double *keytab, uint16_t *perm, uint32_t *cnt, uint32_t *coarse, int n,
                            double kmin, double kmax, double *scratch, int *s_flag) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, T = blockDim.x;
    const int nbuckets = kBucketsPerThread * T, ncoarse = kCoarsePerThread * T;
    if (!(kmax > kmin)) {
        // all keys equal (or one key): stable order is emitter order
        for (int m = tid; m < n; m += T) perm[m] = (uint16_t)m;
        __syncthreads();
        return true;
    }
    const double scale = (double)ncoarse / (kmax - kmin);
    for (int w = tid; w < nbuckets / 2; w += T) cnt[w] = 0u;
    for (int c = tid; c <= ncoarse; c += T) coarse[c] = 0u;
    if (tid == 0) *s_flag = 0;
    __syncthreads();
    for (int j = tid; j < n; j += T)
        atomicAdd(&coarse[coarse_of(__dmul_rn(__dsub_rn(keytab[j], kmin), scale), ncoarse)], 1u);
    __syncthreads();
    uint32_t *wsum = reinterpret_cast<uint32_t *>(scratch);  // 16 words
    {
        // B_c from the exclusive prefix of the coarse counts; thread t owns bins [2t, 2t+2)
        uint32_t cc[kCoarsePerThread], sum = 0;
#pragma unroll
        for (int i = 0; i < kCoarsePerThread; ++i) {
            cc[i] = coarse[tid * kCoarsePerThread + i];
            sum += cc[i];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        uint32_t pre = incl - sum;
        for (int w = 0; w < warp; ++w) pre += wsum[w];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kCoarsePerThread; ++i) {
            const int c = tid * kCoarsePerThread + i;
            coarse[c] = (uint32_t)c + (uint32_t)(((uint64_t)pre * (nbuckets - ncoarse)) / (uint64_t)n);
            pre += cc[i];
        }
        if (tid == T - 1) coarse[ncoarse] = nbuckets;
    }
    __syncthreads();
    // the fine bucket of each of the thread's keys, two 13-bit ids per word,
    // kept for the scatter
    uint32_t fb[kTimeIPT / 2];
#pragma unroll
    for (int i = 0; i < kTimeIPT; ++i) {
        const int j = tid + i * T;
        uint32_t b = 0;
        if (j < n) {
            b = fine_bucket(keytab[j], kmin, scale, coarse, ncoarse);
            atomicAdd(&cnt[b >> 1], (b & 1) ? 0x10000u : 1u);
        }
        if (i & 1) fb[i / 2] |= b << 16;
        else fb[i / 2] = b;
    }
    __syncthreads();
    // exclusive scan of the counters: thread t owns buckets [16t, 16t+16)
    uint32_t loc[kBucketsPerThread];
    uint32_t sum = 0;
#pragma unroll
    for (int i = 0; i < kBucketsPerThread; ++i) {
        loc[i] = cnt_get(cnt, tid * kBucketsPerThread + i);
        sum += loc[i];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t run = incl - sum;
    for (int w = 0; w < warp; ++w) run += wsum[w];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kBucketsPerThread; i += 2) {
        const uint32_t s0 = run, s1 = run + loc[i];
        cnt[(tid * kBucketsPerThread + i) >> 1] = s0 | (s1 << 16);
        if (loc[i] > kMaxBucket || loc[i + 1] > kMaxBucket) *s_flag = 1;
        run = s1 + loc[i + 1];
    }
    __syncthreads();
    if (*s_flag) return false;  // uniform: every thread read the same flag after the barrier
    // scatter: afterwards cnt holds the end (= next start) of every bucket
#pragma unroll
    for (int i = 0; i < kTimeIPT; ++i) {
        const int j = tid + i * T;
        if (j < n) {
            const uint32_t b = (i & 1) ? (fb[i / 2] >> 16) : (fb[i / 2] & 0xFFFFu);
            const uint32_t old = atomicAdd(&cnt[b >> 1], (b & 1) ? 0x10000u : 1u);
            perm[(b & 1) ? (old >> 16) : (old & 0xFFFFu)] = (uint16_t)j;
        }
    }

    __syncthreads();
    // insertion sort inside each bucket by (key, emitter index)
    for (int i = 0; i < kBucketsPerThread; ++i) {
        const uint32_t b = tid * kBucketsPerThread + i;
        const int start = b == 0 ? 0 : (int)cnt_get(cnt, b - 1);
        const int end = (int)cnt_get(cnt, b);
        for (int m = start + 1; m < end; ++m) {
            const uint16_t v = perm[m];
            const double kv = keytab[v];
            int q = m - 1;
            while (q >= start) {
                const uint16_t u = perm[q];
                const double ku = keytab[u];
                if (ku < kv || (ku == kv && u < v)) break;
                perm[q + 1] = u;
                --q;
            }
            perm[q + 1] = v;
        }
    }
    __syncthreads();
    return true;
}

// Stable LSD radix sort (8 passes of 8 bits) of emitter indices by the
// order-preserving 64-bit image of their keys; the fallback of bucket_sort.
// Positions from n on hold kPadKeyBits and stay at the end.
__device__ void radix_sort(double *keytab, uint16_t *perm, uint32_t *H, uint32_t *base, int n, int ipt) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int S = 32 * ipt, T = blockDim.x;
    for (int m = n + tid; m < T * ipt; m += T) keytab[m] = __longlong_as_double(kPadKeyBits);
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint16_t idx[kTimeIPT];
    for (int i = 0; i < ipt; ++i) idx[i] = (uint16_t)(warp * S + i * 32 + lane);
    __syncthreads();
    for (int pass = 0; pass < 8; ++pass) {
        const int shift = pass * 8;
        uint32_t *Hw = H + warp * 256;
        for (int k = lane; k < 256; k += 32) Hw[k] = 0;
        __syncwarp();
        for (int i = 0; i < ipt; ++i) {
            const uint32_t dg = (uint32_t)(sortable(keytab[idx[i]]) >> shift) & 255u;
            const uint32_t peers = __match_any_sync(0xffffffffu, dg);
            if ((peers & lt_mask) == 0) Hw[dg] += __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        for (int k = tid; k < 256; k += T) {
            uint32_t run = 0;
            for (int w = 0; w < T / 32; ++w) {
                const uint32_t h = H[w * 256 + k];
                H[w * 256 + k] = run;
                run += h;
            }
            base[k] = run;
        }
        __syncthreads();
        if (warp == 0) {
            uint32_t v[8], sum = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                v[k] = base[lane * 8 + k];
                sum += v[k];
            }
            uint32_t incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            uint32_t run = incl - sum;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                base[lane * 8 + k] = run;
                run += v[k];
            }
        }
        __syncthreads();
        for (int k = lane; k < 256; k += 32) Hw[k] += base[k];
        __syncwarp();
        for (int i = 0; i < ipt; ++i) {
            const uint32_t dg = (uint32_t)(sortable(keytab[idx[i]]) >> shift) & 255u;
            const uint32_t peers = __match_any_sync(0xffffffffu, dg);
            const uint32_t b0 = Hw[dg];
            const uint32_t rank = b0 + __popc(peers & lt_mask);
            __syncwarp();
            if ((peers & lt_mask) == 0) Hw[dg] = b0 + __popc(peers);
            __syncwarp();
            perm[rank] = idx[i];
        }
        __syncthreads();
        for (int i = 0; i < ipt; ++i) idx[i] = perm[warp * S + i * 32 + lane];
        __syncthreads();
    }
}

// (key, emitter index) order; false both ways for an unordered (NaN) key,
// which then never passes the boundary check and takes the full sort.
__device__ __forceinline__ bool before(double ka, int ja, double kb, int jb) {
    return ka < kb || (ka == kb && ja < jb);
}

// Insertion sort of positions [lo, hi) (hi - lo < 2 ipt) of the
// position-ordered emitter indices P by (key, emitter index), keys from the
// table by emitter.  P comes from the previous pixel's order, so the inner
// loop rarely runs; (kprev, jprev) is the entry at position m - 1
// throughout, and the next position's entry is loaded one step ahead (an
// insertion only rewrites positions up to m).
__device__ __forceinline__ void window_sort(const TimeShape &sh, const double *keytab, uint16_t *P, int lo, int hi) {
    // slots of [lo, hi): contiguous except for the two pad slots at the next
    // multiple of 2 ipt
    const int grp = (int)__umulhi((uint32_t)lo, sh.inv_group), off = 2 * grp, cut = (grp + 1) * 2 * sh.ipt;
    auto sl = [&](int m) { return m + off + (m >= cut ? 2 : 0); };
    int jprev = P[sl(lo)];
    double kprev = keytab[jprev];
    int v = lo + 1 < hi ? P[sl(lo + 1)] : 0;
    double kv = keytab[v];
    for (int m = lo + 1; m < hi; ++m) {
        const int vn = m + 1 < hi ? P[sl(m + 1)] : 0;
        const double kn = keytab[vn];
        if (before(kprev, jprev, kv, v)) {
            kprev = kv;
            jprev = v;
        } else {
            // shift the entries behind v up by one
            int q = m - 1;
            P[sl(m)] = (uint16_t)jprev;
            while (--q >= lo) {
                const int u = P[sl(q)];
                if (before(keytab[u], u, kv, v)) break;
                P[sl(q + 1)] = (uint16_t)u;
            }
            P[sl(q + 1)] = (uint16_t)v;
            // position m now holds (kprev, jprev)
        }
        v = vn;
        kv = kn;
    }
}

// One pixel's direction for the scan.
struct TimePixel {
    double k, inv_tau, dx, dy, dz, dn, q0, q1, q2;
};
// A run of positions as an affine map of the value X that enters it (decayed to
// the run's first position): x_m = D_m X + B_m, and, with w_m = expm1(-2 gap/tau)
// of the gap after m, S1 = sum w D^2, S2 = sum w D B, S3 = sum w |B|^2, so that
// sum w_m |x_m|^2 = |X|^2 S1 + 2 Re(X conj(S2)) + S3 once X is known.
struct RunSums {
    double D = 1.0, Br = 0.0, Bi = 0.0, S1 = 0.0, S2r = 0.0, S2i = 0.0, S3 = 0.0;
    // the gap after the last position, em = expm1(-gap/tau): expm1(-2 gap/tau) = em (2 + em)
    __device__ __forceinline__ void interval(double em) {
        const double w = em * (2.0 + em), wD = w * D;
        S1 = fma(wD, D, S1);
        S2r = fma(wD, Br, S2r);
        S2i = fma(wD, Bi, S2i);
        S3 = fma(w, fma(Br, Br, Bi * Bi), S3);
    }
    // decay over that gap and the next amplitude
    __device__ __forceinline__ void enter(double em, double re, double im) {
        const double dec = 1.0 + em;
        D *= dec;
        Br = fma(dec, Br, re);
        Bi = fma(dec, Bi, im);
    }
};

// Buffer of scan_run's stream: an emitter may stand this many places late.
constexpr int kStream = 4;

// Decaying scan of the positions [m0, m0 + cnt) of the position-ordered emitter
// indices P.  The gaps at the run's two ends are the caller's (the neighbouring
// threads' runs may still change).  STREAM: P holds the previous pixel's order;
// it passes through a sorted buffer of kStream entries, P is rewritten with what
// leaves the buffer, and bad is set when that is not the sorted order.
//
// Two positions at a time: their phases, sines and gap polynomials are
// independent chains, and the rows of a pair are loaded a pair ahead and reduced
// to its phases before the next ones are needed.
template <bool NF, bool SCALE, bool DIGEST, bool STREAM>
__device__ __forceinline__ RunSums scan_run(const TimePixel &px, const TimeShape &sh, const double *keytab, uint16_t *P,
                                            const double4 *__restrict__ atoms4, int n, int m0, int cnt, uint64_t &h,
                                            bool &bad) {
    RunSums r;
    h = 0;
    if (cnt <= 0) return r;
    uint32_t *Pw = reinterpret_cast<uint32_t *>(P) + slot(sh, m0) / 2;
    uint64_t pw = DIGEST ? digest_pow(m0) : 0;
    const double inf = __longlong_as_double(0x7FF0000000000000ll);
    // entry e of the run in the old order; past its end an entry that sorts behind all others
    auto entry = [&](int e, uint32_t w, double &t, int &j) {
        j = e < cnt ? (int)((e & 1) ? w >> 16 : w & 0xFFFFu) : 0x10000 + e;
        t = e < cnt ? keytab[j] : inf;
    };
    double b0, b1, b2, b3, x0, x1;  // STREAM: the buffer and the next two entries
    int i0, i1, i2, i3, y0, y1;
    uint32_t wn = 0;  // the pair of indices after those
    if (STREAM) {
        uint32_t w = Pw[0];
        entry(0, w, b0, i0);
        entry(1, w, b1, i1);
        if (cnt > 2) w = Pw[1];
        entry(2, w, b2, i2);
        entry(3, w, b3, i3);
        bad = !(before(b0, i0, b1, i1) && before(b1, i1, b2, i2) && before(b2, i2, b3, i3));
        if (cnt > 4) w = Pw[2];
        entry(4, w, x0, y0);
        entry(5, w, x1, y1);
        if (cnt > 6) wn = Pw[3];
    } else if (cnt > 2) {
        wn = Pw[1];
    }
    // the next pair in order: emitters ja, jb at times ta, tb
    int ja, jb;
    double ta, tb;
    auto insert = [&](double x, int y, double &t, int &j) {
        t = b0;
        j = i0;
        if (y > 0xFFFF || before(b3, i3, x, y)) {  // (the run's end always goes last)
            b0 = b1; i0 = i1; b1 = b2; i1 = i2; b2 = b3; i2 = i3; b3 = x; i3 = y;
        } else if (before(b2, i2, x, y)) {
            b0 = b1; i0 = i1; b1 = b2; i1 = i2; b2 = x; i2 = y;
        } else if (before(b1, i1, x, y)) {
            b0 = b1; i0 = i1; b1 = x; i1 = y;
        } else if (before(b0, i0, x, y)) {
            b0 = x; i0 = y;
        } else {  // later than the buffer allows (or a NaN key)
            t = x;
            j = y;
            bad = true;
        }
    };
    auto next_pair = [&](int i) {  // entries i, i+1 of the order
        if (STREAM) {
            if (before(b3, i3, x0, y0) && before(x0, y0, x1, y1)) {
                ta = b0; ja = i0; tb = b1; jb = i1;
                b0 = b2; i0 = i2; b1 = b3; i1 = i3; b2 = x0; i2 = y0; b3 = x1; i3 = y1;
            } else {
                insert(x0, y0, ta, ja);
                insert(x1, y1, tb, jb);
            }
            const uint32_t w = wn;
            if (i + 8 < cnt) wn = Pw[i / 2 + 4];
            entry(i + 6, w, x0, y0);
            entry(i + 7, w, x1, y1);
            if (i < cnt) Pw[i / 2] = (uint32_t)ja | ((uint32_t)jb << 16);
        } else {
            const uint32_t w = wn;
            if (i + 2 < cnt) wn = Pw[i / 2 + 1];
            entry(i, w, ta, ja);
            entry(i + 1, w, tb, jb);
        }
    };
    auto row = [&](int j) { return ld_row(atoms4 + min(j, n - 1)); };
    if (!STREAM) {
        const uint32_t w = wn;
        wn = Pw[0];
        next_pair(0);
        wn = w;
    } else {
        next_pair(0);
    }
    double t0 = ta, t1 = tb, em_in = 0.0, th0, th1, r0, r1;  // the pair's times, phases and distances
    uint32_t pj = (uint32_t)ja | ((uint32_t)jb << 16);
    phase_of<NF>(px.k, px.dx, px.dy, px.dz, px.dn, px.q0, px.q1, px.q2, row(ja), th0, r0);
    phase_of<NF>(px.k, px.dx, px.dy, px.dz, px.dn, px.q0, px.q1, px.q2, row(jb), th1, r1);
#pragma unroll 1
    for (int i = 0; i < cnt; i += 2) {
        if (DIGEST) {
            h += (uint64_t)((pj & 0xFFFFu) + 1) * pw;
            pw *= kDigestBase;
            if (i + 1 < cnt) h += (uint64_t)((pj >> 16) + 1) * pw;
            pw *= kDigestBase;
        }
        next_pair(i + 2);
        if (DIGEST) pj = (uint32_t)ja | ((uint32_t)jb << 16);
        const double4 ra = row(ja), rb = row(jb);
        double re0, im0, re1, im1, em0, em1;
        sincos_pair(th0, th1, im0, re0, im1, re1);
        if (NF && SCALE) {
            re0 = __ddiv_rn(re0, r0);
            im0 = __ddiv_rn(im0, r0);
            re1 = __ddiv_rn(re1, r1);
            im1 = __ddiv_rn(im1, r1);
        }
        expm1_neg_pair(__dsub_rn(t1, t0) * px.inv_tau, i + 2 < cnt ? __dsub_rn(ta, t1) * px.inv_tau : 0.0, em0, em1);
        if (i == 0) {
            r.Br = re0;
            r.Bi = im0;
        } else {
            r.enter(em_in, re0, im0);
        }
        if (i + 1 < cnt) {
            r.interval(em0);
            r.enter(em0, re1, im1);
            if (i + 2 < cnt) r.interval(em1);
        }
        em_in = em1;
        t0 = ta;
        t1 = tb;
        phase_of<NF>(px.k, px.dx, px.dy, px.dz, px.dn, px.q0, px.q1, px.q2, ra, th0, r0);
        phase_of<NF>(px.k, px.dx, px.dy, px.dz, px.dn, px.q0, px.q1, px.q2, rb, th1, r1);
    }
    return r;
}

template <bool NF, bool SCALE, bool DIGEST>
__global__ void __launch_bounds__(kTimeThreads, 1) time_kernel(const GeomParams g, const double *__restrict__ atoms,
                                                                const double *__restrict__ times, int n, double c,
                                                                double tau, double *__restrict__ out,
                                                                WsHeader *__restrict__ hdr, int order_pixel,
                                                                int *__restrict__ order_out,
                                                                double *__restrict__ keys_out,
                                                                uint64_t *__restrict__ digest, int chunk, const TimeShape sh) {
    extern __shared__ __align__(16) unsigned char smem[];
    double *keytab = reinterpret_cast<double *>(smem);
    const int T = blockDim.x, nwarps = T / 32, ipt = sh.ipt, cap = T * ipt;
    uint16_t *P = reinterpret_cast<uint16_t *>(smem + (size_t)cap * 8);
    uint32_t *H = reinterpret_cast<uint32_t *>(P + cap + T);
    double *scratch = reinterpret_cast<double *>(H + nwarps * 256);  // 8 doubles per warp
    uint32_t *coarse = reinterpret_cast<uint32_t *>(scratch + 8 * nwarps), *base = coarse;
    __shared__ uint64_t s_dig[kTimeWarps];
    __shared__ int s_pix, s_flag;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int npix = g.nx * g.ny;
    const double ic = 1.0 / c;  // correctly rounded (IEEE division)
    const double4 *atoms4 = reinterpret_cast<const double4 *>(atoms);
    // the scan's exponents use a multiply by 1/tau (1 ulp from the reference's
    // division, ~1e-16 relative in the decay); only the sort keys must match bit for bit
    const double inv_tau = 1.0 / tau;

    // CTA-uniform sort state: whether (K, P) hold the previous pixel's order,
    // and whether warm starts are still tried
    bool have = false;
    int fails = 0, slips = 0;
    // order_pixel >= 0: process that one pixel only, record its sorted order
    // and write its intensity to out[0]
    int iter = 0;
    for (;;) {
        __syncthreads();
        if (tid == 0)
            // (unsigned: every CTA's last claim goes past the end, up to twice npix < 2^31)
            s_pix = order_pixel >= 0 ? (iter == 0 ? 0 : npix)
                                     : (int)min(atomicAdd(&hdr->work_counter, (unsigned)chunk), (unsigned)npix);
        __syncthreads();
        ++iter;
        const int c0 = s_pix;
        if (c0 >= npix) break;
        const int c1 = order_pixel >= 0 ? c0 + 1 : c0 + min(chunk, npix - c0);
        for (int pl = c0; pl < c1; ++pl) {
            int ix, iy;
            if (order_pixel >= 0) {
                ix = order_pixel / g.ny;
                iy = order_pixel - ix * g.ny;
            } else {
                // serpentine walk: odd rows backwards
                ix = pl / g.ny;
                const int r = pl - ix * g.ny;
                iy = (ix & 1) ? g.ny - 1 - r : r;
            }
            const int p = ix * g.ny + iy;
            TimePixel px;
            px.k = g.k;
            px.inv_tau = inv_tau;
            double &dx = px.dx, &dy = px.dy, &dz = px.dz;
            pixel_time(g, ix, iy, dx, dy, dz);
            // time.py:89-91 (np.linalg.norm = sqrt((x*x + y*y) + z*z); q = det/d; q_z -= 1)
            const double dn =
                __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
            const double q0 = __ddiv_rn(dx, dn), q1 = __ddiv_rn(dy, dn), q2 = __dsub_rn(__ddiv_rn(dz, dn), 1.0);
            px.dn = dn;
            px.q0 = q0;
            px.q1 = q1;
            px.q2 = q2;

            // ---- keys: table by emitter index (coalesced) ----
            // (the rows of KB emitters per thread are loaded before any is used; only
            // the last batch checks for the end of the list)
            {
                constexpr int KB = NF ? 4 : 8;
                auto key_batch = [&](int j0, auto last) {
                    constexpr bool kLast = decltype(last)::value;
                    double4 aa[KB];
                    double tt[KB];
#pragma unroll
                    for (int u = 0; u < KB; ++u) {
                        const int j = kLast ? min(j0 + u * T, n - 1) : j0 + u * T;
                        aa[u] = ld_row(atoms4 + j);
                        tt[u] = times[j];
                    }
                    if (!NF) {
                        // far field without branches: the Markstein quotient of every
                        // row, and the IEEE division after the batch for a quotient out of
                        // div_rn's range (a zero path difference, say; the range is tested
                        // on the quotient's exponent)
                        double tq[KB];
                        uint32_t redo = 0;
#pragma unroll
                        for (int u = 0; u < KB; ++u) {
                            const double sp = __fma_rn(q2, aa[u].z, __fma_rn(q1, aa[u].y, __dmul_rn(q0, aa[u].x)));
                            const double qa = __dmul_rn(-sp, ic);
                            tq[u] = __fma_rn(__fma_rn(-c, qa, -sp), ic, qa);
                            redo = max(redo, ((uint32_t)__double2hiint(qa) & 0x7FFFFFFFu) - kDivLow);
                        }
                        if (redo >= kDivSpan) {
#pragma unroll
                            for (int u = 0; u < KB; ++u) {
                                const double sp =
                                    __fma_rn(q2, aa[u].z, __fma_rn(q1, aa[u].y, __dmul_rn(q0, aa[u].x)));
                                tq[u] = div_rn(-sp, c, ic);
                            }
                        }
#pragma unroll
                        for (int u = 0; u < KB; ++u)
                            if (!kLast || j0 + u * T < n) keytab[j0 + u * T] = __dadd_rn(tq[u], tt[u]);
                    } else {
#pragma unroll
                        for (int u = 0; u < KB; ++u) {
                            double t, s, dist;
                            arrival<NF, SCALE>(g, dx, dy, dz, dn, q0, q1, q2, aa[u], tt[u], c, ic, t, s, dist);
                            if (!kLast || j0 + u * T < n) keytab[j0 + u * T] = t;
                        }
                    }
                };
                int j = 0;
#pragma unroll 1
                for (; j + KB * T <= n; j += KB * T) key_batch(j + tid, std::false_type{});
                if (j < n) key_batch(j + tid, std::true_type{});
            }
            __syncthreads();

            // ---- warm start: the previous pixel's order, repaired while it is scanned ----
            // First the few positions around every run's start, so that no emitter has
            // to cross it later.  Then every thread streams its run through a sorted
            // buffer of four and scans what leaves it: an emitter that is less than
            // five places late in the old order comes out in its place; a thread whose
            // stream was not sorted by that sorts its run as a window and scans it again.
            // The order is exact when every run ends before the next begins; otherwise
            // the window passes below repair it and all runs are scanned again.
            const int m0 = tid * ipt, cnt = min(max(n - m0, 0), ipt);
            RunSums run;
            uint64_t h = 0;
            bool sorted = false, scan = true;
            if (have && slips < kWarmMaxFails && fails < kWarmMaxFails && ipt >= 2 * kStream) {
                if (cnt > 0) window_sort(sh, keytab, P, max(m0 - kStream, 0), min(m0 + kStream, n));
                __syncthreads();
                bool bad = false;
                run = scan_run<NF, SCALE, DIGEST, true>(px, sh, keytab, P, atoms4, n, m0, cnt, h, bad);
                if (bad) window_sort(sh, keytab, P, m0, m0 + cnt);
                const int nbad = __syncthreads_count(bad);
                bool apart = true;
                if (m0 > 0 && cnt > 0) {
                    const int u = P[slot(sh, m0 - 1)], v = P[slot(sh, m0)];
                    apart = before(keytab[u], u, keytab[v], v);
                }
                sorted = __syncthreads_and(apart);
                scan = bad || !sorted;
                slips = sorted && nbad <= T / 8 ? 0 : slips + 1;
            }
            // ---- warm start by windows ----
            if (!sorted && have && fails < kWarmMaxFails) {
                // thread t's window: [rt, rt+r) on even passes (r = ipt), [rt-r/2, rt+r/2) on odd
                // ones (the last thread's odd window runs to the end).  After a pass every
                // window is sorted, so a window of the other grid -- two sorted halves --
                // is out of order only if the boundary at its middle is: a thread sorts its
                // window in the first pass, and later only when that boundary was found out
                // of order (dirty).  The boundary a thread checks is the middle of its next
                // window; together the threads check every boundary of the pass's grid.
                bool dirty = true;
                for (int pass = 0; pass < kWarmPasses; ++pass) {
                    const int half = (pass & 1) ? ipt / 2 : 0;
                    const int lo = max(tid * ipt - half, 0);
                    const int hi = min(tid == T - 1 ? cap : (tid + 1) * ipt - half, n);
                    // (the previous pass's __syncthreads_or ordered its reads before these writes)
                    if (dirty && lo < hi) window_sort(sh, keytab, P, lo, hi);
                    __syncthreads();
                    const int b = (pass & 1) ? (tid + 1) * ipt - half : tid * ipt;
                    bool bad = false;
                    if (b >= 1 && b < n) {
                        const int u = P[slot(sh, b - 1)], v = P[slot(sh, b)];
                        bad = !before(keytab[u], u, keytab[v], v);
                    }
                    dirty = bad;
                    if (!__syncthreads_or(bad)) {
                        sorted = true;
                        break;
                    }
                    if (pass == 0) {
                        // Between neighbouring pixels the few pairs still out of order sit
                        // at even boundaries and have moved by a position or two: first a
                        // window of 2 patch positions around each such boundary.  Only
                        // the pairs at those windows' ends can then be out of order; where
                        // one is, the odd window around it (which holds the short one)
                        // takes over in the next pass.
                        const int patch = min(8, ipt / 2);
                        const int plo = max(b - patch, 0), phi = min(b + patch, n);
                        if (bad) window_sort(sh, keytab, P, plo, phi);
                        __syncthreads();
                        bool pbad = false;
                        if (bad) {
                            if (plo >= 1) {
                                const int u = P[slot(sh, plo - 1)], v = P[slot(sh, plo)];
                                pbad = !before(keytab[u], u, keytab[v], v);
                            }
                            if (phi < n) {
                                const int u = P[slot(sh, phi - 1)], v = P[slot(sh, phi)];
                                pbad = pbad || !before(keytab[u], u, keytab[v], v);
                            }
                        }
                        dirty = pbad;
                        if (!__syncthreads_or(pbad)) {
                            sorted = true;
                            break;
                        }
                    }
                }
                fails = sorted ? 0 : fails + 1;
                if (!sorted && tid == 0) atomicAdd(&hdr->work_counter3, 1u);  // warm starts given up
            }
            if (!sorted) {
                // ---- full sort ----
                if (tid == 0) atomicAdd(&hdr->work_counter2, 1u);  // full sorts
                double kmin = __longlong_as_double(0x7FF0000000000000ll), kmax = -kmin;
                for (int j = tid; j < n; j += T) {
                    kmin = fmin(kmin, keytab[j]);
                    kmax = fmax(kmax, keytab[j]);
                }
                block_minmax(kmin, kmax, scratch + 6 * nwarps);
                if (!bucket_sort(keytab, P, H, coarse, n, kmin, kmax, scratch, &s_flag))
                    radix_sort(keytab, P, H, base, n, ipt);
                // P[m] (unpadded) = emitter at sorted position m: move to slots
                uint32_t *P2 = reinterpret_cast<uint32_t *>(P);
                uint32_t pk[kTimeIPT / 2];
#pragma unroll
                for (int i = 0; i < kTimeIPT / 2; ++i) pk[i] = 2 * i < ipt ? P2[tid * (ipt / 2) + i] : 0u;
                __syncthreads();
#pragma unroll
                for (int i = 0; i < kTimeIPT / 2; ++i)
                    if (2 * i < ipt) P2[slot(sh, tid * ipt) / 2 + i] = pk[i];
                __syncthreads();
            }
            have = true;
            // P[slot(sh, m)]: emitter at sorted position m < n

            if (order_pixel >= 0) {
                for (int m = tid; m < n; m += T) {
                    order_out[m] = P[slot(sh, m)];
                    keys_out[m] = keytab[P[slot(sh, m)]];
                }
            }

            if (scan) {
                bool unused = false;
                run = scan_run<NF, SCALE, DIGEST, false>(px, sh, keytab, P, atoms4, n, m0, cnt, h, unused);
            }
            // the gaps at the run's ends (an infinite one before position 0 and after n-1)
            double em_first = -1.0, em_last = -1.0;
            if (cnt > 0) {
                if (m0 > 0)
                    em_first = expm1_neg(__dsub_rn(keytab[P[slot(sh, m0)]], keytab[P[slot(sh, m0 - 1)]]) * inv_tau);
                if (m0 + cnt < n)
                    em_last = expm1_neg(
                        __dsub_rn(keytab[P[slot(sh, m0 + cnt)]], keytab[P[slot(sh, m0 + cnt - 1)]]) * inv_tau);
                run.interval(em_last);
            }
            const double dec0 = 1.0 + em_first;
            const Affine agg = {dec0 * run.D, run.Br, run.Bi};
            // block exclusive scan of the run maps
            Affine incl = agg;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                Affine y;
                y.d = __shfl_up_sync(0xffffffffu, incl.d, o);
                y.br = __shfl_up_sync(0xffffffffu, incl.br, o);
                y.bi = __shfl_up_sync(0xffffffffu, incl.bi, o);
                if (lane >= o) incl = compose(y, incl);
            }
            if (lane == 31) {
                scratch[warp * 3 + 0] = incl.d;
                scratch[warp * 3 + 1] = incl.br;
                scratch[warp * 3 + 2] = incl.bi;
            }
            __syncthreads();
            Affine wpre = {1.0, 0.0, 0.0};  // composition of all earlier warps
            for (int w = 0; w < warp; ++w) {
                const Affine y = {scratch[w * 3 + 0], scratch[w * 3 + 1], scratch[w * 3 + 2]};
                wpre = compose(wpre, y);
            }
            Affine excl;
            excl.d = __shfl_up_sync(0xffffffffu, incl.d, 1);
            excl.br = __shfl_up_sync(0xffffffffu, incl.br, 1);
            excl.bi = __shfl_up_sync(0xffffffffu, incl.bi, 1);
            if (lane == 0) excl = Affine{1.0, 0.0, 0.0};
            excl = compose(wpre, excl);
            // X entering this thread's run = excl applied to x_{-1} = 0, decayed to its
            // first position
            const double Xr = dec0 * excl.br, Xi = dec0 * excl.bi;
            double part = (-tau / 2) *
                          fma(fma(Xr, Xr, Xi * Xi), run.S1, fma(2.0, fma(Xr, run.S2r, Xi * run.S2i), run.S3));
            // block sum (and of the order digest)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                part += __shfl_down_sync(0xffffffffu, part, o);
                if (DIGEST) h += __shfl_down_sync(0xffffffffu, h, o);
            }
            __syncthreads();
            if (lane == 0) {
                scratch[4 * nwarps + warp] = part;
                if (DIGEST) s_dig[warp] = h;
            }
            __syncthreads();
            if (tid == 0) {
                double tot = 0.0;
                uint64_t hh = 0;
                for (int w = 0; w < nwarps; ++w) {
                    tot += scratch[4 * nwarps + w];
                    if (DIGEST) hh += s_dig[w];
                }
                // far field: every amplitude has the pixel's own distance
                out[order_pixel >= 0 ? 0 : p] = !NF && SCALE ? tot / (dn * dn) : tot;
                if (DIGEST && order_pixel < 0) digest[p] = hh;
            }
            // the next pixel's key pass overwrites the key table and P, which the scan reads
            // across runs, and scratch, which thread 0 has just read
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// Large emitter counts (n > kTimeMaxN): the same algorithm with the per-pixel
// arrays in a global workspace slice per CTA -- keys (FP64, by emitter),
// two int32 permutations -- and the bucket counters (uint32, up to
// kLargeBuckets) in shared memory.  Fallback for an overfull bucket: a
// stable LSD radix sort over the whole array in tiles.
// ---------------------------------------------------------------------------
constexpr int kLargeBuckets = 16384;
constexpr int kLargeMaxBucket = 256;
constexpr size_t kLargeSmem = (size_t)kLargeBuckets * 4  // also holds the radix counters
                              + (kCoarse + 4) * 4;      // first fine bucket per coarse bin

__host__ __device__ __forceinline__ int large_buckets(int64_t n) {
    int nb = 8 * kCoarse;  // n > 20480 here: at least 8192 buckets, a multiple of the threads
    while (nb < kLargeBuckets && (int64_t)nb * 4 < n) nb <<= 1;
    return nb;
}

// A CTA's slice: keys (8 B per emitter), the sorted records (16 B) and two
// index arrays for the radix fallback (4 B each).
struct SortRec {
    double key;
    int idx;
    int pad;
};
__host__ __device__ __forceinline__ size_t large_slice_bytes(int64_t n) {
    return ((size_t)n * 32 + 255) & ~(size_t)255;
}

// The two-level map of bucket_sort with nb fine buckets (nb >= 8192 here).
__device__ __forceinline__ uint32_t fine_bucket_n(double t, double kmin, double scale, const uint32_t *coarse) {
    return fine_bucket(t, kmin, scale, coarse, kCoarse);
}

// Sorted (key, emitter) records in rec: the scatter moves each record to its
// bucket and the insertion sort works on the bucket's contiguous records, so
// no pass gathers keys through a permutation.
__device__ bool bucket_sort_large(const double *keys, SortRec *rec, uint32_t *cnt, uint32_t *coarse, int n, int nb,
                                  double kmin, double kmax, double *scratch, int *s_flag) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (!(kmax > kmin)) {
        for (int m = tid; m < n; m += kTimeThreads) rec[m] = SortRec{keys[m], m, 0};
        __syncthreads();
        return true;
    }
    const double scale = (double)kCoarse / (kmax - kmin);
    const int per = nb / kTimeThreads;
    for (int b = tid; b < nb; b += kTimeThreads) cnt[b] = 0u;
    for (int c = tid; c <= kCoarse; c += kTimeThreads) coarse[c] = 0u;
    if (tid == 0) *s_flag = 0;
    __syncthreads();
    for (int j = tid; j < n; j += kTimeThreads)
        atomicAdd(&coarse[coarse_of(__dmul_rn(__dsub_rn(keys[j], kmin), scale), kCoarse)], 1u);
    __syncthreads();
    uint32_t *wsum = reinterpret_cast<uint32_t *>(scratch);
    {
        uint32_t cc[kCoarsePerThread], csum = 0;
#pragma unroll
        for (int i = 0; i < kCoarsePerThread; ++i) {
            cc[i] = coarse[tid * kCoarsePerThread + i];
            csum += cc[i];
        }
        uint32_t cincl = csum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, cincl, o);
            if (lane >= o) cincl += y;
        }
        if (lane == 31) wsum[warp] = cincl;
        __syncthreads();
        uint32_t pre = cincl - csum;
        for (int w = 0; w < warp; ++w) pre += wsum[w];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kCoarsePerThread; ++i) {
            const int c = tid * kCoarsePerThread + i;
            coarse[c] = (uint32_t)c + (uint32_t)(((uint64_t)pre * (uint64_t)(nb - kCoarse)) / (uint64_t)n);
            pre += cc[i];
        }
        if (tid == kTimeThreads - 1) coarse[kCoarse] = (uint32_t)nb;
    }
    __syncthreads();
    for (int j = tid; j < n; j += kTimeThreads) atomicAdd(&cnt[fine_bucket_n(keys[j], kmin, scale, coarse)], 1u);
    __syncthreads();
    uint32_t sum = 0, big = 0;
    for (int i = 0; i < per; ++i) {
        const uint32_t c = cnt[tid * per + i];
        sum += c;
        big |= c > kLargeMaxBucket;
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    if (big) *s_flag = 1;
    __syncthreads();
    uint32_t run = incl - sum;
    for (int w = 0; w < warp; ++w) run += wsum[w];
    __syncthreads();
    for (int i = 0; i < per; ++i) {
        const uint32_t c = cnt[tid * per + i];
        cnt[tid * per + i] = run;
        run += c;
    }
    __syncthreads();
    if (*s_flag) return false;
    // scatter: afterwards cnt[b] is the end of bucket b
    for (int j = tid; j < n; j += kTimeThreads) {
        const double kj = keys[j];
        const uint32_t pos = atomicAdd(&cnt[fine_bucket_n(kj, kmin, scale, coarse)], 1u);
        rec[pos] = SortRec{kj, j, 0};
    }
    __syncthreads();
    for (int i = 0; i < per; ++i) {
        const int b = tid * per + i;
        const int start = b == 0 ? 0 : (int)cnt[b - 1];
        const int end = (int)cnt[b];
        for (int m = start + 1; m < end; ++m) {
            const SortRec v = rec[m];
            int q = m - 1;
            while (q >= start) {
                const SortRec u = rec[q];
                if (u.key < v.key || (u.key == v.key && u.idx < v.idx)) break;
                rec[q + 1] = u;
                --q;
            }
            rec[q + 1] = v;
        }
    }
    __syncthreads();
    return true;
}

// Stable LSD radix sort (8 passes of 8 bits) of emitter indices by the
// order-preserving image of their keys.  Items go through in tiles of
// kTimeThreads * kLargeIPT; inside a tile warp w takes the items
// [w S, (w+1) S), lane-interleaved, so ranks follow item order; digit bases
// carry over from tile to tile.  Result in a (the input order is built here).
constexpr int kLargeIPT = 16;

__device__ void radix_sort_large(const double *keys, int *a, int *b, int n, uint32_t *H, uint32_t *base) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int S = 32 * kLargeIPT, T = kTimeThreads * kLargeIPT;
    const uint32_t lt_mask = (1u << lane) - 1u;
    for (int m = tid; m < n; m += kTimeThreads) a[m] = m;
    __syncthreads();
    for (int pass = 0; pass < 8; ++pass) {
        const int shift = pass * 8;
        // global digit histogram -> exclusive bases
        for (int k = tid; k < 256; k += kTimeThreads) base[k] = 0;
        __syncthreads();
        for (int m = tid; m < n; m += kTimeThreads)
            atomicAdd(&base[(uint32_t)(sortable(keys[a[m]]) >> shift) & 255u], 1u);
        __syncthreads();
        if (warp == 0) {
            uint32_t v[8], sum = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                v[k] = base[lane * 8 + k];
                sum += v[k];
            }
            uint32_t incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            uint32_t run = incl - sum;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                base[lane * 8 + k] = run;
                run += v[k];
            }
        }
        __syncthreads();
        for (int t0 = 0; t0 < n; t0 += T) {
            uint32_t *Hw = H + warp * 256;
            for (int k = lane; k < 256; k += 32) Hw[k] = 0;
            __syncwarp();
            // per-warp digit counts of this tile
            for (int i = 0; i < kLargeIPT; ++i) {
                const int m = t0 + warp * S + i * 32 + lane;
                const uint32_t dg = m < n ? (uint32_t)(sortable(keys[a[m]]) >> shift) & 255u : 256u;
                const uint32_t peers = __match_any_sync(0xffffffffu, dg);
                if (dg < 256u && (peers & lt_mask) == 0) Hw[dg] += __popc(peers);
                __syncwarp();
            }
            __syncthreads();
            // warp offsets inside the tile, and the tile's totals added to the bases
            if (tid < 256) {
                uint32_t run = base[tid];
                for (int w = 0; w < kTimeWarps; ++w) {
                    const uint32_t h = H[w * 256 + tid];
                    H[w * 256 + tid] = run;
                    run += h;
                }
                base[tid] = run;
            }
            __syncthreads();
            for (int i = 0; i < kLargeIPT; ++i) {
                const int m = t0 + warp * S + i * 32 + lane;
                const int e = m < n ? a[m] : 0;
                const uint32_t dg = m < n ? (uint32_t)(sortable(keys[e]) >> shift) & 255u : 256u;
                const uint32_t peers = __match_any_sync(0xffffffffu, dg);
                const uint32_t b0 = dg < 256u ? Hw[dg] : 0u;
                const uint32_t rank = b0 + __popc(peers & lt_mask);
                __syncwarp();
                if (dg < 256u && (peers & lt_mask) == 0) Hw[dg] = b0 + __popc(peers);
                __syncwarp();
                if (m < n) b[rank] = e;
            }
            __syncthreads();
        }
        int *t = a;
        a = b;
        b = t;
    }
    // 8 passes: the sorted order is back in the first array
}

template <bool NF, bool SCALE, bool DIGEST>
__global__ void __launch_bounds__(kTimeThreads, 2) time_kernel_large(
    const GeomParams g, const double *__restrict__ atoms, const double *__restrict__ times, int n, double c,
    double tau, double *__restrict__ out, WsHeader *__restrict__ hdr, int order_pixel, int *__restrict__ order_out,
    double *__restrict__ keys_out, unsigned char *__restrict__ slices, int n_slices, uint64_t *__restrict__ digest) {
    if ((int)blockIdx.x >= n_slices) return;  // one workspace slice per CTA
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t *cnt = reinterpret_cast<uint32_t *>(smem);
    uint32_t *H = cnt;                       // radix fallback: per-warp counters
    uint32_t *base = cnt + kTimeWarps * 256;  // and digit bases
    uint32_t *coarse = cnt + kLargeBuckets;
    __shared__ double scratch[128];
    __shared__ uint64_t s_dig[kTimeWarps];
    __shared__ int s_pix, s_flag;
    unsigned char *slice = slices + (size_t)blockIdx.x * large_slice_bytes(n);
    double *keys = reinterpret_cast<double *>(slice);
    SortRec *rec = reinterpret_cast<SortRec *>(slice + (size_t)n * 8);
    int *perm = reinterpret_cast<int *>(slice + (size_t)n * 24);
    int *perm2 = perm + n;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int npix = g.nx * g.ny;
    const int nb = large_buckets(n);
    const int per = (n + kTimeThreads - 1) / kTimeThreads;
    int iter = 0;
    for (;;) {
        __syncthreads();
        if (tid == 0)
            s_pix = order_pixel >= 0 ? (iter == 0 ? order_pixel : npix)
                                     : (int)min(atomicAdd(&hdr->work_counter, 1u), (unsigned)npix);
        __syncthreads();
        ++iter;
        const int p = s_pix;
        if (p >= npix) break;
        const int ix = p / g.ny, iy = p - ix * g.ny;
        double dx, dy, dz;
        pixel_time(g, ix, iy, dx, dy, dz);
        const double dn = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
        const double q0 = __ddiv_rn(dx, dn), q1 = __ddiv_rn(dy, dn), q2 = __dsub_rn(__ddiv_rn(dz, dn), 1.0);
        const double inv_tau = 1.0 / tau;
        double kmin = __longlong_as_double(0x7FF0000000000000ll), kmax = -kmin;
        for (int j = tid; j < n; j += kTimeThreads) {
            const double4 a = reinterpret_cast<const double4 *>(atoms)[j];
            double t, s, dist;
            arrival<NF, SCALE, false>(g, dx, dy, dz, dn, q0, q1, q2, a, times[j], c, 0.0, t, s, dist);
            kmin = fmin(kmin, t);
            kmax = fmax(kmax, t);
            keys[j] = t;
        }
        block_minmax(kmin, kmax, scratch + 96);
        __syncthreads();
        if (!bucket_sort_large(keys, rec, cnt, coarse, n, nb, kmin, kmax, scratch, &s_flag)) {
            radix_sort_large(keys, perm, perm2, n, H, base);
            for (int m = tid; m < n; m += kTimeThreads) rec[m] = SortRec{keys[perm[m]], perm[m], 0};
            __syncthreads();
        }
        if (p == order_pixel) {
            for (int m = tid; m < n; m += kTimeThreads) {
                order_out[m] = rec[m].idx;
                keys_out[m] = rec[m].key;
            }
        }
        const int m0 = tid * per;
        double Dm = 1.0, Br = 0.0, Bi = 0.0;
        double S1 = 0.0, S2r = 0.0, S2i = 0.0, S3 = 0.0;
        // neighbours' keys carried in registers, the next emitter row loaded one step ahead
        const double4 *atoms4 = reinterpret_cast<const double4 *>(atoms);
        double t_prev = m0 > 0 && m0 - 1 < n ? rec[m0 - 1].key : 0.0;
        SortRec r_next = SortRec{0.0, 0, 0};
        double4 a_next = make_double4(0.0, 0.0, 0.0, 0.0);
        if (m0 < n) {
            r_next = rec[m0];
            a_next = atoms4[r_next.idx];
        }
        uint64_t h = 0, pw = DIGEST && m0 < n ? digest_pow(m0) : 0;
        for (int i = 0; i < per; ++i) {
            const int m = m0 + i;
            if (m >= n) break;
            const double tj = r_next.key;
            const double4 a = a_next;
            if (DIGEST) {
                h += (uint64_t)(r_next.idx + 1) * pw;
                pw *= kDigestBase;
            }
            if (m + 1 < n) {
                r_next = rec[m + 1];
                if (i + 1 < per) a_next = atoms4[r_next.idx];
            }
            double s, dist, re, im;
            path_only<NF>(dx, dy, dz, dn, q0, q1, q2, a, s, dist);
            amplitude<NF, SCALE>(g.k, s, a.w, dist, re, im);
            const double dec = m == 0 ? 0.0 : exp(-__dsub_rn(tj, t_prev) * inv_tau);
            t_prev = tj;
            Dm *= dec;
            Br = fma(dec, Br, re);
            Bi = fma(dec, Bi, im);
            const double w = m < n - 1 ? (-tau / 2) * expm1(-2 * __dsub_rn(r_next.key, tj) * inv_tau) : tau / 2;
            const double wD = w * Dm;
            S1 = fma(wD, Dm, S1);
            S2r = fma(wD, Br, S2r);
            S2i = fma(wD, Bi, S2i);
            S3 = fma(w, fma(Br, Br, Bi * Bi), S3);
        }
        Affine incl = {Dm, Br, Bi};
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            Affine y;
            y.d = __shfl_up_sync(0xffffffffu, incl.d, o);
            y.br = __shfl_up_sync(0xffffffffu, incl.br, o);
            y.bi = __shfl_up_sync(0xffffffffu, incl.bi, o);
            if (lane >= o) incl = compose(y, incl);
        }
        __syncthreads();
        if (lane == 31) {
            scratch[warp * 3 + 0] = incl.d;
            scratch[warp * 3 + 1] = incl.br;
            scratch[warp * 3 + 2] = incl.bi;
        }
        __syncthreads();
        Affine wpre = {1.0, 0.0, 0.0};
        for (int w = 0; w < warp; ++w) {
            const Affine y = {scratch[w * 3 + 0], scratch[w * 3 + 1], scratch[w * 3 + 2]};
            wpre = compose(wpre, y);
        }
        Affine excl;
        excl.d = __shfl_up_sync(0xffffffffu, incl.d, 1);
        excl.br = __shfl_up_sync(0xffffffffu, incl.br, 1);
        excl.bi = __shfl_up_sync(0xffffffffu, incl.bi, 1);
        if (lane == 0) excl = Affine{1.0, 0.0, 0.0};
        excl = compose(wpre, excl);
        const double Xr = excl.br, Xi = excl.bi;
        double part = fma(fma(Xr, Xr, Xi * Xi), S1, fma(2.0, fma(Xr, S2r, Xi * S2i), S3));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            part += __shfl_down_sync(0xffffffffu, part, o);
            if (DIGEST) h += __shfl_down_sync(0xffffffffu, h, o);
        }
        __syncthreads();
        if (lane == 0) {
            scratch[64 + warp] = part;
            if (DIGEST) s_dig[warp] = h;
        }
        __syncthreads();
        if (tid == 0) {
            double tot = 0.0;
            uint64_t hh = 0;
            for (int w = 0; w < kTimeWarps; ++w) {
                tot += scratch[64 + w];
                if (DIGEST) hh += s_dig[w];
            }
            out[order_pixel >= 0 ? 0 : p] = tot;
            if (DIGEST && order_pixel < 0) digest[p] = hh;
        }
    }
}

template <bool NF, bool SCALE>
static void *time_kernel_large_ptr(bool digest) {
    return digest ? (void *)time_kernel_large<NF, SCALE, true> : (void *)time_kernel_large<NF, SCALE, false>;
}

template <bool NF, bool SCALE>
static void *time_kernel_ptr(bool digest) {
    return digest ? (void *)time_kernel<NF, SCALE, true> : (void *)time_kernel<NF, SCALE, false>;
}

static idiwf_status time_validate(const idiwf_geom *geom, const double *atoms, const double *times, int64_t n,
                                  double c, double tau) {
    if (!geom || geom->nx <= 0 || geom->ny <= 0 || (int64_t)geom->nx * geom->ny >= ((int64_t)1 << 31))
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "bad detector size");
    if (geom->offset[0] != 0.0 || geom->offset[1] != 0.0)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "the time path has no detector offset");
    if (geom->flags & IDIWF_SECONDORDER)
        return set_error(IDIWF_ERR_UNSUPPORTED, "secondorder is not defined for the time path");
    if (n < 1) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "the time path needs at least one emitter");
    if (n > ((int64_t)1 << 28)) return set_error(IDIWF_ERR_UNSUPPORTED, "at most 2^28 emitters");
    if (!atoms || !times) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "atoms/times are NULL");
    if (reinterpret_cast<uintptr_t>(atoms) & 31) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "atoms must be 32-byte aligned");
    if (!(c > 0) || !(tau > 0)) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "c and tau must be positive");
    return IDIWF_OK;
}

static void *large_fn(const idiwf_geom *geom, bool digest = false) {
    const bool nf = geom->flags & IDIWF_NF, sc = geom->flags & IDIWF_SCALE;
    return nf ? (sc ? time_kernel_large_ptr<true, true>(digest) : time_kernel_large_ptr<true, false>(digest))
              : (sc ? time_kernel_large_ptr<false, true>(digest) : time_kernel_large_ptr<false, false>(digest));
}

// CTAs of the large-n kernel on this device, each owning one workspace
// slice.  The shared-memory attribute is set before the occupancy query, so
// the workspace size and the launch see the same count (both digest
// instances have the same resources).
static int large_ctas(const idiwf_geom *geom, int order_pixel) {
    if (order_pixel >= 0) return 1;
    void *fn = large_fn(geom);
    int dev = 0, sms = 148, occ = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLargeSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kTimeThreads, kLargeSmem) != cudaSuccess) {
        cudaGetLastError();
        occ = 1;
    }
    return std::max(1, std::min(geom->nx * geom->ny, sms * std::max(occ, 1)));
}

// Threads of a pixel's CTA: 512 / threads pixels share an SM (the kernel's 128
// registers allow 16 warps per SM at any split).  Few threads with long runs cost
// least per pixel -- the fixed costs (barriers, block scan, run ends) are shared by
// more positions and the CTAs of an SM are in different phases -- as long as the
// tables of 512 / threads pixels fit in shared memory.  But a CTA's first pixel
// pays a full sort, so every CTA gets at least two.  100 x 100 pixels, us, 512
// threads against the choice: 500 emitters 400 / 121 (32 threads), 2,000 565 / 273
// (64), 5,000 883 / 590 (128), 10,000 1251 / 1164 (256).  32 x 32 pixels, 1,000
// emitters: 79 (32), 57 (128), 63 (160, the choice), 80 (512).
static TimeShape choose_shape(int n, int npix, int sms) {
    for (const int threads : {32, 64, 128, 160, 256}) {
        const TimeShape s = time_shape(threads, n);
        const int per_sm = kTimeThreads / threads;
        if (s.ipt <= kTimeIPT && per_sm * (s.smem + kCtaShared) <= kSmShared && npix >= 2 * per_sm * sms) return s;
    }
    return time_shape(kTimeThreads, n);
}

static size_t time_ws_bytes(const idiwf_geom *geom, int64_t n, int order_pixel) {
    if (n <= kTimeMaxN) return kWsDataOffset;
    return kWsDataOffset + (size_t)large_ctas(geom, order_pixel) * large_slice_bytes(n);
}

// digest: (nx, ny) uint64 order digests of every pixel, or NULL.
static idiwf_status time_launch(const idiwf_geom *geom, const double *atoms, const double *times, int64_t n,
                                double c, double tau, double *out, void *workspace, size_t workspace_bytes,
                                int order_pixel, int *order_out, double *keys_out, uint64_t *digest,
                                cudaStream_t stream) {
    const int slices_fit = n > kTimeMaxN ? large_ctas(geom, order_pixel) : 0;
    if (!workspace || workspace_bytes < time_ws_bytes(geom, n, order_pixel))
        return set_error(IDIWF_ERR_WORKSPACE, "workspace smaller than idiwf_time_workspace_size()");
    if (reinterpret_cast<uintptr_t>(workspace) & 255)
        return set_error(IDIWF_ERR_WORKSPACE, "workspace must be 256-byte aligned");
    WsHeader *hdr = static_cast<WsHeader *>(workspace);
    const GeomParams g = make_geom(geom);
    const bool nf = geom->flags & IDIWF_NF, sc = geom->flags & IDIWF_SCALE;
    if (n > kTimeMaxN) {
        void *fl = large_fn(geom, digest != nullptr);
        IDIWF_CUDA_CHECK(cudaFuncSetAttribute(fl, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLargeSmem));
        IDIWF_CUDA_CHECK(cudaMemsetAsync(hdr, 0, 2 * sizeof(uint32_t), stream));
        // slices the workspace holds (the caller may pass more than the minimum)
        const size_t avail = (workspace_bytes - kWsDataOffset) / large_slice_bytes(n);
        int n_slices = (int)std::min<size_t>(avail, (size_t)1 << 20);
        const int grid = std::min(slices_fit, n_slices);
        n_slices = grid;
        int ni = (int)n;
        unsigned char *slices = static_cast<unsigned char *>(workspace) + kWsDataOffset;
        void *args[] = {(void *)&g, &atoms, &times, &ni, &c, &tau, &out, &hdr, &order_pixel, &order_out, &keys_out,
                        &slices, &n_slices, &digest};
        IDIWF_CUDA_CHECK(cudaLaunchKernel(fl, dim3(grid), dim3(kTimeThreads), args, kLargeSmem, stream));
        return IDIWF_OK;
    }
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int npix = geom->nx * geom->ny;
    const TimeShape sh = choose_shape((int)n, npix, sms);
    const bool dg = digest != nullptr;
    void *fn = nf ? (sc ? time_kernel_ptr<true, true>(dg) : time_kernel_ptr<true, false>(dg))
                  : (sc ? time_kernel_ptr<false, true>(dg) : time_kernel_ptr<false, false>(dg));
    IDIWF_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kTimeSmemMax));
    // queue counter, error word, and the full-sort / given-up warm-start counts
    IDIWF_CUDA_CHECK(cudaMemsetAsync(hdr, 0, 5 * sizeof(uint32_t), stream));
    const int grid = order_pixel >= 0 ? 1 : std::min(npix, sms * (kTimeThreads / sh.threads));
    // pixels per queue claim: an equal share of the detector per CTA, walked in
    // serpentine order (every pixel of a CTA but its first warm-starts from a
    // neighbour's order; the per-pixel cost hardly varies, so equal shares
    // balance)
    int chunk = (int)(((int64_t)npix + grid - 1) / grid);
    int ni = (int)n;
    void *args[] = {(void *)&g, &atoms, &times, &ni, &c, &tau, &out, &hdr, &order_pixel, &order_out, &keys_out,
                    &digest, &chunk, (void *)&sh};
    IDIWF_CUDA_CHECK(cudaLaunchKernel(fn, dim3(grid), dim3(sh.threads), args, sh.smem, stream));
    return IDIWF_OK;
}

}  // namespace idiwf

using namespace idiwf;

extern "C" int64_t idiwf_time_max_emitters(void) { return kTimeMaxN; }

extern "C" size_t idiwf_time_workspace_size(const idiwf_geom *geom, int64_t n) {
    if (!geom || geom->nx <= 0 || geom->ny <= 0) return kWsDataOffset;
    return time_ws_bytes(geom, n, -1);
}

extern "C" idiwf_status idiwf_time_forward(const idiwf_geom *geom, const double *atoms, const double *times,
                                           int64_t n, double c, double tau, double *out, void *workspace,
                                           size_t workspace_bytes, cudaStream_t stream) {
    idiwf_status st = time_validate(geom, atoms, times, n, c, tau);
    if (st != IDIWF_OK) return st;
    if (!out) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "out is NULL");
    return time_launch(geom, atoms, times, n, c, tau, out, workspace, workspace_bytes, -1, nullptr, nullptr, nullptr,
                       stream);
}

extern "C" idiwf_status idiwf_time_forward_digest(const idiwf_geom *geom, const double *atoms, const double *times,
                                                  int64_t n, double c, double tau, double *out, uint64_t *digest,
                                                  void *workspace, size_t workspace_bytes, cudaStream_t stream) {
    idiwf_status st = time_validate(geom, atoms, times, n, c, tau);
    if (st != IDIWF_OK) return st;
    if (!out || !digest) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "out/digest is NULL");
    return time_launch(geom, atoms, times, n, c, tau, out, workspace, workspace_bytes, -1, nullptr, nullptr, digest,
                       stream);
}

extern "C" idiwf_status idiwf_time_order(const idiwf_geom *geom, const double *atoms, const double *times,
                                         int64_t n, double c, int32_t ix, int32_t iy, int32_t *order,
                                         double *sorted_keys, void *workspace, size_t workspace_bytes,
                                         cudaStream_t stream) {
    idiwf_status st = time_validate(geom, atoms, times, n, c, 1.0);
    if (st != IDIWF_OK) return st;
    if (!order || !sorted_keys) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "order/sorted_keys are NULL");
    if (ix < 0 || iy < 0 || ix >= geom->nx || iy >= geom->ny)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "pixel outside the detector");
    // the intensity of the pixel goes to a scratch slot of the workspace header
    double *scratch = reinterpret_cast<double *>(&static_cast<WsHeader *>(workspace)->pad[0]);
    return time_launch(geom, atoms, times, n, c, 1.0, scratch, workspace, workspace_bytes, ix * geom->ny + iy, order,
                       sorted_keys, nullptr, stream);
}
