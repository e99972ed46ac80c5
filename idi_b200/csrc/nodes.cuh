// Band-limited evaluation of the direct sum: nodes and interpolation.
//
// The field over the detector, with the pixel constant left out, is a sum of
// exp(i phi_j(u, v)) whose phases change along a pixel axis u by at most
//   |d phi / du| <= k |e_u - d_hat (d_hat . e_u)| |r| / |d|   per unit length,
// so an object of a few nanometres is sampled far more finely by its pixels
// than its field needs.  Where that pays, the sum is formed at the n0 x n1
// points of a tensor Chebyshev grid (first kind) laid over the whole
// detector, and the pixels follow by polynomial interpolation, two real
// contractions in FP64: E = L_x V L_y^T.  Measured on a B200, whole calls: two
// images of 50,000 emitters on 1024^2 pixels (64^2 nodes) 0.69 ms against 57.9 ms by
// the direct kernels; eight of 2,000 on 256^2 0.26 against 0.80 ms; field error
// against FP64 9e-8 against 2.1e-7.  The adjoint runs the transpose: the
// pixel weights are contracted onto the nodes, and the adjoint sum runs over
// nodes in place of pixels.
//
// Nodes per axis.  For phi linear in u, exp(i Phi t) on t in [-1, 1] has
// Chebyshev coefficients 2 J_m(Phi): beyond m = Phi they fall
// super-exponentially, over a transition of width Phi^(1/3).  The interpolant
// through n points is off by at most twice the tail of the coefficients
// (aliasing); n = Phi + 2.7 + 6.33 Phi^(1/3) keeps the tail below 1e-8 for
// Phi up to 1000.  The curvature of the detector's directions (d_hat is no linear
// function of u) adds 1 + 14 t, t = half the detector's extent over its plane's
// distance, used up to kNodeMaxT.  tests/test_nodes_math.py holds the rule to
// 1e-8 over random geometries, emitters at the largest distance from the
// origin (an image's other emitters, and the pixels inside, are far below).
//
// The FP64 kernel's images take a finer grid, 5 + 9.6 Phi^(1/3) + 30 t, which holds the
// interpolation to about 2e-15 per emitter, below the rounding of the phases (k r 1e-16).
#pragma once

#include "idiwf_internal.cuh"

namespace idiwf {

constexpr int kPathNodes = 4;        // split_path() continued: nodes and interpolation
constexpr int kNodeMax = 1024;       // nodes per axis
constexpr double kNodeMaxT = 0.6;
constexpr int kNodeThreads = 128;    // node kernel: threads per CTA, nodes per thread, emitters per stage
constexpr int kNodePPT = 4;
constexpr int kNodeTile = kNodeThreads * kNodePPT;
constexpr int kNodeTE = 128;
constexpr int kNodePPT64 = 2;        // FP64: nodes per thread
constexpr int kNodeTile64 = kNodeThreads * kNodePPT64;
constexpr int kNodeBlock = 64;       // emitters per work item and tile
// Largest near-field or second-order phase (radians) that the node kernel's sine
// and cosine polynomials take on top of the half turn (they hold to 1.04 half turns).
constexpr double kNodeMaxExtra = 0.06;

// Node geometry of a detector (host side, make_node_geom): Phi per unit of
// emitter extent, curvature ratios, and the largest |d_hat . e| along each axis.
struct NodeGeom {
    double e[2][3];  // unit vectors of the detector axes
    double phi[2], t[2], s[2];
    double inv_d;
    int32_t ok;
};

struct NodeImage {
    int64_t w0;         // work (tiles x blocks of kNodeBlock emitters) of the images before it
    int32_t path;       // split path of the image
    int32_t n0, n1;     // nodes along x and y
    int32_t ntiles, nblk;
    float scale;        // power of two: the node sums are kept as fixed point, value x scale
};
struct NodePlan {
    int64_t total;      // work of all images
    int64_t pad;
    NodeImage img[kMaxImagesPerLaunch];
};

// Node sums of an image (16 bytes each), and the node limits along each axis that
// the weight and intermediate arrays hold.
__host__ __device__ inline int64_t node_entries(int64_t npix) { return npix / 4 + 4096; }
__host__ __device__ inline int node_cap(int n) { return (n / 2 + 64 < kNodeMax ? n / 2 + 64 : kNodeMax) / 2 * 2; }

NodeGeom make_node_geom(const GeomParams &g);

#if defined(__CUDACC__)

// Nodes along one axis (even, for the 16-byte copies of weight rows) for a phase
// half-range phi; fine: the FP64 kernel's.
__device__ __forceinline__ int node_count(double phi, double t, bool fine) {
    const double n = fine ? phi + 5.0 + 9.6 * cbrt(phi) + 30.0 * t : phi + 3.7 + 6.33 * cbrt(phi) + 14.0 * t;
    return n < (double)(2 * kNodeMax) ? ((int)ceil(n) + 1) / 2 * 2 : 2 * kNodeMax;
}

// Nodes of an image from its largest |r|^2 and largest |r . e| along the two
// detector axes (float bits, rounded up); false when no grid within the limits
// exists.  Along e the phase changes by at most k/|d| (|r . e| + |d_hat . e| |r|),
// and by no more than k/|d| |r|; the near-field and second-order terms add up
// to 2 |r|/|d| of that.
__device__ __forceinline__ bool node_grid(const GeomParams &g, const NodeGeom &ng, uint32_t r2bits, uint32_t xbits,
                                          uint32_t ybits, bool fine, int &n0, int &n1) {
    const double r = sqrt((double)__uint_as_float(r2bits));
    if (!ng.ok || !(r * ng.inv_d <= 0.25)) return false;  // (a NaN fails too)
    if (!fine && (g.flags & (IDIWF_NF | IDIWF_SECONDORDER)) && !(0.5 * g.k * r * r * ng.inv_d <= kNodeMaxExtra)) return false;
    const double f = 1.0 + 2.0 * r * ng.inv_d;
    const double ex = fmin(r, (double)__uint_as_float(xbits) + ng.s[0] * r);
    const double ey = fmin(r, (double)__uint_as_float(ybits) + ng.s[1] * r);
    n0 = node_count(ng.phi[0] * ex * f, ng.t[0], fine);
    n1 = node_count(ng.phi[1] * ey * f, ng.t[1], fine);
    return n0 <= kNodeMax && n1 <= kNodeMax;
}

// Node m of n on [-1, 1], its barycentric weight, and the (fractional) pixel
// index it sits at on an axis of N pixels.
__device__ __forceinline__ double node_x(int n, int m) { return cospi((2 * m + 1) / (2.0 * n)); }
__device__ __forceinline__ double node_w(int n, int m) {
    const double s = sinpi((2 * m + 1) / (2.0 * n));
    return (m & 1) ? -s : s;
}
__device__ __forceinline__ double node_index(int n, int m, int N) { return 0.5 * (N - 1) * (1.0 + node_x(n, m)); }

// Interpolation weights of one axis, row i: L[i][m], m < n, by the barycentric
// formula (Berrut and Trefethen, SIAM Review 46(3), 2004), one warp per row.
__device__ __forceinline__ void node_weights_row(double *__restrict__ L, int n, int N, int i, int lane) {
    const double x = N > 1 ? (2 * i - (N - 1)) / (double)(N - 1) : 0.0;
    double sum = 0.0;
    for (int m = lane; m < n; m += 32) {
        double d = x - node_x(n, m);
        if (fabs(d) < 1e-30) d = 1e-30;  // a pixel on a node: its weight takes the whole sum
        const double c = node_w(n, m) / d;
        L[(size_t)i * n + m] = c;
        sum += c;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const double inv = 1.0 / sum;
    for (int m = lane; m < n; m += 32) L[(size_t)i * n + m] *= inv;
}

// Fewest pairs of an image for which nodes are considered: below it the three
// further kernels cost more than the direct sum (split precision, FP64).
constexpr double kNodeMinPairs = 8e6, kNodeMinPairs64 = 2e6;

// Whether an image of n emitters goes through its n0 x n1 grid: the grid fits
// the buffers, and the pairs saved outweigh the interpolation.  The rates are
// the kernels' measured ones: direct pairs and node pairs per second, FP64
// multiply-adds per second of the interpolation.  The choice depends on
// the image and the geometry alone, as split_path's does.
__device__ __forceinline__ bool nodes_pay(int n, int nx, int ny, int n0, int n1, double direct_rate, double node_rate,
                                          double min_pairs = kNodeMinPairs) {
    const double npix = (double)nx * ny, m = (double)n0 * n1, pairs = (double)n * npix;
    if (n0 > node_cap(nx) || n1 > node_cap(ny) || m > 0.25 * npix + 4096.0 || pairs < min_pairs) return false;
    const double mads = 2.0 * n0 * (npix + (double)n1 * ny);
    return n * m / node_rate + (mads + 100.0 * npix) * (1.0 / 1.2e13) < pairs / direct_rate;
}

// Largest extents of an emitter for the plan: |r|^2, |r . e| along both detector axes, |a|
// (float bits, rounded up), raised per warp into ext (kMaxImagesPerLaunch of each).
struct NodeExtents {
    uint32_t r2 = 0, e0 = 0, e1 = 0, a = 0;
    __device__ __forceinline__ void add(const NodeGeom &ng, const double4 &p, float amp) {
        r2 = max(r2, __float_as_uint(__double2float_ru((p.x * p.x + p.y * p.y) + p.z * p.z)));
        e0 = max(e0, __float_as_uint(__double2float_ru(fabs(p.x * ng.e[0][0] + p.y * ng.e[0][1] + p.z * ng.e[0][2]))));
        e1 = max(e1, __float_as_uint(__double2float_ru(fabs(p.x * ng.e[1][0] + p.y * ng.e[1][1] + p.z * ng.e[1][2]))));
        a = max(a, __float_as_uint(fabsf(amp)));
    }
    __device__ __forceinline__ void raise(uint32_t *ext, int b) const {
        const uint32_t v[4] = {r2, e0, e1, a};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t m = __reduce_max_sync(0xffffffffu, v[k]);
            if ((threadIdx.x & 31) == 0 && m) atomicMax(ext + k * kMaxImagesPerLaunch + b, m);
        }
    }
};
// True in every thread of the grid's last block to get here (a ticket in the header);
// what the other blocks raised is then visible.
__device__ __forceinline__ bool last_block(WsHeader *hdr) {
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&hdr->ticket, 1u) == gridDim.x * gridDim.y - 1;
    __syncthreads();
    return s_last != 0;
}

// Plan of one launch, by one block: every image's path, grid, fixed-point scale and
// share of the work.  fine: the FP64 kernel's images (their direct path counts as
// kPathPixel).  ext: per image max |r|^2, then max |r . e| along the two axes,
// then max |a| (float bits), kMaxImagesPerLaunch each.
__device__ inline void plan_nodes(const BatchParams &bp, const GeomParams &g, const NodeGeom &ng,
                                  const uint32_t *ext, bool fine, WsHeader *hdr, NodePlan *plan) {
    __shared__ long long s_work[kMaxImagesPerLaunch];
    __threadfence();
    const int npix = g.nx * g.ny;
    unsigned long long pairs = 0;
    for (int i = threadIdx.x; i < bp.n_images; i += blockDim.x) {
        const uint32_t r2 = __ldcg(ext + i), amax = __ldcg(ext + 3 * kMaxImagesPerLaunch + i);
        const int n = bp.img[i].n;
        NodeImage ni;
        ni.path = fine ? kPathPixel : split_path(g, r2, bp.groups != 0, false);
        ni.w0 = 0;
        ni.n0 = ni.n1 = ni.ntiles = ni.nblk = 0;
        ni.scale = 1.0f;
        unsigned long long pr = (unsigned long long)n * npix;
        if (bp.nodes && (ni.path == kPathRuns || ni.path == kPathPixel) &&
            // (amplitudes whose fixed-point unit would leave FP32's exponents, infinite or NaN
            // ones take the direct kernels)
            (amax == 0u || (amax >= __float_as_uint(0x1p-40f) && amax <= __float_as_uint(0x1p100f))) &&
            node_grid(g, ng, r2, __ldcg(ext + kMaxImagesPerLaunch + i), __ldcg(ext + 2 * kMaxImagesPerLaunch + i),
                      fine, ni.n0, ni.n1) &&
            (fine ? nodes_pay(n, g.nx, g.ny, ni.n0, ni.n1, 1.6e11, 1.3e11, kNodeMinPairs64)
                  : nodes_pay(n, g.nx, g.ny, ni.n0, ni.n1, ni.path == kPathRuns ? 1.8e12 : 1.5e12, 1.0e12))) {
            ni.path = kPathNodes;
            const int m = ni.n0 * ni.n1;
            const int tile = fine ? kNodeTile64 : kNodeTile;
            ni.ntiles = (m + tile - 1) / tile;
            ni.nblk = (n + kNodeBlock - 1) / kNodeBlock;
            pr = (unsigned long long)n * m;
            // |sum| <= n max |a| [times the largest 1/|d - r| <= 4/(3 D)] < 2^e
            double bound = (double)n * (double)__uint_as_float(amax);
            if ((g.flags & IDIWF_NF) && (g.flags & IDIWF_SCALE)) bound *= 1.4 * ng.inv_d;
            if (bound > 0.0) ni.scale = (float)scalbn(1.0, min(max(60 - (ilogb(bound) + 1), -120), 120));
        }
        pairs += pr;
        s_work[i] = (long long)ni.ntiles * ni.nblk;
        plan->img[i] = ni;
    }
    atomicAdd(&hdr->pairs, pairs);
    __syncthreads();
    if (threadIdx.x == 0) {
        long long w = 0;
        for (int i = 0; i < bp.n_images; ++i) {
            plan->img[i].w0 = w;
            w += s_work[i];
        }
        plan->total = w;
    }
}

// Sine and cosine of pi x, |x| <= 0.52: least-maximum polynomials in x^2, fitted for
// this range (residuals 5.6e-9 and 4e-10; 2.8e-8 rms in FP32), two values at a time.
// On the FMA pipe they cost 5.5 instructions a pair, about what the MUFU pair and
// its argument scaling hold the issue port for, at a fifth of the MUFU's error.
__device__ __forceinline__ void sincospi2(float2 x, float2 &sn, float2 &cs) {
    const float2 z = __fmul2_rn(x, x);
    float2 p = __ffma2_rn(make_float2(0.07687149941921234f, 0.07687149941921234f), z, make_float2(-0.5978690981864929f, -0.5978690981864929f));
    float2 q = __ffma2_rn(make_float2(-0.024310700595378876f, -0.024310700595378876f), z, make_float2(0.23489117622375488f, 0.23489117622375488f));
    p = __ffma2_rn(p, z, make_float2(2.5500025749206543f, 2.5500025749206543f));
    q = __ffma2_rn(q, z, make_float2(-1.3352038860321045f, -1.3352038860321045f));
    p = __ffma2_rn(p, z, make_float2(-5.167705059051514f, -5.167705059051514f));
    q = __ffma2_rn(q, z, make_float2(4.058708667755127f, 4.058708667755127f));
    p = __ffma2_rn(p, z, make_float2(3.141592502593994f, 3.141592502593994f));
    q = __ffma2_rn(q, z, make_float2(-4.934802055358887f, -4.934802055358887f));
    sn = __fmul2_rn(p, x);
    cs = __ffma2_rn(q, z, make_float2(1.0f, 1.0f));
}

// Half-turn angles of a pair of phases from the low words of their FP64 turns (the
// magic binade, +1/4 + 2^-25 turn): bit 31 is the half turn's sign, x = u - 1.5 in half
// turns comes from bits 30..8, plus the 8 bits below (the last 2^-24 takes back the
// half-step rounding offset).
__device__ __forceinline__ float2 half_turns2(uint32_t w0, uint32_t w1) {
    constexpr float kLow = 0x1p-8f - 0x1p-24f;
    const float2 u = make_float2(__uint_as_float(((w0 >> 8) & 0x007FFFFFu) | 0x3F800000u),
                                 __uint_as_float(((w1 >> 8) & 0x007FFFFFu) | 0x3F800000u));
    const float2 v = make_float2(__uint_as_float((w0 & 0xFFu) | 0x3F800000u), __uint_as_float((w1 & 0xFFu) | 0x3F800000u));
    return __ffma2_rn(v, make_float2(kLow, kLow), __fadd2_rn(u, make_float2(-1.50390625f, -1.50390625f)));
}
__device__ __forceinline__ float flip_sign(float x, uint32_t w) {
    return __uint_as_float(__float_as_uint(x) ^ (w & 0x80000000u));
}

// ---------------------------------------------------------------------------
// interpolation: Y[i][j] = sum_k L[i][k] X[j][k], L real (M x K), X complex
// (N x K), both FP64 with k contiguous
// ---------------------------------------------------------------------------
// FP64 tensor-core tiles (mma.m8n8k4): a complex column is two real columns of
// the product, so a thread's accumulator pair is one complex value.  CTA tile
// 64 x 32 complex, 4 warps of 32 x 16, K in blocks of 16 through a
// double-buffered cp.async pipeline; shared rows of 20 elements put the
// fragment loads of a half warp in distinct banks.
constexpr int kGemmM = 64, kGemmN = 32, kGemmK = 16, kGemmThreads = 128;
constexpr int kGemmLd = kGemmK + 4;

__device__ __forceinline__ void cp_async16(void *s, const void *g, bool valid) {
    const int n = valid ? 16 : 0;  // 0: the 16 bytes are filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(s)), "l"(g), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void dmma884(double &c0, double &c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

union GemmSmem {
    struct {
        double a[2][kGemmM * kGemmLd];
        double2 b[2][kGemmN * kGemmLd];
    };
    double2 y[kGemmM * (kGemmN + 1)];  // the finished tile, for stores along rows
};

// One tile at (i0, j0); `store(i, j, re, im)` receives every element inside M x N.
template <class Store>
__device__ __forceinline__ void interp_tile(GemmSmem &sm, const double *__restrict__ L, const double2 *__restrict__ X,
                                            int M, int N, int K, int i0, int j0, const Store &store) {
    const int tid = threadIdx.x, lane = tid & 31, wr = (tid >> 5) >> 1, wc = (tid >> 5) & 1;
    double acc[4][4][2];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
    const int nk = (K + kGemmK - 1) / kGemmK;
    auto issue = [&](int kb) {
        const int s = kb & 1, k0 = kb * kGemmK;
#pragma unroll
        for (int q = 0; q < kGemmM * kGemmK / 2 / kGemmThreads; ++q) {  // 2 doubles per copy (K is even)
            const int c = tid + q * kGemmThreads, r = c / (kGemmK / 2), k = (c % (kGemmK / 2)) * 2;
            const bool ok = i0 + r < M && k0 + k < K;
            cp_async16(&sm.a[s][r * kGemmLd + k], L + (ok ? (size_t)(i0 + r) * K + k0 + k : 0), ok);
        }
#pragma unroll
        for (int q = 0; q < kGemmN * kGemmK / kGemmThreads; ++q) {
            const int c = tid + q * kGemmThreads, r = c / kGemmK, k = c % kGemmK;
            const bool ok = j0 + r < N && k0 + k < K;
            cp_async16(&sm.b[s][r * kGemmLd + k], X + (ok ? (size_t)(j0 + r) * K + k0 + k : 0), ok);
        }
        cp_async_commit();
    };
    issue(0);
    for (int kb = 0; kb < nk; ++kb) {
        if (kb + 1 < nk) {
            issue(kb + 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const double *sa = sm.a[kb & 1] + (wr * 32 + (lane >> 2)) * kGemmLd + (lane & 3);
        const double *sb = reinterpret_cast<const double *>(sm.b[kb & 1] + (wc * 16 + (lane >> 3)) * kGemmLd +
                                                            (lane & 3)) + ((lane >> 2) & 1);
#pragma unroll
        for (int k = 0; k < kGemmK; k += 4) {
            double fa[4], fb[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) fa[t] = sa[t * 8 * kGemmLd + k];
#pragma unroll
            for (int t = 0; t < 4; ++t) fb[t] = sb[(t * 4 * kGemmLd + k) * 2];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) dmma884(acc[a][b][0], acc[a][b][1], fa[a], fb[b]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
            sm.y[(wr * 32 + a * 8 + (lane >> 2)) * (kGemmN + 1) + wc * 16 + b * 4 + (lane & 3)] =
                make_double2(acc[a][b][0], acc[a][b][1]);
    __syncthreads();
#pragma unroll 1
    for (int r = tid >> 5; r < kGemmM; r += kGemmThreads / 32)
        if (i0 + r < M && j0 + lane < N) {
            const double2 v = sm.y[r * (kGemmN + 1) + lane];
            store(i0 + r, j0 + lane, v.x, v.y);
        }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// the transpose: Y[m][n] = sum_k A[k][m] X[k][n], A real (K x M), X complex (K x N),
// both FP64 with m and n contiguous
// ---------------------------------------------------------------------------
// The contraction runs over pixels and the result is small (nodes x pixel columns, then
// nodes x nodes), so tiles are small too, 32 x 16 complex, and the four warps of a CTA
// share each K block of 16 (one k step each); their sums are added in warp order.
constexpr int kGemmTM = 32, kGemmTN = 16;
constexpr int kGemmTLd = 36;
union GemmTSmem {
    struct {
        double a[2][kGemmK * kGemmTLd];
        double b[2][kGemmK * kGemmTLd];
    };
    double2 y[4][kGemmTM * (kGemmTN + 1)];
};

template <class Store>
__device__ __forceinline__ void contract_tile(GemmTSmem &sm, const double *__restrict__ A, const double2 *__restrict__ X,
                                              int M, int N, int K, int i0, int j0, const Store &store) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double acc[4][4][2];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
    const int nk = (K + kGemmK - 1) / kGemmK;
    auto issue = [&](int kb) {
        const int s = kb & 1, k0 = kb * kGemmK;
#pragma unroll
        for (int q = 0; q < 2; ++q) {  // 16 rows x 32 doubles; M is even
            const int c = tid + q * kGemmThreads, k = c >> 4, m = (c & 15) * 2;
            const bool ok = k0 + k < K && i0 + m < M;
            cp_async16(&sm.a[s][k * kGemmTLd + m], A + (ok ? (size_t)(k0 + k) * M + i0 + m : 0), ok);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {  // 16 rows x 16 complex
            const int c = tid + q * kGemmThreads, k = c >> 4, n = c & 15;
            const bool ok = k0 + k < K && j0 + n < N;
            cp_async16(&sm.b[s][k * kGemmTLd + 2 * n], X + (ok ? (size_t)(k0 + k) * N + j0 + n : 0), ok);
        }
        cp_async_commit();
    };
    issue(0);
    for (int kb = 0; kb < nk; ++kb) {
        if (kb + 1 < nk) {
            issue(kb + 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const double *sa = sm.a[kb & 1] + (warp * 4 + (lane & 3)) * kGemmTLd + (lane >> 2);
        const double *sb = sm.b[kb & 1] + (warp * 4 + (lane & 3)) * kGemmTLd + (lane >> 2);
        double fa[4], fb[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) fa[t] = sa[t * 8];
#pragma unroll
        for (int t = 0; t < 4; ++t) fb[t] = sb[t * 8];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) dmma884(acc[a][b][0], acc[a][b][1], fa[a], fb[b]);
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
            sm.y[warp][(a * 8 + (lane >> 2)) * (kGemmTN + 1) + b * 4 + (lane & 3)] =
                make_double2(acc[a][b][0], acc[a][b][1]);
    __syncthreads();
    for (int c = tid; c < kGemmTM * kGemmTN; c += kGemmThreads) {
        const int m = c % kGemmTM, n = c / kGemmTM, at = m * (kGemmTN + 1) + n;
        double2 v = sm.y[0][at];
#pragma unroll
        for (int w = 1; w < 4; ++w) {
            v.x += sm.y[w][at].x;
            v.y += sm.y[w][at].y;
        }
        if (i0 + m < M && j0 + n < N) store(i0 + m, j0 + n, v.x, v.y);
    }
    __syncthreads();
}

#endif  // __CUDACC__

}  // namespace idiwf
