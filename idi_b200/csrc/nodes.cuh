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
// images of 50,000 emitters on 1024^2 pixels (66^2 nodes) 0.69 ms against 57.9 ms by
// the direct kernels, 0.35 ms with the emitters cut into cells (below); eight of 2,000 on
// 256^2 0.22 against 0.80 ms; field error against FP64 9e-8 against 2.1e-7.  The adjoint
// runs the transpose: the pixel weights are contracted onto the nodes, and the adjoint
// sum runs over nodes in place of pixels.
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
// A needle along the beam changes its phase as k r t^2 / 4 T_2(x) over the detector, with
// coefficients J_m of that at twice the order: 2 (a + 5 + 9.6 a^(1/3)) nodes at least, a its size.
//
// An object of next to no phase (Phi below 0.1) still has the near field's amplitude
// 1/|d - r|, whose Chebyshev coefficients fall by rho = e^asinh((1 - r/D) / t) a node, the
// singularity being D - r off the detector: no fewer than 20 / ln rho nodes (1e-8 of its
// variation) or, for FP64, 1 + 35 / ln rho.  FP64 images reach to r = D / 4 (kNodeMaxReach);
// split-precision ones of that amplitude stay far below it (kNfScaleRho2).
#pragma once

#include "idiwf_internal.cuh"

namespace idiwf {

constexpr int kPathNodes = 4;        // split_path() continued: nodes and interpolation
constexpr int kNodeMax = 1024;       // nodes per axis
constexpr double kNodeMaxT = 0.6;
constexpr double kNodeMaxReach = 0.25;  // largest |r| / D
constexpr int kNodeThreads = 128;    // node kernel: threads per CTA, nodes per thread, emitters per stage
constexpr int kNodePPT = 2;
constexpr int kNodeTile = kNodeThreads * kNodePPT;
constexpr int kNodeTE = 128;
constexpr int kNodePPT64 = 2;        // FP64: nodes per thread
constexpr int kNodeTile64 = kNodeThreads * kNodePPT64;
constexpr int kNodeBlock = 64;       // emitters per work item and tile
// Largest near-field or second-order phase (radians) that the node kernel's sine
// and cosine polynomials take on top of the half turn (they hold to 1.04 half turns).
constexpr double kNodeMaxExtra = 0.06;

// Cells: a large or dense object is cut into boxes along the detector axes and the beam.
// A box's field, with the phase of its centre taken out, has the box's band limit, so its
// emitters are summed on a grid of far fewer nodes; the boxes' fields are then
// interpolated to the target grid (the image's nodes, or the pixels themselves) and added
// up with the phases of their centres.  The plan weighs the cells' sums, which shrink
// with the cell, against the interpolation, which grows with their number.  Measured, with
// cells against without (whole calls): 24 images of 1,000 to 100,000 emitters on 512^2
// pixels 3.3 to 3.9 ms by card against 11.7; 300,000 emitters in a micrometre on 128^2
// pixels, which undersample it, 1.16 against 3.30 ms (direct).
constexpr int kCellMax = 512;        // cells per image
constexpr int kCellNodes = 64;       // nodes per axis of a cell's grid
constexpr int kCellMinEmitters = 4096;  // images below this are not cut
constexpr int kCellSort = 1024;      // emitters per block of the sort
constexpr int64_t kCellPixels = 1 << 18;  // most pixels that cells are interpolated to directly

// Node geometry of a detector (host side, make_node_geom): Phi per unit of
// emitter extent, curvature ratios, and the largest |d_hat . e| along each axis.
struct NodeGeom {
    double e[3][3];  // unit vectors of the detector axes and their normal
    double phi[2], t[2], s[2];
    double least[2][2];  // fewest nodes of an axis (split precision, FP64)
    double inv_d;
    double min_pairs;  // fewest pairs of an image that may take nodes
    int32_t ok, ortho;  // ortho: the axes are orthonormal (cells need it)
};

struct NodeImage {
    int32_t path;       // split path of the image
    int32_t n0, n1;     // target grid: nodes along x and y, or (pix) the pixels
    int32_t pix;
    int32_t ntiles, nblk;  // node tiles of a sum (of each cell), blocks of emitters (in all)
    float scale;        // power of two: the node sums are kept as fixed point, value x scale
    int32_t ncell;      // 1: the sum goes straight to the target grid
    int32_t c[3];       // cells along the detector axes and the normal
    int32_t g0, g1;     // nodes of a cell's grid
    uint32_t ticket;    // finished blocks of the sort's count kernel
    double lo[3], size[3], inv[3];  // cells: origin, edges, 1/edges
};
struct NodePlan {
    NodeImage img[kMaxImagesPerLaunch];
};
// Second words of the FP64 kernel's node sums: units of the first word's unit.  A block of
// emitters adds at most half a unit of the first, 2^37 of the second, and an image has at
// most 2^24 blocks.
constexpr double kLowUnit = 0x1p-38;
// What the buffers of an image hold: sums on the target grid, sums of the cells, and the
// cells' sums interpolated along one axis (FP64: f holds the second words of v).
struct NodeCaps {
    int64_t v, f, y;
};

// Node limits along each axis that the weight and intermediate arrays hold, and node sums of
// an image (16 bytes each).
__host__ __device__ inline int node_cap(int n) { return (n / 2 + 64 < kNodeMax ? n / 2 + 64 : kNodeMax) / 2 * 2; }
__host__ __device__ inline int64_t node_entries(int nx, int ny) {
    const int64_t part = (int64_t)nx * ny / 4 + 4096, most = (int64_t)node_cap(nx) * node_cap(ny);
    return part < most ? part : most;
}
// Node buffers of a group of images, and of one image: no more than 512 MB, or than the
// detector's smallest output (4 bytes a pixel); a detector whose images need more (a strip of
// very many columns, say) keeps the direct kernels.
constexpr size_t kNodeGroupBytes = (size_t)512 << 20;
inline bool node_buffers_fit(int nx, int ny, size_t image_bytes) {
    const size_t out = (size_t)nx * ny * 4;
    return image_bytes <= (out > kNodeGroupBytes ? out : kNodeGroupBytes);
}

// Limits of an image's cut, from its own emitter count (not from the others of its batch):
// sums of its cells, and their values interpolated along y (16384 a cell on average: 128
// columns of 128 nodes).
constexpr int64_t kCellSums = 1 << 19, kCellValues = 3 * (1 << 20);
__host__ __device__ inline int64_t cell_most(int64_t n) { return n / 64 < kCellMax ? n / 64 : kCellMax; }
__host__ __device__ inline int64_t cell_values(int64_t n) {
    return cell_most(n) * 16384 < kCellValues ? cell_most(n) * 16384 : kCellValues;
}
// Buffers that hold any cut of images of up to nmax emitters.
inline NodeCaps node_caps(int nx, int ny, int64_t nmax, bool cells) {
    const int64_t npix = (int64_t)nx * ny;
    NodeCaps c;
    c.v = node_entries(nx, ny);
    c.f = c.y = 0;
    if (cells) {
        const int64_t f = cell_most(nmax) * kCellNodes * kCellNodes;
        if (npix <= kCellPixels && c.v < npix) c.v = npix;  // the pixels as the target
        c.f = f < kCellSums ? f : kCellSums;
        c.y = cell_values(nmax);
    }
    return c;
}

NodeGeom make_node_geom(const GeomParams &g);

#if defined(__CUDACC__)

// Nodes along one axis (even, for the 16-byte copies of weight rows) for a phase
// half-range phi and a curved part of up to curve T_2(x); fine: the FP64 kernel's.
__device__ __forceinline__ int node_count(double phi, double curve, double t, const double least[2], bool fine) {
    const double n = fine ? fmax(fmax(phi + 5.0 + 9.6 * cbrt(phi) + 30.0 * t, 2.0 * (curve + 5.0 + 9.6 * cbrt(curve))), least[1])
                          : fmax(phi + 3.7 + 6.33 * cbrt(phi) + 14.0 * t, least[0]);
    return n < (double)(2 * kNodeMax) ? ((int)ceil(n) + 1) / 2 * 2 : 2 * kNodeMax;
}

// Whether an object reaching r from the origin may take nodes at all (a NaN may not).
__device__ __forceinline__ bool node_reach(const GeomParams &g, const NodeGeom &ng, double r, bool fine) {
    if (!ng.ok || !(r * ng.inv_d <= kNodeMaxReach)) return false;
    return fine || !(g.flags & (IDIWF_NF | IDIWF_SECONDORDER)) || 0.5 * g.k * r * r * ng.inv_d <= kNodeMaxExtra;
}
// Nodes along both axes for emitters within rho of a centre, |rho . e| <= ex, ey along the
// axes, of an object reaching r from the origin.  Along e the phase changes by at most
// k/|d| (|rho . e| + |d_hat . e| |rho|), and by no more than k/|d| |rho|; the
// near-field and second-order terms, of the whole r, add up to 2 (|r|/|d|) k |r|/|d|.
__device__ __forceinline__ void node_grid(const NodeGeom &ng, double r, double rho, double ex, double ey, bool fine,
                                          int &n0, int &n1) {
    const double more = 2.0 * r * r * ng.inv_d;
    n0 = node_count(ng.phi[0] * (fmin(rho, ex + ng.s[0] * rho) + more), 0.25 * ng.phi[0] * rho * ng.t[0], ng.t[0], ng.least[0], fine);
    n1 = node_count(ng.phi[1] * (fmin(rho, ey + ng.s[1] * rho) + more), 0.25 * ng.phi[1] * rho * ng.t[1], ng.t[1], ng.least[1], fine);
}

// Node m of n on [-1, 1], its barycentric weight, and the (fractional) pixel
// index it sits at on an axis of N pixels.
__device__ __forceinline__ double node_x(int n, int m) { return cospi((2 * m + 1) / (2.0 * n)); }
__device__ __forceinline__ double node_w(int n, int m) {
    const double s = sinpi((2 * m + 1) / (2.0 * n));
    return (m & 1) ? -s : s;
}
__device__ __forceinline__ double node_index(int n, int m, int N) { return 0.5 * (N - 1) * (1.0 + node_x(n, m)); }

// Pixel i of N on [-1, 1].
__device__ __forceinline__ double pixel_x(int N, int i) { return N > 1 ? (2 * i - (N - 1)) / (double)(N - 1) : 0.0; }

// Interpolation weights of one axis at x, row i: L[i][m], m < n, by the barycentric
// formula (Berrut and Trefethen, SIAM Review 46(3), 2004), one warp per row.
__device__ __forceinline__ void node_weights_row(double *__restrict__ L, int n, double x, int i, int lane) {
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
// further kernels cost more than the direct sum (split precision, FP64).  In
// differentiation (split-precision complex128 fields, and the adjoint) the host's launches
// set the pace of small images, and the direct kernels have fewer: a gradient step of
// 26e6 pairs 0.67 ms direct, 0.69 over nodes, of 47e6 pairs 0.68 and 0.66.
constexpr double kNodeMinPairs = 8e6, kNodeMinPairs64 = 2e6, kNodeMinPairsDiff = 3.2e7;

// Floats as unsigned integers in their order (0 lies below them all).
__device__ __forceinline__ uint32_t float_key(float f) {
    const uint32_t u = __float_as_uint(f);
    return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float key_float(uint32_t k) {
    return __uint_as_float(k & 0x80000000u ? k & 0x7fffffffu : ~k);
}

// Largest extents of an emitter for the plan: |r|^2 and |a| (float bits, rounded up), and
// r . e and -r . e along the three axes (keys, rounded up), raised per block into ext: extent
// k of image b at b * sb + k * sk.
constexpr int kNodeExt = 8;
struct NodeExtents {
    uint32_t v[kNodeExt] = {0, 0, 0, 0, 0, 0, 0, 0};
    __device__ __forceinline__ void add(const NodeGeom &ng, const double4 &p, float amp) {
        v[0] = max(v[0], __float_as_uint(__double2float_ru((p.x * p.x + p.y * p.y) + p.z * p.z)));
        v[1] = max(v[1], __float_as_uint(fabsf(amp)));
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double x = p.x * ng.e[k][0] + p.y * ng.e[k][1] + p.z * ng.e[k][2];
            v[2 + k] = max(v[2 + k], float_key(__double2float_ru(x)));
            v[5 + k] = max(v[5 + k], float_key(__double2float_ru(-x)));
        }
    }
    // (one atomic per block and extent: a warp's own would queue up on the image's words)
    __device__ __forceinline__ void raise(uint32_t *ext, int b, int sb = kNodeExt, int sk = 1) const {
        __shared__ uint32_t s_max[kNodeExt];
        if (threadIdx.x < kNodeExt) s_max[threadIdx.x] = 0;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kNodeExt; ++k) {
            const uint32_t m = __reduce_max_sync(0xffffffffu, v[k]);
            if ((threadIdx.x & 31) == 0 && m) atomicMax(&s_max[k], m);
        }
        __syncthreads();
        if (threadIdx.x < kNodeExt && s_max[threadIdx.x])
            atomicMax(ext + b * sb + threadIdx.x * sk, s_max[threadIdx.x]);
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

// Seconds of an image's evaluation on nodes: the sums, the cells' interpolation to the
// target grid and their phases, and the last interpolation to the pixels; rates
// as measured (node pairs per second; FP64 multiply-adds per second).
__device__ __forceinline__ double node_cost(double n, int nx, int ny, const NodeImage &ni, double pair_rate) {
    const double npix = (double)nx * ny, m = (double)((ni.g0 * ni.g1 + 127) / 128) * 128.0;
    double t = (n + 32.0 * ni.ncell) * m / pair_rate;
    if (ni.ncell > 1) {
        const double t0 = (ni.n0 + 31) / 32 * 32.0, t1 = (ni.n1 + 31) / 32 * 32.0;
        t += ni.ncell * (2.0 * ((ni.n1 + 63) / 64 * 64.0) * ((ni.g0 + 31) / 32 * 32.0) * ni.g1 * (1.0 / 0.9e13) +
                         t0 * t1 * (2.0 * ni.g0 * (1.0 / 0.9e13) + 1.6e-12));
    }
    if (!ni.pix) t += 2.0 * ni.n0 * (npix + (double)ni.n1 * ny) * (1.0 / 1.2e13);
    return t + 100.0 * npix * (1.0 / 1.2e13);
}

// Plan of one launch, by one block: every image's path, grids and fixed-point scale; one warp
// per image, whose lanes try the ways to cut it.  The choice depends on the image and the
// geometry alone, as split_path's does.  fine: the FP64 kernel's images (their direct path
// counts as kPathPixel).
__device__ inline void plan_nodes(const BatchParams &bp, const GeomParams &g, const NodeGeom &ng,
                                  const uint32_t *ext, bool fine, WsHeader *hdr, NodePlan *plan) {
    __threadfence();
    const int npix = g.nx * g.ny, lane = threadIdx.x & 31;
    for (int i = threadIdx.x >> 5; i < bp.n_images; i += blockDim.x >> 5) {
        uint32_t x[kNodeExt];
#pragma unroll
        for (int k = 0; k < kNodeExt; ++k) x[k] = __ldcg(ext + i * kNodeExt + k);
        const int n = bp.img[i].n;
        const uint32_t amax = x[1];
        NodeImage ni;
        ni.path = fine ? kPathPixel : split_path(g, x[0], bp.groups != 0, false);
        ni.n0 = ni.n1 = ni.g0 = ni.g1 = ni.pix = ni.ntiles = ni.nblk = 0;
        ni.scale = 1.0f;
        ni.ncell = ni.c[0] = ni.c[1] = ni.c[2] = 1;
        ni.ticket = 0;
        const double r = sqrt((double)__uint_as_float(x[0]));
        const double pairs = (double)n * npix;
        const int direct = ni.path;
        unsigned long long pr = (unsigned long long)n * npix;
        // (amplitudes whose fixed-point unit would leave FP32's exponents, infinite or NaN
        // ones take the direct kernels)
        if (bp.nodes && n > 0 && (direct == kPathRuns || direct == kPathPixel) &&
            pairs >= ng.min_pairs && node_reach(g, ng, r, fine) &&
            (amax == 0u || (amax >= __float_as_uint(0x1p-40f) && amax <= __float_as_uint(0x1p100f)))) {
            double lo[3], w[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                lo[k] = -(double)key_float(x[5 + k]);
                w[k] = fmax((double)key_float(x[2 + k]) - lo[k], 1e-12 * r);
            }
            // the uncut object, about the origin
            NodeImage best = ni;
            node_grid(ng, r, r, fmax(lo[0] + w[0], -lo[0]), fmax(lo[1] + w[1], -lo[1]), fine, best.n0, best.n1);
            best.g0 = best.n0;
            best.g1 = best.n1;
            const bool whole = best.n0 <= node_cap(g.nx) && best.n1 <= node_cap(g.ny) &&
                               (double)best.n0 * best.n1 <= (double)node_entries(g.nx, g.ny);
            const double rate = fine ? 1.3e11 : 1.0e12;
            double cost = pairs / (fine ? 1.6e11 : (direct == kPathRuns ? 1.8e12 : 1.5e12));
            bool use = false;
            if (whole) {
                const double c = node_cost(n, g.nx, g.ny, best, rate);
                use = c < cost;
                cost = fmin(c, cost);
            }
            if (bp.nodes > 1 && n >= kCellMinEmitters) {
                // lanes 0..15: to the image's nodes, 16..31: to the pixels; edges of 1/2 .. 1/36
                NodeImage cut = best;
                cut.pix = lane >> 4;
                if (cut.pix) {
                    cut.n0 = g.nx;
                    cut.n1 = g.ny;
                }
                const int ci = lane & 15, parts = ci < 6 ? ci + 2 : (ci < 10 ? 2 * ci - 4 : 4 * ci - 24);
                const double edge = fmax(w[0], w[1]) / parts;
                cut.c[0] = (int)fmin(ceil(w[0] / edge - 1e-9), 1e6);
                cut.c[1] = (int)fmin(ceil(w[1] / edge - 1e-9), 1e6);
                cut.c[2] = (int)fmin(ceil(w[2] * fmax(ng.s[0], ng.s[1]) / edge), 1e6);
                cut.c[0] = max(cut.c[0], 1);
                cut.c[1] = max(cut.c[1], 1);
                cut.c[2] = max(cut.c[2], 1);
                const double nc = (double)cut.c[0] * cut.c[1] * cut.c[2];
                double c = 1e30;
                if (nc > 1.0 && nc <= (double)cell_most(n) && (cut.pix ? npix <= kCellPixels : whole)) {
                    cut.ncell = (int)nc;
                    double h[3];
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        cut.lo[k] = lo[k];
                        cut.size[k] = w[k] / cut.c[k];
                        cut.inv[k] = cut.c[k] / w[k];
                        h[k] = 0.5 * cut.size[k] * (1.0 + 1e-9);
                    }
                    node_grid(ng, r, sqrt(h[0] * h[0] + h[1] * h[1] + h[2] * h[2]), h[0], h[1], fine, cut.g0, cut.g1);
                    if (cut.g0 <= kCellNodes && cut.g1 <= kCellNodes && nc * cut.g0 * cut.g1 <= (double)kCellSums &&
                        nc * cut.n1 * cut.g0 <= (double)cell_values(n))
                        c = node_cost(n, g.nx, g.ny, cut, rate);
                }
                double least = c;
#pragma unroll
                for (int o = 16; o; o >>= 1) least = fmin(least, __shfl_xor_sync(0xffffffffu, least, o));
                const int who = __ffs(__ballot_sync(0xffffffffu, c == least)) - 1;
                if (least < 0.95 * cost) {
                    use = true;
                    // the winner's choice, to every lane
                    best.pix = who >> 4;
                    best.n0 = __shfl_sync(0xffffffffu, cut.n0, who);
                    best.n1 = __shfl_sync(0xffffffffu, cut.n1, who);
                    best.g0 = __shfl_sync(0xffffffffu, cut.g0, who);
                    best.g1 = __shfl_sync(0xffffffffu, cut.g1, who);
                    best.ncell = __shfl_sync(0xffffffffu, cut.ncell, who);
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        best.c[k] = __shfl_sync(0xffffffffu, cut.c[k], who);
                        best.lo[k] = lo[k];
                        best.size[k] = w[k] / best.c[k];
                        best.inv[k] = best.c[k] / w[k];
                    }
                }
            }
            if (use) {
                ni = best;
                ni.path = kPathNodes;
                const int m = ni.g0 * ni.g1, tile = fine ? kNodeTile64 : kNodeTile;
                ni.ntiles = (m + tile - 1) / tile;
                ni.nblk = (n + kNodeBlock - 1) / kNodeBlock;  // (the sort replaces it where there are cells)
                pr = (unsigned long long)n * m;
                // |sum| <= n max |a| [times the largest 1/|d - r| <= 4/(3 D)] < 2^e; three bits to
                // spare for the interpolated cells' partial sums
                double bound = (double)n * (double)__uint_as_float(amax);
                if ((g.flags & IDIWF_NF) && (g.flags & IDIWF_SCALE)) bound *= 1.4 * ng.inv_d;
                if (bound > 0.0) ni.scale = (float)scalbn(1.0, min(max(59 - (ilogb(bound) + 1), -120), 120));
            }
        }
        if (lane == 0) {
            atomicAdd(&hdr->pairs, pr);
            if (n > 0 && ni.path != kPathNodes) atomicAdd(&hdr->direct, 1u);
            plan->img[i] = ni;
        }
    }
}

// Cell of an emitter, and a cell's centre; written with explicit roundings so that every
// kernel places an emitter alike.
__device__ __forceinline__ int cell_of(const NodeGeom &ng, const NodeImage &ni, const double4 &p) {
    int id = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double x = __fma_rn(p.z, ng.e[k][2], __fma_rn(p.y, ng.e[k][1], __dmul_rn(p.x, ng.e[k][0])));
        const int c = min(max((int)floor(__dmul_rn(__dsub_rn(x, ni.lo[k]), ni.inv[k])), 0), ni.c[k] - 1);
        id = id * ni.c[k] + c;
    }
    return id;
}
__device__ __forceinline__ void cell_centre(const NodeGeom &ng, const NodeImage &ni, int id, double r[3]) {
    int c[3];
    c[2] = id % ni.c[2];
    c[1] = id / ni.c[2] % ni.c[1];
    c[0] = id / (ni.c[2] * ni.c[1]);
    double x[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) x[k] = __fma_rn(c[k] + 0.5, ni.size[k], ni.lo[k]);
#pragma unroll
    for (int a = 0; a < 3; ++a)
        r[a] = __fma_rn(x[2], ng.e[2][a], __fma_rn(x[1], ng.e[1][a], __dmul_rn(x[0], ng.e[0][a])));
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

// One tile at (i0, j0); `store(i, j, re, im)` receives every element inside M x N.  WORDS: X
// holds fixed-point sums (two 64-bit integers, value / unit) of one word or, the second in
// `low` (kLowUnit of the first's units), of two.
template <int WORDS, class Store>
__device__ __forceinline__ void interp_tile(GemmSmem &sm, const double *__restrict__ L, const double2 *__restrict__ X,
                                            const double2 *__restrict__ low, int M, int N, int K, int i0, int j0,
                                            double unit, const Store &store) {
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
            if (WORDS) {
                longlong2 v = make_longlong2(0, 0);
                if (ok) v = reinterpret_cast<const longlong2 *>(X)[(size_t)(j0 + r) * K + k0 + k];
                double2 x = make_double2((double)v.x, (double)v.y);
                if (WORDS == 2) {
                    // (the first word's part below FP64's 53 bits joins the second)
                    longlong2 w = make_longlong2(0, 0);
                    if (ok) w = reinterpret_cast<const longlong2 *>(low)[(size_t)(j0 + r) * K + k0 + k];
                    x.x += (double)(v.x - (long long)x.x) + (double)w.x * kLowUnit;
                    x.y += (double)(v.y - (long long)x.y) + (double)w.y * kLowUnit;
                }
                sm.b[s][r * kGemmLd + k] = make_double2(x.x * unit, x.y * unit);
            } else {
                cp_async16(&sm.b[s][r * kGemmLd + k], X + (ok ? (size_t)(j0 + r) * K + k0 + k : 0), ok);
            }
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
