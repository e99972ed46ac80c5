// Direct q-space autocorrelation of detector images (the consumers of the
// simulated intensities): idi/reconstruction/cucorrad.py (radial) and
// idi/reconstruction/cucor.py (3d).
//
// Pair set (both): reference pixel (r, c), target (r + dr, c + dc) with
// 0 <= dr < qmax and dc in the column-offset range; one thread per column
// offset walks the row pair and keeps a run: consecutive pairs with the same
// bin are summed in FP32 and the run is added to the FP64 histogram when the
// bin changes -- the radial reference kernel's accumulation, and for the 3d
// one (which adds every pair to FP32 bins) far fewer atomics.
//
//  * qcorr_radial_kernel — CTA = (reference row, group of target
//    rows, up to two images and their mirror rows).  The reference row and each
//    target row are staged in shared memory, q as float4 and the values of all
//    images beside each other.  The bin round(sqrt(d2)) is re-derived
//    only when d2 leaves the current bin's interval (a table of the exact
//    d2 thresholds), since it rarely changes along a row.  Bins go to an FP64
//    shared-memory histogram, added to the output once per CTA.
//  * qcorr_3d_kernel — the same walk over float2 {zd, v} rows; runs go to the
//    FP64 output with global atomics (the 3d histogram does not fit on chip);
//    bins outside the array are dropped.
//  * qcorr_sym_kernel — the reference's symmetrisation about the centre, each
//    mirror pair handled by exactly one thread.
#include <cmath>

#include "idiwf_internal.cuh"

namespace idiwf {

constexpr int kRowsPerCta = 8;  // target rows of a 3d correlator's CTA
constexpr int kQcorrMaxSmemCols = 4096;

// ---------------------------------------------------------------------------
// radial
// ---------------------------------------------------------------------------
// A walk's bins depend on the geometry alone, and finding them costs more than the
// products (two LDS.128, eight FP32 operations and two comparisons per pair against a
// product and a sum), so a walk serves every image value that shares it:
//  * up to kRadialImages images of a stack;
//  * on a detector centred on its rows (q(nr - r, c) = (-qx, qy, qz)(r, c), checked bit for
//    bit by qcorr_mirror_kernel), the mirror walk: reference row nr - t, target row nr - r
//    and column offset -dc visit pairs of the same d2 in the same order, so the walk (r, t, dc)
//    also sums v(nr - t, c + dc) v(nr - r, c).
// Each value keeps its own run in FP32, summed in the reference's order: the sums are
// those of one walk per image, bit for bit.  A thread walks two neighbouring column offsets:
// the second walk's target is the first's next one, so each shared-memory load of a
// target serves both (shared memory bounded the one-offset form: ten wavefronts per
// pair and four values).  Targets are stored by column parity, which keeps the lanes, two
// columns apart, on consecutive addresses.  2 x 512^2, 256 bins: 16.0 ms against 35.5 with
// one walk per image, row pair and offset.  What bounds it now is the bin changes: a lane
// changes bins every 10 to 50 pairs, a warp at every other pair.
constexpr int kRadialImages = 2;

// flag |= 1 where q(nr - r, c) is not (-qx, qy, qz)(r, c), r >= 1.
__global__ void qcorr_mirror_kernel(const float4 *__restrict__ q, int nr, int nc, uint32_t *__restrict__ flag) {
    bool bad = false;
    const int64_t half = (int64_t)(nr / 2) * nc;  // rows 1 .. nr / 2 against nr - 1 .. nr - nr / 2
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < half; i += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(i / nc) + 1, c = (int)(i % nc);
        const float4 a = q[(int64_t)r * nc + c], b = q[(int64_t)(nr - r) * nc + c];
        bad |= !(b.x == -a.x && b.y == a.y && b.z == a.z);
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1u);
}

// One walk's run: V values per position, V = images x (1 or 2).
template <int V>
struct RadialWalk {
    float val[V];
    float lo, hi;  // the current bin's interval of d2
    int dq, dqold;
    bool in_range;
};
template <int V>
struct RadialPoint {
    float x, y, z, v[V];
};
template <int V>
__device__ __forceinline__ RadialPoint<V> radial_point(const float4 *__restrict__ q, const float *__restrict__ v, int i) {
    RadialPoint<V> p;
    const float4 a = q[i];
    p.x = a.x;
    p.y = a.y;
    p.z = a.z;
    if constexpr (V == 4) {
        const float4 t = *reinterpret_cast<const float4 *>(v + 4 * i);
        p.v[0] = t.x;
        p.v[1] = t.y;
        p.v[2] = t.z;
        p.v[3] = t.w;
    } else if constexpr (V == 2) {
        const float2 t = *reinterpret_cast<const float2 *>(v + 2 * i);
        p.v[0] = t.x;
        p.v[1] = t.y;
    } else {
#pragma unroll
        for (int k = 0; k < V; ++k) p.v[k] = v[V * i + k];
    }
    return p;
}

template <int NB, bool MIR>
__device__ __forceinline__ void radial_walks(const float4 *__restrict__ q, const float *__restrict__ images, int nr,
                                             int nc, int qmax, int rows, int refr, float4 *sref, float4 *stgt,
                                             float *vref, float *vtgt, double *hist, const float *bound) {
    constexpr int V = NB * (MIR ? 2 : 1);
    const int tid = threadIdx.x;
    const int64_t npix = (int64_t)nr * nc;
    const int half = (nc + 1) / 2;
    const auto at = [half](int c) { return (c >> 1) + (c & 1) * half; };  // targets by column parity
    const bool row_mirrors = MIR && refr > 0;  // row 0 has no mirror row
    for (int c = tid; c < nc; c += blockDim.x) {
        sref[c] = q[(int64_t)refr * nc + c];
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            vref[c * V + k] = images[k * npix + (int64_t)refr * nc + c];
            if (MIR) vref[c * V + NB + k] = row_mirrors ? images[k * npix + (int64_t)(nr - refr) * nc + c] : 0.0f;
        }
    }
    // column offsets o and o + 1 of -most..most; tc = refc + offset in [0, nc)
    const int most = min(qmax, nc - 1), o = 2 * tid - most;
    const bool active[2] = {o <= most, o + 1 <= most};
    int c0[2], c1[2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        c0[w] = max(0, -(o + w));
        c1[w] = active[w] ? max(min(nc, nc - (o + w)), c0[w]) : c0[w];
    }
    const int both0 = max(c0[0], c0[1]), both1 = min(c1[0], c1[1]);
    const int dr0 = blockIdx.y * rows;
    for (int dr = dr0; dr < min(dr0 + rows, qmax); ++dr) {
        const int tr = refr + dr;
        if (tr >= nr) break;
        // the mirror pair of rows (nr - tr, nr - refr): the smaller reference row walks for both
        if (row_mirrors && refr > nr - tr) continue;
        const bool both = row_mirrors && refr < nr - tr;
        __syncthreads();
        for (int c = tid; c < nc; c += blockDim.x) {
            const int i = at(c);
            stgt[i] = q[(int64_t)tr * nc + c];
#pragma unroll
            for (int k = 0; k < NB; ++k) {
                vtgt[i * V + k] = images[k * npix + (int64_t)tr * nc + c];
                if (MIR) vtgt[i * V + NB + k] = both ? images[k * npix + (int64_t)(nr - tr) * nc + c] : 0.0f;
            }
        }
        __syncthreads();
        if (!active[0]) continue;
        RadialWalk<V> wk[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
#pragma unroll
            for (int k = 0; k < V; ++k) wk[w].val[k] = 0.0f;
            wk[w].dqold = tid;  // any bin (receives an empty run), another for every thread
            wk[w].dq = qmax + 1;
            wk[w].lo = 1.0f;  // empty: the first pair derives its bin
            wk[w].hi = 0.0f;
            wk[w].in_range = false;
        }
        auto flush = [&](const float *val, int bin) {
#pragma unroll
            for (int k = 0; k < NB; ++k) {
                double x = (double)val[k];
                if (MIR && both) x += (double)val[NB + k];
                atomicAdd(&hist[k * (qmax + 1) + bin], x);
            }
        };
        // The reference, per pair: if dq <= qmax { if dq != dqold { add the
        // run to dqold; dqold = dq; val = 0 } val += v v' }.  While the bin
        // stays the same, dq == dqold whenever dq <= qmax, so that test
        // only needs to run when the bin changes.
        auto step = [&](RadialWalk<V> &r, const RadialPoint<V> &a, const RadialPoint<V> &b) {
            const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
            const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
            if (!(d2 >= r.lo && d2 < r.hi)) {  // left the current bin's interval
                r.dq = min((int)rintf(__fsqrt_rn(d2)), qmax + 1);
                r.lo = bound[r.dq];
                r.hi = bound[r.dq + 1];
                r.in_range = r.dq <= qmax;
                if (r.in_range && r.dq != r.dqold) {
                    flush(r.val, r.dqold);
                    r.dqold = r.dq;
#pragma unroll
                    for (int k = 0; k < V; ++k) r.val[k] = 0.0f;
                }
            }
            if (r.in_range)
#pragma unroll
                for (int k = 0; k < V; ++k) r.val[k] = __fadd_rn(r.val[k], __fmul_rn(a.v[k], b.v[k]));
        };
        auto ref = [&](int c) { return radial_point<V>(sref, vref, c); };
        auto tgt = [&](int c) { return radial_point<V>(stgt, vtgt, at(c)); };
        // the pairs before and after the range that both walks share
#pragma unroll
        for (int w = 0; w < 2; ++w)
            for (int c = c0[w]; c < min(both0, c1[w]); ++c) step(wk[w], ref(c), tgt(c + o + w));
        if (both0 < both1) {
            RadialPoint<V> t = tgt(both0 + o);
#pragma unroll 4
            for (int c = both0; c < both1; ++c) {
                const RadialPoint<V> a = ref(c), t1 = tgt(c + o + 1);
                step(wk[0], a, t);
                step(wk[1], a, t1);
                t = t1;
            }
        }
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            for (int c = max(both1, min(both0, c1[w])); c < c1[w]; ++c) step(wk[w], ref(c), tgt(c + o + w));
            if (active[w] && wk[w].dq < qmax) flush(wk[w].val, wk[w].dq);
        }
    }
}

// CTA = (reference row, `rows` target rows, NB images); mirror: flag 0 says that the
// rows mirror (nullptr: not looked at, the rows would not fit in shared memory).
template <int NB, int THREADS, int BLOCKS>
__global__ void __launch_bounds__(THREADS, BLOCKS) qcorr_radial_kernel(const float4 *__restrict__ q,
                                                            const float *__restrict__ images, int nr, int nc,
                                                            int qmax, int rows, double *__restrict__ out,
                                                            const uint32_t *__restrict__ mirror) {
    extern __shared__ __align__(16) unsigned char qsm[];
    const bool mir = mirror && *mirror == 0u;
    const int v = NB * (mirror ? 2 : 1);
    float4 *sref = reinterpret_cast<float4 *>(qsm);
    float4 *stgt = sref + nc;
    float *vref = reinterpret_cast<float *>(stgt + nc + 1);  // (odd nc: the parities take nc + 1 places)
    float *vtgt = vref + (size_t)((nc + 1) * v + 3) / 4 * 4;
    double *hist = reinterpret_cast<double *>(vtgt + (size_t)((nc + 1) * v + 3) / 4 * 4);  // NB x (qmax + 1)
    float *bound = reinterpret_cast<float *>(hist + NB * (qmax + 1));               // qmax + 3 entries
    const int refr = blockIdx.x;
    const int tid = threadIdx.x;
    // rows past the detector, or (mirrored) walked by their mirror rows: nothing to do
    const int dr0 = blockIdx.y * rows;
    if (refr + dr0 >= nr || (mir && refr > 0 && 2 * refr + dr0 > nr)) return;
    for (int i = tid; i < NB * (qmax + 1); i += blockDim.x) hist[i] = 0.0;
    // bound[k]: smallest float d2 >= 0 with rint(sqrt(d2)) >= k, k = 0..qmax+1,
    // by bisection over the (monotone) float bit patterns with the very
    // operations of the bin below; bound[qmax+2] = +inf.  Bins above qmax are
    // one class (the reference only tests dq <= qmax and dq < qmax there).
    for (int k = tid; k <= qmax + 2; k += blockDim.x) {
        float b;
        if (k == 0) {
            b = 0.0f;
        } else if (k == qmax + 2) {
            b = __int_as_float(0x7F800000);
        } else {
            uint32_t lo = 0u, hi = 0x7F800000u;  // rint(sqrt(+0)) = 0 < k <= rint(sqrt(+inf))
            while (hi - lo > 1u) {
                const uint32_t mid = lo + (hi - lo) / 2u;
                if ((int)rintf(__fsqrt_rn(__uint_as_float(mid))) >= k) hi = mid;
                else lo = mid;
            }
            b = __uint_as_float(hi);
        }
        bound[k] = b;
    }
    if (mir) radial_walks<NB, true>(q, images, nr, nc, qmax, rows, refr, sref, stgt, vref, vtgt, hist, bound);
    else radial_walks<NB, false>(q, images, nr, nc, qmax, rows, refr, sref, stgt, vref, vtgt, hist, bound);
    __syncthreads();
    for (int k = 0; k < NB; ++k)
        for (int i = tid; i < qmax; i += blockDim.x)
            if (hist[k * (qmax + 1) + i] != 0.0) atomicAdd(&out[(int64_t)k * qmax + i], hist[k * (qmax + 1) + i]);
}

// Shared memory of the kernel for nb images, with or without the mirror rows.
static size_t radial_smem(int nc, int qmax, int nb, bool mirror) {
    const size_t v = (size_t)nb * (mirror ? 2 : 1);
    return (2 * (size_t)nc + 1) * sizeof(float4) + 2 * (((nc + 1) * v + 3) / 4 * 4) * sizeof(float) +
           (size_t)nb * (qmax + 1) * sizeof(double) + (size_t)(qmax + 3) * sizeof(float);
}

// ---------------------------------------------------------------------------
// 3d
// ---------------------------------------------------------------------------
struct Q3Params {
    int nr, nc, qmax, maxdqz;
    float xcenter, ycenter, z;
};

__device__ __forceinline__ void q3_flush(double *o, int64_t bin, float val) {
    if (bin >= 0) atomicAdd(&o[bin], (double)val);
}

__global__ void __launch_bounds__(1024) qcorr_3d_kernel(const float *__restrict__ zd, const float *__restrict__ images,
                                                        const Q3Params P, double *__restrict__ out) {
    extern __shared__ __align__(16) unsigned char qsm[];
    float2 *sref = reinterpret_cast<float2 *>(qsm);
    float2 *stgt = sref + P.nc;
    const int refr = blockIdx.x;
    const int img = blockIdx.z;
    const int nc = P.nc, qmax = P.qmax;
    const int D0 = 2 * P.maxdqz, D1 = 2 * qmax, D2 = 2 * qmax;
    const float *v = images + (int64_t)img * P.nr * nc;
    double *o = out + (int64_t)img * D0 * D1 * D2;
    const int tid = threadIdx.x;
    for (int c = tid; c < nc; c += blockDim.x)
        sref[c] = make_float2(zd[(int64_t)refr * nc + c], v[(int64_t)refr * nc + c]);
    const float refr2 = __fsub_rn((float)refr, P.xcenter);
    const int dr0 = blockIdx.y * kRowsPerCta;
    for (int dr = dr0; dr < min(dr0 + kRowsPerCta, qmax); ++dr) {
        const int tr = refr + dr;
        if (tr >= P.nr) break;
        __syncthreads();
        for (int c = tid; c < nc; c += blockDim.x)
            stgt[c] = make_float2(zd[(int64_t)tr * nc + c], v[(int64_t)tr * nc + c]);
        __syncthreads();
        const float tr2 = __fsub_rn((float)tr, P.xcenter);
        for (int offsetc = tid - (qmax - 1); offsetc <= qmax - 1; offsetc += blockDim.x) {
            const int c0 = max(0, -offsetc), c1 = min(nc, nc - offsetc);
            int64_t bin = -1;
            float val = 0.0f;
            for (int refc = c0; refc < c1; ++refc) {
                const int tc = refc + offsetc;
                const float2 a = sref[refc];
                const float2 b = stgt[tc];
                const int dqx = qmax + (int)rintf(__fsub_rn(__fmul_rn(tr2, b.x), __fmul_rn(refr2, a.x)));
                const int dqy = qmax + (int)rintf(__fsub_rn(__fmul_rn(__fsub_rn((float)tc, P.ycenter), b.x),
                                                            __fmul_rn(__fsub_rn((float)refc, P.ycenter), a.x)));
                const int dqz = P.maxdqz + (int)rintf(__fmul_rn(P.z, __fsub_rn(a.x, b.x)));
                if (dqz < 0 || dqz >= D0 || dqy < 0 || dqy >= D1 || dqx < 0 || dqx >= D2) continue;
                const int64_t nb = ((int64_t)dqz * D1 + dqy) * D2 + dqx;
                if (nb != bin) {
                    q3_flush(o, bin, val);
                    bin = nb;
                    val = 0.0f;
                }
                val = __fadd_rn(val, __fmul_rn(a.y, b.y));
            }
            q3_flush(o, bin, val);
        }
    }
}

// bins i and -i mod (D0, D1, D2) for i_x in [0, n2) hold the sum of both;
// one thread per mirror pair (the smaller index where both ends are
// visited), a bin that is its own mirror doubles.  n2 is the x extent the
// reference's assemble launch covers: D2/2, or 2 (D2/4) when D2 > 64.
__global__ void qcorr_sym_kernel(double *__restrict__ out, int D0, int D1, int D2, int n2, int n_images) {
    const int64_t per = (int64_t)D0 * D1 * n2;
    const int64_t total = per * n_images;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int img = (int)(t / per);
        int64_t r = t - (int64_t)img * per;
        const int i2 = (int)(r % n2);
        r /= n2;
        const int i1 = (int)(r % D1);
        const int i0 = (int)(r / D1);
        const int m0 = (D0 - i0) % D0, m1 = (D1 - i1) % D1, m2 = (D2 - i2) % D2;
        double *o = out + (int64_t)img * D0 * D1 * D2;
        const int64_t a = ((int64_t)i0 * D1 + i1) * D2 + i2;
        const int64_t b = ((int64_t)m0 * D1 + m1) * D2 + m2;
        if (a == b) {
            o[a] = 2.0 * o[a];
        } else if (m2 >= n2 || a < b) {  // the mirror is visited too only when m2 < n2: take one of the two
            const double s = o[a] + o[b];
            o[a] = s;
            o[b] = s;
        }
    }
}

static int qcorr_sms() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

}  // namespace idiwf

using namespace idiwf;

extern "C" size_t idiwf_qcorr_workspace_size(int32_t nr, int32_t nc) {
    (void)nr;
    (void)nc;
    return 256;
}

extern "C" idiwf_status idiwf_qcorr_radial(const float *q, const float *images, int32_t n_images, int32_t nr,
                                           int32_t nc, int32_t qmax, double *out, void *workspace,
                                           size_t workspace_bytes, cudaStream_t stream) {
    if (!q || !images || !out) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "q, images and out must be non-NULL");
    if (n_images <= 0 || n_images > 65535 || nr <= 0 || nc <= 0)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "n_images in 1..65535, nr and nc positive");
    if (qmax < 1 || qmax > 511) return set_error(IDIWF_ERR_UNSUPPORTED, "qmax must be in 1..511");
    if (nc > kQcorrMaxSmemCols) return set_error(IDIWF_ERR_UNSUPPORTED, "at most 4096 detector columns");
    if (reinterpret_cast<uintptr_t>(q) & 15) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "q must be 16-byte aligned");
    if (!workspace || workspace_bytes < 256) return set_error(IDIWF_ERR_WORKSPACE, "workspace too small");
    IDIWF_CUDA_CHECK(cudaMemsetAsync(out, 0, sizeof(double) * (size_t)n_images * qmax, stream));
    // two of the 2 min(qmax, nc - 1) + 1 column offsets each
    const int threads = (std::min(qmax, nc - 1) + 1 + 31) / 32 * 32;
    const float4 *q4 = reinterpret_cast<const float4 *>(q);
    // as many images per walk, and the mirror rows, as 200 KB of shared memory hold (every
    // detector up to 2048 columns takes 2 images and the mirror rows)
    constexpr size_t kMost = 200 * 1024;
    const bool mirror = radial_smem(nc, qmax, 1, true) <= kMost && nr > 1;
    int nb = std::min(n_images, kRadialImages);
    while (nb > 1 && radial_smem(nc, qmax, nb, mirror) > kMost) --nb;
    uint32_t *flag = mirror ? &static_cast<WsHeader *>(workspace)->work_counter : nullptr;
    if (mirror) {
        IDIWF_CUDA_CHECK(cudaMemsetAsync(flag, 0, sizeof(uint32_t), stream));
        const int64_t half = (int64_t)(nr / 2) * nc;
        const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((half + 255) / 256, 2 * (int64_t)qcorr_sms()));
        qcorr_mirror_kernel<<<blocks, 256, 0, stream>>>(q4, nr, nc, flag);
        IDIWF_CUDA_CHECK(cudaGetLastError());
    }
    // Target rows per CTA: two where that leaves a dozen waves of CTAs (row pairs, half of
    // them walked by their mirror pairs), else one, so that small detectors fill the chip.
    // us with 1, 2 and 8 rows: 2 images of 99 x 64, 103 bins 108, 122, 225; 2 of 72 x 287,
    // 112 bins 226, 285, 621; 3 of 249 x 360, 167 bins 3970, 3998, 4652; 2 of 400 x 400, 256
    // bins 8533, 8350, 8633.
    const int64_t in_reach = std::min(qmax, nr);
    const int64_t row_pairs = in_reach * nr - in_reach * (in_reach - 1) / 2;
    int rows = row_pairs >= 4 * 12 * 4 * (int64_t)qcorr_sms() ? 2 : 1;
    const dim3 grid(nr, ((int)in_reach + rows - 1) / rows);
    for (int b = 0; b < n_images;) {
        const int n = std::min(nb, n_images - b);
        // blocks of up to 288 threads (up to 287 bins) fit four to an SM at 56 registers: bin
        // changes stall a warp for long, so more warps pay although a few values spill (2 x 512^2,
        // 256 bins: 16.0 ms; 16.7 with three at 72 registers, 20.3 with two)
        void *fn = threads <= 288 ? (n == 2 ? (void *)qcorr_radial_kernel<2, 288, 4> : (void *)qcorr_radial_kernel<1, 288, 4>)
                                  : (n == 2 ? (void *)qcorr_radial_kernel<2, 512, 2> : (void *)qcorr_radial_kernel<1, 512, 2>);
        const size_t smem = radial_smem(nc, qmax, n, mirror);
        // (one limit for every call: calls from several threads do not lower it under one another)
        IDIWF_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost));
        const float *im = images + (int64_t)b * nr * nc;
        double *o = out + (int64_t)b * qmax;
        void *args[] = {&q4, &im, &nr, &nc, &qmax, &rows, &o, &flag};
        IDIWF_CUDA_CHECK(cudaLaunchKernel(fn, grid, dim3(threads), args, smem, stream));
        b += n;
    }
    return IDIWF_OK;
}

extern "C" idiwf_status idiwf_qcorr_3d(const float *zd, const float *images, int32_t n_images, int32_t nr, int32_t nc,
                                       int32_t qmax, int32_t maxdqz, float xcenter, float ycenter, float z, double *out,
                                       void *workspace, size_t workspace_bytes, cudaStream_t stream) {
    if (!zd || !images || !out) return set_error(IDIWF_ERR_INVALID_ARGUMENT, "zd, images and out must be non-NULL");
    if (n_images <= 0 || n_images > 65535 || nr <= 0 || nc <= 0)
        return set_error(IDIWF_ERR_INVALID_ARGUMENT, "n_images in 1..65535, nr and nc positive");
    if (qmax < 1 || qmax > 1024) return set_error(IDIWF_ERR_UNSUPPORTED, "qmax must be in 1..1024");
    if (maxdqz < 1 || maxdqz > 4096) return set_error(IDIWF_ERR_UNSUPPORTED, "maxdqz must be in 1..4096");
    if (nc > 2 * kQcorrMaxSmemCols) return set_error(IDIWF_ERR_UNSUPPORTED, "at most 8192 detector columns");
    if (!workspace || workspace_bytes < 256) return set_error(IDIWF_ERR_WORKSPACE, "workspace too small");
    const int64_t D0 = 2 * (int64_t)maxdqz, D1 = 2 * (int64_t)qmax, D2 = 2 * (int64_t)qmax;
    IDIWF_CUDA_CHECK(cudaMemsetAsync(out, 0, sizeof(double) * (size_t)(n_images * D0 * D1 * D2), stream));
    Q3Params P{nr, nc, qmax, maxdqz, xcenter, ycenter, z};
    const size_t smem = 2 * (size_t)nc * sizeof(float2);
    IDIWF_CUDA_CHECK(cudaFuncSetAttribute(qcorr_3d_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int threads = std::min(1024, ((2 * qmax - 1) + 31) / 32 * 32);
    const dim3 grid(nr, (qmax + kRowsPerCta - 1) / kRowsPerCta, n_images);
    qcorr_3d_kernel<<<grid, threads, smem, stream>>>(zd, images, P, out);
    IDIWF_CUDA_CHECK(cudaGetLastError());
    const int n2 = (int)(D2 > 64 ? 2 * (D2 / 4) : D2 / 2);
    const int64_t pairs = n_images * D0 * D1 * n2;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((pairs + 255) / 256, 16 * (int64_t)qcorr_sms()));
    qcorr_sym_kernel<<<blocks, 256, 0, stream>>>(out, (int)D0, (int)D1, (int)D2, n2, n_images);
    IDIWF_CUDA_CHECK(cudaGetLastError());
    return IDIWF_OK;
}
