// Stage (a): XCorr spectrum preprocessing, one CTA per spectrum.
//
// Restates Spectrum/Correlation.hs:37-109 (observedIntensity,
// normaliseByRegion, crossCorrolation) and Spectrum/Data.hs:58-59 (ms2Mass)
// with every float operation an explicit IEEE-rounded intrinsic, so the FP32
// row is bit-identical to the reference's host computation:
//   bin   = round(mz / binWidth)        (ties to even, Haskell `round`)
//   value = max over the bin of sqrt(intensity)
//   norm  = 50 * (e / regionMax)  when regionMax > 1e-6 and i < sel*10
//   x[i]  = norm[i] - (sequential sum of norm over take 151 (drop (i-75)))/150
// The row lives in shared memory while it is built; the output is written
// once as FP32 and, optionally, as BF16 and FP16 copies (round to nearest).
#include "hfx_internal.h"

namespace hfx {

// Host masses, Mass.hs:19-25.
constexpr float kHostH2O = 18.010565f;
constexpr float kHostH = 1.007276f;

__device__ __forceinline__ float spec_cutoff(float last_mz, float pcr, float z) {
    // Correlation.hs:65-67: min (50 + pcr*z) (fromInteger (truncate (last/10) * 10))
    const float mzcut = __fadd_rn(50.0f, __fmul_rn(pcr, z));
    const double t = trunc((double)__fdiv_rn(last_mz, 10.0f));
    const float mzlim = (float)(t * 10.0);
    return (mzcut <= mzlim) ? mzcut : mzlim;
}

// Per-spectrum layout and search window (one thread per spectrum); no `tol`:
// 0.  `lens` and `masses`, where given: the rows' lengths (0 for none) and the
// spectra's masses.
__global__ void k_layout(const float *__restrict__ mz, const int64_t *__restrict__ off,
                         const float *__restrict__ pcr, const float *__restrict__ z,
                         const float *__restrict__ tol, int32_t nspec, LayoutParams lp,
                         SpecMeta *__restrict__ meta, uint32_t *__restrict__ max_len, uint32_t *__restrict__ err,
                         int32_t *__restrict__ lens, float *__restrict__ masses) {
    const int32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nspec) return;
    SpecMeta m;
    const int64_t o0 = off[s], o1 = off[s + 1];
    const float zs = z[s], ps = pcr[s];
    m.npk = (int32_t)(o1 - o0);
    m.status = 0;
    m.len = 0;
    m.cutoff = 0.0f;
    if (m.npk <= 0) {
        m.status = 1;  // empty spectrum: G.last fails in the reference
    } else {
        m.cutoff = spec_cutoff(mz[o1 - 1], ps, zs);
        const float c = lp.custom_bw ? __fdiv_rn(m.cutoff, lp.bw) : m.cutoff;
        const double len = 75.0 + ceil((double)c);
        if (!(len >= 76.0) || len > (double)lp.max_len) {
            m.status = 2;
        } else if (lp.cap_len > 0 && len > (double)lp.cap_len) {
            if (err) atomicOr(err, kErrTooLong);
            m.status = 2;
        } else {
            m.len = (int32_t)len;
            if ((m.len - 75) / 10 <= 0) m.status = 3;  // sel = 0: div by zero
        }
    }
    // Spectrum/Data.hs:58-59 ms2Mass with host constants
    m.mass = __fsub_rn(__fsub_rn(__fmul_rn(ps, zs), __fmul_rn(__fsub_rn(zs, 1.0f), kHostH)),
                       __fadd_rn(kHostH, kHostH2O));
    // tolerance unit: Da (filter.cu:105), ppm, or per spectrum (negative = ppm)
    const float ts = tol ? tol[s] : 0.0f;
    const bool in_ppm = lp.ppm == 1 || (lp.ppm == 2 && ts < 0.0f);
    const float eps = in_ppm ? __fmul_rn(m.mass, __fmul_rn(lp.ppm == 2 ? -ts : ts, 1e-6f)) : ts;
    m.eps = eps;
    m.lo = __fsub_rn(m.mass, eps);  // filter.cu:103-115 (m - eps), (m + eps)
    m.hi = __fadd_rn(m.mass, eps);
    // Search.hs:182 max_chs = round (max 1 (chrg - 1)); ion_series.cu:301-309
    const float zm = __fsub_rn(zs, 1.0f);
    const float mc = (1.0f <= zm) ? zm : 1.0f;
    const float rr = rintf(mc);
    int32_t ch = (rr >= 1.0f) ? (rr > 1000.0f ? 1000 : (int32_t)rr) : 0;
    m.charges_plain = (ch >= 1 && ch <= 4) ? ch : 0;
    m.charges_mod = (int16_t)((ch >= 1 && ch <= 10) ? min(ch, 4) : 0);  // mion_series.cu:303-306, 425-438
    m.nonfinite = 0;
    meta[s] = m;
    if (lens) lens[s] = m.status == 0 ? m.len : 0;
    if (masses) masses[s] = m.mass;
    if (m.status == 0) atomicMax(max_len, (uint32_t)m.len);
}

// Block-wide exclusive scan of one value per thread (blockDim.x <= 1024).
__device__ __forceinline__ int32_t block_excl_scan(int32_t v, int32_t *warp_tot, int32_t &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int32_t t = __shfl_up_sync(0xFFFFFFFFu, x, d);
        if (lane >= d) x += t;
    }
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int32_t w = lane < nw ? warp_tot[lane] : 0;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int32_t t = __shfl_up_sync(0xFFFFFFFFu, w, d);
            if (lane >= d) w += t;
        }
        warp_tot[lane] = w;
    }
    __syncthreads();
    total = warp_tot[nw - 1];
    const int32_t before = (warp ? warp_tot[warp - 1] : 0) + x - v;
    __syncthreads();
    return before;
}

// Zero [from, stride) of a row's copies.
__device__ __forceinline__ void zero_tail(float *o32, __nv_bfloat16 *obf, __half *oh, int64_t from, int64_t stride,
                                          bool vec) {
    int64_t v0 = stride;  // elements from here on in 16-byte stores
    if (vec) v0 = min((from + 7) & ~(int64_t)7, stride);
    for (int64_t i = from + threadIdx.x; i < v0; i += blockDim.x) {
        o32[i] = 0.0f;
        if (obf) obf[i] = __float2bfloat16_rn(0.0f);
        if (oh) oh[i] = __float2half_rn(0.0f);
    }
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    for (int64_t i = v0 + 4 * (int64_t)threadIdx.x; i < stride; i += 4 * (int64_t)blockDim.x)
        *reinterpret_cast<uint4 *>(o32 + i) = z;
    for (int64_t i = v0 + 8 * (int64_t)threadIdx.x; i < stride; i += 8 * (int64_t)blockDim.x) {
        if (obf) *reinterpret_cast<uint4 *>(obf + i) = z;
        if (oh) *reinterpret_cast<uint4 *>(oh + i) = z;
    }
}

// Whether a row's copies take 16-byte stores at multiples of 8 elements.
__device__ __forceinline__ bool row_vectors(const float *o32, const __nv_bfloat16 *obf, const __half *oh) {
    const uint64_t bits = (uint64_t)o32 | (uint64_t)obf | (uint64_t)oh;
    return (bits & 15u) == 0u;
}

// observedIntensity, Correlation.hs:58-71: the bins' maxima into row[0, len),
// zeroed here.
__device__ __forceinline__ void bin_peaks(float *row, int32_t len, const SpecMeta &m, SpecMeta *meta, float ps,
                                          int64_t o0, const float *__restrict__ mz, const float *__restrict__ it,
                                          const LayoutParams &lp) {
    // (up to three words past the row's end, before anything is there)
    for (int32_t i = 4 * threadIdx.x; i < len; i += 4 * blockDim.x)
        *reinterpret_cast<float4 *>(row + i) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncthreads();
    const float plo = __fsub_rn(ps, 15.0f), phi = __fadd_rn(ps, 15.0f);
    for (int32_t i = threadIdx.x; i < m.npk; i += blockDim.x) {
        const float x = mz[o0 + i];
        const bool keep = lp.remove_pcr ? (x <= m.cutoff && (x <= plo || phi <= x)) : (x <= m.cutoff);
        if (!keep) continue;
        const float q = rintf(__fdiv_rn(x, lp.bw));
        if (!(q >= 0.0f) || q >= (float)len) continue;  // the reference raises here
        const float v = __fsqrt_rn(it[o0 + i]);
        if (v >= 0.0f) atomicMax((int *)&row[(int32_t)q], __float_as_int(v));
        if (isinf(v)) meta->nonfinite = 1;
    }
    __syncthreads();
}

// Rows of up to 17,066 bins: one CTA per spectrum.  Every e is >= 0, so
// the left fold over a window (crossCorrolation, Correlation.hs:105-109) equals
// the left fold over its nonzero bins (adding +0 is exact and the sum never is
// -0).  The P nonzero bins are listed once, in bin order, and the row becomes
// the count of them before each bin.  A window's bins [a, b) of the list change
// only where one enters (75 bins below it) or leaves (76 above it), and a and b
// only grow, so a + b names the window's content: its sum is folded once, at
// those up to 2 P + 1 places, and every other bin looks it up.  Bound by the
// instructions issued (82 % of the slots): 10,000 spectra of 225 peaks, FP32 and
// BF16 rows 4,096 long (250 MB), took 0.30 ms folding at each of a row's bins,
// 0.105 ms so.  A list too long for the sums' room beside it is folded at every
// bin.
__global__ void __launch_bounds__(256) k_preprocess(const float *__restrict__ mz, const float *__restrict__ it,
                                                    const int64_t *__restrict__ off,
                                                    const float *__restrict__ pcr, LayoutParams lp,
                                                    SpecMeta *__restrict__ meta, int64_t stride,
                                                    float *__restrict__ out32, __nv_bfloat16 *__restrict__ outbf,
                                                    __half *__restrict__ outh) {
    extern __shared__ __align__(16) uint8_t sm_row[];
    float *row = reinterpret_cast<float *>(sm_row);          // [stride + 1] bin maxima, then
    int32_t *before = reinterpret_cast<int32_t *>(sm_row);   // the nonzero bins before each
    float *val = row + stride + 1;                           // [P] the nonzero bins' values,
    __shared__ float rmax[11];
    __shared__ int32_t warp_n[9];
    const int32_t s = blockIdx.x;
    const SpecMeta m = meta[s];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float *o32 = out32 + (int64_t)s * stride;
    __nv_bfloat16 *obf = outbf ? outbf + (int64_t)s * stride : nullptr;
    __half *oh = outh ? outh + (int64_t)s * stride : nullptr;
    const bool vec = (stride & 7) == 0 && row_vectors(o32, obf, oh);
    const int32_t len = (m.status == 0) ? m.len : 0;
    zero_tail(o32, obf, oh, len, stride, vec);
    if (m.status != 0) return;
    if (tid < 11) rmax[tid] = 0.0f;
    bin_peaks(row, len, m, meta + s, pcr[s], off[s], mz, it, lp);
    // the list of nonzero bins: each warp an eighth of the row
    const int32_t eighth = ((len + 255) >> 8) << 5;
    const int32_t i0 = min(len, warp * eighth), i1 = min(len, i0 + eighth);
    int32_t n = 0;
    for (int32_t i = i0; i < i1; i += 32)
        n += __popc(__ballot_sync(0xFFFFFFFFu, i + lane < i1 && row[i + lane] > 0.0f));
    if (lane == 0) warp_n[warp] = n;
    __syncthreads();
    int32_t pos = 0, P = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w < warp) pos += warp_n[w];
        P += warp_n[w];
    }
    uint16_t *bin = reinterpret_cast<uint16_t *>(val + P);  // [P] their bins
    float *sums = val + P + ((P + 1) >> 1);                 // [2 P + 1] the windows' sums / 150, by a + b
    const bool once = (int64_t)P + ((P + 1) >> 1) + 2 * P + 1 <= stride;
    // i / sel as the upper half of i * (2^32 / sel, up): exact for i * sel < 2^32
    const int32_t sel = (len - 75) / 10;
    const uint32_t inv = sel > 1 ? 0xFFFFFFFFu / (uint32_t)sel + 1u : 0u;
    auto region = [&](int32_t i) { return min(10, inv ? (int32_t)__umulhi((uint32_t)i, inv) : i); };
    for (int32_t i = i0; i < i1; i += 32) {
        const float v = i + lane < i1 ? row[i + lane] : 0.0f;
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, v > 0.0f);
        const int32_t at = pos + __popc(bal & ((1u << lane) - 1u));
        if (i + lane < i1) before[i + lane] = at;
        if (v > 0.0f) {
            val[at] = v;
            if (once) bin[at] = (uint16_t)(i + lane);
            atomicMax((int *)&rmax[region(i + lane)], __float_as_int(v));
        }
        pos += __popc(bal);
    }
    if (tid == 0) before[len] = P;
    __syncthreads();
    // normaliseByRegion, Correlation.hs:84-96
    auto normal = [&](float v, int32_t i) {
        const float mx = rmax[region(i)];
        return (mx > 1e-6f && i < sel * 10) ? __fmul_rn(50.0f, __fdiv_rn(v, mx)) : 0.0f;
    };
    if (once) {
        for (int32_t j = tid; j < P; j += blockDim.x) val[j] = normal(val[j], bin[j]);
    } else {
        for (int32_t i = tid; i < len; i += blockDim.x)
            if (before[i + 1] != before[i]) val[before[i]] = normal(val[before[i]], i);
    }
    auto window = [&](int32_t i, int32_t &a, int32_t &b) {
        const int32_t lo = max(0, i - 75);
        a = before[lo];
        b = before[min(len, lo + 151)];
    };
    // an infinite intensity over itself is no number, and no part of a sum
    const bool inf = (tid < 11 && isinf(rmax[tid]));
    const bool any_inf = __syncthreads_or(inf);
    auto fold = [&](int32_t a, int32_t b) {
        float acc = 0.0f;
        if (any_inf) {
            for (int32_t t = a; t < b; ++t) acc = __fadd_rn(acc, fmaxf(val[t], 0.0f));
        } else {
#pragma unroll 4
            for (int32_t t = a; t < b; ++t) acc = __fadd_rn(acc, val[t]);
        }
        return __fdiv_rn(acc, 150.0f);
    };
    if (once) {
        for (int32_t u = tid; u <= 2 * P; u += blockDim.x) {
            int32_t i = 0;
            if (u < P) i = bin[u] >= 151 ? (int32_t)bin[u] - 75 : -1;
            else if (u < 2 * P) i = (int32_t)bin[u - P] + 76;
            if (i < 0 || i >= len) continue;
            int32_t a, b;
            window(i, a, b);
            sums[a + b] = fold(a, b);
        }
        __syncthreads();
    }
    for (int32_t i = tid; i < len; i += blockDim.x) {
        int32_t a, b;
        window(i, a, b);
        const int32_t at = before[i];
        const float e = before[i + 1] != at ? val[at] : 0.0f;
        const float x = __fsub_rn(e, once ? sums[a + b] : fold(a, b));
        o32[i] = x;
        if (obf) obf[i] = __float2bfloat16_rn(x);
        if (oh) oh[i] = __float2half_rn(x);
    }
}

// Rows too long for that list in shared memory: every window folds all its bins.
__global__ void __launch_bounds__(256) k_preprocess_bins(const float *__restrict__ mz, const float *__restrict__ it,
                                                         const int64_t *__restrict__ off,
                                                         const float *__restrict__ pcr, LayoutParams lp,
                                                         SpecMeta *__restrict__ meta, int64_t stride,
                                                         float *__restrict__ out32, __nv_bfloat16 *__restrict__ outbf,
                                                         __half *__restrict__ outh) {
    extern __shared__ __align__(16) uint8_t sm_row[];
    float *e = reinterpret_cast<float *>(sm_row);  // [len]
    __shared__ float rmax[11];
    const int32_t s = blockIdx.x;
    const SpecMeta m = meta[s];
    const int tid = threadIdx.x;
    float *o32 = out32 + (int64_t)s * stride;
    __nv_bfloat16 *obf = outbf ? outbf + (int64_t)s * stride : nullptr;
    __half *oh = outh ? outh + (int64_t)s * stride : nullptr;
    const bool vec = (stride & 7) == 0 && row_vectors(o32, obf, oh);
    const int32_t len = (m.status == 0) ? m.len : 0;
    zero_tail(o32, obf, oh, len, stride, vec);
    if (m.status != 0) return;
    if (tid < 11) rmax[tid] = 0.0f;
    bin_peaks(e, len, m, meta + s, pcr[s], off[s], mz, it, lp);
    // normaliseByRegion, Correlation.hs:84-96
    const int32_t sel = (len - 75) / 10;
    for (int32_t i = tid; i < len; i += blockDim.x) {
        const int32_t g = min(10, i / sel);
        const float v = e[i];
        if (v > 0.0f) atomicMax((int *)&rmax[g], __float_as_int(v));
    }
    __syncthreads();
    for (int32_t i = tid; i < len; i += blockDim.x) {
        const int32_t g = min(10, i / sel);
        const float mx = rmax[g];
        e[i] = (mx > 1e-6f && i < sel * 10) ? __fmul_rn(50.0f, __fdiv_rn(e[i], mx)) : 0.0f;
    }
    __syncthreads();
    // crossCorrolation, Correlation.hs:105-109
    for (int32_t i = tid; i < len; i += blockDim.x) {
        const int32_t lo = max(0, i - 75);
        const int32_t hi = min(len, lo + 151);
        float acc = 0.0f;
        for (int32_t j = lo; j < hi; ++j) acc = __fadd_rn(acc, e[j]);
        const float x = __fsub_rn(e[i], __fdiv_rn(acc, 150.0f));
        o32[i] = x;
        if (obf) obf[i] = __float2bfloat16_rn(x);
        if (oh) oh[i] = __float2half_rn(x);
    }
}

// ---- long rows (e.g. 0.02 Da bins, ~10^5 bins): the same row, computed sparsely ----
//
// A row that does not fit in shared memory is built from its nonzero bins
// only.  The binned values are the kept peaks' sqrt intensities, max per bin
// (sort the (bin, value) keys, keep the last of each bin); normalisation
// touches only those bins; and x[i] is nonzero only where the 151-bin window
// of i holds a nonzero bin or e[i] != 0.  Every e is >= 0, so the reference's
// left fold over the window equals the left fold over the window's nonzero
// bins (adding +0 is exact and the sum never is -0): the row is bit-identical
// to the dense computation.
constexpr int kSparsePeaks = 4096;
// Peaks of the kernel's small form: its 10 KB of shared memory let eight CTAs
// share an SM, the 80 KB for 4,096 peaks two, and a CTA's sort is a chain of
// barriers.  10,000 spectra of 225 peaks, 10^5-bin FP32 and BF16 rows: 4.5 ms in
// the large form, 3.2 ms in the small one.
constexpr int kSparseFew = 512;
constexpr size_t kDenseRowBytes = 200 * 1024;  // rows up to 51,200 bins are built densely in shared memory

// Spectra of up to kSparseFew peaks, or of more.
template <int kPeaks>
__global__ void __launch_bounds__(256) k_preprocess_sparse(const float *__restrict__ mz, const float *__restrict__ it,
                                                           const int64_t *__restrict__ off,
                                                           const float *__restrict__ pcr, LayoutParams lp,
                                                           const SpecMeta *__restrict__ meta, int64_t stride,
                                                           float *__restrict__ out32,
                                                           __nv_bfloat16 *__restrict__ outbf,
                                                           __half *__restrict__ outh, uint32_t *__restrict__ err) {
    extern __shared__ __align__(16) uint8_t sm_sparse[];
    unsigned long long *keys = reinterpret_cast<unsigned long long *>(sm_sparse);  // [kPeaks]
    int32_t *nzk = reinterpret_cast<int32_t *>(keys + kPeaks);                     // [kPeaks]
    float *nze = reinterpret_cast<float *>(nzk + kPeaks);                          // [kPeaks]
    int32_t *ivs = reinterpret_cast<int32_t *>(nze + kPeaks);                      // [kPeaks + 1]
    __shared__ int32_t warp_tot[32];
    __shared__ float rmax[11];
    const int32_t s = blockIdx.x;
    const SpecMeta m = meta[s];
    if (kPeaks < kSparsePeaks ? m.npk > kPeaks : m.npk <= kSparseFew) return;  // the other form's
    const int tid = threadIdx.x, nt = blockDim.x;
    float *o32 = out32 + (int64_t)s * stride;
    __nv_bfloat16 *obf = outbf ? outbf + (int64_t)s * stride : nullptr;
    __half *oh = outh ? outh + (int64_t)s * stride : nullptr;
    // zero rows (stride is a multiple of 16 elements, rows 16-byte aligned)
    for (int64_t i = (int64_t)tid * 4; i < stride; i += (int64_t)nt * 4)
        *reinterpret_cast<float4 *>(o32 + i) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int64_t i = (int64_t)tid * 8; i < stride; i += (int64_t)nt * 8) {
        if (obf) *reinterpret_cast<uint4 *>(obf + i) = make_uint4(0u, 0u, 0u, 0u);
        if (oh) *reinterpret_cast<uint4 *>(oh + i) = make_uint4(0u, 0u, 0u, 0u);
    }
    if (m.status != 0) return;
    if (m.npk > kPeaks) {
        if (tid == 0) atomicOr(err, kErrTooLong);
        return;
    }
    const int32_t len = m.len;
    // observedIntensity, Correlation.hs:58-71: (bin, sqrt intensity) keys
    const float ps = pcr[s];
    const float plo = __fsub_rn(ps, 15.0f), phi = __fadd_rn(ps, 15.0f);
    const int64_t o0 = off[s];
    int32_t n2 = 1;
    while (n2 < m.npk) n2 <<= 1;
    for (int32_t i = tid; i < n2; i += nt) {
        unsigned long long k = ~0ull;
        if (i < m.npk) {
            const float x = mz[o0 + i];
            const bool keep = lp.remove_pcr ? (x <= m.cutoff && (x <= plo || phi <= x)) : (x <= m.cutoff);
            if (keep) {
                const float q = rintf(__fdiv_rn(x, lp.bw));
                const float v = __fsqrt_rn(it[o0 + i]);
                if (q >= 0.0f && q < (float)len && v >= 0.0f)
                    k = ((unsigned long long)(uint32_t)(int32_t)q << 32) | __float_as_uint(v);
            }
        }
        keys[i] = k;
    }
    if (tid < 11) rmax[tid] = 0.0f;
    __syncthreads();
    // bitonic sort, ascending (bin, then value: non-negative floats order as their bits)
    for (int32_t kk = 2; kk <= n2; kk <<= 1) {
        for (int32_t j = kk >> 1; j > 0; j >>= 1) {
            for (int32_t i = tid; i < n2; i += nt) {
                const int32_t l = i ^ j;
                if (l > i) {
                    const unsigned long long a = keys[i], b = keys[l];
                    const bool up = (i & kk) == 0;
                    if ((a > b) == up) {
                        keys[i] = b;
                        keys[l] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
    // the last key of each bin carries the bin's max; compact them in order
    int32_t nnz = 0;
    for (int32_t base = 0; base < n2; base += nt) {
        const int32_t i = base + tid;
        const unsigned long long k = i < n2 ? keys[i] : ~0ull;
        const bool last = k != ~0ull && (i + 1 >= n2 || (keys[i + 1] >> 32) != (k >> 32));
        int32_t tot = 0;
        const int32_t at = nnz + block_excl_scan(last ? 1 : 0, warp_tot, tot);
        if (last) {
            nzk[at] = (int32_t)(k >> 32);
            nze[at] = __uint_as_float((uint32_t)k);
        }
        nnz += tot;
    }
    __syncthreads();
    // normaliseByRegion, Correlation.hs:84-96
    const int32_t sel = (len - 75) / 10;
    for (int32_t j = tid; j < nnz; j += nt) {
        const float v = nze[j];
        if (v > 0.0f) atomicMax((int *)&rmax[min(10, nzk[j] / sel)], __float_as_int(v));
    }
    __syncthreads();
    for (int32_t j = tid; j < nnz; j += nt) {
        const int32_t k = nzk[j];
        const float mx = rmax[min(10, k / sel)];
        nze[j] = (mx > 1e-6f && k < sel * 10) ? __fmul_rn(50.0f, __fdiv_rn(nze[j], mx)) : 0.0f;
    }
    // positions whose window holds a nonzero bin: [0, 75), and per nonzero
    // bin k the positions i >= 75 with |i - k| <= 75, minus the previous
    // bin's (bins ascending, so the pieces are disjoint)
    const int32_t head = min(75, len);
    int32_t tot = 0;
    for (int32_t base = 0; base < nnz; base += nt) {
        const int32_t j = base + tid;
        int32_t c = 0;
        if (j < nnz) {
            const int32_t k = nzk[j];
            int32_t a = max(head, k - 75);
            if (j > 0) a = max(a, nzk[j - 1] + 76);
            const int32_t b = min(len, k + 76);
            c = max(0, b - a);
        }
        int32_t t = 0;
        const int32_t at = tot + block_excl_scan(c, warp_tot, t);
        if (j < nnz) ivs[j] = at;
        tot += t;
    }
    if (tid == 0) ivs[nnz] = tot;
    __syncthreads();
    // crossCorrolation, Correlation.hs:105-109, at those positions only
    for (int32_t u = tid; u < head + tot; u += nt) {
        int32_t i, first = 0;  // first: a nonzero bin that the window holds, or 0
        if (u < head) {
            i = u;
        } else {
            const int32_t v = u - head;
            int32_t lo = 0, hi = nnz;  // last j with ivs[j] <= v
            while (hi - lo > 1) {
                const int32_t mid = (lo + hi) >> 1;
                if (ivs[mid] <= v) lo = mid; else hi = mid;
            }
            const int32_t k = nzk[lo];
            int32_t a = max(head, k - 75);
            if (lo > 0) a = max(a, nzk[lo - 1] + 76);
            i = a + (v - ivs[lo]);
            first = lo;  // i <= nzk[lo] + 75
        }
        const int32_t wlo = max(0, i - 75);
        const int32_t whi = min(len, wlo + 151);
        while (first > 0 && nzk[first - 1] >= wlo) --first;  // the first nonzero bin >= wlo
        float acc = 0.0f, ei = 0.0f;
        for (int32_t j = first; j < nnz && nzk[j] < whi; ++j) {
            acc = __fadd_rn(acc, nze[j]);
            if (nzk[j] == i) ei = nze[j];
        }
        const float x = __fsub_rn(ei, __fdiv_rn(acc, 150.0f));
        o32[i] = x;
        if (obf) obf[i] = __float2bfloat16_rn(x);
        if (oh) oh[i] = __float2half_rn(x);
    }
}

}  // namespace hfx

using namespace hfx;

int hfx_launch_layout(const float *mz, const int64_t *off, const float *pcr, const float *z,
                      const float *tol, int32_t nspec, const LayoutParams &lp, SpecMeta *meta,
                      uint32_t *max_len, uint32_t *err, cudaStream_t st, int32_t *lens, float *masses) {
    if (nspec <= 0) return 0;
    k_layout<<<(nspec + 127) / 128, 128, 0, st>>>(mz, off, pcr, z, tol, nspec, lp, meta, max_len, err, lens,
                                                   masses);
    return (int)cudaGetLastError();
}

int hfx_launch_preprocess(const float *mz, const float *it, const int64_t *off, const float *pcr,
                          const LayoutParams &lp, SpecMeta *meta, int32_t nspec, int64_t stride,
                          float *out32, __nv_bfloat16 *outbf, __half *outh, uint32_t *err, cudaStream_t st) {
    if (nspec <= 0) return 0;
    size_t smem = (((size_t)stride + 3) & ~(size_t)3) * sizeof(float);
    if (smem > kDenseRowBytes) {
        // long rows: the sparse form (needs the error word for its peak limit)
        if (!err) return (int)cudaErrorInvalidValue;
        auto run = [&](auto f, int peaks) {
            const size_t sm = (size_t)peaks * (8 + 4 + 4 + 4) + 16;
            cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
            f<<<nspec, 256, sm, st>>>(mz, it, off, pcr, lp, meta, stride, out32, outbf, outh, err);
        };
        run(k_preprocess_sparse<kSparseFew>, kSparseFew);
        run(k_preprocess_sparse<kSparsePeaks>, kSparsePeaks);
        return (int)cudaGetLastError();
    }
    // the row, its nonzero bins and their window sums when they fit (up to 17,066
    // bins); otherwise every window folds all its bins
    const bool list = (size_t)stride * 8 + ((size_t)stride + 1) * 4 <= kDenseRowBytes;
    auto fn = list ? k_preprocess : k_preprocess_bins;
    if (list) smem = (2 * (size_t)stride + 1) * 4;
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDenseRowBytes);
    fn<<<nspec, 256, smem, st>>>(mz, it, off, pcr, lp, meta, stride, out32, outbf, outh);
    return (int)cudaGetLastError();
}
