// reduce.cu -- global min/max, the 256-bin histogram, device Otsu, and the
// element-wise ops of the path (greater_constant, binary_and, mask).
#include <cfloat>

#include "common.cuh"
#include "kernels.cuh"

namespace cle {

namespace {

constexpr int kRedThreads = 512;

template <typename T>
__device__ __forceinline__ void minmax_acc(T v, float &a, float &b) {
    float f = to_f32(v);
    a = fminf(a, f);
    b = fmaxf(b, f);
}

template <typename T>
__global__ void __launch_bounds__(kRedThreads)
minmax_partial_kernel(const T *__restrict__ src, int64_t n, float *__restrict__ partial) {
    float a = INFINITY, b = -INFINITY;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if constexpr (sizeof(T) == 4) {
        // 128-bit loads over the aligned body
        const int64_t n4 = ((reinterpret_cast<uintptr_t>(src) & 15) == 0) ? n / 4 : 0;
        const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
        for (int64_t j = i; j < n4; j += stride) {
            uint4 u = __ldcs(s4 + j);
            T v[4];
            memcpy(v, &u, 16);
#pragma unroll
            for (int k = 0; k < 4; ++k) minmax_acc(v[k], a, b);
        }
        for (int64_t j = n4 * 4 + i; j < n; j += stride) minmax_acc(src[j], a, b);
    } else {
        for (int64_t j = i; j < n; j += stride) minmax_acc(src[j], a, b);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = fminf(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    __shared__ float sa[32], sb[32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { sa[w] = a; sb[w] = b; }
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        a = l < nw ? sa[l] : INFINITY;
        b = l < nw ? sb[l] : -INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a = fminf(a, __shfl_xor_sync(0xffffffffu, a, o));
            b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
        }
        if (l == 0) {
            partial[2 * blockIdx.x] = a;
            partial[2 * blockIdx.x + 1] = b;
        }
    }
}

__global__ void minmax_final_kernel(const float *__restrict__ partial, int blocks,
                                    float *__restrict__ out) {
    float a = INFINITY, b = -INFINITY;
    for (int i = threadIdx.x; i < blocks; i += blockDim.x) {
        a = fminf(a, partial[2 * i]);
        b = fmaxf(b, partial[2 * i + 1]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = fminf(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    __shared__ float sa[32], sb[32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { sa[w] = a; sb[w] = b; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
            a = fminf(a, sa[k]);
            b = fmaxf(b, sb[k]);
        }
        out[0] = a;
        out[1] = b;
    }
}

int minmax_blocks(int64_t n) { return launch_blocks(n / 4 + 1, kRedThreads, 4); }

// ---------------------------------------------------------------------------
// Histogram (A6): bin = convert_uint_sat(((v - min) * (bins-1)) / range + 0.5f)
// in float32, per-y-row exact integer partials, then a float32 running sum
// over rows in order (_tier3/_histogram.py:97-128).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cvt_uint_sat_f(float t) {
    if (!(t > 0.0f)) return 0u;
    if (t >= 4294967296.0f) return 0xFFFFFFFFu;
    return (uint32_t)t;
}

__device__ __forceinline__ int hist_bin(float v, float mn, float range, float bm1, int bins) {
    const float a = __fmul_rn(__fsub_rn(v, mn), bm1);
    if (range == 0.0f) return a > 0.0f ? -1 : 0;   // +inf is past the last bin, NaN and -inf are 0
    float t = __fdiv_rn(a, range);
    uint32_t b = cvt_uint_sat_f(__fadd_rn(t, 0.5f));
    return b < (uint32_t)bins ? (int)b : -1;
}

// Up to 256 bins take the bin from q = (v - min) * (bins-1) * (1/range) + 0.5, two
// voxels to a packed operation.  The product is within 1.5 ulp of the IEEE
// quotient and the addition rounds once more on each side, together under 2^-13
// for q < 256: wherever q lies at least 2^-12 from an integer both have the same
// bin.  Adding 2^23 rounded down leaves floor(q) in the low bits, so neither a
// conversion nor a rounding instruction (a quarter of the rate) is needed.
// Everything else (near a bin edge, out of range, NaN, inf, an empty range: 1 in
// 2000 of a smooth image's voxels) is divided exactly.
//
// Each voxel is one shared-memory add of 1 to its warp's copy of the bins, which
// the hardware counts for all lanes on one bin at once: no vote, no branch.
// 512 x 1024 x 1024 float32, smooth: 0.54 ms; with runs of equal bins merged by
// branches and votes 0.87 ms (47 instructions per voxel and lane, issue bound).
// 61 x 479 x 347 (no 128-bit loads, a vote per voxel before): 35 -> 25 us.
constexpr int kHistThreads = 256;
constexpr int kHistPer = 8;   // voxels per thread and round, all loaded first

template <typename T>
__global__ void __launch_bounds__(kHistThreads)
hist_rows_kernel(const T *__restrict__ src, int64_t D, int64_t H, int64_t W, int bins,
                 int zchunk, const float *__restrict__ d_minmax, uint32_t *__restrict__ part,
                 FastDiv fw, FastDiv fw4, uint32_t *__restrict__ done) {
    extern __shared__ uint32_t sh[];   // (warps x bins) when private, else bins
    const int nwarps = kHistThreads / 32;
    const bool priv = bins <= 512;
    const int ncopies = priv ? nwarps : 1;
    for (int i = threadIdx.x; i < ncopies * bins; i += kHistThreads) sh[i] = 0;
    __syncthreads();
    const float mn = d_minmax[0];
    const float range = __fsub_rn(d_minmax[1], mn);
    const float bm1 = (float)(bins - 1);
    const float rr = __frcp_rn(range);
    const int64_t y = blockIdx.x;
    const int64_t z0 = (int64_t)blockIdx.y * zchunk;
    const int64_t z1 = min(D, z0 + zchunk);
    uint32_t *mine = sh + (priv ? (threadIdx.x >> 5) * bins : 0);
    const float2 nmn = make_float2(-mn, -mn), s2 = make_float2(bm1, bm1);
    const float2 r2 = make_float2(rr, rr), h2 = make_float2(0.5f, 0.5f);
    const float2 up = make_float2(8388608.0f, 8388608.0f), dn = make_float2(-8388607.5f, -8388607.5f);

    // ok: bit k set where v[k] is a voxel
    auto bin_all = [&](const float (&v)[kHistPer], uint32_t ok) {
        uint32_t left = ok;   // voxels for the exact division
        if (bins <= 256) {
            left = 0;
#pragma unroll
            for (int k = 0; k < kHistPer; k += 2) {
                const float2 a = __fmul2_rn(__fadd2_rn(make_float2(v[k], v[k + 1]), nmn), s2);
                const float2 q = __fadd2_rn(__fmul2_rn(a, r2), h2);
                const float2 t = __fadd2_rd(q, up);   // 2^23 + floor(q)
                const float2 m = __fadd2_rn(t, dn);   // floor(q) + 0.5, exact
                const float2 d = __fadd2_rn(q, make_float2(-m.x, -m.y));
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const uint32_t b = __float_as_uint(e ? t.y : t.x) - 0x4B000000u;
                    if (ok >> (k + e) & 1u) {
                        if (fabsf(e ? d.y : d.x) <= 0.5f - 0.000244140625f && b < (uint32_t)bins) atomicAdd(&mine[b], 1u);
                        else left |= 1u << (k + e);
                    }
                }
            }
        }
        if (left) {
#pragma unroll
            for (int k = 0; k < kHistPer; ++k) {
                if (left >> k & 1u) {
                    const int b = hist_bin(v[k], mn, range, bm1, bins);
                    if (b >= 0) atomicAdd(&mine[b], 1u);
                }
            }
        }
    };

    bool wide = false;
    if constexpr (std::is_same<T, float>::value) {
        wide = (W & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
        if (wide) {
            // float rows of a multiple of 4 on a 16-byte boundary: 128-bit loads
            const uint32_t W4 = (uint32_t)(W >> 2);
            const uint32_t span4 = (uint32_t)((z1 - z0) * W4);
            for (uint32_t base = 0; base < span4; base += 2 * kHistThreads) {
                float v[kHistPer];
                uint32_t ok = 0;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint32_t j = base + k * kHistThreads + threadIdx.x;
                    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (j < span4) {
                        const uint32_t zz = fw4.div(j), x4 = j - zz * W4;
                        q = __ldg(reinterpret_cast<const float4 *>(src + ((z0 + zz) * H + y) * W) + x4);
                        ok |= 15u << 4 * k;
                    }
                    v[4 * k] = q.x; v[4 * k + 1] = q.y; v[4 * k + 2] = q.z; v[4 * k + 3] = q.w;
                }
                bin_all(v, ok);
            }
        }
    }
    if (!wide) {
        const uint32_t span = (uint32_t)((z1 - z0) * W);
        for (uint32_t base = 0; base < span; base += kHistPer * kHistThreads) {
            float v[kHistPer];
            uint32_t ok = 0;
#pragma unroll
            for (int k = 0; k < kHistPer; ++k) {
                const uint32_t j = base + k * kHistThreads + threadIdx.x;
                v[k] = 0.0f;
                if (j < span) {
                    const uint32_t zz = fw.div(j), xx = j - zz * (uint32_t)W;
                    v[k] = to_f32(src[((z0 + zz) * H + y) * W + xx]);
                    ok |= 1u << k;
                }
            }
            bin_all(v, ok);
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < bins; b += kHistThreads) {
        uint32_t c = 0;
        for (int k = 0; k < ncopies; ++k) c += sh[k * bins + b];
        // a row in one chunk is stored, the chunks of a row are added up
        if (gridDim.y == 1) part[y * bins + b] = c;
        else if (c) atomicAdd(&part[y * bins + b], c);
    }
    if (done && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *done = 0u;
}

// A7: scikit-image Otsu on the histogram, float64, no contraction, numpy's
// sequential cumsum, first-occurrence argmax with NaN as maximum
// (_tier9/_threshold_otsu.py:38-49, :83-106).  Only the four running sums are
// sequential (numpy's cumsum order): one lane of a warp each, from products
// formed before and values loaded 16 at a time, so that a step costs one
// addition; everything else runs in parallel.  A CTA of 256 threads or more
// calls it.  Row sums and Otsu of a 256 x 256 image take 8.4 us in one launch
// (19.4 in two, with two sums to a thread, product and loads inside the chain
// and a sequential argmax).
struct OtsuShared {
    double bc[256], c[256], p[256], w1[256], w2[256], s1[256], s2[256];
    double best[8];
    int at[8];
};

// out[i] = running sum of v in index order (or from the end backwards)
template <bool BACK>
__device__ __forceinline__ void running_sum(const double *v, double *out) {
    double acc = 0.0;
#pragma unroll 2
    for (int i0 = 0; i0 < 256; i0 += 16) {
        double x[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = v[BACK ? 255 - (i0 + k) : i0 + k];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            acc = __dadd_rn(acc, x[k]);
            out[BACK ? 255 - (i0 + k) : i0 + k] = acc;
        }
    }
}

// a beats b in numpy's argmax (b has the smaller index)
__device__ __forceinline__ bool beats(double a, double b) { return b == b && (a != a || a > b); }

__device__ __forceinline__ void otsu_block(OtsuShared &o, const volatile float *hist, const float *d_minmax, double *d_thr,
                                           float *d_thr32) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const float mn = d_minmax[0];
    const float range32 = __fsub_rn(d_minmax[1], mn);
    if (t < 256) {
        o.bc[t] = __dadd_rn(__ddiv_rn(__dmul_rn((double)t, (double)range32), 255.0), (double)mn);
        o.c[t] = (double)hist[t];
        o.p[t] = __dmul_rn(o.c[t], o.bc[t]);
    }
    __syncthreads();
    if (t == 0) running_sum<false>(o.p, o.s1);
    else if (t == 32) running_sum<true>(o.p, o.s2);
    else if (t == 64) running_sum<false>(o.c, o.w1);
    else if (t == 96) running_sum<true>(o.c, o.w2);
    __syncthreads();
    if (t < 256) {
        double v = -INFINITY;   // below every variance (they are squares times counts, or NaN)
        int at = t;
        if (t < 255) {
            const double m1 = __ddiv_rn(o.s1[t], o.w1[t]);
            const double m2 = __ddiv_rn(o.s2[t + 1], o.w2[t + 1]);
            const double d = __dsub_rn(m1, m2);
            v = __dmul_rn(__dmul_rn(o.w1[t], o.w2[t + 1]), __dmul_rn(d, d));
        }
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {   // the lower lane keeps ties: the first occurrence
            const double w = __shfl_down_sync(0xffffffffu, v, k);
            const int wa = __shfl_down_sync(0xffffffffu, at, k);
            if (beats(w, v)) { v = w; at = wa; }
        }
        if (lane == 0) { o.best[warp] = v; o.at[warp] = at; }
    }
    __syncthreads();
    if (t == 0) {
        int idx = o.at[0];
        double v = o.best[0];
        for (int k = 1; k < 8; ++k)
            if (beats(o.best[k], v)) { v = o.best[k]; idx = o.at[k]; }
        const double thr = o.bc[idx];
        if (d_thr) *d_thr = thr;
        if (d_thr32) *d_thr32 = __double2float_rn(thr);
    }
}

// hist[b] = float32 running sum of the row partials over y = 0..H-1 in order
// (the reference's sum_z_projection).  Partials and their running sums are
// integers, so while the running sum stays below 2^24 every float32 addition
// is exact and the result is the exact integer total.  Bins whose total
// reaches 2^24 (at most voxels / 2^24 of them) are summed in row order by one
// warp each; the others take their exact total.  A CTA owns 32 bins: warp w
// adds rows w, w + 32, ... of its lane's bin with 8 loads in flight, so the
// totals take a few memory round trips instead of one per row.
// With OTSU (256 bins) the last CTA to finish runs Otsu on the histogram; `done`
// counts the finished CTAs (0 at the start).
constexpr int kRowsumBins = 32;
template <bool OTSU>
__global__ void __launch_bounds__(1024)
hist_rowsum_kernel(const uint32_t *__restrict__ part, int64_t H, int bins, float *hist,
                   const float *__restrict__ d_minmax, double *__restrict__ d_thr, float *__restrict__ d_thr32,
                   uint32_t *__restrict__ done) {
    __shared__ unsigned long long s_tot[32][kRowsumBins + 1];
    __shared__ unsigned long long s_bin[kRowsumBins];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b = blockIdx.x * kRowsumBins + lane;
    unsigned long long acc = 0;
    if (b < bins) {
        int64_t y = warp;
        for (; y + 7 * 32 < H; y += 8 * 32) {
            uint32_t v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = part[(y + q * 32) * bins + b];
#pragma unroll
            for (int q = 0; q < 8; ++q) acc += v[q];
        }
        for (; y < H; y += 32) acc += part[y * bins + b];
    }
    s_tot[warp][lane] = acc;
    __syncthreads();
    if (warp == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < 32; ++w) t += s_tot[w][lane];
        s_bin[lane] = t;
        if (b < bins && t < (1ull << 24)) hist[b] = (float)t;
    }
    __syncthreads();
    // ordered float32 sums: warp j takes bin j of the CTA when its total is
    // at or above 2^24
    const int bb = blockIdx.x * kRowsumBins + warp;
    if (bb < bins && s_bin[warp] >= (1ull << 24)) {
        float acc32 = 0.0f;
        for (int64_t y0 = 0; y0 < H; y0 += 32) {
            const int64_t y = y0 + lane;
            const uint32_t v = (y < H) ? part[y * bins + bb] : 0u;
            const int n = (H - y0 < 32) ? (int)(H - y0) : 32;
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                const uint32_t x = __shfl_sync(0xffffffffu, v, k);
                if (k < n) acc32 = __fadd_rn(acc32, (float)x);
            }
        }
        if (lane == 0) hist[bb] = acc32;
    }
    if constexpr (OTSU) {
        __shared__ OtsuShared o;
        __shared__ uint32_t s_ticket;
        __threadfence();   // this CTA's bins before its ticket
        __syncthreads();
        if (threadIdx.x == 0) s_ticket = atomicAdd(done, 1u);
        __syncthreads();
        if (s_ticket + 1u != gridDim.x) return;
        __threadfence();   // every other CTA's bins after theirs
        otsu_block(o, hist, d_minmax, d_thr, d_thr32);
    }
}

template <typename Ts, typename Td>
__global__ void greater_kernel(const Ts *__restrict__ src, Td *__restrict__ dst, int64_t n,
                               float c, const float *__restrict__ d_c) {
    const float k = d_c ? *d_c : c;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = (Td)(to_f32(src[i]) > k ? 1 : 0);
}

template <typename Ta, typename Tb, typename Td>
__global__ void and_kernel(const Ta *__restrict__ a, const Tb *__restrict__ b, Td *__restrict__ d,
                           int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        d[i] = (Td)((a[i] != (Ta)0 && b[i] != (Tb)0) ? 1 : 0);
}

// clij_convert_*_sat (_tier0/preamble.cl:505-591)
template <typename Td> __device__ __forceinline__ Td sat_from_f(float v);
template <> __device__ __forceinline__ float sat_from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ uint32_t sat_from_f<uint32_t>(float v) {
    if (v > 4294967295.0f) return 0xFFFFFFFFu;
    if (!(v >= 0.0f)) return 0u;
    return (uint32_t)v;
}
template <> __device__ __forceinline__ uint8_t sat_from_f<uint8_t>(float v) {
    if (v > 255.0f) return 255;
    if (!(v >= 0.0f)) return 0;
    return (uint8_t)v;
}
template <> __device__ __forceinline__ uint16_t sat_from_f<uint16_t>(float v) {
    if (v > 65535.0f) return 65535;
    if (!(v >= 0.0f)) return 0;
    return (uint16_t)v;
}

template <typename Ts, typename Tm, typename Td>
__global__ void mask_kernel(const Ts *__restrict__ s, const Tm *__restrict__ m, Td *__restrict__ d,
                            int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        d[i] = sat_from_f<Td>(m[i] != (Tm)0 ? to_f32(s[i]) : 0.0f);
}

template <typename T>
__device__ __forceinline__ uint32_t label_of(T v) {
    if constexpr (std::is_floating_point<T>::value) return v > (T)0 ? (uint32_t)(int64_t)v : 0u;
    else return (uint32_t)v;
}

// Largest label: four 128-bit loads per thread in flight (4-byte labels on a
// 16-byte boundary), one atomic per CTA.  512 x 1024 x 1024 uint32: 0.54 ms with
// scalar loads and an atomic per warp.
constexpr int kMaxThreads = 512;
template <typename T>
__global__ void __launch_bounds__(kMaxThreads)
label_max_partial(const T *__restrict__ s, int64_t n, uint32_t *__restrict__ out) {
    uint32_t m = 0;
    const int64_t stride = (int64_t)gridDim.x * kMaxThreads, i0 = blockIdx.x * (int64_t)kMaxThreads + threadIdx.x;
    int64_t done = 0;
    if constexpr (sizeof(T) == 4) {
        if ((reinterpret_cast<uintptr_t>(s) & 15) == 0) {
            const int64_t n4 = n / 4;
            const uint4 *s4 = reinterpret_cast<const uint4 *>(s);
            for (int64_t j = i0; j < n4; j += 4 * stride) {
                uint4 u[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) u[k] = j + k * stride < n4 ? __ldcs(s4 + j + k * stride) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    T v[4];
                    memcpy(v, &u[k], 16);
                    m = max(max(m, max(label_of(v[0]), label_of(v[1]))), max(label_of(v[2]), label_of(v[3])));
                }
            }
            done = n4 * 4;
        }
    }
    for (int64_t i = done + i0; i < n; i += stride) m = max(m, label_of(s[i]));
    m = __reduce_max_sync(0xffffffffu, m);
    __shared__ uint32_t s_m[kMaxThreads / 32];
    if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = __reduce_max_sync(0xffffffffu, threadIdx.x < kMaxThreads / 32 ? s_m[threadIdx.x] : 0u);
        if (threadIdx.x == 0 && m) atomicMax(out, m);
    }
}

}  // namespace

// ---------------------------------------------------------------------------

size_t minmax_workspace_bytes(const Img &im) {
    Arena a(nullptr, 0);
    a.take<float>(2 * (size_t)minmax_blocks(im.n()));
    return a.off;
}

int minmax(const Img &im, float *d_out, Arena &ws, cudaStream_t st) {
    const int blocks = minmax_blocks(im.n());
    float *partial = ws.take<float>(2 * (size_t)blocks);
    if (!ws.ok()) { set_error("minimum_maximum: workspace too small"); return CLE_ERR_WORKSPACE; }
    switch (im.dtype) {
        case CLE_F32: minmax_partial_kernel<float><<<blocks, kRedThreads, 0, st>>>((const float *)im.data, im.n(), partial); break;
        case CLE_U16: minmax_partial_kernel<uint16_t><<<blocks, kRedThreads, 0, st>>>((const uint16_t *)im.data, im.n(), partial); break;
        case CLE_U8: minmax_partial_kernel<uint8_t><<<blocks, kRedThreads, 0, st>>>((const uint8_t *)im.data, im.n(), partial); break;
        case CLE_U32: minmax_partial_kernel<uint32_t><<<blocks, kRedThreads, 0, st>>>((const uint32_t *)im.data, im.n(), partial); break;
        default: set_error("minimum_maximum: unsupported dtype %d", im.dtype); return CLE_ERR_DTYPE;
    }
    minmax_final_kernel<<<1, 1024, 0, st>>>(partial, blocks, d_out);
    CLE_LAUNCH_CHECK_N("minmax", 2);
    return CLE_OK;
}

size_t histogram_workspace_bytes(const Img &im, int bins) {
    Arena a(nullptr, 0);
    a.take<uint32_t>((size_t)im.H * bins);
    a.take<uint32_t>(1);
    return a.off;
}

namespace {

struct OtsuOut {
    bool on = false;
    double *thr = nullptr;
    float *thr32 = nullptr;
};

int histogram_impl(const Img &im, int bins, const float *d_minmax, float *d_hist, const OtsuOut &o, Arena &ws,
                   cudaStream_t st) {
    if (bins < 1) { set_error("histogram: num_bins must be >= 1"); return CLE_ERR_ARG; }
    uint32_t *part = ws.take<uint32_t>((size_t)im.H * bins);
    uint32_t *done = ws.take<uint32_t>(1);
    if (!ws.ok()) { set_error("histogram: workspace too small"); return CLE_ERR_WORKSPACE; }
    int dev = 0;
    cudaGetDevice(&dev);
    const int64_t target = (int64_t)num_sms(dev) * 8;
    int64_t zchunks = (target + im.H - 1) / im.H;
    if (zchunks > im.D) zchunks = im.D;
    if (zchunks < 1) zchunks = 1;
    const int zchunk = (int)((im.D + zchunks - 1) / zchunks);
    zchunks = (im.D + zchunk - 1) / zchunk;
    if (im.H > 2147483647 || zchunks > 65535) { set_error("histogram: image too large"); return CLE_ERR_TOO_LARGE; }
    dim3 grid((unsigned)im.H, (unsigned)zchunks);
    const size_t smem = sizeof(uint32_t) * bins * (bins <= 512 ? kHistThreads / 32 : 1);
    if (smem > kMaxSmem) { set_error("histogram: too many bins (%d)", bins); return CLE_ERR_ARG; }
    if (zchunks > 1) CLE_CUDA(cudaMemsetAsync(part, 0, sizeof(uint32_t) * im.H * bins, st));
    const FastDiv fw((uint32_t)im.W), fw4((uint32_t)std::max<int64_t>(1, im.W / 4));
    switch (im.dtype) {
        case CLE_F32:
            CLE_TRY(allow_smem(hist_rows_kernel<float>, smem));
            hist_rows_kernel<float><<<grid, kHistThreads, smem, st>>>((const float *)im.data, im.D, im.H, im.W, bins, zchunk, d_minmax, part, fw, fw4, done);
            break;
        case CLE_U16:
            CLE_TRY(allow_smem(hist_rows_kernel<uint16_t>, smem));
            hist_rows_kernel<uint16_t><<<grid, kHistThreads, smem, st>>>((const uint16_t *)im.data, im.D, im.H, im.W, bins, zchunk, d_minmax, part, fw, fw4, done);
            break;
        case CLE_U8:
            CLE_TRY(allow_smem(hist_rows_kernel<uint8_t>, smem));
            hist_rows_kernel<uint8_t><<<grid, kHistThreads, smem, st>>>((const uint8_t *)im.data, im.D, im.H, im.W, bins, zchunk, d_minmax, part, fw, fw4, done);
            break;
        default: set_error("histogram: unsupported dtype %d", im.dtype); return CLE_ERR_DTYPE;
    }
    CLE_LAUNCH_CHECK("histogram rows");
    const int sums = (bins + kRowsumBins - 1) / kRowsumBins;
    if (o.on) hist_rowsum_kernel<true><<<sums, 1024, 0, st>>>(part, im.H, bins, d_hist, d_minmax, o.thr, o.thr32, done);
    else hist_rowsum_kernel<false><<<sums, 1024, 0, st>>>(part, im.H, bins, d_hist, nullptr, nullptr, nullptr, nullptr);
    CLE_LAUNCH_CHECK("histogram rowsum");
    return CLE_OK;
}

}  // namespace

int histogram(const Img &im, int bins, const float *d_minmax, float *d_hist, Arena &ws,
              cudaStream_t st) {
    return histogram_impl(im, bins, d_minmax, d_hist, OtsuOut(), ws, st);
}

int histogram_otsu(const Img &im, const float *d_minmax, float *d_hist, double *d_thr, float *d_thr32, Arena &ws,
                   cudaStream_t st) {
    OtsuOut o;
    o.on = true;
    o.thr = d_thr;
    o.thr32 = d_thr32;
    return histogram_impl(im, 256, d_minmax, d_hist, o, ws, st);
}

template <typename Ts>
static int greater_dst(const Img &src, const Img &dst, float c, const float *d_c, cudaStream_t st) {
    const int64_t n = src.n();
    const int blocks = launch_blocks(n, 256);
    switch (dst.dtype) {
        case CLE_U8: greater_kernel<Ts, uint8_t><<<blocks, 256, 0, st>>>((const Ts *)src.data, (uint8_t *)dst.data, n, c, d_c); break;
        case CLE_F32: greater_kernel<Ts, float><<<blocks, 256, 0, st>>>((const Ts *)src.data, (float *)dst.data, n, c, d_c); break;
        case CLE_U32: greater_kernel<Ts, uint32_t><<<blocks, 256, 0, st>>>((const Ts *)src.data, (uint32_t *)dst.data, n, c, d_c); break;
        default: set_error("greater_constant: unsupported destination dtype %d", dst.dtype); return CLE_ERR_DTYPE;
    }
    CLE_LAUNCH_CHECK("greater_constant");
    return CLE_OK;
}

int greater_constant(const Img &src, const Img &dst, float c, const float *d_c, cudaStream_t st) {
    CLE_TRY(same_shape(src, dst, "source", "destination"));
    switch (src.dtype) {
        case CLE_F32: return greater_dst<float>(src, dst, c, d_c, st);
        case CLE_U16: return greater_dst<uint16_t>(src, dst, c, d_c, st);
        case CLE_U8: return greater_dst<uint8_t>(src, dst, c, d_c, st);
        case CLE_U32: return greater_dst<uint32_t>(src, dst, c, d_c, st);
        default: set_error("greater_constant: unsupported source dtype %d", src.dtype); return CLE_ERR_DTYPE;
    }
}

template <typename Ta, typename Tb>
static int and_dst(const Img &a, const Img &b, const Img &d, cudaStream_t st) {
    const int64_t n = a.n();
    const int blocks = launch_blocks(n, 256);
    switch (d.dtype) {
        case CLE_U8: and_kernel<Ta, Tb, uint8_t><<<blocks, 256, 0, st>>>((const Ta *)a.data, (const Tb *)b.data, (uint8_t *)d.data, n); break;
        case CLE_F32: and_kernel<Ta, Tb, float><<<blocks, 256, 0, st>>>((const Ta *)a.data, (const Tb *)b.data, (float *)d.data, n); break;
        default: set_error("binary_and: unsupported destination dtype %d", d.dtype); return CLE_ERR_DTYPE;
    }
    CLE_LAUNCH_CHECK("binary_and");
    return CLE_OK;
}

template <typename Ta>
static int and_b(const Img &a, const Img &b, const Img &d, cudaStream_t st) {
    switch (b.dtype) {
        case CLE_U8: return and_dst<Ta, uint8_t>(a, b, d, st);
        case CLE_F32: return and_dst<Ta, float>(a, b, d, st);
        case CLE_U32: return and_dst<Ta, uint32_t>(a, b, d, st);
        default: set_error("binary_and: unsupported dtype %d", b.dtype); return CLE_ERR_DTYPE;
    }
}

int binary_and(const Img &a, const Img &b, const Img &d, cudaStream_t st) {
    CLE_TRY(same_shape(a, b, "operand1", "operand2"));
    CLE_TRY(same_shape(a, d, "operand1", "destination"));
    switch (a.dtype) {
        case CLE_U8: return and_b<uint8_t>(a, b, d, st);
        case CLE_F32: return and_b<float>(a, b, d, st);
        case CLE_U32: return and_b<uint32_t>(a, b, d, st);
        default: set_error("binary_and: unsupported dtype %d", a.dtype); return CLE_ERR_DTYPE;
    }
}

template <typename Ts, typename Tm>
static int mask_dst(const Img &s, const Img &m, const Img &d, cudaStream_t st) {
    const int64_t n = s.n();
    const int blocks = launch_blocks(n, 256);
    switch (d.dtype) {
        case CLE_F32: mask_kernel<Ts, Tm, float><<<blocks, 256, 0, st>>>((const Ts *)s.data, (const Tm *)m.data, (float *)d.data, n); break;
        case CLE_U32: mask_kernel<Ts, Tm, uint32_t><<<blocks, 256, 0, st>>>((const Ts *)s.data, (const Tm *)m.data, (uint32_t *)d.data, n); break;
        case CLE_U8: mask_kernel<Ts, Tm, uint8_t><<<blocks, 256, 0, st>>>((const Ts *)s.data, (const Tm *)m.data, (uint8_t *)d.data, n); break;
        case CLE_U16: mask_kernel<Ts, Tm, uint16_t><<<blocks, 256, 0, st>>>((const Ts *)s.data, (const Tm *)m.data, (uint16_t *)d.data, n); break;
        default: set_error("mask: unsupported destination dtype %d", d.dtype); return CLE_ERR_DTYPE;
    }
    CLE_LAUNCH_CHECK("mask");
    return CLE_OK;
}

template <typename Ts>
static int mask_m(const Img &s, const Img &m, const Img &d, cudaStream_t st) {
    switch (m.dtype) {
        case CLE_U8: return mask_dst<Ts, uint8_t>(s, m, d, st);
        case CLE_F32: return mask_dst<Ts, float>(s, m, d, st);
        case CLE_U32: return mask_dst<Ts, uint32_t>(s, m, d, st);
        default: set_error("mask: unsupported mask dtype %d", m.dtype); return CLE_ERR_DTYPE;
    }
}

int mask_op(const Img &s, const Img &m, const Img &d, cudaStream_t st) {
    CLE_TRY(same_shape(s, m, "source", "mask"));
    CLE_TRY(same_shape(s, d, "source", "destination"));
    switch (s.dtype) {
        case CLE_F32: return mask_m<float>(s, m, d, st);
        case CLE_U32: return mask_m<uint32_t>(s, m, d, st);
        case CLE_U8: return mask_m<uint8_t>(s, m, d, st);
        case CLE_U16: return mask_m<uint16_t>(s, m, d, st);
        default: set_error("mask: unsupported source dtype %d", s.dtype); return CLE_ERR_DTYPE;
    }
}

size_t label_max_workspace_bytes(const Img &) { return 0; }

int label_max(const Img &labels, uint32_t *d_max, Arena &, cudaStream_t st) {
    CLE_CUDA(cudaMemsetAsync(d_max, 0, sizeof(uint32_t), st));
    const int64_t n = labels.n();
    const int blocks = launch_blocks(n / 4 + 1, kMaxThreads, 4);
    switch (labels.dtype) {
        case CLE_U32: label_max_partial<uint32_t><<<blocks, kMaxThreads, 0, st>>>((const uint32_t *)labels.data, n, d_max); break;
        case CLE_F32: label_max_partial<float><<<blocks, kMaxThreads, 0, st>>>((const float *)labels.data, n, d_max); break;
        case CLE_U16: label_max_partial<uint16_t><<<blocks, kMaxThreads, 0, st>>>((const uint16_t *)labels.data, n, d_max); break;
        case CLE_U8: label_max_partial<uint8_t><<<blocks, kMaxThreads, 0, st>>>((const uint8_t *)labels.data, n, d_max); break;
        default: set_error("label_maximum: unsupported dtype %d", labels.dtype); return CLE_ERR_DTYPE;
    }
    CLE_LAUNCH_CHECK("label_maximum");
    return CLE_OK;
}

}  // namespace cle
