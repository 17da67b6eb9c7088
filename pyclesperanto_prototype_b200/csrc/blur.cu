// blur.cu -- separable Gaussian blur (and the uniform-weight box mean used by
// detect_maxima_box with radius > 0).
//
// Semantics (_tier1/_gaussian_blur.py:39-56, _tier1/_execute_separable_kernel.py:7-76):
// passes along x, then y, then z (3D only), each with clamp-to-edge reads and
// float32 intermediates; a pass with sigma <= 0 is a copy.  Inside a pass
// the output is acc = fma(w_i, v_i, acc) for i = -r..r ascending from 0.
//
// Each thread makes 8 consecutive outputs along the pass axis of two lines at
// once (two rows in the x pass, two adjacent columns in the y and z passes), the
// two lines packed (fma.rn.f32x2: two independent round-to-nearest FMAs, the
// rounding of fmaf).  Lines are staged in shared memory as float32; a block of
// 8 taps takes the 8 values of the window already held and the next 8, so 64
// packed FMAs share 8 packed loads.  Taps lie in shared memory as pairs
// (w, w).  Nothing is padded with zero taps: 0 x infinity would be NaN.
// What bounds it: the FMA pipe (sigma 10, 64 x 1024 x 1024: 81 taps x 3 are 0.44 ms
// at 128 FMAs per SM and cycle, three reads and writes 0.25 ms); measured
// 0.85 ms (2.02 with one output per thread and a shared load per FMA), the pipe
// 60% busy, the rest in staging and at the one barrier of each CTA.  Staging
// with all of a thread's loads in flight at once (asynchronous 16-byte copies
// in the y and z passes, batches of 128-bit loads in x) took it from 1.07 ms.
#include "common.cuh"
#include "kernels.cuh"

namespace cle {

namespace {

constexpr int kK = 8;             // outputs per thread along the pass axis, taps per block
constexpr int kSepThreads = 256;
constexpr int kRowMax = 256;      // x pass: most outputs of a row per CTA
constexpr int kBlk = kK + 2;      // x pass: pitch of 8 staged pairs (16-byte lanes on odd granules)

// acc[k] += w * win[k + t] for the 8 outputs; win = lo (8 values) then hi
__device__ __forceinline__ void add_tap(float2 w, int t, const float2 (&lo)[kK], const float2 (&hi)[kK],
                                        float2 (&acc)[kK]) {
#pragma unroll
    for (int k = 0; k < kK; ++k) acc[k] = __ffma2_rn(w, k + t < kK ? lo[(k + t) % kK] : hi[(k + t) % kK], acc[k]);
}

// The taps' chain over a staged line: block(j) loads the window's 8 packed
// values 8j .. 8j + 7 of the thread (values past the last tap's are loaded but
// not used).
template <typename Block>
__device__ __forceinline__ void tap_chain(const float2 *sw, int n, float2 (&acc)[kK], Block block) {
    float2 a[kK], b[kK];
    block(0, a);
    int i = 0;
    // two blocks of taps per round, the window's halves changing places
    for (; i + 2 * kK <= n; i += 2 * kK) {
        block(i / kK + 1, b);
#pragma unroll
        for (int t = 0; t < kK; ++t) add_tap(sw[i + t], t, a, b, acc);
        block(i / kK + 2, a);
#pragma unroll
        for (int t = 0; t < kK; ++t) add_tap(sw[i + kK + t], t, b, a, acc);
    }
    if (i + kK <= n) {
        block(i / kK + 1, b);
#pragma unroll
        for (int t = 0; t < kK; ++t) add_tap(sw[i + t], t, a, b, acc);
        i += kK;
#pragma unroll
        for (int t = 0; t < kK; ++t) a[t] = b[t];
    }
    if (i < n) {
        block(i / kK + 1, b);
#pragma unroll
        for (int t = 0; t < kK - 1; ++t)
            if (i + t < n) add_tap(sw[i + t], t, a, b, acc);
    }
}

__host__ __device__ constexpr int tap_slots(int n) { return (n + 1) & ~1; }   // float2 slots of the taps, 16-byte multiple
// 8-value blocks of a line that tap_chain may load for `out` outputs
__host__ __device__ constexpr int line_blocks(int out, int n) { return out / kK + n / kK + 1; }

// four consecutive aligned source values as float32
__device__ __forceinline__ void load4(const float *p, float (&v)[4]) {
    const float4 f = __ldg(reinterpret_cast<const float4 *>(p));
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
}
__device__ __forceinline__ void load4(const uint16_t *p, float (&v)[4]) {
    const uint2 u = __ldg(reinterpret_cast<const uint2 *>(p));
    v[0] = (float)(u.x & 0xFFFFu); v[1] = (float)(u.x >> 16);
    v[2] = (float)(u.y & 0xFFFFu); v[3] = (float)(u.y >> 16);
}
__device__ __forceinline__ void load4(const uint8_t *p, float (&v)[4]) {
    const uint32_t u = __ldg(reinterpret_cast<const uint32_t *>(p));
    v[0] = (float)(u & 0xFFu); v[1] = (float)((u >> 8) & 0xFFu);
    v[2] = (float)((u >> 16) & 0xFFu); v[3] = (float)(u >> 24);
}

__device__ __forceinline__ void copy_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// x pass: a CTA takes np row pairs and an x tile of `tile` outputs (a
// multiple of 8) of each.
template <typename Tin>
__global__ void __launch_bounds__(kSepThreads)
blur_row_kernel(const Tin *__restrict__ src, float *__restrict__ dst, int64_t rows, int W, int tile, int np,
                FastDiv fc, int vec, const __grid_constant__ Taps taps) {
    extern __shared__ __align__(16) float2 sm[];
    const int n = taps.n, r = (n - 1) / 2;
    float2 *sw = sm, *line = sm + tap_slots(n);
    const int pitch = kBlk * line_blocks(tile, n);
    const int x0 = blockIdx.x * tile;
    const int64_t row0 = ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * (2 * np);
    if (row0 >= rows) return;
    for (int i = threadIdx.x; i < n; i += kSepThreads) sw[i] = make_float2(taps.w[i], taps.w[i]);
    // staging, a warp per row pair: column c of the line is x = x0 - r + c
    const int span = tile + 2 * r, lane = threadIdx.x & 31;
    auto put = [&](float2 *ln, int c, float2 v) { ln[c + 2 * (c / kK)] = v; };
    for (int q = threadIdx.x >> 5; q < np; q += kSepThreads / 32) {
        const Tin *ra = src + min(row0 + 2 * q, rows - 1) * W, *rb = src + min(row0 + 2 * q + 1, rows - 1) * W;
        float2 *ln = line + q * pitch;
        if (vec) {
            // 4 columns per lane from aligned groups (W and x0 are multiples of 4)
            const int xa = x0 - ((r + 3) & ~3), d = x0 - r - xa;
            for (int c0 = 4 * lane; c0 < span + d; c0 += 3 * 128) {
                float va[3][4], vb[3][4];
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    const int c = c0 + 128 * u, x = xa + c;
                    if (c < span + d) {
                        if (x >= 0 && x + 4 <= W) {
                            load4(ra + x, va[u]);
                            load4(rb + x, vb[u]);
                        } else {
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                va[u][k] = to_f32(ra[clampi(x + k, 0, W - 1)]);
                                vb[u][k] = to_f32(rb[clampi(x + k, 0, W - 1)]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < 3; ++u)
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int c = c0 + 128 * u + k - d;
                        if (c >= 0 && c < span) put(ln, c, make_float2(va[u][k], vb[u][k]));
                    }
            }
        } else {
#pragma unroll 4
            for (int c = lane; c < span; c += 32) {
                const int x = clampi(x0 - r + c, 0, W - 1);
                put(ln, c, make_float2(to_f32(ra[x]), to_f32(rb[x])));
            }
        }
    }
    __syncthreads();
    const int per = tile / kK;   // items per row pair
    for (int e = threadIdx.x; e < np * per; e += kSepThreads) {
        const int q = (int)fc.div((uint32_t)e), c = e - q * per;
        const int64_t ra = row0 + 2 * q;
        const int x = x0 + c * kK;
        if (ra >= rows || x >= W) continue;
        const float2 *base = line + q * pitch + c * kBlk;
        float2 acc[kK];
#pragma unroll
        for (int k = 0; k < kK; ++k) acc[k] = make_float2(0.f, 0.f);
        tap_chain(sw, n, acc, [&](int j, float2 (&v)[kK]) {
            const float4 *p = reinterpret_cast<const float4 *>(base + j * kBlk);
#pragma unroll
            for (int k = 0; k < kK / 2; ++k) {
                const float4 f = p[k];
                v[2 * k] = make_float2(f.x, f.y);
                v[2 * k + 1] = make_float2(f.z, f.w);
            }
        });
        float *o = dst + ra * W + x;
        const bool two = ra + 1 < rows;
        if ((W & 3) == 0 && x + kK <= W && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
            for (int k = 0; k < kK; k += 4) {
                *reinterpret_cast<float4 *>(o + k) = make_float4(acc[k].x, acc[k + 1].x, acc[k + 2].x, acc[k + 3].x);
                if (two) *reinterpret_cast<float4 *>(o + W + k) = make_float4(acc[k].y, acc[k + 1].y, acc[k + 2].y, acc[k + 3].y);
            }
        } else {
#pragma unroll
            for (int k = 0; k < kK; ++k)
                if (x + k < W) {
                    o[k] = acc[k].x;
                    if (two) o[W + k] = acc[k].y;
                }
        }
    }
}

// Pass along an axis of length L with element stride `inner`, for a volume
// viewed as [outer][L][inner]: a CTA takes NG x 8 outputs along the axis and
// 2 x NC columns (NG x NC = 256 threads).  tile0: the launch's first tile of the
// axis; ctas: the CTAs of all launches of the pass; clear (optional): a word to
// set to 0 that neither src nor dst holds.
template <typename Tin, int NG>
__global__ void __launch_bounds__(kSepThreads)
blur_col_kernel(const Tin *__restrict__ src, float *__restrict__ dst, int64_t inner, int L, int tile0, int vec,
                const __grid_constant__ Taps taps, MinMaxState *__restrict__ mm, uint32_t ctas, int *clear) {
    constexpr int NC = kSepThreads / NG, COLS = 2 * NC, ROWS = NG * kK;
    extern __shared__ __align__(16) float2 sm[];
    const int n = taps.n, r = (n - 1) / 2;
    float2 *sw = sm;
    float *s = reinterpret_cast<float *>(sm + tap_slots(n));   // [8 * line_blocks][COLS]
    const int64_t c0 = (int64_t)blockIdx.x * COLS;
    const int l0 = (tile0 + (int)blockIdx.y) * ROWS;
    const int64_t base = (int64_t)blockIdx.z * L * inner;
    if (clear && threadIdx.x == 0 && (blockIdx.x | blockIdx.y | blockIdx.z) == 0u) *clear = 0;
    for (int i = threadIdx.x; i < n; i += kSepThreads) sw[i] = make_float2(taps.w[i], taps.w[i]);
    const int span = min(ROWS, L - l0) + 2 * r;
    if (vec) {
        // 4 columns per thread (inner a multiple of 4); most tiles need no clamp
        constexpr int QPR = COLS / 4, STEP = kSepThreads / QPR;
        const int c = 4 * (threadIdx.x % QPR), j0 = threadIdx.x / QPR;
        const Tin *p = src + base + min(c0 + c, inner - 4);
        const bool inside = l0 >= r && l0 - r + span <= L;
        if constexpr (sizeof(Tin) == 4) {
            // float32: asynchronous copies, all in flight at once
            const Tin *q = p + (int64_t)(inside ? l0 - r + j0 : 0) * inner;
            for (int j = j0; j < span; j += STEP, q += (int64_t)STEP * inner)
                copy_async16(s + j * COLS + c, inside ? q : p + (int64_t)clampi(l0 - r + j, 0, L - 1) * inner);
            asm volatile("cp.async.wait_all;" ::: "memory");
        } else {
            for (int j = j0; j < span; j += 4 * STEP) {
                float v[4][4];
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    if (j + b * STEP < span) load4(p + (int64_t)clampi(l0 - r + j + b * STEP, 0, L - 1) * inner, v[b]);
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    if (j + b * STEP < span)
                        *reinterpret_cast<float4 *>(s + (j + b * STEP) * COLS + c) = make_float4(v[b][0], v[b][1], v[b][2], v[b][3]);
            }
        }
    } else {
        constexpr int STEP = kSepThreads / COLS;
        const int c = threadIdx.x % COLS, j0 = threadIdx.x / COLS;
        const Tin *p = src + base + min(c0 + c, inner - 1);
#pragma unroll 8
        for (int j = j0; j < span; j += STEP) s[j * COLS + c] = to_f32(p[(int64_t)clampi(l0 - r + j, 0, L - 1) * inner]);
    }
    __syncthreads();
    const int cp = threadIdx.x % NC, g = threadIdx.x / NC;
    const int64_t c = c0 + 2 * cp;
    float vmin = INFINITY, vmax = -INFINITY;   // of the stored values (when mm)
    if (c < inner && l0 + g * kK < L) {
        const float *col = s + g * kK * COLS + 2 * cp;
        float2 acc[kK];
#pragma unroll
        for (int k = 0; k < kK; ++k) acc[k] = make_float2(0.f, 0.f);
        tap_chain(sw, n, acc, [&](int j, float2 (&v)[kK]) {
#pragma unroll
            for (int k = 0; k < kK; ++k) v[k] = *reinterpret_cast<const float2 *>(col + (j * kK + k) * COLS);
        });
        float *o = dst + base + (int64_t)(l0 + g * kK) * inner + c;
        const int left = L - (l0 + g * kK);
        const bool two = c + 1 < inner;
        const bool pair = (inner & 1) == 0 && (reinterpret_cast<uintptr_t>(dst) & 7) == 0;
#pragma unroll
        for (int k = 0; k < kK; ++k) {
            if (k < left) {
                float *q = o + (int64_t)k * inner;
                if (pair) *reinterpret_cast<float2 *>(q) = acc[k];
                else {
                    q[0] = acc[k].x;
                    if (two) q[1] = acc[k].y;
                }
                if (mm) {
                    vmin = fminf(vmin, acc[k].x);
                    vmax = fmaxf(vmax, acc[k].x);
                    if (two) { vmin = fminf(vmin, acc[k].y); vmax = fmaxf(vmax, acc[k].y); }
                }
            }
        }
    }
    if (mm) {
        __shared__ float s_mn[kSepThreads / 32], s_mx[kSepThreads / 32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            vmin = fminf(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
            vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
        }
        if ((threadIdx.x & 31) == 0) { s_mn[threadIdx.x >> 5] = vmin; s_mx[threadIdx.x >> 5] = vmax; }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < kSepThreads / 32; ++w) { vmin = fminf(vmin, s_mn[w]); vmax = fmaxf(vmax, s_mx[w]); }
            add_minmax(mm, vmin, vmax, ctas);
        }
    }
}

template <typename Tin>
__global__ void convert_kernel(const Tin *__restrict__ src, float *__restrict__ dst, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = to_f32(src[i]);
}

// Thread groups along the axis of a col pass: short axes take fewer outputs and
// more columns per CTA, as far as the staged lines of a long window fit shared
// memory.
int col_groups(int64_t L, int n) { return L <= 32 && n <= 129 ? 4 : L <= 64 && n <= 321 ? 8 : 16; }

template <typename Tin, int NG>
int launch_col(const Tin *src, float *dst, int64_t inner, int L, int64_t outer, const Taps &t, MinMaxState *mm,
               int *clear, cudaStream_t st) {
    constexpr int COLS = 2 * (kSepThreads / NG), ROWS = NG * kK;
    const int64_t cols = (inner + COLS - 1) / COLS, tiles = (L + ROWS - 1) / ROWS;
    const size_t smem = sizeof(float2) * tap_slots(t.n) + sizeof(float) * COLS * kK * line_blocks(ROWS, t.n);
    CLE_TRY(allow_smem(blur_col_kernel<Tin, NG>, smem, sizeof(float) * 2 * (kSepThreads / 32)));
    const int vec = inner % 4 == 0 && reinterpret_cast<uintptr_t>(src) % (4 * sizeof(Tin)) == 0;
    // a grid's second and third axes end at 65535, which the planes of a volume and
    // the tiles of a long axis can pass (one grid axis with divisions in the
    // kernel: 64 x 1024 x 1024, sigma 10, 896 against 888 us)
    constexpr int64_t kMost = 65535;
    for (int64_t o = 0; o < outer; o += kMost)
        for (int64_t tile0 = 0; tile0 < tiles; tile0 += kMost) {
            const dim3 grid((unsigned)cols, (unsigned)std::min(tiles - tile0, kMost), (unsigned)std::min(outer - o, kMost));
            blur_col_kernel<Tin, NG><<<grid, kSepThreads, smem, st>>>(src + o * L * inner, dst + o * L * inner, inner, L,
                                                                      (int)tile0, vec, t, mm, (uint32_t)(cols * tiles * outer), clear);
            CLE_LAUNCH_CHECK("blur pass");
        }
    return CLE_OK;
}

template <typename Tin>
int launch_pass(const Tin *src, float *dst, const Img &im, int axis, const Taps &t, MinMaxState *mm,
                int *clear, cudaStream_t st) {
    if (axis == 2) {
        // the row split evenly into tiles of at most kRowMax outputs
        const int64_t rows = im.D * im.H;
        const int tiles = (int)((im.W + kRowMax - 1) / kRowMax);
        const int tile = (int)(((im.W + tiles - 1) / tiles + kK - 1) / kK * kK);
        // row pairs to fill a CTA's threads, fewer where not even a quarter of the SMs
        // would have a CTA (256 x 256, 801 taps: a call of 83 us with 16 CTAs; two CTAs
        // for every SM cost a batch of tiles, which share the GPU, 2%)
        int dev = 0;
        CLE_CUDA(cudaGetDevice(&dev));
        const int64_t share = rows / 2 * tiles / std::max(1, num_sms(dev) / 4);
        const int np = (int)std::max<int64_t>(1, std::min<int64_t>(std::min(kSepThreads / (tile / kK), 16), share));
        const int64_t ctas = (rows + 2 * np - 1) / (2 * np);
        const dim3 grid((unsigned)((im.W + tile - 1) / tile), (unsigned)std::min<int64_t>(ctas, 65535),
                        (unsigned)((ctas + 65534) / 65535));
        const size_t smem = sizeof(float2) * (tap_slots(t.n) + (size_t)np * kBlk * line_blocks(tile, t.n));
        CLE_TRY(allow_smem(blur_row_kernel<Tin>, smem));
        const int vec = im.W % 4 == 0 && reinterpret_cast<uintptr_t>(src) % (4 * sizeof(Tin)) == 0;
        blur_row_kernel<Tin><<<grid, kSepThreads, smem, st>>>(src, dst, rows, (int)im.W, tile, np,
                                                              FastDiv((uint32_t)(tile / kK)), vec, t);
        CLE_LAUNCH_CHECK("blur pass");
    } else {
        int64_t inner, outer;
        int L;
        if (axis == 1) { inner = im.W; L = (int)im.H; outer = im.D; }
        else { inner = im.W * im.H; L = (int)im.D; outer = 1; }
        switch (col_groups(L, t.n)) {
            case 4: CLE_TRY((launch_col<Tin, 4>(src, dst, inner, L, outer, t, mm, clear, st))); break;
            case 8: CLE_TRY((launch_col<Tin, 8>(src, dst, inner, L, outer, t, mm, clear, st))); break;
            default: CLE_TRY((launch_col<Tin, 16>(src, dst, inner, L, outer, t, mm, clear, st))); break;
        }
    }
    return CLE_OK;
}

template <typename Tin>
int launch_convert(const Tin *src, float *dst, int64_t n, cudaStream_t st) {
    convert_kernel<Tin><<<launch_blocks(n, 256), 256, 0, st>>>(src, dst, n);
    CLE_LAUNCH_CHECK("convert");
    return CLE_OK;
}

template <typename Tin>
int separable_typed(const Img &src, float *dst, const Taps *taps[3], float *t1, float *t2, MinMaxState *mm,
                    int *clear, cudaStream_t st) {
    // pass order x (axis 2), y (axis 1), z (axis 0, 3D only)
    const int passes = (src.ndim == 3) ? 3 : 2;
    const int64_t n = src.n();
    const void *cur = src.data;
    bool cur_is_src = true;
    float *bufs[2] = {t1, t2};
    int which = 0;
    for (int p = 0; p < passes; ++p) {
        float *o = (p == passes - 1) ? dst : bufs[which];
        const Taps *t = taps[p];
        const bool last = p == passes - 1;
        if (cur_is_src) {
            if (t) CLE_TRY(launch_pass<Tin>((const Tin *)cur, o, src, 2 - p, *t, last ? mm : nullptr, last ? clear : nullptr, st));
            else CLE_TRY(launch_convert<Tin>((const Tin *)cur, o, n, st));
        } else {
            if (t) CLE_TRY(launch_pass<float>((const float *)cur, o, src, 2 - p, *t, last ? mm : nullptr, last ? clear : nullptr, st));
            else if (o != cur) CLE_CUDA(cudaMemcpyAsync(o, cur, sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
            if (last && clear && !t) CLE_CUDA(cudaMemsetAsync(clear, 0, sizeof(int), st));
        }
        cur = o;
        cur_is_src = false;
        which ^= 1;
    }
    return CLE_OK;
}

}  // namespace

size_t separable_workspace_bytes(const Img &im) {
    Arena a(nullptr, 0);
    a.take<float>(im.n());
    a.take<float>(im.n());
    return a.off;
}

int separable_filter(const Img &src, float *dst, const Taps *tx, const Taps *ty, const Taps *tz,
                     Arena &ws, cudaStream_t st, MinMaxState *mm, int *clear) {
    float *t1 = ws.take<float>(src.n());
    float *t2 = ws.take<float>(src.n());
    if (!ws.ok()) {
        set_error("gaussian_blur: workspace too small");
        return CLE_ERR_WORKSPACE;
    }
    const Taps *taps[3] = {tx, ty, tz};
    switch (src.dtype) {
        case CLE_F32: return separable_typed<float>(src, dst, taps, t1, t2, mm, clear, st);
        case CLE_U16: return separable_typed<uint16_t>(src, dst, taps, t1, t2, mm, clear, st);
        case CLE_U8: return separable_typed<uint8_t>(src, dst, taps, t1, t2, mm, clear, st);
        default:
            set_error("gaussian_blur: source dtype %d not supported (u8/u16/f32)", src.dtype);
            return CLE_ERR_DTYPE;
    }
}

int gaussian_blur(const Img &src, float *dst, double sx, double sy, double sz, Arena &ws,
                  cudaStream_t st, int *status, bool clear) {
    if (fused_blur_applies(src, sx, sy, sz))
        return fused_blur(src, dst, sx, st, nullptr, status);
    Taps tx, ty, tz;
    const Taps *px = nullptr, *py = nullptr, *pz = nullptr;
    if (sx > 0) { CLE_TRY(make_gauss_taps(sx, tx)); px = &tx; }
    if (sy > 0) { CLE_TRY(make_gauss_taps(sy, ty)); py = &ty; }
    if (src.ndim == 3 && sz > 0) { CLE_TRY(make_gauss_taps(sz, tz)); pz = &tz; }
    return separable_filter(src, dst, px, py, pz, ws, st, nullptr, clear && src.ndim == 3 ? status : nullptr);
}

int separable_minmax(const Img &src, float *dst, double sigma, MinMaxState *mm, Arena &ws, cudaStream_t st) {
    Taps t;
    CLE_TRY(make_gauss_taps(sigma, t));
    return separable_filter(src, dst, &t, &t, src.ndim == 3 ? &t : nullptr, ws, st, mm);
}

}  // namespace cle
