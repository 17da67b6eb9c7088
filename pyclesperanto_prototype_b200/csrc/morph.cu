// morph.cu -- erode_box (_tier1/_erode_box.py:6-47): binary erosion over the
// 3x3 (2D) or 3x3x3 (3D) box.  A voxel of the output is 1 when it and every
// neighbour in its box are nonzero in the source, else 0.  Reads clamp to the
// image edge like every buffer read of the reference; a clamped read lands on
// a voxel of the same box, so only in-range neighbours decide.
//
// One launch: a CTA covers 32 x 8 (x, y) columns and marches a chunk of z.
// Per plane a thread ANDs rows y-1, y, y+1 of its column, takes the x
// neighbours' column results by warp shuffles (the two edge lanes load their
// outer column), and keeps the last three plane results in registers, so each
// source voxel is read about once per plane pass and each output written once.
#include "common.cuh"
#include "kernels.cuh"

namespace cle {

namespace {

constexpr int kEX = 32;   // x columns per CTA (one warp per y row)
constexpr int kEY = 8;    // y rows per CTA

template <typename T>
__device__ __forceinline__ uint32_t nonzero(T v) { return v != T(0) ? 1u : 0u; }

template <typename Ts, typename Td, bool Z>
__global__ void __launch_bounds__(kEX * kEY)
erode_box_kernel(const Ts *__restrict__ src, Td *__restrict__ dst, int D, int H, int W, int zchunk) {
    const int lane = threadIdx.x;
    const int x = blockIdx.x * kEX + lane;
    const int y = blockIdx.y * kEY + threadIdx.y;
    // columns and rows beyond the image repeat the last one (clamp); they
    // take part in the shuffles but store nothing
    const int xc = min(x, W - 1), yc = min(y, H - 1);
    const int ym = max(yc - 1, 0), yp = min(yc + 1, H - 1);
    const int xe = (lane == 0) ? max(xc - 1, 0) : min(xc + 1, W - 1);   // edge lanes' outer column
    const bool edge = lane == 0 || lane == kEX - 1;
    const int64_t plane = (int64_t)H * W;

    auto plane_and = [&](int z) -> uint32_t {
        const Ts *p = src + (int64_t)z * plane;
        const uint32_t c = nonzero(__ldg(p + (int64_t)ym * W + xc)) & nonzero(__ldg(p + (int64_t)yc * W + xc)) &
                           nonzero(__ldg(p + (int64_t)yp * W + xc));
        uint32_t e = 1u;
        if (edge)
            e = nonzero(__ldg(p + (int64_t)ym * W + xe)) & nonzero(__ldg(p + (int64_t)yc * W + xe)) &
                nonzero(__ldg(p + (int64_t)yp * W + xe));
        const uint32_t l = __shfl_up_sync(0xffffffffu, c, 1);
        const uint32_t r = __shfl_down_sync(0xffffffffu, c, 1);
        return c & (lane == 0 ? e : l) & (lane == kEX - 1 ? e : r);
    };

    const bool store = x < W && y < H;
    if constexpr (!Z) {
        const uint32_t o = plane_and(0);
        if (store) dst[(int64_t)y * W + x] = (Td)o;
    } else {
        const int z0 = (int)blockIdx.z * zchunk;
        const int z1 = min(D, z0 + zchunk);
        uint32_t prev = plane_and(max(z0 - 1, 0));
        uint32_t cur = plane_and(z0);
        for (int z = z0; z < z1; ++z) {
            const uint32_t next = plane_and(min(z + 1, D - 1));
            if (store) dst[(int64_t)z * plane + (int64_t)y * W + x] = (Td)(prev & cur & next);
            prev = cur;
            cur = next;
        }
    }
}

template <typename Ts, typename Td>
int launch_erode(const Img &src, const Img &dst, cudaStream_t st) {
    const int64_t gx = (src.W + kEX - 1) / kEX, gy = (src.H + kEY - 1) / kEY;
    if (gy > 65535) { set_error("erode_box: image too large"); return CLE_ERR_TOO_LARGE; }
    const bool z = src.ndim == 3;
    int zchunk = 1;
    int64_t gz = 1;
    if (z) {
        int dev = 0;
        CLE_CUDA(cudaGetDevice(&dev));
        // enough CTAs for 4 waves of 2048-thread SMs, chunks of >= 8 planes
        const int64_t want = (int64_t)num_sms(dev) * 32;
        int64_t chunks = (want + gx * gy - 1) / (gx * gy);
        chunks = std::max<int64_t>(1, std::min<int64_t>(chunks, src.D / 8));
        zchunk = (int)((src.D + chunks - 1) / chunks);
        gz = (src.D + zchunk - 1) / zchunk;
        if (gz > 65535) { set_error("erode_box: image too large"); return CLE_ERR_TOO_LARGE; }
    }
    const dim3 grid((unsigned)gx, (unsigned)gy, (unsigned)gz), block(kEX, kEY);
    if (z)
        erode_box_kernel<Ts, Td, true><<<grid, block, 0, st>>>((const Ts *)src.data, (Td *)dst.data, (int)src.D,
                                                              (int)src.H, (int)src.W, zchunk);
    else
        erode_box_kernel<Ts, Td, false><<<grid, block, 0, st>>>((const Ts *)src.data, (Td *)dst.data, 1,
                                                               (int)src.H, (int)src.W, 1);
    CLE_LAUNCH_CHECK("erode_box");
    return CLE_OK;
}

template <typename Ts>
int erode_dst(const Img &src, const Img &dst, cudaStream_t st) {
    switch (dst.dtype) {
        case CLE_U8: return launch_erode<Ts, uint8_t>(src, dst, st);
        case CLE_U16: return launch_erode<Ts, uint16_t>(src, dst, st);
        case CLE_U32: return launch_erode<Ts, uint32_t>(src, dst, st);
        case CLE_F32: return launch_erode<Ts, float>(src, dst, st);
        default: set_error("erode_box: unsupported destination dtype %d", dst.dtype); return CLE_ERR_DTYPE;
    }
}

// ---- minimum_box / maximum_box (separable, clamped windows) -------------
// _tier1/_minimum_box.py:6-55, _tier1/_maximum_box.py (minimum/maximum_separable_
// {2,3}d_x.cl, absent from the checkout): passes along x, then y, then z (3D), each
// the minimum (maximum) over v + i*e, i = -c..c, c = (N-1)/2 with
// N = int(2*radius + 1), reads clamped to the edge (so the window is the
// in-range part of it); a pass with radius <= 0 is a copy.  min/max are exact,
// so the float32 result does not depend on the order of the comparisons.
// A thread makes 8 consecutive outputs along the pass axis.  Their windows share
// all but 7 values at each end, so it takes the minimum of the shared core once
// and running minima of the two ends: (2r + 8) / 8 loads and about as many
// comparisons per output instead of 2r.  Loads have immediate offsets (a case
// per window length modulo 8).  The first pass reads 8/16-bit sources as they are
// and the last pass of top_hat_box subtracts, so neither has a pass of its own.
// What bounds it: reading and writing the image in each pass.  r = 10 on 100 x 512 x
// 512 uint16: x 55 us a pass (141 with a window scan per output), y and z 41 to 51
// (98), 32 at copy bandwidth; top_hat_box 0.77 -> 0.31 ms, 0.22 with x and y in one
// pass and the minimum and maximum along z in another (below).
constexpr int kBK = 8;            // outputs per thread along the axis
constexpr int kBT = 256;          // threads per CTA
constexpr int kBRow = 256;        // x pass: most outputs of a row per CTA
constexpr int kBPitch = kBK + 1;  // x pass: 8 staged values on 9 words (lanes on different banks)

template <bool MAX>
__device__ __forceinline__ float mm(float a, float b) { return MAX ? fmaxf(a, b) : fminf(a, b); }

// out[k] = min / max of the w = 8 q + S staged values from k on, k = 0..7 (w is odd).
// p: the thread's first value; staged value 8 j + k lies at p + j * BLK + k * STR,
// so that k is an immediate offset.
template <bool MAX, int S, int BLK, int STR>
__device__ __forceinline__ void window_of(const float *p, int q, float (&out)[kBK]) {
    if (q == 0) {
        float v[kBK + S - 1];
#pragma unroll
        for (int i = 0; i < kBK + S - 1; ++i) v[i] = p[i / kBK * BLK + i % kBK * STR];
#pragma unroll
        for (int k = 0; k < kBK; ++k) {
            out[k] = v[k];
#pragma unroll
            for (int i = 1; i < S; ++i) out[k] = mm<MAX>(out[k], v[k + i]);
        }
        return;
    }
    // the core every window holds: values 7 .. w - 1
    float v[kBK];
#pragma unroll
    for (int k = 0; k < kBK; ++k) v[k] = p[k * STR];
    float core = v[7];
    const float *b = p + BLK;
#pragma unroll 2
    for (int j = 1; j < q; ++j, b += BLK) {
        float u[kBK];
#pragma unroll
        for (int k = 0; k < kBK; ++k) u[k] = b[k * STR];
#pragma unroll
        for (int k = 0; k < kBK; k += 2) core = mm<MAX>(mm<MAX>(core, u[k]), u[k + 1]);
    }
    float e[kBK + S - 1];   // from value 8 q on
#pragma unroll
    for (int i = 0; i < kBK + S - 1; ++i) e[i] = b[i / kBK * BLK + i % kBK * STR];
#pragma unroll
    for (int i = 0; i < S; ++i) core = mm<MAX>(core, e[i]);
    // left ends: values k .. 6, right ends: values w .. w + k - 1
    float l = core;
    out[7] = core;
#pragma unroll
    for (int k = 6; k >= 0; --k) {
        l = mm<MAX>(l, v[k]);
        out[k] = l;
    }
    float r = e[S];
    out[1] = mm<MAX>(out[1], r);
#pragma unroll
    for (int k = 2; k < kBK; ++k) {
        r = mm<MAX>(r, e[S + k - 1]);
        out[k] = mm<MAX>(out[k], r);
    }
}
template <bool MAX, int BLK, int STR>
__device__ __forceinline__ void window8(const float *p, int w, float (&out)[kBK]) {
    switch (w % kBK) {
        case 1: window_of<MAX, 1, BLK, STR>(p, w / kBK, out); break;
        case 3: window_of<MAX, 3, BLK, STR>(p, w / kBK, out); break;
        case 5: window_of<MAX, 5, BLK, STR>(p, w / kBK, out); break;
        default: window_of<MAX, 7, BLK, STR>(p, w / kBK, out); break;
    }
}

// x pass: np rows per CTA, an x tile of `tile` outputs (a multiple of 8) of each.
template <bool MAX, typename Tin>
__global__ void __launch_bounds__(kBT)
minmax_row_kernel(const Tin *__restrict__ src, float *__restrict__ dst, int64_t rows, int W, int r, int tile, int np,
                  FastDiv fper) {
    extern __shared__ float sm[];
    const int span = tile + 2 * r, pitch = (span / kBK + 2) * kBPitch;
    const int x0 = blockIdx.x * tile, lane = threadIdx.x & 31;
    const int64_t row0 = ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * np;
    if (row0 >= rows) return;
    for (int q = threadIdx.x >> 5; q < np; q += kBT / 32) {
        const Tin *p = src + min(row0 + q, rows - 1) * W;
        float *ln = sm + q * pitch;
        for (int c0 = lane; c0 < span; c0 += 4 * 32) {
            float v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (c0 + 32 * u < span) v[u] = to_f32(__ldg(p + clampi(x0 - r + c0 + 32 * u, 0, W - 1)));
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = c0 + 32 * u;
                if (c < span) ln[c + c / kBK] = v[u];
            }
        }
    }
    __syncthreads();
    const int per = tile / kBK;
    for (int e = threadIdx.x; e < np * per; e += kBT) {
        const int q = (int)fper.div((uint32_t)e), c = e - q * per, x = x0 + c * kBK;
        if (row0 + q >= rows || x >= W) continue;
        const float *base = sm + q * pitch + c * kBPitch;
        float out[kBK];
        window8<MAX, kBPitch, 1>(base, 2 * r + 1, out);
        float *o = dst + (row0 + q) * W + x;
        if ((W & 3) == 0 && x + kBK <= W && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
            reinterpret_cast<float4 *>(o)[0] = make_float4(out[0], out[1], out[2], out[3]);
            reinterpret_cast<float4 *>(o)[1] = make_float4(out[4], out[5], out[6], out[7]);
        } else {
#pragma unroll
            for (int k = 0; k < kBK; ++k)
                if (x + k < W) o[k] = out[k];
        }
    }
}

// Pass along an axis of length L with element stride `inner`, for a volume
// viewed as [outer][L][inner]: a CTA takes NG x 8 outputs along the axis and
// 2 x 256 / NG columns, a thread two adjacent columns.
template <bool MAX, typename Tin, int NG, typename Ts>
__global__ void __launch_bounds__(kBT)
minmax_col_kernel(const Tin *__restrict__ src, float *__restrict__ dst, int64_t inner, int L, int r, int vec,
                  const Ts *__restrict__ minus) {
    constexpr int NC = kBT / NG, COLS = 2 * NC, ROWS = NG * kBK;
    extern __shared__ __align__(16) float sm[];
    const int64_t c0 = (int64_t)blockIdx.x * COLS, base = (int64_t)blockIdx.z * L * inner;
    const int l0 = blockIdx.y * ROWS;
    const int span = ROWS + 2 * r;   // rows past the axis repeat its last value
    if (vec) {   // float32, inner a multiple of 4: asynchronous 16-byte copies
        constexpr int QPR = COLS / 4, STEP = kBT / QPR;
        const int c = 4 * (threadIdx.x % QPR);
        const Tin *p = src + base + min(c0 + c, inner - 4);
        for (int j = threadIdx.x / QPR; j < span; j += STEP)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(sm + j * COLS + c)),
                         "l"(p + (int64_t)clampi(l0 - r + j, 0, L - 1) * inner)
                         : "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        constexpr int STEP = kBT / COLS;
        const int c = threadIdx.x % COLS;
        const Tin *p = src + base + min(c0 + c, inner - 1);
        for (int j0 = threadIdx.x / COLS; j0 < span; j0 += 8 * STEP) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (j0 + u * STEP < span) v[u] = to_f32(__ldg(p + (int64_t)clampi(l0 - r + j0 + u * STEP, 0, L - 1) * inner));
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (j0 + u * STEP < span) sm[(j0 + u * STEP) * COLS + c] = v[u];
        }
    }
    __syncthreads();
    const int cp = threadIdx.x % NC, g = threadIdx.x / NC;
    const int64_t c = c0 + 2 * cp;
    const int left = L - (l0 + g * kBK);
    if (c >= inner || left <= 0) return;
    const float *col = sm + g * kBK * COLS + 2 * cp;
    float a[kBK], b[kBK];
    const int64_t at = base + (int64_t)(l0 + g * kBK) * inner + c;
    const bool two = c + 1 < inner, pair = (inner & 1) == 0 && (reinterpret_cast<uintptr_t>(dst) & 7) == 0;
    // minus (add_images_weighted(source, opening, 1, -1)): the source's values
    // are on their way while the windows are computed
    Ts sa[kBK], sb[kBK];
    if (minus) {
#pragma unroll
        for (int k = 0; k < kBK; ++k) {
            const int64_t i = at + (int64_t)min(k, left - 1) * inner;
            sa[k] = __ldg(minus + i);
            sb[k] = two ? __ldg(minus + i + 1) : Ts(0);
        }
    }
    window8<MAX, kBK * COLS, COLS>(col, 2 * r + 1, a);
    window8<MAX, kBK * COLS, COLS>(col + 1, 2 * r + 1, b);
    if (minus) {
#pragma unroll
        for (int k = 0; k < kBK; ++k) {
            a[k] = __fsub_rn(to_f32(sa[k]), a[k]);
            b[k] = __fsub_rn(to_f32(sb[k]), b[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < kBK; ++k)
        if (k < left) {
            const int64_t i = at + (int64_t)k * inner;
            if (pair) {
                *reinterpret_cast<float2 *>(dst + i) = make_float2(a[k], b[k]);
            } else {
                dst[i] = a[k];
                if (two) dst[i + 1] = b[k];
            }
        }
}

// Minimum, then maximum along an axis (the opening of top_hat_box along z) in one
// launch: a CTA stages 128 outputs with 2 r on each side, makes the minima in the
// place of the staged values, 128 rows at a time, and the maxima from those.  A
// position outside the axis is none of the maximum's: its minimum is NaN, which
// fmaxf passes over.  100 x 512 x 512, r = 10: 69 us against 93 in two launches;
// 509 x 511 planes (scalar staging) 70 us less.
// NG: groups of 8 outputs along the axis (128 outputs of 32 columns with 16).
template <int NG>
__global__ void __launch_bounds__(kBT)
open_col_kernel(const float *__restrict__ src, float *__restrict__ dst, int64_t inner, int L, int r, int span, int vec) {
    constexpr int NC = kBT / NG, kOCols = 2 * NC, kORows = NG * kBK;
    extern __shared__ __align__(16) float sm[];
    const int64_t c0 = (int64_t)blockIdx.x * kOCols;
    const int l0 = blockIdx.y * kORows, tid = threadIdx.x;
    if (vec) {   // inner a multiple of 4: asynchronous 16-byte copies
        constexpr int QPR = kOCols / 4, STEP = kBT / QPR;
        const int c = 4 * (tid % QPR);
        const float *p = src + min(c0 + c, inner - 4);
        for (int j = tid / QPR; j < span; j += STEP)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(sm + j * kOCols + c)),
                         "l"(p + (int64_t)clampi(l0 - 2 * r + j, 0, L - 1) * inner)
                         : "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        constexpr int STEP = kBT / kOCols;   // (span is a multiple of 8 of them)
        const float *p = src + min(c0 + tid % kOCols, inner - 1);
        float *o = sm + tid;
        for (int j0 = tid / kOCols; j0 < span; j0 += 8 * STEP, o += 8 * STEP * kOCols) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = __ldg(p + (int64_t)clampi(l0 - 2 * r + j0 + u * STEP, 0, L - 1) * inner);
#pragma unroll
            for (int u = 0; u < 8; ++u) o[u * STEP * kOCols] = v[u];
        }
    }
    __syncthreads();
    const int g = tid / NC, w = 2 * r + 1, need = kORows + 2 * r;
    float *col = sm + g * kBK * kOCols + 2 * (tid % NC);
    float a[kBK], b[kBK];
    for (int q = 0; q < need; q += kORows, col += kORows * kOCols) {
        const int row = q + g * kBK, at = l0 - r + row;   // first minimum: its row, its position
        const bool on = row < need && at < L && at + kBK > 0;
        if (on) {
            window8<false, kBK * kOCols, kOCols>(col, w, a);
            window8<false, kBK * kOCols, kOCols>(col + 1, w, b);
        }
        __syncthreads();
        if (row < need) {
#pragma unroll
            for (int k = 0; k < kBK; ++k) {
                const bool in = on && at + k >= 0 && at + k < L;
                col[k * kOCols] = in ? a[k] : NAN;
                col[k * kOCols + 1] = in ? b[k] : NAN;
            }
        }
    }
    __syncthreads();
    const int64_t c = c0 + 2 * (tid % NC);
    const int left = L - (l0 + g * kBK);
    if (c >= inner || left <= 0) return;
    col = sm + g * kBK * kOCols + 2 * (tid % NC);
    window8<true, kBK * kOCols, kOCols>(col, w, a);
    window8<true, kBK * kOCols, kOCols>(col + 1, w, b);
    const bool two = c + 1 < inner, pair = (inner & 1) == 0 && (reinterpret_cast<uintptr_t>(dst) & 7) == 0;
    float *o = dst + (int64_t)(l0 + g * kBK) * inner + c;
#pragma unroll
    for (int k = 0; k < kBK; ++k, o += inner)
        if (k < left) {
            if (pair) {
                *reinterpret_cast<float2 *>(o) = make_float2(a[k], b[k]);
            } else {
                o[0] = a[k];
                if (two) o[1] = b[k];
            }
        }
}

template <int NG>
int launch_open(const float *src, float *dst, const Img &im, int r, cudaStream_t st) {
    constexpr int COLS = 2 * (kBT / NG), ROWS = NG * kBK, STEP = 8 * kBT / COLS;
    const int64_t inner = im.H * im.W;
    const int span = (ROWS + 4 * r + kBK + STEP - 1) / STEP * STEP;
    const size_t smem = sizeof(float) * COLS * (size_t)span;
    CLE_TRY(allow_smem(open_col_kernel<NG>, smem));
    const dim3 grid((unsigned)((inner + COLS - 1) / COLS), (unsigned)((im.D + ROWS - 1) / ROWS));
    const int vec = inner % 4 == 0 && reinterpret_cast<uintptr_t>(src) % 16 == 0;
    open_col_kernel<NG><<<grid, kBT, smem, st>>>(src, dst, inner, (int)im.D, r, span, vec);
    CLE_LAUNCH_CHECK("top_hat_box");
    return CLE_OK;
}

int open_z(const float *src, float *dst, const Img &im, int r, cudaStream_t st) {
    // short axes take fewer outputs and more columns per CTA
    if (im.D <= 32) return launch_open<4>(src, dst, im, r, st);
    if (im.D <= 64) return launch_open<8>(src, dst, im, r, st);
    return launch_open<16>(src, dst, im, r, st);
}

// x and y passes of an image (or of every plane of a volume) in one launch: a CTA
// stages 64 x 64 outputs with their halo, makes the x windows of all staged rows
// (a warp per 8 columns, a lane per row) and the y windows of those (a warp per 8
// rows, a lane per column), so the image crosses memory once instead of twice.
// minus: as in the column kernel.  100 x 512 x 512, r = 10: 72 us (uint16) to 81 (float32
// and subtracting) against 96 and 106 in two launches; bound by issue (64%) and
// the shared-memory loads of the windows.
// Staging takes 96 columns and a multiple of 32 rows whatever the radius, clamped to
// the image, so that it has no guards and strides are immediates.
constexpr int kBP = 64;                 // outputs per CTA along x and y
constexpr int kMaxPlaneR = 16;          // 64 + 2 r staged values are at most 3 warps wide
constexpr int kBIn = (3 * 32 / kBK * kBPitch) | 1;   // pitch of the staged rows (odd: a lane per row meets no bank twice)
inline int plane_rows(int ry) { return (kBP + 2 * ry + 31) / 32 * 32; }

template <bool MAX, typename Tin, typename Ts>
__global__ void __launch_bounds__(kBT, 4)
minmax_plane_kernel(const Tin *__restrict__ src, float *__restrict__ dst, int H, int W, int rx, int ry, int rows,
                    const Ts *__restrict__ minus) {
    constexpr int NW = kBT / 32;
    static_assert(NW == kBP / kBK && kBP == 64, "a warp per 8 columns, then per 8 rows");
    extern __shared__ float sm[];
    const int x0 = blockIdx.x * kBP, y0 = blockIdx.y * kBP, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t plane = (int64_t)blockIdx.z * H * W;
    const uint32_t w = (uint32_t)W;
    {
        const Tin *p = src + plane;
        uint32_t xs[3];
#pragma unroll
        for (int u = 0; u < 3; ++u) xs[u] = (uint32_t)clampi(x0 - rx + lane + 32 * u, 0, W - 1);
        float *o = sm + warp * kBIn + lane + lane / kBK;
        for (int j0 = y0 - ry + warp; j0 < y0 - ry + rows; j0 += 4 * NW, o += 4 * NW * kBIn) {
            Tin v[4][3];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const uint32_t row = (uint32_t)clampi(j0 + a * NW, 0, H - 1) * w;
#pragma unroll
                for (int u = 0; u < 3; ++u) v[a][u] = __ldg(p + (row + xs[u]));
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int u = 0; u < 3; ++u) o[a * NW * kBIn + u * (32 / kBK * kBPitch)] = to_f32(v[a][u]);
        }
    }
    __syncthreads();
    // the x windows take the place of their rows' staged values, 32 rows at a time
    float o[kBK];
    float *p = sm + lane * kBIn;
    for (int q = 0; q < rows; q += 32, p += 32 * kBIn) {
        window8<MAX, kBPitch, 1>(p + warp * kBPitch, 2 * rx + 1, o);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kBK; ++k) p[warp * kBK + k] = o[k];
    }
    __syncthreads();
    const int left = H - (y0 + warp * kBK);
    if (left <= 0) return;
    dst += plane;
    if (minus) minus += plane;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int x = x0 + lane + 32 * h;
        if (x >= W) return;
        const uint32_t at = (uint32_t)(y0 + warp * kBK) * w + (uint32_t)x;
        Ts sv[kBK];
        if (minus) {
#pragma unroll
            for (int k = 0; k < kBK; ++k) sv[k] = __ldg(minus + (at + (uint32_t)min(k, left - 1) * w));
        }
        window8<MAX, kBK * kBIn, kBIn>(sm + warp * kBK * kBIn + lane + 32 * h, 2 * ry + 1, o);
        if (minus) {
#pragma unroll
            for (int k = 0; k < kBK; ++k) o[k] = __fsub_rn(to_f32(sv[k]), o[k]);
        }
        if (left >= kBK) {
#pragma unroll
            for (int k = 0; k < kBK; ++k) dst[at + (uint32_t)k * w] = o[k];
        } else {
#pragma unroll
            for (int k = 0; k < kBK; ++k)
                if (k < left) dst[at + (uint32_t)k * w] = o[k];
        }
    }
}

constexpr int kMaxBoxRadius = 700;

// src (x pass only: any source type) -> dst; axis 0 = x, 1 = y, 2 = z
template <bool MAX, typename Tin, int NG, typename Ts>
int launch_col(const Tin *src, float *dst, int64_t inner, int L, int64_t outer, int r, const Ts *minus, cudaStream_t st) {
    constexpr int COLS = 2 * (kBT / NG), ROWS = NG * kBK;
    auto kern = minmax_col_kernel<MAX, Tin, NG, Ts>;
    const size_t smem = sizeof(float) * COLS * (size_t)(ROWS + 2 * r);
    CLE_TRY(allow_smem(kern, smem));
    const dim3 grid((unsigned)((inner + COLS - 1) / COLS), (unsigned)((L + ROWS - 1) / ROWS), (unsigned)outer);
    const int vec = sizeof(Tin) == 4 && inner % 4 == 0 && reinterpret_cast<uintptr_t>(src) % 16 == 0;
    kern<<<grid, kBT, smem, st>>>(src, dst, inner, L, r, vec, minus);
    return CLE_OK;
}

// axis kXY: radius r along x and ry along y
constexpr int kXY = 3;
constexpr int kOpenZ = 4;   // minimum, then maximum along z
template <bool MAX, typename Tin, typename Ts>
int minmax_pass(const Tin *src, float *dst, const Img &im, int axis, int r, int ry, const Ts *minus, cudaStream_t st) {
    if (im.H > 65535 || im.D > 65535) { set_error("minimum/maximum box: image too large"); return CLE_ERR_TOO_LARGE; }
    if (axis == kXY) {
        auto kern = minmax_plane_kernel<MAX, Tin, Ts>;
        const int rows = plane_rows(ry);
        const size_t smem = sizeof(float) * (size_t)rows * kBIn;
        CLE_TRY(allow_smem(kern, smem));
        const dim3 grid((unsigned)((im.W + kBP - 1) / kBP), (unsigned)((im.H + kBP - 1) / kBP), (unsigned)im.D);
        kern<<<grid, kBT, smem, st>>>(src, dst, (int)im.H, (int)im.W, r, ry, rows, minus);
    } else if (axis == 0) {
        r = (int)std::min<int64_t>(r, im.W - 1);
        const int64_t rows = im.D * im.H;
        const int tiles = (int)((im.W + kBRow - 1) / kBRow);
        const int tile = (int)(((im.W + tiles - 1) / tiles + kBK - 1) / kBK * kBK);
        // rows to fill the CTA's threads, as far as long windows fit 64 KB
        const int pitch = ((tile + 2 * r) / kBK + 2) * kBPitch;
        const int np = (int)std::max<size_t>(1, std::min<size_t>(std::min(kBT / (tile / kBK), 32), 65536 / (sizeof(float) * pitch)));
        const size_t smem = sizeof(float) * (size_t)np * pitch;
        auto kern = minmax_row_kernel<MAX, Tin>;
        CLE_TRY(allow_smem(kern, smem));
        const int64_t ctas = (rows + np - 1) / np;
        const dim3 grid((unsigned)((im.W + tile - 1) / tile), (unsigned)std::min<int64_t>(ctas, 65535),
                        (unsigned)((ctas + 65534) / 65535));
        kern<<<grid, kBT, smem, st>>>(src, dst, rows, (int)im.W, r, tile, np, FastDiv((uint32_t)(tile / kBK)));
    } else {
        const int64_t L = axis == 1 ? im.H : im.D;
        r = (int)std::min<int64_t>(r, L - 1);
        const int64_t inner = axis == 1 ? im.W : im.H * im.W, outer = axis == 1 ? im.D : 1;
        // short axes take fewer outputs and more columns per CTA
        if (L <= 64 && r <= 64) CLE_TRY((launch_col<MAX, Tin, 8, Ts>(src, dst, inner, (int)L, outer, r, minus, st)));
        else CLE_TRY((launch_col<MAX, Tin, 16, Ts>(src, dst, inner, (int)L, outer, r, minus, st)));
    }
    CLE_LAUNCH_CHECK("minimum/maximum box");
    return CLE_OK;
}

template <typename Ts>
__global__ void minus_kernel(const Ts *__restrict__ src, const float *v, float *d, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        d[i] = __fsub_rn(to_f32(src[i]), v[i]);
}
template <typename Ts>
__global__ void to_f32_kernel(const Ts *__restrict__ s, float *__restrict__ d, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) d[i] = to_f32(s[i]);
}

// A sequence of passes over the axes with r > 0, from `src` into `out` (not
// aliasing it), through out and tmp in turn; `minus`: out = *minus - result.
struct Step {
    bool is_max;
    int axis, r, ry;
};
template <typename Ts>
int run_steps(const Ts *src, float *out, float *tmp, const Img &im, const Step *steps, int n, const Ts *minus,
              cudaStream_t st) {
    const int64_t nv = im.n();
    if (n == 0) {
        to_f32_kernel<Ts><<<launch_blocks(nv, 256), 256, 0, st>>>(src, out, nv);
        if (minus) minus_kernel<Ts><<<launch_blocks(nv, 256), 256, 0, st>>>(minus, out, out, nv);
        CLE_LAUNCH_CHECK_N("minimum/maximum box", minus ? 2 : 1);
        return CLE_OK;
    }
    const float *cur = nullptr;
    for (int i = 0; i < n; ++i) {
        // the last pass lands in out
        float *o = ((n - 1 - i) & 1) ? tmp : out;
        // a y or z pass can subtract; an x pass is followed by a pass that does
        const Ts *m = i == n - 1 && steps[i].axis != 0 ? minus : nullptr;
        const Step &t = steps[i];
        if (t.axis == kOpenZ) {   // behind an x, y pass
            CLE_TRY(open_z(cur, o, im, t.r, st));
            cur = o;
            continue;
        }
        if (i == 0) CLE_TRY(t.is_max ? minmax_pass<true>(src, o, im, t.axis, t.r, t.ry, m, st)
                                     : minmax_pass<false>(src, o, im, t.axis, t.r, t.ry, m, st));
        else CLE_TRY(t.is_max ? minmax_pass<true>(cur, o, im, t.axis, t.r, t.ry, m, st)
                              : minmax_pass<false>(cur, o, im, t.axis, t.r, t.ry, m, st));
        cur = o;
    }
    if (minus && steps[n - 1].axis == 0) {
        minus_kernel<Ts><<<launch_blocks(nv, 256), 256, 0, st>>>(minus, out, out, nv);
        CLE_LAUNCH_CHECK("top_hat_box");
    }
    return CLE_OK;
}

}  // namespace

// top_hat_box's opening along z in one launch up to radius 24 (behind an x, y pass),
// where it was the faster form for every size tried; the minima of 2 r more rows
// per 128 outputs outweigh the saved pass from about 32 on (300 x 256 x 256, x and y
// r = 3: r = 10 164 against 178 us, 24 201 : 204, 32 229 : 219).
constexpr int kMaxOpenR = 24;

// x and y in one pass up to radius 16 (its staging's 96 columns), where it was the
// faster form for every size tried: 100 x 512 x 512 r = 1 60 against 92 us, r = 16 82
// against 107; 2048 x 2048 and 1000 planes of 100 x 20, 20 x 100 also.  32-bit
// offsets inside a plane.
static bool plane_pass(const Img &im, int rx, int ry) {
    return rx > 0 && ry > 0 && rx <= kMaxPlaneR && ry <= kMaxPlaneR && im.W > 1 && im.H > 1 &&
           im.H * im.W < (int64_t(1) << 31);
}

size_t box_filter_workspace_bytes(const Img &im) {
    Arena a(nullptr, 0);
    a.take<float>(im.n());      // the source of an in-place call
    a.take<float>(im.n());      // pass temporary
    return a.off;
}

static int radii(const Img &im, double rx, double ry, double rz, int r[3]) {
    const double rr[3] = {rx, ry, rz};
    for (int i = 0; i < 3; ++i) {
        if (!(rr[i] > 0)) { r[i] = 0; continue; }
        const int64_t n = (int64_t)(rr[i] * 2 + 1);     // radius_to_kernel_size
        r[i] = (int)std::min<int64_t>((n - 1) / 2, kMaxBoxRadius);
        if ((n - 1) / 2 > kMaxBoxRadius) {
            set_error("minimum/maximum box: radius above %d", kMaxBoxRadius);
            return CLE_ERR_ARG;
        }
    }
    if (im.ndim == 2) r[2] = 0;
    return CLE_OK;
}

// minimum_box / maximum_box (hat: top_hat_box, source - maximum(minimum)); the
// passes with r > 0 along x, y (, z), for top_hat_box the minima then the maxima
template <typename Ts>
static int box_typed(const Img &src, float *dst, const int r[3], bool is_max, bool hat, Arena &ws, cudaStream_t st) {
    const int64_t n = src.n();
    float *copy = ws.take<float>(n);
    float *tmp = ws.take<float>(n);
    if (!ws.ok()) { set_error("minimum/maximum box: workspace too small"); return CLE_ERR_WORKSPACE; }
    if (n == 0) return CLE_OK;
    const Ts *in = (const Ts *)src.data;
    if (src.data == (void *)dst) {   // float32 in place
        CLE_CUDA(cudaMemcpyAsync(copy, src.data, sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
        in = (const Ts *)copy;
    }
    Step steps[6];
    int k = 0;
    const int64_t len[3] = {src.W, src.H, src.D};
    const bool xy = plane_pass(src, r[0], r[1]);
    const bool open = hat && xy && r[2] > 0 && len[2] > 1 && std::min<int64_t>(r[2], len[2] - 1) <= kMaxOpenR;
    for (int p = 0; p < (hat ? 2 : 1); ++p) {
        const bool mx = hat ? p == 1 : is_max;
        auto pass = [&](int a) {
            if (r[a] > 0 && len[a] > 1) steps[k++] = {mx, a, r[a], 0};
        };
        // the order of the axes does not change a minimum or maximum: the last
        // pass is one that can subtract
        if (open) {
            if (p == 1) steps[k++] = {false, kOpenZ, (int)std::min<int64_t>(r[2], len[2] - 1), 0};
        } else if (p == 1 && xy) {
            pass(2);
        }
        if (xy) steps[k++] = {mx, kXY, r[0], r[1]};
        else { pass(0); pass(1); }
        if ((p == 0 && !open) || !xy) pass(2);
    }
    return run_steps<Ts>(in, dst, tmp, src, steps, k, hat ? in : nullptr, st);
}

static int box_any(const Img &src, const Img &dst, double rx, double ry, double rz, bool is_max, bool hat, const char *name,
                   Arena &ws, cudaStream_t st) {
    CLE_TRY(same_shape(src, dst, "source", "destination"));
    if (dst.dtype != CLE_F32) { set_error("%s: destination must be float32", name); return CLE_ERR_DTYPE; }
    int r[3];
    CLE_TRY(radii(src, rx, ry, rz, r));
    switch (src.dtype) {
        case CLE_F32: return box_typed<float>(src, (float *)dst.data, r, is_max, hat, ws, st);
        case CLE_U16: return box_typed<uint16_t>(src, (float *)dst.data, r, is_max, hat, ws, st);
        case CLE_U8: return box_typed<uint8_t>(src, (float *)dst.data, r, is_max, hat, ws, st);
        default: set_error("box filter: unsupported source dtype %d", src.dtype); return CLE_ERR_DTYPE;
    }
}

int box_filter(const Img &src, const Img &dst, double rx, double ry, double rz, bool is_max, Arena &ws,
               cudaStream_t st) {
    return box_any(src, dst, rx, ry, rz, is_max, false, "minimum/maximum box", ws, st);
}

// top_hat_box: _tier2/_top_hat_box.py:37-43
int top_hat_box(const Img &src, const Img &dst, double rx, double ry, double rz, Arena &ws, cudaStream_t st) {
    return box_any(src, dst, rx, ry, rz, false, true, "top_hat_box", ws, st);
}

int erode_box(const Img &src, const Img &dst, cudaStream_t st) {
    CLE_TRY(same_shape(src, dst, "source", "destination"));
    if (src.n() == 0) return CLE_OK;
    switch (src.dtype) {
        case CLE_U8: return erode_dst<uint8_t>(src, dst, st);
        case CLE_U16: return erode_dst<uint16_t>(src, dst, st);
        case CLE_U32: return erode_dst<uint32_t>(src, dst, st);
        case CLE_I32: return erode_dst<int32_t>(src, dst, st);
        case CLE_F32: return erode_dst<float>(src, dst, st);
        default: set_error("erode_box: unsupported source dtype %d", src.dtype); return CLE_ERR_DTYPE;
    }
}

}  // namespace cle
