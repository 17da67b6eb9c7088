// blur_fused.cu -- one-launch separable Gaussian blur for isotropic sigma.
//
// Same arithmetic as the three-pass path in blur.cu (x pass, then y, then z,
// float32 intermediates, clamp-to-edge, acc = fma(w_i, v_i, acc) for
// i = -R..R from 0), fused so the source is read once and the result written
// once:
//   * a CTA owns a kTX x kTY output tile in (x, y) and marches along z over a
//     chunk of planes (plus R halo planes at each end, clamped);
//   * planes go in groups of P (4, or 2 or 1 where shared memory is short).  The
//     raw (kTY+2R) x (kTX+2R) tiles of a group are staged in shared memory in
//     the source's own type, two groups deep.  On volumes whose rows are a
//     multiple of 16 bytes and whose tiles mostly lie inside the image (tma_pays;
//     when the caller gives a status word) one thread
//     fetches a group with TMA copies (cp.async.bulk.tensor) an interval
//     ahead, completion counted by an mbarrier per stage; otherwise each
//     thread loads its share of a plane into registers through a table of
//     clamped offsets and stores it into the stage;
//   * x pass: an item is 8 x outputs of two rows, the two rows packed
//     (fma.rn.f32x2: two independent round-to-nearest FMAs, the same rounding
//     as fmaf), from 128-bit shared loads of the raw rows, converted in
//     registers (8/16-bit values by a byte permute into 2^23 + v and an exact
//     subtraction).  Column pairs would need an operand pair per odd offset,
//     which the compiler forms again at every use (66 moves an item: 1.92 ms
//     against 1.73 for 512 x 1024 x 1024 at R = 8).  Rows are an odd number of
//     16-byte granules apart, so the eight lanes of a load phase fall on
//     different banks;
//   * every pass runs in transposed form: a value is added to each output it
//     contributes to, output o taking tap i at its i-th step, which is the
//     same ascending chain per output.  So the x and y passes need no window
//     of values, and the z pass keeps 2R partial sums per column; it takes a
//     group's P planes at once, each partial sum moving P slots on;
//   * group g + 1's x pass and group g's y and z passes share one interval
//     between two CTA barriers (the x results are double-buffered).  One
//     barrier per plane instead of one per group left 18% of the warp time in
//     barriers (2.67 against 1.99 ms at that point).
// What bounds it: at R = 8 a voxel takes 59.5 FMAs (x on 48 rows for 32), 0.93 ms
// for 512 x 1024 x 1024 at 128 per SM and cycle; measured 1.73 ms (3.04 with three
// barriers per plane, a float32 tile and a shifted z ring), the FMA pipe 65%
// busy with 4 warps per scheduler, which the 2R partial sums allow (124
// registers).
// Radius R (= sigma_to_kernel_size(sigma)/2) is a template parameter; anisotropic
// sigmas and larger radii use the three-pass path.  In 3D the line is R = 8:
// above it the partial sums leave one CTA per SM and the halos of tile and chunk
// (60 rows for 32, 28 planes) cost more than three passes over memory do: R = 14
// on 61 x 479 x 347 0.251 against 0.152 ms, 64 x 256 x 256 0.106 / 0.062,
// 128 x 512 x 512 0.370 / 0.283, 128 x 1024 x 1024 1.295 / 0.974; R = 8 on the last two
// 0.179 / 0.238 and 0.517 / 0.866.  Given a
// min / max state, each CTA also adds the exact min / max of the values it
// stores and the last CTA writes the result's, which saves threshold_otsu's separate pass over the blurred image.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <atomic>
#include <cstring>

#include "common.cuh"
#include "kernels.cuh"

namespace cle {

namespace {

constexpr int kTX = 32;          // output columns per CTA
constexpr int kTY = 32;          // output rows per CTA
constexpr int kCP = kTX / 2;     // column pairs per tile (y and z passes own a pair)
constexpr int kRY = 2;           // output rows per thread (y and z passes)
constexpr int kThreads = kCP * (kTY / kRY);   // 256
constexpr int kWarps = kThreads / 32;
constexpr int kXS = kTX + 4;     // row stride of the x results (an odd number of 16-byte granules)
constexpr uint64_t kStageWaitNs = 2000000000ull;   // bound of one stage wait

// Resident CTAs per SM the registers allow (2R partial sums per owned column).
template <int R>
constexpr int min_ctas() { return R <= 4 ? 3 : 2; }

template <typename Tin, int R, bool Z>
struct Geom {
    static constexpr int ES = (int)sizeof(Tin);
    // x outputs per x-pass item; a single image has no other plane's work to
    // fill the threads with, so smaller items
    static constexpr int XO = Z ? 8 : 4;
    static constexpr int A = 16 / ES;                             // elements per 16-byte granule
    // the staged row starts at x0 - R - OFF, a multiple of 16 bytes from the row's start
    static constexpr int OFF = (R + A - 1) / A * A - R;
    static constexpr int ROWS = kTY + 2 * R;
    static constexpr int COLS = kTX + 2 * R;
    static constexpr int GR = (OFF + COLS + A - 1) / A;           // granules a row needs
    static constexpr int BX = (GR | 1) * A;                       // row stride (odd granules)
    static constexpr int VB = std::min(16, XO * ES);              // bytes per load of an x item
    static constexpr int VA = VB / ES;                            // elements of one
    static constexpr int NV = (OFF + XO + 2 * R + VA - 1) / VA;  // loads per x item
    static constexpr int ITEMS = ROWS / 2 * (kTX / XO);          // x items per plane (two rows each)
    static constexpr uint32_t BYTES = (uint32_t)(BX * ROWS * ES); // one plane's copy
    static constexpr int STAGE = (int)((BYTES + 127) / 128 * 128);
    static constexpr int LOADS = (ROWS * BX + kThreads - 1) / kThreads;
    static constexpr int XBUF = ROWS * kXS;                       // floats of one plane's x results
    static constexpr size_t TAB = Z ? sizeof(int) * ROWS * BX : 0;   // offset table of the register staging
    static constexpr size_t smem_of(int p) {
        return 128 + (size_t)(Z ? 2 * p : 1) * (STAGE + sizeof(float) * XBUF) + TAB;
    }
    // planes per group: as many as leave room for min_ctas CTAs per SM
    static constexpr int fit(int p) { return p == 1 || (size_t)min_ctas<R>() * (smem_of(p) + 2048) <= 227 * 1024 ? p : fit(p / 2); }
    static constexpr int P = Z ? fit(4) : 1;
    static constexpr size_t SMEM = smem_of(P);
    static_assert((kTX / XO - 1) * XO + NV * VA <= BX, "x item reads inside the staged row");
    static_assert((BX * ES / 16) % 2 == 1 && XO * ES % VB == 0, "aligned x items on odd row strides");
    static_assert(BX <= 256 && ROWS <= 256, "TMA box dimension above 256");
};

// Taps -R..0 (a Gaussian's taps are symmetric: tap i and tap -i come from the
// same i * i), a kernel parameter.
template <int R>
struct HalfTaps {
    float w[R + 1];
};

// ---- TMA staging ------------------------------------------------------------
// The box of a plane starts at x = x0 - R - OFF (OFF rounds it down so that
// x * sizeof(Tin) is a multiple of 16 bytes, the tiled copy's rule for the
// innermost coordinate), y = y0 - R and z = the clamped plane.  Box parts
// outside the image arrive zero-filled; a CTA whose tile reaches over the
// image's x or y edge then overwrites them in the stage with their clamped
// elements, which lie inside both the image and the box.
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0u;
}
// Waits for the phase of `parity` to complete; false after kStageWaitNs.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    while (!mbar_try_wait(bar, parity))
        if (global_ns() - t0 > kStageWaitNs) return false;
    return true;
}
// The same inside a CTA: a wait that runs out raises *fail, and a raised *fail
// ends every wait.
__device__ __forceinline__ void mbar_wait_or_fail(uint64_t *bar, uint32_t parity, int *fail) {
    if (mbar_try_wait(bar, parity)) return;
    const uint64_t t0 = global_ns();
    while (!mbar_try_wait(bar, parity)) {
        if (*(volatile int *)fail != 0) return;
        if (global_ns() - t0 > kStageWaitNs) { *(volatile int *)fail = 1; return; }
    }
}
// Orders this thread's earlier shared-memory accesses before its next
// async-proxy (TMA) write into the same memory.
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tma_load_plane(void *dst, const CUtensorMap *map, int x, int y, int z,
                                               uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar))
        : "memory");
}

// Staged source values as float32 (the same values as to_f32), one of two rows
// each, as a packed pair: element k of the 32-bit words u and v.  An unsigned
// value below 2^23: its bits under the exponent of 2^23 are 2^23 + value
// exactly, and subtracting 2^23 is exact.
__device__ __forceinline__ float2 word_pair(uint32_t u, uint32_t v, int, float) {
    return make_float2(__uint_as_float(u), __uint_as_float(v));
}
__device__ __forceinline__ float2 word_pair(uint32_t u, uint32_t v, int k, uint16_t) {
    const uint32_t sel = k ? 0x7432u : 0x7410u;
    return __fadd2_rn(make_float2(__uint_as_float(__byte_perm(u, 0x4B000000u, sel)), __uint_as_float(__byte_perm(v, 0x4B000000u, sel))),
                      make_float2(-8388608.0f, -8388608.0f));
}
__device__ __forceinline__ float2 word_pair(uint32_t u, uint32_t v, int k, uint8_t) {
    const uint32_t sel = 0x7440u + (uint32_t)k;
    return __fadd2_rn(make_float2(__uint_as_float(__byte_perm(u, 0x4B000000u, sel)), __uint_as_float(__byte_perm(v, 0x4B000000u, sel))),
                      make_float2(-8388608.0f, -8388608.0f));
}
// VB (16, 8 or 4) bytes from shared memory
template <int VB>
__device__ __forceinline__ void load_words(const uint8_t *p, uint32_t *w) {
    if constexpr (VB == 16) {
        const uint4 u = *reinterpret_cast<const uint4 *>(p);
        w[0] = u.x; w[1] = u.y; w[2] = u.z; w[3] = u.w;
    } else if constexpr (VB == 8) {
        const uint2 u = *reinterpret_cast<const uint2 *>(p);
        w[0] = u.x; w[1] = u.y;
    } else {
        w[0] = *reinterpret_cast<const uint32_t *>(p);
    }
}

// TMA: stage planes with the tensor map `tmap` (3D only).  A stage wait that
// runs out raises s_fail: no later wait blocks, no more copies are issued, the
// copies in flight are waited for and *status is set.
// Without TMA, a status word makes the launch the repeat of a TMA launch (same
// grid): it returns at once unless a wait ran out there.
template <typename Tin, int R, bool Z, bool TMA>
__global__ void __launch_bounds__(kThreads, (min_ctas<R>()))
blur_fused_kernel(const Tin *__restrict__ src, const __grid_constant__ CUtensorMap tmap,
                  float *__restrict__ dst, int D, int H, int W, int zchunk,
                  const __grid_constant__ HalfTaps<R> taps, MinMaxState *__restrict__ mm, int *__restrict__ status) {
    static_assert(!TMA || Z, "TMA staging is for volumes");
    using G = Geom<Tin, R, Z>;
    constexpr int BX = G::BX, P = G::P;
    constexpr bool kRegStage = Z && !TMA;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    // raw stages [1 or 2][P][STAGE], x results [1 or 2][P][ROWS][kXS], offsets
    uint8_t *raw = smem_raw + ((128u - (smem_addr(smem_raw) & 127u)) & 127u);
    float *Xo = reinterpret_cast<float *>(raw + (Z ? 2 * P : 1) * G::STAGE);
    int *tab = reinterpret_cast<int *>(Xo + (Z ? 2 * P : 1) * G::XBUF);

    if constexpr (!TMA) {
        if (status != nullptr && *(volatile int *)status == 0) return;
    }
    // CTAs that add to mm, those of the launch that is repeated among them
    const uint32_t ctas = gridDim.x * gridDim.y * gridDim.z * (!TMA && status != nullptr ? 2u : 1u);

    // in 3D the taps stay in registers as packed pairs (w, w), read once
    // through shared memory: taken from the parameter they are fetched for
    // every use, two register moves each
    float2 wr[R + 1];
    if constexpr (Z) {
        __shared__ float s_taps[R + 1];
        if (threadIdx.x <= R) s_taps[threadIdx.x] = taps.w[threadIdx.x];
        __syncthreads();
#pragma unroll
        for (int i = 0; i <= R; ++i) {
            wr[i].x = *(volatile float *)&s_taps[i];
            wr[i].y = *(volatile float *)&s_taps[i];
        }
    }
    auto tap = [&](int i) {
        const int k = i <= R ? i : 2 * R - i;
        if constexpr (Z) return wr[k];
        else return make_float2(taps.w[k], taps.w[k]);
    };

    const int tid = threadIdx.x;
    const int x0 = blockIdx.x * kTX;
    const int y0 = blockIdx.y * kTY;
    const int z0 = Z ? (int)blockIdx.z * zchunk : 0;
    const int z1 = Z ? min(D, z0 + zchunk) : 1;
    // virtual planes z0-R .. z1-1+R (clamped), in groups of P; 2D: the single plane
    const int nvirt = Z ? (z1 - z0) + 2 * R : 1;
    const int ngroups = (nvirt + P - 1) / P;
    const int zbase = Z ? z0 - R : 0;
    const int64_t plane = (int64_t)H * W;
    const int xs = x0 - R - G::OFF, ys = y0 - R;   // image coordinates of the staged tile's first element
    // plane p of group g
    auto stage = [&](int g, int p) { return reinterpret_cast<Tin *>(raw + ((Z ? (g & 1) * P : 0) + p) * G::STAGE); };
    auto xres = [&](int g, int p) { return Xo + ((Z ? (g & 1) * P : 0) + p) * G::XBUF; };

    // register staging: element s of the stage comes from image offset tab[s]
    // (clamped); raw values, so the loads stay in flight until stored
    Tin pre[TMA ? 1 : G::LOADS];
    auto offset_of = [&](int s) {
        const int r = s / BX, c = s - r * BX;
        return clampi(ys + r, 0, H - 1) * W + clampi(xs + c, 0, W - 1);
    };
    auto load_plane = [&](int v) {
        const Tin *p = src + (int64_t)(Z ? clampi(zbase + v, 0, D - 1) : 0) * plane;
#pragma unroll
        for (int k = 0; k < G::LOADS; ++k) {
            const int s = tid + k * kThreads;
            if constexpr (!TMA) pre[k] = s < G::ROWS * BX ? __ldg(p + (Z ? tab[s] : offset_of(s))) : Tin(0);
        }
    };
    auto store_plane = [&](Tin *d) {
#pragma unroll
        for (int k = 0; k < G::LOADS; ++k) {
            const int s = tid + k * kThreads;
            if constexpr (!TMA)
                if (s < G::ROWS * BX) d[s] = pre[k];
        }
    };

    // TMA staging: one barrier per stage; a tile over the image's edge is patched
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ int s_fail;
    const bool patch = xs + G::OFF < 0 || ys < 0 || x0 + kTX + R > W || y0 + kTY + R > H;
    auto issue = [&](int g) {   // one thread: group g into its stage
        const int n = min(P, nvirt - g * P);
        fence_proxy_async_smem();
        mbar_expect_tx(&bars[g & 1], (uint32_t)n * G::BYTES);
        for (int p = 0; p < n; ++p)
            tma_load_plane(stage(g, p), &tmap, xs, ys, clampi(zbase + g * P + p, 0, D - 1), &bars[g & 1]);
    };
    auto patch_plane = [&](Tin *d) {
        // columns left / right of the image, then rows above / below it; an
        // element inside the image is a source only, so the order is free
        const int nl = max(0, -(xs + G::OFF)), nc = nl + max(0, x0 + kTX + R - W);
        for (int e = tid; e < nc * G::ROWS; e += kThreads) {
            const int k = e / G::ROWS, r = e - k * G::ROWS;
            const int c = G::OFF + (k < nl ? k : G::COLS - nc + k);
            d[r * BX + c] = d[(clampi(ys + r, 0, H - 1) - ys) * BX + clampi(xs + c, 0, W - 1) - xs];
        }
        const int nt = max(0, -ys), nr = nt + max(0, y0 + kTY + R - H);
        for (int e = tid; e < nr * G::COLS; e += kThreads) {
            const int k = e / G::COLS, c = G::OFF + e - k * G::COLS;
            const int r = k < nt ? k : G::ROWS - nr + k;
            d[r * BX + c] = d[(clampi(ys + r, 0, H - 1) - ys) * BX + clampi(xs + c, 0, W - 1) - xs];
        }
        fence_proxy_async_smem();
    };
    // TMA: group g has landed (and is patched); its barrier's phase is g / 2
    auto arrive_group = [&](int g) {
        mbar_wait_or_fail(&bars[g & 1], (uint32_t)(g >> 1) & 1u, &s_fail);
        if (patch) {                       // uniform per CTA
            for (int p = 0; p < P; ++p) patch_plane(stage(g, p));
            __syncthreads();
        }
    };

    // x pass of group g: an item is XO outputs of rows r and r + ROWS / 2 of a
    // plane, the two rows packed; column c of the item adds tap c - k to
    // output k
    auto x_pass = [&](int g) {
        constexpr int HR = G::ROWS / 2, EW = 4 / G::ES;     // EW: elements per 32-bit word
        const int n = min(P, nvirt - g * P) * G::ITEMS;
#pragma unroll 1
        for (int e = tid; e < n; e += kThreads) {
            const int p = P == 1 ? 0 : e / G::ITEMS, q0 = e - p * G::ITEMS;
            const int part = q0 / HR, r = q0 - part * HR;
            const uint8_t *pa = reinterpret_cast<const uint8_t *>(stage(g, p) + r * BX + part * G::XO);
            float2 acc[G::XO];
#pragma unroll
            for (int k = 0; k < G::XO; ++k) acc[k] = make_float2(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < G::NV; ++q) {
                uint32_t u[G::VB / 4], w[G::VB / 4];
                load_words<G::VB>(pa + q * G::VB, u);
                load_words<G::VB>(pa + q * G::VB + HR * BX * G::ES, w);
#pragma unroll
                for (int t = 0; t < G::VA; ++t) {
                    const int c = q * G::VA + t - G::OFF;
                    if (c >= 0 && c < G::XO + 2 * R) {
                        const float2 f = word_pair(u[t / EW], w[t / EW], t % EW, Tin());
#pragma unroll
                        for (int k = 0; k < G::XO; ++k)
                            if (c - k >= 0 && c - k <= 2 * R) acc[k] = __ffma2_rn(tap(c - k), f, acc[k]);
                    }
                }
            }
            float *xo = xres(g, p) + r * kXS + part * G::XO;
#pragma unroll
            for (int k = 0; k < G::XO; k += 4) {
                *reinterpret_cast<float4 *>(xo + k) = make_float4(acc[k].x, acc[k + 1].x, acc[k + 2].x, acc[k + 3].x);
                *reinterpret_cast<float4 *>(xo + HR * kXS + k) = make_float4(acc[k].y, acc[k + 1].y, acc[k + 2].y, acc[k + 3].y);
            }
        }
    };

    // y/z ownership: columns tx, tx+1 (a packed pair), rows ry0 .. ry0+kRY-1
    const int tx = (tid % kCP) * 2;
    const int ry0 = (tid / kCP) * kRY;
    const bool c0_ok = (x0 + tx) < W, c1_ok = (x0 + tx + 1) < W;
    // 8-byte stores: rows of an even length in a destination on an 8-byte boundary
    // (a view may start at any element)
    const bool pair_store = c1_ok && (W & 1) == 0 && (reinterpret_cast<uintptr_t>(dst) & 7) == 0;
    float vmin = INFINITY, vmax = -INFINITY;   // of the stored values (when mm)
    auto store2 = [&](float *o, float2 v) {
        if (pair_store) *reinterpret_cast<float2 *>(o) = v;
        else {
            if (c0_ok) o[0] = v.x;
            if (c1_ok) o[1] = v.y;
        }
        if (mm) {
            vmin = fminf(vmin, v.x);
            vmax = fmaxf(vmax, v.x);
            if (c1_ok) { vmin = fminf(vmin, v.y); vmax = fmaxf(vmax, v.y); }
        }
    };
    // rows this thread stores, and the output place that plane 0 of the group would finish
    const int nrow = c0_ok ? min(kRY, H - (y0 + ry0)) : 0;
    float *op = dst + (int64_t)(z0 - (Z ? 2 * R : 0)) * plane + (int64_t)(y0 + ry0) * W + x0 + tx;

    // z partial sums: ring[j][i] of row j belongs to the output plane that has
    // taken taps 0..i (2R of them under way)
    float2 ring[kRY][2 * R];
#pragma unroll
    for (int j = 0; j < kRY; ++j)
#pragma unroll
        for (int i = 0; i < 2 * R; ++i) ring[j][i] = make_float2(0.0f, 0.0f);

    // groups 0 and 1 on their way, group 0 through its x pass
    int issued = 0;   // TMA, thread 0: groups issued
    if constexpr (TMA) {
        if (tid == 0) {
            s_fail = 0;
            mbar_init(&bars[0], 1);
            mbar_init(&bars[1], 1);
            mbar_init_fence();
        }
        __syncthreads();
        if (tid == 0)
            for (; issued < 2 && issued < ngroups; ++issued) issue(issued);
        arrive_group(0);
    } else {
        if constexpr (Z) {
            for (int s = tid; s < G::ROWS * BX; s += kThreads) tab[s] = offset_of(s);
            __syncthreads();
        }
        for (int v = 0; v < nvirt && v < 2 * P; ++v) {
            load_plane(v);
            store_plane(stage(v / P, v % P));
        }
        __syncthreads();
    }
    x_pass(0);
    __syncthreads();
    if constexpr (TMA) {
        if (tid == 0 && issued < ngroups && *(volatile int *)&s_fail == 0) issue(issued++);
    }
    // one group per interval between two barriers: group g + 1's x pass (its
    // stage has landed) and group g's y and z passes; the plane loop is not
    // unrolled (its body stays small enough for the instruction caches)
#pragma unroll 1
    for (int g = 0; g < ngroups; ++g) {
        if (Z && g + 1 < ngroups) {
            if constexpr (TMA) arrive_group(g + 1);
            x_pass(g + 1);
        }
        // y pass: kRY rows of the column pair; row j of the window adds tap
        // j - o to output row o.  Planes past the last one give values that
        // only reach outputs past the last one.
        float2 yv[P][kRY];
#pragma unroll
        for (int p = 0; p < P; ++p) {
            if constexpr (kRegStage) {
                if (g * P + p + 2 * P < nvirt) load_plane(g * P + p + 2 * P);
            }
            const float *xr = xres(g, p) + ry0 * kXS + tx;
#pragma unroll
            for (int o = 0; o < kRY; ++o) yv[p][o] = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < kRY + 2 * R; ++j) {
                const float2 c = *reinterpret_cast<const float2 *>(xr + j * kXS);
#pragma unroll
                for (int o = 0; o < kRY; ++o)
                    if (j - o >= 0 && j - o <= 2 * R) yv[p][o] = __ffma2_rn(tap(j - o), c, yv[p][o]);
            }
            // the stage of group g was consumed an interval ago
            if constexpr (kRegStage) {
                if (g * P + p + 2 * P < nvirt) store_plane(stage(g, p));
            }
        }
        if constexpr (Z) {
            // z pass, P planes at a time: the partial sum with taps 0..a takes
            // taps a + 1.. from the group's planes in order; the one that takes
            // tap 2R is finished by that plane, the others move on P slots
            // (descending a: slot a + P has been read before it is written)
#pragma unroll
            for (int j = 0; j < kRY; ++j) {
                float2 out[P];
#pragma unroll
                for (int a = 2 * R - 1; a >= -P; --a) {
                    float2 t = a >= 0 ? ring[j][a >= 0 ? a : 0] : make_float2(0.f, 0.f);
#pragma unroll
                    for (int p = 0; p < P; ++p) {
                        const int i = a + 1 + p;
                        if (i >= 0 && i <= 2 * R) {
                            t = __ffma2_rn(tap(i), yv[p][j], t);
                            if (i == 2 * R) out[p] = t;
                        }
                    }
                    if (a + P < 2 * R) ring[j][a + P < 2 * R ? a + P : 0] = t;
                }
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const int v = g * P + p;
                    if (v >= 2 * R && v < nvirt && j < nrow) store2(op + (int64_t)p * plane + j * W, out[p]);
                }
            }
            op += P * plane;
        } else {
#pragma unroll
            for (int j = 0; j < kRY; ++j)
                if (j < nrow) store2(op + j * W, yv[0][j]);
        }
        if constexpr (Z) __syncthreads();
        if constexpr (TMA) {
            // group g + 1's stage is consumed: group g + 3 into it
            if (tid == 0 && issued < ngroups && *(volatile int *)&s_fail == 0) issue(issued++);
        }
    }
    if constexpr (TMA) {
        // (the barrier above ordered every s_fail write)
        if (*(volatile int *)&s_fail != 0) {
            // the copies still in flight land before the CTA's shared memory is
            // released: the last group of each stage
            if (tid == 0) {
                for (int q = max(0, issued - 2); q < issued; ++q) mbar_wait(&bars[q & 1], (uint32_t)(q >> 1) & 1u);
                atomicCAS(status, 0, (int)CLE_ERR_ITER_LIMIT);
                if (mm) add_minmax(mm, INFINITY, -INFINITY, ctas);
            }
            return;
        }
    }
    if (mm) {
        __shared__ float s_mn[kWarps], s_mx[kWarps];
        const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            vmin = fminf(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
            vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
        }
        if (lane == 0) { s_mn[warp] = vmin; s_mx[warp] = vmax; }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < kWarps; ++w) { vmin = fminf(vmin, s_mn[w]); vmax = fmaxf(vmax, s_mx[w]); }
            add_minmax(mm, vmin, vmax, ctas);
        }
    }
}

// Upper bound on the z chunks of the fused launch: four waves of four CTAs per
// SM (above what any radius has resident; the most a tile count could use), at most one chunk per plane.
int64_t fused_chunk_cap(int64_t tiles, int64_t D, int sms) {
    return std::max<int64_t>(1, std::min<int64_t>(D, (16 * (int64_t)sms + tiles - 1) / tiles));
}

int resident_ctas(int R) { return R <= 4 ? min_ctas<4>() : min_ctas<8>(); }

// Grid of the fused launch: (x tiles, y tiles, z chunks).  A CTA's time is
// about its planes (chunk + 2R halo), and CTAs run in waves of the resident
// slots, so the chunk count minimises waves x (chunk + 2R): 512 x 1024 x 1024
// at R = 8 takes 2 chunks (2048 CTAs, 6.9 waves of 296) rather than 1
// (1024 CTAs, a half-empty fourth wave).
dim3 fused_grid(const Img &src, int R, int &zchunk) {
    const int gx = (int)((src.W + kTX - 1) / kTX);
    const int gy = (int)((src.H + kTY - 1) / kTY);
    int gz = 1;
    zchunk = 1;
    if (src.ndim == 3) {
        int dev = 0;
        cudaGetDevice(&dev);
        const int sms = num_sms(dev);
        const int64_t slots = (int64_t)sms * resident_ctas(R);
        const int64_t tiles = (int64_t)gx * gy;
        const int64_t cap = fused_chunk_cap(tiles, src.D, sms);
        int64_t best = -1;
        for (int64_t c = 1; c <= cap; ++c) {
            const int64_t zc = (src.D + c - 1) / c;
            const int64_t g = (src.D + zc - 1) / zc;
            const int64_t waves = (tiles * g + slots - 1) / slots;
            const int64_t cost = waves * (zc + 2 * R);
            if (best < 0 || cost < best) {
                best = cost;
                zchunk = (int)zc;
                gz = (int)g;
            }
        }
    }
    return dim3(gx, gy, gz);
}

// The source as a 3D tiled tensor map (x = W innermost) with the box of
// Geom<Tin, R, true>; false when the layout does not allow one (row pitch or base
// address not a multiple of 16 bytes) or the driver lacks the encoder.
// The driver's tensor-map encoder, looked up once outside any stream capture
// (an immutable function pointer; until then, and if the driver lacks it,
// the register-staged path runs).
void *tensor_map_encoder(cudaStream_t st) {
    static std::atomic<void *> fn{nullptr};
    static std::atomic<bool> looked{false};
    if (looked.load(std::memory_order_acquire)) return fn.load(std::memory_order_acquire);
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
        (void)cudaGetLastError();
        return nullptr;
    }
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
        (void)cudaGetLastError();
        f = nullptr;
    }
    fn.store(f, std::memory_order_release);
    looked.store(true, std::memory_order_release);
    return f;
}

template <typename Tin, int R>
bool encode_source_map(const Img &src, CUtensorMap &map, cudaStream_t st) {
    using TG = Geom<Tin, R, true>;
    const uint64_t pitch = (uint64_t)src.W * sizeof(Tin);
    if (pitch % 16 != 0 || (reinterpret_cast<uintptr_t>(src.data) & 15) != 0) return false;
    void *const fn = tensor_map_encoder(st);
    if (fn == nullptr) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)src.W, (cuuint64_t)src.H, (cuuint64_t)src.D};
    const cuuint64_t strides[2] = {(cuuint64_t)pitch, (cuuint64_t)(pitch * (uint64_t)src.H)};
    const cuuint32_t box[3] = {(cuuint32_t)TG::BX, (cuuint32_t)TG::ROWS, 1u};
    const cuuint32_t estride[3] = {1u, 1u, 1u};
    const CUtensorMapDataType dt = sizeof(Tin) == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                 : sizeof(Tin) == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16
                                                    : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    const CUresult r = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn)(
        &map, dt, 3, src.data, dims, strides, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// TMA staging pays where most tiles lie inside the image: a tile on its edge is
// patched behind another barrier in every group.  Interior tiles: half of them
// (8 x 8 tiles) for 8/16-bit sources, three quarters (16 x 16) for float32, whose
// copies are longest.  Microseconds with TMA / through registers, uint16 sigma 2:
// 16 x 16 x 16 29 / 18, 64 x 128 x 128 31 / 29, 512 x 1024 x 16 127 / 92, 64 x 256 x 256 44 / 43,
// 100 x 512 x 512 141 / 157, 4 x 1024 x 1024 73 / 84; float32: 16 x 16 x 16 31 / 21,
// 96 x 256 x 256 68 / 62, 100 x 512 x 512 180 / 178 (sigma 0.5: 63 / 91), 4 x 1024 x 1024 94 / 101.
bool tma_pays(const dim3 &grid, int bytes) {
    const int64_t gx = grid.x, gy = grid.y, inside = std::max<int64_t>(0, gx - 2) * std::max<int64_t>(0, gy - 2);
    return bytes < 4 ? 2 * inside >= gx * gy : 4 * inside >= 3 * gx * gy;
}

template <typename Tin, int R, bool Z>
int launch_fused_r(const Img &src, float *dst, const Taps &t, MinMaxState *mm, int *status, bool repeat, cudaStream_t st) {
    using G = Geom<Tin, R, Z>;
    int zchunk = 1;
    const dim3 grid = fused_grid(src, R, zchunk);
    if (grid.y > 65535 || grid.z > 65535) { set_error("gaussian_blur: image too large for the fused path"); return CLE_ERR_TOO_LARGE; }
    HalfTaps<R> pt;
    for (int i = 0; i <= R; ++i) pt.w[i] = t.w[i];
    alignas(64) CUtensorMap map;
    std::memset(&map, 0, sizeof(map));
    int *gate = nullptr;
    if constexpr (Z) {
        if (status != nullptr && tma_pays(grid, sizeof(Tin)) && encode_source_map<Tin, R>(src, map, st)) {
            auto kern = blur_fused_kernel<Tin, R, true, true>;
            // set on every call: the attribute belongs to the current device's context
            CLE_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::SMEM));
            kern<<<grid, kThreads, G::SMEM, st>>>((const Tin *)src.data, map, dst, (int)src.D, (int)src.H,
                                                        (int)src.W, zchunk, pt, mm, status);
            CLE_LAUNCH_CHECK("gaussian_blur fused (TMA)");
            if (!repeat) return CLE_OK;
            gate = status;
        }
    }
    auto kern = blur_fused_kernel<Tin, R, Z, false>;
    CLE_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::SMEM));
    kern<<<grid, kThreads, G::SMEM, st>>>((const Tin *)src.data, map, dst, (int)src.D, (int)src.H, (int)src.W,
                                                zchunk, pt, mm, gate);
    CLE_LAUNCH_CHECK("gaussian_blur fused");
    return CLE_OK;
}

template <typename Tin, bool Z, int R = 1>
int dispatch_r(const Img &src, float *dst, const Taps &t, int r, MinMaxState *mm, int *status, bool repeat, cudaStream_t st) {
    if constexpr (R > (Z ? kMaxFusedR3 : kMaxFusedR)) {
        set_error("internal: fused radius out of range");
        return CLE_ERR_ARG;
    } else {
        if (r == R) return launch_fused_r<Tin, R, Z>(src, dst, t, mm, status, repeat, st);
        return dispatch_r<Tin, Z, R + 1>(src, dst, t, r, mm, status, repeat, st);
    }
}

}  // namespace

bool fused_blur_applies(const Img &src, double sx, double sy, double sz) {
    if (!(sx > 0) || sx != sy) return false;
    if (src.ndim == 3 && sz != sx) return false;
    if (src.dtype != CLE_F32 && src.dtype != CLE_U16 && src.dtype != CLE_U8) return false;
    const int r = (sigma_to_kernel_size(sx) - 1) / 2;
    return r >= 1 && r <= (src.ndim == 3 ? kMaxFusedR3 : kMaxFusedR) && src.W < (1 << 30) && src.H < (1 << 30);
}

int fused_blur(const Img &src, float *dst, double sigma, cudaStream_t st, MinMaxState *mm, int *status, bool repeat) {
    Taps t;
    CLE_TRY(make_gauss_taps(sigma, t));
    const int r = (t.n - 1) / 2;
    const bool z = src.ndim == 3;
    switch (src.dtype) {
        case CLE_F32: return z ? dispatch_r<float, true>(src, dst, t, r, mm, status, repeat, st) : dispatch_r<float, false>(src, dst, t, r, mm, status, repeat, st);
        case CLE_U16: return z ? dispatch_r<uint16_t, true>(src, dst, t, r, mm, status, repeat, st) : dispatch_r<uint16_t, false>(src, dst, t, r, mm, status, repeat, st);
        case CLE_U8: return z ? dispatch_r<uint8_t, true>(src, dst, t, r, mm, status, repeat, st) : dispatch_r<uint8_t, false>(src, dst, t, r, mm, status, repeat, st);
        default: set_error("gaussian_blur: unsupported source dtype"); return CLE_ERR_DTYPE;
    }
}

int blur_minmax(const Img &src, float *dst, double sigma, MinMaxState *mm, Arena &ws, cudaStream_t st, int *status,
                bool repeat) {
    if (fused_blur_applies(src, sigma, sigma, sigma)) return fused_blur(src, dst, sigma, st, mm, status, repeat);
    if (sigma > 0) return separable_minmax(src, dst, sigma, mm, ws, st);
    CLE_TRY(gaussian_blur(src, dst, sigma, sigma, sigma, ws, st, status));
    Img T = src;
    T.data = dst;
    T.dtype = CLE_F32;
    return minmax(T, mm->out, ws, st);
}

}  // namespace cle
