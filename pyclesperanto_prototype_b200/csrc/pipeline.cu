// pipeline.cu -- voronoi_otsu_labeling (_tier9/_voronoi_otsu_labeling.py:49-73) as one
// stream-ordered sequence with no host round trip:
//   O = gaussian_blur(src, outline_sigma), {min, max}   (blur_fused.cu, blur.cu)
//   histogram -> Otsu -> t32                      (reduce.cu, all on the device)
//   T = gaussian_blur(src, spot_sigma)            (O itself when the sigmas are equal)
//   seg = O > t32; seeds = detect_maxima_box(T) & seg   (maxima.cu, one pass; emits the
//                                                  seed list and the initial CCL keys;
//                                                  mean_box r=0 is a copy)
//   labels(seeds) = CCL                           (ccl.cu, list form)
//   labels = masked Voronoi growth inside seg     (voronoi_bricks.cu)
// The label output buffer is the CCL parent store and the Voronoi state, so
// the only full-size scratch is O (f32), seg (u8), the seed list and a tail the
// phases share: the blurs' temporaries, the spot blur, the growth's lists.
#include "common.cuh"
#include "kernels.cuh"

namespace cle {

namespace {

struct Scalars {
    int status;
    uint32_t seed_count;
    uint32_t nlabels;        // labels of the last call (= its maximum label)
    uint32_t ccl_done;       // CTAs of the seed labelling that have finished
    uint32_t label_bricks;   // growth bricks that hold a label (growth over the whole image)
    uint32_t pad1;
    MinMaxState mm;          // of the outline blur
    float thr32;
    float pad;
    double thr;
    float hist[256];
};

// Seeds of masked_voronoi_labeling with a 0/1 mask: seg = mask != 0,
// seed = binary != 0 inside the mask; seeds get their CCL key and are listed.
template <typename Tb, typename Tm>
__global__ void mask_seeds_kernel(const Tb *__restrict__ bin, const Tm *__restrict__ mask, Geo g,
                                  int64_t n, uint8_t *__restrict__ seg, uint32_t *__restrict__ lab,
                                  uint32_t *__restrict__ seeds, uint32_t *__restrict__ d_count) {
    const int lane = threadIdx.x & 31;
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < n;
         base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = base + threadIdx.x;
        bool seed = false;
        if (i < n) {
            const bool s = mask[i] != (Tm)0;
            seed = s && bin[i] != (Tb)0;
            uint32_t key = 0;
            if (seed) {
                uint32_t x, y, z;
                m2xyz(g, (uint32_t)i, x, y, z);
                key = xyz2k(g, x, y, z) + 1u;
            }
            seg[i] = s ? kMaskByte : 0;
            lab[i] = key;
        }
        const unsigned b = __ballot_sync(0xffffffffu, seed);
        if (b) {
            uint32_t base_pos = 0;
            const int leader = __ffs(b) - 1;
            if (lane == leader) base_pos = atomicAdd(d_count, (uint32_t)__popc(b));
            base_pos = __shfl_sync(0xffffffffu, base_pos, leader);
            if (seed) seeds[base_pos + __popc(b & ((1u << lane) - 1u))] = (uint32_t)i;
        }
    }
}

__global__ void u32_to_f32(const uint32_t *__restrict__ s, float *__restrict__ d, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        d[i] = (float)s[i];
}

struct Layout {
    Scalars *sc;
    float *O;
    uint8_t *seg;
    uint32_t *seeds;
    size_t fixed_end;
};

Layout take_layout(Arena &a, const Img &im) {
    Layout l;
    l.sc = a.take<Scalars>(1);
    l.O = a.take<float>(im.n());
    l.seg = a.take<uint8_t>(im.n());
    l.seeds = a.take<uint32_t>(im.n());
    l.fixed_end = a.off;
    return l;
}

struct BinLayout {
    Scalars *sc;
    uint8_t *seg;
    uint32_t *seeds;
    uint32_t *lab;   // used when the destination is float32
};

BinLayout take_bin_layout(Arena &a, const Img &im) {
    BinLayout l;
    l.sc = a.take<Scalars>(1);
    l.seg = a.take<uint8_t>(im.n());
    l.seeds = a.take<uint32_t>(im.n());
    l.lab = a.take<uint32_t>(im.n());
    return l;
}

template <typename Tb>
int launch_mask_seeds(const Img &bin, const Img &mask, const Geo &g, const BinLayout &l,
                      uint32_t *lab, cudaStream_t st) {
    const int64_t n = bin.n();
    const int b = launch_blocks(n, 256);
    switch (mask.dtype) {
        case CLE_U8: mask_seeds_kernel<Tb, uint8_t><<<b, 256, 0, st>>>((const Tb *)bin.data, (const uint8_t *)mask.data, g, n, l.seg, lab, l.seeds, &l.sc->seed_count); break;
        case CLE_F32: mask_seeds_kernel<Tb, float><<<b, 256, 0, st>>>((const Tb *)bin.data, (const float *)mask.data, g, n, l.seg, lab, l.seeds, &l.sc->seed_count); break;
        case CLE_U32: mask_seeds_kernel<Tb, uint32_t><<<b, 256, 0, st>>>((const Tb *)bin.data, (const uint32_t *)mask.data, g, n, l.seg, lab, l.seeds, &l.sc->seed_count); break;
        default: set_error("masked_voronoi_labeling: unsupported mask dtype %d", mask.dtype); return CLE_ERR_DTYPE;
    }
    CLE_LAUNCH_CHECK("mask seeds");
    return CLE_OK;
}

}  // namespace

size_t masked_voronoi_binary_workspace_bytes(const Img &im) {
    Arena a(nullptr, 0);
    take_bin_layout(a, im);
    size_t tail = std::max(rank_workspace_bytes(fkey_bits_for(im.n())), voronoi_grow_workspace_bytes(im));
    return a.off + tail;
}

int masked_voronoi_binary(const Img &bin, const Img &mask, const Img &dst, Arena &ws, cudaStream_t st,
                          const Limits &lim) {
    CLE_TRY(same_shape(bin, mask, "binary_source", "mask_image"));
    CLE_TRY(same_shape(bin, dst, "binary_source", "labeling_destination"));
    if (dst.dtype != CLE_U32 && dst.dtype != CLE_F32) {
        set_error("masked_voronoi_labeling: destination must be uint32 or float32");
        return CLE_ERR_DTYPE;
    }
    BinLayout l = take_bin_layout(ws, bin);
    const size_t tail_off = ws.off;
    if (!ws.measuring && ws.cap < masked_voronoi_binary_workspace_bytes(bin)) {
        set_error("masked_voronoi_labeling: workspace too small");
        return CLE_ERR_WORKSPACE;
    }
    CLE_CUDA(cudaMemsetAsync(l.sc, 0, sizeof(Scalars), st));
    uint32_t *lab = dst.dtype == CLE_U32 ? (uint32_t *)dst.data : l.lab;
    const Geo g = make_geo(bin);
    switch (bin.dtype) {
        case CLE_U8: CLE_TRY(launch_mask_seeds<uint8_t>(bin, mask, g, l, lab, st)); break;
        case CLE_F32: CLE_TRY(launch_mask_seeds<float>(bin, mask, g, l, lab, st)); break;
        case CLE_U32: CLE_TRY(launch_mask_seeds<uint32_t>(bin, mask, g, l, lab, st)); break;
        default: set_error("masked_voronoi_labeling: unsupported binary dtype %d", bin.dtype); return CLE_ERR_DTYPE;
    }
    CLE_TRY(ccl_list(g, bin.n(), lab, l.seeds, &l.sc->seed_count, bin.n(), ws, st, &l.sc->nlabels,
                     &l.sc->ccl_done, true));
    ws.off = tail_off;
    CLE_TRY(voronoi_grow(bin, lab, l.seg, l.seeds, &l.sc->seed_count, &l.sc->nlabels, &l.sc->status, ws, st,
                         lim));
    if (dst.dtype == CLE_F32) {
        u32_to_f32<<<launch_blocks(dst.n(), 256), 256, 0, st>>>(lab, (float *)dst.data, dst.n());
        CLE_LAUNCH_CHECK("labels to f32");
    }
    return CLE_OK;
}

// ---- extend_labeling_via_voronoi / voronoi_labeling -------------------------
// _tier4/_extend_labeling_via_voronoi.py:13-60: the labels (uint32, any values)
// grow into every zero voxel with the onlyzero_overwrite_maximum box/diamond
// Jacobi steps until a step changes nothing -- the key growth with a mask that
// covers the whole image (labels above 2^24 - 1 and paths above its step range
// take the brick growth behind it).  1024 x 1024 with a spot per 33 x 33 pixels:
// 0.80 ms with the brick growth (two grid barriers a step), 0.27 now.  voronoi_labeling (_tier5/_voronoi_labeling.py:
// 8-40) is connected_components_labeling_box followed by that growth.
namespace {

template <typename T>
__global__ void to_labels_kernel(const T *__restrict__ src, uint32_t *__restrict__ lab, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const T v = src[i];
        uint32_t o;
        if constexpr (std::is_floating_point<T>::value)   // clij_convert_uint_sat
            o = !(v > (T)0) ? 0u : (v >= (T)4294967295.0 ? 0xFFFFFFFFu : (uint32_t)v);
        else if constexpr (std::is_signed<T>::value)
            o = v < (T)0 ? 0u : (uint32_t)v;
        else
            o = (uint32_t)v;
        lab[i] = o;
    }
}

constexpr int kSeedWarps = 8;

// One seed voxel per 8-voxel row segment (x aligned to 8) that holds a label;
// the segment lies in one growth brick (8 x by 4 y, BZ z), so the 3x3x3 brick
// neighbourhood of the seed's brick covers every voxel next to a label of the
// segment.  A warp takes four bricks side by side, all of its rows loaded first.
// Also the mask bytes (arrival step 0 on labels, not yet known elsewhere), the
// largest label and the number of bricks that hold a label.  A few global
// atomics per CTA.
template <int BZ>
__global__ void __launch_bounds__(kSeedWarps * 32)
brick_seeds_kernel(const uint32_t *__restrict__ lab, uint8_t *__restrict__ seg, uint32_t D, uint32_t H, uint32_t W, uint32_t nx,
                   FastDiv fnx, FastDiv fny, uint32_t n, uint32_t *__restrict__ seeds, Scalars *__restrict__ sc) {
    constexpr int ROWS = kBrickY * BZ;
    __shared__ uint32_t s_n, s_base, s_max, s_bricks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_max = s_bricks = 0u;
    for (uint32_t base = blockIdx.x * kSeedWarps; base < n; base += gridDim.x * kSeedWarps) {
        if (threadIdx.x == 0) s_n = 0;
        __syncthreads();
        const uint32_t b = base + warp;
        uint32_t held = 0, pos = 0;   // segments with a label (a row per bit; lanes 0, 8, 16, 24), their place in the CTA's
        uint32_t v[ROWS], at = 0;
        if (b < n) {
            const uint32_t r = fnx.div(b), xb = b - r * nx, zb = fny.div(r), yb = r - zb * fny.d;
            const uint32_t x = xb * 32u + (uint32_t)lane, y0 = yb * kBrickY, z0 = zb * BZ;
            at = (z0 * H + y0) * W + x;
            uint32_t most = 0;
#pragma unroll
            for (int k = 0; k < ROWS; ++k) {
                const bool in = x < W && y0 + k % kBrickY < H && z0 + k / kBrickY < D;
                v[k] = in ? lab[at + ((uint32_t)(k / kBrickY) * H + (uint32_t)(k % kBrickY)) * W] : 0u;
                most = max(most, v[k]);
            }
#pragma unroll
            for (int k = 0; k < ROWS; ++k) {
                if (x < W && y0 + k % kBrickY < H && z0 + k / kBrickY < D)
                    seg[at + ((uint32_t)(k / kBrickY) * H + (uint32_t)(k % kBrickY)) * W] = v[k] ? (uint8_t)0x80 : kMaskByte;
                const unsigned bal = __ballot_sync(0xffffffffu, v[k] != 0u);
                if ((lane & 7) == 0 && (bal >> lane & 0xFFu)) held |= 1u << k;
            }
            most = __reduce_max_sync(0xffffffffu, most);
            const unsigned bricks = __ballot_sync(0xffffffffu, held != 0u);
            if (lane == 0 && most) {
                atomicMax(&s_max, most);
                atomicAdd(&s_bricks, (uint32_t)__popc(bricks));
            }
            if (held) pos = atomicAdd(&s_n, (uint32_t)__popc(held));
        }
        __syncthreads();
        if (threadIdx.x == 0) s_base = s_n ? atomicAdd(&sc->seed_count, s_n) : 0u;
        __syncthreads();
        if (b < n) {
            uint32_t *out = seeds + s_base + pos;
#pragma unroll
            for (int k = 0; k < ROWS; ++k) {
                const unsigned bal = __ballot_sync(0xffffffffu, v[k] != 0u) >> (lane & 24);
                if (held >> k & 1u) *out++ = at + ((uint32_t)(k / kBrickY) * H + (uint32_t)(k % kBrickY)) * W + (uint32_t)__ffs(bal & 0xFFu) - 1u;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_max) {
        atomicMax(&sc->nlabels, s_max);
        atomicAdd(&sc->label_bricks, s_bricks);
    }
}

struct ExtLayout {
    Scalars *sc;
    uint8_t *seg;
    uint32_t *seeds;
    uint32_t *lab;    // used when the destination is float32
};

ExtLayout take_ext_layout(Arena &a, const Img &im) {
    ExtLayout l;
    l.sc = a.take<Scalars>(1);
    l.seg = a.take<uint8_t>(im.n());
    l.seeds = a.take<uint32_t>((im.n() + 7) / 8 + (size_t)(im.D * im.H));
    l.lab = a.take<uint32_t>(im.n());
    return l;
}

// Grows `lab` in place over the whole image; status in l.sc.
int grow_everywhere(const Img &im, uint32_t *lab, ExtLayout &l, Arena &tail, cudaStream_t st,
                    const Limits &lim) {
    const int bz = im.ndim == 3 ? kBrickZ : 1;
    const uint32_t nx = (uint32_t)((im.W + 31) / 32), ny = (uint32_t)((im.H + kBrickY - 1) / kBrickY);
    const uint32_t n = nx * ny * (uint32_t)((im.D + bz - 1) / bz);
    auto kern = im.ndim == 3 ? brick_seeds_kernel<kBrickZ> : brick_seeds_kernel<1>;
    kern<<<launch_blocks((int64_t)n * 32, kSeedWarps * 32), kSeedWarps * 32, 0, st>>>(
        lab, l.seg, (uint32_t)im.D, (uint32_t)im.H, (uint32_t)im.W, nx, FastDiv(nx), FastDiv(ny), n, l.seeds, l.sc);
    CLE_LAUNCH_CHECK("brick seeds");
    return voronoi_grow(im, lab, l.seg, l.seeds, &l.sc->seed_count, &l.sc->nlabels, &l.sc->status, tail, st, lim,
                        &l.sc->label_bricks);
}

}  // namespace

size_t extend_voronoi_workspace_bytes(const Img &im) {
    Arena a(nullptr, 0);
    take_ext_layout(a, im);
    const size_t tail = std::max(ccl_workspace_bytes(im), voronoi_grow_workspace_bytes(im));
    return a.off + tail;
}

int extend_labeling_via_voronoi(const Img &src, const Img &dst, Arena &ws, cudaStream_t st,
                                const Limits &lim) {
    CLE_TRY(same_shape(src, dst, "labeling_source", "labeling_destination"));
    if (dst.dtype != CLE_U32 && dst.dtype != CLE_F32) {
        set_error("extend_labeling_via_voronoi: destination must be uint32 or float32");
        return CLE_ERR_DTYPE;
    }
    ExtLayout l = take_ext_layout(ws, src);
    if (!ws.measuring && ws.cap < extend_voronoi_workspace_bytes(src)) {
        set_error("extend_labeling_via_voronoi: workspace too small");
        return CLE_ERR_WORKSPACE;
    }
    CLE_CUDA(cudaMemsetAsync(l.sc, 0, sizeof(Scalars), st));
    uint32_t *lab = dst.dtype == CLE_U32 ? (uint32_t *)dst.data : l.lab;
    const int64_t n = src.n();
    const int b = launch_blocks(n, 256);
    switch (src.dtype) {
        case CLE_U8: to_labels_kernel<uint8_t><<<b, 256, 0, st>>>((const uint8_t *)src.data, lab, n); break;
        case CLE_U16: to_labels_kernel<uint16_t><<<b, 256, 0, st>>>((const uint16_t *)src.data, lab, n); break;
        case CLE_U32:
            if (src.data != (void *)lab) to_labels_kernel<uint32_t><<<b, 256, 0, st>>>((const uint32_t *)src.data, lab, n);
            break;
        case CLE_I32: to_labels_kernel<int32_t><<<b, 256, 0, st>>>((const int32_t *)src.data, lab, n); break;
        case CLE_F32: to_labels_kernel<float><<<b, 256, 0, st>>>((const float *)src.data, lab, n); break;
        default: set_error("extend_labeling_via_voronoi: unsupported source dtype %d", src.dtype); return CLE_ERR_DTYPE;
    }
    CLE_LAUNCH_CHECK("labels");
    CLE_TRY(grow_everywhere(src, lab, l, ws, st, lim));
    if (dst.dtype == CLE_F32) {
        u32_to_f32<<<launch_blocks(n, 256), 256, 0, st>>>(lab, (float *)dst.data, n);
        CLE_LAUNCH_CHECK("labels to f32");
    }
    return CLE_OK;
}

int voronoi_labeling(const Img &bin, const Img &dst, Arena &ws, cudaStream_t st, const Limits &lim) {
    CLE_TRY(same_shape(bin, dst, "binary_source", "labeling_destination"));
    if (dst.dtype != CLE_U32 && dst.dtype != CLE_F32) {
        set_error("voronoi_labeling: destination must be uint32 or float32");
        return CLE_ERR_DTYPE;
    }
    ExtLayout l = take_ext_layout(ws, bin);
    const size_t tail_off = ws.off;
    if (!ws.measuring && ws.cap < extend_voronoi_workspace_bytes(bin)) {
        set_error("voronoi_labeling: workspace too small");
        return CLE_ERR_WORKSPACE;
    }
    CLE_CUDA(cudaMemsetAsync(l.sc, 0, sizeof(Scalars), st));
    uint32_t *lab = dst.dtype == CLE_U32 ? (uint32_t *)dst.data : l.lab;
    CLE_TRY(ccl_dense(bin, lab, ws, st));
    ws.off = tail_off;
    CLE_TRY(grow_everywhere(bin, lab, l, ws, st, lim));
    if (dst.dtype == CLE_F32) {
        u32_to_f32<<<launch_blocks(dst.n(), 256), 256, 0, st>>>(lab, (float *)dst.data, dst.n());
        CLE_LAUNCH_CHECK("labels to f32");
    }
    return CLE_OK;
}

int *workspace_status_ptr(void *ws) { return &reinterpret_cast<Scalars *>(ws)->status; }
uint32_t *workspace_label_count_ptr(void *ws) { return &reinterpret_cast<Scalars *>(ws)->nlabels; }

size_t vol_workspace_bytes(const Img &im) {
    Arena a(nullptr, 0);
    take_layout(a, im);
    const size_t base = a.off;
    // phase-dependent tail (max over the phases that use it)
    size_t tail = 0;
    tail = std::max(tail, separable_workspace_bytes(im));
    tail = std::max(tail, minmax_workspace_bytes(im) + histogram_workspace_bytes(im, 256));
    tail = std::max(tail, separable_workspace_bytes(im) + minmax_workspace_bytes(im));
    tail = std::max(tail, rank_workspace_bytes(fkey_bits_for(im.n())));
    tail = std::max(tail, voronoi_grow_workspace_bytes(im));
    // 17 bytes per voxel are used (O 4, mask 1, seeds 4, the phases' tail 8); the
    // query answers at least 18, its lower bound since the maxima image was scratch too
    return std::max(base + tail, (18 * (size_t)im.n() + 255) & ~(size_t)255);
}

int voronoi_otsu_labeling(const Img &src, const Img &dst, double spot_sigma, double outline_sigma,
                          Arena &ws, cudaStream_t st, const Limits &lim) {
    CLE_TRY(same_shape(src, dst, "source", "label_image_destination"));
    if (dst.dtype != CLE_U32 && dst.dtype != CLE_F32) {
        set_error("voronoi_otsu_labeling: destination must be uint32 or float32 (got %d)", dst.dtype);
        return CLE_ERR_DTYPE;
    }
    Layout l = take_layout(ws, src);
    const size_t tail_off = ws.off;
    if (!ws.ok() || (!ws.measuring && ws.cap < vol_workspace_bytes(src))) {
        set_error("voronoi_otsu_labeling: workspace too small (%zu < %zu)", ws.cap, vol_workspace_bytes(src));
        return CLE_ERR_WORKSPACE;
    }
    const int64_t n = src.n();
    stage_mark(0, st);
    CLE_CUDA(cudaMemsetAsync(l.sc, 0, sizeof(Scalars), st));

    // 1: the outline blur with its min / max (temporaries in the tail), 2: the
    // threshold, on the device
    CLE_TRY(blur_minmax(src, l.O, outline_sigma, &l.sc->mm, ws, st, &l.sc->status));
    ws.off = tail_off;
    stage_mark(1, st);
    Img Oi = src;
    Oi.data = l.O;
    Oi.dtype = CLE_F32;
    CLE_TRY(histogram_otsu(Oi, l.sc->mm.out, l.sc->hist, &l.sc->thr, &l.sc->thr32, ws, st));
    ws.off = tail_off;
    stage_mark(2, st);

    // 3: the spot blur.  The two blurs build their taps from the float32 sigma
    // and the kernel size int(8 sigma)|1, so equal float32 sigmas with equal
    // kernel sizes give the same image bit for bit: then the outline blur serves
    // both the spot detection and the threshold.  Otherwise the spot blur goes to
    // the tail: to the second of the three-pass blur's temporaries in 2D (its
    // last pass reads the first) and to the first in 3D (it reads the second).
    const bool same_blur = (float)spot_sigma == (float)outline_sigma &&
                           sigma_to_kernel_size(spot_sigma) == sigma_to_kernel_size(outline_sigma);
    Img Ti = Oi;
    if (!same_blur) {
        float *t1 = ws.take<float>(n), *t2 = ws.take<float>(n);
        ws.off = tail_off;
        Ti.data = src.ndim == 3 ? t1 : t2;
        CLE_TRY(gaussian_blur(src, (float *)Ti.data, spot_sigma, spot_sigma, spot_sigma, ws, st, &l.sc->status));
        ws.off = tail_off;
    }
    stage_mark(3, st);

    // 4: segmentation, maxima, seeds, seed keys
    uint32_t *lab = (dst.dtype == CLE_U32) ? (uint32_t *)dst.data : (uint32_t *)l.O;
    const Geo g = make_geo(src);
    const float *O = l.O;
    if (dst.dtype == CLE_F32) {
        // the labels are built in O's buffer; the seed pass reads a copy in dst
        CLE_CUDA(cudaMemcpyAsync(dst.data, l.O, sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
        O = (const float *)dst.data;
        if (same_blur) Ti.data = dst.data;
    }
    CLE_TRY(maxima_seeds(Ti, O, &l.sc->thr32, l.seg, lab, l.seeds, &l.sc->seed_count, st));
    stage_mark(4, st);

    // 5: label the seeds
    CLE_TRY(ccl_list(g, n, lab, l.seeds, &l.sc->seed_count, n, ws, st, &l.sc->nlabels,
                     &l.sc->ccl_done));
    ws.off = tail_off;
    stage_mark(5, st);

    // 6: grow inside the segmentation
    CLE_TRY(voronoi_grow(src, lab, l.seg, l.seeds, &l.sc->seed_count, &l.sc->nlabels, &l.sc->status, ws, st,
                         lim));
    ws.off = tail_off;
    stage_mark(6, st);
    stage_mark(7, st);

    if (dst.dtype == CLE_F32) {
        u32_to_f32<<<launch_blocks(n, 256), 256, 0, st>>>(lab, (float *)dst.data, n);
        CLE_LAUNCH_CHECK("labels to f32");
    }
    return CLE_OK;
}

// ---- gauss_otsu_labeling ------------------------------------------------------
// _tier9/_gauss_otsu_labeling.py:6-45: blur with its min / max, histogram, Otsu,
// connected components of what lies above the threshold.  The labelling compares
// as it loads and the blur reduces as it stores, so the binary image and the pass
// for the extremes are gone: 128 x 1024 x 1024 uint16, sigma 2: 1.46 -> 1.32 ms.
namespace {

struct DenseLayout {
    Scalars *sc;
    float *O;
};

DenseLayout take_dense_layout(Arena &a, const Img &im) {
    DenseLayout l;
    l.sc = a.take<Scalars>(1);
    l.O = a.take<float>(im.n());
    return l;
}

}  // namespace

size_t gauss_otsu_workspace_bytes(const Img &im) {
    Arena a(nullptr, 0);
    take_dense_layout(a, im);
    const size_t tail = std::max(separable_workspace_bytes(im) + minmax_workspace_bytes(im),
                                 std::max(histogram_workspace_bytes(im, 256), ccl_workspace_bytes(im)));
    return a.off + tail;
}

int gauss_otsu_labeling(const Img &src, const Img &dst, double sigma, Arena &ws, cudaStream_t st) {
    CLE_TRY(same_shape(src, dst, "source", "label_image_destination"));
    if (dst.dtype != CLE_U32 && dst.dtype != CLE_F32) {
        set_error("gauss_otsu_labeling: destination must be uint32 or float32");
        return CLE_ERR_DTYPE;
    }
    DenseLayout l = take_dense_layout(ws, src);
    const size_t tail_off = ws.off;
    if (!ws.ok()) { set_error("gauss_otsu_labeling: workspace too small"); return CLE_ERR_WORKSPACE; }
    CLE_CUDA(cudaMemsetAsync(l.sc, 0, sizeof(Scalars), st));
    // the call returns without a word that its caller would have to read, so a blur
    // whose copies did not arrive is made again
    CLE_TRY(blur_minmax(src, l.O, sigma, &l.sc->mm, ws, st, &l.sc->status, true));
    ws.off = tail_off;
    Img Oi = src;
    Oi.data = l.O;
    Oi.dtype = CLE_F32;
    CLE_TRY(histogram_otsu(Oi, l.sc->mm.out, l.sc->hist, &l.sc->thr, &l.sc->thr32, ws, st));
    ws.off = tail_off;
    uint32_t *lab = ws.take<uint32_t>(dst.n());
    if (dst.dtype == CLE_U32) lab = (uint32_t *)dst.data;
    CLE_TRY(ccl_dense(Oi, lab, ws, st, false, &l.sc->thr32));
    return dst.dtype == CLE_F32 ? ccl_to_dst(lab, dst, st) : CLE_OK;
}

}  // namespace cle
