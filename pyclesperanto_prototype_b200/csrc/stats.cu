// stats.cu -- statistics_of_labelled_pixels
// (_tier9/_statistics_of_labelled_pixels.py:7-293, kernels
// _tier9/statistics_per_label_x.cl:1-146, _tier9/standard_deviation_per_label_x.cl:1-96).
//
// Brick reductions: a warp takes a brick of 32 x 8 x 4 voxels (32 x 32 in images),
// every lane a column of 32 voxels in registers, all loads issued at once.  A
// label image is made of compact objects, so a brick holds a few labels: for
// each of them the warp builds every lane's bit mask of matching voxels (the
// coordinate sums and the bounding box are popcounts and bit scans of it), sums
// the intensities, reduces over the lanes and adds the result to the label's
// accumulators, one record, with four atomic instructions.  Where labels are tiny
// (kWorth) the voxels are added by themselves, those that touch along a lane's
// column together.  A label
// that fills half a brick (the background, where it counts as one) is carried
// along in registers from brick to brick.  Two passes, as in the reference (the
// second needs the per-label centroid, mass centre and mean); the second takes
// the labels and masks the first kept, at most kMaxLabels of a brick (3.1 bytes per
// voxel of scratch; images thinner than a brick in some direction keep at least one
// label of each, up to 32 bytes per voxel where a brick holds 4), and does not read
// the label image for those.  Coordinates and 8/16-bit intensities are summed in
// exact 64-bit integers (exact_sums), other intensities in float64; min / max through
// order-preserving unsigned atomics.  The finalise kernels apply the reference's
// float32 column arithmetic and its sentinels for labels absent from the image
// (min FLT_MAX, max -FLT_MAX, sums 0, 0/0 = NaN).
// 512 x 1024 x 1024 uint16, 22% of the voxels in 38000 labels: pass 1 0.87 ms (integer
// pipe 73% busy; 0.49 at copy bandwidth), pass 2 0.74 ms (issue 71%: two exact
// square roots and three float64 sums a voxel).  The sorted form before it
// (voxel indices scattered into label order, then swept) took 2.31 and 0.67 ms.
// 128 x 512 x 512 full of blocks of 3 x 3 x 3, uint16 / float32: 2.07 / 2.24 ms (sorted 2.40 / 2.42; with
// an atomic set per voxel beyond the kept labels 3.22 / 3.30); 5 x 5 x 5 1.05 / 1.36 (1.18 / 1.29); 4 x 4 x 4
// 0.70 / 0.93 (1.38 / 1.40); 2 x 2 x 2 3.44 / 3.15 (4.80 / 4.77); a random label per voxel 3.67 (3.30).
#include <cfloat>

#include "common.cuh"
#include "kernels.cuh"

namespace cle {

namespace {

constexpr int kST = 256;
constexpr int kMaxLabels = 24;   // labels of a brick kept for pass 2 (fewer in thin images)
// Labels are reduced over the warp while they average kWorth voxels of the brick
// (looked at from kTryLabels on): a reduction costs what adding that many voxels
// by themselves does, more for float64 sums.  The largest labels come first, so a
// background that counts as label 1 comes last: with kTryLabels = 4 a few slivers of
// cells sent it to its single voxels (2048 x 1024 float32, 3600 cells of 24 pixels and a
// background: pass 2 20 -> 31 us).
constexpr uint32_t kTryLabels = 16, kWorthInt = 6, kWorthFloat = 12;

// Accumulators of a label: pass 1 ...
struct alignas(32) Acc1 {
    unsigned long long s[4];   // sums of x, y, z, voxel count
    union {                    // sums of intensity, intensity * x, * y, * z
        double v[4];
        unsigned long long u[4];   // (exact: see exact_sums)
    };
    uint32_t lo[4], hi[4];     // smallest / largest x, y, z, ordered intensity
};
// ... and pass 2, with the label's centre and mean (pc) and mass centre and area (pm)
struct alignas(32) Acc2 {
    double s[3];               // distances to centroid, to mass centre, squared deviations
    uint32_t m[2];             // largest distances (bits of non-negative float32)
    float4 pc, pm;
};

// With a device label count (d_L) the init and finalise kernels touch only the
// first min(count, L) labels; L stays the table's row stride.
__device__ __forceinline__ int64_t live_labels(int64_t L, const uint32_t *d_L) {
    return d_L ? ((int64_t)*d_L < L ? (int64_t)*d_L : L) : L;
}

__global__ void stats_init(Acc1 *__restrict__ a, Acc2 *__restrict__ b, int64_t L, const uint32_t *__restrict__ d_L) {
    const int64_t n = live_labels(L, d_L);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        Acc1 &A = a[i];
        Acc2 &B = b[i];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            A.s[k] = 0ull;
            A.v[k] = 0.0;
            A.lo[k] = 0xFFFFFFFFu;
            A.hi[k] = 0u;
        }
        B.s[0] = B.s[1] = B.s[2] = 0.0;
        B.m[0] = B.m[1] = 0u;
    }
}

template <typename T>
__device__ __forceinline__ uint32_t lab_of(T v) {
    if constexpr (std::is_floating_point<T>::value) return v > (T)0 ? (uint32_t)(int64_t)v : 0u;
    else return (uint32_t)v;
}

// Run of equal labels along x inside a warp's 32 voxels: head lane, and
// whether this lane ends its run.
struct Run {
    int head;
    bool tail;
};

__device__ __forceinline__ Run make_run(uint32_t l) {
    const int lane = threadIdx.x & 31;
    const uint32_t lp = __shfl_up_sync(0xffffffffu, l, 1);
    const bool hd = (lane == 0) || (l != lp);
    const unsigned heads = __ballot_sync(0xffffffffu, hd);
    const unsigned upto = (lane == 31) ? 0xffffffffu : ((2u << lane) - 1u);
    Run r;
    r.head = 31 - __clz(heads & upto);
    r.tail = (lane == 31) || ((heads >> (lane + 1)) & 1u);
    return r;
}

// Label of one voxel, 0 for background and for labels above the live count.
template <typename TL>
__device__ __forceinline__ uint32_t live_label(const TL *lab, int64_t m, int64_t L) {
    const uint32_t l = lab_of(lab[m]);
    return (l > (uint32_t)L) ? 0u : l;
}

constexpr int kBatch = 4;   // row segments per warp round (loads in flight)

// Sums of four values over the warp; lane l gets that of value l % 4.  The first two
// steps halve what a lane carries: 6 exchanges instead of 20.
__device__ __forceinline__ double warp_sum4(double a, double b, double c, double d) {
    const int lane = threadIdx.x & 31;
    const bool odd = lane & 1, high = lane & 2;
    double p = odd ? b : a, q = odd ? d : c;
    p += __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
    q += __shfl_xor_sync(0xffffffffu, odd ? c : d, 1);
    double r = high ? q : p;
    r += __shfl_xor_sync(0xffffffffu, high ? p : q, 2);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    return r;
}
// Distances of a voxel to its label's centroid and mass centre in float32
// (relative error a few 1e-7) and its intensity's deviation from the mean; the
// squared deviations are divided by the area once per label.
__device__ __forceinline__ void voxel_moments(const float4 &pc, const float4 &pm, float x, float y, float z, float v,
                                              float &dc, float &dm, double &dv) {
    const float ex = x - pc.x, ey = y - pc.y, ez = z - pc.z;
    const float fx = x - pm.x, fy = y - pm.y, fz = z - pm.z;
    dc = sqrtf(ex * ex + ey * ey + ez * ez);
    dm = sqrtf(fx * fx + fy * fy + fz * fz);
    dv = (double)v - (double)pc.w;
}

// Bricks of the image: 32 x by BY y by BZ z, column voxel k at y = k % BY, z = k / BY.
struct Bricks {
    uint32_t D, H, W, n;       // image, bricks
    uint32_t nx, ny;
    FastDiv fnx, fny;
    uint32_t slots;            // labels of a brick that are kept (below)
};

// What pass 1 keeps of the bricks for pass 2: the labels found and every lane's
// bit mask of matching voxels.
struct Found {
    uint8_t *count;            // labels kept of a brick; kMore: and voxels of others
    uint32_t *label;           // [brick][slots]
    uint32_t *mask;            // [brick][slots][32]
};
constexpr uint32_t kMore = 0x80u;

// A label's sums over bricks: lane k < 4 holds entry k of each group of Acc1.
template <bool INT>
struct Sums {
    unsigned long long s;
    typename std::conditional<INT, unsigned long long, double>::type v;
    uint32_t lo, hi;
    __device__ __forceinline__ void merge(const Sums &o) {
        s += o.s;
        v += o.v;
        lo = min(lo, o.lo);
        hi = max(hi, o.hi);
    }
    __device__ __forceinline__ void add_to(Acc1 *a, bool exact) const {
        const int lane = threadIdx.x & 31;
        if (lane < 4) {
            atomicAdd(a->s + lane, s);
            if (INT && exact) atomicAdd(a->u + lane, (unsigned long long)v);
            else atomicAdd(a->v + lane, (double)v);
            atomicMin(a->lo + lane, lo);
            atomicMax(a->hi + lane, hi);
        }
    }
};

// lane k's entry of four warp-uniform values
template <typename T>
__device__ __forceinline__ T lane4(T a, T b, T c, T d) {
    const int lane = threadIdx.x & 31;
    return lane & 2 ? (lane & 1 ? d : c) : (lane & 1 ? b : a);
}

// What a lane has of a label in its column of the brick.
template <bool INT>
struct Column {
    typename std::conditional<INT, unsigned long long, double>::type v, vy, vz;
    uint32_t n, sy, sz, ylo, yhi, zlo, zhi, vlo, vhi;
    __device__ __forceinline__ void clear() {
        v = vy = vz = 0;
        n = sy = sz = yhi = zhi = vhi = 0u;
        ylo = zlo = vlo = 0xFFFFFFFFu;
    }
    template <typename TI>
    __device__ __forceinline__ void add(uint32_t y, uint32_t z, TI w) {
        const float f = to_f32(w);
        const uint32_t o = f2u(f);
        ++n;
        sy += y;
        sz += z;
        if constexpr (INT) {
            v += (unsigned long long)w;
            vy += (unsigned long long)w * y;
            vz += (unsigned long long)w * z;
        } else {
            v += (double)f;
            vy += (double)f * (double)y;
            vz += (double)f * (double)z;
        }
        ylo = min(ylo, y); yhi = max(yhi, y);
        zlo = min(zlo, z); zhi = max(zhi, z);
        vlo = min(vlo, o); vhi = max(vhi, o);
    }
    __device__ __forceinline__ void add_to(Acc1 *a, uint32_t x, bool exact) const {
        // bounds that the record holds already need no atomic (they only widen, so
        // an older value is as good)
        const uint4 lo = *reinterpret_cast<const uint4 *>(a->lo), hi = *reinterpret_cast<const uint4 *>(a->hi);
        atomicAdd(a->s, (unsigned long long)n * x);
        atomicAdd(a->s + 1, (unsigned long long)sy);
        atomicAdd(a->s + 2, (unsigned long long)sz);
        atomicAdd(a->s + 3, (unsigned long long)n);
        if (INT && exact) {
            atomicAdd(a->u, (unsigned long long)v);
            atomicAdd(a->u + 1, (unsigned long long)v * x);
            atomicAdd(a->u + 2, (unsigned long long)vy);
            atomicAdd(a->u + 3, (unsigned long long)vz);
        } else {
            atomicAdd(a->v, (double)v);
            atomicAdd(a->v + 1, (double)v * (double)x);
            atomicAdd(a->v + 2, (double)vy);
            atomicAdd(a->v + 3, (double)vz);
        }
        if (x < lo.x) atomicMin(a->lo, x);
        if (ylo < lo.y) atomicMin(a->lo + 1, ylo);
        if (zlo < lo.z) atomicMin(a->lo + 2, zlo);
        if (vlo < lo.w) atomicMin(a->lo + 3, vlo);
        if (x > hi.x) atomicMax(a->hi, x);
        if (yhi > hi.y) atomicMax(a->hi + 1, yhi);
        if (zhi > hi.z) atomicMax(a->hi + 2, zhi);
        if (vhi > hi.w) atomicMax(a->hi + 3, vhi);
    }
};

// Pass 1 over the voxels of the bricks.
template <typename TL, typename TI, int BY>
__global__ void __launch_bounds__(kST, 2)
brick_sums_kernel(const TL *__restrict__ lab, const TI *__restrict__ inten, Bricks G, int64_t Lcap,
                  const uint32_t *__restrict__ d_L, Acc1 *__restrict__ a1, Found F, bool exact) {
    constexpr int BZ = 32 / BY;
    constexpr bool INT = sizeof(TI) <= 2 && !std::is_floating_point<TI>::value;
    const uint32_t L = (uint32_t)live_labels(Lcap, d_L);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nwarps = gridDim.x * (kST / 32);
    Sums<INT> carry;
    uint32_t carried = 0;      // label of `carry`
    // warp-uniform brick index: row addresses stay on the uniform datapath
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    for (uint32_t b = blockIdx.x * (kST / 32) + warp; b < G.n; b += nwarps) {
        const uint32_t r = G.fnx.div(b), bx = b - r * G.nx, bz = G.fny.div(r), by = r - bz * G.ny;
        const uint32_t x = bx * 32u + lane, y0 = by * BY, z0 = bz * BZ;
        const uint32_t HW = G.H * G.W, at = z0 * HW + y0 * G.W + bx * 32u;   // the brick's first voxel
        uint32_t l[32];
        bool some = false;
        if (bx * 32u + 32u <= G.W && y0 + BY <= G.H && z0 + BZ <= G.D) {
            const TL *pz = lab + at + lane, *p = pz;
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                l[k] = lab_of(__ldg(p));
                if (k % BY == BY - 1) p = pz += HW;
                else p += G.W;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                const bool in = x < G.W && y0 + k % BY < G.H && z0 + k / BY < G.D;
                l[k] = in ? lab_of(__ldg(lab + at + (uint32_t)(k / BY) * HW + (uint32_t)(k % BY) * G.W + lane)) : 0u;
            }
        }
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            if (l[k] > L) l[k] = 0u;
            some |= l[k] != 0u;
        }
        if (!__any_sync(0xffffffffu, some)) {
            if (lane == 0) F.count[b] = 0;
            continue;
        }
        TI v[32];
        {
            const TI *pz = inten + at + lane, *p = pz;
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                v[k] = l[k] ? __ldg(p) : TI(0);
                if (k % BY == BY - 1) p = pz += HW;
                else p += G.W;
            }
        }
        uint32_t found = 0, covered = 0, more = 0;   // labels, their voxels
        for (;;) {
            // the largest label left in the brick
            uint32_t g = 0;
#pragma unroll
            for (int k = 0; k < 32; ++k) g = max(g, l[k]);
            g = __reduce_max_sync(0xffffffffu, g);
            if (g == 0u) break;
            if (found >= kTryLabels && covered < (INT ? kWorthInt : kWorthFloat) * found) {
                // many tiny labels: the voxels left are added by themselves, those that
                // follow one another in a lane's column together.  (From the registers:
                // a rolled loop that reads the labels again makes the compiler's code of
                // the whole kernel worse, 0.66 against 0.62 ms on sparse labels.)
                more = kMore;
                Column<INT> c;
                c.clear();
#pragma unroll
                for (int k = 0; k < 32; ++k) {
                    if (l[k] == 0u) continue;
                    c.add(y0 + k % BY, z0 + k / BY, v[k]);
                    if (k == 31 || l[k < 31 ? k + 1 : 31] != l[k]) {
                        c.add_to(a1 + (l[k] - 1u), x, exact);
                        c.clear();
                    }
                }
                break;
            }
            Sums<INT> t;
            uint32_t mine = 0;                     // this lane's voxels of label g
            uint32_t vmin = 0xFFFFFFFFu, vmax = 0u;
            uint32_t iv = 0, ivy = 0, ivz = 0;      // 8/16-bit: a brick's sums fit 32 bits
            double dvy = 0.0, dplane[BZ] = {};      // others: per plane, so that z costs nothing per voxel
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                if (l[k] == g) {
                    l[k] = 0u;
                    mine |= 1u << k;
                    if constexpr (INT) {
                        const uint32_t u = (uint32_t)v[k];
                        iv += u;
                        ivy += u * (uint32_t)(k % BY);
                        ivz += u * (uint32_t)(k / BY);
                        vmin = min(vmin, u);
                        vmax = max(vmax, u);
                    } else {
                        const float f = to_f32(v[k]);
                        const double d = (double)f;
                        dplane[k / BY] += d;
                        dvy += d * (double)(y0 + k % BY);
                        vmin = min(vmin, f2u(f));
                        vmax = max(vmax, f2u(f));
                    }
                }
            }
            // sums of k % BY and k / BY over the bits of `mine`
            uint32_t ky = 0, kz = 0;
#pragma unroll
            for (int i = 0; (1 << i) < 32; ++i) {
                uint32_t pat = 0;
#pragma unroll
                for (int k = 0; k < 32; ++k) pat |= ((uint32_t)(k >> i) & 1u) << k;
                if ((1 << i) < BY) ky += (uint32_t)__popc(mine & pat) << i;
                else kz += (uint32_t)__popc(mine & pat) << i;
            }
            kz /= (uint32_t)BY;
            const uint32_t n = (uint32_t)__popc(mine);
            const uint32_t N = __reduce_add_sync(0xffffffffu, n);
            covered += N;
            const unsigned long long xb = bx * 32u;
            {
                const uint32_t sx = __reduce_add_sync(0xffffffffu, n * lane);
                const uint32_t sy = __reduce_add_sync(0xffffffffu, ky), sz = __reduce_add_sync(0xffffffffu, kz);
                t.s = lane4(sx, sy, sz, N) + lane4<unsigned long long>(xb, y0, z0, 0) * N;
            }
            uint32_t lo3, hi3;
            if constexpr (INT) {
                const uint32_t V = __reduce_add_sync(0xffffffffu, iv), Vx = __reduce_add_sync(0xffffffffu, iv * lane);
                const uint32_t Vy = __reduce_add_sync(0xffffffffu, ivy), Vz = __reduce_add_sync(0xffffffffu, ivz);
                t.v = lane4(V, Vx, Vy, Vz) + lane4<unsigned long long>(0, xb, y0, z0) * V;
                lo3 = f2u((float)__reduce_min_sync(0xffffffffu, vmin));
                hi3 = f2u((float)__reduce_max_sync(0xffffffffu, vmax));
            } else {
                // lanes without a voxel of the label add nothing (0 x infinity would)
                double dv = 0.0, dvz = 0.0;
#pragma unroll
                for (int j = 0; j < BZ; ++j) {
                    dv += dplane[j];
                    dvz += dplane[j] * (double)(z0 + j);
                }
                t.v = warp_sum4(dv, mine ? dv * (double)x : 0.0, dvy, dvz);
                lo3 = __reduce_min_sync(0xffffffffu, vmin);
                hi3 = __reduce_max_sync(0xffffffffu, vmax);
            }
            // bounding box: columns (lanes) and the bits of any column
            const unsigned cols = __ballot_sync(0xffffffffu, mine != 0u);
            const uint32_t rows = __reduce_or_sync(0xffffffffu, mine);
            uint32_t ym = 0, zm = 0;
#pragma unroll
            for (int j = 0; j < BZ; ++j) {
                const uint32_t part = BY == 32 ? rows : (rows >> (j * BY)) & ((1u << (BY & 31)) - 1u);
                ym |= part;
                zm |= (part ? 1u : 0u) << j;
            }
            t.lo = lane4(bx * 32u + (uint32_t)__ffs(cols) - 1u, y0 + (uint32_t)__ffs(ym) - 1u, z0 + (uint32_t)__ffs(zm) - 1u, lo3);
            t.hi = lane4(bx * 32u + 31u - (uint32_t)__clz(cols), y0 + 31u - (uint32_t)__clz(ym), z0 + 31u - (uint32_t)__clz(zm), hi3);
            if (g == carried) {
                carry.merge(t);
            } else if (N >= 512u && (!INT || exact)) {
                if (carried) carry.add_to(a1 + (carried - 1u), exact);
                carry = t;
                carried = g;
            } else {
                t.add_to(a1 + (g - 1u), exact);
            }
            if (found < G.slots) {
                F.mask[((size_t)b * G.slots + found) * 32u + lane] = mine;
                if (lane == 0) F.label[(size_t)b * G.slots + found] = g;
            }
            ++found;
        }
        if (lane == 0) F.count[b] = (uint8_t)(min(found, G.slots) | (found > G.slots ? kMore : more));
    }
    if (carried) carry.add_to(a1 + (carried - 1u), exact);
}

// Pass 2 over the labels found in the bricks: the label's voxels are packed
// into a list from the masks, so that every lane works, and their intensities
// gathered; the label image itself is not read again.
template <typename TL, typename TI, int BY>
__global__ void __launch_bounds__(kST, 6)
brick_moments_kernel(const TL *__restrict__ lab, const TI *__restrict__ inten, Bricks G, int64_t Lcap,
                     const uint32_t *__restrict__ d_L, Acc2 *__restrict__ a2, Found F) {
    constexpr int BZ = 32 / BY;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nwarps = gridDim.x * (kST / 32);
    __shared__ uint16_t s_list[kST / 32][1024];
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    uint16_t *list = s_list[warp];
    for (uint32_t b = blockIdx.x * (kST / 32) + warp; b < G.n; b += nwarps) {
        const uint32_t found = F.count[b];
        if (!found) continue;
        const uint32_t r = G.fnx.div(b), bx = b - r * G.nx, bz = G.fny.div(r), by = r - bz * G.ny;
        const uint32_t y0 = by * BY, z0 = bz * BZ, HW = G.H * G.W, at = z0 * HW + y0 * G.W + bx * 32u;
        uint32_t seen = 0;
        for (uint32_t j = 0; j < (found & ~kMore); ++j) {
            const uint32_t g = __ldg(F.label + (size_t)b * G.slots + j);
            uint32_t mine = __ldg(F.mask + ((size_t)b * G.slots + j) * 32u + lane);
            const float4 pc = a2[g - 1u].pc, pm = a2[g - 1u].pm;
            seen |= mine;
            // the label's voxels packed into a list, so that every lane works
            const uint32_t n = (uint32_t)__popc(mine);
            uint32_t pos = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, pos, o);
                if (lane >= (uint32_t)o) pos += y;
            }
            const uint32_t N = __shfl_sync(0xffffffffu, pos, 31);
            pos -= n;
            for (; mine; mine &= mine - 1u) list[pos++] = (uint16_t)(((uint32_t)__ffs(mine) - 1u) * 32u + lane);
            __syncwarp();
            double sdc = 0.0, sdm = 0.0, ssq = 0.0;
            float mdc = 0.0f, mdm = 0.0f;
            // the next entry's intensity is on its way while one is computed
            auto entry = [&](uint32_t i, uint32_t &c, TI &w) {
                c = list[min(i, N - 1u)];
                const uint32_t k = c >> 5;
                w = __ldg(inten + at + (k / BY) * HW + (k % BY) * G.W + (c & 31u));
            };
            uint32_t c;
            TI w;
            entry(lane, c, w);
#pragma unroll 1
            for (uint32_t i = lane; i < N; i += 32u) {
                uint32_t cn;
                TI wn;
                entry(i + 32u, cn, wn);
                const uint32_t k = c >> 5;
                float dc, dm;
                double dv;
                voxel_moments(pc, pm, (float)(bx * 32u + (c & 31u)), (float)(y0 + k % BY), (float)(z0 + k / BY),
                              to_f32(w), dc, dm, dv);
                sdc += (double)dc;
                sdm += (double)dm;
                ssq += dv * dv;
                mdc = fmaxf(mdc, dc);
                mdm = fmaxf(mdm, dm);
                c = cn;
                w = wn;
            }
            __syncwarp();
            const double S = warp_sum4(sdc, sdm, ssq, 0.0);
            const uint32_t M0 = __reduce_max_sync(0xffffffffu, __float_as_uint(mdc));
            const uint32_t M1 = __reduce_max_sync(0xffffffffu, __float_as_uint(mdm));
            Acc2 *a = a2 + (g - 1u);
            if (lane < 3) atomicAdd(a->s + lane, S);
            if (lane < 2) atomicMax(a->m + lane, lane == 0 ? M0 : M1);
        }
        if (found & kMore) {
            // voxels of labels that were not kept: what touches along a lane's column
            // is added at once
            const uint32_t L = (uint32_t)live_labels(Lcap, d_L), x = bx * 32u + lane;
            uint32_t of = 0;   // label at hand
            float4 pc = make_float4(0.f, 0.f, 0.f, 0.f), pm = pc;
            double sdc = 0.0, sdm = 0.0, ssq = 0.0;
            float mdc = 0.0f, mdm = 0.0f;
            auto flush = [&]() {
                Acc2 *a = a2 + (of - 1u);
                const uint2 m = *reinterpret_cast<const uint2 *>(a->m);   // only grow: an older value is as good
                atomicAdd(a->s, sdc);
                atomicAdd(a->s + 1, sdm);
                atomicAdd(a->s + 2, ssq);
                if (__float_as_uint(mdc) > m.x) atomicMax(a->m, __float_as_uint(mdc));
                if (__float_as_uint(mdm) > m.y) atomicMax(a->m + 1, __float_as_uint(mdm));
            };
#pragma unroll 1
            for (int k = 0; k < 32; ++k) {
                const uint32_t y = y0 + k % BY, z = z0 + k / BY, m = at + (uint32_t)(k / BY) * HW + (uint32_t)(k % BY) * G.W + lane;
                uint32_t g = 0;
                if (!(seen >> k & 1u) && x < G.W && y < G.H && z < G.D) g = lab_of(__ldg(lab + m));
                if (g > L) g = 0u;
                if (g != of) {
                    if (of) flush();
                    sdc = sdm = ssq = 0.0;
                    mdc = mdm = 0.0f;
                    of = g;
                    if (g) {
                        pc = a2[g - 1u].pc;
                        pm = a2[g - 1u].pm;
                    }
                }
                if (g) {
                    float dc, dm;
                    double dv;
                    voxel_moments(pc, pm, (float)x, (float)y, (float)z, to_f32(__ldg(inten + m)), dc, dm, dv);
                    sdc += (double)dc;
                    sdm += (double)dm;
                    ssq += dv * dv;
                    mdc = fmaxf(mdc, dc);
                    mdm = fmaxf(mdm, dm);
                }
            }
            if (of) flush();
        }
    }
}

// Row indices of the table (the reference's dict order after label columns).
enum {
    C_BBOX_MIN_X, C_BBOX_MIN_Y, C_BBOX_MIN_Z, C_BBOX_MAX_X, C_BBOX_MAX_Y, C_BBOX_MAX_Z,
    C_BBOX_W, C_BBOX_H, C_BBOX_D, C_MIN_I, C_MAX_I, C_SUM_I, C_AREA, C_MEAN_I,
    C_SUM_IX, C_MASS_X, C_SUM_IY, C_MASS_Y, C_SUM_IZ, C_MASS_Z,
    C_SUM_X, C_CEN_X, C_SUM_Y, C_CEN_Y, C_SUM_Z, C_CEN_Z,
    C_SUM_DC, C_MEAN_DC, C_SUM_DM, C_MEAN_DM, C_STD_I, C_MAX_DC, C_MAX_DM,
    C_RATIO_C, C_RATIO_M, C_NCOLS
};
static_assert(C_NCOLS == CLE_STATS_NCOLS, "table width");

__global__ void stats_final1(const Acc1 *__restrict__ a, Acc2 *__restrict__ b, int64_t L, float *__restrict__ T, const uint32_t *__restrict__ d_L, bool exact) {
    const int64_t n = live_labels(L, d_L);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const Acc1 &A = a[i];
        const bool any = A.s[3] != 0ull;
        const float area = (float)A.s[3];
        auto total = [&](int k) { return exact ? (float)A.u[k] : (float)A.v[k]; };
        const float sum_i = total(0);
        auto put = [&](int c, float v) { T[(int64_t)c * L + i] = v; };
        const float bx0 = any ? (float)A.lo[0] : FLT_MAX, bx1 = any ? (float)A.hi[0] : -FLT_MAX;
        const float by0 = any ? (float)A.lo[1] : FLT_MAX, by1 = any ? (float)A.hi[1] : -FLT_MAX;
        const float bz0 = any ? (float)A.lo[2] : FLT_MAX, bz1 = any ? (float)A.hi[2] : -FLT_MAX;
        put(C_BBOX_MIN_X, bx0); put(C_BBOX_MIN_Y, by0); put(C_BBOX_MIN_Z, bz0);
        put(C_BBOX_MAX_X, bx1); put(C_BBOX_MAX_Y, by1); put(C_BBOX_MAX_Z, bz1);
        put(C_BBOX_W, __fadd_rn(__fsub_rn(bx1, bx0), 1.0f));
        put(C_BBOX_H, __fadd_rn(__fsub_rn(by1, by0), 1.0f));
        put(C_BBOX_D, __fadd_rn(__fsub_rn(bz1, bz0), 1.0f));
        put(C_MIN_I, any ? u2f(A.lo[3]) : FLT_MAX);
        put(C_MAX_I, any ? u2f(A.hi[3]) : -FLT_MAX);
        put(C_SUM_I, sum_i);
        put(C_AREA, area);
        const float mean = __fdiv_rn(sum_i, area);
        put(C_MEAN_I, mean);
        const float six = total(1), siy = total(2), siz = total(3);
        const float mxc = __fdiv_rn(six, sum_i), myc = __fdiv_rn(siy, sum_i), mzc = __fdiv_rn(siz, sum_i);
        put(C_SUM_IX, six); put(C_MASS_X, mxc);
        put(C_SUM_IY, siy); put(C_MASS_Y, myc);
        put(C_SUM_IZ, siz); put(C_MASS_Z, mzc);
        const float sx = (float)A.s[0], sy = (float)A.s[1], sz = (float)A.s[2];
        const float cx = __fdiv_rn(sx, area), cy = __fdiv_rn(sy, area), cz = __fdiv_rn(sz, area);
        put(C_SUM_X, sx); put(C_CEN_X, cx);
        put(C_SUM_Y, sy); put(C_CEN_Y, cy);
        put(C_SUM_Z, sz); put(C_CEN_Z, cz);
        b[i].pc = make_float4(cx, cy, cz, mean);
        b[i].pm = make_float4(mxc, myc, mzc, area);
    }
}

__global__ void stats_final2(const Acc2 *__restrict__ b, int64_t L, float *__restrict__ T, const uint32_t *__restrict__ d_L) {
    const int64_t n = live_labels(L, d_L);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        auto put = [&](int c, float v) { T[(int64_t)c * L + i] = v; };
        const Acc2 &B = b[i];
        const float area = B.pm.w;
        const float sdc = (float)B.s[0], sdm = (float)B.s[1];
        const float mdc = __fdiv_rn(sdc, area), mdm = __fdiv_rn(sdm, area);
        const float xdc = __uint_as_float(B.m[0]);
        const float xdm = __uint_as_float(B.m[1]);
        put(C_SUM_DC, sdc); put(C_MEAN_DC, mdc);
        put(C_SUM_DM, sdm); put(C_MEAN_DM, mdm);
        // sum of squared deviations / area (0 for a label absent from the image)
        put(C_STD_I, (float)sqrt(area > 0.0f ? B.s[2] / (double)area : B.s[2]));
        put(C_MAX_DC, xdc); put(C_MAX_DM, xdm);
        put(C_RATIO_C, __fdiv_rn(xdc, mdc));
        put(C_RATIO_M, __fdiv_rn(xdm, mdm));
    }
}

// ---- centroids of labels (the point list, no second pass) ------------------
// Per row run of label l (1..n): the voxel count and the exact 64-bit sums of
// its x, y and z (x from the run's first voxel in closed form), added once per
// run; then centroid = float32(sum) / float32(count), the division the
// statistics table uses for centroid_x/y/z.
template <typename TL>
__global__ void __launch_bounds__(kST)
centroid_sums_kernel(const TL *__restrict__ lab, uint32_t W, uint32_t H, uint32_t tasks, FastDiv fc,
                     int64_t n, uint32_t *__restrict__ cnt, unsigned long long *__restrict__ sums) {
    const int lane = threadIdx.x & 31;
    const uint32_t chunks = fc.d;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t t0 = warp; t0 < tasks; t0 += kBatch * nwarps) {
        uint32_t lb[kBatch], rb[kBatch], xb[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const uint32_t t = t0 + (uint32_t)k * nwarps;
            const uint32_t row = fc.div(t), x = (t - row * chunks) * 32u + (uint32_t)lane;
            rb[k] = row;
            xb[k] = x;
            lb[k] = (t < tasks && x < W) ? live_label(lab, (int64_t)row * W + x, n) : 0u;
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const uint32_t l = lb[k];
            if (__ballot_sync(0xffffffffu, l != 0u) == 0u) continue;
            const Run r = make_run(l);
            if (r.tail && l) {
                const unsigned long long len = (unsigned long long)(lane - r.head + 1);
                const unsigned long long x0 = xb[k] - (uint32_t)(lane - r.head);
                const uint32_t y = rb[k] % H, z = rb[k] / H;
                const int64_t i = (int64_t)l - 1;
                atomicAdd(cnt + i, (uint32_t)len);
                atomicAdd(sums + 3 * i, len * x0 + len * (len - 1) / 2);
                atomicAdd(sums + 3 * i + 1, len * y);
                atomicAdd(sums + 3 * i + 2, len * z);
            }
        }
    }
}

__global__ void centroid_final_kernel(const uint32_t *__restrict__ cnt, const unsigned long long *__restrict__ sums,
                                      int64_t n, int dims, float *__restrict__ pts) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float area = (float)cnt[i];
        for (int d = 0; d < dims; ++d) pts[d * n + i] = __fdiv_rn((float)sums[3 * i + d], area);
    }
}

struct StatsWs {
    Acc1 *a1;
    Acc2 *a2;
    Found found;
};

Bricks make_bricks(const Img &im) {
    Bricks G;
    const uint32_t by = im.D > 1 ? 8 : 32, bz = 32 / by;
    G.D = (uint32_t)im.D;
    G.H = (uint32_t)im.H;
    G.W = (uint32_t)im.W;
    G.nx = (G.W + 31) / 32;
    G.ny = (G.H + by - 1) / by;
    G.n = G.nx * G.ny * ((G.D + bz - 1) / bz);
    G.fnx = FastDiv(G.nx);
    G.fny = FastDiv(G.ny);
    // kMaxLabels in full bricks (3.1 bytes per voxel), fewer where the image is
    // thinner than a brick
    G.slots = (uint32_t)std::max<int64_t>(1, kMaxLabels * im.n() / ((int64_t)G.n * 1024));
    return G;
}

StatsWs take_stats(Arena &a, const Img &labels, int64_t L) {
    StatsWs w;
    w.a1 = a.take<Acc1>(L);
    w.a2 = a.take<Acc2>(L);
    const Bricks G = make_bricks(labels);
    w.found.count = a.take<uint8_t>(G.n);
    w.found.label = a.take<uint32_t>((size_t)G.n * G.slots);
    w.found.mask = a.take<uint32_t>((size_t)G.n * G.slots * 32u);
    return w;
}

// Intensity totals of 8/16-bit sources are kept in 64-bit integers wherever their
// largest possible value fits (any image of up to 2^31 voxels with sides up to 65536);
// in float64 they pass 2^53 from a label of 16 bits, full scale, in 512 x 1024 x 1024 on,
// and further sums round in the order they arrive.
template <typename TI>
bool exact_sums(const Img &im) {
    if (sizeof(TI) > 2) return false;
    const double most = sizeof(TI) == 1 ? 255.0 : 65535.0;
    return most * (double)im.n() * (double)std::max(im.W, std::max(im.H, im.D)) < 1.8e19;
}

template <typename TL, typename TI, int BY>
int stats_typed(const Img &inten, const Img &lab, int64_t L, float *T, const StatsWs &w, cudaStream_t st,
                const uint32_t *d_L) {
    const Bricks G = make_bricks(lab);
    const int blocks = launch_blocks((int64_t)G.n * 32, kST, 4);
    const bool exact = exact_sums<TI>(lab);
    stage_mark(8, st);
    brick_sums_kernel<TL, TI, BY><<<blocks, kST, 0, st>>>((const TL *)lab.data, (const TI *)inten.data, G, L, d_L,
                                                          w.a1, w.found, exact);
    stage_mark(9, st);
    stats_final1<<<launch_blocks(L, 256), 256, 0, st>>>(w.a1, w.a2, L, T, d_L, exact);
    stage_mark(10, st);
    brick_moments_kernel<TL, TI, BY><<<launch_blocks((int64_t)G.n * 32, kST, 16), kST, 0, st>>>(
        (const TL *)lab.data, (const TI *)inten.data, G, L, d_L, w.a2, w.found);
    stage_mark(11, st);
    stats_final2<<<launch_blocks(L, 256), 256, 0, st>>>(w.a2, L, T, d_L);
    stage_mark(12, st);
    CLE_LAUNCH_CHECK_N("statistics", 4);
    return CLE_OK;
}

template <typename TL, typename TI>
int stats_dims(const Img &inten, const Img &lab, int64_t L, float *T, const StatsWs &w, cudaStream_t st,
               const uint32_t *d_L) {
    return lab.D > 1 ? stats_typed<TL, TI, 8>(inten, lab, L, T, w, st, d_L)
                     : stats_typed<TL, TI, 32>(inten, lab, L, T, w, st, d_L);
}

template <typename TL>
int stats_i(const Img &inten, const Img &lab, int64_t L, float *T, const StatsWs &w, cudaStream_t st,
            const uint32_t *d_L) {
    switch (inten.dtype) {
        case CLE_F32: return stats_dims<TL, float>(inten, lab, L, T, w, st, d_L);
        case CLE_U16: return stats_dims<TL, uint16_t>(inten, lab, L, T, w, st, d_L);
        case CLE_U8: return stats_dims<TL, uint8_t>(inten, lab, L, T, w, st, d_L);
        case CLE_U32: return stats_dims<TL, uint32_t>(inten, lab, L, T, w, st, d_L);
        default: set_error("statistics: unsupported intensity dtype %d", inten.dtype); return CLE_ERR_DTYPE;
    }
}

}  // namespace

size_t stats_workspace_bytes(const Img &labels, int64_t L) {
    Arena a(nullptr, 0);
    take_stats(a, labels, L < 1 ? 1 : L);
    return a.off;
}

int statistics(const Img &inten, const Img &lab, int64_t L, float *T, Arena &ws, cudaStream_t st,
               const uint32_t *d_L) {
    CLE_TRY(same_shape(inten, lab, "intensity_image", "label_image"));
    if (L < 0 || L > 0x7FFFFFFF) { set_error("statistics: bad label count %lld", (long long)L); return CLE_ERR_ARG; }
    if (L == 0) return CLE_OK;
    const StatsWs w = take_stats(ws, lab, L);
    if (!ws.ok()) { set_error("statistics: workspace too small"); return CLE_ERR_WORKSPACE; }
    stats_init<<<launch_blocks(L, 256), 256, 0, st>>>(w.a1, w.a2, L, d_L);
    CLE_LAUNCH_CHECK("statistics init");
    switch (lab.dtype) {
        case CLE_U32: return stats_i<uint32_t>(inten, lab, L, T, w, st, d_L);
        case CLE_F32: return stats_i<float>(inten, lab, L, T, w, st, d_L);
        case CLE_U16: return stats_i<uint16_t>(inten, lab, L, T, w, st, d_L);
        case CLE_U8: return stats_i<uint8_t>(inten, lab, L, T, w, st, d_L);
        default: set_error("statistics: unsupported label dtype %d", lab.dtype); return CLE_ERR_DTYPE;
    }
}

size_t centroids_workspace_bytes(int64_t n) {
    Arena a(nullptr, 0);
    a.take<uint32_t>(n);
    a.take<unsigned long long>(3 * n);
    return a.off;
}

int label_centroids(const Img &lab, int64_t n, float *pts, Arena &ws, cudaStream_t st) {
    if (n < 0 || n > 0x7FFFFFFF) { set_error("centroids: bad label count %lld", (long long)n); return CLE_ERR_ARG; }
    if (n == 0) return CLE_OK;
    uint32_t *cnt = ws.take<uint32_t>(n);
    unsigned long long *sums = ws.take<unsigned long long>(3 * n);
    if (!ws.ok()) { set_error("centroids: workspace too small"); return CLE_ERR_WORKSPACE; }
    CLE_CUDA(cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * n, st));
    CLE_CUDA(cudaMemsetAsync(sums, 0, sizeof(unsigned long long) * 3 * n, st));
    const int64_t rows = lab.D * lab.H;
    const int64_t tasks = rows * ((lab.W + 31) / 32);
    if (tasks > 0xFFFFFFFFll) { set_error("centroids: image too large"); return CLE_ERR_TOO_LARGE; }
    const int blocks = launch_blocks(tasks * 32, kST, 8);
    const FastDiv fc((uint32_t)((lab.W + 31) / 32));
    switch (lab.dtype) {
        case CLE_U32:
            centroid_sums_kernel<uint32_t><<<blocks, kST, 0, st>>>((const uint32_t *)lab.data, (uint32_t)lab.W,
                                                                 (uint32_t)lab.H, (uint32_t)tasks, fc, n, cnt, sums);
            break;
        case CLE_F32:
            centroid_sums_kernel<float><<<blocks, kST, 0, st>>>((const float *)lab.data, (uint32_t)lab.W,
                                                              (uint32_t)lab.H, (uint32_t)tasks, fc, n, cnt, sums);
            break;
        default: set_error("centroids: unsupported label dtype %d", lab.dtype); return CLE_ERR_DTYPE;
    }
    centroid_final_kernel<<<launch_blocks(n, 256), 256, 0, st>>>(cnt, sums, n, lab.ndim == 3 ? 3 : 2, pts);
    CLE_LAUNCH_CHECK_N("centroids", 2);
    return CLE_OK;
}

}  // namespace cle
