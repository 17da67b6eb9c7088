// ccl.cu -- connected_components_labeling_box and relabel_sequential.
//
// Reference semantics (_tier4/_connected_components_labeling_box.py:39-64):
// every foreground voxel starts with its pixel-index key K+1 held in float32
// (set_nonzero_pixels_to_pixelindex, key x-major: K = (x*H + y)*D + z,
// tests/test_set_nonzero_pixels_to_pixelindex.py), Jacobi min-propagation
// over the 3^d box until stable, then relabel_sequential ranks the distinct
// float32 values (_tier3/_relabel_sequential.py:42-57).  So a component's
// label is the rank of float32(min K + 1) among all components, and
// components whose float32 keys round to the same value share a label.
//
// Here: union-find, in tiles for dense masks (below); for small dense masks and
// for a list of seeds the parent pointers are K values (stored as K+1 in the u32 label
// buffer, 0 = background), linked with atomicMin so every root is its
// component's minimum key.  The distinct float32 keys of the components are
// marked in a bitmap over integer-valued floats (fkey_index) and ranked with
// a per-word popcount prefix.  No N-sized float vectors, no host round trips.
#include "common.cuh"
#include "kernels.cuh"

namespace cle {

namespace {

constexpr int kT = 256;

__device__ __forceinline__ uint32_t find_root(const uint32_t *lab, const Geo &g, uint32_t k) {
    uint32_t p = ld_cg(lab + k2m(g, k)) - 1u;
    while (p != k) {
        k = p;
        p = ld_cg(lab + k2m(g, k)) - 1u;
    }
    return k;
}

// find_root with path halving, for the union phase: a visited non-root
// entry is lowered to its grandparent with atomicMin.  Entries only ever move
// to an ancestor in the same tree and roots are never touched, so concurrent
// unions (which link roots only) are unaffected.
__device__ __forceinline__ uint32_t find_root_halve(uint32_t *lab, const Geo &g, uint32_t k) {
    uint32_t mk = k2m(g, k);
    uint32_t p = ld_cg(lab + mk) - 1u;
    while (p != k) {
        const uint32_t mp = k2m(g, p);
        const uint32_t gp = ld_cg(lab + mp) - 1u;
        if (gp == p) return p;
        atomicMin(lab + mk, gp + 1u);
        k = gp;
        mk = k2m(g, k);
        p = ld_cg(lab + mk) - 1u;
    }
    return k;
}

__device__ __forceinline__ void unite(uint32_t *lab, const Geo &g, uint32_t a, uint32_t b) {
    for (;;) {
        a = find_root_halve(lab, g, a);
        b = find_root_halve(lab, g, b);
        if (a == b) return;
        if (a < b) { uint32_t t = a; a = b; b = t; }
        // link root a (larger key) under b
        uint32_t old = atomicMin(lab + k2m(g, a), b + 1u) - 1u;
        if (old == a) return;
        a = old;
    }
}

// Unions voxel (x,y,z) (foreground) with its 13 memory-order predecessors.
__device__ __forceinline__ void union_back(uint32_t *lab, const Geo &g, uint32_t x, uint32_t y,
                                           uint32_t z) {
    const uint32_t kp = xyz2k(g, x, y, z);
#pragma unroll
    for (int dz = -1; dz <= 0; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                if (dz == 0 && (dy > 0 || (dy == 0 && dx >= 0))) continue;
                const int qz = (int)z + dz, qy = (int)y + dy, qx = (int)x + dx;
                if (qz < 0 || qy < 0 || qy >= (int)g.H || qx < 0 || qx >= (int)g.W) continue;
                const uint32_t v = ld_cg(lab + xyz2m(g, qx, qy, qz));
                if (v) unite(lab, g, kp, xyz2k(g, qx, qy, qz));
            }
}

// ---- dense labelling in tiles ----------------------------------------------
// Union-find over the voxels in global memory waits for a chain of L2 loads at
// every union, a few lanes of a warp at a time (134M voxels, 7.5% foreground: 2.66 ms
// for the unions alone, 3.7 ms in all).  Here a CTA first labels a tile of rows in
// shared memory, where a find step takes a few tens of cycles and each thread
// works on a row of its own: a row of 32 voxels is a bit mask, its runs are the
// nodes (named by their first voxel), and the contacts of two rows are bit
// expressions.  Every component of a tile gets a compact id from a device
// counter; only the contacts across tile faces are united in global memory, on
// the ids' parent array, and the row masks say where those lie without reading
// the labels.  The smallest x-major key of a component is kept per id.  Then
// labels cost one gather per foreground voxel.  0.62 ms for the volume above
// (128 x 1024 x 1024): tiles 0.36, faces 0.11, ranks 0.08, labels 0.07; the tiles are
// bound by instruction issue (66%) and the barriers between their phases, the
// pass over the image alone (read 1, write 4 bytes per voxel) is 0.10.
constexpr int kTileThreads = 256;

// Row pairs in contact: the neighbour rows before a row in memory order.
//   k = 0: (y - 1, z)   1: (y - 1, z - 1)   2: (y, z - 1)   3: (y + 1, z - 1)
__host__ __device__ __forceinline__ int row_dy(int k) { return k == 0 ? -1 : k - 2; }
__host__ __device__ __forceinline__ int row_dz(int k) { return k == 0 ? 0 : -1; }

struct Tiles {
    uint32_t nx, ny, nz;   // tiles along x, y, z
    FastDiv fnx, fny;
    uint32_t ws;           // 32-voxel segments per row (= nx)
};

// First voxel of the run of m that holds bit i.
__device__ __forceinline__ uint32_t run_start(uint32_t m, uint32_t i) {
    const uint32_t below = ~m & ((1u << i) - 1u);
    return below ? 32u - (uint32_t)__clz(below) : 0u;
}

__device__ __forceinline__ uint32_t find_plain(volatile uint32_t *p, uint32_t i) {
    uint32_t q = p[i];
    while (q != i) {
        i = q;
        q = p[i];
    }
    return i;
}

// find_plain that hangs every other node of its path from its grandparent.  Only
// nodes that are no roots are written, and only with an ancestor of theirs, so
// a union that is under way elsewhere (which links roots) loses nothing.  In
// shared memory it shortens the chains of random masks (128 x 512 x 512, half
// foreground, whole call: 2.27 -> 1.51 ms; smooth objects 0.53 -> 0.50); on the ids' array in
// global memory its stores get in each other's way (smooth objects 0.50 -> 0.80).
__device__ __forceinline__ uint32_t find_halving(volatile uint32_t *p, uint32_t i) {
    for (;;) {
        const uint32_t q = p[i];
        if (q == i) return i;
        const uint32_t g = p[q];
        if (g == q) return q;
        p[i] = g;
        i = g;
    }
}

// Unites a and b in a forest whose parents are never larger than their nodes.
template <bool HALVING>
__device__ __forceinline__ void unite_plain(uint32_t *p, uint32_t a, uint32_t b) {
    for (;;) {
        a = HALVING ? find_halving(p, a) : find_plain(p, a);
        b = HALVING ? find_halving(p, b) : find_plain(p, b);
        if (a == b) return;
        if (a < b) { const uint32_t t = a; a = b; b = t; }
        const uint32_t old = atomicMin(p + a, b);
        if (old == a) return;
        a = old;
    }
}

// Calls u(i, j) for a set of contacts between bit i of row mask m and bit j of
// row mask q that joins every pair of touching runs: the first voxel of each
// overlap and, unless DIAMOND, contacts that are diagonal only.  `via` is a row
// next to both (below): a contact beside one of its voxels is left out.
// Only contacts of the bits `only` of m.
template <bool DIAMOND, typename U>
__device__ __forceinline__ void row_contacts(uint32_t m, uint32_t q, uint32_t via, uint32_t only, U u) {
    const uint32_t both = m & q;
    for (uint32_t s = both & ~(both << 1) & ~via & only; s; s &= s - 1u) {
        const uint32_t i = (uint32_t)__ffs(s) - 1u;
        u(i, i);
    }
    if constexpr (!DIAMOND) {
        for (uint32_t s = m & (q >> 1) & ~q & ~(m >> 1) & ~(via | via >> 1) & only; s; s &= s - 1u) {
            const uint32_t i = (uint32_t)__ffs(s) - 1u;
            u(i, i + 1u);
        }
        for (uint32_t s = m & (q << 1) & ~q & ~(m << 1) & ~(via | via << 1) & only; s; s &= s - 1u) {
            const uint32_t i = (uint32_t)__ffs(s) - 1u;
            u(i, i - 1u);
        }
    }
}

// Which contacts need no union because other unions imply them; q[k]: the
// masks of the neighbour rows.  With the box, rows 1 and 3 touch row 2 (united
// as row 0 of their plane), so a contact with them beside a voxel of row 2
// follows from the contact with row 2; a contact with row 2 beside a voxel of
// row 0 follows from row 0 and that row's contact with row 2 (its row 3).  With
// face connectivity, row 2 is reached over rows 0 and 1.  Contacts with row 0 are
// always united, and each implication leads to a smaller y, so none is
// circular.  Inside a solid object one union of four remains.
template <bool DIAMOND>
__device__ __forceinline__ uint32_t via_row(int k, const uint32_t (&q)[4]) {
    if (k == 0) return 0u;
    if (DIAMOND) return q[0] & q[1];
    return k == 2 ? q[0] : q[2];
}

// Foreground: what is not zero, or what lies above a threshold on the device (a
// blurred image is labelled without its binary image being written and read).
template <typename T>
struct NonZero {
    using Value = T;
    __device__ __forceinline__ bool operator()(T v) const { return v != T(0); }
};
struct Above {
    using Value = float;
    const float *threshold;
    __device__ __forceinline__ bool operator()(float v) const { return v > __ldg(threshold); }
};

// A tile of 32 x TY x TZ voxels per CTA: lab = compact id + 1 of the voxel's
// component in the tile (0: background), bits = the row masks, parent[id] = id,
// minkey[id] = the component's smallest key.
template <typename FG, int TY, int TZ, bool DIAMOND>
__global__ void __launch_bounds__(kTileThreads, 6)
ccl_tile_kernel(const typename FG::Value *bin, FG fg, uint32_t *lab, uint32_t *__restrict__ bits, uint32_t *__restrict__ parent,
                uint32_t *__restrict__ minkey, uint32_t *__restrict__ d_count, Geo g, Tiles t) {
    // PARTS threads per row: in volumes two share out the neighbour rows, and all
    // the 32 voxels
    constexpr int ROWS = TY * TZ, WARPS = kTileThreads / 32, RPW = ROWS / WARPS, PARTS = kTileThreads / ROWS;
    constexpr int KPARTS = TZ > 1 && !DIAMOND && PARTS > 1 ? 2 : 1, SPARTS = PARTS / KPARTS;
    static_assert(ROWS % WARPS == 0 && kTileThreads % ROWS == 0 && TY % RPW == 0, "rows per warp and threads per row");
    static_assert(PARTS % KPARTS == 0 && 32 % SPARTS == 0, "threads per row");
    __shared__ uint32_t par[ROWS * 32];
    __shared__ uint32_t key[ROWS * 32];
    __shared__ uint32_t mask[ROWS];
    __shared__ uint32_t s_cnt, s_base;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t tyz = t.fnx.div(blockIdx.x), tx = blockIdx.x - tyz * t.nx;
    const uint32_t tz = t.fny.div(tyz), ty = tyz - tz * t.ny;
    const uint32_t x = tx * 32u + lane;
    if (threadIdx.x == 0) s_cnt = 0u;
    // a warp's rows are consecutive y of one plane
    const uint32_t r0 = warp * RPW, z = tz * TZ + r0 / TY, y0 = ty * TY + r0 % TY;
    const uint32_t nrow = z < g.D && y0 < g.H ? min((uint32_t)RPW, g.H - y0) : 0u;   // rows inside the image
    const uint32_t at0 = (z * g.H + y0) * g.W + x, bit0 = (z * g.H + y0) * t.ws + tx;
    const bool xin = x < g.W;
    typename FG::Value v[RPW];
    bool in[RPW], some = false;
#pragma unroll
    for (int k = 0; k < RPW; ++k) {
        in[k] = (uint32_t)k < nrow && xin;
        v[k] = in[k] ? bin[at0 + (uint32_t)k * g.W] : 0;
    }
#pragma unroll
    for (int k = 0; k < RPW; ++k) {
        in[k] = in[k] && fg(v[k]);
        some |= in[k];
    }
    if (!__syncthreads_or(some)) {
        // nothing here (most tiles of a sparse mask)
#pragma unroll
        for (int k = 0; k < RPW; ++k) {
            if ((uint32_t)k < nrow && xin) lab[at0 + (uint32_t)k * g.W] = 0u;
            if ((uint32_t)k < nrow && lane == 0) bits[bit0 + (uint32_t)k * t.ws] = 0u;
        }
        return;
    }
    // row masks; the start of a run is a node of its own
    const uint32_t key0 = xyz2k(g, x, y0, z);
#pragma unroll
    for (int k = 0; k < RPW; ++k) {
        const uint32_t r = r0 + (uint32_t)k;
        const uint32_t m = __ballot_sync(0xffffffffu, in[k]);
        if (lane == 0) {
            mask[r] = m;
            if ((uint32_t)k < nrow) bits[bit0 + (uint32_t)k * t.ws] = m;
        }
        if ((m & ~(m << 1)) >> lane & 1u) {
            par[r * 32 + lane] = r * 32 + lane;
            key[r * 32 + lane] = key0 + (uint32_t)k * g.D;
        }
    }
    __syncthreads();
    const uint32_t row = threadIdx.x % ROWS, part = threadIdx.x / ROWS;
    const uint32_t m = mask[row];
    const int ly = (int)(row % TY), lz = (int)(row / TY);
    if (m) {
        const uint32_t kpart = part % KPARTS;
        const uint32_t only = SPARTS == 1 ? 0xFFFFFFFFu : ((1ull << (32 / SPARTS)) - 1u) << (part / KPARTS * (32 / SPARTS));
        uint32_t q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int qy = ly + row_dy(k), qz = lz + row_dz(k);
            q[k] = qy >= 0 && qy < TY && qz >= 0 ? mask[qz * TY + qy] : 0u;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (TZ == 1 && k > 0) continue;
            if (DIAMOND && (k == 1 || k == 3)) continue;
            if (KPARTS > 1 && (uint32_t)(k % KPARTS) != kpart) continue;
            const uint32_t qr = (uint32_t)((lz + row_dz(k)) * TY + ly + row_dy(k));
            row_contacts<DIAMOND>(m, q[k], via_row<DIAMOND>(k, q), only, [&](uint32_t i, uint32_t j) {
                unite_plain<true>(par, row * 32 + run_start(m, i), qr * 32 + run_start(q[k], j));
            });
        }
    }
    __syncthreads();
    // the components' smallest keys and how many there are
    const uint32_t starts = part == 0 ? m & ~(m << 1) : 0u;
    uint32_t nroot = 0;
    for (uint32_t s = starts; s; s &= s - 1u) {
        const uint32_t node = row * 32 + (uint32_t)__ffs(s) - 1u, root = find_plain(par, node);
        if (root == node) ++nroot;
        else atomicMin(key + root, key[node]);
    }
    uint32_t at = nroot ? atomicAdd(&s_cnt, nroot) : 0u;
    __syncthreads();
    if (threadIdx.x == 0 && s_cnt) s_base = atomicAdd(d_count, s_cnt);
    __syncthreads();
    // ids: the roots first (bit 31 marks an id; a find that meets one has it)
    for (uint32_t s = starts; s; s &= s - 1u) {
        const uint32_t node = row * 32 + (uint32_t)__ffs(s) - 1u;
        if (par[node] == node) {
            const uint32_t id = s_base + at++;
            parent[id] = id;
            minkey[id] = key[node];
            par[node] = 0x80000000u | id;
        }
    }
    __syncthreads();
    for (uint32_t s = starts; s; s &= s - 1u) {
        const uint32_t node = row * 32 + (uint32_t)__ffs(s) - 1u;
        uint32_t q = *(volatile uint32_t *)(par + node);
        while (!(q & 0x80000000u)) q = *(volatile uint32_t *)(par + q);
        *(volatile uint32_t *)(par + node) = q;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RPW; ++k) {
        const uint32_t r = r0 + (uint32_t)k, mr = mask[r];
        if ((uint32_t)k < nrow && xin)
            lab[at0 + (uint32_t)k * g.W] = (mr >> lane & 1u) ? (par[r * 32 + run_start(mr, lane)] & 0x7FFFFFFFu) + 1u : 0u;
    }
}

// Contacts across tile faces, a thread per row segment: whole rows where the
// neighbour row lies in another tile, the segment's two ends everywhere.
template <int TY, int TZ, bool DIAMOND>
__global__ void __launch_bounds__(kT)
ccl_merge_kernel(const uint32_t *__restrict__ lab, const uint32_t *__restrict__ bits, uint32_t *parent, Geo g,
                 Tiles t, FastDiv fws, uint32_t nseg) {
    const uint32_t sgm = blockIdx.x * kT + threadIdx.x;
    const uint32_t m = sgm < nseg ? bits[sgm] : 0u;
    if (!m) return;
    const uint32_t r = fws.div(sgm), xs = sgm - r * t.ws;   // r = z * H + y
    const uint32_t z = g.fH.div(r), y = r - z * g.H;
    const bool first = xs == 0u, last = xs + 1u == t.ws;
    const uint32_t mL = first ? 0u : bits[sgm - 1u], mR = last ? 0u : bits[sgm + 1u];
    const uint32_t *row = lab + (size_t)r * g.W + xs * 32u;
    // neighbouring contacts mostly join the same two components: the pair
    // united last is not walked again
    uint32_t la = 0u, lb = 0u;
    auto join = [&](const uint32_t *p, const uint32_t *q) {
        const uint32_t a = __ldg(p), b = __ldg(q);
        if (a == la && b == lb) return;
        la = a;
        lb = b;
        unite_plain<false>(parent, a - 1u, b - 1u);
    };
    if ((m & 1u) && (mL >> 31)) join(row, row - 1);
    uint32_t q[4], qs[4];
    bool in[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int qy = (int)y + row_dy(k), qz = (int)z + row_dz(k);
        in[k] = (TZ > 1 || k == 0) && qy >= 0 && qy < (int)g.H && qz >= 0;
        qs[k] = in[k] ? ((uint32_t)qz * g.H + (uint32_t)qy) * t.ws + xs : 0u;
        q[k] = in[k] ? bits[qs[k]] : 0u;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (!in[k] || (DIAMOND && (k == 1 || k == 3))) continue;
        const uint32_t qy = y + (uint32_t)row_dy(k), qz = z + (uint32_t)row_dz(k);
        const bool cross = qy / TY != y / TY || qz / TZ != z / TZ;
        const uint32_t *qrow = lab + ((size_t)qz * g.H + qy) * g.W + xs * 32u;
        if (cross)
            row_contacts<DIAMOND>(m, q[k], via_row<DIAMOND>(k, q), 0xFFFFFFFFu, [&](uint32_t i, uint32_t j) { join(row + i, qrow + j); });
        if constexpr (!DIAMOND) {
            // diagonal contacts over the segment's ends that no other
            // contact implies
            if ((m & 1u) && !first && !(q[k] & 1u) && !(mL >> 31) && (bits[qs[k] - 1u] >> 31)) join(row, qrow - 1);
            if ((m >> 31) && !last && !(q[k] >> 31) && !(mR & 1u) && (bits[qs[k] + 1u] & 1u)) join(row + 31, qrow + 32);
        }
    }
}

// Per id: the root, and the component's smallest key at the root.
__global__ void ccl_resolve_kernel(uint32_t *parent, uint32_t *minkey, const uint32_t *__restrict__ d_count) {
    const uint32_t cnt = *d_count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
        const uint32_t root = find_plain(parent, i);
        if (root != i) {
            st_cg(parent + i, root);
            atomicMin(minkey + root, ld_cg(minkey + i));
        }
    }
}

__global__ void ccl_mark_roots(const uint32_t *__restrict__ parent, const uint32_t *__restrict__ minkey,
                               const uint32_t *__restrict__ d_count, uint32_t *__restrict__ bitmap) {
    const uint32_t cnt = *d_count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
        if (parent[i] != i) continue;
        const uint32_t idx = fkey_index((float)(minkey[i] + 1u));   // float32(K + 1)
        atomicOr(bitmap + (idx >> 5), 1u << (idx & 31));
    }
}

__device__ __forceinline__ uint32_t rank_of(const uint32_t *bitmap, const uint32_t *prefix,
                                            uint32_t idx) {
    const uint32_t w = idx >> 5, b = idx & 31;
    return prefix[w] + __popc(bitmap[w] & ((1u << b) - 1u)) + 1u;
}

// Per id: its label, in place of its parent (no other id reads that any more).
__global__ void ccl_label_ids(uint32_t *__restrict__ parent, const uint32_t *__restrict__ minkey,
                              const uint32_t *__restrict__ d_count, const uint32_t *__restrict__ bitmap,
                              const uint32_t *__restrict__ prefix) {
    const uint32_t cnt = *d_count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x)
        parent[i] = rank_of(bitmap, prefix, fkey_index((float)(minkey[parent[i]] + 1u)));
}

// Labels of the foreground voxels: a warp takes the row masks of 32 segments
// and visits the ones that hold foreground, four at a time.
__global__ void __launch_bounds__(kT)
ccl_label_voxels(uint32_t *__restrict__ lab, const uint32_t *__restrict__ bits, const uint32_t *__restrict__ label,
                 uint32_t W, uint32_t ws, FastDiv fws, uint32_t nseg) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (kT / 32);
    for (uint32_t s0 = (blockIdx.x * (kT / 32) + (threadIdx.x >> 5)) * 32u; s0 < nseg; s0 += warps * 32u) {
        const uint32_t m = s0 + lane < nseg ? bits[s0 + lane] : 0u;
        unsigned todo = __ballot_sync(0xffffffffu, m != 0u);
        while (todo) {
            uint32_t at[4], v[4];
            bool on[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int j = todo ? __ffs(todo) - 1 : 0;
                const uint32_t mj = __shfl_sync(0xffffffffu, m, j);
                on[k] = todo != 0u && (mj >> lane & 1u);
                const uint32_t sgm = s0 + (uint32_t)j, r = fws.div(sgm);
                at[k] = r * W + (sgm - r * ws) * 32u + lane;
                v[k] = on[k] ? lab[at[k]] : 0u;
                todo &= todo - 1u;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (on[k]) lab[at[k]] = __ldg(label + (v[k] - 1u));
        }
    }
}

// ---- dense labelling on row runs ------------------------------------------
// Small and thin images: a warp per 32 voxels of a row, parents in the labels
// themselves as keys (x-major, + 1).  In a row, keys grow with x, so the first
// voxel of a run holds the run's smallest key: the first pass links every
// foreground voxel to the start of its run inside the segment.  The union pass
// joins whole runs: a run is united once with every run of each neighbour row
// before it (row_dy, row_dz) that overlaps it, through the first voxel of the
// overlap, with a run of that row that touches it only diagonally and with the
// run that continues it from the previous segment.
constexpr int kRowWarps = 8;   // warps per CTA

struct Rows {
    uint32_t ws;     // segments per row
    FastDiv fws;
    uint32_t nseg;   // D * H * ws
};

template <typename FG>
__global__ void __launch_bounds__(kRowWarps * 32)
ccl_init_rows(const typename FG::Value *bin, FG fg, uint32_t *lab, Geo g, Rows R) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t s = blockIdx.x * kRowWarps + (threadIdx.x >> 5); s < R.nseg; s += gridDim.x * kRowWarps) {
        const uint32_t r = R.fws.div(s), xs = s - r * R.ws;       // r = z * H + y
        const uint32_t z = g.fH.div(r), y = r - z * g.H, x = xs * 32u + lane;
        const bool in = x < g.W, on = in && fg(bin[in ? r * g.W + x : 0u]);
        const uint32_t m = __ballot_sync(0xffffffffu, on);
        if (in) lab[r * g.W + x] = on ? xyz2k(g, xs * 32u + run_start(m, lane), y, z) + 1u : 0u;
    }
}

template <bool DIAMOND>
__global__ void __launch_bounds__(kRowWarps * 32)
ccl_union_rows(uint32_t *lab, Geo g, Rows R) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t xstep = g.H * g.D;                             // key distance of x +- 1
    for (uint32_t s = blockIdx.x * kRowWarps + (threadIdx.x >> 5); s < R.nseg; s += gridDim.x * kRowWarps) {
        const uint32_t r = R.fws.div(s), xs = s - r * R.ws;
        const uint32_t z = g.fH.div(r), y = r - z * g.H, x = xs * 32u + lane;
        const bool in = x < g.W;
        // what is foreground never changes while parents are linked
        const bool on = in && ld_cg(lab + r * g.W + x) != 0u;
        const uint32_t m = __ballot_sync(0xffffffffu, on);
        if (!m) continue;
        const bool is_start = (m & ~(m << 1)) >> lane & 1u, is_end = (m & ~(m >> 1)) >> lane & 1u;
        const uint32_t kp = xyz2k(g, x, y, z);
        // unions start from the run's first voxel (every run voxel points at it)
        const uint32_t ka = on ? kp - (lane - run_start(m, lane)) * xstep : kp;
        if (lane == 0 && on && xs > 0 && ld_cg(lab + r * g.W + x - 1u) != 0u) unite(lab, g, kp, kp - xstep);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (DIAMOND && (k == 1 || k == 3)) continue;
            const int qy = (int)y + row_dy(k), qz = (int)z + row_dz(k);
            if (qy < 0 || qy >= (int)g.H || qz < 0) continue;    // warp-uniform
            const uint32_t *row = lab + ((uint32_t)qz * g.H + (uint32_t)qy) * g.W;
            const bool q = in && ld_cg(row + x) != 0u;
            bool qe = false;                                     // lane 0: row[x - 1], lane 31: row[x + 1]
            if (lane == 0 && xs > 0) qe = ld_cg(row + x - 1u) != 0u;
            if (lane == 31 && x + 1u < g.W) qe = ld_cg(row + x + 1u) != 0u;
            const uint32_t Q = __ballot_sync(0xffffffffu, q);
            const bool qL = lane == 0 ? qe : (Q >> (lane - 1u)) & 1u, qR = lane == 31 ? qe : (Q >> (lane + 1u)) & 1u;
            if (!on) continue;
            const uint32_t kq = xyz2k(g, x, (uint32_t)qy, (uint32_t)qz);
            if (q && (is_start || !qL)) unite(lab, g, ka, kq);         // first voxel of an overlap
            if (DIAMOND) continue;
            if (is_start && qL && !q) unite(lab, g, ka, kq - xstep);   // diagonal contacts
            if (is_end && qR && !q) unite(lab, g, ka, kq + xstep);
        }
    }
}

// Roots: the first voxel of each run walks, its run takes the root by shuffle; a
// root (always the first voxel of its run) is marked in the bitmap.
__global__ void __launch_bounds__(kRowWarps * 32)
ccl_roots_rows(uint32_t *lab, Geo g, Rows R, uint32_t *__restrict__ bitmap) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t s = blockIdx.x * kRowWarps + (threadIdx.x >> 5); s < R.nseg; s += gridDim.x * kRowWarps) {
        const uint32_t r = R.fws.div(s), xs = s - r * R.ws;
        const uint32_t z = g.fH.div(r), y = r - z * g.H, x = xs * 32u + lane;
        const uint32_t v = x < g.W ? ld_cg(lab + r * g.W + x) : 0u;
        const uint32_t m = __ballot_sync(0xffffffffu, v != 0u);
        if (!m) continue;
        uint32_t root = 0u;
        if ((m & ~(m << 1)) >> lane & 1u) {
            const uint32_t k = xyz2k(g, x, y, z);
            root = find_root(lab, g, k) + 1u;
            if (root == k + 1u) {
                const uint32_t idx = fkey_index((float)root);   // float32(K + 1)
                atomicOr(bitmap + (idx >> 5), 1u << (idx & 31));
            }
        }
        root = __shfl_sync(0xffffffffu, root, v != 0u ? (int)run_start(m, lane) : (int)lane);
        if (v != 0u && root != v) st_cg(lab + r * g.W + x, root);
    }
}

__global__ void ccl_label_rows(uint32_t *__restrict__ lab, int64_t n, const uint32_t *__restrict__ bitmap,
                               const uint32_t *__restrict__ prefix) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t v = lab[i];
        if (v) lab[i] = rank_of(bitmap, prefix, fkey_index((float)v));
    }
}

// ---- list variants (sparse seeds) ---------------------------------------
__global__ void ccl_union_list(uint32_t *lab, Geo g, const uint32_t *__restrict__ list,
                               const uint32_t *__restrict__ d_count) {
    const uint32_t cnt = *d_count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
        uint32_t x, y, z;
        m2xyz(g, list[i], x, y, z);
        union_back(lab, g, x, y, z);
    }
}

__global__ void ccl_flatten_list(uint32_t *lab, Geo g, const uint32_t *__restrict__ list,
                                 const uint32_t *__restrict__ d_count) {
    const uint32_t cnt = *d_count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
        const uint32_t m = list[i];
        uint32_t v = ld_cg(lab + m);
        uint32_t r = find_root(lab, g, v - 1u);
        if (r != v - 1u) st_cg(lab + m, r + 1u);
    }
}

__global__ void ccl_mark_list(const uint32_t *__restrict__ lab, Geo g,
                              const uint32_t *__restrict__ list,
                              const uint32_t *__restrict__ d_count, uint32_t *__restrict__ bitmap) {
    const uint32_t cnt = *d_count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
        const uint32_t m = list[i];
        const uint32_t v = lab[m];
        uint32_t x, y, z;
        m2xyz(g, m, x, y, z);
        if (v - 1u != xyz2k(g, x, y, z)) continue;
        uint32_t idx = fkey_index((float)v);
        atomicOr(bitmap + (idx >> 5), 1u << (idx & 31));
    }
}

__global__ void ccl_label_list(uint32_t *__restrict__ lab, const uint32_t *__restrict__ list,
                               const uint32_t *__restrict__ d_count,
                               const uint32_t *__restrict__ bitmap,
                               const uint32_t *__restrict__ prefix) {
    const uint32_t cnt = *d_count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
        const uint32_t m = list[i];
        lab[m] = rank_of(bitmap, prefix, fkey_index((float)lab[m]));
    }
}

// The whole list labelling of a small image in one launch: the unions by a thread
// per listed voxel, then roots, marks, ranks and labels by the CTA that finishes
// last, with block barriers between them, in place of eight launches and a clear.
// That CTA takes 3 to 4 us for every 1024 listed voxels and the launches about 25 us in all,
// so the line is one on the number of listed voxels, which only the device
// knows.  Local maxima are few: voronoi_otsu_labeling of noise (256 x 256 0.18 against 0.23 ms
// for the whole call, 362 x 362 0.20 : 0.24, 32 x 64 x 64 0.28 : 0.31).  A mask's voxels may be all
// of them: masked_voronoi_labeling_binary of 90% masks 64 x 64 0.23 : 0.25, 16 x 32 x 32 0.52 : 0.54,
// 256 x 256 0.31 : 0.27, 32 x 64 x 64 0.76 : 0.61.  With the unions in the one CTA too,
// as this kernel was, the last took 11.1 ms.
constexpr int kListCta = 1024;
constexpr int64_t kListSparseVoxels = int64_t(1) << 17, kListDenseVoxels = int64_t(1) << 15;

__global__ void __launch_bounds__(kListCta)
ccl_list_small(uint32_t *lab, Geo g, const uint32_t *__restrict__ list, const uint32_t *__restrict__ d_count,
               uint32_t *bitmap, uint32_t *prefix, uint32_t words, uint32_t *__restrict__ d_nlabels, uint32_t *d_done) {
    __shared__ uint32_t s_w[kListCta / 32];
    __shared__ uint32_t s_ticket;
    const uint32_t cnt = *d_count;
    const uint32_t t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    const uint32_t ctas = max(1u, min(gridDim.x, (cnt + kListCta - 1) / kListCta));   // that have voxels
    if (blockIdx.x >= ctas) return;
    for (uint32_t i = blockIdx.x * kListCta + t; i < cnt; i += ctas * kListCta) {
        uint32_t x, y, z;
        m2xyz(g, list[i], x, y, z);
        union_back(lab, g, x, y, z);
    }
    if (ctas > 1) {
        __threadfence();   // this CTA's unions before its ticket
        __syncthreads();
        if (t == 0) s_ticket = atomicAdd(d_done, 1u);
        __syncthreads();
        if (s_ticket + 1u != ctas) return;
        __threadfence();   // the other CTAs' unions after theirs
    }
    for (uint32_t w = t; w < words; w += kListCta) st_cg(bitmap + w, 0u);
    __syncthreads();
    for (uint32_t i = t; i < cnt; i += kListCta) {
        const uint32_t m = list[i];
        const uint32_t v = ld_cg(lab + m), r = find_root(lab, g, v - 1u) + 1u;
        uint32_t x, y, z;
        m2xyz(g, m, x, y, z);
        if (r - 1u == xyz2k(g, x, y, z)) {   // a root
            const uint32_t idx = fkey_index((float)r);
            atomicOr(bitmap + (idx >> 5), 1u << (idx & 31));
        }
        if (r != v) st_cg(lab + m, r);
    }
    __syncthreads();
    // bits before each word: every thread a stretch of words
    const uint32_t per = (words + kListCta - 1) / kListCta;
    const uint32_t w0 = min(words, t * per), w1 = min(words, w0 + per);
    uint32_t c = 0;
    for (uint32_t w = w0; w < w1; ++w) c += (uint32_t)__popc(ld_cg(bitmap + w));
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    uint32_t at = incl - c, all = 0;
    for (int k = 0; k < kListCta / 32; ++k) {
        if (k < warp) at += s_w[k];
        all += s_w[k];
    }
    for (uint32_t w = w0; w < w1; ++w) {
        st_cg(prefix + w, at);
        at += (uint32_t)__popc(ld_cg(bitmap + w));
    }
    if (t == 0 && d_nlabels) *d_nlabels = all;
    __syncthreads();
    for (uint32_t i = t; i < cnt; i += kListCta) {
        const uint32_t m = list[i], idx = fkey_index((float)ld_cg(lab + m)), w = idx >> 5;
        st_cg(lab + m, ld_cg(prefix + w) + (uint32_t)__popc(ld_cg(bitmap + w) & ((1u << (idx & 31)) - 1u)) + 1u);
    }
}

// ---- rank machinery -------------------------------------------------------
// Per bitmap word the number of set bits before it, in two launches: bits per
// block of `per` words, then every block adds up the blocks before it (at most
// kRankBlocks of them) and scans its words, 4 per thread and round.  The last
// block also writes the total.
constexpr uint32_t kRankBlocks = 2048, kRankRound = 4 * kT;

__global__ void __launch_bounds__(kT)
rank_sums_kernel(const uint32_t *__restrict__ bitmap, uint32_t words, uint32_t per, uint32_t *__restrict__ sums) {
    const uint32_t w0 = blockIdx.x * per, w1 = min(words, w0 + per);
    uint32_t c = 0;
    for (uint32_t w = w0 + 4 * threadIdx.x; w < w1; w += kRankRound)   // per and w0 are multiples of 4
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (w + k < w1) c += (uint32_t)__popc(bitmap[w + k]);
    c = __reduce_add_sync(0xffffffffu, c);
    __shared__ uint32_t s_c[kT / 32];
    if ((threadIdx.x & 31) == 0) s_c[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kT / 32; ++k) c += s_c[k];
        sums[blockIdx.x] = c;
    }
}

__global__ void __launch_bounds__(kT)
rank_prefix_kernel(const uint32_t *__restrict__ bitmap, uint32_t words, uint32_t per, const uint32_t *__restrict__ sums,
                   uint32_t *__restrict__ prefix, uint32_t *__restrict__ total) {
    __shared__ uint32_t s_w[kT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // bits before this block
    uint32_t before = 0;
    for (uint32_t i = threadIdx.x; i < blockIdx.x; i += kT) before += sums[i];
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) s_w[warp] = before;
    __syncthreads();
    before = 0;
    for (int k = 0; k < kT / 32; ++k) before += s_w[k];
    const uint32_t w0 = blockIdx.x * per, w1 = min(words, w0 + per);
    for (uint32_t base = w0; base < w1; base += kRankRound) {
        const uint32_t w = base + 4 * threadIdx.x;
        uint32_t c[4], x = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            c[k] = x;
            x += w + k < w1 ? (uint32_t)__popc(bitmap[w + k]) : 0u;
        }
        uint32_t incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        __syncthreads();
        if (lane == 31) s_w[warp] = incl;
        __syncthreads();
        uint32_t at = before + incl - x, all = 0;
        for (int k = 0; k < kT / 32; ++k) {
            if (k < warp) at += s_w[k];
            all += s_w[k];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (w + k < w1) prefix[w + k] = at + c[k];
        before += all;
    }
    if (total && blockIdx.x + 1 == gridDim.x && threadIdx.x == 0) *total = before;
}

struct Rank {
    uint32_t *bitmap, *sums, *prefix;
    uint32_t words, per, blocks;
};

Rank take_rank(Arena &ws, uint64_t bits) {
    Rank r;
    r.words = (uint32_t)((bits + 31) / 32 + 1);
    // whole rounds per block
    r.per = ((r.words + kRankBlocks - 1) / kRankBlocks + kRankRound - 1) / kRankRound * kRankRound;
    r.blocks = (r.words + r.per - 1) / r.per;
    r.bitmap = ws.take<uint32_t>(r.words);
    r.sums = ws.take<uint32_t>(r.blocks);
    r.prefix = ws.take<uint32_t>(r.words);
    return r;
}

// prefix from bitmap; *total (optional): the number of set bits
int rank_build(const Rank &r, cudaStream_t st, uint32_t *total = nullptr) {
    rank_sums_kernel<<<r.blocks, kT, 0, st>>>(r.bitmap, r.words, r.per, r.sums);
    rank_prefix_kernel<<<r.blocks, kT, 0, st>>>(r.bitmap, r.words, r.per, r.sums, r.prefix, total);
    CLE_LAUNCH_CHECK_N("rank build", 2);
    return CLE_OK;
}

// Workspace of the dense labelling.
struct Dense {
    uint32_t *count, *bits, *parent, *minkey;
    Rank rank;
};

Dense take_dense(Arena &ws, const Img &im, bool diamond) {
    Dense d;
    // most components the tiles can hold (tiles start at even coordinates):
    // one per 2 x 2 x 2 voxels, or every other voxel with face connectivity
    const int64_t box = ((im.W + 1) / 2) * ((im.H + 1) / 2) * ((im.D + 1) / 2);
    const int64_t most = diamond ? (im.n() + 1) / 2 + im.D * im.H * ((im.W + 31) / 32) : box;
    d.count = ws.take<uint32_t>(1);
    d.bits = ws.take<uint32_t>((size_t)(im.D * im.H * ((im.W + 31) / 32)));
    d.parent = ws.take<uint32_t>((size_t)most);
    d.minkey = ws.take<uint32_t>((size_t)most);
    d.rank = take_rank(ws, fkey_bits_for(im.n()));
    return d;
}

template <typename FG, int TY, int TZ, bool DIAMOND>
int dense_tiles(const Img &bin, FG fg, uint32_t *lab, const Dense &d, const Geo &g, cudaStream_t st) {
    Tiles t;
    t.nx = t.ws = (uint32_t)((bin.W + 31) / 32);
    t.ny = (uint32_t)((bin.H + TY - 1) / TY);
    t.nz = (uint32_t)((bin.D + TZ - 1) / TZ);
    t.fnx = FastDiv(t.nx);
    t.fny = FastDiv(t.ny);
    const uint32_t nseg = (uint32_t)(bin.D * bin.H) * t.ws;
    CLE_CUDA(cudaMemsetAsync(d.count, 0, sizeof(uint32_t), st));
    ccl_tile_kernel<FG, TY, TZ, DIAMOND><<<t.nx * t.ny * t.nz, kTileThreads, 0, st>>>(
        (const typename FG::Value *)bin.data, fg, lab, d.bits, d.parent, d.minkey, d.count, g, t);
    ccl_merge_kernel<TY, TZ, DIAMOND><<<(nseg + kT - 1) / kT, kT, 0, st>>>(lab, d.bits, d.parent, g, t,
                                                                               FastDiv(t.ws), nseg);
    CLE_LAUNCH_CHECK_N("ccl tiles", 2);
    // the id count stays on the device: a grid that fits any count
    const int ib = launch_blocks(std::min<int64_t>(bin.n(), 1 << 20), kT);
    ccl_resolve_kernel<<<ib, kT, 0, st>>>(d.parent, d.minkey, d.count);
    CLE_CUDA(cudaMemsetAsync(d.rank.bitmap, 0, sizeof(uint32_t) * d.rank.words, st));
    ccl_mark_roots<<<ib, kT, 0, st>>>(d.parent, d.minkey, d.count, d.rank.bitmap);
    CLE_LAUNCH_CHECK_N("ccl dense", 2);
    CLE_TRY(rank_build(d.rank, st));
    ccl_label_ids<<<ib, kT, 0, st>>>(d.parent, d.minkey, d.count, d.rank.bitmap, d.rank.prefix);
    ccl_label_voxels<<<launch_blocks(nseg, kT), kT, 0, st>>>(lab, d.bits, d.parent, (uint32_t)bin.W, t.ws, FastDiv(t.ws), nseg);
    CLE_LAUNCH_CHECK_N("ccl label", 2);
    return CLE_OK;
}

template <typename FG, bool DIAMOND>
int dense_rows(const Img &bin, FG fg, uint32_t *lab, const Dense &d, const Geo &g, cudaStream_t st) {
    Rows R;
    R.ws = (uint32_t)((bin.W + 31) / 32);
    R.fws = FastDiv(R.ws);
    R.nseg = (uint32_t)(bin.D * bin.H) * R.ws;
    const int b = launch_blocks((int64_t)R.nseg * 32, kRowWarps * 32);
    ccl_init_rows<FG><<<b, kRowWarps * 32, 0, st>>>((const typename FG::Value *)bin.data, fg, lab, g, R);
    ccl_union_rows<DIAMOND><<<b, kRowWarps * 32, 0, st>>>(lab, g, R);
    CLE_CUDA(cudaMemsetAsync(d.rank.bitmap, 0, sizeof(uint32_t) * d.rank.words, st));
    ccl_roots_rows<<<b, kRowWarps * 32, 0, st>>>(lab, g, R, d.rank.bitmap);
    CLE_LAUNCH_CHECK_N("ccl rows", 3);
    CLE_TRY(rank_build(d.rank, st));
    ccl_label_rows<<<launch_blocks(bin.n(), kT), kT, 0, st>>>(lab, bin.n(), d.rank.bitmap, d.rank.prefix);
    CLE_LAUNCH_CHECK("ccl rows label");
    return CLE_OK;
}

// Tiles of 16 x 8 rows in volumes, of 64 rows in images (and volumes of one plane),
// unless the image is too small to fill the GPU with tiles, whose phases are
// serial (one after another, a row per thread), or so thin that tiles are mostly empty.
// Microseconds of a call on row runs : in tiles, half of the voxels foreground at
// random, then smooth objects: 256 x 256 48 : 112, 42 : 66; 1024 x 1024 157 : 208, 81 : 95;
// 1400 x 1400 260 : 239, 124 : 106; 32 x 64 x 64 73 : 182, 47 : 75; 64 x 100 x 100 243 : 234,
// 104 : 96 (10% foreground 105 : 161); 64 x 128 x 128 334 : 237, 134 : 99 (with face connectivity
// 133 : 150, 100 : 82); 4 x 512 x 512 306 : 220, 118 : 93 (121 : 141, 92 : 86); thin:
// 1 x 4194304 95 : 793, 104 : 526; 8 x 524288 362 : 353, 185 : 165; 16 x 262144 394 : 264,
// 192 : 130; 65536 x 1 x 32 274 : 280; 65536 x 2 x 16 852 : 257; 32768 x 4 x 8 766 : 154.
template <bool DIAMOND, typename FG>
int dense_typed(const Img &bin, FG fg, uint32_t *lab, const Dense &d, const Geo &g, cudaStream_t st) {
    const bool volume = bin.D > 1;
    const int64_t rows = bin.D * bin.H;
    const int64_t tile_rows = volume ? (bin.D + 7) / 8 * 8 * ((bin.H + 15) / 16 * 16) : (bin.H + 63) / 64 * 64;
    const int64_t lanes = rows * ((bin.W + 31) / 32 * 32);   // of the warps on row runs
    if (lanes <= (volume && !DIAMOND ? int64_t(3) << 18 : int64_t(1) << 20) || rows * (volume ? 16 : 8) <= tile_rows)
        return dense_rows<FG, DIAMOND>(bin, fg, lab, d, g, st);
    if (volume) return dense_tiles<FG, 16, 8, DIAMOND>(bin, fg, lab, d, g, st);
    return dense_tiles<FG, 64, 1, DIAMOND>(bin, fg, lab, d, g, st);
}

template <typename T>
int dense_typed(const Img &bin, uint32_t *lab, const Dense &d, const Geo &g, bool diamond, cudaStream_t st) {
    return diamond ? dense_typed<true>(bin, NonZero<T>(), lab, d, g, st) : dense_typed<false>(bin, NonZero<T>(), lab, d, g, st);
}

// ---- relabel ------------------------------------------------------------
template <typename T>
__device__ __forceinline__ uint32_t label_value(T v) {
    if constexpr (std::is_floating_point<T>::value) {
        return v > (T)0 ? (uint32_t)(int64_t)v : 0u;
    } else {
        return (uint32_t)v;
    }
}

template <typename T>
__global__ void relabel_mark_kernel(const T *__restrict__ s, int64_t n, uint32_t maxv,
                                    uint32_t *__restrict__ bitmap) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t v = label_value(s[i]);
        if (v == 0 || v > maxv) continue;
        atomicOr(bitmap + (v >> 5), 1u << (v & 31));
    }
}

template <typename T, typename Td>
__global__ void relabel_apply_kernel(const T *__restrict__ s, Td *__restrict__ d, int64_t n,
                                     uint32_t maxv, const uint32_t *__restrict__ bitmap,
                                     const uint32_t *__restrict__ prefix) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t v = label_value(s[i]);
        uint32_t out = (v == 0 || v > maxv) ? 0u : rank_of(bitmap, prefix, v);
        d[i] = (Td)out;
    }
}

template <typename T>
int relabel_typed(const Img &src, const Img &dst, uint32_t maxv, const Rank &r, cudaStream_t st) {
    const int64_t n = src.n();
    const int b = launch_blocks(n, kT);
    relabel_mark_kernel<T><<<b, kT, 0, st>>>((const T *)src.data, n, maxv, r.bitmap);
    CLE_LAUNCH_CHECK("relabel mark");
    CLE_TRY(rank_build(r, st));
    switch (dst.dtype) {
        case CLE_U32: relabel_apply_kernel<T, uint32_t><<<b, kT, 0, st>>>((const T *)src.data, (uint32_t *)dst.data, n, maxv, r.bitmap, r.prefix); break;
        case CLE_F32: relabel_apply_kernel<T, float><<<b, kT, 0, st>>>((const T *)src.data, (float *)dst.data, n, maxv, r.bitmap, r.prefix); break;
        default: set_error("relabel_sequential: unsupported destination dtype %d", dst.dtype); return CLE_ERR_DTYPE;
    }
    CLE_LAUNCH_CHECK("relabel apply");
    return CLE_OK;
}

__global__ void u32_to_f32_kernel(const uint32_t *__restrict__ s, float *__restrict__ d, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        d[i] = (float)s[i];
}

}  // namespace

size_t rank_workspace_bytes(uint64_t bits) {
    Arena a(nullptr, 0);
    take_rank(a, bits);
    return a.off;
}

size_t ccl_workspace_bytes(const Img &im, bool diamond) {
    Arena a(nullptr, 0);
    a.take<uint32_t>(im.n());   // u32 labels when the destination is f32
    take_dense(a, im, diamond);
    return a.off;
}

int ccl_dense(const Img &bin, uint32_t *lab, Arena &ws, cudaStream_t st, bool diamond, const float *d_above) {
    const Dense d = take_dense(ws, bin, diamond);
    if (!ws.ok()) { set_error("connected_components_labeling_box: workspace too small"); return CLE_ERR_WORKSPACE; }
    if (bin.n() == 0) return CLE_OK;
    const Geo g = make_geo(bin);
    switch (bin.dtype) {
        case CLE_U8: CLE_TRY(dense_typed<uint8_t>(bin, lab, d, g, diamond, st)); break;
        case CLE_U32: CLE_TRY(dense_typed<uint32_t>(bin, lab, d, g, diamond, st)); break;
        case CLE_F32:
            if (d_above) CLE_TRY(dense_typed<false>(bin, Above{d_above}, lab, d, g, st));
            else CLE_TRY(dense_typed<float>(bin, lab, d, g, diamond, st));
            break;
        case CLE_U16: CLE_TRY(dense_typed<uint16_t>(bin, lab, d, g, diamond, st)); break;
        default: set_error("connected_components_labeling_box: unsupported dtype %d", bin.dtype); return CLE_ERR_DTYPE;
    }
    return CLE_OK;
}

int ccl_list(const Geo &g, int64_t n, uint32_t *lab, const uint32_t *list,
             const uint32_t *d_count, int64_t cap, Arena &ws, cudaStream_t st,
             uint32_t *d_nlabels, uint32_t *d_done, bool dense) {
    Rank r = take_rank(ws, fkey_bits_for(n));
    if (!ws.ok()) { set_error("seed labeling: workspace too small"); return CLE_ERR_WORKSPACE; }
    if (n <= (dense ? kListDenseVoxels : kListSparseVoxels)) {
        ccl_list_small<<<(unsigned)((n + kListCta - 1) / kListCta), kListCta, 0, st>>>(lab, g, list, d_count, r.bitmap, r.prefix,
                                                                                   r.words, d_nlabels, d_done);
        CLE_LAUNCH_CHECK("ccl list (one launch)");
        return CLE_OK;
    }
    const int b = launch_blocks(cap, kT);
    ccl_union_list<<<b, kT, 0, st>>>(lab, g, list, d_count);
    ccl_flatten_list<<<b, kT, 0, st>>>(lab, g, list, d_count);
    CLE_CUDA(cudaMemsetAsync(r.bitmap, 0, sizeof(uint32_t) * r.words, st));
    ccl_mark_list<<<b, kT, 0, st>>>(lab, g, list, d_count, r.bitmap);
    CLE_LAUNCH_CHECK_N("ccl list", 3);
    CLE_TRY(rank_build(r, st, d_nlabels));
    ccl_label_list<<<b, kT, 0, st>>>(lab, list, d_count, r.bitmap, r.prefix);
    CLE_LAUNCH_CHECK("ccl list label");
    return CLE_OK;
}

int ccl_to_dst(const uint32_t *lab, const Img &dst, cudaStream_t st) {
    if (dst.dtype == CLE_F32) {
        u32_to_f32_kernel<<<launch_blocks(dst.n(), kT), kT, 0, st>>>(lab, (float *)dst.data, dst.n());
        CLE_LAUNCH_CHECK("u32 to f32");
    }
    return CLE_OK;
}

size_t relabel_workspace_bytes(uint32_t max_label) {
    return rank_workspace_bytes((uint64_t)max_label + 1u);
}

int relabel_sequential(const Img &src, const Img &dst, uint32_t maxv, Arena &ws, cudaStream_t st) {
    CLE_TRY(same_shape(src, dst, "source", "output"));
    Rank r = take_rank(ws, (uint64_t)maxv + 1u);
    if (!ws.ok()) { set_error("relabel_sequential: workspace too small"); return CLE_ERR_WORKSPACE; }
    CLE_CUDA(cudaMemsetAsync(r.bitmap, 0, sizeof(uint32_t) * r.words, st));
    switch (src.dtype) {
        case CLE_U32: return relabel_typed<uint32_t>(src, dst, maxv, r, st);
        case CLE_F32: return relabel_typed<float>(src, dst, maxv, r, st);
        case CLE_U16: return relabel_typed<uint16_t>(src, dst, maxv, r, st);
        case CLE_U8: return relabel_typed<uint8_t>(src, dst, maxv, r, st);
        default: set_error("relabel_sequential: unsupported dtype %d", src.dtype); return CLE_ERR_DTYPE;
    }
}

}  // namespace cle
