// On-device structure generation for scripts/gen_aniso_structures3d.py
// datasets: the random trigonometric field, its porosity quantile and the
// 6-connected percolation test on the 3 x 3 x 3 tiling.
//
// The host draws every random number (wavevectors, phases) with the
// reference's own generator calls; the device does the work that scales with
// the voxel count:
//
//  * field (gen_aniso_structures3d.py:154-176): S = scale * sum_i
//    cos(((2 pi qz_i) z + (2 pi qy_i) y) + (2 pi qx_i) x + phi_i), the terms
//    formed and summed in the reference's order and rounding (this unit is
//    compiled without FMA contraction), modes accumulated in order;
//  * threshold (:179-181): the two order statistics around numpy's linear
//    quantile index, found by an 8-pass radix selection over the sortable
//    bit patterns of the doubles and interpolated in numpy's arithmetic, all
//    on the device; solid where S > t;
//  * percolation (:184-205): the 6-connected components of the pore phase of
//    the 3 x 3 x 3 tiling (no wrap), and whether one touches both faces of an
//    axis.  The tiling repeats one cell, so the cell's components are found
//    once (union-find with atomic minimum links), and the 27 copies of those
//    that touch a cell face are joined across the tiles' common faces.
//
// Every loop over labels is bounded; exceeding the bound reports an error
// instead of spinning.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>

#include "../../include/lbm.h"
#include "engine_host.h"

namespace {

constexpr int GTPB = 256;

// Blocks of `rows` (y, z) rows: the products 2 pi q x coordinate of a row are
// formed once per mode in shared memory, with the roundings of the
// reference's expression.  What is left is the FP64 cosine of every voxel and
// mode: 80^3 with 50 modes, 82 -> 77 us.
constexpr int FIELD_TERMS = 1024;        // row terms in shared memory at a time
__global__ void __launch_bounds__(GTPB) trig_field_kernel(int size, int rows, int n_modes, const int *__restrict__ q,
                                                          const double *__restrict__ phases,
                                                          const double *__restrict__ pts, double scale, double *__restrict__ field)
{
    const double twopi = 2.0 * 3.141592653589793;
    __shared__ double zy[FIELD_TERMS], cx[FIELD_TERMS], ph[FIELD_TERMS];
    const int all = size * size, row0 = blockIdx.x * rows, chunk = FIELD_TERMS / rows;
    // rows > 1: the block's threads cover its rows; rows == 1: its columns in turn
    const int own = rows > 1 ? threadIdx.x / size : 0;
    const bool live = own < rows && row0 + own < all;
    for (int x0 = 0; x0 < (rows > 1 ? 1 : size); x0 += blockDim.x) {
        const int x = rows > 1 ? (int)threadIdx.x % size : x0 + (int)threadIdx.x;
        const bool v = live && x < size;
        const double px = v ? pts[x] : 0.0;
        double acc = 0.0;
        for (int m0 = 0; m0 < n_modes; m0 += chunk) {
            const int mn = min(chunk, n_modes - m0);
            __syncthreads();
            for (int e = threadIdx.x; e < rows * mn; e += blockDim.x) {
                const int r = e / mn, m = e - r * mn, row = min(row0 + r, all - 1);
                const int *qm = q + 3 * (m0 + m);
                zy[e] = (twopi * (double)qm[2]) * pts[row / size] + (twopi * (double)qm[1]) * pts[row % size];
                if (r == 0) {
                    cx[m] = twopi * (double)qm[0];
                    ph[m] = phases[m0 + m];
                }
            }
            __syncthreads();
            if (v)
                for (int m = 0; m < mn; ++m) acc = acc + cos((zy[own * mn + m] + cx[m] * px) + ph[m]);
        }
        if (v) field[(long long)(row0 + own) * size + x] = scale * acc;
    }
}

// order-preserving map of a double's bits to an unsigned key
__device__ __forceinline__ unsigned long long sort_key(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// State of the selection of the order statistic of rank k (0-based) and the
// one after it.
struct Select {
    unsigned long long prefix, pmask;    // bits found so far
    unsigned long long k;                // rank among the keys that match them
    unsigned long long next;             // smallest key above the one found
    double t;                            // the interpolated threshold
    unsigned done;                       // blocks finished in this pass
    unsigned hist[256];
};

__global__ void select_init_kernel(Select *s, unsigned long long k)
{
    s->hist[threadIdx.x] = 0u;
    if (threadIdx.x == 0) {
        s->prefix = s->pmask = 0ull;
        s->k = k;
        s->next = ~0ull;
        s->done = 0u;
    }
}

// One digit: histogram of the matching keys; the last block to finish picks
// the digit of rank k and prepares the next pass.  (One launch per digit and
// no host in between: two order statistics took 16 round trips of some 35 us.)
__global__ void __launch_bounds__(GTPB) select_digit_kernel(const double *__restrict__ field, long long n, int shift, Select *s)
{
    __shared__ unsigned sh[256];
    __shared__ bool last;
    static_assert(GTPB == 256, "one bin per thread");
    sh[threadIdx.x] = 0u;
    const unsigned long long prefix = s->prefix, pmask = s->pmask;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    // whole warps: every lane takes part in the votes of every round
    for (long long w = blockIdx.x * (long long)blockDim.x + threadIdx.x - lane; w < n; w += (long long)gridDim.x * blockDim.x) {
        const unsigned long long k = w + lane < n ? sort_key(field[w + lane]) : 0ull;
        const bool in = w + lane < n && (k & pmask) == prefix;
        const unsigned b = (unsigned)(k >> shift) & 255u;
        // the leading digits of a field take few values, and of the last ones
        // few keys match: one addition where a warp's digits agree
        const unsigned hit = __ballot_sync(0xffffffffu, in);
        if (!hit) continue;
        const int lead = __ffs(hit) - 1;
        const unsigned b0 = __shfl_sync(0xffffffffu, b, lead);
        const bool same = __all_sync(0xffffffffu, !in || b == b0);
        if (in && (!same || lane == lead)) atomicAdd(&sh[b], same ? (unsigned)__popc(hit) : 1u);
    }
    __syncthreads();
    if (sh[threadIdx.x]) atomicAdd(&s->hist[threadIdx.x], sh[threadIdx.x]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&s->done, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // the digit whose keys hold rank k: a scan of the bins, one per thread
    __shared__ unsigned wsum[8];
    const unsigned c = __ldcg(&s->hist[threadIdx.x]);
    unsigned incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) wsum[threadIdx.x >> 5] = incl;
    s->hist[threadIdx.x] = 0u;
    const unsigned long long k = s->k;
    __syncthreads();
    for (int i = 0; i < (int)(threadIdx.x >> 5); ++i) incl += wsum[i];
    if (k < incl && k >= incl - c) {
        const unsigned long long b = threadIdx.x;
        s->k = k - (incl - c);
        s->prefix = prefix | b << shift;
        s->pmask = pmask | 255ull << shift;
        s->done = 0u;
        // after the last digit: the next order statistic is the same key if
        // it occurs again, else the smallest key above it (select_next_kernel)
        if (shift == 0 && k + 1 < incl) s->next = prefix | b;
    }
}

__global__ void __launch_bounds__(GTPB) select_next_kernel(const double *__restrict__ field, long long n, Select *s)
{
    const unsigned long long key = s->prefix;
    unsigned long long best = ~0ull;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long k = sort_key(field[i]);
        if (k > key && k < best) best = k;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0 && best < *(volatile unsigned long long *)&s->next) atomicMin(&s->next, best);
}

__device__ __forceinline__ double key_value(unsigned long long k)
{
    return __longlong_as_double((long long)((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k));
}

// numpy's linear interpolation between the two order statistics (no second
// one after the largest value), gamma = the fractional index.
__global__ void select_threshold_kernel(Select *s, double gamma, int has_next)
{
    const double lo = key_value(s->prefix);
    const double hi = has_next ? key_value(s->next) : lo;
    const double diff = hi - lo;
    double t = lo + diff * gamma;
    if (gamma >= 0.5) t = hi - diff * (1.0 - gamma);
    s->t = t;
}

__global__ void threshold_kernel(const double *__restrict__ field, long long n, const Select *s, uint8_t *__restrict__ solid)
{
    const double t = s->t;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        solid[i] = field[i] > t ? 1 : 0;
}

// ---------------------------------------------------------------- union-find
struct Cell {
    int nx, ny, nz;
};

// root of i: labels only ever point to smaller indices, so a chain is at most
// `limit` long; the walk is bounded by it anyway.  Nodes on the way are moved
// up to their grandparents: such a store may replace a link that another
// thread just lowered, but that thread goes on to join the old link's set
// itself, so no connection is lost.  lab is in global or shared memory;
// volatile accesses see the other threads' links in both.
__device__ __forceinline__ int uf_find(int *labels, int i, long long limit, unsigned *err)
{
    volatile int *lab = labels;
    int p = lab[i];
    for (long long it = 0; it < limit; ++it) {
        if (p == i) return i;
        const int g = lab[p];
        if (g == p) return p;
        lab[i] = g;
        i = p;
        p = g;
    }
    atomicOr(err, 1u);
    return i;
}

// The same without moving nodes up: for passes in which other threads rely on
// the labels they store.
__device__ __forceinline__ int uf_root(const int *lab, int i, long long limit, unsigned *err)
{
    for (long long it = 0; it < limit; ++it) {
        const int p = __ldcg(lab + i);
        if (p == i) return i;
        i = p;
    }
    atomicOr(err, 1u);
    return i;
}

__device__ void uf_union(int *lab, int a, int b, long long limit, unsigned *err)
{
    for (int it = 0; it < (1 << 20); ++it) {
        a = uf_find(lab, a, limit, err);
        b = uf_find(lab, b, limit, err);
        if (a == b) return;
        if (a > b) { const int s = a; a = b; b = s; }
        // link the larger root under the smaller; retry if another thread
        // linked it first (its label then decreased, so progress is made)
        const int old = atomicMin(lab + b, a);
        if (old == b) return;
        b = old;
    }
    atomicOr(err, 2u);
}

// Labels of the cell's pore voxels: the first voxel of the run along x within
// 32 voxels of a row (one warp per 32), -1 for solids; mark = no face bits.
__global__ void uf_init_kernel(const uint8_t *__restrict__ solid, Cell c, int *lab, int *id, unsigned *faces)
{
    const int lane = threadIdx.x & 31, per = (c.nx + 31) / 32;
    const long long items = (long long)c.ny * c.nz * per;
    for (long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; w < items; w += ((long long)gridDim.x * blockDim.x) >> 5) {
        const long long row = w / per;
        const int x = (int)(w % per) * 32 + lane;
        const long long i = row * c.nx + x;
        const bool in = x < c.nx, pore = in && solid[i] == 0;
        const unsigned m = __ballot_sync(0xffffffffu, pore);
        const unsigned below = ~m & ((1u << lane) - 1u);
        const int first = below ? 32 - __clz(below) : 0;
        if (in) {
            lab[i] = pore ? (int)(i - lane + first) : -1;
            id[i] = -1;
            faces[i] = 0u;
        }
    }
}

// Join the runs: across the 32-voxel pieces of a row, and with the rows at
// y - 1 and z - 1.  A voxel whose left neighbour makes the same join leaves
// it to that one.
__global__ void uf_merge_kernel(Cell c, int *lab, unsigned *err)
{
    const long long n = (long long)c.nx * c.ny * c.nz, plane = (long long)c.nx * c.ny;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        if (__ldcg(lab + i) < 0) continue;
        const int x = (int)(i % c.nx);
        const long long r = i / c.nx;
        const int y = (int)(r % c.ny), z = (int)(r / c.ny);
        const bool left = x > 0 && __ldcg(lab + i - 1) >= 0;
        if (left && (x & 31) == 0) uf_union(lab, (int)i, (int)(i - 1), n, err);
        if (y > 0 && __ldcg(lab + i - c.nx) >= 0 && !(left && __ldcg(lab + i - c.nx - 1) >= 0))
            uf_union(lab, (int)i, (int)(i - c.nx), n, err);
        if (z > 0 && __ldcg(lab + i - plane) >= 0 && !(left && __ldcg(lab + i - plane - 1) >= 0))
            uf_union(lab, (int)i, (int)(i - plane), n, err);
    }
}

// face voxel j of axis a (0 = x, 1 = y, 2 = z) on side hi (0/1) of the cell
__device__ __forceinline__ long long face_index(const Cell &c, int a, int hi, long long j)
{
    long long u, v;
    if (a == 0) { u = j % c.ny; v = j / c.ny; return (v * c.ny + u) * c.nx + (hi ? c.nx - 1 : 0); }
    if (a == 1) { u = j % c.nx; v = j / c.nx; return (v * c.ny + (hi ? c.ny - 1 : 0)) * c.nx + u; }
    u = j % c.nx; v = j / c.nx; return ((long long)(hi ? c.nz - 1 : 0) * c.ny + v) * c.nx + u;
}

__host__ __device__ __forceinline__ long long face_count(const Cell &c, int a)
{
    return a == 0 ? (long long)c.ny * c.nz : a == 1 ? (long long)c.nx * c.nz : (long long)c.nx * c.ny;
}

// voxels per row of a face (face_index runs along it first)
__device__ __forceinline__ long long face_width(const Cell &c, int a) { return a == 0 ? c.ny : c.nx; }

// Counters of a percolation call.
struct Perc {
    unsigned bits, err;      // the result, error bits
    int comps, pairs;        // components that touch a face; joins found
};

// Per component that touches a face of the cell: the faces it touches (bit
// 2 a + hi), a compact number and its root.  The face voxels' labels become
// their roots, and nothing else is written to the labels here: a find that
// moved nodes up could put an older label back over a root.
__global__ void face_components_kernel(Cell c, int *lab, unsigned *faces, int *id, int *root, Perc *pc)
{
    const long long n = (long long)c.nx * c.ny * c.nz;
    for (int f = 0; f < 6; ++f) {
        const int a = f >> 1, hi = f & 1;
        const long long m = face_count(c, a);
        for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < m; j += (long long)gridDim.x * blockDim.x) {
            const long long i = face_index(c, a, hi, j);
            if (__ldcg(lab + i) < 0) continue;
            const int r = uf_root(lab, (int)i, n, &pc->err);
            if (r != (int)i) __stcg(lab + i, r);
            if ((__ldcg(faces + r) >> f) & 1u) continue;
            // the first to set a bit of the component numbers it
            if (atomicOr(faces + r, 1u << f) == 0u) {
                const int k = atomicAdd(&pc->comps, 1);
                id[r] = k;
                root[k] = r;
            }
        }
    }
}

// The joins across a common face of neighbouring tiles, (axis, component on
// the high face, component on the low face): where a neighbour on the face
// makes the same join, it is left to that one.
__global__ void face_pairs_kernel(Cell c, const int *lab, const int *id, int2 *pair, Perc *pc)
{
    for (int a = 0; a < 3; ++a) {
        const long long m = face_count(c, a), w = face_width(c, a);
        for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < m; j += (long long)gridDim.x * blockDim.x) {
            const int h = lab[face_index(c, a, 1, j)], l = lab[face_index(c, a, 0, j)];
            if (h < 0 || l < 0) continue;
            if (j % w && lab[face_index(c, a, 1, j - 1)] == h && lab[face_index(c, a, 0, j - 1)] == l) continue;
            if (j >= w && lab[face_index(c, a, 1, j - w)] == h && lab[face_index(c, a, 0, j - w)] == l) continue;
            const int ch = id[h], cl = id[l];
            if (ch < 0 || cl < 0) { atomicOr(&pc->err, 4u); continue; }      // a label that is no numbered root
            pair[atomicAdd(&pc->pairs, 1)] = make_int2((int)((unsigned)ch | (unsigned)a << 30), cl);
        }
    }
}

// The tiling: node t * comps + k is component k of tile t = (tz 3 + ty) 3 + tx.
// Joins of all tiles, then the faces of the tiling that every joined
// component touches, then the axes that one crosses.  The three parts need
// all threads to have finished the one before.
__device__ __forceinline__ int tile_coord(int t, int a) { return a == 0 ? t % 3 : a == 1 ? t / 3 % 3 : t / 9; }

__device__ void tiles_join(const int2 *pair, int np, int nc, int *node, Perc *pc, long long first, long long stride)
{
    for (long long j = first; j < 27ll * np; j += stride) {
        const int t = (int)(j / np);
        const int2 p = pair[j % np];
        const int a = (unsigned)p.x >> 30;
        if (tile_coord(t, a) == 2) continue;
        const int up = a == 0 ? 1 : a == 1 ? 3 : 9;
        uf_union(node, t * nc + (p.x & 0x3fffffff), (t + up) * nc + p.y, 27ll * nc, &pc->err);
    }
}

__device__ void tiles_touch(const unsigned *faces, const int *root, int nc, int *node, unsigned *touch, Perc *pc,
                            long long first, long long stride)
{
    for (long long j = first; j < 27ll * nc; j += stride) {
        const int t = (int)(j / nc);
        unsigned b = faces[root[j % nc]];
        for (int a = 0; a < 3; ++a) {
            const int u = tile_coord(t, a);
            if (u != 0) b &= ~(1u << (2 * a));
            if (u != 2) b &= ~(2u << (2 * a));
        }
        if (b) atomicOr(touch + uf_find(node, (int)j, 27ll * nc, &pc->err), b);
    }
}

__device__ void tiles_check(const unsigned *touch, int nc, Perc *pc, long long first, long long stride)
{
    for (long long j = first; j < 27ll * nc; j += stride) {
        const unsigned b = touch[j] & (touch[j] >> 1);       // both faces of axis a: bit 2 a
        if (b & 0x15u) atomicOr(&pc->bits, (b & 1u) | ((b >> 2 & 1u) << 1) | ((b >> 4 & 1u) << 2));
    }
}

// A few components (the usual case: most pores are one component) are joined
// by one block in shared memory, where the contended links of the large ones
// cost a twentieth of L2's; the rest in global memory, a launch per part.
// 80^3: 399 us for joining every face voxel in global memory -> 19 us for the distinct joins.
constexpr int SMALL_NODES = 5616, SMALL_JOINS = 1 << 17;
__device__ __forceinline__ bool tiles_small(const Perc *pc) { return 27 * (long long)pc->comps <= SMALL_NODES && 27ll * pc->pairs <= SMALL_JOINS; }

__global__ void __launch_bounds__(1024) tiles_small_kernel(const int2 *pair, const unsigned *faces, const int *root, Perc *pc)
{
    __shared__ int node[SMALL_NODES];
    __shared__ unsigned touch[SMALL_NODES];
    if (!tiles_small(pc)) return;
    const int nc = pc->comps;
    for (int j = threadIdx.x; j < 27 * nc; j += blockDim.x) { node[j] = j; touch[j] = 0u; }
    __syncthreads();
    tiles_join(pair, pc->pairs, nc, node, pc, threadIdx.x, blockDim.x);
    __syncthreads();
    tiles_touch(faces, root, nc, node, touch, pc, threadIdx.x, blockDim.x);
    __syncthreads();
    tiles_check(touch, nc, pc, threadIdx.x, blockDim.x);
}

__global__ void tiles_large_kernel(int part, const int2 *pair, const unsigned *faces, const int *root, int *node, unsigned *touch, Perc *pc)
{
    if (tiles_small(pc)) return;
    const int nc = pc->comps;
    const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
    if (part == 0)
        for (long long j = first; j < 27ll * nc; j += stride) { node[j] = (int)j; touch[j] = 0u; }
    else if (part == 1) tiles_join(pair, pc->pairs, nc, node, pc, first, stride);
    else if (part == 2) tiles_touch(faces, root, nc, node, touch, pc, first, stride);
    else tiles_check(touch, nc, pc, first, stride);
}

int grid_for(long long n) { return (int)std::min<long long>((n + GTPB - 1) / GTPB, 148ll * 16); }

}  // namespace

extern "C" int lbm_trig_structure3d(lbm_ctx *ctx, int size, int n_modes, const int32_t *q, const double *phases,
                                    const double *pts, double scale, double porosity, uint8_t *solid_out,
                                    double *threshold)
{
    if (!ctx) return LBM_EINPUT;
    if (!q || !phases || !pts || !solid_out || !threshold) return lbm_fail_input(ctx, "null argument");
    if (size <= 0 || size > 1024 || n_modes <= 0) return lbm_fail_input(ctx, "bad size or mode count");
    if (!(porosity >= 0.0 && porosity <= 1.0)) return lbm_fail_input(ctx, "porosity must lie in [0, 1]");
    CK(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    const long long n = (long long)size * size * size;
    DevMem d_q(s), d_ph(s), d_pts(s), d_field(s), d_sel(s), d_solid(s);
    CK(d_q.alloc(sizeof(int) * 3 * (size_t)n_modes));
    CK(d_ph.alloc(sizeof(double) * (size_t)n_modes));
    CK(d_pts.alloc(sizeof(double) * (size_t)size));
    CK(d_field.alloc(sizeof(double) * (size_t)n));
    CK(d_sel.alloc(sizeof(Select)));
    CK(cudaMemcpyAsync(d_q.p, q, sizeof(int) * 3 * (size_t)n_modes, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(d_ph.p, phases, sizeof(double) * (size_t)n_modes, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(d_pts.p, pts, sizeof(double) * (size_t)size, cudaMemcpyHostToDevice, s));
    auto *field = static_cast<double *>(d_field.p);
    auto *sel = static_cast<Select *>(d_sel.p);
    // as many rows as fit a block; a longer row takes a block by itself
    const int rows = std::max(1, std::min(GTPB / size, 16));
    const int threads = rows > 1 ? (rows * size + 31) / 32 * 32 : std::min(GTPB, (size + 31) / 32 * 32);
    trig_field_kernel<<<(size * size + rows - 1) / rows, threads, 0, s>>>(
        size, rows, n_modes, static_cast<const int *>(d_q.p), static_cast<const double *>(d_ph.p),
        static_cast<const double *>(d_pts.p), scale, field);
    CK(cudaGetLastError());

    // numpy's linear quantile: virtual index (n - 1) q, its floor and the next
    const double vi = (double)(n - 1) * porosity;
    const long long lo = (long long)std::floor(vi);
    const double gamma = vi - (double)lo;
    select_init_kernel<<<1, 256, 0, s>>>(sel, (unsigned long long)lo);
    CK(cudaGetLastError());
    // few blocks of several keys per thread: every block adds 256 bins
    const int sgrid = (int)std::min<long long>((n + 8 * GTPB - 1) / (8 * GTPB), 148ll * 4);
    for (int shift = 56; shift >= 0; shift -= 8) {
        select_digit_kernel<<<sgrid, GTPB, 0, s>>>(field, n, shift, sel);
        CK(cudaGetLastError());
    }
    const int has_next = lo + 1 < n ? 1 : 0;
    if (has_next) {
        select_next_kernel<<<sgrid, GTPB, 0, s>>>(field, n, sel);
        CK(cudaGetLastError());
    }
    select_threshold_kernel<<<1, 1, 0, s>>>(sel, gamma, has_next);
    CK(cudaGetLastError());

    uint8_t *dst = solid_out;
    const bool dev = lbm_is_device_ptr(solid_out);
    if (!dev) {
        CK(d_solid.alloc((size_t)n));
        dst = static_cast<uint8_t *>(d_solid.p);
    }
    threshold_kernel<<<grid_for(n), GTPB, 0, s>>>(field, n, sel, dst);
    CK(cudaGetLastError());
    double t = 0.0;
    CK(cudaMemcpyAsync(&t, &sel->t, sizeof(double), cudaMemcpyDeviceToHost, s));
    if (!dev) CK(cudaMemcpyAsync(solid_out, dst, (size_t)n, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    *threshold = t;
    return LBM_OK;
}

extern "C" int lbm_percolates3d(lbm_ctx *ctx, const uint8_t *solid, int nx, int ny, int nz, int perc[3])
{
    if (!ctx) return LBM_EINPUT;
    if (!solid || !perc) return lbm_fail_input(ctx, "null argument");
    if (nx <= 0 || ny <= 0 || nz <= 0) return lbm_fail_input(ctx, "bad dimensions");
    const long long n = 27ll * nx * ny * nz;
    if (n >= (1ll << 31)) return lbm_fail_input(ctx, "3x3x3 tiling exceeds 2^31 voxels");
    CK(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    const long long cell = (long long)nx * ny * nz;
    DevMem d_solid(s), d_cell(s), d_nodes(s), d_pc(s);
    const uint8_t *src = solid;
    if (!lbm_is_device_ptr(solid)) {
        CK(d_solid.alloc((size_t)cell));
        CK(cudaMemcpyAsync(d_solid.p, solid, (size_t)cell, cudaMemcpyHostToDevice, s));
        src = static_cast<const uint8_t *>(d_solid.p);
    }
    const Cell c{nx, ny, nz};
    // components that touch a face: at most one per face voxel; joins: at
    // most one per voxel of three faces
    const long long joins = face_count(c, 0) + face_count(c, 1) + face_count(c, 2);
    const long long comps = std::min(2 * joins, cell);
    CK(d_cell.alloc(sizeof(int) * 3 * (size_t)cell));
    CK(d_nodes.alloc(sizeof(int) * ((2 * 27 + 1) * (size_t)comps + 2 * (size_t)joins)));
    CK(d_pc.alloc(sizeof(Perc)));
    CK(cudaMemsetAsync(d_pc.p, 0, sizeof(Perc), s));
    auto *lab = static_cast<int *>(d_cell.p), *id = lab + cell;
    auto *faces = reinterpret_cast<unsigned *>(id + cell);
    auto *pair = static_cast<int2 *>(d_nodes.p);
    auto *root = reinterpret_cast<int *>(pair + joins), *node = root + comps;
    auto *touch = reinterpret_cast<unsigned *>(node + 27 * comps);
    auto *pc = static_cast<Perc *>(d_pc.p);
    const long long warps = (long long)ny * nz * ((nx + 31) / 32);
    uf_init_kernel<<<grid_for(32 * warps), GTPB, 0, s>>>(src, c, lab, id, faces);
    CK(cudaGetLastError());
    uf_merge_kernel<<<grid_for(cell), GTPB, 0, s>>>(c, lab, &pc->err);
    CK(cudaGetLastError());
    const long long fmax = std::max({face_count(c, 0), face_count(c, 1), face_count(c, 2)});
    face_components_kernel<<<grid_for(fmax), GTPB, 0, s>>>(c, lab, faces, id, root, pc);
    CK(cudaGetLastError());
    face_pairs_kernel<<<grid_for(fmax), GTPB, 0, s>>>(c, lab, id, pair, pc);
    CK(cudaGetLastError());
    tiles_small_kernel<<<1, 1024, 0, s>>>(pair, faces, root, pc);
    CK(cudaGetLastError());
    for (int part = 0; part < 4; ++part) {
        tiles_large_kernel<<<grid_for(27 * fmax), GTPB, 0, s>>>(part, pair, faces, root, node, touch, pc);
        CK(cudaGetLastError());
    }
    Perc h{};
    CK(cudaMemcpyAsync(&h, pc, sizeof(h), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (h.err) return lbm_fail_input(ctx, "percolation labelling did not settle (iteration bound reached)");
    for (int a = 0; a < 3; ++a) perc[a] = (h.bits >> a) & 1u;
    return LBM_OK;
}
