// Reduced-precision D3Q19 kernels: shifted populations stored as FP32, FP16
// (power-of-two scaled) or BF16, collision in FP32, flux reduced in FP64.
#include <algorithm>

#include "step3d_slots.cuh"

namespace lbm {

cudaError_t launch_init3d_f64(void *A, long long plane, long long n, cudaStream_t s);
cudaError_t launch_canon3d_f64(const Solve3 &S, long long done, double *f, float *u, cudaStream_t s);

#define LBM_ODD(ST, V, W) step3d_odd_kernel<ST, odd_lp(V).npt, odd_lp(V).minb, W>
#define LBM_ODDP(ST, W) step3d_odd_pair_kernel<ST, odd_lp(3).minb, W>
#define LBM_EVEN(ST, V, W) step3d_even_kernel<ST, even_lp(V).minb, W, even_meta(V)>
#define LBM_EVENA(ST, V, W) step3d_even_async_kernel<ST, even_lp(V).minb, W>
#define LBM_EVENG(ST, V, W) step3d_even_group_kernel<ST, even_lp(V).minb, W, even_meta(V)>
#define LBM_EVENL(ST, V, W) step3d_even_links_kernel<ST, even_lp(V).minb, W, even_meta(V), even_pair(V)>
#define LBM_EVENW(ST, V, W) step3d_even_links1_kernel<ST, even_lp(V).minb, W, even_meta(V)>
#define LBM_ODDB(ST, W, L) step3d_odd_bulk_kernel<ST, odd_lp(4).minb, W, L>
#define LBM_PULL(ST, Q, W) step3d_pull_kernel<ST, pull_minb(Q), W, pull_meta(Q)>
#define LBM_PULL1(ST, Q, W) step3d_pull1_kernel<ST, pull_minb(Q), W, pull_meta(Q)>
#define LBM_PULLG(ST, Q, W) step3d_pull_group_kernel<ST, pull_minb(Q), W, pull_meta(Q)>

// Persistent CTAs of the bulk-staged odd kernel per (storage, tau = 1, device),
// set by prepare_bulk once its shared-memory ring has been allowed.
static int g_bulk_ctas[3][2][64];

template <class ST, bool W>
static int prepare_bulk(int dev)
{
    using T = typename ST::T;
    const void *k[2] = {(const void *)LBM_ODDB(ST, W, false), (const void *)LBM_ODDB(ST, W, true)};
    const unsigned smem = odd_bulk_smem<T>();
    int nb = 0, sms = 0;
    for (const void *f : k) {
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, f, ODD_BULK_THREADS, smem) != cudaSuccess) return 0;
    }
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    g_bulk_ctas[ST::code - 1][W ? 1 : 0][dev] = nb * sms;
    return nb;
}

cudaError_t prepare_step3d_lp(int dev)
{
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    const bool ok = prepare_bulk<StoreF32, true>(dev) > 0 && prepare_bulk<StoreF32, false>(dev) > 0
                 && prepare_bulk<StoreF16, true>(dev) > 0 && prepare_bulk<StoreF16, false>(dev) > 0
                 && prepare_bulk<StoreBF16, true>(dev) > 0 && prepare_bulk<StoreBF16, false>(dev) > 0;
    return ok ? cudaSuccess : cudaErrorInvalidConfiguration;
}

template <class ST, bool W, bool L>
static cudaError_t launch_bulk(dim3 grid, cudaStream_t s, const SlotArgs<L> &a)
{
    int dev = 0;
    cudaGetDevice(&dev);
    const int ctas = (dev >= 0 && dev < 64) ? g_bulk_ctas[ST::code - 1][W ? 1 : 0][dev] : 0;
    if (ctas <= 0) return cudaErrorInvalidConfiguration;   // prepare_step3d_lp not run on this device
    grid.x = std::min<unsigned>(grid.x, (unsigned)ctas);
    return launch_pdl(LBM_ODDB(ST, W, L), grid, ODD_BULK_THREADS, odd_bulk_smem<typename ST::T>(), s, a);
}

template <class ST, bool W>
static cudaError_t launch_lp(int v, bool odd, dim3 grid, cudaStream_t s, const StepArgs &a)
{
    if (v < 0 || v >= NVAR_LP + NVAR_PULL) return cudaErrorInvalidValue;
    if (v >= NVAR_LP) {
        switch (v - NVAR_LP) {
        case 0: LBM_PULL(ST, 0, W)<<<grid, TPB, 0, s>>>(a); break;
        // 1 runs step3d_pull_slots_kernel, or without neighbour records as 2
        case 2: LBM_PULL(ST, 2, W)<<<grid, TPB, 0, s>>>(a); break;
        case 3: LBM_PULL1(ST, 3, W)<<<grid, TPB, 0, s>>>(a); break;
        case 4: LBM_PULLG(ST, 4, W)<<<grid, TPB, 0, s>>>(a); break;
        case 5: LBM_PULLG(ST, 5, W)<<<grid, TPB, 0, s>>>(a); break;
        default: return cudaErrorInvalidValue;
        }
        return cudaGetLastError();
    }
    const int vo = v / NVAR_EVEN_LP, ve = v % NVAR_EVEN_LP;
    if (odd) {
        switch (vo) {
        case 0: LBM_ODD(ST, 0, W)<<<grid, TPB, 0, s>>>(a); break;
        case 1: LBM_ODD(ST, 1, W)<<<grid, TPB, 0, s>>>(a); break;
        case 2: LBM_ODD(ST, 2, W)<<<grid, TPB, 0, s>>>(a); break;
        case 3: LBM_ODDP(ST, W)<<<grid, TPB, 0, s>>>(a); break;
        default: {
            const cudaError_t e = launch_bulk<ST, W, true>(grid, s, SlotArgs<true>{a});
            if (e != cudaSuccess) return e;
        } break;
        }
    } else {
        switch (ve) {
        case 0: LBM_EVEN(ST, 0, W)<<<grid, TPB, 0, s>>>(a); break;
        case 1: LBM_EVEN(ST, 1, W)<<<grid, TPB, 0, s>>>(a); break;
        case 2: LBM_EVEN(ST, 2, W)<<<grid, TPB, 0, s>>>(a); break;
        case 3: LBM_EVEN(ST, 3, W)<<<grid, TPB, 0, s>>>(a); break;
        case 4: LBM_EVENA(ST, 4, W)<<<grid, TPB, 0, s>>>(a); break;
        case 5: LBM_EVENA(ST, 5, W)<<<grid, TPB, 0, s>>>(a); break;
        case 6: LBM_EVENG(ST, 6, W)<<<grid, TPB, 0, s>>>(a); break;
        case 7: LBM_EVENG(ST, 7, W)<<<grid, TPB, 0, s>>>(a); break;
        case 8: LBM_EVENL(ST, 8, W)<<<grid, TPB, 0, s>>>(a); break;
        case 9: LBM_EVENL(ST, 9, W)<<<grid, TPB, 0, s>>>(a); break;
        case 10: LBM_EVENL(ST, 10, W)<<<grid, TPB, 0, s>>>(a); break;
        case 11: LBM_EVENL(ST, 11, W)<<<grid, TPB, 0, s>>>(a); break;
        case 12: LBM_EVENL(ST, 12, W)<<<grid, TPB, 0, s>>>(a); break;
        case 13: LBM_EVENW(ST, 13, W)<<<grid, 2 * TPB, 0, s>>>(a); break;
        default: LBM_EVENW(ST, 14, W)<<<grid, 2 * TPB, 0, s>>>(a); break;
        }
    }
    return cudaGetLastError();
}

// Step of a single solve whose records travel in the launch (variants with
// slots_variant): the pull form, or the bulk-staged odd and grouped link-slot
// even steps.  a.a.nwork: items of the bulk-staged launch.
template <class ST, bool W>
static cudaError_t launch_slots_lp(bool pull, bool odd, bool split, int ntiles, int ndir, cudaStream_t s, SlotArgs<false> a)
{
    if (pull)
        return split ? launch_pdl(step3d_pull_slots_kernel<ST, W, true, 128, 6, false>, dim3(2 * ntiles, ndir), 128, 0, s, a)
                     : launch_pdl(step3d_pull_slots_kernel<ST, W, false, 256, 3, false>, dim3(ntiles, ndir), 256, 0, s, a);
    if (odd) {
        a.a.nwork = ntiles * ndir;
        return launch_bulk<ST, W, false>(dim3(a.a.nwork), s, a);
    }
    return split ? launch_pdl(step3d_links_slots_kernel<ST, W, true, 256, 4, false>, dim3(2 * ntiles), 256, 0, s, a)
                 : launch_pdl(step3d_links_slots_kernel<ST, W, false, 256, 4, false>, dim3(ntiles), 256, 0, s, a);
}

cudaError_t launch_slots3d_lp(int prec, bool pull, bool w1, bool odd, bool split, int ntiles, int ndir, cudaStream_t s,
                              const SlotArgs<false> &a)
{
    switch (prec) {
    case 1: return w1 ? launch_slots_lp<StoreF32, true>(pull, odd, split, ntiles, ndir, s, a) : launch_slots_lp<StoreF32, false>(pull, odd, split, ntiles, ndir, s, a);
    case 2: return w1 ? launch_slots_lp<StoreF16, true>(pull, odd, split, ntiles, ndir, s, a) : launch_slots_lp<StoreF16, false>(pull, odd, split, ntiles, ndir, s, a);
    case 3: return w1 ? launch_slots_lp<StoreBF16, true>(pull, odd, split, ntiles, ndir, s, a) : launch_slots_lp<StoreBF16, false>(pull, odd, split, ntiles, ndir, s, a);
    default: return cudaErrorInvalidValue;
    }
}

template <class ST, bool W>
static cudaError_t launch_list_lp(bool pull, bool odd, dim3 grid, cudaStream_t s, const SlotArgs<true> &a)
{
    if (pull) return launch_pdl(step3d_pull_slots_kernel<ST, W, false, 256, 3, true>, grid, 256, 0, s, a);
    if (odd) return launch_bulk<ST, W, true>(grid, s, a);
    return launch_pdl(step3d_links_slots_kernel<ST, W, false, 256, 4, true>, grid, 256, 0, s, a);
}

cudaError_t launch_slots3d_list(int prec, bool pull, bool w1, bool odd, dim3 grid, cudaStream_t s, const StepArgs &args)
{
    const SlotArgs<true> a{args};
    switch (prec) {
    case 0: return launch_slots3d_list_f64(w1, odd, grid, s, a);
    case 1: return w1 ? launch_list_lp<StoreF32, true>(pull, odd, grid, s, a) : launch_list_lp<StoreF32, false>(pull, odd, grid, s, a);
    case 2: return w1 ? launch_list_lp<StoreF16, true>(pull, odd, grid, s, a) : launch_list_lp<StoreF16, false>(pull, odd, grid, s, a);
    case 3: return w1 ? launch_list_lp<StoreBF16, true>(pull, odd, grid, s, a) : launch_list_lp<StoreBF16, false>(pull, odd, grid, s, a);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_step3d_lp(int prec, int variant, bool w1, bool odd, dim3 grid, cudaStream_t s, const StepArgs &a)
{
    variant = kernel_variant(prec, variant);     // the two-lattice AA form runs the in-place kernels
    switch (prec) {
    case 1: return w1 ? launch_lp<StoreF32, true>(variant, odd, grid, s, a) : launch_lp<StoreF32, false>(variant, odd, grid, s, a);
    case 2: return w1 ? launch_lp<StoreF16, true>(variant, odd, grid, s, a) : launch_lp<StoreF16, false>(variant, odd, grid, s, a);
    case 3: return w1 ? launch_lp<StoreBF16, true>(variant, odd, grid, s, a) : launch_lp<StoreBF16, false>(variant, odd, grid, s, a);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_init3d(int prec, void *A, long long plane, long long n, cudaStream_t s)
{
    switch (prec) {
    case 0: return launch_init3d_f64(A, plane, n, s);
    case 1: init3d_kernel<StoreF32><<<1184, 256, 0, s>>>(A, plane, n); break;
    case 2: init3d_kernel<StoreF16><<<1184, 256, 0, s>>>(A, plane, n); break;
    case 3: init3d_kernel<StoreBF16><<<1184, 256, 0, s>>>(A, plane, n); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_canon3d(int prec, const Solve3 &S, long long done, double *f, float *u, cudaStream_t s)
{
    switch (prec) {
    case 0: return launch_canon3d_f64(S, done, f, u, s);
    case 1: canon3d_kernel<StoreF32><<<1184, 256, 0, s>>>(S, done, f, u); break;
    case 2: canon3d_kernel<StoreF16><<<1184, 256, 0, s>>>(S, done, f, u); break;
    case 3: canon3d_kernel<StoreBF16><<<1184, 256, 0, s>>>(S, done, f, u); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Pore voxels per block of SCAN_WORDS mask words.
__global__ void word_sums_kernel(const uint32_t *mask, long long nwords, unsigned *bsum)
{
    __shared__ unsigned sh[TPB / 32];
    unsigned c = 0;
    for (int q = threadIdx.x; q < SCAN_WORDS; q += TPB) {
        const long long w = (long long)blockIdx.x * SCAN_WORDS + q;
        if (w < nwords) c += __popc(~mask[w]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = 0;
        for (int i = 0; i < TPB / 32; ++i) t += sh[i];
        bsum[blockIdx.x] = t;
    }
}

// wpre[w] = pore voxels before word w (exclusive scan), from per-block offsets.
__global__ void word_scan_kernel(const uint32_t *mask, long long nwords, const unsigned *boff, uint32_t *wpre)
{
    constexpr int PER = SCAN_WORDS / TPB;       // consecutive words per thread
    __shared__ unsigned sh[TPB / 32];
    const long long w0 = (long long)blockIdx.x * SCAN_WORDS + (long long)threadIdx.x * PER;
    unsigned c[PER], t = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        c[q] = (w0 + q < nwords) ? __popc(~mask[w0 + q]) : 0u;
        t += c[q];
    }
    // exclusive scan of t across the block
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned incl = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) sh[wid] = incl;
    __syncthreads();
    unsigned wbase = 0;
    for (int i = 0; i < wid; ++i) wbase += sh[i];
    unsigned run = boff[blockIdx.x] + wbase + incl - t;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        if (w0 + q < nwords) wpre[w0 + q] = run;
        run += c[q];
    }
}

// fnode[rank] = linear index of every pore voxel.
__global__ void scatter_fnode_kernel(const uint32_t *mask, const uint32_t *wpre, long long nwords, int wpr,
                                     int nx, uint32_t *fnode)
{
    for (long long w = blockIdx.x * (long long)blockDim.x + threadIdx.x; w < nwords;
         w += (long long)gridDim.x * blockDim.x) {
        uint32_t f = ~mask[w];
        unsigned at = wpre[w];
        const long long row = w / wpr;
        const int x0 = (int)(w - row * wpr) * 32;
        while (f) {
            const int b = __ffs(f) - 1;
            f &= f - 1u;
            fnode[at++] = (uint32_t)(row * nx + x0 + b);
        }
    }
}

// Neighbour records of every pore voxel (see meta_nbrs).
__global__ void build_meta_kernel(Solve3 S, uint4 *meta, uint2 *meta2)
{
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < (unsigned)S.nfluid;
         i += gridDim.x * blockDim.x) {
        int x, y, z;
        coords3(S, S.fnode[i], x, y, z);
        CNb nb;
        compact_nbrs(S, i, x, y, z, nb);
        const int ny = S.ny, nz = S.nz, wpr = S.wpr;
        const int row = z * ny + y;
        const int ym = y == 0 ? ny - 1 : y - 1, yp = y == ny - 1 ? 0 : y + 1;
        const int zm = z == 0 ? nz - 1 : z - 1, zp = z == nz - 1 ? 0 : z + 1;
        auto off = [&](int yy, int zz, int k) -> unsigned {
            return nb.idx[k] - S.wpre[(unsigned)(zz * ny + yy) * wpr];
        };
        unsigned link = nb.solid & 0x7ffffu;
        link |= (x == 0 ? LK_XLO : 0u) | (x == S.nx - 1 ? LK_XHI : 0u) | (y == 0 ? LK_YLO : 0u) |
                (y == ny - 1 ? LK_YHI : 0u) | (z == 0 ? LK_ZLO : 0u) | (z == nz - 1 ? LK_ZHI : 0u);
        meta[i] = make_uint4((unsigned)row, link,
                             off(ym, z, k_of(0, -1, 0)) | (off(yp, z, k_of(0, 1, 0)) << 16),
                             off(y, zm, k_of(0, 0, -1)) | (off(y, zp, k_of(0, 0, 1)) << 16));
        meta2[i] = make_uint2(off(ym, zm, k_of(0, -1, -1)) | (off(yp, zm, k_of(0, 1, -1)) << 16),
                              off(ym, zp, k_of(0, -1, 1)) | (off(yp, zp, k_of(0, 1, 1)) << 16));
    }
}

__global__ void advance3d_kernel(Solve3 *solves, int nsolves, long long steps)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nsolves && solves[i].st->phase < PH_DONE) solves[i].st->s_base += steps;
}

}  // namespace lbm
