// Step kernels that start early: the steps, slots and bits of the kernels of
// engine3d.cuh, arranged so that a block's first population load is not the
// last of a chain of dependent ones.
//
// The kernels of engine3d.cuh read the work item, then the solve record it
// names, then that solve's state, then the neighbour record and the row
// starts, and only then populations: five trips to L2 or DRAM, some 3 us of
// the 7 us a tile of the 128^3 workload takes.  Here
//   - a single solve's records travel in the launch parameters (constant
//     bank) and the item is the block index; a batch's item and record are
//     read as before (LIST);
//   - all that does not change during a solve (item, record, neighbour
//     records, row starts, slots) is read before griddepcontrol.wait, so that
//     with programmatic launches it overlaps the end of the step before;
//   - populations are requested before the solve's state has arrived (a
//     single solve launches its unfinished directions only; a batch lists
//     finished solves until they are polled, their record says so);
//   - whether a step reduces is one bit of State3::redm instead of a division
//     of the 64-bit step number per thread, and the flux sums of steps that
//     do not reduce are not formed.
// Per step (before -> after, B200, all directions; the first figure of FP64
// includes only the operator of d3q19.cuh): FP64 one direction of 32^3 7.5 ->
// 3.8 us, 64^3 28.2 -> 20.6, 80^3 74.0 -> 62.7 (86 % of the copy bandwidth);
// FP32 pull 96^3 47.0 -> 41.2 (82 %), 97 x 61 x 75 with four directions 30.6
// -> 23.7; BF16 128^3 62.8 -> 56.4; FP16 batch of eight structures 119.8 ->
// 106.8 (all directions in every step; stepped in groups that fit L2, see
// plain_group, 80^3 takes 47.7, 96^3 34.7 and 97 x 61 x 75 22).  What is left:
// FP64 and FP32 run near the copy bandwidth where the lattices exceed L2; the
// 16-bit even step waits on its scattered accesses.
#pragma once
#include "engine3d.cuh"

namespace lbm {

// Step number, and whether the step reduces, of a running solve.
struct StepHead {
    long long n;
    bool run, red;
};
__device__ __forceinline__ StepHead step_head(const Solve3 &S, const StepArgs &a)
{
    const State3 &st = *S.st;
    StepHead h;
    h.n = st.s_base + a.step + 1;
    h.run = st.phase < PH_DONE;
    h.red = (st.redm >> a.bit) & 1ull;
    return h;
}
// Step number modulo 4 (the lattices of the two-lattice forms): known from
// the launch where every solve of it starts at a multiple of 4, so that the
// populations' addresses do not wait for the state.
__device__ __forceinline__ int step_n4(const Solve3 &S, const StepArgs &a)
{
    return a.n4 >= 0 ? a.n4 : (int)((S.st->s_base + a.step + 1) & 3);
}
// Lattice the AA step reads and the one it writes (aa_src, aa_dst).
template <class T>
__device__ __forceinline__ const T *slots_src(const Solve3 &S, int n4) { return static_cast<const T *>((S.aa2 && (((n4 + 3) >> 1) & 1)) ? S.B : S.A); }
template <class T>
__device__ __forceinline__ T *slots_dst(const Solve3 &S, int n4) { return static_cast<T *>((S.aa2 && ((n4 >> 1) & 1)) ? S.B : S.A); }

// Split tiles (SPLIT, Solve3::split): a tile's 512 voxels over several short
// blocks.  Whole tiles fill a few waves badly (64^3 in FP64: 924 tiles on 296
// block slots), and a small lattice leaves SMs idle (32^3: 40 tiles).  A
// block then holds virtual threads t = part * HT .. + HT - 1 of the canonical
// order (thread t sums voxels t and t + TPB, a warp's 32 sums meet in a
// shuffle tree, the 8 warps' in order) in its lower half, their second voxels
// in its upper half, and leaves the sums of its warps one by one: 8 partials
// per tile, which reduce3d_kernel adds in order, so the flux has the same bits.
// Whole tiles stay for batches and large lattices, whose partials would take
// 12 KB per tile (DEFER_SLOTS x 8 x 3 doubles).  Against whole tiles: one
// direction of 32^3 in FP64 6.2 -> 4.0 us per step (blocks of 128), 64^3 23.4
// -> 20.6, BF16 128^3 60.3 -> 56.4.

// Voxel (within the tile) of thread tid of part `part` of a split tile, NT
// threads, V adjacent voxels each.
template <int NT, int V>
__device__ __forceinline__ unsigned split_voxel(int part, unsigned tid)
{
    constexpr unsigned HT = NT / 2;
    return part * (HT * V) + (tid < HT ? tid * V : TPB + (tid - HT) * V);
}

__device__ __forceinline__ double *partial_slot(const Solve3 &S, const StepArgs &a, int tile, int warp)
{
    const int per = S.split ? TPB / 32 : 1;
    return S.partials + 3ll * (((long long)defer_slot(a) * S.ntiles + tile) * per + warp);
}

// Flux partial of a whole tile from the sums of a full block (finish_tile's
// deferred branch).  Needs a barrier before the next use.
__device__ __forceinline__ void tile_partial(const Solve3 &S, int tile, const StepArgs &a, double (&acc)[3])
{
    __shared__ double sh[TPB / 32][3];
    warp_sum3(acc, sh[threadIdx.x >> 5]);
    __syncthreads();
    if (threadIdx.x < 3) {
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < TPB / 32; ++w) x += sh[w][threadIdx.x];
        partial_slot(S, a, tile, 0)[threadIdx.x] = x;
    }
}

// The 18 link slots of pore voxel i from its neighbour record (see
// step3d_even_links_kernel: slot k - 1 is read for population k and written
// with population opp k).
__device__ __forceinline__ void link_slots(const Solve3 &S, unsigned i, unsigned P, uint4 m, uint2 m2,
                                           unsigned (&sl)[Q3 - 1])
{
    CNb nb;
    meta_nbrs(S, i, m, m2, nb);
#pragma unroll
    for (int k = 1; k < Q3; ++k) {
        const int o = opp3(k);
        sl[k - 1] = ((nb.solid >> o) & 1u) ? (k * P + i) : (o * P + nb.idx[o]);
    }
}

// Stores of populations k and k + 1 at two slots: the 16-bit types round
// both in one conversion, with the bits store_pop would give each.
template <class ST>
__device__ __forceinline__ void store_pops(typename ST::T *A, unsigned s0, typename ST::C v0, unsigned s1, typename ST::C v1,
                                           uint32_t hv, int k)
{
    if constexpr (ST::stochastic) {
        const uint32_t d = ST::sr2(v0, v1, dir_bits(hv, k), dir_bits(hv, k + 1));
        __stcs(reinterpret_cast<unsigned short *>(A + s0), (unsigned short)(d & 0xffffu));
        __stcs(reinterpret_cast<unsigned short *>(A + s1), (unsigned short)(d >> 16));
    } else {
        ST::st(A + s0, v0);
        ST::st(A + s1, v1);
    }
}

// The item of a block: solve record and tile.  False: no item (a batch's
// launch of an empty work list).
template <bool LIST>
__device__ __forceinline__ bool slots_item(const SlotArgs<LIST> &ka, const Solve3 *&S, int &tile, int block)
{
    if constexpr (LIST) {
        if (block >= (ka.a.nwork_dev ? *ka.a.nwork_dev : ka.a.nwork)) return false;
        const int2 item = ka.a.work[block];
        S = ka.a.solves + item.x;
        tile = item.y;
    } else {
        S = ka.s + blockIdx.y;
        tile = block;
    }
    return true;
}

// Does the record say that the solve has finished (control3d_kernel)?  Read
// before the wait, so the note of a pass that is still running may be missed:
// the solve's state, read after the wait, decides then.
__device__ __forceinline__ bool noted_done(const Solve3 &S) { return *static_cast<const volatile int *>(&S.done) != 0; }

// AA step, odd (local: slot k is the voxel's own, written with opp k) or even
// (neighbour: link slots), one voxel per thread at a time: the voxel of a
// split tile's thread, or voxels t and t + TPB of a whole tile.
template <class ST, bool W1, bool EVEN, bool SPLIT, int NT, int MINB, bool LIST>
__global__ void __launch_bounds__(NT, MINB) step3d_aa_kernel(const __grid_constant__ SlotArgs<LIST> ka)
{
    using T = typename ST::T;
    using Cp = typename ST::C;
    static_assert(SPLIT || NT == TPB, "a whole tile takes a full block");
    constexpr int PARTS = SPLIT ? TPB * TILE_NPT / NT : 1, VPT = SPLIT ? 1 : TILE_NPT;
    const StepArgs &a = ka.a;
    const Solve3 *Sp;
    int tile;
    pdl_launch();
    if (!slots_item<LIST>(ka, Sp, tile, blockIdx.x / PARTS)) { pdl_wait(); return; }
    const Solve3 &S = *Sp;
    if (LIST && noted_done(S)) { pdl_wait(); return; }
    const int part = blockIdx.x % PARTS;
    const unsigned P = (unsigned)S.plane, nf = (unsigned)S.nfluid;
    const unsigned i0 = (unsigned)tile * (TPB * TILE_NPT) + (SPLIT ? split_voxel<NT, 1>(part, threadIdx.x) : threadIdx.x);
    uint4 mr[VPT];
    uint2 mr2[VPT];
    unsigned sl[Q3 - 1];
    if constexpr (EVEN) {
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
            const bool v = i0 + j * TPB < nf;
            mr[j] = v ? __ldg(S.meta + (i0 + j * TPB)) : make_uint4(0, 0, 0, 0);
            mr2[j] = v ? __ldg(S.meta2 + (i0 + j * TPB)) : make_uint2(0, 0);
        }
        if (i0 < nf) link_slots(S, i0, P, mr[0], mr2[0], sl);
    }
    pdl_wait();
    const int n4 = step_n4(S, a);
    const T *R = slots_src<T>(S, n4);
    T *W = slots_dst<T>(S, n4);
    const StepHead h = step_head(S, a);
    double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
        const unsigned i = i0 + j * TPB;
        const bool v = i < nf;
        if (EVEN && j && v) link_slots(S, i, P, mr[j], mr2[j], sl);
        Cp g[Q3];
        if (v) {
            g[0] = ST::ld(R + i);
#pragma unroll
            for (int k = 1; k < Q3; ++k) g[k] = ST::ld(R + (EVEN ? sl[k - 1] : k * P + i));
        }
        if (!h.run) return;            // after the loads, which do not wait for the state
        if (!v) continue;
        Cp ux, uy, uz;
        collide3<ST, W1>(g, S, ux, uy, uz);
        const uint32_t hv = voxel_bits<ST>(i, h.n);
        store_pop<ST>(W, i, g[0], hv, 0);
#pragma unroll
        for (int k = 1; k < Q3; k += 2)
            store_pops<ST>(W, EVEN ? sl[opp3(k) - 1] : opp3(k) * P + i, g[k],
                           EVEN ? sl[opp3(k + 1) - 1] : opp3(k + 1) * P + i, g[k + 1], hv, k);
        if (h.red) { acc[0] += (double)ux; acc[1] += (double)uy; acc[2] += (double)uz; }
    }
    if (!h.red) return;
    if constexpr (SPLIT) {
        constexpr int HT = NT / 2;
        __shared__ double su[3][HT];
        if (threadIdx.x >= HT) {
#pragma unroll
            for (int c = 0; c < 3; ++c) su[c][threadIdx.x - HT] = acc[c];
        }
        __syncthreads();
        if (threadIdx.x >= HT) return;
        // a missing second voxel adds +0, which changes no sum of this kind
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] += su[c][threadIdx.x];
        warp_sum3(acc, partial_slot(S, a, tile, part * (HT / 32) + (threadIdx.x >> 5)));
    } else {
        tile_partial(S, tile, a, acc);
    }
}

// Pull step (see step3d_pull_kernel): a thread gathers, collides and stores
// an adjacent voxel pair.
template <class ST, bool W1, bool SPLIT, int NT, int MINB, bool LIST>
__global__ void __launch_bounds__(NT, MINB) step3d_pull_slots_kernel(const __grid_constant__ SlotArgs<LIST> ka)
{
    using T = typename ST::T;
    static_assert(ST::shifted && TILE_NPT == 2, "the pull form is a reduced-precision voxel-pair kernel");
    static_assert(SPLIT || NT == TPB, "a whole tile takes a full block");
    constexpr int PARTS = TPB / NT;
    const StepArgs &a = ka.a;
    const Solve3 *Sp;
    int tile;
    pdl_launch();
    if (!slots_item<LIST>(ka, Sp, tile, blockIdx.x / PARTS)) { pdl_wait(); return; }
    const Solve3 &S = *Sp;
    if (LIST && noted_done(S)) { pdl_wait(); return; }
    const int part = blockIdx.x % PARTS;
    const unsigned tid = threadIdx.x;
    const unsigned P = (unsigned)S.plane, nf = (unsigned)S.nfluid;
    const unsigned i = (unsigned)tile * (TPB * TILE_NPT) + (SPLIT ? split_voxel<NT, 2>(part, tid) : 2u * tid);
    const bool v = i < nf;
    unsigned sa[Q3], sb[Q3];
    if (v) {
        pull_sources<true>(S, i, P, sa);
        if (i + 1u < nf) {
            pull_sources<true>(S, i + 1u, P, sb);
        } else {
#pragma unroll
            for (int k = 0; k < Q3; ++k) sb[k] = k * P + i + 1u;
        }
    }
    pdl_wait();
    // the parity of a step is its launch's (s_base is even)
    const bool odd = !(a.step & 1);
    const T *R = static_cast<const T *>(odd ? S.A : S.B);
    T *W = static_cast<T *>(odd ? S.B : S.A);
    const StepHead h = step_head(S, a);
    float2 g[Q3], u[3] = {};
    if (v) {
        ST::ld2(R + i, g[0].x, g[0].y);
#pragma unroll
        for (int k = 1; k < Q3; ++k) {
            g[k].x = ST::ld(R + sa[k]);
            g[k].y = ST::ld(R + sb[k]);
        }
    }
    if (!h.run) return;
    if (v) {
        collide3x2<ST, W1>(g, S, u);
        const uint32_t h0 = voxel_bits<ST>(i, h.n), h1 = voxel_bits<ST>(i + 1u, h.n);
#pragma unroll
        for (int k = 0; k < Q3; ++k)
            ST::st2(W + (k * P + i), g[k].x, g[k].y, dir_bits(h0, k), dir_bits(h1, k));
    }
    if (!h.red) return;
    // virtual threads: tid < NT of this part, first voxel NT * part + tid of
    // the tile (split: the block's pairs are voxels NT * part .. + NT - 1 and
    // the same + TPB)
    __shared__ float su[3][2 * NT];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        su[c][2 * tid] = u[c].x;
        su[c][2 * tid + 1] = u[c].y;
    }
    __syncthreads();
    const unsigned t0 = (unsigned)tile * (TPB * TILE_NPT) + part * NT + tid;
    double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (t0 < nf) acc[c] += (double)su[c][tid];
        if (t0 + TPB < nf) acc[c] += (double)su[c][tid + NT];
    }
    if constexpr (SPLIT) warp_sum3(acc, partial_slot(S, a, tile, part * (NT / 32) + (tid >> 5)));
    else tile_partial(S, tile, a, acc);
}

// Even step with the link slots of a block's voxels in shared memory, found
// once for all directions of the structure (see step3d_even_links_kernel);
// the directions are stepped one after another.
template <class ST, bool W1, bool SPLIT, int NT, int MINB, bool LIST>
__global__ void __launch_bounds__(NT, MINB) step3d_links_slots_kernel(const __grid_constant__ SlotArgs<LIST> ka)
{
    using T = typename ST::T;
    using Cp = typename ST::C;
    static_assert(SPLIT || NT == TPB, "a whole tile takes a full block");
    constexpr int PARTS = SPLIT ? TPB * TILE_NPT / NT : 1, VPT = SPLIT ? 1 : TILE_NPT;
    __shared__ unsigned sl[Q3 - 1][VPT * NT];
    __shared__ float su[MAX_GROUP][3][SPLIT ? NT : 1];      // split: velocities of reduction steps
    const StepArgs &a = ka.a;
    const Solve3 *Sp;
    int tile;
    pdl_launch();
    if (!slots_item<LIST>(ka, Sp, tile, blockIdx.x / PARTS)) { pdl_wait(); return; }
    const Solve3 &S0 = *Sp;
    const int part = blockIdx.x % PARTS;
    const unsigned tid = threadIdx.x;
    const unsigned P = (unsigned)S0.plane, nf = (unsigned)S0.nfluid;
    const unsigned i0 = (unsigned)tile * (TPB * TILE_NPT) + (SPLIT ? split_voxel<NT, 1>(part, tid) : tid);
    const int ng = min(S0.group, MAX_GROUP);
    if constexpr (LIST) {
        bool done = true;
#pragma unroll
        for (int d = 0; d < MAX_GROUP; ++d)
            if (d < ng) done = noted_done(Sp[d]) && done;
        if (done) { pdl_wait(); return; }
    }
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
        const unsigned i = i0 + j * TPB;
        if (i >= nf) continue;
        unsigned q[Q3 - 1];
        link_slots(S0, i, P, __ldg(S0.meta + i), __ldg(S0.meta2 + i), q);
#pragma unroll
        for (int k = 0; k < Q3 - 1; ++k) sl[k][j * NT + tid] = q[k];
    }
    pdl_wait();
    unsigned redm = 0;                 // split: directions that reduce
#pragma unroll 1
    for (int d = 0; d < ng; ++d) {
        const Solve3 &S = Sp[d];
        const int n4 = step_n4(S, a);  // the direction's own: a finished leader's step count stands still
        const T *R = slots_src<T>(S, n4);
        T *W = slots_dst<T>(S, n4);
        const StepHead h = step_head(S, a);
        double acc[3] = {0.0, 0.0, 0.0};
        if (!h.run) continue;
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
            const unsigned i = i0 + j * TPB;
            if (i >= nf) continue;
            Cp g[Q3];
            g[0] = ST::ld(R + i);
#pragma unroll
            for (int k = 1; k < Q3; ++k) g[k] = ST::ld(R + sl[k - 1][j * NT + tid]);
            Cp ux, uy, uz;
            collide3<ST, W1>(g, S, ux, uy, uz);
            const uint32_t hv = voxel_bits<ST>(i, h.n);
            store_pop<ST>(W, i, g[0], hv, 0);
#pragma unroll
            for (int k = 1; k < Q3; k += 2)
                store_pops<ST>(W, sl[opp3(k) - 1][j * NT + tid], g[k], sl[opp3(k + 1) - 1][j * NT + tid], g[k + 1], hv, k);
            if constexpr (SPLIT) {
                if (h.red) { su[d][0][tid] = ux; su[d][1][tid] = uy; su[d][2][tid] = uz; }
            } else {
                if (h.red) { acc[0] += (double)ux; acc[1] += (double)uy; acc[2] += (double)uz; }
            }
        }
        if (!h.red) continue;
        if constexpr (SPLIT) {
            redm |= 1u << d;
        } else {
            tile_partial(S, tile, a, acc);
            __syncthreads();           // its scratch is the next direction's
        }
    }
    if constexpr (SPLIT) {
        // the warps share out the (direction, virtual warp) sums: one barrier for all
        if (!redm) return;
        __syncthreads();
        constexpr unsigned HT = NT / 2, VW = HT / 32;
        const unsigned t0 = (unsigned)tile * (TPB * TILE_NPT) + part * HT;
#pragma unroll 1
        for (unsigned w = tid >> 5; w < MAX_GROUP * VW; w += NT / 32) {
            const unsigned d = w / VW, vw = w % VW, t = vw * 32 + (tid & 31);
            if (!((redm >> d) & 1u)) continue;
            double v[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (t0 + t < nf) v[c] += (double)su[d][c][t];
                if (t0 + t + TPB < nf) v[c] += (double)su[d][c][HT + t];
            }
            warp_sum3(v, partial_slot(Sp[d], a, tile, part * VW + vw));
        }
    }
}

// Step of a single solve: ndir directions (a.s), with split or whole tiles.
cudaError_t launch_slots3d_f64(bool w1, bool odd, bool split, int ntiles, int ndir, cudaStream_t s, const SlotArgs<false> &a);
cudaError_t launch_slots3d_lp(int prec, bool pull, bool w1, bool odd, bool split, int ntiles, int ndir, cudaStream_t s,
                              const SlotArgs<false> &a);
// Step of a batch: the items of its work list.
cudaError_t launch_slots3d_list(int prec, bool pull, bool w1, bool odd, dim3 grid, cudaStream_t s, const StepArgs &a);
cudaError_t launch_slots3d_list_f64(bool w1, bool odd, dim3 grid, cudaStream_t s, const SlotArgs<true> &a);

}  // namespace lbm
