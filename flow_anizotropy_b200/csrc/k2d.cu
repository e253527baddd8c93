// D2Q9 kernels.  Compiled with -fmad=false: every float operation of the
// collision rounds as in the reference build (plain -O3, no FMA), so a step
// is bit-identical to LMB2d/lbm.cpp:563-632.
#include "engine2d.cuh"

namespace lbm {

// AA slots of a cell's links (k = 1..8): population k is read from, and
// population inv k written to, its own slot [k] across a solid link, else the
// neighbour's slot [inv k] at x - e_k.
__device__ __forceinline__ void slots2(const Solve2 &S, int nd, int x, int y, uint32_t sol, unsigned (&sl)[Q2])
{
    const int nx = S.nx, ny = S.ny;
    const int dx[3] = {x == 0 ? nx - 1 : -1, 0, x == nx - 1 ? 1 - nx : 1};
    const int dy[3] = {y == 0 ? (ny - 1) * nx : -nx, 0, y == ny - 1 ? -(ny - 1) * nx : nx};
    sl[0] = (unsigned)nd;
#pragma unroll
    for (int k = 1; k < Q2; ++k) {
        const int o = inv2(k);
        sl[k] = ((sol >> o) & 1u) ? k * S.plane + (unsigned)nd : o * S.plane + (unsigned)(nd + dx[ex2(o) + 1] + dy[ey2(o) + 1]);
    }
}

// One step (odd: local, even: neighbour) of one tile of one solve.  A thread
// steps an adjacent cell pair in packed FP32; all that does not change during
// a solve (record, solid bits, slots) is read before the wait for the step
// before, and the step's flags are bits of State2 (a 64-bit division per
// thread and flag took a fifth of the step).  Bound by latency on one image
// (512 blocks), by instructions on many.  Per step: one 256^2 image, both
// directions, 5.3 -> 3.0 us; 16 images 58 (47 while averaging) -> 25 us.
// (7 blocks of 72 registers per SM: with 8 of 64 the slots spill, 4.3 and 29.7 us.)
template <bool ODD>
__global__ void __launch_bounds__(THREADS2, 7) step2d_kernel(const StepArgs2 a)
{
    __shared__ double sh[TPB / 32][2];
    __shared__ float su[2][TPB];
    pdl_launch();
    const Solve2 &S = a.solves[blockIdx.y];
    const int tile = blockIdx.x, tid = threadIdx.x;
    const int nd = tile * TPB + 2 * tid, nn = S.nn;
    const unsigned P = S.plane;
    float *A = S.A;
    // solid bits of both cells (nd is even; the table is padded)
    const uint32_t both = nd < nn ? *reinterpret_cast<const uint32_t *>(S.nbm + nd) : 0x00010001u;
    const uint32_t s0 = both & 0xffffu, s1 = nd + 1 < nn ? both >> 16 : 1u;
    const bool l0 = !(s0 & 1u), l1 = !(s1 & 1u);
    unsigned sa[Q2], sb[Q2];
    if constexpr (!ODD) {
        const int y = S.dvx.div(nd), x = nd - y * S.nx;
        const bool wrap = x + 1 == S.nx;
        if (l0) slots2(S, nd, x, y, s0, sa);
        if (l1) slots2(S, nd + 1, wrap ? 0 : x + 1, wrap ? y + 1 : y, s1, sb);
    }
    pdl_wait();
    const State2 &st = *S.st;
    const int phase = st.phase;
    const long long n = st.s_base + a.step + 1;
    bool red, keep;
    if (a.bit >= 0) {
        red = (st.redm[a.bit >> 6] >> (a.bit & 63)) & 1ull;
        keep = (st.keepm[a.bit >> 6] >> (a.bit & 63)) & 1ull;
    } else {
        red = reduce2(S.c, st, n);
        keep = snap2(S.c, st, n) || last2(S.c, st, n);
    }
    float2 g[Q2], U = make_float2(0.0f, 0.0f), V = U;
    if constexpr (ODD) {
        if (l0 || l1)
#pragma unroll
            for (int k = 0; k < Q2; ++k) g[k] = *reinterpret_cast<const float2 *>(A + (k * P + (unsigned)nd));
    } else {
#pragma unroll
        for (int k = 0; k < Q2; ++k) {
            g[k].x = l0 ? A[sa[k]] : w2(k);
            g[k].y = l1 ? A[sb[k]] : w2(k);
        }
    }
    if (phase >= PH_DONE) return;
    if (l0 || l1) {
        collide2(g, S.fxt, S.fyt, S.itau, U, V);
        if constexpr (ODD) {
            // a solid partner's slots are never read
#pragma unroll
            for (int k = 0; k < Q2; ++k) *reinterpret_cast<float2 *>(A + (inv2(k) * P + (unsigned)nd)) = g[k];
        } else {
#pragma unroll
            for (int k = 0; k < Q2; ++k) {
                if (l0) A[sa[inv2(k)]] = g[k].x;
                if (l1) A[sb[inv2(k)]] = g[k].y;
            }
        }
    }
    if (!(red || keep)) return;
    if (!l0) U.x = V.x = 0.0f;
    if (!l1) U.y = V.y = 0.0f;
    if (keep) {
        const bool snap = snap2(S.c, st, n), last = last2(S.c, st, n);
        if (nd < nn) {
            if (snap) { S.snap[2 * nd] = U.x; S.snap[2 * nd + 1] = V.x; }
            if (last) { S.last[2 * nd] = U.x; S.last[2 * nd + 1] = V.x; }
        }
        if (nd + 1 < nn) {
            if (snap) { S.snap[2 * nd + 2] = U.y; S.snap[2 * nd + 3] = V.y; }
            if (last) { S.last[2 * nd + 2] = U.y; S.last[2 * nd + 3] = V.y; }
        }
    }
    if (!red) return;
    su[0][2 * tid] = U.x; su[0][2 * tid + 1] = U.y;
    su[1][2 * tid] = V.x; su[1][2 * tid + 1] = V.y;
    __syncthreads();
    double acc[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int c = 0; c < 2; ++c) acc[h][c] = (double)su[c][h * THREADS2 + tid];
    finish_tile2(S, tile, n, acc, sh);
}

__global__ void nbmask2d_kernel(const uint32_t *mask, int nx, int ny, int wpr, uint16_t *nbm)
{
    const int nn = nx * ny;
    for (int nd = blockIdx.x * blockDim.x + threadIdx.x; nd < nn; nd += gridDim.x * blockDim.x) {
        const int y = nd / nx, x = nd - y * nx;
        const int X[3] = {x == 0 ? nx - 1 : x - 1, x, x == nx - 1 ? 0 : x + 1};
        const int Yr[3] = {y == 0 ? ny - 1 : y - 1, y, y == ny - 1 ? 0 : y + 1};
        uint32_t sol = 0;
#pragma unroll
        for (int k = 0; k < Q2; ++k) {
            const int yy = Yr[ey2(k) + 1], xx = X[ex2(k) + 1];
            sol |= (uint32_t)mbit(mask + (size_t)yy * wpr, xx) << k;
        }
        nbm[nd] = (uint16_t)sol;
    }
}

cudaError_t launch_nbmask2d(const uint32_t *mask, int nx, int ny, uint16_t *nbm, cudaStream_t s)
{
    const int nn = nx * ny;
    nbmask2d_kernel<<<(nn + 255) / 256 < 1184 ? (nn + 255) / 256 : 1184, 256, 0, s>>>(mask, nx, ny, (nx + 31) / 32, nbm);
    return cudaGetLastError();
}

__global__ void init2d_kernel(float *A, unsigned plane, int nn)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x)
#pragma unroll
        for (int k = 0; k < Q2; ++k) A[k * plane + (unsigned)i] = w2(k);
}

// Populations the next step will read, in the reference's pre-collision
// (post-transport) form: after a local step A[opp k][x] holds f*_k(x), which
// streams to x + e_k; after a neighbour step A[k][x] already holds them.
__global__ void canon2d_kernel(const Solve2 S, long long done, float *f_out)
{
    for (int nd = blockIdx.x * blockDim.x + threadIdx.x; nd < S.nn; nd += gridDim.x * blockDim.x) {
        const int y = S.dvx.div(nd);
        const int x = nd - y * S.nx;
        if (mbit(S.mask + (size_t)y * S.wpr, x)) {
            for (int k = 0; k < Q2; ++k) f_out[nd * Q2 + k] = 0.0f;
            continue;
        }
        for (int k = 0; k < Q2; ++k) {
            float v;
            if (!(done & 1ll)) {
                v = S.A[k * S.plane + (unsigned)nd];
            } else {
                // pre-collision f_k(x) = f*_k(x - e_k), or f*_inv(k)(x) if x - e_k is solid
                const int sx = (x - ex2(k) + S.nx) % S.nx, sy = (y - ey2(k) + S.ny) % S.ny;
                const int o = inv2(k);
                if (mbit(S.mask + (size_t)sy * S.wpr, sx)) v = S.A[k * S.plane + (unsigned)nd];
                else v = S.A[o * S.plane + (unsigned)(sy * S.nx + sx)];
            }
            f_out[nd * Q2 + k] = v;
        }
    }
}

// field_residual (LMB2d/lbm.cpp:217-229): out[0] = sum (du^2 + dv^2), out[1] = sum (u^2 + v^2)
__global__ void fieldres2d_kernel(const float *snap, const float *last, int nn, double *out)
{
    __shared__ double sh[TPB / 32][3];
    double v[2] = {0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
        const float u = last[2 * i], w = last[2 * i + 1];
        const double du = u - snap[2 * i];
        const double dv = w - snap[2 * i + 1];
        v[0] += du * du + dv * dv;
        v[1] += (double)u * u + (double)w * w;
    }
    block_sum2(v, sh);
    if (threadIdx.x == 0) { atomicAdd(out, v[0]); atomicAdd(out + 1, v[1]); }
}

// s_base += steps for every solve (the step numbers of a replayed chunk of
// step launches are relative to s_base), and the flags of the next MASK2
// steps, one thread per step.
__global__ void __launch_bounds__(MASK2) advance2d_kernel(const Solve2 *solves, long long steps)
{
    const Solve2 &S = solves[blockIdx.x];
    pdl_launch();
    pdl_wait();
    State2 &st = *S.st;
    const long long base = st.s_base + steps, n = base + 1 + threadIdx.x;
    const bool run = st.phase < PH_DONE;
    const unsigned red = __ballot_sync(0xffffffffu, run && reduce2(S.c, st, n));
    const unsigned keep = __ballot_sync(0xffffffffu, run && (snap2(S.c, st, n) || last2(S.c, st, n)));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        reinterpret_cast<unsigned *>(st.redm)[threadIdx.x >> 5] = red;
        reinterpret_cast<unsigned *>(st.keepm)[threadIdx.x >> 5] = keep;
    }
    if (threadIdx.x == 0) st.s_base = base;
}

cudaError_t launch_advance2d(const Solve2 *solves, int nsolves, long long steps, cudaStream_t s)
{
    return launch_pdl(advance2d_kernel, dim3(nsolves), MASK2, 0, s, solves, steps);
}

cudaError_t launch_step2d(bool odd, int ntiles, int nsolves, cudaStream_t s, const StepArgs2 &a)
{
    if (nsolves > 65535) {
        // beyond one grid's second dimension: a launch per 65535 solves
        for (int j = 0; j < nsolves; j += 65535) {
            StepArgs2 x = a;
            x.solves += j;
            const cudaError_t e = launch_step2d(odd, ntiles, nsolves - j < 65535 ? nsolves - j : 65535, s, x);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    const dim3 grid(ntiles, nsolves);
    return odd ? launch_pdl(step2d_kernel<true>, grid, THREADS2, 0, s, a) : launch_pdl(step2d_kernel<false>, grid, THREADS2, 0, s, a);
}

}  // namespace lbm
