// Deferred flux reduction of the 3D step kernels (StepArgs::defer): after a
// run of at most DEFER_SLOTS launches, one block per (solve, launch) sums the
// tile partials a reduction step left in its slot, in the order the last
// tile of an immediate reduction uses (thread t takes tiles t, t + TPB, ...,
// then the fixed-order block sum), and one block per solve runs the
// controller over the steps in order.  So a deferred solve takes the same
// decisions and reports the same bits as one reduced at every step; only the
// work moves out of the step kernels (LMB3d/lbm3d-perm.cpp:298-303 is the
// reduction, :320-398 the controller).
#include "engine3d.cuh"

namespace lbm {

// The steps of a pass that were reduced are the bits of State3::redm, noted by
// the controller pass before it (or with the initial state).
__global__ void __launch_bounds__(TPB) reduce3d_kernel(const Solve3 *solves, long long step0, double *qbuf)
{
    __shared__ double sh[TPB / 32][3];
    const int j = blockIdx.x, r = blockIdx.y;
    const Solve3 &S = solves[j];
    double *out = qbuf + 4ll * ((long long)j * DEFER_SLOTS + r);
    pdl_launch();
    pdl_wait();
    if (S.st->phase >= PH_DONE || !((S.st->redm >> r) & 1ull)) {
        if (threadIdx.x == 0) out[3] = 0.0;
        return;
    }
    const int per = S.split ? TPB / 32 : 1;      // a split tile left its 8 warps' sums: add them as a block would
    const double *p = S.partials + 3ll * (long long)((step0 + r) & (DEFER_SLOTS - 1)) * S.ntiles * per;
    double v[3] = {0.0, 0.0, 0.0};
    for (int t = threadIdx.x; t < S.ntiles; t += TPB) {
        double x[3];
        if (S.split) {
            const double *w = p + 3ll * per * t;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                x[c] = 0.0;
#pragma unroll
                for (int q = 0; q < TPB / 32; ++q) x[c] += w[3 * q + c];
            }
        } else {
            x[0] = p[3ll * t]; x[1] = p[3ll * t + 1]; x[2] = p[3ll * t + 2];
        }
        v[0] += x[0];
        v[1] += x[1];
        v[2] += x[2];
    }
    block_sum3<TPB>(v, sh);
    if (threadIdx.x == 0) {
        const double inv = (double)S.nn;
        out[0] = v[0] / inv;
        out[1] = v[1] / inv;
        out[2] = v[2] / inv;
        out[3] = 1.0;
    }
}

// One block per solve: the pass's fluxes come to shared memory together,
// then one thread runs the controller over the steps in order on a shared
// copy of the state (the controller acts on a step when the phase it has
// reached by then needs that step: which steps phase 1 needs is found by all
// threads at once, the 64-bit divisions of one thread for 64 steps took most
// of the pass).  The pass ends by noting, one thread per step, which of the
// next DEFER_SLOTS steps reduce (State3::redm), so that the step kernels test
// one bit, and with advance != 0 moves s_base on.
static_assert(DEFER_SLOTS == 64, "two warps, one bit of a 64-bit mask per thread");
__device__ __forceinline__ unsigned long long ballot64(unsigned (&bits)[2], bool x)
{
    const unsigned m = __ballot_sync(0xffffffffu, x);
    if ((threadIdx.x & 31) == 0) bits[threadIdx.x >> 5] = m;
    __syncthreads();
    const unsigned long long r = (unsigned long long)bits[1] << 32 | bits[0];
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(DEFER_SLOTS) control3d_kernel(Solve3 *solves, long long step0, int nsteps,
                                                                  const double *qbuf, int mode, long long advance)
{
    __shared__ double q[DEFER_SLOTS][4];
    __shared__ State3 st;
    __shared__ unsigned bits[2];
    const int j = blockIdx.x;
    Solve3 &S = solves[j];
    pdl_launch();
    pdl_wait();
    for (int r = threadIdx.x; r < nsteps; r += blockDim.x)
        for (int c = 0; c < 4; ++c) q[r][c] = qbuf[4ll * ((long long)j * DEFER_SLOTS + r) + c];
    if (threadIdx.x == 0) st = *S.st;
    __syncthreads();
    // for the step kernels' blocks, which may be reading it (noted_done); here
    // too, since a batch's records are written anew when its work list changes
    auto note_done = [&] { *static_cast<volatile int *>(&S.done) = 1; };
    if (st.phase >= PH_DONE) {
        if (threadIdx.x == 0) note_done();
        return;
    }
    const long long first = st.s_base + step0 + 1;
    const unsigned long long run = ballot64(bits, (int)threadIdx.x < nsteps && needs_reduction(S.c, PH_RUN, first + threadIdx.x));
    if (threadIdx.x == 0)
        for (int r = 0; r < nsteps && st.phase < PH_DONE; ++r) {
            if (st.phase == PH_RUN) {
                const unsigned long long rest = run >> r;
                if (!rest) break;
                r += __ffsll((long long)rest) - 1;
            }
            const long long n = first + r;
            if (q[r][3] == 0.0) {            // a needed step without partials: cannot happen by construction
                st.status = STATUS_WAIT_TIMEOUT;
                st.phase = PH_ERR;
                st.steps = n;
                break;
            }
            controller3(S.c, st, n, q[r]);
        }
    __syncthreads();
    const long long done = first + nsteps - 1;
    const unsigned long long next = ballot64(bits, deferred_reduces(S.c, st.phase, done + threadIdx.x + 1, done, mode));
    if (threadIdx.x != 0) return;
    st.redm = next;
    if (st.phase < PH_DONE) st.s_base += advance;
    else note_done();
    *S.st = st;
}

cudaError_t launch_deferred3d(Solve3 *solves, int nsolves, long long step0, int nsteps, double *qbuf,
                              int mode, long long advance, cudaStream_t s)
{
    if (nsolves <= 0 || nsteps <= 0) return cudaSuccess;
    if (nsteps > DEFER_SLOTS) return cudaErrorInvalidValue;
    const cudaError_t e = launch_pdl(reduce3d_kernel, dim3(nsolves, nsteps), TPB, 0, s, solves, step0, qbuf);
    if (e != cudaSuccess) return e;
    return launch_pdl(control3d_kernel, dim3(nsolves), DEFER_SLOTS, 0, s, solves, step0, nsteps, (const double *)qbuf, mode, advance);
}

}  // namespace lbm
