// FP64 D3Q19 kernels.  This translation unit is compiled with -fmad=false:
// the collision keeps the reference's rounding step by step
// (LMB3d/lbm3d-perm.cpp:218-245), so one step matches the CPU oracle bit for bit.
#include "step3d_slots.cuh"

namespace lbm {

#define LBM_ODD(V) step3d_odd_kernel<StoreF64, odd_f64(V).npt, odd_f64(V).minb, W1>
#define LBM_EVEN(V) step3d_even_kernel<StoreF64, even_f64(V).minb, W1, even_meta(V)>

template <bool W1>
static void launch_f64(int vo, int ve, bool odd, dim3 grid, cudaStream_t s, const StepArgs &a)
{
    if (odd) {
        switch (vo) {
        case 0: LBM_ODD(0)<<<grid, TPB, 0, s>>>(a); break;
        case 1: LBM_ODD(1)<<<grid, TPB, 0, s>>>(a); break;
        default: LBM_ODD(2)<<<grid, TPB, 0, s>>>(a); break;
        }
    } else {
        switch (ve) {
        case 0: LBM_EVEN(0)<<<grid, TPB, 0, s>>>(a); break;
        case 1: LBM_EVEN(1)<<<grid, TPB, 0, s>>>(a); break;
        case 2: LBM_EVEN(2)<<<grid, TPB, 0, s>>>(a); break;
        case 3: LBM_EVEN(3)<<<grid, TPB, 0, s>>>(a); break;
        // FP64 staging would exceed the static shared-memory limit: variants
        // 4-5 run the register-staged kernel with the same record reads
        case 4: LBM_EVEN(0)<<<grid, TPB, 0, s>>>(a); break;
        default: LBM_EVEN(1)<<<grid, TPB, 0, s>>>(a); break;
        }
    }
}

cudaError_t launch_step3d_f64(int variant, bool w1, bool odd, dim3 grid, cudaStream_t s, const StepArgs &a)
{
    if (variant < 0 || variant >= 2 * NVAR_F64) return cudaErrorInvalidValue;
    variant = kernel_variant(0, variant);        // the two-lattice AA form runs the in-place kernels
    const int vo = variant / NVAR_EVEN, ve = variant % NVAR_EVEN;
    if (w1) launch_f64<true>(vo, ve, odd, grid, s, a);
    else launch_f64<false>(vo, ve, odd, grid, s, a);
    return cudaGetLastError();
}

template <bool W1, bool EVEN>
static cudaError_t launch_slots(bool split, int ntiles, int ndir, cudaStream_t s, const SlotArgs<false> &a)
{
    return split ? launch_pdl(step3d_aa_kernel<StoreF64, W1, EVEN, true, 128, 4, false>, dim3(4 * ntiles, ndir), 128, 0, s, a)
                 : launch_pdl(step3d_aa_kernel<StoreF64, W1, EVEN, false, 256, 2, false>, dim3(ntiles, ndir), 256, 0, s, a);
}

cudaError_t launch_slots3d_f64(bool w1, bool odd, bool split, int ntiles, int ndir, cudaStream_t s, const SlotArgs<false> &a)
{
    return w1 ? (odd ? launch_slots<true, false>(split, ntiles, ndir, s, a) : launch_slots<true, true>(split, ntiles, ndir, s, a))
              : (odd ? launch_slots<false, false>(split, ntiles, ndir, s, a) : launch_slots<false, true>(split, ntiles, ndir, s, a));
}

cudaError_t launch_slots3d_list_f64(bool w1, bool odd, dim3 grid, cudaStream_t s, const SlotArgs<true> &a)
{
    return w1 ? (odd ? launch_pdl(step3d_aa_kernel<StoreF64, true, false, false, 256, 2, true>, grid, 256, 0, s, a)
                     : launch_pdl(step3d_aa_kernel<StoreF64, true, true, false, 256, 2, true>, grid, 256, 0, s, a))
              : (odd ? launch_pdl(step3d_aa_kernel<StoreF64, false, false, false, 256, 2, true>, grid, 256, 0, s, a)
                     : launch_pdl(step3d_aa_kernel<StoreF64, false, true, false, 256, 2, true>, grid, 256, 0, s, a));
}

cudaError_t launch_init3d_f64(void *A, long long plane, long long n, cudaStream_t s)
{
    init3d_kernel<StoreF64><<<1184, 256, 0, s>>>(A, plane, n);
    return cudaGetLastError();
}

cudaError_t launch_canon3d_f64(const Solve3 &S, long long done, double *f, float *u, cudaStream_t s)
{
    canon3d_kernel<StoreF64><<<1184, 256, 0, s>>>(S, done, f, u);
    return cudaGetLastError();
}

}  // namespace lbm
