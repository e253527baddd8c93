// liblbm host engine: contexts, structure upload and bit packing, the plain
// solve loops (one launch per step, on-device convergence controller, one
// host synchronisation per convergence check), velocity export and the
// diagnostic entry points.  The C ABI is declared in include/lbm.h.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/lbm.h"
#include "engine2d.cuh"
#include "engine_host.h"
#include "engine_m.cuh"
#include "engine_md.cuh"
#include "step3d_slots.cuh"

using namespace lbm;

// ------------------------------------------------------------- utilities ----
int lbm_fail_cuda(lbm_ctx *ctx, cudaError_t e, const char *what, int line)
{
    if (ctx)
        ctx->err = std::string("CUDA error: ") + cudaGetErrorString(e) + " in " + what +
                   " (engine line " + std::to_string(line) + ")";
    return LBM_ECUDA;
}

int lbm_fail_input(lbm_ctx *ctx, const std::string &msg)
{
    if (ctx) ctx->err = msg;
    return LBM_EINPUT;
}

bool lbm_is_device_ptr(const void *p)
{
    if (!p) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// Pack a byte mask (x fastest, 1 = solid) into rows of 32-bit words, count
// the pore voxels and flag any value other than 0/1 (LMB3d/lbm3d-perm.cpp:190-192).
__global__ void pack_mask_kernel(const uint8_t *__restrict__ solid, int nx, long long rows, int wpr,
                                 uint32_t *__restrict__ mask, unsigned long long *npore, unsigned *bad)
{
    // one count per block: a global atomic per word took 1.7 ms of a 512^3 mask
    __shared__ unsigned long long s_cnt;
    __shared__ unsigned s_bad;
    if (threadIdx.x == 0) { s_cnt = 0ull; s_bad = 0u; }
    __syncthreads();
    const long long total = rows * wpr;
    unsigned long long all = 0ull;
    unsigned b = 0;
    for (long long w = blockIdx.x * (long long)blockDim.x + threadIdx.x; w < total;
         w += (long long)gridDim.x * blockDim.x) {
        const long long r = w / wpr;
        const int c = (int)(w - r * wpr);
        const int x0 = c * 32;
        const uint8_t *row = solid + r * nx;
        uint32_t bits = 0;
        unsigned cnt = 0;
        for (int i = 0; i < 32; ++i) {
            if (x0 + i >= nx) { bits |= 1u << i; continue; }   // past the row end: solid
            const uint8_t v = row[x0 + i];
            b |= v > 1;
            if (v) bits |= 1u << i; else ++cnt;
        }
        mask[w] = bits;
        all += cnt;
    }
    if (all) atomicAdd(&s_cnt, all);
    if (b) atomicOr(&s_bad, 1u);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_cnt) atomicAdd(npore, s_cnt);
        if (s_bad) atomicOr(bad, 1u);
    }
}

int lbm_upload_mask(lbm_ctx *ctx, const uint8_t *solid, int nx, long long rows, DevMem &mask,
                    long long &npore)
{
    const long long nn = (long long)nx * rows;
    const int wpr = (nx + 31) / 32;
    DevMem staging(ctx->stream), scratch(ctx->stream);
    const uint8_t *src = solid;
    if (!lbm_is_device_ptr(solid)) {
        CK(staging.alloc((size_t)nn));
        CK(cudaMemcpyAsync(staging.p, solid, (size_t)nn, cudaMemcpyHostToDevice, ctx->stream));
        src = static_cast<const uint8_t *>(staging.p);
    }
    CK(mask.alloc(sizeof(uint32_t) * (size_t)rows * wpr));
    CK(scratch.alloc(16));
    CK(cudaMemsetAsync(scratch.p, 0, 16, ctx->stream));
    auto *cnt = static_cast<unsigned long long *>(scratch.p);
    auto *bad = reinterpret_cast<unsigned *>(cnt + 1);
    const long long words = rows * wpr;
    const int blocks = (int)std::min<long long>((words + 255) / 256, 4L * 1184);
    pack_mask_kernel<<<blocks, 256, 0, ctx->stream>>>(src, nx, rows, wpr, static_cast<uint32_t *>(mask.p), cnt, bad);
    CK(cudaGetLastError());
    unsigned long long h[2] = {0, 0};
    CK(cudaMemcpyAsync(h, scratch.p, 16, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if ((unsigned)h[1]) return lbm_fail_input(ctx, "non-binary voxel");
    npore = (long long)h[0];
    if (npore == 0) return lbm_fail_input(ctx, "structure has no pore space");
    return LBM_OK;
}

// ------------------------------------------------------------- context ------
extern "C" int lbm_version(void) { return LBM_API_VERSION; }

extern "C" int lbm_create(lbm_ctx **out, int device)
{
    if (!out) return LBM_EINPUT;
    *out = nullptr;
    lbm_ctx *ctx = new lbm_ctx();
    ctx->device = device;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&ctx->sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = prepare_step3d_lp(device);
    if (e == cudaSuccess) {
        // keep up to 4 GiB of freed lattices in the device's stream-ordered
        // pool between solves instead of returning them to the driver at
        // every synchronisation (repeated solves then reuse mapped memory)
        cudaMemPool_t pool = nullptr;
        e = cudaDeviceGetDefaultMemPool(&pool, device);
        unsigned long long keep = 4ull << 30;
        if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    if (e != cudaSuccess) {
        lbm_last_error_global() = std::string("CUDA error: ") + cudaGetErrorString(e);
        delete ctx;
        return LBM_ECUDA;
    }
    *out = ctx;
    return LBM_OK;
}

extern "C" void lbm_destroy(lbm_ctx *ctx)
{
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    cudaStreamDestroy(ctx->stream);
    delete ctx;
}

std::string &lbm_last_error_global()
{
    static std::string s;
    return s;
}

extern "C" void *lbm_stream(const lbm_ctx *ctx) { return ctx ? (void *)ctx->stream : nullptr; }

extern "C" const char *lbm_last_error(const lbm_ctx *ctx)
{
    return ctx ? ctx->err.c_str() : lbm_last_error_global().c_str();
}

// --------------------------------------------------------------- 3D ---------
int lbm_check_params3d(lbm_ctx *ctx, const lbm_params3d &p)
{
    if (!(p.tau > 0.5)) return lbm_fail_input(ctx, "tau must exceed 0.5");
    if (p.lag <= 0) return lbm_fail_input(ctx, "--lag must be positive");
    if (p.precision < LBM_FP64 || p.precision > LBM_MD32) return lbm_fail_input(ctx, "unknown precision");
    if ((is_moment(p.precision) || is_dense_m(p.precision)) && p.tau != 1.0)
        return lbm_fail_input(ctx, "moment-projected storage needs tau = 1");
    if (p.criterion != LBM_CRIT_DRIFT && p.criterion != LBM_CRIT_BLOCK && p.criterion != LBM_CRIT_BATCH)
        return lbm_fail_input(ctx, "unknown criterion");
    if (p.criterion != LBM_CRIT_DRIFT && (p.sample <= 0 || p.lag % p.sample != 0))
        return lbm_fail_input(ctx, "block criterion needs sample > 0 dividing lag");
    if (p.variant != LBM_VARIANT_DEFAULT && (p.variant < 0 || p.variant >= variant_count(p.precision)))
        return lbm_fail_input(ctx, "unknown step-kernel variant");
    return LBM_OK;
}

// The autotuner's pick on the 128^3 tensor workload: FP32 the pull form
// (voxel pairs, ranks from the neighbour record, 3 blocks per SM); 16-bit
// the two-lattice AA form of the bulk-staged odd step + the grouped even
// step with the link slots shared by the directions (4 blocks per SM).
int lbm_default_variant(int prec)
{
    if (prec == LBM_FP32) return NVAR_LP + 1;
    if (prec == LBM_FP16 || prec == LBM_BF16) return AA2_BASE_LP + 4 * NVAR_EVEN_LP + 9;
    return 0;
}

// The batch's default: the solve default (its 16-bit pick has a grouped even
// step, which the batch runs over runs of a structure's consecutive slots).
int lbm_default_batch_variant(int prec)
{
    return lbm_default_variant(prec);
}

static lbm_params3d lbm_resolve_variant(lbm_params3d p)
{
    if (p.variant == LBM_VARIANT_DEFAULT) p.variant = lbm_default_variant(p.precision);
    return p;
}

// Pore voxels x directions up to which a single 16-bit solve takes the pull form.
constexpr long long SMALL_16BIT = 500000;

static size_t elem_size(int prec) { return prec == LBM_FP64 ? 8 : (prec == LBM_FP32 ? 4 : 2); }

long long lbm_plane_elems(long long nn) { return (nn + 63) / 64 * 64; }

// Lattice bytes of one direction over n pore voxels.
long long lbm_lattice_bytes3d(long long n, int prec)
{
    if (is_moment(prec)) return 2ll * mom_buffer_bytes(prec, n);
    return (long long)Q3 * lbm_plane_elems(n) * (long long)elem_size(prec);
}

// Lattice bytes of one direction of a filled solve record (both lattices of
// the pull and two-lattice AA forms).
long long lbm_lattice_bytes(const Solve3 &S)
{
    if (is_dense_m(S.prec)) return md_lattice_bytes(S.md);
    return lbm_lattice_bytes3d(S.nfluid, S.prec) * ((S.pull || S.aa2) ? 2 : 1);
}

// Point a solve record at its lattice memory (lbm_lattice_bytes(S) bytes);
// the second lattice of the two-lattice forms follows the first.
void lbm_attach_lattice(Solve3 &S, void *p)
{
    S.A = p;
    S.B = (S.pull || S.aa2) ? static_cast<char *>(p) + lbm_lattice_bytes3d(S.nfluid, S.prec) : nullptr;
}

// Plane stride (populations) or record slots per buffer (moments).
long long lbm_plane_for(int prec, long long n)
{
    return is_moment(prec) ? mom_slots(n) : lbm_plane_elems(n);
}

// A variant whose even kernel reads neighbour records needs them built.
int lbm_effective_variant(int prec, int variant, bool have_meta)
{
    if (is_moment(prec) || is_dense_m(prec) || have_meta) return variant;
    if (is_aa2_variant(prec, variant))
        return aa2_base(prec) + lbm_effective_variant(prec, kernel_variant(prec, variant), false);
    if (is_pull_variant(prec, variant))
        return pull_meta(variant - NVAR_LP) ? NVAR_LP + 2 : variant;   // pull, ranks from the mask
    const int ve = variant % nvar_even(prec);
    if (!even_meta(ve)) return variant;
    if (even_wide(ve)) return variant - ve + 14;        // link slots, one voxel per thread, ranks from the mask
    if (even_links(ve)) return variant - ve + 10;       // grouped link slots (one voxel at a time), ranks from the mask
    if (even_grouped(ve)) return variant - ve + 6;      // grouped, ranks from the mask
    return variant - ve + (ve & 1) + 2;                 // same budget, ranks from the mask
}

// Does this (effective) variant run the grouped even kernel?
bool lbm_grouped_variant(int prec, int variant)
{
    if (is_pull_variant(prec, variant)) return pull_grouped(variant - NVAR_LP);
    variant = kernel_variant(prec, variant);
    return prec >= LBM_FP32 && prec <= LBM_BF16 && even_grouped(variant % NVAR_EVEN_LP);
}

// Do all launches (not only the even ones) of this variant take the grouped work list?
bool lbm_grouped_all(int prec, int variant)
{
    return is_pull_variant(prec, variant) && pull_grouped(variant - NVAR_LP);
}

// Work list of the grouped even step over solves that share one structure:
// runs of up to MAX_GROUP consecutive records, led by the first of each run.
static void lbm_group_items(std::vector<Solve3> &hs, std::vector<int2> &items)
{
    const int n = (int)hs.size();
    for (auto &S : hs) S.group = 0;
    for (int j = 0; j < n; j += MAX_GROUP) {
        hs[j].group = std::min(MAX_GROUP, n - j);
        for (int t = 0; t < hs[j].ntiles; ++t) items.push_back(make_int2(j, t));
    }
}

cudaError_t lbm_launch_step(int prec, int variant, bool w1, bool odd, dim3 grid, cudaStream_t s, const StepArgs &a)
{
    if (prec == LBM_FP64) return launch_step3d_f64(variant, w1, odd, grid, s, a);
    if (is_dense_m(prec)) return launch_stepmd(variant, grid, s, a);
    if (is_moment(prec)) return launch_stepm(prec, variant, grid, s, a);
    return launch_step3d_lp(prec, variant, w1, odd, grid, s, a);
}

cudaError_t lbm_init_lattice(int prec, const Solve3 &S, cudaStream_t s)
{
    if (is_dense_m(prec)) return init_md_lattice(S, s);   // tensor maps; step 1 writes the records
    if (is_moment(prec)) return cudaSuccess;        // step 1 writes the moments from scratch
    return launch_init3d(prec, S.A, S.plane, S.nfluid, s);
}

cudaError_t lbm_canon(int prec, const Solve3 &S, long long done, double *f, float *u, cudaStream_t s)
{
    if (is_dense_m(prec)) return launch_canonmd(S, done, f, u, s);
    if (is_moment(prec)) return launch_canonm(prec, S, done, f, u, s);
    return launch_canon3d(prec, S, done, f, u, s);
}

void lbm_fill_solve3(Solve3 &S, int nx, int ny, int nz, const double F[3], const lbm_params3d &p, int npt)
{
    memset(&S, 0, sizeof(S));
    S.prec = p.precision;
    S.pull = is_pull_variant(p.precision, p.variant) ? 1 : 0;
    S.aa2 = is_aa2_variant(p.precision, p.variant) ? 1 : 0;
    S.nx = nx; S.ny = ny; S.nz = nz;
    S.wpr = (nx + 31) / 32;
    S.nn = (long long)nx * ny * nz;
    S.plane = lbm_plane_elems(S.nn);
    S.ntiles = (int)((S.nn + TPB * npt - 1) / (TPB * npt));
    if (is_dense_m(p.precision)) md_fill_geom(S.md, nx, ny, nz, p.variant, S.ntiles);
    S.dvx.init(nx);
    S.dvy.init(ny);
    Phys3 &P = S.P;
    for (int c = 0; c < 3; ++c) { P.F[c] = F[c]; P.Ff[c] = (float)F[c]; }
    P.tau = p.tau;
    P.pref = 1.0 - 0.5 / p.tau;
    P.itau = 1.0 / p.tau;
    P.wp[0] = w3(0) * P.pref; P.wp[1] = w3(1) * P.pref; P.wp[2] = w3(7) * P.pref;
    for (int j = 0; j < 9; ++j) {
        // zero products dropped, as the collision's (x + 0 == x)
        const int k = 2 * j + 1, e[3] = {ex3(k), ey3(k), ez3(k)};
        double eF = 0.0;
        bool first = true;
        for (int c = 0; c < 3; ++c) {
            if (!e[c]) continue;
            const double t = e[c] > 0 ? F[c] : -F[c];
            eF = first ? t : eF + t;
            first = false;
        }
        P.eF[j] = eF;
    }
    P.omega = (float)(1.0 / p.tau);
    P.preff = (float)P.pref;
    // FP16 keeps h * scale; scale puts the largest plausible deviation
    // (Poiseuille peak |F| L^2 / 8 nu over the longest axis) near 2^12, far
    // from both the overflow at 65504 and the subnormal range.
    double scale = 1.0;
    if (p.precision == LBM_FP16) {
        const double nu = (p.tau - 0.5) / 3.0;
        const double L = (double)std::max(nx, std::max(ny, nz));
        const double fmag = std::sqrt(F[0] * F[0] + F[1] * F[1] + F[2] * F[2]);
        const double uest = fmag * L * L / (8.0 * nu);
        scale = uest > 0 ? std::exp2(std::round(std::log2(4096.0 / uest))) : 1.0;
        scale = std::min(std::max(scale, 1.0), std::exp2(40.0));
    }
    S.scale = (float)scale;
    S.inv_scale = (float)(1.0 / scale);
    Ctl3 &c = S.c;
    c.eps = p.eps; c.lag = p.lag; c.min_steps = p.min_steps; c.max_steps = p.max_steps;
    c.avg_steps = p.avg_steps; c.hold = p.hold; c.criterion = p.criterion;
    c.sample = p.sample > 0 ? p.sample : 1; c.ksigma = p.ksigma;
}

void lbm_init_state3(State3 &st, const Ctl3 &c, int mode)
{
    memset(&st, 0, sizeof(st));
    st.phase = PH_RUN;
    if (c.max_steps <= 0) {
        // no run-in steps: converged iff hold <= 0 (LMB3d/lbm3d-perm.cpp:362)
        st.converged = 0 >= c.hold ? 1 : 0;
        if (c.avg_steps <= 0) { st.phase = PH_DONE; st.steps = 0; }
        else { st.phase = PH_AVG; st.avg_start = 0; }
    }
    // reductions of the first pass (the controller pass notes the later ones)
    for (int r = 0; r < DEFER_SLOTS; ++r)
        if (deferred_reduces(c, st.phase, r + 1, 0, mode)) st.redm |= 1ull << r;
}

int lbm_pick_npt(const lbm_params3d &p) { return variant_npt(p.precision, p.variant); }

int lbm_build_pores(lbm_ctx *ctx, Solve3 &S, int npt, DevMem &wpre, DevMem &fnode, DevMem &meta, DevMem &meta2)
{
    const long long nwords = (long long)S.wpr * S.ny * S.nz;
    const int blocks = (int)((nwords + SCAN_WORDS - 1) / SCAN_WORDS);
    DevMem bsum(ctx->stream), boff(ctx->stream);
    CK(bsum.alloc(sizeof(unsigned) * (size_t)blocks));
    CK(boff.alloc(sizeof(unsigned) * (size_t)blocks));
    CK(wpre.alloc(sizeof(uint32_t) * (size_t)(nwords + 1)));
    word_sums_kernel<<<blocks, TPB, 0, ctx->stream>>>(S.mask, nwords, static_cast<unsigned *>(bsum.p));
    CK(cudaGetLastError());
    std::vector<unsigned> h(blocks);
    CK(cudaMemcpyAsync(h.data(), bsum.p, sizeof(unsigned) * blocks, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    unsigned long long total = 0;
    for (int b = 0; b < blocks; ++b) { const unsigned c = h[b]; h[b] = (unsigned)total; total += c; }
    const uint32_t tot32 = (uint32_t)total;
    CK(cudaMemcpyAsync(boff.p, h.data(), sizeof(unsigned) * blocks, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(static_cast<uint32_t *>(wpre.p) + nwords, &tot32, sizeof(uint32_t),
                       cudaMemcpyHostToDevice, ctx->stream));
    word_scan_kernel<<<blocks, TPB, 0, ctx->stream>>>(S.mask, nwords, static_cast<const unsigned *>(boff.p),
                                                      static_cast<uint32_t *>(wpre.p));
    CK(cudaGetLastError());
    CK(fnode.alloc(sizeof(uint32_t) * (size_t)std::max<unsigned long long>(total, 1)));
    const int sb = (int)std::min<long long>((nwords + 255) / 256, 8L * 1184);
    scatter_fnode_kernel<<<sb, 256, 0, ctx->stream>>>(S.mask, static_cast<const uint32_t *>(wpre.p), nwords,
                                                      S.wpr, S.nx, static_cast<uint32_t *>(fnode.p));
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(ctx->stream));   // host staging must outlive the copies
    S.wpre = static_cast<const uint32_t *>(wpre.p);
    S.fnode = static_cast<const uint32_t *>(fnode.p);
    S.nfluid = (int)total;
    if (is_dense_m(S.prec)) {
        // dense moment form: tiles cover the box; the padded byte mask
        // replaces the neighbour records
        S.meta = nullptr;
        S.meta2 = nullptr;
        CK(meta.alloc((size_t)md_pmask_bytes(S.md, S.ny, S.nz)));
        S.md.pmask = static_cast<const uint8_t *>(meta.p);
        CK(launch_padmask(S, ctx->stream));
        return LBM_OK;
    }
    S.plane = lbm_plane_for(S.prec, (long long)total);
    S.ntiles = (int)((total + (unsigned long long)TPB * npt - 1) / ((unsigned long long)TPB * npt));
    if (S.ntiles == 0) S.ntiles = 1;
    S.meta = nullptr;
    S.meta2 = nullptr;
    // neighbour records (24 B per pore voxel) for the even-step kernels that
    // read them; in-row offsets are 16-bit, so rows up to 65535 voxels
    if (S.nx <= 65535 && total > 0) {
        CK(meta.alloc(sizeof(uint4) * (size_t)total));
        CK(meta2.alloc(sizeof(uint2) * (size_t)total));
        const int mb = (int)std::min<unsigned long long>((total + 255) / 256, 8ull * 1184);
        build_meta_kernel<<<mb, 256, 0, ctx->stream>>>(S, static_cast<uint4 *>(meta.p), static_cast<uint2 *>(meta2.p));
        CK(cudaGetLastError());
        S.meta = static_cast<const uint4 *>(meta.p);
        S.meta2 = static_cast<const uint2 *>(meta2.p);
    }
    return LBM_OK;
}

void lbm_copy_pores(Solve3 &dst, const Solve3 &src)
{
    dst.wpre = src.wpre; dst.fnode = src.fnode; dst.nfluid = src.nfluid;
    dst.meta = src.meta; dst.meta2 = src.meta2;
    dst.plane = src.plane; dst.ntiles = src.ntiles;
    dst.md.pmask = src.md.pmask;
}

// Run a set of 3D solves sharing one mask to completion, one launch per step.
// The host synchronises only where the controller can change phase: on lag
// multiples and max_steps in phase 1, at the end of the averaging phase.  In
// between, whole chunks of kGraphSteps3 launches (an even count, starting on
// an even step, plus the s_base advance) are replayed from a CUDA graph, which
// removes the per-launch overhead that dominates small structures; the step
// numbers and kernels are those of single launches.
constexpr int kGraphSteps3 = 64;

// Does a solve of this precision reduce its flux through deferred slots (its
// partials buffer then holds DEFER_SLOTS x ntiles x 3 doubles)?  The dense
// moment form keeps the immediate reduction (its tiles have their own block
// size).
bool lbm_defers(int prec) { return !is_dense_m(prec); }

long long lbm_partial_doubles(int prec, int ntiles, bool split)
{
    return 3ll * ntiles * (lbm_defers(prec) ? DEFER_SLOTS : 1) * (split ? TPB / 32 : 1);
}

// Do solves of this (effective) variant run the kernels of step3d_slots.cuh?
// The default variants do, and their one- and two-lattice counterparts: FP64
// variants 0 and 18, the pull form with ranks from the record, the bulk-staged
// odd + link-slot even pair (69 in place, 150).  The others, and structures
// without neighbour records (whose effective variant computes ranks), run the
// work-list kernels of engine3d.cuh.
bool lbm_slots_variant(int prec, int variant)
{
    if (prec == LBM_FP64) return kernel_variant(prec, variant) == 0;
    if (prec > LBM_BF16) return false;
    return variant == NVAR_LP + 1 || kernel_variant(prec, variant) == 4 * NVAR_EVEN_LP + 9;
}

// Are the tiles of a single solve split over several blocks (Solve3::split)?
// Up to SPLIT_MAX_TILES tiles in all of a call's directions: 100 MB of
// partials at most, and beyond it the last wave of whole tiles is a small
// part of a step.  The pull form's whole tiles pack better (its split tiles
// measured the same at 96^3, 42.5 against 42.6 us per step), so it splits
// only where whole tiles do not fill the SMs' block slots once.
constexpr int SPLIT_MAX_TILES = 8192, SPLIT_MAX_TILES_PULL = 3 * 148;   // 3 blocks per SM
static bool plain_split(int prec, int variant, const Solve3 &S, int ndir)
{
    variant = lbm_effective_variant(prec, variant, S.meta != nullptr);
    return lbm_slots_variant(prec, variant) &&
           (long long)S.ntiles * ndir <= (is_pull_variant(prec, variant) ? SPLIT_MAX_TILES_PULL : SPLIT_MAX_TILES);
}

// Directions of a single solve stepped together (slots variants): as many as
// fit in L2 (126 MB) side by side, each group taking a chunk of steps in turn,
// so that a step finds its lattices there instead of in DRAM.  Against all
// three directions per step (us per step of all, B200): FP64 72^3 at 32 MB a
// direction 36.9 -> 27.7 in pairs, 80^3 (56 MB) 65.3 -> 47.7 one at a time,
// 96^3 (71 MB) 82.2 -> 69.2; FP32 (two lattices) 96^3 (71 MB) 42.1 -> 34.7,
// 112^3 (102 MB) 62.6 -> 57.5.  A direction that does not fit gains nothing
// (FP64 104^3, 98 MB: 113.7 -> 117.4; the pull form still does at 102 MB), and
// where all fit together more of them fill the SMs better (FP64 64^3, 23 MB:
// 20.8 together, 23.4 one at a time).  Two lattices a step apart hold 80 MB as
// well as one does, but not 96 (FP64 72^3 with 100 MB allowed: 36.6).  The
// 16-bit even step shares a voxel's link slots between the directions and is
// not bound by DRAM (51 GLUPS in and out of L2), so it keeps them together.
// An uneven split costs little: four FP64 directions of 64^3 (23 MB each) take
// 30.4 us as 3 + 1, 29.7 as 2 + 2, 33.4 all together and 34.7 one at a time;
// of 56^3 (19 MB) 25.4 all together, 25.2 as 3 + 1, 25.0 as 2 + 2.
constexpr long long L2_GROUP_BYTES = 80ll << 20, L2_ONE_BYTES = 88ll << 20, L2_ONE_BYTES_PULL = 112ll << 20;
static int plain_group(int prec, int variant, const Solve3 &S, int ndir)
{
    if (!lbm_slots_variant(prec, variant) || lbm_grouped_variant(prec, variant)) return ndir;
    const long long one = lbm_lattice_bytes(S);
    if (one > (S.pull ? L2_ONE_BYTES_PULL : L2_ONE_BYTES)) return ndir;
    return (int)std::max(1ll, std::min<long long>(ndir, L2_GROUP_BYTES / one));
}

// One step of solves j0 .. j0 + nj - 1 of hs by the kernels of step3d_slots.cuh.
static cudaError_t launch_plain_slots(const std::vector<Solve3> &hs, int j0, int nj, int prec, int variant, bool w1,
                                      const StepArgs &a, cudaStream_t s)
{
    const bool pull = is_pull_variant(prec, variant);
    // directions per launch: a structure's group where the even step is
    // grouped, else as many as the parameters hold
    const int per = lbm_grouped_variant(prec, variant) ? MAX_GROUP : MAX_PLAIN;
    cudaError_t e = cudaSuccess;
    for (int j = j0; j < j0 + nj && e == cudaSuccess; j += per) {
        SlotArgs<false> x;
        const int m = std::min(per, j0 + nj - j);
        for (int d = 0; d < m; ++d) x.s[d] = hs[j + d];
        x.a = a;
        const bool odd = a.n4 & 1;
        e = prec == LBM_FP64 ? launch_slots3d_f64(w1, odd, hs[j].split, hs[j].ntiles, m, s, x)
                             : launch_slots3d_lp(prec, pull, w1, odd, hs[j].split, hs[j].ntiles, m, s, x);
    }
    return e;
}

// Step launches of one call's solves (run_plain3d and the autotuner).
struct PlainSteps {
    int prec, variant;                // the effective variant
    bool w1;
    StepArgs a, ae;                   // work lists: (solve, tile) items, and the even steps' (grouped variants')
    cudaStream_t stream;
    bool slots, gall;
    std::vector<Solve3> live;         // slots variants: the records to step, their groups set

    PlainSteps(int prec_, int variant_, bool w1_, const StepArgs &a_, const StepArgs &ae_, cudaStream_t s)
        : prec(prec_), variant(variant_), w1(w1_), a(a_), ae(ae_), stream(s),
          slots(lbm_slots_variant(prec_, variant_)), gall(lbm_grouped_all(prec_, variant_)) {}

    // `count` steps from relative step rel on (the step after s0 steps done, bit
    // `bit` of the masks): every group of directions in turn takes all of
    // them, so that its lattices stay in L2 from step to step
    cudaError_t launch(long long rel, long long s0, int bit, int count) const
    {
        cudaError_t e = cudaSuccess;
        const int m = slots ? (int)live.size() : 1;
        const int group = slots ? plain_group(prec, variant, live[0], m) : 1;
        for (int j = 0; j < m && e == cudaSuccess; j += group)
            for (int i = 0; i < count && e == cudaSuccess; ++i) {
                const int n4 = (int)((s0 + i + 1) & 3);
                const bool odd = n4 & 1;
                StepArgs x = (slots || (odd && !gall)) ? a : ae;
                x.step = rel + i;
                if (slots) {
                    x.bit = bit + i; x.n4 = n4;
                    e = launch_plain_slots(live, j, std::min(group, m - j), prec, variant, w1, x, stream);
                } else {
                    e = lbm_launch_step(prec, variant, w1, odd, dim3(x.nwork), stream, x);
                }
            }
        return e;
    }
};

static int run_plain3d(lbm_ctx *ctx, std::vector<Solve3> &hs, Solve3 *d_solves, State3 *d_states,
                       const int2 *d_work, int nwork, int prec, int variant, std::vector<State3> &hst)
{
    const int n = (int)hs.size();
    bool w1 = true;
    for (const Solve3 &S : hs) w1 = w1 && S.P.tau == 1.0;
    variant = lbm_effective_variant(prec, variant, hs.empty() || hs[0].meta != nullptr);
    long long s = 0, base = 0;        // steps done; s_base of the unfinished solves (host copy)
    const bool defer = lbm_defers(prec);
    DevMem qbuf(ctx->stream);
    if (defer) CK(qbuf.alloc(sizeof(double) * 4 * DEFER_SLOTS * (size_t)std::max(1, n)));
    double *qb = static_cast<double *>(qbuf.p);
    long long pend0 = 0;              // deferred single launches not yet reduced: [pend0, pend0 + pending)
    int pending = 0;
    StepArgs a;
    a.solves = d_solves; a.work = d_work; a.nwork_dev = nullptr; a.nwork = nwork;
    a.defer = defer ? 1 : 0;
    StepArgs ae = a;                  // even steps (grouped work list for grouped variants)
    DevMem gwork(ctx->stream);
    if (lbm_grouped_variant(prec, variant)) {
        std::vector<int2> items;
        lbm_group_items(hs, items);
        CK(gwork.alloc(sizeof(int2) * items.size()));
        CK(cudaMemcpyAsync(gwork.p, items.data(), sizeof(int2) * items.size(), cudaMemcpyHostToDevice, ctx->stream));
        CK(cudaMemcpyAsync(d_solves, hs.data(), sizeof(Solve3) * n, cudaMemcpyHostToDevice, ctx->stream));
        ae.work = static_cast<const int2 *>(gwork.p);
        ae.nwork = (int)items.size();
    }
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    struct GraphGuard {
        cudaGraph_t &g; cudaGraphExec_t &e;
        ~GraphGuard() { if (e) cudaGraphExecDestroy(e); if (g) cudaGraphDestroy(g); }
    } guard{graph, exec};
    a.wait_ns = ctx->test_wait_ns;
    a.starve = ctx->test_starve;
    ae.wait_ns = a.wait_ns;
    ae.starve = a.starve;
    PlainSteps steps(prec, variant, w1, a, ae, ctx->stream);
    // slots variants launch the records of the unfinished solves only.  (Their
    // kernels request populations before they know whether the solve runs, so a
    // finished one would go on reading its lattice: one direction of 64^3 at
    // porosity 0.8 beside three that had finished took 19.2 us per step in FP64
    // and 11.7 in FP32, now 12.2 and 6.5; alone 10.7 and 5.4.)
    auto relist = [&] {
        steps.live.clear();
        for (int j = 0; j < n; ++j)
            if (hst[j].phase < PH_DONE) steps.live.push_back(hs[j]);
        const int m = (int)steps.live.size();
        for (int j = 0; j < m; ++j) steps.live[j].group = j % MAX_GROUP ? 0 : std::min(MAX_GROUP, m - j);
    };
    // reduce and control the deferred single launches (before s_base moves,
    // before a chunk reuses their slots, and before the states are read)
    auto flush = [&]() -> cudaError_t {
        if (!pending) return cudaSuccess;
        const cudaError_t e = launch_deferred3d(d_solves, n, pend0, pending, qb, 1, 0, ctx->stream);
        pending = 0;
        return e;
    };
    bool stale = false;               // the graph launches solves that have finished
    auto capture = [&]() -> int {
        if (exec) CK(cudaGraphExecDestroy(exec));     // a running one is freed when it has ended
        exec = nullptr;
        if (graph) CK(cudaGraphDestroy(graph));
        graph = nullptr;
        CK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        // launch i of a chunk runs step i + 1 after s_base (a multiple of 4)
        cudaError_t e = steps.launch(0, 0, 0, kGraphSteps3);
        if (e == cudaSuccess && defer) e = launch_deferred3d(d_solves, n, 0, kGraphSteps3, qb, 1, kGraphSteps3, ctx->stream);
        if (e == cudaSuccess && !defer) {
            advance3d_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(d_solves, n, kGraphSteps3);
            e = cudaGetLastError();
        }
        const cudaError_t e2 = cudaStreamEndCapture(ctx->stream, &graph);
        CK(e);
        CK(e2);
        CK(cudaGraphInstantiate(&exec, graph, 0));
        stale = false;
        return LBM_OK;
    };
    for (;;) {
        CK(cudaMemcpyAsync(hst.data(), d_states, sizeof(State3) * n, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        const size_t had = steps.live.size();
        relist();
        stale = stale || (steps.slots && exec && steps.live.size() != had);
        long long target = LLONG_MAX;
        for (int j = 0; j < n; ++j) {
            const State3 &st = hst[j];
            const Ctl3 &c = hs[j].c;
            if (st.phase == PH_RUN) {
                long long nx = (s / c.lag + 1) * c.lag;
                if (c.max_steps > s) nx = std::min(nx, c.max_steps);
                target = std::min(target, nx);
            } else if (st.phase == PH_AVG) {
                target = std::min(target, st.avg_start + c.avg_steps);
            }
        }
        if (target == LLONG_MAX) break;
        if (!exec && target - s >= 2 * kGraphSteps3) {
            const int rc = capture();
            if (rc) return rc;
        }
        while (s < target) {
            if (exec && (s & 3) == 0 && target - s >= kGraphSteps3) {
                CK(flush());
                if (base != s) {
                    // a chunk numbers its steps from s_base: catch up with the single steps
                    advance3d_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(d_solves, n, s - base);
                    CK(cudaGetLastError());
                    base = s;
                }
                CK(cudaGraphLaunch(exec, ctx->stream));
                s += kGraphSteps3;
                base += kGraphSteps3;
                if (stale) {           // made anew while a chunk of the old one runs
                    const int rc = capture();
                    if (rc) return rc;
                }
            } else {
                // every unfinished solve of the call is at step s + 1 (they start
                // together); single launches up to the next chunk, pass or target
                int count = 1;
                if (defer) {
                    while (count < DEFER_SLOTS - pending && s + count < target &&
                           !(exec && ((s + count) & 3) == 0 && target - s - count >= kGraphSteps3)) ++count;
                    if (!pending) pend0 = s - base;
                }
                CK(steps.launch(s - base, s, pending, count));
                s += count;
                if (defer && (pending += count) == DEFER_SLOTS) CK(flush());
            }
        }
        CK(flush());
    }
    return LBM_OK;
}

extern "C" int lbm_solve3d(lbm_ctx *ctx, const uint8_t *solid, int nx, int ny, int nz,
                           int ndir, const double *forces, const lbm_params3d *params,
                           lbm_result3d *results, float *vel_out)
{
    if (!ctx) return LBM_EINPUT;
    if (!solid || !forces || !params || !results || ndir <= 0)
        return lbm_fail_input(ctx, "null argument");
    CK(cudaSetDevice(ctx->device));
    if (nx <= 0 || ny <= 0 || nz <= 0) return lbm_fail_input(ctx, "bad dimensions");
    const long long nn = (long long)nx * ny * nz;
    if (nn >= (1ll << 31) || (long long)Q3 * lbm_plane_elems(nn) >= (1ll << 32))
        return lbm_fail_input(ctx, "lattice too large (19 x nodes must stay below 2^32)");
    int rc = lbm_check_params3d(ctx, *params);
    if (rc) return rc;
    lbm_params3d p = lbm_resolve_variant(*params);
    const int prec = p.precision, npt = lbm_pick_npt(p);

    DevMem mask(ctx->stream);
    long long npore = 0;
    rc = lbm_upload_mask(ctx, solid, nx, (long long)ny * nz, mask, npore);
    if (rc) return rc;
    // 16-bit storage: small structures are bound by the time of one short
    // launch, where the pull form's single kernel is the faster one (three
    // directions at porosity 0.5, us per step, pull / AA pair: 32^3 3.5 / 5.1,
    // 48^3 4.3 / 6.4, 64^3 9.3 / 9.8, 80^3 17.1 / 16.3)
    if (params->variant == LBM_VARIANT_DEFAULT && (prec == LBM_FP16 || prec == LBM_BF16) && npore * ndir <= SMALL_16BIT)
        p.variant = NVAR_LP + 1;

    std::vector<Solve3> hs(ndir);
    std::vector<State3> hst(ndir);
    std::vector<DevMem> lat, part;
    lat.reserve(ndir); part.reserve(ndir);
    DevMem d_states(ctx->stream), d_solves(ctx->stream), d_work(ctx->stream);
    DevMem wpre(ctx->stream), fnode(ctx->stream), meta(ctx->stream), meta2(ctx->stream);
    Solve3 proto;
    lbm_fill_solve3(proto, nx, ny, nz, forces, p, npt);
    proto.mask = static_cast<const uint32_t *>(mask.p);
    rc = lbm_build_pores(ctx, proto, npt, wpre, fnode, meta, meta2);
    if (rc) return rc;
    CK(d_states.alloc(sizeof(State3) * ndir));
    for (int j = 0; j < ndir; ++j) {
        Solve3 &S = hs[j];
        lbm_fill_solve3(S, nx, ny, nz, forces + 3 * j, p, npt);
        lbm_copy_pores(S, proto);
        lat.emplace_back(ctx->stream);
        part.emplace_back(ctx->stream);
        S.split = plain_split(prec, p.variant, S, ndir) ? 1 : 0;
        CK(lat.back().alloc((size_t)lbm_lattice_bytes(S)));
        CK(part.back().alloc(sizeof(double) * (size_t)lbm_partial_doubles(prec, S.ntiles, S.split)));
        lbm_attach_lattice(S, lat.back().p);
        S.mask = static_cast<const uint32_t *>(mask.p);
        S.partials = static_cast<double *>(part.back().p);
        S.st = static_cast<State3 *>(d_states.p) + j;
        lbm_init_state3(hst[j], S.c, 1);
        CK(lbm_init_lattice(prec, S, ctx->stream));
    }
    std::vector<int2> work;
    for (int j = 0; j < ndir; ++j)
        for (int t = 0; t < hs[j].ntiles; ++t) work.push_back(make_int2(j, t));
    CK(d_solves.alloc(sizeof(Solve3) * ndir));
    CK(d_work.alloc(sizeof(int2) * work.size()));
    CK(cudaMemcpyAsync(d_solves.p, hs.data(), sizeof(Solve3) * ndir, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(d_work.p, work.data(), sizeof(int2) * work.size(), cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(d_states.p, hst.data(), sizeof(State3) * ndir, cudaMemcpyHostToDevice, ctx->stream));

    rc = run_plain3d(ctx, hs, static_cast<Solve3 *>(d_solves.p), static_cast<State3 *>(d_states.p),
                     static_cast<const int2 *>(d_work.p), (int)work.size(), prec, p.variant, hst);
    if (rc) return rc;

    if (vel_out) {
        const bool dev = lbm_is_device_ptr(vel_out);
        DevMem vbuf(ctx->stream);
        if (!dev) CK(vbuf.alloc(sizeof(float) * 3 * (size_t)nn));
        for (int j = 0; j < ndir; ++j) {
            float *dst = dev ? vel_out + 3 * nn * j : static_cast<float *>(vbuf.p);
            CK(cudaMemsetAsync(dst, 0, sizeof(float) * 3 * (size_t)nn, ctx->stream));   // solids: u = 0
            CK(lbm_canon(prec, hs[j], hst[j].steps, nullptr, dst, ctx->stream));
            if (!dev)
                CK(cudaMemcpyAsync(vel_out + 3 * nn * j, vbuf.p, sizeof(float) * 3 * nn,
                                   cudaMemcpyDeviceToHost, ctx->stream));
        }
        CK(cudaStreamSynchronize(ctx->stream));
    }

    int out = LBM_OK;
    for (int j = 0; j < ndir; ++j) {
        const State3 &st = hst[j];
        lbm_result3d &r = results[j];
        for (int c = 0; c < 3; ++c) { r.q[c] = st.q[c]; r.se[c] = st.se[c]; }
        r.steps = st.steps;
        r.converged = st.converged;
        r.status = st.status;
        if (st.status == STATUS_WAIT_TIMEOUT) {
            ctx->err = "run " + std::to_string(j) + ": a step kernel gave up waiting for its shared-memory copies";
            out = LBM_ECUDA;
        } else if (st.status) {
            ctx->err = "non-finite flux in run " + std::to_string(j) + " at step " + std::to_string(st.steps);
            out = LBM_EINPUT;
        } else if (!st.converged && out == LBM_OK) {
            out = LBM_NOT_CONVERGED;
        }
    }
    CK(cudaStreamSynchronize(ctx->stream));
    return out;
}

extern "C" int lbm_debug_bulk_wait(lbm_ctx *ctx, unsigned long long wait_ns, int starve)
{
    if (!ctx) return LBM_EINPUT;
    ctx->test_wait_ns = wait_ns;
    ctx->test_starve = starve ? 1 : 0;
    return LBM_OK;
}

extern "C" int lbm_debug_steps3d(lbm_ctx *ctx, const uint8_t *solid, int nx, int ny, int nz,
                                 const double force[3], double tau, int precision, int variant,
                                 long long nsteps, double *f_out, float *u_out, double q_out[3])
{
    if (!ctx) return LBM_EINPUT;
    CK(cudaSetDevice(ctx->device));
    if (nx <= 0 || ny <= 0 || nz <= 0) return lbm_fail_input(ctx, "bad dimensions");
    const long long nn = (long long)nx * ny * nz;
    if (nn >= (1ll << 31) || (long long)Q3 * lbm_plane_elems(nn) >= (1ll << 32))
        return lbm_fail_input(ctx, "lattice too large");
    lbm_params3d p;
    memset(&p, 0, sizeof(p));
    p.tau = tau; p.eps = 0.0; p.lag = LLONG_MAX / 4; p.hold = 1 << 30;
    p.min_steps = 0; p.max_steps = nsteps; p.avg_steps = 0;
    p.precision = precision; p.criterion = LBM_CRIT_DRIFT; p.variant = variant; p.sample = 1;
    int rc = lbm_check_params3d(ctx, p);
    if (rc) return rc;
    p = lbm_resolve_variant(p);
    variant = p.variant;
    const int npt = lbm_pick_npt(p);
    DevMem mask(ctx->stream);
    long long npore = 0;
    rc = lbm_upload_mask(ctx, solid, nx, (long long)ny * nz, mask, npore);
    if (rc) return rc;
    std::vector<Solve3> hs(1);
    std::vector<State3> hst(1);
    Solve3 &S = hs[0];
    lbm_fill_solve3(S, nx, ny, nz, force, p, npt);
    DevMem lat(ctx->stream), part(ctx->stream), d_states(ctx->stream), d_solves(ctx->stream), d_work(ctx->stream);
    DevMem wpre(ctx->stream), fnode(ctx->stream), meta(ctx->stream), meta2(ctx->stream);
    S.mask = static_cast<const uint32_t *>(mask.p);
    rc = lbm_build_pores(ctx, S, npt, wpre, fnode, meta, meta2);
    if (rc) return rc;
    CK(lat.alloc((size_t)lbm_lattice_bytes(S)));
    S.split = plain_split(precision, variant, S, 1) ? 1 : 0;
    CK(part.alloc(sizeof(double) * (size_t)lbm_partial_doubles(precision, S.ntiles, S.split)));
    CK(d_states.alloc(sizeof(State3)));
    lbm_attach_lattice(S, lat.p);
    S.mask = static_cast<const uint32_t *>(mask.p);
    S.partials = static_cast<double *>(part.p); S.st = static_cast<State3 *>(d_states.p);
    lbm_init_state3(hst[0], S.c, 1);
    CK(lbm_init_lattice(precision, S, ctx->stream));
    std::vector<int2> work;
    for (int t = 0; t < S.ntiles; ++t) work.push_back(make_int2(0, t));
    CK(d_solves.alloc(sizeof(Solve3)));
    CK(d_work.alloc(sizeof(int2) * work.size()));
    CK(cudaMemcpyAsync(d_solves.p, &S, sizeof(Solve3), cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(d_work.p, work.data(), sizeof(int2) * work.size(), cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(d_states.p, hst.data(), sizeof(State3), cudaMemcpyHostToDevice, ctx->stream));
    rc = run_plain3d(ctx, hs, static_cast<Solve3 *>(d_solves.p), static_cast<State3 *>(d_states.p),
                     static_cast<const int2 *>(d_work.p), (int)work.size(), precision, variant, hst);
    if (rc) return rc;
    DevMem fb(ctx->stream), ub(ctx->stream);
    if (f_out) {
        CK(fb.alloc(sizeof(double) * Q3 * (size_t)nn));
        CK(cudaMemsetAsync(fb.p, 0, sizeof(double) * Q3 * (size_t)nn, ctx->stream));
    }
    if (u_out) {
        CK(ub.alloc(sizeof(float) * 3 * (size_t)nn));
        CK(cudaMemsetAsync(ub.p, 0, sizeof(float) * 3 * (size_t)nn, ctx->stream));
    }
    CK(lbm_canon(precision, S, nsteps, static_cast<double *>(fb.p), static_cast<float *>(ub.p), ctx->stream));
    if (f_out) CK(cudaMemcpyAsync(f_out, fb.p, sizeof(double) * Q3 * nn, cudaMemcpyDeviceToHost, ctx->stream));
    if (u_out) CK(cudaMemcpyAsync(u_out, ub.p, sizeof(float) * 3 * nn, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if (q_out) for (int c = 0; c < 3; ++c) q_out[c] = hst[0].q[c];
    return LBM_OK;
}

extern "C" int lbm_variant_count(int precision)
{
    return (precision >= LBM_FP64 && precision <= LBM_MD32) ? variant_count(precision) : 0;
}

// Autotuner: every variant runs the same fixed number of steps on the same
// resident lattices with the launches of a tensor solve, timed with CUDA
// events on the launch stream.
extern "C" int lbm_tune3d(lbm_ctx *ctx, const uint8_t *solid, int nx, int ny, int nz, int ndir,
                          int precision, int nsteps, double *ms_per_step, int *best)
{
    if (!ctx) return LBM_EINPUT;
    CK(cudaSetDevice(ctx->device));
    if (nx <= 0 || ny <= 0 || nz <= 0 || ndir <= 0 || nsteps <= 0) return lbm_fail_input(ctx, "bad arguments");
    if (precision < LBM_FP64 || precision > LBM_MD32) return lbm_fail_input(ctx, "unknown precision");
    const long long nn = (long long)nx * ny * nz;
    if (nn >= (1ll << 31) || (long long)Q3 * lbm_plane_elems(nn) >= (1ll << 32))
        return lbm_fail_input(ctx, "lattice too large");
    DevMem mask(ctx->stream);
    long long npore = 0;
    int rc = lbm_upload_mask(ctx, solid, nx, (long long)ny * nz, mask, npore);
    if (rc) return rc;
    const int nv = variant_count(precision);
    // lattice bytes and tile count bounds over the variants
    long long lat_bytes = 0, max_tiles = (nn + TPB - 1) / TPB + 1;
    for (int v = 0; v < nv; ++v) {
        lbm_params3d pv;
        memset(&pv, 0, sizeof(pv));
        pv.tau = 1.0; pv.precision = precision; pv.variant = v;
        Solve3 g;
        const double F0[3] = {0, 0, 0};
        lbm_fill_solve3(g, nx, ny, nz, F0, pv, variant_npt(precision, v));
        g.nfluid = (int)npore;
        lat_bytes = std::max(lat_bytes, lbm_lattice_bytes(g));
        max_tiles = std::max<long long>(max_tiles, g.ntiles);
    }
    std::vector<DevMem> lat;
    lat.reserve(ndir);
    for (int j = 0; j < ndir; ++j) {
        lat.emplace_back(ctx->stream);
        CK(lat.back().alloc((size_t)lat_bytes));
    }
    DevMem d_states(ctx->stream), d_solves(ctx->stream), d_work(ctx->stream), part(ctx->stream);
    CK(d_states.alloc(sizeof(State3) * ndir));
    CK(d_solves.alloc(sizeof(Solve3) * ndir));
    CK(part.alloc(sizeof(double) * 3 * (size_t)max_tiles * ndir));
    cudaEvent_t e0, e1;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    double best_ms = 1e300;
    int best_v = 0;
    for (int v = 0; v < nv; ++v) {
        lbm_params3d p;
        memset(&p, 0, sizeof(p));
        p.tau = 1.0; p.lag = LLONG_MAX / 4; p.hold = 1 << 30; p.max_steps = LLONG_MAX / 4;
        p.precision = precision; p.variant = v; p.sample = 1;
        const int npt = variant_npt(precision, v);
        DevMem wpre(ctx->stream), fnode(ctx->stream), meta(ctx->stream), meta2(ctx->stream);
        Solve3 proto;
        const double F0[3] = {1e-6, 0, 0};
        lbm_fill_solve3(proto, nx, ny, nz, F0, p, npt);
        proto.mask = static_cast<const uint32_t *>(mask.p);
        rc = lbm_build_pores(ctx, proto, npt, wpre, fnode, meta, meta2);
        if (rc) break;
        std::vector<Solve3> hs(ndir);
        std::vector<State3> hst(ndir);
        std::vector<int2> work;
        for (int j = 0; j < ndir; ++j) {
            double F[3] = {0, 0, 0};
            F[j % 3] = 1e-6;
            lbm_fill_solve3(hs[j], nx, ny, nz, F, p, npt);
            lbm_copy_pores(hs[j], proto);
            hs[j].split = plain_split(precision, v, hs[j], ndir) ? 1 : 0;
            lbm_attach_lattice(hs[j], lat[j].p);
            hs[j].mask = proto.mask;
            hs[j].partials = static_cast<double *>(part.p) + 3ll * j * max_tiles;
            hs[j].st = static_cast<State3 *>(d_states.p) + j;
            lbm_init_state3(hst[j], hs[j].c, 1);
            CK(lbm_init_lattice(precision, hs[j], ctx->stream));
            for (int t = 0; t < hs[j].ntiles; ++t) work.push_back(make_int2(j, t));
        }
        DevMem w(ctx->stream);
        CK(w.alloc(sizeof(int2) * work.size()));
        CK(cudaMemcpyAsync(w.p, work.data(), sizeof(int2) * work.size(), cudaMemcpyHostToDevice, ctx->stream));
        CK(cudaMemcpyAsync(d_solves.p, hs.data(), sizeof(Solve3) * ndir, cudaMemcpyHostToDevice, ctx->stream));
        CK(cudaMemcpyAsync(d_states.p, hst.data(), sizeof(State3) * ndir, cudaMemcpyHostToDevice, ctx->stream));
        StepArgs a;
        a.solves = static_cast<const Solve3 *>(d_solves.p);
        a.work = static_cast<const int2 *>(w.p);
        a.nwork_dev = nullptr;
        a.nwork = (int)work.size();
        // no step reduces (no lag multiple comes, redm = 0): the partials, of
        // one slot of whole tiles per direction, are never written
        if (lbm_defers(precision)) { a.defer = 1; a.bit = 0; }
        const int ev = lbm_effective_variant(precision, v, proto.meta != nullptr);
        StepArgs ae = a;
        DevMem gw(ctx->stream);
        if (lbm_grouped_variant(precision, ev)) {
            std::vector<int2> items;
            lbm_group_items(hs, items);
            CK(gw.alloc(sizeof(int2) * items.size()));
            CK(cudaMemcpyAsync(gw.p, items.data(), sizeof(int2) * items.size(), cudaMemcpyHostToDevice, ctx->stream));
            CK(cudaMemcpyAsync(d_solves.p, hs.data(), sizeof(Solve3) * ndir, cudaMemcpyHostToDevice, ctx->stream));
            ae.work = static_cast<const int2 *>(gw.p);
            ae.nwork = (int)items.size();
        }
        // the launches of a solve: directions in groups, a pass of steps at a time
        PlainSteps steps(precision, ev, true, a, ae, ctx->stream);
        steps.live = hs;
        long long s = 0;
        auto run = [&](int count) -> cudaError_t {
            cudaError_t e = cudaSuccess;
            for (int i = 0; i < count && e == cudaSuccess; i += DEFER_SLOTS) {
                const int c = std::min(DEFER_SLOTS, count - i);
                e = steps.launch(s, s, 0, c);
                s += c;
            }
            return e;
        };
        CK(run(std::max(2, nsteps / 4)));
        CK(cudaEventRecord(e0, ctx->stream));
        CK(run(nsteps));
        CK(cudaEventRecord(e1, ctx->stream));
        CK(cudaEventSynchronize(e1));
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, e0, e1));
        const double per = (double)ms / nsteps;
        if (ms_per_step) ms_per_step[v] = per;
        if (per < best_ms) { best_ms = per; best_v = v; }
        CK(cudaStreamSynchronize(ctx->stream));
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    if (best) *best = best_v;
    return LBM_OK;
}
