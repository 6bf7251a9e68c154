// lcmc_launch.h - host-side launchers exported by the kernel translation units.
#pragma once
#include <cuda_runtime.h>

#include "lcmc_internal.h"

namespace lcmc {

// Launch of a kernel of the FP64 colour phases.  The next such kernel in the
// stream may be launched while this one runs: each calls phase_begin() first,
// which waits until all that came before it in the stream is complete and
// visible, so only the launch itself overlaps (8192 particles, 27 phases of two
// kernels: 0.465 -> 0.350 ms per sweep).  The FP32 phase kernels gained 1 % from
// it in small systems and lost 4 % in batches, where the early blocks of the
// hand-over kernel took the other streams' shared memory: they are launched
// plainly.
template <typename... P, typename... A>
inline void launch_phase(void (*f)(P...), int grid, int block, int smem, cudaStream_t s, const A &...a)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, f, P(a)...);
}

#ifdef __CUDACC__
__device__ __forceinline__ void phase_begin()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

// lcmc_rebin.cu
void launch_rebin(const DevView &v, cudaStream_t s, int grid, bool trials); // trials: the sweep's trial moves too
// per-cell results of the colour phases into the statistics and the running
// energy (before the volume move); then the sweep counter and adaptive step
void launch_sweep_stats(const DevView &v, cudaStream_t s);
void launch_sweep_advance(const DevView &v, cudaStream_t s);

// lcmc_sweep_exact.cu (FP64, bit-identical to the CPU oracle)
void exact_init(); // before the first FP64 colour phase
constexpr long long EX_MOST = 256ll << 20 >> 9; // rows (512 bytes) of a batch
void exact_scratch_size(int ntot, long long most, long long *cap, long long *alloc, int *nb);
void launch_exact_offsets(const DevView &v, cudaStream_t s); // after the rebin, before the colour phases
void launch_phase_exact(const DevView &v, cudaStream_t s, int ci, int grid);
void launch_volume_energies(const DevView &v, cudaStream_t s, double *e0, double *e1, int *hard, int grid,
                            bool per_particle);
void launch_total_energy(const DevView &v, cudaStream_t s, double *e0, double *e1, int *hard, int grid, bool cells,
                         bool by_cells, bool per_particle);
int energy_exact_blocks_per_sm(); // resident blocks of 128 threads per SM

// lcmc_sweep_fast.cu (FP32)
struct FastVariant {
    int amax; // active-cell capacity of a class
};
// The FP32 phase kernel a context runs
struct FastChoice {
    int cls = 0;        // capacity class
    bool spec21 = true; // mu = 2, nu = 1, sigma0 = 1 in every replica
    bool one_k = true;  // the same pair constants in every replica: they come with the launch
    int shape = 2;      // block shape: 0 for cells of a gas, 1 for at most 40 particles, 2 + class by class
    bool wide = false;  // 512 threads per cell: at most a cell per SM
    // the same kernel (the class is only a capacity)
    bool same_kernel(const FastChoice &o) const
    {
        return spec21 == o.spec21 && one_k == o.one_k && wide == o.wide && shape == o.shape;
    }
    bool operator==(const FastChoice &o) const { return cls == o.cls && same_kernel(o); }
};
constexpr int FAST_SHAPES = 5;
constexpr int FAST_SPARSE = 32; // most particles of a cell of shape 0
int fast_shape_candidates(int shape); // places of the static cells' particles
int fast_variant_count();
FastVariant fast_variant(int i);
void launch_phase_fast(const FastChoice &c, const GBConsts &k, const DevView &v, cudaStream_t s, int ci, int grid);
int fast_blocks_per_sm(const FastChoice &c);
// retries (FP32, the largest capacity) and FP64 attempts of the cells the FP32 kernel left in colour phase ci
void launch_phase_rescue(bool spec21, const DevView &v, cudaStream_t s, int ci, int grid);
void rescue_init(); // once per process before the first hand-over launch

// lcmc_misc.cu
void launch_q_chunk_sums(const DevView &v, cudaStream_t s); // Q-tensor chunk sums of every replica
// chunk sums of (e0, e1, hard) of the NPT replicas not rejected at stage 1
void launch_chunk_sums_volume(const DevView &v, cudaStream_t s, const double *e0, const double *e1, const int *hard);
// FP32-pair screen of the volume move: energies at V and V', chunk sums, stage 1
void launch_screen(const DevView &v, cudaStream_t s, int grid, bool spec21);
void launch_chunk_sums_screen(const DevView &v, cudaStream_t s);
int screen_blocks_per_sm();
// from launch_total_energy's sums (its `cells`)
void launch_energy_reduce(const DevView &v, cudaStream_t s, const double *e0, int replica_only, bool cells);
// FP64 energy check of the due replicas (all = every replica) from launch_total_energy's sums with cells = true
void launch_energy_check(const DevView &v, cudaStream_t s, const double *e0, int all);
void launch_order_sums(const DevView &v, cudaStream_t s, int r, double *out);
void launch_to_id_order(const DevView &v, cudaStream_t s, int r, int grid);
void launch_validate_upload(const double *const x[6], int *id, int n, const double L[3], double R2, int *flag,
                            cudaStream_t s, int grid);

} // namespace lcmc
struct lcmc_mlp;
namespace lcmc {
// lcmc_mlp.cu (in-sweep surrogate inference)
unsigned wait_limit(); // what lcmc_set_wait_limit set
void *mlp_input(lcmc_mlp *m);
int mlp_ld(lcmc_mlp *m);
int mlp_bmax(lcmc_mlp *m);
int mlp_n_in(lcmc_mlp *m);
const float *mlp_forward_device(lcmc_mlp *m, int B, cudaStream_t s);
int *mlp_err(lcmc_mlp *m);

// lcmc_da.cu (surrogate features, delayed acceptance, recordings)
void launch_features(const DevView &v, cudaStream_t s, void *X, int ldx, int grid);
void launch_da_stage1(const DevView &v, cudaStream_t s, const float *y);
void launch_record_samples(const DevView &v, cudaStream_t s);
void launch_hist_record(const DevView &v, cudaStream_t s);
void launch_volume_propose(const DevView &v, cudaStream_t s);
void launch_volume_finish(const DevView &v, cudaStream_t s, double *e0, double *e1, int *hard, int grid,
                          bool per_particle);

// lcmc_noalloc.cu (allocation-free FP64 total energy on a caller's stream)
int total_energy_noalloc(const GBConsts &k, int n, const double *px, const double *py, const double *pz,
                         const double *ox, const double *oy, const double *oz, const double box[3], double *d_out,
                         cudaStream_t st, char *msg, size_t len);

// lcmc_pairtest.cu / lcmc_pairtest64.cu (pair term on given inputs)
void launch_pair_terms32(const GBConsts &k, int n, const double *d, const double *ei, const double *ej, double *out,
                         cudaStream_t s);
void launch_pair_terms64(const GBConsts &k, int n, const double *d, const double *ei, const double *ej, double *out,
                         cudaStream_t s);

} // namespace lcmc
