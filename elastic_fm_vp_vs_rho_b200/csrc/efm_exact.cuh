// Table entry of the exact-adjoint kernels (efm_exact.cu, efm_exact_stream.cu), one per
// instance.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "efm_internal.cuh"

struct EfmExact {
    int nx, ny, nz, W;
    int tiles_x, tiles_z, tiles_y, tile_begin;   // one-thread-per-cell kernels
    int st_tx, st_tz, st_ty, st_begin, ychunk;   // plane-streaming kernels (efm_exact_stream.cu)
    int nt;
    float k;
    const float *lam, *mu, *rho, *cpml;
    float *bv[3], *bt[6];   // nine consecutive volumes (the streaming kernels use stride N)
    const float *pin;   // adjoint memory variables, read (x, y, z slab families, 6 vars each)
    float *pout;        // ... written
    int64_t psx_n, psy_n, psz_n;
    const float *seg;   // forward (vx vy vz txx tyy tzz txy txz tyz) per slot
    int64_t slot_stride;
    float *g_lam, *g_mu, *g_rho;
    float *scr;         // 9 volumes: ubar (velocity transpose) or k C taubar's 6 entries + 3 shear products
    const float *avg;   // 6 volumes: harmonic mu_xy, mu_xz, mu_yz, buoyancy x, y, z
    int nsrc;
    int sx[EFM_NSRC], sy[EFM_NSRC], sz[EFM_NSRC];
    float mt[EFM_NSRC][6];
    const float *wav;
    double *mtg;
    int nrec;
    const int *rec_lin, *rec_id;
    const float *res;
};

// Launch as a programmatic dependent (EFM_OPT_PDL of the calling context): the kernel's prologue
// overlaps the tail of the preceding one.  Every thread of such a kernel waits in efm_pdl_wait, so
// that its completion implies the preceding kernel's.
extern "C" int efm_stream_pdl();

template <typename... KArgs, typename... Args>
cudaError_t efm_launch_pdl(void (*k)(KArgs...), int grid, int threads, int smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = efm_stream_pdl() ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k, args...);
    const cudaError_t l = cudaGetLastError();
    return e != cudaSuccess ? e : l;
}
