// The batched WBP form: persistent stage kernels over many series.
#pragma once
#include "recon_kernels.cuh"
#include "wbp_bp.cuh"

namespace at3r {

// ---------------------------------------------------------------------------
// Batched WBP: persistent stage kernels over many series.  A wave holds one
// slab of every series in the batch (series of fewer slabs drop out of later
// waves); each of the five WBP stages runs as one launch over the whole wave,
// whose persistent CTAs pull virtual blocks — (series' slab, block of that
// stage) — from a counter until none is left, and run the same block body
// the per-series kernels run, so every result is bit-identical to the
// per-series launches.
// ---------------------------------------------------------------------------
struct WbpSlab {
    const float* proj;        // series projections [T][ny][nx]
    size_t tilt_stride;
    int row_pitch, y0;        // nx; first row of the slab
    const float2* cs;
    int T, N, Nx, Nz, S;
    const float* h;           // R-weight transfer function
    void* filt;               // staged, filtered sinogram (storage type of the batch)
    float* scale;
    int* flags;
    float* g2;                // 2x grid, then the cropped spectrum
    float2* y;                // row spectra
    float* vol;               // the slab's first output slice
    size_t vol_slice;
    int b_rweight, b_row, b_xc2r, zcrop_cb, zcrop_pitch, packed;
    float norm;
    WbpBpArgs bp;
    FftPlan fN, f2x, f2z, fz, fx;
    int gx[5];                // virtual grid x of each stage (y is the slab's slices; the BP's y, z below)
    int bp_gy, bp_gz;
};

constexpr int WBP_WAVE_SLICES = 4;   // slices a back-projection block carries
constexpr int kWbpStages = 5;   // rweight, bp, row_r2c, zcrop, x_c2r

// Flags of every slab of the wave to zero (run_slab_t's memset); grid = slabs.
__global__ void k_wave_flags(const WbpSlab* __restrict__ w)
{
    const WbpSlab& d = w[blockIdx.x];
    for (int i = threadIdx.x; i < d.S; i += blockDim.x) d.flags[i] = 0;
}

// Stage STAGE of a wave: start[k] is the first virtual block of slab k
// (start[nslabs] the total); counter starts at 0.
template <int STAGE, typename ST, int RS>
__global__ void __launch_bounds__(STAGE == 1 ? WBP_THREADS : 512, STAGE == 1 ? 3 : (RS < 2 ? 2 : 1))
    k_wbp_wave(const WbpSlab* __restrict__ w, const int* __restrict__ start, int nslabs, int* __restrict__ counter)
{
    __shared__ int s_item;
    const int total = start[nslabs];
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
        __syncthreads();
        const int item = s_item;
        __syncthreads();
        if (item >= total) return;
        int lo = 0, hi = nslabs - 1;   // the slab whose block range holds item
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (start[mid] <= item) lo = mid;
            else hi = mid - 1;
        }
        const WbpSlab& d = w[lo];
        const int v = item - start[lo];
        const int bx = v % d.gx[STAGE], by = v / d.gx[STAGE];
        if constexpr (STAGE == 0) {
            rweight_block<ST, RS>(d.proj, d.tilt_stride, d.row_pitch, d.y0, d.cs, d.T, d.N, d.Nz, d.h, d.fN,
                                  d.b_rweight, static_cast<ST*>(d.filt), d.scale, d.flags, bx, by);
        } else if constexpr (STAGE == 1) {
            wbp_bp_tile<ST, WBP_WAVE_SLICES>(d.bp, bx, by % d.bp_gy, by / d.bp_gy);
        } else if constexpr (STAGE == 2) {
            row_r2c_block<RS>(d.g2, d.Nx, d.Nz, d.f2x, d.b_row, d.y, bx, by);
        } else if constexpr (STAGE == 3) {
            const float2* yv = d.y;
            zcrop_block<RS>(yv, d.Nx, d.Nz, d.zcrop_cb, d.zcrop_pitch, d.f2z, d.fz, d.norm,
                            reinterpret_cast<float2*>(d.g2), bx, by);
        } else {
            x_c2r_block<RS>(reinterpret_cast<const float2*>(d.g2), d.Nx, d.Nz, d.fx, d.b_xc2r, d.packed, d.vol,
                            d.vol_slice, bx, by);
        }
        __syncthreads();   // shared memory is reused by the next block
    }
}

}  // namespace at3r
