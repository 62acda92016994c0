// WBP back-projection onto the 2x grid (AreTomo/Recon/GBackProjWbp.cu:14-53):
// the mean over the tilts of the lerped filtered sinogram, 0 where no tilt
// contributes.
//
// A CTA covers 32 x 32 voxels of WB slices (the geometry is every slice's); a
// thread carries a block of 2 x 2 voxels for all of them.  On the 2x grid the
// block's detector positions lie within (cos + |sin|) / 2 <= 0.71 of one another, so
// three consecutive samples hold all its taps and voxel v takes sample k
// with the hat weight max(0, 1 - |x_v - k|): the lerp's own two weights, and zero.
// Tilts go in chunks of WBP_CHUNK: the CTA stages each tilt's detector window (the
// tile's corners bound it) in shared memory, four slices to a 16-byte entry, and a
// thread's three loads serve four voxels and four slices — 3 bytes a voxel, tilt and
// slice against 8 when every voxel loads its own pair of samples.  Lanes are 8 x 4
// blocks, so that a quarter-warp's entries are few and neighbouring.  Positions,
// index and weights are formed once for the WB slices; sums run in the reference's
// (tilt) order with packed multiply-adds.
// Measured (4096 x 128 rows x 41, thickness 1200): 31.6 ms with a pair of samples a voxel
// (two shared wavefronts a voxel and slice, the LSU path at 76 %) -> 18.8 ms; 512 x 512 x
// 41 x 128: 1.82 -> 1.06 ms; the FP16 form, which staged half-precision values and
// differences, 1440 x 512 x 51 x 400: 16.9 -> 13.1 ms with half the error.  Bound by the
// multiply-adds (FMA pipe 72-77 % busy, issue 66 %, shared-memory wavefronts 57 %).
// Slices whose sinogram holds values near the -1e10 "empty" marker, infinities or
// NaN (flag bits) are summed sample by sample as the reference tests them.
#pragma once
#include "recon_kernels.cuh"

namespace at3r {

constexpr int WBP_T = 32, WBP_THREADS = 256, WBP_CHUNK = 16;
constexpr int WBP_WW = 28;   // window stride: 31 (cos + |sin|) / 2 + 6 < 28 samples

struct WbpBpArgs {
    const void* sino;        // [slices][T][N] of the storage type
    const float* scale;      // [slices][T] row scales (16-bit storage), else null
    const float2* cs;
    const int* flags;        // per-slice flag bits
    int* seen;               // run summary (may be null)
    float* out;              // [slices][GZ][GX]
    int T, N, GX, GZ, S;
};

template <int WB>
__host__ __device__ constexpr size_t wbp_bp_smem()
{
    return (sizeof(float2) + sizeof(int)) * WBP_CHUNK + sizeof(float) * WB * WBP_CHUNK * WBP_WW;
}

// First voxel of a thread's block.
__device__ __forceinline__ int wbp_x(int X0, int warp, int lane) { return X0 + 16 * (warp & 1) + 2 * (lane & 7); }
__device__ __forceinline__ int wbp_z(int Z0, int warp, int lane) { return Z0 + 8 * (warp >> 1) + 2 * (lane >> 3); }

// Tile (X0, Z0) of tilt (c): positions of its four corners on the detector.
__device__ __forceinline__ void wbp_span(float2 c, int X0, int Z0, float hx, float hz, float cent, float& lo, float& hi)
{
    lo = 3.0e38f;
    hi = -3.0e38f;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float cX = (float)(X0 + ((k & 1) ? WBP_T - 1 : 0)) - hx;
        const float cZ = (float)(Z0 + ((k & 2) ? WBP_T - 1 : 0)) - hz;
        const float xp = bp_xp<1>(cX, __fmul_rn(cZ, c.y), c.x, cent);
        lo = fminf(lo, xp);
        hi = fmaxf(hi, xp);
    }
}

// Windows of tilts [c0, c0 + nc) of slices [ys, ys + n), n <= 4, into win[nc][WBP_WW]; zero off the detector.
// NAN_STAYS: slices of the mask `nan` keep a stored NaN, the 16-bit types' code of a missing value.
template <typename ST, bool NAN_STAYS = false>
__device__ __forceinline__ void wbp_stage(const WbpBpArgs& p, float4* win, const int* ws, int c0, int nc, int ys, int n,
                                          unsigned nan = 0)
{
    for (int e = threadIdx.x; e < nc * WBP_WW; e += WBP_THREADS) {
        const int t = e / WBP_WW, x = ws[t] + (e - t * WBP_WW);
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const size_t row = (size_t)(ys + q) * p.T + c0 + t;
            v[q] = 0.f;
            if (q < n && x >= 0 && x < p.N) {
                const ST* src = static_cast<const ST*>(p.sino) + row * p.N + x;
                const float sc = std::is_same<ST, float>::value ? 1.f : __ldg(p.scale + row);
                v[q] = NAN_STAYS && ((nan >> q) & 1) ? static_cast<float>(__ldg(src)) * sc : Stor<ST>::ld(src, sc);
            }
        }
        win[e] = make_float4(v[0], v[1], v[2], v[3]);
    }
}

// The tile of four slices from ys on, every sample tested as the reference does, for the
// slices in `mask`.  The whole CTA takes part: windows are staged as in the untested sums,
// and one pair of 16-byte entries serves the four slices.  Measured (reconstruction of 4096 x
// 64 rows x 41, thickness 1200, an infinite pixel in every row): 113.7 ms voxel by voxel
// from global memory, 44.2 ms; 22.6 ms with none.
template <typename ST>
__device__ __noinline__ void wbp_quad_tested(const WbpBpArgs& p, int bx, int by, int ys, unsigned mask)
{
    const int n = min(4, p.S - ys);
    extern __shared__ float4 bsm4[];
    float4* win = bsm4;                                                      // [WBP_CHUNK][WBP_WW]
    float2* cs_s = reinterpret_cast<float2*>(win + WBP_CHUNK * WBP_WW);      // [WBP_CHUNK]
    int* ws = reinterpret_cast<int*>(cs_s + WBP_CHUNK);                      // [WBP_CHUNK]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int X0 = bx * WBP_T, Z0 = by * WBP_T, X = wbp_x(X0, warp, lane), Z = wbp_z(Z0, warp, lane);
    const float cent = (float)(p.N / 2), endX = (float)(p.N - 2);
    const float hx = (float)p.GX / 2.0f, hz = (float)p.GZ / 2.0f;
    // a slice with no value near the empty marker holds no missing value: its NaNs are NaNs
    unsigned nan = 0;
    for (int q = 0; q < n; q++)
        if (!(__ldg(p.flags + ys + q) & kFlagRawLow)) nan |= 1u << q;
    float sum[4][4], cnt[4][4];   // [voxel 2 dz + dx][slice]
#pragma unroll
    for (int v = 0; v < 4; v++)
#pragma unroll
        for (int q = 0; q < 4; q++) sum[v][q] = cnt[v][q] = 0.f;
    for (int c0 = 0; c0 < p.T; c0 += WBP_CHUNK) {
        const int nc = min(WBP_CHUNK, p.T - c0);
        if (tid < nc) {
            const float2 c = __ldg(&p.cs[c0 + tid]);
            float lo, hi;
            wbp_span(c, X0, Z0, hx, hz, cent, lo, hi);
            ws[tid] = (int)floorf(lo) - 1;
            cs_s[tid] = c;
        }
        __syncthreads();
        wbp_stage<ST, true>(p, win, ws, c0, nc, ys, n, nan);
        __syncthreads();
        for (int t = 0; t < nc; t++) {
            const float2 c = cs_s[t];
#pragma unroll
            for (int v = 0; v < 4; v++) {
                const float fX = (float)(X + (v & 1)) - hx, fZ = (float)(Z + (v >> 1)) - hz;
                const float xp = bp_xp<1>(fX, __fmul_rn(fZ, c.y), c.x, cent);
                if (!(xp >= 0.f && xp <= endX)) continue;
                const int i = (int)xp;
                const float fr = __fsub_rn(xp, (float)i), om = __fsub_rn(1.f, fr);
                const float4 f0 = win[t * WBP_WW + i - ws[t]], f1 = win[t * WBP_WW + i - ws[t] + 1];
                const float a0[4] = {f0.x, f0.y, f0.z, f0.w}, a1[4] = {f1.x, f1.y, f1.z, f1.w};
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float s = __fmaf_rn(a0[q], om, __fmul_rn(a1[q], fr));
                    if (s <= kSentinelTest) continue;   // a NaN sample is summed
                    sum[v][q] = __fadd_rn(sum[v][q], s);
                    cnt[v][q] += 1.f;
                }
            }
        }
        __syncthreads();
    }
    if (X >= p.GX || Z >= p.GZ) return;
    float* out = p.out + ((size_t)ys * p.GZ + Z) * p.GX + X;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if (!((mask >> q) & 1)) continue;
        float r[4];
#pragma unroll
        for (int v = 0; v < 4; v++) r[v] = cnt[v][q] > 0.f ? __fmul_rn(sum[v][q], __fdiv_rn(1.f, cnt[v][q])) : 0.f;
        float* o = out + (size_t)q * p.GZ * p.GX;
        *reinterpret_cast<float2*>(o) = make_float2(r[0], r[1]);
        *reinterpret_cast<float2*>(o + p.GX) = make_float2(r[2], r[3]);
    }
}

template <typename ST, int WB>
__device__ __forceinline__ void wbp_bp_tile(const WbpBpArgs& p, int bx, int by, int bz)
{
    extern __shared__ float4 bsm4[];
    float4* win = bsm4;                                                      // [WB / 4][WBP_CHUNK][WBP_WW]
    float2* cs_s = reinterpret_cast<float2*>(win + WB / 4 * WBP_CHUNK * WBP_WW);   // [WBP_CHUNK]
    int* ws = reinterpret_cast<int*>(cs_s + WBP_CHUNK);                      // [WBP_CHUNK]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ys0 = bz * WB, nsl = min(WB, p.S - ys0);
    const int X0 = bx * WBP_T, Z0 = by * WBP_T;
    const int X = wbp_x(X0, warp, lane), Z = wbp_z(Z0, warp, lane);
    const float cent = (float)(p.N / 2), endX = (float)(p.N - 2);
    const float hx = (float)p.GX / 2.0f, hz = (float)p.GZ / 2.0f;
    const float fX0 = (float)X - hx, fX1 = (float)(X + 1) - hx, fZ0 = (float)Z - hz, fZ1 = (float)(Z + 1) - hz;

    if (p.seen && bx == 0 && by == 0 && tid < nsl) atomicOr(p.seen, __ldg(p.flags + ys0 + tid) & kFlagsReported);

    float2 acc[4][WB / 2];   // voxel 2 dz + dx
    int cnt[4];
#pragma unroll
    for (int v = 0; v < 4; v++) {
        cnt[v] = 0;
#pragma unroll
        for (int q = 0; q < WB / 2; q++) acc[v][q] = make_float2(0.f, 0.f);
    }
    for (int c0 = 0; c0 < p.T; c0 += WBP_CHUNK) {
        const int nc = min(WBP_CHUNK, p.T - c0);
        int inside = 1;
        if (tid < nc) {
            const float2 c = __ldg(&p.cs[c0 + tid]);
            float lo, hi;
            wbp_span(c, X0, Z0, hx, hz, cent, lo, hi);
            ws[tid] = (int)floorf(lo) - 1;
            cs_s[tid] = c;
            inside = lo >= 0.01f && hi <= endX - 0.01f;
        }
        inside = __syncthreads_and(inside);   // the whole tile on the detector in every tilt of the chunk
#pragma unroll
        for (int h = 0; h < WB / 4; h++)
            wbp_stage<ST>(p, win + h * WBP_CHUNK * WBP_WW, ws, c0, nc, ys0 + 4 * h, nsl - 4 * h);
        __syncthreads();
        // EDGE: samples off the detector take no part
        auto sum_tilt = [&](int t, auto edge) {
            constexpr bool EDGE = decltype(edge)::value;
            const float2 c = cs_s[t];
            const float s0 = __fmul_rn(fZ0, c.y), s1 = __fmul_rn(fZ1, c.y);
            const float xp[4] = {bp_xp<1>(fX0, s0, c.x, cent), bp_xp<1>(fX1, s0, c.x, cent),
                                 bp_xp<1>(fX0, s1, c.x, cent), bp_xp<1>(fX1, s1, c.x, cent)};
            const float lo = c.y >= 0.f ? xp[0] : xp[2];   // the block's leftmost position
            float kf;
            int e = t * WBP_WW - ws[t];
            if constexpr (EDGE) {
                kf = floorf(lo);
                e += (int)kf;
            } else {
                const float tr = __fadd_rd(lo, kMagic);   // floor(lo) from the bits of lo + 2^23
                kf = __fsub_rn(tr, kMagic);
                e += __float_as_int(tr) - kMagicBits;
            }
            float d[4];
#pragma unroll
            for (int v = 0; v < 4; v++) {
                d[v] = __fsub_rn(xp[v], kf);
                if constexpr (EDGE) {
                    const bool in = xp[v] >= 0.f && xp[v] <= endX;
                    d[v] = in ? d[v] : -8.f;   // weight 0 everywhere
                    cnt[v] += in;
                }
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                float2 a[WB / 2];
#pragma unroll
                for (int h = 0; h < WB / 4; h++) {
                    const float4 f = win[h * WBP_CHUNK * WBP_WW + e + k];
                    a[2 * h] = make_float2(f.x, f.y);
                    a[2 * h + 1] = make_float2(f.z, f.w);
                }
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const float w = __saturatef(1.f - fabsf(d[v] - (float)k));
                    const float2 w2 = make_float2(w, w);
#pragma unroll
                    for (int q = 0; q < WB / 2; q++) fma2(acc[v][q], w2, a[q]);
                }
            }
        };
        if (inside) {
            for (int t = 0; t < nc; t++) sum_tilt(t, std::false_type{});
#pragma unroll
            for (int v = 0; v < 4; v++) cnt[v] += nc;
        } else {
            for (int t = 0; t < nc; t++) sum_tilt(t, std::true_type{});
        }
        __syncthreads();
    }

    // (GX and GZ are even: blocks lie in the grid or outside it)
    const int nout = X < p.GX && Z < p.GZ ? nsl : 0;
    float k[4];
    const bool same = cnt[0] == cnt[1] && cnt[0] == cnt[2] && cnt[0] == cnt[3];
    k[0] = cnt[0] > 0 ? __fdiv_rn(1.f, (float)cnt[0]) : 0.f;
#pragma unroll
    for (int v = 1; v < 4; v++) k[v] = same ? k[0] : cnt[v] > 0 ? __fdiv_rn(1.f, (float)cnt[v]) : 0.f;
    float* out = p.out + ((size_t)ys0 * p.GZ + Z) * p.GX + X;
#pragma unroll
    for (int q = 0; q < WB; q++) {
        if (q >= nout) break;
        float r[4];
#pragma unroll
        for (int v = 0; v < 4; v++) r[v] = __fmul_rn((q & 1) ? acc[v][q / 2].y : acc[v][q / 2].x, k[v]);
        float* o = out + (size_t)q * p.GZ * p.GX;
        *reinterpret_cast<float2*>(o) = make_float2(r[0], r[1]);
        *reinterpret_cast<float2*>(o + p.GX) = make_float2(r[2], r[3]);
    }
    // slices summed sample by sample (the same for the whole CTA): a pass of its own, over what is stored
    // above.  Lane q looks at slice q, and only here: known from the start, or read slice by slice,
    // the mask cost the sums above registers (1440 x 512 x 51 x 400 in FP16: 13.07 ms as it is,
    // 13.48 and 13.31; 13.03 with the test in line, per voxel)
    const int lq = lane & 7;
    const unsigned tested = __ballot_sync(0xffffffffu, lane < nsl && (__ldg(p.flags + ys0 + min(lq, nsl - 1)) &
                                                                      (kFlagRawLow | kFlagRawSpecial)));
#pragma unroll
    for (int h = 0; h < WB / 4; h++)
        if ((tested >> (4 * h)) & 15)
            wbp_quad_tested<ST>(p, bx, by, ys0 + 4 * h, (tested >> (4 * h)) & 15);
}

// Grid (tiles x, tiles z, ceil(slices / WB)).
template <typename ST, int WB>
__global__ void __launch_bounds__(WBP_THREADS, 3) k_bp_wbp(const __grid_constant__ WbpBpArgs p)
{
    wbp_bp_tile<ST, WB>(p, blockIdx.x, blockIdx.y, blockIdx.z);
}

}  // namespace at3r
