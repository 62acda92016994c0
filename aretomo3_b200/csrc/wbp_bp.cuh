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
// (two shared wavefronts a voxel and slice, the LSU path at 76 %) -> 19.1 ms; 512 x 512 x
// 41 x 128: 1.82 -> 1.12 ms; the FP16 form, which staged half-precision values and
// differences, 1440 x 512 x 51 x 400: 16.9 -> 15.2 ms with half the error.
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

// One voxel of one slice, every sample tested as the reference does.
template <typename ST>
__device__ __noinline__ float wbp_voxel_tested(const WbpBpArgs& p, int ys, float fX, float fZ, float cent, int* count)
{
    float sum = 0.f;
    int n = 0;
    const float endX = (float)(p.N - 2);
    for (int t = 0; t < p.T; t++) {
        const float2 c = __ldg(&p.cs[t]);
        const float xp = bp_xp<1>(fX, __fmul_rn(fZ, c.y), c.x, cent);
        if (!(xp >= 0.f && xp <= endX)) continue;
        const int i = (int)xp;
        const size_t row = (size_t)ys * p.T + t;
        const float sc = std::is_same<ST, float>::value ? 1.f : __ldg(p.scale + row);
        const ST* q = static_cast<const ST*>(p.sino) + row * p.N + i;
        const float fr = __fsub_rn(xp, (float)i);
        const float v = __fmaf_rn(Stor<ST>::ld(q, sc), __fsub_rn(1.f, fr), __fmul_rn(Stor<ST>::ld(q + 1, sc), fr));
        if (v <= kSentinelTest) continue;   // a NaN sample is summed
        sum = __fadd_rn(sum, v);
        n++;
    }
    *count = n;
    return sum;
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
    const int X = X0 + 16 * (warp & 1) + 2 * (lane & 7), Z = Z0 + 8 * (warp >> 1) + 2 * (lane >> 3);
    const float cent = (float)(p.N / 2), endX = (float)(p.N - 2);
    const float hx = (float)p.GX / 2.0f, hz = (float)p.GZ / 2.0f;
    const float fX0 = (float)X - hx, fX1 = (float)(X + 1) - hx, fZ0 = (float)Z - hz, fZ1 = (float)(Z + 1) - hz;

    unsigned tested = 0;   // slices summed sample by sample
    for (int q = 0; q < nsl; q++)
        if (__ldg(p.flags + ys0 + q) & (kFlagRawLow | kFlagRawSpecial)) tested |= 1u << q;
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
            float lo = 3.0e38f, hi = -3.0e38f;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float cX = (float)(X0 + ((k & 1) ? WBP_T - 1 : 0)) - hx;
                const float cZ = (float)(Z0 + ((k & 2) ? WBP_T - 1 : 0)) - hz;
                const float xp = bp_xp<1>(cX, __fmul_rn(cZ, c.y), c.x, cent);
                lo = fminf(lo, xp);
                hi = fmaxf(hi, xp);
            }
            ws[tid] = (int)floorf(lo) - 1;
            cs_s[tid] = c;
            inside = lo >= 0.01f && hi <= endX - 0.01f;
        }
        inside = __syncthreads_and(inside);   // the whole tile on the detector in every tilt of the chunk
#pragma unroll
        for (int h = 0; h < WB / 4; h++)
            for (int e = tid; e < nc * WBP_WW; e += WBP_THREADS) {
                const int t = e / WBP_WW, x = ws[t] + (e - t * WBP_WW);
                float v[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const size_t row = (size_t)(ys0 + 4 * h + q) * p.T + c0 + t;
                    v[q] = 0.f;
                    if (4 * h + q < nsl && x >= 0 && x < p.N)
                        v[q] = Stor<ST>::ld(static_cast<const ST*>(p.sino) + row * p.N + x,
                                            std::is_same<ST, float>::value ? 1.f : __ldg(p.scale + row));
                }
                win[h * WBP_CHUNK * WBP_WW + e] = make_float4(v[0], v[1], v[2], v[3]);
            }
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

    if (X >= p.GX || Z >= p.GZ) return;   // (GX and GZ are even: blocks lie in the grid or outside it)
    float k[4];
    const bool same = cnt[0] == cnt[1] && cnt[0] == cnt[2] && cnt[0] == cnt[3];
    k[0] = cnt[0] > 0 ? __fdiv_rn(1.f, (float)cnt[0]) : 0.f;
#pragma unroll
    for (int v = 1; v < 4; v++) k[v] = same ? k[0] : cnt[v] > 0 ? __fdiv_rn(1.f, (float)cnt[v]) : 0.f;
    float* out = p.out + ((size_t)ys0 * p.GZ + Z) * p.GX + X;
#pragma unroll
    for (int q = 0; q < WB; q++) {
        if (q >= nsl) break;
        float r[4];
#pragma unroll
        for (int v = 0; v < 4; v++) r[v] = __fmul_rn((q & 1) ? acc[v][q / 2].y : acc[v][q / 2].x, k[v]);
        if ((tested >> q) & 1) {
            for (int v = 0; v < 4; v++) {
                int n;
                const float sum = wbp_voxel_tested<ST>(p, ys0 + q, (v & 1) ? fX1 : fX0, (v >> 1) ? fZ1 : fZ0, cent, &n);
                const float y = n > 0 ? __fmul_rn(sum, __fdiv_rn(1.f, (float)n)) : 0.f;
                if (v == 0) r[0] = y; else if (v == 1) r[1] = y; else if (v == 2) r[2] = y; else r[3] = y;
            }
        }
        float* o = out + (size_t)q * p.GZ * p.GX;
        *reinterpret_cast<float2*>(o) = make_float2(r[0], r[1]);
        *reinterpret_cast<float2*>(o + p.GX) = make_float2(r[2], r[3]);
    }
}

// Grid (tiles x, tiles z, ceil(slices / WB)).
template <typename ST, int WB>
__global__ void __launch_bounds__(WBP_THREADS, 3) k_bp_wbp(const __grid_constant__ WbpBpArgs p)
{
    wbp_bp_tile<ST, WB>(p, blockIdx.x, blockIdx.y, blockIdx.z);
}

}  // namespace at3r
