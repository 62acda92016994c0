// SART kernels for FP32 series of many rows: slices on the lanes.
//
// Every y-slice has the same geometry, so the interpolation weights of a
// voxel or a ray serve all slices.  Here the slices are the innermost index:
//   volume    W[group][Nz][Nx][G]   rows z flipped, G slices of a group
//   sinogram  R[group][T][N][G]     weighted rows and residual
// with G = 16, 32 or 64 (slabs of fewer slices: 8 or 4): a few lanes share a position and
// carry its G slices, read as contiguous runs.  Every load is then fully coalesced whatever the tilt (with
// rays or voxels on the lanes, a warp's samples lie 1/cos or cos apart and a
// 16-byte tap load took 6.6 to 8.1 wavefronts for 4), and a thread that carries a
// few neighbouring rays or voxels loads the taps they share once.  What a slice's
// result is made of does not depend on G, so every G gives the same bits.
// Measured (B200, ms in the two projectors, four-slice kernels first): 4096 x 64 x 41 x
// 1200, 15 iterations, forward 184 -> 99, back 84 -> 61; 1024 x 256 x 61 x 300,
// 15 iterations, 64 -> 43 and 31 -> 22.  FP32 only: with a 16-bit copy of the volume the
// forward projector's conversions took what the bytes saved (2048 x 96 x 41 x
// 600, 10 iterations: 33.6 ms against 31.3 for the four-slice 16-bit kernel).
#pragma once
#include "recon_kernels.cuh"

#include <algorithm>

namespace at3r {

constexpr int WIDE_THREADS = 256, WIDE_WARPS = WIDE_THREADS / 32;
constexpr int FPW_RAYS = 2;                  // rays a thread carries
constexpr int FPW_LP = 4;                    // lanes that share its rays
constexpr int FPW_WARP_RAYS = FPW_RAYS * 32 / FPW_LP, FPW_PAIRS = 32 / FPW_LP;
constexpr int FPW_MAX_COLS = 32;             // columns of a ray pair's window; wider: sample by sample
constexpr int FPW_MAX_ROWS = 8;              // volume rows per weight table
constexpr int WIDE_POLLS = 1 << 22;          // polls of a wait for a bulk copy before it gives up

// Back-projector: slices of a thread, NS = 8 as two runs of four at 4 LP k + 4 lp
// (each 16-byte load of the LP lanes is contiguous).
template <int LP>
__device__ __forceinline__ int bpw_slice(int lp, int k)
{
    return 4 * LP * k + 4 * lp;
}
// Forward projector: slices of register group b (four slices) of lane lp of pair
// `pair`, NS slices a thread.  Neighbouring pairs, whose lanes share a quarter-warp, take
// the 64-byte chunks of a column in swapped order: both would otherwise hit the
// same banks.
template <int NS>
__device__ __forceinline__ int fpw_slice(int lp, int pair, int b)
{
    return NS <= 4 ? NS * lp : 16 * (b ^ (pair & 1)) + 4 * lp;
}

// Columns that rays up to d detector samples apart can touch in one volume row of
// tilt (c, s): they lie 1/c apart, and the samples of one row span 2 tan.
__device__ inline int fpw_cols(int d, float c, float s, int N, int Nx)
{
    const double dc = c, t = fabs((double)s) / dc;
    const double span = d / dc + 2.01 * t + 0.02 + 2.4e-7 * (double)N / dc;
    const double n = floor(span) + 3.0;
    return n > (double)Nx ? Nx : (int)n;
}

// ---------------------------------------------------------------------------
// Staging: R[g][t][u][G] = proj[t][y0 + ys][u] * (cos_t / Nz), zero for the
// slices that fill up the last group (CDoSartRecon.cpp:100-117,
// GWeightProjs.cu:7-19).  A 32 x G tile through shared memory.  Bound by
// HBM; grid (ceil(N / 32), T, groups).
// ---------------------------------------------------------------------------
template <int G>
__global__ void __launch_bounds__(256) k_gather_wide(const float* __restrict__ proj, size_t tilt_stride,
                                                     int row_pitch, int y0, const float2* __restrict__ cs, int T,
                                                     int N, int Nz, int S, float* __restrict__ raw,
                                                     int* __restrict__ flags)
{
    __shared__ float tile[G][33];
    const int t = blockIdx.y, g = blockIdx.z, u0 = blockIdx.x * 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float w = __ldg(&cs[t].x) / (float)Nz;
    const float* src = proj + (size_t)t * tilt_stride + (size_t)(y0 + g * G) * row_pitch + u0 + lane;
    for (int q = warp; q < G; q += 8) {
        float v = 0.f;
        if (g * G + q < S && u0 + lane < N) v = __ldg(src + (size_t)q * row_pitch) * w;
        tile[q][lane] = v;
        const bool low = __any_sync(0xffffffffu, v <= kLowValue), special = __any_sync(0xffffffffu, !(fabsf(v) < kSpecial));
        if (lane == 0 && (low || special))
            atomicOr(flags + g * G + q, (low ? kFlagRawLow : 0) | (special ? kFlagRawSpecial : 0));
    }
    __syncthreads();
    float* dst = raw + (((size_t)g * T + t) * N + u0) * G;
    for (int i = threadIdx.x; i < 32 * G; i += 256) {
        const int u = i / G, q = i % G;
        if (u0 + u < N) dst[i] = tile[q][u];
    }
}

// W[g][row][x][G] -> vol[ys][row][x].  Grid (ceil(Nx / 32), Nz, groups).
template <int G>
__global__ void __launch_bounds__(256) k_ungroup_wide(const float* __restrict__ w, float* __restrict__ vol, int Nx,
                                                      int Nz, int S)
{
    __shared__ float tile[G][33];
    const int row = blockIdx.y, g = blockIdx.z, x0 = blockIdx.x * 32;
    const float* src = w + (((size_t)g * Nz + row) * Nx + x0) * G;
    for (int i = threadIdx.x; i < 32 * G; i += 256) {
        const int x = i / G, q = i % G;
        if (x0 + x < Nx) tile[q][x] = __ldcs(src + i);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int q = threadIdx.x >> 5; q < G; q += 8)
        if (g * G + q < S && x0 + lane < Nx)
            vol[((size_t)(g * G + q) * Nz + row) * Nx + x0 + lane] = tile[q][lane];
}

// Group size for a slab of S slices: the cheapest once the last group is filled up.  Time
// per slice against G = 64, measured on 4096 x 64 x 41 and 1024 x 256 x 61
// reconstructions: 1.18 for 32 (fewer slices share a weight and a position), 1.65 for 16.
// From `smallest` on: 16 for a series; a slab of fewer slices also takes 8 (2.6 and 3.2) and 4
// (4.8 and 6.2), so that slab_slices of a few slices costs neither the work nor the memory
// of 16.  Measured (2 iterations of 4096 x 64 x 41 x 1200; four-slice kernels / filled
// up to 16 / now): slabs of 1 slice 377 / 729 / 486 ms, of 4 97 / 182 / 122, of 8 63 / 91 / 65;
// 2048 x 32 x 41 x 600, 3 iterations: of 4 29.2 / - / 27.6, of 8 16.5 / - / 14.3.
inline double wide_cost(int S, int smallest, int* group = nullptr)
{
    const double rate[5] = {1.0, 1.18, 1.65, 2.8, 5.2};
    double best = 1e30;
    for (int k = 0; 64 >> k >= smallest; k++) {
        const int G = 64 >> k;
        const double c = rate[k] * ((S + G - 1) / G * G);
        if (c < best) {
            best = c;
            if (group) *group = G;
        }
    }
    return best;
}
inline int wide_group(int S)
{
    int G = 64;
    wide_cost(S, 4, &G);
    return G;
}
// Slices the workspace holds for slabs of up to S, filled-up groups included (a slab of 64
// slices fewer is no larger, filled up, than one that is not filled up at all).
inline int wide_slices(int S)
{
    int m = S;
    for (int s = std::max(1, S - 63); s <= S; s++) m = std::max(m, (s + wide_group(s) - 1) / wide_group(s) * wide_group(s));
    return m;
}

// V = 4, 2 or 1 values in one access.
template <int V>
using VecOf = std::conditional_t<V == 4, float4, std::conditional_t<V == 2, float2, float>>;
template <int V>
__device__ __forceinline__ void unpack(const VecOf<V>& a, float (&v)[V])
{
    if constexpr (V == 4) { v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; }
    else if constexpr (V == 2) { v[0] = a.x; v[1] = a.y; }
    else v[0] = a;
}
template <int V>
__device__ __forceinline__ VecOf<V> pack(const float (&v)[V])
{
    if constexpr (V == 4) return make_float4(v[0], v[1], v[2], v[3]);
    else if constexpr (V == 2) return make_float2(v[0], v[1]);
    else return v[0];
}

// NS slices of one column in pairs of slices; even: the address of the lane's part of its
// pair's first chunk, odd: of the second (fpw_slice).
template <int NS>
__device__ __forceinline__ void fpw_load(const float* even, const float* odd, float2 (&v)[(NS + 1) / 2])
{
    if constexpr (NS == 2) v[0] = *reinterpret_cast<const float2*>(even);
    if constexpr (NS == 1) v[0] = make_float2(*even, 0.f);
#pragma unroll
    for (int b = 0; b < NS / 4; b++) {
        const float4 a = *reinterpret_cast<const float4*>((b & 1 ? odd : even) + 32 * (b >> 1));
        v[2 * b] = make_float2(a.x, a.y);
        v[2 * b + 1] = make_float2(a.z, a.w);
    }
}

// ---------------------------------------------------------------------------
// Forward projection of tilts [t0, t0 + nt) and residual (GForProj.cu:10-76,
// GDiffProj.cu:7-21).  A warp carries 16 neighbouring rays of one tilt, each thread
// two of them (a pair) for G / 4 slices, and walks the volume rows they cross.
// The samples of a ray that touch volume row Z (at most ceil(2 / cos)) read columns
// that overlap: their bilinear weights are merged into one weight per (ray, column),
// so a pair's window of C = 1 / cos + 2 tan + 3 columns is loaded once for both rays
// and all their samples (three to four column loads a ray and row become two, and the
// 4 / cos multiply-adds of separate samples 2 + 2 tan).  The weights of up to
// FPW_MAX_ROWS rows at a time go through a table of the warp's in shared memory;
// samples and their validity are the reference's (fp_ray_setup), every value is
// FP32, and a column that a ray does not touch has weight zero.
// The window of the warp's rays in a row is one contiguous run of the volume:
// the lane that holds the row's bounds fetches it with one bulk asynchronous copy into a
// ring of rows, ahead of their use.  The ring holds 80 columns, which the window of 16 rays
// exceeds from about 77 degrees on (in volumes wider than that); such tilts go sample by sample,
// and so do those whose pair window exceeds FPW_MAX_COLS (about 84 degrees).  A warp shares nothing with the others of its CTA, so no
// block-wide barrier is needed and short rays leave no one waiting.
// The rows are cut into segments of seg_rows, one warp each: the segments that a ray
// block crosses leave their sums in `part`, and the last of them to finish adds
// them up in order and forms the residual.  Short walks keep the concurrent warps
// of all tilts near one another in z, within what L2 holds of the volume, and give
// small volumes enough warps.
// Grid (ceil(N / FPW_CTA_RAYS) * tilts, segments, groups), the tilts of a ray block
// next to one another.
// ---------------------------------------------------------------------------
struct FpwArgs {
    const float* vol;        // W
    const float* raw;
    float* diff;
    const float2* cs;
    double* rf;              // R-factor sums or null
    int* flags;
    float* part;             // ray sums of the segments [segment][group][nt][N][G]
    int* arrived;            // [group][nt][ray warps]: segments done; zero between launches
    int seg_rows;            // volume rows a warp walks
    int Nx, Nz, T, N, t0, nt;
    int polls;               // limit of a wait for a bulk copy (WIDE_POLLS)
};

constexpr int FPW_THREADS = 128, FPW_WARPS = FPW_THREADS / 32, FPW_CTA_RAYS = FPW_WARPS * FPW_WARP_RAYS;
constexpr int FPW_MAX_STAGES = 4;
// Shared memory of a warp: a ring that holds two rows of its window at 60 degrees, the
// weight table, barriers and window starts.  CTAs per SM as it allows.
template <int G>
struct Fpw {
    static constexpr int NS = G / FPW_LP;
    static constexpr int RING = 80 * G * (int)sizeof(float);
    static constexpr int TABLE = G == 64 ? 5 << 10 : 3 << 10;
    static constexpr int WARP_BYTES = RING + TABLE + 8 * FPW_MAX_STAGES + 8 * FPW_MAX_ROWS * FPW_PAIRS + 4 * FPW_MAX_ROWS;
    static constexpr size_t SMEM = (size_t)FPW_WARPS * WARP_BYTES;
    static constexpr int CTAS = G == 64 ? 2 : G >= 16 ? 4 : 5;   // (G 4 and 8: 2 to 12 % faster than 4 or 6)
    static_assert(WARP_BYTES % 16 == 0, "16-byte aligned regions");
};

// Sums and counts of four slices summed sample by sample.
struct TestedQuad {
    float s[4], n[4];
};

// Samples [lo, hi] of a ray for four slices, one by one (the path of slices that hold empty,
// infinite or NaN voxels).  EMPTY: with the reference's empty test; otherwise, for slices
// without empty voxels, as the four-slice kernel sums them, with no difference of two taps, so
// that a sample between infinite voxels is infinite and not NaN.  One 16-byte load a tap
// serves the four slices, and the taps of FPT samples are in flight together: the walk
// waits on L2, which it reads with little reuse (beside the rings, L1 holds a few KB a warp).
// Measured (forward projections of 2 iterations of 4096 x 64 x 41 x 1200): with a NaN pixel in every
// row 441 ms one slice at a time, 139 ms, the four-slice kernel 80 ms; in one row 39 and 35
// ms (32 ms); in none 13.2 ms (25 ms).
constexpr int FPT = 4;
template <bool EMPTY>
__device__ __noinline__ TestedQuad fpw_quad_tested(const float* v0, int G, int Nx, RayPos r, int lo, int hi)
{
    TestedQuad o{};
    const ptrdiff_t row = (ptrdiff_t)G * Nx;
    for (int i0 = lo; i0 <= hi; i0 += FPT) {
        float4 f[FPT][4];
        float wx[FPT], wz[FPT];
#pragma unroll
        for (int k = 0; k < FPT; k++) {
            const int i = min(i0 + k, hi);   // (a sample past the last one is not added)
            const float fX = r.x(i), fZ = r.z(i);
            const int iX = (int)fX, iZ = (int)fZ;
            const float* p = v0 + (ptrdiff_t)G * iX - iZ * row;
            wx[k] = fX - (float)iX;
            wz[k] = fZ - (float)iZ;
            f[k][0] = __ldg(reinterpret_cast<const float4*>(p));
            f[k][1] = __ldg(reinterpret_cast<const float4*>(p + G));
            f[k][2] = __ldg(reinterpret_cast<const float4*>(p - row));
            f[k][3] = __ldg(reinterpret_cast<const float4*>(p - row + G));
        }
#pragma unroll
        for (int k = 0; k < FPT; k++) {
            if (i0 + k > hi) break;
            const float ux = 1.f - wx[k], uz = 1.f - wz[k];
            const float w00 = ux * uz, w10 = wx[k] * uz, w01 = ux * wz[k], w11 = wx[k] * wz[k];
            auto add = [&](int q, float a00, float a10, float a01, float a11) {
                if constexpr (EMPTY) {
                    const float val = bilerp(a00, a10, a01, a11, wx[k], wz[k]);
                    const bool in = !(val < kSentinelTest);   // a NaN sample is summed
                    o.s[q] = in ? o.s[q] + val : o.s[q];
                    o.n[q] += in ? 1.f : 0.f;
                } else {
                    o.s[q] = __fmaf_rn(w11, a11, __fmaf_rn(w01, a01, __fmaf_rn(w10, a10, __fmaf_rn(w00, a00, o.s[q]))));
                    o.n[q] += 1.f;
                }
            };
            add(0, f[k][0].x, f[k][1].x, f[k][2].x, f[k][3].x);
            add(1, f[k][0].y, f[k][1].y, f[k][2].y, f[k][3].y);
            add(2, f[k][0].z, f[k][1].z, f[k][2].z, f[k][3].z);
            add(3, f[k][0].w, f[k][1].w, f[k][2].w, f[k][3].w);
        }
    }
    return o;
}

__device__ __forceinline__ void bulk_row_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// The warp's rays for the quads (four slices) of a group in `quads`, sample by sample, into
// res[ray][half][quad].  The four lanes of a pair share out its rays, halves of a ray and quads, so that
// all work where one slice of a group is tested, and neighbouring lanes take neighbouring
// quads where many are.
template <int G>
__device__ __noinline__ void fpw_rays_tested(const float* v00, const int* flags, int Nx, RayPos ray, int rlo, int rhi,
                                             unsigned quads, TestedQuad* res)
{
    const int lane = threadIdx.x & 31, lp = lane % FPW_LP, pair = lane / FPW_LP, nq = __popc(quads);
    for (int k = lp; k < FPW_RAYS * 2 * nq; k += FPW_LP) {   // (as many rounds for every lane)
        const int quad = __fns(quads, 0, k % nq + 1), r = k / nq >> 1, half = k / nq & 1, src = FPW_RAYS * pair + r;
        RayPos rp = ray;
        rp.tx = __shfl_sync(0xffffffffu, ray.tx, src);
        const int lo = __shfl_sync(0xffffffffu, rlo, src), hi = __shfl_sync(0xffffffffu, rhi, src), mid = (lo + hi) >> 1;
        const int4 f4 = __ldg(reinterpret_cast<const int4*>(flags + 4 * quad));
        const int f[4] = {f4.x, f4.y, f4.z, f4.w};
        const int i0 = half ? mid + 1 : lo, i1 = half ? hi : mid;
        bool empty = false, plain = false;   // slices of the quad that may and that do not hold empty voxels
#pragma unroll
        for (int q = 0; q < 4; q++) {
            empty |= (f[q] & kFlagVolEmpty) != 0;
            plain |= !(f[q] & kFlagVolEmpty) && (f[q] & (kFlagRawSpecial | kFlagVolSpecial));
        }
        TestedQuad& o = res[(src * 2 + half) * (G / 4) + quad];
        if (plain) o = fpw_quad_tested<false>(v00 + 4 * quad, G, Nx, rp, i0, i1);
        if (empty) {
            const TestedQuad t = fpw_quad_tested<true>(v00 + 4 * quad, G, Nx, rp, i0, i1);
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (f[q] & kFlagVolEmpty) { o.s[q] = t.s[q]; o.n[q] = t.n[q]; }
        }
    }
    __syncwarp();
}

// Samples [lo, hi] of a ray for a thread's slices, one by one, into sum (steep tilts).  Two samples at a
// time: their taps come from L2 (1 subset of tilts to +-80 degrees, 1024 x 64 x 61 x 300, 5 iterations: 9.0
// ms one at a time, 7.7; the four-slice kernels 8.4).  Not in line, where it takes registers from
// the row loop (10 forward projections of 4096 x 64 x 1200 without steep tilts: 13.8 ms in line, 13.2).
template <int G>
__device__ __noinline__ void fpw_ray_steep(const float* v00, int Nx, RayPos ray, int lo, int hi, int even, int odd,
                                           float2* sum)
{
    constexpr int NS = Fpw<G>::NS, NP = (NS + 1) / 2;
    float2 acc[NP];
#pragma unroll
    for (int q = 0; q < NP; q++) acc[q] = make_float2(0.f, 0.f);
#pragma unroll 2
    for (int i = lo; i <= hi; i++) {
        const float fX = ray.x(i), fZ = ray.z(i);
        const int iX = (int)fX, iZ = (int)fZ;
        const float wx = fX - (float)iX, wz = fZ - (float)iZ, ux = 1.f - wx, uz = 1.f - wz;
        const float* v = v00 + ((ptrdiff_t)iX - (ptrdiff_t)iZ * Nx) * G;
        const float wt[4] = {ux * uz, wx * uz, ux * wz, wx * wz};
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const float* vm = v + (m & 1) * G - (ptrdiff_t)(m >> 1) * Nx * G;
            float2 a[NP];
            fpw_load<NS>(vm + even, vm + odd, a);
            const float2 w2 = make_float2(wt[m], wt[m]);
#pragma unroll
            for (int q = 0; q < NP; q++) fma2(acc[q], w2, a[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < NP; q++) sum[q] = acc[q];
}

template <int G>
__global__ void __launch_bounds__(FPW_THREADS, Fpw<G>::CTAS) k_fp_wide(FpwArgs p)
{
    using F = Fpw<G>;
    constexpr int NS = F::NS, RW = FPW_WARP_RAYS;
    constexpr int NP = (NS + 1) / 2, V = NS < 4 ? NS : 4;   // pairs of slices a thread sums; slices in one access
    extern __shared__ float4 wsm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    char* region = reinterpret_cast<char*>(wsm) + warp * F::WARP_BYTES;
    float2* tab = reinterpret_cast<float2*>(region + F::RING);                        // [rows][FPW_PAIRS][CP]
    uint64_t* mbar = reinterpret_cast<uint64_t*>(region + F::RING + F::TABLE);
    int* s_k0 = reinterpret_cast<int*>(mbar + FPW_MAX_STAGES);                        // [FPW_MAX_ROWS][FPW_PAIRS] first column of a window
    int* s_off = s_k0 + FPW_MAX_ROWS * FPW_PAIRS;                                     // and its place in the row fetched
    int* s_cnt = s_off + FPW_MAX_ROWS * FPW_PAIRS;                                    // [FPW_MAX_ROWS] columns of the row's windows
    const int tb = blockIdx.x % p.nt, u0 = (blockIdx.x / p.nt) * FPW_CTA_RAYS + warp * RW, g = blockIdx.z;
    const int t = p.t0 + tb, Nx = p.Nx, Nz = p.Nz, N = p.N;
    if (u0 >= N) return;
    const float2 cc = __ldg(&p.cs[t]);
    const float c = cc.x, s = cc.y, inv_c = 1.f / c;
    const int L = (int)((float)Nz / c + 1.5f);
    const float halfL = (float)L * 0.5f, tz = (float)Nz * 0.5f;
    auto zpos = [&](int i) { return __fmaf_rn((float)i - halfL, c, tz); };

    // ray lane % RW: position and in-volume samples
    RayPos ray;
    int rlo, rhi;
    fp_ray_setup(min(u0 + lane % RW, N - 1), N, Nx, Nz, c, s, ray, rlo, rhi);
    if (u0 + lane % RW >= N) { rlo = 1; rhi = 0; }
    // rows the warp's rays cross, and those of this segment
    int z0 = __reduce_min_sync(0xffffffffu, rlo <= rhi ? (int)zpos(rlo) : INT_MAX);
    int z1 = __reduce_max_sync(0xffffffffu, rlo <= rhi ? (int)zpos(rhi) + 1 : -1);

    const int lp = lane % FPW_LP, pair = lane / FPW_LP;
    const int even = fpw_slice<NS>(lp, pair, 0), odd = fpw_slice<NS>(lp, pair, 1);
    float2 acc[FPW_RAYS][NP];
#pragma unroll
    for (int r = 0; r < FPW_RAYS; r++)
#pragma unroll
        for (int q = 0; q < NP; q++) acc[r][q] = make_float2(0.f, 0.f);

    const size_t gvol = (size_t)g * Nz * Nx * G;
    const float* v00 = p.vol + gvol + (size_t)(Nz - 1) * Nx * G;   // voxel (0, 0)
    const int C = fpw_cols(FPW_RAYS - 1, c, s, N, Nx), W = min(Nx, fpw_cols(RW - 1, c, s, N, Nx) + 2);
    const uint32_t row_bytes = (uint32_t)(W * G * sizeof(float));
    const bool blocked = C <= FPW_MAX_COLS && row_bytes <= F::RING;
    // segments that take part: those the rays cross (one if none)
    const int seg = blockIdx.y, seg0 = z1 < z0 ? 0 : z0 / p.seg_rows;
    const int nseg = z1 < z0 ? 1 : z1 / p.seg_rows - seg0 + 1;
    if (seg < seg0 || seg >= seg0 + nseg) return;
    z0 = max(z0, seg * p.seg_rows);
    z1 = min(z1, (seg + 1) * p.seg_rows - 1);
    if (blocked && z1 >= z0) {
        const int ns = min(FPW_MAX_STAGES, (int)(F::RING / row_bytes));
        if (lane == 0) {
            for (int k = 0; k < ns; k++)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar + k)) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        // (columns past a row's window are read with weight zero: they must hold finite values)
        for (int e = lane; e < F::RING / 16; e += 32) reinterpret_cast<float4*>(region)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        const int CP = C | 1;   // odd pitch: the table's stores spread over the banks
        const int rows = min(FPW_MAX_ROWS, F::TABLE / (8 * FPW_PAIRS * CP));
        // in a row of samples [ia, ib], the first column of ray tx, clamped so that n columns from it lie in
        // the volume, and the last one
        auto left = [&](float tx, int ia, int ib, int n) {
            const float xl = __fmaf_rn(-((float)(s >= 0.f ? ib : ia) - halfL), s, tx);
            return (int)fminf(fmaxf(floorf(xl), 0.f), (float)(Nx - n));
        };
        auto right = [&](float tx, int ia, int ib) {
            const float xr = __fmaf_rn(-((float)(s >= 0.f ? ia : ib) - halfL), s, tx);
            return (int)fminf(fmaxf(floorf(xr) + 1.f, 0.f), (float)(Nx - 1));
        };
        // lane j < rows: the samples [ia, ib] with z in [Z - 1, Z + 1) of row Z = zc + j, the warp's
        // window there, its address and bytes
        const float tx0 = __shfl_sync(0xffffffffu, ray.tx, 0), tx1 = __shfl_sync(0xffffffffu, ray.tx, RW - 1);
        struct Row {
            int ia, ib, kw;
            uint32_t bytes;
            const float* src;
        };
        auto row_info = [&](int zc) {
            Row r;
            const float Z1 = (float)(zc + lane - 1);
            r.ia = first_true(0, L - 1, est_index(ceilf(__fmaf_rn(Z1 - tz, inv_c, halfL))), [&](int i) { return zpos(i) >= Z1; });
            r.ib = __shfl_down_sync(0xffffffffu, r.ia, 2) - 1;
            r.kw = left(tx0, r.ia, r.ib, W);
            r.src = v00 + ((ptrdiff_t)r.kw - (ptrdiff_t)(zc + lane) * Nx) * G;
            r.bytes = (uint32_t)(min(max(right(tx1, r.ia, r.ib) - r.kw + 1, 1), W) * G * sizeof(float));
            return r;
        };
        Row row = row_info(z0), next{};   // this chunk's rows and the next one's
        const uint32_t ring0 = smem_u32(region), bar0 = smem_u32(mbar);
        const int lead = min(ns, rows);   // rows fetched ahead: within this chunk and the next
        int sf = 0;                       // stage the next row goes to
        auto fetch = [&](bool mine, const float* src, uint32_t bytes) {
            if (mine) bulk_row_copy(ring0 + sf * row_bytes, src, bytes, bar0 + 8 * sf);
            sf = sf + 1 == ns ? 0 : sf + 1;
        };
        for (int k = 0; k < lead; k++) fetch(lane == k && z0 + k <= z1, row.src, row.bytes);
        int sc = 0;                       // stage of the row in use
        uint32_t phase = 0;
        bool ok = true;
        const int rk = lane % RW, rp = rk / FPW_RAYS, half = lane / RW;
        for (int zc = z0; zc <= z1; zc += rows) {
            const int nr = min(rows, z1 - zc + 1);
            next = row_info(zc + rows);
            // the pairs' windows
            for (int e0 = 0; e0 < nr * FPW_PAIRS; e0 += 32) {
                const int e = e0 + lane, j = min(e / FPW_PAIRS, rows - 1), q = e % FPW_PAIRS;
                const int a = __shfl_sync(0xffffffffu, row.ia, j), b = __shfl_sync(0xffffffffu, row.ib, j);
                const int kwj = __shfl_sync(0xffffffffu, row.kw, j);
                const int k0 = left(__shfl_sync(0xffffffffu, ray.tx, FPW_RAYS * q), a, b, C);
                int n = min(right(__shfl_sync(0xffffffffu, ray.tx, FPW_RAYS * q + FPW_RAYS - 1), a, b) - k0 + 1, C);
#pragma unroll
                for (int o = 1; o < FPW_PAIRS; o <<= 1) n = max(n, __shfl_xor_sync(0xffffffffu, n, o));
                if (e < nr * FPW_PAIRS) {
                    if (q == 0) s_cnt[j] = n;
                    s_k0[e] = k0;
                    s_off[e] = (k0 - kwj) * G;
                }
            }
            for (int e = lane; e < nr * FPW_PAIRS * CP / 2; e += 32)
                reinterpret_cast<float4*>(tab)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            __syncwarp();
            // weights: the chunk's samples in turn, every lane its ray; a sample adds to rows iZ and iZ + 1
            // (the two halves of the warp)
            const int i1 = __shfl_sync(0xffffffffu, row.ib, nr - 1);
            int i = __shfl_sync(0xffffffffu, row.ia, 0);
            float fd = (float)i - halfL;   // (exact, as are its increments)
            for (; i <= i1; i++, fd += 1.f) {
                const float fX = __fmaf_rn(-fd, s, ray.tx), fZ = __fmaf_rn(fd, c, tz);
                const float tX = __fadd_rd(fX, kMagic), zf = floorf(fZ);
                const int j = (int)zf + half - zc;
                if ((unsigned)j < (unsigned)nr && i >= rlo && i <= rhi) {
                    const float wx = fX - (tX - kMagic), wz = fZ - zf, m = half ? wz : 1.f - wz;
                    const int e = __float_as_int(tX) - kMagicBits - s_k0[j * FPW_PAIRS + rp];
                    float* w = reinterpret_cast<float*>(tab + (j * FPW_PAIRS + rp) * CP + e) + rk % FPW_RAYS;
                    if ((unsigned)e < (unsigned)(C - 1)) {
                        w[0] = __fmaf_rn(1.f - wx, m, w[0]);
                        w[2] = __fmaf_rn(wx, m, w[2]);
                    }
                }
                __syncwarp();
            }
            int j = 0;
            for (; j < nr; j++) {
                ok = mbar_wait(bar0 + 8 * sc, phase, p.polls);
                if (!__all_sync(0xffffffffu, ok)) break;
                const float* v = reinterpret_cast<const float*>(region + sc * row_bytes) + s_off[j * FPW_PAIRS + pair];
                const float2* w = tab + (j * FPW_PAIRS + pair) * CP;
                const float *ve = v + even, *vo = v + odd;
                const int cols = s_cnt[j];
                // (the next column is loaded ahead; past the last one it reads on within the warp's region)
                float2 wt = w[0], a[NP];
                fpw_load<NS>(ve, vo, a);
#pragma unroll 2
                for (int e = 0; e < cols; e++) {
                    ve += G;
                    vo += G;
                    const float2 wn = w[e + 1];
                    float2 an[NP];
                    fpw_load<NS>(ve, vo, an);
                    const float2 w0 = make_float2(wt.x, wt.x), w1 = make_float2(wt.y, wt.y);
#pragma unroll
                    for (int q = 0; q < NP; q++) {
                        fma2(acc[0][q], w0, a[q]);
                        fma2(acc[1][q], w1, a[q]);
                    }
                    wt = wn;
#pragma unroll
                    for (int q = 0; q < NP; q++) a[q] = an[q];
                }
                __syncwarp();   // the stage is free: fetch the row `lead` ahead into the next free stage
                const int jf = j + lead;
                const bool in = jf < rows;
                fetch(lane == (in ? jf : jf - rows) && zc + jf <= z1, in ? row.src : next.src,
                      in ? row.bytes : next.bytes);
                if (++sc == ns) { sc = 0; phase ^= 1; }
            }
            if (!__all_sync(0xffffffffu, ok)) {
                // a copy did not arrive: the run is flagged.  Row zc + j and the rows fetched ahead of it are
                // in flight, in the stages from sc on, the parity changing where the ring starts over: wait
                // for each (bounded), so that none lands in another CTA's memory.  The warp's sums become
                // zero and it goes on, so that the segments of its rays still count up to their last one
                for (int k = 0; k < lead && zc + j + k <= z1; k++) {
                    const int sg = sc + k;
                    mbar_wait(bar0 + 8 * (sg < ns ? sg : sg - ns), sg < ns ? phase : phase ^ 1, WIDE_POLLS);
                }
                if (lane == 0) atomicOr(p.flags + g * G, kFlagStageTimeout);
#pragma unroll
                for (int r = 0; r < FPW_RAYS; r++)
#pragma unroll
                    for (int q = 0; q < NP; q++) acc[r][q] = make_float2(0.f, 0.f);
                break;
            }
            row = next;
        }
    } else if (!blocked) {
        // steep tilts: sample by sample, a segment the samples whose lower row it holds
        const float Z0 = (float)(seg * p.seg_rows), Z1 = (float)((seg + 1) * p.seg_rows);
        const int slo = first_true(rlo, rhi, est_index(ceilf(__fmaf_rn(Z0 - tz, inv_c, halfL))), [&](int i) { return zpos(i) >= Z0; });
        const int shi = first_true(slo, rhi, est_index(ceilf(__fmaf_rn(Z1 - tz, inv_c, halfL))), [&](int i) { return zpos(i) >= Z1; }) - 1;
#pragma unroll
        for (int r = 0; r < FPW_RAYS; r++) {
            const int k = FPW_RAYS * pair + r;
            RayPos rp = ray;
            rp.tx = __shfl_sync(0xffffffffu, ray.tx, k);
            const int lo = __shfl_sync(0xffffffffu, slo, k), hi = __shfl_sync(0xffffffffu, shi, k);
            float2 sum[NP];
            fpw_ray_steep<G>(v00, Nx, rp, lo, hi, even, odd, sum);
#pragma unroll
            for (int q = 0; q < NP; q++) acc[r][q] = sum[q];
        }
    }

    // the sums of the segments, added up by the last one to arrive
    if (nseg > 1) {
        const int groups = gridDim.z;
        const size_t pitch = (size_t)groups * p.nt * N * G;
        float* mine = p.part + (((size_t)g * p.nt + tb) * N + u0) * G;
        auto at = [&](int sg, int r, int b) {
            return reinterpret_cast<VecOf<V>*>(mine + sg * pitch + (size_t)(FPW_RAYS * pair + r) * G + fpw_slice<NS>(lp, pair, b));
        };
#pragma unroll
        for (int r = 0; r < FPW_RAYS; r++)
            if (u0 + FPW_RAYS * pair + r < N) {
#pragma unroll
                for (int b = 0; b < NS / V; b++) {
                    float v[V];
#pragma unroll
                    for (int q = 0; q < V; q++) v[q] = q & 1 ? acc[r][(V * b + q) / 2].y : acc[r][(V * b + q) / 2].x;
                    *at(seg, r, b) = pack<V>(v);
                }
            }
        __threadfence();
        __syncwarp();
        int last = 0;
        if (lane == 0) {
            int* count = p.arrived + ((size_t)g * p.nt + tb) * ((N + RW - 1) / RW) + u0 / RW;
            last = atomicAdd(count, 1) == nseg - 1;
            if (last) *count = 0;
        }
        if (!__shfl_sync(0xffffffffu, last, 0)) return;
        __threadfence();
#pragma unroll
        for (int r = 0; r < FPW_RAYS; r++)
#pragma unroll
            for (int q = 0; q < NP; q++) acc[r][q] = make_float2(0.f, 0.f);
#pragma unroll 2
        for (int sg = seg0; sg < seg0 + nseg; sg++)
#pragma unroll
            for (int r = 0; r < FPW_RAYS; r++)
                if (u0 + FPW_RAYS * pair + r < N) {
#pragma unroll
                    for (int b = 0; b < NS / V; b++) {
                        float v[V];
                        unpack<V>(__ldcg(at(sg, r, b)), v);
#pragma unroll
                        for (int q = 0; q < V; q++) {
                            float2& s2 = acc[r][(V * b + q) / 2];
                            if (q & 1) s2.y += v[q];
                            else s2.x += v[q];
                        }
                    }
                }
    }

    // mean along the ray, residual and R-factor sums
    float ad = 0.f, ar = 0.f;
    unsigned tested = 0, quads = 0;   // slices summed sample by sample; quads of the group that hold some
    int ys[NS / V];
#pragma unroll
    for (int k = 0; k < NS / V; k++) {
        ys[k] = g * G + fpw_slice<NS>(lp, pair, k);
        float fl[V];
        unpack<V>(__ldg(reinterpret_cast<const VecOf<V>*>(p.flags + ys[k])), fl);
#pragma unroll
        for (int q = 0; q < V; q++)
            if (__float_as_int(fl[q]) & (kFlagVolEmpty | kFlagRawSpecial | kFlagVolSpecial)) {
                tested |= 1u << (V * k + q);
                quads |= 1u << ((ys[k] - g * G) / 4);
            }
    }
    quads = __reduce_or_sync(0xffffffffu, quads);
    TestedQuad* res = reinterpret_cast<TestedQuad*>(region);   // (the ring: no copy is in flight any more)
    static_assert(RW * 2 * (G / 4) * sizeof(TestedQuad) <= F::RING, "sums of the tested slices");
    if (quads) fpw_rays_tested<G>(v00, p.flags + g * G, Nx, ray, rlo, rhi, quads, res);
#pragma unroll
    for (int r = 0; r < FPW_RAYS; r++) {
        const int k = FPW_RAYS * pair + r, u = u0 + k;
        const int lo = __shfl_sync(0xffffffffu, rlo, k), hi = __shfl_sync(0xffffffffu, rhi, k);
        if (u >= N) continue;
        const float n = (float)max(hi - lo + 1, 0);
#pragma unroll
        for (int b = 0; b < NS / V; b++) {
            const size_t o = (((size_t)g * p.T + t) * N + u) * G + (ys[b] - g * G);
            float rw[V], d[V];
            unpack<V>(*reinterpret_cast<const VecOf<V>*>(p.raw + o), rw);
            const TestedQuad* tq = res + 2 * k * (G / 4) + (ys[b] - g * G) / 4;
#pragma unroll
            for (int q = 0; q < V; q++) {
                float sum = q & 1 ? acc[r][(V * b + q) / 2].y : acc[r][(V * b + q) / 2].x, cnt = n;
                if ((tested >> (V * b + q)) & 1) {
                    const int e = V == 4 ? q : (ys[b] + q) & 3;
                    sum = tq[0].s[e] + tq[G / 4].s[e];
                    cnt = tq[0].n[e] + tq[G / 4].n[e];
                }
                const float fp = cnt <= 0.f ? kSentinelValue : sum / cnt;
                d[q] = 0.f;
                if (!(fp < kSentinelTest) && !(rw[q] < kSentinelTest)) {
                    d[q] = rw[q] - fp;
                    ad += fabsf(d[q]);
                    ar += fabsf(rw[q]);
                    if (d[q] <= kLowValue) atomicOr(p.flags + ys[b] + q, kFlagDiffLow);
                    if (!(fabsf(d[q]) < kSpecial)) atomicOr(p.flags + ys[b] + q, kFlagDiffSpecial);
                }
            }
            *reinterpret_cast<VecOf<V>*>(p.diff + o) = pack<V>(d);
        }
    }
    if (p.rf) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ad += __shfl_xor_sync(0xffffffffu, ad, o);
            ar += __shfl_xor_sync(0xffffffffu, ar, o);
        }
        if (lane == 0) {
            atomicAdd(p.rf, (double)ad);
            atomicAdd(p.rf + 1, (double)ar);
        }
    }
}

// ---------------------------------------------------------------------------
// Back-projection and update (GBackProj.cu:12-60, bSart) of tilts [t0, t1).
// A thread carries a block of 2 x 2 voxels for NS slices: their detector
// positions lie within cos + |sin| <= 1.42 of one another, so four consecutive
// samples hold all their taps, and voxel v takes sample k with the hat weight
// max(0, 1 - |x_v - k|) — the lerp's own two weights, zero elsewhere.  Four loads
// of NS slices serve four voxels (eight one voxel at a time).  The CTA's windows
// (16 c + 8 |s| + 4 samples a tilt) come to shared memory by bulk copies, three tilts
// ahead (below).  Bound by the multiply-adds: pipe 64 % busy, issue 67 %, shared-memory wavefronts
// 54 %; the volume read and written once is 47 % of its time at the copy rate.
// Positions are the reference's FP32 ones and sums run in its (tilt) order.
// Grid (x tiles, z tiles, groups).
// ---------------------------------------------------------------------------
struct BpwArgs {
    const float* sino;       // raw or residual, [groups][T][N][G]
    const float2* cs;
    float* vol;              // W
    int* flags;
    int T, N, t0, t1, Nx, Nz, low_bit;
    int polls;               // limit of a wait for a bulk copy (WIDE_POLLS)
    float relax;
};

template <int LP>
__host__ __device__ constexpr int bpw_tile_x() { return 4 * (32 / LP); }
constexpr int BPW_TILE_Z = 8;

// One voxel of four slices, every sample tested as the reference does; a tap is one 16-byte
// load.  Measured (back-projections of 2 iterations of 4096 x 64 x 41 x 1200 with a missing pixel
// in every row): 54.6 ms one slice at a time, 17.7 ms; the four-slice kernel 19.8 ms.
__device__ __noinline__ TestedQuad bpw_quad_tested(const float* row0, size_t tilt_pitch, int G, int N, const float2* cs,
                                                   int t0, int t1, float fX, float fZ, float cent)
{
    TestedQuad o{};
    const float endX = (float)(N - 2);
#pragma unroll 4
    for (int t = t0; t < t1; t++) {
        const float2 c = __ldg(&cs[t]);
        const float xp = bp_xp<0>(fX, __fmul_rn(fZ, c.y), c.x, cent);
        const bool in = xp >= 0.f && xp <= endX;
        const int i = in ? (int)xp : 0;
        const float fr = __fsub_rn(xp, (float)i), om = __fsub_rn(1.f, fr);
        const float* p = row0 + (size_t)t * tilt_pitch + (size_t)i * G;
        const float4 f0 = __ldg(reinterpret_cast<const float4*>(p)), f1 = __ldg(reinterpret_cast<const float4*>(p + G));
        const float a0[4] = {f0.x, f0.y, f0.z, f0.w}, a1[4] = {f1.x, f1.y, f1.z, f1.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float v = __fmaf_rn(a0[q], om, __fmul_rn(a1[q], fr));
            if (!in || v <= kSentinelTest) continue;   // a NaN sample is summed
            o.s[q] = __fadd_rn(o.s[q], v);
            o.n[q] += 1.f;
        }
    }
    return o;
}

// Staging of a tile, all by bulk asynchronous copies: the sinogram windows of
// two chunks of BPW_CHUNK tilts (each window one contiguous run), and the old
// volume rows of the tile, which arrive while the tilts are summed.
constexpr int BPW_CHUNK = 3;
template <int LP>
__host__ __device__ constexpr int bpw_window() { return LP == 8 ? 22 : LP == 4 ? 38 : LP == 2 ? 70 : 134; }   // |(TX - 1, TZ - 1)| + 6 samples
template <int LP, int NS>
__host__ __device__ constexpr size_t bpw_smem()
{
    return sizeof(float) * LP * NS * ((size_t)2 * BPW_CHUNK * bpw_window<LP>() + bpw_tile_x<LP>() * BPW_TILE_Z) + 64;
}

// The value of a voxel after an update to y, with the flags of a value that is not ordinary (set once:
// where a whole slice becomes empty, one atomic per voxel would wait for all others).
__device__ __forceinline__ float bpw_value(const BpwArgs& p, int slice, float y)
{
    if (!(y > kSentinelTest && y < kSpecial)) {
        const int bit = y > kSentinelTest ? kFlagVolSpecial : kFlagVolEmpty;
        if (!(*reinterpret_cast<volatile int*>(p.flags + slice) & bit)) atomicOr(p.flags + slice, bit);
    }
    return y > kSentinelTest ? fmaxf(y, 0.f) : kSentinelValue;
}

// The update of the slices in `bits`-flagged quads (four slices) of the group, sample by
// sample.  The LP lanes of a block of 2 x 2 voxels share out its voxels and the quads,
// neighbouring lanes neighbouring quads.  A pass of its own: beside the untested update it
// would cost that one registers.
template <int LP, int NS>
__device__ __noinline__ void bpw_update_tested(const BpwArgs& p, const float* tile, int X, int Z, int bits, unsigned quads)
{
    constexpr int G = LP * NS, TX = bpw_tile_x<LP>(), TZ = BPW_TILE_Z;
    const int g = blockIdx.z, X0 = blockIdx.x * TX, Z0 = blockIdx.y * TZ, nq = __popc(quads);
    const float cent = (float)p.N / 2.0f, hx = (float)p.Nx * 0.5f, hz = (float)p.Nz * 0.5f;
    const size_t tilt_pitch = (size_t)p.N * G;
    for (int k = threadIdx.x % LP; k < 4 * nq; k += LP) {
        const int sl = 4 * __fns(quads, 0, k % nq + 1), v = k / nq, x = X + (v & 1), z = Z + (v >> 1);
        if (x >= p.Nx || z >= p.Nz) continue;
        const TestedQuad t = bpw_quad_tested(p.sino + (size_t)g * p.T * tilt_pitch + sl, tilt_pitch, G, p.N, p.cs, p.t0,
                                             p.t1, (float)x - hx, (float)z - hz, cent);
        const int4 f4 = __ldg(reinterpret_cast<const int4*>(p.flags + g * G + sl));
        const int f[4] = {f4.x, f4.y, f4.z, f4.w};
        const float4 o4 = *reinterpret_cast<const float4*>(tile + ((z - Z0) * TX + (x - X0)) * G + sl);
        const float old[4] = {o4.x, o4.y, o4.z, o4.w};
        float* dst = p.vol + (((size_t)g * p.Nz + (p.Nz - 1 - z)) * p.Nx + x) * G + sl;
#pragma unroll
        for (int q = 0; q < 4; q++)
            if ((f[q] & bits) && t.n[q] > 0.f)
                dst[q] = bpw_value(p, g * G + sl + q, __fmaf_rn(t.s[q], __fdiv_rn(p.relax, t.n[q]), old[q]));
    }
}

template <int LP, int NS>
__global__ void __launch_bounds__(WIDE_THREADS, 3) k_bp_wide(const __grid_constant__ BpwArgs p)
{
    constexpr int G = LP * NS, TX = bpw_tile_x<LP>(), TZ = BPW_TILE_Z;
    extern __shared__ float4 wsm[];
    float* win = reinterpret_cast<float*>(wsm);                                 // [2][BPW_CHUNK][window][G]
    float* tile = win + 2 * BPW_CHUNK * bpw_window<LP>() * G;                   // [TZ][TX][G]
    uint64_t* mbar = reinterpret_cast<uint64_t*>(tile + TX * TZ * G);           // [3]: the two chunks, the tile
    int* s_kw = reinterpret_cast<int*>(mbar + 3);                               // [2][BPW_CHUNK] window starts
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = blockIdx.z;
    const int lp = lane % LP;
    const int X0 = blockIdx.x * TX, Z0 = blockIdx.y * TZ;
    const int X = X0 + 2 * ((warp & 1) * (32 / LP) + lane / LP), Z = Z0 + 2 * (warp >> 1);
    const int N = p.N, Nx = p.Nx, Nz = p.Nz;
    const float cent = (float)N / 2.0f, endX = (float)(N - 2);
    const float hx = (float)Nx * 0.5f, hz = (float)Nz * 0.5f;
    const float fX0 = (float)X - hx, fX1 = (float)(X + 1) - hx;
    const float fZ0 = (float)Z - hz, fZ1 = (float)(Z + 1) - hz;
    const float kmax = (float)(N - 4);
    const int WN = min(N, bpw_window<LP>());   // samples of a window
    const size_t tilt_pitch = (size_t)N * G;
    const float* gsino = p.sino + (size_t)g * p.T * tilt_pitch;

    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(BPW_CHUNK) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar + 1)), "r"(BPW_CHUNK) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar + 2)), "r"(TZ) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // threads [0, BPW_CHUNK): the window of tilt tc + tid into buffer b
    auto fetch = [&](int tc, int b) {
        if (tid >= BPW_CHUNK) return;
        const uint32_t bar = smem_u32(mbar + b);
        int kw = -1;   // no sample of the tile on the detector
        if (tc + tid < p.t1) {
            const float2 c = __ldg(&p.cs[tc + tid]);
            const float za = __fmul_rn((float)(c.y >= 0.f ? Z0 : Z0 + TZ - 1) - hz, c.y);
            const float zb = __fmul_rn((float)(c.y >= 0.f ? Z0 + TZ - 1 : Z0) - hz, c.y);
            const float lo = bp_xp<0>((float)X0 - hx, za, c.x, cent), hi = bp_xp<0>((float)(X0 + TX - 1) - hx, zb, c.x, cent);
            if (hi >= 0.f && lo <= endX) kw = (int)fminf(fmaxf(floorf(lo), 0.f), (float)(N - WN));
        }
        s_kw[b * BPW_CHUNK + tid] = kw;
        if (kw >= 0)
            bulk_row_copy(smem_u32(win + (b * BPW_CHUNK + tid) * bpw_window<LP>() * G),
                          gsino + (size_t)(tc + tid) * tilt_pitch + (size_t)kw * G, (uint32_t)(WN * G * sizeof(float)), bar);
        else
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
    };
    fetch(p.t0, 0);
    fetch(p.t0 + BPW_CHUNK, 1);
    const int nx = min(TX, Nx - X0);
    if (warp == 1 && lane < TZ) {   // row Z0 + lane of the old tile
        if (Z0 + lane < Nz)
            bulk_row_copy(smem_u32(tile + lane * TX * G), p.vol + (((size_t)g * Nz + (Nz - 1 - Z0 - lane)) * Nx + X0) * G,
                          (uint32_t)(nx * G * sizeof(float)), smem_u32(mbar + 2));
        else
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar + 2)) : "memory");
    }
    __syncthreads();   // s_kw

    float2 acc[4][NS / 2];   // voxel 2 dz + dx
    int cnt[4];
#pragma unroll
    for (int v = 0; v < 4; v++) {
        cnt[v] = 0;
#pragma unroll
        for (int q = 0; q < NS / 2; q++) acc[v][q] = make_float2(0.f, 0.f);
    }
    bool ok = true;
    uint32_t phase = 0;
    for (int tc = p.t0, b = 0; tc < p.t1; tc += BPW_CHUNK) {
        if (ok && !mbar_wait(smem_u32(mbar + b), phase, p.polls)) {
            // a window did not arrive: wait (bounded) for this chunk's copies and, where there is
            // a next chunk, its own, which are in flight too (buffer 0 of it is a phase on)
            ok = false;
            mbar_wait(smem_u32(mbar + b), phase, WIDE_POLLS);
            if (tc + BPW_CHUNK < p.t1) mbar_wait(smem_u32(mbar + (b ^ 1)), b ? phase ^ 1 : phase, WIDE_POLLS);
        }
        const int nc = min(BPW_CHUNK, p.t1 - tc);
        for (int j = 0; j < nc; j++) {
            const int kw = s_kw[b * BPW_CHUNK + j];
            if (kw < 0) continue;
            const float2 c = __ldg(&p.cs[tc + j]);
            const float s0 = __fmul_rn(fZ0, c.y), s1 = __fmul_rn(fZ1, c.y);
            const float xp[4] = {bp_xp<0>(fX0, s0, c.x, cent), bp_xp<0>(fX1, s0, c.x, cent),
                                 bp_xp<0>(fX0, s1, c.x, cent), bp_xp<0>(fX1, s1, c.x, cent)};
            const float lo = c.y >= 0.f ? xp[0] : xp[2], hi = c.y >= 0.f ? xp[3] : xp[1];
            // four samples from kf hold every tap of the block; x[v] relative to them,
            // or far from them all (weights 0) off the detector
            const float kf = fminf(fmaxf(floorf(lo), 0.f), kmax);
            float d[4];
            if (__all_sync(0xffffffffu, lo >= 0.f && hi <= endX)) {
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    d[v] = __fsub_rn(xp[v], kf);
                    cnt[v]++;
                }
            } else {
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const bool in = xp[v] >= 0.f && xp[v] <= endX;
                    d[v] = in ? __fsub_rn(xp[v], kf) : -8.f;
                    cnt[v] += in;
                }
            }
            const float* src = win + ((b * BPW_CHUNK + j) * bpw_window<LP>() + ((int)kf - kw)) * G + 4 * lp;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                float2 a[NS / 2];
#pragma unroll
                for (int q = 0; q < NS / 4; q++) {
                    const float4 f = *reinterpret_cast<const float4*>(src + k * G + 4 * LP * q);
                    a[2 * q] = make_float2(f.x, f.y);
                    a[2 * q + 1] = make_float2(f.z, f.w);
                }
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const float w = __saturatef(1.f - fabsf(d[v] - (float)k));
                    const float2 w2 = make_float2(w, w);
#pragma unroll
                    for (int q = 0; q < NS / 2; q++) fma2(acc[v][q], w2, a[q]);
                }
            }
        }
        if (b) phase ^= 1;
        if (tc + 2 * BPW_CHUNK < p.t1) {
            // the buffer is free; nothing more is fetched once a wait of any thread ran out
            if (!__syncthreads_and(ok)) { ok = false; break; }
            fetch(tc + 2 * BPW_CHUNK, b);
            __syncthreads();   // s_kw
        }
        b ^= 1;
    }
    ok = ok && mbar_wait(smem_u32(mbar + 2), 0, p.polls);
    if (!ok) {   // a copy did not arrive: the run is flagged, the voxels keep their values
        mbar_wait(smem_u32(mbar + 2), 0, WIDE_POLLS);
        atomicOr(p.flags + g * G, kFlagStageTimeout);
        return;
    }

    unsigned tested = 0, quads = 0;   // slices summed sample by sample; quads of the group that hold some
    const int bits = p.low_bit | kFlagRawSpecial | kFlagDiffSpecial;
#pragma unroll
    for (int b = 0; b < NS / 4; b++) {
        const int4 f = __ldg(reinterpret_cast<const int4*>(p.flags + g * G + bpw_slice<LP>(lp, b)));
        const int fl[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (fl[q] & bits) {
                tested |= 1u << (4 * b + q);
                quads |= 1u << (bpw_slice<LP>(lp, b) / 4);
            }
    }
    // update: old + sum * (relax / count), clamped at 0
    const bool same = cnt[0] == cnt[1] && cnt[0] == cnt[2] && cnt[0] == cnt[3];
    float k[4];
    k[0] = __fdiv_rn(p.relax, (float)max(cnt[0], 1));
#pragma unroll
    for (int v = 1; v < 4; v++) k[v] = same ? k[0] : __fdiv_rn(p.relax, (float)max(cnt[v], 1));
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const int x = X + (v & 1), z = Z + (v >> 1);
        if (x >= Nx || z >= Nz || cnt[v] <= 0) continue;
        const size_t o = (((size_t)g * Nz + (Nz - 1 - z)) * Nx + x) * G;
#pragma unroll
        for (int b = 0; b < NS / 4; b++) {
            const int sl = bpw_slice<LP>(lp, b);
            float4* dst = reinterpret_cast<float4*>(p.vol + o + sl);
            const float4 o4 = *reinterpret_cast<const float4*>(tile + ((z - Z0) * TX + (x - X0)) * G + sl);
            const float2 kk = make_float2(k[v], k[v]);
            float2 f01 = make_float2(o4.x, o4.y), f23 = make_float2(o4.z, o4.w);
            fma2(f01, acc[v][2 * b], kk);
            fma2(f23, acc[v][2 * b + 1], kk);
            const float f[4] = {f01.x, f01.y, f23.x, f23.y};
            const unsigned mask = (tested >> (4 * b)) & 15;
            // ordinary values only (a NaN or an infinity makes the sum one)
            if (mask || !((fabsf(f[0]) + fabsf(f[1])) + (fabsf(f[2]) + fabsf(f[3])) < -kSentinelTest)) {
                // (the tested slices are another lane's to write)
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (!((mask >> q) & 1)) reinterpret_cast<float*>(dst)[q] = bpw_value(p, g * G + sl + q, f[q]);
                continue;
            }
            *dst = make_float4(fmaxf(f[0], 0.f), fmaxf(f[1], 0.f), fmaxf(f[2], 0.f), fmaxf(f[3], 0.f));
        }
    }
    quads = __reduce_or_sync(0xffffffffu, quads);
    if (quads) bpw_update_tested<LP, NS>(p, tile, X, Z, bits, quads);
}

}  // namespace at3r
