// volume_kernels.cu -- volume ingest and per-volume resources on the GPU:
// synthetic fBm generation, the 9-level density pyramid, the majorant, the
// empty-space occupancy bricks, the transmittance (TR) mips, the HG phase LUT
// and the baked NEE transmittance grid.
//
// The reference builds the pyramid on the CPU (VolumeRender::Update,
// core/volume.cu:1474-1515) and the TR mips / LUT / baked TR with legacy
// texture + surface references (core/volume.cu:1322-1400, 1535-1696).  Here
// every resource is a plain z-fastest fp32 array in HBM, built on the volume's
// stream: the pyramid's levels by a launch each, the TR levels by one, the
// occupancy of the grid and of the mips by two each.
#include <algorithm>
#include <cmath>
#include <vector>

#include "kernels.h"

namespace mrp {

// ---------------------------------------------------------------------------
// fBm value noise (synthetic benchmark volumes; not part of the reference).
// PCG-RXS-M-XS lattice hash (Jarzynski & Olano, JCGT 2020), quintic fade.
// ---------------------------------------------------------------------------
MRP_D uint32_t pcg(uint32_t v) {
    uint32_t s = v * 747796405u + 2891336453u;
    uint32_t w = ((s >> ((s >> 28u) + 4u)) ^ s) * 277803737u;
    return (w >> 22u) ^ w;
}
MRP_D float lattice(uint32_t seed, int ix, int iy, int iz) {
    uint32_t h = pcg(pcg(pcg(pcg(seed) + (uint32_t)ix) + (uint32_t)iy) + (uint32_t)iz);
    return fm((float)(h >> 8), 5.9604644775390625e-8f);
}
MRP_D float quintic(float f) { return fm(fm(fm(f, f), f), fa(fm(f, fs(fm(f, 6.0f), 15.0f)), 10.0f)); }
MRP_D float value_noise(float px, float py, float pz, uint32_t seed) {
    float fx = floorf(px), fy = floorf(py), fz = floorf(pz);
    int ix = (int)fx, iy = (int)fy, iz = (int)fz;
    float wx = quintic(fs(px, fx)), wy = quintic(fs(py, fy)), wz = quintic(fs(pz, fz));
    float c00 = lerp(lattice(seed, ix, iy, iz), lattice(seed, ix, iy, iz + 1), wz);
    float c01 = lerp(lattice(seed, ix, iy + 1, iz), lattice(seed, ix, iy + 1, iz + 1), wz);
    float c10 = lerp(lattice(seed, ix + 1, iy, iz), lattice(seed, ix + 1, iy, iz + 1), wz);
    float c11 = lerp(lattice(seed, ix + 1, iy + 1, iz), lattice(seed, ix + 1, iy + 1, iz + 1), wz);
    return lerp(lerp(c00, c01, wy), lerp(c10, c11, wy), wx);
}
MRP_D float fbm_voxel(int R, int x, int y, int z, uint32_t seed, float base_freq, int octaves, float gain) {
    float Rf = (float)R;
    float u = fd(fa((float)x, 0.5f), Rf), v = fd(fa((float)y, 0.5f), Rf), w = fd(fa((float)z, 0.5f), Rf);
    float sum = 0, norm = 0, amp = 1.0f, freq = base_freq;
    for (int o = 0; o < octaves; ++o) {
        sum = fa(sum, fm(amp, value_noise(fm(u, freq), fm(v, freq), fm(w, freq), seed + (uint32_t)o * 1013u)));
        norm = fa(norm, amp);
        amp = fm(amp, gain);
        freq = fm(freq, 2.0f);
    }
    float n = fd(sum, norm);
    float dx = fs(u, 0.5f), dy = fs(v, 0.5f), dz = fs(w, 0.5f);
    float d = fsq(fa(fa(fm(dx, dx), fm(dy, dy)), fm(dz, dz)));
    float t = fd(fs(d, 0.4f), fs(0.32f, 0.4f));
    t = fminf(fmaxf(t, 0.0f), 1.0f);
    float fall = fm(fm(t, t), fs(3.0f, fm(2.0f, t)));
    return fminf(fmaxf(fm(n, fall), 0.0f), 1.0f);
}
// Stores of a grid texel: fp32, or fp16 storage (round to nearest even).
MRP_D void st_f(float* p, float v) { *p = v; }
MRP_D void st_f(__half* p, float v) { *p = __float2half_rn(v); }
template <class T>
__global__ void k_fbm(T* __restrict__ out, int R, uint32_t seed, float base_freq, int octaves, float gain) {
    size_t n = (size_t)R * R * R;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        int z = (int)(i % R), y = (int)((i / R) % R), x = (int)(i / ((size_t)R * R));
        st_f(out + i, fbm_voxel(R, x, y, z, seed, base_freq, octaves, gain));
    }
}
// fp32 <-> fp16 storage of a grid (set_data into an fp16 volume, readback).
__global__ void k_narrow(const float* __restrict__ in, size_t n, __half* __restrict__ out) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = __float2half_rn(in[i]);
}
__global__ void k_widen(const __half* __restrict__ in, size_t n, float* __restrict__ out) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = __half2float(in[i]);
}

// ---------------------------------------------------------------------------
// Pyramid level from a source grid: the reference's CPU trilinear Sample()
// (border 0, negative values clamped, core/volume.cu:835-863) at texel
// centres u = (i + 0.5) / res (ParallelFill, core/omp.cpp:11-13).
// ---------------------------------------------------------------------------
template <class T>
MRP_D float cpu_fetch(const T* __restrict__ d, int res, int x, int y, int z) {
    if (x < 0 || y < 0 || z < 0 || x >= res || y >= res || z >= res) return 0.0f;
    return fmaxf(0.0f, ldg_f(d + ((size_t)x * res + y) * res + z));
}
// res = 1 << lg (256 >> m, or 512 and 1024 on the way down to 256): one
// thread per texel, k fastest.  The source coordinate of an index is the same
// for all three axes, so a block works the (double) coordinates of the res
// indices out once; per texel that leaves the eight loads and the lerps.
// DRAM bound where the source is the grid: 512^3 -> 256^3 takes 95 us (5.7 TB/s), and all nine
// levels 133 us against 281 with the coordinates worked out per texel.
constexpr int kResampleThreads = 256, kResampleMax = 1024;
template <class T>
__global__ void __launch_bounds__(kResampleThreads) k_resample(float* __restrict__ out, int lg, const T* __restrict__ src,
                                                               int src_res) {
    __shared__ int at[kResampleMax];
    __shared__ float wt[kResampleMax];
    const int res = 1 << lg;
    const float sr = (float)src_res;
    for (int q = threadIdx.x; q < res; q += kResampleThreads) {
        const float u = (float)(((double)q + 0.5) / res);
        const float px = fs(fm(u, sr), 0.5f);
        const int x = (int)floorf(px);
        at[q] = x;
        wt[q] = fs(px, (float)x);
    }
    __syncthreads();
    const int n = 1 << (3 * lg);
    const size_t sx = (size_t)src_res * src_res, sy = src_res;
    for (int i = blockIdx.x * kResampleThreads + threadIdx.x; i < n; i += gridDim.x * kResampleThreads) {
        const int k = i & (res - 1), j = (i >> lg) & (res - 1), q = i >> (2 * lg);
        const int x = at[q], y = at[j], z = at[k];
        const float wx = wt[q], wy = wt[j], wz = wt[k];
        float t[8];
        if ((unsigned)x < (unsigned)(src_res - 1) && (unsigned)y < (unsigned)(src_res - 1) &&
            (unsigned)z < (unsigned)(src_res - 1)) {
            const T* p = src + x * sx + y * sy + z;
            t[0] = ldg_f(p); t[1] = ldg_f(p + 1); t[2] = ldg_f(p + sy); t[3] = ldg_f(p + sy + 1);
            t[4] = ldg_f(p + sx); t[5] = ldg_f(p + sx + 1); t[6] = ldg_f(p + sx + sy); t[7] = ldg_f(p + sx + sy + 1);
#pragma unroll
            for (int c = 0; c < 8; ++c) t[c] = fmaxf(0.0f, t[c]);
        } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) t[c] = cpu_fetch(src, src_res, x + (c >> 2), y + ((c >> 1) & 1), z + (c & 1));
        }
        const float a = lerp(lerp(t[0], t[1], wz), lerp(t[2], t[3], wz), wy);
        const float b = lerp(lerp(t[4], t[5], wz), lerp(t[6], t[7], wz), wy);
        out[i] = lerp(a, b, wx);
    }
}

// Mip level L and TR level L - 1 side by side per texel, L = 1..4
// (VolumeDev::mip_tr).
__global__ void k_interleave_mip_tr(const float* __restrict__ mips, const float* __restrict__ trs,
                                    float2* __restrict__ out) {
    const int total = mip_tr_offset(5);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        int L = 1;
        while (L < 4 && i >= mip_tr_offset(L + 1)) ++L;
        const int j = i - mip_tr_offset(L);
        out[i] = make_float2(mips[mip_offset(L) + j], trs[tr_offset(L - 1) + j]);
    }
}

// The padded mips and TR levels side by side (VolumeDev::pad_pair).
__global__ void k_pair_padded(const float* __restrict__ a, const float* __restrict__ b, float2* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kPadLevelFloats; i += gridDim.x * blockDim.x)
        out[i] = make_float2(a[i], b[i]);
}

// Padded copies of three levels of edge 8, 4, 2 (blockIdx.y picks one): the
// texel of (x, y, z) in [-1, n + 1]^3 is the level's texel under border
// addressing (0 outside) or clamp addressing (nearest edge texel).
__global__ void k_pad_levels(const float* __restrict__ l8, const float* __restrict__ l4, const float* __restrict__ l2,
                             int clamp, float* __restrict__ out) {
    const int n = 8 >> blockIdx.y, P = n + 3;
    const float* src = blockIdx.y == 0 ? l8 : blockIdx.y == 1 ? l4 : l2;
    float* dst = out + pad_offset(n);
    for (int i = threadIdx.x; i < P * P * P; i += blockDim.x) {
        int x = i / (P * P) - 1, y = (i / P) % P - 1, z = i % P - 1;
        float val;
        if (clamp) {
            x = min(max(x, 0), n - 1); y = min(max(y, 0), n - 1); z = min(max(z, 0), n - 1);
            val = src[(x * n + y) * n + z];
        } else {
            const bool in = (unsigned)x < (unsigned)n && (unsigned)y < (unsigned)n && (unsigned)z < (unsigned)n;
            val = in ? src[(x * n + y) * n + z] : 0.0f;
        }
        dst[i] = val;
    }
}

// ---------------------------------------------------------------------------
// One pass over a grid for everything Update derives from single voxels: the
// majorant, the bounds of the nonzero voxels, and per row (x, y) which bricks
// along z the row's nonzero voxels occupy.
//
// Majorant: max density floored at the reference's default 1e-5
// (core/volume.hpp:104).  Densities are compared as int bits, which orders
// non-negative floats; negative (SDF) values never win.
//
// Occupancy bricks for exact empty-space skipping in the first-hit march.
// Brick b covers voxels [8b, 8b + 8) per axis.  A trilinear fetch whose base
// voxel lies in brick b reads voxels base..base+1, i.e. at most one voxel
// past the brick; the brick is marked occupied when any voxel in
// [8b - 1, 8b + 9] holds a non-zero value, one voxel more on each side than
// the fetch needs, so that a base voxel found from a coordinate that may be
// off by less than one voxel still picks a brick whose apron holds the whole
// footprint.  A zero brick therefore guarantees Density() == 0 exactly for
// every sample whose base voxel is in it or within one voxel of it (border
// texels are 0 by addressing).
//
// DRAM bound: each voxel is read once (k_scan_rows), then the rows' masks are
// combined over 11 x 11 rows per brick column (k_occ_bricks).  A row's masks
// take 16 bytes per started 1024 voxels: a 32nd of the grid from 128^3 in fp32
// and 256^3 in fp16 on, more below (an eighth at 32^3).  512^3 fp32 and the five mips: 160 us (the grid alone
// 118 us, 4.6 TB/s) against 1.94 ms when the majorant, the bounds and each
// brick's 11^3 voxels were read by kernels of their own.
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 256, kScanBlocks = 6;   // resident blocks per SM: one wave
constexpr int kSegVoxels = 1024;   // voxels of a row that a warp masks at a time
struct ScanJobs {
    OccJob job[kMaxOccJobs];
};
// One warp per row; lane l keeps the 32-bit mask of voxels 32 l .. 32 l + 31
// of each segment, widens it by the aprons' voxels, and the warp leaves four
// words per segment: bit l of word b is brick 4 l + b of the segment.
// stats (or null): the bounds {min x, y, z, max x, y, z}, then the majorant's bits.
template <class T>
__global__ void __launch_bounds__(kScanThreads, kScanBlocks) k_scan_rows(const T* __restrict__ only, ScanJobs jobs,
                                                            int* __restrict__ stats) {
    const OccJob J = jobs.job[blockIdx.y];
    const T* __restrict__ d = only ? only : reinterpret_cast<const T*>(J.src);
    const int R = J.R, lane = threadIdx.x & 31;
    const int warps = gridDim.x * (kScanThreads / 32);
    const int segs = (R + kSegVoxels - 1) / kSegVoxels;   // 1 or 2 (R <= 2048)
    int lo[3] = {R, R, R}, hi[3] = {-1, -1, -1};
    float top = 0.00001f;
    for (int row = blockIdx.x * (kScanThreads / 32) + threadIdx.x / 32; row < R * R; row += warps) {
        const T* p = d + (size_t)row * R;
        uint32_t m[2] = {0u, 0u};
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            if (s >= segs) break;
            const int nw = min((R - s * kSegVoxels + 31) / 32, 32);
            for (int c0 = 0; c0 < nw; c0 += 16) {   // sixteen loads in flight per lane
                float v[16];
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    const int z = s * kSegVoxels + 32 * (c0 + c) + lane;
                    v[c] = z < R ? ldg_f(p + z) : 0.0f;
                }
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    top = fmaxf(top, v[c]);
                    const uint32_t b = __ballot_sync(0xffffffffu, v[c] != 0.0f);
                    if (lane == c0 + c) m[s] = b;
                }
            }
        }
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            if (s >= segs) break;
            uint32_t up = __shfl_up_sync(0xffffffffu, m[s], 1), dn = __shfl_down_sync(0xffffffffu, m[s], 1);
            const uint32_t last0 = __shfl_sync(0xffffffffu, m[0], 31), first1 = __shfl_sync(0xffffffffu, m[1], 0);
            if (lane == 0) up = s ? last0 : 0u;
            if (lane == 31) dn = s ? 0u : first1;
            const uint32_t w = m[s] | (m[s] << 1) | (up >> 31) | (m[s] >> 1) | (dn << 31) | (m[s] >> 2) | (dn << 30);
            uint4 o;
            o.x = __ballot_sync(0xffffffffu, (w & 0x000000ffu) != 0u);
            o.y = __ballot_sync(0xffffffffu, (w & 0x0000ff00u) != 0u);
            o.z = __ballot_sync(0xffffffffu, (w & 0x00ff0000u) != 0u);
            o.w = __ballot_sync(0xffffffffu, (w & 0xff000000u) != 0u);
            if (lane == 0) J.rows[row * segs + s] = o;
            const uint32_t any = __ballot_sync(0xffffffffu, m[s] != 0u);
            if (stats && any) {
                const int f = __ffs(any) - 1, l = 31 - __clz(any);
                const uint32_t mf = __shfl_sync(0xffffffffu, m[s], f), ml = __shfl_sync(0xffffffffu, m[s], l);
                const int x = row / R, y = row % R, z0 = s * kSegVoxels;
                lo[0] = min(lo[0], x); hi[0] = max(hi[0], x);
                lo[1] = min(lo[1], y); hi[1] = max(hi[1], y);
                lo[2] = min(lo[2], z0 + 32 * f + __ffs(mf) - 1); hi[2] = max(hi[2], z0 + 32 * l + 31 - __clz(ml));
            }
        }
    }
    if (!stats) return;
    for (int o = 16; o; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (lane == 0) {
        atomicMax(stats + 6, __float_as_int(top));
        if (hi[0] >= 0)
            for (int a = 0; a < 3; ++a) {
                atomicMin(stats + a, lo[a]);
                atomicMax(stats + 3 + a, hi[a]);
            }
    }
}
// One block per 4 x 4 brick columns, one column a warp: the column's bricks
// from the masks of its 11 x 11 rows, and of the block's sixteen columns the
// coarse bricks (4^3 bricks each: coarse brick C is empty when the 64 bricks
// 4C..4C+3 per axis are; their aprons together are the coarse brick's own
// apron, so a zero coarse brick carries the same guarantee over its span).
__global__ void __launch_bounds__(512) k_occ_bricks(ScanJobs jobs) {
    const OccJob J = jobs.job[blockIdx.y];
    const int R = J.R, nb = (R + 7) >> 3, nc = (nb + 3) >> 2, segs = (R + kSegVoxels - 1) / kSegVoxels;
    if ((int)blockIdx.x >= nc * nc) return;
    __shared__ uint32_t coarse[64];
    if (threadIdx.x < 64) coarse[threadIdx.x] = 0u;
    __syncthreads();
    const int cx = blockIdx.x / nc, cy = blockIdx.x % nc, warp = threadIdx.x / 32, lane = threadIdx.x & 31;
    const int bx = 4 * cx + warp / 4, by = 4 * cy + warp % 4;
    if (bx < nb && by < nb) {
        for (int s = 0; s < segs; ++s) {
            uint4 o = make_uint4(0u, 0u, 0u, 0u);
            for (int t = lane; t < 121; t += 32) {
                const int x = 8 * bx - 1 + t / 11, y = 8 * by - 1 + t % 11;
                if ((unsigned)x < (unsigned)R && (unsigned)y < (unsigned)R) {
                    const uint4 r = J.rows[(x * R + y) * segs + s];
                    o.x |= r.x; o.y |= r.y; o.z |= r.z; o.w |= r.w;
                }
            }
            o.x = __reduce_or_sync(0xffffffffu, o.x); o.y = __reduce_or_sync(0xffffffffu, o.y);
            o.z = __reduce_or_sync(0xffffffffu, o.z); o.w = __reduce_or_sync(0xffffffffu, o.w);
            const uint32_t b[4] = {(o.x >> lane) & 1u, (o.y >> lane) & 1u, (o.z >> lane) & 1u, (o.w >> lane) & 1u};
            const int bz = s * (kSegVoxels / 8) + 4 * lane;
            uint8_t* dst = J.occ + (bx * nb + by) * nb;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (bz + q < nb) dst[bz + q] = (uint8_t)b[q];
            if (b[0] | b[1] | b[2] | b[3]) coarse[s * 32 + lane] = 1u;
        }
    }
    __syncthreads();
    if (J.coarse && (int)threadIdx.x < nc) J.coarse[(cx * nc + cy) * nc + threadIdx.x] = (uint8_t)coarse[threadIdx.x];
}

// ---------------------------------------------------------------------------
// Fill_TR (core/volume.cu:1535-1560): transmittance of TR level `level`
// (res 128>>level) marched 128 steps toward the light through density level
// level+1 with alpha scaled by 1.73^(level+1) (core/volume.cu:1636-1653).
//
// One launch for all eight levels, the small ones first: their 128 steps in
// series take about as long as a level of any size (28 to 56 us each when
// launched one after the other), so they run beside level 0's blocks.  Bound
// by level 0's instructions (2 M voxels x 128 steps).  The levels are read
// from copies with a border of zeros (tr_pad_off): a voxel at a face takes
// 128 tiny steps there, and with another kind of fetch for the edge one such
// lane sends its whole warp through both.  All levels of a 256^3 cloud:
// 1.13 ms in eight launches, 0.84 ms in one, 0.51 ms from the padded copies
// with floor taken by an addition, 0.43 ms with the steps cut to the box of
// nonzero voxels, 0.39 ms with the texels in z pairs.
// ---------------------------------------------------------------------------
constexpr int kTrLevels = 8, kTrThreads = 128;
__host__ __device__ constexpr int tr_blocks(int lv) {   // blocks of level lv
    const int n = 128 >> lv;
    return (n * n * n + kTrThreads - 1) / kTrThreads;
}
__host__ __device__ constexpr int tr_first_block(int lv) {   // levels 7, 6, ..., 0 in that order
    int o = 0;
    for (int l = kTrLevels - 1; l > lv; --l) o += tr_blocks(l);
    return o;
}
// Padded copy of mip lv + 1 (edge n = 128 >> lv): (n + 2)^3 pairs, texels
// (x, y, z) and (x, y, z + 1) at ((x + 1) P + y + 1) P + z + 1 with P = n + 2,
// zeros around: a fetch takes four loads, each a lerp's two operands.
__host__ __device__ constexpr int tr_pad_off(int lv) {
    int o = 0;
    for (int l = 0; l < lv; ++l) { const int p = (128 >> l) + 2; o += p * p * p; }
    return o;
}
static_assert(tr_pad_off(kTrLevels) == (int)kTrPadTexels, "padded pyramid size");
__global__ void k_pad_pyramid(const float* __restrict__ mips, float2* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < (int)kTrPadTexels; i += gridDim.x * blockDim.x) {
        int lv = 0;
        while (lv + 1 < kTrLevels && i >= tr_pad_off(lv + 1)) ++lv;
        const int n = 128 >> lv, P = n + 2, j = i - tr_pad_off(lv);
        const int x = j / (P * P) - 1, y = (j / P) % P - 1, z = j % P - 1;
        const float* m = mips + mip_offset(lv + 1);
        out[i] = make_float2(fetch_border(m, n, x, y, z), fetch_border(m, n, x, y, z + 1));
    }
}


// Sum of the density over 128 steps of d from p through level LV, in tex3's
// arithmetic: the edge is a power of two, so u N is exact and u N - 0.5 one
// fused operation, and adding 1.5 2^23 rounding down leaves floor in the low
// mantissa bits (the offsets of those bits fold into the addresses).  An
// empty brick adds exactly 0 and is skipped.  Steps before `first` only move
// p, steps from `last` on are left out (both read 0).  The steps must stay
// within a quarter of a texel of the unit cube.
template <int LV>
MRP_D float tr_march(const float2* __restrict__ pad, const uint8_t* __restrict__ occ, f3 p, f3 d, int first, int last) {
    constexpr int N = 128 >> LV, P = N + 2, NB = (N + 7) >> 3;
    constexpr float kFloor = 12582912.0f;
    constexpr uint32_t kBits = 0x4B400000u;
    constexpr uint32_t kBase = (kBits - 1u) * (uint32_t)(P * P + P + 1);
    constexpr uint32_t kBrick = (kBits >> 3) * (uint32_t)(NB * NB + NB + 1);
    float acc = 0.0f;
    int s = 0;
    for (; s < first; ++s) p = add(p, d);
    for (; s < last; ++s) {
        p = add(p, d);
        const float px = fmaf(fa(p.x, 0.5f), (float)N, -0.5f), py = fmaf(fa(p.y, 0.5f), (float)N, -0.5f),
                    pz = fmaf(fa(p.z, 0.5f), (float)N, -0.5f);
        const float tx = __fadd_rd(px, kFloor), ty = __fadd_rd(py, kFloor), tz = __fadd_rd(pz, kFloor);
        const uint32_t x = __float_as_uint(tx), y = __float_as_uint(ty), z = __float_as_uint(tz);
        if (occ) {   // voxel -1 belongs to brick 0
            const uint32_t bx = max(x, kBits) >> 3, by = max(y, kBits) >> 3, bz = max(z, kBits) >> 3;
            if (__ldg(occ + ((bx * NB + by) * NB + bz - kBrick)) == 0) continue;
        }
        const float wx = fs(px, fs(tx, kFloor)), wy = fs(py, fs(ty, kFloor)), wz = fs(pz, fs(tz, kFloor));
        const float ox = fs(1.0f, wx), oy = fs(1.0f, wy), oz = fs(1.0f, wz);
        const float2* b = pad + ((x * P + y) * P + z - kBase);
        const float2 t00 = __ldg(b), t01 = __ldg(b + P), t10 = __ldg(b + P * P), t11 = __ldg(b + P * P + P);
        const float c00 = lerp_w(t00.x, t00.y, wz, oz), c01 = lerp_w(t01.x, t01.y, wz, oz);
        const float c10 = lerp_w(t10.x, t10.y, wz, oz), c11 = lerp_w(t11.x, t11.y, wz, oz);
        acc = fa(acc, lerp_w(lerp_w(c00, c01, wy, oy), lerp_w(c10, c11, wy, oy), wx, ox));
    }
    return acc;
}
// The same by general fetches, for rays that leave the cube (a light
// direction that is not a number).
__device__ __noinline__ float tr_march_any(const float* __restrict__ mip, int n, f3 p, f3 d) {
    float acc = 0.0f;
    for (int s = 0; s < 128; ++s) {
        p = add(p, d);
        acc = fa(acc, tex3<false>(mip, n, p));
    }
    return acc;
}
// One voxel of level LV; mip_occ (may be null): 8^3 brick flags of mip levels 0..kOccMips-1.
template <int LV>
MRP_D void tr_voxel(float* __restrict__ trs, const float* __restrict__ mips, const float2* __restrict__ mips_tr,
                    const uint8_t* __restrict__ mip_occ, const TrArgs& A) {
    constexpr int N = 128 >> LV;
    const f3 L = A.L;
    const int i = ((int)blockIdx.x - tr_first_block(LV)) * kTrThreads + (int)threadIdx.x;
    if (i >= N * N * N) return;
    const int z = i % N, y = (i / N) % N, x = i / (N * N);
    const f3 uv = div(adds(mk3((float)x, (float)y, (float)z), 0.5f), (float)N);
    const f3 ori = subs(uv, 0.5f);
    const float dis = ray_box_distance(ori, L);
    const float step = fd(dis, 128.0f);
    const f3 d = mul(L, step);
    constexpr float lim = 0.5f + 0.25f / N;
    const bool inside = fabsf(ori.x + 128.0f * d.x) <= lim && fabsf(ori.y + 128.0f * d.y) <= lim &&
                        fabsf(ori.z + 128.0f * d.z) <= lim;
    // the steps whose fetch can touch a nonzero texel: a nonzero voxel lies
    // within 1/R + 2/N of it (a voxel of every level on the way down, half as
    // large each, and the fetch's own footprint); the box of nonzero voxels
    // has 2/R of margin already, and two steps cover the divisions' rounding
    const float o[3] = {ori.x, ori.y, ori.z}, dd[3] = {d.x, d.y, d.z}, lo[3] = {A.lo.x, A.lo.y, A.lo.z},
                hi[3] = {A.hi.x, A.hi.y, A.hi.z};
    constexpr float grow = 2.25f / N;
    float s0 = 0.0f, s1 = 128.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float l = lo[a] - grow - o[a], h = hi[a] + grow - o[a];
        if (fabsf(dd[a]) < 1e-30f) {   // does not move along this axis
            if (l > 0.0f || h < 0.0f) s1 = -1.0f;
        } else {
            const float r = 1.0f / dd[a], ta = l * r, tb = h * r;
            s0 = fmaxf(s0, fminf(ta, tb));
            s1 = fminf(s1, fmaxf(ta, tb));
        }
    }
    const int last = s0 > s1 ? 0 : (int)fminf(s1 + 2.0f, 128.0f), first = (int)fmaxf(fminf(s0, 128.0f) - 3.0f, 0.0f);
    const float acc =
        inside ? tr_march<LV>(mips_tr + tr_pad_off(LV),
                              LV + 1 < kOccMips && mip_occ ? mip_occ + mip_occ_offset(LV + 1) : nullptr, ori, d,
                              first, last)
               : tr_march_any(mips + mip_offset(LV + 1), N, ori, d);
    trs[tr_offset(LV) + i] = fm(1.0f, fm(expf(fm(fm(-acc, A.alpha[LV]), step)), 1.0f));
}
__global__ void __launch_bounds__(kTrThreads) k_tr_levels(float* __restrict__ trs, const float* __restrict__ mips,
                                                          const float2* __restrict__ mips_tr,
                                                          const uint8_t* __restrict__ mip_occ,
                                                          const __grid_constant__ TrArgs A) {
    const int b = (int)blockIdx.x;
    if (b >= tr_first_block(0)) tr_voxel<0>(trs, mips, mips_tr, mip_occ, A);
    else if (b >= tr_first_block(1)) tr_voxel<1>(trs, mips, mips_tr, mip_occ, A);
    else if (b >= tr_first_block(2)) tr_voxel<2>(trs, mips, mips_tr, mip_occ, A);
    else if (b >= tr_first_block(3)) tr_voxel<3>(trs, mips, mips_tr, mip_occ, A);
    else if (b >= tr_first_block(4)) tr_voxel<4>(trs, mips, mips_tr, mip_occ, A);
    else if (b >= tr_first_block(5)) tr_voxel<5>(trs, mips, mips_tr, mip_occ, A);
    else if (b >= tr_first_block(6)) tr_voxel<6>(trs, mips, mips_tr, mip_occ, A);
    else tr_voxel<7>(trs, mips, mips_tr, mip_occ, A);
}

// ---------------------------------------------------------------------------
// Fill_Hg (core/volume.cu:1322-1400): 512x512 LUT of the HG phase averaged
// over a cone, 1024 scrambled-Halton samples per texel.  The digit
// permutations are the reference's (core/volume.cu:1195, from the model
// file), the per-texel shift bn comes from the texel's LUT stream instead of
// a curand draw.
// ---------------------------------------------------------------------------
constexpr int kHgSamples = 1024;
// The scrambled radical inverses of samples 0..1023 in bases 2, 3, 5 and 11
// (x, y, z, w), the same for every texel: filled from the host.
__device__ float4 d_halton[kHgSamples];

static float scrambled_radical_inverse(uint32_t base, const uint32_t* perm, uint32_t a) {
    const float inv_base = 1.0f / (float)base;
    uint32_t rev = 0;
    float inv_base_n = 1.0f;
    while (a) {
        uint32_t next = a / base;
        uint32_t digit = a - next * base;
        rev = rev * base + perm[digit];
        inv_base_n = inv_base_n * inv_base;
        a = next;
    }
    const float tail = (inv_base * (float)perm[0]) / (1.0f - inv_base);
    return std::fmin(inv_base_n * ((float)rev + tail), 0.99999994f);
}
// frac(f) = f - (float)(long)f for 0 <= f < 2
MRP_D float frac2(float f) { return f >= 1.0f ? fs(f, 1.0f) : f; }

// One texel's constants and its two sample estimators.  The arithmetic is
// Fill_Hg's; terms that its vectors carry without effect are left out: the
// view direction is (1, 0, 0) and the texel's direction has no z, so of
// sample_hg's vector only x = cos and y = -sin sin(phi) + 0 cos enter the dot
// product, and dot(normalize(p), view) is p.x / length(p).
struct HgTexel {
    float g, radius, bn;
    f3 dir;
    MRP_D float phase_sample(float4 q) const {   // a direction drawn from the phase function
        const float e0 = frac2(fa(q.x, bn)), e1 = frac2(fa(q.y, bn));
        float cost;
        if (fabsf(g) < 0.0001) {
            cost = fs(fm(e0, 2.0f), 1.0f);
        } else {
            const float g2 = fm(g, g);
            const float t0 = fd(fs(1.0f, g2), fa(fs(1.0f, g), fm(fm(2.0f, g), e0)));
            cost = fd(fs(fa(1.0f, g2), fm(t0, t0)), fm(2.0f, g));
        }
        const float phi = (float)(2.0 * 3.14159265359 * (double)e1);
        const float sint = fsq(fmaxf(0.0f, fs(1.0f, fm(cost, cost))));
        const float y = fa(-fm(sint, sinf(phi)), fm(0.0f, cost));   // (not a number where cost is infinite, |g| > 1)
        const float sdotl = fa(fm(dir.x, cost), fm(dir.y, y));
        const float p = fa(fs(fm(radius, radius), 1.0f), fm(sdotl, sdotl));
        if (p <= 0) return 0.0f;
        const float w = fsq(p);
        float d0 = fs(sdotl, w);
        const float d1 = fd(fa(sdotl, w), radius);
        d0 = fd(fmaxf(0.0f, d0), radius);
        const float d = fs(fm(fm(d1, d1), d1), fm(fm(d0, d0), d0));
        return fmaxf(0.0f, fd(d, 4.0f));
    }
    MRP_D float cone_sample(float4 q) const {    // a point of the ball around the direction
        const float rx = frac2(fa(q.x, bn)), ry = frac2(fa(q.y, bn)), rz = frac2(fa(q.z, bn));
        const float theta = (float)((double)rx * 2.0 * 3.1415926535);
        const float phi = (float)acos(2.0 * (double)ry - 1.0);
        const float r = powf(rz, fd(1.0f, 3.0f));
        float st_, ct, sp, cp;
        sincosf(theta, &st_, &ct);
        sincosf(phi, &sp, &cp);
        const float rr = fm(radius, r), rs = fm(rr, sp);
        const f3 rp = add(mk3(fm(rs, ct), fm(rs, st_), fm(rr, cp)), dir);
        return hg(fd(rp.x, length(rp)), g);
    }
};

// One texel a thread, 128 texels of a row a block, 32 samples at a time.  A
// sample is of one kind or the other (frac(w + bn) < mis); lanes disagree on
// almost every sample, so the kinds are taken apart: each lane runs through
// its own phase samples, then through its own cone samples, leaves the terms
// in its column of shared memory and adds them there in sample order, which
// keeps the sum's rounding.  Bound by the estimators' instructions (double
// acos, powf twice, sines and cosines in a cone sample).  One table: 12.85 ms
// with the digits of every inverse worked out per texel and both kinds run in
// turn for every sample, 3.96 ms this way (the same bits).
constexpr int kHgChunk = 32;
__global__ void __launch_bounds__(128) k_hg_lut(float* __restrict__ lut, float g, uint32_t seed) {
    __shared__ float4 pts[kHgSamples];
    __shared__ float term[kHgChunk][128];
    for (int k = threadIdx.x; k < kHgSamples; k += 128) pts[k] = d_halton[k];
    const int i = blockIdx.x * 128 + threadIdx.x, j = blockIdx.y;
    const float costheta = (float)((((double)(float)i + 0.5) / kLut) * 2.0 - 1.0);
    const float aa = (float)(((double)(float)j + 0.5) / kLut);
    const float angle = (float)((double)aa * 3.1415926535 * 60.0 / 180.0);
    Stream st(kLutStream, (uint32_t)(j * kLut + i), 0, 0, seed);
    HgTexel T;
    T.g = g;
    T.bn = st.next();
    T.radius = tanf(angle);
    T.dir = mk3(costheta, fsq(fs(1.0f, fm(costheta, costheta))), 0.0f);
    float mis = 0;
    {
        float p = fa(fs(fm(T.radius, T.radius), 1.0f), fm(T.dir.x, T.dir.x));
        if (p > 0) {
            float sdotl = g > 0 ? T.dir.x : -T.dir.x;
            float w = fsq(p);
            float d0 = fd(fmaxf(0.0f, fs(sdotl, w)), T.radius);
            float d1 = fd(fa(sdotl, w), T.radius);
            float d = fs(fm(fm(d1, d1), d1), fm(fm(d0, d0), d0));
            mis = fm((float)(d1 > d0), d);
        }
        mis = fminf(fmaxf(mis, 1e-8f), 1.0f);
        float a = fabsf(g);
        double ad = a;
        a = (float)(ad < 0.6 ? 0.0 : (ad < 0.7 ? (ad - 0.6) * 9 : (pow((ad - 0.7) / 0.3, 0.05) * 0.1 + 0.9)));
        mis = fs(1.0f, fd(1.0f, fa(1.0f, fd(fm(a, mis), fs(1.0f, a)))));
    }
    __syncthreads();
    float h = 0.0f;
    float* own = &term[0][threadIdx.x];
    for (int k0 = 0; k0 < kHgSamples; k0 += kHgChunk) {
        uint32_t phase = 0;
#pragma unroll 8
        for (int k = 0; k < kHgChunk; ++k) phase |= (uint32_t)(frac2(fa(pts[k0 + k].w, T.bn)) < mis) << k;
        for (uint32_t m = phase; m; m &= m - 1) {
            const int k = __ffs(m) - 1;
            own[k * 128] = T.phase_sample(pts[k0 + k]);
        }
        for (uint32_t m = ~phase; m; m &= m - 1) {
            const int k = __ffs(m) - 1;
            own[k * 128] = T.cone_sample(pts[k0 + k]);
        }
#pragma unroll 8
        for (int k = 0; k < kHgChunk; ++k) h = fa(h, own[k * 128]);
    }
    lut[j * kLut + i] = fd(h, (float)kHgSamples);
}

MRP_D float density(const VolumeDev& v, f3 p) { return density_tex(v, p); }

// The part [t_in, t_out] of the ray p + t L outside which Density() is
// exactly 0 (the nonzero voxels' box, VolumeDev::nz_lo / nz_hi, whose margin
// of a voxel is far above the rounding here); t_in > t_out when the ray
// misses it, everything when no box was computed.
struct BoxSpan { float t_in, t_out; };
MRP_D BoxSpan nonzero_span(const VolumeDev& v, f3 p, f3 L) {
    BoxSpan b{0.0f, 3.0e38f};
    if (!v.has_bounds) return b;
    const float o[3] = {p.x, p.y, p.z}, d[3] = {L.x, L.y, L.z};
    const float lo[3] = {v.nz_lo.x, v.nz_lo.y, v.nz_lo.z}, hi[3] = {v.nz_hi.x, v.nz_hi.y, v.nz_hi.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (d[a] == 0.0f) {
            if (o[a] < lo[a] || o[a] > hi[a]) b.t_in = 3.0e38f, b.t_out = -1.0f;
        } else {
            const float ta = (lo[a] - o[a]) / d[a], tb = (hi[a] - o[a]) / d[a];
            b.t_in = fmaxf(b.t_in, fminf(ta, tb));
            b.t_out = fminf(b.t_out, fmaxf(ta, tb));
        }
    }
    return b;
}

// Tr (transmittance, common.cuh) over the steps that can change it: the same
// draws and the same estimate.  Density 0 leaves tr as it is in both loops,
// so no texel is read before t_in, and past t_out the walk can end: its
// remaining steps only use up draws that nobody reads.  (Needs t to grow:
// smax > 0 and tr_scale > 0.)
template <class DT>
MRP_D float transmittance_span(const VolumeDev& v, Stream& st, f3 pos, f3 dir, float dis, float alpha, BoxSpan span) {
    const float smax = fm(v.max_density, alpha);
    float tr = 1.0f, t = 0.0f;
    if (span.t_in > span.t_out) return tr;
    const float end = fminf(dis, span.t_out);
    int loop = 0;
    while (loop++ < 10000 && tr > 0.5) {
        float rk = st.next();
        t = fs(t, fm(fd(logf(fs(1.0f, rk)), smax), v.tr_scale));
        if (t > end) return tr;
        float d = t < span.t_in ? 0.0f : density_occ<DT>(v, add(pos, mul(dir, t)));
        float S = fm(d, alpha);
        tr = fm(tr, fs(1.0f, fmaxf(0.0f, fd(S, smax))));
        if (d < 0) t = fs(t, d);
    }
    while (loop++ < 10000 && tr > 0.001) {
        float rk = st.next();
        t = fs(t, fm(fd(logf(fs(1.0f, rk)), smax), v.tr_scale));
        if (t > end) break;
        float d = t < span.t_in ? 0.0f : density_occ<DT>(v, add(pos, mul(dir, t)));
        float S = fm(d, alpha);
        if (st.next() < fmaxf(0.0f, fd(S, smax))) { tr = 0.0f; break; }
        if (d < 0) t = fs(t, d);
    }
    return tr;
}

// Fill_BakeTR (core/volume.cu:1562-1587) over voxels [first, first+count):
// the mean of 5 (density > 0) or 2 estimates of Tr from the voxel.
// replicate != 0 restarts the voxel's stream for every estimate, as InitRand
// inside the reference's loop does: the estimates are identical, so one walk
// gives them all, and only their float sum is formed as often as the loop
// would (which matters for 5 of them: v + v over 2 is v).
//
// Bound by the walks' instructions (Philox, log and division per step, lanes
// of a warp ending apart).  768^3 over a 128^3 cloud: 262 -> 63 ms from one walk instead of 2 or 5 and
// from walks that end with the box.
//
// GROWS: every step moves the walk on (launch_baked_tr).  A walk that goes
// backwards or stands still (a negative or zero extinction or step scale)
// takes transmittance as it is: it reads the density behind the voxel, and
// carried past the far side by a negative density it comes back.  An instance
// of its own: with a way back out of its first loop the other took 175 instead
// of 125 ms for two bakes of 768^3.
template <class DT, bool GROWS>
__global__ void __launch_bounds__(128) k_baked_tr(float* __restrict__ out, const __grid_constant__ VolumeDev v,
                                                  int bake_res, float alpha, f3 L, uint32_t seed, int replicate,
                                                  int64_t first, int64_t count) {
    float rf = (float)bake_res;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < count; q += (int64_t)gridDim.x * blockDim.x) {
        int64_t vi = first + q;
        int x = (int)(vi / ((int64_t)bake_res * bake_res)), y = (int)((vi / bake_res) % bake_res), z = (int)(vi % bake_res);
        f3 uv = div(adds(mk3((float)x, (float)y, (float)z), 0.5f), rf);
        f3 p = subs(uv, 0.5f);
        uint32_t hi = (uint32_t)(vi >> 32) * 8u;
        const float md = ray_box_distance(p, L);
        const BoxSpan span = GROWS ? nonzero_span(v, p, L) : BoxSpan{};
        auto walk = [&](Stream& st) {
            if constexpr (GROWS) return transmittance_span<DT>(v, st, p, L, md, alpha, span);
            else return transmittance<DT>(v, st, p, L, md, alpha);
        };
        float res;
        if (replicate) {
            Stream st(kBakeStream, (uint32_t)vi, hi, 0, seed);
            res = walk(st);
            // five equal terms: 0 and 1 sum exactly, others round on the way
            if (res != 0.0f && res != 1.0f && density(v, p) > 0) {
                float acc = 0.0f;
                for (int i = 0; i < 5; ++i) acc = fa(acc, res);
                res = fd(acc, 5.0f);
            }
        } else {
            int cnt = density(v, p) > 0 ? 5 : 2;
            float acc = 0.0f;
            for (int i = 0; i < cnt; ++i) {
                Stream st(kBakeStream, (uint32_t)vi, hi + (uint32_t)i, 0, seed);
                acc = fa(acc, walk(st));
            }
            res = fd(acc, (float)cnt);
        }
        out[vi] = res;
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static int grid_for(size_t n, int block, int sms) {
    size_t g = (n + block - 1) / block;
    size_t cap = (size_t)sms * 32;
    return (int)(g < cap ? (g ? g : 1) : cap);
}

template <class T>
static cudaError_t fbm_t(T* out, int R, uint32_t seed, float base_freq, int octaves, float gain, int sms,
                         cudaStream_t s) {
    k_fbm<T><<<grid_for((size_t)R * R * R, 256, sms), 256, 0, s>>>(out, R, seed, base_freq, octaves, gain);
    return cudaGetLastError();
}
cudaError_t launch_fbm(float* out, int R, uint32_t seed, float base_freq, int octaves, float gain, int sms,
                       cudaStream_t s) {
    return fbm_t(out, R, seed, base_freq, octaves, gain, sms, s);
}
cudaError_t launch_fbm(__half* out, int R, uint32_t seed, float base_freq, int octaves, float gain, int sms,
                       cudaStream_t s) {
    return fbm_t(out, R, seed, base_freq, octaves, gain, sms, s);
}
cudaError_t launch_narrow(const float* in, size_t n, __half* out, int sms, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_narrow<<<grid_for(n, 256, sms), 256, 0, s>>>(in, n, out);
    return cudaGetLastError();
}
cudaError_t launch_widen(const __half* in, size_t n, float* out, int sms, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_widen<<<grid_for(n, 256, sms), 256, 0, s>>>(in, n, out);
    return cudaGetLastError();
}
template <class T>
static cudaError_t resample_t(float* out, int res, const T* src, int src_res, int sms, cudaStream_t s) {
    int lg = 0;
    while ((1 << lg) < res) ++lg;
    if ((1 << lg) != res || res > kResampleMax) return cudaErrorInvalidValue;
    k_resample<T><<<grid_for((size_t)res * res * res, kResampleThreads, sms), kResampleThreads, 0, s>>>(out, lg, src, src_res);
    return cudaGetLastError();
}
cudaError_t launch_resample(float* out, int res, const float* src, int src_res, int sms, cudaStream_t s) {
    return resample_t(out, res, src, src_res, sms, s);
}
cudaError_t launch_resample(float* out, int res, const __half* src, int src_res, int sms, cudaStream_t s) {
    return resample_t(out, res, src, src_res, sms, s);
}
cudaError_t launch_interleave_mip_tr(const float* mips, const float* trs, float2* out, int sms, cudaStream_t s) {
    k_interleave_mip_tr<<<sms * 8, 256, 0, s>>>(mips, trs, out);
    return cudaGetLastError();
}
cudaError_t launch_pair_padded(const float* mips_pad, const float* trs_pad, float2* out, cudaStream_t s) {
    k_pair_padded<<<(kPadLevelFloats + 255) / 256, 256, 0, s>>>(mips_pad, trs_pad, out);
    return cudaGetLastError();
}
cudaError_t launch_pad_levels(const float* l8, const float* l4, const float* l2, bool clamp, float* out,
                              cudaStream_t s) {
    k_pad_levels<<<dim3(1, 3), 256, 0, s>>>(l8, l4, l2, clamp ? 1 : 0, out);
    return cudaGetLastError();
}
static unsigned coarse_columns(int R) {   // blocks of k_occ_bricks
    const unsigned nc = (unsigned)(((R + 7) >> 3) + 3) >> 2;
    return nc * nc;
}
template <class T>
static cudaError_t scan_grid_t(const T* d, const OccJob& job, int* stats, int sms, cudaStream_t s) {
    ScanJobs J{};
    J.job[0] = job;
    const int rows = job.R * job.R, need = (rows + kScanThreads / 32 - 1) / (kScanThreads / 32);
    k_scan_rows<T><<<std::min(need, sms * kScanBlocks), kScanThreads, 0, s>>>(d, J, stats);
    k_occ_bricks<<<coarse_columns(job.R), 512, 0, s>>>(J);
    return cudaGetLastError();
}
cudaError_t launch_scan_grid(const float* d, const OccJob& job, int* stats, int sms, cudaStream_t s) {
    return scan_grid_t(d, job, stats, sms, s);
}
cudaError_t launch_scan_grid(const __half* d, const OccJob& job, int* stats, int sms, cudaStream_t s) {
    return scan_grid_t(d, job, stats, sms, s);
}
cudaError_t launch_scan_levels(const OccJob* job, int count, int sms, cudaStream_t s) {
    if (count < 1 || count > kMaxOccJobs) return cudaErrorInvalidValue;
    ScanJobs J{};
    int need = 0;
    unsigned columns = 0;
    for (int i = 0; i < count; ++i) {
        J.job[i] = job[i];
        need = std::max(need, (job[i].R * job[i].R + kScanThreads / 32 - 1) / (kScanThreads / 32));
        columns = std::max(columns, coarse_columns(job[i].R));
    }
    k_scan_rows<float><<<dim3(std::min(need, sms * kScanBlocks), count), kScanThreads, 0, s>>>(nullptr, J, nullptr);
    k_occ_bricks<<<dim3(columns, count), 512, 0, s>>>(J);
    return cudaGetLastError();
}
cudaError_t launch_pad_pyramid(const float* mips, float2* mips_tr, int sms, cudaStream_t s) {
    k_pad_pyramid<<<grid_for(kTrPadTexels, 256, sms), 256, 0, s>>>(mips, mips_tr);
    return cudaGetLastError();
}
cudaError_t launch_tr_levels(float* trs, const float* mips, const float2* mips_tr, const uint8_t* mip_occ,
                             const TrArgs& args, cudaStream_t s) {
    k_tr_levels<<<tr_first_block(0) + tr_blocks(0), kTrThreads, 0, s>>>(trs, mips, mips_tr, mip_occ, args);
    return cudaGetLastError();
}
cudaError_t set_halton_permutations(const uint32_t perm[28]) {
    std::vector<float4> h(kHgSamples);
    for (uint32_t k = 0; k < (uint32_t)kHgSamples; ++k)
        h[k] = make_float4(scrambled_radical_inverse(2, perm, k), scrambled_radical_inverse(3, perm + 2, k),
                           scrambled_radical_inverse(5, perm + 5, k), scrambled_radical_inverse(11, perm + 17, k));
    return cudaMemcpyToSymbol(d_halton, h.data(), kHgSamples * sizeof(float4));
}
cudaError_t launch_hg_lut(float* lut, float g, uint32_t seed, cudaStream_t s) {
    k_hg_lut<<<dim3(kLut / 128, kLut), 128, 0, s>>>(lut, g, seed);
    return cudaGetLastError();
}
cudaError_t launch_baked_tr(float* out, const VolumeDev& v, int bake_res, float alpha, const float L[3], uint32_t seed,
                            int replicate, int sms, cudaStream_t s) {
    int64_t total = (int64_t)bake_res * bake_res * bake_res;
    // bounded chunks keep every launch short
    const int64_t chunk = (int64_t)1 << 26;
    const bool grows = v.max_density * alpha > 0.0f && v.tr_scale > 0.0f;   // every step's length is positive
    for (int64_t first = 0; first < total; first += chunk) {
        int64_t cnt = total - first < chunk ? total - first : chunk;
        const int grid = grid_for((size_t)cnt, 128, sms);
        const f3 l = mk3(L[0], L[1], L[2]);
        auto kernel = v.density_h ? (grows ? k_baked_tr<__half, true> : k_baked_tr<__half, false>)
                                  : (grows ? k_baked_tr<float, true> : k_baked_tr<float, false>);
        kernel<<<grid, 128, 0, s>>>(out, v, bake_res, alpha, l, seed, replicate, first, cnt);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace mrp
