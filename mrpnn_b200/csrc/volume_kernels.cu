// volume_kernels.cu -- volume ingest and per-volume resources on the GPU:
// synthetic fBm generation, the 9-level density pyramid, the majorant, the
// empty-space occupancy bricks, the transmittance (TR) mips, the HG phase LUT
// and the baked NEE transmittance grid.
//
// The reference builds the pyramid on the CPU (VolumeRender::Update,
// core/volume.cu:1474-1515) and the TR mips / LUT / baked TR with legacy
// texture + surface references (core/volume.cu:1322-1400, 1535-1696).  Here
// every resource is a plain z-fastest fp32 array in HBM produced by one
// kernel launch per level, on the volume's stream.
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
template <class T>
__global__ void k_resample(float* __restrict__ out, int res, const T* __restrict__ src, int src_res) {
    size_t n = (size_t)res * res * res;
    float sr = (float)src_res;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        int k = (int)(i % res), j = (int)((i / res) % res), q = (int)(i / ((size_t)res * res));
        float u = (float)(((double)q + 0.5) / res), v = (float)(((double)j + 0.5) / res),
              w = (float)(((double)k + 0.5) / res);
        float px = fs(fm(u, sr), 0.5f), py = fs(fm(v, sr), 0.5f), pz = fs(fm(w, sr), 0.5f);
        int x = (int)floorf(px), y = (int)floorf(py), z = (int)floorf(pz);
        float wx = fs(px, (float)x), wy = fs(py, (float)y), wz = fs(pz, (float)z);
        float a = lerp(lerp(cpu_fetch(src, src_res, x, y, z), cpu_fetch(src, src_res, x, y, z + 1), wz),
                       lerp(cpu_fetch(src, src_res, x, y + 1, z), cpu_fetch(src, src_res, x, y + 1, z + 1), wz), wy);
        float b = lerp(lerp(cpu_fetch(src, src_res, x + 1, y, z), cpu_fetch(src, src_res, x + 1, y, z + 1), wz),
                       lerp(cpu_fetch(src, src_res, x + 1, y + 1, z), cpu_fetch(src, src_res, x + 1, y + 1, z + 1), wz), wy);
        out[i] = lerp(a, b, wx);
    }
}

// ---------------------------------------------------------------------------
// max density (the delta-tracking majorant), floored at the reference's
// default 1e-5 (core/volume.hpp:104).  Densities are compared as int bits,
// which orders non-negative floats; negative (SDF) values never win.
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_max_density(const T* __restrict__ d, size_t n, int* __restrict__ out_bits) {
    float m = 0.00001f;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        m = fmaxf(m, ldg_f(d + i));
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out_bits, __float_as_int(m));
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

// One warp per grid row (x, y): the lanes scan z, the warp keeps the bounds
// of the nonzero voxels it saw and adds them with six atomics at the end.
template <class T>
__global__ void k_nonzero_bounds(const T* __restrict__ d, int R, int* __restrict__ out6) {
    const int lane = threadIdx.x & 31;
    const long long warps = (long long)gridDim.x * (blockDim.x / 32);
    int lo[3] = {R, R, R}, hi[3] = {-1, -1, -1};
    for (long long row = blockIdx.x * (long long)(blockDim.x / 32) + threadIdx.x / 32; row < (long long)R * R;
         row += warps) {
        const T* p = d + row * R;
        int zlo = R, zhi = -1;
        for (int z = lane; z < R; z += 32)
            if (ldg_f(p + z) != 0.0f) { zlo = min(zlo, z); zhi = max(zhi, z); }
        zlo = __reduce_min_sync(0xffffffffu, zlo);
        zhi = __reduce_max_sync(0xffffffffu, zhi);
        if (zhi >= 0) {
            const int x = (int)(row / R), y = (int)(row % R);
            lo[0] = min(lo[0], x); hi[0] = max(hi[0], x);
            lo[1] = min(lo[1], y); hi[1] = max(hi[1], y);
            lo[2] = min(lo[2], zlo); hi[2] = max(hi[2], zhi);
        }
    }
    if (lane == 0 && hi[0] >= 0) {
        for (int a = 0; a < 3; ++a) {
            atomicMin(out6 + a, lo[a]);
            atomicMax(out6 + 3 + a, hi[a]);
        }
    }
}

// ---------------------------------------------------------------------------
// Occupancy bricks for exact empty-space skipping in the first-hit march.
// Brick b covers voxels [b*B, b*B + B) per axis.  A trilinear fetch whose
// base voxel lies in brick b reads voxels base..base+1, i.e. at most one
// voxel past the brick; the brick is marked occupied when any voxel in
// [b*B - 1, b*B + B + 1] holds a non-zero value, one voxel more on each
// side than the fetch needs, so that a base voxel found from a coordinate
// that may be off by less than one voxel still picks a brick whose apron
// holds the whole footprint.  A zero brick therefore guarantees Density() ==
// 0 exactly for every sample whose base voxel is in it or within one voxel
// of it (border texels are 0 by addressing).
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_occupancy(const T* __restrict__ d, int R, int shift, int nb, uint8_t* __restrict__ occ) {
    int total = nb * nb * nb;
    for (int b = blockIdx.x; b < total; b += gridDim.x) {
        int bz = b % nb, by = (b / nb) % nb, bx = b / (nb * nb);
        int B = 1 << shift;
        int x0 = bx * B - 1, y0 = by * B - 1, z0 = bz * B - 1;
        int span = B + 3;
        int any = 0;
        for (int t = threadIdx.x; t < span * span * span && !any; t += blockDim.x) {
            int z = z0 + t % span, y = y0 + (t / span) % span, x = x0 + t / (span * span);
            if ((unsigned)x < (unsigned)R && (unsigned)y < (unsigned)R && (unsigned)z < (unsigned)R)
                any |= ldg_f(d + ((size_t)x * R + y) * R + z) != 0.0f;
        }
        any = __syncthreads_or(any);
        if (threadIdx.x == 0) occ[b] = any ? 1 : 0;
    }
}

// Coarse bricks of 4^3 occupancy bricks (edge 4B): coarse brick C is empty
// when the 64 bricks 4C..4C+3 per axis are.  Their aprons together cover
// voxels [4CB - 1, 4CB + 4B + 1], the coarse brick's own apron, so a zero
// coarse brick carries the same guarantee as a zero brick, over its span.
__global__ void k_occupancy_coarse(const uint8_t* __restrict__ occ, int nb, int nc, uint8_t* __restrict__ out) {
    const int total = nc * nc * nc;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < total; c += gridDim.x * blockDim.x) {
        const int cz = c % nc, cy = (c / nc) % nc, cx = c / (nc * nc);
        int any = 0;
        for (int k = 0; k < 64 && !any; ++k) {
            const int x = 4 * cx + k / 16, y = 4 * cy + (k / 4) % 4, z = 4 * cz + k % 4;
            if (x < nb && y < nb && z < nb) any = occ[(x * nb + y) * nb + z];
        }
        out[c] = any ? 1 : 0;
    }
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
// nonzero voxels.
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
// Padded copy of mip lv + 1 (edge n = 128 >> lv): (n + 2)^3 floats, texel
// (x, y, z) at ((x + 1) P + y + 1) P + z + 1 with P = n + 2, zeros around.
__host__ __device__ constexpr int tr_pad_off(int lv) {
    int o = 0;
    for (int l = 0; l < lv; ++l) { const int p = (128 >> l) + 2; o += p * p * p; }
    return o;
}
static_assert(tr_pad_off(kTrLevels) == (int)kTrPadFloats, "padded pyramid size");
__global__ void k_pad_pyramid(const float* __restrict__ mips, float* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < (int)kTrPadFloats; i += gridDim.x * blockDim.x) {
        int lv = 0;
        while (lv + 1 < kTrLevels && i >= tr_pad_off(lv + 1)) ++lv;
        const int n = 128 >> lv, P = n + 2, j = i - tr_pad_off(lv);
        const int x = j / (P * P) - 1, y = (j / P) % P - 1, z = j % P - 1;
        out[i] = fetch_border(mips + mip_offset(lv + 1), n, x, y, z);
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
MRP_D float tr_march(const float* __restrict__ pad, const uint8_t* __restrict__ occ, f3 p, f3 d, int first, int last) {
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
        const float* b = pad + ((x * P + y) * P + z - kBase);
        const float c00 = lerp_w(__ldg(b), __ldg(b + 1), wz, oz), c01 = lerp_w(__ldg(b + P), __ldg(b + P + 1), wz, oz);
        const float c10 = lerp_w(__ldg(b + P * P), __ldg(b + P * P + 1), wz, oz),
                    c11 = lerp_w(__ldg(b + P * P + P), __ldg(b + P * P + P + 1), wz, oz);
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
MRP_D void tr_voxel(float* __restrict__ trs, const float* __restrict__ mips, const float* __restrict__ mips_tr,
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
                                                          const float* __restrict__ mips_tr,
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
// sample_hg's vector only x = cos and y = -sin sin(phi) enter the dot
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
        const float sdotl = fa(fm(dir.x, cost), fm(dir.y, -fm(sint, sinf(phi))));
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
        const float st_ = sinf(theta), ct = cosf(theta), sp = sinf(phi), cp = cosf(phi);
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
// turn for every sample, 4.19 ms this way (the same bits).
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
// remaining steps only use up draws that nobody reads.  (Needs t to grow,
// smax > 0 and tr_scale > 0; the caller opens the span otherwise.)
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
template <class DT>
__global__ void __launch_bounds__(128) k_baked_tr(float* __restrict__ out, const __grid_constant__ VolumeDev v,
                                                  int bake_res, float alpha, f3 L, uint32_t seed, int replicate,
                                                  int64_t first, int64_t count) {
    float rf = (float)bake_res;
    const bool grows = v.max_density * alpha > 0.0f && v.tr_scale > 0.0f;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < count; q += (int64_t)gridDim.x * blockDim.x) {
        int64_t vi = first + q;
        int x = (int)(vi / ((int64_t)bake_res * bake_res)), y = (int)((vi / bake_res) % bake_res), z = (int)(vi % bake_res);
        f3 uv = div(adds(mk3((float)x, (float)y, (float)z), 0.5f), rf);
        f3 p = subs(uv, 0.5f);
        uint32_t hi = (uint32_t)(vi >> 32) * 8u;
        const float md = ray_box_distance(p, L);
        const BoxSpan span = grows ? nonzero_span(v, p, L) : BoxSpan{0.0f, 3.0e38f};
        float res;
        if (replicate) {
            Stream st(kBakeStream, (uint32_t)vi, hi, 0, seed);
            res = transmittance_span<DT>(v, st, p, L, md, alpha, span);
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
                acc = fa(acc, transmittance_span<DT>(v, st, p, L, md, alpha, span));
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
cudaError_t launch_resample(float* out, int res, const float* src, int src_res, int sms, cudaStream_t s) {
    k_resample<float><<<grid_for((size_t)res * res * res, 256, sms), 256, 0, s>>>(out, res, src, src_res);
    return cudaGetLastError();
}
cudaError_t launch_resample(float* out, int res, const __half* src, int src_res, int sms, cudaStream_t s) {
    k_resample<__half><<<grid_for((size_t)res * res * res, 256, sms), 256, 0, s>>>(out, res, src, src_res);
    return cudaGetLastError();
}
cudaError_t launch_max_density(const float* d, size_t n, int* out_bits, int sms, cudaStream_t s) {
    k_max_density<float><<<grid_for(n, 256, sms), 256, 0, s>>>(d, n, out_bits);
    return cudaGetLastError();
}
cudaError_t launch_max_density(const __half* d, size_t n, int* out_bits, int sms, cudaStream_t s) {
    k_max_density<__half><<<grid_for(n, 256, sms), 256, 0, s>>>(d, n, out_bits);
    return cudaGetLastError();
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
template <class T>
static cudaError_t nonzero_bounds_t(const T* d, int R, int* out6, int sms, cudaStream_t s) {
    long long rows = (long long)R * R;
    int blocks = (int)((rows + 7) / 8 < sms * 16 ? (rows + 7) / 8 : sms * 16);
    k_nonzero_bounds<T><<<blocks, 256, 0, s>>>(d, R, out6);
    return cudaGetLastError();
}
cudaError_t launch_nonzero_bounds(const float* d, int R, int* out6, int sms, cudaStream_t s) {
    return nonzero_bounds_t(d, R, out6, sms, s);
}
cudaError_t launch_nonzero_bounds(const __half* d, int R, int* out6, int sms, cudaStream_t s) {
    return nonzero_bounds_t(d, R, out6, sms, s);
}
template <class T>
static cudaError_t occupancy_t(const T* d, int R, int shift, int nb, uint8_t* occ, int sms, cudaStream_t s) {
    int total = nb * nb * nb;
    k_occupancy<T><<<total < sms * 16 ? total : sms * 16, 256, 0, s>>>(d, R, shift, nb, occ);
    return cudaGetLastError();
}
cudaError_t launch_occupancy(const float* d, int R, int shift, int nb, uint8_t* occ, int sms, cudaStream_t s) {
    return occupancy_t(d, R, shift, nb, occ, sms, s);
}
cudaError_t launch_occupancy(const __half* d, int R, int shift, int nb, uint8_t* occ, int sms, cudaStream_t s) {
    return occupancy_t(d, R, shift, nb, occ, sms, s);
}
cudaError_t launch_occupancy_coarse(const uint8_t* occ, int nb, uint8_t* coarse, int sms, cudaStream_t s) {
    const int nc = (nb + 3) / 4, total = nc * nc * nc;
    k_occupancy_coarse<<<grid_for((size_t)total, 128, sms), 128, 0, s>>>(occ, nb, nc, coarse);
    return cudaGetLastError();
}
cudaError_t launch_pad_pyramid(const float* mips, float* mips_tr, int sms, cudaStream_t s) {
    k_pad_pyramid<<<grid_for(kTrPadFloats, 256, sms), 256, 0, s>>>(mips, mips_tr);
    return cudaGetLastError();
}
cudaError_t launch_tr_levels(float* trs, const float* mips, const float* mips_tr, const uint8_t* mip_occ,
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
    for (int64_t first = 0; first < total; first += chunk) {
        int64_t cnt = total - first < chunk ? total - first : chunk;
        const int grid = grid_for((size_t)cnt, 128, sms);
        const f3 l = mk3(L[0], L[1], L[2]);
        if (v.density_h) k_baked_tr<__half><<<grid, 128, 0, s>>>(out, v, bake_res, alpha, l, seed, replicate, first, cnt);
        else k_baked_tr<float><<<grid, 128, 0, s>>>(out, v, bake_res, alpha, l, seed, replicate, first, cnt);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace mrp
