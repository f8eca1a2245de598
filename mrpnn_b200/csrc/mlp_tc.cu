// mlp_tc.cu -- the MRPNN network (RadiancePredictInternal,
// core/radiancePredict.cu:301-422) on the 5th-generation tensor cores.
//
// Layout of the work.  A persistent kernel with one CTA per SM holds every
// layer's weights in shared memory as UMMA operand images (K-major, no
// swizzle: 8-row x 16-byte core matrices).  Three groups of 128 threads (two
// for coloured albedos) each own one 128-pixel tile at a time; thread t of a
// group owns pixel row t of its tile and TMEM lane t.  Per layer step the
// group writes its A rows (activations, rounded to BF16 or quantised to
// FP8-E4M3) to shared memory, an elected thread a layer issues tcgen05.mma into
// the group's TMEM columns and commits to an mbarrier, and every thread reads its
// row of the FP32 accumulator back with tcgen05.ld for the epilogue (bias,
// ReLU, residuals, gates), all in FP32 on the CUDA cores.  The SE gate MLPs,
// pooling, the LSEFin gate and the last 16->1 layer stay in FP32.
//
// What bounds it: the latency of each tile's chain of dependent steps, so the
// tiles in flight on an SM decide.  Three instead of two need a group's state
// in 160 instead of 256 TMEM columns (residuals where the accumulators go,
// comb where LC0's accumulator goes) and a thread's in 168 registers instead
// of 248 (LC0..LX rows made 32 values at a time); the element-wise work in
// register pairs (f32x2) takes 13 % of the instructions away.  BF16 network of
// a 1920 x 1080 frame (966 K hits): 1.44 -> 1.10 ms, the same bits.
//
// Layers (58): per SE block three branch layers w x w (main widths 8, 8, 16,
// 16, 16, 32, 32, 32; direct-illumination 4 x 8), the three final 32x32 and
// 8x8 layers, then LC0 128x128, LC1 64x128, LC2 32x64, LX 16x32, LX0..LX11
// 16x16.  N and K are padded to the MMA granularity with zeros.
#include <cmath>
#include <cstring>
#include <vector>

#include <cuda_fp16.h>

#include "kernels.h"
#include "mlp_tc.h"
#include "tc_ptx.cuh"

namespace mrp {

// ---------------------------------------------------------------------------
// layer table (shared by the host packer and the kernel)
// ---------------------------------------------------------------------------
constexpr int kLayers = 58;
// main SE block widths (kMainW) and packed fp32 offsets, usable at run time in device code
__host__ __device__ constexpr int mw(int k) { return k < 2 ? 8 : k < 5 ? 16 : 32; }
__host__ __device__ constexpr int mblk_off(int k) { int o = 0; for (int i = 0; i < k; ++i) o += 64 + 24 + 3 * (mw(i) * mw(i) + mw(i)); return o; }
static_assert(mblk_off(8) == kMainFinalOff, "block offsets");
constexpr int kL81 = 24, kLD41 = 39, kLC0 = 42, kLC1 = 43, kLC2 = 44, kLX = 45, kLX0 = 46;
__host__ __device__ constexpr int layer_n(int i) {
    return i < 24 ? mw(i / 3) : i < 27 ? 32 : i < 42 ? 8 : i == kLC0 ? 128 : i == kLC1 ? 64 : i == kLC2 ? 32 : 16;
}
__host__ __device__ constexpr int layer_k(int i) {
    return i < 24 ? mw(i / 3) : i < 27 ? 32 : i < 42 ? 8 : i == kLC0 ? 128 : i == kLC1 ? 128 : i == kLC2 ? 64 :
           i == kLX ? 32 : 16;
}
__host__ __device__ constexpr int pad_to(int x, int m) { return (x + m - 1) / m * m; }
// operand element bytes: 2 (BF16) or 1 (E4M3); K granularity 16 / 32 elements
__host__ __device__ constexpr int kpad(int i, int eb) { return pad_to(layer_k(i), eb == 2 ? 16 : 32); }
__host__ __device__ constexpr int npad(int i) { return pad_to(layer_n(i), 16); }
__host__ __device__ constexpr int layer_bytes(int i, int eb) { return npad(i) * kpad(i, eb) * eb; }
__host__ __device__ constexpr int layer_off(int i, int eb) {
    int o = 0;
    for (int j = 0; j < i; ++j) o += layer_bytes(j, eb);
    return o;
}
__host__ __device__ constexpr int image_bytes(int eb) { return layer_off(kLayers, eb); }
// FP8 weight scales: one per output channel, layer i's at scale_off(i)
__host__ __device__ constexpr int scale_off(int i) {
    int o = 0;
    for (int j = 0; j < i; ++j) o += npad(j);
    return o;
}
constexpr int kScaleCount = scale_off(kLayers);
// The fp32 constants the CUDA-core parts read, packed for shared memory:
// FP8 weight scales, layer biases (both indexed by scale_off), the 12 SE gate
// MLPs (input-major: 8 x 8, then 8 x 3 padded to 8 x 4), LSEFin1 / LSEFin2,
// LGGS and the 16 -> 1 head.
constexpr int kAuxSEBlock = 96;
constexpr int kAuxScale = 0, kAuxBias = kScaleCount, kAuxSE = 2 * kScaleCount, kAuxLSE1 = kAuxSE + 12 * kAuxSEBlock,
              kAuxLSE2 = kAuxLSE1 + 1200, kAuxLGGSW = kAuxLSE2 + 96, kAuxLGGSB = kAuxLGGSW + 24,
              kAuxLX12W = kAuxLGGSB + 8, kAuxLX12B = kAuxLX12W + 16, kAuxCount = (kAuxLX12B + 1 + 3) / 4 * 4;
// fp32 weight / bias of layer i in the packed fp32 layout (common.cuh)
__host__ __device__ constexpr int layer_w32(int i) {
    return i < 24 ? mblk_off(i / 3) + 88 + (i % 3) * (mw(i / 3) * mw(i / 3) + mw(i / 3))
         : i < 27 ? kMainFinalOff + (i - 24) * (1024 + 32)
         : i < 39 ? di_block_off((i - 27) / 3) + 88 + ((i - 27) % 3) * 72
         : i < 42 ? kDiFinalOff + (i - 39) * 72
         : i == kLC0 ? kLC0W : i == kLC1 ? kLC1W : i == kLC2 ? kLC2W : i == kLX ? kLXW : lxw(i - kLX0);
}
__host__ __device__ constexpr int layer_b32(int i) { return layer_w32(i) + layer_n(i) * layer_k(i); }
static_assert(layer_b32(kLC0) == kLC0B && layer_b32(kLX0 + 11) == lxb(11), "layer table");
static_assert(image_bytes(2) <= 110 * 1024, "BF16 weight image must fit shared memory");
static_assert(kAuxBias % 4 == 0 && kAuxSE % 4 == 0 && kAuxLSE1 % 4 == 0 && kAuxLSE2 % 4 == 0 && kAuxSEBlock % 4 == 0,
              "constants read as float4 start on 16-byte boundaries");

// Byte offset of element (row m, k) in a K-major no-swizzle operand tile of
// padded width Kp: 8-row groups SBO = Kp*eb*8 bytes apart, 16-byte K chunks
// 128 bytes apart, rows of a core matrix 16 bytes apart.
__host__ __device__ constexpr int op_off(int m, int k, int kp, int eb) {
    return (m / 8) * (kp * eb * 8) + (k * eb / 16) * 128 + (m % 8) * 16 + (k * eb) % 16;
}

// ---------------------------------------------------------------------------
// host: operand images
// ---------------------------------------------------------------------------
static uint16_t bf16_bits(float f) {   // round to nearest even
    uint32_t u;
    std::memcpy(&u, &f, 4);
    if ((u & 0x7F800000u) == 0x7F800000u) return (uint16_t)(u >> 16 | ((u & 0xFFFF) ? 0x40 : 0));
    u += 0x7FFFu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}
// E4M3 (bias 7, no infinities, max 448), round to nearest even, saturating.
static uint8_t e4m3_bits(float f) {
    uint8_t s = std::signbit(f) ? 0x80 : 0;
    double a = std::fabs((double)f);
    if (!(a == a)) return 0x7F;
    if (a >= 448.0) return s | 0x7E;
    if (a < std::ldexp(1.0, -10)) return s;   // below half the smallest subnormal
    int e;
    std::frexp(a, &e);                        // a = m * 2^e, m in [0.5, 1)
    int ex = e - 1;                           // a in [2^ex, 2^(ex+1))
    if (ex < -6) ex = -6;                     // subnormal range shares 2^-6 * 0.mmm
    double q = std::ldexp(1.0, ex - 3);       // quantum of 3 mantissa bits
    double n = std::nearbyint(a / q);         // ties to even (default rounding)
    double v = n * q;
    if (v >= 448.0) return s | 0x7E;
    if (v == 0) return s;
    int vex;
    std::frexp(v, &vex);
    vex -= 1;
    if (vex < -6) return s | (uint8_t)(v / std::ldexp(1.0, -9));   // subnormal: mantissa / 8 * 2^-6
    uint8_t mant = (uint8_t)(v / std::ldexp(1.0, vex) * 8.0 - 8.0);
    return s | (uint8_t)((vex + 7) << 3) | mant;
}

static cudaError_t upload_layer_descs();
cudaError_t tc_prepare_weights(const float* w32, TcWeights& w) {
    std::vector<uint8_t> img16(image_bytes(2), 0), img8(image_bytes(1), 0);
    // FP8: each output channel (weight row) scaled by its own amax / 448
    std::vector<float> scales(kScaleCount, 1.0f);
    for (int i = 0; i < kLayers; ++i) {
        int n = layer_n(i), k = layer_k(i);
        const float* W = w32 + layer_w32(i);   // [n][k], row-major (Out, In)
        for (int r = 0; r < n; ++r) {
            float amax = 0.0f;
            for (int c = 0; c < k; ++c) amax = std::fmax(amax, std::fabs(W[r * k + c]));
            float s = amax > 0 ? amax / 448.0f : 1.0f;
            scales[scale_off(i) + r] = s;
            for (int c = 0; c < k; ++c) {
                uint16_t b = bf16_bits(W[r * k + c]);
                std::memcpy(&img16[layer_off(i, 2) + op_off(r, c, kpad(i, 2), 2)], &b, 2);
                img8[layer_off(i, 1) + op_off(r, c, kpad(i, 1), 1)] = e4m3_bits(W[r * k + c] / s);
            }
        }
    }
    std::vector<float> aux(kAuxCount, 0.0f);
    for (int i = 0; i < kScaleCount; ++i) aux[kAuxScale + i] = scales[i];
    for (int i = 0; i < kLayers; ++i)
        for (int r = 0; r < layer_n(i); ++r) aux[kAuxBias + scale_off(i) + r] = w32[layer_b32(i) + r];
    for (int b = 0; b < 12; ++b) {
        const float* src = w32 + (b < 8 ? mblk_off(b) : di_block_off(b - 8));
        float* dst = &aux[kAuxSE + kAuxSEBlock * b];
        for (int j = 0; j < 8; ++j) {
            for (int o = 0; o < 8; ++o) dst[8 * j + o] = src[8 * o + j];
            for (int o = 0; o < 3; ++o) dst[64 + 4 * j + o] = src[64 + 8 * o + j];
        }
    }
    // LSEFin1 [16][75] (out, in) stored input-major [75][16]
    for (int o = 0; o < 16; ++o)
        for (int j = 0; j < 75; ++j) aux[kAuxLSE1 + 16 * j + o] = w32[kLSEFin1W + o * 75 + j];
    std::memcpy(&aux[kAuxLSE2], w32 + kLSEFin2W, 96 * sizeof(float));
    std::memcpy(&aux[kAuxLGGSW], w32 + kLGGSW, 24 * sizeof(float));
    std::memcpy(&aux[kAuxLGGSB], w32 + kLGGSB, 8 * sizeof(float));
    std::memcpy(&aux[kAuxLX12W], w32 + kLX12W, 16 * sizeof(float));
    aux[kAuxLX12B] = w32[kLX12B];
    cudaError_t e;
    if (!w.d_aux && (e = mrp::dev_malloc(&w.d_aux, kAuxCount * sizeof(float))) != cudaSuccess) return e;
    if ((e = cudaMemcpy(w.d_aux, aux.data(), kAuxCount * sizeof(float), cudaMemcpyHostToDevice)) != cudaSuccess)
        return e;
    if (!w.d_bf16 && (e = mrp::dev_malloc(&w.d_bf16, img16.size())) != cudaSuccess) return e;
    if (!w.d_fp8 && (e = mrp::dev_malloc(&w.d_fp8, img8.size())) != cudaSuccess) return e;
    if (!w.d_err && (e = mrp::dev_malloc(&w.d_err, sizeof(int))) != cudaSuccess) return e;
    if (!w.d_counter && (e = mrp::dev_malloc(&w.d_counter, sizeof(int))) != cudaSuccess) return e;
    if ((e = cudaMemcpy(w.d_bf16, img16.data(), img16.size(), cudaMemcpyHostToDevice)) != cudaSuccess) return e;
    if ((e = cudaMemcpy(w.d_fp8, img8.data(), img8.size(), cudaMemcpyHostToDevice)) != cudaSuccess) return e;
    if ((e = cudaMemset(w.d_err, 0, sizeof(int))) != cudaSuccess) return e;
    if ((e = upload_layer_descs()) != cudaSuccess) return e;
    w.ready = true;
    return cudaSuccess;
}
cudaError_t tc_ensure_scratch(TcScratch& s) {
    if (s.d) return cudaSuccess;
    cudaError_t e = mrp::dev_malloc(&s.d, 2 * sizeof(int));
    if (e != cudaSuccess) { s.d = nullptr; return e; }
    return cudaMemset(s.d, 0, 2 * sizeof(int));
}
void tc_free_scratch(TcScratch& s) {
    if (s.d) mrp::dev_free(s.d);
    s.d = nullptr;
}

// ---------------------------------------------------------------------------
// device: layer descriptors, group synchronisation, one MMA round
//
// Code size matters here: the whole network runs inside one kernel and its
// groups (two or three) execute different layers at once, so every layer of
// one shape shares one routine and takes its layer index at run time from a
// constant table (instead of one template instance per layer).
// ---------------------------------------------------------------------------
constexpr int kGroupThreads = 128;
constexpr int kTmemCols = 512;
// Groups of a block (tiles in flight on an SM) and their share of tensor
// memory: three where the pixels' albedo is grey, two where it is not, whose
// tail runs once per channel and so keeps comb beside LC0's accumulator.
template <bool COL> constexpr int kGroups = COL ? 2 : 3;
template <bool COL> constexpr int kTmemColsPerGroup = COL ? 256 : 160;
static_assert(kGroups<false> * kTmemColsPerGroup<false> <= kTmemCols && kGroups<true> * kTmemColsPerGroup<true> <= kTmemCols,
              "tensor memory columns");
constexpr uint32_t kWaitLimit = 1u << 22;   // polls before an MMA round is declared lost
constexpr int kABytes = 128 * 128 * 2;      // one group's A buffer (largest: 128 x 128 BF16)

// Where a layer's biases and FP8 scales lie in the shared-memory constants.
// (The tables are read at every step of the chain, so their size counts: with
// 32 bytes a layer 100 001 coloured sets in BF16 took 294 us, with these 276;
// 300 sets in FP8 68 and 64.)
struct LayerDesc { int abias, soff; };
__constant__ LayerDesc c_layer_desc[kLayers];
// What issuing a layer's MMAs takes ([0] BF16, [1] E4M3): the weight image's
// offset and the rows' group stride as the shared-memory descriptor holds
// them (16-byte units), the instruction descriptor, the number of MMAs (32
// bytes of K each).
struct MmaDesc { uint32_t b_off, sbo, idesc, steps; };
__constant__ uint4 c_mma_desc[2][kLayers];

static cudaError_t upload_layer_descs() {
    LayerDesc descs[kLayers];
    MmaDesc mma[2][kLayers];
    for (int i = 0; i < kLayers; ++i) {
        descs[i] = LayerDesc{kAuxBias + scale_off(i), scale_off(i)};
        for (int e = 0; e < 2; ++e) {
            const int eb = e == 0 ? 2 : 1, kb = kpad(i, eb) * eb;   // bytes of a row
            mma[e][i] = MmaDesc{(uint32_t)layer_off(i, eb) >> 4, (uint32_t)(kb * 8) >> 4,
                                tc::instr_desc(128, npad(i), eb == 2 ? tc::kFmtBF16 : tc::kFmtE4M3), (uint32_t)(kb / 32)};
        }
    }
    static_assert(sizeof mma == sizeof c_mma_desc, "one 16-byte constant a layer");
    cudaError_t e = cudaMemcpyToSymbol(c_mma_desc, mma, sizeof mma);
    return e != cudaSuccess ? e : cudaMemcpyToSymbol(c_layer_desc, descs, sizeof descs);
}

// barrier 0 is __syncthreads, 1 to 3 the groups', 4 the split tile's
__device__ __forceinline__ void split_bar() {
    asm volatile("bar.sync %0, %1;" ::"r"(4), "r"(3 * kGroupThreads) : "memory");
}
__device__ __forceinline__ void group_bar(int g) {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "r"(kGroupThreads) : "memory");
}
// The same barrier; true for the whole group when `x` is for one of its threads.
__device__ __forceinline__ bool group_any(int g, bool x) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %3, 0;\n\tbar.red.or.pred p, %1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(r) : "r"(1 + g), "r"(kGroupThreads), "r"((uint32_t)x) : "memory");
    return r != 0;
}

// Per-thread constants of a group, passed by value into the per-block
// routines (a reference would put them in local memory and make every use a
// load).  The mutable part -- mbarrier phase (bit 0) and "a wait timed out"
// (bit 1) -- travels as an int through the calls.
struct Group {
    int g, t;             // group index, thread within the group
    uint32_t a_s;         // A buffer (shared address)
    uint32_t wimg_s;      // weight image (shared address)
    uint32_t mbar_s;      // the group's mbarrier (shared address)
    uint32_t tmem;        // TMEM address of this thread's lane, column 0 of the group
    int* err;
};
constexpr int kStFailed = 2;

// The MMAs of one layer (COUNT = 1) or of the three channels' layers (3; A
// sub-tiles a_stride bytes and accumulators d_stride columns apart), issued
// after all A rows are in shared memory and awaited by the whole group.  The
// first thread of warp q issues layer l0 + q, so three layers' issue runs side
// by side; the mbarrier takes kArrivals arrivals a round.
// SPLIT: all three groups wrote the rows and wait (G.g is a thread's share of
// its row there, and the first group's threads issue).
constexpr int kArrivals = 3;
template <int EB, int COUNT, bool SPLIT = false>
__device__ __noinline__ int mma_round(const Group G, int st, int l0, int a_stride, int d0, int d_stride) {
    static_assert(COUNT == 1 || COUNT == kArrivals, "arrivals a round");
    tc::fence_proxy_async();
    tc::fence_before_sync();
    if (SPLIT) split_bar();
    else group_bar(G.g);
    if ((G.t & 31) == 0 && G.t < 32 * COUNT && (!SPLIT || G.g == 0)) {
        tc::fence_after_sync();
        const int q = G.t >> 5;
        const uint4 m = c_mma_desc[EB == 2 ? 0 : 1][l0 + q];
        // (LBO: 128 bytes between the two 16-byte K chunks of one MMA)
        const uint64_t hi = ((uint64_t)(128 >> 4) << 16) | ((uint64_t)m.y << 32) | (1ull << 46);
        uint64_t ad = hi | (((G.a_s + (uint32_t)(q * a_stride)) >> 4) & 0x3FFFu);
        uint64_t bd = hi | (((G.wimg_s >> 4) + m.x) & 0x3FFFu);
        const uint32_t dc = (G.tmem & 0xFFFFu) + (uint32_t)(d0 + q * d_stride);   // lane 0, the group's columns
#pragma unroll 1
        for (uint32_t s = 0; s < m.w; ++s, ad += 256 >> 4, bd += 256 >> 4) {
            if (EB == 2) tc::mma_bf16(dc, ad, bd, m.z, s > 0);
            else tc::mma_fp8(dc, ad, bd, m.z, s > 0);
        }
#pragma unroll
        for (int i = 0; i < kArrivals / COUNT; ++i) tc::mma_commit_s(G.mbar_s);
    }
    bool done = tc::mbar_wait_s(G.mbar_s, (uint32_t)(st & 1), kWaitLimit);
    st ^= 1;
    if (!done) {
        st |= kStFailed;
        atomicExch(G.err, 1);
    }
    tc::fence_after_sync();
    return st;
}

// Writes this thread's row of an A operand: v[0..n) (zero padded to kp) at
// sub-tile byte offset `off`.  FP8 rows are scaled by 1/s (s = row amax/448),
// returned so the epilogue can undo it.
template <int EB, int N, int KP>
__device__ __forceinline__ float write_row(uint32_t a_s, int off, int row, const float* v) {
    float inv = 1.0f, s = 1.0f;
    if (EB == 1) {
        float amax = 0.0f;
#pragma unroll
        for (int i = 0; i < N; ++i) amax = fmaxf(amax, fabsf(v[i]));
        s = amax > 0.0f ? amax * (1.0f / 448.0f) : 1.0f;
        inv = 1.0f / s;
    }
    constexpr int E = 16 / EB;   // elements per 16-byte chunk
#pragma unroll
    for (int c = 0; c < KP / E; ++c) {
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (EB == 2) {
                int i0 = c * 8 + 2 * q;
                float lo = i0 < N ? v[i0] : 0.0f, hi = i0 + 1 < N ? v[i0 + 1] : 0.0f;
                w[q] = tc::pack_bf16(lo, hi);
            } else {
                int i0 = c * 16 + 4 * q;
                float x0 = i0 < N ? v[i0] * inv : 0.0f, x1 = i0 + 1 < N ? v[i0 + 1] * inv : 0.0f;
                float x2 = i0 + 2 < N ? v[i0 + 2] * inv : 0.0f, x3 = i0 + 3 < N ? v[i0 + 3] * inv : 0.0f;
                w[q] = (uint32_t)tc::pack_e4m3(x0, x1) | ((uint32_t)tc::pack_e4m3(x2, x3) << 16);
            }
        }
        tc::st_shared_v4(a_s + (uint32_t)(off + op_off(row, c * E, KP, EB)), w[0], w[1], w[2], w[3]);
    }
    return s;
}

// Values [32 p, 32 p + 32) of this thread's A row of N (a multiple of 32).
template <int EB, int N>
MRP_D void store_part(const Group& G, int p, const float (&v)[32], float inv) {
    constexpr int E = 16 / EB;
#pragma unroll
    for (int c = 0; c < 32 / E; ++c) {
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (EB == 2) {
                w[q] = tc::pack_bf16(v[8 * c + 2 * q], v[8 * c + 2 * q + 1]);
            } else {
                const int i = 16 * c + 4 * q;
                w[q] = (uint32_t)tc::pack_e4m3(v[i] * inv, v[i + 1] * inv) |
                       ((uint32_t)tc::pack_e4m3(v[i + 2] * inv, v[i + 3] * inv) << 16);
            }
        }
        tc::st_shared_v4(G.a_s + (uint32_t)op_off(G.t, 32 * p + c * E, N, EB), w[0], w[1], w[2], w[3]);
    }
}

MRP_D float sigmoid_d(float o) { return 1.0f / (1.0f + __expf(-o)); }

// relu(D * scale + b) for N columns of layer L (runtime), in place.
// The constants live in shared memory but reach the routines as a generic
// pointer; reading them with shared-space loads (the address converted once
// per access) keeps them off the generic load path, whose results the
// scheduler tracks like global loads.
MRP_D float4 lds4_at(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
MRP_D float4 lds4(const float* p) { return lds4_at((uint32_t)__cvta_generic_to_shared(p)); }
MRP_D float lds1(const float* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}

// Element-wise work, which is what the threads of a row spend their
// instructions on, runs in register pairs.
MRP_D void add_to(float& a0, float& a1, float b0, float b1) { upk2(add2(pk2(a0, a1), pk2(b0, b1)), a0, a1); }
// a = x * g + a
MRP_D void fma_to(float& a0, float& a1, float x0, float x1, f32x2 g) { upk2(fma2(pk2(x0, x1), g, pk2(a0, a1)), a0, a1); }

// Biases and scales start on 16-float boundaries (scale_off), so they are
// read four at a time.  off: first output of the part at hand.
template <int EB, int N>
MRP_D void bias_relu(float* d, int L, float rs, const float* aux, int off = 0) {
    static_assert(N % 4 == 0, "layer widths are multiples of 4");
    const int ab = c_layer_desc[L].abias + off, so = c_layer_desc[L].soff + off;
#pragma unroll
    for (int q = 0; q < N / 4; ++q) {
        const float4 b = lds4(aux + ab + 4 * q);
        f32x2 lo = pk2(d[4 * q], d[4 * q + 1]), hi = pk2(d[4 * q + 2], d[4 * q + 3]);
        if (EB == 1) {
            const float4 w = lds4(aux + kAuxScale + so + 4 * q);
            const f32x2 r2 = pk2(rs, rs);
            lo = fma2(lo, mul2(r2, pk2(w.x, w.y)), pk2(b.x, b.y));
            hi = fma2(hi, mul2(r2, pk2(w.z, w.w)), pk2(b.z, b.w));
        } else {
            lo = add2(lo, pk2(b.x, b.y));
            hi = add2(hi, pk2(b.z, b.w));
        }
        upk2(lo, d[4 * q], d[4 * q + 1]);
        upk2(hi, d[4 * q + 2], d[4 * q + 3]);
#pragma unroll
        for (int i = 0; i < 4; ++i) d[4 * q + i] = fmaxf(d[4 * q + i], 0.0f);
    }
}
// n consecutive constants (16-byte aligned, n a multiple of 4) into registers.
template <int N>
MRP_D void aux_row(const float* aux, int off, float* out) {
#pragma unroll
    for (int q = 0; q < N / 4; ++q) {
        const float4 v = lds4(aux + off + 4 * q);
        out[4 * q] = v.x; out[4 * q + 1] = v.y; out[4 * q + 2] = v.z; out[4 * q + 3] = v.w;
    }
}

// Asynchronous copies into shared memory (dst a shared address).
MRP_D void copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
MRP_D void copy4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
MRP_D void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
constexpr int kStageStride = 3 * kGroupThreads * 16;   // bytes between a thread's chunks in SplitScratch::stage
MRP_D void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Feature sources (rows may be invalid: zeros); FROM is a run-time offset.
// Row-major features are read 16 bytes at a time where the rows start on 16
// bytes: a load of 4 bytes a lane touches 32 lines for 128 bytes.  (100 001
// sets, coloured, BF16: 468 -> 309 us; 300 sets, FP8: 121 -> 87 us.)
struct RowFeatures {           // [n][576] row-major
    const float* x;
    bool valid, vec;
    template <int W>
    MRP_D void load(int c, int from, float* xs) const {
        const float* p = x + c * 192 + from;
        if (valid && vec) {
#pragma unroll
            for (int i = 0; i < W / 4; ++i) {
                const float4 q = __ldg(reinterpret_cast<const float4*>(p) + i);
                xs[4 * i] = q.x; xs[4 * i + 1] = q.y; xs[4 * i + 2] = q.z; xs[4 * i + 3] = q.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < W; ++i) xs[i] = valid ? __ldg(p + i) : 0.0f;
        }
    }
    MRP_D void prefetch(int, int) const {}   // (a line holds several blocks' slices: no gain)
    // the slice as 16-byte chunks, chunk i at slot + i * kStageStride; staged
    // reads them back
    MRP_D void stage(int c, int from, int w, uint32_t slot) const {
        if (!valid) return;
        const float* p = x + c * 192 + from;
        if (vec) {
            for (int i = 0; i < w / 4; ++i) copy16(slot + i * kStageStride, p + 4 * i);
        } else {
            for (int i = 0; i < w; ++i) copy4(slot + (i >> 2) * kStageStride + (i & 3) * 4, p + i);
        }
    }
    template <int W>
    MRP_D void staged(uint32_t slot, float* xs) const {
#pragma unroll
        for (int i = 0; i < W / 4; ++i) {
            float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (valid) q = lds4_at(slot + i * kStageStride);
            xs[4 * i] = q.x; xs[4 * i + 1] = q.y; xs[4 * i + 2] = q.z; xs[4 * i + 3] = q.w;
        }
    }
};
struct TileFeatures {          // FP16 pairs of the staged predictor's tiled layout
    const __half2* x;          // already offset to (r / 32) * 288 * 32 + r % 32
    bool valid;
    template <int W>
    MRP_D void load(int c, int from, float* xs) const {
#pragma unroll
        for (int k = 0; k < W / 2; ++k) {
            const float2 p = valid ? __half22float2(__ldg(x + (c * 96 + (from >> 1) + k) * 32)) : make_float2(0.0f, 0.0f);
            xs[2 * k] = p.x;
            xs[2 * k + 1] = p.y;
        }
    }
    // Asks L2 for the next block's slices, a lane a line (a pair's 32 lanes
    // share it): the features of a large frame come from HBM.  1080p frame
    // 2.480 -> 2.461 ms; two blocks ahead 2.467.
    MRP_D void prefetch(int from, int w) const {
        const int k = threadIdx.x & 31;
        if (!valid || k >= w / 2) return;
#pragma unroll
        for (int c = 0; c < 3; ++c) prefetch_l2(x + (c * 96 + (from >> 1) + k) * 32);
    }
    MRP_D void stage(int c, int from, int w, uint32_t slot) const {
        if (!valid) return;
        for (int k = 0; k < w / 2; ++k)
            copy4(slot + (k >> 2) * kStageStride + (k & 3) * 4, x + (c * 96 + (from >> 1) + k) * 32);
    }
    template <int W>
    MRP_D void staged(uint32_t slot, float* xs) const {
#pragma unroll
        for (int i = 0; i < W / 8; ++i) {
            float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (valid) q = lds4_at(slot + i * kStageStride);
            const float f[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t u = __float_as_uint(f[k]);
                const float2 p = __half22float2(*reinterpret_cast<const __half2*>(&u));
                xs[8 * i + 2 * k] = p.x;
                xs[8 * i + 2 * k + 1] = p.y;
            }
        }
    }
};

// Per-row state that lives in TMEM between blocks.  Of a group's columns the
// main chain has 0..95, 32 a channel, the direct-illumination chain
// 112..159, 16 a channel: a channel's residual lies where the MMAs put its
// accumulator, since it has gone into the A row before the MMA that
// overwrites it is issued.  96..111 hold the LSEFin1 partial sums.  In the
// tail of a grey albedo comb lies in 0..119 until LC0's accumulator (0..127)
// takes its place, the LSEFin1 sums in 128..143 and the residual pairs' state
// in 144..159; of a coloured one comb lies in 136..255, the sums are put into
// 96..111 again before each channel, and the pairs' state follows them there.
constexpr int kColHf = 96, kColDi = 112;
template <bool COL> constexpr int kColComb = COL ? 136 : 0;
template <bool COL> constexpr int kColHfTail = COL ? 96 : 128;
template <bool COL> constexpr int kColA16 = COL ? 96 : 144;
template <int N>
MRP_D void tmem_get(const Group& G, int col, float* out) {
    if constexpr (N == 8) {
        uint32_t r[8];
        tc::tmem_ld8_nowait(G.tmem + col, r);
        tc::tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = __uint_as_float(r[i]);
    } else {
        uint32_t r[N / 16][16];
#pragma unroll
        for (int c = 0; c < N / 16; ++c) tc::tmem_ld16_nowait(G.tmem + col + 16 * c, r[c]);
        tc::tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < N / 16; ++c)
#pragma unroll
            for (int i = 0; i < 16; ++i) out[16 * c + i] = __uint_as_float(r[c][i]);
    }
}
template <int N>
MRP_D void tmem_put(const Group& G, int col, const float* v) {
    if constexpr (N == 8) {
        float t[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) t[i] = v[i];
        tc::tmem_st8(G.tmem + col, t);
    } else {
#pragma unroll
        for (int c = 0; c < N / 16; ++c) {
            float t[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) t[i] = v[16 * c + i];
            tc::tmem_st16(G.tmem + col + 16 * c, t);
        }
    }
}

struct BlockDesc { int w, from, widen, has_prev, l0, col, stride, se_off, pid; };
__constant__ BlockDesc c_blocks[12] = {
    {8, 0, 0, 0, 0, 0, 32, kAuxSE + kAuxSEBlock * 0, 0},      {8, 8, 1, 1, 3, 0, 32, kAuxSE + kAuxSEBlock * 1, 3},
    {16, 16, 0, 1, 6, 0, 32, kAuxSE + kAuxSEBlock * 2, 6},    {16, 32, 0, 1, 9, 0, 32, kAuxSE + kAuxSEBlock * 3, 9},
    {16, 48, 1, 1, 12, 0, 32, kAuxSE + kAuxSEBlock * 4, 12},  {32, 64, 0, 1, 15, 0, 32, kAuxSE + kAuxSEBlock * 5, 15},
    {32, 96, 0, 1, 18, 0, 32, kAuxSE + kAuxSEBlock * 6, 18},  {32, 128, 0, 1, 21, 0, 32, kAuxSE + kAuxSEBlock * 7, 21},
    {8, 160, 0, 0, 27, kColDi, 16, kAuxSE + kAuxSEBlock * 8, 24}, {8, 168, 0, 1, 30, kColDi, 16, kAuxSE + kAuxSEBlock * 9, 27},
    {8, 176, 0, 1, 33, kColDi, 16, kAuxSE + kAuxSEBlock * 10, 30}, {8, 184, 0, 1, 36, kColDi, 16, kAuxSE + kAuxSEBlock * 11, 33},
};

// One SE block over the three channels (SE / SERES + ADD3 / REP3,
// core/radiancePredict.cu:240-294): gate from the slice pools, branch layers
// l0..l0+2 on the tensor cores (accumulators at col, stride columns a channel
// on), then prev <- relu(D + b) + slice (ADD3) or concat(relu(D + b), slice)
// (REP3), left where the accumulator was.
template <int EB, int W, class Src>
__device__ __noinline__ int tc_block(const Group G, int st, const Src src, const float* aux, int b, float g,
                                     float gamma) {
    const BlockDesc bd = c_blocks[b];
    constexpr int KP = pad_to(W, EB == 2 ? 16 : 32);
    constexpr int SUB = 128 * KP * EB;   // bytes of one branch's A sub-tile
    float xs[3][W];                      // the block's feature slice, loaded once
    float p8[8];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        src.template load<W>(c, bd.from, xs[c]);
        float s = 0.0f, m = -10000.0f;
#pragma unroll
        for (int i = 0; i < W; ++i) { s += xs[c][i]; m = fmaxf(m, xs[c][i]); }
        p8[c] = s / (float)W;
        p8[3 + c] = m;
    }
    if (b < 11) src.prefetch(c_blocks[b + 1].from, c_blocks[b + 1].w);
    p8[6] = g;
    p8[7] = gamma;
    // LSEFin1 (75 -> 16) accumulated block by block in TMEM: pool[pid + c] =
    // avg, pool[36 + pid + c] = max; LSEFin1 is stored input-major (the 16
    // weights of input j at kAuxLSE1 + 16 j), outputs in pairs
    {
        float hf[16];
        tmem_get<16>(G, kColHf, hf);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const f32x2 av = pk2(p8[c], p8[c]), mx = pk2(p8[3 + c], p8[3 + c]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 wa = lds4(aux + kAuxLSE1 + 16 * (bd.pid + c) + 4 * q);
                const float4 wm = lds4(aux + kAuxLSE1 + 16 * (36 + bd.pid + c) + 4 * q);
                fma_to(hf[4 * q], hf[4 * q + 1], wa.x, wa.y, av);
                fma_to(hf[4 * q + 2], hf[4 * q + 3], wa.z, wa.w, av);
                fma_to(hf[4 * q], hf[4 * q + 1], wm.x, wm.y, mx);
                fma_to(hf[4 * q + 2], hf[4 * q + 3], wm.z, wm.w, mx);
            }
        }
        tmem_put<16>(G, kColHf, hf);
    }
    f32x2 gate[3];
    {
        float h[8], a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int o = 0; o < 8; ++o) h[o] = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float4 u = lds4(aux + bd.se_off + 8 * j), v = lds4(aux + bd.se_off + 8 * j + 4);
            const f32x2 p = pk2(p8[j], p8[j]);
            fma_to(h[0], h[1], u.x, u.y, p);
            fma_to(h[2], h[3], u.z, u.w, p);
            fma_to(h[4], h[5], v.x, v.y, p);
            fma_to(h[6], h[7], v.z, v.w, p);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float4 u = lds4(aux + bd.se_off + 64 + 4 * j);
            h[j] = fmaxf(h[j], 0.0f);
            fma_to(a[0], a[1], u.x, u.y, pk2(h[j], h[j]));
            a[2] = fmaf(h[j], u.z, a[2]);
        }
#pragma unroll
        for (int o = 0; o < 3; ++o) {
            const float q = sigmoid_d(a[o]);
            gate[o] = pk2(q, q);
        }
    }
    float rs[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float in[W];
        if (bd.has_prev) {
            tmem_get<W>(G, bd.col + c * bd.stride, in);
#pragma unroll
            for (int i = 0; i < W; i += 2) fma_to(in[i], in[i + 1], xs[c][i], xs[c][i + 1], gate[c]);
        } else {
#pragma unroll
            for (int i = 0; i < W; i += 2) upk2(mul2(pk2(xs[c][i], xs[c][i + 1]), gate[c]), in[i], in[i + 1]);
        }
        rs[c] = write_row<EB, W, KP>(G.a_s, c * SUB, G.t, in);
    }
    st = mma_round<EB, 3>(G, st, bd.l0, SUB, bd.col, bd.stride);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float d[W];
        tmem_get<W>(G, bd.col + c * bd.stride, d);
        bias_relu<EB, W>(d, bd.l0 + c, rs[c], aux);
        if (bd.widen) {
            float nv[2 * W];
#pragma unroll
            for (int o = 0; o < W; ++o) { nv[o] = d[o]; nv[W + o] = xs[c][o]; }
            tmem_put<2 * W>(G, bd.col + c * bd.stride, nv);
        } else {
#pragma unroll
            for (int o = 0; o < W; o += 2) add_to(d[o], d[o + 1], xs[c][o], xs[c][o + 1]);
            tmem_put<W>(G, bd.col + c * bd.stride, d);
        }
    }
    tc::tmem_wait_st();
    return st;
}

// Residual pair k of the tail: a += relu(LX(2k+1) relu(LX(2k) a + b) + b),
// a (16 values) kept in TMEM columns kColA16.
template <int EB, bool COL>
__device__ __noinline__ int tc_residual_pair(const Group G, int st, const float* aux, int k) {
    constexpr int KP = EB == 2 ? 16 : 32;
    const int La = kLX0 + 2 * k, Lb = La + 1;
    float a16[16];
    tmem_get<16>(G, kColA16<COL>, a16);
    float r0 = write_row<EB, 16, KP>(G.a_s, 0, G.t, a16);
    st = mma_round<EB, 1>(G, st, La, 0, 64, 0);
    float u[16];
    tmem_get<16>(G, 64, u);
    bias_relu<EB, 16>(u, La, r0, aux);
    float r1 = write_row<EB, 16, KP>(G.a_s, 0, G.t, u);
    st = mma_round<EB, 1>(G, st, Lb, 0, 80, 0);
    float z[16];
    tmem_get<16>(G, 80, z);
    bias_relu<EB, 16>(z, Lb, r1, aux);
#pragma unroll
    for (int i = 0; i < 16; i += 2) add_to(a16[i], a16[i + 1], z[i], z[i + 1]);
    tmem_put<16>(G, kColA16<COL>, a16);
    tc::tmem_wait_st();
    return st;
}

// The tail from LX's accumulator (columns 32..47) on: six residual pairs and
// the 16 -> 1 head.
struct TailOut { float p; int st; };
template <int EB, bool COL>
MRP_D TailOut tc_tail_end(const Group& G, int st, float r, const float* aux) {
    float a16[16];
    tmem_get<16>(G, 32, a16);
    bias_relu<EB, 16>(a16, kLX, r, aux);
    tmem_put<16>(G, kColA16<COL>, a16);
    tc::tmem_wait_st();
#pragma unroll 1
    for (int k = 0; k < 6; ++k) st = tc_residual_pair<EB, COL>(G, st, aux, k);
    tmem_get<16>(G, kColA16<COL>, a16);
    float a = 0.0f;
#pragma unroll
    for (int j = 0; j < 16; ++j) a = fmaf(a16[j], lds1(aux + kAuxLX12W + j), a);
    return TailOut{fmaxf(a + lds1(aux + kAuxLX12B), 0.0f), st};
}

// An A row of N values that come in parts of 32: get(part, v) makes part
// `part`.  FP8 rows need their scale first: with HOLD the row is held
// meanwhile (the coloured form's threads have the registers: one set 119 ->
// 108 us, 100 001 sets 353 -> 345); otherwise it is made twice and never held
// whole.
template <int EB, int N, bool HOLD, class F>
MRP_D float write_parts(const Group& G, F get) {
    constexpr int PARTS = N / 32, KEEP = EB == 1 && HOLD ? PARTS : 1;
    float v[KEEP][32];
    if (EB == 2) {
#pragma unroll
        for (int p = 0; p < PARTS; ++p) {
            get(p, v[0]);
            store_part<EB, N>(G, p, v[0], 1.0f);
        }
        return 1.0f;
    }
    float amax = 0.0f;
#pragma unroll
    for (int p = 0; p < PARTS; ++p) {
        get(p, v[p % KEEP]);
#pragma unroll
        for (int i = 0; i < 32; ++i) amax = fmaxf(amax, fabsf(v[p % KEEP][i]));
    }
    const float s = amax > 0.0f ? amax * (1.0f / 448.0f) : 1.0f, inv = 1.0f / s;
#pragma unroll
    for (int p = 0; p < PARTS; ++p) {
        if (!HOLD) get(p, v[0]);
        store_part<EB, N>(G, p, v[p % KEEP], inv);
    }
    return s;
}

// The tail of one albedo channel (core/radiancePredict.cu:375-419): LSEFin
// gate, LC0 over [comb * gate, LGGS], LC1, LC2, LX, six residual pairs and
// the 16 -> 1 head.  comb (kColComb) and the LSEFin1 sums (kColHfTail) come
// from TMEM.
template <int EB, bool COL>
__device__ __noinline__ TailOut tc_tail(const Group G, int st, const float* aux, float g, float gamma, float s4) {
    float gf[6];
    {
        float h[16];
        tmem_get<16>(G, kColHfTail<COL>, h);
#pragma unroll
        for (int o = 0; o < 16; ++o) {
            float a = h[o];
            a = fmaf(lds1(aux + kAuxLSE1 + 16 * 72 + o), g, a);
            a = fmaf(lds1(aux + kAuxLSE1 + 16 * 73 + o), gamma, a);
            a = fmaf(lds1(aux + kAuxLSE1 + 16 * 74 + o), s4, a);
            h[o] = fmaxf(a, 0.0f);
        }
#pragma unroll
        for (int o = 0; o < 6; ++o) {
            float w[16];
            aux_row<16>(aux, kAuxLSE2 + o * 16, w);
            float a = 0.0f;
#pragma unroll
            for (int j = 0; j < 16; ++j) a = fmaf(h[j], w[j], a);
            gf[o] = sigmoid_d(a);
        }
    }
    // LC0's A row: [comb * gate segment, LGGS (3 -> 8)]
    float r = write_parts<EB, 128, COL>(G, [&](int p, float (&v)[32]) {
        if (p < 3) {
            tmem_get<32>(G, kColComb<COL> + 32 * p, v);
            const f32x2 q = pk2(gf[p], gf[p]);
#pragma unroll
            for (int i = 0; i < 32; i += 2) upk2(mul2(pk2(v[i], v[i + 1]), q), v[i], v[i + 1]);
        } else {
            float e[24];
            tmem_get<16>(G, kColComb<COL> + 96, e);
            tmem_get<8>(G, kColComb<COL> + 112, e + 16);
#pragma unroll
            for (int i = 0; i < 24; ++i) v[i] = e[i] * gf[3 + i / 8];
#pragma unroll
            for (int o = 0; o < 8; ++o) {
                float a = 0.0f;
                a = fmaf(g, lds1(aux + kAuxLGGSW + o * 3), a);
                a = fmaf(gamma, lds1(aux + kAuxLGGSW + o * 3 + 1), a);
                a = fmaf(s4, lds1(aux + kAuxLGGSW + o * 3 + 2), a);
                v[24 + o] = fmaxf(a + lds1(aux + kAuxLGGSB + o), 0.0f);
            }
        }
    });
    st = mma_round<EB, 1>(G, st, kLC0, 0, 0, 0);
    float rn = write_parts<EB, 128, COL>(G, [&](int p, float (&v)[32]) {
        tmem_get<32>(G, 32 * p, v);
        if (p == 0) bias_relu<EB, 32>(v, kLC0, r, aux, 0);
        else if (p == 1) bias_relu<EB, 32>(v, kLC0, r, aux, 32);
        else if (p == 2) bias_relu<EB, 32>(v, kLC0, r, aux, 64);
        else bias_relu<EB, 32>(v, kLC0, r, aux, 96);
    });
    st = mma_round<EB, 1>(G, st, kLC1, 0, 0, 0);
    r = rn;
    rn = write_parts<EB, 64, COL>(G, [&](int p, float (&v)[32]) {
        tmem_get<32>(G, 32 * p, v);
        if (p == 0) bias_relu<EB, 32>(v, kLC1, r, aux, 0);
        else bias_relu<EB, 32>(v, kLC1, r, aux, 32);
    });
    st = mma_round<EB, 1>(G, st, kLC2, 0, 0, 0);
    r = rn;
    rn = write_parts<EB, 32, COL>(G, [&](int, float (&v)[32]) {
        tmem_get<32>(G, 0, v);
        bias_relu<EB, 32>(v, kLC2, r, aux);
    });
    st = mma_round<EB, 1>(G, st, kLX, 0, 32, 0);
    return tc_tail_end<EB, COL>(G, st, rn, aux);
}

// ---------------------------------------------------------------------------
// A tile split over the three groups, for calls of no more tiles than SMs,
// where nothing hides the chain of a tile's dependent steps: three threads a
// row, G.g the channel that a thread takes through the SE blocks and its part
// of the rows behind them (all in the first group's A buffer and columns).
// What they have to tell one another goes through the other groups' A
// buffers.  Every value is made by the operations, in the order, that one
// thread a row uses.  One FP8 tile of 300 sets: 111 k cycles with one thread
// a row, two thirds of them in the SE blocks (9 to 10 k a block of width 32, a
// third of that for its features to arrive; 4 k split, the next block's
// features copied to shared memory meanwhile).  The call 83.5 -> 70 us, and a
// 163 x 97 FP8 frame of four launches 587 -> 528; since there is no loop over
// tiles, around which its state spilled, another 63.6 -> 60.6 and 475 -> 468.
// (With twice as many sets, two tiles in turn an SM, that loop took 127 us, the
// other form 107.)
// ---------------------------------------------------------------------------
struct SplitScratch {
    float4 stage[8][3 * kGroupThreads];   // the threads' slices of the next block (chunk, thread)
    float hf[16][128];                    // LSEFin1 sums
    union {
        float pool[2][6][128];    // slice pools (block parity; average, maximum of a channel)
        float amax[2][3][128];    // behind the blocks, FP8: largest value of a thread's part
    };
};
static_assert(sizeof(SplitScratch) <= 2 * kABytes, "the other groups' A buffers hold it");

template <int EB, int W, class Src>
__device__ __noinline__ int split_block(const Group G, int st, const Src src, const float* aux, SplitScratch* X, int b,
                                        float g, float gamma) {
    const BlockDesc bd = c_blocks[b];
    constexpr int KP = pad_to(W, EB == 2 ? 16 : 32);
    const int c = G.g, col = bd.col + c * bd.stride;
    float (*pool)[128] = X->pool[b & 1];
    // (asked for a block ago)
    float xs[W];
    const uint32_t slot = tc::smem_addr(&X->stage[0][c * kGroupThreads + G.t]);
    copies_wait();
    src.template staged<W>(slot, xs);
    {
        float s = 0.0f, m = -10000.0f;
#pragma unroll
        for (int i = 0; i < W; ++i) { s += xs[i]; m = fmaxf(m, xs[i]); }
        pool[c][G.t] = s / (float)W;
        pool[3 + c][G.t] = m;
    }
    split_bar();
    if (b < 11) src.stage(c, c_blocks[b + 1].from, c_blocks[b + 1].w, slot);
    float p8[8];
#pragma unroll
    for (int i = 0; i < 6; ++i) p8[i] = pool[i][G.t];
    p8[6] = g;
    p8[7] = gamma;
    float gate;
    {
        float h[8], a = 0.0f;
#pragma unroll
        for (int o = 0; o < 8; ++o) h[o] = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float4 u = lds4(aux + bd.se_off + 8 * j), v = lds4(aux + bd.se_off + 8 * j + 4);
            const f32x2 p = pk2(p8[j], p8[j]);
            fma_to(h[0], h[1], u.x, u.y, p);
            fma_to(h[2], h[3], u.z, u.w, p);
            fma_to(h[4], h[5], v.x, v.y, p);
            fma_to(h[6], h[7], v.z, v.w, p);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) a = fmaf(fmaxf(h[j], 0.0f), lds1(aux + bd.se_off + 64 + 4 * j + c), a);
        gate = sigmoid_d(a);
    }
    float rs;
    {
        float in[W];
        const f32x2 q = pk2(gate, gate);
        if (bd.has_prev) {
            tmem_get<W>(G, col, in);
#pragma unroll
            for (int i = 0; i < W; i += 2) fma_to(in[i], in[i + 1], xs[i], xs[i + 1], q);
        } else {
#pragma unroll
            for (int i = 0; i < W; i += 2) upk2(mul2(pk2(xs[i], xs[i + 1]), q), in[i], in[i + 1]);
        }
        rs = write_row<EB, W, KP>(G.a_s, c * 128 * KP * EB, G.t, in);
    }
    // LSEFin1, eight outputs for each of two of a row's threads
    if (c < 2) {
        float hf[8];
#pragma unroll
        for (int o = 0; o < 8; ++o) hf[o] = b == 0 ? 0.0f : X->hf[8 * c + o][G.t];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const f32x2 av = pk2(p8[k], p8[k]), mx = pk2(p8[3 + k], p8[3 + k]);
            const float* wa = aux + kAuxLSE1 + 16 * (bd.pid + k) + 8 * c;
            const float* wm = wa + 16 * 36;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float4 u = lds4(wa + 4 * q), v = lds4(wm + 4 * q);
                fma_to(hf[4 * q], hf[4 * q + 1], u.x, u.y, av);
                fma_to(hf[4 * q + 2], hf[4 * q + 3], u.z, u.w, av);
                fma_to(hf[4 * q], hf[4 * q + 1], v.x, v.y, mx);
                fma_to(hf[4 * q + 2], hf[4 * q + 3], v.z, v.w, mx);
            }
        }
#pragma unroll
        for (int o = 0; o < 8; ++o) X->hf[8 * c + o][G.t] = hf[o];
    }
    st = mma_round<EB, 3, true>(G, st, bd.l0, 128 * KP * EB, bd.col, bd.stride);
    float d[W];
    tmem_get<W>(G, col, d);
    bias_relu<EB, W>(d, bd.l0 + c, rs, aux);
    if (bd.widen) {
        float nv[2 * W];
#pragma unroll
        for (int o = 0; o < W; ++o) { nv[o] = d[o]; nv[W + o] = xs[o]; }
        tmem_put<2 * W>(G, col, nv);
    } else {
#pragma unroll
        for (int o = 0; o < W; o += 2) add_to(d[o], d[o + 1], xs[o], xs[o + 1]);
        tmem_put<W>(G, col, d);
    }
    tc::tmem_wait_st();
    return st;
}

// The row's FP8 scale from what its three threads hold (1 in BF16).
template <int EB>
MRP_D float split_scale(const Group& G, float (&part)[3][128], float amax) {
    if (EB == 2) return 1.0f;
    part[G.g][G.t] = amax;
    split_bar();
    amax = fmaxf(fmaxf(part[0][G.t], part[1][G.t]), part[2][G.t]);
    return amax > 0.0f ? amax * (1.0f / 448.0f) : 1.0f;
}
template <int N>
MRP_D float abs_max(const float* v, float a) {
#pragma unroll
    for (int i = 0; i < N; ++i) a = fmaxf(a, fabsf(v[i]));
    return a;
}
// Values [k, k + N) of this row's A operand of KP (N 8 or a multiple of 16).
template <int EB, int KP, int N>
MRP_D void split_store(const Group& G, int k, const float* v, float inv) {
    if (EB == 2) {
#pragma unroll
        for (int i = 0; i < N; i += 8)
            tc::st_shared_v4(G.a_s + (uint32_t)op_off(G.t, k + i, KP, EB), tc::pack_bf16(v[i], v[i + 1]),
                             tc::pack_bf16(v[i + 2], v[i + 3]), tc::pack_bf16(v[i + 4], v[i + 5]),
                             tc::pack_bf16(v[i + 6], v[i + 7]));
    } else {
        uint32_t w[N / 4];
#pragma unroll
        for (int q = 0; q < N / 4; ++q)
            w[q] = (uint32_t)tc::pack_e4m3(v[4 * q] * inv, v[4 * q + 1] * inv) |
                   ((uint32_t)tc::pack_e4m3(v[4 * q + 2] * inv, v[4 * q + 3] * inv) << 16);
        if constexpr (N == 8) {
            tc::st_shared_v2(G.a_s + (uint32_t)op_off(G.t, k, KP, EB), w[0], w[1]);
        } else {
#pragma unroll
            for (int i = 0; i < N / 16; ++i)
                tc::st_shared_v4(G.a_s + (uint32_t)op_off(G.t, k + 16 * i, KP, EB), w[4 * i], w[4 * i + 1], w[4 * i + 2],
                                 w[4 * i + 3]);
        }
    }
}
// The next layer's A row (N values, relu(D + b) of layer L) from the
// accumulator in columns [0, N), in parts of 16: thread c of a row takes parts
// c, c + 3, ...; returns the row's scale.
template <int EB, int N>
MRP_D float split_relu_row(const Group& G, int L, float r, const float* aux, float (&part)[3][128]) {
    constexpr int MINE = (N / 16 + 2) / 3;
    float v[MINE][16], amax = 0.0f;
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
        const int p = G.g + 3 * i;
        if (p < N / 16) {
            tmem_get<16>(G, 16 * p, v[i]);
            bias_relu<EB, 16>(v[i], L, r, aux, 16 * p);
            if (EB == 1) amax = abs_max<16>(v[i], amax);
        }
    }
    const float s = split_scale<EB>(G, part, amax), inv = 1.0f / s;
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
        const int p = G.g + 3 * i;
        if (p < N / 16) split_store<EB, N, 16>(G, 16 * p, v[i], inv);
    }
    return s;
}

// tc_network of a grey albedo for a split tile; the first group's threads
// return the result.
template <int EB, class Src>
__device__ __noinline__ TailOut split_network(const Group G, int st, const Src src, const float* aux, SplitScratch* X,
                                              float gamma, float g, float s4) {
    const int c = G.g;
    src.stage(c, c_blocks[0].from, c_blocks[0].w, tc::smem_addr(&X->stage[0][c * kGroupThreads + G.t]));
#pragma unroll 1
    for (int b = 0; b < 8; ++b) {
        const int w = c_blocks[b].w;
        if (w == 8) st = split_block<EB, 8>(G, st, src, aux, X, b, g, gamma);
        else if (w == 16) st = split_block<EB, 16>(G, st, src, aux, X, b, g, gamma);
        else st = split_block<EB, 32>(G, st, src, aux, X, b, g, gamma);
    }
    float m[32], e[8], rs;
    {
        constexpr int KP = pad_to(32, EB == 2 ? 16 : 32), SUB = 128 * KP * EB;
        tmem_get<32>(G, 32 * c, m);
        rs = write_row<EB, 32, KP>(G.a_s, c * SUB, G.t, m);
        st = mma_round<EB, 3, true>(G, st, kL81, SUB, 0, 32);
    }
    tmem_get<32>(G, 32 * c, m);
    bias_relu<EB, 32>(m, kL81 + c, rs, aux);
    tmem_put<32>(G, 32 * c, m);
    tc::tmem_wait_st();
#pragma unroll 1
    for (int b = 8; b < 12; ++b) st = split_block<EB, 8>(G, st, src, aux, X, b, g, gamma);
    {
        constexpr int KP = pad_to(8, EB == 2 ? 16 : 32), SUB = 128 * KP * EB;
        tmem_get<8>(G, kColDi + 16 * c, e);
        rs = write_row<EB, 8, KP>(G.a_s, c * SUB, G.t, e);
        st = mma_round<EB, 3, true>(G, st, kLD41, SUB, kColDi, 16);
    }
    tmem_get<8>(G, kColDi + 16 * c, e);
    bias_relu<EB, 8>(e, kLD41 + c, rs, aux);
    tmem_get<32>(G, 32 * c, m);
    // LSEFin: of its six gates a thread needs its channel's two
    float gf[2];
    {
        float h[16];
#pragma unroll
        for (int o = 0; o < 16; ++o) {
            float a = X->hf[o][G.t];
            a = fmaf(lds1(aux + kAuxLSE1 + 16 * 72 + o), g, a);
            a = fmaf(lds1(aux + kAuxLSE1 + 16 * 73 + o), gamma, a);
            a = fmaf(lds1(aux + kAuxLSE1 + 16 * 74 + o), s4, a);
            h[o] = fmaxf(a, 0.0f);
        }
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            float w[16];
            aux_row<16>(aux, kAuxLSE2 + (c + 3 * o) * 16, w);
            float a = 0.0f;
#pragma unroll
            for (int j = 0; j < 16; ++j) a = fmaf(h[j], w[j], a);
            gf[o] = sigmoid_d(a);
        }
    }
    // LC0's A row: a channel's 32 and 8 gated values each, LGGS by the last
    {
        const f32x2 q = pk2(gf[0], gf[0]);
#pragma unroll
        for (int i = 0; i < 32; i += 2) upk2(mul2(pk2(m[i], m[i + 1]), q), m[i], m[i + 1]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) e[i] *= gf[1];
    float lg[8];
#pragma unroll
    for (int o = 0; o < 8; ++o) {
        float a = 0.0f;
        a = fmaf(g, lds1(aux + kAuxLGGSW + o * 3), a);
        a = fmaf(gamma, lds1(aux + kAuxLGGSW + o * 3 + 1), a);
        a = fmaf(s4, lds1(aux + kAuxLGGSW + o * 3 + 2), a);
        lg[o] = fmaxf(a + lds1(aux + kAuxLGGSB + o), 0.0f);
    }
    float r;
    {
        float amax = 0.0f;
        if (EB == 1) amax = abs_max<8>(lg, abs_max<8>(e, abs_max<32>(m, 0.0f)));
        r = split_scale<EB>(G, X->amax[0], amax);
        const float inv = 1.0f / r;
        split_store<EB, 128, 32>(G, 32 * c, m, inv);
        split_store<EB, 128, 8>(G, 96 + 8 * c, e, inv);
        if (c == 2) split_store<EB, 128, 8>(G, 120, lg, inv);
    }
    st = mma_round<EB, 1, true>(G, st, kLC0, 0, 0, 0);
    r = split_relu_row<EB, 128>(G, kLC0, r, aux, X->amax[1]);
    st = mma_round<EB, 1, true>(G, st, kLC1, 0, 0, 0);
    r = split_relu_row<EB, 64>(G, kLC1, r, aux, X->amax[0]);
    st = mma_round<EB, 1, true>(G, st, kLC2, 0, 0, 0);
    r = split_relu_row<EB, 32>(G, kLC2, r, aux, X->amax[1]);
    st = mma_round<EB, 1, true>(G, st, kLX, 0, 32, 0);
    // the 16-wide rest is one thread's work a row
    return c == 0 ? tc_tail_end<EB, false>(G, st, r, aux) : TailOut{0.0f, st};
}

template <int EB, class Src>
MRP_D int run_block(const Group& G, int st, const Src& src, const float* aux, int b, float g, float gamma) {
    const int w = c_blocks[b].w;
    if (w == 8) return tc_block<EB, 8>(G, st, src, aux, b, g, gamma);
    if (w == 16) return tc_block<EB, 16>(G, st, src, aux, b, g, gamma);
    return tc_block<EB, 32>(G, st, src, aux, b, g, gamma);
}

MRP_D float radiance(float p, float s4) { return fmaxf(expf(p) - 1.0f, 0.0f) * s4; }

template <int EB, bool COL, class Src>
MRP_D int tc_network(const Group& G, int st, const Src& src, const float* aux,
                      float gamma, float g, f3 sr, float out[3]) {
    {
        float z[16];
#pragma unroll
        for (int o = 0; o < 16; ++o) z[o] = 0.0f;
        tmem_put<16>(G, kColHf, z);
        tc::tmem_wait_st();
    }
    // main branch, X[0:160], and its three 32x32 finals
#pragma unroll 1
    for (int b = 0; b < 8; ++b) st = run_block<EB>(G, st, src, aux, b, g, gamma);
    float rs_main[3];
    {
        constexpr int KP = pad_to(32, EB == 2 ? 16 : 32), SUB = 128 * KP * EB;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float pv[32];
            tmem_get<32>(G, 32 * c, pv);
            rs_main[c] = write_row<EB, 32, KP>(G.a_s, c * SUB, G.t, pv);
        }
        st = mma_round<EB, 3>(G, st, kL81, SUB, 0, 32);
    }
    // direct-illumination branch, X[160:192], and its 8x8 finals
#pragma unroll 1
    for (int b = 8; b < 12; ++b) st = run_block<EB>(G, st, src, aux, b, g, gamma);
    float rs_di[3];
    {
        constexpr int KP = pad_to(8, EB == 2 ? 16 : 32), SUB = 128 * KP * EB;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float pv[8];
            tmem_get<8>(G, kColDi + 16 * c, pv);
            rs_di[c] = write_row<EB, 8, KP>(G.a_s, c * SUB, G.t, pv);
        }
        st = mma_round<EB, 3>(G, st, kLD41, SUB, kColDi, 16);
    }
    // comb[120] = relu(finals + b): the direct-illumination part behind the
    // main one, once it and the LSEFin1 sums have been read
    float hf[16];
    {
        float e[3][8];
        tmem_get<16>(G, kColHf, hf);
#pragma unroll
        for (int c = 0; c < 3; ++c) tmem_get<8>(G, kColDi + 16 * c, e[c]);
        tmem_put<16>(G, kColHfTail<COL>, hf);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            bias_relu<EB, 8>(e[c], kLD41 + c, rs_di[c], aux);
            tmem_put<8>(G, kColComb<COL> + 96 + 8 * c, e[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float m[32];
        tmem_get<32>(G, 32 * c, m);
        bias_relu<EB, 32>(m, kL81 + c, rs_main[c], aux);
        tmem_put<32>(G, kColComb<COL> + 32 * c, m);
    }
    tc::tmem_wait_st();
    // tail, once per distinct albedo channel (core/radiancePredict.cu:375-419)
    const float srv[3] = {sr.x, sr.y, sr.z};
    float P[3];
#pragma unroll
    for (int ch = 0; ch < (COL ? 3 : 1); ++ch) {
        if (ch == 1 && srv[1] == srv[0]) { P[1] = P[0]; continue; }
        if (ch == 2 && srv[2] == srv[0]) { P[2] = P[0]; continue; }
        if (ch == 2 && srv[2] == srv[1]) { P[2] = P[1]; continue; }
        if (ch > 0) {   // the previous tail's accumulators covered the sums
            tmem_put<16>(G, kColHfTail<COL>, hf);
            tc::tmem_wait_st();
        }
        TailOut t = tc_tail<EB, COL>(G, st, aux, g, gamma, powf(srv[ch], 4.0f));
        st = t.st;
        P[ch] = t.p;
    }
    if (!COL) P[1] = P[2] = P[0];
#pragma unroll
    for (int c = 0; c < 3; ++c) out[c] = radiance(P[c], powf(srv[c], 4.0f));
    return st;
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
struct TcArgs {
    const uint8_t* wimg;        // operand image (global)
    int wimg_bytes;
    const float* aux;           // fp32 constants of the CUDA-core parts (kAux* layout)
    int* err;
    int* tile_counter;
    // inputs: either row-major features [n][576] + gamma, or staged records
    const float* feat;
    bool feat_vec;              // feat on a 16-byte boundary
    const float* gamma;
    int n;
    float g;
    f3 sr;
    float* out3;                // row-major [n][3]
    // staged records: segs[0, nseg), or seg0 alone when segs is null
    const TcSegment* segs;
    int nseg;
    TcSegment seg0;
};

// One tile of `rows` rows: st = eval(features, gamma, g, sr, o) for row t, and,
// with `stores`, its result.
template <bool STAGED, class F>
MRP_D int tile_work(const TcArgs& A, const TcSegment* segs, const int* seg_start, int rows, int tile, int t, bool stores,
                    F eval) {
    int st;
    float o[3];
    if constexpr (STAGED) {
        int q = 0;
        while (tile >= seg_start[q + 1]) ++q;
        const TcSegment* S = segs + q;
        const int r = (tile - seg_start[q]) * rows + t;
        const bool valid = t < rows && r < *S->rec_count;
        const size_t cap = S->rec_cap;
        float gamma = valid ? S->rec_f[15 * cap + r] : 0.0f;
        TileFeatures src{reinterpret_cast<const __half2*>(S->feat) + (size_t)(r >> 5) * 288 * 32 + (r & 31), valid};
        st = eval(src, gamma, S->g, S->sr, o);
        if (valid && stores && !(st & kStFailed)) {
            int pix = S->rec_pix[r];
            f3 hit = mk3(S->rec_f[r], S->rec_f[cap + r], S->rec_f[2 * cap + r]);
            f3 res = mul(mul(mk3(o[0], o[1], o[2]), S->light_color), S->scatter_rate);
            float4 v4 = make_float4(fmaxf(res.x, 0.0f), fmaxf(res.y, 0.0f), fmaxf(res.z, 0.0f),
                                    fmaxf(length(sub(S->ori, hit)), 0.0f));
            const int mean_k = S->mean_k;
            float rate = 1.0f / (float)(1 + mean_k);
            float4 a = mean_k == 0 ? make_float4(0, 0, 0, 0) : S->accum[pix];
            S->accum[pix] = make_float4(lerp(a.x, v4.x, rate), lerp(a.y, v4.y, rate), lerp(a.z, v4.z, rate),
                                        lerp(a.w, v4.w, rate));
        }
    } else {
        const int r = tile * rows + t;
        const bool valid = t < rows && r < A.n;
        float gamma = valid ? A.gamma[r] : 0.0f;
        RowFeatures src{A.feat + (size_t)r * 576, valid, A.feat_vec};
        st = eval(src, gamma, A.g, A.sr, o);
        if (valid && stores && !(st & kStFailed)) {
            A.out3[3 * (size_t)r] = o[0];
            A.out3[3 * (size_t)r + 1] = o[1];
            A.out3[3 * (size_t)r + 2] = o[2];
        }
    }
    return st;
}

// Rows of a split tile: 32 or 64 of the 128 where the sets then still fit one
// tile an SM (an SM takes a tile's features in at 64 bytes a cycle).
MRP_D int split_rows(int tiles64, int tiles32, int sms) { return tiles32 <= sms ? 32 : tiles64 <= sms ? 64 : 128; }

// SPLIT (grey albedos): the groups share each tile, for calls of at most one
// tile an SM.  A form of its own: beside the other in one kernel it cost that
// one 1 % of a 1080p frame.
template <int EB, bool STAGED, bool COL, bool SPLIT>
__global__ void __launch_bounds__(kGroups<COL> * kGroupThreads, 1) k_mlp_tc(const __grid_constant__ TcArgs A) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int wbytes = (A.wimg_bytes + 1023) & ~1023;
    uint8_t* wimg = smem;
    uint8_t* abuf = smem + wbytes;
    uint64_t* mbar = reinterpret_cast<uint64_t*>(abuf + kGroups<COL> * kABytes);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + kGroups<COL>);
    int* tile_slot = reinterpret_cast<int*>(tslot + 1);
    int* seg_start = tile_slot + kGroups<COL>;   // staged: first tile of each segment, [nseg + 1]
    float* aux_s = reinterpret_cast<float*>(seg_start + kTcMaxSegments + 1 + 3);   // 16-byte aligned below
    const TcSegment* segs = A.segs ? A.segs : &A.seg0;
    const int nseg = A.segs ? A.nseg : 1;

    const int tid = threadIdx.x, warp = tid / 32;
    // weights -> shared memory
    const uint32_t wimg_at = tc::smem_addr(wimg);
    for (int i = tid * 16; i < A.wimg_bytes; i += blockDim.x * 16) copy16(wimg_at + (uint32_t)i, A.wimg + i);
    aux_s = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(aux_s) + 15) & ~(uintptr_t)15);
    for (int i = tid * 4; i < kAuxCount; i += blockDim.x * 4)
        *reinterpret_cast<float4*>(aux_s + i) = __ldg(reinterpret_cast<const float4*>(A.aux + i));
    if (warp == 0) {
        tc::tmem_alloc(tslot, kTmemCols);
        tc::tmem_relinquish();
    }
    if (tid < kGroups<COL>) tc::mbar_init(mbar + tid, kArrivals);
    if (STAGED && tid == 32) {
        int acc[3] = {0, 0, 0}, rows = 128;   // tiles of 128, 64 and 32 rows
        for (int q = 0; SPLIT && q < nseg; ++q)
            for (int k = 0; k < 3; ++k) acc[k] += (*segs[q].rec_count + (128 >> k) - 1) >> (7 - k);
        if (SPLIT) rows = split_rows(acc[1], acc[2], (int)gridDim.x);
        int start = 0;
        for (int q = 0; q < nseg; ++q) {
            seg_start[q] = start;
            start += (*segs[q].rec_count + rows - 1) / rows;
        }
        seg_start[nseg] = start;
        seg_start[kTcMaxSegments + 1] = rows;
    }
    tc::mbar_fence_init();
    copies_wait();
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = *tslot;

    Group G;
    G.g = tid / kGroupThreads;
    G.t = tid % kGroupThreads;
    G.a_s = tc::smem_addr(abuf + G.g * kABytes);
    G.wimg_s = tc::smem_addr(wimg);
    G.mbar_s = tc::smem_addr(mbar + G.g);
    G.tmem = tbase + (uint32_t)(G.g * kTmemColsPerGroup<COL>) + ((uint32_t)(32 * ((tid / 32) % 4)) << 16);
    G.err = A.err;
    int st = 0;

    const int rows = !SPLIT ? 128 : STAGED ? seg_start[kTcMaxSegments + 1]
                                           : split_rows((A.n + 63) / 64, (A.n + 31) / 32, (int)gridDim.x);
    const int total_tiles = STAGED ? seg_start[nseg] : (A.n + rows - 1) / rows;
    if constexpr (SPLIT) {
        static_assert(!COL, "three groups");
        SplitScratch* X = reinterpret_cast<SplitScratch*>(abuf + kABytes);
        G.a_s = tc::smem_addr(abuf);
        G.mbar_s = tc::smem_addr(mbar);
        G.tmem = tbase + ((uint32_t)(32 * (warp % 4)) << 16);
        if ((int)blockIdx.x < total_tiles)   // at most one tile a block (launch_tc)
            st = tile_work<STAGED>(A, segs, seg_start, rows, (int)blockIdx.x, G.t, G.g == 0,
                                   [&](const auto& src, float gamma, float g, f3 sr, float* o) {
                                       const float s4 = powf(sr.x, 4.0f);
                                       const TailOut t = split_network<EB>(G, st, src, aux_s, X, gamma, g, s4);
                                       o[0] = o[1] = o[2] = radiance(t.p, s4);
                                       return t.st;
                                   });
    }
    // the first tiles go round the blocks, the rest to whichever group is free
    for (bool first = true; !SPLIT; first = false) {
        if (G.t == 0)
            tile_slot[G.g] = first ? G.g * (int)gridDim.x + (int)blockIdx.x
                                   : kGroups<COL> * (int)gridDim.x + atomicAdd(A.tile_counter, 1);
        group_bar(G.g);
        int tile = tile_slot[G.g];
        // (a wait may have timed out for some of a group's threads only: they
        // stop together, or the others would wait at the barrier for them)
        const bool lost = group_any(G.g, st & kStFailed);
        if (tile >= total_tiles || lost) break;
        // staged records from the last tile down: the gather wrote its
        // features in record order just before, so the last tiles' features
        // are still in L2 when the first groups ask for them
        if (STAGED) tile = total_tiles - 1 - tile;
        st = tile_work<STAGED>(A, segs, seg_start, rows, tile, G.t, true,
                               [&](const auto& src, float gamma, float g, f3 sr, float* o) {
                                   return tc_network<EB, COL>(G, st, src, aux_s, gamma, g, sr, o);
                               });
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tbase, kTmemCols);
    }
}

static size_t tc_smem_bytes(int eb, int groups) {
    return (size_t)((image_bytes(eb) + 1023) & ~1023) + groups * kABytes + groups * 8 + 16 +
           (kTcMaxSegments + 1 + 3) * sizeof(int) + 16 + kAuxCount * sizeof(float);
}

template <int EB, bool STAGED, bool COL, bool SPLIT = false>
static cudaError_t launch_tc(TcArgs& a, int sms, cudaStream_t s) {
    auto kernel = k_mlp_tc<EB, STAGED, COL, SPLIT>;
    size_t smem = tc_smem_bytes(EB, kGroups<COL>);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if (!SPLIT && (e = cudaMemsetAsync(a.tile_counter, 0, sizeof(int), s)) != cudaSuccess) return e;
    kernel<<<sms, kGroups<COL> * kGroupThreads, smem, s>>>(a);
    return cudaGetLastError();
}
// most: the most sets or records there can be, each segment's rounded up to a
// tile.  Up to one tile an SM a tile's latency is the call's, and the groups
// share it; from there on more tiles in flight are worth more.  Of a frame the
// host knows its pixels only, not how many of them hit: one whose hits would
// fit but whose pixels do not takes the other form.
template <bool STAGED>
static cudaError_t launch_tc(TcArgs& a, bool fp8, bool coloured, size_t most, int sms, cudaStream_t s) {
    if (coloured) return fp8 ? launch_tc<1, STAGED, true>(a, sms, s) : launch_tc<2, STAGED, true>(a, sms, s);
    if (most <= (size_t)sms * 128)
        return fp8 ? launch_tc<1, STAGED, false, true>(a, sms, s) : launch_tc<2, STAGED, false, true>(a, sms, s);
    return fp8 ? launch_tc<1, STAGED, false>(a, sms, s) : launch_tc<2, STAGED, false>(a, sms, s);
}
static bool is_coloured(f3 sr) { return !(sr.x == sr.y && sr.x == sr.z); }

static TcArgs base_args(const TcWeights& w, bool fp8) {
    TcArgs a{};
    a.wimg = (const uint8_t*)(fp8 ? w.d_fp8 : w.d_bf16);
    a.wimg_bytes = image_bytes(fp8 ? 1 : 2);
    a.aux = w.d_aux;
    a.err = w.d_err;
    a.tile_counter = w.d_counter;
    return a;
}

cudaError_t tc_launch_mlp(const TcWeights& w, bool fp8, const float* feat, const float* gamma, float g, const float sr[3],
                          int n, float* out3, int sms, cudaStream_t s) {
    if (!w.ready) return cudaErrorNotReady;
    TcArgs a = base_args(w, fp8);
    a.feat = feat;
    a.feat_vec = (reinterpret_cast<uintptr_t>(feat) & 15) == 0;
    a.gamma = gamma;
    a.n = n;
    a.g = g;
    a.sr = mk3(sr[0], sr[1], sr[2]);
    a.out3 = out3;
    return launch_tc<false>(a, fp8, is_coloured(a.sr), (size_t)n, sms, s);
}

cudaError_t tc_launch_mlp_at(const TcWeights& w, bool fp8, const float* feat, const float* gamma, float g,
                             const float sr[3], int n, float* out3, int* tile_counter, int* err, int sms,
                             cudaStream_t s) {
    if (!w.ready || !tile_counter || !err) return cudaErrorNotReady;
    TcArgs a = base_args(w, fp8);
    a.err = err;
    a.tile_counter = tile_counter;
    a.feat = feat;
    a.feat_vec = (reinterpret_cast<uintptr_t>(feat) & 15) == 0;
    a.gamma = gamma;
    a.n = n;
    a.g = g;
    a.sr = mk3(sr[0], sr[1], sr[2]);
    a.out3 = out3;
    cudaError_t e = cudaMemsetAsync(err, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
    return launch_tc<false>(a, fp8, is_coloured(a.sr), (size_t)n, sms, s);
}

TcSegment tc_segment(const VolumeDev& v, const ViewDev& view, const HitRecords& rec, const float* feat,
                     float4* accum) {
    TcSegment q{};
    q.feat = feat;
    q.rec_count = rec.count;
    q.rec_pix = rec.pix;
    q.rec_f = rec.f;
    q.rec_cap = rec.cap;
    q.accum = accum;
    q.sr = mk3(v.scatter_rate.x / 1.001f, v.scatter_rate.y / 1.001f, v.scatter_rate.z / 1.001f);
    q.light_color = view.light_color;
    q.scatter_rate = v.scatter_rate;
    q.ori = view.ori;
    q.g = view.g;
    q.mean_k = view.mean_k;
    q.most = (size_t)view.width * view.height;
    return q;
}

cudaError_t tc_launch_mlp_rec(const TcWeights& w, bool fp8, const VolumeDev& v, const ViewDev& view,
                              const HitRecords& rec, const float* feat, float4* accum, const TcScratch& sc, int sms,
                              cudaStream_t s) {
    if (!w.ready || !sc.d) return cudaErrorNotReady;
    TcArgs a = base_args(w, fp8);
    a.tile_counter = sc.d;
    a.err = sc.d + 1;
    a.segs = nullptr;
    a.nseg = 1;
    a.seg0 = tc_segment(v, view, rec, feat, accum);
    return launch_tc<true>(a, fp8, is_coloured(a.seg0.sr), a.seg0.most, sms, s);
}

cudaError_t tc_launch_mlp_segments(const TcWeights& w, bool fp8, const TcSegment* d_segs, const TcSegment* h_segs,
                                   int nseg, const TcScratch& sc, int sms, cudaStream_t s) {
    if (!w.ready || !sc.d || !d_segs || !h_segs) return cudaErrorNotReady;
    if (nseg < 1 || nseg > kTcMaxSegments) return cudaErrorInvalidValue;
    TcArgs a = base_args(w, fp8);
    a.tile_counter = sc.d;
    a.err = sc.d + 1;
    a.segs = d_segs;
    a.nseg = nseg;
    bool coloured = false;
    size_t most = 0;   // (up to 127 rows of a segment's last tile stay empty)
    for (int q = 0; q < nseg; ++q) {
        coloured = coloured || is_coloured(h_segs[q].sr);
        most += (h_segs[q].most + 127) / 128 * 128;
    }
    return launch_tc<true>(a, fp8, coloured, most, sms, s);
}

// ---------------------------------------------------------------------------
// self-test: one M=128 GEMM D = A * B^T through the same descriptors
// ---------------------------------------------------------------------------
template <int EB>
__global__ void __launch_bounds__(128, 1) k_tc_gemm_test(const float* __restrict__ A, const float* __restrict__ B,
                                                         int n, int k, float* __restrict__ D, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int kp = k;   // multiple of 16 (BF16) / 32 (E4M3)
    uint8_t* sa = smem;
    uint8_t* sb = smem + 128 * kp * EB;
    uint64_t* mbar = reinterpret_cast<uint64_t*>(sb + 128 * kp * EB);
    uint32_t* slot = reinterpret_cast<uint32_t*>(mbar + 1);
    int t = threadIdx.x;
    if (t < 32) { tc::tmem_alloc(slot, 128); tc::tmem_relinquish(); }
    if (t == 0) tc::mbar_init(mbar, 1);
    tc::mbar_fence_init();
    for (int idx = t; idx < 128 * kp; idx += 128) {
        int m = idx / kp, kk = idx % kp;
        float va = A[m * k + kk];
        float vb = m < n ? B[m * k + kk] : 0.0f;
        if (EB == 2) {
            uint32_t pa = tc::pack_bf16(va, 0.0f), pb = tc::pack_bf16(vb, 0.0f);
            *reinterpret_cast<unsigned short*>(sa + op_off(m, kk, kp, 2)) = (unsigned short)(pa & 0xFFFF);
            *reinterpret_cast<unsigned short*>(sb + op_off(m, kk, kp, 2)) = (unsigned short)(pb & 0xFFFF);
        } else {
            sa[op_off(m, kk, kp, 1)] = (uint8_t)(tc::pack_e4m3(va, 0.0f) & 0xFF);
            sb[op_off(m, kk, kp, 1)] = (uint8_t)(tc::pack_e4m3(vb, 0.0f) & 0xFF);
        }
    }
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    uint32_t tbase = *slot;
    if (t == 0) {
        uint32_t idesc = tc::instr_desc(128, n, EB == 2 ? tc::kFmtBF16 : tc::kFmtE4M3);
        uint32_t sbo = (uint32_t)(kp * EB * 8);
        for (int s = 0; s < kp * EB / 32; ++s) {
            uint64_t ad = tc::smem_desc(tc::smem_addr(sa) + s * 256, 128, sbo);
            uint64_t bd = tc::smem_desc(tc::smem_addr(sb) + s * 256, 128, sbo);
            if (EB == 2) tc::mma_bf16(tbase, ad, bd, idesc, s > 0);
            else tc::mma_fp8(tbase, ad, bd, idesc, s > 0);
        }
        tc::mma_commit(mbar);
    }
    bool ok = tc::mbar_wait(mbar, 0, kWaitLimit);
    if (!ok && t == 0) atomicExch(err, 1);
    tc::fence_after_sync();
    if (ok) {
        uint32_t lane_addr = tbase + ((uint32_t)(32 * (t / 32)) << 16);
        for (int c0 = 0; c0 < n; c0 += 16) {
            float v[16];
            tc::tmem_ld16(lane_addr + c0, v);
            for (int i = 0; i < 16; ++i) D[t * n + c0 + i] = v[i];
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (t < 32) { tc::fence_after_sync(); tc::tmem_dealloc(tbase, 128); }
}

cudaError_t tc_gemm_test(bool fp8, const float* A, const float* B, int n, int k, float* D, int* err, cudaStream_t s) {
    int eb = fp8 ? 1 : 2;
    size_t smem = (size_t)2 * 128 * k * eb + 64;
    cudaError_t e;
    if (fp8) {
        if ((e = cudaFuncSetAttribute(k_tc_gemm_test<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess) return e;
        k_tc_gemm_test<1><<<1, 128, smem, s>>>(A, B, n, k, D, err);
    } else {
        if ((e = cudaFuncSetAttribute(k_tc_gemm_test<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess) return e;
        k_tc_gemm_test<2><<<1, 128, smem, s>>>(A, B, n, k, D, err);
    }
    return cudaGetLastError();
}

}  // namespace mrp
