// mlp_fp32.cu -- the MRPNN network (RadiancePredictInternal,
// core/radiancePredict.cu:301-422) in FP32 on the CUDA cores, the drop-in form.
//
// Every output is the reference's own sum: its bias (or 0) first, then the
// inputs in index order, one fused multiply-add each.  Only who computes what
// is arranged here, so the result does not depend on the tiling.
//
// What bounds it: the FP32 pipes and, next to them, shared-memory reads.
// 48.5 K multiply-adds a pixel are 0.66 ms for the 509 K hits of the headline
// frame at 74.4 TFLOP/s.  One thread per pixel with weights from L1 (the form
// before this one) spent its time waiting for those weights (5.69 ms).  Here
// a block of eight warps takes a tile of 64 pixels (32 for few pixels):
// activations [row][pixel] and the weights of the layer at hand in shared
// memory; a thread makes 8 pixels x 4 outputs of a wide layer in registers, 4
// pixels x up to 4 outputs of a narrow one, and issues its multiply-adds in
// pairs (fma.rn.f32x2: two IEEE fused multiply-adds).  A shared-memory load
// costs a warp one wavefront per float a lane gets, whatever the lanes share,
// so floats loaded per multiply-add decide (12 for 32 in the wide layers).
// 509 K hits: 1.86 ms; 2.02 with 8 pixels a thread in the narrow layers too;
// 1.98 with four warps of 8 x 8 a thread (two warps a scheduler do not hide
// the latencies, and coloured albedos take 1.17 instead of 0.98 ms per 100
// 001 sets); 3.03 with 128 pixels a tile and features loaded where they are
// used.  200 003 sets in rows: 3.25 -> 0.87 ms.
//
// Weights stream through two 8 KB stages in 28 chunks (laid out input-major
// on the host) and the SE blocks' feature slices through two 24 KB regions,
// both by asynchronous copies ahead of their use; the barrier that hands a
// chunk over is also what separates most layers.  The SE blocks' three
// channels are independent chains: two warps each, meeting at a barrier of
// their own; the remaining two warps run the direct-illumination chain.
#include <cmath>
#include <cstring>
#include <vector>

#include "kernels.h"

namespace mrp {

namespace {

constexpr int kThreads = 256;   // eight warps
constexpr int kChunk = 2048;   // floats of a stage
enum Chunk { kCGate = 0, kCFin1 = 1, kCHead = 2, kCB2 = 3, kCB4 = 4, kCB5 = 5, kCFinal = 11, kCLC0 = 13, kCLC1 = 21,
             kCLC2 = 25, kCRes0 = 26, kCRes1 = 27, kChunks = 28 };
// kCHead holds main blocks 0 and 1.  The direct-illumination layers ride along:
// block 0 in kCHead, 1 in kCB2, 2 and 3 in kCB4, the finals in kCB5, at these
// offsets.
constexpr int kHeadDi = 384, kB2Di = 1536, kB4Di = 768, kB5Di = 1536;
// Constants of the kernels: the layers' biases, LSEFin1's last
// row (albedo^4), LSEFin2, LGGS and the 16 -> 1 head.
constexpr int mw(int k) { return k < 2 ? 8 : k < 5 ? 16 : 32; }
constexpr int kBMain = 0;   // block b, channel c at main_bias(b) + c * mw(b)
constexpr int main_bias(int b) { int o = kBMain; for (int i = 0; i < b; ++i) o += 3 * mw(i); return o; }
constexpr int kBFinal = main_bias(8), kBDi = kBFinal + 96, kBDiFinal = kBDi + 96, kBLC0 = kBDiFinal + 24,
              kBLC1 = kBLC0 + 128, kBLC2 = kBLC1 + 64, kBLX = kBLC2 + 32, kBRes = kBLX + 16, kFin1Last = kBRes + 192,
              kFin2 = kFin1Last + 16, kLggsW = kFin2 + 96, kLggsB = kLggsW + 24, kHeadW = kLggsB + 8,
              kHeadB = kHeadW + 16, kConst = (kHeadB + 1 + 3) / 4 * 4;
__constant__ float c_con[kConst];

}  // namespace

size_t fp32_weight_floats() { return (size_t)kChunks * kChunk; }

// Packed weights (common.cuh) -> chunks (d_out) and the kernels' constants.
cudaError_t fp32_prepare_weights(const float* w, float* d_out) {
    std::vector<float> stream(fp32_weight_floats() + kConst);
    float* out = stream.data();
    auto chunk = [&](int c) { return out + (size_t)c * kChunk; };
    // rows [k0, k1) of a layer with weights W [n][K] (out, in): [k][n]
    auto rows = [](float* dst, const float* W, int n, int K, int k0, int k1) {
        for (int k = k0; k < k1; ++k)
            for (int o = 0; o < n; ++o) dst[(k - k0) * n + o] = W[o * K + k];
    };
    auto block = [&](int b) { return w + (b < 8 ? main_block_off(b) : di_block_off(b - 8)); };
    for (int b = 0; b < 12; ++b) std::memcpy(chunk(kCGate) + 88 * b, block(b), 88 * sizeof(float));
    rows(chunk(kCFin1), w + kLSEFin1W, 16, 75, 0, 74);
    // three channels of a W x W block layer
    auto channels = [&](float* dst, const float* W, int n, int k0, int k1) {
        for (int c = 0; c < 3; ++c) rows(dst + c * (k1 - k0) * n, W + c * (n * n + n), n, n, k0, k1);
    };
    channels(chunk(kCHead), block(0) + 88, 8, 0, 8);
    channels(chunk(kCHead) + 192, block(1) + 88, 8, 0, 8);
    channels(chunk(kCHead) + kHeadDi, block(8) + 88, 8, 0, 8);
    channels(chunk(kCB2) + kB2Di, block(9) + 88, 8, 0, 8);
    channels(chunk(kCB4) + kB4Di, block(10) + 88, 8, 0, 8);
    channels(chunk(kCB4) + kB4Di + 192, block(11) + 88, 8, 0, 8);
    channels(chunk(kCB5) + kB5Di, w + kDiFinalOff, 8, 0, 8);
    channels(chunk(kCB2), block(2) + 88, 16, 0, 16);
    channels(chunk(kCB2) + 768, block(3) + 88, 16, 0, 16);
    channels(chunk(kCB4), block(4) + 88, 16, 0, 16);
    for (int b = 5; b < 9; ++b)
        for (int h = 0; h < 2; ++h)
            channels(chunk(kCB5 + 2 * (b - 5) + h), b < 8 ? block(b) + 88 : w + kMainFinalOff, 32, 16 * h, 16 * h + 16);
    for (int q = 0; q < 8; ++q) rows(chunk(kCLC0 + q), w + kLC0W, 128, 128, 16 * q, 16 * q + 16);
    for (int q = 0; q < 4; ++q) rows(chunk(kCLC1 + q), w + kLC1W, 64, 128, 32 * q, 32 * q + 32);
    rows(chunk(kCLC2), w + kLC2W, 32, 64, 0, 64);
    rows(chunk(kCRes0), w + kLXW, 16, 32, 0, 32);
    for (int k = 0; k < 12; ++k)
        rows(k < 6 ? chunk(kCRes0) + 512 + 256 * k : chunk(kCRes1) + 256 * (k - 6), w + lxw(k), 16, 16, 0, 16);
    float* c = out + (size_t)kChunks * kChunk;
    auto bias3 = [&](int at, const float* W, int n) {
        for (int ch = 0; ch < 3; ++ch) std::memcpy(c + at + ch * n, W + ch * (n * n + n) + n * n, n * sizeof(float));
    };
    for (int b = 0; b < 8; ++b) bias3(main_bias(b), block(b) + 88, kMainW[b]);
    bias3(kBFinal, w + kMainFinalOff, 32);
    for (int b = 0; b < 4; ++b) bias3(kBDi + 24 * b, block(8 + b) + 88, 8);
    bias3(kBDiFinal, w + kDiFinalOff, 8);
    std::memcpy(c + kBLC0, w + kLC0B, 128 * sizeof(float));
    std::memcpy(c + kBLC1, w + kLC1B, 64 * sizeof(float));
    std::memcpy(c + kBLC2, w + kLC2B, 32 * sizeof(float));
    std::memcpy(c + kBLX, w + kLXB, 16 * sizeof(float));
    for (int k = 0; k < 12; ++k) std::memcpy(c + kBRes + 16 * k, w + lxb(k), 16 * sizeof(float));
    for (int o = 0; o < 16; ++o) c[kFin1Last + o] = w[kLSEFin1W + o * 75 + 74];
    std::memcpy(c + kFin2, w + kLSEFin2W, 96 * sizeof(float));
    std::memcpy(c + kLggsW, w + kLGGSW, 24 * sizeof(float));
    std::memcpy(c + kLggsB, w + kLGGSB, 8 * sizeof(float));
    std::memcpy(c + kHeadW, w + kLX12W, 16 * sizeof(float));
    c[kHeadB] = w[kLX12B];
    cudaError_t e = cudaMemcpyToSymbol(c_con, c, kConst * sizeof(float));
    return e != cudaSuccess ? e : cudaMemcpy(d_out, out, fp32_weight_floats() * sizeof(float), cudaMemcpyHostToDevice);
}

namespace {

MRP_D float lo_of(f32x2 v) { float a, b; upk2(v, a, b); return a; }
MRP_D float hi_of(f32x2 v) { float a, b; upk2(v, a, b); return b; }
MRP_D float relu(float a) { return a >= 0.0f ? a : 0.0f; }
MRP_D float sigmoid_ref(float o) { return (float)(1.0 / (1.0 + (double)expf(-o))); }
MRP_D void cp16(float* dst, const float* src, int bytes) {   // bytes: 16, or 0 for zeros
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

// N consecutive pixels of a row, N = 1 or 2 (the element-wise phases: lane l
// of a warp has pixels N l ..).
template <int N>
struct Vec { float v[N]; };
template <int N>
MRP_D Vec<N> ldv(const float* p) {
    Vec<N> r;
    if constexpr (N == 2) { const float2 q = *reinterpret_cast<const float2*>(p); r.v[0] = q.x; r.v[1] = q.y; }
    else r.v[0] = *p;
    return r;
}
template <int N>
MRP_D void stv(float* p, const Vec<N>& r) {
    if constexpr (N == 2) *reinterpret_cast<float2*>(p) = make_float2(r.v[0], r.v[1]);
    else *p = r.v[0];
}

// The layer phases.  Wide layers: a thread has H groups of four pixels, lane
// l's at 32 h + 4 (l % 8), and outputs by l / 8 (of four).  Narrow layers:
// one group of four pixels, at 4 (l % (8 H)), and outputs by l / (8 H) (of
// 4 / H), twice as many for H = 2: fewer floats loaded per multiply-add.
template <int H>
struct Px { float v[4 * H]; };
template <int H>
MRP_D Px<H> ldp(const float* row, int pg) {
    Px<H> r;
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const float4 q = *reinterpret_cast<const float4*>(row + 32 * h + 4 * pg);
        r.v[4 * h] = q.x; r.v[4 * h + 1] = q.y; r.v[4 * h + 2] = q.z; r.v[4 * h + 3] = q.w;
    }
    return r;
}
template <int H>
MRP_D void stp(float* row, int pg, const Px<H>& r) {
#pragma unroll
    for (int h = 0; h < H; ++h)
        *reinterpret_cast<float4*>(row + 32 * h + 4 * pg) =
            make_float4(r.v[4 * h], r.v[4 * h + 1], r.v[4 * h + 2], r.v[4 * h + 3]);
}

// NO outputs of a thread's pixels, two pixels to a register pair.
template <int H, int NO>
struct Acc {
    f32x2 a[NO][2 * H];
    MRP_D void bias(int at) {
#pragma unroll
        for (int n = 0; n < NO; ++n) {
            const float b = c_con[at + n];
#pragma unroll
            for (int p = 0; p < 2 * H; ++p) a[n][p] = pk2(b, b);
        }
    }
    MRP_D Px<H> out(int n) const {   // relu of output n
        Px<H> r;
#pragma unroll
        for (int p = 0; p < 2 * H; ++p) { r.v[2 * p] = relu(lo_of(a[n][p])); r.v[2 * p + 1] = relu(hi_of(a[n][p])); }
        return r;
    }
    // K inputs: row k of the tile at s + k * T (s at the lane's pixels), this
    // thread's weights at w + k * R
    template <int K>
    MRP_D void mul(const float* s, int T, const float* w, int R) {
#pragma unroll 8
        for (int k = 0; k < K; ++k) {
            f32x2 x[2 * H];
#pragma unroll
            for (int h = 0; h < H; ++h) {
                const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(s + k * T + 32 * h);
                x[2 * h] = q.x; x[2 * h + 1] = q.y;
            }
            float wk[NO];
            if constexpr (NO == 4) { const float4 q = *reinterpret_cast<const float4*>(w + k * R); wk[0] = q.x; wk[1] = q.y; wk[2] = q.z; wk[3] = q.w; }
            else if constexpr (NO == 2) { const float2 q = *reinterpret_cast<const float2*>(w + k * R); wk[0] = q.x; wk[1] = q.y; }
            else wk[0] = w[k * R];
#pragma unroll
            for (int n = 0; n < NO; ++n) {
                const f32x2 ww = pk2(wk[n], wk[n]);
#pragma unroll
                for (int p = 0; p < 2 * H; ++p) a[n][p] = fma2(x[p], ww, a[n][p]);
            }
        }
    }
};

// Feature sources: element (channel c, sample i) of pixel r of the launch is
// sample f = c * 192 + i.  Pixels past the end read as 0.  A slice region of
// the tile in shared memory holds 32 samples of each channel (kRegion floats
// a channel).
struct TiledSource {   // the staged predictor's tiled layout (launch_gather_rec); region: [sample][pixel]
    const float* feat;
    int count;
    MRP_D bool group(int r) const { return (r & ~31) < count; }   // a started group of 32 is allocated whole
    MRP_D const float* at(int r, int f) const { return feat + ((size_t)(r >> 5) * 576 + f) * 32 + (r & 31); }
    // eight samples of one pixel
    MRP_D void eight(int r, int f, float (&v)[8]) const {
        const float* p = at(r, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = group(r) ? __ldg(p + 32 * e) : 0.0f;
    }
    // one sample of a thread's pixels
    template <int H>
    MRP_D Px<H> sample(int r0, int pg, int f) const {
        Px<H> x;
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int r = r0 + 32 * h + 4 * pg;
            const float4 q = group(r) ? __ldg(reinterpret_cast<const float4*>(at(r, f))) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            x.v[4 * h] = q.x; x.v[4 * h + 1] = q.y; x.v[4 * h + 2] = q.z; x.v[4 * h + 3] = q.w;
        }
        return x;
    }
    // samples [f, f + n) of the tile's pixels into row `row` on of a channel's
    // region, by threads t of nt
    template <int H>
    MRP_D void stage(float* reg, int row, int r0, int f, int n, int t, int nt) const {
        for (int q = t; q < n * 8 * H; q += nt) {
            const int i = q / (8 * H), h = (q / 8) % H, r = r0 + 32 * h + 4 * (q % 8);
            cp16(reg + (row + i) * 32 * H + 32 * h + 4 * (q % 8), group(r) ? at(r, f + i) : feat, group(r) ? 16 : 0);
        }
    }
    // NO samples from row o of a channel's region for a thread's pixels
    // (G: the thread's groups of four pixels, H or 1)
    template <int H, int G, int NO>
    static MRP_D void region(const float* reg, int o, int pg, Px<G> (&x)[NO]) {
#pragma unroll
        for (int n = 0; n < NO; ++n) x[n] = ldp<G>(reg + (o + n) * 32 * H, pg);
    }
};
// [n][576], a pixel's features in a row; region: [pixel slot][32 samples] in
// 16-byte pieces, piece j of slot s at j ^ (s % 8), slots ordered so that the
// lanes' pixels lie in consecutive ones.
struct RowSource {
    const float* feat;
    int count;
    bool vec;   // rows start on 16-byte boundaries
    MRP_D void eight(int r, int f, float (&v)[8]) const {   // f a multiple of 8
        const float* p = feat + (size_t)r * 576 + f;
        if (r < count && vec) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = r < count ? __ldg(p + e) : 0.0f;
        }
    }
    template <int H>
    MRP_D Px<H> sample(int r0, int pg, int f) const {
        Px<H> x;
#pragma unroll
        for (int p = 0; p < 4 * H; ++p) {
            const int r = r0 + 32 * (p / 4) + 4 * pg + p % 4;
            x.v[p] = r < count ? __ldg(feat + (size_t)r * 576 + f) : 0.0f;
        }
        return x;
    }
    template <int H>
    static MRP_D int slot(int px) { return (px & 3) * 8 * H + (px >> 2); }
    template <int H>
    MRP_D void stage(float* reg, int row, int r0, int f, int n, int t, int nt) const {
        const int per = n / 4;   // 16-byte pieces of a pixel
        for (int q = t; q < per * 32 * H; q += nt) {
            const int px = q / per, j = q % per, r = r0 + px, s = slot<H>(px);
            float* d = reg + s * 32 + (((row >> 2) + j) ^ (s & 7)) * 4;
            const float* src = feat + (size_t)r * 576 + f + 4 * j;
            if (vec || r >= count) {
                // (an address of a copy of no bytes must be aligned too)
                const float* none = reinterpret_cast<const float*>(reinterpret_cast<uintptr_t>(feat) & ~(uintptr_t)15);
                cp16(d, r < count ? src : none, r < count ? 16 : 0);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint32_t a = (uint32_t)__cvta_generic_to_shared(d + e);
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(a), "l"(src + e) : "memory");
                }
            }
        }
    }
    template <int H, int G, int NO>
    static MRP_D void region(const float* reg, int o, int pg, Px<G> (&x)[NO]) {   // o a multiple of NO
#pragma unroll
        for (int p = 0; p < 4 * G; ++p) {
            const int s = (p & 3) * 8 * H + (p >> 2) * 8 + pg;
            const float* d = reg + s * 32 + ((o >> 2) ^ (pg & 7)) * 4 + (o & 3);
            if constexpr (NO == 4) { const float4 q = *reinterpret_cast<const float4*>(d); x[0].v[p] = q.x; x[1].v[p] = q.y; x[2].v[p] = q.z; x[3].v[p] = q.w; }
            else if constexpr (NO == 2) { const float2 q = *reinterpret_cast<const float2*>(d); x[0].v[p] = q.x; x[1].v[p] = q.y; }
            else x[0].v[p] = *d;
        }
    }
};

// What becomes of a pixel's three outputs.
struct FrameSink {   // the running mean at the record's pixel (k_hit's record r)
    VolumeDev v;
    ViewDev w;
    HitRecords rec;
    float4* accum;
    MRP_D float gamma(int r) const { return rec.f[15 * rec.cap + r]; }
    MRP_D void put(int r, const float (&o)[3]) const {
        const int pix = rec.pix[r];
        const f3 hit = mk3(rec.f[r], rec.f[rec.cap + r], rec.f[2 * rec.cap + r]);
        const f3 pr = mrp::mul(mk3(o[0], o[1], o[2]), 1.0f);   // alphaMult == 1 (core/render.cuh:844-848)
        const f3 res = mrp::mul(mrp::mul(pr, w.light_color), v.scatter_rate);
        running_mean(accum, pix, w.mean_k, make_float4(res.x, res.y, res.z, length(sub(w.ori, hit))));
    }
};
struct RowSink {
    const float* gam;
    float* out3;
    MRP_D float gamma(int r) const { return gam[r]; }
    MRP_D void put(int r, const float (&o)[3]) const {
        out3[3 * (size_t)r] = o[0]; out3[3 * (size_t)r + 1] = o[1]; out3[3 * (size_t)r + 2] = o[2];
    }
};

// The 36 (block, channel) slices in descending width: first sample, width,
// pool index.
struct Slice { short f, w, pid; };
constexpr int kSlices = 36;
constexpr int kBlockFrom[12] = {0, 8, 16, 32, 48, 64, 96, 128, 160, 168, 176, 184};
constexpr int kBlockW[12] = {8, 8, 16, 16, 16, 32, 32, 32, 8, 8, 8, 8};
struct SliceTable {
    Slice s[kSlices];
    constexpr SliceTable() : s{} {
        int n = 0;
        for (int w = 32; w >= 8; w /= 2)
            for (int b = 0; b < 12; ++b)
                if (kBlockW[b] == w)
                    for (int c = 0; c < 3; ++c) {
                        s[n].f = (short)(c * 192 + kBlockFrom[b]);
                        s[n].w = (short)w;
                        s[n].pid = (short)(3 * b + c);
                        ++n;
                    }
    }
};
__constant__ SliceTable c_slices = SliceTable();

template <int H, bool COLOURED>
struct Layout {   // shared memory, floats
    static constexpr int T = 32 * H;
    static constexpr int kAct = 0;                       // activations [128][T]; pools and their constants [74][T]
    static constexpr int kAct2 = kAct + 128 * T;         // coloured: the gated inputs and what follows, per channel
    static constexpr int kRegion = 32 * T;               // a channel's part of a slice region
    static constexpr int kSlice = kAct2 + (COLOURED ? 128 * T : 0);   // slice regions [2][3][kRegion]
    static constexpr int kGates = kSlice + 6 * kRegion;  // SE gates [36][T], then the 6 LSEFin gates
    static constexpr int kFin = kGates + 36 * T;         // LSEFin1 over the first 74 inputs [16][T]
    static constexpr int kRing = kFin + 16 * T;
    static constexpr int kFloats = kRing + 2 * kChunk;
};
static_assert(2 * (Layout<2, false>::kFloats * 4 + 1024) <= 228 * 1024, "two blocks of an SM");

// Where main block b's slice lies: region, first row of each channel's part.
// Blocks 0..2 fill region 0, 3 and 4 region 1; then 5, 6, 7 take turns.
MRP_D int slice_region(int b) { return b == 3 || b == 4 || b == 6; }
MRP_D int slice_row(int b) { return b == 1 ? 8 : b == 2 || b == 4 ? 16 : 0; }

template <int H, bool COLOURED, class Source, class Sink>
struct Net {
    using L = Layout<H, COLOURED>;
    static constexpr int T = L::T;
    float* sm;
    const float* wts;   // chunks in global memory
    int q;              // chunks handed over so far

    MRP_D void copy(int chunk) const {   // 8 KB into the stage of the chunk after the current one
        const float* src = wts + (size_t)chunk * kChunk;
        float* dst = sm + L::kRing + (q & 1) * kChunk;
#pragma unroll
        for (int i = 0; i < kChunk / (4 * kThreads); ++i) {
            const int o = 4 * (i * kThreads + (int)threadIdx.x);
            cp16(dst + o, src + o, 16);
        }
    }
    // All warps: everything before is done, every copy issued before has
    // landed, the next chunk is in shared memory (returned), and the one
    // after it (`upcoming`, or -1) is on its way.
    MRP_D const float* next(int upcoming) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        const float* cur = sm + L::kRing + (q & 1) * kChunk;
        ++q;
        if (upcoming >= 0) copy(upcoming);
        return cur;
    }
    static MRP_D void group_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(1 + id) : "memory"); }
    MRP_D float* region(int b, int c) const { return sm + L::kSlice + (3 * slice_region(b) + c) * L::kRegion; }
    MRP_D float* act(int row) const { return sm + L::kAct + row * T; }

    // The slices of main blocks 0..4 of a tile (256 threads).
    MRP_D void stage_first(const Source& src, int r0) const {
#pragma unroll 1
        for (int b = 0; b < 5; ++b)
#pragma unroll 1
            for (int c = 0; c < 3; ++c)
                src.template stage<H>(region(b, c), slice_row(b), r0, c * 192 + main_from(b), main_w(b), threadIdx.x, kThreads);
    }
    // The slice of block b of one channel, by its two warps, once both are
    // past their last read of the region (a group_sync in between).
    MRP_D void stage_next(const Source& src, int r0, int b, int c, int half, int lane) const {
        src.template stage<H>(region(b, c), 0, r0, c * 192 + main_from(b), 32, 32 * half + lane, 64);
    }
    static MRP_D int main_w(int b) { return b < 2 ? 8 : b < 5 ? 16 : 32; }
    static MRP_D int main_from(int b) { return b < 2 ? 8 * b : b < 5 ? 16 * (b - 1) : 64 + 32 * (b - 5); }
    static MRP_D int main_bias_at(int b) { return b < 2 ? 24 * b : b < 5 ? 48 + 48 * (b - 2) : 192 + 96 * (b - 5); }
    static_assert(main_bias(1) == 24 && main_bias(2) == 48 && main_bias(5) == 192 && main_bias(7) == 384, "bias offsets");

    // ---- SE chains -------------------------------------------------------
    MRP_D void gated(Px<H>& x, const Px<H>& g) const {
#pragma unroll
        for (int p = 0; p < 4 * H; ++p) x.v[p] = x.v[p] * g.v[p];
    }
    // Main block b, channel c: layer, then the next block's inputs in place:
    // out = relu(acc) (+ slice, or beside it when the block widens), next
    // input = next slice * next gate + out.  This warp: outputs half * W / 2 on.
    template <int W, bool WIDEN>
    MRP_D void main_block(const float* w, int b, int c, int half, int lane) {   // W = 8, 16
        constexpr int NO = W * H / 8;
        const int pg = lane % (8 * H), o = half * (W / 2) + lane / (8 * H) * NO;
        Acc<1, NO> acc;
        acc.bias(main_bias_at(b) + c * W + o);
        acc.template mul<W>(act(32 * c) + 4 * pg, T, w + c * W * W + o, W);
        group_sync(c);   // both halves have read the inputs
        main_step<1, NO, W, WIDEN, false>(acc, b, c, o, pg);
        group_sync(c);
    }
    template <int G, int NO, int W, bool WIDEN, bool LAST>
    MRP_D void main_step(const Acc<G, NO>& acc, int b, int c, int o, int pg) {
        Px<G> x[NO], y[NO], z[NO], g;
        Source::template region<H, G, NO>(region(b, c), slice_row(b) + o, pg, x);
        if (!LAST) {
            Source::template region<H, G, NO>(region(b + 1, c), slice_row(b + 1) + o, pg, y);
            if (WIDEN) Source::template region<H, G, NO>(region(b + 1, c), slice_row(b + 1) + W + o, pg, z);
            g = ldp<G>(sm + L::kGates + (3 * (b + 1) + c) * T, pg);
        }
#pragma unroll
        for (int n = 0; n < NO; ++n) {
            Px<G> a = acc.out(n), e;
#pragma unroll
            for (int p = 0; p < 4 * G; ++p) {
                if (!WIDEN) a.v[p] = a.v[p] + x[n].v[p];
                if (!LAST) a.v[p] = fmaf(y[n].v[p], g.v[p], a.v[p]);
                if (WIDEN) e.v[p] = fmaf(z[n].v[p], g.v[p], x[n].v[p]);
            }
            stp<G>(act(32 * c + o + n), pg, a);
            if (WIDEN) stp<G>(act(32 * c + W + o + n), pg, e);
        }
    }
    // A layer of the direct-illumination chain (b = 4: the finals): two warps,
    // four of the eight outputs of every channel each; rows 96 + 8 c.
    template <bool LAST>
    MRP_D void di_layer(const Source& src, int r0, const float* w, int b, int half, int lane) {
        const int pg = lane % (8 * H), o = 4 * half + lane / (8 * H) * H;
        Acc<1, H> acc[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            acc[c].bias(kBDi + 24 * b + 8 * c + o);
            acc[c].template mul<8>(act(96 + 8 * c) + 4 * pg, T, w + 64 * c + o, 8);
        }
        group_sync(3);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            Px<1> g;
            if (b < 4 && !LAST) g = ldp<1>(sm + L::kGates + (3 * (9 + b) + c) * T, pg);
#pragma unroll
            for (int n = 0; n < H; ++n) {
                Px<1> a = acc[c].out(n);
                if (b < 4) {
                    const Px<1> x = src.template sample<1>(r0, pg, c * 192 + 160 + 8 * b + o + n);
#pragma unroll
                    for (int p = 0; p < 4; ++p) a.v[p] = a.v[p] + x.v[p];
                    if (!LAST) {
                        const Px<1> y = src.template sample<1>(r0, pg, c * 192 + 168 + 8 * b + o + n);
#pragma unroll
                        for (int p = 0; p < 4; ++p) a.v[p] = fmaf(y.v[p], g.v[p], a.v[p]);
                    }
                }
                stp<1>(act(96 + 8 * c + o + n), pg, a);
            }
        }
        group_sync(3);
    }
    static_assert(kBDiFinal == kBDi + 96, "the finals' biases follow the blocks'");
    // All chains of a tile (every warp calls it: the chunk hand-overs are the
    // block's barriers).
    MRP_D void se_chains(const Source& src, int r0, int role, int lane) {
        const int c = role >> 1, half = role & 1, pg = lane & 7, og = lane >> 3;
        const bool main = role < 6;
        const float* w = next(kCB2);
        if (main) {
            Px<H> x[1];
            Source::template region<H, H, 1>(region(0, c), 4 * half + og, pg, x);
            gated(x[0], ldp<H>(sm + L::kGates + c * T, pg));
            stp<H>(act(32 * c + 4 * half + og), pg, x[0]);
            group_sync(c);
            main_block<8, false>(w, 0, c, half, lane);
            main_block<8, true>(w + 192, 1, c, half, lane);
        } else {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                Px<H> x = src.template sample<H>(r0, pg, d * 192 + 160 + 4 * half + og);
                gated(x, ldp<H>(sm + L::kGates + (24 + d) * T, pg));
                stp<H>(act(96 + 8 * d + 4 * half + og), pg, x);
            }
            group_sync(3);
            di_layer<false>(src, r0, w + kHeadDi, 0, half, lane);
        }
        w = next(kCB4);
        if (main) {
            main_block<16, false>(w, 2, c, half, lane);
            stage_next(src, r0, 5, c, half, lane);   // region 0: slice 2 was its last
            main_block<16, false>(w + 768, 3, c, half, lane);
        } else {
            di_layer<false>(src, r0, w + kB2Di, 1, half, lane);
        }
        w = next(kCB5);
        if (main) {
            main_block<16, true>(w, 4, c, half, lane);
            stage_next(src, r0, 6, c, half, lane);
        } else {
            di_layer<false>(src, r0, w + kB4Di, 2, half, lane);
            di_layer<true>(src, r0, w + kB4Di + 192, 3, half, lane);
        }
        const int o = half * 16 + og * 4;
#pragma unroll 1
        for (int b = 5; b < 9; ++b) {   // b = 8: the finals, whose biases follow
            Acc<H, 4> acc;
            const float* a = act(32 * c) + 4 * pg;
            w = next(kCB5 + 2 * (b - 5) + 1);
            if (main) {
                acc.bias(main_bias_at(b) + c * 32 + o);
                acc.template mul<16>(a, T, w + c * 512 + o, 32);
            } else if (b == 5) {
                di_layer<true>(src, r0, w + kB5Di, 4, half, lane);
            }
            w = next(kCB5 + 2 * (b - 5) + 2);   // after the last: kCLC0
            if (main) {
                acc.template mul<16>(a + 16 * T, T, w + c * 512 + o, 32);
                group_sync(c);
                if (b < 7) {
                    main_step<H, 4, 32, false, false>(acc, b, c, o, pg);
                    group_sync(c);
                    if (b == 5) stage_next(src, r0, 7, c, half, lane);
                } else if (b == 7) {
                    main_step<H, 4, 32, false, true>(acc, b, c, o, pg);
                } else {
                    store(acc, act(32 * c + o), pg);
                }
            }
        }
    }
    static_assert(kCFinal == kCB5 + 6 && kCLC0 == kCFinal + 2 && main_bias(7) + 96 == kBFinal, "chunk order");
    template <int G, int NO>
    MRP_D void store(const Acc<G, NO>& acc, float* dst, int pg) const {
#pragma unroll
        for (int n = 0; n < NO; ++n) stp<G>(dst + n * T, pg, acc.out(n));
    }

    // ---- pools, gates, LSEFin1 ---------------------------------------------
    // thread: pixel t % T, every G-th slice; sums run in sample order
    MRP_D void pools(const Source& src, int r0) {
        constexpr int G = kThreads / T;
        const int px = (int)threadIdx.x % T, grp = (int)threadIdx.x / T;
#pragma unroll 1
        for (int i = grp; i < kSlices; i += G) {
            const Slice S = c_slices.s[i];
            float s = 0.0f, m = -10000.0f;
            if (S.w == 32) pool<32>(src, r0 + px, S.f, s, m);
            else if (S.w == 16) pool<16>(src, r0 + px, S.f, s, m);
            else pool<8>(src, r0 + px, S.f, s, m);
            act(S.pid)[px] = s / (float)S.w;
            act(36 + S.pid)[px] = m;
        }
    }
    template <int W>
    static MRP_D void pool(const Source& src, int r, int f, float& s, float& m) {
        float x[W / 8][8];
#pragma unroll
        for (int j = 0; j < W / 8; ++j) src.eight(r, f + 8 * j, x[j]);
#pragma unroll
        for (int j = 0; j < W / 8; ++j)
#pragma unroll
            for (int e = 0; e < 8; ++e) { s += x[j][e]; m = fmaxf(m, x[j][e]); }
    }
    // SE gates of block b: 8 -> 8 relu -> 3 sigmoid per pixel.
    MRP_D void gates(const float* w, int b, float g, const Vec<H>& gam, int lane) {
        Vec<H> p8[8], a3[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            p8[c] = ldv<H>(act(3 * b + c) + lane * H);
            p8[3 + c] = ldv<H>(act(36 + 3 * b + c) + lane * H);
#pragma unroll
            for (int p = 0; p < H; ++p) a3[c].v[p] = 0.0f;
        }
#pragma unroll
        for (int p = 0; p < H; ++p) { p8[6].v[p] = g; p8[7].v[p] = gam.v[p]; }
        const float* wb = w + 88 * b;
#pragma unroll
        for (int o = 0; o < 8; ++o) {   // hidden unit o joins the three sums as their o-th term
            float h[H];
#pragma unroll
            for (int p = 0; p < H; ++p) h[p] = 0.0f;
            const float4 u = *reinterpret_cast<const float4*>(wb + 8 * o), t = *reinterpret_cast<const float4*>(wb + 8 * o + 4);
            const float wj[8] = {u.x, u.y, u.z, u.w, t.x, t.y, t.z, t.w};
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int p = 0; p < H; ++p) h[p] = fmaf(p8[j].v[p], wj[j], h[p]);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float v = wb[64 + 8 * k + o];
#pragma unroll
                for (int p = 0; p < H; ++p) a3[k].v[p] = fmaf(relu(h[p]), v, a3[k].v[p]);
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
#pragma unroll
            for (int p = 0; p < H; ++p) a3[k].v[p] = sigmoid_ref(a3[k].v[p]);
            stv<H>(sm + L::kGates + (3 * b + k) * T + lane * H, a3[k]);
        }
    }
    // LSEFin1 over the 74 inputs that no albedo channel changes: two of the
    // sixteen sums a warp.
    MRP_D void lsefin1(const float* w, int warp, int lane) {
        Vec<H> s[2];
#pragma unroll
        for (int p = 0; p < H; ++p) s[0].v[p] = s[1].v[p] = 0.0f;
#pragma unroll 8
        for (int k = 0; k < 74; ++k) {
            const Vec<H> x = ldv<H>(act(k) + lane * H);
            const float2 u = *reinterpret_cast<const float2*>(w + 16 * k + 2 * warp);
#pragma unroll
            for (int p = 0; p < H; ++p) { s[0].v[p] = fmaf(x.v[p], u.x, s[0].v[p]); s[1].v[p] = fmaf(x.v[p], u.y, s[1].v[p]); }
        }
        stv<H>(sm + L::kFin + 2 * warp * T + lane * H, s[0]);
        stv<H>(sm + L::kFin + (2 * warp + 1) * T + lane * H, s[1]);
    }

    // ---- one tile: pixels r0 .. r0 + T - 1; next_r0 < 0: no tile after it ----
    MRP_D void tile(const Source& src, const Sink& sink, int r0, int next_r0, float g, f3 sr, int role, int count) {
        const int warp = (int)threadIdx.x / 32, lane = (int)threadIdx.x & 31;
        Vec<H> gam;   // of the element-wise phases' pixels
#pragma unroll
        for (int p = 0; p < H; ++p) gam.v[p] = r0 + lane * H + p < count ? sink.gamma(r0 + lane * H + p) : 0.0f;
        pools(src, r0);
        if (warp == 0) {
            Vec<H> gg;
#pragma unroll
            for (int p = 0; p < H; ++p) gg.v[p] = g;
            stv<H>(act(72) + lane * H, gg);
            stv<H>(act(73) + lane * H, gam);
        }
        const float* w = next(kCFin1);
        gates(w, warp, g, gam, lane);
        if (warp < 4) gates(w, 8 + warp, g, gam, lane);
        lsefin1(next(kCHead), warp, lane);
        // (the hand-over that starts the chains waits for these reads of the pools)
        se_chains(src, r0, role, lane);
        __syncthreads();   // comb [120][T]; the slice regions are free
        if (next_r0 >= 0) stage_first(src, next_r0);
        const float srv[3] = {sr.x, sr.y, sr.z};
        float P[3];
#pragma unroll 1
        for (int ch = 0; ch < 3; ++ch) {
            if (ch == 1 && srv[1] == srv[0]) { P[1] = P[0]; continue; }
            if (ch == 2 && srv[2] == srv[0]) { P[2] = P[0]; continue; }
            if (ch == 2 && srv[2] == srv[1]) { P[2] = P[1]; continue; }
            const bool last = ch == 2 || (srv[1] == srv[0] ? srv[2] == srv[0] : ch == 1 && (srv[2] == srv[0] || srv[2] == srv[1]));
            const float p = tail(powf(ch == 0 ? srv[0] : ch == 1 ? srv[1] : srv[2], 4.0f), g, gam, warp, lane,
                                 !last ? (int)kCLC0 : next_r0 >= 0 ? (int)kCGate : -1);
            if (ch == 0) P[0] = p; else if (ch == 1) P[1] = p; else P[2] = p;
        }
        const int r = r0 + (int)threadIdx.x;
        if ((int)threadIdx.x < T && r < count) {
            float o[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) o[c] = fmaxf(expf(P[c]) - 1.0f, 0.0f) * powf(srv[c], 4.0f);
            sink.put(r, o);
        }
        // (the next tile's pools overwrite rows 0..73, last read before the
        // hand-over of the tail's last chunk)
    }
    // The tail of one albedo channel; thread t < T returns pixel t's output.
    MRP_D float tail(float s4, float g, const Vec<H>& gam, int warp, int lane, int after) {
        const int pg = lane & 7, og = lane >> 3;
        float* dst = sm + (COLOURED ? L::kAct2 : L::kAct);
        // LSEFin gates, one pixel a thread, spare threads share the six gates out
        {
            constexpr int G = kThreads / T >= 6 ? 6 : 3, PER = 6 / G;
            const int px = (int)threadIdx.x % T, grp = (int)threadIdx.x / T;
            if (grp < G) {
                float hf[16];
#pragma unroll
                for (int o = 0; o < 16; ++o) hf[o] = relu(fmaf(s4, c_con[kFin1Last + o], sm[L::kFin + o * T + px]));
#pragma unroll
                for (int q2 = 0; q2 < PER; ++q2) {
                    const int o = grp * PER + q2;
                    float a = 0.0f;
#pragma unroll
                    for (int j = 0; j < 16; ++j) a = fmaf(hf[j], c_con[kFin2 + o * 16 + j], a);
                    sm[L::kGates + o * T + px] = sigmoid_ref(a);
                }
            }
        }
        __syncthreads();
        // x = concat(main_c * gate_c, di_c * gate_{3+c}, LGGS(g, gamma, albedo^4))
#pragma unroll 4
        for (int i = 0; i < 16; ++i) {
            const int row = 16 * warp + i;
            Vec<H> x;
            if (row < 120) {
                const Vec<H> gt = ldv<H>(sm + L::kGates + (row < 96 ? row >> 5 : 3 + ((row - 96) >> 3)) * T + lane * H);
                x = ldv<H>(act(row) + lane * H);
#pragma unroll
                for (int p = 0; p < H; ++p) x.v[p] = x.v[p] * gt.v[p];
            } else {   // LGGS 3 -> 8: sum first, bias last (LinearReLU, :41-56)
                const int o = row - 120;
#pragma unroll
                for (int p = 0; p < H; ++p) {
                    float a = fmaf(g, c_con[kLggsW + 3 * o], 0.0f);
                    a = fmaf(gam.v[p], c_con[kLggsW + 3 * o + 1], a);
                    a = fmaf(s4, c_con[kLggsW + 3 * o + 2], a);
                    a += c_con[kLggsB + o];
                    x.v[p] = relu(a);
                }
            }
            stv<H>(dst + row * T + lane * H, x);
        }
        const float* in = dst + 4 * pg;
        const float* w;
        {
            Acc<H, 4> acc;
            acc.bias(kBLC0 + 16 * warp + 4 * og);
#pragma unroll 1
            for (int k = 0; k < 8; ++k) {
                w = next(kCLC0 + k + 1);   // after the last: kCLC1
                acc.template mul<16>(in + 16 * k * T, T, w + 16 * warp + 4 * og, 128);
            }
            __syncthreads();
            store(acc, dst + (16 * warp + 4 * og) * T, pg);
        }
        const int qg = lane % (8 * H), qo = lane / (8 * H);   // the narrow layers' pixels and outputs
        {
            Acc<1, 2 * H> acc;
            const int o = 8 * warp + 2 * H * qo;
            acc.bias(kBLC1 + o);
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                w = next(kCLC1 + k + 1);   // after the last: kCLC2
                acc.template mul<32>(dst + 4 * qg + 32 * k * T, T, w + o, 64);
            }
            __syncthreads();
            store(acc, dst + o * T, qg);
        }
        {
            Acc<1, H> acc;
            const int o = 4 * warp + H * qo;
            acc.bias(kBLC2 + o);
            w = next(kCRes0);
            acc.template mul<64>(dst + 4 * qg, T, w + o, 32);
            __syncthreads();
            store(acc, dst + o * T, qg);
        }
        // LX (rows 0..31 -> 96..111) and the six residual pairs (96..111 ->
        // 112..127 -> 96..111): 32 pixels a warp, 4 pixels x 4 outputs a
        // thread, whose own four sums stay in registers (rows that the next
        // tile's pools, which other warps may have begun, leave alone)
        float P = 0.0f;
        w = next(kCRes1);
        const bool mine = warp < H;
        float* col = dst + 32 * warp;   // this warp's pixels (mine)
        Px<1> a[4];
        if (mine) {
            Acc<1, 4> acc;
            acc.bias(kBLX + 4 * og);
            acc.template mul<32>(col + 4 * pg, T, w + 4 * og, 16);
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                a[n] = acc.out(n);
                stp<1>(col + (96 + 4 * og + n) * T, pg, a[n]);
            }
            __syncwarp();
#pragma unroll 1
            for (int k = 0; k < 3; ++k) residual(a, col, w + 512 + 512 * k, kBRes + 32 * k, pg, og);
        }
        w = next(after);
        if (mine) {
#pragma unroll 1
            for (int k = 0; k < 3; ++k) residual(a, col, w + 512 * k, kBRes + 96 + 32 * k, pg, og);
            float p = 0.0f;
#pragma unroll
            for (int j = 0; j < 16; ++j) p = fmaf(col[(96 + j) * T + lane], c_con[kHeadW + j], p);
            P = relu(p + c_con[kHeadB]);
        }
        return P;
    }
    static MRP_D void residual(Px<1> (&a)[4], float* col, const float* w, int b, int pg, int og) {
        Acc<1, 4> y, z;
        y.bias(b + 4 * og);
        y.template mul<16>(col + 96 * T + 4 * pg, T, w + 4 * og, 16);
#pragma unroll
        for (int n = 0; n < 4; ++n) stp<1>(col + (112 + 4 * og + n) * T, pg, y.out(n));
        __syncwarp();
        z.bias(b + 16 + 4 * og);
        z.template mul<16>(col + 112 * T + 4 * pg, T, w + 256 + 4 * og, 16);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const Px<1> o = z.out(n);
#pragma unroll
            for (int p = 0; p < 4; ++p) a[n].v[p] += o.v[p];
            stp<1>(col + (96 + 4 * og + n) * T, pg, a[n]);
        }
        __syncwarp();
    }
};

template <int H, bool COLOURED, class Source, class Sink>
MRP_D void run_net(const float* __restrict__ wts, const Source& source, const Sink& sink, int count, float g, f3 sr) {
    extern __shared__ __align__(16) float sm[];
    using N = Net<H, COLOURED, Source, Sink>;
    constexpr int T = N::T;
    const int tiles = (count + T - 1) / T;
    if ((int)blockIdx.x >= tiles) return;
    N net{sm, wts, 0};
    net.copy(kCGate);
    net.stage_first(source, (int)blockIdx.x * T);
    // warps 4 j + s of a block share an SM quarter: the second half of the
    // grid turns the chains' roles by two warps, so that of two blocks on an
    // SM the two-warp chain (little work) falls on different quarters
    const int turn = blockIdx.x >= gridDim.x / 2 ? 2 : 0;
    const int role = ((int)threadIdx.x / 32 + turn) & 7;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x)
        net.tile(source, sink, t * T, t + (int)gridDim.x < tiles ? (t + (int)gridDim.x) * T : -1, g, sr, role, count);
}

template <int H, bool COLOURED>
__global__ void __launch_bounds__(kThreads, COLOURED ? 1 : 2)
    k_mlp_rec(const __grid_constant__ FrameSink sink, const float* __restrict__ feat, const float* __restrict__ wts) {
    const int count = *sink.rec.count;
    run_net<H, COLOURED>(wts, TiledSource{feat, count}, sink, count, sink.w.g, div(sink.v.scatter_rate, 1.001f));
}
template <int H, bool COLOURED>
__global__ void __launch_bounds__(kThreads, COLOURED ? 1 : 2)
    k_mlp_rows(RowSource source, RowSink sink, float g, f3 sr, const float* __restrict__ wts) {
    run_net<H, COLOURED>(wts, source, sink, source.count, g, sr);
}

int sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 148;
    return sms;
}
// Calls launch(pxt, coloured, smem bytes, blocks) for n pixels at most.
template <class F>
cudaError_t pick(int n, f3 sr, F launch) {
    const int sms = sm_count();
    const bool coloured = !(sr.x == sr.y && sr.x == sr.z);
    // Tiles of 64 pixels use the FP32 pipes best; of 32 pixels, they fill the
    // SMs sooner: taken while 64-pixel tiles would not give every SM two.
    const bool small = n < 128 * sms;
    const int tile = small ? 32 : 64;
    const int tiles = (n + tile - 1) / tile;
    const int per_sm = coloured ? 1 : 2;
    return launch(small, coloured, tiles < per_sm * sms ? tiles : per_sm * sms);
}
template <class K, class... A>
cudaError_t start(K kernel, int floats, int blocks, cudaStream_t s, A... args) {
    const int bytes = floats * (int)sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    kernel<<<blocks, kThreads, bytes, s>>>(args...);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_mlp_fp32(const float* weights, const float* feat, const float* gamma, float g, const float sr[3],
                            int n, float* out3, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const f3 a = mk3(sr[0], sr[1], sr[2]);
    const RowSource src{feat, n, (reinterpret_cast<uintptr_t>(feat) & 15) == 0};
    const RowSink sink{gamma, out3};
    return pick(n, a, [&](bool small, bool coloured, int blocks) {
        if (small) return coloured ? start(k_mlp_rows<1, true>, Layout<1, true>::kFloats, blocks, s, src, sink, g, a, weights)
                                   : start(k_mlp_rows<1, false>, Layout<1, false>::kFloats, blocks, s, src, sink, g, a, weights);
        return coloured ? start(k_mlp_rows<2, true>, Layout<2, true>::kFloats, blocks, s, src, sink, g, a, weights)
                        : start(k_mlp_rows<2, false>, Layout<2, false>::kFloats, blocks, s, src, sink, g, a, weights);
    });
}

cudaError_t launch_mlp_rec_fp32(const VolumeDev& v, const ViewDev& view, HitRecords rec, const float* feat,
                                const float* weights, float4* accum, cudaStream_t s) {
    const int n = view.width * view.height;
    if (n <= 0) return cudaSuccess;
    const FrameSink sink{v, view, rec, accum};
    return pick(n, v.scatter_rate, [&](bool small, bool coloured, int blocks) {
        if (small) return coloured ? start(k_mlp_rec<1, true>, Layout<1, true>::kFloats, blocks, s, sink, feat, weights)
                                   : start(k_mlp_rec<1, false>, Layout<1, false>::kFloats, blocks, s, sink, feat, weights);
        return coloured ? start(k_mlp_rec<2, true>, Layout<2, true>::kFloats, blocks, s, sink, feat, weights)
                        : start(k_mlp_rec<2, false>, Layout<2, false>::kFloats, blocks, s, sink, feat, weights);
    });
}

}  // namespace mrp
