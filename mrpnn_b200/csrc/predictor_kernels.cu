// predictor_kernels.cu -- the MRPNN radiance predictor on the GPU, FP32 form.
//
// One launch renders one frame of RenderCamera<true, MRPNN>
// (core/volume.cu:198-228 -> core/render.cuh:808-875):
//   camera ray -> first estimated hit (DeterminateEstimatedHit) -> random
//   bases (GetMatrixFromNormal) -> 192-point stencil gather of density, TR
//   and HG features (SetupInputData) -> SE-gated MLP
//   (RadiancePredictInternal) -> running mean.
// Everything up to the features keeps the reference's float rounding order
// (common.cuh), so hits and features match the CPU oracle to the bit except
// where a transcendental's last bit differs.  The networks are in
// mlp_fp32.cu and mlp_tc.cu.
#include <cfloat>
#include <cmath>

#include <cuda_fp16.h>

#include "kernels.h"

namespace mrp {

// Stencil tables (GetSamples23_ / SphereRandom3, core/vector.cu:82-405),
// filled from the host: per sample offset, mip layer, and the HG-LUT row
// coordinate v (depends only on the sample), plus the 160 unit directions of
// the model file.
__constant__ float c_offset[192];
__constant__ int c_layer[192];
__constant__ float c_lutv[192];
__constant__ float c_dirs[160 * 3];
__constant__ float c_udirs[160 * 3];   // the same directions normalised (host, double precision)
// The fast gather's per-point constants packed for one 16-byte load each:
// (direction x, y, z, offset) and (unit direction x, y, z, LUT row v); the
// directions are 0 for the light-ray points 160..191.
__constant__ float4 c_pt0[192], c_pt1[192];

// The 192 points as the runs of GetSamples23_'s layout: layers 0..7 over the
// 160 rotated directions (8, 8, 16, 16, 16, 32, 32, 32 points), then layers
// 0..3 on the light ray (8 points each); the runs of 32 in halves, for the
// parts below.  set_stencil_tables checks that the tables it loads have this
// layout.
constexpr int kRuns = 15;
#define MRP_STENCIL_RUNS                                                                                              \
    {{0, 0, 8}, {1, 8, 16}, {2, 16, 32}, {3, 32, 48}, {4, 48, 64}, {5, 64, 80}, {5, 80, 96}, {6, 96, 112},            \
     {6, 112, 128}, {7, 128, 144}, {7, 144, 160}, {0, 160, 168}, {1, 168, 176}, {2, 176, 184}, {3, 184, 192}}
constexpr int kStencilRuns[kRuns][3] = MRP_STENCIL_RUNS;
__constant__ int c_stencil_runs[kRuns][3] = MRP_STENCIL_RUNS;
#undef MRP_STENCIL_RUNS
// The runs in six parts of 32 points each and in twelve of 16: first run of
// part p, and the end.
__constant__ int c_stencil_parts[2][13] = {{0, 3, 5, 7, 9, 11, kRuns}, {0, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 13, kRuns}};
cudaError_t set_stencil_tables(const StencilTables& t) {
    cudaError_t e;
    // the staged gather is compiled for the runs of kStencilRuns
    for (const auto& run : kStencilRuns)
        for (int i = run[1]; i < run[2]; ++i)
            if (t.layer[i] != run[0]) return cudaErrorInvalidValue;
    if ((e = cudaMemcpyToSymbol(c_offset, t.offset, sizeof t.offset)) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(c_layer, t.layer, sizeof t.layer)) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(c_lutv, t.lut_v, sizeof t.lut_v)) != cudaSuccess) return e;
    float ud[160 * 3];
    for (int i = 0; i < 160; ++i) {
        double x = t.dirs[3 * i], y = t.dirs[3 * i + 1], z = t.dirs[3 * i + 2];
        double l = std::sqrt(x * x + y * y + z * z);
        if (!(l > 0)) {   // the hit point itself (point 0, whose X_Hg is HG(X . L))
            if (i != 0) return cudaErrorInvalidValue;
            l = 1.0;
        }
        ud[3 * i] = (float)(x / l); ud[3 * i + 1] = (float)(y / l); ud[3 * i + 2] = (float)(z / l);
    }
    if ((e = cudaMemcpyToSymbol(c_udirs, ud, sizeof ud)) != cudaSuccess) return e;
    float4 p0[192], p1[192];
    for (int i = 0; i < 192; ++i) {
        const bool rot = i < 160;
        p0[i] = make_float4(rot ? t.dirs[3 * i] : 0.0f, rot ? t.dirs[3 * i + 1] : 0.0f, rot ? t.dirs[3 * i + 2] : 0.0f,
                            t.offset[i]);
        p1[i] = make_float4(rot ? ud[3 * i] : 0.0f, rot ? ud[3 * i + 1] : 0.0f, rot ? ud[3 * i + 2] : 0.0f, t.lut_v[i]);
    }
    if ((e = cudaMemcpyToSymbol(c_pt0, p0, sizeof p0)) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(c_pt1, p1, sizeof p1)) != cudaSuccess) return e;
    return cudaMemcpyToSymbol(c_dirs, t.dirs, sizeof t.dirs);
}

MRP_D float density(const VolumeDev& v, f3 p) { return density_tex(v, p); }
MRP_D const float* mip_level(const VolumeDev& v, int m) { return v.mips + mip_offset(m); }
MRP_D const float* tr_level(const VolumeDev& v, int m) { return v.trs + tr_offset(m); }

// RenderCamera ray (core/volume.cu:208-216): jitter = first two draws of the
// pixel stream.
MRP_D f3 camera_ray(const ViewDev& w, int row, int col) { return camera_ray_dir(w, row, col); }

// Density() at pos + dir * t for the march, skipping the 8 texel loads when
// an occupancy brick proves the trilinear footprint all zero.  The brick is
// found from X = c + sR * t per axis (c = (pos + 0.5) * R - 0.5, sR = dir *
// R, one FMA), which differs from the fetch's own texel coordinate by far
// less than one voxel; the bricks carry one voxel of apron more than a
// fetch needs, so the brick of floor(X) (clamped to the grid) holds the
// fetch's whole footprint either way.  lerp(0, 0, w) is exactly +0, so the
// skip returns the value the fetch would, and otherwise the fetch runs on
// the exact position.
struct MarchRay {
    f3 pos, dir;
    f3 c, sR;   // texel coordinate X(t) = c + sR * t, per axis
    f3 isR;     // 1 / sR (0 where sR == 0)
};
MRP_D MarchRay march_ray(const VolumeDev& v, f3 pos, f3 dir) {
    const float nf = (float)v.res;
    MarchRay m;
    m.pos = pos;
    m.dir = dir;
    m.c = mk3((pos.x + 0.5f) * nf - 0.5f, (pos.y + 0.5f) * nf - 0.5f, (pos.z + 0.5f) * nf - 0.5f);
    m.sR = mk3(dir.x * nf, dir.y * nf, dir.z * nf);
    m.isR = mk3(m.sR.x != 0.0f ? 1.0f / m.sR.x : 0.0f, m.sR.y != 0.0f ? 1.0f / m.sR.y : 0.0f,
                m.sR.z != 0.0f ? 1.0f / m.sR.z : 0.0f);
    return m;
}
// The largest t up to which X(t) stays inside brick b (base voxels
// [b << sh, (b + 1) << sh)) on one axis, with a 1/64-voxel margin: X(t) is
// a single rounded FMA, monotone in t, and the margin is far above the
// rounding of X or of this bound.
MRP_D float brick_exit(float c, float sR, float isR, int b, int sh) {
    const float m = 1.0f / 64.0f;
    if (sR > 0.0f) return ((float)((b + 1) << sh) - m - c) * isR;
    if (sR < 0.0f) return ((float)(b << sh) + m - c) * isR;
    return 3.0e38f;
}
// *t_brick: when the brick proves the value 0 and the base voxel lies inside
// the grid, the t up to which the ray stays in that brick -- or in its
// coarse brick of 4^3 bricks, when that one is empty as well -- (the march's
// next steps there read 0 as well); else -1.  The coarse brick is looked up
// only after an empty brick, so steps inside the cloud pay nothing for it.
template <class DT>
MRP_D float density_skip(const VolumeDev& v, const MarchRay& m, float t, Tally* tl, float* t_brick) {
    const int R1 = v.res - 1, sh = v.occ_shift, nb = v.occ_res;
    const int xi = __float2int_rd(fmaf(m.sR.x, t, m.c.x));
    const int yi = __float2int_rd(fmaf(m.sR.y, t, m.c.y));
    const int zi = __float2int_rd(fmaf(m.sR.z, t, m.c.z));
    const int x = min(max(xi, 0), R1) >> sh, y = min(max(yi, 0), R1) >> sh, z = min(max(zi, 0), R1) >> sh;
    *t_brick = -1.0f;
    if (__ldg(v.occ + (x * nb + y) * nb + z) == 0) {
        if ((unsigned)xi <= (unsigned)R1 && (unsigned)yi <= (unsigned)R1 && (unsigned)zi <= (unsigned)R1) {
            int bx = x, by = y, bz = z, bs = sh;
            const int nc = v.occ2_res;
            if (v.occ2 && __ldg(v.occ2 + ((x >> 2) * nc + (y >> 2)) * nc + (z >> 2)) == 0) {
                bx = x >> 2; by = y >> 2; bz = z >> 2; bs = sh + 2;
            }
            *t_brick = fminf(brick_exit(m.c.x, m.sR.x, m.isR.x, bx, bs),
                             fminf(brick_exit(m.c.y, m.sR.y, m.isR.y, by, bs), brick_exit(m.c.z, m.sR.z, m.isR.z, bz, bs)));
        }
        return 0.0f;
    }
    if (tl) tl->fetches++;
    return density_as<DT>(v, add(m.pos, mul(m.dir, t)));
}

// The march's runs of empty steps, `while (loop < lim && t <= b_le && t <
// b_lt) { ++loop; t += e; }`, in closed form.  When e = 1 / res is a power
// of two and t a multiple of it, every one of those additions is exact (t
// stays a small integer times e), so the run ends at the first multiple of
// e past the bounds, or after lim - loop steps: the same t and loop as the
// additions one by one.  inv_e = res.  False (nothing done) when t is not a
// multiple of e; the caller then adds step by step.
MRP_D bool replay_empty(float& t, int& loop, float inv_e, float e, float b_le, float b_lt, int lim) {
    const float j0 = t * inv_e;   // exact: inv_e is a power of two
    if (j0 != floorf(j0)) return false;
    const float cap = 16777216.0f;  // 2^24: beyond any reachable step count
    const float j_le = floorf(fminf(b_le * inv_e, cap));
    const float j_lt = ceilf(fminf(b_lt * inv_e, cap)) - 1.0f;
    const float jm = fminf(j_le, j_lt);
    int k = jm >= j0 ? (int)(jm - j0) + 1 : 0;
    k = min(k, max(lim - loop, 0));
    loop += k;
    t = (j0 + (float)k) * e;        // exact: an integer below 2^24 times a power of two
    return true;
}

// DeterminateEstimatedHit(float& alpha, ...) (core/render.cuh:105-197).
// pass_rate = exp(-t_step * SMax) is computed once on the host.  DT: the
// density grid's storage type (void: read from the volume per fetch).
template <class DT = void>
MRP_D bool estimated_hit(const VolumeDev& v, float alpha, float pass_rate, f3 pos, f3 dir, float dis, f3* next,
                         Tally* tl = nullptr) {
    float smax = fm(v.max_density, alpha);
    float t = 0.0f, last_non_empty_t = 0.0f, prob = 1.0f, last_dens = 0.0f;
    float rf = (float)v.res;
    float t_step = fd(2.0f, rf), empty_step = fd(1.0f, rf);
    // runs of empty steps replay in closed form on power-of-two grids (the
    // counting copy adds step by step: it tallies every step)
    const bool pow2 = !tl && (v.res & (v.res - 1)) == 0;
    const MarchRay mr = march_ray(v, pos, dir);
    int loop = 0;
    float t_exit = 3.0e38f;   // beyond it (and within dis) every step reads 0
    if (v.has_bounds) {
        // Up to where the ray enters the box outside which Density() is 0,
        // every step reads 0 and only advances t by empty_step (last_dens,
        // prob and last_non_empty_t stay at their initial values), so those
        // steps are replayed as additions alone, in the same float order.
        float t0 = 0.0f, t1 = dis;
        const float o[3] = {pos.x, pos.y, pos.z}, dd[3] = {dir.x, dir.y, dir.z};
        const float lo[3] = {v.nz_lo.x, v.nz_lo.y, v.nz_lo.z}, hi[3] = {v.nz_hi.x, v.nz_hi.y, v.nz_hi.z};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (dd[a] == 0.0f) {
                if (o[a] < lo[a] || o[a] > hi[a]) t0 = 3.0e38f;
            } else {
                const float ta = (lo[a] - o[a]) / dd[a], tb = (hi[a] - o[a]) / dd[a];
                t0 = fmaxf(t0, fminf(ta, tb));
                t1 = fminf(t1, fmaxf(ta, tb));
            }
        }
        const bool never = t0 > t1;   // the march segment [0, dis] stays where the density is 0
        if (never && !tl) {           // it would step until t > dis and report no hit
            *next = mk3(0, 0, 0);
            return false;
        }
        const float t_enter = never ? 3.0e38f : t0;
        if (!never) t_exit = t1;
        if (pow2) replay_empty(t, loop, rf, empty_step, dis, t_enter, 10000);
        while (loop < 10000 && t <= dis && t < t_enter) {
            ++loop;
            if (tl) tl->steps++;
            t = fa(t, empty_step);
        }
    }
    while (loop++ < 10000) {
        if (t > dis) {
            if (last_non_empty_t != 0.0f) { t = last_non_empty_t; break; }
            *next = mk3(0, 0, 0);
            return false;
        }
        if (!tl && t > t_exit && !(last_dens > 0.0f)) {
            // Past the nonzero box every step reads 0 and, with no pending
            // transition from density, only advances t by empty_step; each
            // step advances t by at least empty_step, so the loop cannot
            // reach its iteration bound before t > dis: the outcome is the
            // one the t > dis test above gives.
            if (last_non_empty_t != 0.0f) { t = last_non_empty_t; break; }
            *next = mk3(0, 0, 0);
            return false;
        }
        if (tl) tl->steps++;
        float d, t_brick = -1.0f;
        if (v.occ) {
            d = density_skip<DT>(v, mr, t, tl, &t_brick);
        } else {
            d = density_as<DT>(v, add(pos, mul(dir, t)));
            if (tl) tl->fetches++;
        }
        if (d > 0) {
            float S = fm(d, alpha);
            float step_p = fa(pass_rate, fm(fs(1.0f, pass_rate), fs(1.0f, fd(S, smax))));
            float next_p = fm(prob, step_p);
            if (next_p < 0.5f) {
                float offset = fs(1.0f, fd(logf(fd(0.5f, prob)), logf(step_p)));
                t = fs(t, fm(t_step, offset));
                break;
            }
            prob = next_p;
            t = fa(t, t_step);
        } else {
            if (last_dens > 0) {
                float S = fm(last_dens, alpha);
                float ts = fa(t_step, d);
                // exp(-(ts*SMax)) == pass_rate when d == 0 (same argument)
                float pr = d == 0.0f ? pass_rate : expf(-fm(ts, smax));
                float step_p = fa(pr, fm(fs(1.0f, pr), fs(1.0f, fd(S, smax))));
                float next_p = fm(prob, step_p);
                if (next_p < 0.5f) {
                    float offset = fs(1.0f, fd(logf(fd(0.5f, prob)), logf(step_p)));
                    t = fs(t, fm(ts, offset));
                    break;
                }
                prob = next_p;
                last_non_empty_t = fa(t, d);
            }
            t = fa(t, fmaxf(fm(-d, 1.0f), empty_step));
        }
        last_dens = d;
        // The step read 0 from an empty brick: the following steps that
        // start inside the brick read 0 too and, last_dens being 0, only
        // advance t by empty_step -- replayed as additions alone.
        if (pow2 && t_brick >= 0.0f) replay_empty(t, loop, rf, empty_step, fminf(t_brick, dis), 3.0e38f, 10000);
        while (t <= t_brick && t <= dis && loop < 10000) {
            ++loop;
            if (tl) tl->steps++;
            t = fa(t, empty_step);
        }
    }
    *next = add(mul(dir, t), pos);
    return true;
}

// GetSamplePoint (core/render.cuh:436-462)
template <class DT = void>
MRP_D bool first_hit(const VolumeDev& v, f3 ori, f3 dir, float alpha, float pass_rate, f3* hit, Tally* tl = nullptr) {
    dir = normalize(dir);
    *hit = mk3(0, 0, 0);
    float dis = ray_box_offset(ori, dir);
    if (dis < 0) return false;
    f3 sp = add(ori, mul(dir, dis));
    float md = ray_box_distance(sp, dir);
    f3 p;
    bool in = estimated_hit<DT>(v, alpha, pass_rate, sp, dir, md, &p, tl);
    if (in) *hit = p;
    return in;
}

// GetMatrixFromNormal (core/render.cuh:694-708)
MRP_D void basis(f3 v1, float spread, Stream& st, f3* b0, f3* b1, f3* b2) {
    v1 = normalize(v1);
    f3 v2 = mk3(0, 0, 0), v3 = mk3(0, 0, 0);
    for (int guard = 0; guard < 1000; ++guard) {
        float ex = fm(st.next(), spread);
        float ey = fm(st.next(), spread);
        f3 r = uniform_sphere(ex, ey);
        if (fabsf(dot(r, v1)) < 0.00001) continue;
        v2 = normalize(cross(v1, r));
        v3 = cross(v2, v1);
        break;
    }
    *b0 = v1; *b1 = v2; *b2 = v3;
}

// ShadowTerm_TRTex(...).x with unit light colour (core/renderResources.cu:254-272)
MRP_D float shadow_tr(const VolumeDev& v, f3 p, f3 light, int mip) {
    const float* g = tr_level(v, mip);
    int n = 128 >> mip;
    if (p.x < -0.5f || p.y < -0.5f || p.z < -0.5f || p.x > 0.5f || p.y > 0.5f || p.z > 0.5f) {
        float off = ray_box_offset(p, light);
        if (off >= 0) return fm(1.0f, tex3<true>(g, n, add(p, mul(light, off))));
        return 1.0f;
    }
    return fm(1.0f, tex3<true>(g, n, p));
}

// One stencil point of SetupInputData (core/radiancePredict.cu:433-471):
// density (X_Val), TR (X_Val_Sub) and HG (X_Val_Hg) features of sample i.
struct PixelFrame { f3 pos, X, Y, Z, LX, L; float g, alpha; };

MRP_D void gather_sample(const VolumeDev& v, const PixelFrame& f, int i, float* fd_, float* fs_, float* fh_) {
    float off = c_offset[i];
    int layer = c_layer[i];
    f3 cur;
    if (i < 160) {
        f3 p = mk3(c_dirs[3 * i], c_dirs[3 * i + 1], c_dirs[3 * i + 2]);
        cur = add(f.pos, mul(add(add(mul(f.X, p.x), mul(f.Y, p.y)), mul(f.Z, p.z)), off));
    } else {
        cur = add(f.pos, mul(f.L, off));
    }
    // plain fetch: brick tests here cost more than the skipped loads (measured)
    float d = tex3<false>(mip_level(v, layer), 256 >> layer, cur);
    // x / 64 == x * 2^-6 exactly (both round the same real number)
    *fd_ = logf(fa(1.0f, fm(fm(f.alpha, d), 0.015625f)));
    if (i == 0) {
        *fh_ = logf(fa(hg(dot(f.X, f.L), f.g), 1.0f));
    } else {
        f3 ms = normalize(sub(cur, f.pos));
        float c1 = dot(f.X, ms), c2 = dot(f.LX, ms);
        float u = fa(fm(c1, 0.5f), 0.5f), u2 = fa(fm(c2, 0.5f), 0.5f);
        float lv = c_lutv[i];
        *fh_ = logf(fa(fm(tex_lut(v.lut, u, lv), tex_lut(v.lut, u2, lv)), 1.0f));
    }
    *fs_ = shadow_tr(v, cur, f.LX, layer > 1 ? layer - 1 : 0);
}
// The same stencil point with contracted arithmetic (FMA positions and
// lerps, rsqrt direction), used by the staged gather of the render path:
// the features stay within 1e-5 relative of gather_sample.
// The fp16 path's per-record constants of X_Hg.  A rotated point's
// direction from the hit is X px + Y py + Z pz for its unit stencil
// direction (px, py, pz), so its cosine with X is px (a per-point constant:
// its LUT factor is lut_dirs[i]) and its cosine with LX is q . (px, py, pz),
// q = (LX.X, LX.Y, LX.Z); a light-ray point's direction is L itself.  The
// exact form normalises cur - pos; the two differ by rounding (< 1e-6 in
// the cosine), far below an fp16 step of the feature.
struct HgFast {
    f3 q;
    float u1L, u2L;          // LUT coordinates of the light-ray points
    const float* lut_dirs;
};
MRP_D HgFast hg_fast(const VolumeDev& v, const PixelFrame& f) {
    HgFast h;
    h.q = mk3(dot(f.LX, f.X), dot(f.LX, f.Y), dot(f.LX, f.Z));
    h.u1L = fmaf(dot(f.X, f.L), 0.5f, 0.5f);
    h.u2L = fmaf(dot(f.LX, f.L), 0.5f, 0.5f);
    h.lut_dirs = v.lut_dirs;
    return h;
}
__global__ void k_lut_dirs(const float* __restrict__ lut, float* __restrict__ out) {
    int i = threadIdx.x;
    if (blockIdx.x == 192) {
        if (i < 160) out[i] = tex_lut_fast(lut, fmaf(c_udirs[3 * i], 0.5f, 0.5f), c_lutv[i]);
        return;
    }
    // point blockIdx.x's row: tex_lut_fast's y and its blend of two texels
    const float py = fmaf(c_lutv[blockIdx.x], (float)kLut, -0.5f), fly = floorf(py), wy = py - fly;
    const int y = (int)fly;
    const float* r0 = lut + min(max(y, 0), kLut - 1) * kLut;
    const float* r1 = lut + min(max(y + 1, 0), kLut - 1) * kLut;
    float* row = out + (kLutRows - kLut * kLut) + blockIdx.x * kLutRow;
    for (int x = i - 1; x <= kLut; x += blockDim.x) {
        const int x0 = min(max(x, 0), kLut - 1);
        row[x + 1] = lerp_fast(r0[x0], r1[x0], wy);
    }
}
MRP_D const float* lut_row(const VolumeDev& v, int i) {
    return v.lut_dirs + (kLutRows - kLut * kLut) + i * kLutRow;
}
cudaError_t launch_lut_dirs(const float* lut, float* out, cudaStream_t s) {
    k_lut_dirs<<<193, 256, 0, s>>>(lut, out);
    return cudaGetLastError();
}

// Stencil point i with the sizes and levels of its run hoisted by the
// caller: mip level m (n^3 texels), TR level (tn^3), and whether the point
// lies on the light ray (i >= 160) rather than along a rotated direction.
struct RunLevels {
    const float* mip;
    const float* tr;
    int n, tn;
    bool light;
    bool mip_pad, tr_pad;   // mip / tr point at a padded copy (tex3_padded)
    const float2* pair;     // the run's (mip, TR) texel pairs (mip_tr or pad_pair), or null
    bool pair_pad;          // pair is a padded pair level
};
// FP16: the features are stored as fp16, so the two logs use the hardware
// log2 (__logf, absolute error < 4e-7 on the arguments here, all >= 1), which
// is below half an fp16 step of every output above 1e-3.
template <bool FP16>
MRP_D float feature_log(float x) { return FP16 ? __logf(x) : logf(x); }

template <bool FP16>
MRP_D void gather_point_fast(const VolumeDev& v, const PixelFrame& f, const RunLevels& R, const HgFast& H, f3 iLX,
                             int i, float* fd_, float* fs_, float* fh_) {
    const float4 p0 = c_pt0[i], p1 = c_pt1[i];
    const float off = p0.w;
    f3 d;   // offset from the point
    if (!R.light) {
        const float px = p0.x, py = p0.y, pz = p0.z;
        d = mk3(fmaf(f.Z.x, pz, fmaf(f.Y.x, py, f.X.x * px)) * off, fmaf(f.Z.y, pz, fmaf(f.Y.y, py, f.X.y * px)) * off,
                fmaf(f.Z.z, pz, fmaf(f.Y.z, py, f.X.z * px)) * off);
    } else {
        d = mk3(f.L.x * off, f.L.y * off, f.L.z * off);
    }
    const f3 cur = mk3(f.pos.x + d.x, f.pos.y + d.y, f.pos.z + d.z);
    // ShadowTerm_TRs reads the TR at the point itself inside the box, else
    // where the light ray enters the box
    const bool outside = cur.x < -0.5f || cur.y < -0.5f || cur.z < -0.5f || cur.x > 0.5f || cur.y > 0.5f || cur.z > 0.5f;
    float dens, tr_pair = 0.0f;
    bool paired = false;
    if (R.pair && !outside) {
        if (R.pair_pad) {
            tex3_padded_pair(R.pair, R.n, cur, &dens, &tr_pair);
            paired = true;
        } else {
            paired = tex3_pair_interior(R.pair, R.n, cur, &dens, &tr_pair);
        }
    }
    if (!paired) dens = R.mip_pad ? tex3_padded(R.mip, R.n, cur) : tex3_fast<false>(R.mip, R.n, cur);
    *fd_ = feature_log<FP16>(fmaf(f.alpha * dens, 0.015625f, 1.0f));
    if (i == 0) {
        *fh_ = feature_log<FP16>(hg(dot(f.X, f.L), f.g) + 1.0f);
    } else if (FP16) {
        const float* row = lut_row(v, i);
        float a, b;
        if (!R.light) {
            const float c2 = fmaf(H.q.z, p1.z, fmaf(H.q.y, p1.y, H.q.x * p1.x));
            a = __ldg(H.lut_dirs + i);
            b = lut_row_fast(row, fmaf(c2, 0.5f, 0.5f));
        } else {
            a = lut_row_fast(row, H.u1L);
            b = lut_row_fast(row, H.u2L);
        }
        *fh_ = feature_log<FP16>(fmaf(a, b, 1.0f));
    } else {
        f3 ms = mk3(cur.x - f.pos.x, cur.y - f.pos.y, cur.z - f.pos.z);
        float rl = rsqrtf(fmaf(ms.z, ms.z, fmaf(ms.y, ms.y, ms.x * ms.x)));
        ms = mk3(ms.x * rl, ms.y * rl, ms.z * rl);
        float c1 = fmaf(f.X.z, ms.z, fmaf(f.X.y, ms.y, f.X.x * ms.x));
        float c2 = fmaf(f.LX.z, ms.z, fmaf(f.LX.y, ms.y, f.LX.x * ms.x));
        const float* row = lut_row(v, i);
        *fh_ = feature_log<FP16>(fmaf(lut_row_fast(row, fmaf(c1, 0.5f, 0.5f)), lut_row_fast(row, fmaf(c2, 0.5f, 0.5f)), 1.0f));
    }
    // ShadowTerm_TRs: outside the box, the TR where the light ray enters it
    const f3 p = cur, light = f.LX;
    float tr = 1.0f;
    if (paired) {
        tr = tr_pair;
    } else {
        f3 q = p;
        bool fetch = true;
        if (outside) {
            float o = ray_box_offset_inv(p, iLX);   // iLX = inv(light), once per record
            fetch = o >= 0;
            q = mk3(fmaf(light.x, o, p.x), fmaf(light.y, o, p.y), fmaf(light.z, o, p.z));
        }
        if (fetch) tr = R.tr_pad ? tex3_padded(R.tr, R.tn, q) : tex3_fast<true>(R.tr, R.tn, q);
    }
    *fs_ = tr;
}
// The points of runs [first_run, end_run) (0, kRuns: all 192), run by run (GetSamples23_'s layout: layers 0..7 over the
// 160 rotated directions, then layers 0..3 on the light ray), into a tiled
// feature layout: fp32 (record r, channel c, sample i at word
// ((r / 32) * 576 + c * 192 + i) * 32 + r % 32), or FP16 pairs (samples 2k,
// 2k + 1 of channel c as one half2 at word ((r / 32) * 288 + c * 96 + k) * 32
// + r % 32).  Either way a warp of 32 records writes 128 contiguous bytes.
template <bool FP16>
MRP_D void gather_all_fast(const VolumeDev& v, const PixelFrame& f, float* feat, int r, int first_run, int end_run) {
    float* out = feat + (size_t)(r >> 5) * 576 * 32 + (r & 31);
    __half2* out2 = reinterpret_cast<__half2*>(feat) + (size_t)(r >> 5) * 288 * 32 + (r & 31);
    float pa = 0.0f, pb = 0.0f, pc = 0.0f;   // the even sample of a pair
    const HgFast H = FP16 ? hg_fast(v, f) : HgFast{mk3(0, 0, 0), 0.0f, 0.0f, nullptr};
    const f3 iLX = inv(f.LX);
#pragma unroll 1
    for (int run = first_run; run < end_run; ++run) {
        const int layer = c_stencil_runs[run][0], from = c_stencil_runs[run][1], to = c_stencil_runs[run][2];
        const int tl = layer > 1 ? layer - 1 : 0;
        // edge <= 8 (mips 5..7, TR levels 4..6): most footprints touch the
        // grid's edge, so those runs read the padded copies when present
        const bool mp = v.mips_pad && layer >= 5, tp = v.trs_pad && tl >= 4;
        // layers 1..4: mip level and TR level share the edge 256 >> layer
        // layers 5..7: the padded pairs (mips 5..7 with TR levels 4..6)
        const bool pp = mp && tp && v.pad_pair;
        const float2* pr = pp ? v.pad_pair + pad_offset(256 >> layer)
                           : v.mip_tr && layer >= 1 && layer <= 4 ? v.mip_tr + mip_tr_offset(layer) : nullptr;
        const RunLevels R{mp ? v.mips_pad + pad_offset(256 >> layer) : mip_level(v, layer),
                          tp ? v.trs_pad + pad_offset(128 >> tl) : tr_level(v, tl), 256 >> layer, 128 >> tl,
                          from >= 160, mp, tp, pr, pp};
#pragma unroll 1
        for (int i = from; i < to; ++i) {
            float a, b, c;
            gather_point_fast<FP16>(v, f, R, H, iLX, i, &a, &b, &c);
            if (!FP16) {
                out[i * 32] = a;
                out[(192 + i) * 32] = b;
                out[(384 + i) * 32] = c;
            } else if (i & 1) {   // runs start on even samples
                const int k = i >> 1;
                out2[k * 32] = __floats2half2_rn(pa, a);
                out2[(96 + k) * 32] = __floats2half2_rn(pb, b);
                out2[(192 + k) * 32] = __floats2half2_rn(pc, c);
            } else {
                pa = a; pb = b; pc = c;
            }
        }
    }
}
// The fp16-feature gather through the texture unit (gather_filter): the
// reference's own sampling in SetupInputData (core/radiancePredict.cu:
// 433-471) -- tex3D on Mip(layer) (border) and TR_Mip(layer - 1) (clamp),
// tex2D on _HGLut (clamp), weights quantised by the filter to 1/256 -- in
// place of the software trilinear of gather_point_fast.  Layers 1..7 read
// mip and TR from one pair texture (one fetch for both where the point is
// inside the volume); layer 0 (mip 256^3, TR 128^3) from two textures.
// Everything around the fetches is gather_point_fast's: stencil positions,
// X_Hg's per-record constants, ShadowTerm_TRTex's box entry for points
// outside the volume.
MRP_D float tex_at(cudaTextureObject_t t, f3 p) { return tex3D<float>(t, p.z + 0.5f, p.y + 0.5f, p.x + 0.5f); }
// pair texel coordinate of p on a level of edge n: (p + 0.5) n + 1, the
// padded grid's unnormalized coordinate (voxel i centred at i + 1.5)
MRP_D float2 pair_at(cudaTextureObject_t t, float n, float c, f3 p) {
    return tex3D<float2>(t, fmaf(p.z, n, c), fmaf(p.y, n, c), fmaf(p.x, n, c));
}
struct TexRun {
    cudaTextureObject_t a, b;   // layer 0: mip, TR; else the pair (a) of the run's layer
    float n, c;                 // the pair level's edge and coordinate offset n / 2 + 1
    bool pair, light;
};
MRP_D void gather_point_tex(const VolumeDev& v, const PixelFrame& f, const TexRun& R, const HgFast& H, f3 iLX, int i,
                            float* fd_, float* fs_, float* fh_) {
    const float4 p0 = c_pt0[i], p1 = c_pt1[i];
    const float off = p0.w;
    f3 d;
    if (!R.light) {
        const float px = p0.x, py = p0.y, pz = p0.z;
        d = mk3(fmaf(f.Z.x, pz, fmaf(f.Y.x, py, f.X.x * px)) * off, fmaf(f.Z.y, pz, fmaf(f.Y.y, py, f.X.y * px)) * off,
                fmaf(f.Z.z, pz, fmaf(f.Y.z, py, f.X.z * px)) * off);
    } else {
        d = mk3(f.L.x * off, f.L.y * off, f.L.z * off);
    }
    const f3 cur = mk3(f.pos.x + d.x, f.pos.y + d.y, f.pos.z + d.z);
    // ShadowTerm_TRTex: the TR at the point inside the volume, else where the
    // light ray from it enters the volume (1 where it misses)
    const bool outside = cur.x < -0.5f || cur.y < -0.5f || cur.z < -0.5f || cur.x > 0.5f || cur.y > 0.5f || cur.z > 0.5f;
    float o = 0.0f;
    if (outside) o = ray_box_offset_inv(cur, iLX);
    const f3 q = mk3(fmaf(f.LX.x, o, cur.x), fmaf(f.LX.y, o, cur.y), fmaf(f.LX.z, o, cur.z));
    float dens, tr = 1.0f;
    if (R.pair) {
        const float2 m = pair_at(R.a, R.n, R.c, cur);
        dens = m.x;
        if (!outside) tr = m.y;
        else if (o >= 0) tr = pair_at(R.a, R.n, R.c, q).y;
    } else {
        dens = tex_at(R.a, cur);
        if (!outside || o >= 0) tr = tex_at(R.b, q);
    }
    *fd_ = __logf(fmaf(f.alpha * dens, 0.015625f, 1.0f));
    *fs_ = tr;
    if (i == 0) {
        *fh_ = __logf(hg(dot(f.X, f.L), f.g) + 1.0f);
    } else {
        const float lv = p1.w;
        float a, b;
        if (!R.light) {
            // this LUT read in software from the fp32 table, the light-ray
            // points' two through the texture unit: the stencil's trilinear
            // fetches keep the texture pipe the gather's tighter limit, and
            // this split balances it against the load pipe (1024^2 frame:
            // 0.468 ms all through the texture unit, 0.460 this way, 0.512
            // with every LUT read in software)
            const float c2 = fmaf(H.q.z, p1.z, fmaf(H.q.y, p1.y, H.q.x * p1.x));
            a = __ldg(H.lut_dirs + i);
            b = tex_lut_fast(v.lut, fmaf(c2, 0.5f, 0.5f), lv);
        } else {
            a = tex2D<float>(v.glut_tex, H.u1L, lv);
            b = tex2D<float>(v.glut_tex, H.u2L, lv);
        }
        *fh_ = __logf(fmaf(a, b, 1.0f));
    }
}
MRP_D void gather_all_tex(const VolumeDev& v, const PixelFrame& f, float* feat, int r, int first_run, int end_run) {
    __half2* out2 = reinterpret_cast<__half2*>(feat) + (size_t)(r >> 5) * 288 * 32 + (r & 31);
    float pa = 0.0f, pb = 0.0f, pc = 0.0f;   // the even sample of a pair
    const HgFast H = hg_fast(v, f);
    const f3 iLX = inv(f.LX);
#pragma unroll 1
    for (int run = first_run; run < end_run; ++run) {
        const int layer = c_stencil_runs[run][0], from = c_stencil_runs[run][1], to = c_stencil_runs[run][2];
        const float n = (float)(256 >> layer);
        const TexRun R = layer == 0 ? TexRun{v.gmip0_tex, v.gtr0_tex, 0.0f, 0.0f, false, from >= 160}
                                    : TexRun{v.gpair_tex[layer], 0, n, fmaf(n, 0.5f, 1.0f), true, from >= 160};
#pragma unroll 1
        for (int i = from; i < to; ++i) {
            float a, b, c;
            gather_point_tex(v, f, R, H, iLX, i, &a, &b, &c);
            if (i & 1) {   // runs start on even samples
                const int k = i >> 1;
                out2[k * 32] = __floats2half2_rn(pa, a);
                out2[(96 + k) * 32] = __floats2half2_rn(pb, b);
                out2[(192 + k) * 32] = __floats2half2_rn(pc, c);
            } else {
                pa = a; pb = b; pc = c;
            }
        }
    }
}
MRP_D float gamma_of(const PixelFrame& f) { return acosf(fminf(1.0f, fmaxf(-1.0f, dot(f.X, f.LX)))); }

// All 192 points; feature i of channel c to out[c * stride + i].
MRP_D void gather(const VolumeDev& v, const PixelFrame& f, float* out, int stride, float* gamma) {
    for (int i = 0; i < 192; ++i) gather_sample(v, f, i, out + i, out + stride + i, out + 2 * stride + i);
    *gamma = gamma_of(f);
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
__global__ void k_first_hit(VolumeDev v, const float* __restrict__ ori, const float* __restrict__ dir, float alpha,
                            float pass_rate, int n, float* __restrict__ hit4) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    f3 h;
    bool in = first_hit(v, ld3(ori + 3 * i), ld3(dir + 3 * i), alpha, pass_rate, &h);
    hit4[4 * i] = h.x; hit4[4 * i + 1] = h.y; hit4[4 * i + 2] = h.z; hit4[4 * i + 3] = in ? 1.0f : 0.0f;
}

// bases: [n][15] = X, Y, Z (main basis), LX (light basis x), unused
__global__ void k_gather(VolumeDev v, const float* __restrict__ pos, const float* __restrict__ bases,
                         const float* __restrict__ light, float g, float alpha, int n, float* __restrict__ feat,
                         float* __restrict__ gamma) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* b = bases + 12 * i;
    PixelFrame f{ld3(pos + 3 * i), ld3(b), ld3(b + 3), ld3(b + 6), ld3(b + 9), ld3(light), g, alpha};
    gather(v, f, feat + (size_t)576 * i, 192, gamma + i);
}

// ---------------------------------------------------------------------------
// Staged predictor: one launch of RenderCamera<true, MRPNN> is
//   k_hit     per pixel: ray, first hit, bases; hit pixels appended to a
//             compact record list, missed pixels resolved to the sky;
//   k_gather  per record: the 192-point stencil -> tiled features;
//   k_mlp_*   per record: the network -> running mean at the record's pixel.
// ---------------------------------------------------------------------------
// 128-thread blocks, eight resident per SM (64 registers), each warp taking
// 32 pixels at a time: march lengths vary from 0 to ~1000 steps.
constexpr int kHitThreads = 128;
// One warp's 32 pixels (lane = pixel pix); every lane of the warp calls it.
template <bool COUNT, class DT, bool ENV>
MRP_D void hit_pixels(const VolumeDev& v, const ViewDev& w, const HitRecords& rec, float4* __restrict__ accum,
                      int pix) {
    Tally tally;
    int npix = w.width * w.height;
    bool valid = pix >= 0 && pix < npix && pixel_selected(w, pix / w.width, pix % w.width);
    bool active = false;
    f3 hit = mk3(0, 0, 0), X, Y, Z, LX;
    if (valid) {
        int row = pix / w.width, col = pix % w.width;
        f3 ori = w.ori, dir;
        if (w.ray_dir) {                                     // GetRadiances: explicit rays
            ori = mk3(w.ray_ori[3 * pix], w.ray_ori[3 * pix + 1], w.ray_ori[3 * pix + 2]);
            dir = normalize(mk3(w.ray_dir[3 * pix], w.ray_dir[3 * pix + 1], w.ray_dir[3 * pix + 2]));
        } else {
            dir = normalize(camera_ray(w, row, col));        // NNPredict: dir = normalize(dir)
        }
        f3 L = normalize(w.light_dir);
        Stream st(kPixelStream, (uint32_t)pix, 0, (uint32_t)w.frame, w.seed);   // InitRand again
        active = first_hit<DT>(v, ori, dir, w.alpha, w.pass_rate, &hit, COUNT ? &tally : nullptr);
        if (COUNT) {
            tally.events += active ? 1 : 0;
            tally.lookups += active ? 192 : 0;
            flush_tally(w.counters, tally);
        }
        if (active) {   // the bases only matter for a hit (they draw after the march)
            f3 LY, LZ;
            basis(dir, 0.1f, st, &X, &Y, &Z);
            basis(L, 0.1f, st, &LX, &LY, &LZ);
        } else {        // NNPredict returns SkyBox(dir) for a ray that finds no hit
            // (the map lookup only in the copy compiled for volumes with an
            // environment map: its call would cost the march registers)
            const f3 sk = ENV ? sky_map(v.hdri, v.hdri_w, v.hdri_h, v.env_exp, dir) : v.sky;
            running_mean(accum, pix, w.mean_k, make_float4(sk.x, sk.y, sk.z, -1.0f));
        }
    }
    // warp-aggregated append of the hit pixels
    unsigned lane = threadIdx.x & 31;
    unsigned m = __ballot_sync(0xffffffffu, active);
    if (m == 0) return;
    int base = 0;
    if (lane == (unsigned)(__ffs(m) - 1)) base = atomicAdd(rec.count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
    if (!active) return;
    int r = base + __popc(m & ((1u << lane) - 1u));
    size_t cap = rec.cap;
    rec.pix[r] = pix;
    float* f = rec.f + r;
    float vals[16] = {hit.x, hit.y, hit.z, X.x, X.y, X.z, Y.x, Y.y, Y.z, Z.x, Z.y, Z.z, LX.x, LX.y, LX.z,
                      gamma_of(PixelFrame{hit, X, Y, Z, LX, mk3(0, 0, 0), 0.0f, 0.0f})};
#pragma unroll
    for (int k = 0; k < 16; ++k) f[k * cap] = vals[k];
}
// Persistent warps: each takes the next tile of 2^lsx x 2^lsy pixels (8 x 4;
// fewer in small launches, launch_hit) from a counter (rec.count[1]) as soon
// as its previous rays have ended, so a
// long march holds one warp, not a whole block, and the SMs stay full until
// the last tiles are handed out; the rays of a square-ish tile march more
// alike than 32 pixels of a row.  (Explicit rays, a width x 1 launch, come
// in a row.)
template <bool COUNT, class DT, bool ENV = false>
__global__ void __launch_bounds__(kHitThreads, 8) k_hit(VolumeDev v, ViewDev w, HitRecords rec, float4* __restrict__ accum,
                                                       int lsx, int lsy) {
    const int sx = 1 << lsx, sy = 1 << lsy;
    const int tx = (w.width + sx - 1) >> lsx, nchunks = tx * ((w.height + sy - 1) >> lsy);
    const int lane = (int)(threadIdx.x & 31);
    const int lx = lane & (sx - 1), ly = lane >> lsx;
    for (;;) {
        int c = 0;
        if (lane == 0) c = atomicAdd(rec.count + 1, 1);
        c = __shfl_sync(0xffffffffu, c, 0);
        if (c >= nchunks) return;
        const int col = (c % tx) * sx + lx, row = (c / tx) * sy + ly;
        hit_pixels<COUNT, DT, ENV>(v, w, rec, accum, ly < sy && col < w.width && row < w.height ? row * w.width + col : -1);
    }
}

MRP_D PixelFrame record_frame(const HitRecords& rec, int r, f3 L, float g, float alpha) {
    const float* f = rec.f + r;
    size_t c = rec.cap;
    PixelFrame pf;
    pf.pos = mk3(f[0], f[c], f[2 * c]);
    pf.X = mk3(f[3 * c], f[4 * c], f[5 * c]);
    pf.Y = mk3(f[6 * c], f[7 * c], f[8 * c]);
    pf.Z = mk3(f[9 * c], f[10 * c], f[11 * c]);
    pf.LX = mk3(f[12 * c], f[13 * c], f[14 * c]);
    pf.L = L;
    pf.g = g;
    pf.alpha = alpha;
    return pf;
}

template <bool FP16, bool TEX = false>
__global__ void __launch_bounds__(128) k_gather_rec(VolumeDev v, ViewDev w, HitRecords rec, float* __restrict__ feat) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= *rec.count) return;
    PixelFrame pf = record_frame(rec, r, normalize(w.light_dir), w.g, w.alpha);
    int first_run = 0, end_run = kRuns;
    if (gridDim.y > 1) {   // one of six or twelve parts of the stencil
        const int* parts = c_stencil_parts[gridDim.y == 6 ? 0 : 1];
        first_run = parts[blockIdx.y];
        end_run = parts[blockIdx.y + 1];
    }
    if (TEX) gather_all_tex(v, pf, feat, r, first_run, end_run);
    else gather_all_fast<FP16>(v, pf, feat, r, first_run, end_run);
}

// Per-pixel intermediates for the debug entry point: aux [npix][20] = hit
// xyz, hit flag, gamma, X, Y, Z, LX; feat [npix][576].
template <bool FP16>
__global__ void k_debug_scatter(HitRecords rec, const float* __restrict__ feat, float* __restrict__ aux,
                                float* __restrict__ feat_out) {
    int r = blockIdx.x;
    if (r >= *rec.count) return;
    int pix = rec.pix[r];
    const float* f = rec.f + r;
    float* a = aux + (size_t)pix * 20;
    if (threadIdx.x == 0) {
        a[0] = f[0]; a[1] = f[rec.cap]; a[2] = f[2 * rec.cap]; a[3] = 1.0f; a[4] = f[15 * rec.cap];
        for (int k = 0; k < 12; ++k) a[5 + k] = f[(3 + k) * rec.cap];
    }
    if (FP16) {   // fp16 pairs: word ((r / 32) * 288 + c * 96 + k) * 32 + r % 32 holds samples 2k, 2k + 1
        const __half2* src = reinterpret_cast<const __half2*>(feat) + (size_t)(r >> 5) * 288 * 32 + (r & 31);
        for (int j = threadIdx.x; j < 288; j += blockDim.x) {
            const float2 p = __half22float2(src[j * 32]);
            feat_out[(size_t)pix * 576 + 2 * j] = p.x;
            feat_out[(size_t)pix * 576 + 2 * j + 1] = p.y;
        }
    } else {
        const float* src = feat + (size_t)(r >> 5) * 576 * 32 + (r & 31);
        for (int i = threadIdx.x; i < 576; i += blockDim.x) feat_out[(size_t)pix * 576 + i] = src[i * 32];
    }
}

cudaError_t launch_first_hit(const VolumeDev& v, const float* ori, const float* dir, float alpha, float pass_rate, int n,
                             float* hit4, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_first_hit<<<(n + 127) / 128, 128, 0, s>>>(v, ori, dir, alpha, pass_rate, n, hit4);
    return cudaGetLastError();
}
cudaError_t launch_gather(const VolumeDev& v, const float* pos, const float* bases, const float* light, float g,
                          float alpha, int n, float* feat, float* gamma, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_gather<<<(n + 127) / 128, 128, 0, s>>>(v, pos, bases, light, g, alpha, n, feat, gamma);
    return cudaGetLastError();
}
cudaError_t launch_hit(const VolumeDev& v, const ViewDev& view, HitRecords rec, float4* accum, cudaStream_t s) {
    int n = view.width * view.height;
    if (n <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(rec.count, 0, 2 * sizeof(int), s);   // records, pixel chunks handed out
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
    // A warp's pixels: 8 x 4, or 4 x 4 or 4 x 2 (explicit rays: in a row) where
    // that makes at most sixteen warps an SM.  There the longest march of a
    // warp is the launch's time, and fewer lanes share its branches: 163 x 97
    // over 100^3, four launches, 529 -> 510 us, 128 x 128 over 256^3 228 -> 213;
    // from 256 x 256 on full warps are as fast (268 both) and then faster
    // (512 x 512: 500 against 543 with half of the lanes).
    const int lp = n <= sms * 128 ? 3 : n <= sms * 256 ? 4 : 5;
    const int lsy = view.height > 1 ? lp / 2 : 0, lsx = lp - lsy;
    const int chunks = ((view.width + (1 << lsx) - 1) >> lsx) * ((view.height + (1 << lsy) - 1) >> lsy);
    const int need = (chunks + kHitThreads / 32 - 1) / (kHitThreads / 32);
    const int blocks = need < sms * 8 ? need : sms * 8;   // eight resident per SM
    // one copy of the march per counting mode and density storage type, and
    // for volumes with an environment map
    if (v.hdri) {
        if (v.density_h) k_hit<false, __half, true><<<blocks, kHitThreads, 0, s>>>(v, view, rec, accum, lsx, lsy);
        else k_hit<false, float, true><<<blocks, kHitThreads, 0, s>>>(v, view, rec, accum, lsx, lsy);
    } else if (v.density_h) {
        if (view.counters) k_hit<true, __half><<<blocks, kHitThreads, 0, s>>>(v, view, rec, accum, lsx, lsy);
        else k_hit<false, __half><<<blocks, kHitThreads, 0, s>>>(v, view, rec, accum, lsx, lsy);
    } else {
        if (view.counters) k_hit<true, float><<<blocks, kHitThreads, 0, s>>>(v, view, rec, accum, lsx, lsy);
        else k_hit<false, float><<<blocks, kHitThreads, 0, s>>>(v, view, rec, accum, lsx, lsy);
    }
    return cudaGetLastError();
}
// ---------------------------------------------------------------------------
// Tile gather of the tile network (GatherData -> GatherSamples ->
// NNGatherSamples, core/volume.cu:257-282; core/render.cuh:199-397, 464-485,
// 1006-1142; SetupInputData2, core/radiancePredict.cu:487-553): per 8 x
// 8-pixel tile 773 floats: X_Val[192], X_Val_Hg[192], X_Val_Sub[192],
// 5 angle / depth-gradient terms, 192 t-grid values.  nl = {-log 0.76,
// -log 0.75, -log 0.25} from the host's logf.
// ---------------------------------------------------------------------------
struct TauState { float tau, target; bool first; };

// CheckExitCondition (core/render.cuh:199-297): trapezoid optical depth over
// the step; the crossing of the 50 % (then 25 %) survival threshold solved in
// the step.
MRP_D float exit_offset(float A, float B, float C, float dq, float dt, float S, float lastS) {
    if (fabsf(A) < 1e-6f) return fd(dq, fm(fm(dt, fa(S, lastS)), 0.5f));
    float D = fs(fm(B, B), fm(fm(4.0f, A), C));
    D = fmaxf(D, 0.0f);
    float sq = fsq(D);
    float q = fm(-0.5f, fa(B, sq));   // (float)(-0.5 * (double)(B + sq)): exact halving
    float u1 = fd(q, A), u2 = fd(C, q);
    return u1 == fminf(fmaxf(u1, 0.0f), 1.0f) ? u1 : u2;
}
MRP_D bool check_exit(float S, float lastS, float dt, float t, TauState& st, float ts[4], float tau_second) {
    float tau_next = fa(st.tau, fm(fm(fa(S, lastS), 0.5f), dt));
    if (tau_next >= st.target) {
        float dtau = fs(st.target, st.tau);
        float A = fm(fm(0.5f, dt), fs(S, lastS)), B = fm(dt, lastS);
        float off = exit_offset(A, B, -dtau, dtau, dt, S, lastS);
        off = fminf(fmaxf(off, 0.0f), 1.0f);
        float hit_t = fs(t, fm(dt, fs(1.0f, off)));
        if (st.first) {
            ts[0] = hit_t;
            st.target = tau_second;
            st.first = false;
            if (tau_next >= st.target) {
                float d2 = fs(st.target, st.tau);
                float off2 = exit_offset(A, B, -d2, d2, dt, S, lastS);
                ts[1] = fs(t, fm(dt, fs(1.0f, off2)));
                return true;
            }
        } else {
            ts[1] = hit_t;
            return true;
        }
    }
    st.tau = tau_next;
    return false;
}

// DeterminateEstimatedHit(alpha, pos, dir, dis) -> float4 (core/render.cuh:298-397).
// A step that reads 0 (and no transition from density pending) only advances
// t by half a voxel, so the march skips such steps exactly as the first-hit
// march does (estimated_hit): up to the box of nonzero voxels, through empty
// bricks, and past the box's far side, where it ends with what the t > dis
// test gives.
template <class DT>
MRP_D void estimated_hit_ts(const VolumeDev& v, float alpha, f3 pos, f3 dir, float dis, const float nl[3],
                            float ts[4]) {
    float smax = fm(v.max_density, alpha);
    float t = 0.0f;
    ts[0] = 0.0f; ts[1] = 0.0f; ts[2] = FLT_MAX; ts[3] = 0.0f;
    float last_non_empty_t = 0.0f;
    float rf = (float)v.res;
    float t_step = fd(1.0f, rf);
    if (fm(smax, t_step) > nl[0]) t_step = fd(nl[0], smax);
    const float half = fd(0.5f, rf);
    const bool pow2 = (v.res & (v.res - 1)) == 0;
    const MarchRay mr = march_ray(v, pos, dir);
    TauState st{0.0f, nl[1], true};
    int loop = 0;
    float last = 0.0f, t_exit = 3.0e38f;
    if (v.has_bounds && v.occ) {
        float t0 = 0.0f, t1 = dis;
        const float o[3] = {pos.x, pos.y, pos.z}, dd[3] = {dir.x, dir.y, dir.z};
        const float lo[3] = {v.nz_lo.x, v.nz_lo.y, v.nz_lo.z}, hi[3] = {v.nz_hi.x, v.nz_hi.y, v.nz_hi.z};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (dd[a] == 0.0f) {
                if (o[a] < lo[a] || o[a] > hi[a]) t0 = 3.0e38f;
            } else {
                const float ta = (lo[a] - o[a]) / dd[a], tb = (hi[a] - o[a]) / dd[a];
                t0 = fmaxf(t0, fminf(ta, tb));
                t1 = fminf(t1, fmaxf(ta, tb));
            }
        }
        const float t_enter = t0 > t1 ? 3.0e38f : t0;
        t_exit = t0 > t1 ? 0.0f : t1;
        if (pow2) replay_empty(t, loop, 2.0f * rf, half, dis, t_enter, 10000);
        while (loop < 10000 && t <= dis && t < t_enter) {
            ++loop;
            t = fa(t, half);
        }
    }
    while (loop++ < 10000) {
        // past the box: only empty steps are left, and fewer than the
        // bound allows (each advances t by half a voxel)
        if (t > dis || (t > t_exit && !(last > 0.0f) && (float)(10000 - loop) > (dis - t) * (2.0f * rf) + 2.0f)) {
            if (st.first) ts[0] = last_non_empty_t;
            else ts[1] = last_non_empty_t;
            break;
        }
        float t_brick = -1.0f;
        const float d = v.occ ? density_skip<DT>(v, mr, t, nullptr, &t_brick) : density_as<DT>(v, add(pos, mul(dir, t)));
        if (d > 0) {
            float S = fm(d, alpha);
            if (check_exit(S, last, t_step, t, st, ts, nl[2])) break;
            ts[2] = fminf(t, ts[2]);
            t = fa(t, t_step);
            last = S;
        } else {
            if (last > 0) {
                float ts_ = fa(t_step, d);
                if (ts_ > 0) {
                    if (check_exit(0.0f, last, ts_, t, st, ts, nl[2])) break;
                    last_non_empty_t = fa(t, ts_);
                } else {
                    last_non_empty_t = t;
                }
            }
            t = fa(t, fmaxf(fm(-d, 1.0f), half));
            last = 0.0f;
        }
        if (pow2 && t_brick >= 0.0f) replay_empty(t, loop, 2.0f * rf, half, fminf(t_brick, dis), 3.0e38f, 10000);
        while (t <= t_brick && t <= dis && loop < 10000) {
            ++loop;
            t = fa(t, half);
        }
    }
    if (ts[2] == FLT_MAX) ts[2] = 0.0f;
    float survival = expf(-st.tau);
    ts[3] = fminf(fd(fmaxf(fs(1.0f, survival), 0.0f), 0.75f), 1.0f);
}

// GetSampleT (core/render.cuh:464-485)
template <class DT>
MRP_D void sample_t(const VolumeDev& v, f3 ori, f3 dir, float alpha, const float nl[3], float ts[4]) {
    float dis = ray_box_offset(ori, dir);
    if (dis < 0) { ts[0] = ts[1] = ts[2] = ts[3] = 0.0f; return; }
    f3 sp = add(ori, mul(dir, dis));
    float md = ray_box_distance(sp, dir);
    estimated_hit_ts<DT>(v, alpha, sp, dir, md, nl, ts);
    if (ts[0] > 0) { ts[0] = fa(ts[0], dis); ts[2] = fa(ts[2], dis); }
    if (ts[1] > 0) ts[1] = fa(ts[1], dis);
}

struct TileView {
    int W, H, px, py, frame;
    uint32_t seed;
    f3 ori, up, right, L;
    float alpha, g;
    float nl[3];
};

// One block of 64 threads per tile: a thread marches one of the tile's 64 rays
// (PrepareRay, core/render.cuh:1006-1040: sample `sid`'s base ray and its
// three neighbours), the sums over the rays run in the reference's order on
// one thread per component, and the 192 stencil points are spread over the
// block.  Bound by the marches (lanes of a warp end apart).  128 x 128 tiles
// of a 256^3 cloud: 13.9 ms with one thread per tile, 0.64 ms.
constexpr int kTileThreads = 64;
template <class DT>
__global__ void __launch_bounds__(kTileThreads) k_gather_tiles(const __grid_constant__ VolumeDev v,
                                                               const __grid_constant__ TileView T,
                                                               float* __restrict__ out) {
    __shared__ float ray[64][4];      // direction, t of the ray's threshold (0: none)
    __shared__ float ray_t[64][2];    // ts[0], ts[1]
    __shared__ float samples[16][4], total[5];
    __shared__ float box[2][4];       // per warp: min x, min y, max x, max y of the rays that hit
    const int idx = blockIdx.x, tid = threadIdx.x;
    const int i = idx / T.W, j = idx % T.W;
    float* ob = out + (size_t)idx * 773;
    float u = fs(1.0f, fd(fa(fa((float)j, fd((float)T.px, 8.0f)), 0.5f), (float)T.W));
    float w = fs(1.0f, fd(fa(fa((float)i, fd((float)T.py, 8.0f)), 0.5f), (float)T.H));
    f3 fwd = normalize(neg(T.ori));
    f3 dir = add(add(fwd, mul(T.right, fs(fm(u, 2.0f), 1.0f))), mul(T.up, fs(fm(w, 2.0f), 1.0f)));
    const float rw = fm((float)T.W, 4.0f), rh = fm((float)T.H, 4.0f);
    f3 ro = mk3(fd(-T.right.x, rw), fd(-T.right.y, rw), fd(-T.right.z, rw));
    f3 uo = mk3(fd(-T.up.x, rh), fd(-T.up.y, rh), fd(-T.up.z, rh));
    {
        // sample sid at (x, y) in {-3, -1, 1, 3}^2, its ray q at (+-0.5, +-0.5)
        // around it; t-grid place: 4 floats a sample, 16 more a row
        const int sid = tid >> 2, q = tid & 3;
        const int x = -3 + 2 * (sid & 3), y = -3 + 2 * (sid >> 2), cb = (sid >> 2) & 1;
        const bool p25 = ((sid + cb) & 1) != 0;
        const float ox = (float)x + (q & 1 ? 0.5f : -0.5f), oy = (float)y + (q & 2 ? 0.5f : -0.5f);
        const int gid = 4 * sid + 16 * (sid >> 2) + (q & 1 ? 2 : 0) + (q & 2 ? 16 : 0);
        const f3 sd = normalize(add(add(dir, mul(ro, ox)), mul(uo, oy)));
        float ts[4];
        sample_t<DT>(v, T.ori, sd, T.alpha, T.nl, ts);
        const float rt = p25 ? ts[1] : ts[0];
        ray[tid][0] = sd.x; ray[tid][1] = sd.y; ray[tid][2] = sd.z; ray[tid][3] = rt;
        ray_t[tid][0] = ts[0]; ray_t[tid][1] = ts[1];
        const float rn = fd(1.0f, 3.0f);
        const float min_t = fm(ts[2], rn), max_t = fm(fmaxf(ts[0], ts[1]), rn);
        float* tg = ob + 192 * 3 + 5;
        tg[gid] = fm(fa(min_t, max_t), 0.5f);
        tg[gid + 1] = fs(max_t, min_t);
        tg[gid / 2 + 128] = ts[3];
        const bool in = rt != 0;
        float b[4] = {in ? ox : FLT_MAX, in ? oy : FLT_MAX, in ? ox : -FLT_MAX, in ? oy : -FLT_MAX};
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            b[0] = fminf(b[0], __shfl_xor_sync(0xffffffffu, b[0], o));
            b[1] = fminf(b[1], __shfl_xor_sync(0xffffffffu, b[1], o));
            b[2] = fmaxf(b[2], __shfl_xor_sync(0xffffffffu, b[2], o));
            b[3] = fmaxf(b[3], __shfl_xor_sync(0xffffffffu, b[3], o));
        }
        if ((tid & 31) == 0)
            for (int k = 0; k < 4; ++k) box[tid >> 5][k] = b[k];
    }
    __syncthreads();
    const float bx0 = fminf(box[0][0], box[1][0]), by0 = fminf(box[0][1], box[1][1]);
    const float bx1 = fmaxf(box[0][2], box[1][2]), by1 = fmaxf(box[0][3], box[1][3]);
    if (bx0 == FLT_MAX) {   // all 64 rays miss
        if (tid == 0) ob[0] = -1000.0f;
        return;
    }
    // (the tile's first value starts at 0, which the reference's multiplies
    // of tile 0 by 1.00001 before this point leave as it is)
    if (tid < 3) {          // component tid of the mean direction
        float a = 0.0f;
        for (int k = 0; k < 64; ++k)
            if (ray[k][3] != 0) a = fa(a, ray_t[k][1] > 0 ? fm(ray[k][tid], 2.0f) : ray[k][tid]);
        total[tid] = a;
    } else if (tid >= 32 && tid < 34) {   // depth gradients: horizontal, vertical
        float a = 0.0f;
        for (int s = 0; s < 16; ++s) {
            float h = 0.0f;
            for (int k = 4 * s; k < 4 * s + 4; ++k)
                if (ray[k][3] != 0) h = fa(h, fa(ray_t[k][0], ray_t[k][1]));
            a = fa(a, (tid == 32 ? (s & 3) >= 2 : (s >> 2) >= 2) ? h : -h);
        }
        total[3 + (tid - 32)] = a;
    } else if (tid >= 40 && tid < 56) {   // the ray that stands for a sample
        const int s = tid - 40;
        const bool p25 = ((s + ((s >> 2) & 1)) & 1) != 0;
        int best = 4 * s;
        for (int k = 4 * s + 1; k < 4 * s + 4; ++k) {
            const float c = ray[k][3], r = ray[best][3];
            if ((c != 0 && ((c < r) != p25)) || r == 0) best = k;
        }
        const int fill = s / 2 + (p25 ? 8 : 0);
        for (int k = 0; k < 4; ++k) samples[fill][k] = ray[best][k];
    }
    __syncthreads();
    Stream st(kPixelStream, (uint32_t)idx, 0, (uint32_t)T.frame, T.seed);
    f3 X, Y, Z, LX, LY, LZ;
    basis(mk3(total[0], total[1], total[2]), 0.0f, st, &X, &Y, &Z);
    basis(T.L, 0.0f, st, &LX, &LY, &LZ);
    if (tid == 0) {
        float minx = fs(bx0, 0.5f), miny = fs(by0, 0.5f), maxx = fa(bx1, 0.5f), maxy = fa(by1, 0.5f);
        f3 blc = normalize(add(add(dir, mul(ro, minx)), mul(uo, miny)));
        f3 rc = normalize(add(dir, mul(ro, maxx))), uc = normalize(add(dir, mul(uo, maxy)));
        auto cl = [](float x) { return fmaxf(-1.0f, fminf(1.0f, x)); };
        float* go = ob + 192 * 3;
        go[0] = acosf(cl(dot(X, T.L)));
        float gbl = acosf(cl(dot(blc, T.L)));
        go[1] = fs(acosf(cl(dot(rc, T.L))), gbl);
        go[2] = fs(acosf(cl(dot(uc, T.L))), gbl);
        go[3] = total[3];
        go[4] = total[4];
    }
    // the samples that have a hit, in order: point k >= 16 takes them in turn
    uint32_t have = 0;
#pragma unroll
    for (int s = 0; s < 16; ++s) have |= (uint32_t)(samples[s][3] != 0) << s;
    const int n = __popc(have);
    // SetupInputData2: X_Val [0, 192), X_Val_Hg [192, 384), X_Val_Sub [384, 576)
    for (int k = tid; k < 192; k += kTileThreads) {
        float fdv = 0.0f, fsv = 0.0f, fhv = 0.0f;
        if (k < 16) {
            const float* sm = samples[k];
            if (sm[3] != 0) {
                f3 sd = mk3(sm[0], sm[1], sm[2]);
                f3 sp = add(T.ori, mul(sd, sm[3]));
                float d = tex3<false>(mip_level(v, 0), 256, sp);
                fdv = logf(fa(1.0f, fm(fm(T.alpha, d), 0.015625f)));
                fhv = logf(fa(hg(dot(sd, T.L), T.g), 1.0f));
                fsv = shadow_tr(v, sp, T.L, 0);
            }
        } else {
            uint32_t m = have;
            for (int q = (k - 16) % n; q; --q) m &= m - 1;
            const float* sm = samples[__ffs(m) - 1];
            PixelFrame pf{add(T.ori, mul(mk3(sm[0], sm[1], sm[2]), sm[3])), X, Y, Z, T.L, T.L, T.g, T.alpha};
            gather_sample(v, pf, k, &fdv, &fsv, &fhv);
        }
        if (idx == 0 && k == 0) fdv = fm(fdv, 1.00001f);   // the reference's debug multiply of tile 0
        ob[k] = fdv;
        ob[192 + k] = fhv;
        ob[384 + k] = fsv;
    }
}

cudaError_t launch_gather_tiles(const VolumeDev& v, const ViewDev& view, int px, int py, const float nl[3], float* out,
                                cudaStream_t s) {
    int n = view.width * view.height;
    if (n <= 0) return cudaSuccess;
    TileView T{view.width, view.height, px, py, view.frame, view.seed, view.ori, view.up, view.right,
               view.light_dir, view.alpha, view.g, {nl[0], nl[1], nl[2]}};
    if (v.density_h) k_gather_tiles<__half><<<n, kTileThreads, 0, s>>>(v, T, out);
    else k_gather_tiles<float><<<n, kTileThreads, 0, s>>>(v, T, out);
    return cudaGetLastError();
}

cudaError_t launch_gather_rec(const VolumeDev& v, const ViewDev& view, HitRecords rec, float* feat, bool fp16,
                              cudaStream_t s) {
    int n = view.width * view.height;
    if (n <= 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
    // A record's 192 points in series take 100 us (texture form; 170 us the
    // FP32 form) however few records there are; six threads a record, 32
    // points each, take 28 us (53 us) for small frames and still 239 against
    // 249 us at 724^2 pixels.  At 1024^2 (half of them hits) the records fill
    // the SMs by themselves: 465 against 444 us for the texture form, while
    // the FP32 form, waiting for its loads, still gains (961 against 978 us).
    // The line lies between them, at 4054 pixels an SM (600 000 of 148).
    // Twelve threads of 16 points where even six leave the SMs short of warps:
    // 163 x 97, four launches, 510 -> 487 us, 128 x 128 213 -> 208, 256 x 256
    // 269 -> 266, 320 x 240 as before, 384 x 384 451 -> 460.
    const int parts = n <= sms * 512 ? 12 : !fp16 || n <= sms * 4054 ? 6 : 1;
    const dim3 grid((n + 127) / 128, parts);
    if (fp16 && v.glut_tex) k_gather_rec<true, true><<<grid, 128, 0, s>>>(v, view, rec, feat);
    else if (fp16) k_gather_rec<true><<<grid, 128, 0, s>>>(v, view, rec, feat);
    else k_gather_rec<false><<<grid, 128, 0, s>>>(v, view, rec, feat);
    return cudaGetLastError();
}
cudaError_t launch_debug_scatter(HitRecords rec, const float* feat, bool fp16, int npix, float* aux, float* feat_out,
                                 cudaStream_t s) {
    if (npix > 0) {
        if (fp16) k_debug_scatter<true><<<npix, 128, 0, s>>>(rec, feat, aux, feat_out);
        else k_debug_scatter<false><<<npix, 128, 0, s>>>(rec, feat, aux, feat_out);
    }
    return cudaGetLastError();
}

}  // namespace mrp
