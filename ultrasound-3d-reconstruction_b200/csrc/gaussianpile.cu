// GaussianPile projected-slice ("us_focus") additive splatting: binning, forward, backward.
//
// Reference behaviour restated here (paths inside KevinWCCC/ultrasound-3d-reconstruction,
// ops/gaussianplie_renderer):
//   include/shader/us_focus_device.cuh:88-316     conditional footprint of a 3D Gaussian on
//                                                 the slice under an elevational beam PSF
//   include/shader/plane_cond2d_device.cuh:14-98  world covariance, probe-frame covariance
//   include/shader/shared.cuh:6-34                quaternion -> rotation, normalisation
//   src/mapper/core_tile.cu:25-234                tile rectangles, keys, ranges
//   src/shader/forward.cu:27-210                  per-tile additive forward
//   src/shader/us_focus.cu:129-803, 805-966       sufficient-statistics backward, per-Gaussian
//                                                 finalize with finite-difference shape grads
//
// B200 design: each Gaussian's footprint is computed once per call and cached (the reference
// recomputes it in the mapper, once per tile in the forward and again per tile in the
// backward); tiles are filled in Gaussian order on small grids, else scattered and sorted like the UltraGauss
// path (see fills); the backward writes one record of nine moments per (tile, Gaussian) instance, from which the
// per-Gaussian finalize forms the gradient terms in instance order (the reference adds ~35 float
// atomics per instance into a per-Gaussian workspace).
//
// Arithmetic that decides integer outputs or that the forward image depends on (footprint,
// rectangles, window test, weights) uses the reference's operations in the reference's
// order, so that with the same --use_fast_math flags rectangles, sorted ids and tile ranges
// are bit-exact and images match to rounding of the summation.
#include <algorithm>

#include <float.h>
#include <type_traits>

#include "f32x2.cuh"
#include "us3d_common.cuh"
#include "scan.cuh"
#include "binning.cuh"
#include "stable_bins.cuh"

namespace us3d {
namespace gp {

// Slice grid pack layout (reference include/shader/slice_grid_geometry.cuh:4-16).
enum { SG_PROBE_TYPE = 0, SG_H = 1, SG_W = 2, SG_DELTA_LAT_MM = 3, SG_DELTA_AX_MM = 4, SG_NEAR_MM = 5,
       SG_LAT_COL_OFFSET = 6, SG_CENTER_LATERAL = 7 };
// us_focus parameter vector layout (reference include/shader/us_focus_device.cuh:9-23).
enum { UF_SIGMA_ELE_0 = 0, UF_SIGMA_ELE_1 = 1, UF_SIGMA_ELE_MIN = 2, UF_SIGMA_ELE_MAX = 3, UF_SIGMA_LAT_0 = 4,
       UF_SIGMA_LAT_1 = 5, UF_SIGMA_LAT_MIN = 6, UF_SIGMA_LAT_MAX = 7, UF_DET_GAMMA = 8, UF_DET_EPS = 9,
       UF_WEIGHT_MIN = 10, UF_USE_LATERAL_FOCUS = 11, UF_INFLATE_LAT_MM = 12, UF_INFLATE_AX_MM = 13 };

constexpr int FWD_BATCH = 256;
constexpr int PARTIAL_F4 = 3;  // per-instance partial record: nine moments in 12 floats
constexpr float GRAD_CLAMP = 1e3f;

struct Workspace {
    long long* header;
    int4* rects;        // G
    uint32_t* dkey;     // G
    int* touched;       // G
    int* inst_offset;   // G + 1
    long long* bs_g;
    int* tile_count;    // T
    int* tile_start;    // T + 1
    int* tile_cursor;   // T
    long long* bs_t;
    float4* cand;       // G x 3: (base_weight, intensity, mu2_lat, mu2_ax) (inv00, inv01, inv11, r_lat) (r_ax, valid)
    float4* bfp;        // G x 4, what the backward needs of the forward's footprint:
                        // (mu2_lat, mu2_ax, r_lat (< 0: no footprint), r_ax) (inv00, inv01, inv11, bno_const)
                        // (s2_00, s2_01, s2_11, 1 / det_norm) (mu_ele, 1 / denom_ele, dsigma_ele/dax, sigma_ele)
    StableScratch stable;    // small bucket grids (stable_bins)
    unsigned long long* keys;  // the other ones, and few elements with depth keys: instances before the sort
    int* slot_inst;
    int* sorted_gid;
    int* sorted_inst;
    size_t bytes;
};

// Whether the buckets are filled in element order (stable_bins.cuh) or sorted one by one. With depth keys the fill
// needs the radix sort's twelve launches, and a slice's lists are short: the whole forward with the sort /
// with the fill, us: 64x64 pixels 89 / 122 for 20k Gaussians, 112 / 146 for 45k, 187 / 165 for 70k; 256x256 89 / 129,
// 119 / 158, 142 / 181 and 198 / 226 for 120k; 512x512 141 / 174, 214 / 242, 276 / 302, 417 / 426; 720x704 206 / 224,
// 334 / 338, 443 / 456, 715 / 674.
constexpr int64_t FILL_MIN_KEYED = 65536;
static inline bool fills(int64_t G, int64_t T, bool keyed) {
    return stable_bins(G, T, keyed) && (!keyed || G >= FILL_MIN_KEYED);
}

static Workspace carve(void* base, int64_t G, int64_t T, int64_t cap) {
    Carver c(base);
    Workspace w;
    w.header = c.take<long long>(H_WORDS);
    w.rects = c.take<int4>((size_t)G);
    w.dkey = c.take<uint32_t>((size_t)G);
    w.touched = c.take<int>((size_t)G);
    w.inst_offset = c.take<int>((size_t)G + 1);
    w.bs_g = c.take<long long>((size_t)scan_num_blocks(G) + 1);
    w.tile_count = c.take<int>((size_t)T);
    w.tile_start = c.take<int>((size_t)T + 1);
    w.tile_cursor = c.take<int>((size_t)T);
    w.bs_t = c.take<long long>((size_t)scan_num_blocks(T) + 1);
    w.cand = c.take<float4>((size_t)G * 3);
    w.bfp = c.take<float4>((size_t)G * 4);
    // a workspace serves calls with depth keys (sort_by_v) and without: a small one has both
    const bool all = fills(G, T, true);
    w.stable = fills(G, T, false) ? stable_carve(c, G, T, all) : StableScratch{};
    w.keys = all ? nullptr : c.take<unsigned long long>((size_t)cap);
    w.slot_inst = all ? nullptr : c.take<int>((size_t)cap);
    w.sorted_gid = c.take<int>((size_t)cap);
    w.sorted_inst = c.take<int>((size_t)cap);
    w.bytes = align_up(c.off, 256);
    return w;
}

// ---- geometry helpers (reference include/shader/shared.cuh:6-34) ----

__device__ __forceinline__ float3 normalize3(const float3 v) {
    const float n = sqrtf(fmaxf(1e-12f, f3_dot(v, v)));
    return make_float3(v.x / n, v.y / n, v.z / n);
}

// Probe axes are the normalised columns of the 4x4 pose, the origin its translation column.
struct Axes {
    float3 raw_lat, raw_ax, raw_ele, lat, ax, ele, origin;
};

__device__ __forceinline__ Axes axes_from_pose(const float* __restrict__ pose) {
    Axes a;
    a.raw_lat = make_float3(pose[0], pose[4], pose[8]);
    a.raw_ax = make_float3(pose[1], pose[5], pose[9]);
    a.raw_ele = make_float3(pose[2], pose[6], pose[10]);
    a.lat = normalize3(a.raw_lat);
    a.ax = normalize3(a.raw_ax);
    a.ele = normalize3(a.raw_ele);
    a.origin = make_float3(pose[3], pose[7], pose[11]);
    return a;
}

// Rotation from a (w, x, y, z) quaternion normalised with rsqrt.
__device__ __forceinline__ void quat_rot(const float q0, const float q1, const float q2, const float q3, float R[9]) {
    const float nq = rsqrtf(fmaxf(1e-12f, q0 * q0 + q1 * q1 + q2 * q2 + q3 * q3));
    const float w = q0 * nq, x = q1 * nq, y = q2 * nq, z = q3 * nq;
    const float xx = x * x, yy = y * y, zz = z * z;
    const float xy = x * y, xz = x * z, yz = y * z;
    const float wx = w * x, wy = w * y, wz = w * z;
    R[0] = 1.f - 2.f * (yy + zz);
    R[1] = 2.f * (xy - wz);
    R[2] = 2.f * (xz + wy);
    R[3] = 2.f * (xy + wz);
    R[4] = 1.f - 2.f * (xx + zz);
    R[5] = 2.f * (yz - wx);
    R[6] = 2.f * (xz - wy);
    R[7] = 2.f * (yz + wx);
    R[8] = 1.f - 2.f * (xx + yy);
}

// Sigma_w = R diag(s^2) R^T (reference plane_cond2d_device.cuh:48-69).
__device__ __forceinline__ void sigma_world(float sx, float sy, float sz, const float R[9], float S[9]) {
    float M[9];
    M[0] = R[0] * sx * sx; M[1] = R[1] * sy * sy; M[2] = R[2] * sz * sz;
    M[3] = R[3] * sx * sx; M[4] = R[4] * sy * sy; M[5] = R[5] * sz * sz;
    M[6] = R[6] * sx * sx; M[7] = R[7] * sy * sy; M[8] = R[8] * sz * sz;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) S[i * 3 + j] = M[i * 3 + 0] * R[j] + M[i * 3 + 1] * R[3 + j] + M[i * 3 + 2] * R[6 + j];
}

// Sc = A^T Sigma_w A with A = [lat ax ele] (reference plane_cond2d_device.cuh:71-98).
__device__ __forceinline__ void sigma_probe(const float S[9], float3 a0, float3 a1, float3 a2, float Sc[9]) {
    const float3 c0 = make_float3(S[0] * a0.x + S[1] * a0.y + S[2] * a0.z, S[3] * a0.x + S[4] * a0.y + S[5] * a0.z,
                                  S[6] * a0.x + S[7] * a0.y + S[8] * a0.z);
    const float3 c1 = make_float3(S[0] * a1.x + S[1] * a1.y + S[2] * a1.z, S[3] * a1.x + S[4] * a1.y + S[5] * a1.z,
                                  S[6] * a1.x + S[7] * a1.y + S[8] * a1.z);
    const float3 c2 = make_float3(S[0] * a2.x + S[1] * a2.y + S[2] * a2.z, S[3] * a2.x + S[4] * a2.y + S[5] * a2.z,
                                  S[6] * a2.x + S[7] * a2.y + S[8] * a2.z);
    Sc[0] = a0.x * c0.x + a0.y * c0.y + a0.z * c0.z;
    Sc[1] = a0.x * c1.x + a0.y * c1.y + a0.z * c1.z;
    Sc[2] = a0.x * c2.x + a0.y * c2.y + a0.z * c2.z;
    Sc[3] = a1.x * c0.x + a1.y * c0.y + a1.z * c0.z;
    Sc[4] = a1.x * c1.x + a1.y * c1.y + a1.z * c1.z;
    Sc[5] = a1.x * c2.x + a1.y * c2.y + a1.z * c2.z;
    Sc[6] = a2.x * c0.x + a2.y * c0.y + a2.z * c0.z;
    Sc[7] = a2.x * c1.x + a2.y * c1.y + a2.z * c1.z;
    Sc[8] = a2.x * c2.x + a2.y * c2.y + a2.z * c2.z;
}

// Adjugate inverse of a 3x3 matrix; false unless det > 1e-12 and finite
// (reference us_focus_device.cuh:115-151).
__device__ __forceinline__ bool inv3(const float M[9], float Mi[9]) {
    const float a00 = M[0], a01 = M[1], a02 = M[2], a10 = M[3], a11 = M[4], a12 = M[5], a20 = M[6], a21 = M[7],
                a22 = M[8];
    const float c00 = a11 * a22 - a12 * a21;
    const float c01 = a02 * a21 - a01 * a22;
    const float c02 = a01 * a12 - a02 * a11;
    const float c10 = a12 * a20 - a10 * a22;
    const float c11 = a00 * a22 - a02 * a20;
    const float c12 = a02 * a10 - a00 * a12;
    const float c20 = a10 * a21 - a11 * a20;
    const float c21 = a01 * a20 - a00 * a21;
    const float c22 = a00 * a11 - a01 * a10;
    const float det = a00 * c00 + a01 * c10 + a02 * c20;
    if (!(det > 1e-12f) || !isfinite(det)) return false;
    const float id = 1.f / det;
    Mi[0] = c00 * id; Mi[1] = c01 * id; Mi[2] = c02 * id;
    Mi[3] = c10 * id; Mi[4] = c11 * id; Mi[5] = c12 * id;
    Mi[6] = c20 * id; Mi[7] = c21 * id; Mi[8] = c22 * id;
    return true;
}

__device__ __forceinline__ float det_norm_factor(float d, float gamma) {
    if (gamma == 0.f) return 1.f;
    if (fabsf(gamma - 0.25f) < 1e-7f) return 1.f / sqrtf(sqrtf(d));
    if (fabsf(gamma - 0.5f) < 1e-7f) return 1.f / sqrtf(d);
    if (fabsf(gamma - 1.f) < 1e-7f) return 1.f / d;
    return powf(d, -gamma);
}

__device__ __forceinline__ float clampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }

struct Footprint {
    float mu2_lat, mu2_ax, s2_00, s2_01, s2_11, inv00, inv01, inv11, det2;
    float sigma_ele, sigma_lat, mu_lat, mu_ax, mu_ele, sc22;
    float Lc[9], Se[9];
    float r_lat, r_ax;
};

// Elevational-PSF conditional footprint (reference us_focus_device.cuh:179-316):
// Sc = A^T Sigma_w A + 1e-6 I, Lc = Sc^-1, Le = Lc + diag(lat focus, 0, 1/sigma_ele^2),
// Se = Le^-1, mu_e = Se Lc mu_c, Sigma_2 = Se[0:2, 0:2] (symmetrised), radii from it.
__device__ __forceinline__ bool footprint(const float m0, const float m1, const float m2, const float s0,
                                          const float s1, const float s2, const float q0, const float q1,
                                          const float q2, const float q3, const Axes& A, float near_mm, float k_sigma,
                                          const float* __restrict__ P, Footprint& F) {
    const float3 d = make_float3(m0 - A.origin.x, m1 - A.origin.y, m2 - A.origin.z);
    F.mu_lat = f3_dot(d, A.lat);
    F.mu_ax = f3_dot(d, A.ax);
    F.mu_ele = f3_dot(d, A.ele);
    float R[9];
    quat_rot(q0, q1, q2, q3, R);
    const float sx = fmaxf(s0, 1e-6f), sy = fmaxf(s1, 1e-6f), sz = fmaxf(s2, 1e-6f);
    float Sw[9], Sc[9];
    sigma_world(sx, sy, sz, R, Sw);
    sigma_probe(Sw, A.lat, A.ax, A.ele, Sc);
    Sc[0] += 1e-6f;
    Sc[4] += 1e-6f;
    Sc[8] += 1e-6f;
    if (!inv3(Sc, F.Lc)) return false;
    const float depth = fmaxf(F.mu_ax - near_mm, 0.f);
    F.sigma_ele = clampf(P[UF_SIGMA_ELE_0] + P[UF_SIGMA_ELE_1] * depth, P[UF_SIGMA_ELE_MIN], P[UF_SIGMA_ELE_MAX]);
    F.sigma_lat = clampf(P[UF_SIGMA_LAT_0] + P[UF_SIGMA_LAT_1] * depth, P[UF_SIGMA_LAT_MIN], P[UF_SIGMA_LAT_MAX]);
    float Le[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) Le[i] = F.Lc[i];
    if (P[UF_USE_LATERAL_FOCUS] != 0.f) Le[0] += 1.f / fmaxf(F.sigma_lat * F.sigma_lat, 1e-12f);
    Le[8] += 1.f / fmaxf(F.sigma_ele * F.sigma_ele, 1e-12f);
    if (!inv3(Le, F.Se)) return false;
    const float mc[3] = {F.mu_lat, F.mu_ax, F.mu_ele};
    const float t0 = F.Lc[0] * mc[0] + F.Lc[1] * mc[1] + F.Lc[2] * mc[2];
    const float t1 = F.Lc[3] * mc[0] + F.Lc[4] * mc[1] + F.Lc[5] * mc[2];
    const float t2 = F.Lc[6] * mc[0] + F.Lc[7] * mc[1] + F.Lc[8] * mc[2];
    F.mu2_lat = F.Se[0] * t0 + F.Se[1] * t1 + F.Se[2] * t2;
    F.mu2_ax = F.Se[3] * t0 + F.Se[4] * t1 + F.Se[5] * t2;
    const float il = fmaxf(P[UF_INFLATE_LAT_MM], 0.f), ia = fmaxf(P[UF_INFLATE_AX_MM], 0.f);
    F.s2_00 = F.Se[0] + il * il;
    F.s2_01 = 0.5f * (F.Se[1] + F.Se[3]);
    F.s2_11 = F.Se[4] + ia * ia;
    F.det2 = F.s2_00 * F.s2_11 - F.s2_01 * F.s2_01;
    if (!(F.det2 > P[UF_DET_EPS]) || !isfinite(F.det2)) return false;
    const float idet = 1.f / F.det2;
    F.inv00 = F.s2_11 * idet;
    F.inv01 = -F.s2_01 * idet;
    F.inv11 = F.s2_00 * idet;
    F.sc22 = Sc[8];
    const float cross = fabsf(F.s2_01);
    F.r_lat = k_sigma * sqrtf(fmaxf(F.s2_00 + cross, 1e-12f));
    F.r_ax = k_sigma * sqrtf(fmaxf(F.s2_11 + cross, 1e-12f));
    return true;
}

// ------------------------------------------------------------------------------------
// Binning
// ------------------------------------------------------------------------------------

__global__ void init_kernel(int64_t T, int* __restrict__ tile_count, int* __restrict__ tile_cursor,
                            long long* __restrict__ header, int64_t cap, int64_t G) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0 && threadIdx.x < H_WORDS) {
        long long v = 0;
        if (threadIdx.x == H_CAP) v = cap;
        if (threadIdx.x == H_G) v = G;
        if (threadIdx.x == H_T) v = T;
        header[threadIdx.x] = v;
    }
    if (t >= T) return;
    tile_count[t] = 0;
    tile_cursor[t] = 0;
}

// Footprint, tile rectangle, depth key and forward candidate of every Gaussian
// (reference src/mapper/core_tile.cu:25-174 and src/shader/forward.cu:27-86).
__global__ void __launch_bounds__(256)
preprocess_kernel(int64_t G, int H, int W, int tile, int tiles_x, int tiles_y, float lat_mm, float ax_mm,
                  float near_mm, float k_sigma, int sort_by_v, const float* __restrict__ means,
                  const float* __restrict__ scales, const float* __restrict__ quats, const float* __restrict__ opac,
                  const float* __restrict__ inten, const float* __restrict__ pose, const float* __restrict__ grid,
                  const float* __restrict__ params, int4* __restrict__ rects, uint32_t* __restrict__ dkey,
                  int* __restrict__ touched, int* __restrict__ tile_count, float4* __restrict__ cand,
                  float4* __restrict__ bfp) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    const Axes A = axes_from_pose(pose);
    const float* m = means + 3 * g;
    const float* s = scales + 3 * g;
    const float* q = quats + 4 * g;
    Footprint F;
    rects[g] = make_int4(0, 0, 0, 0);
    touched[g] = 0;
    dkey[g] = 0;
    if (!footprint(m[0], m[1], m[2], s[0], s[1], s[2], q[0], q[1], q[2], q[3], A, near_mm, k_sigma, params, F)) return;
    const float u_pix = F.mu2_lat / lat_mm + grid[SG_LAT_COL_OFFSET];
    const float v_pix = (F.mu2_ax - near_mm) / ax_mm;
    const float r_lat_pix = fmaxf(1.0f, F.r_lat / fmaxf(1e-8f, lat_mm));
    const float r_ax_pix = fmaxf(1.0f, F.r_ax / fmaxf(1e-8f, ax_mm));
    const float ts = (float)tile;
    int x0 = (int)floorf((u_pix - r_lat_pix) / ts);
    int y0 = (int)floorf((v_pix - r_ax_pix) / ts);
    int x1 = (int)ceilf((u_pix + r_lat_pix) / ts);
    int y1 = (int)ceilf((v_pix + r_ax_pix) / ts);
    x0 = max(0, x0);
    y0 = max(0, y0);
    x1 = min(tiles_x, x1);
    y1 = min(tiles_y, y1);
    (void)H;
    (void)W;
    if (x0 >= x1 || y0 >= y1) return;
    rects[g] = make_int4(x0, y0, x1, y1);
    dkey[g] = sort_by_v ? f32_to_u32_sat((v_pix + 500.0f) * 1000.0f) : 0u;
    touched[g] = (x1 - x0) * (y1 - y0);
    (void)tile_count;  // counted per block by rect_count_kernel
    // Forward candidate, computed with the forward's own near plane (the grid pack's);
    // the mapper's footprint is reused when the two near planes agree.
    Footprint Ff = F;
    bool okf = true;
    if (grid[SG_NEAR_MM] != near_mm)
        okf = footprint(m[0], m[1], m[2], s[0], s[1], s[2], q[0], q[1], q[2], q[3], A, grid[SG_NEAR_MM], k_sigma,
                        params, Ff);
    float bw = 0.f;
    bool valid = okf;
    if (okf) {
        const float det_eps = params[UF_DET_EPS];
        const float denom_ele = fmaxf(Ff.sc22 + Ff.sigma_ele * Ff.sigma_ele + det_eps, 1e-12f);
        const float slice_response = expf(-0.5f * Ff.mu_ele * Ff.mu_ele / denom_ele);
        const float norm = det_norm_factor(Ff.det2 + det_eps, params[UF_DET_GAMMA]);
        bw = opac[g] * slice_response * norm;
        valid = isfinite(bw);
    }
    cand[3 * g + 0] = make_float4(bw, inten[g], Ff.mu2_lat, Ff.mu2_ax);
    cand[3 * g + 1] = make_float4(Ff.inv00, Ff.inv01, Ff.inv11, Ff.r_lat);
    cand[3 * g + 2] = make_float4(Ff.r_ax, valid ? 1.f : 0.f, 0.f, 0.f);
    // The backward's per-Gaussian factors (reference us_focus.cu:398-477), with the grid's near
    // plane as the backward uses it.
    {
        const float det_eps = params[UF_DET_EPS], det_gamma = params[UF_DET_GAMMA];
        const float near_b = grid[SG_NEAR_MM];
        const float denom_ele = fmaxf(Ff.sc22 + Ff.sigma_ele * Ff.sigma_ele + det_eps, 1e-12f);
        const float slice_response = expf(-0.5f * Ff.mu_ele * Ff.mu_ele / denom_ele);
        const float norm = det_norm_factor(Ff.det2 + det_eps, det_gamma);
        const float depth = fmaxf(Ff.mu_ax - near_b, 0.f);
        const float se_raw = params[UF_SIGMA_ELE_0] + params[UF_SIGMA_ELE_1] * depth;
        const float dse_dax = (Ff.mu_ax > near_b && se_raw > params[UF_SIGMA_ELE_MIN] &&
                               se_raw < params[UF_SIGMA_ELE_MAX]) ? params[UF_SIGMA_ELE_1] : 0.f;
        bfp[4 * g + 0] = make_float4(Ff.mu2_lat, Ff.mu2_ax, okf ? Ff.r_lat : -1.f, Ff.r_ax);
        bfp[4 * g + 1] = make_float4(Ff.inv00, Ff.inv01, Ff.inv11, slice_response * norm);
        bfp[4 * g + 2] = make_float4(Ff.s2_00, Ff.s2_01, Ff.s2_11, 1.f / fmaxf(Ff.det2 + det_eps, 1e-12f));
        bfp[4 * g + 3] = make_float4(Ff.mu_ele, 1.f / denom_ele, dse_dax, Ff.sigma_ele);
    }
}

// ------------------------------------------------------------------------------------
// Forward
// ------------------------------------------------------------------------------------

// One block of four warps per 8x4 block of a tile's pixels. The sum over a pixel's candidates is split by
// Gaussian index into 16 classes (g mod 16), each summed in list order, and the class sums are added
// in class order. The grouping does not depend on the tile size, so the image does not either (the
// reference sums the whole list in order, src/shader/forward.cu:88-210: the results agree up to rounding).
//
// Every batch of candidates is tested once (its box against the pixel block's extent, with a margin for the
// rounding of the per-pixel test) and queued by class, in list order. A quarter-warp then walks its
// class's queue, lane l holding the four pixels of column l in packed FP32 pairs: four candidates are
// visited by one instruction, and the lateral part of the test and of the quadratic form is formed once
// for four pixels. With one candidate and one pixel per lane the kernel executed 226M warp instructions for
// a 256x256 slice of 200k Gaussians, in 711 us; 117M and 268 us so, bound by issue and, at the end, by the
// blocks with the longest lists (1.5 times the mean). 768x768, 200k: 2.10 -> 0.91 ms. Two, four and eight
// pixel blocks sharing the staged candidates took 315, 394 and 535 us (more warps wait for each
// batch); 8 classes 336 us, 32 classes 314 us; batches of 128 / 512 337 / 328 us; unrolled 1 / 2 / 4 times
// 331 / 305 / 272 us; compiled for 10 / 12 blocks per SM 319 / 341 us.
constexpr int CLASSES = 16, GROUP_WARPS = CLASSES / 4, GROUP = GROUP_WARPS * 32;
constexpr int FWD_CTAS = 8;
constexpr int BLK_W = 8, BLK_H = 4;
constexpr int FWD_ROUNDS = FWD_BATCH / 32;  // warp-wide tests of a batch
static_assert(FWD_BATCH <= 256 && FWD_ROUNDS % 4 == 0 && FWD_ROUNDS % GROUP_WARPS == 0, "queue entries and counts are bytes");

__global__ void __launch_bounds__(GROUP, FWD_CTAS)
forward_kernel(int H, int W, int tile, int tiles_x, const float* __restrict__ grid, const float* __restrict__ params,
               const int* __restrict__ tile_start, const int* __restrict__ sorted_gid,
               const long long* __restrict__ header, const float4* __restrict__ cand, float* __restrict__ image) {
    __shared__ float4 sc0[FWD_BATCH + 1], sc1[FWD_BATCH + 1];  // the last candidate reaches no pixel
    __shared__ float2 sc2[FWD_BATCH + 1];
    __shared__ unsigned char s_cls[FWD_BATCH];
    __shared__ unsigned s_cnt[CLASSES][FWD_ROUNDS / 4];  // per class: a byte per warp-wide test, its candidates
    __shared__ __align__(16) unsigned char s_queue[CLASSES][FWD_BATCH];
    static_assert(sizeof(s_queue) >= sizeof(float) * CLASSES * BLK_W * BLK_H, "the class sums reuse the queues");
    if (header[H_FLAGS] != 0) return;
    const int bx = (tile + BLK_W - 1) / BLK_W, by = (tile + BLK_H - 1) / BLK_H;
    const int t = blockIdx.x / (bx * by), kb = blockIdx.x % (bx * by);  // tile and its pixel block
    const int tx = t % tiles_x, ty = t / tiles_x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, col = lane & (BLK_W - 1);
    const int cls = warp * 4 + (lane >> 3);
    const int lx = (kb % bx) * BLK_W + col, ly = (kb / bx) * BLK_H;
    const int x = tx * tile + lx, y = ty * tile + ly;
    const bool col_ok = lx < tile && x < W;
    const float weight_min = params[UF_WEIGHT_MIN];
    const float xi_lat = (static_cast<float>(x) - grid[SG_LAT_COL_OFFSET]) * grid[SG_DELTA_LAT_MM];
    float xi_ax[BLK_H];
    // the block's extent in mm
    float lat_lo = 3.0e38f, lat_hi = -3.0e38f, ax_lo = 3.0e38f, ax_hi = -3.0e38f;
#pragma unroll
    for (int r = 0; r < BLK_H; ++r) {
        xi_ax[r] = static_cast<float>(y + r) * grid[SG_DELTA_AX_MM] + grid[SG_NEAR_MM];
        if (col_ok && ly + r < tile && y + r < H) {
            lat_lo = lat_hi = xi_lat;
            ax_lo = fminf(ax_lo, xi_ax[r]);
            ax_hi = fmaxf(ax_hi, xi_ax[r]);
        }
    }
#pragma unroll
    for (int o = 1; o < BLK_W; o <<= 1) {
        lat_lo = fminf(lat_lo, __shfl_xor_sync(0xffffffffu, lat_lo, o));
        lat_hi = fmaxf(lat_hi, __shfl_xor_sync(0xffffffffu, lat_hi, o));
        ax_lo = fminf(ax_lo, __shfl_xor_sync(0xffffffffu, ax_lo, o));
        ax_hi = fmaxf(ax_hi, __shfl_xor_sync(0xffffffffu, ax_hi, o));
    }
    const f32x2 AX0 = pk2(xi_ax[0], xi_ax[1]), AX1 = pk2(xi_ax[2], xi_ax[3]);
    const f32x2 CE = dup2(-0.72134752044448170f);  // -log2(e) / 2
    const int s0 = tile_start[t], n = tile_start[t + 1] - s0;
    f32x2 acc0 = dup2(0.f), acc1 = acc0;
    if (threadIdx.x == 0) {
        sc0[FWD_BATCH] = make_float4(0.f, 0.f, 0.f, 0.f);
        sc1[FWD_BATCH] = make_float4(0.f, 0.f, 0.f, -1.f);
        sc2[FWD_BATCH] = make_float2(-1.f, 0.f);
    }
    const unsigned char* queue = s_queue[cls];
    for (int b0 = 0; b0 < n; b0 += FWD_BATCH) {
        const int nb = min(FWD_BATCH, n - b0);
        __syncthreads();
        for (int j = threadIdx.x; j < nb; j += GROUP) {
            const int g = sorted_gid[s0 + b0 + j];
            sc0[j] = cand[3 * g];
            sc1[j] = cand[3 * g + 1];
            const float4 c2 = cand[3 * g + 2];
            sc2[j] = make_float2(c2.x, c2.y);
            s_cls[j] = (unsigned char)(g % CLASSES);
        }
        if (threadIdx.x < CLASSES * (FWD_ROUNDS / 4)) (&s_cnt[0][0])[threadIdx.x] = 0u;
        __syncthreads();
        // the candidates that reach this pixel block, queued by class in list order
        int place[FWD_ROUNDS / GROUP_WARPS], of[FWD_ROUNDS / GROUP_WARPS];
#pragma unroll
        for (int i = 0; i < FWD_ROUNDS / GROUP_WARPS; ++i) {
            const int round = i * GROUP_WARPS + warp, j = round * 32 + lane;
            bool near = false;
            if (j < nb) {
                const float4 c0 = sc0[j];
                const float2 c2 = sc2[j];
                const float rl = sc1[j].w;
                const float ml = 1e-5f * (fabsf(c0.z) + rl + fabsf(lat_lo) + fabsf(lat_hi)) + 1e-30f;
                const float ma = 1e-5f * (fabsf(c0.w) + c2.x + fabsf(ax_lo) + fabsf(ax_hi)) + 1e-30f;
                near = c2.y != 0.f && lat_hi >= c0.z - rl - ml && lat_lo <= c0.z + rl + ml &&
                       ax_hi >= c0.w - c2.x - ma && ax_lo <= c0.w + c2.x + ma;
            }
            of[i] = near ? s_cls[j] : CLASSES;
            const unsigned same = __match_any_sync(0xffffffffu, of[i]);
            place[i] = __popc(same & ((1u << lane) - 1u));
            if (near && place[i] == 0)
                reinterpret_cast<unsigned char*>(s_cnt[of[i]])[round] = (unsigned char)__popc(same);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < FWD_ROUNDS / GROUP_WARPS; ++i) {
            if (of[i] == CLASSES) continue;
            const int round = i * GROUP_WARPS + warp;
            int pos = place[i];
#pragma unroll
            for (int w = 0; w < FWD_ROUNDS / 4; ++w) {
                const int in = min(max(round - 4 * w, 0), 4);  // rounds of this word that come before
                pos = __dp4a(s_cnt[of[i]][w], (unsigned)(0x01010101ull & ((1ull << (8 * in)) - 1ull)), (unsigned)pos);
            }
            s_queue[of[i]][pos] = (unsigned char)(round * 32 + lane);
        }
        int n_mine = 0;
#pragma unroll
        for (int w = 0; w < FWD_ROUNDS / 4; ++w) n_mine = __dp4a(s_cnt[cls][w], 0x01010101u, (unsigned)n_mine);
        int n_max = max(n_mine, __shfl_xor_sync(0xffffffffu, n_mine, 8));
        n_max = max(n_max, __shfl_xor_sync(0xffffffffu, n_max, 16));
        __syncthreads();
        // With a positive weight_min an infinite quad fails the weight test by itself.
        auto run = [&](auto positive_t) {
            constexpr bool POSITIVE = decltype(positive_t)::value;
#pragma unroll 8
            for (int k = 0; k < n_max; ++k) {
                const int j = k < n_mine ? queue[k] : FWD_BATCH;
                const float4 c0 = sc0[j], c1 = sc1[j];
                const float r_ax = sc2[j].x;
                const float dlat = xi_lat - c0.z;
                const float lim = fabsf(dlat) <= c1.w ? r_ax : -1.f;
                const f32x2 L = dup2(dlat), QL0 = dup2(c1.x * dlat), QA0 = dup2(c1.y * dlat);
                auto rows = [&](f32x2 AX, f32x2& acc) {
                    const f32x2 D = sub2(AX, dup2(c0.w));
                    const f32x2 QL = fma2(dup2(c1.y), D, QL0), QA = fma2(dup2(c1.z), D, QA0);
                    const f32x2 Q = fma2(D, QA, mul2(L, QL));
                    const f32x2 Wt = mul2(dup2(c0.x), ex2_2(mul2(Q, CE)));
                    float d0, d1, q0, q1, w0, w1, v0, v1;
                    up2(D, d0, d1);
                    up2(Q, q0, q1);
                    up2(Wt, w0, w1);
                    up2(mul2(dup2(c0.y), Wt), v0, v1);
                    const bool k0 = fabsf(d0) <= lim && q0 >= 0.f && (POSITIVE || q0 <= FLT_MAX) && !(w0 < weight_min);
                    const bool k1 = fabsf(d1) <= lim && q1 >= 0.f && (POSITIVE || q1 <= FLT_MAX) && !(w1 < weight_min);
                    acc = add2(acc, pk2(k0 ? v0 : 0.f, k1 ? v1 : 0.f));
                };
                rows(AX0, acc0);
                rows(AX1, acc1);
            }
        };
        if (weight_min > 0.f)
            run(std::true_type{});
        else
            run(std::false_type{});
    }
    __syncthreads();
    float(*s_sum)[BLK_W * BLK_H] = reinterpret_cast<float(*)[BLK_W * BLK_H]>(&s_queue[0][0]);
    float v[BLK_H];
    up2(acc0, v[0], v[1]);
    up2(acc1, v[2], v[3]);
#pragma unroll
    for (int r = 0; r < BLK_H; ++r) s_sum[cls][r * BLK_W + col] = v[r];
    __syncthreads();
    if (warp != 0 || !col_ok) return;
    const int r = lane >> 3;  // warp 0: lane (row, column)
    if (ly + r >= tile || y + r >= H) return;
    float total = s_sum[0][lane];
#pragma unroll
    for (int c = 1; c < CLASSES; ++c) total += s_sum[c][lane];
    image[(y + r) * W + x] = total;
}

// ------------------------------------------------------------------------------------
// Backward
// ------------------------------------------------------------------------------------

// Every term of a Gaussian's adjoint is a fixed combination of nine sums over its contributing pixels, which an
// instance's record holds: ub = up * bno (bno = the weight without the opacity) times q_lat, q_ax,
// q_lat^2, q_lat q_ax, q_ax^2 (q = inv2 d), dlat^2, dlat dax, dax^2 and 1. The finalize
// forms the terms (the reference keeps 35 of them per instance).
// The q-weighted sums are taken per pixel, not expanded from moments of d: for an elongated
// footprint q nearly cancels along the long axis, and the expansion inv00^2 S(dlat^2) + 2 inv00 inv01
// S(dlat dax) + ... loses in fp32 the digits that the chain through Se and Lc (with entries in
// the hundreds for such footprints) then amplifies.
enum { M_QL = 0, M_QA, M_QLL, M_QLA, M_QAA, M_XX, M_XY, M_YY, M_ONE, M_COUNT };

// One half-warp per instance of the sorted instance list (tile by tile): its lanes share the pixels of the
// footprint's bounding box within the instance's tile, lane l the pixels l and l + 16 of every 32 in a packed
// FP32 pair, and accumulate the per-pixel adjoint of the footprint (reference src/shader/us_focus.cu:398-477,
// 805-966); the sums are then reduced over the half-warp in a fixed order. The footprints are the
// forward's (cached per Gaussian by the preprocess). A whole warp per instance, one pixel per lane and
// 19 terms written per instance executed 369M warp instructions for a 256x256 slice of 200k Gaussians, at
// 74 % of the issue rate, a good part of them for the reduction and the terms: 453 us, and 16 us to sum the
// records. With half-warps, the box walked in floats and nine moments per instance 282 us, bound by
// issue (72 %); the finalize, which now forms the terms, 44 -> 61 us.
constexpr int BWD_WARPS = 8;  // warps per CTA

__global__ void __launch_bounds__(BWD_WARPS * 32, 4)
backward_inst_kernel(int T, int W, int tile, int tiles_x, const float* __restrict__ opac,
                     const float4* __restrict__ bfp,
                     const float* __restrict__ grid, const float* __restrict__ params,
                     const int* __restrict__ tile_start, const int* __restrict__ sorted_gid,
                     const int* __restrict__ sorted_inst, const long long* __restrict__ header,
                     const float* __restrict__ grad_image, float* __restrict__ partial, int H) {
    if (header[H_FLAGS] != 0) return;
    const int lane = threadIdx.x & 31, l = lane & 15, half = lane >> 4;
    const int total = tile_start[T];
    const float weight_min = params[UF_WEIGHT_MIN];
    const float lat_delta = grid[SG_DELTA_LAT_MM], ax_delta = grid[SG_DELTA_AX_MM];
    const float col_off = grid[SG_LAT_COL_OFFSET], near_mm = grid[SG_NEAR_MM];
    // Each warp owns a contiguous run of instances, so the instance's tile (the last t with
    // tile_start[t] <= k; empty tiles share a start) is found by one binary search per warp and
    // then followed forward as k advances.
    const int n_warps = (int)(gridDim.x * blockDim.x) >> 5;
    const int wid = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int chunk = (int)(((int64_t)total + n_warps - 1) / n_warps);
    const int k_begin = (int)min((int64_t)total, (int64_t)wid * chunk), k_end = min(total - k_begin, chunk) + k_begin;
    int t = 0;
    if (k_begin < k_end) {
        int lo = 0, hi = T;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (tile_start[mid] <= k_begin) lo = mid; else hi = mid;
        }
        t = lo;
    }
    const f32x2 CE = dup2(-0.72134752044448170f);  // -log2(e) / 2
    int x0 = 0, y0 = 0, x1 = 0, y1 = 0, t_end = k_begin < k_end ? k_begin : 0;
    for (int k0 = k_begin; k0 < k_end; k0 += 2) {
        const bool live = half < k_end - k0;
        const int k = live ? k0 + half : k0;
        if (k >= t_end) {  // another tile (the first one included)
            while (t + 1 < T && (t_end = tile_start[t + 1]) <= k) ++t;
            t_end = tile_start[t + 1];
            const int tx = t % tiles_x, ty = t / tiles_x;
            x0 = tx * tile;
            y0 = ty * tile;
            x1 = min(W, x0 + tile);
            y1 = min(H, y0 + tile);
        }
        const int g = sorted_gid[k];
        const float4 f0 = bfp[4 * (int64_t)g], f1 = bfp[4 * (int64_t)g + 1];
        const float mu2_lat = f0.x, mu2_ax = f0.y, r_lat = f0.z, r_ax = f0.w;
        const float inv00 = f1.x, inv01 = f1.y, inv11 = f1.z, bno_const = f1.w;
        f32x2 M0 = dup2(0.f), SL = M0, SA = M0, SLL = M0, SLA = M0, SAA = M0, MXX = M0, MXY = M0, MYY = M0;
        if (r_lat >= 0.f) {
            const int cx0 = max(x0, (int)ceilf((mu2_lat - r_lat) / lat_delta + col_off));
            const int cx1 = min(x1, (int)floorf((mu2_lat + r_lat) / lat_delta + col_off) + 1);
            const int cy0 = max(y0, (int)ceilf((mu2_ax - r_ax - near_mm) / ax_delta));
            const int cy1 = min(y1, (int)floorf((mu2_ax + r_ax - near_mm) / ax_delta) + 1);
            const int bw = cx1 - cx0, npx = bw > 0 && cy1 > cy0 ? bw * (cy1 - cy0) : 0;
            const float o = opac[g];
            // Pixels l + 32 i and l + 16 + 32 i of the box, row-major: (row, column) of each stepped without
            // divisions, in whole floats. The quotients of at most 32.5 by at most 32 are 1/64
            // away from a whole number or more.
            const float rbw = bw > 0 ? (float)bw : 1.f;
            const int ra = (int)__fdividef((float)l + 0.5f, rbw), rb = (int)__fdividef((float)l + 16.5f, rbw);
            const int step_y = (int)__fdividef(32.5f, rbw), step_x = 32 - step_y * bw;
            float xa = (float)(cx0 + l - ra * bw), xb = (float)(cx0 + l + 16 - rb * bw);
            float ya = (float)(cy0 + ra), yb = (float)(cy0 + rb);
            const float fx = (float)step_x, fy = (float)step_y, x_end = (float)cx1;
            int at_a = (cy0 + ra) * W + cx0 + l - ra * bw, at_b = (cy0 + rb) * W + cx0 + l + 16 - rb * bw;
            const int step = step_y * W + step_x, wrap = W - bw;
            const f32x2 ML = dup2(mu2_lat), MA = dup2(mu2_ax), I00 = dup2(inv00), I01 = dup2(inv01), I11 = dup2(inv11);
            const f32x2 CO = dup2(col_off), LD = dup2(lat_delta), AD = dup2(ax_delta), NR = dup2(near_mm);
            // Ordinary: a pixel that does not contribute adds exact zeros, and an infinite quad or weight
            // fails the weight test, without tests of their own.
            const bool ordinary = weight_min > 0.f && fabsf(o * bno_const) <= FLT_MAX && fabsf(bno_const) <= FLT_MAX &&
                                  (fabsf(inv00) + fabsf(inv01) + fabsf(inv11)) * (r_lat + r_ax) <= 1e30f;
            auto sweep = [&](auto ordinary_t) {
                constexpr bool ORD = decltype(ordinary_t)::value;
                for (int pi = l; pi < npx; pi += 32) {
                    const bool second = pi + 16 < npx;
                    const f32x2 GI = pk2(grad_image[at_a], second ? grad_image[at_b] : 0.f);
                    const f32x2 XC = sub2(pk2(xa, xb), CO), YF = pk2(ya, yb);
                    const f32x2 DL = fma2(XC, LD, neg2(ML)), D = sub2(fma2(YF, AD, NR), MA);
                    xa += fx;
                    ya += fy;
                    at_a += step;
                    if (xa >= x_end) {
                        xa -= rbw;
                        ya += 1.f;
                        at_a += wrap;
                    }
                    xb += fx;
                    yb += fy;
                    at_b += step;
                    if (xb >= x_end) {
                        xb -= rbw;
                        yb += 1.f;
                        at_b += wrap;
                    }
                    // the contractions of the compiled scalar expressions: every sum is the one a whole warp with
                    // one pixel per lane forms (the finite differences of the finalize magnify rounding)
                    f32x2 QL = fma2(I01, D, mul2(I00, DL)), QA = fma2(I11, D, mul2(I01, DL));
                    const f32x2 Q = fma2(DL, QL, mul2(D, QA));
                    const f32x2 BNO = mul2(dup2(bno_const), ex2_2(mul2(Q, CE)));
                    float e0, e1, d0, d1, q0, q1, w0, w1, u0, u1;
                    up2(DL, e0, e1);
                    up2(D, d0, d1);
                    up2(Q, q0, q1);
                    up2(mul2(dup2(o), BNO), w0, w1);
                    up2(mul2(GI, BNO), u0, u1);
                    bool in0 = fabsf(e0) <= r_lat && fabsf(d0) <= r_ax && q0 >= 0.f && !(w0 < weight_min);
                    bool in1 = second && fabsf(e1) <= r_lat && fabsf(d1) <= r_ax && q1 >= 0.f && !(w1 < weight_min);
                    if (!ORD) {
                        in0 = in0 && q0 <= FLT_MAX && fabsf(w0) <= FLT_MAX;
                        in1 = in1 && q1 <= FLT_MAX && fabsf(w1) <= FLT_MAX;
                        float a0, a1, b0, b1;
                        up2(QL, a0, a1);
                        up2(QA, b0, b1);
                        QL = pk2(in0 ? a0 : 0.f, in1 ? a1 : 0.f);
                        QA = pk2(in0 ? b0 : 0.f, in1 ? b1 : 0.f);
                    }
                    const f32x2 UB = pk2(in0 ? u0 : 0.f, in1 ? u1 : 0.f);
                    const f32x2 UL = mul2(UB, QL), UA = mul2(UB, QA), UX = mul2(UB, DL), UY = mul2(UB, D);
                    M0 = add2(M0, UB);
                    SL = add2(SL, UL);
                    SA = add2(SA, UA);
                    SLL = fma2(UL, QL, SLL);
                    SLA = fma2(UL, QA, SLA);
                    SAA = fma2(UA, QA, SAA);
                    MXX = fma2(UX, DL, MXX);
                    MXY = fma2(UX, D, MXY);
                    MYY = fma2(UY, D, MYY);
                }
            };
            if (ordinary)
                sweep(std::true_type{});
            else
                sweep(std::false_type{});
        }
        __syncwarp();
        // Reduction of the nine sums over the half-warp: eight of them transposed (each exchange halves
        // the values a lane carries, so lanes 2j and 2j + 1 end with sum j), the ninth plainly.
        const unsigned FULL = 0xffffffffu;
        const float v[8] = {sum2(SL), sum2(SA), sum2(SLL), sum2(SLA), sum2(SAA), sum2(MXX), sum2(MXY), sum2(MYY)};
        float m0 = sum2(M0), b4[4], c2[2];
        const bool h8 = lane & 8, h4 = lane & 4, h2 = lane & 2;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            b4[i] = (h8 ? v[4 + i] : v[i]) + __shfl_xor_sync(FULL, h8 ? v[i] : v[4 + i], 8);
#pragma unroll
        for (int i = 0; i < 2; ++i)
            c2[i] = (h4 ? b4[2 + i] : b4[i]) + __shfl_xor_sync(FULL, h4 ? b4[i] : b4[2 + i], 4);
        float d = (h2 ? c2[1] : c2[0]) + __shfl_xor_sync(FULL, h2 ? c2[0] : c2[1], 2);
        d += __shfl_xor_sync(FULL, d, 1);
#pragma unroll
        for (int x = 8; x >= 1; x >>= 1) m0 += __shfl_xor_sync(FULL, m0, x);
        // value j = bits 3..1 of the lane within its half (bit 3 selected the upper four, bit 2 the upper two)
        if (live && ((l & 1) == 0 || l == 1))
            partial[(int64_t)(4 * PARTIAL_F4) * sorted_inst[k] + (l == 1 ? (int)M_ONE : l >> 1)] = l == 1 ? m0 : d;
    }
}

__device__ __forceinline__ float sanitize(float g) {
    if (!isfinite(g)) return 0.f;
    if (fabsf(g) > GRAD_CLAMP) return copysignf(GRAD_CLAMP, g);
    return g;
}

// g_M -= Inv^T g_Inv Inv^T: adjoint of a 3x3 inverse (reference us_focus.cu:375-396).
__device__ __forceinline__ void inv3_bwd(const float Inv[9], const float gInv[9], float gM[9]) {
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float acc = 0.f;
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) acc += Inv[a * 3 + r] * gInv[a * 3 + b] * Inv[c * 3 + b];
            gM[r * 3 + c] -= acc;
        }
}

struct FpAdjoint {
    float mu2_lat, mu2_ax, inv00, inv01, inv11, det2, mu_ele, sc22, sigma_ele;
};

__device__ __forceinline__ float fp_dot(const Footprint& F, const FpAdjoint& a) {
    return a.mu2_lat * F.mu2_lat + a.mu2_ax * F.mu2_ax + a.inv00 * F.inv00 + a.inv01 * F.inv01 +
           a.inv11 * F.inv11 + a.det2 * F.det2 + a.mu_ele * F.mu_ele + a.sc22 * F.sc22 + a.sigma_ele * F.sigma_ele;
}

// Central difference (step eps) of the footprint/adjoint dot product with respect to one
// scale or quaternion component (reference us_focus.cu:313-373).
__device__ float shape_fd(const float* m, const float* s, const float* q, bool is_quat, int idx, float eps,
                          const Axes& A, float near_mm, float k_sigma, const float* P, const FpAdjoint& a) {
    float sp[3] = {s[0], s[1], s[2]}, sm[3] = {s[0], s[1], s[2]};
    float qp[4] = {q[0], q[1], q[2], q[3]}, qm[4] = {q[0], q[1], q[2], q[3]};
    if (is_quat) {
        qp[idx] += eps;
        qm[idx] -= eps;
    } else {
        sp[idx] += eps;
        sm[idx] -= eps;
    }
    Footprint Fp, Fm;
    const bool okp = footprint(m[0], m[1], m[2], sp[0], sp[1], sp[2], qp[0], qp[1], qp[2], qp[3], A, near_mm, k_sigma, P, Fp);
    const bool okm = footprint(m[0], m[1], m[2], sm[0], sm[1], sm[2], qm[0], qm[1], qm[2], qm[3], A, near_mm, k_sigma, P, Fm);
    const float lp = okp ? fp_dot(Fp, a) : 0.f;
    const float lm = okm ? fp_dot(Fm, a) : 0.f;
    return (lp - lm) / (2.f * eps);
}

// Exact shape gradient (analytic mode; the reference has only the central differences
// above): the adjoint of the probe-frame covariance, g_Sc (from the same chain through Se and
// Lc that gives the mean and pose gradients), is carried back through Sc = A^T Sigma_w A +
// 1e-6 I (Sc_ij = a_i^T Sigma_w a_j), the world covariance exactly as sigma_world forms it,
// Sigma_w = R D R with D = diag(s^2) (the reference's product, R from quat_rot), and
// R = rot(q / |q|):
//   G = dL/dSigma_w = sum_ij g_Sc[i][j] a_i a_j^T,
//   dL/ds_k = 2 s_k sum_ij G_ij R_ik R_kj (0 where the 1e-6 floor of the scale is active),
//   dL/dR = G R^T D + D R^T G, and dL/dq through the rotation of the normalised quaternion and
//   the normalisation.
__device__ void shape_analytic(const float* s, const float* q, const Axes& A, const float g_Sc[9], float d_s[3],
                               float d_q[4]) {
    const float3 ax[3] = {A.lat, A.ax, A.ele};
    float G[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float acc = 0.f;
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const float ai = r == 0 ? ax[i].x : (r == 1 ? ax[i].y : ax[i].z);
                    const float aj = c == 0 ? ax[j].x : (c == 1 ? ax[j].y : ax[j].z);
                    acc += g_Sc[i * 3 + j] * ai * aj;
                }
            G[r * 3 + c] = acc;
        }
    float R[9];
    quat_rot(q[0], q[1], q[2], q[3], R);
    const float sv[3] = {s[0], s[1], s[2]};
    float D[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float sk = fmaxf(sv[k], 1e-6f);
        D[k] = sk * sk;
        float acc = 0.f;  // sum_ij G_ij R_ik R_kj
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) acc += G[i * 3 + j] * R[i * 3 + k] * R[k * 3 + j];
        d_s[k] = sv[k] > 1e-6f ? 2.f * sk * acc : 0.f;
    }
    float gR[9];  // dL/dR = G R^T D + D R^T G
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            float u = 0.f, v = 0.f;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                u += G[a * 3 + c] * R[b * 3 + c];
                v += R[c * 3 + a] * G[c * 3 + b];
            }
            gR[a * 3 + b] = u * D[b] + D[a] * v;
        }
    // R of the unit quaternion (w, x, y, z) as in quat_rot; derivative per component
    const float n2 = q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
    const float nq = rsqrtf(fmaxf(1e-12f, n2));
    const float w = q[0] * nq, x = q[1] * nq, y = q[2] * nq, z = q[3] * nq;
    const float gw = 2.f * (-z * gR[1] + y * gR[2] + z * gR[3] - x * gR[5] - y * gR[6] + x * gR[7]);
    const float gx = 2.f * (y * gR[1] + z * gR[2] + y * gR[3] - 2.f * x * gR[4] - w * gR[5] + z * gR[6] + w * gR[7] -
                            2.f * x * gR[8]);
    const float gy = 2.f * (-2.f * y * gR[0] + x * gR[1] + w * gR[2] + x * gR[3] + z * gR[5] - w * gR[6] + z * gR[7] -
                            2.f * y * gR[8]);
    const float gz = 2.f * (-2.f * z * gR[0] - w * gR[1] + x * gR[2] + w * gR[3] - 2.f * z * gR[4] + y * gR[5] +
                            x * gR[6] + y * gR[7]);
    // through the normalisation u = q / |q| (no normalisation term where the 1e-12 floor is active)
    const float dot = (n2 > 1e-12f) ? (w * gw + x * gx + y * gy + z * gz) : 0.f;
    d_q[0] = nq * (gw - w * dot);
    d_q[1] = nq * (gx - x * dot);
    d_q[2] = nq * (gy - y * dot);
    d_q[3] = nq * (gz - z * dot);
}

__device__ __forceinline__ float3 normalize3_bwd(const float3 raw, const float3 n, const float3 g) {
    const float len = sqrtf(fmaxf(1e-12f, f3_dot(raw, raw)));
    const float il = 1.f / len;
    const float dn = f3_dot(n, g);
    return make_float3((g.x - n.x * dn) * il, (g.y - n.y * dn) * il, (g.z - n.z * dn) * il);
}

// The terms of one instance (reference us_focus.cu:398-477: per pixel up * weight, up c bno and cm = up c weight
// times the footprint derivatives) from its moments; cm = co * up * bno.
enum { P_MU_PROBE1 = 0, P_MU_PROBE2, P_SC22, P_MU_E0, P_MU_E1, P_SE00, P_SE01, P_SE11, P_OPACITY, P_INTENSITY,
       P_FP_MU2_LAT, P_FP_MU2_AX, P_FP_INV00, P_FP_INV01, P_FP_INV11, P_FP_DET2, P_FP_MU_ELE, P_FP_SC22,
       P_FP_SIGMA_ELE, P_COUNT };

__device__ __forceinline__ void instance_terms(const float4 a, const float4 b, const float m0, const float4 f2,
                                               const float4 f3, const float o, const float c, const float det_gamma,
                                               float acc[P_COUNT]) {
    const float s2_00 = f2.x, s2_01 = f2.y, s2_11 = f2.z, inv_det_norm = f2.w;
    const float mu_ele = f3.x, inv_de = f3.y, dse_dax = f3.z, sigma_ele = f3.w;
    const float ql = a.x, qa = a.y, qll = a.z, qla = a.w, qaa = b.x, mxx = b.y, mxy = b.z, myy = b.w;
    const float co = c * o;  // cm = co * up * bno
    const float ele2 = mu_ele * mu_ele * inv_de * inv_de;
    acc[P_INTENSITY] = o * m0;
    acc[P_OPACITY] = c * m0;
    acc[P_MU_E0] = co * ql;
    acc[P_MU_E1] = co * qa;
    acc[P_FP_MU2_LAT] = co * ql;
    acc[P_FP_MU2_AX] = co * qa;
    acc[P_FP_INV00] = co * (-0.5f * mxx);
    acc[P_FP_INV01] = co * (-mxy);
    acc[P_FP_INV11] = co * (-0.5f * myy);
    acc[P_FP_DET2] = co * m0 * (-det_gamma * inv_det_norm);
    acc[P_SE00] = co * (0.5f * qll - det_gamma * s2_11 * inv_det_norm * m0);
    acc[P_SE01] = 0.5f * co * (qla + 2.f * det_gamma * s2_01 * inv_det_norm * m0);
    acc[P_SE11] = co * (0.5f * qaa - det_gamma * s2_00 * inv_det_norm * m0);
    acc[P_MU_PROBE2] = co * m0 * (-mu_ele * inv_de);
    acc[P_SC22] = co * m0 * (0.5f * ele2);
    acc[P_MU_PROBE1] = co * m0 * (ele2 * dse_dax);
    acc[P_FP_MU_ELE] = co * m0 * (-mu_ele * inv_de);
    acc[P_FP_SC22] = co * m0 * (0.5f * ele2);
    acc[P_FP_SIGMA_ELE] = co * m0 * (ele2 * sigma_ele);
}

// Per Gaussian: the terms of its instances summed in instance order, then the chain rule
// through Se and Lc, finite-difference shape gradients, sanitising, and the pose contribution
// (reference us_focus.cu:479-803).
__global__ void __launch_bounds__(128)
finalize_kernel(int64_t G, float k_sigma, const int* __restrict__ inst_offset, const int4* __restrict__ rects,
                const float* __restrict__ means, const float* __restrict__ scales, const float* __restrict__ quats,
                const float* __restrict__ opac, const float* __restrict__ inten, const float4* __restrict__ bfp,
                const float* __restrict__ pose, const float* __restrict__ grid, const float* __restrict__ params,
                const long long* __restrict__ header, const float4* __restrict__ partial, int pose_grad,
                int shape_analytic_mode, float* __restrict__ d_means, float* __restrict__ d_scales, float* __restrict__ d_quats,
                float* __restrict__ d_opac, float* __restrict__ d_inten, float* __restrict__ pose_partial) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    float* pp = pose_grad ? pose_partial + 12 * g : nullptr;
    if (pp) {
#pragma unroll
        for (int i = 0; i < 12; ++i) pp[i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        d_means[3 * g + i] = 0.f;
        d_scales[3 * g + i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) d_quats[4 * g + i] = 0.f;
    d_opac[g] = 0.f;
    d_inten[g] = 0.f;
    if (header[H_FLAGS] != 0) return;
    if ((int)(grid[SG_PROBE_TYPE] + 0.5f) != 0) return;  // linear probes only, as the reference
    const int4 rect = rects[g];
    if (rect.x >= rect.z || rect.y >= rect.w) return;
    const Axes A = axes_from_pose(pose);
    const float near_mm = grid[SG_NEAR_MM];
    const float* m = means + 3 * g;
    const float* s = scales + 3 * g;
    const float* q = quats + 4 * g;
    Footprint F;
    if (!footprint(m[0], m[1], m[2], s[0], s[1], s[2], q[0], q[1], q[2], q[3], A, near_mm, k_sigma, params, F)) return;

    float acc[P_COUNT];
#pragma unroll
    for (int i = 0; i < P_COUNT; ++i) acc[i] = 0.f;
    {
        const float4 f2 = bfp[4 * g + 2], f3 = bfp[4 * g + 3];
        const float det_gamma = params[UF_DET_GAMMA], c_opac = opac[g], c_inten = inten[g];
        const int i1 = inst_offset[g + 1];
        for (int i = inst_offset[g]; i < i1; ++i) {
            const float4* r = partial + (int64_t)PARTIAL_F4 * i;
            float v[P_COUNT];
            instance_terms(r[0], r[1], reinterpret_cast<const float*>(r)[M_ONE], f2, f3, c_opac, c_inten, det_gamma, v);
#pragma unroll
            for (int k = 0; k < P_COUNT; ++k) acc[k] = __fadd_rn(acc[k], v[k]);
        }
    }

    const float depth = fmaxf(F.mu_ax - near_mm, 0.f);
    const bool depth_active = F.mu_ax > near_mm;
    const float se_raw = params[UF_SIGMA_ELE_0] + params[UF_SIGMA_ELE_1] * depth;
    const float sl_raw = params[UF_SIGMA_LAT_0] + params[UF_SIGMA_LAT_1] * depth;
    const bool use_lat = params[UF_USE_LATERAL_FOCUS] != 0.f;
    const float dse = (depth_active && se_raw > params[UF_SIGMA_ELE_MIN] && se_raw < params[UF_SIGMA_ELE_MAX])
                          ? params[UF_SIGMA_ELE_1] : 0.f;
    const float dsl = (use_lat && depth_active && sl_raw > params[UF_SIGMA_LAT_MIN] && sl_raw < params[UF_SIGMA_LAT_MAX])
                          ? params[UF_SIGMA_LAT_1] : 0.f;
    const float dlam_ele = -2.f * dse / fmaxf(F.sigma_ele * F.sigma_ele * F.sigma_ele, 1e-12f);
    const float dlam_lat = use_lat ? -2.f * dsl / fmaxf(F.sigma_lat * F.sigma_lat * F.sigma_lat, 1e-12f) : 0.f;

    const float mu_c[3] = {F.mu_lat, F.mu_ax, F.mu_ele};
    const float* Lc = F.Lc;
    const float* Se = F.Se;
    float g_mu_probe[3] = {0.f, acc[P_MU_PROBE1], acc[P_MU_PROBE2]};
    float g_Sc[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, acc[P_SC22]};
    const float g_mu_e[3] = {acc[P_MU_E0], acc[P_MU_E1], 0.f};
    float g_Se[9] = {acc[P_SE00], acc[P_SE01], 0.f, acc[P_SE01], acc[P_SE11], 0.f, 0.f, 0.f, 0.f};
    const float y_lc[3] = {Lc[0] * mu_c[0] + Lc[1] * mu_c[1] + Lc[2] * mu_c[2],
                           Lc[3] * mu_c[0] + Lc[4] * mu_c[1] + Lc[5] * mu_c[2],
                           Lc[6] * mu_c[0] + Lc[7] * mu_c[1] + Lc[8] * mu_c[2]};
    const float g_y[3] = {Se[0] * g_mu_e[0] + Se[3] * g_mu_e[1] + Se[6] * g_mu_e[2],
                          Se[1] * g_mu_e[0] + Se[4] * g_mu_e[1] + Se[7] * g_mu_e[2],
                          Se[2] * g_mu_e[0] + Se[5] * g_mu_e[1] + Se[8] * g_mu_e[2]};
    float g_Lc[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) g_Lc[i * 3 + j] = g_y[i] * mu_c[j];
    g_mu_probe[0] += Lc[0] * g_y[0] + Lc[3] * g_y[1] + Lc[6] * g_y[2];
    g_mu_probe[1] += Lc[1] * g_y[0] + Lc[4] * g_y[1] + Lc[7] * g_y[2];
    g_mu_probe[2] += Lc[2] * g_y[0] + Lc[5] * g_y[1] + Lc[8] * g_y[2];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) g_Se[i * 3 + j] += g_mu_e[i] * y_lc[j];
    float g_Le[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    inv3_bwd(Se, g_Se, g_Le);
#pragma unroll
    for (int i = 0; i < 9; ++i) g_Lc[i] += g_Le[i];
    g_mu_probe[1] += g_Le[0] * dlam_lat + g_Le[8] * dlam_ele;
    inv3_bwd(Lc, g_Lc, g_Sc);

    d_inten[g] = sanitize(acc[P_INTENSITY]);
    d_opac[g] = sanitize(acc[P_OPACITY]);
    const FpAdjoint adj = {acc[P_FP_MU2_LAT], acc[P_FP_MU2_AX], acc[P_FP_INV00], acc[P_FP_INV01], acc[P_FP_INV11],
                           acc[P_FP_DET2], acc[P_FP_MU_ELE], acc[P_FP_SC22], acc[P_FP_SIGMA_ELE]};
    if (shape_analytic_mode) {
        float ds[3], dq[4];
        shape_analytic(s, q, A, g_Sc, ds, dq);
        for (int k = 0; k < 3; ++k) d_scales[3 * g + k] = sanitize(ds[k]);
        for (int k = 0; k < 4; ++k) d_quats[4 * g + k] = sanitize(dq[k]);
    } else {
        for (int k = 0; k < 3; ++k)
            d_scales[3 * g + k] = sanitize(shape_fd(m, s, q, false, k, 1e-3f, A, near_mm, k_sigma, params, adj));
        for (int k = 0; k < 4; ++k)
            d_quats[4 * g + k] = sanitize(shape_fd(m, s, q, true, k, 1e-3f, A, near_mm, k_sigma, params, adj));
    }
    const float3 g_delta = make_float3(g_mu_probe[0] * A.lat.x + g_mu_probe[1] * A.ax.x + g_mu_probe[2] * A.ele.x,
                                       g_mu_probe[0] * A.lat.y + g_mu_probe[1] * A.ax.y + g_mu_probe[2] * A.ele.y,
                                       g_mu_probe[0] * A.lat.z + g_mu_probe[1] * A.ax.z + g_mu_probe[2] * A.ele.z);
    d_means[3 * g + 0] = sanitize(g_delta.x);
    d_means[3 * g + 1] = sanitize(g_delta.y);
    d_means[3 * g + 2] = sanitize(g_delta.z);
    if (!pp) return;

    // Pose contribution of this Gaussian (reference us_focus.cu:754-802); reduced over
    // Gaussians by pose_reduce_kernel instead of float atomics.
    float R[9];
    quat_rot(q[0], q[1], q[2], q[3], R);
    const float sx = fmaxf(s[0], 1e-6f), sy = fmaxf(s[1], 1e-6f), sz = fmaxf(s[2], 1e-6f);
    float Sw[9];
    sigma_world(sx, sy, sz, R, Sw);
    const float3 axes[3] = {A.lat, A.ax, A.ele};
    float3 ga[3] = {make_float3(0.f, 0.f, 0.f), make_float3(0.f, 0.f, 0.f), make_float3(0.f, 0.f, 0.f)};
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            const float gij = g_Sc[i * 3 + j];
            const float3 ai = axes[i], aj = axes[j];
            const float3 Sai = make_float3(Sw[0] * ai.x + Sw[1] * ai.y + Sw[2] * ai.z, Sw[3] * ai.x + Sw[4] * ai.y + Sw[5] * ai.z,
                                           Sw[6] * ai.x + Sw[7] * ai.y + Sw[8] * ai.z);
            const float3 Saj = make_float3(Sw[0] * aj.x + Sw[1] * aj.y + Sw[2] * aj.z, Sw[3] * aj.x + Sw[4] * aj.y + Sw[5] * aj.z,
                                           Sw[6] * aj.x + Sw[7] * aj.y + Sw[8] * aj.z);
            ga[i].x += gij * Saj.x; ga[i].y += gij * Saj.y; ga[i].z += gij * Saj.z;
            ga[j].x += gij * Sai.x; ga[j].y += gij * Sai.y; ga[j].z += gij * Sai.z;
        }
    const float3 dw = make_float3(m[0] - A.origin.x, m[1] - A.origin.y, m[2] - A.origin.z);
    const float3 g_lat = normalize3_bwd(A.raw_lat, A.lat, make_float3(g_mu_probe[0] * dw.x + ga[0].x, g_mu_probe[0] * dw.y + ga[0].y, g_mu_probe[0] * dw.z + ga[0].z));
    const float3 g_ax = normalize3_bwd(A.raw_ax, A.ax, make_float3(g_mu_probe[1] * dw.x + ga[1].x, g_mu_probe[1] * dw.y + ga[1].y, g_mu_probe[1] * dw.z + ga[1].z));
    const float3 g_ele = normalize3_bwd(A.raw_ele, A.ele, make_float3(g_mu_probe[2] * dw.x + ga[2].x, g_mu_probe[2] * dw.y + ga[2].y, g_mu_probe[2] * dw.z + ga[2].z));
    // 4x4 row-major pose indices: column 0 = lateral, 1 = axial, 2 = elevational, 3 = origin.
    pp[0] = g_lat.x; pp[1] = g_lat.y; pp[2] = g_lat.z;
    pp[3] = g_ax.x; pp[4] = g_ax.y; pp[5] = g_ax.z;
    pp[6] = g_ele.x; pp[7] = g_ele.y; pp[8] = g_ele.z;
    pp[9] = -g_delta.x; pp[10] = -g_delta.y; pp[11] = -g_delta.z;
}

// Sums the per-Gaussian pose contributions in a fixed order, in two launches: block b of
// POSE_BLOCKS reduces the contiguous chunk b of Gaussians and leaves its 12 sums in the chunk's
// first slot of pose_partial; one block then adds the chunk sums in block order.
constexpr int POSE_BLOCKS = 512;

// The pose gradient is a sum over all Gaussians of terms with long lever arms that largely
// cancel, so the sums run in double: per-Gaussian float contributions, chunk sums and the final
// sum accumulate in double (fixed order), and the chunk sums stay in double (two float slots
// each, in the chunk's own first Gaussians' slots; chunks hold at least two Gaussians).
__device__ __forceinline__ void pose_block_sum(double a[12]) {
    __shared__ double red[256][13];
#pragma unroll
    for (int i = 0; i < 12; ++i) red[threadIdx.x][i] = a[i];
    __syncthreads();
    for (int stride = 128; stride > 0; stride >>= 1) {
        if (threadIdx.x < stride)
#pragma unroll
            for (int i = 0; i < 12; ++i) red[threadIdx.x][i] += red[threadIdx.x + stride][i];
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 12; ++i) a[i] = red[0][i];
}

__global__ void __launch_bounds__(256)
pose_chunk_kernel(int64_t G, int64_t chunk, float* __restrict__ pose_partial) {
    const int64_t g0 = (int64_t)blockIdx.x * chunk;
    if (g0 >= G) return;
    const int64_t g1 = g0 + chunk < G ? g0 + chunk : G;
    double a[12];
#pragma unroll
    for (int i = 0; i < 12; ++i) a[i] = 0.0;
    for (int64_t g = g0 + threadIdx.x; g < g1; g += blockDim.x)
#pragma unroll
        for (int i = 0; i < 12; ++i) a[i] += (double)pose_partial[12 * g + i];
    pose_block_sum(a);  // ends with every read of the chunk done
    double* out = reinterpret_cast<double*>(pose_partial + 12 * g0);
    if (threadIdx.x < 12) out[threadIdx.x] = a[threadIdx.x];
}

__global__ void __launch_bounds__(256)
pose_final_kernel(int64_t G, int64_t chunk, const float* __restrict__ pose_partial, float* __restrict__ d_pose) {
    const int nb = (int)((G + chunk - 1) / chunk);
    double a[12];
#pragma unroll
    for (int i = 0; i < 12; ++i) a[i] = 0.0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        const double* in = reinterpret_cast<const double*>(pose_partial + 12 * (int64_t)b * chunk);
#pragma unroll
        for (int i = 0; i < 12; ++i) a[i] += in[i];
    }
    pose_block_sum(a);
    if (threadIdx.x == 0) {
        const int idx[12] = {0, 4, 8, 1, 5, 9, 2, 6, 10, 3, 7, 11};
        for (int i = 0; i < 16; ++i) d_pose[i] = 0.f;
        for (int i = 0; i < 12; ++i) d_pose[idx[i]] = (float)a[i];
    }
}

__global__ void export_kernel(int T, const int* __restrict__ tile_start, const int* __restrict__ sorted_gid,
                              int* __restrict__ out_ids, int* __restrict__ rs, int* __restrict__ re) {
    const int t = blockIdx.x;
    if (t >= T) return;
    const int s0 = tile_start[t], s1 = tile_start[t + 1];
    if (threadIdx.x == 0) {
        rs[t] = (s1 > s0) ? s0 : -1;
        re[t] = (s1 > s0) ? s1 : -1;
    }
    for (int s = s0 + threadIdx.x; s < s1; s += blockDim.x) out_ids[s] = sorted_gid[s];
}

}  // namespace gp
}  // namespace us3d

using namespace us3d;
using namespace us3d::gp;

static BinAttr g_gp_sort_attr;

static int gp_sizes(int H, int W, int tile, int* tx, int* ty) {
    US3D_CHECK_ARG(H > 0 && W > 0, "H/W must be positive");
    US3D_CHECK_ARG(tile > 0 && tile * tile <= 1024, "tile_size_px must be in [1, 32]");
    *tx = (W + tile - 1) / tile;
    *ty = (H + tile - 1) / tile;
    return US3D_OK;
}

extern "C" size_t us3d_gp_workspace_bytes(int64_t n_gauss, int32_t H, int32_t W, int32_t tile, int64_t cap) {
    if (n_gauss < 0 || cap < 0 || H <= 0 || W <= 0 || tile <= 0) return 0;
    const int64_t T = (int64_t)((W + tile - 1) / tile) * ((H + tile - 1) / tile);
    return carve(nullptr, n_gauss, T, cap).bytes;
}

extern "C" size_t us3d_gp_backward_scratch_bytes(int64_t n_gauss, int64_t cap) {
    if (n_gauss < 0 || cap < 0) return 0;
    // + 2 Gaussians' pose slots: a chunk's double sums span two slots, also for a last chunk of one
    return (size_t)cap * PARTIAL_F4 * sizeof(float4) + (size_t)(n_gauss + 2) * 12 * sizeof(float) + 256;
}

static int gp_forward_impl(void* workspace, size_t workspace_bytes, int64_t n_gauss, const float* means,
                           const float* scales, const float* quats, const float* opacities, const float* intensities,
                           const float* pose, const float* grid_pack, const float* focus_params, int32_t H, int32_t W,
                           float lateral_spacing, float axial_spacing, float axial_near, int32_t tile_size,
                           float k_sigma, int32_t sort_by_v, int64_t cap, float* out_image, StatusRead* status,
                           void* stream_) {
    int tx, ty;
    int st = gp_sizes(H, W, tile_size, &tx, &ty);
    if (st != US3D_OK) return st;
    US3D_CHECK_ARG(workspace && out_image && pose && grid_pack && focus_params, "NULL pointer argument");
    US3D_CHECK_ARG(n_gauss >= 0 && n_gauss <= 0x7fffffffLL, "n_gauss out of range");
    US3D_CHECK_ARG(n_gauss == 0 || (means && scales && quats && opacities && intensities), "NULL parameter pointer");
    US3D_CHECK_ARG(cap >= 0 && cap <= 0x7fffffffLL, "instance capacity must be in [0, 2^31)");
    US3D_CHECK_ARG(lateral_spacing > 0.f && axial_spacing > 0.f, "pixel spacing must be > 0");
    const int64_t T = (int64_t)tx * ty;
    const Workspace w = carve(workspace, n_gauss, T, cap);
    US3D_CHECK_ARG(workspace_bytes >= w.bytes, "workspace too small: %zu < %zu", workspace_bytes, w.bytes);
    cudaStream_t stream = (cudaStream_t)stream_;
    const int prof = prof_begin("gp_forward", stream);
    init_kernel<<<(unsigned)((T + 255) / 256), 256, 0, stream>>>(T, w.tile_count, w.tile_cursor, w.header, cap, n_gauss);
    const unsigned gb = (unsigned)((n_gauss + 255) / 256);
    if (n_gauss > 0)
        preprocess_kernel<<<gb, 256, 0, stream>>>(n_gauss, H, W, tile_size, tx, ty, lateral_spacing, axial_spacing,
                                                  axial_near, k_sigma, sort_by_v, means, scales, quats, opacities,
                                                  intensities, pose, grid_pack, focus_params, w.rects, w.dkey,
                                                  w.touched, w.tile_count, w.cand, w.bfp);
    US3D_CHECK_LAUNCH("gp preprocess");
    const bool fill = fills(n_gauss, T, sort_by_v != 0);
    US3D_CHECK_CUDA(launch_bins(n_gauss, tx, T, RectOf4{w.rects}, sort_by_v ? w.dkey : nullptr, w.touched, w.stable,
                                w.tile_count, w.tile_start, w.tile_cursor, w.inst_offset, w.bs_g, w.bs_t, w.header, cap,
                                fill ? nullptr : w.keys, w.slot_inst, w.sorted_gid, w.sorted_inst, g_gp_sort_attr, stream));
    if (status != nullptr) {
        const int rc = status->record(w.header, stream);
        if (rc != US3D_OK) return rc;
    }
    const int blocks = ((tile_size + BLK_W - 1) / BLK_W) * ((tile_size + BLK_H - 1) / BLK_H);  // pixel blocks per tile
    forward_kernel<<<(unsigned)(T * blocks), GROUP, 0, stream>>>(H, W, tile_size, tx, grid_pack, focus_params,
                                                                 w.tile_start, w.sorted_gid, w.header, w.cand, out_image);
    US3D_CHECK_LAUNCH("gp forward");
    prof_end(prof, stream);
    count_launches(1 + (n_gauss > 0) + bins_launches(n_gauss, T, fill, sort_by_v != 0) + 1);
    return US3D_OK;
}

extern "C" int us3d_gp_forward(void* workspace, size_t workspace_bytes, int64_t n_gauss, const float* means,
                               const float* scales, const float* quats, const float* opacities,
                               const float* intensities, const float* pose, const float* grid_pack,
                               const float* focus_params, int32_t H, int32_t W, float lateral_spacing,
                               float axial_spacing, float axial_near, int32_t tile_size, float k_sigma,
                               int32_t sort_by_v, int64_t cap, float* out_image, void* stream_) {
    return gp_forward_impl(workspace, workspace_bytes, n_gauss, means, scales, quats, opacities, intensities, pose,
                           grid_pack, focus_params, H, W, lateral_spacing, axial_spacing, axial_near, tile_size,
                           k_sigma, sort_by_v, cap, out_image, nullptr, stream_);
}

extern "C" int us3d_gp_forward_checked(void* workspace, size_t workspace_bytes, int64_t n_gauss, const float* means,
                                       const float* scales, const float* quats, const float* opacities,
                                       const float* intensities, const float* pose, const float* grid_pack,
                                       const float* focus_params, int32_t H, int32_t W, float lateral_spacing,
                                       float axial_spacing, float axial_near, int32_t tile_size, float k_sigma,
                                       int32_t sort_by_v, int64_t cap, float* out_image, int64_t* total,
                                       int32_t* flags, void* stream_) {
    StatusRead status;
    const int st = gp_forward_impl(workspace, workspace_bytes, n_gauss, means, scales, quats, opacities, intensities,
                                   pose, grid_pack, focus_params, H, W, lateral_spacing, axial_spacing, axial_near,
                                   tile_size, k_sigma, sort_by_v, cap, out_image, &status, stream_);
    return st != US3D_OK ? st : wait_status(status, total, flags);
}

extern "C" int us3d_gp_read_status(const void* workspace, int64_t* total, int32_t* flags, void* stream_) {
    US3D_CHECK_ARG(workspace != nullptr, "workspace is NULL");
    long long hdr[H_WORDS];
    cudaStream_t stream = (cudaStream_t)stream_;
    US3D_CHECK_CUDA(cudaMemcpyAsync(hdr, workspace, sizeof(hdr), cudaMemcpyDeviceToHost, stream));
    US3D_CHECK_CUDA(cudaStreamSynchronize(stream));
    if (total) *total = hdr[H_TOTAL];
    if (flags) *flags = (int32_t)hdr[H_FLAGS];
    return US3D_OK;
}

extern "C" int us3d_gp_backward(void* workspace, int64_t n_gauss, const float* means, const float* scales,
                                const float* quats, const float* opacities, const float* intensities,
                                const float* pose, const float* grid_pack, const float* focus_params, int32_t H,
                                int32_t W, int32_t tile_size, float k_sigma, int64_t cap, const float* grad_image,
                                int32_t grad_flags, void* scratch, size_t scratch_bytes, float* d_means,
                                float* d_scales, float* d_quats, float* d_opacities, float* d_intensities,
                                float* d_pose, void* stream_) {
    US3D_CHECK_ARG((grad_flags & ~(US3D_GP_GRAD_POSE | US3D_GP_GRAD_SHAPE_ANALYTIC)) == 0,
                   "unknown gradient flags 0x%x", (unsigned)grad_flags);
    const int pose_grad = (grad_flags & US3D_GP_GRAD_POSE) ? 1 : 0;
    const int shape_analytic_mode = (grad_flags & US3D_GP_GRAD_SHAPE_ANALYTIC) ? 1 : 0;
    int tx, ty;
    int st = gp_sizes(H, W, tile_size, &tx, &ty);
    if (st != US3D_OK) return st;
    US3D_CHECK_ARG(workspace && grad_image && pose && grid_pack && focus_params, "NULL pointer argument");
    US3D_CHECK_ARG(n_gauss >= 0 && n_gauss <= 0x7fffffffLL, "n_gauss out of range");
    US3D_CHECK_ARG(cap >= 0 && cap <= 0x7fffffffLL, "instance capacity must be in [0, 2^31)");
    US3D_CHECK_ARG(scratch_bytes >= us3d_gp_backward_scratch_bytes(n_gauss, cap), "backward scratch too small");
    US3D_CHECK_ARG(n_gauss == 0 || (means && scales && quats && opacities && intensities && d_means && d_scales &&
                                    d_quats && d_opacities && d_intensities), "NULL gradient/parameter pointer");
    US3D_CHECK_ARG(!pose_grad || d_pose, "d_pose is NULL");
    const int64_t T = (int64_t)tx * ty;
    const Workspace w = carve(workspace, n_gauss, T, cap);
    float* partial = reinterpret_cast<float*>(scratch);
    float* pose_partial = partial + (size_t)cap * PARTIAL_F4 * 4;
    pose_partial = reinterpret_cast<float*>(align_up(reinterpret_cast<uintptr_t>(pose_partial), 256));
    cudaStream_t stream = (cudaStream_t)stream_;
    const int prof = prof_begin("gp_backward", stream);
    int launches = 0;
    if (T > 0) {
        backward_inst_kernel<<<148 * 8, BWD_WARPS * 32, 0, stream>>>(
            (int)T, W, tile_size, tx, opacities, w.bfp, grid_pack, focus_params, w.tile_start,
            w.sorted_gid, w.sorted_inst, w.header, grad_image, partial, H);
        US3D_CHECK_LAUNCH("gp backward instances");
        launches = 1;
    }
    if (n_gauss > 0) {
        finalize_kernel<<<(unsigned)((n_gauss + 127) / 128), 128, 0, stream>>>(
            n_gauss, k_sigma, w.inst_offset, w.rects, means, scales, quats, opacities, intensities, w.bfp, pose, grid_pack,
            focus_params, w.header, reinterpret_cast<const float4*>(partial), pose_grad, shape_analytic_mode, d_means, d_scales, d_quats, d_opacities, d_intensities,
            pose_partial);
        US3D_CHECK_LAUNCH("gp finalize");
        ++launches;
    }
    if (pose_grad) {
        const int64_t chunk = std::max<int64_t>(2, (n_gauss + POSE_BLOCKS - 1) / POSE_BLOCKS);
        if (n_gauss > 0) {
            pose_chunk_kernel<<<(unsigned)((n_gauss + chunk - 1) / chunk), 256, 0, stream>>>(n_gauss, chunk,
                                                                                             pose_partial);
            ++launches;
        }
        pose_final_kernel<<<1, 256, 0, stream>>>(n_gauss, chunk, pose_partial, d_pose);
        US3D_CHECK_LAUNCH("gp pose reduce");
        ++launches;
    }
    prof_end(prof, stream);
    count_launches(launches);
    return US3D_OK;
}

extern "C" int us3d_gp_export_bins(const void* workspace, int64_t n_gauss, int32_t H, int32_t W, int32_t tile_size,
                                   int64_t cap, int32_t* out_sorted_ids, int32_t* out_range_start,
                                   int32_t* out_range_end, int32_t* out_rects, void* stream_) {
    int tx, ty;
    int st = gp_sizes(H, W, tile_size, &tx, &ty);
    if (st != US3D_OK) return st;
    US3D_CHECK_ARG(workspace && out_range_start && out_range_end, "NULL pointer argument");
    const int64_t T = (int64_t)tx * ty;
    const Workspace w = carve(const_cast<void*>(workspace), n_gauss, T, cap);
    cudaStream_t stream = (cudaStream_t)stream_;
    export_kernel<<<(unsigned)T, 256, 0, stream>>>((int)T, w.tile_start, w.sorted_gid, out_sorted_ids,
                                                   out_range_start, out_range_end);
    if (out_rects && n_gauss > 0)
        US3D_CHECK_CUDA(cudaMemcpyAsync(out_rects, w.rects, sizeof(int4) * n_gauss, cudaMemcpyDeviceToDevice, stream));
    US3D_CHECK_LAUNCH("gp export");
    count_launches(1);
    return US3D_OK;
}
