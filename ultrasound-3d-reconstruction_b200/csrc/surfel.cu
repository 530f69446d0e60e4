// UltraGS baseline: 2D-Gaussian-surfel rasterisation (ray-splat intersection, front-to-back
// alpha compositing, seven auxiliary maps) with its backward.
//
// Reference behaviour restated here (paths inside KevinWCCC/ultrasound-3d-reconstruction,
// ops/ultrags_baseline_renderer):
//   cuda_rasterizer/forward.cu:20-65       SH -> RGB (degree-2 "ultrasound" terms), clamp
//   cuda_rasterizer/forward.cu:69-107      splat-to-pixel homography T = S2W^T * W2N * N2P
//   cuda_rasterizer/forward.cu:109-139     screen-space AABB of the 3-sigma ellipse
//   cuda_rasterizer/forward.cu:141-246     preprocess: near cull, dual-visible normal, radius
//   cuda_rasterizer/forward.cu:249-439     tile compositing, early termination, aux maps
//   cuda_rasterizer/rasterizer_impl.cu:70-137  keys (tile << 32 | depth bits), tile ranges
//   cuda_rasterizer/backward.cu:103-404    back-to-front replay and per-pair gradients
//   cuda_rasterizer/backward.cu:406-602    homography / AABB / rotation / SH gradients
//
// B200 design. Binning gives every tile its (tile, Gaussian) instances in (depth bits, Gaussian index) order,
// the order the reference's stable radix sort produces: on small grids by ordering the Gaussians once
// and filling the tiles in that order, else by sorting each tile's bucket in shared memory. The
// forward gives each thread one pixel; every warp keeps, of 32 surfels of the list at a time, those whose
// exact reach box meets its 8x4 pixels and stages their 80-byte records itself, independently of
// the other warps. The backward keeps the reference's per-pixel back-to-front replay (its recurrences
// need it) on the same kind of lists, but replaces the per-pair float atomics by a fixed-order
// reduction: two surfels at a time, each warp reduces its 32 pixels' 18 gradient terms of both with
// one transposed butterfly (37 shuffles), the sums of the warps that replayed a surfel are added in
// warp order into one per-instance partial, and per Gaussian the instances are summed in order and the
// preprocess backward follows. Results are deterministic.
//
// Matrix products are evaluated with the summation order of the GLM operators the
// reference uses (column-major, k ascending, zero entries included), so that pixel
// rectangles, keys and contributor counts agree bit for bit under the same compiler flags.
#include "us3d_common.cuh"
#include "scan.cuh"
#include "binning.cuh"
#include "stable_bins.cuh"

namespace us3d {
namespace gs {

constexpr int TILE = 16;
constexpr int BLOCK = TILE * TILE;
constexpr int REC_F4 = 5;        // 80-byte per-Gaussian render record
constexpr int BWD_BATCH = 64;    // Gaussians staged per backward batch
constexpr int NGRAD = 18;        // per-instance gradient terms
constexpr int PARTIAL_F4 = 5;    // 20 floats per instance partial (2 pad)
constexpr float NEAR_N = 0.2f;
constexpr float FAR_N = 100.0f;
constexpr float FILTER_SIZE = 0.707106f;
constexpr float FILTER_INV_SQUARE = 2.0f;
constexpr float SH_C0 = 0.28209479177387814f;
constexpr float SH_C1 = 0.4886025119029199f;
enum { FLAG_PREFILTERED = 4 };

// Column-major small matrix: m[c][r] is column c, row r (C columns, R rows).
template <int C, int R>
struct Mat {
    float m[C][R];
};

// (C1 x R1) * (C2 x C1): out[c][r] = sum_k a[k][r] * b[c][k], k ascending, left to right.
template <int C1, int R1, int C2>
__device__ __forceinline__ Mat<C2, R1> mmul(const Mat<C1, R1>& a, const Mat<C2, C1>& b) {
    Mat<C2, R1> o;
#pragma unroll
    for (int c = 0; c < C2; ++c)
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            float acc = a.m[0][r] * b.m[c][0];
#pragma unroll
            for (int k = 1; k < C1; ++k) acc = acc + a.m[k][r] * b.m[c][k];
            o.m[c][r] = acc;
        }
    return o;
}

template <int C, int R>
__device__ __forceinline__ Mat<R, C> transpose(const Mat<C, R>& a) {
    Mat<R, C> o;
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
        for (int r = 0; r < R; ++r) o.m[r][c] = a.m[c][r];
    return o;
}

struct V3 {
    float x, y, z;
};
__device__ __forceinline__ V3 v3(float x, float y, float z) { return V3{x, y, z}; }
__device__ __forceinline__ V3 vmul(const V3 a, const V3 b) { return v3(a.x * b.x, a.y * b.y, a.z * b.z); }
__device__ __forceinline__ V3 vscale(float s, const V3 a) { return v3(s * a.x, s * a.y, s * a.z); }
__device__ __forceinline__ V3 vadd(const V3 a, const V3 b) { return v3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ V3 vsub(const V3 a, const V3 b) { return v3(a.x - b.x, a.y - b.y, a.z - b.z); }
// Dot product as a product vector summed x + y + z (the GLM form).
__device__ __forceinline__ float vdot(const V3 a, const V3 b) {
    const V3 t = vmul(a, b);
    return t.x + t.y + t.z;
}
__device__ __forceinline__ V3 vcross(const V3 a, const V3 b) {
    return v3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ V3 col3(const Mat<3, 3>& a, int c) { return v3(a.m[c][0], a.m[c][1], a.m[c][2]); }

// Rotation of the (w,x,y,z) quaternion stored as (q.x, q.y, q.z, q.w), column-major
// (gsplat's quat_to_rotmat, reference auxiliary.h:199-222).
__device__ __forceinline__ Mat<3, 3> quat_rot(const float4 q) {
    const float s = rsqrtf(q.w * q.w + q.x * q.x + q.y * q.y + q.z * q.z);
    const float w = q.x * s, x = q.y * s, y = q.z * s, z = q.w * s;
    Mat<3, 3> R;
    R.m[0][0] = 1.f - 2.f * (y * y + z * z);
    R.m[0][1] = 2.f * (x * y + w * z);
    R.m[0][2] = 2.f * (x * z - w * y);
    R.m[1][0] = 2.f * (x * y - w * z);
    R.m[1][1] = 1.f - 2.f * (x * x + z * z);
    R.m[1][2] = 2.f * (y * z + w * x);
    R.m[2][0] = 2.f * (x * z + w * y);
    R.m[2][1] = 2.f * (y * z - w * x);
    R.m[2][2] = 1.f - 2.f * (x * x + y * y);
    return R;
}

// Vector-Jacobian product of quat_rot given dL/dR (column-major), returned in the same
// (w,x,y,z)-in-(x,y,z,w) storage (reference auxiliary.h:225-271).
__device__ __forceinline__ float4 quat_rot_vjp(const float4 q, const Mat<3, 3>& g) {
    const float s = rsqrtf(q.w * q.w + q.x * q.x + q.y * q.y + q.z * q.z);
    const float w = q.x * s, x = q.y * s, y = q.z * s, z = q.w * s;
    float4 o;
    o.x = 2.f * (x * (g.m[1][2] - g.m[2][1]) + y * (g.m[2][0] - g.m[0][2]) + z * (g.m[0][1] - g.m[1][0]));
    o.y = 2.f * (-2.f * x * (g.m[1][1] + g.m[2][2]) + y * (g.m[0][1] + g.m[1][0]) + z * (g.m[0][2] + g.m[2][0]) +
                 w * (g.m[1][2] - g.m[2][1]));
    o.z = 2.f * (x * (g.m[0][1] + g.m[1][0]) - 2.f * y * (g.m[0][0] + g.m[2][2]) + z * (g.m[1][2] + g.m[2][1]) +
                 w * (g.m[2][0] - g.m[0][2]));
    o.w = 2.f * (x * (g.m[0][2] + g.m[2][0]) + y * (g.m[1][2] + g.m[2][1]) - 2.f * z * (g.m[0][0] + g.m[1][1]) +
                 w * (g.m[0][1] - g.m[1][0]));
    return o;
}

__device__ __forceinline__ Mat<3, 3> scale_mat(float sx, float sy, float mod) {
    Mat<3, 3> S;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < 3; ++r) S.m[c][r] = (c == r) ? 1.f : 0.f;
    S.m[0][0] = mod * sx;
    S.m[1][1] = mod * sy;
    return S;
}

// world -> NDC as a column-major 4x4 from the row-major projection array.
__device__ __forceinline__ Mat<4, 4> world2ndc(const float* pm) {
    Mat<4, 4> w;
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int r = 0; r < 4; ++r) w.m[c][r] = pm[4 * r + c];
    return w;
}

__device__ __forceinline__ Mat<3, 4> ndc2pix(int W, int H) {
    Mat<3, 4> n;
    n.m[0][0] = (float)((double)W / 2.0); n.m[0][1] = 0.f; n.m[0][2] = 0.f; n.m[0][3] = (float)((double)(W - 1) / 2.0);
    n.m[1][0] = 0.f; n.m[1][1] = (float)((double)H / 2.0); n.m[1][2] = 0.f; n.m[1][3] = (float)((double)(H - 1) / 2.0);
    n.m[2][0] = 0.f; n.m[2][1] = 0.f; n.m[2][2] = 0.f; n.m[2][3] = 1.f;
    return n;
}

__device__ __forceinline__ Mat<3, 4> splat2world(const Mat<3, 3>& L, const float3 p) {
    Mat<3, 4> s;
    s.m[0][0] = L.m[0][0]; s.m[0][1] = L.m[0][1]; s.m[0][2] = L.m[0][2]; s.m[0][3] = 0.f;
    s.m[1][0] = L.m[1][0]; s.m[1][1] = L.m[1][1]; s.m[1][2] = L.m[1][2]; s.m[1][3] = 0.f;
    s.m[2][0] = p.x; s.m[2][1] = p.y; s.m[2][2] = p.z; s.m[2][3] = 1.f;
    return s;
}

__device__ __forceinline__ float3 xform_point(const float3 p, const float* m) {
    return make_float3(m[0] * p.x + m[4] * p.y + m[8] * p.z + m[12], m[1] * p.x + m[5] * p.y + m[9] * p.z + m[13],
                       m[2] * p.x + m[6] * p.y + m[10] * p.z + m[14]);
}
__device__ __forceinline__ V3 xform_vec(const V3 p, const float* m) {
    return v3(m[0] * p.x + m[4] * p.y + m[8] * p.z, m[1] * p.x + m[5] * p.y + m[9] * p.z,
              m[2] * p.x + m[6] * p.y + m[10] * p.z);
}
__device__ __forceinline__ V3 xform_vec_t(const V3 p, const float* m) {
    return v3(m[0] * p.x + m[1] * p.y + m[2] * p.z, m[4] * p.x + m[5] * p.y + m[6] * p.z,
              m[8] * p.x + m[9] * p.y + m[10] * p.z);
}

// SH colour with the reference's degree-2 "ultrasound" terms (forward.cu:20-65).
// Returns the clamp flags as bits 0..2.
__device__ __forceinline__ int sh_color(int g, int deg, int M, const float* means, const float* campos,
                                        const float* shs, float* rgb) {
    const V3 pos = v3(means[3 * g], means[3 * g + 1], means[3 * g + 2]);
    V3 dir = vsub(pos, v3(campos[0], campos[1], campos[2]));
    const float len = sqrtf(vdot(dir, dir));
    dir = v3(dir.x / len, dir.y / len, dir.z / len);
    const float* sh = shs + (int64_t)g * M * 3;
    auto c = [&](int k) { return v3(sh[3 * k], sh[3 * k + 1], sh[3 * k + 2]); };
    V3 res = vscale(SH_C0, c(0));
    if (deg > 0) {
        const float x = dir.x, y = dir.y, z = dir.z;
        res = vsub(vadd(vsub(res, vscale(SH_C1 * y, c(1))), vscale(SH_C1 * z, c(2))), vscale(SH_C1 * x, c(3)));
        if (deg > 1) {
            const float depth = x;
            const float refl_var = x * x + y * y + z * z;
            const float sc_x = x * y, sc_y = z * y, sc_z = x * z;
            const float att = __expf(-depth);
            const float refl = -refl_var;
            res = vsub(vadd(vsub(vadd(vsub(res, vscale(att, c(4))), vscale(refl, c(5))), vscale(sc_z, c(6))),
                            vscale(sc_x, c(7))),
                       vscale(sc_y, c(8)));
        }
    }
    res = v3(res.x + 0.5f, res.y + 0.5f, res.z + 0.5f);
    const int clamped = (res.x < 0) | ((res.y < 0) << 1) | ((res.z < 0) << 2);
    rgb[0] = fmaxf(res.x, 0.0f);
    rgb[1] = fmaxf(res.y, 0.0f);
    rgb[2] = fmaxf(res.z, 0.0f);
    return clamped;
}

struct Workspace {
    long long* header;
    float4* rec;           // G x 5; the last two floats hold the reach box
    float* depth;          // G (view depth, key bits)
    int4* rect;            // G tile rectangle [x0, y0, x1, y1)
    int* clamped;          // G (bits 0..2)
    int* touched;          // G
    int* inst_offset;      // G + 1
    long long* bs_g;
    int* tile_count;       // T
    int* tile_start;       // T + 1
    int* tile_cursor;      // T
    long long* bs_t;
    StableScratch stable;    // small bucket grids (stable_bins)
    unsigned long long* keys;  // the other ones: instances before the sort
    int* slot_inst;
    int* sorted_gid;
    int* sorted_inst;
    float* accum;          // 3P: final T, M1, M2
    uint32_t* n_contrib;   // 2P: last contributor, median contributor
    size_t bytes;
};

static Workspace carve(void* base, int64_t G, int64_t T, int64_t P, int64_t cap) {
    Carver c(base);
    Workspace w;
    w.header = c.take<long long>(H_WORDS);
    w.rec = c.take<float4>((size_t)G * REC_F4);
    w.depth = c.take<float>((size_t)G);
    w.rect = c.take<int4>((size_t)G);
    w.clamped = c.take<int>((size_t)G);
    w.touched = c.take<int>((size_t)G);
    w.inst_offset = c.take<int>((size_t)G + 1);
    w.bs_g = c.take<long long>((size_t)scan_num_blocks(G) + 1);
    w.tile_count = c.take<int>((size_t)T);
    w.tile_start = c.take<int>((size_t)T + 1);
    w.tile_cursor = c.take<int>((size_t)T);
    w.bs_t = c.take<long long>((size_t)scan_num_blocks(T) + 1);
    if (stable_bins(G, T, true)) {
        w.stable = stable_carve(c, G, T, true);
        w.keys = nullptr;
        w.slot_inst = nullptr;
    } else {
        w.stable = {};
        w.keys = c.take<unsigned long long>((size_t)cap);
        w.slot_inst = c.take<int>((size_t)cap);
    }
    w.sorted_gid = c.take<int>((size_t)cap);
    w.sorted_inst = c.take<int>((size_t)cap);
    w.accum = c.take<float>((size_t)P * 3);
    w.n_contrib = c.take<uint32_t>((size_t)P * 2);
    w.bytes = align_up(c.off, 256);
    return w;
}

struct Params {
    int P, D, M, W, H, gx, gy;
    float scale_modifier;
    int prefiltered;
    const float* means;
    const float* shs;
    const float* colors;
    const float* opacities;
    const float* scales;
    const float* rotations;
    const float* transmat;
    const float* view;
    const float* proj;
    const float* campos;
};

// ------------------------------------------------------------------------------------
// Preprocess + binning
// ------------------------------------------------------------------------------------

__global__ void init_kernel(int64_t T, int* __restrict__ tile_count, int* __restrict__ tile_cursor,
                            long long* __restrict__ header, int64_t cap, int64_t G, int64_t P) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0 && threadIdx.x < H_WORDS) {
        long long v = 0;
        if (threadIdx.x == H_CAP) v = cap;
        if (threadIdx.x == H_G) v = G;
        if (threadIdx.x == H_T) v = T;
        if (threadIdx.x == H_P) v = P;
        header[threadIdx.x] = v;
    }
    if (t >= T) return;
    tile_count[t] = 0;
    tile_cursor[t] = 0;
}

// Pixel columns [x0, x1] and rows [y0, y1] that hold every pixel whose alpha with this surfel can
// reach 1/255, as four 16-bit numbers: the box of {rho3d <= c} (the screen box of forward.cu:109-139
// with the cutoff c = 2 ln(255 opacity) in the place of 9) together with the filter's disc
// {rho2d <= c}, in double precision and half a pixel wider than that, which covers the float
// rounding of the per-pixel test (about 1e-3 pixel). Everything when the box is unbounded (the
// splat's plane passes the camera) or not finite; nothing when the opacity is below 1/255. An end that
// does not fit 16 bits stands for all pixels beyond (see reaches).
__device__ __forceinline__ uint2 reach_box(const V3 T0, const V3 T1, const V3 T2, float px, float py, float opacity) {
    const uint2 all = make_uint2(0x7fff8000u, 0x7fff8000u);  // low half: first, high half: last
    if (opacity * 255.0f < 0.999f) return make_uint2(0x80007fffu, 0x80007fffu);
    const double c = 2.0 * (double)logf(255.0f * opacity) * 1.0001 + 1e-3;
    const double x0 = T0.x, x1 = T0.y, x2 = T0.z, y0 = T1.x, y1 = T1.y, y2 = T1.z, w0 = T2.x, w1 = T2.y, w2 = T2.z;
    const double d = c * (w0 * w0 + w1 * w1) - w2 * w2;
    if (!(d < -1e-6 * w2 * w2)) return all;
    const double id = 1.0 / d;
    const double ux = (c * (x0 * w0 + x1 * w1) - x2 * w2) * id, uy = (c * (y0 * w0 + y1 * w1) - y2 * w2) * id;
    const double hx = sqrt(fmax(0.0, ux * ux - (c * (x0 * x0 + x1 * x1) - x2 * x2) * id));
    const double hy = sqrt(fmax(0.0, uy * uy - (c * (y0 * y0 + y1 * y1) - y2 * y2) * id));
    const double r = sqrt(c / FILTER_INV_SQUARE);
    const double a = floor(fmin(ux - hx, px - r) - 0.5), b = ceil(fmax(ux + hx, px + r) + 0.5);
    const double e = floor(fmin(uy - hy, py - r) - 0.5), f = ceil(fmax(uy + hy, py + r) + 0.5);
    if (!(a <= b) || !(e <= f)) return all;  // not finite
    auto half = [](double v) { return (unsigned)(int)fmin(fmax(v, -32768.0), 32767.0) & 0xffffu; };
    return make_uint2(half(a) | (half(b) << 16), half(e) | (half(f) << 16));
}

// Whether a reach box meets columns [bx, bx + w) and rows [by, by + h). A last column or row of 32,767 is not
// an end: frames may be wider, and such a box goes on.
__device__ __forceinline__ bool reaches(unsigned xr, unsigned yr, int bx, int by, int w, int h) {
    return (int)(short)(xr & 0xffffu) < bx + w && (int)(short)(xr >> 16) >= min(bx, 0x7fff) &&
           (int)(short)(yr & 0xffffu) < by + h && (int)(short)(yr >> 16) >= min(by, 0x7fff);
}

// Per Gaussian: near cull, homography, dual-visible normal, AABB radius, tile rectangle,
// colour, render record, per-tile counts (forward.cu:141-246).
__global__ void __launch_bounds__(256)
preprocess_kernel(Params p, int* __restrict__ radii, float4* __restrict__ rec, float* __restrict__ depth_out,
                  int4* __restrict__ rect_out, int* __restrict__ clamped_out, int* __restrict__ touched,
                  int* __restrict__ tile_count, long long* __restrict__ header) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= p.P) return;
    radii[g] = 0;
    touched[g] = 0;
    clamped_out[g] = 0;
    depth_out[g] = 0.f;
    rect_out[g] = make_int4(0, 0, 0, 0);
    const float3 po = make_float3(p.means[3 * g], p.means[3 * g + 1], p.means[3 * g + 2]);
    const float3 pv = xform_point(po, p.view);
    if (pv.z <= 0.2f) {
        if (p.prefiltered) atomicOr(reinterpret_cast<unsigned long long*>(header + H_FLAGS), (unsigned long long)FLAG_PREFILTERED);
        return;
    }
    Mat<3, 3> T;
    V3 normal;
    if (p.transmat == nullptr) {
        const float4 q = make_float4(p.rotations[4 * g], p.rotations[4 * g + 1], p.rotations[4 * g + 2],
                                     p.rotations[4 * g + 3]);
        const Mat<3, 3> R = quat_rot(q);
        const Mat<3, 3> S = scale_mat(p.scales[2 * g], p.scales[2 * g + 1], p.scale_modifier);
        const Mat<3, 3> L = mmul(R, S);
        const Mat<4, 3> A = mmul(transpose(splat2world(L, po)), world2ndc(p.proj));
        T = mmul(A, ndc2pix(p.W, p.H));
        normal = xform_vec(col3(L, 2), p.view);
    } else {
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int r = 0; r < 3; ++r) T.m[c][r] = p.transmat[9 * g + 3 * c + r];
        normal = v3(0.f, 0.f, 1.f);
    }
    // dual-visible: orient the normal towards the camera
    const float cosv = -(pv.x * normal.x + pv.y * normal.y + pv.z * normal.z);
    if (cosv == 0) return;
    const float mult = cosv > 0 ? 1.f : -1.f;
    normal = vscale(mult, normal);
    // AABB of the cutoff ellipse (forward.cu:109-139), cutoff 3
    const float cutoff = 3.0f;
    const V3 t = v3(cutoff * cutoff, cutoff * cutoff, -1.0f);
    const V3 T0 = col3(T, 0), T1 = col3(T, 1), T2 = col3(T, 2);
    const float d = vdot(t, vmul(T2, T2));
    if (d == 0.0f) return;
    const V3 f = vscale(1.0f / d, t);
    const float px = vdot(f, vmul(T0, T2)), py = vdot(f, vmul(T1, T2));
    const float h0x = px * px - vdot(f, vmul(T0, T0));
    const float h0y = py * py - vdot(f, vmul(T1, T1));
    const float hx = sqrtf((1e-4f < h0x) ? h0x : 1e-4f);
    const float hy = sqrtf((1e-4f < h0y) ? h0y : 1e-4f);
    const float radius = ceilf(fmaxf(fmaxf(hx, hy), cutoff * FILTER_SIZE));
    const int r = (int)radius;
    const int x0 = min(p.gx, max(0, (int)((px - (float)r) / (float)TILE)));
    const int y0 = min(p.gy, max(0, (int)((py - (float)r) / (float)TILE)));
    const int x1 = min(p.gx, max(0, (int)((((px + (float)r) + (float)TILE) - 1.0f) / (float)TILE)));
    const int y1 = min(p.gy, max(0, (int)((((py + (float)r) + (float)TILE) - 1.0f) / (float)TILE)));
    if ((x1 - x0) * (y1 - y0) == 0) return;
    float rgb[3];
    int clamped = 0;
    if (p.colors == nullptr) {
        clamped = sh_color(g, p.D, p.M, p.means, p.campos, p.shs, rgb);
    } else {
        rgb[0] = p.colors[3 * g];
        rgb[1] = p.colors[3 * g + 1];
        rgb[2] = p.colors[3 * g + 2];
    }
    clamped_out[g] = clamped;
    depth_out[g] = pv.z;
    radii[g] = r;
    float4* o = rec + (int64_t)REC_F4 * g;
    o[0] = make_float4(T0.x, T0.y, T0.z, px);
    o[1] = make_float4(T1.x, T1.y, T1.z, py);
    o[2] = make_float4(T2.x, T2.y, T2.z, p.opacities[g]);
    o[3] = make_float4(normal.x, normal.y, normal.z, rgb[0]);
    const uint2 box = reach_box(T0, T1, T2, px, py, p.opacities[g]);
    o[4] = make_float4(rgb[1], rgb[2], __uint_as_float(box.x), __uint_as_float(box.y));
    rect_out[g] = make_int4(x0, y0, x1, y1);
    touched[g] = (x1 - x0) * (y1 - y0);
    (void)tile_count;  // counted per block by rect_count_kernel
}

// ------------------------------------------------------------------------------------
// Forward compositing
// ------------------------------------------------------------------------------------

// Ray-splat intersection of pixel (pxf, pyf) with the splat of homography rows Tu, Tv, Tw
// (forward.cu:335-350). Returns false when the pair is skipped before alpha.
struct Hit {
    V3 k, l, p;
    float sx, sy, rho3d, rho2d, dx, dy, depth;
};

__device__ __forceinline__ bool intersect(float pxf, float pyf, const float4 r0, const float4 r1, const float4 r2,
                                          Hit& h) {
    const V3 Tu = v3(r0.x, r0.y, r0.z), Tv = v3(r1.x, r1.y, r1.z), Tw = v3(r2.x, r2.y, r2.z);
    h.k = vsub(vscale(pxf, Tw), Tu);
    h.l = vsub(vscale(pyf, Tw), Tv);
    h.p = vcross(h.k, h.l);
    if (h.p.z == 0.0f) return false;
    h.sx = h.p.x / h.p.z;
    h.sy = h.p.y / h.p.z;
    h.rho3d = h.sx * h.sx + h.sy * h.sy;
    h.dx = r0.w - pxf;
    h.dy = r1.w - pyf;
    h.rho2d = FILTER_INV_SQUARE * (h.dx * h.dx + h.dy * h.dy);
    h.depth = (h.sx * Tw.x + h.sy * Tw.y) + Tw.z;
    return !(h.depth < NEAR_N);
}

// Asynchronous global -> shared copies (cp.async, sm_80 and later): the next batch of render
// records is gathered into the second staging buffer while the current one is shaded.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// A warp shades a block of 8 columns x 4 rows (warp w: column block w & 1, row block w >> 1).
constexpr int BLK_W = 8, BLK_H = 4;
__device__ __forceinline__ int block_x(int t) { return ((t >> 5) & 1) * BLK_W + (t & (BLK_W - 1)); }
__device__ __forceinline__ int block_y(int t) { return (t >> 6) * BLK_H + ((t & 31) >> 3); }

// One CTA per tile, one pixel per thread, the warps independent of one another: of every 32 surfels of the tile's
// list a warp keeps, by ballot and in order, those whose reach box meets its 8x4 pixels, copies their
// records into its own staging buffer while it composites the ones before, and stops when its pixels are
// done. The others fail the alpha test on all its pixels (decisions and sums are those of the whole list, and
// a contributor's number is its place in the tile's list). The intersections of two kept surfels are
// evaluated together. What bounds the kernel is the dependent chain of the longest list (a
// clustered scene of 200k surfels at 256x256: 1.053 ms with one list for the tile, 0.452 ms with lists per
// warp of batches staged by the whole CTA, whose warps then spent half their stall cycles waiting
// for one another at its barriers (SMs 345k cycles busy on average, 895k at most); 0.294 ms so).
__global__ void __launch_bounds__(BLOCK)
forward_kernel(int W, int H, int gx, const int* __restrict__ tile_start, const int* __restrict__ sorted_gid,
               const long long* __restrict__ header, const float4* __restrict__ rec, const float* __restrict__ bg,
               float* __restrict__ out_color, float* __restrict__ out_others, float* __restrict__ accum,
               uint32_t* __restrict__ n_contrib) {
    __shared__ float4 s_rec[BLOCK / 32][2][REC_F4][32];  // per warp: double-buffered staging
    __shared__ unsigned char s_list[BLOCK / 32][2][32];  // their places among the 32
    if (header[H_FLAGS] != 0) return;
    const int tile = blockIdx.x;
    const int tx = tile % gx, ty = tile / gx;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bx = tx * TILE + (warp & 1) * BLK_W, by = ty * TILE + (warp >> 1) * BLK_H;
    const uint32_t pxi = (uint32_t)(tx * TILE + block_x(threadIdx.x)), pyi = (uint32_t)(ty * TILE + block_y(threadIdx.x));
    const bool inside = pxi < (uint32_t)W && pyi < (uint32_t)H;
    const float pxf = (float)pxi, pyf = (float)pyi;
    bool done = !inside;
    const int s0 = tile_start[tile], n = tile_start[tile + 1] - s0;
    float T = 1.0f;
    uint32_t last_contributor = 0;
    float C[3] = {0.f, 0.f, 0.f};
    float N[3] = {0.f, 0.f, 0.f};
    float D = 0.f, M1 = 0.f, M2 = 0.f, distortion = 0.f, median_depth = 0.f, median_contributor = -1.f;
    const float mscale = FAR_N / (FAR_N - NEAR_N);
    const unsigned FULL = 0xffffffffu;
    auto load_gid = [&](int c) {
        const int k = 32 * c + lane;
        return k < n ? sorted_gid[s0 + k] : -1;
    };
    auto load_box = [&](int gid) {
        return gid >= 0 ? reinterpret_cast<const uint2*>(rec + (int64_t)REC_F4 * gid + 4)[1] : make_uint2(0u, 0u);
    };
    // the kept ones of 32 surfels into buffer b; returns their number
    auto stage = [&](int gid, uint2 box, int b) {
        const bool mine = gid >= 0 && reaches(box.x, box.y, bx, by, BLK_W, BLK_H);
        const unsigned bits = __ballot_sync(FULL, mine);
        if (mine) {
            const int at = __popc(bits & ((1u << lane) - 1u));
            const float4* r = rec + (int64_t)REC_F4 * gid;
#pragma unroll
            for (int f = 0; f < REC_F4; ++f) cp_async16(&s_rec[warp][b][f][at], r + f);
            s_list[warp][b][at] = (unsigned char)lane;
        }
        cp_async_commit();
        return __popc(bits);
    };
    // chunk c is composited while the records of chunk c + 1 are copied, the boxes of chunk c + 2 and the
    // indices of chunk c + 3 are read
    const int chunks = __all_sync(FULL, done) ? 0 : (n + 31) / 32;
    int g1 = load_gid(0), g2 = load_gid(1), g3 = load_gid(2);
    uint2 b1 = load_box(g1), b2 = load_box(g2);
    int nl_next = stage(g1, b1, 0);
    for (int c = 0; c < chunks; ++c) {
        const int nl = nl_next;
        nl_next = stage(g2, b2, (c + 1) & 1);
        g2 = g3;
        b2 = load_box(g3);
        g3 = load_gid(c + 3);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // this lane's copies of chunk c have landed
        __syncwarp();                                           // ... and every lane's
        const float4(*sr)[32] = s_rec[warp][c & 1];
        const unsigned char* list = s_list[warp][c & 1];
        // alpha of surfel j at this pixel, 0 when the pair is skipped
        auto alpha_of = [&](int j, float& depth) {
            const float4 r2 = sr[2][j];
            Hit h = {};
            const bool ok = intersect(pxf, pyf, sr[0][j], sr[1][j], r2, h);
            const float power = -0.5f * fminf(h.rho3d, h.rho2d);
            const float alpha = fminf(0.99f, r2.w * __expf(power));
            depth = h.depth;
            return ok && !(power > 0.0f) && !(alpha < 1.0f / 255.0f) ? alpha : 0.0f;
        };
        auto composite = [&](int j, float alpha, float depth) {
            if (alpha == 0.0f || done) return;
            const float test_T = T * (1 - alpha);
            if (test_T < 0.0001f) {
                done = true;
                return;
            }
            const float w = alpha * T;
            const float A = 1 - T;
            const float m = mscale * (1 - NEAR_N / depth);
            distortion += (m * m * A + M2 - 2 * m * M1) * w;
            D += depth * w;
            M1 += m * w;
            M2 += m * m * w;
            last_contributor = (uint32_t)(32 * c + list[j] + 1);
            if (T > 0.5) {
                median_depth = depth;
                median_contributor = (float)last_contributor;
            }
            const float4 r3 = sr[3][j];
            const float2 r4 = *reinterpret_cast<const float2*>(&sr[4][j]);
            N[0] += r3.x * w;
            N[1] += r3.y * w;
            N[2] += r3.z * w;
            C[0] += r3.w * w;
            C[1] += r4.x * w;
            C[2] += r4.y * w;
            T = test_T;
        };
        int e = 0;
        for (; e + 2 <= nl; e += 2) {
            float da, db;
            const float aa = alpha_of(e, da), ab = alpha_of(e + 1, db);
            composite(e, aa, da);
            composite(e + 1, ab, db);
        }
        if (e < nl) {
            float da;
            const float aa = alpha_of(e, da);
            composite(e, aa, da);
        }
        if (__all_sync(FULL, done)) break;  // (also: every lane has left buffer c & 1)
    }
    cp_async_wait_all();
    if (inside) {
        const int64_t HW = (int64_t)H * W;
        const int64_t pix = (int64_t)W * pyi + pxi;
        accum[pix] = T;
        accum[pix + HW] = M1;
        accum[pix + 2 * HW] = M2;
        n_contrib[pix] = last_contributor;
        n_contrib[pix + HW] = f32_to_u32_sat(median_contributor);
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) out_color[ch * HW + pix] = C[ch] + T * bg[ch];
        out_others[pix] = D;
        out_others[pix + HW] = 1 - T;
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) out_others[pix + (2 + ch) * HW] = N[ch];
        out_others[pix + 5 * HW] = median_depth;
        out_others[pix + 6 * HW] = distortion;
    }
}

// ------------------------------------------------------------------------------------
// Backward
// ------------------------------------------------------------------------------------

// Sums of va[0..17] and vb[0..17] over the 32 lanes of a warp, transposed: the first exchange gives
// lanes 0-15 the terms of a and lanes 16-31 those of b, the next ones halve the terms that a lane
// carries, 37 shuffles for both (27 for each alone). On return a lane holds the totals of
// terms [base, base + count) of its instance in o[0..1], see PairSlot.
__device__ __forceinline__ void warp_reduce_pair(const float (&va)[NGRAD], const float (&vb)[NGRAD], float (&o)[2]) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4, h2 = lane & 2, h1 = lane & 1;
    float x[18], y[10], z[6], w[4];
#pragma unroll
    for (int i = 0; i < 18; ++i) x[i] = (h16 ? vb[i] : va[i]) + __shfl_xor_sync(FULL, h16 ? va[i] : vb[i], 16);
#pragma unroll
    for (int i = 0; i < 9; ++i) y[i] = (h8 ? x[9 + i] : x[i]) + __shfl_xor_sync(FULL, h8 ? x[i] : x[9 + i], 8);
    y[9] = 0.f;
#pragma unroll
    for (int i = 0; i < 5; ++i) z[i] = (h4 ? y[5 + i] : y[i]) + __shfl_xor_sync(FULL, h4 ? y[i] : y[5 + i], 4);
    z[5] = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) w[i] = (h2 ? z[3 + i] : z[i]) + __shfl_xor_sync(FULL, h2 ? z[i] : z[3 + i], 2);
    w[3] = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) o[i] = (h1 ? w[2 + i] : w[i]) + __shfl_xor_sync(FULL, h1 ? w[i] : w[2 + i], 1);
}

// The terms that a lane holds after warp_reduce_pair.
struct PairSlot {
    int base, count;
};
__device__ __forceinline__ PairSlot pair_slot(int lane) {
    const int n8 = 9, n4 = (lane & 4) ? 4 : 5;
    const int n2 = (lane & 2) ? max(n4 - 3, 0) : min(n4, 3);
    const int n1 = (lane & 1) ? max(n2 - 2, 0) : min(n2, 2);
    return PairSlot{((lane & 8) ? n8 : 0) + ((lane & 4) ? 5 : 0) + ((lane & 2) ? 3 : 0) + ((lane & 1) ? 2 : 0), n1};
}

// One CTA per tile, one pixel per thread, Gaussians replayed back to front
// (backward.cu:103-404). As in the forward, a warp holds 8x4 pixels and replays only the surfels whose
// reach box meets them, two at a time: their intersections are independent, and their gradient terms
// share one transposed warp reduction. Per staged Gaussian the sums of the warps that replayed it are
// added in warp order into the instance's 18-term partial:
//   [0..2] dL/dTu  [3..5] dL/dTv  [6..8] dL/dTw  [9..10] dL/dmean2D  [11..13] dL/dnormal
//   [14] dL/dopacity  [15..17] dL/dcolor
// Bound by the replay chain of the longest tile list: on 200k clustered surfels at 256x256, 1.732 -> 0.924 ms.
__global__ void __launch_bounds__(BLOCK)
backward_kernel(int W, int H, int gx, const int* __restrict__ tile_start, const int* __restrict__ sorted_gid,
                const int* __restrict__ sorted_inst, const long long* __restrict__ header,
                const float4* __restrict__ rec, const float* __restrict__ bg, const float* __restrict__ accum,
                const uint32_t* __restrict__ n_contrib, const float* __restrict__ dL_dpix,
                const float* __restrict__ dL_dothers, float4* __restrict__ partial) {
    __shared__ float4 s_rec[2][REC_F4][BWD_BATCH];  // double-buffered staging
    __shared__ int s_inst[2][BWD_BATCH];
    __shared__ float s_red[BWD_BATCH][BLOCK / 32][NGRAD];
    __shared__ unsigned s_who[BWD_BATCH];  // warps that wrote their sums
    __shared__ unsigned char s_list[BLOCK / 32][BWD_BATCH];
    __shared__ int s_last;
    if (header[H_FLAGS] != 0) return;
    const int tile = blockIdx.x;
    const int tx = tile % gx, ty = tile / gx;
    const uint32_t pxi = (uint32_t)(tx * TILE + block_x(threadIdx.x)), pyi = (uint32_t)(ty * TILE + block_y(threadIdx.x));
    const bool inside = pxi < (uint32_t)W && pyi < (uint32_t)H;
    const float pxf = (float)pxi, pyf = (float)pyi;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bx = tx * TILE + (warp & 1) * BLK_W, by = ty * TILE + (warp >> 1) * BLK_H;
    const PairSlot slot = pair_slot(lane);
    const int s0 = tile_start[tile], n = tile_start[tile + 1] - s0;
    const int64_t HW = (int64_t)H * W;
    const int64_t pix = (int64_t)W * pyi + pxi;

    const float T_final = inside ? accum[pix] : 0.f;
    float T = T_final;
    const int last_contributor = inside ? (int)n_contrib[pix] : 0;
    // No pixel of the tile has a contributor at or beyond the largest last contributor: the
    // back-to-front replay starts there (its state changes only at contributors), and the
    // instances behind it get zero partials.
    if (threadIdx.x == 0) s_last = 0;
    __syncthreads();
    if (last_contributor > 0) atomicMax(&s_last, last_contributor);
    __syncthreads();
    const int n_live = min(s_last, n);
    const int warp_last = __reduce_max_sync(0xffffffffu, last_contributor);
    for (int k = n_live + threadIdx.x; k < n; k += BLOCK) {
        float4* out = partial + (int64_t)PARTIAL_F4 * sorted_inst[s0 + k];
#pragma unroll
        for (int f = 0; f < PARTIAL_F4; ++f) out[f] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int median_contributor = inside ? (int)n_contrib[pix + HW] : 0;
    float dpix[3] = {0.f, 0.f, 0.f};
    float dd_depth = 0.f, dd_accum = 0.f, dd_reg = 0.f, dd_median = 0.f;
    float dd_normal[3] = {0.f, 0.f, 0.f};
    if (inside) {
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) dpix[ch] = dL_dpix[ch * HW + pix];
        dd_depth = dL_dothers[pix];
        dd_accum = dL_dothers[pix + HW];
        dd_reg = dL_dothers[pix + 6 * HW];
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) dd_normal[ch] = dL_dothers[pix + (2 + ch) * HW];
        dd_median = dL_dothers[pix + 5 * HW];
    }
    const float final_D = inside ? accum[pix + HW] : 0.f;
    const float final_D2 = inside ? accum[pix + 2 * HW] : 0.f;
    const float final_A = 1 - T_final;
    float accum_rec[3] = {0.f, 0.f, 0.f}, last_color[3] = {0.f, 0.f, 0.f};
    float last_depth = 0.f, accum_depth_rec = 0.f, accum_alpha_rec = 0.f;
    float last_normal[3] = {0.f, 0.f, 0.f}, accum_normal_rec[3] = {0.f, 0.f, 0.f};
    float last_dL_dT = 0.f, last_alpha = 0.f;
    const float bg_dot_dpixel = bg[0] * dpix[0] + bg[1] * dpix[1] + bg[2] * dpix[2];
    const float mscale = FAR_N / (FAR_N - NEAR_N);

    // batch k (staged from the back of the tile list's live part) goes to buffer k & 1: thread
    // jj < BWD_BATCH copies Gaussian jj's record and instance id. The copies of batch k + 1 are
    // issued after batch k's first barrier (every thread is then done with that buffer's
    // previous batch) and run while batch k is replayed; the Gaussian index each copy needs is
    // read one batch earlier still, so no thread waits on it.
    static_assert(BWD_BATCH <= BLOCK, "one staging thread per batch entry");
    auto load_gid = [&](int b0) {
        const int jj = threadIdx.x;
        return (jj < BWD_BATCH && b0 + jj < n_live) ? sorted_gid[s0 + n_live - 1 - (b0 + jj)] : -1;
    };
    auto stage = [&](int b0, int buf, int gid) {
        const int jj = threadIdx.x;
        if (gid >= 0) {
            const float4* r = rec + (int64_t)REC_F4 * gid;
#pragma unroll
            for (int f = 0; f < REC_F4; ++f) cp_async16(&s_rec[buf][f][jj], r + f);
            cp_async4(&s_inst[buf][jj], sorted_inst + (s0 + n_live - 1 - (b0 + jj)));
        }
        cp_async_commit();
    };
    int gid_next = 0;
    if (n_live > 0) {
        stage(0, 0, load_gid(0));
        gid_next = load_gid(BWD_BATCH);
    }
    for (int b0 = 0, k = 0; b0 < n_live; b0 += BWD_BATCH, ++k) {
        const int nb = min(BWD_BATCH, n_live - b0);
        cp_async_wait_all();  // this thread's copies of batch k have landed
        __syncthreads();      // ... and everyone's; the previous batch's partials are written
        if (b0 + BWD_BATCH < n_live) {
            stage(b0 + BWD_BATCH, (k + 1) & 1, gid_next);
            gid_next = load_gid(b0 + 2 * BWD_BATCH);
        }
        const float4(*sr)[BWD_BATCH] = s_rec[k & 1];
        const int* si = s_inst[k & 1];
        if (threadIdx.x < BWD_BATCH) s_who[threadIdx.x] = 0u;
        __syncthreads();
        int nl = 0;
#pragma unroll
        for (int jc = 0; jc < BWD_BATCH; jc += 32) {
            const int jl = jc + lane;
            // entry jl is contributor n_live - b0 - jl (counted from one): none of the warp's pixels
            // has a contributor beyond warp_last
            const bool mine = jl < nb && n_live - b0 - jl <= warp_last &&
                              reaches(__float_as_uint(sr[4][jl].z), __float_as_uint(sr[4][jl].w), bx, by, BLK_W, BLK_H);
            const unsigned bits = __ballot_sync(0xffffffffu, mine);
            if (mine) s_list[warp][nl + __popc(bits & ((1u << lane) - 1u))] = (unsigned char)jl;
            nl += __popc(bits);
        }
        __syncwarp();
        // the pair (this pixel, entry jj): whether it contributes, and its weight
        auto evaluate = [&](int jj, Hit& h, float& G, float& alpha) {
            h = {};
            const float4 r2 = sr[2][jj];
            const bool hit = intersect(pxf, pyf, sr[0][jj], sr[1][jj], r2, h);
            const float power = -0.5f * fminf(h.rho3d, h.rho2d);
            G = __expf(power);
            alpha = fminf(0.99f, r2.w * G);
            return n_live - b0 - jj <= last_contributor && hit && !(power > 0.0f) && !(alpha < 1.0f / 255.0f);
        };
        // one step of the replay: the gradient terms of the pair
        auto replay = [&](int jj, const Hit& h, float G, float alpha, float (&v)[NGRAD]) {
            const float4 r2 = sr[2][jj], r3 = sr[3][jj];
            const float2 r4 = *reinterpret_cast<const float2*>(&sr[4][jj]);
            const float col[3] = {r3.w, r4.x, r4.y};
            const float nrm[3] = {r3.x, r3.y, r3.z};
            T = T / (1.f - alpha);
            const float wT = alpha * T;
            float dL_dalpha = 0.0f;
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                accum_rec[ch] = last_alpha * last_color[ch] + (1.f - last_alpha) * accum_rec[ch];
                last_color[ch] = col[ch];
                dL_dalpha += (col[ch] - accum_rec[ch]) * dpix[ch];
                v[15 + ch] = wT * dpix[ch];
            }
            float dL_dz = 0.0f;
            const float c_d = h.depth;
            const float m_d = mscale * (1 - NEAR_N / c_d);
            const float dmd_dd = (FAR_N * NEAR_N) / ((FAR_N - NEAR_N) * c_d * c_d);
            if (n_live - b0 - jj == median_contributor) dL_dz += dd_median;
            const float dL_dweight = (final_D2 + m_d * m_d * final_A - 2 * m_d * final_D) * dd_reg;
            dL_dalpha += dL_dweight - last_dL_dT;
            last_dL_dT = dL_dweight * alpha + (1 - alpha) * last_dL_dT;
            const float dL_dmd = 2.0f * (T * alpha) * (m_d * final_A - final_D) * dd_reg;
            dL_dz += dL_dmd * dmd_dd;
            accum_depth_rec = last_alpha * last_depth + (1.f - last_alpha) * accum_depth_rec;
            last_depth = c_d;
            dL_dalpha += (c_d - accum_depth_rec) * dd_depth;
            // the reference adds last_alpha * 1.0 in double precision
            accum_alpha_rec = (float)((double)last_alpha + (double)__fmul_rn(1.f - last_alpha, accum_alpha_rec));
            dL_dalpha += (1 - accum_alpha_rec) * dd_accum;
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                accum_normal_rec[ch] = last_alpha * last_normal[ch] + (1.f - last_alpha) * accum_normal_rec[ch];
                last_normal[ch] = nrm[ch];
                dL_dalpha += (nrm[ch] - accum_normal_rec[ch]) * dd_normal[ch];
                v[11 + ch] = alpha * T * dd_normal[ch];
            }
            dL_dalpha *= T;
            last_alpha = alpha;
            dL_dalpha += (-T_final / (1.f - alpha)) * bg_dot_dpixel;
            const float dL_dG = r2.w * dL_dalpha;
            dL_dz += alpha * T * dd_depth;
            if (h.rho3d <= h.rho2d) {
                const float dsx = dL_dG * -G * h.sx + dL_dz * r2.x;
                const float dsy = dL_dG * -G * h.sy + dL_dz * r2.y;
                const float dsx_pz = dsx / h.p.z, dsy_pz = dsy / h.p.z;
                const V3 dL_dp = v3(dsx_pz, dsy_pz, -(dsx_pz * h.sx + dsy_pz * h.sy));
                const V3 dL_dk = vcross(h.l, dL_dp);
                const V3 dL_dl = vcross(dL_dp, h.k);
                v[0] = -dL_dk.x; v[1] = -dL_dk.y; v[2] = -dL_dk.z;
                v[3] = -dL_dl.x; v[4] = -dL_dl.y; v[5] = -dL_dl.z;
                v[6] = pxf * dL_dk.x + pyf * dL_dl.x + dL_dz * h.sx;
                v[7] = pxf * dL_dk.y + pyf * dL_dl.y + dL_dz * h.sy;
                v[8] = pxf * dL_dk.z + pyf * dL_dl.z + dL_dz * 1.0f;
            } else {
                const float dG_ddelx = -G * FILTER_INV_SQUARE * h.dx;
                const float dG_ddely = -G * FILTER_INV_SQUARE * h.dy;
                v[9] = dL_dG * dG_ddelx;
                v[10] = dL_dG * dG_ddely;
                v[6] = h.sx * dL_dz;
                v[7] = h.sy * dL_dz;
                v[8] = dL_dz;
            }
            v[14] = G * dL_dalpha;
        };
        for (int e = 0; e < nl; e += 2) {
            const int ja = s_list[warp][e], jb = e + 1 < nl ? s_list[warp][e + 1] : -1;
            Hit ha, hb;
            float Ga, Gb, aa, ab;
            const bool ca = evaluate(ja, ha, Ga, aa);
            bool cb = evaluate(jb >= 0 ? jb : ja, hb, Gb, ab);
            cb = cb && jb >= 0;
            const bool wa = __any_sync(0xffffffffu, ca), wb = __any_sync(0xffffffffu, cb);
            if (!wa && !wb) continue;
            float va[NGRAD], vb[NGRAD];
#pragma unroll
            for (int q = 0; q < NGRAD; ++q) va[q] = vb[q] = 0.f;
            if (ca) replay(ja, ha, Ga, aa, va);
            if (cb) replay(jb, hb, Gb, ab, vb);
            float o[2];
            warp_reduce_pair(va, vb, o);
            const int jj = (lane & 16) ? jb : ja;
            if ((lane & 16) ? wb : wa) {
                if (slot.count > 0) s_red[jj][warp][slot.base] = o[0];
                if (slot.count > 1) s_red[jj][warp][slot.base + 1] = o[1];
                if ((lane & 15) == 0) atomicOr(&s_who[jj], 1u << warp);
            }
        }
        __syncthreads();
        // term q of entry jj: the sums of the warps that replayed it, in warp order
        for (int i = threadIdx.x; i < nb * 4 * PARTIAL_F4; i += BLOCK) {
            const int jj = i / (4 * PARTIAL_F4), q = i - jj * (4 * PARTIAL_F4);
            float a = 0.f;
            if (q < NGRAD)
                for (unsigned who = s_who[jj]; who != 0u; who &= who - 1u) a += s_red[jj][__ffs(who) - 1][q];
            reinterpret_cast<float*>(partial + (int64_t)PARTIAL_F4 * si[jj])[q] = a;
        }
    }
}

// d|v|/dv applied to dv (reference auxiliary.h:110-121).
__device__ __forceinline__ V3 dnormvdv(const V3 v, const V3 dv) {
    const float sum2 = v.x * v.x + v.y * v.y + v.z * v.z;
    const float invsum32 = 1.0f / sqrtf(sum2 * sum2 * sum2);
    return v3(((+sum2 - v.x * v.x) * dv.x - v.y * v.x * dv.y - v.z * v.x * dv.z) * invsum32,
              (-v.x * v.y * dv.x + (sum2 - v.y * v.y) * dv.y - v.z * v.y * dv.z) * invsum32,
              (-v.x * v.z * dv.x - v.y * v.z * dv.y + (sum2 - v.z * v.z) * dv.z) * invsum32);
}

// One thread per Gaussian: sum its instance partials in order, then the preprocess backward
// (backward.cu:406-602): mean2D -> homography, homography -> mean / scale / rotation, normal
// -> rotation, SH -> colour and mean, and the reference's screen-space mean gradient.
// Per-Gaussian sums of its instances' partials, in instance order, written over its first
// instance's partial: PARTIAL_F4 threads per Gaussian, thread f summing float4 column f, so that
// the threads of a Gaussian read each 80-byte partial together and many Gaussians' loads are in
// flight (the sums are the ones a thread summing all columns would form).
constexpr int REDUCE_THREADS = 32 * PARTIAL_F4;  // 32 Gaussians per block
__global__ void __launch_bounds__(REDUCE_THREADS)
reduce_partials_kernel(int64_t n_gauss, const int* __restrict__ radii, const int* __restrict__ inst_offset,
                       const long long* __restrict__ header, float4* __restrict__ partial) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t g = t / PARTIAL_F4;
    const int f = (int)(t % PARTIAL_F4);
    if (g >= n_gauss || radii[g] <= 0 || header[H_FLAGS] != 0) return;
    const int i0 = inst_offset[g], i1 = inst_offset[g + 1];
    if (i1 <= i0) return;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    int i = i0;
    for (; i + 4 <= i1; i += 4) {  // four instances' loads in flight
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = partial[(int64_t)PARTIAL_F4 * (i + u) + f];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            s.x += v[u].x;
            s.y += v[u].y;
            s.z += v[u].z;
            s.w += v[u].w;
        }
    }
    for (; i < i1; ++i) {
        const float4 v = partial[(int64_t)PARTIAL_F4 * i + f];
        s.x += v.x;
        s.y += v.y;
        s.z += v.z;
        s.w += v.w;
    }
    partial[(int64_t)PARTIAL_F4 * i0 + f] = s;
}

__global__ void __launch_bounds__(128)
reduce_preprocess_kernel(Params p, float focal_x, float focal_y, float tan_fovx, float tan_fovy,
                         const int* __restrict__ radii, const int* __restrict__ inst_offset,
                         const long long* __restrict__ header, const float4* __restrict__ partial,
                         const float4* __restrict__ rec, const int* __restrict__ clamped_bits,
                         float* __restrict__ d_mean2D, float* __restrict__ d_colors, float* __restrict__ d_opacity,
                         float* __restrict__ d_means3D, float* __restrict__ d_transmat, float* __restrict__ d_sh,
                         float* __restrict__ d_scales, float* __restrict__ d_rot) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= p.P) return;
    float s[20];
#pragma unroll
    for (int q = 0; q < 20; ++q) s[q] = 0.f;
    const bool vis = radii[g] > 0 && header[H_FLAGS] == 0;
    if (vis) {  // the instance sums reduce_partials_kernel left in the first instance's partial
        const int i0 = inst_offset[g];
        if (inst_offset[g + 1] > i0) {
            const float4* r = partial + (int64_t)PARTIAL_F4 * i0;
#pragma unroll
            for (int f = 0; f < PARTIAL_F4; ++f) {
                const float4 x = r[f];
                s[4 * f] = x.x;
                s[4 * f + 1] = x.y;
                s[4 * f + 2] = x.z;
                s[4 * f + 3] = x.w;
            }
        }
    }
    // defaults: everything zero, render sums passed through
    float dT[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) dT[q] = s[q];
    float dmean3[3] = {0.f, 0.f, 0.f};
    float dscale[2] = {0.f, 0.f};
    float4 drot = make_float4(0.f, 0.f, 0.f, 0.f);
    float m2x = 0.f, m2y = 0.f;
    const int M = p.M;
    if (p.shs != nullptr)
        for (int k = 0; k < M * 3; ++k) d_sh[(int64_t)g * M * 3 + k] = 0.f;
    float dcol[3] = {s[15], s[16], s[17]};
    if (vis) {
        const int Wb = (int)(focal_x * tan_fovx * 2);
        const int Hb = (int)(focal_y * tan_fovy * 2);
        const bool precomp = (p.scales == nullptr);
        const float3 po = make_float3(p.means[3 * g], p.means[3 * g + 1], p.means[3 * g + 2]);
        Mat<3, 3> T, R, Lm;
        Mat<3, 4> Pm;
        V3 normal;
        float4 rot = make_float4(0.f, 0.f, 0.f, 0.f);
        float scx = 0.f, scy = 0.f;
        if (precomp) {
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int r = 0; r < 3; ++r) T.m[c][r] = p.transmat[9 * g + 3 * c + r];
            normal = v3(0.f, 0.f, 0.f);
        } else {
            rot = make_float4(p.rotations[4 * g], p.rotations[4 * g + 1], p.rotations[4 * g + 2], p.rotations[4 * g + 3]);
            scx = p.scales[2 * g];
            scy = p.scales[2 * g + 1];
            R = quat_rot(rot);
            Lm = mmul(R, scale_mat(scx, scy, 1.0f));
            Pm = mmul(world2ndc(p.proj), ndc2pix(Wb, Hb));
            T = mmul(transpose(splat2world(Lm, po)), Pm);
            normal = xform_vec(col3(Lm, 2), p.view);
        }
        Mat<3, 3> dLT;
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int r = 0; r < 3; ++r) dLT.m[c][r] = dT[3 * c + r];
        const float dmx = s[9], dmy = s[10];
        bool early = false;
        if (dmx != 0 || dmy != 0) {
            const V3 tv = v3(9.0f, 9.0f, -1.0f);
            const V3 T0 = col3(T, 0), T1 = col3(T, 1), T2 = col3(T, 2);
            const float d = vdot(tv, vmul(T2, T2));
            const V3 fv = vscale(1.0f / d, tv);
            const V3 dT0 = vmul(vscale(dmx, fv), T2);
            const V3 dT1 = vmul(vscale(dmy, fv), T2);
            V3 dT3 = vadd(vmul(vscale(dmx, fv), T0), vmul(vscale(dmy, fv), T1));
            const V3 dL_df = vadd(vmul(vscale(dmx, T0), T2), vmul(vscale(dmy, T1), T2));
            const float dL_dd = (float)((double)vdot(dL_df, fv) * (-1.0 / (double)d));
            const V3 dd_dT3 = v3((tv.x * T2.x) * 2.0f, (tv.y * T2.y) * 2.0f, (tv.z * T2.z) * 2.0f);
            dT3 = vadd(dT3, vscale(dL_dd, dd_dT3));
            dLT.m[0][0] += dT0.x; dLT.m[0][1] += dT0.y; dLT.m[0][2] += dT0.z;
            dLT.m[1][0] += dT1.x; dLT.m[1][1] += dT1.y; dLT.m[1][2] += dT1.z;
            dLT.m[2][0] += dT3.x; dLT.m[2][1] += dT3.y; dLT.m[2][2] += dT3.z;
            if (precomp) {
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int r = 0; r < 3; ++r) dT[3 * c + r] = dLT.m[c][r];
                early = true;
            }
        }
        if (!precomp && !early) {
            const Mat<3, 4> dM = mmul(Pm, transpose(dLT));
            V3 dtn = xform_vec_t(v3(s[11], s[12], s[13]), p.view);
            const float3 pv = xform_point(po, p.view);
            const float cosv = -(pv.x * normal.x + pv.y * normal.y + pv.z * normal.z);
            const float mult = cosv > 0 ? 1.f : -1.f;
            dtn = vscale(mult, dtn);
            const V3 dRS0 = v3(dM.m[0][0], dM.m[0][1], dM.m[0][2]);
            const V3 dRS1 = v3(dM.m[1][0], dM.m[1][1], dM.m[1][2]);
            Mat<3, 3> dR;
            dR.m[0][0] = dRS0.x * scx; dR.m[0][1] = dRS0.y * scx; dR.m[0][2] = dRS0.z * scx;
            dR.m[1][0] = dRS1.x * scy; dR.m[1][1] = dRS1.y * scy; dR.m[1][2] = dRS1.z * scy;
            dR.m[2][0] = dtn.x; dR.m[2][1] = dtn.y; dR.m[2][2] = dtn.z;
            drot = quat_rot_vjp(rot, dR);
            dscale[0] = vdot(dRS0, col3(R, 0));
            dscale[1] = vdot(dRS1, col3(R, 1));
            dmean3[0] = dM.m[2][0];
            dmean3[1] = dM.m[2][1];
            dmean3[2] = dM.m[2][2];
        }
        // SH backward (backward.cu:20-98), with the reference's degree-2 gradient terms
        if (p.shs != nullptr) {
            const int deg = p.D;
            const V3 pos = v3(po.x, po.y, po.z);
            const V3 dir_orig = vsub(pos, v3(p.campos[0], p.campos[1], p.campos[2]));
            const float len = sqrtf(vdot(dir_orig, dir_orig));
            const V3 dir = v3(dir_orig.x / len, dir_orig.y / len, dir_orig.z / len);
            const float* sh = p.shs + (int64_t)g * M * 3;
            auto c = [&](int k) { return v3(sh[3 * k], sh[3 * k + 1], sh[3 * k + 2]); };
            const int cl = clamped_bits[g];
            V3 dRGB = v3(dcol[0] * ((cl & 1) ? 0.f : 1.f), dcol[1] * ((cl & 2) ? 0.f : 1.f),
                         dcol[2] * ((cl & 4) ? 0.f : 1.f));
            V3 dRGBdx = v3(0, 0, 0), dRGBdy = v3(0, 0, 0), dRGBdz = v3(0, 0, 0);
            const float x = dir.x, y = dir.y, z = dir.z;
            float* dsh = d_sh + (int64_t)g * M * 3;
            auto put = [&](int k, const V3 a) {
                dsh[3 * k] = a.x;
                dsh[3 * k + 1] = a.y;
                dsh[3 * k + 2] = a.z;
            };
            put(0, vscale(SH_C0, dRGB));
            if (deg > 0) {
                put(1, vscale(-SH_C1 * y, dRGB));
                put(2, vscale(SH_C1 * z, dRGB));
                put(3, vscale(-SH_C1 * x, dRGB));
                dRGBdx = vscale(-SH_C1, c(3));
                dRGBdy = vscale(-SH_C1, c(1));
                dRGBdz = vscale(SH_C1, c(2));
                if (deg > 1) {
                    const float depth = x;
                    const float d4 = __expf(-depth);
                    put(4, vscale(d4, dRGB));
                    const float d5 = x * x + y * y + z * z;
                    put(5, vscale(d5, dRGB));
                    const float d6 = x * y, d7 = y * z, d8 = x * z;
                    put(6, vscale(d6, dRGB));
                    put(7, vscale(d7, dRGB));
                    put(8, vscale(d8, dRGB));
                    // vector minus scalar, componentwise, as the reference writes it
                    auto sub = [](V3 a, float b) { return v3(a.x - b, a.y - b, a.z - b); };
                    auto add = [](V3 a, float b) { return v3(a.x + b, a.y + b, a.z + b); };
                    dRGBdx = sub(add(sub(sub(dRGBdx, d4), d5), d6), d8);
                    dRGBdy = add(sub(sub(dRGBdy, d5), d6), d7);
                    dRGBdz = add(sub(sub(dRGBdz, d5), d7), d8);
                }
            }
            const V3 dL_ddir = v3(vdot(dRGBdx, dRGB), vdot(dRGBdy, dRGB), vdot(dRGBdz, dRGB));
            const V3 dm = dnormvdv(dir_orig, dL_ddir);
            dmean3[0] += dm.x;
            dmean3[1] += dm.y;
            dmean3[2] += dm.z;
        }
        // screen-space mean gradient as the reference reports it (backward.cu:558-560)
        const float depth = rec[(int64_t)REC_F4 * g + 2].z;
        m2x = (float)(((double)(dT[2] * depth) * 0.5) * (double)(float)Wb);
        m2y = (float)(((double)(dT[5] * depth) * 0.5) * (double)(float)Hb);
    }
    d_mean2D[3 * g] = m2x;
    d_mean2D[3 * g + 1] = m2y;
    d_mean2D[3 * g + 2] = 0.f;
    d_colors[3 * g] = dcol[0];
    d_colors[3 * g + 1] = dcol[1];
    d_colors[3 * g + 2] = dcol[2];
    d_opacity[g] = s[14];
    d_means3D[3 * g] = dmean3[0];
    d_means3D[3 * g + 1] = dmean3[1];
    d_means3D[3 * g + 2] = dmean3[2];
#pragma unroll
    for (int q = 0; q < 9; ++q) d_transmat[9 * g + q] = dT[q];
    if (d_scales) {
        d_scales[2 * g] = dscale[0];
        d_scales[2 * g + 1] = dscale[1];
    }
    if (d_rot) {
        d_rot[4 * g] = drot.x;
        d_rot[4 * g + 1] = drot.y;
        d_rot[4 * g + 2] = drot.z;
        d_rot[4 * g + 3] = drot.w;
    }
}

// Reference-format binning and per-pixel state (rasterizer_impl.cu:116-137, ImageState).
__global__ void export_kernel(int T, const int* __restrict__ tile_start, const float* __restrict__ depth,
                              const int* __restrict__ sorted_gid, uint32_t* __restrict__ point_list,
                              unsigned long long* __restrict__ ref_keys, uint32_t* __restrict__ ranges) {
    const int t = blockIdx.x;
    if (t >= T) return;
    const int s0 = tile_start[t], s1 = tile_start[t + 1];
    if (threadIdx.x == 0) {
        ranges[2 * t] = s1 > s0 ? (uint32_t)s0 : 0u;
        ranges[2 * t + 1] = s1 > s0 ? (uint32_t)s1 : 0u;
    }
    for (int s = s0 + threadIdx.x; s < s1; s += blockDim.x) {
        point_list[s] = (uint32_t)sorted_gid[s];
        if (ref_keys) ref_keys[s] = ((unsigned long long)(uint32_t)t << 32) | __float_as_uint(depth[sorted_gid[s]]);
    }
}

__global__ void mark_visible_kernel(int P, const float* __restrict__ means, const float* __restrict__ view,
                                    uint8_t* __restrict__ present) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= P) return;
    const float3 po = make_float3(means[3 * g], means[3 * g + 1], means[3 * g + 2]);
    present[g] = (xform_point(po, view).z <= 0.2f) ? 0 : 1;
}

}  // namespace gs
}  // namespace us3d

using namespace us3d;
using namespace us3d::gs;

static BinAttr g_gs_sort_attr;

static inline int64_t gs_tiles(int32_t W, int32_t H) {
    return (int64_t)((W + TILE - 1) / TILE) * ((H + TILE - 1) / TILE);
}

extern "C" size_t us3d_gs_workspace_bytes(int64_t n_gauss, int32_t width, int32_t height, int64_t cap) {
    if (n_gauss < 0 || width <= 0 || height <= 0 || cap < 0) return 0;
    return carve(nullptr, n_gauss, gs_tiles(width, height), (int64_t)width * height, cap).bytes;
}

extern "C" size_t us3d_gs_backward_scratch_bytes(int64_t cap) {
    return cap < 0 ? 0 : (size_t)cap * PARTIAL_F4 * sizeof(float4);
}

static Params make_params(int64_t P, int32_t D, int32_t M, int32_t W, int32_t H, const float* means,
                          const float* shs, const float* colors, const float* opac, const float* scales, float mod,
                          const float* rots, const float* transmat, const float* view, const float* proj,
                          const float* campos, int32_t prefiltered) {
    Params p;
    p.P = (int)P; p.D = D; p.M = M; p.W = W; p.H = H;
    p.gx = (W + TILE - 1) / TILE;
    p.gy = (H + TILE - 1) / TILE;
    p.scale_modifier = mod;
    p.prefiltered = prefiltered;
    p.means = means; p.shs = shs; p.colors = colors; p.opacities = opac; p.scales = scales;
    p.rotations = rots; p.transmat = transmat; p.view = view; p.proj = proj; p.campos = campos;
    return p;
}

static int gs_forward_impl(void* workspace, size_t workspace_bytes, int64_t n_gauss, int32_t sh_degree,
                           int32_t sh_coeffs, const float* background, int32_t width, int32_t height,
                           const float* means3D, const float* shs, const float* colors_precomp,
                           const float* opacities, const float* scales, float scale_modifier, const float* rotations,
                           const float* transmat_precomp, const float* viewmatrix, const float* projmatrix,
                           const float* campos, int32_t prefiltered, int64_t cap, float* out_color, float* out_others,
                           int32_t* out_radii, StatusRead* status, void* stream_) {
    US3D_CHECK_ARG(width > 0 && height > 0, "image_width/image_height must be positive");
    US3D_CHECK_ARG(n_gauss >= 0 && n_gauss <= 0x7fffffffLL, "n_gauss out of range");
    US3D_CHECK_ARG(cap >= 0 && cap <= 0x7fffffffLL, "instance capacity must be in [0, 2^31)");
    US3D_CHECK_ARG(workspace && background && viewmatrix && projmatrix && out_color && out_others,
                   "NULL pointer argument");
    US3D_CHECK_ARG(n_gauss == 0 || (means3D && opacities && out_radii), "NULL Gaussian pointer");
    US3D_CHECK_ARG(n_gauss == 0 || (colors_precomp != nullptr) != (shs != nullptr),
                   "Please provide excatly one of either SHs or precomputed colors!");
    US3D_CHECK_ARG(n_gauss == 0 || ((scales && rotations) != (transmat_precomp != nullptr)),
                   "Please provide exactly one of either scale/rotation pair or precomputed 3D covariance!");
    US3D_CHECK_ARG(shs == nullptr || (sh_coeffs >= 1 && campos != nullptr && sh_degree >= 0 &&
                                      (sh_degree < 1 || sh_coeffs >= 4) && (sh_degree < 2 || sh_coeffs >= 9)),
                   "SH coefficients too few for the requested degree");
    const int64_t T = gs_tiles(width, height), P = (int64_t)width * height;
    const Workspace w = carve(workspace, n_gauss, T, P, cap);
    US3D_CHECK_ARG(workspace_bytes >= w.bytes, "workspace too small: %zu < %zu", workspace_bytes, w.bytes);
    cudaStream_t stream = (cudaStream_t)stream_;
    const Params p = make_params(n_gauss, sh_degree, sh_coeffs, width, height, means3D, shs, colors_precomp,
                                 opacities, scales, scale_modifier, rotations, transmat_precomp, viewmatrix,
                                 projmatrix, campos, prefiltered);
    const int prof = prof_begin("gs_forward", stream);
    init_kernel<<<(unsigned)((T + 255) / 256), 256, 0, stream>>>(T, w.tile_count, w.tile_cursor, w.header, cap,
                                                                 n_gauss, P);
    const unsigned gb = (unsigned)((n_gauss + 255) / 256);
    if (n_gauss > 0)
        preprocess_kernel<<<gb, 256, 0, stream>>>(p, out_radii, w.rec, w.depth, w.rect, w.clamped, w.touched,
                                                  w.tile_count, w.header);
    US3D_CHECK_LAUNCH("gs preprocess");
    US3D_CHECK_CUDA(launch_bins(n_gauss, p.gx, T, RectOf4{w.rect}, reinterpret_cast<const uint32_t*>(w.depth), w.touched, w.stable, w.tile_count,
                                w.tile_start, w.tile_cursor, w.inst_offset, w.bs_g, w.bs_t, w.header, cap, w.keys, w.slot_inst,
                                w.sorted_gid, w.sorted_inst, g_gs_sort_attr, stream));
    if (status != nullptr) {
        const int rc = status->record(w.header, stream);
        if (rc != US3D_OK) return rc;
    }
    forward_kernel<<<(unsigned)T, BLOCK, 0, stream>>>(width, height, p.gx, w.tile_start, w.sorted_gid, w.header, w.rec,
                                                      background, out_color, out_others, w.accum, w.n_contrib);
    US3D_CHECK_LAUNCH("gs forward");
    prof_end(prof, stream);
    count_launches(1 + (n_gauss > 0) + bins_launches(n_gauss, T, w.keys == nullptr, true) + 1);
    return US3D_OK;
}

extern "C" int us3d_gs_forward(void* workspace, size_t workspace_bytes, int64_t n_gauss, int32_t sh_degree,
                               int32_t sh_coeffs, const float* background, int32_t width, int32_t height,
                               const float* means3D, const float* shs, const float* colors_precomp,
                               const float* opacities, const float* scales, float scale_modifier,
                               const float* rotations, const float* transmat_precomp, const float* viewmatrix,
                               const float* projmatrix, const float* campos, int32_t prefiltered, int64_t cap,
                               float* out_color, float* out_others, int32_t* out_radii, void* stream_) {
    return gs_forward_impl(workspace, workspace_bytes, n_gauss, sh_degree, sh_coeffs, background, width, height,
                           means3D, shs, colors_precomp, opacities, scales, scale_modifier, rotations,
                           transmat_precomp, viewmatrix, projmatrix, campos, prefiltered, cap, out_color, out_others,
                           out_radii, nullptr, stream_);
}

extern "C" int us3d_gs_forward_checked(void* workspace, size_t workspace_bytes, int64_t n_gauss, int32_t sh_degree,
                                       int32_t sh_coeffs, const float* background, int32_t width, int32_t height,
                                       const float* means3D, const float* shs, const float* colors_precomp,
                                       const float* opacities, const float* scales, float scale_modifier,
                                       const float* rotations, const float* transmat_precomp, const float* viewmatrix,
                                       const float* projmatrix, const float* campos, int32_t prefiltered, int64_t cap,
                                       float* out_color, float* out_others, int32_t* out_radii, int64_t* total,
                                       int32_t* flags, void* stream_) {
    StatusRead status;
    const int st = gs_forward_impl(workspace, workspace_bytes, n_gauss, sh_degree, sh_coeffs, background, width,
                                   height, means3D, shs, colors_precomp, opacities, scales, scale_modifier, rotations,
                                   transmat_precomp, viewmatrix, projmatrix, campos, prefiltered, cap, out_color,
                                   out_others, out_radii, &status, stream_);
    return st != US3D_OK ? st : wait_status(status, total, flags);
}

extern "C" int us3d_gs_read_status(const void* workspace, int64_t* total, int32_t* flags, void* stream_) {
    US3D_CHECK_ARG(workspace != nullptr, "workspace is NULL");
    long long hdr[H_WORDS];
    cudaStream_t stream = (cudaStream_t)stream_;
    US3D_CHECK_CUDA(cudaMemcpyAsync(hdr, workspace, sizeof(hdr), cudaMemcpyDeviceToHost, stream));
    US3D_CHECK_CUDA(cudaStreamSynchronize(stream));
    if (total) *total = hdr[H_TOTAL];
    if (flags) *flags = (int32_t)hdr[H_FLAGS];
    return US3D_OK;
}

extern "C" int us3d_gs_backward(void* workspace, int64_t n_gauss, int32_t sh_degree, int32_t sh_coeffs,
                                const float* background, int32_t width, int32_t height, const float* means3D,
                                const float* shs, const float* colors_precomp, const float* scales,
                                float scale_modifier, const float* rotations, const float* transmat_precomp,
                                const float* viewmatrix, const float* projmatrix, const float* campos,
                                float tan_fovx, float tan_fovy, const int32_t* radii, int64_t cap,
                                const float* dL_dcolor, const float* dL_dothers, void* scratch, size_t scratch_bytes,
                                float* d_means2D, float* d_colors, float* d_opacity, float* d_means3D,
                                float* d_transmat, float* d_sh, float* d_scales, float* d_rotations, void* stream_) {
    US3D_CHECK_ARG(width > 0 && height > 0 && n_gauss >= 0 && cap >= 0, "bad sizes");
    US3D_CHECK_ARG(workspace && background && viewmatrix && projmatrix && dL_dcolor && dL_dothers,
                   "NULL pointer argument");
    US3D_CHECK_ARG(scratch_bytes >= us3d_gs_backward_scratch_bytes(cap), "backward scratch too small");
    US3D_CHECK_ARG(n_gauss == 0 || (means3D && radii && d_means2D && d_colors && d_opacity && d_means3D && d_transmat),
                   "NULL gradient pointer");
    US3D_CHECK_ARG(shs == nullptr || (d_sh && campos), "NULL SH gradient pointer");
    (void)colors_precomp;
    (void)scale_modifier;  // the reference's backward rebuilds the homography at scale 1
    const int64_t T = gs_tiles(width, height), P = (int64_t)width * height;
    const Workspace w = carve(workspace, n_gauss, T, P, cap);
    cudaStream_t stream = (cudaStream_t)stream_;
    const Params p = make_params(n_gauss, sh_degree, sh_coeffs, width, height, means3D, shs, colors_precomp, nullptr,
                                 scales, scale_modifier, rotations, transmat_precomp, viewmatrix, projmatrix, campos, 0);
    // focal lengths exactly as the reference computes them on the host
    const float focal_y = (float)height / (2.0f * tan_fovy);
    const float focal_x = (float)width / (2.0f * tan_fovx);
    float4* partial = reinterpret_cast<float4*>(scratch);
    const int prof = prof_begin("gs_backward", stream);
    backward_kernel<<<(unsigned)T, BLOCK, 0, stream>>>(width, height, p.gx, w.tile_start, w.sorted_gid,
                                                       w.sorted_inst, w.header, w.rec, background, w.accum,
                                                       w.n_contrib, dL_dcolor, dL_dothers, partial);
    if (n_gauss > 0) {
        reduce_partials_kernel<<<(unsigned)((n_gauss * PARTIAL_F4 + REDUCE_THREADS - 1) / REDUCE_THREADS),
                                 REDUCE_THREADS, 0, stream>>>(n_gauss, radii, w.inst_offset, w.header, partial);
        reduce_preprocess_kernel<<<(unsigned)((n_gauss + 127) / 128), 128, 0, stream>>>(
            p, focal_x, focal_y, tan_fovx, tan_fovy, radii, w.inst_offset, w.header, partial, w.rec, w.clamped,
            d_means2D, d_colors, d_opacity, d_means3D, d_transmat, d_sh, d_scales, d_rotations);
    }
    US3D_CHECK_LAUNCH("gs backward");
    prof_end(prof, stream);
    count_launches(1 + 2 * (n_gauss > 0));
    return US3D_OK;
}

extern "C" int us3d_gs_export(const void* workspace, int64_t n_gauss, int32_t width, int32_t height, int64_t cap,
                              uint32_t* out_point_list, uint64_t* out_keys, uint32_t* out_ranges,
                              uint32_t* out_n_contrib, float* out_accum, float* out_records, void* stream_) {
    US3D_CHECK_ARG(workspace && out_point_list && out_ranges && width > 0 && height > 0, "bad argument");
    const int64_t T = gs_tiles(width, height), P = (int64_t)width * height;
    const Workspace w = carve(const_cast<void*>(workspace), n_gauss, T, P, cap);
    cudaStream_t stream = (cudaStream_t)stream_;
    export_kernel<<<(unsigned)T, 256, 0, stream>>>((int)T, w.tile_start, w.depth, w.sorted_gid, out_point_list,
                                                   reinterpret_cast<unsigned long long*>(out_keys), out_ranges);
    US3D_CHECK_LAUNCH("gs export");
    if (out_n_contrib)
        US3D_CHECK_CUDA(cudaMemcpyAsync(out_n_contrib, w.n_contrib, sizeof(uint32_t) * 2 * P, cudaMemcpyDeviceToDevice, stream));
    if (out_accum)
        US3D_CHECK_CUDA(cudaMemcpyAsync(out_accum, w.accum, sizeof(float) * 3 * P, cudaMemcpyDeviceToDevice, stream));
    if (out_records && n_gauss > 0)
        US3D_CHECK_CUDA(cudaMemcpyAsync(out_records, w.rec, sizeof(float4) * REC_F4 * n_gauss, cudaMemcpyDeviceToDevice,
                                        stream));
    count_launches(1);
    return US3D_OK;
}

extern "C" int us3d_gs_mark_visible(int64_t n_gauss, const float* means3D, const float* viewmatrix,
                                    uint8_t* out_present, void* stream_) {
    US3D_CHECK_ARG(n_gauss >= 0 && n_gauss <= 0x7fffffffLL, "n_gauss out of range");
    if (n_gauss == 0) return US3D_OK;
    US3D_CHECK_ARG(means3D && viewmatrix && out_present, "NULL pointer argument");
    mark_visible_kernel<<<(unsigned)((n_gauss + 255) / 256), 256, 0, (cudaStream_t)stream_>>>((int)n_gauss, means3D,
                                                                                             viewmatrix, out_present);
    US3D_CHECK_LAUNCH("gs mark_visible");
    count_launches(1);
    return US3D_OK;
}
