// The denoiser fallback: renderer/src/denoise.rs `denoise` (edge-avoiding a-trous wavelet filter, Dammertz et al.
// 2010, guided by first-hit albedo and normal, its luminance edge-stopping width from the variance filtered over 3 x 3
// pixels as in SVGF), run on the scene's accum on the device. main.rs:548-557 calls it with 4 iterations on the Frame
// (gpu.rs:4219-4232: each Pixel over its count, the normal normalised or zero). Included by pathtrace.cu.
//
// Arithmetic is denoise.rs's in f32, with the two edge-stopping exponentials taken as one of the summed exponents, their
// divisors as factors, and the sums as fused multiply-adds; `exp` is the device's expf (within a few ulps of libm).
// Results match the oracle's restatement to ~1e-5 relative, not bit for bit.
#pragma once

namespace trt {

constexpr float DN_EPS = 1e-3f;
// denoise.rs:16 K: the B3 spline's taps 3/8, 1/4, 1/16 by distance
__device__ __forceinline__ float dn_k(int a) { return a == 0 ? 0.375f : (a == 1 ? 0.25f : 0.0625f); }

struct DenoiseBufs {
    float4* cur[2];   // demodulated irradiance (xyz), its luminance (w)
    float* var[2];    // its variance
    float4* nrm_a;    // first-hit normal, normalised or zero (xyz); the first-hit albedo's x (w)
    float2* alb_yz;   // the albedo's y and z (the Frame's)
};

__device__ __forceinline__ float dn_fin(float v) { return (__float_as_uint(v) & 0x7f800000u) == 0x7f800000u ? 0.0f : v; }
__device__ __forceinline__ V3 dn_max_eps(V3 a) { return V3{fmaxf(a.x, DN_EPS), fmaxf(a.y, DN_EPS), fmaxf(a.z, DN_EPS)}; }

// gpu.rs:4219-4232 (the Frame of a Pixel) and denoise.rs:11-15 (demodulation, the variance in irradiance units).
__global__ void k_dn_prep(const float4* __restrict__ accum, uint32_t n, DenoiseBufs D) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 c = accum[5ull * i], a = accum[5ull * i + 1], nn = accum[5ull * i + 2];
    float cnt = fmaxf(dn_fin(c.w), 1.0f);
    V3 color = V3{dn_fin(c.x) / cnt, dn_fin(c.y) / cnt, dn_fin(c.z) / cnt};
    V3 albedo = V3{dn_fin(a.x) / cnt, dn_fin(a.y) / cnt, dn_fin(a.z) / cnt};
    V3 normal = V3{dn_fin(nn.x) / cnt, dn_fin(nn.y) / cnt, dn_fin(nn.z) / cnt};
    float mean = dn_fin(a.w) / cnt;
    float variance = fmaxf(dn_fin(nn.w) / cnt - mean * mean, 0.0f) / cnt;
    // glam normalize_or_zero: v / |v| where 1 / |v| is finite and positive
    float len = sqrtf(dot(normal, normal));
    float rcp = 1.0f / len;
    normal = (rcp > 0.0f && (__float_as_uint(rcp) & 0x7f800000u) != 0x7f800000u) ? normal * rcp : v3(0.0f);
    V3 ae = dn_max_eps(albedo);
    V3 demod = V3{color.x / ae.x, color.y / ae.y, color.z / ae.z};
    float la = dot(ae, V3{0.2126f, 0.7152f, 0.0722f});
    D.cur[0][i] = f4(demod, luminance(demod));
    D.var[0][i] = variance / (la * la);
    D.nrm_a[i] = f4(normal, albedo.x);
    D.alb_yz[i] = make_float2(albedo.y, albedo.z);
}

// denoise.rs:20-35: the variance over 3 x 3 pixels, weights 0.5 / 0.25 a tap along each axis, over the taps inside.
__device__ __forceinline__ float dn_var3(const float* __restrict__ var, int x, int y, int w, int h) {
    float s = 0.0f, ws = 0.0f;
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            int qx = x + dx, qy = y + dy;
            if (qx < 0 || qy < 0 || qx >= w || qy >= h) continue;
            float k = (dx == 0 ? 0.5f : 0.25f) * (dy == 0 ? 0.5f : 0.25f);
            s += k * __ldg(var + (uint32_t)qy * (uint32_t)w + (uint32_t)qx);
            ws += k;
        }
    return s / ws;
}

__device__ __forceinline__ float pow64(float x) {
    // x^64 by six squarings (what powi(64) comes to)
    x = x * x; x = x * x; x = x * x; x = x * x; x = x * x;
    return x * x;
}

// denoise.rs:36-68: one a-trous iteration at `step`, 5 x 5 taps of the B3 spline kernel, after the variance's filter; the
// last iteration writes the irradiance times the albedo again (denoise.rs:72), as RGB floats.
// Bound: issue (25 taps of about 50 instructions; the taps' loads are L1 hits of a 32 x 8 tile's neighbourhood). With a
// division and an exponential for each of the two edge-stops, a luminance a tap, products and sums unfused, and bounds
// checked on every tap it was about 95: 140 us an iteration at 1280 x 720 under ncu, and 8 more for the variance.
// INSIDE: every tap lies in the image (all but the tiles at its border).
struct DnSum { float x, y, z, w, v; };
template <bool INSIDE>
__device__ __forceinline__ DnSum dn_taps(const DenoiseBufs& D, const float4* __restrict__ cur, const float* __restrict__ var,
                                         int x, int y, int w, int h, int step, float lp, float inv_sigma, V3 np, V3 ap) {
    DnSum t{0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int dy = -2; dy <= 2; ++dy) {
        const int qy = y + dy * step;
        if (!INSIDE && (qy < 0 || qy >= h)) continue;
        const uint32_t row = (uint32_t)qy * (uint32_t)w;
#pragma unroll
        for (int dx = -2; dx <= 2; ++dx) {
            const int qx = x + dx * step;
            if (!INSIDE && (qx < 0 || qx >= w)) continue;
            const uint32_t q = row + (uint32_t)qx;
            const float4 c = __ldg(cur + q), g = __ldg(D.nrm_a + q);
            const float2 a = __ldg(D.alb_yz + q);
            const float wn = pow64(fmaxf(__fmaf_rn(np.z, g.z, __fmaf_rn(np.y, g.y, np.x * g.x)), 0.0f));
            const float ax = ap.x - g.w, ay = ap.y - a.x, az = ap.z - a.y;
            const float d2 = __fmaf_rn(az, az, __fmaf_rn(ay, ay, ax * ax));
            const float e = expf(__fmaf_rn(d2, -100.0f, -(fabsf(lp - c.w) * inv_sigma)));
            const float wt = dn_k(dx < 0 ? -dx : dx) * dn_k(dy < 0 ? -dy : dy) * wn * e;
            t.x = __fmaf_rn(c.x, wt, t.x);
            t.y = __fmaf_rn(c.y, wt, t.y);
            t.z = __fmaf_rn(c.z, wt, t.z);
            t.w += wt;
            t.v = __fmaf_rn(wt * wt, __ldg(var + q), t.v);
        }
    }
    return t;
}
constexpr uint32_t DN_TILE_X = 32u, DN_TILE_Y = 8u;
__global__ void __launch_bounds__(DN_TILE_X * DN_TILE_Y) k_dn_atrous(DenoiseBufs D, uint32_t src, uint32_t w, uint32_t h,
                                                                     int step, float* __restrict__ rgb) {
    // (tiles in rows, one grid dimension: an image may be 2^26 pixels high)
    const uint32_t tiles_x = (w + DN_TILE_X - 1u) / DN_TILE_X;
    const int x = (int)(blockIdx.x % tiles_x * DN_TILE_X + threadIdx.x % DN_TILE_X);
    const int y = (int)(blockIdx.x / tiles_x * DN_TILE_Y + threadIdx.x / DN_TILE_X);
    if (x >= (int)w || y >= (int)h) return;
    const uint32_t i = (uint32_t)y * w + (uint32_t)x;
    const float4* cur = src ? D.cur[1] : D.cur[0];
    const float* var = src ? D.var[1] : D.var[0];
    const float4 cp = cur[i], g = D.nrm_a[i];
    const float2 a = D.alb_yz[i];
    const V3 np = xyz(g), ap{g.w, a.x, a.y};
    const float var_f = dn_var3(var, x, y, (int)w, (int)h);
    const float inv_sigma = 1.0f / (4.0f * sqrtf(fmaxf(var_f, 0.0f)) + 1e-4f);
    const bool inside = x >= 2 * step && y >= 2 * step && x + 2 * step < (int)w && y + 2 * step < (int)h;
    const DnSum t = inside ? dn_taps<true>(D, cur, var, x, y, (int)w, (int)h, step, cp.w, inv_sigma, np, ap)
                           : dn_taps<false>(D, cur, var, x, y, (int)w, (int)h, step, cp.w, inv_sigma, np, ap);
    const bool any = t.w > 0.0f;
    const V3 c = any ? V3{t.x / t.w, t.y / t.w, t.z / t.w} : xyz(cp);
    if (rgb) {
        const V3 ae = dn_max_eps(ap);
        rgb[3ull * i] = c.x * ae.x;
        rgb[3ull * i + 1] = c.y * ae.y;
        rgb[3ull * i + 2] = c.z * ae.z;
    } else {
        (src ? D.cur[0] : D.cur[1])[i] = f4(c, luminance(c));
        (src ? D.var[0] : D.var[1])[i] = any ? t.v / (t.w * t.w) : var[i];
    }
}

// denoise.rs:72 with no iterations: the irradiance times the albedo again.
__global__ void k_dn_remod(DenoiseBufs D, uint32_t n, float* rgb) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const V3 c = xyz(D.cur[0][i]);
    const float2 a = D.alb_yz[i];
    const V3 ae = dn_max_eps(V3{D.nrm_a[i].w, a.x, a.y});
    rgb[3ull * i] = c.x * ae.x;
    rgb[3ull * i + 1] = c.y * ae.y;
    rgb[3ull * i + 2] = c.z * ae.z;
}

}  // namespace trt
