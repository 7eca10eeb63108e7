// env_tex.cuh -- the environment map lookup, shared by the host table build
// and the device kernels: HDRTexture2D::evaluate_impl
// (src/texture/hdr_texture.cpp:27-30) behind Texture2D::evaluate with the
// repeat wrap (src/core/texture.hpp:57-95), i.e. LinearSampler::Sample2D
// (src/utility/sampler.hpp:16-29) in double with float texels: each
// texel-times-weight product is a double product rounded to float
// (Point3<float>::operator*(double), src/utility/geometry.hpp:268-271), the
// sums are float.
//
// A lookup is some 60 double operations, and FP64 runs at a small fraction of
// the FP32 rate. But a coordinate in [0, 1] that is zero or at least 2^-20 is a
// multiple of 2^-44, so the weights are too: integers of 45 bits, exactly (the
// doubles hold them exactly as well). A byte texel's weighted value is then
// integer arithmetic; a float texel's is a product of the weight's two float
// parts with the rounding test of exact32.cuh. What is outside the safe range
// (coordinates below 2^-20, NaN, texels that are negative, tiny, huge or not
// finite) or too close to a rounding boundary takes the double expressions, out
// of line. Maps on every material under a sky map 1001x563x4 7.66 -> 6.94 ms,
// all material kinds under the sky map 320x180x8 4.80 -> 4.52 ms.
#pragma once

#include <cuda_runtime.h>

#include "exact32.cuh"

namespace trg {

// One axis of the lookup: the two texels and their weights, d of the second and
// e = 1 - d of the first, in units of 2^-44: high 23 and low 22 bits.
struct TexAxis {
  int i0, i1;
  uint32_t dh, dl, eh, el;
};
// t: the wrapped coordinate. False outside the exact range.
TR_HD bool tex_axis(float t, int n, TexAxis& A) {
  const uint32_t b = fbits(t);
  if (!(b == 0u || (b >= 0x35800000u && b <= 0x3f800000u)) || n > (1 << 18)) return false;  // 0, [2^-20, 1]
  const uint64_t m = (b & 0x7fffffu) | 0x800000u;
  const uint64_t U = b ? m << ((b >> 23) - 106u) : 0u;  // t 2^44
  const uint64_t x = U * (uint32_t)(n - 1);             // t (n - 1), below 2^62
  const uint64_t one = 1ull << 44, d = x & (one - 1), e = one - d;
  A.i0 = (int)(x >> 44);
  A.i1 = A.i0 + 1 > n - 1 ? n - 1 : A.i0 + 1;
  A.dh = (uint32_t)(d >> 22);
  A.dl = (uint32_t)d & 0x3fffffu;
  A.eh = (uint32_t)(e >> 22);
  A.el = (uint32_t)e & 0x3fffffu;
  return true;
}

// A weight as two floats, h its rounding and h + l the weight.
struct TexWeight {
  float h, l;
};
TR_HD TexWeight tex_weight(uint32_t hi, uint32_t lo) {
  const float a = (float)hi * 2.38418579e-07f, b = (float)lo * 5.68434189e-14f;  // 2^-22, 2^-44: exact
  TexWeight w;
  w.h = a + b;
  w.l = b - (w.h - a);
  return w;
}
// float(double(w) * double(x)) for x zero or in [2^-40, 2^61]; ok cleared
// when not proven. With p = RN(w.h x) the rest is e + w.l x, below 2^-22 p:
// its rounding, the ends' in ziv and the double product's are together below
// 6 * 2^-48 p.
TR_HD float tex_mul(TexWeight w, float x, bool& ok) {
  const float p = w.h * x;
  const float r = ffma(w.l, x, ffma(w.h, x, -p));
  float y;
  ok &= ziv(p, r, 5.68434189e-14f * p, y);  // 2^-44
  return y;
}

TR_HD void tex_wrap(float u_in, float v_in, float& uw, float& vw) {
  // wrap_repeat: clamp(x - floor(x), 0, 1)
  uw = u_in - floorf(u_in);
  vw = v_in - floorf(v_in);
  uw = uw < 0.0f ? 0.0f : (1.0f < uw ? 1.0f : uw);
  vw = vw < 0.0f ? 0.0f : (1.0f < vw ? 1.0f : vw);
}

// The lookups as the reference writes them. Texel (x, y) at tex[x + y * w];
// (uw, vw): wrapped coordinates.
TR_HD_COLD f3 env_tex_eval_d(const float4* tex, int w, int h, float uw, float vw) {
  double u = (double)uw, v = (double)vw;
  u = (u < 0.0 ? 0.0 : (1.0 < u ? 1.0 : u)) * (double)(w - 1);
  v = (v < 0.0 ? 0.0 : (1.0 < v ? 1.0 : v)) * (double)(h - 1);
  int u0 = (int)u, v0 = (int)v;
  u0 = u0 < 0 ? 0 : (u0 > w - 1 ? w - 1 : u0);
  v0 = v0 < 0 ? 0 : (v0 > h - 1 ? h - 1 : v0);
  const int u1 = u0 + 1 > w - 1 ? w - 1 : u0 + 1;
  const int v1 = v0 + 1 > h - 1 ? h - 1 : v0 + 1;
  const double du = u - u0, dv = v - v0;
  const double eu = 1.0 - du, ev = 1.0 - dv;
  const float4 a = tex[u0 + (size_t)v0 * w], b = tex[u1 + (size_t)v0 * w];
  const float4 c = tex[u0 + (size_t)v1 * w], d = tex[u1 + (size_t)v1 * w];
  // ((a eu + b du) ev) + ((c eu + d du) dv), per channel
  const float tr = (float)(eu * a.x) + (float)(du * b.x), br = (float)(eu * c.x) + (float)(du * d.x);
  const float tg = (float)(eu * a.y) + (float)(du * b.y), bg = (float)(eu * c.y) + (float)(du * d.y);
  const float tb = (float)(eu * a.z) + (float)(du * b.z), bb = (float)(eu * c.z) + (float)(du * d.z);
  return mk3((float)(ev * tr) + (float)(dv * br), (float)(ev * tg) + (float)(dv * bg),
             (float)(ev * tb) + (float)(dv * bb));
}

// ImageTexture2D::evaluate_impl (src/texture/image_texture2d.cpp:26-30) over
// Image2D<Color3b>: the same bilinear weights, but each weighted texel is a
// Point3<uint8_t> (the double product truncated to a byte) and the sums are
// bytes; the result is divided by 255.
TR_HD_COLD f3 env_tex_eval8_d(const uchar4* tex, int w, int h, float uw, float vw) {
  double u = (double)uw, v = (double)vw;
  u = (u < 0.0 ? 0.0 : (1.0 < u ? 1.0 : u)) * (double)(w - 1);
  v = (v < 0.0 ? 0.0 : (1.0 < v ? 1.0 : v)) * (double)(h - 1);
  int u0 = (int)u, v0 = (int)v;
  u0 = u0 < 0 ? 0 : (u0 > w - 1 ? w - 1 : u0);
  v0 = v0 < 0 ? 0 : (v0 > h - 1 ? h - 1 : v0);
  const int u1 = u0 + 1 > w - 1 ? w - 1 : u0 + 1;
  const int v1 = v0 + 1 > h - 1 ? h - 1 : v0 + 1;
  const double du = u - u0, dv = v - v0;
  const double eu = 1.0 - du, ev = 1.0 - dv;
  const uchar4 a = tex[u0 + (size_t)v0 * w], b = tex[u1 + (size_t)v0 * w];
  const uchar4 c = tex[u0 + (size_t)v1 * w], d = tex[u1 + (size_t)v1 * w];
  auto by = [](double f, int x) { return (int)(f * (double)x) & 0xff; };
  auto ch = [&](int ta, int tb, int tc, int td) {
    const int top = (by(eu, ta) + by(du, tb)) & 0xff, bot = (by(eu, tc) + by(du, td)) & 0xff;
    return (float)((by(ev, top) + by(dv, bot)) & 0xff) / 255.0f;
  };
  return mk3(ch(a.x, b.x, c.x, d.x), ch(a.y, b.y, c.y, d.y), ch(a.z, b.z, c.z, d.z));
}

// The same results (texture coordinates as given).
TR_HD_COLD f3 env_tex_eval(const float4* tex, int w, int h, float u_in, float v_in) {
  float uw, vw;
  tex_wrap(u_in, v_in, uw, vw);
  TexAxis U, V;
  if (!tex_axis(uw, w, U) || !tex_axis(vw, h, V)) return env_tex_eval_d(tex, w, h, uw, vw);
  const float4 a = tex[U.i0 + (size_t)V.i0 * w], b = tex[U.i1 + (size_t)V.i0 * w];
  const float4 c = tex[U.i0 + (size_t)V.i1 * w], d = tex[U.i1 + (size_t)V.i1 * w];
  const TexWeight du = tex_weight(U.dh, U.dl), eu = tex_weight(U.eh, U.el);
  const TexWeight dv = tex_weight(V.dh, V.dl), ev = tex_weight(V.eh, V.el);
  bool ok = true;
  uint32_t least = 0xffffffffu, most = 0u;  // of the factors' bits (less one: zero passes)
  auto row = [&](float x, float y) {
    const uint32_t bx = fbits(x), by = fbits(y);
    least = umin3(least, bx - 1u, by - 1u);
    most = most > bx ? most : bx;
    most = most > by ? most : by;
    return tex_mul(eu, x, ok) + tex_mul(du, y, ok);
  };
  auto col = [&](float x, float y) {
    least = umin3(least, fbits(x) - 1u, fbits(y) - 1u);
    return tex_mul(ev, x, ok) + tex_mul(dv, y, ok);
  };
  const f3 top = mk3(row(a.x, b.x), row(a.y, b.y), row(a.z, b.z));
  const f3 bot = mk3(row(c.x, d.x), row(c.y, d.y), row(c.z, d.z));
  const f3 r = mk3(col(top.x, bot.x), col(top.y, bot.y), col(top.z, bot.z));
  // texels zero or in [2^-40, 2^60], rows zero or at least 2^-40
  if (ok && least >= 0x2b800000u - 1u && most <= 0x5d800000u) return r;
  return env_tex_eval_d(tex, w, h, uw, vw);
}

TR_HD_COLD f3 env_tex_eval8(const uchar4* tex, int w, int h, float u_in, float v_in) {
  float uw, vw;
  tex_wrap(u_in, v_in, uw, vw);
  TexAxis U, V;
  if (!tex_axis(uw, w, U) || !tex_axis(vw, h, V)) return env_tex_eval8_d(tex, w, h, uw, vw);
  const uchar4 a = tex[U.i0 + (size_t)V.i0 * w], b = tex[U.i1 + (size_t)V.i0 * w];
  const uchar4 c = tex[U.i0 + (size_t)V.i1 * w], d = tex[U.i1 + (size_t)V.i1 * w];
  // floor(weight * x): (h 2^22 + l) x / 2^44
  auto by = [](uint32_t h22, uint32_t l22, uint32_t x) { return (h22 * x + (l22 * x >> 22)) >> 22; };
  auto ch = [&](uint32_t ta, uint32_t tb, uint32_t tc, uint32_t td) {
    const uint32_t top = (by(U.eh, U.el, ta) + by(U.dh, U.dl, tb)) & 0xffu;
    const uint32_t bot = (by(U.eh, U.el, tc) + by(U.dh, U.dl, td)) & 0xffu;
    return (float)((by(V.eh, V.el, top) + by(V.dh, V.dl, bot)) & 0xffu) / 255.0f;
  };
  return mk3(ch(a.x, b.x, c.x, d.x), ch(a.y, b.y, c.y, d.y), ch(a.z, b.z, c.z, d.z));
}

}  // namespace trg
