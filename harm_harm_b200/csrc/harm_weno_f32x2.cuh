// harm_weno_f32x2.cuh -- the FP32 WENO5 weights and edge values of two cells at once on
// Blackwell's packed FP32 pipe (add/mul/fma on float2: one instruction, two lanes).
//
// The algorithm is that of smono_indicator / weno5_cell_weights / weno3_unopt / weno_frac /
// weno5_edges (harm_device.cuh) for T = float, lane by lane, in the differences of the stencil
// to its centre (exact for neighbouring values within a factor of two, so a constant line
// gives its value exactly); operations without a packed form (reciprocals, compares, selects,
// min/max) run on each lane.  Where the scalar code branches on a lane's value (monotone
// cells, the WENO3 blend of the stencil reduction), the packed code evaluates both sides when
// either lane needs them and blends with exact zeros and ones, so that a lane's value never
// depends on its partner.
//
// What bounds it is the FMA pipe (a packed operation takes two of its cycles), then the ALU
// (compares and min/max at half rate) and the special-function unit (a reciprocal takes eight
// cycles of a warp's quarter of the SM).  So the derivatives come from the sums and
// differences of opposite neighbours (19 packed operations instead of 54), min-mods of
// magnitudes are sign tests and minima, the three 1/beta^2 share their denominators, and the
// weight ratios are divided out only where one exceeds the threshold.
#pragma once
#include "harm_device.cuh"

namespace hb {

// F2 is a float2: the compiler's float2 intrinsics of the packed pipe (add, mul, fma with
// round-to-nearest; no contraction across them) let it keep the pairs in adjacent registers,
// so packing and unpacking cost no moves
using F2 = float2;

__device__ __forceinline__ F2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ F2 f2(float a) { return make_float2(a, a); }
// 1/x for x and 1/x normal (the hardware approximation, 1 ulp; every operand here is a sum with
// the smallest normal number or larger)
__device__ __forceinline__ float rcp_ftz(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void f2split(F2 x, float& a, float& b) {
  a = x.x;
  b = x.y;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return __fadd2_rn(a, b); }
// a - b as fma(b, -1, a): one packed instruction, where negating a pair takes two more
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ F2 ffma2(F2 a, F2 b, F2 c) { return __ffma2_rn(a, b, c); }
// lane-wise helpers
template <typename Fn>
__device__ __forceinline__ F2 lanes(F2 x, Fn fn) {
  float a, b;
  f2split(x, a, b);
  return f2(fn(a), fn(b));
}
template <typename Fn>
__device__ __forceinline__ F2 lanes(F2 x, F2 y, Fn fn) {
  float a, b, c, d;
  f2split(x, a, b);
  f2split(y, c, d);
  return f2(fn(a, c), fn(b, d));
}
__device__ __forceinline__ F2 rcp2(F2 x) { return f2(rcp_ftz(x.x), rcp_ftz(x.y)); }

__device__ __forceinline__ F2 symsum3(F2 a0, F2 a1, F2 a2) { return (a0 + a2) + a1; }

// The constants of the packed arithmetic, as pairs.  A packed operation takes its operands from
// register pairs only, and the compiler rebuilds a literal pair with two moves at a use, so a
// kernel makes the constants that are used often once, by an assembly statement that it cannot
// repeat, and carries them in registers; a constant used once scales each lane by an immediate.
struct WenoK {
  F2 m1, m2, m4, c3, c6, k133, eps4, tiny, weps, m13, m10, p10, p5;
};
__device__ __forceinline__ F2 kept(float c) {
  unsigned long long r;
  asm volatile("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(c));
  return make_float2(__uint_as_float((unsigned)r), __uint_as_float((unsigned)(r >> 32)));
}
// both lanes times a literal, as scalar products with an immediate operand
__device__ __forceinline__ F2 scaled(F2 a, float k) { return f2(a.x * k, a.y * k); }
__device__ __forceinline__ WenoK weno_consts() {
  WenoK k;
  k.m1 = kept(-1.0f); k.m2 = kept(-2.0f); k.m4 = kept(-4.0f);
  k.c3 = kept(3.0f); k.c6 = kept(6.0f); k.k133 = kept((float)(13. / 3.)); k.eps4 = kept(4.0f * WenoEps<float>::eps);
  k.tiny = kept(WenoEps<float>::tiny); k.weps = kept(WenoEps<float>::weps);
  k.m13 = kept(-1.3f); k.m10 = kept(-10.0f); k.p10 = kept(10.0f); k.p5 = kept(5.0f);
  return k;
}

// the five-point stencil of two cells: its centre u0, the differences m2 .. p2 of the others to
// it, and the sums s and differences a of opposite ones
struct Sten {
  F2 u0, m2, m1, p1, p2, s1, a1, s2, a2;
};
// u points at the cells' centre values (u[-2..2])
__device__ __forceinline__ Sten stencil_of(const WenoK& K, const F2* u) {
  Sten s;
  s.u0 = u[0];
  s.m2 = ffma2(u[0], K.m1, u[-2]);
  s.m1 = ffma2(u[0], K.m1, u[-1]);
  s.p1 = ffma2(u[0], K.m1, u[1]);
  s.p2 = ffma2(u[0], K.m1, u[2]);
  s.s1 = s.p1 + s.m1;
  s.a1 = ffma2(s.m1, K.m1, s.p1);
  s.s2 = s.p2 + s.m2;
  s.a2 = ffma2(s.m2, K.m1, s.p2);
  return s;
}

__device__ __forceinline__ float fma_sat(float a, float b, float c) {
  float r;
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// limit_weight<float> (0 | ramp to avg | avg | ramp to 1) of ORDER weights w[k] * r at most 1, in
// units of avg: the lower ramp saturated to [0, 1] plus (1 - avg)/avg times the upper one; the
// saturation is part of the multiply-add, where min/max would load the half-rate ALU
template <int ORDER>
__device__ __forceinline__ void limit_weights_f2(F2* w, F2 r) {
  constexpr float avg = 1.0f / (float)ORDER, w1 = 0.2f * avg, w2 = (1.0f - 0.2f) * avg, w3 = (1.0f + 0.2f) * avg,
                  w4 = 1.0f, kl = 1.0f / (w2 - w1), ku = 1.0f / (w4 - w3);
  const float lx = r.x * kl, ly = r.y * kl, ux = r.x * ku, uy = r.y * ku;
#pragma unroll
  for (int k = 0; k < ORDER; k++) {
    const F2 lo = f2(fma_sat(w[k].x, lx, -kl * w1), fma_sat(w[k].y, ly, -kl * w1));
    const F2 up = f2(fma_sat(w[k].x, ux, -ku * w3), fma_sat(w[k].y, uy, -ku * w3));
    w[k] = lo + up;
    if (ORDER == 3) w[k] = w[k] + up;
  }
}

// the smoothness weights 1/t^2 of three stencils up to the common factor (t0 t1 t2)^2, limited,
// in units of avg; b: the regularised measures.  The t sum to one and none is below weps, so the
// largest of the three is at least (weps/3)^2, a normal FP32 number, and a product that
// underflows belongs to a weight below 1e-18 of it, which the limiter sets to zero.
__device__ __forceinline__ void smooth3_f2(const WenoK& K, const F2* b, F2* w) {
  const F2 rb = rcp2(symsum3(b[0], b[1], b[2]));
  const F2 t0 = ffma2(b[0], rb, K.weps), t1 = ffma2(b[1], rb, K.weps), t2 = ffma2(b[2], rb, K.weps);
  const F2 q0 = t1 * t2, q1 = t0 * t2, q2 = t0 * t1;
  w[0] = q0 * q0;
  w[1] = q1 * q1;
  w[2] = q2 * q2;
  limit_weights_f2<3>(w, rcp2(symsum3(w[0], w[1], w[2])));
}

__device__ __forceinline__ float min_abs3(float a, float b, float c) {
  float r;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// smono_indicator<float> of two cells.  Six times the left and right edge derivatives of orders
// 1..3 of the 5-point polynomial, each pair a sum and a difference of the same two terms built
// from the third and fourth differences h, e; the smallest magnitude of a min-mod chain is the
// smallest of all where the signs agree and zero where any differs.
__device__ __forceinline__ F2 smono_indicator_f2(const WenoK& K, const Sten& s, const F2* u) {
  const F2 e = ffma2(K.m4, s.s1, s.s2), h = ffma2(K.m2, s.a1, s.a2), g = scaled(s.s2, 1.5f);
  const F2 z = g + e, y = ffma2(e, K.m1, g), x = s.a1 + s.a2;
  const F2 l1 = ffma2(y, K.m1, x), r1 = x + y;
  const F2 h3 = K.c3 * h;
  const F2 l2 = ffma2(h3, K.m1, z), r2 = z + h3;
  const F2 l3 = K.c3 * ffma2(K.m2, e, h), r3 = ffma2(K.c6, e, h3);
  const F2 dl = K.c6 * ffma2(s.m2, K.m1, s.m1), dr = K.c6 * ffma2(s.p1, K.m1, s.p2);
  auto one = [](float l1, float r1, float l2, float r2, float l3, float r3, float dl, float dr, float cut, bool& part) {
    const unsigned a = __float_as_uint(l1);
    const unsigned differ = (a ^ __float_as_uint(r1)) | (a ^ __float_as_uint(dl)) | (a ^ __float_as_uint(dr)) |
                            (__float_as_uint(l2) ^ __float_as_uint(r2)) | (__float_as_uint(l3) ^ __float_as_uint(r3));
    float v = min_abs3(min_abs3(l1, r1, dl), min_abs3(dr, l2, r2), min_abs3(l3, r3, l3));
    v = ((int)differ < 0) ? 0.0f : v;
    part = part || (v > 0.0f && v < cut);
    return v;
  };
  auto cutoff = [](float u0, float um1, float up1, float um2, float up2) {
    const float norm = fabsf(u0) + ((fabsf(um1) + fabsf(up1)) + (fabsf(um2) + fabsf(up2)));
    return fmaf(norm, 6.0f * WenoEps<float>::smono, 6.0f * WenoEps<float>::tiny);
  };
  const float ca = cutoff(u[0].x, u[-1].x, u[1].x, u[-2].x, u[2].x), cb = cutoff(u[0].y, u[-1].y, u[1].y, u[-2].y, u[2].y);
  bool part = false;
  const float va = one(l1.x, r1.x, l2.x, r2.x, l3.x, r3.x, dl.x, dr.x, ca, part);
  const float vb = one(l1.y, r1.y, l2.y, r2.y, l3.y, r3.y, dl.y, dr.y, cb, part);
  if (part)  // rare: derivatives within 500 epsilons of the stencil's size
    return f2(va < ca ? __fdividef(va, ca) : 1.0f, vb < cb ? __fdividef(vb, cb) : 1.0f);
  return f2(va >= ca ? 1.0f : 0.0f, vb >= cb ? 1.0f : 0.0f);
}

// weno5_cell_weights<float> of two cells: the unoptimised weights blended towards 1/3 by m
// ((1 - m) w + m/3 is w itself for m = 0 and exactly 1/3 for m = 1), skipped when both cells
// are monotone.  The smoothness measures are 4 times the reference's (they are only ever
// normalised by their sum), their regularisation with them; the smallest normal number is
// added to each instead of to their sum, so that a zero line has equal weights.
__device__ __forceinline__ void weno5_cell_weights_f2(const WenoK& K, const Sten& s, const F2* u, F2 m, F2* w) {
  if (m.x == 1.0f && m.y == 1.0f) {
    w[0] = w[1] = w[2] = f2(1.0f / 3.0f);
    return;
  }
  const F2 fd0 = ffma2(K.m4, s.p1, s.p2), fd2 = ffma2(K.m4, s.m1, s.m2);
  const F2 sd0 = ffma2(K.m2, s.p1, s.p2), sd2 = ffma2(K.m2, s.m1, s.m2);
  const F2 normu = ffma2(u[0], u[0], ffma2(u[-1], u[-1], u[1] * u[1]) + ffma2(u[-2], u[-2], u[2] * u[2]));
  const F2 ee = ffma2(normu, K.eps4, K.tiny);
  F2 b[3];
  b[0] = ffma2(K.k133 * sd0, sd0, ffma2(fd0, fd0, ee));
  b[1] = ffma2(K.k133 * s.s1, s.s1, ffma2(s.a1, s.a1, ee));
  b[2] = ffma2(K.k133 * sd2, sd2, ffma2(fd2, fd2, ee));
  smooth3_f2(K, b, w);
  const F2 r = rcp2(symsum3(w[0], w[1], w[2])) * f2(1.0f - m.x, 1.0f - m.y), mt = scaled(m, 1.0f / 3.0f);
#pragma unroll
  for (int k = 0; k < 3; k++) w[k] = ffma2(w[k], r, mt);
}

// weno_frac<float> of two cells from their outer weights and their neighbours' (at distance 2)
// inner ones: the smaller weight ratio on a ramp from 1.3 to 1.6
__device__ __forceinline__ F2 weno_frac_f2(const WenoK& K, F2 w0, F2 w2, F2 wm0, F2 wp2) {
  const F2 el = ffma2(K.m13, wm0, w2), er = ffma2(K.m13, wp2, w0);  // ratio above 1.3 where positive
  const float ea = fminf(el.x, er.x), eb = fminf(el.y, er.y);
  if (fmaxf(ea, eb) > 0.0f) {
    constexpr float E = WenoEps<float>::eps, s = 1.0f / (1.6f - 1.3f);
    const float xa = fminf(el.x * rcp_ftz(wm0.x + E), er.x * rcp_ftz(wp2.x + E));
    const float xb = fminf(el.y * rcp_ftz(wm0.y + E), er.y * rcp_ftz(wp2.y + E));
    return f2(__saturatef(xa * s), __saturatef(xb * s));
  }
  return f2(0.0f);
}

// weno5_edges<float> of two cells from their weights w, final lower-order fractions f and
// SMONO indicators m.  (1 - m) out + m y5 is out for m = 0 and y5 for m = 1 (finite out), so
// the packed code blends both lanes; it skips the WENO sums when both cells are monotone and
// the 5-point values when neither is partly monotone.  Every edge value is the cell's value
// plus a weighted combination of the differences (each stencil's coefficients sum to one), so
// the rounding of the weights' normalisation scales only the offsets: the reconstruction
// carries no bias of that rounding times the value, which a near-steady flow would accumulate
// step after step.  The combinations are 8 (WENO5), 2 (WENO3) and 128 (5-point) times their
// values, the weights 16 and 4 times theirs.
__device__ __forceinline__ void weno5_edges_f2(const WenoK& K, const Sten& s, const F2* u, const F2* w, F2 f, F2 m, F2& yl,
                                               F2& yr) {
  F2 o5l = f2(0.0f), o5r = f2(0.0f);
  if (fmaxf(m.x, m.y) > 0.0f) {
    const F2 a = ffma2(s.s2, K.m1, scaled(s.s1, 20.0f)), c = K.m4 * ffma2(K.m10, s.a1, s.a2);
    constexpr float k = 1.0f / 128.0f;
    const F2 mk = scaled(m, k);
    o5l = ffma2(c, K.m1, a) * mk;  // 60 d-1 - 20 d1 - 5 d-2 + 3 d2, and mirrored
    o5r = (a + c) * mk;
    if (fminf(m.x, m.y) >= 1.0f) {
      yl = s.u0 + o5l;
      yr = s.u0 + o5r;
      return;
    }
  }
  // optimal face weights (1, 10, 5)/16 and mirrored; the stencils' edge values less u_0 are
  // (-10 d1 + 3 d2)/8, (3 d-1 - d1)/8, (-d-2 + 6 d-1)/8
  const F2 w1 = K.p10 * w[1], wl2 = K.p5 * w[2], wr0 = K.p5 * w[0];
  const F2 sl = rcp2((w[0] + w1) + wl2), sr = rcp2((w[2] + w1) + wr0);
  const F2 l0 = ffma2(K.m10, s.p1, K.c3 * s.p2), l1 = ffma2(s.p1, K.m1, K.c3 * s.m1), l2 = ffma2(s.m2, K.m1, K.c6 * s.m1);
  const F2 r0 = ffma2(s.p2, K.m1, K.c6 * s.p1), r1 = ffma2(s.m1, K.m1, K.c3 * s.p1), r2 = ffma2(K.m10, s.m1, K.c3 * s.m2);
  const F2 nl = scaled(sl, 0.125f), nr = scaled(sr, 0.125f);
  F2 outl = ffma2(w1, l1, ffma2(w[0], l0, wl2 * l2)) * nl;
  F2 outr = ffma2(w1, r1, ffma2(w[2], r2, wr0 * r0)) * nr;
  if (fmaxf(f.x, f.y) > 0.0f) {
    // the WENO3 blend: unoptimised weights of the two 2-point stencils, optimal weights (1, 3)/4
    const F2 normu = ffma2(u[0], u[0], ffma2(u[-1], u[-1], u[1] * u[1]));
    const F2 ee = ffma2(normu, f2(WenoEps<float>::eps), K.tiny);
    const F2 b0 = ffma2(s.p1, s.p1, ee), b1 = ffma2(s.m1, s.m1, ee);
    const F2 rb = rcp2(b0 + b1);
    const F2 t0 = ffma2(b0, rb, K.weps), t1 = ffma2(b1, rb, K.weps);
    F2 v[2] = {t1 * t1, t0 * t0};
    limit_weights_f2<2>(v, rcp2(v[0] + v[1]));
    const F2 v0 = K.c3 * v[0], v1 = K.c3 * v[1];
    const F2 nl3 = rcp2(v[0] + v1), nr3 = rcp2(v0 + v[1]);
    // -d1 and d-1 of the left edge, d1 and -d-1 of the right one, each times 1/2
    const F2 t3l = ffma2(v1, s.m1, (v[0] * K.m1) * s.p1) * scaled(nl3, 0.5f);
    const F2 t3r = ffma2(v0, s.p1, (v[1] * K.m1) * s.m1) * scaled(nr3, 0.5f);
    const F2 omf = f2(1.0f - f.x, 1.0f - f.y);
    outl = ffma2(omf, outl, f * t3l);
    outr = ffma2(omf, outr, f * t3r);
  }
  const F2 omm = f2(1.0f - m.x, 1.0f - m.y);
  yl = s.u0 + ffma2(omm, outl, o5l);
  yr = s.u0 + ffma2(omm, outr, o5r);
}

}  // namespace hb
