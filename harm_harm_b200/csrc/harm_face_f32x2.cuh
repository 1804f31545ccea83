// harm_face_f32x2.cuh -- the FP32 face physics with a face's left and right states as the two
// lanes of packed FP32 operations (the same formulas as limit_gamma, get_state, primtoflux,
// vchar of harm_device.cuh and the HLL flux of flux.c:852, vchar.c:34, fluxcompute.c:243).
//
// The stress-energy flux is written as T^d_mu = k1 u_mu - k2 B_mu + delta^d_mu (p + b^2/2) with
//   k1 = w u^d + (B^2 u^d - (u.B) B^d) / (u^0)^2,  k2 = (B^d + (u.B) u^d) / (u^0)^2
// (w without the density for mu = 0, whose rest-mass part rho u^d (1 + u_t) is separate), the
// conserved state with u^0 for u^d and no B^d: two multiply-adds per component.  sqrt(-g) is
// multiplied in once, on the combination of the two states.
#pragma once
#include "harm_weno_f32x2.cuh"

namespace hb {

// the metric fields of one face that its physics reads; ialpha = 1/alpha
struct FaceGeo {
  float g[10];  // g_mu nu
  float n00, n0d, ndd;  // g^00, g^0d, g^dd
  float pert, alpha, ialpha, bsaa, b1, b2, b3, gdet;
};

template <int DIR>
__device__ __forceinline__ void load_face_geo(const float* __restrict__ tab, size_t plane, size_t c, FaceGeo& g) {
#pragma unroll
  for (int f = 0; f < 10; f++) g.g[f] = (f == 8) ? 0.0f : __ldg(tab + (size_t)(HARM_G_GCOV + f) * plane + c);
  g.n00 = __ldg(tab + (size_t)HARM_G_GCON * plane + c);
  g.n0d = __ldg(tab + (size_t)(HARM_G_GCON + sym(0, DIR)) * plane + c);
  g.ndd = __ldg(tab + (size_t)(HARM_G_GCON + sym(DIR, DIR)) * plane + c);
  g.pert = __ldg(tab + (size_t)HARM_G_GCOVPERT_TT * plane + c);
  g.alpha = __ldg(tab + (size_t)HARM_G_ALPHA * plane + c);
  g.ialpha = 1.0f / g.alpha;
  g.bsaa = __ldg(tab + (size_t)HARM_G_BETASQOALPHASQ * plane + c);
  g.b1 = __ldg(tab + (size_t)(HARM_G_BETA + 0) * plane + c);
  g.b2 = __ldg(tab + (size_t)(HARM_G_BETA + 1) * plane + c);
  g.b3 = __ldg(tab + (size_t)(HARM_G_BETA + 2) * plane + c);
  g.gdet = __ldg(tab + (size_t)HARM_G_GDET * plane + c);
}

__device__ __forceinline__ F2 neg2(F2 a) { return a * f2(-1.0f); }
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float sqrt_ftz(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// g_ij U^i U^j of the two states (g_23 = 0 in these coordinates)
__device__ __forceinline__ F2 qsq_f2(const FaceGeo& g, F2 u1, F2 u2, F2 u3) {
  const F2 t = ffma2(f2(g.g[5]), u2, f2(g.g[6]) * u3);
  const F2 a = ffma2(f2(g.g[4]) * u1, u1, (u1 * f2(2.0f)) * t);
  return ffma2(f2(g.g[7]) * u2, u2, ffma2(f2(g.g[9]) * u3, u3, a));
}

// HLL (laxf: LAXF) flux of one face from its states pl, pr into F (times sqrt(-g)); returns
// ctop, the larger of the two wave speeds
template <int DIR>
__device__ __forceinline__ float face_flux_f2(const FaceGeo& g, const float* pl, const float* pr, float gam, float gmax,
                                              int laxf, float* F) {
  const F2 rho = f2(pl[HARM_RHO], pr[HARM_RHO]), uu = f2(pl[HARM_UU], pr[HARM_UU]);
  F2 U[3], B[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    U[i] = f2(pl[HARM_U1 + i], pr[HARM_U1 + i]);
    B[i] = f2(pl[HARM_B1 + i], pr[HARM_B1 + i]);
  }
  const float bd = 0.5f * (pl[HARM_B1 + DIR - 1] + pr[HARM_B1 + DIR - 1]);
  B[DIR - 1] = f2(bd);
  F2 q = qsq_f2(g, U[0], U[1], U[2]);
  q = f2(fmaxf(q.x, 0.0f), fmaxf(q.y, 0.0f));
  const float qmax = gmax * gmax - 1.0f;
  if (gmax > 1.0f && (q.x > qmax || q.y > qmax)) {  // limit_gamma, rare
    const F2 f = f2(q.x > qmax ? sqrtf(qmax / q.x) : 1.0f, q.y > qmax ? sqrtf(qmax / q.y) : 1.0f);
#pragma unroll
    for (int i = 0; i < 3; i++) U[i] = U[i] * f;
    q = qsq_f2(g, U[0], U[1], U[2]);
    q = f2(fmaxf(q.x, 0.0f), fmaxf(q.y, 0.0f));
  }
  // u^mu, u_mu, 1 + u_t
  const F2 g2 = f2(1.0f) + q, rs = f2(rsqrt_ftz(g2.x), rsqrt_ftz(g2.y));
  // gamma and u^0 to their last bit, each by one correction from its remainder: every component
  // of u^mu carries u^0's rounding, coherently
  const F2 gs = g2 * rs, gamma = ffma2(ffma2(neg2(gs), gs, g2), rs * f2(0.5f), gs);
  const F2 us = gamma * f2(g.ialpha), u0 = ffma2(ffma2(us, f2(-g.alpha), gamma), f2(g.ialpha), us);
  const F2 iu0 = rs * f2(g.alpha), ig2 = iu0 * iu0;
  const F2 mu0 = neg2(u0);
  const F2 u[4] = {u0, ffma2(mu0, f2(g.b1), U[0]), ffma2(mu0, f2(g.b2), U[1]), ffma2(mu0, f2(g.b3), U[2])};
  const F2 ut = ffma2(U[0], f2(g.g[1]), ffma2(U[1], f2(g.g[2]), U[2] * f2(g.g[3])));
  const float alphasq = g.alpha * g.alpha;
  const F2 onep = ffma2(ffma2(f2(-alphasq), f2(g.bsaa) + q, f2(g.pert)), rcp2(ffma2(gamma, f2(g.alpha), f2(1.0f))), ut);
  // the normal observer has no covariant spatial components, so u_i = g_ij U^j; lowering u^mu
  // would cancel g_0i u^0 against it, and leave the rounding of the larger terms in slow flow
  const F2 d0 = onep + f2(-1.0f);
  const F2 d1 = ffma2(f2(g.g[4]), U[0], ffma2(f2(g.g[5]), U[1], f2(g.g[6]) * U[2]));
  const F2 d2 = ffma2(f2(g.g[5]), U[0], f2(g.g[7]) * U[1]);
  const F2 d3 = ffma2(f2(g.g[6]), U[0], f2(g.g[9]) * U[2]);
  const F2 dv[4] = {d0, d1, d2, d3};
  // B_mu, B^2, u.B, b^2
  F2 Bc[4];
  Bc[0] = ffma2(B[0], f2(g.g[1]), ffma2(B[1], f2(g.g[2]), B[2] * f2(g.g[3])));
  Bc[1] = ffma2(B[0], f2(g.g[4]), ffma2(B[1], f2(g.g[5]), B[2] * f2(g.g[6])));
  Bc[2] = ffma2(B[0], f2(g.g[5]), B[1] * f2(g.g[7]));
  Bc[3] = ffma2(B[0], f2(g.g[6]), B[2] * f2(g.g[9]));
  const F2 Bsq = ffma2(B[0], Bc[1], ffma2(B[1], Bc[2], B[2] * Bc[3]));
  const F2 uB = ffma2(B[0], d1, ffma2(B[1], d2, B[2] * d3));
  const F2 bsq = ffma2(uB, uB, Bsq) * ig2;
  const F2 P = f2(gam - 1.0f) * uu, Pu = P + uu;
  const F2 ptot = ffma2(f2(0.5f), bsq, P);
  // wave speeds (vchar.c:34, simplefast :260)
  float cmax = 0.0f, cmin = 0.0f;
  {
    constexpr float small = Eps<float>::small, eps = Eps<float>::eps;
    const F2 up = f2(fmaxf(uu.x, 0.0f), fmaxf(uu.y, 0.0f));
    const F2 rp = f2(rho.x < 0.0f ? small : rho.x, rho.y < 0.0f ? small : rho.y);
    const F2 pp = f2(gam - 1.0f) * up, h = (rp + up) + pp;
    F2 W = (rp + up) + P;
    F2 cs2 = (f2(gam) * pp) * rcp2(h);
    cs2 = f2(W.x > 0.0f ? fminf(fmaxf(cs2.x, small), 1.0f - eps * 10.0f) : small,
             W.y > 0.0f ? fminf(fmaxf(cs2.y, small), 1.0f - eps * 10.0f) : small);
    W = f2(W.x > 0.0f ? W.x : small, W.y > 0.0f ? W.y : small);
    const F2 e = bsq + W;
    const F2 va2 = bsq * rcp2(f2(small + fabsf(e.x), small + fabsf(e.y)));
    F2 c2 = ffma2(neg2(cs2), va2, cs2 + va2);
    auto clamp = [&](float c, float sum, float r) {
      if (c < 0.0f && c / sum > -eps * 100.0f) c = 0.0f;
      if (c > 1.0f && (c < 1.0f + eps * 100.0f || r < 0.0f)) c = 1.0f;
      return c;
    };
    if (c2.x < 0.0f || c2.x > 1.0f || c2.y < 0.0f || c2.y > 1.0f)  // rare
      c2 = f2(clamp(c2.x, cs2.x + va2.x, rp.x), clamp(c2.y, cs2.y + va2.y, rp.y));
    const float AA = g.ndd, BB = g.n00, AB = g.n0d;
    const F2 ud = u[DIR], omc = f2(1.0f) - c2, AuBu = ud * u0;
    const F2 hb = ffma2(AuBu, omc, f2(-AB) * c2);                 // half of vchar.c's B
    const F2 a = ffma2(u0 * u0, omc, f2(-BB) * c2);
    const F2 x = ffma2(f2(2.0f * AB), AuBu, ffma2(f2(-AA) * u0, u0, (f2(-BB) * ud) * ud));
    const F2 disc = c2 * ffma2(f2(AB * AB - AA * BB), c2, neg2(x * omc));  // a quarter of its discriminant
    const F2 rt = f2(sqrt_ftz(fmaxf(disc.x, 0.0f)), sqrt_ftz(fmaxf(disc.y, 0.0f)));
    const F2 ia = rcp2(a);
    const F2 vp = (hb + rt) * ia, vm = (hb - rt) * ia;
    cmax = fmaxf(fmaxf(fmaxf(vp.x, vm.x), fmaxf(vp.y, vm.y)), 0.0f);
    cmin = fmaxf(-fminf(fminf(vp.x, vm.x), fminf(vp.y, vm.y)), 0.0f);
  }
  const float ctop = fmaxf(cmax, cmin);
  // F = Fr + ca (Fl - Fr) + cc (Ul - Ur): the rounding of the weights scales only the jump
  // between the two states, which is small where the flow is smooth
  float ca = 0.5f, cc = 0.5f * ctop;
  if (!laxf && cmax + cmin != 0.0f) {
    ca = cmax / (cmax + cmin);
    cc = ca * cmin;
  }
  const F2 ud = u[DIR];
  const F2 em = ffma2(Bsq, ud, neg2(uB) * f2(bd)) * ig2;
  const F2 k1 = ffma2(Pu + rho, ud, em), k1e = ffma2(Pu, ud, em), k2 = ffma2(uB, ud, f2(bd)) * ig2;
  const F2 et = Bsq * iu0;
  const F2 c1 = ffma2(Pu + rho, u0, et), c1e = ffma2(Pu, u0, et), c2 = uB * iu0;
  const F2 rud = rho * ud, ru0 = rho * u0;
  auto put = [&](int p, F2 f, F2 c) {
    F[p] = g.gdet * fmaf(ca, f.x - f.y, fmaf(cc, c.x - c.y, f.y));
  };
  put(HARM_RHO, rud, ru0);
  {
    const F2 f = ffma2(rud, onep, ffma2(k1e, d0, neg2(k2) * Bc[0]));
    const F2 c = ffma2(ru0, onep, ffma2(c1e, d0, neg2(c2) * Bc[0])) + ptot;
    put(HARM_UU, f, c);
  }
#pragma unroll
  for (int i = 1; i <= 3; i++) {
    F2 f = ffma2(k1, dv[i], neg2(k2) * Bc[i]);
    if (i == DIR) f = f + ptot;
    put(HARM_UU + i, f, ffma2(c1, dv[i], neg2(c2) * Bc[i]));
  }
#pragma unroll
  for (int i = 1; i <= 3; i++) {
    if (i == DIR) put(HARM_B1 + i - 1, f2(0.0f), B[i - 1]);
    else put(HARM_B1 + i - 1, ffma2(B[i - 1], ud, neg2(f2(bd) * u[i])) * iu0, B[i - 1]);
  }
  return ctop;
}

// the minimum of cour dx / ctop over the faces whose largest finite ctop is given (division is
// monotone), as a block: one atomicMin on the bits of the double
__device__ __forceinline__ void block_dt_atomic(double ctop, double cour_dx, unsigned long long* slot) {
  __shared__ double red[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ctop = fmax(ctop, __shfl_xor_sync(0xffffffffu, ctop, o));
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) red[w] = ctop;
  __syncthreads();
  if (w == 0) {
    double v = (lane < (int)(blockDim.x >> 5)) ? red[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    const double dt = cour_dx / v;
    if (lane == 0 && dt < 1.e300) atomicMin(slot, (unsigned long long)__double_as_longlong(dt));
  }
}

}  // namespace hb
