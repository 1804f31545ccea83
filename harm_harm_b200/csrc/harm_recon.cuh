// harm_recon.cuh -- the flux stage of one direction as two kernels: k_recon, the left and right
// edge value of every primitive in every cell, and k_face, the face states' physics.
//
// Along x2 and x3 k_recon marches: a thread owns one primitive on one line (FP64) or on two
// lines (FP32, the two lanes of the packed operations), holds its stencil and the weights of the
// cells around it in registers, and reads each value from memory once.  A warp is one primitive
// on 32 or 64 lines with neighbouring i, so every access is coalesced.
// Along x1 (k_recon_x1) a warp is one primitive on 64 consecutive cells of a line, two to a
// lane; neighbours' values and weights go through rows of shared memory private to the warp.
// What bounds both is arithmetic (FP32: the ALU and FMA pipes; FP64: the FP64 pipe and its
// latency), so each cell's weights are computed once: a tile of 32 faces staged in shared
// memory (k_fluxt) computes 40 cells' for 33, spends as much again on indexing and moves every
// weight through shared memory.  The edge values cost a round trip through memory that the
// arithmetic hides.  The warps of a block are one primitive: a primitive whose lines take a
// slower path (zero lines, steep ones) holds up no other's.
// Flux stage of a substep (EMFs included) against the tiles it replaces: FP32 WENO5 at 256x128x64
// 1214 -> 756 us (recon 143 + 161 + 166, faces 3 x 48, cell pass and coefficients 97), FP64 WENO5 at
// 192x96x64 3550 -> 1412 us, FP32 PARALINE at 192x96x64 404 -> 337 us; with the three directions in
// joint launches FP32 WENO5 at 120x72x40 287 -> 195 us (212 with separate ones).
#pragma once
#include "harm_common.cuh"
#include "harm_face_f32x2.cuh"

// ------------------------------------------------------------------ k_recon

// The cells whose edges are wanted (extended indices): c0 .. c1 along the direction, and the
// lines (t, o), t = t0 .. t0+nt-1 fastest (i for x2 and x3, j for x1) and o = o0 .. (k, or j for
// x3); lines are numbered t fastest.  chunk: edge cells per thread.
struct ReconBox {
  int c0, c1, t0, nt, o0, nlines, chunk;
};

// n / d for 0 <= n < 2^31 by one multiplication: m = floor(2^(31+s) / d) + 1 with
// 2^(s-1) < d <= 2^s (T. Granlund and P. Montgomery, PLDI 1994)
struct FastDiv {
  unsigned m, s, d;
};
static inline FastDiv fast_div(unsigned d) {
  FastDiv f;
  f.d = d;
  f.s = 0;
  while ((1ull << f.s) < d) f.s++;
  f.m = (unsigned)((1ull << (31 + f.s)) / d + 1);
  if (d == 1) f.m = 0x80000001u;
  return f;
}
__device__ __forceinline__ unsigned operator/(unsigned n, const FastDiv& f) {
  return (unsigned)(((unsigned long long)n * f.m) >> (31 + f.s));
}

template <typename T>
struct ReconLanes;
template <>
struct ReconLanes<double> {
  using V = double;
  static constexpr int N = 1;
};
template <>
struct ReconLanes<float> {
  using V = F2;
  static constexpr int N = 2;
};

// cells past an edge cell that its edges need, and the length of the window that holds them
template <int LIM>
struct ReconWin {
  static constexpr int D = (LIM == HARM_LIM_WENO5) ? 5 : (LIM == HARM_LIM_MC) ? 1 : 2;
  static constexpr int W = (LIM == HARM_LIM_WENO5) ? 8 : 2 * D + 1;
  static constexpr bool S = (LIM == HARM_LIM_WENO5 || LIM == HARM_LIM_PARALINE);  // a per-cell coefficient
  static constexpr int R = (LIM == HARM_LIM_PARALINE) ? 3 : D;  // the reach of edges and coefficient
};

// edges of the cell at y[0] by the limiters that need no weights
template <int LIM>
__device__ __forceinline__ void simple_edges(const double* y, double s, double& l, double& r) {
  if constexpr (LIM == HARM_LIM_PARA) para4_cell<double>(y, l, r);
  else if constexpr (LIM == HARM_LIM_PARALINE) paraline_cell<double>(y, s, l, r);
  else {
    const double dq = mc_slope(y[-1], y[0], y[1]);
    l = y[0] - 0.5 * dq;
    r = y[0] + 0.5 * dq;
  }
}
template <int LIM>
__device__ __forceinline__ void simple_edges(const F2* y, F2 s, F2& l, F2& r) {
  constexpr int D = ReconWin<LIM>::D;
  float a[2 * D + 1], b[2 * D + 1], la, lb, ra, rb;
#pragma unroll
  for (int q = -D; q <= D; q++) f2split(y[q], a[q + D], b[q + D]);
  if constexpr (LIM == HARM_LIM_PARA) {
    para4_cell<float>(a + D, la, ra);
    para4_cell<float>(b + D, lb, rb);
  } else if constexpr (LIM == HARM_LIM_PARALINE) {
    paraline_cell<float>(a + D, s.x, la, ra);
    paraline_cell<float>(b + D, s.y, lb, rb);
  } else {
    const float qa = mc_slope(a[0], a[1], a[2]), qb = mc_slope(b[0], b[1], b[2]);
    la = a[1] - 0.5f * qa; ra = a[1] + 0.5f * qa;
    lb = b[1] - 0.5f * qb; rb = b[1] + 0.5f * qb;
  }
  l = f2(la, lb);
  r = f2(ra, rb);
}

// WENO5BND along a line: the weights of the newest cells, their lower-order fractions, and the
// edges of the cell five behind the newest.  u[0..7]: the newest eight cells (u[7] the newest,
// n); w, m: weights and SMONO indicators of n-5 .. n-2; wz: the first weight of n-6; f: the
// fractions of n-6 .. n-4.
template <typename V>
struct WenoLine {
  V u[8], w[4][3], m[4], wz, f[3];
};

struct NoConsts {};
template <int LIM, typename T>
__device__ __forceinline__ auto recon_consts() {
  if constexpr (LIM == HARM_LIM_WENO5 && sizeof(T) == 4) return weno_consts();
  else return NoConsts{};
}
__device__ __forceinline__ void weno_new_weights(const NoConsts&, WenoLine<double>& s) {
  s.m[3] = smono_indicator<double>(s.u + 5);
  weno5_cell_weights<double>(s.u + 5, s.m[3], s.w[3]);
}
__device__ __forceinline__ void weno_new_weights(const WenoK& K, WenoLine<F2>& s) {
  const Sten st = stencil_of(K, s.u + 5);
  s.m[3] = smono_indicator_f2(K, st, s.u + 5);
  weno5_cell_weights_f2(K, st, s.u + 5, s.m[3], s.w[3]);
}
__device__ __forceinline__ void weno_new_frac(const NoConsts&, WenoLine<double>& s) {
  const double wm[3] = {s.wz, 0.0, 0.0}, wp[3] = {0.0, 0.0, s.w[3][2]};
  s.f[2] = weno_frac<double>(s.w[1], wm, wp);
}
__device__ __forceinline__ void weno_new_frac(const WenoK& K, WenoLine<F2>& s) {
  s.f[2] = weno_frac_f2(K, s.w[1][0], s.w[1][2], s.wz, s.w[3][2]);
}
__device__ __forceinline__ void weno_line_edges(const NoConsts&, const WenoLine<double>& s, double ss, double& l, double& r) {
  double f = s.f[1];
  if (ss > 0.0) f = weno_lof<double>(f, s.f[0], s.f[2], ss);
  weno5_edges<double>(s.u + 2, s.w[0], f, s.m[0], l, r);
}
__device__ __forceinline__ void weno_line_edges(const WenoK& K, const WenoLine<F2>& s, F2 ss, F2& l, F2& r) {
  F2 f = s.f[1];
  if (ss.x > 0.0f) f.x = weno_lof<float>(f.x, s.f[0].x, s.f[2].x, ss.x);  // rare: a jump above 0.25
  if (ss.y > 0.0f) f.y = weno_lof<float>(f.y, s.f[0].y, s.f[2].y, ss.y);
  weno5_edges_f2(K, stencil_of(K, s.u + 2), s.u + 2, s.w[0], f, s.m[0], l, r);
}

// The window of one line: fill takes the first 2D cells of a chunk, step the next one, after which
// l and r are the edges of the cell D behind it (s: its coefficient).
template <int LIM, typename V>
struct ReconLine {
  V u[ReconWin<LIM>::W];
  template <typename C>
  __device__ __forceinline__ void fill(const C&, V v, int) {
    constexpr int W = ReconWin<LIM>::W;
#pragma unroll
    for (int q = 0; q + 1 < W; q++) u[q] = u[q + 1];
    u[W - 1] = v;
  }
  template <typename C>
  __device__ __forceinline__ void step(const C& K, V v, V s, V& l, V& r) {
    fill(K, v, 0);
    simple_edges<LIM>(u + ReconWin<LIM>::W / 2, s, l, r);
  }
};
template <typename V>
struct ReconLine<HARM_LIM_WENO5, V> {
  WenoLine<V> a;
  template <typename C>
  __device__ __forceinline__ void weights(const C& K, V v) {
#pragma unroll
    for (int q = 0; q < 7; q++) a.u[q] = a.u[q + 1];
    a.u[7] = v;
    a.wz = a.w[0][0];
#pragma unroll
    for (int q = 0; q < 3; q++) {
#pragma unroll
      for (int k = 0; k < 3; k++) a.w[q][k] = a.w[q + 1][k];
      a.m[q] = a.m[q + 1];
    }
    weno_new_weights(K, a);
  }
  template <typename C>
  __device__ __forceinline__ void frac(const C& K) {
    a.f[0] = a.f[1];
    a.f[1] = a.f[2];
    weno_new_frac(K, a);
  }
  // n: cells taken before this one (the weights need five, the fractions four cells' weights)
  template <typename C>
  __device__ __forceinline__ void fill(const C& K, V v, int n) {
    if (n < 4) {
#pragma unroll
      for (int q = 0; q < 7; q++) a.u[q] = a.u[q + 1];
      a.u[7] = v;
      return;
    }
    weights(K, v);
    if (n >= 8) frac(K);
  }
  template <typename C>
  __device__ __forceinline__ void step(const C& K, V v, V s, V& l, V& r) {
    weights(K, v);
    frac(K);
    weno_line_edges(K, a, s, l, r);
  }
};

// Warps per block and blocks per SM the marching kernel is compiled for.  FP32: 4 (the window of
// WENO5, 56 registers beside its temporaries, fits 128 without spills; 5 spill, and a full step at
// 256x128x64 takes 3095 us instead of 2867; 3 are the same).  FP64: 5 (102 registers with a few
// spills, 25 % more warps to hide the divisions: 330 us a direction at 192x96x64 against 350 at 4).
constexpr int kReconWarps = 4;
template <typename T>
constexpr int kReconBlocks = sizeof(T) == 4 ? 4 : 5;
// steps unrolled: an unrolled loop saves moves and misses the instruction cache (FP32 WENO5 at
// 256x128x64, full step: 1 step 2861 us, 2 2821, 4 2867, 8 3320; FP64's step is long)
template <typename T>
constexpr int kReconUnroll = sizeof(T) == 4 ? 2 : 1;

// CLAMP: for fewer ghost zones than the stencil reaches (recon_narrow); cells beyond the grid are
// the grid's last one in that direction.  It serves x1 too, whose rows have no ends to stop at.
template <int DIR, int LIM, typename T, bool CLAMP>
__device__ __forceinline__ void recon_march(const Dims& d, const ReconBox& rb, const double* __restrict__ P,
                                            const T* __restrict__ S, T* __restrict__ EL, T* __restrict__ ER, int group,
                                            int chunk, int prim) {
  static_assert(DIR != 1 || CLAMP, "x1: k_recon_x1");
  using V = typename ReconLanes<T>::V;
  constexpr int N = ReconLanes<T>::N, D = ReconWin<LIM>::D;
  constexpr bool HAS_S = ReconWin<LIM>::S;
  const int lane = threadIdx.x & 31;
  const int line0 = (group * kReconWarps + (int)(threadIdx.x >> 5)) * 32 * N;
  if (line0 >= rb.nlines) return;
  const int a = rb.c0 + chunk * rb.chunk, b = min(a + rb.chunk - 1, rb.c1);
  const unsigned stride = (DIR == 1) ? 1u : (DIR == 2) ? (unsigned)d.n1e : (unsigned)d.plane;
  [[maybe_unused]] const int cells_along = (DIR == 1) ? d.n1e : (DIR == 2) ? d.n2e : d.n3e;
  const double* Pp = P + (size_t)prim * d.cells;
  T* el = EL + (size_t)prim * d.cells;
  T* er = ER + (size_t)prim * d.cells;
  // offset within one primitive of the newest cell of each line (lines past the last repeat it)
  unsigned at[N];
#pragma unroll
  for (int q = 0; q < N; q++) {
    const int l = min(line0 + 32 * q + lane, rb.nlines - 1);
    const unsigned t = rb.t0 + l % rb.nt, o = rb.o0 + l / rb.nt;
    const unsigned first = (DIR == 1) ? o * (unsigned)d.plane + t * (unsigned)d.n1e
                         : (DIR == 2) ? o * (unsigned)d.plane + t : o * (unsigned)d.n1e + t;
    at[q] = first + (unsigned)(a - D) * stride;
  }
  // the value at cell c of line q, whose offset is at[q]
  auto value = [&](int q, int c) -> double {
    if constexpr (CLAMP) return __ldg(Pp + (at[q] + (unsigned)(min(max(c, 0), cells_along - 1) - c) * stride));
    else return __ldg(Pp + at[q]);
  };
  const bool ok0 = line0 + lane < rb.nlines, ok1 = N == 2 && line0 + 32 + lane < rb.nlines;
  const auto K = recon_consts<LIM, T>();
  ReconLine<LIM, V> ln;
  // Loads run ahead: a cell's values two steps, its coefficient one (a step is shorter than the
  // memory's latency times the warps that share the scheduler).
  const int last = b + D;  // the chunk's last cell
  int cell = a - D;        // the newest loaded cell
  double nx[2][N];
#pragma unroll
  for (int q = 0; q < N; q++) {
    nx[0][q] = value(q, cell);
    at[q] += stride;
    nx[1][q] = value(q, cell + 1);
  }
  cell++;
  // takes the next cell and loads the one two after it
  auto next = [&]() -> V {
    V v;
    if constexpr (N == 2) v = f2((float)nx[0][0], (float)nx[0][1]);
    else v = nx[0][0];
    const bool more = cell < last;
    cell++;
#pragma unroll
    for (int q = 0; q < N; q++) {
      nx[0][q] = nx[1][q];
      at[q] += stride;
      if (more) nx[1][q] = value(q, cell);
    }
    return v;
  };
#pragma unroll 1
  for (int n = 0; n < 2 * D; n++) ln.fill(K, next(), n);
  // the steady loop has no conditions on its position, so that the window's shifts become
  // renamings (with them, moves were 30 % of its instructions)
  constexpr int U = kReconUnroll<T>;
  V sn{};
  unsigned c0 = at[0] - (unsigned)(D + 1) * stride, c1 = at[N - 1] - (unsigned)(D + 1) * stride;  // the edge cell
  auto coef = [&]() -> V {
    if constexpr (N == 2) return f2(__ldg(S + c0), __ldg(S + c1));
    else return __ldg(S + c0);
  };
  if constexpr (HAS_S) sn = coef();
#pragma unroll 1
  for (int c = a; c <= b; c += U) {
#pragma unroll
    for (int q = 0; q < U; q++) {
      const bool in = U == 1 || c + q <= b;
      const V s = sn;
      const unsigned e0 = c0, e1 = c1;
      c0 += stride;
      c1 += stride;
      if (HAS_S && c + q < b) sn = coef();
      V l, r;
      ln.step(K, next(), s, l, r);
      if constexpr (N == 2) {
        if (ok0 && in) { el[e0] = l.x; er[e0] = r.x; }
        if (ok1 && in) { el[e1] = l.y; er[e1] = r.y; }
      } else {
        if (ok0 && in) { el[e0] = l; er[e0] = r; }
      }
    }
  }
}

template <int DIR, int LIM, typename T, bool CLAMP = false, int TU = HARM_TU>
__global__ void __launch_bounds__(32 * kReconWarps, kReconBlocks<T>) k_recon(Dims d, ReconBox rb, const double* __restrict__ P,
                                                                             const T* __restrict__ S, T* __restrict__ EL,
                                                                             T* __restrict__ ER) {
  recon_march<DIR, LIM, T, CLAMP>(d, rb, P, S, EL, ER, blockIdx.x, blockIdx.y, blockIdx.z);
}

// x1: the rows of a plane's lines are one contiguous range of memory, ghost cells included; a warp
// takes segments of 64 of its cells (positions), wherever rows end in them: the edges of ghost
// cells beyond c0 .. c1 are computed from whatever is next to them and never read.  WENO5: the
// weights of all 64 positions and the edges of those whose neighbours' weights (at distance 3 at
// most) are among them, otherwise the edges of all.  Each lane has positions `lane` and
// `lane + 32`.  (Segments of single lines left up to a third of the last one's lanes idle, and
// cost two integer divisions each.)
template <int LIM>
struct ReconRow {
  static constexpr int M = (LIM == HARM_LIM_WENO5) ? 3 : 0;  // positions without edges at either end
  static constexpr int H = (LIM == HARM_LIM_MC) ? 1 : 2;     // stencil half width
  static constexpr int E = 64 - 2 * M;                        // edge cells per segment
};
constexpr int kRowWarps = 8;
// FP64: 3 blocks per SM (80 registers; left to itself 94 and 2 blocks, 330 us against 299 at
// 192x96x64)
template <typename T>
constexpr int kRowBlocks = sizeof(T) == 4 ? 1 : 3;
template <typename T>
struct ReconRowSmem {
  T u[68];
  T w0[64], w2[64], f[64];
};

// the segments it, it + nw, ... of the box
template <int LIM, typename T>
__device__ __forceinline__ void recon_rows(const Dims& d, const ReconBox& rb, const FastDiv& dseg,
                                           const double* __restrict__ P, const T* __restrict__ S, T* __restrict__ EL,
                                           T* __restrict__ ER, ReconRowSmem<T>& w, int it, int nw, int prim) {
  using R = ReconRow<LIM>;
  constexpr int H = R::H, M = R::M;
  constexpr bool HAS_S = ReconWin<LIM>::S;
  const int lane = threadIdx.x & 31;
  const double* Pp = P + (size_t)prim * d.cells;
  T* el = EL + (size_t)prim * d.cells;
  T* er = ER + (size_t)prim * d.cells;
  const int items = rb.nlines / rb.nt * (int)dseg.d;  // segments of the box
  const unsigned plane = (unsigned)d.plane, row0 = (unsigned)rb.t0 * (unsigned)d.n1e;
  const unsigned ncell = (unsigned)rb.nt * (unsigned)d.n1e, top = (unsigned)d.cells - 1u;
  double nx[3];
  unsigned nb = 0, nend = 0;  // position 0 of the loaded segment, and the end of its plane's range
  auto load = [&](int q) {    // cells nb - H .. nb + 63 + H (those past the array repeat its last)
    const unsigned o = (unsigned)q / dseg, sg = (unsigned)q - o * dseg.d;
    const unsigned first = ((unsigned)rb.o0 + o) * plane + row0;
    nb = first + sg * (unsigned)R::E - (unsigned)M;
    nend = first + ncell;
#pragma unroll
    for (int k = 0; k < 3; k++)
      if (k < 2 || lane < 2 * H) nx[k] = __ldg(Pp + min(nb - (unsigned)H + (unsigned)(lane + 32 * k), top));
  };
  [[maybe_unused]] const auto K = recon_consts<LIM, T>();
  if (it < items) load(it);
  for (; it < items; it += nw) {
    const unsigned c0 = nb + (unsigned)lane, c1 = c0 + 32u, end = nend;
    __syncwarp();
    w.u[lane] = (T)nx[0];
    w.u[lane + 32] = (T)nx[1];
    if (lane < 2 * H) w.u[lane + 64] = (T)nx[2];
    if (it + nw < items) load(it + nw);
    __syncwarp();
    const int x0 = lane, x1 = lane + 32;
    const bool e0 = x0 >= M && c0 < end, e1 = x1 < 64 - M && c1 < end;
    T l0, r0, l1, r1;
    if constexpr (sizeof(T) == 4) {
      F2 u[2 * H + 1], l, r;
#pragma unroll
      for (int q = 0; q <= 2 * H; q++) u[q] = f2((float)w.u[x0 + q], (float)w.u[x1 + q]);
      F2 s = f2(0.0f);
      if (HAS_S) s = f2(e0 ? (float)__ldg(S + c0) : 0.0f, e1 ? (float)__ldg(S + c1) : 0.0f);
      if constexpr (LIM == HARM_LIM_WENO5) {
        const Sten st = stencil_of(K, u + 2);
        F2 wt[3];
        const F2 m = smono_indicator_f2(K, st, u + 2);
        weno5_cell_weights_f2(K, st, u + 2, m, wt);
        w.w0[x0] = wt[0].x; w.w0[x1] = wt[0].y;
        w.w2[x0] = wt[2].x; w.w2[x1] = wt[2].y;
        __syncwarp();
        // positions 2 .. 61 have both neighbours at distance 2
        const F2 wm = f2(w.w0[max(x0 - 2, 0)], w.w0[x1 - 2]), wp = f2(w.w2[x0 + 2], w.w2[min(x1 + 2, 63)]);
        F2 f = weno_frac_f2(K, wt[0], wt[2], wm, wp);
        const bool jump = (e0 && s.x > 0.0f) || (e1 && s.y > 0.0f);
        if (__any_sync(0xffffffffu, jump)) {
          w.f[x0] = f.x; w.f[x1] = f.y;
          __syncwarp();
          if (e0 && s.x > 0.0f) f.x = weno_lof<float>(f.x, w.f[x0 - 1], w.f[x0 + 1], s.x);
          if (e1 && s.y > 0.0f) f.y = weno_lof<float>(f.y, w.f[x1 - 1], w.f[x1 + 1], s.y);
        }
        weno5_edges_f2(K, st, u + 2, wt, f, m, l, r);
      } else {
        simple_edges<LIM>(u + H, s, l, r);
      }
      l0 = l.x; l1 = l.y; r0 = r.x; r1 = r.y;
    } else if constexpr (LIM == HARM_LIM_WENO5) {
      T u[2][5], wt[2][3], m[2], f[2], ll[2], rr[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int x = lane + 32 * h;
#pragma unroll
        for (int q = 0; q < 5; q++) u[h][q] = w.u[x + q];
        m[h] = smono_indicator<T>(u[h] + 2);
        weno5_cell_weights<T>(u[h] + 2, m[h], wt[h]);
        w.w0[x] = wt[h][0];
        w.w2[x] = wt[h][2];
      }
      __syncwarp();
      bool jump = false;
      T s[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int x = lane + 32 * h;
        const T wm[3] = {w.w0[max(x - 2, 0)], T(0), T(0)}, wp[3] = {T(0), T(0), w.w2[min(x + 2, 63)]};
        f[h] = weno_frac<T>(wt[h], wm, wp);
        s[h] = (h ? e1 : e0) ? __ldg(S + (h ? c1 : c0)) : T(0);
        jump = jump || s[h] > T(0);
      }
      if (__any_sync(0xffffffffu, jump)) {
        w.f[x0] = f[0];
        w.f[x1] = f[1];
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int x = lane + 32 * h;
          if (s[h] > T(0)) f[h] = weno_lof<T>(f[h], w.f[x - 1], w.f[x + 1], s[h]);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; h++) weno5_edges<T>(u[h] + 2, wt[h], f[h], m[h], ll[h], rr[h]);
      l0 = ll[0]; l1 = ll[1]; r0 = rr[0]; r1 = rr[1];
    } else {
      T u[2 * H + 1];
#pragma unroll
      for (int q = 0; q <= 2 * H; q++) u[q] = w.u[x0 + q];
      simple_edges<LIM>(u + H, (HAS_S && e0) ? __ldg(S + c0) : T(0), l0, r0);
#pragma unroll
      for (int q = 0; q <= 2 * H; q++) u[q] = w.u[x1 + q];
      simple_edges<LIM>(u + H, (HAS_S && e1) ? __ldg(S + c1) : T(0), l1, r1);
    }
    if (e0) { el[c0] = l0; er[c0] = r0; }
    if (e1) { el[c1] = l1; er[c1] = r1; }
  }
}

template <int LIM, typename T, int TU = HARM_TU>
__global__ void __launch_bounds__(32 * kRowWarps, kRowBlocks<T>) k_recon_x1(Dims d, ReconBox rb, FastDiv dseg,
                                                             const double* __restrict__ P,
                                                             const T* __restrict__ S, T* __restrict__ EL,
                                                             T* __restrict__ ER) {
  __shared__ ReconRowSmem<T> rows[kRowWarps];
  const int warp = threadIdx.x >> 5;
  recon_rows<LIM, T>(d, rb, dseg, P, S, EL, ER, rows[warp], (int)blockIdx.x * kRowWarps + warp, (int)gridDim.x * kRowWarps,
                     blockIdx.z);
}

// ------------------------------------------------------------------ per-cell coefficients

// S of direction DIR for edge cell t of a ReconBox, from the cell pass L (k_cellprep): the
// strength of WENO5BND's momentum-flux reduction, or PARALINE's flattening coefficient (CLAMP: as
// k_recon's)
template <int DIR, int LIM, typename T, bool CLAMP = false>
__device__ __forceinline__ void recon_coef(const Dims& d, const ReconBox& rb, const double* __restrict__ P,
                                           const T* __restrict__ L, T* __restrict__ S, long long t) {
  const int nc = rb.c1 - rb.c0 + 1;
  if (t >= (long long)nc * rb.nlines) return;
  int c, l;
  if (DIR == 1) { c = (int)(t % nc); l = (int)(t / nc); }
  else { l = (int)(t % rb.nlines); c = (int)(t / rb.nlines); }
  c += rb.c0;
  const int tt = rb.t0 + l % rb.nt, o = rb.o0 + l / rb.nt;
  const long long stride = (DIR == 1) ? 1 : (DIR == 2) ? (long long)d.n1e : (long long)d.plane;
  const size_t id = (DIR == 1) ? cidx(d, c, tt, o) : (DIR == 2) ? cidx(d, tt, c, o) : cidx(d, tt, o, c);
  [[maybe_unused]] const int cells_along = (DIR == 1) ? d.n1e : (DIR == 2) ? d.n2e : d.n3e;
  auto along = [&](int q) { return id + (CLAMP ? min(max(c + q, 0), cells_along - 1) - c : q) * stride; };
  if constexpr (LIM == HARM_LIM_WENO5) {
    const T* Lq = L + (size_t)3 * (DIR - 1) * d.cells;
    const T* ve = Lq + d.cells;
    const T* up = Lq + 2 * d.cells;
    S[id] = weno_dp_strength<T>(weno_dp<T>((T)__ldg(P + (size_t)HARM_RHO * d.cells + id), __ldg(Lq + id), __ldg(up + id),
                                           __ldg(ve + along(-1)), __ldg(ve + along(1)), __ldg(up + along(-1)),
                                           __ldg(up + along(1))));
  } else {
    const T* Vd = L + (size_t)DIR * d.cells;
    T v[7], pp[7];
#pragma unroll
    for (int q = 0; q < 7; q++) {
      const size_t at = along(q - 3);
      v[q] = (q >= 1 && q <= 5) ? __ldg(Vd + at) : T(0);
      pp[q] = __ldg(L + at);
    }
    S[id] = paraline_fi<T>(v, pp);
  }
}
template <int DIR, int LIM, typename T, bool CLAMP = false, int TU = HARM_TU>
__global__ void __launch_bounds__(256) k_recon_coef(Dims d, ReconBox rb, const double* __restrict__ P,
                                                    const T* __restrict__ L, T* __restrict__ S) {
  recon_coef<DIR, LIM, T, CLAMP>(d, rb, P, L, S, (long long)blockIdx.x * 256 + threadIdx.x);
}

// ------------------------------------------------------------------ k_face

// One thread per (i, j) of the face box and kb consecutive k: the face's metric is loaded once
// for them (FP32; x3-independent).  Bounded by the FMA pipe in FP32, by the FP64 pipe in FP64.
// Blocks of 128 threads per SM, in whose registers the next face's states are loaded under this
// one's physics: FP32 5 (49 us at 256x128x64; 4: 51, 3: 55), FP64 4 (126 us at 192x96x64, with
// spills; 3: 132, 2: 160).
template <typename T>
constexpr int kFaceBlocks = sizeof(T) == 4 ? 5 : 4;
constexpr int kFaceThreads = 128;
// Block (bx, by) of a direction's faces: their fluxes, and the minimum of their time-step limits.
template <int DIR, typename T, typename GT>
__device__ __forceinline__ void face_block(const Dims& d, const Phys& ph, const FaceBox& fb, const T* __restrict__ EL,
                                           const T* __restrict__ ER, const GT* __restrict__ geom, T* __restrict__ F,
                                           unsigned long long* __restrict__ dtslot, int kb, int bx, int by) {
  const int t = bx * kFaceThreads + (int)threadIdx.x;
  const int i = t % fb.cnt[0] + fb.lo[0], j = t / fb.cnt[0] + fb.lo[1];
  const int k0 = by * kb, k1 = min(k0 + kb, fb.cnt[2]);
  constexpr int loc = (DIR == 1) ? HARM_LOC_FACE1 : (DIR == 2) ? HARM_LOC_FACE2 : HARM_LOC_CENT;
  const GT* tab = geom + (size_t)loc * HARM_NGF * d.plane;
  double top = 0.0;
  if (j <= fb.hi[1]) {
    const int ii = i + d.ng, jj = j + d.ng;
    const size_t c2 = (size_t)jj * d.n1e + ii;
    const size_t stride = (DIR == 1) ? 1 : (DIR == 2) ? (size_t)d.n1e : d.plane;
    if constexpr (sizeof(T) == 4) {
      FaceGeo g;
      load_face_geo<DIR>(tab, d.plane, c2, g);
      float mx = 0.0f;
      float nl[NPR], nr[NPR];
      auto load = [&](int k) {
        const size_t id = (size_t)(k + fb.lo[2] + d.ng3) * d.plane + c2;
#pragma unroll
        for (int p = 0; p < NPR; p++) {
          nl[p] = __ldg(ER + (size_t)p * d.cells + id - stride);
          nr[p] = __ldg(EL + (size_t)p * d.cells + id);
        }
      };
      load(k0);
#pragma unroll 1
      for (int k = k0; k < k1; k++) {
        const size_t id = (size_t)(k + fb.lo[2] + d.ng3) * d.plane + c2;
        float pl[NPR], pr[NPR], Fo[NPR];
#pragma unroll
        for (int p = 0; p < NPR; p++) {
          pl[p] = nl[p];
          pr[p] = nr[p];
        }
        if (k + 1 < k1) load(k + 1);
        const float ct = face_flux_f2<DIR>(g, pl, pr, (float)ph.gam, (float)ph.gammamax, ph.laxf, Fo);
        if (ct <= 3.402823466e38f) mx = fmaxf(mx, ct);
#pragma unroll
        for (int p = 0; p < NPR; p++) F[(size_t)p * d.cells + id] = Fo[p];
      }
      top = (double)mx;
    } else {
      for (int k = k0; k < k1; k++) {
        const size_t id = (size_t)(k + fb.lo[2] + d.ng3) * d.plane + c2;
        T pl[NPR], pr[NPR];
#pragma unroll
        for (int p = 0; p < NPR; p++) {
          pl[p] = __ldg(ER + (size_t)p * d.cells + id - stride);
          pr[p] = __ldg(EL + (size_t)p * d.cells + id);
        }
        const double ct = face_hll<DIR, T, GT>(d, ph, geom, F, id, ii, jj, pl, pr);
        if (ct <= 1.7976931348623157e308) top = fmax(top, ct);
      }
    }
  }
  block_dt_atomic(top, ph.cour * ((DIR == 1) ? ph.dx1 : (DIR == 2) ? ph.dx2 : ph.dx3), dtslot);
}
template <int DIR, typename T, typename GT, int TU = HARM_TU>
__global__ void __launch_bounds__(kFaceThreads, kFaceBlocks<T>) k_face(Dims d, Phys ph, FaceBox fb, const T* __restrict__ EL,
                                                              const T* __restrict__ ER, const GT* __restrict__ geom,
                                                              T* __restrict__ F, unsigned long long* __restrict__ dtslot,
                                                              int kb) {
  face_block<DIR, T, GT>(d, ph, fb, EL, ER, geom, F, dtslot, kb, blockIdx.x, blockIdx.y);
}

// ------------------------------------------------------------------ small grids

// The stages of the three directions in one launch each, for grids whose launches take longer to
// start than to run (one_launch_fluxes): a block belongs to one direction.
struct ReconAll {
  ReconBox rb[3];
  unsigned blocks[3];  // of each direction (0 without x3)
  unsigned groups[3];  // of a march's chunk
  FastDiv dseg;
};
struct FaceAll {
  FaceBox fb[3];
  unsigned blocks[3], bx[3];
};

template <int LIM, typename T, int TU = HARM_TU>
__global__ void __launch_bounds__(256) k_recon_coef_all(Dims d, ReconAll ra, const double* __restrict__ P,
                                                        const T* __restrict__ L, T* __restrict__ S) {
  unsigned b = blockIdx.x;
  if (b < ra.blocks[0]) return recon_coef<1, LIM, T>(d, ra.rb[0], P, L, S, (long long)b * 256 + threadIdx.x);
  b -= ra.blocks[0];
  if (b < ra.blocks[1]) return recon_coef<2, LIM, T>(d, ra.rb[1], P, L, S + d.cells, (long long)b * 256 + threadIdx.x);
  b -= ra.blocks[1];
  recon_coef<3, LIM, T>(d, ra.rb[2], P, L, S + 2 * d.cells, (long long)b * 256 + threadIdx.x);
}

// E: [direction][left, right][8][cells]
template <int LIM, typename T, int TU = HARM_TU>
__global__ void __launch_bounds__(32 * kReconWarps, kReconBlocks<T>) k_recon_all(Dims d, ReconAll ra, const double* __restrict__ P,
                                                                                 const T* __restrict__ S, T* __restrict__ E) {
  __shared__ ReconRowSmem<T> rows[kReconWarps];
  const size_t ne = (size_t)NPR * d.cells;
  unsigned b = blockIdx.x;
  if (b < ra.blocks[0]) {
    const int warp = threadIdx.x >> 5;
    return recon_rows<LIM, T>(d, ra.rb[0], ra.dseg, P, S, E, E + ne, rows[warp], (int)b * kReconWarps + warp,
                              (int)ra.blocks[0] * kReconWarps, blockIdx.y);
  }
  b -= ra.blocks[0];
  if (b < ra.blocks[1])
    return recon_march<2, LIM, T, false>(d, ra.rb[1], P, S + d.cells, E + 2 * ne, E + 3 * ne, (int)(b % ra.groups[1]),
                                         (int)(b / ra.groups[1]), blockIdx.y);
  b -= ra.blocks[1];
  recon_march<3, LIM, T, false>(d, ra.rb[2], P, S + 2 * d.cells, E + 4 * ne, E + 5 * ne, (int)(b % ra.groups[2]),
                                (int)(b / ra.groups[2]), blockIdx.y);
}

template <typename T, typename GT, int TU = HARM_TU>
__global__ void __launch_bounds__(kFaceThreads, kFaceBlocks<T>) k_face_all(Dims d, Phys ph, FaceAll fa, const T* __restrict__ E,
                                                                  const GT* __restrict__ geom, T* __restrict__ F1,
                                                                  T* __restrict__ F2, T* __restrict__ F3,
                                                                  unsigned long long* __restrict__ slots) {
  const size_t ne = (size_t)NPR * d.cells;
  unsigned b = blockIdx.x;
  if (b < fa.blocks[0])
    return face_block<1, T, GT>(d, ph, fa.fb[0], E, E + ne, geom, F1, slots + 0, 1, (int)(b % fa.bx[0]), (int)(b / fa.bx[0]));
  b -= fa.blocks[0];
  if (b < fa.blocks[1])
    return face_block<2, T, GT>(d, ph, fa.fb[1], E + 2 * ne, E + 3 * ne, geom, F2, slots + 1, 1, (int)(b % fa.bx[1]),
                                (int)(b / fa.bx[1]));
  b -= fa.blocks[1];
  face_block<3, T, GT>(d, ph, fa.fb[2], E + 4 * ne, E + 5 * ne, geom, F3, slots + 2, 1, (int)(b % fa.bx[2]), (int)(b / fa.bx[2]));
}

// ------------------------------------------------------------------ launchers

template <int DIR>
static inline ReconBox recon_box(const Dims& d, const FaceBox& fb) {
  ReconBox rb;
  const int ax = DIR - 1, ta = (DIR == 1) ? 1 : 0, oa = (DIR == 3) ? 1 : 2;
  const int g[3] = {d.ng, d.ng, d.ng3};
  rb.c0 = fb.lo[ax] - 1 + g[ax];
  rb.c1 = fb.hi[ax] + g[ax];
  rb.t0 = fb.lo[ta] + g[ta];
  rb.nt = fb.cnt[ta];
  rb.o0 = fb.lo[oa] + g[oa];
  rb.nlines = fb.cnt[ta] * fb.cnt[oa];
  rb.chunk = rb.c1 - rb.c0 + 1;
  return rb;
}

// Whether the stencils of a direction reach beyond its ghost zones (a caller's own grid:
// harm_grid_setup gives as many as they need).  Grids of WENO5 and PARALINE are created with
// enough of them in x1 and x2 only.
template <int DIR, int LIM>
constexpr bool recon_may_be_narrow = DIR == 3 || LIM == HARM_LIM_MC || LIM == HARM_LIM_PARA;
template <int DIR, int LIM>
static inline bool recon_narrow(const Dims& d) {
  return recon_may_be_narrow<DIR, LIM> && (DIR == 3 ? d.ng3 : d.ng) <= ReconWin<LIM>::R;
}

// Cuts a box's lines into chunks and gives their number.  Each chunk costs its first cell's window
// again (10 loads and 4 cells' weights for WENO5), so a line is cut only as far as the chip needs
// blocks: eight per SM (two waves; the other limiters, lighter in registers and bound by the
// latency of their loads, 24), and at least 12 cells (the others 4: a march of a small grid is a
// chain of load latencies).
template <int LIM>
static inline int cut_marches(ReconBox& rb, int groups, int num_sms) {
  const int nc = rb.c1 - rb.c0 + 1;
  constexpr int per_sm = (LIM == HARM_LIM_WENO5) ? 8 : 24;
  int chunks = (per_sm * num_sms + groups * NPR - 1) / (groups * NPR);
  chunks = std::max(1, std::min(chunks, nc / ((LIM == HARM_LIM_WENO5) ? 12 : 4)));
  rb.chunk = (nc + chunks - 1) / chunks;
  return (nc + rb.chunk - 1) / rb.chunk;
}
// the segments of the x1 rows of a plane
template <int LIM>
static inline long long row_segments(const Dims& d, const ReconBox& rb) {
  return ((long long)rb.nt * d.n1e + ReconRow<LIM>::E - 1) / ReconRow<LIM>::E;
}

// The two kernels of one direction on a face box; E: scratch of 2 x 8 x cells of T, S of cells.  The cell
// pass L has to be there for the box's stencils (WENO5, PARALINE).
// x1: segments are independent, and a warp takes the next one's loads under its own.
template <int DIR, int LIM, typename T, typename GT>
static inline cudaError_t launch_flux_dir(const Dims& d, const Phys& ph, const FaceBox& fb, const double* P, const GT* geom,
                                          T* F, unsigned long long* slot, cudaStream_t st, const T* L, T* S, T* E,
                                          int num_sms, unsigned long long& launches) {
  if (d.cells > 0xFFFFFFFFull) return cudaErrorInvalidValue;  // 32-bit offsets within a primitive
  ReconBox rb = recon_box<DIR>(d, fb);
  const int nc = rb.c1 - rb.c0 + 1;
  T* EL = E;
  T* ER = E + (size_t)NPR * d.cells;
  cudaError_t e;
  if constexpr (ReconWin<LIM>::S) {
    auto k = k_recon_coef<DIR, LIM, T>;
    if constexpr (DIR == 3)
      if (recon_narrow<DIR, LIM>(d)) k = k_recon_coef<DIR, LIM, T, true>;
    k<<<nblk((long long)nc * rb.nlines), 256, 0, st>>>(d, rb, P, L, S);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    launches++;
  }
  if (recon_narrow<DIR, LIM>(d)) {
    if constexpr (recon_may_be_narrow<DIR, LIM>) {
      constexpr int LN = 32 * ReconLanes<T>::N * kReconWarps;
      k_recon<DIR, LIM, T, true><<<dim3((rb.nlines + LN - 1) / LN, 1, NPR), 32 * kReconWarps, 0, st>>>(d, rb, P, S, EL, ER);
    }
  } else if constexpr (DIR == 1) {
    const long long nseg = row_segments<LIM>(d, rb), items = nseg * (rb.nlines / rb.nt);
    if (items > 0x7FFFFFFF) return cudaErrorInvalidValue;
    const long long blocks = std::min<long long>((items + kRowWarps - 1) / kRowWarps, 4LL * num_sms);
    k_recon_x1<LIM, T><<<dim3((unsigned)blocks, 1, NPR), 32 * kRowWarps, 0, st>>>(d, rb, fast_div((unsigned)nseg), P, S, EL, ER);
  } else {
    constexpr int LN = 32 * ReconLanes<T>::N * kReconWarps;
    const int groups = (rb.nlines + LN - 1) / LN, chunks = cut_marches<LIM>(rb, groups, num_sms);
    k_recon<DIR, LIM, T><<<dim3(groups, chunks, NPR), 32 * kReconWarps, 0, st>>>(d, rb, P, S, EL, ER);
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  const unsigned int bx = nblk((long long)fb.cnt[0] * fb.cnt[1], kFaceThreads);
  int kb = 1;
  while (kb < 4 && (long long)bx * ((fb.cnt[2] + 2 * kb - 1) / (2 * kb)) >= 16LL * num_sms) kb *= 2;
  k_face<DIR, T, GT><<<dim3(bx, (fb.cnt[2] + kb - 1) / kb), kFaceThreads, 0, st>>>(d, ph, fb, EL, ER, geom, F, slot, kb);
  launches += 2;
  return cudaGetLastError();
}

// The three directions of a small grid, a launch per stage.
template <int LIM, typename T, typename GT>
static inline cudaError_t launch_flux_all(const Dims& d, const Phys& ph, const double* P, const GT* geom, T* F1, T* F2, T* F3,
                                          unsigned long long* slots, cudaStream_t st, int num_sms,
                                          unsigned long long& launches, const T* L, T* S, T* E) {
  ReconAll ra{};
  FaceAll fa{};
  const int dirs = d.n3 > 1 ? 3 : 2;
  for (int q = 0; q < dirs; q++) {
    fa.fb[q] = face_box(d, q + 1);
    fa.bx[q] = nblk((long long)fa.fb[q].cnt[0] * fa.fb[q].cnt[1], kFaceThreads);
    fa.blocks[q] = fa.bx[q] * fa.fb[q].cnt[2];
  }
  ra.rb[0] = recon_box<1>(d, fa.fb[0]);
  ra.rb[1] = recon_box<2>(d, fa.fb[1]);
  if (dirs == 3) ra.rb[2] = recon_box<3>(d, fa.fb[2]);
  cudaError_t e;
  if constexpr (ReconWin<LIM>::S) {
    for (int q = 0; q < dirs; q++) ra.blocks[q] = nblk((long long)(ra.rb[q].c1 - ra.rb[q].c0 + 1) * ra.rb[q].nlines);
    k_recon_coef_all<LIM, T><<<ra.blocks[0] + ra.blocks[1] + ra.blocks[2], 256, 0, st>>>(d, ra, P, L, S);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    launches++;
  }
  const long long nseg = row_segments<LIM>(d, ra.rb[0]), items = nseg * (ra.rb[0].nlines / ra.rb[0].nt);
  ra.dseg = fast_div((unsigned)nseg);
  ra.blocks[0] = (unsigned)std::min<long long>((items + kReconWarps - 1) / kReconWarps, 8LL * num_sms);
  for (int q = 1; q < dirs; q++) {
    constexpr int LN = 32 * ReconLanes<T>::N * kReconWarps;
    ra.groups[q] = (ra.rb[q].nlines + LN - 1) / LN;
    ra.blocks[q] = ra.groups[q] * cut_marches<LIM>(ra.rb[q], ra.groups[q], num_sms);
  }
  k_recon_all<LIM, T><<<dim3(ra.blocks[0] + ra.blocks[1] + ra.blocks[2], NPR), 32 * kReconWarps, 0, st>>>(d, ra, P, S, E);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  k_face_all<T, GT><<<fa.blocks[0] + fa.blocks[1] + fa.blocks[2], kFaceThreads, 0, st>>>(d, ph, fa, E, geom, F1, F2, F3, slots);
  launches += 2;
  return cudaGetLastError();
}

// The three directions on the whole grid.
template <int LIM, typename T, typename GT>
static inline cudaError_t launch_flux_dirs(const Dims& d, const Phys& ph, const double* pb, const GT* geom, T* F1, T* F2,
                                           T* F3, unsigned long long* slots, cudaStream_t st, int num_sms,
                                           unsigned long long& launches, T* L, T* S, T* E) {
  cudaError_t e;
  if constexpr (ReconWin<LIM>::S) {
    if ((e = launch_cellprep<LIM, T, GT>(d, ph, pb, geom, L, 0, d.n3e, st)) != cudaSuccess) return e;
    launches++;
  }
  if (one_launch_fluxes(d, LIM, sizeof(T) == 8) && !recon_narrow<1, LIM>(d) && !recon_narrow<2, LIM>(d) && (d.n3 == 1 || !recon_narrow<3, LIM>(d)))
    return launch_flux_all<LIM, T, GT>(d, ph, pb, geom, F1, F2, F3, slots, st, num_sms, launches, L, S, E);
  const FaceBox b1 = face_box(d, 1), b2 = face_box(d, 2), b3 = face_box(d, 3);
  if ((e = launch_flux_dir<1, LIM, T, GT>(d, ph, b1, pb, geom, F1, slots + 0, st, L, S, E, num_sms, launches)) != cudaSuccess) return e;
  if ((e = launch_flux_dir<2, LIM, T, GT>(d, ph, b2, pb, geom, F2, slots + 1, st, L, S, E, num_sms, launches)) != cudaSuccess) return e;
  if (d.n3 > 1)
    return launch_flux_dir<3, LIM, T, GT>(d, ph, b3, pb, geom, F3, slots + 2, st, L, S, E, num_sms, launches);
  return cudaSuccess;
}

// The three flux directions of one substep while the state is still arriving in k-slabs
// (SlabWait): after each slab's copy, the x1 and x2 faces of its planes (their stencils stay in
// the plane) and every row of A x3 faces whose stencils' planes have all arrived.  Same kernels
// and results as the whole-grid launches.
// L (WENO5, PARALINE): the cell pass's output buffer; each slab's cell pass runs once the slab
// has arrived, before the kernels that read its planes.
template <int LIM, typename T, typename GT>
static inline cudaError_t launch_flux_slabs(const Dims& d, const Phys& ph, const double* pb, const GT* geom, T* F1,
                                            T* F2, T* F3, unsigned long long* slots, cudaStream_t st,
                                            const SlabWait& sw, int num_sms, unsigned long long& launches, T* L, T* S,
                                            T* E) {
  constexpr int A = 32, X = ReconGeom<LIM>::X;
  const FaceBox b1 = face_box(d, 1), b2 = face_box(d, 2), b3 = face_box(d, 3);
  int f3 = b3.lo[2];  // first x3 face not launched yet
  cudaError_t e;
  if (sw.nslab == 1) {
    if ((e = cudaStreamWaitEvent(st, sw.ev[0], 0)) != cudaSuccess) return e;
    if (sw.aos && hp_harm_to_soa(sw.ctx, sw.aos, sw.soa, 0, d.n3e)) return cudaErrorLaunchFailure;
    return launch_flux_dirs<LIM, T, GT>(d, ph, pb, geom, F1, F2, F3, slots, st, num_sms, launches, L, S, E);
  }
  for (int s = 0; s < sw.nslab; s++) {
    if ((e = cudaStreamWaitEvent(st, sw.ev[s], 0)) != cudaSuccess) return e;
    const int resident = (s + 1) * sw.planes;  // planes [0, resident) are on the device
    const int klo = s * sw.planes - d.ng3, khi = resident - 1 - d.ng3;
    if (sw.aos && hp_harm_to_soa(sw.ctx, sw.aos, sw.soa, s * sw.planes, resident < d.n3e ? resident : d.n3e))
      return cudaErrorLaunchFailure;
    if constexpr (ReconWin<LIM>::S) {
      const int k1 = resident < d.n3e ? resident : d.n3e;
      if ((e = launch_cellprep<LIM, T, GT>(d, ph, pb, geom, L, s * sw.planes, k1, st)) != cudaSuccess) return e;
      launches++;
    }
    FaceBox sb;
    if (face_box_k(b1, klo, khi, &sb)) {
      if ((e = launch_flux_dir<1, LIM, T, GT>(d, ph, sb, pb, geom, F1, slots + 0, st, L, S, E, num_sms, launches)) != cudaSuccess) return e;
    }
    if (face_box_k(b2, klo, khi, &sb)) {
      if ((e = launch_flux_dir<2, LIM, T, GT>(d, ph, sb, pb, geom, F2, slots + 1, st, L, S, E, num_sms, launches)) != cudaSuccess) return e;
    }
    // x3 rows of faces f0 .. last read planes up to last + ng3 + X (clamped); a row takes the
    // sweep's last face when it is the only one left after it
    while (d.n3 > 1 && f3 <= b3.hi[2]) {
      int last = f3 + A - 1;
      if (b3.hi[2] - last == 1) last = b3.hi[2];
      int top = last + d.ng3 + X;
      if (top > d.n3e - 1) top = d.n3e - 1;
      if (top >= resident && s + 1 < sw.nslab) break;
      if (face_box_k(b3, f3, last, &sb)) {
        if ((e = launch_flux_dir<3, LIM, T, GT>(d, ph, sb, pb, geom, F3, slots + 2, st, L, S, E, num_sms, launches)) != cudaSuccess) return e;
      }
      f3 = last + 1;
    }
  }
  return cudaSuccess;
}

