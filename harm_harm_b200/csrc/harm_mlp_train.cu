// harm_mlp_train.cu -- training and inference plumbing of the learned inversion guess.
//
// Training runs in FP32 with hand-written kernels:
//   k_mlp_grad   forward and backward pass of the 10-64-64-64-2 SiLU network over a
//                minibatch; each block owns a slice of the samples, keeps the parameters and
//                activations in shared memory (147 KB) and its gradients in registers, and
//                writes one partial gradient, so the reduction order is fixed
//                (deterministic gradients);
//   k_mlp_adam   sums the partial gradients in a fixed order and applies Adam;
//   k_mlp_norm   feature/target means and standard deviations (one block, FP64 sums);
//   k_mlp_init   Glorot-uniform weights, zero biases, from a counter-based hash.
// Loss: L = 1/(2n) sum_samples sum_outputs (y - t~)^2 over the standardised targets t~.
// Inference: k_mlp_pack writes the BF16 fragment-ordered record of harm_mlp.cuh;
// k_mlp_predict evaluates it on the tensor cores (mma.sync m16n8k16, FP32 accumulation),
// the same device function the inversion kernels call.
#include <algorithm>
#include <vector>
#include "harm_common.cuh"
#include "harm_mlp.cuh"
#include "harm_mlp_tc.cuh"

int hb_setmsg(const char* msg, int code);

namespace {

constexpr int TS = 64;           // samples per chunk
constexpr int TP = TS + 4;       // row pitch of the shared-memory matrices
constexpr int TR_GRID = 148;     // blocks of one training step at most
// parameters (W2, W3 with padded rows), then activations [feature][sample]: inputs, the three
// layers' outputs, and their derivatives, which become the layers' deltas in place
constexpr int TM = MLP_H * TP;   // floats of one 64 x 64 matrix
constexpr size_t TR_SMEM = (size_t)(MLP_IN * MLP_H + 3 * MLP_H + MLP_H * MLP_OUT + 4 + 8 * TM + MLP_IN * TP + 4 * TS + 8) * 4;

__device__ __forceinline__ uint64_t smix(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// 4 x 4 register tiles of 64 x 64 products; thread (tx, ty) of 16 x 16.  All matrices have rows
// of TP floats, activations [feature][sample].  Each 16-byte load feeds eight multiply-adds, and
// the rows' padding keeps the loads of neighbouring lanes in different banks.
//
// acc[a][b] += sum_k W[k][4 tx + a] H[k][4 ty + b]
template <int K>
__device__ __forceinline__ void mm_rows(const float* W, int wp, const float* H, int tx, int ty, float (&acc)[4][4]) {
#pragma unroll 8
  for (int k = 0; k < K; k++) {
    const float4 w = *reinterpret_cast<const float4*>(W + k * wp + 4 * tx);
    const float4 h = *reinterpret_cast<const float4*>(H + k * TP + 4 * ty);
    const float wv[4] = {w.x, w.y, w.z, w.w}, hv[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) acc[a][b] = fmaf(wv[a], hv[b], acc[a][b]);
  }
}
// acc[a][b] += sum_o W[tx + 16 a][o] D[o][4 ty + b]
__device__ __forceinline__ void mm_back(const float* W, const float* D, int tx, int ty, float (&acc)[4][4]) {
#pragma unroll 2
  for (int o = 0; o < MLP_H; o += 4) {
    float4 w[4], d[4];
#pragma unroll
    for (int a = 0; a < 4; a++) w[a] = *reinterpret_cast<const float4*>(W + (tx + 16 * a) * TP + o);
#pragma unroll
    for (int q = 0; q < 4; q++) d[q] = *reinterpret_cast<const float4*>(D + (o + q) * TP + 4 * ty);
#pragma unroll
    for (int a = 0; a < 4; a++) {
      const float wv[4] = {w[a].x, w[a].y, w[a].z, w[a].w};
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float dv[4] = {d[q].x, d[q].y, d[q].z, d[q].w};
#pragma unroll
        for (int b = 0; b < 4; b++) acc[a][b] = fmaf(wv[q], dv[b], acc[a][b]);
      }
    }
  }
}
// acc[a][b] += sum_s H[ty + 16 a][s] D[tx + 16 b][s]: the weights' gradient of a chunk
__device__ __forceinline__ void mm_grad(const float* H, const float* D, int tx, int ty, float (&acc)[4][4]) {
#pragma unroll 2
  for (int s = 0; s < TS; s += 4) {
    float4 h[4], d[4];
#pragma unroll
    for (int a = 0; a < 4; a++) h[a] = *reinterpret_cast<const float4*>(H + (ty + 16 * a) * TP + s);
#pragma unroll
    for (int b = 0; b < 4; b++) d[b] = *reinterpret_cast<const float4*>(D + (tx + 16 * b) * TP + s);
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) {
        acc[a][b] = fmaf(h[a].x, d[b].x, acc[a][b]);
        acc[a][b] = fmaf(h[a].y, d[b].y, acc[a][b]);
        acc[a][b] = fmaf(h[a].z, d[b].z, acc[a][b]);
        acc[a][b] = fmaf(h[a].w, d[b].w, acc[a][b]);
      }
  }
}

// the outputs o = 4 tx + a of a layer for samples 4 ty + b from their pre-activations: SiLU into
// H, its derivative into S
__device__ __forceinline__ void put_layer(float* H, float* S, int tx, int ty, const float (&z)[4][4]) {
#pragma unroll
  for (int a = 0; a < 4; a++) {
    float h[4], d[4];
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const float s = 1.0f / (1.0f + expf(-z[a][b]));
      h[b] = z[a][b] * s;
      d[b] = s * (1.0f + z[a][b] * (1.0f - s));
    }
    *reinterpret_cast<float4*>(H + (4 * tx + a) * TP + 4 * ty) = make_float4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<float4*>(S + (4 * tx + a) * TP + 4 * ty) = make_float4(d[0], d[1], d[2], d[3]);
  }
}
// the deltas of rows i = tx + 16 a: S (the derivatives) times acc, in place
__device__ __forceinline__ void put_delta(float* S, int tx, int ty, const float (&acc)[4][4]) {
#pragma unroll
  for (int a = 0; a < 4; a++) {
    float4* p = reinterpret_cast<float4*>(S + (tx + 16 * a) * TP + 4 * ty);
    const float4 d = *p;
    *p = make_float4(acc[a][0] * d.x, acc[a][1] * d.y, acc[a][2] * d.z, acc[a][3] * d.w);
  }
}

// Forward and backward of the network over a block's samples, 64 at a time, in FP32.  Bounded by
// the FMA pipe and the shared-memory loads that feed it, about evenly: one block of 256 threads
// fills an SM's shared memory, each thread a 4 x 4 tile of every 64 x 64 product; the gradients
// stay in registers over the block's chunks.  (With two scalar loads per multiply-add, from
// layouts of one product each, a step of 8192 samples took 98 us and a pass over 131,072 samples
// 1332 us; now 36 and 318 us.  512 threads with tiles of 4 x 2 took 43 and 378 us.)
__global__ void __launch_bounds__(256, 1) k_mlp_grad(size_t ndata, const float* __restrict__ feat,
                                                     const float* __restrict__ targ, const float* __restrict__ norm,
                                                     const float* __restrict__ params, long long nbatch,
                                                     uint64_t seed, long long step, float inv_n,
                                                     float* __restrict__ partial, double* __restrict__ partial_loss) {
  extern __shared__ __align__(16) float sm[];
  float* W1 = sm;                       // [10][64]
  float* Bs = W1 + MLP_IN * MLP_H;      // b1, b2, b3
  float* W4 = Bs + 3 * MLP_H;           // [64][2]
  float* B4 = W4 + MLP_H * MLP_OUT;
  float* W2 = B4 + 4;
  float* W3 = W2 + TM;
  float* H1 = W3 + TM;
  float* H2 = H1 + TM;
  float* H3 = H2 + TM;
  float* S1 = H3 + TM;
  float* S2 = S1 + TM;
  float* S3 = S2 + TM;
  float* X = S3 + TM;                   // [10][TP]
  float* T = X + MLP_IN * TP;           // targets [2][TS]
  float* DY = T + 2 * TS;               // output errors [2][TS]
  float* red = DY + 2 * TS;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  for (int i = tid; i < MLP_IN * MLP_H; i += 256) W1[i] = params[MLP_OFF_W1 + i];
  for (int i = tid; i < MLP_H; i += 256) {
    Bs[i] = params[MLP_OFF_B1 + i];
    Bs[MLP_H + i] = params[MLP_OFF_B2 + i];
    Bs[2 * MLP_H + i] = params[MLP_OFF_B3 + i];
  }
  for (int i = tid; i < MLP_H * MLP_OUT; i += 256) W4[i] = params[MLP_OFF_W4 + i];
  if (tid < MLP_OUT) B4[tid] = params[MLP_OFF_B4 + tid];
  for (int i = tid; i < MLP_H * MLP_H; i += 256) {
    W2[(i >> 6) * TP + (i & 63)] = params[MLP_OFF_W2 + i];
    W3[(i >> 6) * TP + (i & 63)] = params[MLP_OFF_W3 + i];
  }
  float g2[4][4] = {}, g3[4][4] = {};   // gradients of W[ty + 16 a][tx + 16 b]
  float g1[3] = {}, gb = 0.0f, g4 = 0.0f;  // W1 entries tid + 256 q; a bias (tid < 192); W4 and b4 (tid < 130)
  const long long per = (nbatch + gridDim.x - 1) / gridDim.x;
  const long long s0 = (long long)blockIdx.x * per, s1 = min(nbatch, s0 + per);
  float lacc = 0.0f;
  for (long long c0 = s0; c0 < s1; c0 += TS) {
    const int nc = (int)min((long long)TS, s1 - c0);
    __syncthreads();
    for (int e = tid; e < TS * 12; e += 256) {
      const int s = e / 12, col = e % 12;
      float v = 0.0f;
      if (s < nc) {
        const long long j = c0 + s;
        const size_t idx = seed ? (size_t)(smix(seed ^ smix((uint64_t)(step * nbatch + j))) % ndata) : (size_t)j;
        if (col < MLP_IN) v = (feat[idx * MLP_IN + col] - norm[col]) / norm[MLP_IN + col];
        else v = (targ[idx * MLP_OUT + col - MLP_IN] - norm[2 * MLP_IN + col - MLP_IN]) / norm[2 * MLP_IN + 2 + col - MLP_IN];
      }
      if (col < MLP_IN) X[col * TP + s] = v;
      else T[(col - MLP_IN) * TS + s] = v;
    }
    __syncthreads();
    auto bias = [&](const float* b, float (&z)[4][4]) {
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int q = 0; q < 4; q++) z[a][q] = b[4 * tx + a];
    };
    {
      float z[4][4];
      bias(Bs, z);
      mm_rows<MLP_IN>(W1, MLP_H, X, tx, ty, z);
      put_layer(H1, S1, tx, ty, z);
    }
    __syncthreads();
    {
      float z[4][4];
      bias(Bs + MLP_H, z);
      mm_rows<MLP_H>(W2, TP, H1, tx, ty, z);
      put_layer(H2, S2, tx, ty, z);
    }
    __syncthreads();
    {
      float z[4][4];
      bias(Bs + 2 * MLP_H, z);
      mm_rows<MLP_H>(W3, TP, H2, tx, ty, z);
      put_layer(H3, S3, tx, ty, z);
    }
    __syncthreads();
    // output and its error
    if (tid < TS * 2) {
      const int o = tid >> 6, s = tid & 63;
      float y0 = B4[o], y1 = 0.0f, y2 = 0.0f, y3 = 0.0f;
#pragma unroll 4
      for (int k = 0; k < MLP_H; k += 4) {
        y0 = fmaf(H3[k * TP + s], W4[k * 2 + o], y0);
        y1 = fmaf(H3[(k + 1) * TP + s], W4[k * 2 + 2 + o], y1);
        y2 = fmaf(H3[(k + 2) * TP + s], W4[k * 2 + 4 + o], y2);
        y3 = fmaf(H3[(k + 3) * TP + s], W4[k * 2 + 6 + o], y3);
      }
      float dy = 0.0f;
      if (s < nc) {
        const float r = ((y0 + y1) + (y2 + y3)) - T[tid];
        lacc += 0.5f * r * r;
        dy = r * inv_n;
      }
      DY[tid] = dy;
    }
    __syncthreads();
    {  // delta of layer 3, in place of its derivatives
      float acc[4][4];
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++)
          acc[a][b] = DY[4 * ty + b] * W4[(tx + 16 * a) * 2] + DY[TS + 4 * ty + b] * W4[(tx + 16 * a) * 2 + 1];
      put_delta(S3, tx, ty, acc);
    }
    // W4[k][o] (threads 2k + o) and b4
    if (tid < MLP_H * 2) {
      const int k = tid >> 1, o = tid & 1;
      float a0 = 0.0f, a1 = 0.0f;
#pragma unroll 8
      for (int q = 0; q < TS; q += 2) {  // rotated by k: neighbouring rows in different banks
        const int s = (q + 2 * k) & (TS - 1);
        a0 = fmaf(H3[k * TP + s], DY[o * TS + s], a0);
        a1 = fmaf(H3[k * TP + s + 1], DY[o * TS + s + 1], a1);
      }
      g4 += a0 + a1;
    } else if (tid < MLP_H * 2 + 2) {
      float a = 0.0f;
      for (int s = 0; s < TS; s++) a += DY[(tid - MLP_H * 2) * TS + s];
      g4 += a;
    }
    __syncthreads();
    mm_grad(H2, S3, tx, ty, g3);
    {
      float acc[4][4] = {};
      mm_back(W3, S3, tx, ty, acc);
      put_delta(S2, tx, ty, acc);
    }
    __syncthreads();
    mm_grad(H1, S2, tx, ty, g2);
    {
      float acc[4][4] = {};
      mm_back(W2, S2, tx, ty, acc);
      put_delta(S1, tx, ty, acc);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const int e = tid + 256 * q;
      if (e < MLP_IN * MLP_H) {
        const float* x = X + (e >> 6) * TP;
        const float* d = S1 + (e & 63) * TP;
        float a0 = 0.0f, a1 = 0.0f;
#pragma unroll 4
        for (int s = 0; s < TS; s += 4) {
          const float4 xv = *reinterpret_cast<const float4*>(x + s), dv = *reinterpret_cast<const float4*>(d + s);
          a0 = fmaf(xv.x, dv.x, a0);
          a1 = fmaf(xv.y, dv.y, a1);
          a0 = fmaf(xv.z, dv.z, a0);
          a1 = fmaf(xv.w, dv.w, a1);
        }
        g1[q] += a0 + a1;
      }
    }
    if (tid < 3 * MLP_H) {  // the biases: sums of the deltas' rows
      const float* d = (tid < MLP_H ? S1 : tid < 2 * MLP_H ? S2 : S3) + (tid & 63) * TP;
      float a0 = 0.0f, a1 = 0.0f;
#pragma unroll 4
      for (int s = 0; s < TS; s += 4) {
        const float4 v = *reinterpret_cast<const float4*>(d + s);
        a0 += v.x + v.z;
        a1 += v.y + v.w;
      }
      gb += a0 + a1;
    }
  }
  float* out = partial + (size_t)blockIdx.x * MLP_NPARAMS;
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const int e = (ty + 16 * a) * MLP_H + tx + 16 * b;
      out[MLP_OFF_W2 + e] = g2[a][b];
      out[MLP_OFF_W3 + e] = g3[a][b];
    }
#pragma unroll
  for (int q = 0; q < 3; q++)
    if (tid + 256 * q < MLP_IN * MLP_H) out[MLP_OFF_W1 + tid + 256 * q] = g1[q];
  if (tid < 3 * MLP_H) out[(tid < MLP_H ? MLP_OFF_B1 : tid < 2 * MLP_H ? MLP_OFF_B2 : MLP_OFF_B3) + (tid & 63)] = gb;
  if (tid < MLP_H * 2) out[MLP_OFF_W4 + tid] = g4;
  else if (tid < MLP_H * 2 + 2) out[MLP_OFF_B4 + tid - MLP_H * 2] = g4;
  // block loss in a fixed order
  __syncthreads();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lacc += __shfl_xor_sync(0xffffffffu, lacc, o);
  if ((tid & 31) == 0) red[tid >> 5] = lacc;
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
    for (int w = 0; w < 8; w++) s += red[w];
    partial_loss[blockIdx.x] = s;
  }
}

// sum of the partial gradients, then Adam when lr > 0.  A block sums 32 parameters, its eight
// warps an eighth of the partials each, combined in their order (fixed, so the gradient stays
// deterministic): 8 us; with one thread per parameter over all partials the 36 blocks' serial
// loads took 15 us.
__global__ void __launch_bounds__(256) k_mlp_adam(int nb, const float* __restrict__ partial,
                                                  const double* __restrict__ partial_loss, float* __restrict__ params,
                                                  float* __restrict__ m, float* __restrict__ v, float lr, float b1, float b2,
                                                  float eps, float bc1, float bc2, float inv_n,
                                                  float* __restrict__ grad_out, double* __restrict__ loss_out) {
  __shared__ float part[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int p = blockIdx.x * 32 + lane;
  float a = 0.0f;
  if (p < MLP_NPARAMS) {
    const int per = (nb + 7) / 8, q1 = min(nb, (w + 1) * per);
#pragma unroll 8
    for (int q = w * per; q < q1; q++) a += partial[(size_t)q * MLP_NPARAMS + p];
  }
  part[w][lane] = a;
  __syncthreads();
  if (w == 0 && p < MLP_NPARAMS) {
    float g = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; q++) g += part[q][lane];
    if (grad_out) grad_out[p] = g;
    if (lr > 0.0f) {
      const float mm = b1 * m[p] + (1.0f - b1) * g;
      const float vv = b2 * v[p] + (1.0f - b2) * g * g;
      m[p] = mm;
      v[p] = vv;
      params[p] -= lr * (mm / bc1) / (sqrtf(vv / bc2) + eps);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 32 && loss_out) {
    double s = 0.0;
    for (int b = 0; b < nb; b++) s += partial_loss[b];
    *loss_out = s * (double)inv_n;
  }
}

__global__ void k_mlp_norm(size_t n, const float* __restrict__ feat, const float* __restrict__ targ,
                           float* __restrict__ norm) {
  __shared__ double s1[MLP_IN + MLP_OUT][32], s2[MLP_IN + MLP_OUT][32];
  double a1[MLP_IN + MLP_OUT], a2[MLP_IN + MLP_OUT];
  for (int c = 0; c < MLP_IN + MLP_OUT; c++) { a1[c] = 0.0; a2[c] = 0.0; }
  for (size_t t = threadIdx.x; t < n; t += blockDim.x) {
    for (int c = 0; c < MLP_IN; c++) {
      double x = feat[t * MLP_IN + c];
      a1[c] += x; a2[c] += x * x;
    }
    for (int c = 0; c < MLP_OUT; c++) {
      double x = targ[t * MLP_OUT + c];
      a1[MLP_IN + c] += x; a2[MLP_IN + c] += x * x;
    }
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int c = 0; c < MLP_IN + MLP_OUT; c++) {
    double x = a1[c], y = a2[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      y += __shfl_xor_sync(0xffffffffu, y, o);
    }
    if (lane == 0) { s1[c][w] = x; s2[c][w] = y; }
  }
  __syncthreads();
  if (threadIdx.x < MLP_IN + MLP_OUT) {
    const int c = threadIdx.x;
    double x = 0.0, y = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) { x += s1[c][q]; y += s2[c][q]; }
    const double mean = x / (double)n, var = fmax(y / (double)n - mean * mean, 0.0);
    double sd = sqrt(var);
    if (!(sd > 1e-6)) sd = 1.0;
    if (c < MLP_IN) { norm[c] = (float)mean; norm[MLP_IN + c] = (float)sd; }
    else { norm[2 * MLP_IN + c - MLP_IN] = (float)mean; norm[2 * MLP_IN + MLP_OUT + c - MLP_IN] = (float)sd; }
  }
}

__global__ void k_mlp_init(uint64_t seed, float* __restrict__ params) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= MLP_NPARAMS) return;
  int fin = 0, fout = 0;
  if (p < MLP_OFF_B1) { fin = MLP_IN; fout = MLP_H; }
  else if (p >= MLP_OFF_W2 && p < MLP_OFF_B2) { fin = MLP_H; fout = MLP_H; }
  else if (p >= MLP_OFF_W3 && p < MLP_OFF_B3) { fin = MLP_H; fout = MLP_H; }
  else if (p >= MLP_OFF_W4 && p < MLP_OFF_B4) { fin = MLP_H; fout = MLP_OUT; }
  if (fin == 0) { params[p] = 0.0f; return; }
  const double u = (double)(smix(seed ^ smix((uint64_t)p)) >> 11) * (1.0 / 9007199254740992.0);
  const double a = sqrt(6.0 / (double)(fin + fout));
  params[p] = (float)((2.0 * u - 1.0) * a);
}

// BF16 fragments (mma.sync m16n8k16 .col B operand), biases, normalisation, start bias
__global__ void k_mlp_pack(const float* __restrict__ params, const float* __restrict__ norm, float start_bias,
                           MlpPacked* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < MLP_TILES * 32) {
    const int tile = t >> 5, lane = t & 31;
    int woff, K, N, kt, nt;
    if (tile < MLP_TILE_L2) { woff = MLP_OFF_W1; K = MLP_IN; N = MLP_H; kt = 0; nt = tile; }
    else if (tile < MLP_TILE_L3) { woff = MLP_OFF_W2; K = MLP_H; N = MLP_H; kt = (tile - MLP_TILE_L2) >> 3; nt = (tile - MLP_TILE_L2) & 7; }
    else if (tile < MLP_TILE_L4) { woff = MLP_OFF_W3; K = MLP_H; N = MLP_H; kt = (tile - MLP_TILE_L3) >> 3; nt = (tile - MLP_TILE_L3) & 7; }
    else { woff = MLP_OFF_W4; K = MLP_H; N = MLP_OUT; kt = tile - MLP_TILE_L4; nt = 0; }
    const int k0 = kt * 16 + 2 * (lane & 3), n = nt * 8 + (lane >> 2);
    const float scale = (tile < MLP_TILE_L4) ? 0.5f : 1.0f;  // layers 1-3 halved (mlp_tanh)
    auto W = [&](int k) -> float { return (k < K && n < N) ? scale * params[woff + k * N + n] : 0.0f; };
    uint32_t* f = reinterpret_cast<uint32_t*>(&out->frag[tile >> 1][lane]) + 2 * (tile & 1);
    f[0] = pack_bf16x2(W(k0), W(k0 + 1));
    f[1] = pack_bf16x2(W(k0 + 8), W(k0 + 9));
  }
  if (t < MLP_NBIAS) {
    float b = 0.0f;
    if (t < MLP_H) b = 0.5f * params[MLP_OFF_B1 + t];
    else if (t < 2 * MLP_H) b = 0.5f * params[MLP_OFF_B2 + t - MLP_H];
    else if (t < 3 * MLP_H) b = 0.5f * params[MLP_OFF_B3 + t - 2 * MLP_H];
    else if (t < 3 * MLP_H + MLP_OUT) b = params[MLP_OFF_B4 + t - 3 * MLP_H];
    out->bias[t] = b;
  }
  if (t < MLP_NNORM) out->norm[t] = norm[t];
  if (t == 0) {
    out->start_bias = start_bias;
    out->pad[0] = out->pad[1] = out->pad[2] = 0.0f;
  }
}

// BF16 B operands in the tensor-core canonical layout of harm_mlp_tc.cuh (one 16-byte chunk of
// 8 K-consecutive weights per thread), biases, normalisation, start bias
__global__ void k_mlp_pack_tc(const float* __restrict__ params, const float* __restrict__ norm, float start_bias,
                              MlpTc* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < TC_WBYTES / 16) {
    const int off = t * 16;
    int base, kc, woff, K, N;
    if (off < TC_W2) { base = TC_W1; kc = 2; woff = MLP_OFF_W1; K = MLP_IN; N = MLP_H; }
    else if (off < TC_W3) { base = TC_W2; kc = 8; woff = MLP_OFF_W2; K = MLP_H; N = MLP_H; }
    else if (off < TC_W4) { base = TC_W3; kc = 8; woff = MLP_OFF_W3; K = MLP_H; N = MLP_H; }
    else { base = TC_W4; kc = 8; woff = MLP_OFF_W4; K = MLP_H; N = MLP_OUT; }
    const int rel = off - base, cm = rel >> 7;
    const int n = (cm / kc) * 8 + ((rel & 127) >> 4), k0 = (cm % kc) * 8;  // tc_off(n, k0, kc) == rel
    const float scale = (base < TC_W4) ? 0.5f : 1.0f;  // layers 1-3 halved (mlp_tanh)
    auto W = [&](int k) -> float { return (k < K && n < N) ? scale * params[woff + k * N + n] : 0.0f; };
    uint4 v;
    v.x = pack_bf16x2(W(k0), W(k0 + 1));
    v.y = pack_bf16x2(W(k0 + 2), W(k0 + 3));
    v.z = pack_bf16x2(W(k0 + 4), W(k0 + 5));
    v.w = pack_bf16x2(W(k0 + 6), W(k0 + 7));
    out->w[t] = v;
  }
  if (t < MLP_NBIAS) {
    float b = 0.0f;
    if (t < MLP_H) b = 0.5f * params[MLP_OFF_B1 + t];
    else if (t < 2 * MLP_H) b = 0.5f * params[MLP_OFF_B2 + t - MLP_H];
    else if (t < 3 * MLP_H) b = 0.5f * params[MLP_OFF_B3 + t - 2 * MLP_H];
    else if (t < 3 * MLP_H + MLP_OUT) b = params[MLP_OFF_B4 + t - 3 * MLP_H];
    out->bias[t] = b;
  }
  if (t < MLP_NNORM) out->norm[t] = norm[t];
  if (t == 0) {
    out->start_bias = start_bias;
    out->pad[0] = out->pad[1] = out->pad[2] = 0.0f;
  }
}

__global__ void __launch_bounds__(256) k_mlp_predict(size_t n, const float* __restrict__ feat,
                                                     const MlpPacked* __restrict__ mlp, float* __restrict__ out) {
  __shared__ MlpPacked sm;
  __shared__ MlpWarpScratch ws[8];
  mlp_load_packed(sm, mlp);
  __syncthreads();
  for (size_t base = (size_t)blockIdx.x * 256; base < n; base += (size_t)gridDim.x * 256) {
    const size_t t = base + threadIdx.x;
    const bool valid = t < n;
    float f[MLP_IN];
#pragma unroll
    for (int i = 0; i < MLP_IN; i++) f[i] = valid ? feat[t * MLP_IN + i] : 0.0f;
    float y[MLP_OUT];
    mlp_warp_eval(sm, ws[threadIdx.x >> 5], f, valid, y);
    if (valid) {
      out[t * MLP_OUT + 0] = y[0];
      out[t * MLP_OUT + 1] = y[1];
    }
  }
}

int ensure_train_scratch(harm_ctx* c) {
  if (!c->d_mlp_adam) {
    CK(cudaMalloc(&c->d_mlp_adam, 2 * (size_t)MLP_NPARAMS * sizeof(float)));
  }
  if (!c->d_mlp_work) {
    // partial gradients of up to TR_GRID blocks, their partial losses (doubles) and the loss
    c->mlp_work_n = (size_t)TR_GRID * MLP_NPARAMS + 2 * TR_GRID + 4;
    CK(cudaMalloc(&c->d_mlp_work, c->mlp_work_n * sizeof(float)));
  }
  static std::atomic<unsigned long long> raised{0};
  CK(raise_smem_limit_once(raised, (const void*)k_mlp_grad, (int)TR_SMEM));
  return 0;
}

double* partial_loss_of(harm_ctx* c) {
  return reinterpret_cast<double*>(c->d_mlp_work + (size_t)TR_GRID * MLP_NPARAMS + 2);  // 8-byte aligned
}

}  // namespace

extern "C" int harm_b200_mlp_init(harm_ctx* c, uint64_t seed, float* d_params) {
  if (!c || !d_params) return hb_setmsg("null argument", 1);
  k_mlp_init<<<nblk(MLP_NPARAMS), 256, 0, c->stream>>>(seed, d_params);
  c->launches++;
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(c->stream));
  return 0;
}

extern "C" int harm_b200_mlp_norm(harm_ctx* c, size_t n, const float* d_feat, const float* d_targ, float* d_norm) {
  if (!c || !d_feat || !d_targ || !d_norm) return hb_setmsg("null argument", 1);
  if (n == 0) return hb_setmsg("no samples", 2);
  k_mlp_norm<<<1, 1024, 0, c->stream>>>(n, d_feat, d_targ, d_norm);
  c->launches++;
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(c->stream));
  return 0;
}

extern "C" int harm_b200_mlp_loss_grad(harm_ctx* c, size_t n, const float* d_feat, const float* d_targ,
                                       const float* d_params, const float* d_norm, double* loss, float* d_grad) {
  if (!c || !d_feat || !d_targ || !d_params || !d_norm || !d_grad) return hb_setmsg("null argument", 1);
  if (n == 0) return hb_setmsg("no samples", 2);
  if (ensure_train_scratch(c)) return 1;
  const int nb = (int)std::min<size_t>((n + TS - 1) / TS, (size_t)TR_GRID);
  float* partial = c->d_mlp_work;
  double* ploss = partial_loss_of(c);
  double* dloss = ploss + TR_GRID;
  const float inv_n = (float)(1.0 / (double)n);
  k_mlp_grad<<<nb, 256, TR_SMEM, c->stream>>>(n, d_feat, d_targ, d_norm, d_params, (long long)n, 0ull, 0ll, inv_n,
                                              partial, ploss);
  k_mlp_adam<<<nblk(MLP_NPARAMS, 32), 256, 0, c->stream>>>(nb, partial, ploss, nullptr, nullptr, nullptr, 0.0f, 0.f, 0.f,
                                                       0.f, 1.f, 1.f, inv_n, d_grad, dloss);
  c->launches += 2;
  CK(cudaGetLastError());
  double h = 0.0;
  CK(cudaMemcpyAsync(&h, dloss, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  if (loss) *loss = h;
  return 0;
}

extern "C" int harm_b200_mlp_train(harm_ctx* c, size_t n, const float* d_feat, const float* d_targ,
                                   const float* d_norm, float* d_params, int steps, int batch, float lr,
                                   uint64_t seed, float* loss_hist) {
  if (!c || !d_feat || !d_targ || !d_norm || !d_params) return hb_setmsg("null argument", 1);
  if (n == 0 || steps < 1 || batch < 1) return hb_setmsg("need n, steps and batch >= 1", 2);
  if (seed == 0) seed = 0x5eedull;
  if (ensure_train_scratch(c)) return 1;
  float* m = c->d_mlp_adam;
  float* v = m + MLP_NPARAMS;
  CK(cudaMemsetAsync(m, 0, 2 * (size_t)MLP_NPARAMS * sizeof(float), c->stream));
  float* partial = c->d_mlp_work;
  double* ploss = partial_loss_of(c);
  double* dloss = ploss + TR_GRID;
  std::vector<double> hist;
  double* d_hist = nullptr;
  if (loss_hist) {
    CK(cudaMalloc(&d_hist, (size_t)steps * sizeof(double)));
  }
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const int nb = (int)std::min<long long>(((long long)batch + TS - 1) / TS, (long long)TR_GRID);
  const float inv_n = (float)(1.0 / (double)batch);
  double p1 = 1.0, p2 = 1.0;
  for (int s = 0; s < steps; s++) {
    // cosine decay to lr/100
    const double frac = (double)s / (double)steps;
    const float lr_s = (float)(lr * (0.01 + 0.99 * 0.5 * (1.0 + cos(3.141592653589793 * frac))));
    p1 *= b1;
    p2 *= b2;
    k_mlp_grad<<<nb, 256, TR_SMEM, c->stream>>>(n, d_feat, d_targ, d_norm, d_params, (long long)batch, seed,
                                                (long long)s, inv_n, partial, ploss);
    k_mlp_adam<<<nblk(MLP_NPARAMS, 32), 256, 0, c->stream>>>(nb, partial, ploss, d_params, m, v, lr_s, b1, b2, eps,
                                                         (float)(1.0 - p1), (float)(1.0 - p2), inv_n, nullptr,
                                                         d_hist ? d_hist + s : dloss);
    c->launches += 2;
  }
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && d_hist) {
    hist.resize(steps);
    e = cudaMemcpyAsync(hist.data(), d_hist, (size_t)steps * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (d_hist) cudaFree(d_hist);
  if (e != cudaSuccess) return hb_seterr("mlp training", e);
  if (loss_hist)
    for (int s = 0; s < steps; s++) loss_hist[s] = (float)hist[s];
  return 0;
}

extern "C" int harm_b200_mlp_set(harm_ctx* c, const float* d_params, const float* d_norm, double start_bias) {
  if (!c || !d_params || !d_norm) return hb_setmsg("null argument", 1);
  if (!c->d_mlp) {
    CK(cudaMalloc(&c->d_mlp, sizeof(MlpPacked) + sizeof(MlpTc)));
  }
  if (!c->d_wpg) {
    CK(cudaMalloc(&c->d_wpg, (size_t)c->g.n1 * c->g.n2 * c->g.n3 * sizeof(double)));
  }
  k_mlp_pack<<<nblk(MLP_TILES * 32), 256, 0, c->stream>>>(d_params, d_norm, (float)start_bias,
                                                         reinterpret_cast<MlpPacked*>(c->d_mlp));
  k_mlp_pack_tc<<<nblk(TC_WBYTES / 16), 256, 0, c->stream>>>(d_params, d_norm, (float)start_bias, mlp_tc_of(c));
  c->launches += 2;
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(c->stream));
  c->mlp_step = 1;  // a packed network is present
  return 0;
}

// Network outputs for n feature rows (the tensor-core counterpart of k_mlp_predict).
__global__ void __launch_bounds__(256) k_mlp_predict_tc(size_t n, const float* __restrict__ feat,
                                                        const MlpTc* __restrict__ mlp, float* __restrict__ out,
                                                        unsigned int* __restrict__ status) {
  extern __shared__ __align__(128) unsigned char tc_smem[];
  MlpTcBlock& B = *reinterpret_cast<MlpTcBlock*>(tc_smem);
  mlp_tc_begin(B, mlp);
  const int wg = threadIdx.x >> 7, r = threadIdx.x & 127;
  const long long ntiles = (long long)((n + 127) / 128);
  TcState st = {0u, false};
  for (long long tile = 2ll * blockIdx.x + wg; tile < ntiles; tile += 2ll * gridDim.x) {
    const size_t t = (size_t)tile * 128 + r;
    const bool valid = t < n;
    float f[MLP_IN], x[MLP_IN];
#pragma unroll
    for (int i = 0; i < MLP_IN; i++) f[i] = valid ? feat[t * MLP_IN + i] : 0.0f;
    mlp_tc_standardise(B.net, f, valid, x);
    float y[MLP_OUT];
    if (!mlp_tc_eval(B, x, st, status, y)) break;
    if (valid) {
      out[t * MLP_OUT + 0] = y[0];
      out[t * MLP_OUT + 1] = y[1];
    }
  }
  mlp_tc_end(B, st);
}

extern "C" int harm_b200_mlp_predict(harm_ctx* c, size_t n, const float* d_feat, float* d_out) {
  if (!c || !d_feat || !d_out) return hb_setmsg("null argument", 1);
  if (!c->d_mlp || !c->mlp_step) return hb_setmsg("no network set (harm_b200_mlp_set)", 3);
  if (n == 0) return 0;
  if (c->mlp_tc == 1 || c->mlp_tc == 2) {  // the tcgen05 engines: their network kernel
    static std::atomic<unsigned long long> configured{0};
    static std::atomic<int> per_sm{1};
    if (int rc = tc_blocks_per_sm(c, k_mlp_predict_tc, configured, per_sm)) return rc;
    const size_t pairs = (n + 255) / 256;
    const unsigned int nb = (unsigned int)std::min<size_t>(pairs, (size_t)per_sm.load() * c->num_sms);
    k_mlp_predict_tc<<<nb, 256, sizeof(MlpTcBlock), c->stream>>>(n, d_feat, mlp_tc_of(c), d_out, c->d_status);
  } else {
    const unsigned int nb = (unsigned int)std::min<size_t>((n + 255) / 256, (size_t)4 * c->num_sms);
    k_mlp_predict<<<nb, 256, 0, c->stream>>>(n, d_feat, reinterpret_cast<const MlpPacked*>(c->d_mlp), d_out);
  }
  c->launches++;
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(c->stream));
  unsigned int st = 0;
  CK(cudaMemcpy(&st, c->d_status, sizeof(st), cudaMemcpyDeviceToHost));
  if (st) {
    CK(cudaMemset(c->d_status, 0, sizeof(st)));
    return hb_setmsg("a tensor-core MMA of the network did not complete", 5);
  }
  return 0;
}
