// learned.cu -- the kernels of the learned initial guess: a small periodic 3D convolutional
// network (U-Net) that maps a voxel image's material fields to the periodic fluctuation of the
// solution of every load case, trained and run by these kernels only.
//
// The reference finds initial guesses by solving the image coarsened by 2 per axis
// (chfem/src/femhmg/femhmg.c:561-846); the network replaces that search, PCG still runs to the
// same tolerance, so results do not change -- only where the iteration starts.
//
// Tensors are FP32, [N][C][D][H][W] with W fastest; every kernel takes the element stride
// between samples (nstride), so a channel slice of a wider tensor (the U-Net's skip
// concatenation) is addressed in place.  Convolutions are periodic (the images are periodic
// cells), 3x3x3 or 1x1x1, cross-correlation: out[co][p] = b[co] + sum_ci sum_o w[co][ci][o]
// in[ci][p + o - 1].
//
// B200 design: direct convolution on the CUDA cores (FP32 throughout) with shared-memory tiles and
// packed FP32 multiply-adds (two output channels per instruction, the rounding of two scalar
// ones).  Inside a chunk shared-memory bandwidth stands against FP32 issue, so a thread accumulates
// 8 positions along H x 16 output channels in registers: a row of weights (16 channels of one
// tap) is read once for 8 positions and an input value once for 3 taps x 16 channels, and lanes
// run along W so that input reads are free of bank conflicts.  (4 positions along W per thread
// read inputs with up to 4 conflicts and weights twice as often: 14 TFLOP/s.)  The weight gradient keeps the 27 taps of 4 output channels x 1 input channel
// per thread in registers and slides along W, so that a position costs 9 new input values instead
// of 27; the 4 warps of a CTA take its 4 planes and are summed in shared memory in warp order
// before the CTA adds into the global gradient with FP32 atomics (training, unlike the solver,
// does not need bitwise reproducibility).  What bounds them now is the staging between the chunks,
// which is not overlapped with the arithmetic: the FMA pipe is busy 43 % (convolution at 32^3, 11 %
// occupancy) and 41 % (weight gradient at 64^3, 18 %) of the cycles.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <string>

#include "device_cfg.h"

namespace {

std::string g_err;

constexpr int NTH = 128;                     // threads per CTA
constexpr int CO_T = 16;                     // output channels per CTA
constexpr int TX = 16, TY = 8;               // output tile along W and H; TZ planes along D
constexpr int HX = TX + 2, HY = TY + 2;

__device__ __forceinline__ int pmod(int v, int n) { v %= n; return v < 0 ? v + n : v; }

// Forward convolution (also the backward-data pass, with flipped and transposed weights).
// grid: (tiles of 16 x 8 x PY positions, ceil(Cout / 16), N).  PY: positions along H per thread
// (and planes per tile); 8 for full use of each weight read, fewer where 8 leaves SMs without a
// CTA (the launch chooses).  The plane pitch puts the two half-warps, one plane apart, on
// different banks.  Forward and backward of the whole network on two 64^3 samples: 12.4 -> 5.2 ms
// with these three kernels, 8 positions per thread in all but the deepest levels.
constexpr int CV_CI = 4;                     // input channels per shared-memory chunk
constexpr int CV_PL = 208;                   // words of a staged plane (180 used; 16 mod 32)
template <int K, int PY>
__global__ void __launch_bounds__(NTH) k_conv(const float* __restrict__ in, long in_ns, int Cin, int D, int H, int W,
                                               const float* __restrict__ w, const float* __restrict__ bias, int Cout,
                                               float* __restrict__ out, long out_ns, int relu, int accumulate) {
  constexpr int KK = K * K * K, OFF = K / 2, TZ = PY, HZ = TZ + 2;
  __shared__ float sIn[CV_CI * HZ * CV_PL];
  __shared__ __align__(16) float sW[CV_CI * KK * CO_T];
  const int tilesX = (W + TX - 1) / TX, tilesY = (H + TY - 1) / TY;
  const int tile = blockIdx.x;
  const int x0 = (tile % tilesX) * TX, y0 = ((tile / tilesX) % tilesY) * TY, z0 = (tile / (tilesX * tilesY)) * TZ;
  const int co0 = blockIdx.y * CO_T, n = blockIdx.z;
  const int tid = threadIdx.x;
  // lanes: 16 along W, 2 planes; then the groups of PY rows and the other planes
  const int lx = tid % TX, lz = ((tid / TX) & 1) + 2 * (tid / (2 * TX * (TY / PY))), ly = ((tid / (2 * TX)) % (TY / PY)) * PY;
  const float* inb = in + (long)n * in_ns;
  const long S = (long)D * H * W;
  float2 acc[CO_T / 2][PY];
#pragma unroll
  for (int c = 0; c < CO_T / 2; c++)
#pragma unroll
    for (int p = 0; p < PY; p++) acc[c][p] = make_float2(0.f, 0.f);
  for (int ci0 = 0; ci0 < Cin; ci0 += CV_CI) {
    const int nci = min(CV_CI, Cin - ci0);
    __syncthreads();
    // input chunk with periodic halo
    for (int t = tid; t < HZ * HY * HX; t += NTH) {
      const int hx = t % HX, hy = (t / HX) % HY, hz = t / (HX * HY);
      const int gx = pmod(x0 + hx - 1, W), gy = pmod(y0 + hy - 1, H), gz = pmod(z0 + hz - 1, D);
      const float* p = inb + (long)ci0 * S + ((long)gz * H + gy) * W + gx;
      float* q = sIn + hz * CV_PL + hy * HX + hx;
      for (int c = 0; c < nci; c++) q[c * HZ * CV_PL] = p[c * S];
    }
    // weights of the chunk: sW[(c * KK + o) * CO_T + co]
    for (int t = tid; t < nci * KK * CO_T; t += NTH) {
      const int co = t % CO_T, o = (t / CO_T) % KK, c = t / (CO_T * KK);
      sW[t] = co0 + co < Cout ? w[((long)(co0 + co) * Cin + (ci0 + c)) * KK + o] : 0.f;
    }
    __syncthreads();
    for (int c = 0; c < nci; c++) {
#pragma unroll 1
      for (int kzx = 0; kzx < K * K; kzx++) {
        const int kz = kzx / K, kx = kzx - kz * K;
        const float* col = sIn + c * HZ * CV_PL + (lz + kz + 1 - OFF) * CV_PL + (ly + 1 - OFF) * HX + lx + kx + 1 - OFF;
        float2 iv[PY + K - 1];
#pragma unroll
        for (int j = 0; j < PY + K - 1; j++) { const float v = col[j * HX]; iv[j] = make_float2(v, v); }
#pragma unroll
        for (int ky = 0; ky < K; ky++) {
          const float4* wv = reinterpret_cast<const float4*>(sW + (c * KK + (kz * K + ky) * K + kx) * CO_T);
#pragma unroll
          for (int u = 0; u < CO_T / 4; u++) {
            const float4 wq = wv[u];
            const float2 w0 = make_float2(wq.x, wq.y), w1 = make_float2(wq.z, wq.w);
#pragma unroll
            for (int p = 0; p < PY; p++) {
              acc[2 * u][p] = __ffma2_rn(w0, iv[p + ky], acc[2 * u][p]);
              acc[2 * u + 1][p] = __ffma2_rn(w1, iv[p + ky], acc[2 * u + 1][p]);
            }
          }
        }
      }
    }
  }
  const int gz = z0 + lz, gx = x0 + lx;
  if (gz >= D || gx >= W) return;
  float* outb = out + (long)n * out_ns;
#pragma unroll
  for (int co = 0; co < CO_T; co++) {
    if (co0 + co >= Cout) break;
    const float b = bias ? bias[co0 + co] : 0.f;
#pragma unroll
    for (int p = 0; p < PY; p++) {
      const int gy = y0 + ly + p;
      if (gy >= H) break;
      const long idx = (long)(co0 + co) * S + ((long)gz * H + gy) * W + gx;
      float v = ((co & 1) ? acc[co / 2][p].y : acc[co / 2][p].x) + b;
      if (accumulate) v += outb[idx];
      if (relu) v = fmaxf(v, 0.f);
      outb[idx] = v;
    }
  }
}

// Backward-data weights: wt[ci][co][o] = w[co][ci][KK - 1 - o] (flip every axis, swap channels).
__global__ void k_flip_weights(const float* w, int Cout, int Cin, int KK, float* wt) {
  const long n = (long)Cout * Cin * KK;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    const int o = (int)(t % KK), ci = (int)((t / KK) % Cin), co = (int)(t / ((long)KK * Cin));
    wt[((long)ci * Cout + co) * KK + (KK - 1 - o)] = w[t];
  }
}

// Weight gradient: dw[co][ci][o] += sum_n sum_p g[n][co][p] in[n][ci][p + o - 1]; db[co] += sum g.
// grid: (spatial tiles of 16 x 8 x 4, ceil(Cout/16) * ceil(Cin/8), N).  Warp: one plane of the
// tile; lane: input channel lane % 8, output channels 4 (lane / 8) .. + 3.
constexpr int WG_CI = 8, WG_TZ = 4, WG_HP = HX * HY * (WG_TZ + 2), WG_PI = WG_HP + 1;  // odd pitch: a bank per channel
constexpr int WG_TP = TX * TY * WG_TZ, WG_PG = CO_T + 4;  // gradients by position, 16-byte rows
template <int K>
__global__ void __launch_bounds__(NTH) k_conv_wgrad(const float* __restrict__ in, long in_ns, int Cin, int D, int H, int W,
                                                     const float* __restrict__ g, long g_ns, int Cout, float* dw, float* db) {
  constexpr int KK = K * K * K, OFF = K / 2;
  extern __shared__ __align__(16) float smem_w[];
  float* sG = smem_w;                     // [WG_TP][WG_PG]
  float* sIn = smem_w + WG_TP * WG_PG;    // [WG_CI][WG_PI], then the CTA's sums [KK][CO_T][WG_CI]
  const int tilesX = (W + TX - 1) / TX, tilesY = (H + TY - 1) / TY;
  const int tile = blockIdx.x;
  const int x0 = (tile % tilesX) * TX, y0 = ((tile / tilesX) % tilesY) * TY, z0 = (tile / (tilesX * tilesY)) * WG_TZ;
  const int nci_t = (Cin + WG_CI - 1) / WG_CI;
  const int co0 = (blockIdx.y / nci_t) * CO_T, ci0 = (blockIdx.y % nci_t) * WG_CI, n = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, lz = tid >> 5;
  const long S = (long)D * H * W;
  const float* inb = in + (long)n * in_ns;
  const float* gb = g + (long)n * g_ns;
  const int nci = min(WG_CI, Cin - ci0), nco = min(CO_T, Cout - co0);
  for (int t = tid; t < WG_HP; t += NTH) {
    const int hx = t % HX, hy = (t / HX) % HY, hz = t / (HX * HY);
    const int gx = pmod(x0 + hx - 1, W), gy = pmod(y0 + hy - 1, H), gz = pmod(z0 + hz - 1, D);
    const float* p = inb + (long)ci0 * S + ((long)gz * H + gy) * W + gx;
    for (int c = 0; c < WG_CI; c++) sIn[c * WG_PI + t] = c < nci ? p[c * S] : 0.f;
  }
  for (int t = tid; t < WG_TP; t += NTH) {
    const int gx = x0 + t % TX, gy = y0 + (t / TX) % TY, gz = z0 + t / (TX * TY);
    const bool ok = gx < W && gy < H && gz < D;
    const float* p = gb + (long)co0 * S + ((long)gz * H + gy) * W + gx;
    for (int c = 0; c < CO_T; c++) sG[t * WG_PG + c] = ok && c < nco ? p[c * S] : 0.f;
  }
  __syncthreads();
  const int ci = lane % WG_CI, cg = 4 * (lane / WG_CI);
  float2 a[KK][2];
#pragma unroll
  for (int o = 0; o < KK; o++) a[o][0] = a[o][1] = make_float2(0.f, 0.f);
  for (int py = 0; py < TY; py++) {
    const float* gp = sG + ((lz * TY + py) * TX) * WG_PG + cg;
    const float* ip = sIn + ci * WG_PI + ((lz + 1 - OFF) * HY + (py + 1 - OFF)) * HX + 1 - OFF;
    float win[K * K][K];  // the K columns of input under the position, K x K rows
#pragma unroll
    for (int j = 0; j < K - 1; j++)
#pragma unroll
      for (int r = 0; r < K * K; r++) win[r][j + 1] = ip[((r / K) * HY + r % K) * HX + j];
#pragma unroll
    for (int px = 0; px < TX; px++) {
#pragma unroll
      for (int r = 0; r < K * K; r++) {
#pragma unroll
        for (int j = 0; j < K - 1; j++) win[r][j] = win[r][j + 1];
        win[r][K - 1] = ip[((r / K) * HY + r % K) * HX + px + K - 1];
      }
      const float4 gv = *reinterpret_cast<const float4*>(gp + px * WG_PG);
      const float2 g0 = make_float2(gv.x, gv.y), g1 = make_float2(gv.z, gv.w);
#pragma unroll
      for (int r = 0; r < K * K; r++)
#pragma unroll
        for (int j = 0; j < K; j++) {
          const float2 v = make_float2(win[r][j], win[r][j]);
          a[r * K + j][0] = __ffma2_rn(g0, v, a[r * K + j][0]);
          a[r * K + j][1] = __ffma2_rn(g1, v, a[r * K + j][1]);
        }
    }
  }
  // the 4 planes' sums in warp order, then one atomic per weight
  __syncthreads();
  float* sum = sIn;
  for (int q = 0; q < WG_TZ; q++) {
    if (lz == q) {
#pragma unroll
      for (int o = 0; o < KK; o++) {
        float* d = sum + (o * CO_T + cg) * WG_CI + ci;
        const float v[4] = {a[o][0].x, a[o][0].y, a[o][1].x, a[o][1].y};
#pragma unroll
        for (int u = 0; u < 4; u++) d[u * WG_CI] = q ? d[u * WG_CI] + v[u] : v[u];
      }
    }
    __syncthreads();
  }
  for (int t = tid; t < KK * CO_T * WG_CI; t += NTH) {
    const int c = t % WG_CI, co = (t / WG_CI) % CO_T, o = t / (WG_CI * CO_T);
    if (c < nci && co < nco) atomicAdd(dw + ((long)(co0 + co) * Cin + (ci0 + c)) * KK + o, sum[t]);
  }
  // bias gradient from the CTAs of the first input-channel chunk
  if (db && ci0 == 0) {
    const int co = tid % CO_T, part = tid / CO_T;
    float v = 0.f;
    for (int p = part; p < WG_TP; p += NTH / CO_T) v += sG[p * WG_PG + co];
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    __shared__ float sb[NTH / 32][CO_T];  // one atomic per channel and CTA
    if (lane < CO_T) sb[lz][co] = v;
    __syncthreads();
    if (tid < nco) atomicAdd(db + co0 + tid, (sb[0][tid] + sb[1][tid]) + (sb[2][tid] + sb[3][tid]));
  }
}

__global__ void k_relu_bwd(const float* y, long y_ns, float* g, long g_ns, long per_sample, int N) {
  const long tot = per_sample * N;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < tot; t += (long)gridDim.x * blockDim.x) {
    const long n = t / per_sample, i = t % per_sample;
    if (!(y[n * y_ns + i] > 0.f)) g[n * g_ns + i] = 0.f;
  }
}

// 2x2x2 average pool (D, H, W even) and its adjoint (optionally accumulating).
__global__ void k_pool2(const float* in, long in_ns, int C, int D, int H, int W, float* out, long out_ns, int N) {
  const int d = D / 2, h = H / 2, w = W / 2;
  const long per = (long)C * d * h * w, tot = per * N;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < tot; t += (long)gridDim.x * blockDim.x) {
    const long n = t / per, r = t % per;
    const int x = (int)(r % w), y = (int)((r / w) % h), z = (int)((r / ((long)w * h)) % d), c = (int)(r / ((long)w * h * d));
    const float* p = in + n * in_ns + (long)c * D * H * W;
    float s = 0.f;
    for (int dz = 0; dz < 2; dz++)
      for (int dy = 0; dy < 2; dy++)
        for (int dx = 0; dx < 2; dx++) s += p[((long)(2 * z + dz) * H + 2 * y + dy) * W + 2 * x + dx];
    out[n * out_ns + r] = 0.125f * s;
  }
}
__global__ void k_pool2_bwd(const float* g, long g_ns, int C, int D, int H, int W, float* gin, long gin_ns, int N, int accumulate) {
  const long per = (long)C * D * H * W, tot = per * N;
  const int d = D / 2, h = H / 2, w = W / 2;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < tot; t += (long)gridDim.x * blockDim.x) {
    const long n = t / per, r = t % per;
    const int x = (int)(r % W), y = (int)((r / W) % H), z = (int)((r / ((long)W * H)) % D), c = (int)(r / ((long)W * H * D));
    const float v = 0.125f * g[n * g_ns + (((long)c * d + z / 2) * h + y / 2) * w + x / 2];
    float* o = gin + n * gin_ns + r;
    *o = accumulate ? *o + v : v;
  }
}
// nearest 2x upsample (coarse D, H, W -> 2D, 2H, 2W) and its adjoint
__global__ void k_up2(const float* in, long in_ns, int C, int D, int H, int W, float* out, long out_ns, int N) {
  const int D2 = 2 * D, H2 = 2 * H, W2 = 2 * W;
  const long per = (long)C * D2 * H2 * W2, tot = per * N;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < tot; t += (long)gridDim.x * blockDim.x) {
    const long n = t / per, r = t % per;
    const int x = (int)(r % W2), y = (int)((r / W2) % H2), z = (int)((r / ((long)W2 * H2)) % D2), c = (int)(r / ((long)W2 * H2 * D2));
    out[n * out_ns + r] = in[n * in_ns + (((long)c * D + z / 2) * H + y / 2) * W + x / 2];
  }
}
__global__ void k_up2_bwd(const float* g, long g_ns, int C, int D, int H, int W, float* gin, long gin_ns, int N) {
  const int H2 = 2 * H, W2 = 2 * W;
  const long per = (long)C * D * H * W, tot = per * N;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < tot; t += (long)gridDim.x * blockDim.x) {
    const long n = t / per, r = t % per;
    const int x = (int)(r % W), y = (int)((r / W) % H), z = (int)((r / ((long)W * H)) % D), c = (int)(r / ((long)W * H * D));
    const float* p = g + n * g_ns + (long)c * (2 * D) * H2 * W2;
    float s = 0.f;
    for (int dz = 0; dz < 2; dz++)
      for (int dy = 0; dy < 2; dy++)
        for (int dx = 0; dx < 2; dx++) s += p[((long)(2 * z + dz) * H2 + 2 * y + dy) * W2 + 2 * x + dx];
    gin[n * gin_ns + r] = s;
  }
}

// loss = sum (pred - target)^2 / count (FP64 accumulation); grad = 2 (pred - target) / count.  One
// atomic per CTA of a grid of 8 CTAs per SM: one per warp of a grid over all elements queued
// 295 thousand FP64 atomics on one address (455 us for 9.4 million elements).
__global__ void __launch_bounds__(256) k_mse(const float* pred, const float* target, long n, double inv_count, float* grad, double* loss) {
  __shared__ double sred[8];
  double s = 0.0;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    const float d = pred[t] - target[t];
    s += (double)d * d;
    if (grad) grad[t] = (float)(2.0 * inv_count) * d;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sred[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) s += sred[w];
    atomicAdd(loss, s * inv_count);
  }
}

__global__ void k_adam(float* p, const float* g, float* m, float* v, long n, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    const float gv = g[t];
    const float mv = b1 * m[t] + (1.f - b1) * gv, vv = b2 * v[t] + (1.f - b2) * gv * gv;
    m[t] = mv;
    v[t] = vv;
    p[t] -= lr * (mv / c1) / (sqrtf(vv / c2) + eps);
  }
}

// Material features of a voxel image: out[n][f][voxel] = table[label][f] (f < F) where the label
// of each voxel is its uint8 colour.
__global__ void k_features(const uint8_t* img, long img_ns, long S, const float* table, int F, float* out, long out_ns, int N) {
  const long tot = S * N;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < tot; t += (long)gridDim.x * blockDim.x) {
    const long n = t / S, i = t % S;
    const int lab = img[n * img_ns + i];
    for (int f = 0; f < F; f++) out[n * out_ns + (long)f * S + i] = table[lab * F + f];
  }
}

// Initial guesses from the network output: x_k[node * 3 + comp] = out[3k + comp][node] plus, on
// the displaced component of load case k, its macroscopic ramp (col for x, (R - row) mod R for y,
// (L - layer) mod L for z; node = row + col R + layer R C).
struct GuessPtrs { double* x[6]; };
__global__ void k_assemble_guess(const float* out, int L, int C, int R, GuessPtrs xs) {
  const long S = (long)L * C * R;
  const int AX[6] = {0, 1, 2, 1, 2, 1}, CO[6] = {0, 1, 2, 2, 0, 0};
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < S; i += (long)gridDim.x * blockDim.x) {
    const int r = (int)(i % R), c = (int)((i / R) % C), l = (int)(i / ((long)R * C));
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const double ramp = AX[k] == 0 ? (double)c : (AX[k] == 1 ? (double)((R - r) % R) : (double)((L - l) % L));
#pragma unroll
      for (int comp = 0; comp < 3; comp++)
        xs.x[k][3 * i + comp] = (double)out[(long)(3 * k + comp) * S + i] + (comp == CO[k] ? ramp : 0.0);
    }
  }
}

int grid1(long n) { long g = (n + 255) / 256; return (int)(g < 1 ? 1 : (g > 65535 ? 65535 : g)); }
bool check(const char* who) {
  const cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) { g_err = std::string(who) + ": " + cudaGetErrorString(e); return false; }
  return true;
}
int conv_tiles(int D, int H, int W, int planes) { return ((W + TX - 1) / TX) * ((H + TY - 1) / TY) * ((D + planes - 1) / planes); }
// Positions along H per thread (planes per tile) of k_conv: the most that still gives every SM a
// CTA, since fewer read each weight more often.
int conv_planes(int N, int D, int H, int W, int Cout) {
  const int sms = chfem::device_sms();
  const long per = (long)((Cout + CO_T - 1) / CO_T) * N;
  for (int p = 8; p > 2; p /= 2)
    if (conv_tiles(D, H, W, p) * per >= sms) return p;
  return 2;
}
template <int K, int PY>
void conv(const float* in, long in_ns, int N, int Cin, int D, int H, int W, const float* w, const float* bias, int Cout, int relu,
          int accumulate, float* out, long out_ns, cudaStream_t st) {
  const dim3 g(conv_tiles(D, H, W, PY), (Cout + CO_T - 1) / CO_T, N);
  k_conv<K, PY><<<g, NTH, 0, st>>>(in, in_ns, Cin, D, H, W, w, bias, Cout, out, out_ns, relu, accumulate);
}

}  // namespace

extern "C" {

const char* chfemB200NnLastError(void) { return g_err.c_str(); }

// out = conv(in) (+ bias) (ReLU when relu) for ksize 3 or 1; accumulate adds into out first.
int chfemB200NnConv3d(const float* in, long in_ns, int N, int Cin, int D, int H, int W, const float* w, const float* bias, int Cout,
                      int ksize, int relu, int accumulate, float* out, long out_ns, void* stream) {
  if (!in || !w || !out || N < 1 || Cin < 1 || Cout < 1 || D < 1 || H < 1 || W < 1 || (ksize != 1 && ksize != 3)) {
    g_err = "chfemB200NnConv3d: bad arguments"; return 0;
  }
  const cudaStream_t st = (cudaStream_t)stream;
  const int py = conv_planes(N, D, H, W, Cout);
  auto go = [&](auto f8, auto f4, auto f2) {
    (py == 8 ? f8 : py == 4 ? f4 : f2)(in, in_ns, N, Cin, D, H, W, w, bias, Cout, relu, accumulate, out, out_ns, st);
  };
  if (ksize == 3) go(&conv<3, 8>, &conv<3, 4>, &conv<3, 2>);
  else go(&conv<1, 8>, &conv<1, 4>, &conv<1, 2>);
  return check("chfemB200NnConv3d") ? 1 : 0;
}

// grad_in = conv^T(grad_out): the forward kernel on flipped, transposed weights (wt: caller
// scratch of Cout*Cin*k^3 floats); accumulate adds into grad_in.
int chfemB200NnConv3dBackwardData(const float* grad_out, long g_ns, int N, int Cout, int D, int H, int W, const float* w, int Cin,
                                  int ksize, float* wt, int accumulate, float* grad_in, long gin_ns, void* stream) {
  if (!grad_out || !w || !wt || !grad_in || (ksize != 1 && ksize != 3)) { g_err = "chfemB200NnConv3dBackwardData: bad arguments"; return 0; }
  const int KK = ksize * ksize * ksize;
  k_flip_weights<<<grid1((long)Cout * Cin * KK), 256, 0, (cudaStream_t)stream>>>(w, Cout, Cin, KK, wt);
  return chfemB200NnConv3d(grad_out, g_ns, N, Cout, D, H, W, wt, nullptr, Cin, ksize, 0, accumulate, grad_in, gin_ns, stream);
}

// dw += dL/dw, db += dL/db (db may be NULL); the caller zeroes them before the first call.
int chfemB200NnConv3dBackwardWeight(const float* in, long in_ns, int N, int Cin, int D, int H, int W, const float* grad_out, long g_ns,
                                    int Cout, int ksize, float* dw, float* db, void* stream) {
  if (!in || !grad_out || !dw || (ksize != 1 && ksize != 3)) { g_err = "chfemB200NnConv3dBackwardWeight: bad arguments"; return 0; }
  const dim3 g(conv_tiles(D, H, W, WG_TZ), ((Cout + CO_T - 1) / CO_T) * ((Cin + WG_CI - 1) / WG_CI), N);
  const size_t smem = (size_t)(WG_CI * WG_PI + WG_TP * WG_PG) * sizeof(float);
  static chfem::PerDevice kept3, kept1;
  if (!(ksize == 3 ? chfem::ctas_per_sm(kept3, k_conv_wgrad<3>, NTH, smem) : chfem::ctas_per_sm(kept1, k_conv_wgrad<1>, NTH, smem))) {
    g_err = "chfemB200NnConv3dBackwardWeight: shared-memory attribute refused"; return 0;
  }
  if (ksize == 3) k_conv_wgrad<3><<<g, NTH, smem, (cudaStream_t)stream>>>(in, in_ns, Cin, D, H, W, grad_out, g_ns, Cout, dw, db);
  else k_conv_wgrad<1><<<g, NTH, smem, (cudaStream_t)stream>>>(in, in_ns, Cin, D, H, W, grad_out, g_ns, Cout, dw, db);
  return check("chfemB200NnConv3dBackwardWeight") ? 1 : 0;
}

int chfemB200NnReluBackward(const float* y, long y_ns, float* g, long g_ns, long per_sample, int N, void* stream) {
  k_relu_bwd<<<grid1(per_sample * N), 256, 0, (cudaStream_t)stream>>>(y, y_ns, g, g_ns, per_sample, N);
  return check("chfemB200NnReluBackward") ? 1 : 0;
}
int chfemB200NnPool2(const float* in, long in_ns, int N, int C, int D, int H, int W, float* out, long out_ns, void* stream) {
  if ((D | H | W) & 1) { g_err = "chfemB200NnPool2: even sizes only"; return 0; }
  k_pool2<<<grid1((long)C * D * H * W / 8 * N), 256, 0, (cudaStream_t)stream>>>(in, in_ns, C, D, H, W, out, out_ns, N);
  return check("chfemB200NnPool2") ? 1 : 0;
}
int chfemB200NnPool2Backward(const float* g, long g_ns, int N, int C, int D, int H, int W, float* gin, long gin_ns, int accumulate, void* stream) {
  k_pool2_bwd<<<grid1((long)C * D * H * W * N), 256, 0, (cudaStream_t)stream>>>(g, g_ns, C, D, H, W, gin, gin_ns, N, accumulate);
  return check("chfemB200NnPool2Backward") ? 1 : 0;
}
int chfemB200NnUpsample2(const float* in, long in_ns, int N, int C, int D, int H, int W, float* out, long out_ns, void* stream) {
  k_up2<<<grid1((long)C * D * H * W * 8 * N), 256, 0, (cudaStream_t)stream>>>(in, in_ns, C, D, H, W, out, out_ns, N);
  return check("chfemB200NnUpsample2") ? 1 : 0;
}
int chfemB200NnUpsample2Backward(const float* g, long g_ns, int N, int C, int D, int H, int W, float* gin, long gin_ns, void* stream) {
  k_up2_bwd<<<grid1((long)C * D * H * W * N), 256, 0, (cudaStream_t)stream>>>(g, g_ns, C, D, H, W, gin, gin_ns, N);
  return check("chfemB200NnUpsample2Backward") ? 1 : 0;
}
// loss (device double, accumulated) and grad (may be NULL) of the mean squared error
int chfemB200NnMse(const float* pred, const float* target, long n, float* grad, double* loss, void* stream) {
  k_mse<<<std::min(grid1(n), 8 * chfem::device_sms()), 256, 0, (cudaStream_t)stream>>>(pred, target, n, 1.0 / (double)n, grad, loss);
  return check("chfemB200NnMse") ? 1 : 0;
}
int chfemB200NnAdam(float* p, const float* g, float* m, float* v, long n, float lr, float b1, float b2, float eps, int step, void* stream) {
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  k_adam<<<grid1(n), 256, 0, (cudaStream_t)stream>>>(p, g, m, v, n, lr, b1, b2, eps, c1, c2);
  return check("chfemB200NnAdam") ? 1 : 0;
}
int chfemB200NnFeatures(const uint8_t* img, long img_ns, long S, const float* table, int F, float* out, long out_ns, int N, void* stream) {
  k_features<<<grid1(S * N), 256, 0, (cudaStream_t)stream>>>(img, img_ns, S, table, F, out, out_ns, N);
  return check("chfemB200NnFeatures") ? 1 : 0;
}

// The six elastic initial-guess vectors (device, 3 L C R doubles each) from the network's output
// [18][L][C][R] (device).
int chfemB200NnAssembleGuess(const float* out, int L, int C, int R, double* const* x, void* stream) {
  if (!out || !x) { g_err = "chfemB200NnAssembleGuess: null argument"; return 0; }
  GuessPtrs p;
  for (int k = 0; k < 6; k++) { if (!x[k]) { g_err = "chfemB200NnAssembleGuess: null vector"; return 0; } p.x[k] = x[k]; }
  k_assemble_guess<<<grid1((long)L * C * R), 256, 0, (cudaStream_t)stream>>>(out, L, C, R, p);
  return check("chfemB200NnAssembleGuess") ? 1 : 0;
}

}  // extern "C"
