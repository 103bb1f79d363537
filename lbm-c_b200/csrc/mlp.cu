// Training and inference kernels of the learned subgrid closure (lbmc_mlp_*).
// No counterpart in the reference.
//
// Training is plain mini-batch Adam on the mean squared error, all on the
// GPU with hand-written kernels:
//   mlp_grad_kernel      a few samples per warp, lane = hidden neuron:
//                        forward pass with the BF16 weights (FP32
//                        accumulation), backward pass, gradient sums in
//                        registers, one FP32 partial per block;
//   mlp_update_kernel    sums the block partials in a fixed order
//                        (deterministic gradients), Adam on the FP32 master
//                        weights, refreshes the BF16 copy the forward pass
//                        uses.
// The gradient is that of the loss as computed with the BF16-rounded
// weights, which is what the CPU check (oracle/mlp_oracle.py) reproduces.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <random>
#include <string>
#include <vector>

#include "../../include/lbmc.h"
#include "engine_internal.h"
#include "launch.cuh"
#include "mlp.cuh"

using namespace lbmc;

namespace {

constexpr int GRAD_BLOCK = 256;
constexpr int GRAD_SLOTS = MLP_PARAMS + 1;  // parameters + loss

lbmc_status merr(lbmc_status s, const std::string &m) {
  lbmc::set_last_error(m);
  return s;
}

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }

__global__ void normalise_kernel(const float *raw, const float *y, long long n, MlpClosure c, float *xn,
                                 float *yn) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  for (int i = 0; i < MLP_IN; i++) xn[k * MLP_IN + i] = (raw[k * MLP_IN + i] - c.mean[i]) * c.inv_std[i];
  if (y) yn[k] = y[k] / c.target_scale;
}

// Gradient of sum over the batch of (y_hat - t)^2 / B with respect to the
// (BF16-rounded) parameters; idx selects the batch's samples.
//
// A sample's whole pass stays in one warp, lane = hidden neuron, GRAD_GROUP
// samples at a time: lane j keeps row j and column j of W2 and row j of W1
// and of their gradients in registers, so a layer is 32 broadcast 128-bit
// shared-memory reads (the group's values of one neuron) with 4 FP32 FMAs
// each, and the gradient needs no atomics.  The warps' sums meet in shared
// memory once per block (rows padded to 33 so that neither the lane-wise
// writes nor the parameter-wise reads conflict).  Bound by latency: a batch
// of 4096 samples is one pass of 1024 warps (7.5 KFLOP a sample, 0.4 us of
// the chip's FP32 rate).  One sample per thread with a shared-memory atomic
// per parameter and sample, 16 blocks for a batch of 4096, took ~2200 us a
// batch (32 lanes on one address); this kernel takes 10.8 us and the chained
// update 6.4 us (cold).  Eight epochs of 196608 samples in batches of 4096,
// staging and the host's shuffles included: 840 -> 9 ms.
constexpr int GRAD_WARPS = GRAD_BLOCK / 32;
constexpr int GRAD_GROUP = 4;                         // samples a warp takes at a time
constexpr int GRAD_SAMPLES = GRAD_WARPS * GRAD_GROUP;  // per block and pass
// The block's sums in shared memory: element (row i, lane j) of a matrix at i * 33 + j.
constexpr int RED_W2 = 0, RED_W1 = RED_W2 + MLP_H * 33, RED_B1 = RED_W1 + MLP_IN * 33, RED_B2 = RED_B1 + MLP_H,
              RED_W3 = RED_B2 + MLP_H, RED_B3 = RED_W3 + MLP_H, RED_LOSS = RED_B3 + 1, RED_SIZE = RED_LOSS + 1;

// Where parameter p (or the loss, p = MLP_PARAMS) lies in the block's sums.
__device__ __forceinline__ int red_index(int p) {
  if (p < MLP_B1) return RED_W1 + (p % MLP_IN) * 33 + p / MLP_IN;
  if (p < MLP_W2) return RED_B1 + (p - MLP_B1);
  if (p < MLP_B2) return RED_W2 + ((p - MLP_W2) % MLP_H) * 33 + (p - MLP_W2) / MLP_H;
  if (p < MLP_W3) return RED_B2 + (p - MLP_B2);
  if (p < MLP_B3) return RED_W3 + (p - MLP_W3);
  return p == MLP_B3 ? RED_B3 : RED_LOSS;
}

__device__ __forceinline__ float f4_get(const float4 &v, int s) {
  return s == 0 ? v.x : s == 1 ? v.y : s == 2 ? v.z : v.w;
}

__global__ void __launch_bounds__(GRAD_BLOCK, 1)
    mlp_grad_kernel(const float *xn, const float *tn, const int *idx, int B, const __nv_bfloat16 *w,
                    float *partials) {
  __shared__ float4 h1_of[GRAD_WARPS][MLP_H], d2_of[GRAD_WARPS][MLP_H];
  __shared__ float x_of[GRAD_WARPS][GRAD_GROUP][8];  // inputs, then the target
  __shared__ float red[GRAD_WARPS / 2][RED_SIZE];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  release_successor();
  // The samples do not depend on the previous training step: the first group
  // is fetched before waiting for the weights.
  auto fetch = [&](long long first) {
    // 8 lanes a sample: six inputs, the target, one idle
    const int s = lane >> 3, q = lane & 7;
    float v = 0.f;
    if (first + s < B && q < 7) {
      const long long k = idx ? idx[first + s] : first + s;
      v = q < MLP_IN ? xn[k * MLP_IN + q] : tn[k];
    }
    x_of[warp][s][q] = v;
  };
  const long long stride = (long long)gridDim.x * GRAD_SAMPLES;
  long long first = blockIdx.x * GRAD_SAMPLES + warp * GRAD_GROUP;
  fetch(first);
  wait_for_predecessor();
  float w1[MLP_IN], w2row[MLP_H], w2col[MLP_H];
#pragma unroll
  for (int q = 0; q < MLP_IN; q++) w1[q] = __bfloat162float(w[MLP_W1 + lane * MLP_IN + q]);
#pragma unroll
  for (int i = 0; i < MLP_H; i++) {
    w2row[i] = __bfloat162float(w[MLP_W2 + lane * MLP_H + i]);
    w2col[i] = __bfloat162float(w[MLP_W2 + i * MLP_H + lane]);
  }
  const float b1 = __bfloat162float(w[MLP_B1 + lane]), b2 = __bfloat162float(w[MLP_B2 + lane]);
  const float w3 = __bfloat162float(w[MLP_W3 + lane]), b3 = __bfloat162float(w[MLP_B3]);
  float gw1[MLP_IN], gw2[MLP_H], gb1 = 0.f, gb2 = 0.f, gw3 = 0.f, gb3 = 0.f, loss = 0.f;
#pragma unroll
  for (int q = 0; q < MLP_IN; q++) gw1[q] = 0.f;
#pragma unroll
  for (int i = 0; i < MLP_H; i++) gw2[i] = 0.f;
  const float inv_b = 1.0f / (float)B;
  for (; first < B; first += stride) {
    // Samples past the batch count nothing, also where the network overflows
    // on their zero inputs.
    auto live = [&](int s) { return first + s < B; };
    __syncwarp();
    // Layer 1: a = W1 x + b1; h1 = silu(a), p1 = silu'(a).
    float p1[GRAD_GROUP], h[GRAD_GROUP];
#pragma unroll
    for (int s = 0; s < GRAD_GROUP; s++) {
      float a = b1;
#pragma unroll
      for (int q = 0; q < MLP_IN; q++) a += w1[q] * x_of[warp][s][q];
      const float sg = sigmoidf_(a);
      h[s] = live(s) ? a * sg : 0.f;
      p1[s] = sg + h[s] * (1.0f - sg);
    }
    h1_of[warp][lane] = make_float4(h[0], h[1], h[2], h[3]);
    __syncwarp();
    // Layer 2 and the output: y = W3 silu(W2 h1 + b2) + b3.
    float a2[GRAD_GROUP] = {b2, b2, b2, b2};
#pragma unroll
    for (int i = 0; i < MLP_H; i++) {
      const float4 v = h1_of[warp][i];
#pragma unroll
      for (int s = 0; s < GRAD_GROUP; s++) a2[s] += w2row[i] * f4_get(v, s);
    }
    float d2[GRAD_GROUP];
#pragma unroll
    for (int s = 0; s < GRAD_GROUP; s++) {
      const float sg = sigmoidf_(a2[s]);
      const float h2 = live(s) ? a2[s] * sg : 0.f;
      float y = w3 * h2;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) y += __shfl_xor_sync(0xffffffffu, y, off);
      const float r = live(s) ? y + b3 - x_of[warp][s][MLP_IN] : 0.f;
      const float dy = 2.0f * r * inv_b;
      loss += r * r * inv_b;
      gb3 += dy;
      gw3 += dy * h2;
      d2[s] = live(s) ? dy * w3 * (sg + h2 * (1.0f - sg)) : 0.f;
      gb2 += d2[s];
    }
    d2_of[warp][lane] = make_float4(d2[0], d2[1], d2[2], d2[3]);
    __syncwarp();
    // Backward through W2, and the gradients of both layers.
    float d1[GRAD_GROUP] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < MLP_H; i++) {
      const float4 v = h1_of[warp][i], d = d2_of[warp][i];
#pragma unroll
      for (int s = 0; s < GRAD_GROUP; s++) {
        gw2[i] += d2[s] * f4_get(v, s);
        d1[s] += w2col[i] * f4_get(d, s);
      }
    }
#pragma unroll
    for (int s = 0; s < GRAD_GROUP; s++) {
      const float d = d1[s] * p1[s];
      gb1 += d;
#pragma unroll
      for (int q = 0; q < MLP_IN; q++) gw1[q] += d * x_of[warp][s][q];
    }
    __syncwarp();
    fetch(first + stride);
  }
  // Warps 4..7 hand their sums to warps 0..3, then the block adds four rows.
  auto each = [&](auto &&f) {
#pragma unroll
    for (int i = 0; i < MLP_H; i++) f(gw2[i], RED_W2 + i * 33 + lane);
#pragma unroll
    for (int q = 0; q < MLP_IN; q++) f(gw1[q], RED_W1 + q * 33 + lane);
    f(gb1, RED_B1 + lane);
    f(gb2, RED_B2 + lane);
    f(gw3, RED_W3 + lane);
    if (lane == 0) {
      f(gb3, RED_B3);
      f(loss, RED_LOSS);
    }
  };
  float *row = red[warp % (GRAD_WARPS / 2)];
  if (warp >= GRAD_WARPS / 2) each([&](float &v, int k) { row[k] = v; });
  __syncthreads();
  if (warp < GRAD_WARPS / 2) each([&](float &v, int k) { row[k] += v; });
  __syncthreads();
  for (int p = threadIdx.x; p < GRAD_SLOTS; p += GRAD_BLOCK) {
    const int k = red_index(p);
    partials[(long long)blockIdx.x * GRAD_SLOTS + p] = (red[0][k] + red[1][k]) + (red[2][k] + red[3][k]);
  }
}

// Adam's constants of one step.
struct AdamStep {
  float lr, b1, b2, eps, c1, c2;
};

// Sums the block partials in a fixed order (deterministic gradients) and,
// in a training step, applies Adam to the FP32 master weights and refreshes
// the BF16 copy the forward pass uses; the loss goes to loss_out as well
// where that is given.  REDUCE_PARAMS parameters a block, REDUCE_SLICES
// threads to a parameter, so that the ~128 partials of a batch are read 16
// deep instead of one after the other.
constexpr int REDUCE_PARAMS = 32, REDUCE_SLICES = 8;
__global__ void __launch_bounds__(REDUCE_PARAMS *REDUCE_SLICES)
    mlp_update_kernel(const float *partials, int nblocks, float *grad, float *loss_out, bool train, AdamStep s,
                      float *master, float *m, float *v, __nv_bfloat16 *w) {
  __shared__ float sum[REDUCE_SLICES][REDUCE_PARAMS];
  const int lane = threadIdx.x % REDUCE_PARAMS, slice = threadIdx.x / REDUCE_PARAMS;
  const int p = blockIdx.x * REDUCE_PARAMS + lane;
  release_successor();
  wait_for_predecessor();
  float t = 0.f;
  if (p < GRAD_SLOTS) {
#pragma unroll 16
    for (int b = slice; b < nblocks; b += REDUCE_SLICES) t += partials[(long long)b * GRAD_SLOTS + p];
  }
  sum[slice][lane] = t;
  __syncthreads();
  if (slice != 0 || p >= GRAD_SLOTS) return;
  float g = sum[0][lane];
#pragma unroll
  for (int k = 1; k < REDUCE_SLICES; k++) g += sum[k][lane];
  grad[p] = g;
  if (p == MLP_PARAMS) {
    if (loss_out) *loss_out = g;
    return;
  }
  if (!train) return;
  const float mi = s.b1 * m[p] + (1.0f - s.b1) * g;
  const float vi = s.b2 * v[p] + (1.0f - s.b2) * g * g;
  m[p] = mi;
  v[p] = vi;
  const float step = s.lr * (mi / s.c1) / (sqrtf(vi / s.c2) + s.eps);
  master[p] -= step;
  w[p] = __float2bfloat16_rn(master[p]);
}

__global__ void mlp_predict_kernel(const float *xn, long long n, const __nv_bfloat16 *w, float scale,
                                   float *out) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  float x[MLP_IN];
  for (int i = 0; i < MLP_IN; i++) x[i] = xn[k * MLP_IN + i];
  out[k] = scale * mlp_forward(w, x);
}

// The in-step evaluation (mlp_forward_warp) over a batch: 32 samples per
// warp, lanes past n feed zeros.
constexpr int STEP_PREDICT_BLOCK = 128;
__global__ void __launch_bounds__(STEP_PREDICT_BLOCK)
    mlp_predict_step_kernel(const float *raw, long long n, const MlpStep *cl, const MlpConsts kc, float *out) {
  __shared__ __align__(16) unsigned stage[STEP_PREDICT_BLOCK / 32][128];
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  float x[MLP_IN];
  for (int i = 0; i < MLP_IN; i++) x[i] = k < n ? fmaf(raw[k * MLP_IN + i], kc.scale[i], kc.shift[i]) : 0.0f;
  const float y = mlp_forward_warp(cl, x, stage[threadIdx.x >> 5]) + kc.b3;
  if (k < n) out[k] = kc.target_scale * y;
}

__global__ void features_kernel(const float *S, const float *rho, long long n, float *out) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  strain_features(S + k * 6, rho ? rho[k] : 1.0f, out + k * MLP_IN);
}

}  // namespace

struct lbmc_mlp {
  int device = 0;
  MlpClosure host;  // weights (BF16) + normalisation
  std::vector<float> master;
  float *d_master = nullptr, *d_m = nullptr, *d_v = nullptr, *d_grad = nullptr;
  __nv_bfloat16 *d_w = nullptr;
  long long adam_t = 0;
  unsigned long long seed = 0;
  int sms = 1;
  cudaStream_t stream = nullptr;  // the training kernels' (calls return when it is idle)
};

namespace {

template <class T>
cudaError_t upload(T **dst, const T *src, size_t count) {
  cudaError_t e = cudaMalloc(dst, count * sizeof(T) + 16);
  if (e == cudaSuccess && src) e = cudaMemcpy(*dst, src, count * sizeof(T), cudaMemcpyHostToDevice);
  return e;
}

void sync_host_weights(lbmc_mlp *m) {
  for (int p = 0; p < MLP_PARAMS; p++) m->host.w[p] = __float2bfloat16_rn(m->master[p]);
}

}  // namespace

const MlpClosure *lbmc_mlp_closure(const lbmc_mlp *m) { return m ? &m->host : nullptr; }

namespace lbmc {

void mlp_step_layout(const MlpClosure &cl, int iterations, MlpStep &s, MlpConsts &kc) {
  memset(&s, 0, sizeof(s));
  memset(&kc, 0, sizeof(kc));
  // BF16 bit pattern of parameter p, times `scale` (1 or the exact 1/2 that
  // the in-step SiLU expects folded into layers 1 and 2).
  auto bits = [&](int p, float scale) -> unsigned {
    if (p < 0) return 0u;
    const __nv_bfloat16 v = __float2bfloat16_rn(scale * __bfloat162float(cl.w[p]));
    unsigned short b;
    memcpy(&b, &v, sizeof(b));
    return b;
  };
  auto pair = [&](int p0, int p1, float scale) -> unsigned {
    return bits(p0, scale) | (bits(p1, scale) << 16);
  };
  auto set = [](uint4 &v, int j, unsigned w) { (j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w) = w; };
  for (int lane = 0; lane < 32; lane++) {
    const int g = lane >> 2, c = lane & 3;
    for (int j = 0; j < 4; j++) {
      const int n = 8 * j + g, k = 2 * c, col = 8 * j + 2 * c;
      // input 6 is the constant 1 that the bias goes with
      set(s.w1[lane], j, k < MLP_IN ? pair(MLP_W1 + n * MLP_IN + k, MLP_W1 + n * MLP_IN + k + 1, 0.5f)
                                    : pair(MLP_B1 + n, -1, 0.5f));
      for (int kt = 0; kt < 2; kt++)
        for (int r = 0; r < 2; r++) {
          const int kk = 16 * kt + 8 * r + 2 * c;
          set(s.w2[j][lane], 2 * kt + r, pair(MLP_W2 + n * MLP_H + kk, MLP_W2 + n * MLP_H + kk + 1, 0.5f));
        }
      set(s.b2[lane], j, pair(MLP_B2 + col, MLP_B2 + col + 1, 0.5f));
    }
    for (int kt = 0; kt < 2; kt++)
      for (int r = 0; r < 2; r++) {
        const int kk = 16 * kt + 8 * r + 2 * c;
        set(s.w3[lane], 2 * kt + r, g == 0 ? pair(MLP_W3 + kk, MLP_W3 + kk + 1, 1.0f) : 0u);
      }
  }
  for (int i = 0; i < MLP_IN; i++) {
    kc.scale[i] = cl.inv_std[i];
    kc.shift[i] = -cl.mean[i] * cl.inv_std[i];
    kc.lo[i] = cl.lo[i];
    kc.hi[i] = cl.hi[i];
  }
  kc.b3 = __bfloat162float(cl.w[MLP_B3]);
  kc.target_scale = cl.target_scale;
  kc.iterations = iterations;
}

}  // namespace lbmc

extern "C" lbmc_status lbmc_mlp_create(int device, unsigned long long seed, lbmc_mlp **out) {
  if (!out) return merr(LBMC_ERR_INVALID_ARG, "lbmc_mlp_create: out is NULL");
  *out = nullptr;
  if (cudaSetDevice(device) != cudaSuccess) {
    cudaGetLastError();
    return merr(LBMC_ERR_NO_DEVICE, "lbmc_mlp_create: no such device");
  }
  lbmc_mlp *m = new lbmc_mlp();
  m->device = device;
  m->seed = seed;
  m->master.assign(MLP_PARAMS, 0.f);
  std::mt19937_64 rng(seed);
  auto xavier = [&](int off, int fan_in, int fan_out, int count) {
    const float a = std::sqrt(6.0f / (float)(fan_in + fan_out));
    std::uniform_real_distribution<float> u(-a, a);
    for (int k = 0; k < count; k++) m->master[off + k] = u(rng);
  };
  xavier(MLP_W1, MLP_IN, MLP_H, MLP_H * MLP_IN);
  xavier(MLP_W2, MLP_H, MLP_H, MLP_H * MLP_H);
  xavier(MLP_W3, MLP_H, 1, MLP_H);
  memset(&m->host, 0, sizeof(m->host));
  for (int i = 0; i < MLP_IN; i++) {
    m->host.inv_std[i] = 1.f;
    m->host.lo[i] = -1e30f;
    m->host.hi[i] = 1e30f;
  }
  m->host.target_scale = 1.f;
  m->host.iterations = 2;
  sync_host_weights(m);
  cudaError_t e = cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = upload(&m->d_master, m->master.data(), MLP_PARAMS);
  std::vector<float> zeros(GRAD_SLOTS, 0.f);
  if (e == cudaSuccess) e = upload(&m->d_m, zeros.data(), MLP_PARAMS);
  if (e == cudaSuccess) e = upload(&m->d_v, zeros.data(), MLP_PARAMS);
  if (e == cudaSuccess) e = upload(&m->d_grad, zeros.data(), GRAD_SLOTS);
  if (e == cudaSuccess) e = upload(&m->d_w, m->host.w, MLP_PARAMS);
  if (e != cudaSuccess) {
    lbmc_mlp_destroy(m);
    return merr(LBMC_ERR_ALLOC, std::string("lbmc_mlp_create: ") + cudaGetErrorString(e));
  }
  *out = m;
  return LBMC_OK;
}

extern "C" lbmc_status lbmc_mlp_set_normalization(lbmc_mlp *m, const float *mean, const float *std,
                                                  const float *lo, const float *hi, float target_scale) {
  if (!m || !mean || !std || !(target_scale > 0)) return merr(LBMC_ERR_INVALID_ARG, "lbmc_mlp_set_normalization");
  for (int i = 0; i < MLP_IN; i++) {
    if (!(std[i] > 0)) return merr(LBMC_ERR_INVALID_ARG, "lbmc_mlp_set_normalization: std must be > 0");
    m->host.mean[i] = mean[i];
    m->host.inv_std[i] = 1.0f / std[i];
    m->host.lo[i] = lo ? lo[i] : -1e30f;
    m->host.hi[i] = hi ? hi[i] : 1e30f;
  }
  m->host.target_scale = target_scale;
  return LBMC_OK;
}

// Normalised copies of host features / targets on the device.
static lbmc_status stage(lbmc_mlp *m, const float *features, const float *target, long long n, float **xn,
                         float **yn) {
  float *raw = nullptr, *ty = nullptr;
  cudaError_t e = upload(&raw, features, (size_t)n * MLP_IN);
  if (e == cudaSuccess && target) e = upload(&ty, target, (size_t)n);
  if (e == cudaSuccess) e = cudaMalloc(xn, (size_t)n * MLP_IN * sizeof(float));
  if (e == cudaSuccess && target) e = cudaMalloc(yn, (size_t)n * sizeof(float));
  if (e == cudaSuccess) {
    normalise_kernel<<<(unsigned)((n + 255) / 256), 256>>>(raw, ty, n, m->host, *xn, target ? *yn : nullptr);
    e = cudaDeviceSynchronize();
  }
  cudaFree(raw);
  cudaFree(ty);
  if (e != cudaSuccess) return merr(LBMC_ERR_CUDA, std::string("mlp staging: ") + cudaGetErrorString(e));
  return LBMC_OK;
}

// Blocks of the gradient kernel for B samples: one pass of GRAD_SAMPLES a
// block until every SM has one (its registers fill the SM), then several
// passes a block.
static int gradient_blocks(const lbmc_mlp *m, long long B) {
  return (int)std::max(1LL, std::min((B + GRAD_SAMPLES - 1) / GRAD_SAMPLES, (long long)m->sms));
}

// Gradient (and loss) of one batch into d_grad; with `adam` also the step.
static cudaError_t gradient(lbmc_mlp *m, const float *xn, const float *yn, const int *idx, int B, float *partials,
                            const AdamStep *adam, float *loss_out) {
  const int nb = gradient_blocks(m, B);
  cudaError_t e = launch_chained(mlp_grad_kernel, dim3(nb), dim3(GRAD_BLOCK), m->stream, xn, yn, idx, B, m->d_w, partials);
  if (e != cudaSuccess) return e;
  return launch_chained(mlp_update_kernel, dim3((GRAD_SLOTS + REDUCE_PARAMS - 1) / REDUCE_PARAMS),
                        dim3(REDUCE_PARAMS * REDUCE_SLICES), m->stream, partials, nb, m->d_grad, loss_out, adam != nullptr,
                        adam ? *adam : AdamStep{}, m->d_master, m->d_m, m->d_v, m->d_w);
}

extern "C" lbmc_status lbmc_mlp_gradients(lbmc_mlp *m, const float *features, const float *target, long long n,
                                          float *grads, float *loss) {
  if (!m || !features || !target || n < 1 || n > (1 << 24)) return merr(LBMC_ERR_INVALID_ARG, "lbmc_mlp_gradients");
  cudaSetDevice(m->device);
  float *xn = nullptr, *yn = nullptr, *partials = nullptr;
  lbmc_status s = stage(m, features, target, n, &xn, &yn);
  if (s != LBMC_OK) return s;
  cudaError_t e = cudaMalloc(&partials, (size_t)gradient_blocks(m, n) * GRAD_SLOTS * sizeof(float));
  if (e == cudaSuccess) e = gradient(m, xn, yn, nullptr, (int)n, partials, nullptr, nullptr);
  std::vector<float> out(GRAD_SLOTS);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(out.data(), m->d_grad, GRAD_SLOTS * sizeof(float), cudaMemcpyDeviceToHost, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  cudaFree(xn);
  cudaFree(yn);
  cudaFree(partials);
  if (e != cudaSuccess) return merr(LBMC_ERR_CUDA, std::string("lbmc_mlp_gradients: ") + cudaGetErrorString(e));
  if (grads) memcpy(grads, out.data(), MLP_PARAMS * sizeof(float));
  if (loss) *loss = out[MLP_PARAMS];
  return LBMC_OK;
}

extern "C" lbmc_status lbmc_mlp_train(lbmc_mlp *m, const float *features, const float *target, long long n,
                                      int epochs, int batch, float lr, float *loss_history) {
  if (!m || !features || !target || n < 1 || epochs < 1 || batch < 1 || !(lr > 0))
    return merr(LBMC_ERR_INVALID_ARG, "lbmc_mlp_train");
  cudaSetDevice(m->device);
  float *xn = nullptr, *yn = nullptr, *partials = nullptr, *losses = nullptr;
  int *idx = nullptr;
  lbmc_status s = stage(m, features, target, n, &xn, &yn);
  if (s != LBMC_OK) return s;
  // Every LOSS_EVERY-th batch's loss counts in the history; the losses of up to
  // `kept` epochs stay on the device before they are read, so that no batch
  // waits for the host (read after every epoch: 20 batches of 100, 3 epochs,
  // 692 us instead of 664).
  constexpr long long LOSS_EVERY = 16, LOSS_BUFFER = 1 << 12;
  const long long sampled = loss_history ? (n / batch + LOSS_EVERY - 1) / LOSS_EVERY : 0;
  const int kept = (int)std::min<long long>(epochs, std::max(1LL, LOSS_BUFFER / std::max(1LL, sampled)));
  cudaError_t e = cudaMalloc(&partials, (size_t)gradient_blocks(m, batch) * GRAD_SLOTS * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&idx, (size_t)n * sizeof(int));
  if (e == cudaSuccess && sampled > 0) e = cudaMalloc(&losses, (size_t)(sampled * kept) * sizeof(float));
  std::vector<float> loss_of((size_t)(sampled * kept));
  auto fetch_losses = [&]() {
    if (e == cudaSuccess && sampled > 0)
      e = cudaMemcpyAsync(loss_of.data(), losses, loss_of.size() * sizeof(float), cudaMemcpyDeviceToHost, m->stream);
  };
  auto record_epochs = [&](int first, int end) {  // the stream is idle
    for (int ep = first; loss_history && ep < end; ep++) {
      double sum = 0;
      for (long long k = 0; k < sampled; k++) sum += loss_of[(ep - first) * sampled + k];
      loss_history[ep] = (float)(sum / (double)std::max(1LL, sampled));
    }
  };
  std::vector<int> perm(n);
  std::iota(perm.begin(), perm.end(), 0);
  std::mt19937_64 rng(m->seed ^ 0x9E3779B97F4A7C15ull);
  AdamStep a = {lr, 0.9f, 0.999f, 1e-8f, 0.f, 0.f};
  for (int ep = 0; ep < epochs && e == cudaSuccess; ep++) {
    // the host shuffles while the device runs the previous epoch
    std::shuffle(perm.begin(), perm.end(), rng);
    const bool full = ep > 0 && ep % kept == 0;
    if (full) fetch_losses();
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(idx, perm.data(), (size_t)n * sizeof(int), cudaMemcpyHostToDevice, m->stream);
    // perm is pageable: the copy may still read it until the stream is idle
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    if (full && e == cudaSuccess) record_epochs(ep - kept, ep);
    long long batches = 0;
    for (long long off = 0; off + batch <= n && e == cudaSuccess; off += batch, batches++) {
      m->adam_t++;
      a.c1 = 1.0f - std::pow(a.b1, (float)m->adam_t);
      a.c2 = 1.0f - std::pow(a.b2, (float)m->adam_t);
      e = gradient(m, xn, yn, idx + off, batch, partials, &a,
                   losses && batches % LOSS_EVERY == 0 ? losses + ep % kept * sampled + batches / LOSS_EVERY : nullptr);
    }
  }
  fetch_losses();
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(m->master.data(), m->d_master, MLP_PARAMS * sizeof(float), cudaMemcpyDeviceToHost, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  cudaFree(xn);
  cudaFree(yn);
  cudaFree(partials);
  cudaFree(losses);
  cudaFree(idx);
  if (e != cudaSuccess) return merr(LBMC_ERR_CUDA, std::string("lbmc_mlp_train: ") + cudaGetErrorString(e));
  record_epochs((epochs - 1) / kept * kept, epochs);
  sync_host_weights(m);
  return LBMC_OK;
}

extern "C" lbmc_status lbmc_mlp_predict(lbmc_mlp *m, const float *features, long long n, float *out) {
  if (!m || !features || !out || n < 1) return merr(LBMC_ERR_INVALID_ARG, "lbmc_mlp_predict");
  cudaSetDevice(m->device);
  float *xn = nullptr, *yn = nullptr, *res = nullptr;
  lbmc_status s = stage(m, features, nullptr, n, &xn, &yn);
  if (s != LBMC_OK) return s;
  cudaError_t e = cudaMalloc(&res, (size_t)n * sizeof(float));
  if (e == cudaSuccess) {
    mlp_predict_kernel<<<(unsigned)((n + 255) / 256), 256>>>(xn, n, m->d_w, m->host.target_scale, res);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, res, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(xn);
  cudaFree(res);
  if (e != cudaSuccess) return merr(LBMC_ERR_CUDA, std::string("lbmc_mlp_predict: ") + cudaGetErrorString(e));
  return LBMC_OK;
}

extern "C" lbmc_status lbmc_mlp_predict_step(lbmc_mlp *m, const float *features, long long n, float *out) {
  if (!m || !features || !out || n < 1) return merr(LBMC_ERR_INVALID_ARG, "lbmc_mlp_predict_step");
  cudaSetDevice(m->device);
  MlpStep hs;
  MlpConsts kc;
  mlp_step_layout(m->host, 1, hs, kc);
  float *raw = nullptr, *res = nullptr;
  MlpStep *ds = nullptr;
  cudaError_t e = upload(&raw, features, (size_t)n * MLP_IN);
  if (e == cudaSuccess) e = upload(&ds, &hs, 1);
  if (e == cudaSuccess) e = cudaMalloc(&res, (size_t)n * sizeof(float));
  if (e == cudaSuccess) {
    const long long blocks = (n + STEP_PREDICT_BLOCK - 1) / STEP_PREDICT_BLOCK;
    mlp_predict_step_kernel<<<(unsigned)blocks, STEP_PREDICT_BLOCK>>>(raw, n, ds, kc, res);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, res, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(raw);
  cudaFree(ds);
  cudaFree(res);
  if (e != cudaSuccess) return merr(LBMC_ERR_CUDA, std::string("lbmc_mlp_predict_step: ") + cudaGetErrorString(e));
  return LBMC_OK;
}

extern "C" lbmc_status lbmc_mlp_features(int device, const float *strain6, const float *rho, long long n,
                                         float *features6) {
  if (!strain6 || !features6 || n < 1) return merr(LBMC_ERR_INVALID_ARG, "lbmc_mlp_features");
  if (cudaSetDevice(device) != cudaSuccess) return merr(LBMC_ERR_NO_DEVICE, "lbmc_mlp_features");
  float *S = nullptr, *r = nullptr, *f = nullptr;
  cudaError_t e = upload(&S, strain6, (size_t)n * 6);
  if (e == cudaSuccess && rho) e = upload(&r, rho, (size_t)n);
  if (e == cudaSuccess) e = cudaMalloc(&f, (size_t)n * MLP_IN * sizeof(float));
  if (e == cudaSuccess) {
    features_kernel<<<(unsigned)((n + 255) / 256), 256>>>(S, r, n, f);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(features6, f, (size_t)n * MLP_IN * sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(S);
  cudaFree(r);
  cudaFree(f);
  if (e != cudaSuccess) return merr(LBMC_ERR_CUDA, std::string("lbmc_mlp_features: ") + cudaGetErrorString(e));
  return LBMC_OK;
}

extern "C" lbmc_status lbmc_mlp_get_params(lbmc_mlp *m, float *params) {
  if (!m || !params) return merr(LBMC_ERR_INVALID_ARG, "lbmc_mlp_get_params");
  for (int p = 0; p < MLP_PARAMS; p++) params[p] = __bfloat162float(m->host.w[p]);
  return LBMC_OK;
}

extern "C" lbmc_status lbmc_mlp_set_params(lbmc_mlp *m, const float *params) {
  if (!m || !params) return merr(LBMC_ERR_INVALID_ARG, "lbmc_mlp_set_params");
  cudaSetDevice(m->device);
  for (int p = 0; p < MLP_PARAMS; p++) m->master[p] = params[p];
  sync_host_weights(m);
  cudaError_t e = cudaMemcpy(m->d_master, m->master.data(), MLP_PARAMS * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(m->d_w, m->host.w, MLP_PARAMS * sizeof(__nv_bfloat16), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(m->d_m, 0, MLP_PARAMS * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(m->d_v, 0, MLP_PARAMS * sizeof(float));
  m->adam_t = 0;
  if (e != cudaSuccess) return merr(LBMC_ERR_CUDA, "lbmc_mlp_set_params");
  return LBMC_OK;
}

extern "C" lbmc_status lbmc_mlp_destroy(lbmc_mlp *m) {
  if (!m) return LBMC_OK;
  cudaSetDevice(m->device);
  cudaFree(m->d_master);
  cudaFree(m->d_m);
  cudaFree(m->d_v);
  cudaFree(m->d_grad);
  cudaFree(m->d_w);
  if (m->stream) cudaStreamDestroy(m->stream);
  delete m;
  return LBMC_OK;
}
