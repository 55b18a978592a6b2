// screen.cu - the learned screen: a per-pixel MLP B -> 64 -> 32 -> 1 that
// proposes candidate pixels for the plain ACE detector to re-score.
//
// No counterpart in the reference.  Trained on the device on the plain
// detector's own ACE decisions over synthetic frames, by the kernels here:
//   normaliser   per band: mean and a power-of-two scale s_b ~ 1/sigma_b
//                (power of two, so that it folds exactly into fp16 weights);
//   batch        training samples: positives drawn from the detector's
//                compacted positive list, the rest uniform over the frame;
//   gather       features (x_b - mean_b) s_b rounded to bfloat16, band-major
//                [Bp][n], and the 0/1 labels from the score map;
//   gradients    forward (bfloat16 weights, FP32 accumulation, h1 rounded to
//                bfloat16 as inference does), deltas and dW = delta^T act in
//                one kernel over chunks of samples; per-CTA partials added in
//                a fixed order;
//   adam         FP32 master weights; the forward reads them rounded.
// Inference (screen_tc_kernel, below) runs layers 1 and 2 on the tensor
// cores straight from the fp16 cube.
//
// Parameter layout (FP32), Bp = bands rounded up to 64:
//   W1[64][Bp] | b1[64] | W2[32][64] | b2[32] | w3[32] | b3
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "synth.h"
#include "launch_state.h"
#include "tc.cuh"

namespace hsi_b200 {
namespace {

constexpr int kH1 = 64, kH2 = 32;

__host__ __device__ inline int padded_bands(int B) { return (B + 63) / 64 * 64; }
__host__ __device__ inline int64_t param_count(int B) {
  return static_cast<int64_t>(kH1) * padded_bands(B) + kH1 + kH2 * kH1 + kH2 + kH2 + 1;
}

struct ParamView {
  float *W1, *b1, *W2, *b2, *w3, *b3;
};
__host__ __device__ inline ParamView view(float* p, int B) {
  ParamView v;
  v.W1 = p;
  v.b1 = v.W1 + static_cast<int64_t>(kH1) * padded_bands(B);
  v.W2 = v.b1 + kH1;
  v.b2 = v.W2 + kH2 * kH1;
  v.w3 = v.b2 + kH2;
  v.b3 = v.w3 + kH2;
  return v;
}

__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// ---- initialisation: He-uniform from a counter hash, padding columns zero ----
__global__ void init_kernel(float* __restrict__ p, int B, uint64_t seed) {
  const int Bp = padded_bands(B);
  const int64_t n = param_count(B);
  const ParamView v = view(p, B);
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const double u = static_cast<double>(hsi_mix64(seed ^ (0x9E3779B97F4A7C15ull * (i + 1))) >> 11) * 0x1.0p-53;
    float val = 0.0f;
    float* q = p + i;
    if (q < v.b1) {
      const int b = static_cast<int>(i % Bp);
      if (b < B) val = static_cast<float>((2.0 * u - 1.0) * sqrt(6.0 / B));
    } else if (q >= v.W2 && q < v.b2) {
      val = static_cast<float>((2.0 * u - 1.0) * sqrt(6.0 / kH1));
    } else if (q >= v.w3 && q < v.b3) {
      val = static_cast<float>((2.0 * u - 1.0) * sqrt(6.0 / kH2));
    }
    p[i] = val;  // biases start at zero
  }
}

// ---- normaliser: mean and power-of-two scale from raw FP64 moments ----------
__global__ void normaliser_kernel(const double* __restrict__ m, int B, float* __restrict__ norm) {
  const int Bp = padded_bands(B);
  const double N = m[B + static_cast<int64_t>(B) * B];
  for (int b = threadIdx.x; b < Bp; b += blockDim.x) {
    float mu = 0.0f, s = 0.0f;
    if (b < B && N > 0.0) {
      const double mean = m[b] / N;
      const double var = m[B + static_cast<int64_t>(b) * B + b] / N - mean * mean;
      mu = static_cast<float>(mean);
      // s = 2^round(-log2 sigma): exact in fp16 weights; 1 for a constant band;
      // clamped so that |bfloat16 weight| * s stays inside the fp16 range
      s = var > 0.0 ? static_cast<float>(exp2(rint(-0.5 * log2(var)))) : 1.0f;
      s = fminf(fmaxf(s, 0x1.0p-14f), 0x1.0p12f);
    }
    norm[b] = mu;
    norm[Bp + b] = s;
  }
}

// ---- training batch: n_pos draws from the positive list, the rest uniform ----
__global__ void batch_kernel(const hsi_detection* __restrict__ pos, const uint32_t* __restrict__ pos_count,
                             int pos_capacity, int width, int64_t pixels, const float* __restrict__ score,
                             float threshold, uint64_t seed, int n_pos, int n, int32_t* __restrict__ index,
                             float* __restrict__ labels) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const uint32_t np = min(*pos_count, static_cast<uint32_t>(pos_capacity));
  const uint64_t h = hsi_mix64(seed * 0x100000001B3ull + static_cast<uint64_t>(s));
  int64_t p;
  if (s < n_pos && np > 0) {
    const hsi_detection d = pos[h % np];
    p = static_cast<int64_t>(d.y) * width + d.x;
  } else {
    p = static_cast<int64_t>(h % static_cast<uint64_t>(pixels));
  }
  index[s] = static_cast<int32_t>(p);
  labels[s] = score[p] >= threshold ? 1.0f : 0.0f;
}

// ---- gather: features [Bp][n], (x - mean) s rounded to bfloat16 --------------
template <typename T>
__global__ void gather_kernel(const T* __restrict__ cube, int64_t stride, int B, const float* __restrict__ norm,
                              const int32_t* __restrict__ index, int n, float* __restrict__ features) {
  const int Bp = padded_bands(B);
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (s >= n) return;
  float v = 0.0f;
  if (b < B) {
    float x;
    if constexpr (sizeof(T) == 4) {
      x = cube[static_cast<int64_t>(b) * stride + index[s]];
    } else {
      x = __half2float(cube[static_cast<int64_t>(b) * stride + index[s]]);
    }
    v = bf16r((x - norm[b]) * norm[Bp + b]);
  }
  features[static_cast<int64_t>(b) * n + s] = v;
}

// ---- one training pass: forward, deltas and gradient partials ----------------
//
// A CTA takes chunks of S samples with the whole network in shared memory:
// the chunk's features, W1 and W2 rounded to bfloat16, and the activations
// and deltas, which never reach global memory.  All five products run from
// shared memory in FP32 register tiles; the weight gradients stay in registers
// over a CTA's chunks, and each CTA writes one partial of every parameter that
// reduce_kernel adds in a fixed order (deterministic, and shorter sums than
// one chain over the batch).
// 8192 samples of 224 bands: 28 us here and 3.4 us in reduce_kernel, where a
// one-thread-per-sample forward, six row-dot launches (20 blocks, each one
// chain over the whole batch) and a loss launch took 1.58 ms.
// Bound: shared-memory reads, then FP32 FMA.  Layer 1 and dW1 are 64 x Bp products per sample each,
// 7.5 us on 128 SMs for 8192 samples of 224 bands; the tiles read one shared
// value per 8 (layer 1) or 16 (dW1) FMAs, so shared memory keeps up.  S = 64
// amortises the 64 KB of W1 a CTA stages; 32 up to 4736 samples (148 chunks),
// where 64 would leave more than half of the SMs without one.
constexpr int kTrainThreads = 256;
constexpr int kTrainMaxCtas = 148;  // partials in the workspace; more chunks than that are looped over
constexpr int kW1Stride = kH1 + 2;  // W1^T rows [b][64]: 2-way conflicts on the transposing store, float2 reads
constexpr int kW2Stride = kH2 + 4;  // W2^T rows [j][32]: float4 reads along k

__host__ __device__ inline int train_chunk(int n) { return n <= 32 * kTrainMaxCtas ? 32 : 64; }
__host__ __device__ inline int train_ctas(int n) {
  const int chunks = (n + train_chunk(n) - 1) / train_chunk(n);
  return chunks < kTrainMaxCtas ? chunks : kTrainMaxCtas;
}
// floats of one CTA's partial: every parameter, then the loss sum, padded to 128 bytes
__host__ __device__ inline int64_t partial_stride(int B) { return (param_count(B) + 1 + 31) / 32 * 32; }

template <int S>
struct TrainSmem {
  static constexpr int kS = S + 4;  // sample-minor rows: 16-byte aligned, 8 rows apart in the banks
  static __host__ __device__ constexpr int floats(int bp) {
    return bp * kS + bp * kW1Stride + kH1 * kW2Stride + kH1 * kS /* h1 */ + S * (kH1 + 4) /* delta1^T */ +
           2 * kH2 * kS /* z2 -> delta2, h2 */ + 2 * S /* delta3, loss */ + kH1 + 2 * kH2 /* b1, b2, w3 */;
  }
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(valid ? 4 : 0)
               : "memory");
}

// NB = Bp / 64.  `vec`: the features' rows start on 16 bytes (n a multiple of 4).
template <int NB, int S>
__global__ void __launch_bounds__(kTrainThreads, 1)
    train_kernel(const float* __restrict__ params, int B, const float* __restrict__ X,
                 const float* __restrict__ labels, int n, float pos_weight, int vec, float* __restrict__ partials) {
  constexpr int Bp = 64 * NB;
  constexpr int kS = TrainSmem<S>::kS;
  constexpr int kD = kH1 + 4;  // delta1^T row: [s][64]
  extern __shared__ __align__(16) float sw[];
  float* xs = sw;                         // [Bp][kS]
  float* w1t = xs + Bp * kS;              // [Bp][kW1Stride], bfloat16 values
  float* w2t = w1t + Bp * kW1Stride;      // [64][kW2Stride], bfloat16 values
  float* h1 = w2t + kH1 * kW2Stride;      // [64][kS]
  float* d1t = h1 + kH1 * kS;             // [S][kD]
  float* d2 = d1t + S * kD;               // [32][kS]: z2, then delta2
  float* h2 = d2 + kH2 * kS;              // [32][kS]
  float* d3 = h2 + kH2 * kS;              // [S]
  float* ls = d3 + S;                     // [S]
  float* b1 = ls + S;
  float* b2 = b1 + kH1;
  float* w3 = b2 + kH2;
  const ParamView v = view(const_cast<float*>(params), B);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunks = (n + S - 1) / S;

  auto load_features = [&](int chunk) {
    const int s0 = chunk * S;
    if (vec) {
      for (int e = tid; e < Bp * (S / 4); e += kTrainThreads) {
        const int b = e / (S / 4), s = e % (S / 4) * 4;
        const bool in = s0 + s < n;
        cp_async16(xs + b * kS + s, X + static_cast<int64_t>(b) * n + (in ? s0 + s : 0), in);
      }
    } else {
      for (int e = tid; e < Bp * S; e += kTrainThreads) {
        const int b = e / S, s = e % S;
        const bool in = s0 + s < n;
        cp_async4(xs + b * kS + s, X + static_cast<int64_t>(b) * n + (in ? s0 + s : 0), in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load_features(blockIdx.x);
#pragma unroll 16
  for (int e = tid; e < Bp * kH1; e += kTrainThreads) {  // 16 loads in flight a thread
    const int j = e / Bp, b = e % Bp;
    w1t[b * kW1Stride + j] = bf16r(v.W1[e]);
  }
  for (int e = tid; e < kH2 * kH1; e += kTrainThreads) w2t[(e % kH1) * kW2Stride + e / kH1] = bf16r(v.W2[e]);
  if (tid < kH1) b1[tid] = v.b1[tid];
  if (tid < kH2) {
    b2[tid] = v.b2[tid];
    w3[tid] = bf16r(v.w3[tid]);
  }
  const float b3 = v.b3[0];

  // gradients of this CTA: dW1 rows 8 warp .. + 7 by columns lane + 32 i (row
  // pairs packed), dW2 rows 4 warp .. + 3 by columns lane and lane + 32, and
  // one bias / w3 / loss element on each of the first threads
  float2 g1[4][2 * NB];
  float g2[4][2];
  float gs = 0.0f;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
#pragma unroll
    for (int i = 0; i < 2 * NB; ++i) g1[r][i] = make_float2(0.0f, 0.0f);
    g2[r][0] = g2[r][1] = 0.0f;
  }

  for (int chunk = blockIdx.x; chunk < chunks; chunk += gridDim.x) {
    const int s0 = chunk * S;
    if (chunk != static_cast<int>(blockIdx.x)) {
      __syncthreads();  // the previous chunk's features and deltas are done with
      load_features(chunk);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // layer 1: 4 hidden units x S/16 samples a thread, bands in order
    {
      constexpr int kQ = S / 16;
      const int ss = (tid & 15) * kQ, j0 = (tid >> 4) * 4;
      float2 z[2][kQ];
#pragma unroll
      for (int q = 0; q < kQ; ++q) {
        z[0][q] = make_float2(b1[j0], b1[j0 + 1]);
        z[1][q] = make_float2(b1[j0 + 2], b1[j0 + 3]);
      }
#pragma unroll 8
      for (int b = 0; b < B; ++b) {
        const float2 wa = *reinterpret_cast<const float2*>(w1t + b * kW1Stride + j0);
        const float2 wb = *reinterpret_cast<const float2*>(w1t + b * kW1Stride + j0 + 2);
        float x[kQ];
        if constexpr (kQ == 4) {
          const float4 t = *reinterpret_cast<const float4*>(xs + b * kS + ss);
          x[0] = t.x, x[1] = t.y, x[2] = t.z, x[3] = t.w;
        } else {
          const float2 t = *reinterpret_cast<const float2*>(xs + b * kS + ss);
          x[0] = t.x, x[1] = t.y;
        }
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
          const float2 xx = make_float2(x[q], x[q]);
          z[0][q] = ffma2(wa, xx, z[0][q]);
          z[1][q] = ffma2(wb, xx, z[1][q]);
        }
      }
#pragma unroll
      for (int q = 0; q < kQ; ++q) {
        const bool in = s0 + ss + q < n;
        h1[j0 * kS + ss + q] = in ? bf16r(fmaxf(z[0][q].x, 0.0f)) : 0.0f;
        h1[(j0 + 1) * kS + ss + q] = in ? bf16r(fmaxf(z[0][q].y, 0.0f)) : 0.0f;
        h1[(j0 + 2) * kS + ss + q] = in ? bf16r(fmaxf(z[1][q].x, 0.0f)) : 0.0f;
        h1[(j0 + 3) * kS + ss + q] = in ? bf16r(fmaxf(z[1][q].y, 0.0f)) : 0.0f;
      }
    }
    __syncthreads();
    // layer 2: 4 units x S/32 samples a thread
    {
      constexpr int kQ = S / 32;
      const int k0 = warp * 4;
      float z[4][kQ];
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int q = 0; q < kQ; ++q) z[k][q] = b2[k0 + k];
#pragma unroll 8
      for (int j = 0; j < kH1; ++j) {
        const float4 w = *reinterpret_cast<const float4*>(w2t + j * kW2Stride + k0);
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
          const float h = h1[j * kS + lane + 32 * q];
          z[0][q] = fmaf(w.x, h, z[0][q]);
          z[1][q] = fmaf(w.y, h, z[1][q]);
          z[2][q] = fmaf(w.z, h, z[2][q]);
          z[3][q] = fmaf(w.w, h, z[3][q]);
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
          d2[(k0 + k) * kS + lane + 32 * q] = z[k][q];
          h2[(k0 + k) * kS + lane + 32 * q] = fmaxf(z[k][q], 0.0f);
        }
    }
    __syncthreads();
    // layer 3, the loss and delta3: one thread a sample
    if (tid < S) {
      const bool in = s0 + tid < n;
      float z3 = b3;
#pragma unroll
      for (int k = 0; k < kH2; ++k) z3 = fmaf(w3[k], h2[k * kS + tid], z3);
      const float y = in ? labels[s0 + tid] : 0.0f, w = y > 0.5f ? pos_weight : 1.0f;
      const float sp = z3 > 0.0f ? z3 + log1pf(expf(-z3)) : log1pf(expf(z3));
      ls[tid] = in ? w * (sp - y * z3) : 0.0f;
      d3[tid] = in ? w * (1.0f / (1.0f + expf(-z3)) - y) / static_cast<float>(n) : 0.0f;
    }
    __syncthreads();
    for (int e = tid; e < kH2 * S; e += kTrainThreads) {
      const int k = e / S, s = e % S;
      const float z = d2[k * kS + s];
      d2[k * kS + s] = (z > 0.0f && s0 + s < n) ? d3[s] * w3[k] : 0.0f;
    }
    __syncthreads();
    // delta1_j = [h1_j > 0] sum_k delta2_k W2_kj: 8 units (4 rows of two warps' halves) x S/32 samples a thread
    {
      constexpr int kQ = S / 32;
      const int j0 = warp * 8;
#pragma unroll
      for (int jj = 0; jj < 8; jj += 4) {
        float acc[4][kQ];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int q = 0; q < kQ; ++q) acc[j][q] = 0.0f;
#pragma unroll 2
        for (int k = 0; k < kH2; k += 4) {
          float w[4][4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float4 t = *reinterpret_cast<const float4*>(w2t + (j0 + jj + j) * kW2Stride + k);
            w[j][0] = t.x, w[j][1] = t.y, w[j][2] = t.z, w[j][3] = t.w;
          }
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int q = 0; q < kQ; ++q) {
              const float d = d2[(k + kk) * kS + lane + 32 * q];
#pragma unroll
              for (int j = 0; j < 4; ++j) acc[j][q] = fmaf(d, w[j][kk], acc[j][q]);
            }
        }
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
          const int s = lane + 32 * q;
          float4 t;
          t.x = h1[(j0 + jj) * kS + s] > 0.0f ? acc[0][q] : 0.0f;
          t.y = h1[(j0 + jj + 1) * kS + s] > 0.0f ? acc[1][q] : 0.0f;
          t.z = h1[(j0 + jj + 2) * kS + s] > 0.0f ? acc[2][q] : 0.0f;
          t.w = h1[(j0 + jj + 3) * kS + s] > 0.0f ? acc[3][q] : 0.0f;
          *reinterpret_cast<float4*>(d1t + s * kD + j0 + jj) = t;
        }
      }
    }
    __syncthreads();
    // dW1 += delta1 X^T, four samples at a time: X by float4 along the samples
    // (rows of kS floats: 8 lanes cover the banks), delta1 broadcast
#pragma unroll 1
    for (int s = 0; s < S; s += 4) {
      float2 d[4][4];  // [sample][row pair]
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 a = *reinterpret_cast<const float4*>(d1t + (s + q) * kD + warp * 8);
        const float4 c = *reinterpret_cast<const float4*>(d1t + (s + q) * kD + warp * 8 + 4);
        d[q][0] = make_float2(a.x, a.y), d[q][1] = make_float2(a.z, a.w);
        d[q][2] = make_float2(c.x, c.y), d[q][3] = make_float2(c.z, c.w);
      }
#pragma unroll
      for (int i = 0; i < 2 * NB; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(xs + (lane + 32 * i) * kS + s);
        const float xq[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 xx = make_float2(xq[q], xq[q]);
#pragma unroll
          for (int r = 0; r < 4; ++r) g1[r][i] = ffma2(d[q][r], xx, g1[r][i]);
        }
      }
    }
    // dW2 += delta2 h1^T, the same way
#pragma unroll 2
    for (int s = 0; s < S; s += 4) {
      const float4 ha = *reinterpret_cast<const float4*>(h1 + lane * kS + s);
      const float4 hb = *reinterpret_cast<const float4*>(h1 + (lane + 32) * kS + s);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float4 d = *reinterpret_cast<const float4*>(d2 + (warp * 4 + r) * kS + s);
        g2[r][0] = fmaf(d.w, ha.w, fmaf(d.z, ha.z, fmaf(d.y, ha.y, fmaf(d.x, ha.x, g2[r][0]))));
        g2[r][1] = fmaf(d.w, hb.w, fmaf(d.z, hb.z, fmaf(d.y, hb.y, fmaf(d.x, hb.x, g2[r][1]))));
      }
    }
    // db1 (threads 0..63), db2 (64..95), dw3 (96..127), db3 (128), loss (160)
    if (tid < kH1) {
#pragma unroll 8
      for (int s = 0; s < S; ++s) gs += d1t[s * kD + tid];
    } else if (tid < kH1 + kH2) {
      const float* r = d2 + (tid - kH1) * kS;
#pragma unroll 8
      for (int s = 0; s < S; ++s) gs += r[s];
    } else if (tid < kH1 + 2 * kH2) {
      const float* r = h2 + (tid - kH1 - kH2) * kS;
#pragma unroll 8
      for (int s = 0; s < S; ++s) gs = fmaf(d3[s], s0 + s < n ? r[s] : 0.0f, gs);
    } else if (tid == kH1 + 2 * kH2 || tid == kH1 + 3 * kH2) {
      const float* r = tid == kH1 + 2 * kH2 ? d3 : ls;
#pragma unroll 8
      for (int s = 0; s < S; ++s) gs += r[s];
    }
  }

  const ParamView g = view(partials + static_cast<int64_t>(blockIdx.x) * partial_stride(B), B);
#pragma unroll
  for (int i = 0; i < 2 * NB; ++i)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      g.W1[(warp * 8 + 2 * r) * Bp + lane + 32 * i] = g1[r][i].x;
      g.W1[(warp * 8 + 2 * r + 1) * Bp + lane + 32 * i] = g1[r][i].y;
    }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    g.W2[(warp * 4 + r) * kH1 + lane] = g2[r][0];
    g.W2[(warp * 4 + r) * kH1 + lane + 32] = g2[r][1];
  }
  if (tid < kH1) g.b1[tid] = gs;
  else if (tid < kH1 + kH2) g.b2[tid - kH1] = gs;
  else if (tid < kH1 + 2 * kH2) g.w3[tid - kH1 - kH2] = gs;
  else if (tid == kH1 + 2 * kH2) g.b3[0] = gs;
  else if (tid == kH1 + 3 * kH2) g.b3[1] = gs;
}

// out[i] = sum over the CTAs' partials; 32 parameters by 8 slices of the
// partials a block, so a thread has its few loads in flight together (one
// thread per parameter would chain 128 of them).  The element after the last
// parameter is the loss sum.
__global__ void __launch_bounds__(256) reduce_kernel(const float* __restrict__ partials, int nparts, int64_t stride,
                                                    int64_t count, int n, float* __restrict__ grads,
                                                    float* __restrict__ loss) {
  __shared__ float s[8][33];
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 32 + lane;
  float t = 0.0f;
  if (i <= count) {
#pragma unroll 8
    for (int c = slice; c < nparts; c += 8) t += partials[c * stride + i];
  }
  s[slice][lane] = t;
  __syncthreads();
  if (slice == 0 && i <= count) {
    float r = s[0][lane];
#pragma unroll
    for (int w = 1; w < 8; ++w) r += s[w][lane];
    if (i < count) grads[i] = r;
    else if (loss) *loss = r / static_cast<float>(n);
  }
}

template <int NB, int S>
cudaError_t launch_train(const float* params, int B, const float* X, const float* labels, int n, float pos_weight,
                         int vec, float* partials, cudaStream_t s) {
  constexpr int smem = static_cast<int>(sizeof(float)) * TrainSmem<S>::floats(64 * NB);
  const cudaError_t e = raise_smem_limit(train_kernel<NB, S>, smem);
  if (e != cudaSuccess) return e;
  train_kernel<NB, S><<<train_ctas(n), kTrainThreads, smem, s>>>(params, B, X, labels, n, pos_weight, vec, partials);
  return cudaGetLastError();
}

// Room for the partials of any batch of up to n samples at any band count, as the
// callers' workspace had before: batches of 32-sample chunks (up to 4736 samples)
// leave up to 148 partials, 8192 samples in 64-sample chunks 128, so that the
// latter's own would be too small for a shorter batch.
size_t train_bytes(int n) {
  const int chunks = n / 32 + (n % 32 != 0);
  return sizeof(float) * static_cast<size_t>(std::min(chunks, kTrainMaxCtas)) *
             static_cast<size_t>(partial_stride(HSI_MAX_BANDS)) +
         256;
}

__global__ void adam_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                            const float* __restrict__ g, int64_t n, float lr, float b1, float b2, float eps, float c1,
                            float c2) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// ---- inference on the tensor cores -------------------------------------------
//
// Per 128-pixel tile:  layer 1 on the tensor cores straight from the fp16
// cube: two 64-pixel x Bp-band TMA boxes with the 128-byte swizzle are an
// MN-major A operand; B = W1' = bf16(W1) diag(s) in fp16 (exact: s is a
// power of two), b1' = b1 - W1' mean.  Layer 2: h1 = relu(.) rounded to
// bfloat16 into a K-major shared tile, times bf16(W2).  Layer 3 (32 -> 1) on
// the CUDA cores.  Output: one FP32 logit per pixel.
// Warps: 0 TMA, 1 MMA issuer (+ TMEM), 2-5 epilogue (one per TMEM lane
// quarter).  TMEM: layer-1 accumulators double-buffered at columns 0 / 64,
// layer 2 at 128.
constexpr int kScrTile = 128, kScrBox = 64;
constexpr int kScrThreads = 6 * 32;
constexpr uint32_t kScrTmemCols = 256;

struct ScreenOps {
  unsigned char w1[4][kH1 * 128];  // up to 4 K-blocks of 64 bands: 64 rows x 128 B, fp16, swizzled K-major
  unsigned char w2[kH2 * 128];     // 32 rows x 64 hidden bf16, swizzled K-major
  float b1[kH1];
  float b2[kH2];
  float w3[kH2];
  float b3;
};

__device__ __forceinline__ uint32_t sw128(int row, int byte) {
  return static_cast<uint32_t>((row >> 3) * 1024 + (row & 7) * 128 + ((((byte >> 4) ^ (row & 7))) << 4) + (byte & 15));
}

// Fold the normaliser into layer 1, round and lay out the weights: one block
// per hidden unit of layer 1 and one for the rest.  One block for everything
// took 45 us ahead of the inference (64 dependent rounds of loads, then the
// FP64 sums of 64 units on 8 warps); 65 blocks take 4.
__global__ void __launch_bounds__(256) pack_kernel(const float* __restrict__ params, int B,
                                                  const float* __restrict__ norm, ScreenOps* __restrict__ ops) {
  __shared__ float used[256];  // the unit's fp16 weights
  const int Bp = padded_bands(B);
  const ParamView v = view(const_cast<float*>(params), B);
  const int j = blockIdx.x, b = threadIdx.x;
  if (j < kH1) {
    if (b < Bp) {
      const float w = b < B ? bf16r(v.W1[static_cast<int64_t>(j) * Bp + b]) * norm[Bp + b] : 0.0f;
      const __half h = __float2half_rn(w);
      *reinterpret_cast<__half*>(&ops->w1[b >> 6][sw128(j, (b & 63) * 2)]) = h;
      used[b] = __half2float(h);
    }
    __syncthreads();
    // b1' = b1 - sum_b W1'_jb mean_b in FP64, from the fp16 weights actually used
    if (threadIdx.x < 32) {
      double acc = 0.0;
      for (int i = threadIdx.x; i < B; i += 32) acc += static_cast<double>(used[i]) * static_cast<double>(norm[i]);
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (threadIdx.x == 0) ops->b1[j] = static_cast<float>(static_cast<double>(v.b1[j]) - acc);
    }
    return;
  }
  for (int e = threadIdx.x; e < kH2 * kH1; e += blockDim.x)
    *reinterpret_cast<__nv_bfloat16*>(&ops->w2[sw128(e / kH1, e % kH1 * 2)]) = __float2bfloat16_rn(v.W2[e]);
  if (threadIdx.x < kH2) {
    ops->b2[threadIdx.x] = v.b2[threadIdx.x];
    ops->w3[threadIdx.x] = bf16r(v.w3[threadIdx.x]);
  }
  if (threadIdx.x == 0) ops->b3 = v.b3[0];
}

struct ScreenArgs {
  int64_t pixels;
  int bands_padded;
  const ScreenOps* ops;
  float* logits;
  int* status;
};

__global__ void __launch_bounds__(kScrThreads, 1)
    screen_tc_kernel(const __grid_constant__ CUtensorMap cube_map, const ScreenArgs args) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int Bp = args.bands_padded;
  const int kb_count = Bp / 64;
  const uint32_t box_bytes = static_cast<uint32_t>(Bp) * 128;  // Bp bands x 64 px x 2 B
  const uint32_t stage_bytes = 2 * box_bytes;
  const int kIn = (128 * 1024) / stage_bytes < 4 ? (128 * 1024) / stage_bytes : 4;  // 2 or 4 stages
  unsigned char* in = smem;                                   // kIn stages
  unsigned char* w1 = in + kIn * stage_bytes;                  // kb_count x 8 KB
  unsigned char* w2 = w1 + kb_count * kH1 * 128;               // 4 KB
  unsigned char* h1 = w2 + kH2 * 128;                          // 2 x 16 KB (1024-aligned)
  float* cst = reinterpret_cast<float*>(h1 + 2 * kScrTile * 128);  // b1, b2, w3, b3
  uint64_t* bars = reinterpret_cast<uint64_t*>(cst + kH1 + 2 * kH2 + 4);
  uint64_t* in_full = bars;
  uint64_t* in_empty = bars + 4;
  uint64_t* acc1_full = bars + 8;
  uint64_t* acc1_empty = bars + 10;
  uint64_t* h1_full = bars + 12;
  uint64_t* h1_empty = bars + 14;
  uint64_t* acc2_full = bars + 16;
  uint64_t* acc2_empty = bars + 17;
  uint64_t* w_full = bars + 18;
  uint64_t* mma_done = bars + 19;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 21);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t P = args.pixels;
  const int64_t ntiles = div_up<int64_t>(P, kScrTile);
  const int n = ntiles > blockIdx.x ? static_cast<int>((ntiles - 1 - blockIdx.x) / gridDim.x + 1) : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kIn; ++s) {
      mbar_init(&in_full[s], 1);
      mbar_init(&in_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc1_full[b], 1);
      mbar_init(&acc1_empty[b], 4);
      mbar_init(&h1_full[b], 4);
      mbar_init(&h1_empty[b], 1);
    }
    mbar_init(acc2_full, 1);
    mbar_init(acc2_empty, 4);
    mbar_init(w_full, 1);
    mbar_init(mma_done, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  for (int i = threadIdx.x; i < kH1 + 2 * kH2 + 1; i += blockDim.x) cst[i] = args.ops->b1[i];
  if (warp == 1) tmem_alloc(tmem_slot, kScrTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      prefetch_tensormap(&cube_map);
      mbar_arrive_expect_tx(w_full, kb_count * kH1 * 128 + kH2 * 128);
      for (int kb = 0; kb < kb_count; ++kb) bulk_g2s(w1 + kb * kH1 * 128, args.ops->w1[kb], kH1 * 128, w_full);
      bulk_g2s(w2, args.ops->w2, kH2 * 128, w_full);
      uint32_t pending = 0, parity = 0;
      for (int i = 0; i < n; ++i) {
        const int s = i % kIn;
        const uint32_t ph = (i / kIn) & 1u;
        if (*abort_flag || !mbar_wait_idle(&in_empty[s], ph ^ 1u)) {
          record_error(args.status, HSI_E_TIMEOUT);
          *abort_flag = 1;
          break;
        }
        const int64_t tile = blockIdx.x + static_cast<int64_t>(i) * gridDim.x;
        mbar_arrive_expect_tx(&in_full[s], stage_bytes);
        for (int h = 0; h < 2; ++h)
          tma_load_2d(in + s * stage_bytes + h * box_bytes, &cube_map, static_cast<int>(tile * kScrTile + h * kScrBox),
                      0, &in_full[s]);
        pending |= 1u << s;
        parity = (parity & ~(1u << s)) | (ph << s);
      }
      for (int s = 0; s < kIn; ++s)
        if ((pending >> s) & 1u) mbar_wait_idle(&in_full[s], (parity >> s) & 1u);
      mbar_wait_idle(w_full, 0);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t id1 = idesc_f16_amn(kScrTile, kH1);
      const uint32_t id2 = idesc_bf16_f32(kScrTile, kH2);
      bool issued = false;
      if (n > 0 && !mbar_wait_idle(w_full, 0)) {
        record_error(args.status, HSI_E_TIMEOUT);
        *abort_flag = 1;
      }
      const uint64_t dw2 = smem_desc_sw128(w2);
      // layer 2 of tile j
      auto layer2 = [&](int j) -> bool {
        const int pb = j & 1;
        if (!mbar_wait_idle(&h1_full[pb], (j >> 1) & 1u) || !mbar_wait_idle(acc2_empty, (j & 1u) ^ 1u)) return false;
        tc_fence_after();
        const uint64_t dh = smem_desc_sw128(h1 + pb * kScrTile * 128);
#pragma unroll
        for (int ks = 0; ks < kH1 / 16; ++ks) umma_f16(tmem + 128, dh + 2 * ks, dw2 + 2 * ks, id2, ks > 0 ? 1u : 0u);
        umma_commit(&h1_empty[pb]);
        umma_commit(acc2_full);
        return true;
      };
      for (int i = 0; i < n && !*abort_flag; ++i) {
        const int s = i % kIn, pb = i & 1;
        if (!mbar_wait_idle(&in_full[s], (i / kIn) & 1u) || !mbar_wait_idle(&acc1_empty[pb], ((i >> 1) & 1u) ^ 1u)) {
          record_error(args.status, HSI_E_TIMEOUT);
          *abort_flag = 1;
          break;
        }
        tc_fence_after();
        unsigned char* a = in + s * stage_bytes;
        for (int ks = 0; ks < Bp / 16; ++ks) {
          const uint64_t da = smem_desc_mn_sw128(a + ks * 2048, box_bytes);
          const uint64_t db = smem_desc_sw128(w1 + (ks >> 2) * kH1 * 128) + 2 * (ks & 3);
          umma_f16(tmem + pb * kH1, da, db, id1, ks > 0 ? 1u : 0u);
        }
        umma_commit(&in_empty[s]);
        umma_commit(&acc1_full[pb]);
        issued = true;
        if (i > 0 && !layer2(i - 1)) {
          record_error(args.status, HSI_E_TIMEOUT);
          *abort_flag = 1;
          break;
        }
      }
      if (n > 0 && !*abort_flag && !layer2(n - 1)) {
        record_error(args.status, HSI_E_TIMEOUT);
        *abort_flag = 1;
      }
      if (issued) {
        umma_commit(mma_done);
        if (!mbar_wait_idle(mma_done, 0)) record_error(args.status, HSI_E_TIMEOUT);
      }
    }
  } else {
    // epilogue: warp -> TMEM lane quarter q, thread -> pixel q*32 + lane
    const int q = warp & 3;
    const int px = q * 32 + lane;
    const uint32_t trow = tmem + (static_cast<uint32_t>(q * 32) << 16);
    const float* b1 = cst;
    const float* b2 = cst + kH1;
    const float* w3 = b2 + kH2;
    const float b3 = w3[kH2];
    for (int i = 0; i < n; ++i) {
      const int pb = i & 1;
      if (!mbar_wait_idle(&acc1_full[pb], (i >> 1) & 1u)) {
        record_error(args.status, HSI_E_TIMEOUT);
        *abort_flag = 1;
        break;
      }
      tc_fence_after();
      uint32_t r0[32], r1[32];
      tmem_ld32(trow + pb * kH1, r0);
      tmem_ld32(trow + pb * kH1 + 32, r1);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc1_empty[pb]);
      // h1 = relu(acc + b1') as bfloat16, one 128-byte row per pixel
      uint32_t packed[32];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float a0 = fmaxf(__uint_as_float(r0[2 * j]) + b1[2 * j], 0.0f);
        const float a1 = fmaxf(__uint_as_float(r0[2 * j + 1]) + b1[2 * j + 1], 0.0f);
        const __nv_bfloat162 v2 = __floats2bfloat162_rn(a0, a1);
        packed[j] = *reinterpret_cast<const uint32_t*>(&v2);
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float a0 = fmaxf(__uint_as_float(r1[2 * j]) + b1[32 + 2 * j], 0.0f);
        const float a1 = fmaxf(__uint_as_float(r1[2 * j + 1]) + b1[32 + 2 * j + 1], 0.0f);
        const __nv_bfloat162 v2 = __floats2bfloat162_rn(a0, a1);
        packed[16 + j] = *reinterpret_cast<const uint32_t*>(&v2);
      }
      if (!mbar_wait_idle(&h1_empty[pb], ((i >> 1) & 1u) ^ 1u)) {
        record_error(args.status, HSI_E_TIMEOUT);
        *abort_flag = 1;
        break;
      }
      unsigned char* ht = h1 + pb * kScrTile * 128;
#pragma unroll
      for (int c = 0; c < 8; ++c)
        *reinterpret_cast<uint4*>(ht + sw128(px, c * 16)) =
            make_uint4(packed[4 * c], packed[4 * c + 1], packed[4 * c + 2], packed[4 * c + 3]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&h1_full[pb]);
      if (!mbar_wait_idle(acc2_full, i & 1u)) {
        record_error(args.status, HSI_E_TIMEOUT);
        *abort_flag = 1;
        break;
      }
      tc_fence_after();
      uint32_t r2[32];
      tmem_ld32(trow + 128, r2);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc2_empty);
      float z = b3;
#pragma unroll
      for (int k = 0; k < kH2; ++k) z = fmaf(w3[k], fmaxf(__uint_as_float(r2[k]) + b2[k], 0.0f), z);
      const int64_t p = (blockIdx.x + static_cast<int64_t>(i) * gridDim.x) * kScrTile + px;
      if (p < P) args.logits[p] = z;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kScrTmemCols);
  }
}

size_t screen_smem_bytes(int Bp) {
  const size_t stage = 2 * static_cast<size_t>(Bp) * 128;
  const size_t k_in = (128 * 1024) / stage < 4 ? (128 * 1024) / stage : 4;
  return k_in * stage + static_cast<size_t>(Bp / 64) * kH1 * 128 + kH2 * 128 + 2 * kScrTile * 128 +
         sizeof(float) * (kH1 + 2 * kH2 + 4) + 22 * sizeof(uint64_t) + 1024;
}

// ---- gather candidate pixels into a compact BSQ cube --------------------------
template <typename T>
__global__ void pick_kernel(const T* __restrict__ cube, int64_t stride, int B, int width,
                            const hsi_detection* __restrict__ cand, const uint32_t* __restrict__ count, int capacity,
                            T* __restrict__ out, int64_t out_stride) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (i >= capacity || b >= B) return;
  const uint32_t nc = min(*count, static_cast<uint32_t>(capacity));
  T v;
  if (static_cast<uint32_t>(i) < nc) {
    const int64_t p = static_cast<int64_t>(cand[i].y) * width + cand[i].x;
    v = cube[static_cast<int64_t>(b) * stride + p];
  } else {
    v = cube[static_cast<int64_t>(b) * stride];  // padding: a real pixel, its scores are ignored
  }
  out[static_cast<int64_t>(b) * out_stride + i] = v;
}

}  // namespace
}  // namespace hsi_b200

using namespace hsi_b200;

extern "C" HSI_API int64_t hsi_screen_param_count(int bands) {
  if (bands <= 0 || bands > HSI_MAX_BANDS) return 0;
  return param_count(bands);
}

extern "C" HSI_API int hsi_screen_init(float* d_params, int bands, uint64_t seed, hsi_stream_t stream) {
  if (!d_params || bands <= 0 || bands > HSI_MAX_BANDS) return HSI_E_INVALID;
  init_kernel<<<64, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(d_params, bands, seed);
  return static_cast<int>(cudaGetLastError());
}

extern "C" HSI_API int hsi_screen_normaliser(const double* d_moments, int bands, float* d_norm, hsi_stream_t stream) {
  if (!d_moments || !d_norm || bands <= 0 || bands > HSI_MAX_BANDS) return HSI_E_INVALID;
  normaliser_kernel<<<1, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(d_moments, bands, d_norm);
  return static_cast<int>(cudaGetLastError());
}

extern "C" HSI_API int hsi_screen_batch(const hsi_detection* d_positives, const uint32_t* d_positive_count,
                                        int positive_capacity, int height, int width, const float* d_score,
                                        float threshold, uint64_t seed, int num_positive_draws, int n,
                                        int32_t* d_index, float* d_labels, hsi_stream_t stream) {
  if (!d_positives || !d_positive_count || positive_capacity <= 0 || height <= 0 || width <= 0 || !d_score ||
      n <= 0 || num_positive_draws < 0 || !d_index || !d_labels)
    return HSI_E_INVALID;
  const int64_t P = static_cast<int64_t>(height) * width;
  if (P > 0x7fffffff) return HSI_E_CAPACITY;
  batch_kernel<<<(n + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      d_positives, d_positive_count, positive_capacity, width, P, d_score, threshold, seed, num_positive_draws, n,
      d_index, d_labels);
  return static_cast<int>(cudaGetLastError());
}

extern "C" HSI_API int hsi_screen_gather(const void* d_cube, int dtype, int64_t plane_stride, int bands,
                                         const float* d_norm, const int32_t* d_index, int n, float* d_features,
                                         hsi_stream_t stream) {
  if (!d_cube || !d_norm || !d_index || !d_features || n <= 0 || bands <= 0 || bands > HSI_MAX_BANDS)
    return HSI_E_INVALID;
  const dim3 grid((n + 255) / 256, padded_bands(bands));
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == HSI_F32)
    gather_kernel<float><<<grid, 256, 0, s>>>(static_cast<const float*>(d_cube), plane_stride, bands, d_norm,
                                              d_index, n, d_features);
  else if (dtype == HSI_F16)
    gather_kernel<__half><<<grid, 256, 0, s>>>(static_cast<const __half*>(d_cube), plane_stride, bands, d_norm,
                                               d_index, n, d_features);
  else
    return HSI_E_INVALID;
  return static_cast<int>(cudaGetLastError());
}

extern "C" HSI_API size_t hsi_screen_train_workspace_bytes(int bands, int n) {
  if (bands <= 0 || n <= 0) return 0;
  return train_bytes(n);
}

extern "C" HSI_API int hsi_screen_gradients(const float* d_params, int bands, const float* d_features,
                                            const float* d_labels, int n, float pos_weight, float* d_grads,
                                            float* d_loss, void* d_workspace, size_t workspace_bytes,
                                            hsi_stream_t stream) {
  if (!d_params || !d_features || !d_labels || !d_grads || n <= 0 || bands <= 0 || bands > HSI_MAX_BANDS)
    return HSI_E_INVALID;
  if (!d_workspace || workspace_bytes < train_bytes(n)) return HSI_E_WORKSPACE;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  float* partials = static_cast<float*>(d_workspace);
  // 16-byte feature copies need every row on 16 bytes
  const int vec = (n & 3) == 0 && (reinterpret_cast<uintptr_t>(d_features) & 15u) == 0;
  const auto launch = [&](auto nb) {
    constexpr int NB = decltype(nb)::value;
    return train_chunk(n) == 32
               ? launch_train<NB, 32>(d_params, bands, d_features, d_labels, n, pos_weight, vec, partials, s)
               : launch_train<NB, 64>(d_params, bands, d_features, d_labels, n, pos_weight, vec, partials, s);
  };
  cudaError_t e;
  switch (padded_bands(bands) / 64) {
    case 1: e = launch(std::integral_constant<int, 1>{}); break;
    case 2: e = launch(std::integral_constant<int, 2>{}); break;
    case 3: e = launch(std::integral_constant<int, 3>{}); break;
    default: e = launch(std::integral_constant<int, 4>{}); break;
  }
  if (e != cudaSuccess) return static_cast<int>(e);
  const int64_t count = param_count(bands);
  reduce_kernel<<<static_cast<int>(count / 32 + 1), 256, 0, s>>>(partials, train_ctas(n), partial_stride(bands), count,
                                                                 n, d_grads, d_loss);
  return static_cast<int>(cudaGetLastError());
}

extern "C" HSI_API int hsi_screen_adam(float* d_params, float* d_adam_state, const float* d_grads, int bands,
                                       float lr, int step, hsi_stream_t stream) {
  if (!d_params || !d_adam_state || !d_grads || bands <= 0 || bands > HSI_MAX_BANDS || step < 1) return HSI_E_INVALID;
  const int64_t n = param_count(bands);
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.0f - powf(b1, static_cast<float>(step)), c2 = 1.0f - powf(b2, static_cast<float>(step));
  adam_kernel<<<64, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(d_params, d_adam_state, d_adam_state + n,
                                                                      d_grads, n, lr, b1, b2, 1e-8f, c1, c2);
  return static_cast<int>(cudaGetLastError());
}

extern "C" HSI_API size_t hsi_screen_infer_workspace_bytes(int bands) {
  if (bands <= 0 || bands > HSI_MAX_BANDS) return 0;
  return (sizeof(ScreenOps) + 255) & ~static_cast<size_t>(255);
}

namespace hsi_b200 {
namespace {

// Screen inference on at most max_ctas CTAs (0: one per SM).  The kernel's
// static tile schedule covers every tile for any grid size.
int screen_infer(const void* d_cube, int height, int width, int bands, int dtype, int64_t plane_stride,
                 const float* d_norm, const float* d_params, float* d_logits, void* d_workspace,
                 size_t workspace_bytes, int max_ctas, hsi_stream_t stream) {
  if (max_ctas < 0) return HSI_E_INVALID;
  if (!d_cube || !d_norm || !d_params || !d_logits || height <= 0 || width <= 0 || bands <= 0 ||
      bands > HSI_MAX_BANDS)
    return HSI_E_INVALID;
  if (dtype != HSI_F16) return HSI_E_INVALID;  // the first layer reads fp16 cubes as its MMA operand
  const int64_t P = static_cast<int64_t>(height) * width;
  if (plane_stride < P || (plane_stride & 7) != 0) return HSI_E_INVALID;  // 16-byte TMA strides
  if ((reinterpret_cast<uintptr_t>(d_cube) & 15u) != 0) return HSI_E_INVALID;
  if (!d_workspace || workspace_bytes < hsi_screen_infer_workspace_bytes(bands)) return HSI_E_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(d_workspace) & 255u) != 0) return HSI_E_INVALID;
  const int Bp = padded_bands(bands);
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  ScreenOps* ops = static_cast<ScreenOps*>(d_workspace);
  pack_kernel<<<kH1 + 1, 256, 0, s>>>(d_params, bands, d_norm, ops);
  CUtensorMap map;
  if (encode_cube_map_sw128(&map, d_cube, HSI_F16, P, bands, plane_stride, kScrBox, Bp) != 0) return HSI_E_INVALID;
  const size_t smem = screen_smem_bytes(Bp);
  const cudaError_t e = raise_smem_limit(screen_tc_kernel, static_cast<int>(smem));
  if (e != cudaSuccess) return static_cast<int>(e);
  const int sms = device_sm_count();
  const int cap = max_ctas > 0 && max_ctas < sms ? max_ctas : sms;
  const int64_t ntiles = (P + kScrTile - 1) / kScrTile;
  const int grid = static_cast<int>(ntiles < cap ? ntiles : cap);
  ScreenArgs a{P, Bp, ops, d_logits, nullptr};
  screen_tc_kernel<<<grid, kScrThreads, smem, s>>>(map, a);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace
}  // namespace hsi_b200

extern "C" HSI_API int hsi_screen_infer(const void* d_cube, int height, int width, int bands, int dtype,
                                        int64_t plane_stride, const float* d_norm, const float* d_params,
                                        float* d_logits, void* d_workspace, size_t workspace_bytes,
                                        hsi_stream_t stream) {
  return screen_infer(d_cube, height, width, bands, dtype, plane_stride, d_norm, d_params, d_logits, d_workspace,
                      workspace_bytes, 0, stream);
}

extern "C" HSI_API int hsi_screen_infer_ctas(const void* d_cube, int height, int width, int bands, int dtype,
                                             int64_t plane_stride, const float* d_norm, const float* d_params,
                                             float* d_logits, void* d_workspace, size_t workspace_bytes,
                                             int max_ctas, hsi_stream_t stream) {
  return screen_infer(d_cube, height, width, bands, dtype, plane_stride, d_norm, d_params, d_logits, d_workspace,
                      workspace_bytes, max_ctas, stream);
}

extern "C" HSI_API int hsi_gather_candidates(const void* d_cube, int dtype, int64_t plane_stride, int bands,
                                             int width, const hsi_detection* d_candidates,
                                             const uint32_t* d_count, int capacity, void* d_out,
                                             int64_t out_stride, hsi_stream_t stream) {
  if (!d_cube || !d_candidates || !d_count || !d_out || capacity <= 0 || bands <= 0 || bands > HSI_MAX_BANDS ||
      width <= 0 || out_stride < capacity)
    return HSI_E_INVALID;
  const dim3 grid((capacity + 255) / 256, bands);
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == HSI_F32)
    pick_kernel<float><<<grid, 256, 0, s>>>(static_cast<const float*>(d_cube), plane_stride, bands, width,
                                            d_candidates, d_count, capacity, static_cast<float*>(d_out), out_stride);
  else if (dtype == HSI_F16)
    pick_kernel<__half><<<grid, 256, 0, s>>>(static_cast<const __half*>(d_cube), plane_stride, bands, width,
                                             d_candidates, d_count, capacity, static_cast<__half*>(d_out),
                                             out_stride);
  else
    return HSI_E_INVALID;
  return static_cast<int>(cudaGetLastError());
}
