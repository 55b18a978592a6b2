// rxace.cu - RX and ACE scoring (whitening pass).
//
// Per pixel, with y = x - mu and the FP64-built statistics (factor.cu):
//   z = W y (W = L^-1, lower triangular);  RX = |z|^2
//   zu_t = z . u_t = y . v_t with v_t = W^T u_t (precomputed per frame)
//   ACE_t = zu_t^2 / (|u_t|^2 RX), skipped (0) when |u_t|^2 <= 0 or RX <= 0;
//   best = max with strict '>' so the lowest t wins ties, clamp to [0, 1],
//   0 and target -1 when no target is valid
// (reference rx_cpu / ace_best_cpu, src/detectors_cpu.cpp:95-156, which
// whiten in double with float statistics).
//
// Both paths treat the scoring as one GEMM  Zaug = Waug . Y  with
// Waug = [W ; V^T] ((B + T) x B): the first B rows give z, the last T rows the
// ACE numerators, and an epilogue per pixel reduces them to RX / ACE.
//
// This file holds the preparation kernel and the plain FP32 CUDA-core path,
// the comparator for the tensor-core path in rxace_tc.cu and the scorer of
// frames above its 127 bands.
//
// Plain path.  The rows of Waug go in groups of eight; group G multiplies only
// the bands up to its last row (W is lower triangular; target rows are dense).
// A persistent block holds all groups' weights in shared memory (118 KB at 224
// bands and 16 targets) beside the 64 centred pixels of its tile, so the tile's
// product runs without a barrier, and the next tile's pixels are on their way
// to registers meanwhile.  A half-warp takes all 64 pixels (four per lane) of
// one "chain", the groups G, G + 16, G + 32, whose squares form one partial sum
// of RX.  Chains differ in length, so the host deals them out: neighbours in
// length share a warp, and each SM sub-partition gets a long and a short warp.
// Bound: FP32 FMA (B^2 / 2 + T B per pixel).  1024 x 1024 x 224 fp16, 16
// targets: 3.24 ms with 128 x 128 tiles that staged W and the cube per 16-band
// chunk for every row tile (16-way conflicts on W's transposing store, a
// barrier per chunk, warps idling above the diagonal); see the launch below
// for the time now.
#include "common.cuh"
#include "launch_state.h"

#include <algorithm>

namespace hsi_b200 {
namespace {

constexpr int kPxTile = 64;     // pixels per tile
constexpr int kThreads = 256;
constexpr int kGroupRows = 8;   // output rows (bands + targets) per group
constexpr int kChains = 16;     // partial sums of RX per pixel, a half-warp each
constexpr int kMaxGroups = (HSI_MAX_BANDS + HSI_MAX_FILTERS_PER_PASS) / kGroupRows;

// Where the groups' weights lie (floats from the panels' start, [k][8 rows] of
// `bands[g]` bands) and which half-warp takes which chain.
struct Panels {
  int groups;
  int kpad;                       // bands rounded up to 8
  int floats;                     // of all panels
  int offset[kMaxGroups];
  short bands[kMaxGroups];
  unsigned char chain[kChains];   // chain of half-warp h
};

// Prepared operands in the workspace (FP32 path).
struct SimtOperands {
  float* panels;   // 16-byte aligned
  float* mean_hi;  // mu = hi + lo (double-float)
  float* mean_lo;
  float* uu;       // [T]
};

__host__ __device__ inline int round_up(int v, int m) { return (v + m - 1) / m * m; }

Panels make_panels(int B, int T) {
  Panels p{};
  p.groups = (B + T + kGroupRows - 1) / kGroupRows;
  p.kpad = round_up(B, kGroupRows);
  int cost[kChains] = {}, order[kChains];
  for (int g = 0; g < p.groups; ++g) {
    // rows above B end their dot product at the diagonal; target rows are dense
    p.bands[g] = static_cast<short>(std::min((g + 1) * kGroupRows, p.kpad));
    cost[g % kChains] += p.bands[g];
  }
  for (int c = 0; c < kChains; ++c) order[c] = c;
  std::stable_sort(order, order + kChains, [&](int a, int b) { return cost[a] > cost[b]; });
  // pairs of neighbours, longest first: pair i on warp i of the first four,
  // then the remaining pairs shortest first, so that warps w and w + 4 (one
  // sub-partition) add up alike
  for (int i = 0; i < kChains / 2; ++i) {
    const int w = i < 4 ? i : 4 + (7 - i);
    p.chain[2 * w] = static_cast<unsigned char>(order[2 * i]);
    p.chain[2 * w + 1] = static_cast<unsigned char>(order[2 * i + 1]);
  }
  // the two halves of a warp read their weights at the same band: the second
  // halves' panels start 64 bytes off, on other banks
  for (int half = 0; half < 2; ++half) {
    if (half) p.floats += 16;
    for (int w = 0; w < kChains / 2; ++w)
      for (int g = p.chain[2 * w + half]; g < p.groups; g += kChains) {
        p.offset[g] = p.floats;
        p.floats += p.bands[g] * kGroupRows;
      }
  }
  return p;
}

// One thread per weight: rows < B copy W, rows B + t hold v_t = W^T u_t in
// FP64; the rest are zero.  blockIdx.x: the group, blockIdx.y: 256 weights of
// its panel.
__global__ void __launch_bounds__(256) prep_simt_kernel(const double* __restrict__ stats, int B, int T,
                                                       const __grid_constant__ Panels pn, SimtOperands op) {
  const int g = blockIdx.x;
  const double* mean = stats;
  const double* W = stats + B;
  const double* tw = W + static_cast<size_t>(B) * B;
  const double* tn = tw + static_cast<size_t>(T) * B;
  const int e = blockIdx.y * 256 + threadIdx.x;
  if (e < pn.bands[g] * kGroupRows) {
    const int k = e / kGroupRows, n = g * kGroupRows + e % kGroupRows;
    double v = 0.0;
    if (k < B) {
      if (n < B) {
        v = W[static_cast<size_t>(n) * B + k];
      } else if (n < B + T) {
        const double* u = tw + static_cast<size_t>(n - B) * B;
#pragma unroll 16
        for (int i = k; i < B; ++i) v += W[static_cast<size_t>(i) * B + k] * u[i];
      }
    }
    op.panels[pn.offset[g] + e] = static_cast<float>(v);
  }
  if (g == 0 && blockIdx.y == 0) {
    for (int b = threadIdx.x; b < B; b += blockDim.x) {
      const float hi = static_cast<float>(mean[b]);
      op.mean_hi[b] = hi;
      op.mean_lo[b] = static_cast<float>(mean[b] - static_cast<double>(hi));
    }
    for (int t = threadIdx.x; t < T; t += blockDim.x) op.uu[t] = static_cast<float>(tn[t]);
  }
}

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) {
  return v;
}
template <>
__device__ __forceinline__ float to_f<__half>(__half v) {
  return __half2float(v);
}

struct ScoreOut {
  float* rx;            // nullable
  float* ace_best;      // nullable
  int32_t* ace_target;  // nullable
  float* ace_maps;      // nullable, T maps at map_stride
  int64_t map_stride;
};

// V pixels of band row b from pixel p on, centred; zero past the frame.
template <typename T>
constexpr int kVec = 16 / static_cast<int>(sizeof(T));

struct SimtSmem {
  float mean_hi[HSI_MAX_BANDS], mean_lo[HSI_MAX_BANDS];
  float uu[HSI_MAX_FILTERS_PER_PASS];
  float rx[kChains][kPxTile];
  float zu[HSI_MAX_FILTERS_PER_PASS][kPxTile];
  // then y[kpad][kPxTile], the panels
};

// BANDS: the instance's largest padded band count, which sizes the register
// prefetch.  `aligned`: the cube starts on 16 bytes.
template <typename T, int BANDS>
__global__ void __launch_bounds__(kThreads, BANDS <= 128 ? 2 : 1)
    rxace_simt_kernel(const T* __restrict__ cube, int64_t pixels, int64_t stride, int B, int Tn, int aligned,
                      const __grid_constant__ Panels pn, SimtOperands op, ScoreOut out) {
  constexpr int V = kVec<T>;
  constexpr int kRowVecs = kPxTile / V;                                    // 16-byte groups per band row
  constexpr int kLoads = (BANDS * kRowVecs + kThreads - 1) / kThreads;     // per thread and tile
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SimtSmem& sm = *reinterpret_cast<SimtSmem*>(smem_raw);
  float* ys = reinterpret_cast<float*>(smem_raw + sizeof(SimtSmem));  // [kpad][kPxTile]
  float* ws = ys + pn.kpad * kPxTile;                                 // panels
  const int tid = threadIdx.x, lane = tid & 31;
  const int64_t tiles = div_up<int64_t>(pixels, kPxTile);

  for (int i = tid; i < pn.floats / 4; i += kThreads)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(ws + 4 * i)), "l"(op.panels + 4 * i)
                 : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int b = tid; b < B; b += kThreads) {
    sm.mean_hi[b] = op.mean_hi[b];
    sm.mean_lo[b] = op.mean_lo[b];
  }
  if (tid < Tn) sm.uu[tid] = op.uu[tid];

  // this thread's share of a tile: group m of row (tid + 256 m) / kRowVecs
  uint4 raw[kLoads];
  auto fetch = [&](int64_t tile) {
    const int64_t p0 = tile * kPxTile;
#pragma unroll
    for (int m = 0; m < kLoads; ++m) {
      const int e = tid + kThreads * m, b = e / kRowVecs;
      const int64_t p = p0 + e % kRowVecs * V;
      raw[m] = make_uint4(0u, 0u, 0u, 0u);
      if (b >= B || p >= pixels) continue;
      const T* src = cube + static_cast<int64_t>(b) * stride + p;
      if (aligned && p + V <= pixels) {
        raw[m] = __ldg(reinterpret_cast<const uint4*>(src));
      } else {
        T v[V];
#pragma unroll
        for (int j = 0; j < V; ++j) v[j] = p + j < pixels ? src[j] : T(0.0f);
        raw[m] = *reinterpret_cast<const uint4*>(v);
      }
    }
  };
  auto commit = [&](int64_t tile) {
    const int64_t p0 = tile * kPxTile;
#pragma unroll
    for (int m = 0; m < kLoads; ++m) {
      const int e = tid + kThreads * m, b = e / kRowVecs, px = e % kRowVecs * V;
      if (b >= pn.kpad) continue;
      T v[V];
      *reinterpret_cast<uint4*>(v) = raw[m];
      const float hi = b < B ? sm.mean_hi[b] : 0.0f, lo = b < B ? sm.mean_lo[b] : 0.0f;
      float y[V];
#pragma unroll
      for (int j = 0; j < V; ++j) y[j] = b < B && p0 + px + j < pixels ? (to_f<T>(v[j]) - hi) - lo : 0.0f;
#pragma unroll
      for (int j = 0; j < V; j += 4)
        *reinterpret_cast<float4*>(ys + b * kPxTile + px + j) = make_float4(y[j], y[j + 1], y[j + 2], y[j + 3]);
    }
  };

  int64_t tile = blockIdx.x;
  fetch(tile);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  commit(tile);
  __syncthreads();
  const int px = 4 * (lane & 15);
  const int chain = pn.chain[2 * (tid >> 5) + (lane >> 4)];
  for (; tile < tiles; tile += gridDim.x) {
    const int64_t next = tile + gridDim.x;
    if (next < tiles) fetch(next);
    float rx_part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int g = chain; g < pn.groups; g += kChains) {
      float2 acc[kGroupRows][2];  // row i, pixel pairs of this lane's four: packed FMAs
#pragma unroll
      for (int i = 0; i < kGroupRows; ++i) acc[i][0] = acc[i][1] = make_float2(0.0f, 0.0f);
      const float* w = ws + pn.offset[g];
      const float* y = ys + px;
      const int bands = pn.bands[g];  // a multiple of 8
#pragma unroll 1
      for (int k0 = 0; k0 < bands; k0 += 8, w += 8 * kGroupRows, y += 8 * kPxTile) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float4 wa = *reinterpret_cast<const float4*>(w + k * kGroupRows);
          const float4 wb = *reinterpret_cast<const float4*>(w + k * kGroupRows + 4);
          const float4 yk = *reinterpret_cast<const float4*>(y + k * kPxTile);
          const float wv[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
          const float2 y0 = make_float2(yk.x, yk.y), y1 = make_float2(yk.z, yk.w);
#pragma unroll
          for (int i = 0; i < kGroupRows; ++i) {
            const float2 wi = make_float2(wv[i], wv[i]);
            acc[i][0] = ffma2(wi, y0, acc[i][0]);
            acc[i][1] = ffma2(wi, y1, acc[i][1]);
          }
        }
      }
      // fold: rows < B -> RX partials; rows B..B+T-1 -> ACE numerators
#pragma unroll
      for (int i = 0; i < kGroupRows; ++i) {
        const int row = g * kGroupRows + i;
        const float z[4] = {acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y};
        if (row < B) {
#pragma unroll
          for (int j = 0; j < 4; ++j) rx_part[j] = fmaf(z[j], z[j], rx_part[j]);
        } else if (row < B + Tn) {
          *reinterpret_cast<float4*>(&sm.zu[row - B][px]) = make_float4(z[0], z[1], z[2], z[3]);
        }
      }
    }
    *reinterpret_cast<float4*>(&sm.rx[chain][px]) = make_float4(rx_part[0], rx_part[1], rx_part[2], rx_part[3]);
    __syncthreads();  // the tile's sums are in, its pixels done with
    if (next < tiles) commit(next);
    // RX and ACE of one pixel by four lanes, a quarter of the targets each
    // (reference src/detectors_cpu.cpp:127-156)
    {
      const int q = tid & 3, epx = tid >> 2;
      const int64_t p = tile * kPxTile + epx;
      float rx = 0.0f;
#pragma unroll
      for (int c = 0; c < kChains; ++c) rx += sm.rx[c][epx];
      float best = -1.0f;
      int32_t best_t = -1;
      const int t0 = q * Tn / 4, t1 = (q + 1) * Tn / 4;
      for (int t = t0; t < t1; ++t) {
        float a = 0.0f;
        if (sm.uu[t] > 0.0f && rx > 0.0f) {
          const float zu = sm.zu[t][epx];
          a = (zu * zu) / (sm.uu[t] * rx);
          if (a > best) {
            best = a;
            best_t = t;
          }
        }
        if (out.ace_maps && p < pixels) out.ace_maps[static_cast<int64_t>(t) * out.map_stride + p] = a;
      }
      // lowest target on ties: a later quarter wins only when strictly larger
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int32_t ot = __shfl_xor_sync(0xffffffffu, best_t, o);
        const bool other_first = (q & o) != 0;
        if (ob > best || (other_first && ob == best && ot >= 0)) {
          best = ob;
          best_t = ot;
        }
      }
      if (q == 0 && p < pixels) {
        if (out.rx) out.rx[p] = rx;
        if (out.ace_best) out.ace_best[p] = best < 0.0f ? 0.0f : fminf(best, 1.0f);
        if (out.ace_target) out.ace_target[p] = best_t;
      }
    }
    __syncthreads();  // the next tile's pixels are in, this one's sums read
  }
}

size_t align256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

// The size callers have always been asked for (row tiles of 128, bands rounded
// up to 16); the panels take less than half of it.
size_t simt_bytes(int B, int T) {
  return align256(sizeof(float) * static_cast<size_t>(round_up(B + T, 128)) * round_up(B, 16)) +
         3 * align256(sizeof(float) * HSI_MAX_BANDS);
}

SimtOperands carve_simt(void* ws, const Panels& pn) {
  SimtOperands op;
  const uintptr_t base = (reinterpret_cast<uintptr_t>(ws) + 15u) & ~static_cast<uintptr_t>(15u);
  op.panels = reinterpret_cast<float*>(base);
  op.mean_hi = op.panels + round_up(pn.floats, 4);
  op.mean_lo = op.mean_hi + HSI_MAX_BANDS;
  op.uu = op.mean_lo + HSI_MAX_BANDS;
  return op;
}

template <typename T, int BANDS>
cudaError_t launch_simt(const void* cube, int64_t P, int64_t stride, int B, int Tn, const Panels& pn,
                        const SimtOperands& op, const ScoreOut& o, cudaStream_t s) {
  // in steps of 8 KB, so that few layouts are ever asked about
  const size_t need = sizeof(SimtSmem) + sizeof(float) * (static_cast<size_t>(pn.kpad) * kPxTile + pn.floats);
  const size_t smem = std::min<size_t>((need + 8191) / 8192 * 8192, 232448);
  const int resident = device_residency(rxace_simt_kernel<T, BANDS>, kThreads, smem);
  if (resident <= 0) {
    const cudaError_t e = raise_smem_limit(rxace_simt_kernel<T, BANDS>, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
  }
  const int64_t tiles = div_up<int64_t>(P, kPxTile);
  const int64_t wave = static_cast<int64_t>(std::max(resident, 1)) * device_sm_count();
  const int aligned = (reinterpret_cast<uintptr_t>(cube) & 15u) == 0;
  rxace_simt_kernel<T, BANDS><<<static_cast<unsigned>(std::min(tiles, wave)), kThreads, smem, s>>>(
      static_cast<const T*>(cube), P, stride, B, Tn, aligned, pn, op, o);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_simt_bands(const void* cube, int64_t P, int64_t stride, int B, int Tn, const Panels& pn,
                              const SimtOperands& op, const ScoreOut& o, cudaStream_t s) {
  if (pn.kpad <= 64) return launch_simt<T, 64>(cube, P, stride, B, Tn, pn, op, o, s);
  if (pn.kpad <= 128) return launch_simt<T, 128>(cube, P, stride, B, Tn, pn, op, o, s);
  return launch_simt<T, 256>(cube, P, stride, B, Tn, pn, op, o, s);
}

}  // namespace

// Shared with rxace_tc.cu.
int rxace_check(const void* cube, int height, int width, int bands, int dtype, int64_t stride, const double* stats,
                int T) {
  if (!cube || !stats || height <= 0 || width <= 0 || bands <= 0 || bands > HSI_MAX_BANDS) return HSI_E_INVALID;
  if (T < 0 || T > HSI_MAX_FILTERS_PER_PASS) return HSI_E_INVALID;
  if (dtype != HSI_F32 && dtype != HSI_F16) return HSI_E_INVALID;
  const int64_t P = static_cast<int64_t>(height) * width;
  if (stride < P || (stride & 7) != 0) return HSI_E_INVALID;
  return HSI_OK;
}

}  // namespace hsi_b200

using namespace hsi_b200;

extern "C" HSI_API size_t hsi_rx_ace_simt_workspace_bytes(int bands, int num_targets) {
  if (bands <= 0 || bands > HSI_MAX_BANDS || num_targets < 0) return 0;
  return simt_bytes(bands, num_targets);
}

extern "C" HSI_API int hsi_rx_ace_simt(const void* d_cube, int height, int width, int bands, int dtype,
                                       int64_t plane_stride, const double* d_stats64, int num_targets,
                                       float* d_rx, float* d_ace_best, int32_t* d_ace_target, float* d_ace_maps,
                                       int64_t map_stride, void* d_workspace, size_t workspace_bytes,
                                       hsi_stream_t stream) {
  const int rc = rxace_check(d_cube, height, width, bands, dtype, plane_stride, d_stats64, num_targets);
  if (rc != HSI_OK) return rc;
  const int64_t P = static_cast<int64_t>(height) * width;
  if (d_ace_maps && map_stride < P) return HSI_E_INVALID;
  if (!d_workspace || workspace_bytes < simt_bytes(bands, num_targets)) return HSI_E_WORKSPACE;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const Panels pn = make_panels(bands, num_targets);
  const SimtOperands op = carve_simt(d_workspace, pn);
  prep_simt_kernel<<<dim3(pn.groups, (pn.kpad * kGroupRows + 255) / 256), 256, 0, s>>>(d_stats64, bands, num_targets,
                                                                                     pn, op);
  ScoreOut o{d_rx, d_ace_best, d_ace_target, d_ace_maps, map_stride};
  const cudaError_t e =
      dtype == HSI_F32 ? launch_simt_bands<float>(d_cube, P, plane_stride, bands, num_targets, pn, op, o, s)
                       : launch_simt_bands<__half>(d_cube, P, plane_stride, bands, num_targets, pn, op, o, s);
  return static_cast<int>(e);
}
