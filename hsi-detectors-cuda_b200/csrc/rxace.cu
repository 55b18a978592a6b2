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
// product runs without a block barrier, and the next tile's pixels are on their
// way to registers meanwhile.  A half-warp takes all 64 pixels (four per lane)
// of one group, a warp a pair of neighbours; the host deals the pairs out so
// that every warp has the same number of bands to go through (240 each at 224
// bands and 16 targets: with two warps per sub-partition, one that ends early
// leaves the other's latencies bare).  The squares of groups G, G + 16, G + 32
// form one partial sum of RX; a pair waits for the pair eight before it, which
// is always started earlier, before it adds its own.
// Bound: FP32 FMA (B^2 / 2 + T B per pixel; the pipe is 72 % busy) and the
// shared-memory reads beside it (71 %: eight weights and four pixels per lane
// for 16 packed FMAs; sixteen rows by two pixels needed ten wavefronts where
// this tile needs eight, and was 13 % slower).  1024 x 1024 x 224 fp16, 16
// targets: 1.28 ms; 3.24 with 128 x 128 tiles that staged W and the cube per
// 16-band chunk for every row tile (16-way conflicts on W's transposing store,
// a barrier per chunk, warps idling above the diagonal).
#include "common.cuh"
#include "launch_state.h"
#include "rxace_panels.h"

#include <algorithm>

namespace hsi_b200 {
namespace {

constexpr int kPxTile = 64;     // pixels per tile
constexpr int kThreads = 256;
constexpr int kWarps = kSimtWarps;
static_assert(kThreads == 32 * kWarps, "a list of pairs per warp");

// Prepared operands in the workspace (FP32 path).
struct SimtOperands {
  float* panels;   // 16-byte aligned
  float* mean_hi;  // mu = hi + lo (double-float)
  float* mean_lo;
  float* uu;       // [T]
};

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
  __shared__ double su[kGroupRows][HSI_MAX_BANDS + 1];  // the group's u_t, its rows on different banks
  const bool dense = (g + 1) * kGroupRows > B;
  if (dense) {
    for (int i = threadIdx.x; i < kGroupRows * B; i += 256) {
      const int n = g * kGroupRows + i / B;
      if (n >= B && n < B + T) su[i / B][i % B] = tw[static_cast<size_t>(n - B) * B + i % B];
    }
    __syncthreads();
  }
  const int e = blockIdx.y * 256 + threadIdx.x;
  if (e < pn.bands[g] * kGroupRows) {
    const int k = e / kGroupRows, n = g * kGroupRows + e % kGroupRows;
    double v = 0.0;
    if (k < B) {
      if (n < B) {
        v = W[static_cast<size_t>(n) * B + k];
      } else if (n < B + T) {
        // v_k = sum_{i >= k} W_ik u_i in ascending i: 32 rows of W in flight at a
        // time (a load per term of the chain: 23 us at 224 bands, now 9.6 us)
        const double* u = su[e % kGroupRows];
        for (int i0 = k & ~3; i0 < B; i0 += 32) {
          double w[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) w[j] = W[static_cast<size_t>(min(i0 + j, B - 1)) * B + k];
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (i0 + j >= k && i0 + j < B) v += w[j] * u[i0 + j];
        }
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

template <typename T>
constexpr int kVec = 16 / static_cast<int>(sizeof(T));

struct SimtSmem {
  float2 mean[HSI_MAX_BANDS];  // (hi, lo)
  float uu[HSI_MAX_FILTERS_PER_PASS];
  float rx[kChains][kPxTile];
  float zu[HSI_MAX_FILTERS_PER_PASS][kPxTile];
  int done[kMaxPairs + 1];  // tiles whose squares pair i has added (per block, in order)
  int gave_up;              // a wait ran out: sums are missing
  int pad;                  // y starts on 16 bytes
  // then y[kpad][kPxTile], the panels, 8 floats that the last band's prefetch reads
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
  for (int b = tid; b < B; b += kThreads) sm.mean[b] = make_float2(op.mean_hi[b], op.mean_lo[b]);
  if (tid < Tn) sm.uu[tid] = op.uu[tid];
  if (tid <= kMaxPairs) sm.done[tid] = 0;
  if (tid == 0) sm.gave_up = 0;

  // this thread's share of a tile: V pixels from px0 on of bands b0, b0 + step, ..
  constexpr int kStep = kThreads / kRowVecs;
  const int b0 = tid / kRowVecs, px0 = tid % kRowVecs * V;
  const T* src0 = cube + static_cast<int64_t>(b0) * stride + px0;
  const int64_t src_step = kStep * stride;
  uint4 raw[kLoads];
  const auto whole = [&](int64_t tile) { return aligned && tile * kPxTile + px0 + V <= pixels; };
  auto fetch = [&](int64_t tile) {
    if (!whole(tile)) return;  // such pixels are read when the tile is stored
    const T* src = src0 + tile * kPxTile;
#pragma unroll
    for (int m = 0; m < kLoads; ++m, src += src_step)
      if (b0 + m * kStep < B) raw[m] = __ldg(reinterpret_cast<const uint4*>(src));
  };
  auto store = [&](int b, const float (&x)[V], int64_t inside) {
    const float2 mean = sm.mean[b];
    float y[V];
#pragma unroll
    for (int j = 0; j < V; ++j) y[j] = j < inside ? (x[j] - mean.x) - mean.y : 0.0f;
#pragma unroll
    for (int j = 0; j < V; j += 4)
      *reinterpret_cast<float4*>(ys + b * kPxTile + px0 + j) = make_float4(y[j], y[j + 1], y[j + 2], y[j + 3]);
  };
  auto commit = [&](int64_t tile) {
    float x[V];
    if (whole(tile)) {
#pragma unroll
      for (int m = 0; m < kLoads; ++m) {
        if (b0 + m * kStep >= B) break;
        T v[V];
        *reinterpret_cast<uint4*>(v) = raw[m];
#pragma unroll
        for (int j = 0; j < V; ++j) x[j] = to_f<T>(v[j]);
        store(b0 + m * kStep, x, V);
      }
    } else {
      const int64_t inside = pixels - (tile * kPxTile + px0);  // may be negative
      const T* src = src0 + tile * kPxTile;
#pragma unroll 1
      for (int b = b0; b < B; b += kStep, src += src_step) {
#pragma unroll
        for (int j = 0; j < V; ++j) x[j] = j < inside ? to_f<T>(src[j]) : 0.0f;
        store(b, x, inside);
      }
    }
  };
  // bands past B multiply zero weights: zero once
  for (int i = B * kPxTile + tid; i < pn.kpad * kPxTile; i += kThreads) ys[i] = 0.0f;

  int64_t tile = blockIdx.x;
  fetch(tile);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  commit(tile);
  __syncthreads();
  const int px = 4 * (lane & 15), half = lane >> 4, warp = tid >> 5;
  for (int turn = 1; tile < tiles; tile += gridDim.x, ++turn) {
    const int64_t next = tile + gridDim.x;
    if (next < tiles) fetch(next);
    for (int i = pn.first[warp]; i < pn.first[warp + 1]; ++i) {
      const int pair = pn.pair[i], g = 2 * pair + half;
      // packed FMAs over row pairs: their weights lie side by side as they are
      // read, and only the four pixels have to be doubled into a register pair
      float2 acc[kGroupRows / 2][4];
#pragma unroll
      for (int r = 0; r < kGroupRows / 2; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[r][j] = make_float2(0.0f, 0.0f);
      const int bands = g < pn.groups ? pn.bands[g] : 0;  // a multiple of 8
      const float* w = ws + pn.offset[g < pn.groups ? g : 0];
      const float* y = ys + px;
      // the next band's operands are read one band ahead
      float4 wa = *reinterpret_cast<const float4*>(w), wb = *reinterpret_cast<const float4*>(w + 4);
      float4 yk = *reinterpret_cast<const float4*>(y);
#pragma unroll 1
      for (int k0 = 0; k0 < bands; k0 += 8) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          w += kGroupRows;
          y += kPxTile;
          const float2 wv[4] = {make_float2(wa.x, wa.y), make_float2(wa.z, wa.w), make_float2(wb.x, wb.y),
                                make_float2(wb.z, wb.w)};
          const float yv[4] = {yk.x, yk.y, yk.z, yk.w};
          wa = *reinterpret_cast<const float4*>(w);
          wb = *reinterpret_cast<const float4*>(w + 4);
          yk = *reinterpret_cast<const float4*>(y);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 yj = make_float2(yv[j], yv[j]);
#pragma unroll
            for (int r = 0; r < kGroupRows / 2; ++r) acc[r][j] = ffma2(wv[r], yj, acc[r][j]);
          }
        }
      }
      __syncwarp();
      // fold: rows < B -> RX partials; rows B..B+T-1 -> ACE numerators
      float4 part = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      float* sum = &sm.rx[g % kChains][px];
      if (pair >= kChains / 2) {
        // the chain's earlier groups; the wait ends: their warp has them ahead
        // of anything that waits, and the lowest pair in work waits for none.
        // Should it run out all the same, the block ends with this tile and its
        // scores become NaN (there is no status word to set).
        volatile const int* before = &sm.done[pair - kChains / 2];
        uint32_t n = 0;
        while (*before < turn && n < kWaitLimit) ++n;
        if (n == kWaitLimit) sm.gave_up = 1;
        __threadfence_block();
        part = *reinterpret_cast<const float4*>(sum);
      }
      const auto z_of = [&](int r) {
        const float2(&a)[4] = acc[r / 2];
        return r % 2 ? make_float4(a[0].y, a[1].y, a[2].y, a[3].y) : make_float4(a[0].x, a[1].x, a[2].x, a[3].x);
      };
      const auto add_square = [&](const float4& z) {
        part.x = fmaf(z.x, z.x, part.x);
        part.y = fmaf(z.y, z.y, part.y);
        part.z = fmaf(z.z, z.z, part.z);
        part.w = fmaf(z.w, z.w, part.w);
      };
      if ((g + 1) * kGroupRows <= B) {
#pragma unroll
        for (int r = 0; r < kGroupRows; ++r) add_square(z_of(r));
      } else {
#pragma unroll
        for (int r = 0; r < kGroupRows; ++r) {
          const int row = g * kGroupRows + r;
          if (row < B) add_square(z_of(r));
          else if (row < B + Tn) *reinterpret_cast<float4*>(&sm.zu[row - B][px]) = z_of(r);
        }
      }
      *reinterpret_cast<float4*>(sum) = part;
      __threadfence_block();
      __syncwarp();
      if (lane == 0) *const_cast<volatile int*>(&sm.done[pair]) = turn;
    }
    __syncthreads();  // the tile's sums are in, its pixels done with
    if (next < tiles) commit(next);
    // RX and ACE of one pixel by four lanes, a quarter of the targets each
    // (reference src/detectors_cpu.cpp:127-156)
    {
      const int q = tid & 3, epx = tid >> 2;
      const int64_t p = tile * kPxTile + epx;
      float rx = 0.0f;
#pragma unroll
      for (int c = 0; c < kChains; ++c) rx += c < pn.groups ? sm.rx[c][epx] : 0.0f;
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
    if (sm.gave_up) break;
  }
  if (sm.gave_up) {
    const float nan = __int_as_float(0x7fc00000);
    for (tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int64_t p = tile * kPxTile + tid;
      if (tid >= kPxTile || p >= pixels) continue;
      if (out.rx) out.rx[p] = nan;
      if (out.ace_best) out.ace_best[p] = nan;
      if (out.ace_target) out.ace_target[p] = -1;
      for (int t = 0; out.ace_maps && t < Tn; ++t) out.ace_maps[static_cast<int64_t>(t) * out.map_stride + p] = nan;
    }
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
  const size_t need = sizeof(SimtSmem) + sizeof(float) * (static_cast<size_t>(pn.kpad) * kPxTile + pn.floats + kGroupRows);
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
