// rxace_tc.cu - RX and ACE whitening on the 5th-generation tensor cores.
//
// Per pixel x (reference rx_cpu / ace_best_cpu, src/detectors_cpu.cpp:95-156):
//   z = W (x - mean),  RX = |z|^2,  ACE_t = (z . u_t)^2 / (|u_t|^2 |z|^2),
// with W = L^-1 of the loaded scene covariance and u_t = W (d_t - mean).
// Since z . u_t = (x - mean) . v_t with v_t = W^T u_t, one contraction with the
// augmented matrix A = [W; v_0^T; ...] (N = B + T rows, K = B bands) gives both
// z and the ACE numerators.
//
// Precision.  RX/ACE amplify relative errors by the conditioning of W (its
// rows hold large entries of alternating sign), and the tensor cores' FP32
// accumulation truncates, so the contraction is done in exact integers:
//   data:  d = x - mean (FP32), per pixel p a power-of-two scale 2^t_p that
//          puts its largest |d_b| in [2^21, 2^22); q = rint(d 2^t_p) split into
//          balanced signed bytes q = L0 2^16 + L1 2^8 + L2;
//   rows:  per row n a power-of-two scale 2^f_n with |A_nb| 2^f_n < 2^23 - 2^16,
//          w = rint(A_nb 2^f_n) = M0 2^16 + M1 2^8 + M2 (computed in FP64);
//   MMAs:  tcgen05.mma.kind::i8, INT32 accumulators by limb weight
//          S_k = sum_{a+b=k} La Mb^T for k = 0..3 (the weight-1 pair L2 M2 is
//          dropped: ~2^-32 of the leading term); S0..S3 and M0..M2 are adjacent,
//          so the eight limb products are three instructions per 32 bands;
//   epilogue: z_n = ((S0 256 + S1) 2^16 + (S2 256 + S3)) 2^(8 - f_n - t_p)
//          + (A_n . (mean32 - mean)): both halves are exact int32 sums, then FP32.
// Measured against the FP64 oracle: |RX error| / max(1, RX) and |ACE error|
// are a few 1e-5 at 113 bands (the fixed-point data step and the 24-bit rows).
//
// Kernel roles (one CTA per SM, persistent over 128-pixel tiles):
//   warp 0      TMA producer: 64-pixel boxes of the BSQ cube, all bands
//   warp 1      TMEM allocator + single-thread MMA issuer
//   warps 2-9   converters: per-pixel scale, limb tiles in the UMMA layout; four
//               warps (32 bands each) per 64-pixel half of the tile, so that one
//               half's loads and scale exchange run beside the other's conversion
//   warps 10-17 epilogue: TMEM -> z -> RX, ACE maps, best target; four warps for
//               output rows 0-63, four for rows 64-127
// Two MMA rounds per tile, each into its own half of TMEM: round h covers rows
// [32h, 32h + 32) and [64 + 32h, 64 + 32h + 32), so that both sets of epilogue
// warps drain it at once.  They give its columns back after the arithmetic of its
// last eight columns; the other round's products run under that arithmetic, and the
// next tile's under the output of the targets.
// Round h writes S0 to columns [256h, 256h + 64), S1 the next 64, S2 and S3
// after them.  The whitener limbs lie in shared memory by round, [M0 | M1 | M2]
// of its 64 rows (8 KB each).  Bands are padded to a multiple of 32 only: short
// spectra take fewer MMA steps and converter warps, and smaller boxes in a
// deeper ring.
// What bounds it: shared memory feeds the MMAs (28 KB per round and 32 bands),
// the converters and the epilogue's row constants, about 4900 of the 5500 cycles
// that a 128-pixel tile takes at 113 bands.  2048 x 1024 x 113 FP32 with 8 targets:
// 340 us; 391 us when each half of TMEM was drained by four warps alone and held
// until the tile's output, an operand was read by five instructions per 32 bands, and the
// epilogue's output took the targets one at a time.  1024 x 1024 x 16: 95 us,
// 154 us before.
#include <cuda_fp16.h>

#include <type_traits>

#include "tc.cuh"
#include "launch_state.h"

namespace hsi_b200 {
namespace {

constexpr int kRows = 128;   // output rows (N): whitener rows + target rows
constexpr int kK = 128;      // bands (K), zero-padded
constexpr int kTilePx = 128; // pixels per tile (M)
constexpr int kBoxPx = 64;   // pixels per TMA box
constexpr int kOpStages = 2;
constexpr int kConvWarps = 8;
constexpr int kEpiWarps = 8;
constexpr int kWarpTma = 0, kWarpMma = 1, kWarpConv0 = 2, kWarpEpi0 = kWarpConv0 + kConvWarps;
constexpr int kThreads = (kWarpEpi0 + kEpiWarps) * 32;  // 576
constexpr int kLimbBytes = kRows * kK;                  // 16 KB per limb tile
constexpr int kMaxTargetsPerPass = HSI_MAX_FILTERS_PER_PASS;
constexpr uint32_t kTmemCols = 512;

constexpr int kInBytes = 2 * kK * kBoxPx * 4;           // the ring of input boxes: 64 KB
constexpr int kMaxIn = 8;                               // boxes in the ring, at most
constexpr int kBandStep = 32;                           // bands per MMA (and per converter warp)
constexpr int kConvPerBox = kConvWarps / 2;             // converter warps of a box

// Per-frame operands written by the prep kernel (workspace) and staged into
// shared memory by every CTA.
struct TcOperands {
  unsigned char limbs[3][kLimbBytes];  // M0 | M1 | M2 tiles, UMMA 128B-swizzled K-major
  float gain[kRows];                   // 2^(8 - f_n) (0 for unused rows)
  float offset[kRows];                 // A_n . (mean32 - mean)
  float mean32[kK];                    // mean rounded to float (0 past B)
  float uu[kMaxTargetsPerPass];        // |u_t|^2 of this pass's targets
};

struct Smem {
  size_t w_off, a_off, in_off, red_off, t_off, ops_off, zz_off, zb_off, bar_off, slot_off, total;
};

__host__ __device__ inline Smem smem_layout() {
  Smem s;
  size_t off = 0;
  s.w_off = off;                    // 48 KB, 1024-aligned
  off += 3 * kLimbBytes;
  s.a_off = off;                    // kOpStages x 48 KB
  off += static_cast<size_t>(kOpStages) * 3 * kLimbBytes;
  s.in_off = off;
  off += kInBytes;
  s.red_off = off;                  // [2 halves][2][4][64] floats: pixel maxima over a warp's bands
  off += 2 * kConvWarps * kBoxPx * sizeof(float);
  s.t_off = off;                    // [kOpStages][128] ints: pixel scale exponents
  off += kOpStages * kTilePx * sizeof(int);
  s.ops_off = off;                  // gain, offset, mean32, uu, 1 / uu
  off += (3 * kRows + 2 * kMaxTargetsPerPass) * sizeof(float);
  s.zz_off = off;                   // [128] |z|^2 over rows 64-127
  off += kTilePx * sizeof(float);
  s.zb_off = off;                   // [16][128] ACE numerators
  off += kMaxTargetsPerPass * kTilePx * sizeof(float);
  s.bar_off = off;
  off += (2 * kMaxIn + 2 * kOpStages + 6 + 4 + 8) * sizeof(uint64_t);
  s.slot_off = off;
  off += 16;
  s.total = off + 1024;
  return s;
}

struct TcArgs {
  int64_t pixels;
  int bands;
  int steps;     // bands in steps of kBandStep
  int rows;      // B + targets of this pass
  int ntarg;     // targets of this pass
  int t0;        // first target index of this pass
  int first, last;
  const TcOperands* ops;
  float* rx;
  float* ace_best;
  int32_t* ace_target;
  float* ace_maps;
  int64_t map_stride;
  int* status;
};

// Where output row n lies among the limb tiles' rows: by MMA round, see above.
__device__ __forceinline__ int limb_row(int n) { return ((n >> 5) & 1) * 64 + (n >> 6) * 32 + (n & 31); }

__device__ __forceinline__ uint32_t sw128_byte(int row, int k) {
  return static_cast<uint32_t>((row >> 3) * 1024 + (row & 7) * 128 + ((((k >> 4) ^ (row & 7))) << 4) + (k & 15));
}

__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<uint64_t&>(r))
      : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<uint64_t&>(r))
      : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
  return r;
}
// max(a, |b|, |c|)
__device__ __forceinline__ float max_abs(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(fabsf(b)), "f"(fabsf(c)));
  return r;
}
// Two consecutive elements (8- or 4-byte aligned) as floats.
__device__ __forceinline__ float2 load2f(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 load2f(const __half* p) { return __half22float2(*reinterpret_cast<const __half2*>(p)); }


// ---- prep: the augmented matrix in fixed point, FP64 ------------------------
// One block per output row n; thread k = band.
__global__ void __launch_bounds__(128) tc_prep_kernel(const double* __restrict__ stats, int B, int T, int t0,
                                                      int ntarg, TcOperands* __restrict__ ops) {
  const int n = blockIdx.x, k = threadIdx.x;
  const double* mean = stats;
  const double* W = stats + B;
  const double* tw = W + static_cast<size_t>(B) * B;
  const double* tn = tw + static_cast<size_t>(T) * B;
  __shared__ double red[128];
  double a = 0.0;
  if (n < B) {
    if (k < B) a = W[static_cast<size_t>(n) * B + k];
  } else if (n < B + ntarg) {
    // v_k = sum_{i >= k} W_ik u_i in ascending i: 32 rows of W in flight at a time
    // (a load per term of the chain took most of the launch: 17 us, now 4.5 us)
    __shared__ double u[128];
    if (k < B) u[k] = tw[static_cast<size_t>(t0 + n - B) * B + k];
    __syncthreads();
    const double* col = W + min(k, B - 1);
    for (int i0 = k & ~31; i0 < B; i0 += 32) {
      double w[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) w[j] = col[static_cast<size_t>(min(i0 + j, B - 1)) * B];
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (i0 + j >= k && i0 + j < B) a += w[j] * u[i0 + j];
    }
  }
  const double m32 = k < B ? static_cast<double>(static_cast<float>(mean[k])) : 0.0;
  const double dm = k < B ? m32 - mean[k] : 0.0;
  // row maximum
  red[k] = fabs(a);
  __syncthreads();
  for (int s = 64; s > 0; s >>= 1) {
    if (k < s) red[k] = fmax(red[k], red[k + s]);
    __syncthreads();
  }
  const double amax = red[0];
  __syncthreads();
  int f = 0;
  if (amax > 0.0) {
    f = static_cast<int>(floor(log2((8388608.0 - 65536.0) / amax)));
    while (ldexp(amax, f) >= 8388608.0 - 65536.0) --f;  // guard the log2 rounding
  }
  const int w = amax > 0.0 ? static_cast<int>(rint(ldexp(a, f))) : 0;
  const int m2 = ((w + 128) & 255) - 128;
  const int w1 = (w - m2) >> 8;
  const int m1 = ((w1 + 128) & 255) - 128;
  const int m0 = (w1 - m1) >> 8;
  const uint32_t o = sw128_byte(limb_row(n), k);
  ops->limbs[0][o] = static_cast<unsigned char>(m0 & 255);
  ops->limbs[1][o] = static_cast<unsigned char>(m1 & 255);
  ops->limbs[2][o] = static_cast<unsigned char>(m2 & 255);
  // offset = A_n . (mean32 - mean), FP64
  red[k] = a * dm;
  __syncthreads();
  for (int s = 64; s > 0; s >>= 1) {
    if (k < s) red[k] += red[k + s];
    __syncthreads();
  }
  if (k == 0) {
    ops->gain[n] = amax > 0.0 ? static_cast<float>(ldexp(1.0, 8 - f)) : 0.0f;
    ops->offset[n] = static_cast<float>(red[0]);
  }
  if (n == 0) {
    ops->mean32[k] = static_cast<float>(m32);
    if (k < kMaxTargetsPerPass) ops->uu[k] = k < ntarg ? static_cast<float>(tn[t0 + k]) : 0.0f;
  }
}

// ---- the contraction ------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kThreads, 1)
    rxace_tc_kernel(const __grid_constant__ CUtensorMap cube_map, const TcArgs args) {
  // the ring of input boxes: a power of two of them
  const int steps = args.steps;
  const uint32_t box_bytes = static_cast<uint32_t>(steps) * kBandStep * kBoxPx * sizeof(T);
  int in_log = 1;
  while ((2 << in_log) <= kMaxIn && (2u << in_log) * box_bytes <= kInBytes) ++in_log;
  const int kIn = 1 << in_log;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const Smem L = smem_layout();
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L.bar_off);
  uint64_t* in_full = bars;
  uint64_t* in_empty = in_full + kMaxIn;
  uint64_t* op_full = in_empty + kMaxIn;
  uint64_t* op_empty = op_full + kOpStages;
  uint64_t* acc_full = op_empty + kOpStages;  // [2]: one per MMA round
  uint64_t* acc_empty = acc_full + 2;         // [2]
  uint64_t* w_full = acc_empty + 2;
  uint64_t* mma_done = w_full + 1;
  uint64_t* red_bar = mma_done + 1;    // [2 halves][2]: a box's per-warp maxima written
  uint64_t* half_full = red_bar + 4;   // [4]: rows 64-127 of a TMEM lane quarter's pixels are in zzp, zbuf
  uint64_t* half_empty = half_full + 4;  // [4]: and have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L.slot_off);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L.slot_off + 8);
  float* red = reinterpret_cast<float*>(smem + L.red_off);
  int* tvec = reinterpret_cast<int*>(smem + L.t_off);
  float* gain = reinterpret_cast<float*>(smem + L.ops_off);
  float* offset = gain + kRows;
  float* mean32 = offset + kRows;
  float* uu = mean32 + kK;
  float* uinv = uu + kMaxTargetsPerPass;
  float* zzp = reinterpret_cast<float*>(smem + L.zz_off);
  float* zbuf = reinterpret_cast<float*>(smem + L.zb_off);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t P = args.pixels;
  const int64_t ntiles = div_up<int64_t>(P, kTilePx);
  // static persistent schedule: tiles blockIdx.x, blockIdx.x + gridDim.x, ...
  const int n = ntiles > blockIdx.x ? static_cast<int>((ntiles - 1 - blockIdx.x) / gridDim.x + 1) : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kIn; ++s) {
      mbar_init(&in_full[s], 1);
      mbar_init(&in_empty[s], steps);
    }
    for (int s = 0; s < kOpStages; ++s) {
      mbar_init(&op_full[s], 2 * steps);
      mbar_init(&op_empty[s], 1 + kEpiWarps);  // MMA done with the limbs + epilogue done with the scales
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(&acc_full[h], 1);
      mbar_init(&acc_empty[h], kEpiWarps);
    }
    mbar_init(w_full, 1);
    mbar_init(mma_done, 1);
    for (int b = 0; b < 4; ++b) {
      mbar_init(&red_bar[b], steps);
      mbar_init(&half_full[b], 1);
      mbar_init(&half_empty[b], 1);
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  for (int i = threadIdx.x; i < 3 * kRows + kMaxTargetsPerPass; i += blockDim.x) gain[i] = args.ops->gain[i];
  if (threadIdx.x < kMaxTargetsPerPass) {
    const float v = args.ops->uu[threadIdx.x];
    uinv[threadIdx.x] = v > 0.0f ? 1.0f / v : 0.0f;
  }
  if (warp == kWarpMma) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == kWarpTma) {
    if (lane == 0) {
      prefetch_tensormap(&cube_map);
      // the whitener limbs, once, by MMA round: limb l of round h at (3h + l) x 8 KB
      mbar_arrive_expect_tx(w_full, 3 * kLimbBytes);
      for (int h = 0; h < 2; ++h)
        for (int l = 0; l < 3; ++l)
          bulk_g2s(smem + L.w_off + (3 * h + l) * (kLimbBytes / 2), args.ops->limbs[l] + h * (kLimbBytes / 2),
                   kLimbBytes / 2, w_full);
      uint32_t pending = 0, parity = 0;
      for (int i = 0; i < 2 * n; ++i) {
        const int s = i & (kIn - 1);
        const uint32_t ph = (i >> in_log) & 1u;
        if (*abort_flag || !mbar_wait_idle(&in_empty[s], ph ^ 1u)) {
          record_error(args.status, HSI_E_TIMEOUT);
          *abort_flag = 1;
          break;
        }
        const int64_t tile = blockIdx.x + static_cast<int64_t>(i >> 1) * gridDim.x;
        mbar_arrive_expect_tx(&in_full[s], box_bytes);
        tma_load_2d(smem + L.in_off + static_cast<size_t>(s) * box_bytes, &cube_map,
                    static_cast<int>(tile * kTilePx + (i & 1) * kBoxPx), 0, &in_full[s]);
        pending |= 1u << s;
        parity = (parity & ~(1u << s)) | (ph << s);
      }
      for (int s = 0; s < kIn; ++s)
        if ((pending >> s) & 1u) mbar_wait_idle(&in_full[s], (parity >> s) & 1u);
      mbar_wait_idle(w_full, 0);
    }
  } else if (warp == kWarpMma) {
    if (lane == 0) {
      const uint32_t id192 = idesc_s8_s32(kTilePx, 192);  // [M0; M1; M2] of a round
      const uint32_t id128 = idesc_s8_s32(kTilePx, 128);  // [M0; M1]
      const uint32_t id64 = idesc_s8_s32(kTilePx, 64);    // M2
      const int rounds = args.rows > 32 ? 2 : 1;
      bool issued = false;
      if (n > 0 && !mbar_wait_idle(w_full, 0)) {
        record_error(args.status, HSI_E_TIMEOUT);
        *abort_flag = 1;
      }
      bool ok = true;
      for (int i = 0; i < n && ok && !*abort_flag; ++i) {
        const int so = i % kOpStages;
        if (!mbar_wait_idle(&op_full[so], (i / kOpStages) & 1u)) {
          record_error(args.status, HSI_E_TIMEOUT);
          *abort_flag = 1;
          break;
        }
        unsigned char* a = smem + L.a_off + static_cast<size_t>(so) * 3 * kLimbBytes;
        const uint64_t a0 = smem_desc_sw128(a), a1 = smem_desc_sw128(a + kLimbBytes);
        const uint64_t a2 = smem_desc_sw128(a + 2 * kLimbBytes);
        for (int h = 0; h < rounds; ++h) {
          if (!mbar_wait_idle(&acc_empty[h], (i & 1u) ^ 1u)) {
            record_error(args.status, HSI_E_TIMEOUT);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem + 256u * h;  // S0 | S1 | S2 | S3 of this round's rows, 64 columns each
          const uint64_t bw = smem_desc_sw128(smem + L.w_off + 3 * h * (kLimbBytes / 2));         // [M0; M1; M2]
          const uint64_t bw2 = smem_desc_sw128(smem + L.w_off + (3 * h + 2) * (kLimbBytes / 2));  // M2
          umma_i8(d + 128, a2, bw, id128, 0u);  // S2 = L2 M0, S3 = L2 M1
          umma_i8(d + 0, a0, bw, id128, 0u);    // S0 = L0 M0, S1 = L0 M1
          umma_i8(d + 128, a0, bw2, id64, 1u);  // S2 += L0 M2
          umma_i8(d + 64, a1, bw, id192, 1u);   // S1 += L1 M0, S2 += L1 M1, S3 += L1 M2
          for (int k = 1; k < steps; ++k) {
            const uint64_t adv = static_cast<uint64_t>(k * 2);  // 32 bytes of K in 16-byte units
            umma_i8(d + 128, a2 + adv, bw + adv, id128, 1u);
            umma_i8(d + 0, a0 + adv, bw + adv, id192, 1u);
            umma_i8(d + 64, a1 + adv, bw + adv, id192, 1u);
          }
          umma_commit(&acc_full[h]);
          issued = true;
        }
        if (!ok) break;
        umma_commit(&op_empty[so]);
      }
      if (issued) {
        umma_commit(mma_done);
        if (!mbar_wait_idle(mma_done, 0)) record_error(args.status, HSI_E_TIMEOUT);
      }
    }
  } else if (warp < kWarpEpi0) {
    // ---------------- converters ----------------
    // Four warps per half of a tile: warp w of half `half` owns bands [32w, 32w + 32)
    // of the half's boxes; lane l reads box pixels 2l and 2l + 1 (one 64- or 32-bit
    // load per band for both) and stores them as operand rows l and l + 32: the 32
    // rows of one limb store then fall evenly on the eight 16-byte slots of the
    // 128-byte swizzle (row & 7), four conflict-free wavefronts.
    const int c = warp - kWarpConv0, half = c / kConvPerBox, w = c % kConvPerBox;
    constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
    const int wbias = __float_as_int(kMagic) - 0x8080;
    const float4* mu = reinterpret_cast<const float4*>(mean32 + w * kBandStep);
    for (int i = 0; i < n && w < steps; ++i) {
      const int j = 2 * i + half, s = j & (kIn - 1), so = i % kOpStages;
      if (!mbar_wait_idle(&in_full[s], (j >> in_log) & 1u)) {
        record_error(args.status, HSI_E_TIMEOUT);
        *abort_flag = 1;
        break;
      }
      const T* in = reinterpret_cast<const T*>(smem + L.in_off + static_cast<size_t>(s) * box_bytes) +
                    w * kBandStep * kBoxPx + 2 * lane;
      const int64_t tile = blockIdx.x + static_cast<int64_t>(i) * gridDim.x;
      float* r = red + (half * 2 + (i & 1)) * kConvPerBox * kBoxPx;
      float2 d[2][kBandStep / 2];  // band pairs
#pragma unroll
      for (int g = 0; g < kBandStep / 4; ++g) {
        const float4 m4 = mu[g];
        float2 x[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = load2f(in + (g * 4 + e) * kBoxPx);
        d[0][2 * g] = add2(make_float2(x[0].x, x[1].x), make_float2(-m4.x, -m4.y));
        d[1][2 * g] = add2(make_float2(x[0].y, x[1].y), make_float2(-m4.x, -m4.y));
        d[0][2 * g + 1] = add2(make_float2(x[2].x, x[3].x), make_float2(-m4.z, -m4.w));
        d[1][2 * g + 1] = add2(make_float2(x[2].y, x[3].y), make_float2(-m4.z, -m4.w));
      }
      // pixels past the frame (last tile only) convert as zeros
      const int64_t left = P - tile * kTilePx - half * kBoxPx - 2 * lane;
      if (left <= 1) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int jj = 0; jj < kBandStep / 2; ++jj)
            if (h >= left) d[h][jj] = make_float2(0.0f, 0.0f);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float m = 0.0f;
#pragma unroll
        for (int jj = 0; jj < kBandStep / 2; ++jj) m = max_abs(m, d[h][jj].x, d[h][jj].y);
        r[w * kBoxPx + 32 * h + lane] = m;
      }
      // the input box is consumed (values are in registers); maxima published
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&in_empty[s]);
        mbar_arrive(&red_bar[half * 2 + (i & 1)]);
      }
      if (!mbar_wait_idle(&red_bar[half * 2 + (i & 1)], (i >> 1) & 1u) ||
          !mbar_wait_idle(&op_empty[so], ((i / kOpStages) & 1u) ^ 1u)) {
        record_error(args.status, HSI_E_TIMEOUT);
        *abort_flag = 1;
        break;
      }
      unsigned char* a = smem + L.a_off + static_cast<size_t>(so) * 3 * kLimbBytes;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float m = 0.0f;
#pragma unroll
        for (int cc = 0; cc < kConvPerBox; ++cc)
          if (cc < steps) m = fmaxf(m, r[cc * kBoxPx + 32 * h + lane]);
        // 2^t with m 2^t in [2^21, 2^22): |q| <= 2^22, exact through the FMA rounding
        int t = 0;
        if (m > 0.0f) t = min(max(21 - (static_cast<int>((__float_as_uint(m) >> 23) & 255u) - 127), -100), 100);
        const float sc = __int_as_float((t + 127) << 23);
        const int row = half * kBoxPx + 32 * h + lane;
#pragma unroll
        for (int u = 0; u < kBandStep / 16; ++u) {
          uint32_t l0[4], l1[4], l2[4];
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const float2 v01 = ffma2(d[h][u * 8 + g * 2], make_float2(sc, sc), make_float2(kMagic, kMagic));
            const float2 v23 = ffma2(d[h][u * 8 + g * 2 + 1], make_float2(sc, sc), make_float2(kMagic, kMagic));
            const int q[4] = {__float_as_int(v01.x) - wbias, __float_as_int(v01.y) - wbias,
                              __float_as_int(v23.x) - wbias, __float_as_int(v23.y) - wbias};
            const uint32_t p01 = __byte_perm(q[0], q[1], 0x5140), p23 = __byte_perm(q[2], q[3], 0x5140);
            const uint32_t h01 = __byte_perm(q[0], q[1], 0x7362), h23 = __byte_perm(q[2], q[3], 0x7362);
            l2[g] = __byte_perm(p01, p23, 0x5410) ^ 0x80808080u;
            l1[g] = __byte_perm(p01, p23, 0x7632) ^ 0x80808080u;
            l0[g] = __byte_perm(h01, h23, 0x5410);
          }
          const uint32_t o = sw128_byte(row, w * kBandStep + u * 16);
          *reinterpret_cast<uint4*>(a + o) = make_uint4(l0[0], l0[1], l0[2], l0[3]);
          *reinterpret_cast<uint4*>(a + kLimbBytes + o) = make_uint4(l1[0], l1[1], l1[2], l1[3]);
          *reinterpret_cast<uint4*>(a + 2 * kLimbBytes + o) = make_uint4(l2[0], l2[1], l2[2], l2[3]);
        }
        if (w == 0) tvec[so * kTilePx + row] = t;
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&op_full[so]);
    }
  } else {
    // ---------------- epilogue ----------------
    const int e = warp - kWarpEpi0;
    const int q = warp & 3;         // TMEM lane quarter this warp may access
    const int hf = e >> 2;          // row half: rows [64 hf, 64 hf + 64)
    const int px = q * 32 + lane;   // operand row, and the tile's pixel in it
    const int pixel = (q >> 1) * kBoxPx + 2 * lane + (q & 1);
    const uint32_t trow = tmem + (static_cast<uint32_t>(q * 32) << 16);
    const int B = args.bands, rows = args.rows, nt = args.ntarg;
    const int rounds = rows > 32 ? 2 : 1;
    uint32_t valid = 0;  // this pass's targets with a norm above zero
    for (int k = 0; k < nt; ++k) valid |= (uu[k] > 0.0f ? 1u : 0u) << k;
    for (int i = 0; i < n; ++i) {
      const int so = i % kOpStages;
      // the scales were published with the limbs (already complete: the MMA waited on it)
      if (!mbar_wait_idle(&op_full[so], (i / kOpStages) & 1u)) {
        record_error(args.status, HSI_E_TIMEOUT);
        *abort_flag = 1;
        break;
      }
      const int t = tvec[so * kTilePx + px];
      __syncwarp();
      if (lane == 0) mbar_arrive(&op_empty[so]);  // scales read
      const float tau = __int_as_float((127 - t) << 23);
      float zz = 0.0f;
      bool ok = true;
      bool mine = hf == 0;  // zzp and zbuf may be written: the last tile's have been read
#pragma unroll 1
      for (int h = 0; h < rounds && ok; ++h) {
        if (!mbar_wait_idle(&acc_full[h], i & 1u)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const int m0 = hf * 64 + h * 32;                      // the round's first row here
        const uint32_t col = trow + 256u * h + 32u * hf;      // S0 of it; S1, S2, S3 64 columns apart
        auto load = [&](int cb, uint32_t (&v)[4][8]) {
#pragma unroll
          for (int k = 0; k < 4; ++k) tmem_ld8(col + 8u * cb + 64u * k, v[k]);
        };
        // all_bands: every row of the block is a whitened band (the common case: no
        // per-row test); otherwise rows past B are ACE numerators, past `rows` unused
        auto block = [&](auto all_bands, int n0, const uint32_t (&v)[4][8]) {
#pragma unroll
          for (int w = 0; w < 2; ++w) {
            // four rows' gains and offsets per float4 broadcast
            const float4 gv = *reinterpret_cast<const float4*>(gain + n0 + 4 * w);
            const float4 ov = *reinterpret_cast<const float4*>(offset + n0 + 4 * w);
#pragma unroll
            for (int jj = 0; jj < 4; jj += 2) {
              const int j = 4 * w + jj;
              const int nn = n0 + j;
              // u = S0 2^24 + S1 2^16 + S2 2^8 + S3 as (S0 256 + S1) 2^16 + (S2 256 + S3):
              // |S0| <= 2^20, |S1| < 2^21.6, |S2| < 2^22.3, |S3| <= 2^22 (128 bands of
              // |L0| <= 64, other limbs <= 128 in magnitude), so both halves are exact int32
              float2 hi, lo;
              hi.x = __int2float_rn(static_cast<int>(v[0][j]) * 256 + static_cast<int>(v[1][j]));
              hi.y = __int2float_rn(static_cast<int>(v[0][j + 1]) * 256 + static_cast<int>(v[1][j + 1]));
              lo.x = __int2float_rn(static_cast<int>(v[2][j]) * 256 + static_cast<int>(v[3][j]));
              lo.y = __int2float_rn(static_cast<int>(v[2][j + 1]) * 256 + static_cast<int>(v[3][j + 1]));
              const float2 u = ffma2(hi, make_float2(65536.0f, 65536.0f), lo);
              const float2 z = ffma2(mul2(u, make_float2(tau, tau)), jj ? make_float2(gv.z, gv.w) : make_float2(gv.x, gv.y),
                                     jj ? make_float2(ov.z, ov.w) : make_float2(ov.x, ov.y));
              if (decltype(all_bands)::value) {
                zz = fmaf(z.x, z.x, zz);
                zz = fmaf(z.y, z.y, zz);
              } else {
                zz = nn < B ? fmaf(z.x, z.x, zz) : zz;
                if (nn >= B && nn < rows) zbuf[(nn - B) * kTilePx + px] = z.x;
                zz = nn + 1 < B ? fmaf(z.y, z.y, zz) : zz;
                if (nn + 1 >= B && nn + 1 < rows) zbuf[(nn + 1 - B) * kTilePx + px] = z.y;
              }
            }
          }
        };
        uint32_t v[4][8];
#pragma unroll 1
        for (int cb = 0; cb < 4; ++cb) {
          const int n0 = m0 + 8 * cb;
          if (n0 >= rows) break;  // warp-uniform
          load(cb, v);
          tmem_wait_ld();
          if (n0 + 8 <= B) {
            block(std::true_type{}, n0, v);
          } else {
            if (!mine && !mbar_wait_idle(&half_empty[q], (i & 1u) ^ 1u)) {
              ok = false;
              break;
            }
            mine = true;
            block(std::false_type{}, n0, v);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[h]);
      }
      if (ok && !mine) ok = mbar_wait_idle(&half_empty[q], (i & 1u) ^ 1u);
      if (ok && hf == 1) {
        zzp[px] = zz;
        __syncwarp();
        if (lane == 0) mbar_arrive(&half_full[q]);
        continue;
      }
      if (!ok || !mbar_wait_idle(&half_full[q], i & 1u)) {
        record_error(args.status, HSI_E_TIMEOUT);
        *abort_flag = 1;
        break;
      }
      const int64_t tile = blockIdx.x + static_cast<int64_t>(i) * gridDim.x;
      const int64_t p = tile * kTilePx + pixel;
      if (p < P) {
        const float rx = zz + zzp[px];
        if (args.rx && args.first) args.rx[p] = rx;
        if (nt > 0) {
          float best = -1.0f;
          int32_t best_t = -1;
          if (!args.first) {
            if (args.ace_best) best = args.ace_best[p];
            if (args.ace_target) best_t = args.ace_target[p];
          }
          // (z.u)^2 / (|u|^2 |z|^2) as (z.u)^2 (1 / |u|^2) (1 / |z|^2): one division per
          // pixel instead of one per target
          const float rinv = rx > 0.0f ? 1.0f / rx : 0.0f;
          const uint32_t live = rx > 0.0f ? valid : 0u;  // targets that score here
          float* map = args.ace_maps ? args.ace_maps + static_cast<int64_t>(args.t0) * args.map_stride + p : nullptr;
          // four targets' numerators and scales in flight (slots past nt are readable)
          for (int k0 = 0; k0 < nt; k0 += 4) {
            const float4 ui = *reinterpret_cast<const float4*>(uinv + k0);
            const float uk[4] = {ui.x, ui.y, ui.z, ui.w};
            float zu[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) zu[k] = zbuf[(k0 + k) * kTilePx + px];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const bool on = (live >> (k0 + k)) & 1u;
              const float a = on ? (zu[k] * zu[k]) * (uk[k] * rinv) : 0.0f;
              const bool better = on && a > best;
              best = better ? a : best;
              best_t = better ? args.t0 + k0 + k : best_t;
              if (map && k0 + k < nt) map[static_cast<int64_t>(k0 + k) * args.map_stride] = a;
            }
          }
          if (args.ace_best) args.ace_best[p] = args.last ? (best < 0.0f ? 0.0f : fminf(best, 1.0f)) : best;
          if (args.ace_target) args.ace_target[p] = best_t;
        }
      }
      // zzp / zbuf free for the next tile
      __syncwarp();
      if (lane == 0) mbar_arrive(&half_empty[q]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kWarpMma) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

size_t tc_ws_bytes() { return (sizeof(TcOperands) + 255) & ~size_t(255); }

int sm_count() { return device_sm_count(); }

template <typename T>
int launch_tc(const void* cube, int64_t P, int B, int64_t stride, const double* stats, int ntargets, float* rx,
              float* ace_best, int32_t* ace_target, float* ace_maps, int64_t map_stride, void* ws, cudaStream_t s) {
  CUtensorMap map;
  const int steps = div_up(B, kBandStep);
  const int dt = sizeof(T) == 4 ? HSI_F32 : HSI_F16;
  if (encode_cube_map(&map, cube, dt, P, B, stride, kBoxPx, steps * kBandStep) != 0) return HSI_E_INVALID;
  const Smem L = smem_layout();
  // set once per device and element type
  const cudaError_t configured = raise_smem_limit(rxace_tc_kernel<T>, static_cast<int>(L.total));
  if (configured != cudaSuccess) return static_cast<int>(configured);
  TcOperands* ops = static_cast<TcOperands*>(ws);
  const int per_pass = kRows - B < kMaxTargetsPerPass ? kRows - B : kMaxTargetsPerPass;
  const int passes = ntargets > 0 ? (ntargets + per_pass - 1) / per_pass : 1;
  const int64_t ntiles = div_up<int64_t>(P, kTilePx);
  const int grid = static_cast<int>(ntiles < sm_count() ? ntiles : sm_count());
  for (int pass = 0; pass < passes; ++pass) {
    const int t0 = pass * per_pass;
    const int nt = ntargets > 0 ? (ntargets - t0 < per_pass ? ntargets - t0 : per_pass) : 0;
    tc_prep_kernel<<<kRows, 128, 0, s>>>(stats, B, ntargets, t0, nt, ops);
    TcArgs a;
    a.pixels = P;
    a.bands = B;
    a.steps = steps;
    a.rows = B + nt;
    a.ntarg = nt;
    a.t0 = t0;
    a.first = pass == 0;
    a.last = pass == passes - 1;
    a.ops = ops;
    a.rx = rx;
    a.ace_best = ace_best;
    a.ace_target = ace_target;
    a.ace_maps = ace_maps;
    a.map_stride = map_stride;
    a.status = nullptr;
    rxace_tc_kernel<T><<<grid, kThreads, L.total, s>>>(map, a);
  }
  return static_cast<int>(cudaGetLastError());
}

}  // namespace
}  // namespace hsi_b200

using namespace hsi_b200;

extern "C" HSI_API size_t hsi_rx_ace_workspace_bytes(int bands, int num_targets) {
  if (bands <= 0 || num_targets < 0) return 0;
  return tc_ws_bytes();
}

extern "C" HSI_API int hsi_rx_ace(const void* d_cube, int height, int width, int bands, int dtype,
                                  int64_t plane_stride, const double* d_stats64, int num_targets, float* d_rx,
                                  float* d_ace_best, int32_t* d_ace_target, float* d_ace_maps, int64_t map_stride,
                                  void* d_workspace, size_t workspace_bytes, hsi_stream_t stream) {
  if (!d_cube || !d_stats64 || height <= 0 || width <= 0 || bands <= 0) return HSI_E_INVALID;
  if (dtype != HSI_F32 && dtype != HSI_F16) return HSI_E_INVALID;
  if (bands > kK - 1 || num_targets < 0 || num_targets > 64) return HSI_E_CAPACITY;
  const int64_t P = static_cast<int64_t>(height) * width;
  if (plane_stride < P || (plane_stride & 7) != 0) return HSI_E_INVALID;
  if (num_targets > 0 && d_ace_maps && map_stride < P) return HSI_E_INVALID;
  if (!d_workspace || workspace_bytes < tc_ws_bytes()) return HSI_E_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(d_workspace) & 255u) != 0 || (reinterpret_cast<uintptr_t>(d_cube) & 15u) != 0)
    return HSI_E_INVALID;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == HSI_F32)
    return launch_tc<float>(d_cube, P, bands, plane_stride, d_stats64, num_targets, d_rx, d_ace_best, d_ace_target,
                            d_ace_maps, map_stride, d_workspace, s);
  return launch_tc<__half>(d_cube, P, bands, plane_stride, d_stats64, num_targets, d_rx, d_ace_best, d_ace_target,
                           d_ace_maps, map_stride, d_workspace, s);
}
