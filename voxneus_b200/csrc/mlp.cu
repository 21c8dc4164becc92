// Radiance MLP [hash 32 | SH 16 | normal 3] -> 64 ReLU -> 3 Sigmoid (models/radiance_mlp.py:42-53,
// 81-98) on the 5th-generation tensor cores (tcgen05, kind::tf32, accumulators in TMEM).
//
// Accuracy: every product runs as a 3-term split x = hi + lo (hi, lo tf32), a*b ~ ah*bh + ah*bl +
// al*bh, accumulated in f32 — about 21 bits per product, the FP32 parity bar (colours 1e-5, weight
// gradients 1e-4 of their scale) holds where a single tf32 pass (11 bits) would not.
//
// Operands are K-major canonical no-swizzle layouts (tc.cuh; kind::tf32 with an MN-major operand
// writes nothing on this part, so every operand is staged with its contraction dimension
// contiguous). A 16-byte chunk holds 4 consecutive K elements of one row:
//   X    (128 sample rows, K = features): chunk (m, 4f..4f+3) at (f*16 + m/8)*128 + (m%8)*16
//   W0   [hi; lo] (128 rows: hidden unit n's hi part in row n, its lo part in row 64 + n, K =
//        features): element (r, k) at ((k/4)*16 + r/8)*128 + (r%8)*16 + (k%4)*4
// The stacked hi/lo operand lets one N = 128 MMA form two of the three products:
//   Z   = X W0^T   A = X_hi, B = [W_hi; W_lo] (N = 128) + A = X_lo, B = W_hi (N = 64), K = 56 in 7
//                  steps; Z = columns [0, 64) + [64, 128)
// The forward writes the colours and, for the adjoint (mlp_adjoint.cuh), the input rows (52 floats, or
// the compact 36-float rows of the fused appearance path) and each sample's ReLU mask; the adjoint
// writes dL/d(hash), dL/d(normal) and per-block weight-gradient partials that k_mlp_wgrad_reduce sums in
// a fixed order (deterministic). The folded variant (compact rows whose tiles each lie inside one ray)
// contracts K = 40 features [hash | normal | 0] in 5 steps, with SH(d) as a per-ray bias of the hidden
// layer.
#include "hashgrid.cuh"
#include "tc.cuh"

namespace vx {

constexpr int KIN = 51;  // input features
constexpr int KP = 52;   // row width of the input rows (column 51 is padding)
// Compact rows of the fused appearance path: [hash 32 | normal 3 | pad], 144 bytes. The 16 SH(d)
// features (columns 32..47 of a full row) depend on the ray only. When a ray's samples fill whole
// 128-row tiles the folded MLP (fold_col below) adds them as a per-ray hidden bias;
// otherwise the MLP kernels rebuild them from the ray's direction while they stage a tile, the same
// function on the same operands as the row writer, so that both layouts give the same bits.
constexpr int KC = 36;
constexpr int NH = 64;   // hidden units
constexpr int NO = 3;    // colours
constexpr int TM = 128;  // samples per tile (TMEM lanes)
constexpr int WG = NH * KP + NO * NH + NH + NO;  // per-block weight-gradient partial size
constexpr uint32_t kWaitLimit = 1u << 22;       // default mbarrier polls before a tile gives up
// After a block gives up on a wait, the copy or MMA it waited for may still be running: the
// block waits for it (at most this many polls) before it frees tensor memory and exits, so no
// asynchronous write lands in memory that another block owns next.
constexpr uint32_t kDrainLimit = 1u << 22;

constexpr uint32_t kXBytes = 16 * 16 * 128;  // one tf32 part of X (or DZ)
constexpr uint32_t kWBytes = 16 * 16 * 128;  // W0 (or W0^T) as [hi; lo]

__device__ int g_tc_timeouts = 0;

// The wait policy of the MMA kernels: polls per mbarrier wait, and a caller's device status word
// (nullable) that every block which gave up increments.
struct TcGuard {
  int* status;
  uint32_t limit;
};

// The guard the host launchers of this thread pass (vx_tc_guard).
thread_local TcGuard t_guard{nullptr, kWaitLimit};

// Whether this thread's launches take the caller's poll limit (a kernel variant that reads it) or
// the default (a compile-time bound, which keeps the waits' loops as tight as before).
inline bool custom_wait() { return t_guard.limit != kWaitLimit; }

__device__ __forceinline__ void report_timeout(int* status) {
  atomicAdd(&g_tc_timeouts, 1);
  if (status) atomicAdd(status, 1);
}

// Where a kernel's full rows come from: rays_d == nullptr, rows of KP floats; otherwise compact
// rows of KC floats whose SH features are recomputed from rays_d of the sample's ray (i / S; the
// entry points keep the sample count below 2^32).
struct RowSrc {
  const float* rays_d;
  int64_t S;
};

// Feature chunk c = (hh ? 7 : 0) + j (0..12, four features each) of a staged sample: chunks 0..7
// the hash features, 8..11 SH(d), 12 the normal and the pad column. j is a constant of the
// unrolled staging loop, so each SH group is built only where it is stored.
template <bool kCompact>
__device__ __forceinline__ float4 x_chunk(const float4* rrow, bool hh, int j, float3 dir) {
  if (kCompact && hh) {
    if (j == 0) return rrow[7];
    if (j <= 4) return sh_chunk(dir.x, dir.y, dir.z, j - 1);
    return rrow[8];
  }
  return rrow[(hh ? 7 : 0) + j];
}

// The ray direction of sample i, for the thread that stages the sample's chunks 7..12.
template <bool kCompact>
__device__ __forceinline__ float3 stage_dir(const RowSrc& src, int64_t i, bool need) {
  float3 d = make_float3(0.0f, 0.0f, 0.0f);
  if (kCompact && need) {
    const uint32_t r = (uint32_t)i / (uint32_t)src.S;
    d = make_float3(__ldg(src.rays_d + 3 * (size_t)r), __ldg(src.rays_d + 3 * (size_t)r + 1),
                    __ldg(src.rays_d + 3 * (size_t)r + 2));
  }
  return d;
}

struct MlpW {
  const float* W0;  // (64, 51)
  const float* b0;  // (64)
  const float* W1;  // (3, 64)
  const float* b1;  // (3)
};

// The folded MLP (compact rows whose 128-row tiles each lie inside one ray, so SH(d) is constant
// over a tile): the 16 SH columns leave the contraction and become a per-ray bias of the hidden
// layer, b0 + W0[:, 32:48] SH(d) (columns summed in order). Its input features are [hash 32 | normal 3 | 0 x 5], K = 40
// (the adjoint puts a one after the normal).
// Folded feature k comes from column fold_col(k) of W0 (-1: none).
__device__ __forceinline__ int fold_col(int k) { return k < 32 ? k : (k < 35 ? 48 + (k - 32) : -1); }

__device__ __forceinline__ uint32_t x_off(int f, int m) { return (uint32_t)((f * 16 + (m >> 3)) * 128 + (m & 7) * 16); }
// row r of [W_hi; W_lo] (r < 64: hi of hidden unit r, else lo of hidden unit r - 64), feature k
__device__ __forceinline__ uint32_t w_off(int r, int k) {
  return (uint32_t)(((k >> 2) * 16 + (r >> 3)) * 128 + (r & 7) * 16 + (k & 3) * 4);
}

__device__ __forceinline__ void st_split4(uint8_t* hi, uint8_t* lo, uint32_t off, float a, float b, float c, float d) {
  float4 h, l;
  tc::split_tf32(a, h.x, l.x);
  tc::split_tf32(b, h.y, l.y);
  tc::split_tf32(c, h.z, l.z);
  tc::split_tf32(d, h.w, l.w);
  *reinterpret_cast<float4*>(hi + off) = h;
  *reinterpret_cast<float4*>(lo + off) = l;
}

// W0 as [hi; lo] tf32 (features 51..63 zero), b0, W1, b1; X feature chunks 13..15 (columns 52..63,
// never written by the tiles) zeroed.
__device__ void stage_weights(const MlpW& w, uint8_t* W2, uint8_t* XH, uint8_t* XL, float* B0, float* W1s, float* B1,
                              int tid, int nt) {
  for (int e = tid; e < NH * 64; e += nt) {
    const int n = e >> 6, k = e & 63;
    float h, l;
    tc::split_tf32(k < KIN ? w.W0[n * KIN + k] : 0.0f, h, l);
    *reinterpret_cast<float*>(W2 + w_off(n, k)) = h;
    *reinterpret_cast<float*>(W2 + w_off(NH + n, k)) = l;
  }
  for (int e = tid; e < 3 * TM; e += nt) {
    const uint32_t off = x_off(13 + e / TM, e % TM);
    *reinterpret_cast<float4*>(XH + off) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    *reinterpret_cast<float4*>(XL + off) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  for (int i = tid; i < NH; i += nt) B0[i] = w.b0[i];
  for (int i = tid; i < NO * NH; i += nt) W1s[i] = w.W1[i];
  if (tid < NO) B1[tid] = w.b1[tid];
}

constexpr uint32_t kId128 = tc::idesc_tf32(TM, 2 * NH, false, false);
constexpr uint32_t kId64 = tc::idesc_tf32(TM, NH, false, false);

// A [hi | lo] K-major operand times a stacked [hi; lo] B: columns [t, t + 64) receive
// A_hi B_hi + A_lo B_hi and [t + 64, t + 128) receive A_hi B_lo (one N = 128 and one N = 64 MMA per
// 8-wide K step; the result is the sum of the two column halves). Issued by one thread.
__device__ __forceinline__ void issue_split(uint32_t t, uint32_t ah0, uint32_t al0, uint32_t b0, int ksteps) {
#pragma unroll 1
  for (int ks = 0; ks < ksteps; ++ks) {
    const uint64_t ah = tc::sdesc(ah0 + ks * 4096, 2048, 128), al = tc::sdesc(al0 + ks * 4096, 2048, 128);
    const uint64_t b = tc::sdesc(b0 + ks * 4096, 2048, 128);
    tc::mma_tf32(t, ah, b, kId128, ks > 0);
    tc::mma_tf32(t, al, b, kId64, true);
  }
}

// Z = X W0^T into TMEM columns [tz, tz + 128) as two halves to add (same sequence in both passes).
__device__ __forceinline__ void issue_z(uint32_t tz, uint32_t xh, uint32_t xl, uint32_t w2) {
  issue_split(tz, xh, xl, w2, 7);
}

// 32 columns of a split result: TMEM columns [col, col + 32) + [col + 64, col + 96) of this warp's lanes
__device__ __forceinline__ void tmem_ld_sum32(uint32_t taddr, float v[32]) {
  float u[32];
  tc::tmem_ld32(taddr, v);
  tc::tmem_ld32(taddr + 64, u);
  tc::tmem_wait_ld();
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] += u[j];
}

// Where a forward's outputs go: colours (row stride ldc; may be null when mask is given) and, when mask is given, each sample's ReLU
// mask (bit j of word k: hidden unit 32 k + j is active; two words a sample, row stride ldm).
struct MlpOut {
  float* colors;
  int64_t ldc;
  uint32_t* mask;
  int64_t ldm;
};

// This thread's half of the colour pre-activation: hidden units 32*hh..32*hh+31 of sample lane; kMask:
// their ReLU bits.
template <bool kMask>
__device__ __forceinline__ uint32_t colour_partial(const float z[32], int hh, const float* B0, const float* W1s,
                                                   float& p0, float& p1, float& p2) {
  p0 = p1 = p2 = 0.0f;
  uint32_t bits = 0;
#pragma unroll
  for (int j4 = 0; j4 < 8; ++j4) {
    const int n = 32 * hh + 4 * j4;
    const float4 b = *reinterpret_cast<const float4*>(B0 + n);
    const float4 u0 = *reinterpret_cast<const float4*>(W1s + n);
    const float4 u1 = *reinterpret_cast<const float4*>(W1s + NH + n);
    const float4 u2 = *reinterpret_cast<const float4*>(W1s + 2 * NH + n);
    const float bb[4] = {b.x, b.y, b.z, b.w}, w0[4] = {u0.x, u0.y, u0.z, u0.w};
    const float w1[4] = {u1.x, u1.y, u1.z, u1.w}, w2[4] = {u2.x, u2.y, u2.z, u2.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float h = fmaxf(z[4 * j4 + i] + bb[i], 0.0f);
      if (kMask) bits |= (h > 0.0f ? 1u : 0u) << (4 * j4 + i);
      p0 = fmaf(w0[i], h, p0);
      p1 = fmaf(w1[i], h, p1);
      p2 = fmaf(w2[i], h, p2);
    }
  }
  return bits;
}

// The ReLU bits alone, of the same pre-activations.
__device__ __forceinline__ uint32_t relu_bits(const float z[32], int hh, const float* B0) {
  uint32_t bits = 0;
#pragma unroll
  for (int j4 = 0; j4 < 8; ++j4) {
    const float4 b = *reinterpret_cast<const float4*>(B0 + 32 * hh + 4 * j4);
    const float bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) bits |= (z[4 * j4 + i] + bb[i] > 0.0f ? 1u : 0u) << (4 * j4 + i);
  }
  return bits;
}

// Forward with the 51 features of a tile built in place: two threads per sample, 8 hash levels each; SH of the view
// direction; the normal. 256 threads: warp w reads TMEM lanes 32*(w%4).. and hidden columns 32*(w/4)..; the two
// column halves meet in shared memory.
template <bool kCustomWait>
__global__ void __launch_bounds__(256, 2) k_mlp_fwd_tc(HashArgs a, int64_t P, MlpW w, MlpOut out, TcGuard g) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t wait_limit = kCustomWait ? g.limit : kWaitLimit;  // a constant bound unless a caller set one
  uint8_t* XH = smem;
  uint8_t* XL = XH + kXBytes;
  uint8_t* W2 = XL + kXBytes;
  float* B0 = reinterpret_cast<float*>(W2 + kWBytes);
  float* W1s = B0 + NH;
  float* B1 = W1s + NO * NH;
  float* RED = B1 + 4;  // [2][TM][4]
  uint64_t* bar = reinterpret_cast<uint64_t*>(RED + 2 * TM * 4);
  uint32_t* s_taddr = reinterpret_cast<uint32_t*>(bar + 1);
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31, q = wid & 3, hh = wid >> 2;
  stage_weights(w, W2, XH, XL, B0, W1s, B1, tid, blockDim.x);
  if (tid == 0) tc::mbar_init(bar, 1);
  if (wid == 0) tc::tmem_alloc(s_taddr, 128);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *s_taddr;
  const uint32_t xh = tc::smem_u32(XH), xl = tc::smem_u32(XL), w2 = tc::smem_u32(W2);
  const uint32_t mask = (1u << a.log2T) - 1u;
  const size_t T = (size_t)1 << a.log2T;
  uint32_t phase = 0;
  const int64_t ntiles = (P + TM - 1) / TM;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t m0 = t * TM;
    const int m = tid & (TM - 1), half = tid >> 7;
    const int64_t i = m0 + m;
    float feat[16], extra[16];
    if (i < P) {
      float x[3];
      sample_pos(a, i, x);
#pragma unroll
      for (int qq = 0; qq < 8; ++qq) {
        const int l = 8 * half + qq;
        const float lw = a.lw[l];
        float f0 = 0.0f, f1 = 0.0f;
        if (lw != 0.0f) {
          LevelCell c;
          level_cell(x, a.res[l], mask, c);
          const float2* tab = reinterpret_cast<const float2*>(a.table) + (size_t)l * T;
          gather_level(tab, c, f0, f1);
          if (lw < 1.0f) {
            f0 *= lw;
            f1 *= lw;
          }
        }
        feat[2 * qq] = f0;
        feat[2 * qq + 1] = f1;
      }
      if (half == 0) {
        const int64_t r = i / a.S;
        sh16(__ldg(a.rays_d + 3 * r), __ldg(a.rays_d + 3 * r + 1), __ldg(a.rays_d + 3 * r + 2), extra);
      } else {
        extra[0] = a.normals[3 * i];
        extra[1] = a.normals[3 * i + 1];
        extra[2] = a.normals[3 * i + 2];
        extra[3] = 0.0f;
      }
    } else {
#pragma unroll
      for (int qq = 0; qq < 16; ++qq) feat[qq] = extra[qq] = 0.0f;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
      st_split4(XH, XL, x_off(4 * half + c, m), feat[4 * c], feat[4 * c + 1], feat[4 * c + 2], feat[4 * c + 3]);
    if (half == 0) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        st_split4(XH, XL, x_off(8 + c, m), extra[4 * c], extra[4 * c + 1], extra[4 * c + 2], extra[4 * c + 3]);
    } else {
      st_split4(XH, XL, x_off(12, m), extra[0], extra[1], extra[2], extra[3]);
    }
    tc::fence_smem_to_async();
    __syncthreads();
    if (tid == 0) {
      tc::fence_after_sync();
      issue_z(tbase, xh, xl, w2);
      tc::commit(bar);
    }
    const bool ok = tc::mbar_wait(bar, phase, wait_limit);
    phase ^= 1u;
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        if (!ok) tc::mbar_wait(bar, phase ^ 1u, kDrainLimit);  // this tile's Z MMA, before TMEM is freed
        report_timeout(g.status);
      }
      break;
    }
    tc::fence_after_sync();
    float z[32];
    tmem_ld_sum32(tbase + ((uint32_t)(32 * q) << 16) + 32 * hh, z);
    float p0, p1, p2;
    colour_partial<false>(z, hh, B0, W1s, p0, p1, p2);
    float* r = RED + (hh * TM + 32 * q + lane) * 4;
    r[0] = p0;
    r[1] = p1;
    r[2] = p2;
    tc::fence_before_sync();
    __syncthreads();
    if (tid < TM && m0 + tid < P) {
#pragma unroll
      for (int c = 0; c < NO; ++c) {
        const float o = (B1[c] + RED[tid * 4 + c]) + RED[(TM + tid) * 4 + c];
        out.colors[(m0 + tid) * out.ldc + c] = sigmoidf_ref(o);
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (wid == 0) tc::tmem_dealloc(tbase, 128);
}

constexpr size_t kFwdSmem = 2 * kXBytes + kWBytes + sizeof(float) * (NH + NO * NH + 4 + 2 * TM * 4) + 16;

// Forward on rows (52 floats, compact, or any stride from 51 on): one CTA per SM holding two independent tile slots
// of 256 worker threads, which share the stacked weights and the tensor core, and one issuing warp a slot
// (16 + slot), which issues the slot's MMAs and row copies (issuing blocks while the tensor core's queue
// is full; warp-issued, tc.cuh). A slot has two X operands (the lo part in shared memory, the hi part in
// TMEM columns, sample lanes, written with tcgen05.st), one accumulator of 128 columns and one or two
// row buffers that a bulk copy fills. A worker stages tile t+1 while the MMAs of tile t run, reads
// Z(t) out, hands both facts to the issuing warp (one arrival a warp on `ready`) and forms the colours
// while the MMAs of tile t+1 run, so no MMA is waited for unless the staging and the epilogue are
// shorter. What bounds it: the latency of the workers' chain (rows -> parts, accumulators -> colours) at
// 16 warps an SM, ~2,300 cycles a tile. 1,048,576 samples: 91 us (with masks 98; one X a slot, MMAs
// issued by one of its threads between two barriers, ~115 cycles apart: 2,000 of a tile's 5,600 cycles in
// its slot) -> 76 us; 61,440,000 samples 5.01 -> 3.89 ms.
template <bool kCompact, bool kFold>
struct FwdShape {
  static constexpr int kLd = kCompact ? KC : KP;                 // floats per row
  static constexpr int kKSteps = kFold ? 5 : 7;                  // of 8 features
  static constexpr int kBufs = kFold ? 2 : 1;                    // row buffers a slot
  static constexpr uint32_t kX = kKSteps * 2 * 2048;             // X_lo of a tile
  static constexpr uint32_t kRows = TM * kLd * 4;
  static constexpr uint32_t kOffHead = 16 * 2048;                // after W0 [hi; lo] (64 features)
  static constexpr uint32_t kOffSh = kOffHead + 4 * (NH + NO * NH + 4);  // folded: W0's SH columns [16][64]
  static constexpr uint32_t kOffBeta = kOffSh + (kFold ? 16 * NH * 4 : 0);    // folded: [slot][2][64]
  static constexpr uint32_t kOffRed = kOffBeta + (kFold ? 2 * 2 * NH * 4 : 0);  // [slot][2][2][TM][4]
  static constexpr uint32_t kOffBar = kOffRed + 2 * 2 * 2 * TM * 16;
  static constexpr uint32_t kOffSlot = (kOffBar + 96 + 1023) / 1024 * 1024;
  static constexpr uint32_t kSlot = 2 * kX + kBufs * kRows;
  static constexpr uint32_t kSmem = kOffSlot + 2 * kSlot;
};
static_assert(FwdShape<true, true>::kSmem <= 227 * 1024 && FwdShape<false, false>::kSmem <= 227 * 1024,
              "the forward's shared memory exceeds a CTA's");
static_assert(FwdShape<true, true>::kSmem > 116 * 1024, "two forward CTAs would fit on an SM and contend for TMEM");
static_assert(FwdShape<true, true>::kOffRed % 16 == 0 && FwdShape<true, true>::kOffBeta % 16 == 0 &&
                  FwdShape<false, false>::kOffRed % 16 == 0 && FwdShape<true, true>::kRows % 128 == 0 &&
                  FwdShape<false, false>::kRows % 128 == 0 && FwdShape<true, true>::kOffBar % 8 == 0 &&
                  FwdShape<false, false>::kOffBar % 8 == 0,
              "shared-memory alignment");
constexpr int kFwdThreads = 512 + 64;

// The rows of a forward: compact and folded, compact, contiguous 52 floats, any other stride. The last are brought in by
// the workers' asynchronous copies of 4 bytes, or 16 where the rows are aligned, a tile ahead: 1,000,000 rows 116 us
// (by the issuing warp alone 175; a kernel of its own with rows through registers 150), contiguous 75.
enum FwdRows { kFwdFold = 0, kFwdCompact = 1, kFwdFull = 2, kFwdStrided = 3 };

// A barrier of a slot's workers that also agrees on whether any of them gave up a wait. Like the tensor-memory loads
// and stores it is an instruction of a converged warp: __syncwarp() first wherever lanes can have parted.
__device__ __forceinline__ bool slot_sync_or(int slot, bool v) {
  uint32_t r;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, %2, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"(v ? 1u : 0u), "r"(1 + slot)
      : "memory");
  return r != 0;
}

template <bool kCustomWait, FwdRows kRows, bool kMask>
__global__ void __launch_bounds__(kFwdThreads, 1)
    k_mlp_fwd_rows2(const float* __restrict__ X, int64_t ldx, int xvec, int64_t P, MlpW w, MlpOut out, TcGuard g,
                    RowSrc src) {
  constexpr bool kFold = kRows == kFwdFold, kCompact = kRows == kFwdFold || kRows == kFwdCompact;
  constexpr bool kStrided = kRows == kFwdStrided;
  using S = FwdShape<kCompact, kFold>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t wait_limit = kCustomWait ? g.limit : kWaitLimit;
  uint8_t* W2 = smem;
  float* B0 = reinterpret_cast<float*>(smem + S::kOffHead);
  float* W1s = B0 + NH;
  float* B1 = W1s + NO * NH;
  float* WSH = reinterpret_cast<float*>(smem + S::kOffSh);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // in a uniform register: warp-uniform branches
  const bool issuer = warp >= 16;
  const int slot = issuer ? warp - 16 : warp >> 3;
  const int wid = warp & 7, q = wid & 3, hh = wid >> 2, stid = 32 * wid + lane;
  const int m = 32 * q + lane;  // this thread's sample in its slot's tile
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kOffBar) + 4 * slot;
  uint64_t* bar = bars;            // the slot's MMAs of a tile
  uint64_t* ready = bars + 1;      // X of a tile staged and the previous Z read (8 arrivals)
  uint64_t* bar_rows = bars + 2;   // [2]
  volatile int* s_fail = reinterpret_cast<volatile int*>(smem + S::kOffBar + 64);  // [2]
  uint32_t* s_taddr = reinterpret_cast<uint32_t*>(smem + S::kOffBar + 72);
  uint8_t* SL = smem + S::kOffSlot + slot * S::kSlot;
  uint8_t* ROWS = SL + 2 * S::kX;
  float* RED = reinterpret_cast<float*>(smem + S::kOffRed) + slot * (2 * 2 * TM * 4);
  float* BETA = reinterpret_cast<float*>(smem + S::kOffBeta) + slot * 2 * NH;
  for (int e = tid; e < NH * 64; e += kFwdThreads) {
    const int n = e >> 6, k = e & 63;
    const int col = kFold ? fold_col(k) : (k < KIN ? k : -1);
    float h, l;
    tc::split_tf32(col >= 0 ? w.W0[n * KIN + col] : 0.0f, h, l);
    *reinterpret_cast<float*>(W2 + w_off(n, k)) = h;
    *reinterpret_cast<float*>(W2 + w_off(NH + n, k)) = l;
  }
  if (kFold)
    for (int e = tid; e < 16 * NH; e += kFwdThreads) WSH[(e & 15) * NH + (e >> 4)] = w.W0[(e >> 4) * KIN + 32 + (e & 15)];
  for (int i = tid; i < NH; i += kFwdThreads) B0[i] = w.b0[i];
  for (int i = tid; i < NO * NH; i += kFwdThreads) W1s[i] = w.W1[i];
  if (tid < NO) B1[tid] = w.b1[tid];
  if (issuer && lane == 0) {
    tc::mbar_init(bar, 1);
    tc::mbar_init(ready, 8);
    tc::mbar_init(bar_rows, kStrided ? 256 : 1);
    tc::mbar_init(bar_rows + 1, 1);
    s_fail[slot] = 0;
  }
  __syncwarp();
  if (warp == 0) tc::tmem_alloc(s_taddr, 512);
  tc::fence_smem_to_async();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tb = __shfl_sync(0xffffffffu, *s_taddr, 0);
  const uint32_t tcol = tb + 128 * slot;        // Z accumulator (two halves)
  const uint32_t acol = tb + 256 + 128 * slot;  // X_hi: feature f of buffer b in column acol + 64 b + f
  const uint32_t lane_base = (uint32_t)(32 * q) << 16;
  const int64_t ntiles = (P + TM - 1) / TM;
  const int64_t t0 = 2 * (int64_t)blockIdx.x + slot, tstride = 2 * (int64_t)gridDim.x;
  if (issuer) {
    const bool lead = tc::elect_lead();
    const uint64_t dal = tc::sdesc(tc::smem_u32(SL), 2048, 128), db = tc::sdesc(tc::smem_u32(W2), 2048, 128);
    int n_mma = 0, n_rows[2] = {0, 0};
    auto fetch_rows = [&](int64_t t, int buf) {
      if (lead) {
        const int64_t m0 = t * TM;
        const uint32_t bytes = (uint32_t)(P - m0 < TM ? P - m0 : TM) * (uint32_t)(S::kLd * 4);
        tc::mbar_arrive_expect_tx(bar_rows + buf, bytes);
        tc::bulk_g2s(ROWS + buf * S::kRows, X + m0 * S::kLd, bytes, bar_rows + buf);
      }
      ++n_rows[buf];
    };
#pragma unroll
    for (int b = 0; b < S::kBufs; ++b)
      if (!kStrided && t0 + b * tstride < ntiles) fetch_rows(t0 + b * tstride, b);
    int it = 0;
    bool bad = false;
    for (int64_t t = t0; t < ntiles; t += tstride, ++it) {
      bool ok = tc::mbar_wait_unless(ready, it & 1, wait_limit, s_fail + slot);
      // a worker that gave up a wait said so before it arrived: nothing more is issued, so that no barrier has
      // two phases outstanding
      if (__shfl_sync(0xffffffffu, (int)(!ok || s_fail[slot] != 0), 0)) {
        bad = true;
        break;
      }
      tc::fence_after_sync();
      const uint32_t ah = acol + 64 * (it & 1);
      const uint64_t al = dal + (it & 1) * (S::kX / 16);
      // Z = X W0^T: per step of 8 features X_hi [W_hi; W_lo] (N = 128) and X_lo W_hi (N = 64)
#pragma unroll
      for (int ks = 0; ks < S::kKSteps; ++ks) {
        tc::mma_tf32_ts_warp(lead, tcol, ah + 8 * ks, db + ks * 256, kId128, ks > 0);
        tc::mma_tf32_warp(lead, tcol, al + ks * 256, db + ks * 256, kId64, true);
      }
      tc::commit_warp(lead, bar);
      ++n_mma;
      const int64_t tn = t + S::kBufs * tstride;  // the tile's rows have been read
      if (!kStrided && tn < ntiles) fetch_rows(tn, S::kBufs == 2 ? it & 1 : 0);
    }
    if (bad && lane == 0) s_fail[slot] = 1;
    // the workers leave on their own or see the flag; then nothing of this slot may still be in flight
    tc::fence_before_sync();
    __syncthreads();
    if (s_fail[slot] && lane == 0) {
      if (n_mma > 0) tc::mbar_wait(bar, (n_mma - 1) & 1, kDrainLimit);
#pragma unroll
      for (int b = 0; b < 2; ++b)
        if (n_rows[b] > 0) tc::mbar_wait(bar_rows + b, (n_rows[b] - 1) & 1, kDrainLimit);
      report_timeout(g.status);
    }
  } else {
    float dnx = 0.0f, dny = 0.0f, dnz = 0.0f;  // kFold, threads 0..63: a tile's ray direction, a tile ahead
    auto load_dir = [&](int64_t t) {
      if (kFold && stid < NH) {
        const int64_t r = t * TM / src.S;
        dnx = __ldg(src.rays_d + 3 * r);
        dny = __ldg(src.rays_d + 3 * r + 1);
        dnz = __ldg(src.rays_d + 3 * r + 2);
      }
    };
    bool ok = true;  // no wait of this thread has given up
    auto load_rows = [&](int64_t t) {  // kStrided: this thread's part of tile t's rows
      const float* from = X + t * TM * ldx;
      const int nrows = (int)(P - t * TM < TM ? P - t * TM : TM);
      if (xvec) {  // 12 chunks of 16 bytes and three columns (the row may end there)
        constexpr int kCh = KP / 4;
        for (int e = stid; e < nrows * kCh; e += 256) {
          const int r = e / kCh, c = 4 * (e - r * kCh);
          const uint32_t to = tc::smem_u32(ROWS) + (r * KP + c) * 4;
          const float* p = from + r * ldx + c;
          if (c < 48) {
            tc::async16(to, p);
          } else {
#pragma unroll
            for (int k = 0; k < 3; ++k) tc::async4(to + 4 * k, p + k);
          }
        }
      } else {
        int r = stid / KIN, k = stid - r * KIN;
#pragma unroll 4
        for (; r < nrows;) {
          tc::async4(tc::smem_u32(ROWS) + (r * KP + k) * 4, from + r * ldx + k);
          k += 256 % KIN;
          r += 256 / KIN;
          if (k >= KIN) {
            k -= KIN;
            ++r;
          }
        }
      }
      tc::async_arrive(bar_rows);
    };
    auto stage = [&](int64_t t, int i) {  // tile t, number i of this slot: rows -> X_hi / X_lo
      const int buf = i & 1;
      const bool valid = t * TM + m < P;
      ok = tc::mbar_wait(bar_rows + (S::kBufs == 2 ? buf : 0), S::kBufs == 2 ? (i >> 1) & 1 : buf, wait_limit) && ok;
      __syncwarp();
      const float4* rrow = reinterpret_cast<const float4*>(ROWS + (S::kBufs == 2 ? buf : 0) * S::kRows + m * (S::kLd * 4));
      uint8_t* XL = SL + buf * S::kX;
      constexpr int kN = kFold ? 5 : 7;  // chunks of 4 features a thread
      const int c0 = hh ? kN : 0;
      float3 dir = make_float3(0.0f, 0.0f, 0.0f);
      if (!kFold) dir = stage_dir<kCompact>(src, t * TM + m, valid && hh);
      float xh[4 * kN];
#pragma unroll
      for (int j = 0; j < kN; ++j) {
        const int c = c0 + j;
        float4 u = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (kFold) {  // [hash 32 | normal 3 | 0 | 0 x 4]
          if (valid && c < 9) u = rrow[c];
          if (c == 8) u.w = 0.0f;
        } else {  // column 51 zero (the padding column may hold anything), chunk 13 zero
          if (valid && c < 13) u = x_chunk<kCompact>(rrow, hh, j, dir);
          if (c == 12) u.w = 0.0f;
        }
        const float v[4] = {u.x, u.y, u.z, u.w};
        float lo[4];
#pragma unroll
        for (int i4 = 0; i4 < 4; ++i4) tc::split_tf32(v[i4], xh[4 * j + i4], lo[i4]);
        *reinterpret_cast<float4*>(XL + x_off(c, m)) = make_float4(lo[0], lo[1], lo[2], lo[3]);
      }
      __syncwarp();
      // stores aligned to their widths (the column base is a multiple of 64)
      const uint32_t ta = acol + 64 * buf + lane_base + 4 * c0;
      if (kFold && hh == 0) {
        tc::tmem_st16(ta, xh);
        tc::tmem_st4(ta + 16, xh + 16);
      } else if (kFold) {
        tc::tmem_st4(ta, xh);
        tc::tmem_st8(ta + 4, xh + 4);
        tc::tmem_st8(ta + 12, xh + 12);
      } else if (hh == 0) {
        tc::tmem_st16(ta, xh);
        tc::tmem_st8(ta + 16, xh + 16);
        tc::tmem_st4(ta + 24, xh + (kFold ? 0 : 24));
      } else {
        tc::tmem_st4(ta, xh);
        tc::tmem_st16(ta + 4, xh + 4);
        tc::tmem_st8(ta + 20, xh + (kFold ? 0 : 20));
      }
      if (kFold && stid < NH) {  // the tile's hidden bias
        float sh[16];
        sh16(dnx, dny, dnz, sh);
        float b = B0[stid];
#pragma unroll
        for (int k = 0; k < 16; ++k) b = fmaf(WSH[k * NH + stid], sh[k], b);
        BETA[NH * buf + stid] = b;
        if (t + tstride < ntiles) load_dir(t + tstride);
      }
      __syncwarp();
      tc::tmem_wait_st();
    };
    auto tell = [&]() {  // to the issuing warp: what this warp wrote and read is done
      if (!ok) s_fail[slot] = 1;
      tc::fence_smem_to_async();
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(ready);
    };
    if (t0 < ntiles) {
      load_dir(t0);
      if (kStrided) load_rows(t0);
      stage(t0, 0);
      tell();
      slot_sync_or(slot, false);  // the first tile's bias is written, its rows are read
      if (kStrided && t0 + tstride < ntiles) load_rows(t0 + tstride);
    }
    int it = 0;
    for (int64_t t = t0; t < ntiles; t += tstride, ++it) {
      const int par = it & 1;
      const int64_t m0 = t * TM;
      const bool valid = m0 + m < P, more = t + tstride < ntiles;
      if (more) stage(t + tstride, it + 1);
      ok = tc::mbar_wait_unless(bar, par, wait_limit, s_fail + slot) && ok;
      __syncwarp();
      tc::fence_after_sync();
      float z[32];
      tmem_ld_sum32(tcol + lane_base + 32 * hh, z);
      if (more) tell();
      const float* b0 = kFold ? BETA + NH * par : B0;
      const bool colours = !kMask || out.colors;
      float* red = RED + par * (2 * TM * 4);
      uint32_t bits;
      if (colours) {
        float p0, p1, p2;
        bits = colour_partial<kMask>(z, hh, b0, W1s, p0, p1, p2);
        *reinterpret_cast<float4*>(red + (hh * TM + m) * 4) = make_float4(p0, p1, p2, 0.0f);
      } else {
        bits = relu_bits(z, hh, b0);
      }
      if (kMask && valid) out.mask[(m0 + m) * out.ldm + hh] = bits;
      if (slot_sync_or(slot, !ok)) {
        if (stid == 0) s_fail[slot] = 1;
        break;
      }
      if (kStrided && t + 2 * tstride < ntiles) load_rows(t + 2 * tstride);  // the next tile's have been read
      if (valid && colours) {  // hh = 0: colours 0 and 1, hh = 1: colour 2
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int cc = 2 * hh + c;
          if (cc < NO) {
            const float o = (B1[cc] + red[m * 4 + cc]) + red[(TM + m) * 4 + cc];
            out.colors[(m0 + m) * out.ldc + cc] = sigmoidf_ref(o);
          }
        }
      }
    }
    if (kStrided) tc::async_wait_all();
    tc::fence_before_sync();
    __syncthreads();
  }
  tc::fence_before_sync();
  __syncthreads();
  __syncwarp();
  if (warp == 0) tc::tmem_dealloc(tb, 512);
}

}  // namespace vx

#include "mlp_adjoint.cuh"

namespace vx {

// Sum the per-block partials into dW0 (64,51), dW1 (3,64), db0 (64), db1 (3), in a fixed order
// (deterministic): a block of 32 x 8 threads takes 32 consecutive elements; thread (x, y) sums
// the partials of blocks y, y + 8, y + 16, ... in increasing order, and the 8 slice sums are then
// added in slice order. Loads are coalesced along the elements.
constexpr int kReduceSlices = 8;

__global__ void __launch_bounds__(256) k_mlp_wgrad_reduce(const float* __restrict__ partials, int nblocks,
                                                          float* __restrict__ dW0, float* __restrict__ db0,
                                                          float* __restrict__ dW1, float* __restrict__ db1) {
  __shared__ double part[kReduceSlices][32];
  const int e = blockIdx.x * 32 + threadIdx.x;
  double acc = 0.0;
  if (e < WG)
    for (int b = threadIdx.y; b < nblocks; b += kReduceSlices) acc += (double)__ldg(partials + (int64_t)b * WG + e);
  part[threadIdx.y][threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.y != 0 || e >= WG) return;
  double sum = 0.0;
#pragma unroll
  for (int y = 0; y < kReduceSlices; ++y) sum += part[y][threadIdx.x];
  const float v = (float)sum;
  if (e < NH * KP) {
    const int n = e / KP, k = e % KP;
    if (k < KIN) dW0[n * KIN + k] = v;
  } else if (e < NH * KP + NO * NH) {
    dW1[e - NH * KP] = v;
  } else if (e < NH * KP + NO * NH + NH) {
    db0[e - NH * KP - NO * NH] = v;
  } else {
    db1[e - NH * KP - NO * NH - NH] = v;
  }
}

// MLP input rows [hash 32 | SH 16 | normal 3 | 0] of the training forward. A block of 256 threads
// covers 64 consecutive samples: warp w gathers levels 4(w/2)..4(w/2)+3 for the samples
// 32(w%2)..32(w%2)+31, so each gather instruction reads one level for 32 consecutive samples of
// a ray, and neighbouring samples that share a coarse-level cell share its request. Warps of
// level group 0 also evaluate the SH of the view direction, group 1 copies the normal; the rows
// meet in shared memory and leave as one contiguous block (or row by row for a wider stride), evicted first
// from L2, where the 64 MB table is to stay: 1 M samples 229 -> 224 us, a view's 61 M 11.79 -> 11.65 ms. Bound by
// the table's sector requests from L1 to L2, 78% of the rate that random reads reach.
constexpr int kRowsPerBlock = 64;

template <bool kCompact>
__global__ void __launch_bounds__(256) k_hash_rows(HashArgs a) {
  constexpr int kChunks = kCompact ? KC / 4 : 13;  // float4 chunks per row
  __shared__ float4 srow[kRowsPerBlock * kChunks];
  const uint32_t mask = (1u << a.log2T) - 1u;
  const size_t T = (size_t)1 << a.log2T;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = w >> 1;
  const int ls = 32 * (w & 1) + lane;  // this thread's sample in the block
  for (int64_t base = (int64_t)blockIdx.x * kRowsPerBlock; base < a.P; base += (int64_t)gridDim.x * kRowsPerBlock) {
    const int64_t i = base + ls;
    if (i < a.P) {
      float x[3];
      sample_pos(a, i, x);
      float f[8];
#pragma unroll
      for (int qq = 0; qq < 4; ++qq) {
        const int l = 4 * g + qq;
        const float lw = a.lw[l];
        float f0 = 0.0f, f1 = 0.0f;
        if (lw != 0.0f) {
          LevelCell c;
          level_cell(x, a.res[l], mask, c);
          const float2* tab = reinterpret_cast<const float2*>(a.table) + (size_t)l * T;
          gather_level(tab, c, f0, f1);
          if (lw < 1.0f) {
            f0 *= lw;
            f1 *= lw;
          }
        }
        f[2 * qq] = f0;
        f[2 * qq + 1] = f1;
      }
      srow[ls * kChunks + 2 * g] = make_float4(f[0], f[1], f[2], f[3]);
      srow[ls * kChunks + 2 * g + 1] = make_float4(f[4], f[5], f[6], f[7]);
      if (g == 0 && !kCompact) {
        const int64_t r = i / a.S;
        float o[16];
        sh16(__ldg(a.rays_d + 3 * r), __ldg(a.rays_d + 3 * r + 1), __ldg(a.rays_d + 3 * r + 2), o);
#pragma unroll
        for (int c = 0; c < 4; ++c)
          srow[ls * kChunks + 8 + c] = make_float4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
      } else if (g == 1) {
        srow[ls * kChunks + kChunks - 1] = make_float4(a.normals[3 * i], a.normals[3 * i + 1], a.normals[3 * i + 2],
                                                       0.0f);
      }
    }
    __syncthreads();
    const int nrows = (int)(a.P - base < kRowsPerBlock ? a.P - base : kRowsPerBlock);
    if (a.ld == 4 * kChunks) {
      float4* out = reinterpret_cast<float4*>(a.out + base * (4 * kChunks));
      for (int k = tid; k < nrows * kChunks; k += 256) __stcs(out + k, srow[k]);
    } else {
      for (int k = tid; k < nrows * kChunks; k += 256)
        reinterpret_cast<float4*>(a.out + (base + k / kChunks) * a.ld)[k % kChunks] = srow[k];
    }
    __syncthreads();
  }
}

// k_hash_rows over a.P samples, one wave of resident blocks; compact rows when a.ld == KC.
void launch_hash_rows(const HashArgs& a, cudaStream_t st) {
  static int rows_per_sm[2] = {0, 0};
  const bool compact = a.ld == KC;
  auto kern = compact ? k_hash_rows<true> : k_hash_rows<false>;
  if (rows_per_sm[compact] == 0) {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, 256, 0) != cudaSuccess || nb < 1) nb = 4;
    rows_per_sm[compact] = nb;
  }
  kern<<<grid_for((a.P + kRowsPerBlock - 1) / kRowsPerBlock * 256, 256, rows_per_sm[compact]), 256, 0, st>>>(a);
}

// Rows [hash 32 | view 16 | normal 3 | 0] of the modules' separate inputs, 52 floats each, so that the MLP
// kernels take them by bulk copies: a thread per 16-byte chunk. Bound by memory: 200,003 rows 13 us, and 26 us of cat plus 39 us of gradient
// copies are gone.
__global__ void __launch_bounds__(256) k_radiance_rows(const float* __restrict__ hash, const float* __restrict__ view,
                                                       const float* __restrict__ normal, int64_t n, int vec,
                                                       float4* __restrict__ rows) {
  constexpr int kChunks = KP / 4;
  for (int64_t e = blockIdx.x * (int64_t)256 + threadIdx.x; e < n * kChunks; e += (int64_t)gridDim.x * 256) {
    const int64_t r = e / kChunks;
    const int c = (int)(e - r * kChunks);
    float4 v;
    if (c == kChunks - 1) {
      v = make_float4(__ldg(normal + 3 * r), __ldg(normal + 3 * r + 1), __ldg(normal + 3 * r + 2), 0.0f);
    } else {
      const float* p = c < 8 ? hash + 32 * r + 4 * c : view + 16 * r + 4 * (c - 8);
      v = vec ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
    }
    rows[e] = v;
  }
}

template <bool kCustomWait, bool kMask>
auto rows2_kernel(FwdRows rows) {
  return rows == kFwdFold      ? k_mlp_fwd_rows2<kCustomWait, kFwdFold, kMask>
         : rows == kFwdCompact ? k_mlp_fwd_rows2<kCustomWait, kFwdCompact, kMask>
         : rows == kFwdFull    ? k_mlp_fwd_rows2<kCustomWait, kFwdFull, kMask>
                               : k_mlp_fwd_rows2<kCustomWait, kFwdStrided, kMask>;
}

// The forward on rows X (row stride ldx, or compact rows when src.rays_d is given).
int launch_fwd(const float* X, int64_t ldx, int64_t P, const MlpW& w, const MlpOut& out, cudaStream_t st,
               RowSrc src = RowSrc{nullptr, 0}) {
  const bool aligned = (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  // folded: compact rows whose tiles each lie inside one ray (samples per ray a multiple of the tile)
  const FwdRows rows = src.rays_d ? (src.S % TM == 0 ? kFwdFold : kFwdCompact)
                                  : (ldx == KP && aligned ? kFwdFull : kFwdStrided);
  const bool cw = custom_wait();
  auto kern = out.mask ? (cw ? rows2_kernel<true, true>(rows) : rows2_kernel<false, true>(rows))
                       : (cw ? rows2_kernel<true, false>(rows) : rows2_kernel<false, false>(rows));
  const int smem = rows == kFwdFold      ? (int)FwdShape<true, true>::kSmem
                   : rows == kFwdCompact ? (int)FwdShape<true, false>::kSmem
                                         : (int)FwdShape<false, false>::kSmem;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return set_error(VX_ERR_CUDA, "mlp forward: %s", cudaGetErrorString(e));
  const int64_t pairs = ((P + TM - 1) / TM + 1) / 2;
  const unsigned blocks = (unsigned)(pairs < (int64_t)kSMs ? pairs : (int64_t)kSMs);
  kern<<<blocks, kFwdThreads, smem, st>>>(X, ldx, ldx % 4 == 0 && aligned, P, w, out, t_guard, src);
  return VX_OK;
}

// The forward from the hash table and the ray, nothing but the colours written (inference of a C caller without rows).
int launch_fwd_hash(const HashArgs& a, int64_t P, const MlpW& w, const MlpOut& out, cudaStream_t st) {
  const int64_t tiles = (P + TM - 1) / TM;
  auto kern = custom_wait() ? k_mlp_fwd_tc<true> : k_mlp_fwd_tc<false>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwdSmem);
  if (e != cudaSuccess) return set_error(VX_ERR_CUDA, "mlp forward: %s", cudaGetErrorString(e));
  const unsigned blocks = (unsigned)(tiles < (int64_t)kSMs * 2 ? tiles : (int64_t)kSMs * 2);
  kern<<<blocks, 256, kFwdSmem, st>>>(a, P, w, out, t_guard);
  return VX_OK;
}

template <int kMode>
int launch_adjoint(const float* x, int64_t ldx, int64_t P, const MlpW& w, const float* d_colors, const float* y,
                   int64_t ldy, const uint32_t* mask, int64_t ldm, float* d_hash, float* d_normal, float* partials,
                   int blocks, cudaStream_t st, RowSrc src, const char* what) {
  constexpr int smem = (int)AdjShape<kMode>::kSmem;
  auto kern = custom_wait() ? k_mlp_adjoint<kMode, true> : k_mlp_adjoint<kMode, false>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return set_error(VX_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  kern<<<blocks, kAdjThreads, smem, st>>>(x, ldx, P, w, d_colors, y, ldy, mask, ldm, d_hash, d_normal, partials,
                                          t_guard, src);
  return VX_OK;
}

// The adjoint and its weight-gradient reduction. Full rows (src.rays_d == nullptr, any stride
// >= 51: 52-float contiguous rows arrive by bulk copies) or compact rows (bulk copies only; folded
// when the samples of a ray fill whole tiles, as in the forward). A caller without the forward's
// mask (or colours) gets them from a forward launch that leaves them in d_hash's rows (words 0..1
// and floats 2..4 of each), which the adjoint reads before it writes them.
int mlp_backward_launch(const float* x, int64_t ldx, int64_t n_points, const float* W0, const float* b0,
                        const float* W1, const float* b1, const float* d_colors, const float* colors,
                        const uint32_t* mask, float* d_hash, float* d_normal, float* dW0, float* db0, float* dW1,
                        float* db1, float* partials, int64_t n_partial_floats, cudaStream_t st, RowSrc src,
                        const char* what) {
  VX_REQUIRE(x && W0 && b0 && W1 && b1 && d_colors && d_hash && d_normal && dW0 && db0 && dW1 && db1 && partials,
             "null pointer");
  VX_REQUIRE((reinterpret_cast<uintptr_t>(d_hash) & 15) == 0, "d_hash must be 16-byte aligned");
  const int nb = vx_mlp_blocks(n_points);
  VX_REQUIRE(n_partial_floats >= (int64_t)nb * WG, "partials buffer holds %lld floats, need %lld",
             (long long)n_partial_floats, (long long)nb * WG);
  MlpW w{W0, b0, W1, b1};
  const bool compact = src.rays_d != nullptr;
  int launches = 1;
  if (n_points > 0) {
    const float* y = colors;
    int64_t ldy = NO, ldm = 2;
    if (!mask || !colors) {
      uint32_t* dm = reinterpret_cast<uint32_t*>(d_hash);
      if (int s = launch_fwd(x, ldx, n_points, w, MlpOut{colors ? nullptr : d_hash + 2, 32, dm, 32}, st, src)) return s;
      mask = dm;
      ldm = 32;
      if (!colors) {
        y = d_hash + 2;
        ldy = 32;
      }
      ++launches;
    }
    const bool bulk = ldx == KP && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    // folded: whole tiles, each inside one ray, whose d_colors, colours and mask rows are bulk copies too
    const bool fold = compact && src.S % TM == 0 && n_points % TM == 0 && ldy == NO && ldm == 2 &&
                      ((reinterpret_cast<uintptr_t>(d_colors) | reinterpret_cast<uintptr_t>(y) |
                        reinterpret_cast<uintptr_t>(mask)) & 15) == 0;
    auto go = compact ? (fold ? launch_adjoint<kAdjFold> : launch_adjoint<kAdjCompact>)
                      : (bulk ? launch_adjoint<kAdjFull> : launch_adjoint<kAdjStrided>);
    if (int s = go(x, ldx, n_points, w, d_colors, y, ldy, mask, ldm, d_hash, d_normal, partials, nb, st, src, what))
      return s;
    ++launches;
  } else {
    cudaMemsetAsync(partials, 0, sizeof(float) * WG, st);
  }
  k_mlp_wgrad_reduce<<<(WG + 31) / 32, dim3(32, kReduceSlices), 0, st>>>(partials, n_points > 0 ? nb : 1, dW0, db0,
                                                                        dW1, db1);
  count_launches(launches);
  return check_launch(what);
}

}  // namespace vx

using namespace vx;

static int appearance_forward(const float* table, int n_levels, int log2_size, int n_features,
                              const int32_t* level_res, const float* level_weights, const float* rays_o,
                              const float* rays_d, const float* mid, int n_samples, const float xyz_min[3],
                              const float xyz_max[3], int64_t n_points, const float* normals, const float* W0,
                              const float* b0, const float* W1, const float* b1, float* colors, float* rows,
                              int64_t ld_rows, uint32_t* mask, void* stream) {
  HashArgs a{};
  if (int s = fill_hash(a, table, n_levels, log2_size, n_features, level_res, level_weights)) return s;
  VX_REQUIRE(n_levels == 16, "the fused appearance MLP takes 16 hash levels x 2 features (got %d)", n_levels);
  VX_REQUIRE(n_points >= 0 && n_samples >= 1, "bad sizes");
  if (n_points == 0) return VX_OK;
  VX_REQUIRE(table && rays_o && rays_d && mid && xyz_min && xyz_max && normals && W0 && b0 && W1 && b1 && colors,
             "null pointer");
  VX_REQUIRE(!rows || ((ld_rows == KC || ld_rows >= KP) && ld_rows % 4 == 0 && ((uintptr_t)rows & 15) == 0),
             "rows need a row stride of 36 floats (compact) or >= 52, a multiple of 4, and 16-byte alignment");
  VX_REQUIRE(!rows || ld_rows != KC || n_points < (int64_t(1) << 32), "compact rows take fewer than 2^32 samples");
  fill_positions(a, nullptr, rays_o, rays_d, mid, n_samples, xyz_min, xyz_max);
  a.P = n_points;
  a.out = rows;
  a.ld = ld_rows;
  a.normals = normals;
  MlpW w{W0, b0, W1, b1};
  const MlpOut out{colors, NO, mask, 2};
  cudaStream_t st = (cudaStream_t)stream;
  if (rows) {  // training: rows gathered at high occupancy, then the MLP on the rows
    launch_hash_rows(a, st);
    const RowSrc src{ld_rows == KC ? rays_d : nullptr, n_samples};
    if (int s = launch_fwd(rows, ld_rows, n_points, w, out, st, src)) return s;
    count_launches(2);
  } else {  // inference: features built in shared memory, nothing else written
    if (int s = launch_fwd_hash(a, n_points, w, out, st)) return s;
    count_launches(1);
  }
  return check_launch("appearance_mlp_forward");
}

static int radiance_forward(const float* x, int64_t ldx, int64_t n_points, const float* W0, const float* b0,
                            const float* W1, const float* b1, float* colors, uint32_t* mask, void* stream) {
  MlpW w{W0, b0, W1, b1};
  if (int s = launch_fwd(x, ldx, n_points, w, MlpOut{colors, NO, mask, 2}, (cudaStream_t)stream)) return s;
  count_launches(1);
  return check_launch("radiance_mlp_forward");
}

extern "C" {

int vx_appearance_mlp_forward(const float* table, int n_levels, int log2_size, int n_features,
                              const int32_t* level_res, const float* level_weights, const float* rays_o,
                              const float* rays_d, const float* mid, int n_samples, const float xyz_min[3],
                              const float xyz_max[3], int64_t n_points, const float* normals, const float* W0,
                              const float* b0, const float* W1, const float* b1, float* colors, float* rows,
                              int64_t ld_rows, void* stream) {
  return appearance_forward(table, n_levels, log2_size, n_features, level_res, level_weights, rays_o, rays_d, mid,
                            n_samples, xyz_min, xyz_max, n_points, normals, W0, b0, W1, b1, colors, rows, ld_rows,
                            nullptr, stream);
}

int vx_appearance_mlp_forward_masked(const float* table, int n_levels, int log2_size, int n_features,
                                     const int32_t* level_res, const float* level_weights, const float* rays_o,
                                     const float* rays_d, const float* mid, int n_samples, const float xyz_min[3],
                                     const float xyz_max[3], int64_t n_points, const float* normals, const float* W0,
                                     const float* b0, const float* W1, const float* b1, float* colors, float* rows,
                                     int64_t ld_rows, uint32_t* relu_mask, void* stream) {
  VX_REQUIRE(n_points <= 0 || (rows && relu_mask), "null pointer");
  return appearance_forward(table, n_levels, log2_size, n_features, level_res, level_weights, rays_o, rays_d, mid,
                            n_samples, xyz_min, xyz_max, n_points, normals, W0, b0, W1, b1, colors, rows, ld_rows,
                            relu_mask, stream);
}

int vx_appearance_mlp_forward_chunked(const float* table, int n_levels, int log2_size, int n_features,
                                      const int32_t* level_res, const float* level_weights, const float* rays_o,
                                      const float* rays_d, const float* mid, int n_samples, const float xyz_min[3],
                                      const float xyz_max[3], int64_t n_points, const float* normals,
                                      const float* W0, const float* b0, const float* W1, const float* b1,
                                      float* colors, float* scratch_rows, int64_t scratch_count, void* stream) {
  HashArgs a{};
  if (int s = fill_hash(a, table, n_levels, log2_size, n_features, level_res, level_weights)) return s;
  VX_REQUIRE(n_levels == 16, "the fused appearance MLP takes 16 hash levels x 2 features (got %d)", n_levels);
  VX_REQUIRE(n_points >= 0 && n_samples >= 1, "bad sizes");
  VX_REQUIRE(n_points % n_samples == 0, "n_points must be whole rays (a multiple of n_samples)");
  if (n_points == 0) return VX_OK;
  VX_REQUIRE(table && rays_o && rays_d && mid && xyz_min && xyz_max && normals && W0 && b0 && W1 && b1 && colors &&
                 scratch_rows,
             "null pointer");
  VX_REQUIRE(((uintptr_t)scratch_rows & 15) == 0, "scratch rows must be 16-byte aligned");
  VX_REQUIRE(scratch_count >= n_samples, "scratch holds %lld rows, fewer than one ray's %d samples",
             (long long)scratch_count, n_samples);
  VX_REQUIRE(scratch_count < (int64_t(1) << 32), "the scratch takes fewer than 2^32 rows");
  fill_positions(a, nullptr, rays_o, rays_d, mid, n_samples, xyz_min, xyz_max);
  a.ld = KC;  // compact rows: SH(d) is recomputed from rays_d by the MLP kernel
  a.out = scratch_rows;
  MlpW w{W0, b0, W1, b1};
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t chunk = (scratch_count / n_samples) * n_samples;  // whole rays per pass
  int launches = 0;
  for (int64_t c0 = 0; c0 < n_points; c0 += chunk) {
    const int64_t len = n_points - c0 < chunk ? n_points - c0 : chunk;
    HashArgs ac = a;
    const int64_t r0 = c0 / n_samples;
    ac.rays_o = rays_o + 3 * r0;
    ac.rays_d = rays_d + 3 * r0;
    ac.mid = mid + c0;
    ac.normals = normals + 3 * c0;
    ac.P = len;
    launch_hash_rows(ac, st);
    if (int s = launch_fwd(scratch_rows, KC, len, w, MlpOut{colors + 3 * c0, NO, nullptr, 0}, st,
                           RowSrc{ac.rays_d, n_samples}))
      return s;
    launches += 2;
  }
  count_launches(launches);
  return check_launch("appearance_mlp_forward_chunked");
}

int vx_mlp_blocks(int64_t n_points) {
  const int64_t tiles = (n_points + TM - 1) / TM;
  const int64_t cap = (int64_t)kSMs;
  return (int)(tiles < 1 ? 1 : (tiles < cap ? tiles : cap));
}

int vx_mlp_partial_floats(void) { return WG; }

int vx_tc_guard(int* status, int64_t wait_polls) {
  VX_REQUIRE(wait_polls <= (int64_t)UINT32_MAX, "wait_polls above 2^32 - 1");
  t_guard.status = status;
  t_guard.limit = wait_polls < 0 ? kWaitLimit : (uint32_t)wait_polls;
  return VX_OK;
}

int vx_tensor_core_timeouts(void) {
  int h = 0;
  const int zero = 0;
  if (cudaMemcpyFromSymbol(&h, g_tc_timeouts, sizeof(int)) != cudaSuccess) return -1;
  if (cudaMemcpyToSymbol(g_tc_timeouts, &zero, sizeof(int)) != cudaSuccess) return -1;
  return h;
}

int vx_radiance_rows(const float* hash, const float* view, const float* normal, int64_t n_points, float* rows,
                     void* stream) {
  VX_REQUIRE(n_points >= 0, "bad sizes");
  if (n_points == 0) return VX_OK;
  VX_REQUIRE(hash && view && normal && rows, "null pointer");
  VX_REQUIRE((reinterpret_cast<uintptr_t>(rows) & 15) == 0, "rows must be 16-byte aligned");
  const int vec = ((reinterpret_cast<uintptr_t>(hash) | reinterpret_cast<uintptr_t>(view)) & 15) == 0;
  k_radiance_rows<<<grid_for(n_points * (KP / 4), 256, 32), 256, 0, (cudaStream_t)stream>>>(
      hash, view, normal, n_points, vec, reinterpret_cast<float4*>(rows));
  count_launches(1);
  return check_launch("radiance_rows");
}

int vx_radiance_mlp_forward(const float* x, int64_t ldx, int64_t n_points, int in_dim, int hidden, int out_dim,
                            const float* W0, const float* b0, const float* W1, const float* b1, float* colors,
                            void* stream) {
  VX_REQUIRE(in_dim == KIN && hidden == NH && out_dim == NO, "the fused MLP is %d -> %d -> %d (got %d -> %d -> %d)",
             KIN, NH, NO, in_dim, hidden, out_dim);
  VX_REQUIRE(n_points >= 0 && ldx >= KIN, "bad sizes");
  if (n_points == 0) return VX_OK;
  VX_REQUIRE(x && W0 && b0 && W1 && b1 && colors, "null pointer");
  return radiance_forward(x, ldx, n_points, W0, b0, W1, b1, colors, nullptr, stream);
}

int vx_radiance_mlp_forward_masked(const float* x, int64_t ldx, int64_t n_points, int in_dim, int hidden, int out_dim,
                                   const float* W0, const float* b0, const float* W1, const float* b1, float* colors,
                                   uint32_t* relu_mask, void* stream) {
  VX_REQUIRE(in_dim == KIN && hidden == NH && out_dim == NO, "the fused MLP is %d -> %d -> %d (got %d -> %d -> %d)",
             KIN, NH, NO, in_dim, hidden, out_dim);
  VX_REQUIRE(n_points >= 0 && ldx >= KIN, "bad sizes");
  if (n_points == 0) return VX_OK;
  VX_REQUIRE(x && W0 && b0 && W1 && b1 && colors && relu_mask, "null pointer");
  return radiance_forward(x, ldx, n_points, W0, b0, W1, b1, colors, relu_mask, stream);
}

int vx_radiance_mlp_backward(const float* x, int64_t ldx, int64_t n_points, int in_dim, int hidden, int out_dim,
                             const float* W0, const float* b0, const float* W1, const float* b1, const float* d_colors,
                             const float* colors, float* d_hash, float* d_normal, float* dW0, float* db0, float* dW1,
                             float* db1, float* partials, int64_t n_partial_floats, void* stream) {
  return vx_radiance_mlp_backward_masked(x, ldx, n_points, in_dim, hidden, out_dim, W0, b0, W1, b1, d_colors, colors,
                                         nullptr, d_hash, d_normal, dW0, db0, dW1, db1, partials, n_partial_floats,
                                         stream);
}

int vx_radiance_mlp_backward_masked(const float* x, int64_t ldx, int64_t n_points, int in_dim, int hidden, int out_dim,
                                    const float* W0, const float* b0, const float* W1, const float* b1,
                                    const float* d_colors, const float* colors, const uint32_t* relu_mask,
                                    float* d_hash, float* d_normal, float* dW0, float* db0, float* dW1, float* db1,
                                    float* partials, int64_t n_partial_floats, void* stream) {
  VX_REQUIRE(in_dim == KIN && hidden == NH && out_dim == NO, "the fused MLP is %d -> %d -> %d", KIN, NH, NO);
  VX_REQUIRE(n_points >= 0 && ldx >= KIN, "bad sizes");
  return mlp_backward_launch(x, ldx, n_points, W0, b0, W1, b1, d_colors, colors, relu_mask, d_hash, d_normal, dW0, db0,
                             dW1, db1, partials, n_partial_floats, (cudaStream_t)stream, RowSrc{nullptr, 0},
                             "radiance_mlp_backward");
}

int vx_appearance_mlp_backward(const float* rows, const float* rays_d, int n_samples, int64_t n_points,
                               const float* W0, const float* b0, const float* W1, const float* b1,
                               const float* d_colors, const float* colors, float* d_hash, float* d_normal, float* dW0,
                               float* db0, float* dW1, float* db1, float* partials, int64_t n_partial_floats,
                               void* stream) {
  return vx_appearance_mlp_backward_masked(rows, rays_d, n_samples, n_points, W0, b0, W1, b1, d_colors, colors, nullptr,
                                           d_hash, d_normal, dW0, db0, dW1, db1, partials, n_partial_floats, stream);
}

int vx_appearance_mlp_backward_masked(const float* rows, const float* rays_d, int n_samples, int64_t n_points,
                                      const float* W0, const float* b0, const float* W1, const float* b1,
                                      const float* d_colors, const float* colors, const uint32_t* relu_mask,
                                      float* d_hash, float* d_normal, float* dW0, float* db0, float* dW1, float* db1,
                                      float* partials, int64_t n_partial_floats, void* stream) {
  VX_REQUIRE(n_points >= 0 && n_samples >= 1, "bad sizes");
  VX_REQUIRE(rays_d && rows, "null pointer");
  VX_REQUIRE(((uintptr_t)rows & 15) == 0, "compact rows must be 16-byte aligned");
  VX_REQUIRE(n_points < (int64_t(1) << 32), "compact rows take fewer than 2^32 samples");
  return mlp_backward_launch(rows, KC, n_points, W0, b0, W1, b1, d_colors, colors, relu_mask, d_hash, d_normal, dW0,
                             db0, dW1, db1, partials, n_partial_floats, (cudaStream_t)stream,
                             RowSrc{rays_d, n_samples}, "appearance_mlp_backward");
}

}  // extern "C"
