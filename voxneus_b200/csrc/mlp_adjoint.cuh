// Adjoint of the radiance MLP [hash 32 | SH 16 | normal 3] -> 64 ReLU -> 3 Sigmoid on the tensor
// cores (tcgen05, kind::f16 on bf16 parts, f32 accumulators in TMEM). Included by mlp.cu.
//
// With m[s,n] = 1 where hidden unit n of sample s is active (kept by the forward, one bit each) and
// d[s,c] = dL/d(pre-sigmoid colour c), the ReLU makes the hidden layer linear in m, and both
// contractions of the adjoint have the 0/1 matrix m as one operand, which a bf16 holds exactly:
//   dX[s,k]  = sum_c d[s,c] (m V_c)[s,k],  V_c[n,k] = W1[c,n] W0[n,k] (a constant of the launch)
//   G_c[n,k] = sum_s m[s,n] (d[s,c] x[s,k]), with x's last feature 1
//   dW0[n,k] = sum_c W1[c,n] G_c[n,k],  db0 the same of the ones column
//   dW1[c,n] = sum_k W0[n,k] G_c[n,k] + b0[n] G_c[n,ones]   (relu(z) = m (W0 x + b0))
// so the hidden layer is not recomputed, no 64-wide dL/dz is split or transposed, and the other
// operand needs three bf16 parts only: a float32's 24 bits cut into 8 + 8 + 8 (cut3), which
// is exact, where a tf32 hi + lo pair carries 22 of them.
//
// A product with the mask is no selection: 0 times an infinity or a NaN is a NaN, and d x overflows where d W1 x does
// not. So a sample of which no unit is active takes part with d = 0, and a block whose sums are not finite
// forms them again on the CUDA cores, selecting (adj_plain_sums): units that such a sample leaves inactive keep
// their gradients, as ReLU's adjoint has it.
//
// Layouts (no swizzle, 16-byte units; tc.cuh). The operands of G are written once, sample by sample,
// and read with their sample index as the contraction: kind::f16 takes MN-major operands.
//   A (G)    row r = c * stride + k of the 3 x features matrix, element (r, s) at
//            (r/8)*2048 + s*16 + (r%8)*2: a thread's 8 rows are one 16-byte store, a warp's
//            consecutive samples consecutive (no bank conflicts)
//   M        element (s, n) at (n/8)*2048 + s*16 + (n%8)*2: MN-major B of G, K-major A of dX
//   V        column j (hash feature k of colour c: 32 c + k; normal: 96 + 4 c + k), element (j, n)
//            at (n/8)*1792 + (j/8)*128 + (j%8)*16 + (n%8)*2: K-major B of dX
// G runs as M = 128 (the 108 rows; two overlapping row ranges for the 156 rows of the unfolded
// form) x N = 64 x K = 128 samples, dX as 128 samples x N = 112 x K = 64, three parts each into one
// accumulator.
//
// A persistent CTA per SM: 512 worker threads, thread (s, hh) forming features 8 hh .. of all colours for
// sample s, and one warp that issues the MMAs and the bulk copies (issuing blocks while the tensor core's
// queue is full). The queue is G(t), dX(t+1), G(t+1), ...: dX(t+1) runs while A(t+1) is staged; dX(t) and
// G(t-1) are read out and the next mask staged while G(t) runs. d_hash leaves through shared memory in
// whole lines: written from the TMEM lanes (32 rows an instruction) it held the load/store unit for
// longer than G takes.
//
// What bounds it: the shared-memory port. A tile writes and reads A once (92 KB each way), reads V (43 KB)
// and M (48 KB), about 2,100 cycles at 128 bytes a cycle, and staging A and running G alternate on the
// one A buffer that fits: ~4,200 cycles a tile. 1,048,576 samples: 317 us (the adjoint that recomputed the
// hidden layer and split dL/dz) -> 137 us; 262,144 samples: 90 -> 40 us; 200,003 contiguous rows: 92 -> 53 us.
// Tried: 24 bf16 products held in registers over the tile boundary (spills in a 96-register budget,
// 218 us); the G sums left in tensor memory (its truncated additions put 3e-6 of error in dW1, against
// 2.5e-7); the MMAs issued by a branch of one thread (163 us).
#pragma once

namespace vx {

enum AdjRows { kAdjFold = 0, kAdjCompact = 1, kAdjFull = 2, kAdjStrided = 3 };

constexpr int kAdjWork = 512;               // worker threads; one more warp issues the MMAs and copies
constexpr int kAdjThreads = kAdjWork + 32;
constexpr uint32_t kAdjChunk = TM * 16;          // 8 rows x 128 samples of bf16
constexpr uint32_t kAdjMask = 8 * kAdjChunk;     // 64 hidden units
constexpr int kVCols = 112;                      // 96 hash + 12 normal columns, padded to a multiple of 16
constexpr uint32_t kVChunk = kVCols * 16;
constexpr uint32_t kVPart = 8 * kVChunk;

constexpr uint32_t kAdjAux = TM * (NO + NO + 2) * 4;

template <int kMode>
struct AdjShape {
  static constexpr bool kFold = kMode == kAdjFold;
  static constexpr bool kCompact = kMode == kAdjFold || kMode == kAdjCompact;
  static constexpr bool kBulk = kMode != kAdjStrided;
  static constexpr int kStride = kFold ? 40 : KP;  // rows of A per colour (the last 4 of 40 are zero)
  static constexpr int kChunks = (3 * kStride + 7) / 8;
  static constexpr int kRow2 = kChunks * 8 - TM;   // first row of the second G range (unfolded)
  static constexpr int kLd = kCompact ? KC : KP;   // floats per row in shared memory
  static constexpr int kBufs = kFold ? 2 : 1;      // row buffers
  static constexpr uint32_t kPart = kChunks * kAdjChunk;
  static constexpr uint32_t kOffMask = 3 * kPart;
  static constexpr uint32_t kOffV = kOffMask + 2 * kAdjMask;
  static constexpr uint32_t kOffRows = kOffV + 3 * kVPart;
  static constexpr uint32_t kRowBytes = kLd * 4;
  static constexpr uint32_t kOffCur = kOffRows + kBufs * TM * kRowBytes;  // folded: ones rows of G [2][3][64]
  static constexpr uint32_t kOffSh = kOffCur + (kFold ? 2 * 3 * NH * 4 : 0);
  static constexpr uint32_t kOffAux = kOffSh + (kFold ? 4 * 16 * 4 : 0);  // folded: [2] d_out, y, mask of a tile
  static constexpr uint32_t kOffH = kOffAux + (kFold ? 2 * kAdjAux : 0);  // folded: d_hash of a tile
  static constexpr uint32_t kOffBar = kOffH + (kFold ? TM * 32 * 4 : 0);
  static constexpr uint32_t kSmem = kOffBar + 48;
};
static_assert(AdjShape<kAdjFold>::kSmem <= 227 * 1024 && AdjShape<kAdjCompact>::kSmem <= 227 * 1024 &&
                  AdjShape<kAdjFull>::kSmem <= 227 * 1024,
              "the adjoint's shared memory exceeds a CTA's");
// one CTA per SM: two would contend for TMEM with their staging out of step
static_assert(AdjShape<kAdjFold>::kSmem > 116 * 1024, "two adjoint CTAs would fit on an SM");
// G's M = 128 descriptors read whole chunks: the folded form's 16th chunk of the last part lies in
// the mask buffer that follows (its rows 120..127 of G are not used)
static_assert(AdjShape<kAdjFold>::kChunks == 15 && AdjShape<kAdjFull>::kChunks == 20, "A layout");
static_assert(AdjShape<kAdjFull>::kRow2 == 32, "the second row range starts on a chunk");
static_assert(AdjShape<kAdjFold>::kOffBar % 8 == 0 && AdjShape<kAdjFull>::kOffBar % 8 == 0 &&
                  AdjShape<kAdjCompact>::kOffBar % 8 == 0 && AdjShape<kAdjFold>::kOffCur % 16 == 0 &&
                  AdjShape<kAdjFold>::kOffRows % 128 == 0 && AdjShape<kAdjFull>::kOffRows % 128 == 0,
              "shared-memory alignment");

// tensor-memory columns: G of even tiles (two row ranges of 64 columns), dX, M as dX's A operand, G of
// odd tiles (a tile's G is read out while the next one's runs)
constexpr uint32_t kAdjDx = 128, kAdjMk = 256, kAdjG1 = 384;
constexpr uint32_t kIdG = tc::idesc_bf16(TM, NH, true, true);
constexpr uint32_t kIdDx = tc::idesc_bf16(TM, kVCols, false, false);

__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// Four float32 into their three bf16 parts, packed in pairs. A remainder after a rounded part has at
// most 16 (then 8) significant bits, so the three parts sum to the value exactly. (Conversions in
// pairs: five ALU instructions a pair; cutting by masks and byte permutes takes seven.)
__device__ __forceinline__ void cut3(const float v[4], uint32_t h[2], uint32_t m[2], uint32_t l[2]) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float a = v[2 * i], b = v[2 * i + 1];
    h[i] = bf16x2(a, b);
    const float ra = a - __uint_as_float(h[i] << 16), rb = b - __uint_as_float(h[i] & 0xffff0000u);
    m[i] = bf16x2(ra, rb);
    l[i] = bf16x2(ra - __uint_as_float(m[i] << 16), rb - __uint_as_float(m[i] & 0xffff0000u));
  }
}

// 16 mask bits of a sample (hidden units 16 hh ..) as bf16 0/1: two chunks of M in shared memory, and the
// same pairs as eight columns of M in tensor memory (the A operand of dX).
__device__ __forceinline__ void stage_mask(uint8_t* M, uint32_t taddr, int m, int hh, uint32_t bits) {
  float o[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t t = bits >> (2 * i);
    o[i] = __uint_as_float(((t & 1u) | ((t & 2u) << 15)) * 0x3f80u);
  }
  tc::tmem_st8(taddr, o);
#pragma unroll
  for (int f = 0; f < 2; ++f)
    *reinterpret_cast<float4*>(M + (2 * hh + f) * kAdjChunk + m * 16) =
        make_float4(o[4 * f], o[4 * f + 1], o[4 * f + 2], o[4 * f + 3]);
  tc::tmem_wait_st();
}

constexpr int kAdjShTid = 5;  // the worker that evaluates SH(d) of a tile's ray

// Named barriers: 1 once a tile's A is staged (the workers go on, the issuing warp waits), 2 at the end
// of a tile, which also agrees on whether any thread gave up a wait. They, and the tensor-memory loads and stores, are
// instructions of a converged warp: __syncwarp() first wherever lanes can have parted before (polls that
// end at different times, a branch of some lanes), because nothing else makes them meet again.
__device__ __forceinline__ void adj_staged_arrive() {
  asm volatile("bar.arrive 1, %0;" ::"n"(kAdjThreads) : "memory");
}
__device__ __forceinline__ void adj_staged_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kAdjThreads) : "memory");
}
__device__ __forceinline__ void adj_workers_sync() {
  __syncwarp();
  asm volatile("bar.sync 3, %0;" ::"n"(kAdjWork) : "memory");
}
__device__ __forceinline__ bool adj_sync_or(bool v) {
  uint32_t r;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 2, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"(v ? 1u : 0u), "n"(kAdjThreads)
      : "memory");
  return r != 0;
}

// The weight gradients of this block's tiles in plain float32, for blocks in which the products above leave the finite
// range: dz = active ? sum_c d_c W1[c] : 0, dW0 = dz^T x, db0 = sum dz, dW1 = d^T h, db1 = sum d, in the layout of
// pb. y and mask are formed again where the caller's launch kept them in d_hash's rows (row strides of 32), which
// are overwritten by now. By the whole block; sm: its shared memory. 16 warps: z with four samples a warp at a time, two
// hidden units a lane; the sums with thread (n, kg) holding hidden unit n, features 8 kg .. (1,048,576 samples: 1,180 us
// in all where a block or all blocks do this, 138 us where none does).
template <int kMode>
__device__ __noinline__ void adj_plain_sums(float* sm, const float* X, int64_t ldx, int64_t P, MlpW w, const float* d_out,
                                            const float* y, int64_t ldy, const uint32_t* mask, int64_t ldm, float* pb,
                                            RowSrc src) {
  using S = AdjShape<kMode>;
  constexpr int kXp = 60, kZp = 65, kWp = 53;  // pitches
  constexpr int kPer = 8, kGroups = 7;         // features a thread, thread groups with features (the last forms dW1, db1)
  float* XS = sm;                              // x [128][kXp], feature 51 the one of db0, 0 from there on
  float* WS = XS + TM * kXp;                   // W0 [64][kWp], 0 from feature 51 on
  float* DZ = WS + NH * kWp;                   // [128][kZp]
  float* HS = DZ + TM * kZp;                   // relu(z) [128][kZp]
  float* DS = HS + TM * kZp;                   // d [128][3]
  uint32_t* MS = reinterpret_cast<uint32_t*>(DS + TM * NO);  // mask [128][2]
  static_assert((TM * (kXp + 2 * kZp + NO + 2) + NH * kWp) * 4 <= 200 * 1024, "the block's shared memory");
  static_assert(kGroups * kPer >= KP && kGroups * kPer <= kXp && (kGroups + 1) * NH == kAdjWork, "the threads' features");
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, n = tid & (NH - 1), kg = tid / NH;
  for (int e = tid; e < NH * kWp; e += kAdjThreads) WS[e] = e % kWp < KIN ? w.W0[e / kWp * KIN + e % kWp] : 0.0f;
  float acc[kPer], acc1[NO];
#pragma unroll
  for (int j = 0; j < kPer; ++j) acc[j] = 0.0f;
#pragma unroll
  for (int c = 0; c < NO; ++c) acc1[c] = 0.0f;
  const int64_t ntiles = (P + TM - 1) / TM;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    __syncthreads();  // the previous tile's values are read
    const int64_t r0 = t * TM;
    const int nrows = (int)(P - r0 < TM ? P - r0 : TM);
    for (int e = tid; e < TM * KIN; e += kAdjThreads) {
      const int r = e / KIN, k = e - r * KIN;
      if (S::kCompact && k >= 32 && k < 48) continue;
      XS[r * kXp + k] = r >= nrows ? 0.0f : S::kCompact ? X[(r0 + r) * KC + (k < 32 ? k : k - 16)] : X[(r0 + r) * ldx + k];
    }
    for (int e = tid; e < TM * NO; e += kAdjThreads) {
      const bool in = e < nrows * NO;
      const float v = in && ldy == NO ? y[r0 * NO + e] : 0.0f;
      DS[e] = in ? d_out[r0 * NO + e] * (ldy == NO ? (1.0f - v) * v : 1.0f) : 0.0f;
      if (e < TM * 2) MS[e] = ldm == 2 && e < nrows * 2 ? mask[r0 * 2 + e] : 0u;
    }
    if (tid < TM) {
      for (int k = KIN; k < kXp; ++k) XS[tid * kXp + k] = k == KIN && tid < nrows ? 1.0f : 0.0f;
      if (S::kCompact) {
        float sh[16];
        const float* dir = src.rays_d + 3 * ((r0 + (tid < nrows ? tid : nrows - 1)) / src.S);
        sh16(dir[0], dir[1], dir[2], sh);
#pragma unroll
        for (int k = 0; k < 16; ++k) XS[tid * kXp + 32 + k] = sh[k];
      }
    }
    __syncthreads();
    if (wid < kAdjWork / 32) {
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
        const int rq = 8 * wid + 4 * q;
        float z[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int u = 0; u < 2; ++u) z[i][u] = w.b0[lane + 32 * u];
#pragma unroll 1
        for (int k = 0; k < KP; k += 4) {  // feature 51: W0's padding is 0
          float w0[4], w1[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            w0[j] = WS[lane * kWp + k + j];
            w1[j] = WS[(lane + 32) * kWp + k + j];
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 v = *reinterpret_cast<const float4*>(XS + (rq + i) * kXp + k);
            const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              z[i][0] = fmaf(w0[j], x[j], z[i][0]);
              z[i][1] = fmaf(w1[j], x[j], z[i][1]);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = rq + i;
          const bool in = r < nrows;
          float h[2], d[NO];
          bool on[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            on[u] = in && (ldm == 2 ? (MS[r * 2 + u] >> lane & 1u) != 0 : z[i][u] > 0.0f);
            h[u] = on[u] ? z[i][u] : 0.0f;
          }
#pragma unroll
          for (int c = 0; c < NO; ++c) {
            d[c] = DS[r * NO + c];
            if (ldy != NO) {
              const float o = w.b1[c] + warp_sum(fmaf(w.W1[c * NH + lane], h[0], w.W1[c * NH + lane + 32] * h[1]));
              const float v = __shfl_sync(0xffffffffu, sigmoidf_ref(o), 0);
              d[c] *= (1.0f - v) * v;
              __syncwarp();
              if (lane == 0) DS[r * NO + c] = d[c];
            }
          }
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int m = lane + 32 * u;
            const float dh = d[0] * w.W1[m] + d[1] * w.W1[NH + m] + d[2] * w.W1[2 * NH + m];
            DZ[r * kZp + m] = on[u] ? dh : 0.0f;
            HS[r * kZp + m] = h[u];
          }
        }
      }
    }
    __syncthreads();
    if (tid < kAdjWork) {  // rows past P: x, h and d are 0
      float part[kPer], part1[NO];
#pragma unroll
      for (int j = 0; j < kPer; ++j) part[j] = 0.0f;
#pragma unroll
      for (int c = 0; c < NO; ++c) part1[c] = 0.0f;
      if (kg < kGroups) {
#pragma unroll 4
        for (int r = 0; r < TM; ++r) {
          const float dz = DZ[r * kZp + n];
#pragma unroll
          for (int f = 0; f < 2; ++f) {
            const float4 v = *reinterpret_cast<const float4*>(XS + r * kXp + kPer * kg + 4 * f);
            part[4 * f] = fmaf(dz, v.x, part[4 * f]);
            part[4 * f + 1] = fmaf(dz, v.y, part[4 * f + 1]);
            part[4 * f + 2] = fmaf(dz, v.z, part[4 * f + 2]);
            part[4 * f + 3] = fmaf(dz, v.w, part[4 * f + 3]);
          }
        }
      } else {  // dW1 of hidden unit n, and db1[n]
#pragma unroll 4
        for (int r = 0; r < TM; ++r) {
          const float h = HS[r * kZp + n];
#pragma unroll
          for (int c = 0; c < NO; ++c) part1[c] = fmaf(DS[r * NO + c], h, part1[c]);
          part[0] += n < NO ? DS[r * NO + n] : 0.0f;
        }
      }
#pragma unroll
      for (int j = 0; j < kPer; ++j) acc[j] += part[j];
#pragma unroll
      for (int c = 0; c < NO; ++c) acc1[c] += part1[c];
    }
  }
  if (tid < kGroups * NH) {
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int k = kPer * kg + j;
      if (k < KP) pb[n * KP + k] = k == KIN ? 0.0f : acc[j];
      if (k == KIN) pb[NH * KP + NO * NH + n] = acc[j];
    }
  } else if (tid < kAdjWork) {
#pragma unroll
    for (int c = 0; c < NO; ++c) pb[NH * KP + c * NH + n] = acc1[c];
    if (n < NO) pb[NH * KP + NO * NH + NH + n] = acc[0];
  }
}

// X (P rows), d_out (P,3), the forward's colours y (row stride ldy) and mask bits (two words a row,
// stride ldm) -> d_hash (P,32), d_normal (P,3), per-block weight-gradient partials
// [dW0 (64 x 52) | dW1 (3 x 64) | db0 (64) | db1 (3)]. y and mask may lie in d_hash's own rows (a
// tile's are read before its d_hash is written).
template <int kMode, bool kCustomWait>
__global__ void __launch_bounds__(kAdjThreads, 1)
    k_mlp_adjoint(const float* __restrict__ X, int64_t ldx, int64_t P, MlpW w, const float* __restrict__ d_out,
                  const float* y, int64_t ldy, const uint32_t* mask, int64_t ldm, float* d_hash,
                  float* __restrict__ d_normal, float* __restrict__ partials, TcGuard g, RowSrc src) {
  using S = AdjShape<kMode>;
  constexpr bool kFold = S::kFold;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t wait_limit = kCustomWait ? g.limit : kWaitLimit;
  uint8_t* A = smem;
  uint8_t* MK = smem + S::kOffMask;
  uint8_t* V = smem + S::kOffV;
  uint8_t* ROWS = smem + S::kOffRows;
  float* CUR = reinterpret_cast<float*>(smem + S::kOffCur);
  float* SHT = reinterpret_cast<float*>(smem + S::kOffSh);
  float* AUX = reinterpret_cast<float*>(smem + S::kOffAux);
  uint8_t* HT = smem + S::kOffH;
  uint64_t* bar_g = reinterpret_cast<uint64_t*>(smem + S::kOffBar);
  uint64_t* bar_dx = bar_g + 1;
  uint64_t* bar_rows = bar_g + 2;  // [2]
  uint32_t* s_taddr = reinterpret_cast<uint32_t*>(bar_g + 4);
  volatile int* s_fail = reinterpret_cast<volatile int*>(s_taddr + 1);  // a worker gave up a wait before staging A
  const int tid = threadIdx.x, lane = tid & 31;
  const int wid = __shfl_sync(0xffffffffu, tid >> 5, 0);  // in a uniform register: warp-uniform branches
  const int q = wid & 3, hh = wid >> 2;
  const int m = 32 * q + lane;  // this thread's sample in the tile (its TMEM lane)
  // V, a warp per hidden unit, lanes over the features (coalesced rows of W0); columns 99, 103, 107 and
  // 108.. are zero
#pragma unroll 4
  for (int n = wid; n < NH; n += kAdjThreads / 32) {
    const float w0 = __ldg(w.W0 + n * KIN + lane);
    const float wn = lane < 3 ? __ldg(w.W0 + n * KIN + 48 + lane) : 0.0f;
#pragma unroll
    for (int c = 0; c < NO; ++c) {
      const float w1 = __ldg(w.W1 + c * NH + n);
      const float v[4] = {w1 * w0, w1 * wn, 0.0f, 0.0f};
      uint32_t h[2], mi[2], l[2];
      cut3(v, h, mi, l);
      uint8_t* o = V + (n >> 3) * kVChunk + (n & 7) * 2;
      const uint32_t oh = (32 * c + lane) * 16, on = (96 + 4 * c + lane) * 16;
      *reinterpret_cast<uint16_t*>(o + oh) = (uint16_t)h[0];
      *reinterpret_cast<uint16_t*>(o + kVPart + oh) = (uint16_t)mi[0];
      *reinterpret_cast<uint16_t*>(o + 2 * kVPart + oh) = (uint16_t)l[0];
      if (lane < (c == 2 ? 8 : 4)) {  // with the zero columns up to 111
        *reinterpret_cast<uint16_t*>(o + on) = (uint16_t)(h[0] >> 16);
        *reinterpret_cast<uint16_t*>(o + kVPart + on) = (uint16_t)(mi[0] >> 16);
        *reinterpret_cast<uint16_t*>(o + 2 * kVPart + on) = (uint16_t)(l[0] >> 16);
      }
    }
  }
  if (tid == 0) {
    tc::mbar_init(bar_g, 1);
    tc::mbar_init(bar_dx, 1);
    tc::mbar_init(bar_rows, 1);
    tc::mbar_init(bar_rows + 1, 1);
    *s_fail = 0;
  }
  __syncwarp();
  if (wid == 0) tc::tmem_alloc(s_taddr, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tb = __shfl_sync(0xffffffffu, *s_taddr, 0), lane_base = (uint32_t)(32 * q) << 16;
  const uint32_t a0 = tc::smem_u32(A), mk0 = tc::smem_u32(MK), v0 = tc::smem_u32(V);
  const int64_t ntiles = (P + TM - 1) / TM, tstep = gridDim.x, t0 = blockIdx.x;
  bool failed = false;
  int it = 0;  // tiles done
  // The issuing warp: phases issued on each barrier. A worker that gave up a wait says so before it arrives at the
  // staged barrier, and then nothing more is issued: no barrier ever has two phases outstanding, so that the
  // drain after a give-up can wait for the last one.
  int n_g = 0, n_dx = 0, n_rows[2] = {0, 0};
  // the workers' sums over the tiles. G of every tile is added up in registers (rounded to nearest; the
  // tensor core's own accumulation truncates, a bias that grows with the number of additions): thread
  // (m, hh) holds row m, hidden units 16 hh ..; unfolded, warps with q = 3 also rows m + kRow2 >= 128 of
  // the second range. kFold: the SH columns of G are each tile's ones row of colour c, hidden unit n,
  // times SH(d) of the tile's ray; thread tid < 384 holds pair (c, n) = tid / 2, SH values 8 (tid % 2) ..
  float acc[16], acc2[kFold ? 1 : 16], shacc[8], sb = 0.0f;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    acc[k] = 0.0f;
    if (!kFold) acc2[k] = 0.0f;
    if (k < 8) shacc[k] = 0.0f;
  }
  const int pair = tid >> 1, sh0 = 8 * (tid & 1);
  // after G of a tile: this thread's part of the accumulators, then (once loaded) into the sums
  auto load_g = [&](int buf, float v[16]) { tc::tmem_ld16(tb + lane_base + buf * kAdjG1 + 16 * hh, v); };
  auto add_g = [&](int buf, float v[16]) {
#pragma unroll
    for (int k = 0; k < 16; ++k) acc[k] += v[k];
    if (kFold) {
      if (q >= 1 && lane == 3 + 8 * (q - 1)) {  // row 40 c + 35, c = q - 1
        float4* o = reinterpret_cast<float4*>(CUR + (buf * 3 + q - 1) * NH + 16 * hh);
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
      }
    } else if (q == 3) {
      tc::tmem_ld16(tb + lane_base + buf * kAdjG1 + 64 + 16 * hh, v);
      tc::tmem_wait_ld();
#pragma unroll
      for (int k = 0; k < 16; ++k) acc2[k] += v[k];
    }
  };
  auto add_sh = [&](int i) {  // tile i of this block, a barrier after its add_g
    if (hh < 3) {
      const float s = CUR[(i & 1) * 3 * NH + pair];
#pragma unroll
      for (int k = 0; k < 8; ++k) shacc[k] = fmaf(s, SHT[16 * (i & 3) + sh0 + k], shacc[k]);
    }
  };
  if (wid == kAdjWork / 32) {  // the issuing warp, converged throughout
    const bool lead = tc::elect_lead();
    // a descriptor's address field is its low 14 bits (16-byte units) and every offset below keeps it
    // there, so one base per operand and constant steps
    const uint64_t da_g = tc::sdesc(a0, 128, kAdjChunk), db_g = tc::sdesc(mk0, 128, kAdjChunk);
    const uint64_t db_x = tc::sdesc(v0, kVChunk, 128);
    auto fetch_rows = [&](int64_t t, int buf) {
      if (lead) {
        const int64_t r0 = t * TM;
        const uint32_t bytes = (uint32_t)(P - r0 < TM ? P - r0 : TM) * S::kRowBytes;
        tc::mbar_arrive_expect_tx(bar_rows + buf, bytes + (kFold ? kAdjAux : 0));
        if (kFold) {
          float* aux = AUX + buf * (kAdjAux / 4);
          tc::bulk_g2s(aux, d_out + r0 * NO, TM * NO * 4, bar_rows + buf);
          tc::bulk_g2s(aux + TM * NO, y + r0 * NO, TM * NO * 4, bar_rows + buf);
          tc::bulk_g2s(aux + 2 * TM * NO, mask + r0 * 2, TM * 2 * 4, bar_rows + buf);
        }
        tc::bulk_g2s(ROWS + buf * TM * S::kRowBytes, X + r0 * S::kLd, bytes, bar_rows + buf);
      }
      ++n_rows[buf];
    };
    auto issue_dx = [&]() {
      tc::fence_after_sync();
#pragma unroll
      for (int p = 2; p >= 0; --p)  // the small parts first
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          tc::mma_bf16_ts_warp(lead, tb + kAdjDx, tb + kAdjMk + 8 * ks, db_x + (p * kVPart + ks * 2 * kVChunk) / 16, kIdDx,
                               p != 2 || ks != 0);
      tc::commit_warp(lead, bar_dx);
      ++n_dx;
    };
    auto issue_g = [&](int buf) {
      tc::fence_after_sync();
      const uint64_t b = db_g + buf * (kAdjMask / 16);
#pragma unroll
      for (int p = 2; p >= 0; --p)
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const bool acc_on = p != 2 || ks != 0;
          tc::mma_bf16_warp(lead, tb + buf * kAdjG1, da_g + (p * S::kPart + ks * 256) / 16, b + ks * 16, kIdG, acc_on);
          if (!kFold)
            tc::mma_bf16_warp(lead, tb + buf * kAdjG1 + 64, da_g + (p * S::kPart + (S::kRow2 / 8) * kAdjChunk + ks * 256) / 16,
                              b + ks * 16, kIdG, acc_on);
        }
      tc::commit_warp(lead, bar_g);
      ++n_g;
    };
    if (S::kBulk)
#pragma unroll
      for (int b = 0; b < S::kBufs; ++b)
        if (t0 + b * tstep < ntiles) fetch_rows(t0 + b * tstep, b);
    adj_sync_or(false);
    if (t0 < ntiles) issue_dx();
    for (int64_t t = t0; t < ntiles; t += tstep, ++it) {
      const int par = it & 1;
      adj_staged_sync();  // A of this tile is staged, its rows are read
      if (!__any_sync(0xffffffffu, *s_fail)) {
        issue_g(par);
        if (S::kBulk && t + S::kBufs * tstep < ntiles) fetch_rows(t + S::kBufs * tstep, S::kBufs == 2 ? par : 0);
      }
      if (__shfl_sync(0xffffffffu, (int)adj_sync_or(false), 0)) {  // uniform, so that the loop stays so
        failed = true;
        break;
      }
      if (t + tstep < ntiles) issue_dx();  // queued behind G
    }
  } else {
    // What a tile needs besides its rows: dL/dcolour, the forward's colours and 16 mask bits a thread.
    // Folded: they arrive with the rows. Otherwise loaded here a tile ahead of their use (and, for
    // kAdjStrided, this thread's share of the rows).
    float dy[NO], yv[NO], d[NO];
    uint32_t bits[2] = {0, 0};
    float pre[13], dir[3] = {0.0f, 0.0f, 0.0f};  // dir: kFold, one thread, the tile's ray
    auto load_tile = [&](int64_t t) {
      if (kFold) {
        if (tid == kAdjShTid) {
#pragma unroll
          for (int c = 0; c < 3; ++c) dir[c] = __ldg(src.rays_d + 3 * (t * TM / src.S) + c);
        }
        return;
      }
      const int64_t i = t * TM + m;
      const bool in = i < P;
#pragma unroll
      for (int c = 0; c < NO; ++c) {
        dy[c] = in ? __ldg(d_out + i * NO + c) : 0.0f;
        yv[c] = in ? y[i * ldy + c] : 0.0f;
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) bits[k] = in ? mask[i * ldm + k] : 0u;
      if (!S::kBulk) {
#pragma unroll
        for (int k = 0; k < 13; ++k) {
          const int e = tid + kAdjWork * k, r = e / KIN;
          pre[k] = e < TM * KIN && t * TM + r < P ? __ldg(X + (t * TM + r) * ldx + (e - r * KIN)) : 0.0f;
        }
      }
    };
    bool ok = true;                 // no wait of this thread has given up
    auto stage_tile = [&](int i) {  // tile i of this block
      const int buf = i & 1;
      if (kFold) {
        ok = tc::mbar_wait(bar_rows + buf, (i >> 1) & 1, wait_limit) && ok;
        const float* aux = AUX + buf * (kAdjAux / 4);
#pragma unroll
        for (int c = 0; c < NO; ++c) {
          dy[c] = aux[NO * m + c];
          yv[c] = aux[NO * (TM + m) + c];
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) bits[k] = __float_as_uint(aux[2 * NO * TM + 2 * m + k]);
        if (tid == kAdjShTid) {
          float sh[16];
          sh16(dir[0], dir[1], dir[2], sh);
#pragma unroll
          for (int k = 0; k < 16; ++k) SHT[16 * (i & 3) + k] = sh[k];
        }
      }
#pragma unroll
      for (int c = 0; c < NO; ++c) d[c] = dy[c] * ((1.0f - yv[c]) * yv[c]);  // 0 on rows past P
      sb += hh == 0 ? d[0] : (hh == 1 ? d[1] : d[2]);
      if ((bits[0] | bits[1]) == 0u) d[0] = d[1] = d[2] = 0.0f;  // no unit is active: nothing to pass on
      __syncwarp();
      stage_mask(MK + buf * kAdjMask, tb + lane_base + kAdjMk + 8 * hh, m, hh, bits[hh >> 1] >> (16 * (hh & 1)));
      if (!S::kBulk) {
#pragma unroll
        for (int k = 0; k < 13; ++k) {
          const int e = tid + kAdjWork * k, r = e / KIN;
          if (e < TM * KIN) reinterpret_cast<float*>(ROWS)[r * KP + (e - r * KIN)] = pre[k];
        }
      }
    };
    auto row_of = [&](int buf) {
      return reinterpret_cast<const float4*>(ROWS + buf * TM * S::kRowBytes + m * S::kRowBytes);
    };
    if (t0 < ntiles) {
      load_tile(t0);
      stage_tile(0);
      if (t0 + tstep < ntiles) load_tile(t0 + tstep);  // a tile ahead of its use
    }
    tc::fence_smem_to_async();
    tc::fence_before_sync();
    adj_sync_or(false);
    for (int64_t t = t0; t < ntiles; t += tstep, ++it) {
      const int par = it & 1;
      const int64_t m0 = t * TM;
      const bool valid = m0 + m < P, more = t + tstep < ntiles;
      // 1: G of the previous tile (A is free), this tile's rows. A wait that gives up is agreed on at the
      // end of the tile; until then the block goes on with whatever the memory holds, but issues nothing.
      if (it > 0) ok = tc::mbar_wait(bar_g, par ^ 1, wait_limit) && ok;
      if (S::kBulk && !kFold) ok = tc::mbar_wait(bar_rows, par, wait_limit) && ok;
      if (!ok) *s_fail = 1;
      __syncwarp();
      tc::fence_after_sync();
      // 2: the rows of A
      const float d0 = d[0], d1 = d[1], d2 = d[2];
      if constexpr (kFold) {
        const float4* rrow = row_of(par) + 2 * hh;  // features 8 hh ..
        const float4 x0 = rrow[0], x1 = rrow[1];
#pragma unroll
        for (int c = 0; c < NO; ++c) {
          const float v0[4] = {d[c] * x0.x, d[c] * x0.y, d[c] * x0.z, d[c] * x0.w};
          const float v1[4] = {d[c] * x1.x, d[c] * x1.y, d[c] * x1.z, d[c] * x1.w};
          uint32_t h[4], mi[4], l[4];
          cut3(v0, h, mi, l);
          cut3(v1, h + 2, mi + 2, l + 2);
          uint8_t* o = A + (5 * c + hh) * kAdjChunk + m * 16;
          *reinterpret_cast<uint4*>(o) = make_uint4(h[0], h[1], h[2], h[3]);
          *reinterpret_cast<uint4*>(o + S::kPart) = make_uint4(mi[0], mi[1], mi[2], mi[3]);
          *reinterpret_cast<uint4*>(o + 2 * S::kPart) = make_uint4(l[0], l[1], l[2], l[3]);
        }
        if (hh < NO) {  // the last chunk of colour hh: the normal and the ones feature
          float4 x = row_of(par)[8];
          x.w = 1.0f;
          const float dc = hh == 0 ? d[0] : (hh == 1 ? d[1] : d[2]);
          const float v[4] = {dc * x.x, dc * x.y, dc * x.z, dc * x.w};
          uint32_t h[2], mi[2], l[2];
          cut3(v, h, mi, l);
          uint8_t* o = A + (5 * hh + 4) * kAdjChunk + m * 16;
          *reinterpret_cast<uint4*>(o) = make_uint4(h[0], h[1], 0u, 0u);
          *reinterpret_cast<uint4*>(o + S::kPart) = make_uint4(mi[0], mi[1], 0u, 0u);
          *reinterpret_cast<uint4*>(o + 2 * S::kPart) = make_uint4(l[0], l[1], 0u, 0u);
        }
      } else {
        const float4* rrow = row_of(0);
        float3 dir = make_float3(0.0f, 0.0f, 0.0f);
        if (S::kCompact && valid) {
          const uint32_t r = (uint32_t)(m0 + m) / (uint32_t)src.S;
          dir = make_float3(__ldg(src.rays_d + 3 * (size_t)r), __ldg(src.rays_d + 3 * (size_t)r + 1),
                            __ldg(src.rays_d + 3 * (size_t)r + 2));
        }
#pragma unroll
        for (int i = 0; i < 13; ++i) {  // chunks of 4 features: 3 hh .. 3 hh + 2, and 12 for hh = 3
          if (i < 12 ? i / 3 != hh : hh != 3) continue;
          float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (valid) {
            if (S::kCompact)
              x = i < 8 ? rrow[i] : (i < 12 ? sh_chunk(dir.x, dir.y, dir.z, i - 8) : rrow[8]);
            else
              x = rrow[i];
          }
          if (i == 12) x.w = valid ? 1.0f : 0.0f;
#pragma unroll
          for (int c = 0; c < NO; ++c) {
            const float v[4] = {d[c] * x.x, d[c] * x.y, d[c] * x.z, d[c] * x.w};
            uint32_t h[2], mi[2], l[2];
            cut3(v, h, mi, l);
            const int r0 = KP * c + 4 * i;
            uint8_t* o = A + (r0 >> 3) * kAdjChunk + m * 16 + (r0 & 4) * 2;
            *reinterpret_cast<uint2*>(o) = make_uint2(h[0], h[1]);
            *reinterpret_cast<uint2*>(o + S::kPart) = make_uint2(mi[0], mi[1]);
            *reinterpret_cast<uint2*>(o + 2 * S::kPart) = make_uint2(l[0], l[1]);
          }
        }
      }
      tc::fence_smem_to_async();
      tc::fence_before_sync();
      if (!kFold) __syncwarp();
      adj_staged_arrive();
      // 3: G of this tile runs; G of the previous tile and dX of this one are read out (their loads in
      // flight together), the next tile's mask is staged
      ok = tc::mbar_wait(bar_dx, par, wait_limit) && ok;
      __syncwarp();
      tc::fence_after_sync();
      {
        float gv[16], r[8], u[8], v[8];
        if (kFold && it > 0) load_g(par ^ 1, gv);
        tc::tmem_ld8(tb + lane_base + kAdjDx + 8 * hh, r);
        tc::tmem_ld8(tb + lane_base + kAdjDx + 32 + 8 * hh, u);
        tc::tmem_ld8(tb + lane_base + kAdjDx + 64 + 8 * hh, v);
        if (kFold && it > 1) add_sh(it - 2);
        tc::tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 8; ++k) r[k] = fmaf(d2, v[k], fmaf(d1, u[k], d0 * r[k]));
        if constexpr (kFold) {  // 16-byte chunk k of a row at k ^ (row % 8): no bank conflicts either way
          *reinterpret_cast<float4*>(HT + m * 128 + ((2 * hh) ^ (m & 7)) * 16) = make_float4(r[0], r[1], r[2], r[3]);
          *reinterpret_cast<float4*>(HT + m * 128 + ((2 * hh + 1) ^ (m & 7)) * 16) = make_float4(r[4], r[5], r[6], r[7]);
        } else if (valid) {
          float4* o = reinterpret_cast<float4*>(d_hash + (m0 + m) * 32 + 8 * hh);
          o[0] = make_float4(r[0], r[1], r[2], r[3]);
          o[1] = make_float4(r[4], r[5], r[6], r[7]);
        }
        if (!kFold && it > 0) {  // (not in flight together: the unfolded forms have no registers left)
          __syncwarp();
          load_g(par ^ 1, gv);
          tc::tmem_wait_ld();
        }
        if (it > 0) add_g(par ^ 1, gv);
        __syncwarp();
      }
      if (hh == 3) {
        float r[4], u[4], v[4];
        tc::tmem_ld4(tb + lane_base + kAdjDx + 96, r);
        tc::tmem_ld4(tb + lane_base + kAdjDx + 100, u);
        tc::tmem_ld4(tb + lane_base + kAdjDx + 104, v);
        tc::tmem_wait_ld();
        if (kFold || valid) {
#pragma unroll
          for (int k = 0; k < 3; ++k) d_normal[(m0 + m) * 3 + k] = fmaf(d2, v[k], fmaf(d1, u[k], d0 * r[k]));
        }
      }
      if constexpr (kFold) {  // the four warps of 32 samples: their rows leave in whole lines
        asm volatile("bar.sync %0, 128;" ::"r"(4 + q) : "memory");
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int row = 32 * q + 8 * hh + 4 * s + (lane >> 3), k = lane & 7;
          *reinterpret_cast<float4*>(d_hash + (m0 + row) * 32 + 4 * k) =
              *reinterpret_cast<const float4*>(HT + row * 128 + (k ^ (row & 7)) * 16);
        }
      }
      if (!S::kBulk) adj_workers_sync();  // every worker has read this tile's rows: they are overwritten next
      if (more) {
        stage_tile(it + 1);
        if (t + 2 * tstep < ntiles) load_tile(t + 2 * tstep);
      }
      tc::fence_smem_to_async();
      tc::fence_before_sync();
      if (adj_sync_or(!ok)) {
        failed = true;
        break;
      }
    }
    if (!failed && it > 0) failed = !tc::mbar_wait(bar_g, (it - 1) & 1, wait_limit);
    __syncwarp();
  }
  failed = __syncthreads_or(failed);
  if (failed && tid == kAdjWork) {
    // MMAs and row copies may still run: let them finish (bounded) before tensor memory is freed and
    // the block leaves
    if (n_g > 0) tc::mbar_wait(bar_g, (n_g - 1) & 1, kDrainLimit);
    if (n_dx > 0) tc::mbar_wait(bar_dx, (n_dx - 1) & 1, kDrainLimit);
#pragma unroll
    for (int b = 0; b < 2; ++b)
      if (n_rows[b] > 0) tc::mbar_wait(bar_rows + b, (n_rows[b] - 1) & 1, kDrainLimit);
    report_timeout(g.status);
  }
  __syncthreads();
  tc::fence_after_sync();
  // weight-gradient partials of this block: G (and the SH sums) through shared memory
  const bool have = it > 0 && !failed;
  float* pb = partials + (int64_t)blockIdx.x * WG;
  float* GD = reinterpret_cast<float*>(smem);                       // [3 * kStride rows][65]
  float* SHD = GD + 160 * 65;                                       // kFold: [3 * 64][17]
  float* SB = SHD + 3 * NH * 17;                                    // [3][4]
  if (have && kFold) {
    if (it > 1) add_sh(it - 2);
  }
  if (have && tid < kAdjWork) {
    float gv[16];
    load_g((it - 1) & 1, gv);
    tc::tmem_wait_ld();
    add_g((it - 1) & 1, gv);
  }
  if (have && kFold) {
    __syncthreads();
    add_sh(it - 1);
  }
  if (have && tid < kAdjWork) {
    if (m < 3 * S::kStride) {
#pragma unroll
      for (int i = 0; i < 16; ++i) GD[m * 65 + 16 * hh + i] = acc[i];
    }
    if (!kFold && q == 3) {
#pragma unroll
      for (int i = 0; i < 16; ++i) GD[(m + S::kRow2) * 65 + 16 * hh + i] = acc2[i];
    }
  }
  if (kFold && hh < 3) {
#pragma unroll
    for (int k = 0; k < 8; ++k) SHD[pair * 17 + sh0 + k] = shacc[k];
  }
  bool finite = fabsf(sb) < INFINITY;
#pragma unroll
  for (int i = 0; i < 16; ++i) {  // rows past 3 * kStride hold nothing
    finite = finite && (m >= 3 * S::kStride || fabsf(acc[i]) < INFINITY);
    if (!kFold) finite = finite && (m + S::kRow2 >= 3 * S::kStride || fabsf(acc2[i]) < INFINITY);
    if (kFold && i < 8) finite = finite && fabsf(shacc[i]) < INFINITY;
  }
  sb = warp_sum(sb);
  if (hh < NO && lane == 0) SB[hh * 4 + q] = sb;
  const bool plain = __syncthreads_or(have && !finite);
  constexpr int kOnes = kFold ? 35 : 51;
  // a warp per hidden unit, lanes over the 51 columns of W0 (and the padding column, 0)
#pragma unroll 4
  for (int n = plain ? NH : wid; n < NH; n += kAdjThreads / 32) {
    float w1[NO], s[NO];
#pragma unroll
    for (int c = 0; c < NO; ++c) {
      w1[c] = __ldg(w.W1 + c * NH + n);
      s[c] = 0.0f;
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int col = lane + 32 * half;
      if (col < KP) {
        const int k = kFold ? (col < 32 ? col : (col < 48 ? -1 : col - 16)) : col;
        const float w0 = col < KIN ? __ldg(w.W0 + n * KIN + col) : 0.0f;
        float v = 0.0f;
#pragma unroll
        for (int c = 0; c < NO; ++c) {
          float gv = 0.0f;
          if (have && col < KIN) gv = k >= 0 ? GD[(c * S::kStride + k) * 65 + n] : SHD[(c * NH + n) * 17 + col - 32];
          v = fmaf(w1[c], gv, v);
          s[c] = fmaf(w0, gv, s[c]);
        }
        pb[n * KP + col] = v;
      }
    }
    float db = 0.0f;
#pragma unroll
    for (int c = 0; c < NO; ++c) {
      const float ones = have ? GD[(c * S::kStride + kOnes) * 65 + n] : 0.0f;
      db = fmaf(w1[c], ones, db);
      s[c] = fmaf(__ldg(w.b0 + n), ones, warp_sum(s[c]));
      if (lane == 0) pb[NH * KP + c * NH + n] = s[c];
    }
    if (lane == 0) pb[NH * KP + NO * NH + n] = db;
  }
  if (tid < NO && !plain) {
    const float* s = SB + tid * 4;
    pb[NH * KP + NO * NH + NH + tid] = have ? (s[0] + s[1]) + (s[2] + s[3]) : 0.0f;
  }
  if (plain) adj_plain_sums<kMode>(reinterpret_cast<float*>(smem), X, ldx, P, w, d_out, y, ldy, mask, ldm, pb, src);
  tc::fence_before_sync();
  __syncthreads();
  __syncwarp();
  if (wid == 0) tc::tmem_dealloc(tb, 512);
}

}  // namespace vx
