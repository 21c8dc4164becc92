// SDF + Eq.7 gradient/normal queries (models/sdf_grid.py:90-160) of a large batch of scattered
// points, in spatial order. When the grid does not fit in L2 (a 512^3 grid is 512 MiB), a batch of
// random points reads every stencil from a different DRAM row, and any 32 of them touch ~20 lines with
// each of their 32 loads. Here the points are brought into bricks of 16^3 cells; a block stages a brick's
// voxels (19^3 with their neighbours) in shared memory and answers its points from there. The per-point
// arithmetic is the plain query's (common.cuh), so the outputs are bit-identical to it; the order of the
// points inside a brick is not fixed and does not show.
//
// Random accesses to DRAM run at ~45 G reads or ~22 G writes a second on this part, to an L2-resident
// window at 200-260 G (a probe of 2^24 accesses over 32 MB .. 1 GB), and returning atomics on a few
// thousand counters at 75 G. So the permutation goes there and back in two steps of bounded reach:
//   count      points per brick, from per-block histograms in shared memory
//   partition  points -> at most 256 buckets of consecutive bricks, a block's points of one bucket side by
//              side: records (x, y, z) at place k, k kept per point
//   bricks     within each bucket (a window of a few MB) -> brick order, with k
//   query      a brick's points from shared memory, or those of sparse bricks from the grid; results at k,
//              inside the bucket's window
//   collect    each point's result from its k: neighbours of a partition block read the same 256 runs
// Points that crowd into a few cells, 32 neighbours at a time, as a caller's own order or the clamp of points outside
// the box may have them, are answered in the order they came (kCrowded).
// What bounds it: DRAM traffic (records, grid, results: ~180 bytes a point with normals and the grid once)
// and, with normals, issue. 2^24 uniform points of a 512^3 grid, one query of
// the SDF and one of gradient and normal: 4.40 ms (Morton keys, a four-pass radix sort, queries through
// L1) -> 1.94 ms; with the points scattered to bricks in one step 3.03 ms.
#include "common.cuh"

namespace vx {
namespace {

constexpr int kBrick = 16;                  // cells per axis
constexpr int kReg = kBrick + 3;            // voxels per axis: lower neighbours, upper corners and theirs
constexpr int kPitch = 24;                  // floats per row: a row may start up to 3 voxels early (16 bytes)
constexpr int kChunk = 2048;                // points of a brick that one block takes
constexpr int kQueryThreads = 256;
constexpr int kTile = 4096;                 // points of a partition or brick-order block
constexpr int kTileThreads = 512;
constexpr int kCountThreads = 1024;
constexpr int kBuckets = 256;               // at most
// Bricks with at least this many points are staged, the others' points read the grid themselves: at 128 points
// a brick (2^22 of a 512^3 grid) 341 us staged against 269 with normals and 194 against 116 without, at 512
// points 536 against ~1080 and 270 against ~460. From a mean of kDenseMean on all are staged, which saves
// the other pass over the records.
constexpr int kDenseNormals = 160, kDenseSdf = 256, kDenseMean = 400;
// With at most this many cells among 32 consecutive points on average, the points are queried in the order they came,
// with nothing moved. 2^24 points with gradients and normals, all in one cell (1 cell in 32 points), 9 in 10 there and the
// rest anywhere (4.2), 8 in 10 (7.4): 564, 1009 and 1150 us so, 1101, 1324 and 1291 us by bricks. The line lies lower than
// where these meet because crowded and scattered stretches may also follow one another (8 in 10 so: ~1730 us).
constexpr int kCrowded = 5;
constexpr int kSmemBins = 48 * 1024;        // bins of a block's histogram in shared memory
constexpr int64_t kBatch = int64_t(1) << 24;  // points per pass: bounds the workspace
constexpr int kMaxAxis = 1 << 24;             // longer axes (float32 cell numbers): the plain kernel
constexpr int kMaxBins = 1 << 22;             // more bricks (grids a few voxels thick): the plain kernel

struct Bins {
  int n[3];
  __host__ __device__ int64_t total() const { return (int64_t)n[0] * n[1] * n[2]; }
};

Bins make_bins(const int32_t res[3]) {
  Bins b;
  for (int a = 0; a < 3; ++a) b.n[a] = (res[a] + kBrick - 1) / kBrick;
  return b;
}

// Bricks of a bucket: 2^bucket_shift.
inline int bucket_shift(int64_t nbins) {
  int shift = 0;
  while (((nbins - 1) >> shift) >= kBuckets) ++shift;
  return shift;
}

// Dynamic shared memory of k_brick_order: a tile's records with their bricks, and two counters a brick of the bucket.
constexpr size_t order_bytes(int shift) { return (size_t)kTile * 18 + ((size_t)8 << shift); }
static_assert(kMaxBins / kBuckets == 1 << 14 && order_bytes(14) <= 220 * 1024, "the largest bucket's counters fit");

// Grids that the bricks do not take and the plain kernel does: axes too long for exact cell numbers, and more
// bricks than the buckets' counters hold (2 x 65 x 16,000,000 has 5 M, a cube of 2^31 voxels 0.5 M).
inline bool plain_grid(const int32_t res[3]) {
  return res[0] > kMaxAxis || res[1] > kMaxAxis || res[2] > kMaxAxis || make_bins(res).total() > kMaxBins;
}

__device__ __forceinline__ int point_bin(const Grid& g, const Bins& b, float px, float py, float pz) {
  // cell indices (the clamp of gs_coord keeps them in [0, R-1]; NaN reads as 0)
  const int x = (int)gs_coord(px, g.lo[0], g.den[0], g.inv_den[0], g.rx) / kBrick;
  const int y = (int)gs_coord(py, g.lo[1], g.den[1], g.inv_den[1], g.ry) / kBrick;
  const int z = (int)gs_coord(pz, g.lo[2], g.den[2], g.inv_den[2], g.rz) / kBrick;
  return (x * b.n[1] + y) * b.n[2] + z;
}

// What k_bin_count saw of the points' order, every fourth run of 32 of a block's: how many runs, and their cells.
struct Sample {
  int runs, cells;
};

__device__ __forceinline__ bool crowded(const Sample* s) {
  const int runs = __ldg(&s->runs);
  return runs > 0 && __ldg(&s->cells) <= kCrowded * runs;
}

// Points per brick. kSmem: a histogram per block (one block per SM), added up at its end; otherwise (more
// bricks than fit) straight into the counts.
template <bool kSmem>
__global__ void __launch_bounds__(kCountThreads) k_bin_count(const float* __restrict__ xyz, int64_t n, Grid g, Bins b,
                                                            int* __restrict__ counts, Sample* __restrict__ sample) {
  extern __shared__ int hist[];
  __shared__ int seen[2];
  const int nbins = (int)b.total(), lane = threadIdx.x & 31;
  int runs = 0, cells = 0;
  if (threadIdx.x < 2) seen[threadIdx.x] = 0;
  if (kSmem)
    for (int i = threadIdx.x; i < nbins; i += kCountThreads) hist[i] = 0;
  __syncthreads();
  constexpr int kPer = 4;  // points a thread, their loads in flight together
  const int64_t step = (int64_t)gridDim.x * kCountThreads;
  for (int64_t i0 = blockIdx.x * (int64_t)kCountThreads + threadIdx.x; i0 - lane < n; i0 += kPer * step) {  // whole warps
    float p[kPer][3];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int64_t i = i0 + u * step;
#pragma unroll
      for (int a = 0; a < 3; ++a) p[u][a] = i < n ? __ldg(xyz + 3 * i + a) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int64_t i = i0 + u * step;
      const int x = (int)gs_coord(p[u][0], g.lo[0], g.den[0], g.inv_den[0], g.rx);
      const int y = (int)gs_coord(p[u][1], g.lo[1], g.den[1], g.inv_den[1], g.ry);
      const int z = (int)gs_coord(p[u][2], g.lo[2], g.den[2], g.inv_den[2], g.rz);
      if (i < n) atomicAdd((kSmem ? hist : counts) + (x / kBrick * b.n[1] + y / kBrick) * b.n[2] + z / kBrick, 1);
      if (u == 0 && i - lane + 32 <= n) {
        const unsigned same = __match_any_sync(0xffffffffu, lin3(g, x, y, z));
        cells += __popc(__ballot_sync(0xffffffffu, __ffs(same) - 1 == lane));
        ++runs;
      }
    }
  }
  if (lane == 0) {
    atomicAdd(seen, runs);
    atomicAdd(seen + 1, cells);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(&sample->runs, seen[0]);
    atomicAdd(&sample->cells, seen[1]);
  }
  if (kSmem) {
    for (int i = threadIdx.x; i < nbins; i += kCountThreads)
      if (hist[i]) atomicAdd(counts + i, hist[i]);
  }
}

constexpr int kScanBins = 4096;  // bins of a scan block, 4 a thread

// Counts -> their exclusive starts, and the work list of bricks with at least `dense` points: {brick, first
// record} of every chunk, nchunks entries in any order (none for crowded points). A block adds up the counts before its own bins
// itself (L2 reads, all in flight at once) instead of waiting for the blocks before it: 32,768 bins take
// 6 us, 26 as one block's loop over carries.
__global__ void __launch_bounds__(1024) k_bin_scan(const int* __restrict__ counts, int64_t nbins, int dense,
                                                   int* __restrict__ starts, int* __restrict__ nchunks,
                                                   int2* __restrict__ list, const Sample* __restrict__ sample) {
  if (crowded(sample)) return;
  __shared__ int2 part[32];
  __shared__ int before[32], first;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t base = blockIdx.x * (int64_t)kScanBins;
  const int4* c4 = reinterpret_cast<const int4*>(counts);
  int pre = 0;
#pragma unroll 4
  for (int64_t i = tid; i < base / 4; i += 1024) {
    const int4 v = __ldg(c4 + i);
    pre += v.x + v.y + v.z + v.w;
  }
  const int64_t i0 = base + 4 * tid;
  int c[4] = {0, 0, 0, 0};
  int2 mine = make_int2(0, 0);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (i0 + j < nbins) c[j] = __ldg(counts + i0 + j);
    mine.x += c[j];
    mine.y += c[j] >= dense ? (c[j] + kChunk - 1) / kChunk : 0;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) pre += __shfl_xor_sync(0xffffffffu, pre, o);
  int2 inc = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, inc.x, o), y = __shfl_up_sync(0xffffffffu, inc.y, o);
    if (lane >= o) {
      inc.x += x;
      inc.y += y;
    }
  }
  if (lane == 31) part[warp] = inc;
  if (lane == 0) before[warp] = pre;
  __syncthreads();
  int2 at = make_int2(inc.x - mine.x, inc.y - mine.y);
  for (int w = 0; w < 32; ++w) {
    at.x += before[w] + (w < warp ? part[w].x : 0);
    at.y += w < warp ? part[w].y : 0;
  }
  if (tid == 1023) first = atomicAdd(nchunks, at.y + mine.y);
  __syncthreads();
  at.y += first;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (i0 + j < nbins) starts[i0 + j] = at.x;
    if (c[j] > 0 && c[j] >= dense)
      for (int q = 0; q < c[j]; q += kChunk) list[at.y++] = make_int2((int)(i0 + j), at.x + q);
    at.x += c[j];
    if (i0 + j == nbins - 1) starts[nbins] = at.x;
  }
}

// Exclusive scan of cnt[0, width) into loc by the block (kTileThreads threads).
__device__ __forceinline__ void scan_counts(const int* cnt, int* loc, int width) {
  __shared__ int part[kTileThreads / 32], total;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int carry = 0;
  for (int base = 0; base < width; base += kTileThreads) {
    const int v = base + tid < width ? cnt[base + tid] : 0;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) part[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      const int p = lane < kTileThreads / 32 ? part[lane] : 0;
      int q = p;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, q, o);
        if (lane >= o) q += t;
      }
      if (lane < kTileThreads / 32) part[lane] = q - p;
      if (lane == 31) total = q;
    }
    __syncthreads();
    if (base + tid < width) loc[base + tid] = carry + part[warp] + inc - v;
    carry += total;
    __syncthreads();
  }
}

// Points into buckets of 2^shift bricks: a block reserves a run per bucket, puts its points side by side in
// shared memory and writes the runs from there (whole sectors: a 16-byte store into an absent sector makes
// L2 read it from DRAM first).
__global__ void __launch_bounds__(kTileThreads, 2) k_partition(const float* __restrict__ xyz, int64_t n, Grid g, Bins b,
                                                               int shift, const int* __restrict__ starts,
                                                               int* __restrict__ cursor, int* __restrict__ place,
                                                               float4* __restrict__ rec, const Sample* __restrict__ sample) {
  if (crowded(sample)) return;
  extern __shared__ __align__(16) float4 stage[];  // [kTile]
  uint8_t* which = reinterpret_cast<uint8_t*>(stage + kTile);  // [kTile] bucket of a staged record
  __shared__ int cnt[kBuckets], loc[kBuckets], delta[kBuckets];
  const int tid = threadIdx.x;
  const int64_t i0 = blockIdx.x * (int64_t)kTile;
  const int m = (int)(n - i0 < kTile ? n - i0 : kTile);
  if (tid < kBuckets) cnt[tid] = 0;
  __syncthreads();
  float p[kTile / kTileThreads][3];
  int at[kTile / kTileThreads];  // bucket << 16 | rank in the block's run
#pragma unroll
  for (int u = 0; u < kTile / kTileThreads; ++u) {
    const int e = u * kTileThreads + tid;
#pragma unroll
    for (int a = 0; a < 3; ++a) p[u][a] = e < m ? __ldg(xyz + 3 * (i0 + e) + a) : 0.0f;
  }
#pragma unroll
  for (int u = 0; u < kTile / kTileThreads; ++u) {
    if (u * kTileThreads + tid >= m) continue;
    const int k = point_bin(g, b, p[u][0], p[u][1], p[u][2]) >> shift;
    at[u] = k << 16 | atomicAdd(cnt + k, 1);
  }
  __syncthreads();
  int got = 0;
  if (tid < kBuckets && cnt[tid] > 0) got = __ldg(starts + ((int64_t)tid << shift)) + atomicAdd(cursor + tid, cnt[tid]);
  scan_counts(cnt, loc, kBuckets);
  if (tid < kBuckets) delta[tid] = got - loc[tid];
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kTile / kTileThreads; ++u) {
    const int e = u * kTileThreads + tid;
    if (e >= m) continue;
    const int k = at[u] >> 16, l = loc[k] + (at[u] & 0xffff);
    stage[l] = make_float4(p[u][0], p[u][1], p[u][2], 0.0f);
    which[l] = (uint8_t)k;
    place[i0 + e] = delta[k] + l;
  }
  __syncthreads();
  for (int e = tid; e < m; e += kTileThreads) rec[delta[which[e]] + e] = stage[e];
}

// One bucket's tile of records into brick order, each with its place k. The block finds its tile from
// the buckets' sizes.
__global__ void __launch_bounds__(kTileThreads, 2) k_brick_order(const float4* __restrict__ rec, Grid g, Bins b, int shift,
                                                              int nbuckets, const int* __restrict__ starts,
                                                              int* __restrict__ cursor, float4* __restrict__ out,
                                                              const Sample* __restrict__ sample) {
  if (crowded(sample)) return;
  extern __shared__ __align__(16) float4 stage[];  // [kTile]
  uint16_t* which = reinterpret_cast<uint16_t*>(stage + kTile);  // [kTile] bin of a staged record
  int* hist = reinterpret_cast<int*>(which + kTile);              // [2^shift] counts, then deltas
  __shared__ int range[2], bucket, part[kBuckets / 32];
  const int tid = threadIdx.x, lane = tid & 31, nbins = (int)b.total(), width = 1 << shift;
  int* loc = hist + width;                                        // [2^shift]
  if (tid == 0) bucket = -1;
  __syncthreads();
  int s0 = 0, tiles = 0, inc = 0;
  if (tid < kBuckets) {
    if (tid < nbuckets) {
      s0 = __ldg(starts + ((int64_t)tid << shift));
      const int s1 = __ldg(starts + min((int64_t)(tid + 1) << shift, (int64_t)nbins));
      tiles = (s1 - s0 + kTile - 1) / kTile;
    }
    inc = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    if (lane == 31) part[tid >> 5] = inc;
  }
  __syncthreads();
  if (tid < kBuckets) {
    for (int w = 0; w < (tid >> 5); ++w) inc += part[w];
    const int first = inc - tiles;
    if ((int)blockIdx.x >= first && (int)blockIdx.x < inc) {
      bucket = tid;
      range[0] = s0 + ((int)blockIdx.x - first) * kTile;
      range[1] = min(range[0] + kTile, __ldg(starts + min((int64_t)(tid + 1) << shift, (int64_t)nbins)));
    }
  }
  __syncthreads();
  if (bucket < 0) return;
  const int bin0 = bucket << shift, k0 = range[0], k1 = range[1];
  for (int i = tid; i < width; i += kTileThreads) hist[i] = 0;
  __syncthreads();
  float4 q[kTile / kTileThreads];
  int bin[kTile / kTileThreads], rank[kTile / kTileThreads];
#pragma unroll
  for (int u = 0; u < kTile / kTileThreads; ++u) {
    const int k = k0 + u * kTileThreads + tid;
    q[u] = k < k1 ? __ldg(rec + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
#pragma unroll
  for (int u = 0; u < kTile / kTileThreads; ++u) {
    if (k0 + u * kTileThreads + tid >= k1) continue;
    bin[u] = point_bin(g, b, q[u].x, q[u].y, q[u].z) - bin0;
    rank[u] = atomicAdd(hist + bin[u], 1);
  }
  __syncthreads();
  scan_counts(hist, loc, width);
  for (int i = tid; i < width; i += kTileThreads)
    if (hist[i] > 0) hist[i] = __ldg(starts + bin0 + i) + atomicAdd(cursor + bin0 + i, hist[i]) - loc[i];
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kTile / kTileThreads; ++u) {
    const int k = k0 + u * kTileThreads + tid;
    if (k >= k1) continue;
    const int l = loc[bin[u]] + rank[u];
    stage[l] = make_float4(q[u].x, q[u].y, q[u].z, __int_as_float(k));
    which[l] = (uint16_t)bin[u];
  }
  __syncthreads();
  for (int e = tid; e < k1 - k0; e += kTileThreads) out[hist[which[e]] + e] = stage[e];
}

// A record's SDF (of the corner values where the cells agree), normal and gradient: one 32-byte store, so the
// sector is written whole.
__device__ __forceinline__ void store_normals(const float* f, const Grid& g, const Tri& t, const Eq7& e,
                                              const float (&c)[8], const float (&gr)[3], int want_sdf, int want_normal,
                                              float4* to) {
  float s = 0.0f, nn[3] = {0.0f, 0.0f, 0.0f}, len;
  if (want_sdf) {
    if (t.inb == 0xffu && t.x0 == e.x0 && t.y0 == e.y0 && t.z0 == e.z0) {
#pragma unroll
      for (int k = 0; k < 8; ++k) s = fmaf(c[k], t.w[k], s);
    } else {
      s = gs_sample(f, g, t);
    }
  }
  if (want_normal) normalize_eps(gr, nn, len);
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(to), "f"(nn[0]), "f"(nn[1]), "f"(nn[2]),
               "f"(s), "f"(gr[0]), "f"(gr[1]), "f"(gr[2]), "f"(0.0f)
               : "memory");
}

// One chunk of a brick per block: 34 KB of voxels and at most 64 registers keep four blocks or more on an SM,
// one staging while others compute. 2^24 points: 536 us with normals (1.74 ms in Morton order through L1),
// 270 us without (1.08 ms). kNormals: the results of the record with place k go to res[2 k] = (normal,
// sdf) and res[2 k + 1] = (gradient, 0), one 32-byte sector; otherwise its SDF to sdf[k].
template <bool kNormals>
__global__ void __launch_bounds__(kQueryThreads, kNormals ? 4 : 6)
    k_brick_query(const float* __restrict__ f, Grid g, Bins b, int vec, const int* __restrict__ starts,
                  const int* __restrict__ nchunks, const int2* __restrict__ list, const float4* __restrict__ rec,
                  float4* __restrict__ res, int want_sdf, int want_normal, float* __restrict__ sdf) {
  __shared__ __align__(16) float vox[kReg * kReg * kPitch];
  if ((int)blockIdx.x >= __ldg(nchunks)) return;
  const int tid = threadIdx.x;
  const int2 item = __ldg(list + blockIdx.x);
  const int bz = item.x % b.n[2], by = item.x / b.n[2] % b.n[1], bx = item.x / b.n[2] / b.n[1];
  const int end = min(item.y + kChunk, __ldg(starts + item.x + 1));
  // the brick's voxels, clipped to the grid
  const int x_lo = max(bx * kBrick - 1, 0), y_lo = max(by * kBrick - 1, 0);
  const int z_lo = max(bz * kBrick - 1, 0) & (vec ? ~3 : ~0);
  const int x_n = min(bx * kBrick + kBrick + 1, g.rx - 1) - x_lo + 1;
  const int y_n = min(by * kBrick + kBrick + 1, g.ry - 1) - y_lo + 1;
  const int z_n = min(bz * kBrick + kBrick + 1, g.rz - 1) - z_lo + 1;
  const float* src = f + lin3(g, x_lo, y_lo, z_lo);
  if (vec) {  // grid rows of whole float4, 6 a row (the last may run past the region, inside the grid's row)
    for (int e = tid; e < x_n * kReg * (kPitch / 4); e += kQueryThreads) {
      const int c4 = 4 * (e % (kPitch / 4)), r = e / (kPitch / 4), y = r % kReg, x = r / kReg;
      if (y < y_n && c4 < z_n)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(vox + r * kPitch + c4)),
                     "l"(src + (x * g.ry + y) * g.rz + c4)
                     : "memory");
    }
  } else {
    for (int e = tid; e < x_n * kReg * kReg; e += kQueryThreads) {
      const int z = e % kReg, r = e / kReg, y = r % kReg, x = r / kReg;
      if (y < y_n && z < z_n)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(vox + r * kPitch + z)),
                     "l"(src + (x * g.ry + y) * g.rz + z)
                     : "memory");
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  for (int j = item.y + tid; j < end; j += kQueryThreads) {
    const float4 q = __ldg(rec + j);
    const int64_t at = __float_as_int(q.w);
    Tri t;
    gs_setup(g, q.x, q.y, q.z, t);
    // the whole stencil lies in the region and in the grid
    const bool in_t = t.inb == 0xffu && t.x0 >= x_lo && t.y0 >= y_lo && t.z0 >= z_lo && t.x0 + 1 < x_lo + x_n &&
                      t.y0 + 1 < y_lo + y_n && t.z0 + 1 < z_lo + z_n;
    if (!kNormals) {
      float s = 0.0f;
      if (in_t) {
        const float* p = vox + ((t.x0 - x_lo) * kReg + (t.y0 - y_lo)) * kPitch + (t.z0 - z_lo);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          s = fmaf(p[((k & 4) ? kReg * kPitch : 0) + ((k & 2) ? kPitch : 0) + (k & 1)], t.w[k], s);
      } else {
        s = gs_sample(f, g, t);
      }
      sdf[at] = s;
      continue;
    }
    Eq7 e;
    eq7_setup(g, q.x, q.y, q.z, e);
    float w[8], c[8], gr[3] = {0.0f, 0.0f, 0.0f};
    eq7_weights(e, w);
    const bool in = e.x0 >= 1 && e.y0 >= 1 && e.z0 >= 1 && e.x0 + 2 < g.rx && e.y0 + 2 < g.ry && e.z0 + 2 < g.rz &&
                    e.x0 - 1 >= x_lo && e.y0 - 1 >= y_lo && e.z0 - 1 >= z_lo && e.x0 + 2 < x_lo + x_n &&
                    e.y0 + 2 < y_lo + y_n && e.z0 + 2 < z_lo + z_n;
    bool done = false;
    if (in) {
      constexpr int sx = kReg * kPitch, sy = kPitch;
      const float* p = vox + (e.x0 - x_lo) * sx + (e.y0 - y_lo) * sy + (e.z0 - z_lo);
#pragma unroll
      for (int k = 0; k < 8; ++k) c[k] = p[((k & 4) ? sx : 0) + ((k & 2) ? sy : 0) + (k & 1)];
      done = g.fd_r[0] != 0.0f && eq7_gradient_columns(p, sx, sy, g, w, c, gr);
    }
    if (!done) {
      eq7_load_block(f, g, e, c);
      eq7_gradient_block(f, g, e, w, c, gr);
    }
    store_normals(f, g, t, e, c, gr, want_sdf, want_normal, res + 2 * at);
  }
}

// A pass's outputs, null where not asked for.
struct PointOut {
  float *sdf, *grad, *normal;
};

// The records of bricks with fewer than `dense` points, a thread each, from the grid itself: staging a brick
// costs 34 KB of reads. Crowded points: all of them, from xyz to the caller's outputs.
template <bool kNormals>
__global__ void __launch_bounds__(256) k_sparse_query(const float* __restrict__ f, Grid g, Bins b, int dense,
                                                      const int* __restrict__ starts, const float4* __restrict__ rec,
                                                      int64_t n, float4* __restrict__ res, int want_sdf, int want_normal,
                                                      float* __restrict__ sdf, const Sample* __restrict__ sample,
                                                      const float* __restrict__ xyz, PointOut out) {
  if (crowded(sample)) {
    for (int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
      const float px = __ldg(xyz + 3 * i), py = __ldg(xyz + 3 * i + 1), pz = __ldg(xyz + 3 * i + 2);
      if (!kNormals) {
        out.sdf[i] = query_sdf(f, g, px, py, pz);
        continue;
      }
      Eq7 e;
      eq7_setup(g, px, py, pz, e);
      float w[8], c[8], gr[3], nn[3], len;
      eq7_load_block(f, g, e, c);
      if (out.sdf) out.sdf[i] = query_sdf_block(f, g, px, py, pz, e, c);
      eq7_weights(e, w);
      eq7_gradient_block(f, g, e, w, c, gr);
      normalize_eps(gr, nn, len);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (out.grad) out.grad[3 * i + a] = gr[a];
        if (out.normal) out.normal[3 * i + a] = nn[a];
      }
    }
    return;
  }
  if (dense <= 1) return;
  for (int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
    const float4 q = __ldg(rec + i);
    const int bin = point_bin(g, b, q.x, q.y, q.z);
    if (__ldg(starts + bin + 1) - __ldg(starts + bin) >= dense) continue;
    const int64_t at = __float_as_int(q.w);
    Tri t;
    gs_setup(g, q.x, q.y, q.z, t);
    if (!kNormals) {
      sdf[at] = gs_sample(f, g, t);
      continue;
    }
    Eq7 e;
    eq7_setup(g, q.x, q.y, q.z, e);
    float w[8], c[8], gr[3];
    eq7_weights(e, w);
    eq7_load_block(f, g, e, c);
    eq7_gradient_block(f, g, e, w, c, gr);
    store_normals(f, g, t, e, c, gr, want_sdf, want_normal, res + 2 * at);
  }
}

// Each point's results from its place.
template <bool kNormals>
__global__ void __launch_bounds__(256) k_collect(const int* __restrict__ place, int64_t n, const float4* __restrict__ res,
                                                 const float* __restrict__ s, PointOut out,
                                                 const Sample* __restrict__ sample) {
  if (crowded(sample)) return;
  float *sdf = out.sdf, *grad = out.grad, *normal = out.normal;
  constexpr int kPer = 4;  // points a thread, their loads in flight together
  for (int64_t i0 = blockIdx.x * (int64_t)(256 * kPer) + threadIdx.x; i0 < n; i0 += (int64_t)gridDim.x * 256 * kPer) {
    int64_t k[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) k[u] = i0 + 256 * u < n ? __ldg(place + i0 + 256 * u) : 0;
    float4 a[kPer], b[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      if (!kNormals) {
        a[u].w = __ldg(s + k[u]);
      } else {
        if (sdf || normal) a[u] = __ldg(res + 2 * k[u]);
        if (grad) b[u] = __ldg(res + 2 * k[u] + 1);
      }
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int64_t i = i0 + 256 * u;
      if (i >= n) break;
      if (!kNormals || sdf) sdf[i] = a[u].w;
      if (kNormals && normal) {
        normal[3 * i] = a[u].x;
        normal[3 * i + 1] = a[u].y;
        normal[3 * i + 2] = a[u].z;
      }
      if (kNormals && grad) {
        grad[3 * i] = b[u].x;
        grad[3 * i + 1] = b[u].y;
        grad[3 * i + 2] = b[u].z;
      }
    }
  }
}

constexpr int64_t kAlign = 256;
inline int64_t align_up(int64_t b) { return (b + kAlign - 1) / kAlign * kAlign; }

// Workspace: bucket-order records (16 bytes a point) and later the results (32) in one place, brick-order
// records (16), places (4), starts, counts, cursors of bricks and buckets and the work list's length, the
// work list.
struct Layout {
  int64_t rec, place, starts, counts, cursor, list, bytes, zeroed;
};

Layout make_layout(int64_t batch, int64_t nbins) {
  Layout l;
  l.rec = align_up(batch * 32);
  l.place = l.rec + align_up(batch * 16);
  l.starts = l.place + align_up(batch * 4);
  l.counts = l.starts + align_up((nbins + 1) * 4);
  l.cursor = l.counts + align_up(nbins * 4);
  l.zeroed = align_up(nbins * 4) + (nbins + kBuckets + 3) * 4;  // counts, cursors and sample
  l.list = l.counts + align_up(l.zeroed);
  l.bytes = l.list + align_up(((nbins < batch ? nbins : batch) + batch / kChunk) * 8);
  return l;
}

}  // namespace
}  // namespace vx

using namespace vx;

extern "C" {

int64_t vx_field_query_sorted_workspace(int64_t n, const int32_t res[3]) {
  if (n <= 0 || n > INT32_MAX || !res) return 0;
  if (res[0] < 2 || res[1] < 2 || res[2] < 2) return 0;
  if (plain_grid(res)) return kAlign;
  return make_layout(n < kBatch ? n : kBatch, make_bins(res).total()).bytes;
}

int vx_field_query_sorted(const float* grid, const int32_t res[3], const float xyz_min[3], const float xyz_max[3],
                          const float* xyz, int64_t n, float* sdf, float* grad, float* normal, void* workspace,
                          int64_t workspace_bytes, void* stream) {
  if (int s = check_grid(res)) return s;
  VX_REQUIRE(n >= 0 && n <= INT32_MAX, "n out of range (0 .. 2^31-1)");
  if (n == 0 || (!sdf && !grad && !normal)) return VX_OK;
  VX_REQUIRE(grid && xyz && xyz_min && xyz_max && workspace, "null pointer");
  const int64_t need = vx_field_query_sorted_workspace(n, res);
  VX_REQUIRE(need > 0, "sort workspace size query failed");
  VX_REQUIRE(workspace_bytes >= need, "workspace holds %lld bytes, need %lld", (long long)workspace_bytes,
             (long long)need);
  VX_REQUIRE(((uintptr_t)workspace & (kAlign - 1)) == 0, "workspace must be 256-byte aligned");
  if (plain_grid(res))
    return vx_field_query(grid, res, xyz_min, xyz_max, xyz, n, sdf, grad, normal, nullptr, nullptr, stream);
  const Bins b = make_bins(res);
  const int64_t nbins = b.total();
  Grid g = make_grid(res, xyz_min, xyz_max);
  const Layout l = make_layout(n < kBatch ? n : kBatch, nbins);
  char* w = static_cast<char*>(workspace);
  float4* res0 = reinterpret_cast<float4*>(w);  // bucket-order records, then the results
  float4* rec = reinterpret_cast<float4*>(w + l.rec);
  int* place = reinterpret_cast<int*>(w + l.place);
  int* starts = reinterpret_cast<int*>(w + l.starts);
  int* counts = reinterpret_cast<int*>(w + l.counts);
  int* cursor = reinterpret_cast<int*>(w + l.cursor);  // [nbins] bricks, [kBuckets], the work list's length
  int* nchunks = cursor + nbins + kBuckets;
  Sample* sample = reinterpret_cast<Sample*>(nchunks + 1);
  int2* list = reinterpret_cast<int2*>(w + l.list);
  const bool normals = grad || normal;
  const int vec = res[2] % 4 == 0 && (reinterpret_cast<uintptr_t>(grid) & 15) == 0;
  const int shift = bucket_shift(nbins);
  const int nbuckets = (int)((nbins - 1) >> shift) + 1;
  const size_t count_smem = nbins <= kSmemBins ? (size_t)nbins * 4 : 0, order_smem = order_bytes(shift);
  constexpr int part_smem = kTile * 17;
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaFuncSetAttribute(k_bin_count<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBins * 4);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_brick_order, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)order_bytes(bucket_shift(kMaxBins)));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_partition, cudaFuncAttributeMaxDynamicSharedMemorySize, part_smem);
  int launches = 0;
  for (int64_t i0 = 0; i0 < n && e == cudaSuccess; i0 += kBatch) {
    const int64_t m = n - i0 < kBatch ? n - i0 : kBatch;
    const float* p = xyz + 3 * i0;
    e = cudaMemsetAsync(counts, 0, (size_t)l.zeroed, st);
    if (e != cudaSuccess) break;
    const unsigned tiles = (unsigned)((m + kTile - 1) / kTile);
    const int dense = m < (int64_t)kDenseMean * nbins ? (normals ? kDenseNormals : kDenseSdf) : 1;
    if (count_smem)
      k_bin_count<true><<<tiles < kSMs ? tiles : kSMs, kCountThreads, count_smem, st>>>(p, m, g, b, counts, sample);
    else
      k_bin_count<false><<<grid_for(m, kCountThreads, 2), kCountThreads, 0, st>>>(p, m, g, b, counts, sample);
    k_bin_scan<<<(unsigned)((nbins + kScanBins - 1) / kScanBins), 1024, 0, st>>>(counts, nbins, dense, starts, nchunks,
                                                                               list, sample);
    k_partition<<<tiles, kTileThreads, part_smem, st>>>(p, m, g, b, shift, starts, cursor + nbins, place, res0, sample);
    k_brick_order<<<tiles + nbuckets, kTileThreads, order_smem, st>>>(res0, g, b, shift, nbuckets, starts, cursor, rec,
                                                                             sample);
    launches += 6;
    e = cudaGetLastError();  // what follows stores at the places that these four wrote
    if (e != cudaSuccess) break;
    // at least the work list's length
    const unsigned blocks = (unsigned)((nbins < m / dense ? nbins : m / dense) + m / kChunk);
    const PointOut out{sdf ? sdf + i0 : nullptr, grad ? grad + 3 * i0 : nullptr, normal ? normal + 3 * i0 : nullptr};
    float* s = reinterpret_cast<float*>(res0);
    if (normals) {
      if (blocks)
        k_brick_query<true><<<blocks, kQueryThreads, 0, st>>>(grid, g, b, vec, starts, nchunks, list, rec, res0,
                                                              sdf != nullptr, normal != nullptr, nullptr);
      k_sparse_query<true><<<grid_for(m, 256), 256, 0, st>>>(grid, g, b, dense, starts, rec, m, res0, sdf != nullptr,
                                                             normal != nullptr, nullptr, sample, p, out);
      k_collect<true><<<grid_for(m, 256), 256, 0, st>>>(place, m, res0, nullptr, out, sample);
    } else {
      if (blocks)
        k_brick_query<false><<<blocks, kQueryThreads, 0, st>>>(grid, g, b, vec, starts, nchunks, list, rec, nullptr, 1, 0,
                                                               s);
      k_sparse_query<false><<<grid_for(m, 256), 256, 0, st>>>(grid, g, b, dense, starts, rec, m, nullptr, 1, 0, s, sample,
                                                              p, out);
      k_collect<false><<<grid_for(m, 256), 256, 0, st>>>(place, m, nullptr, s, out, sample);
    }
    launches += 1;
  }
  if (e != cudaSuccess) return set_error(VX_ERR_CUDA, "field_query_sorted: %s", cudaGetErrorString(e));
  count_launches(launches);
  return check_launch("field_query_sorted");
}

}  // extern "C"
