// Closed-form eikonal (Eq.10-11, regularization/eikonal.py:13-171) and Laplacian curvature
// (Eq.12-14, regularization/curvature.py:13-165) gradients written straight into the grid
// gradient.
//
// Two forms:
//  * list form (the reference's kernel interface, eikonal_grad.cu / curvature_grad.cu):
//    one thread per listed vertex, atomics into the gradient, scale 2/|list|;
//  * fused gather form for the training step: one pass over 32x4x4 voxel tiles of the
//    grid, skipping tiles with no active vertex. Each output voxel sums, in a fixed order, the
//    contributions of the <= 7 active interior vertices whose stencil touches it (itself
//    and its 6 face neighbours) and is added to the gradient once: the result is
//    deterministic. The active set is the V_R bitmap with the relax and narrow-band
//    predicates, and |V_R| comes from the device-side counts.
// Both forms also reduce the monitoring losses (mean over interior vertices) through partials.
#include <cooperative_groups.h>

#include "common.cuh"

namespace vx {

struct RegOut {
  double* partials;       // 3 per block: eikonal sum, curvature sum, interior count
  unsigned int* counter;  // zero before the first launch; reset by the last block
  float* losses;          // [eikonal, curvature]
};

__device__ void reduce_losses(const RegOut& o, double e, double c, double n) {
  __shared__ double s[3][32];
  __shared__ bool is_last;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nthreads = blockDim.x * blockDim.y * blockDim.z;
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int wl = tid & 31, ww = tid >> 5;
  (void)lane;
  (void)warp;
  e = warp_sum_d(e);
  c = warp_sum_d(c);
  n = warp_sum_d(n);
  if (wl == 0) {
    s[0][ww] = e;
    s[1][ww] = c;
    s[2][ww] = n;
  }
  __syncthreads();
  const unsigned nblocks = gridDim.x * gridDim.y * gridDim.z;
  const unsigned bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  if (tid == 0) {
    double a = 0, b = 0, k = 0;
    for (int w = 0; w < (nthreads + 31) / 32; ++w) {
      a += s[0][w];
      b += s[1][w];
      k += s[2][w];
    }
    o.partials[3 * bid] = a;
    o.partials[3 * bid + 1] = b;
    o.partials[3 * bid + 2] = k;
    __threadfence();
    is_last = (atomicAdd(o.counter, 1u) == nblocks - 1);
  }
  __syncthreads();
  if (!is_last) return;
  // last block: every thread sums a fixed strided subset, then a fixed-order warp/block tree
  // (deterministic for a given launch shape)
  __threadfence();
  const volatile double* p = o.partials;
  double a = 0, b = 0, k = 0;
  for (unsigned i = tid; i < nblocks; i += nthreads) {
    a += p[3 * i];
    b += p[3 * i + 1];
    k += p[3 * i + 2];
  }
  a = warp_sum_d(a);
  b = warp_sum_d(b);
  k = warp_sum_d(k);
  __syncthreads();
  if (wl == 0) {
    s[0][ww] = a;
    s[1][ww] = b;
    s[2][ww] = k;
  }
  __syncthreads();
  if (tid == 0) {
    a = b = k = 0;
    for (int w = 0; w < (nthreads + 31) / 32; ++w) {
      a += s[0][w];
      b += s[1][w];
      k += s[2][w];
    }
    if (o.losses) {
      o.losses[0] = k > 0 ? (float)(a / k) : 0.0f;
      o.losses[1] = k > 0 ? (float)(b / k) : 0.0f;
    }
    *o.counter = 0u;
  }
}

// ------------------------------------ list form --------------------------------------------

__global__ void __launch_bounds__(256) k_eikonal_list(const float* __restrict__ f, Grid g,
                                                      const int64_t* __restrict__ verts, int64_t nv,
                                                      float* __restrict__ gg, float weight, RegOut o) {
  double e = 0, n = 0;
  const float dx = 2.0f * g.eps[0], dy = 2.0f * g.eps[1], dz = 2.0f * g.eps[2];
  const int nblk = gridDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nv; i += (int64_t)nblk * blockDim.x) {
    const int64_t vx_ = verts[3 * i], vy_ = verts[3 * i + 1], vz_ = verts[3 * i + 2];
    if (vx_ <= 0 || vx_ >= g.rx - 1 || vy_ <= 0 || vy_ >= g.ry - 1 || vz_ <= 0 || vz_ >= g.rz - 1) continue;
    const int x = (int)vx_, y = (int)vy_, z = (int)vz_;
    const float nx = (__ldg(f + lin3(g, x + 1, y, z)) - __ldg(f + lin3(g, x - 1, y, z))) / dx;
    const float ny = (__ldg(f + lin3(g, x, y + 1, z)) - __ldg(f + lin3(g, x, y - 1, z))) / dy;
    const float nz = (__ldg(f + lin3(g, x, y, z + 1)) - __ldg(f + lin3(g, x, y, z - 1))) / dz;
    const float len = sqrtf(nx * nx + ny * ny + nz * nz);
    const float scale = (2.0f / (float)nv) * (1.0f - 1.0f / (len + 1e-8f)) * weight;
    const float ax = scale * nx, ay = scale * ny, az = scale * nz;
    if (gg) {
      atomicAdd(gg + lin3(g, x + 1, y, z), ax / dx);
      atomicAdd(gg + lin3(g, x - 1, y, z), -ax / dx);
      atomicAdd(gg + lin3(g, x, y + 1, z), ay / dy);
      atomicAdd(gg + lin3(g, x, y - 1, z), -ay / dy);
      atomicAdd(gg + lin3(g, x, y, z + 1), az / dz);
      atomicAdd(gg + lin3(g, x, y, z - 1), -az / dz);
    }
    const double l = sqrt((double)nx * nx + (double)ny * ny + (double)nz * nz + 1e-16);
    e += (l - 1.0) * (l - 1.0);
    n += 1.0;
  }
  reduce_losses(o, e, 0.0, n);
}

__global__ void __launch_bounds__(256) k_curvature_list(const float* __restrict__ f, Grid g,
                                                        const int64_t* __restrict__ verts, int64_t nv,
                                                        float* __restrict__ gg, float weight, RegOut o) {
  double c = 0, n = 0;
  const float ex2 = g.eps[0] * g.eps[0], ey2 = g.eps[1] * g.eps[1], ez2 = g.eps[2] * g.eps[2];
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nv; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t vx_ = verts[3 * i], vy_ = verts[3 * i + 1], vz_ = verts[3 * i + 2];
    if (vx_ <= 0 || vx_ >= g.rx - 1 || vy_ <= 0 || vy_ >= g.ry - 1 || vz_ <= 0 || vz_ >= g.rz - 1) continue;
    const int x = (int)vx_, y = (int)vy_, z = (int)vz_;
    const float fc = __ldg(f + lin3(g, x, y, z));
    const float Lx = (__ldg(f + lin3(g, x + 1, y, z)) + __ldg(f + lin3(g, x - 1, y, z)) - 2.0f * fc) / ex2;
    const float Ly = (__ldg(f + lin3(g, x, y + 1, z)) + __ldg(f + lin3(g, x, y - 1, z)) - 2.0f * fc) / ey2;
    const float Lz = (__ldg(f + lin3(g, x, y, z + 1)) + __ldg(f + lin3(g, x, y, z - 1)) - 2.0f * fc) / ez2;
    const float scale = (2.0f / (float)nv) * weight;
    if (gg) {
      atomicAdd(gg + lin3(g, x, y, z), scale * (-2.0f * Lx / ex2 - 2.0f * Ly / ey2 - 2.0f * Lz / ez2));
      atomicAdd(gg + lin3(g, x + 1, y, z), scale * (Lx / ex2));
      atomicAdd(gg + lin3(g, x - 1, y, z), scale * (Lx / ex2));
      atomicAdd(gg + lin3(g, x, y + 1, z), scale * (Ly / ey2));
      atomicAdd(gg + lin3(g, x, y - 1, z), scale * (Ly / ey2));
      atomicAdd(gg + lin3(g, x, y, z + 1), scale * (Lz / ez2));
      atomicAdd(gg + lin3(g, x, y, z - 1), scale * (Lz / ez2));
    }
    c += (double)Lx * Lx + (double)Ly * Ly + (double)Lz * Lz;
    n += 1.0;
  }
  reduce_losses(o, 0.0, c, n);
}

// ------------------------------------ gather form ------------------------------------------

constexpr int TZ = 32, TY = 4, TX = 4;  // output tile (z fastest)
constexpr int MY = TY + 2, MX = TX + 2;  // halo-1 box extents in y and x

struct StencilArgs {
  const float* f;
  const uint32_t* fb;  // filtered V_R bitmaps from vx_vr_count: [bits & band | bits & band & relax]
  int64_t nwords;
  Grid g;
  const unsigned long long* counts;  // from vx_vr_count
  float relax_r;
  float w_eik, w_curv;
  float* gg;
  int tiles_z, tiles_y, tiles_x;
};

__device__ __forceinline__ void tile_origin(const StencilArgs& a, int t, int& x0, int& y0, int& z0) {
  const int tz = t % a.tiles_z;
  const int ty = (t / a.tiles_z) % a.tiles_y;
  const int tx = t / (a.tiles_z * a.tiles_y);
  z0 = tz * TZ;
  y0 = ty * TY;
  x0 = tx * TX;
}

struct StencilConsts {
  float inv_nv, dx, dy, dz, ex2, ey2, ez2, sc, w_eik;
};

// What active vertex (x, y, z) adds to its face neighbours: e[a] + c[a] to v + e_a and c[a] - e[a] to v - e_a
// (eikonal e = scale n_a / (2 eps_a), curvature c = scale L_a / eps_a^2), and -2 (c[0] + c[1] + c[2]) to
// itself, with scale = 2/|V_R| (1 - 1/(|n| + 1e-8)) w_eik and sc = 2/|V_R| w_curv (eikonal_grad.cu,
// curvature_grad.cu); also its two loss terms.
__device__ __forceinline__ void vertex_terms(const StencilArgs& a, const StencilConsts& k, int x, int y, int z,
                                             float e[3], float c[3], double* loss) {
  const float* f = a.f + lin3(a.g, x, y, z);
  const int sx = a.g.ry * a.g.rz, sy = a.g.rz;
  const float fc = __ldg(f);
  const float fxp = __ldg(f + sx), fxm = __ldg(f - sx);
  const float fyp = __ldg(f + sy), fym = __ldg(f - sy);
  const float fzp = __ldg(f + 1), fzm = __ldg(f - 1);
  const float Lx = (fxp + fxm - 2.0f * fc) / k.ex2;
  const float Ly = (fyp + fym - 2.0f * fc) / k.ey2;
  const float Lz = (fzp + fzm - 2.0f * fc) / k.ez2;
  const float nx = (fxp - fxm) / k.dx, ny = (fyp - fym) / k.dy, nz = (fzp - fzm) / k.dz;
  const float len = sqrtf(nx * nx + ny * ny + nz * nz);
  const float se = k.inv_nv * (1.0f - 1.0f / (len + 1e-8f)) * k.w_eik;
  e[0] = (se * nx) / k.dx;
  e[1] = (se * ny) / k.dy;
  e[2] = (se * nz) / k.dz;
  c[0] = k.sc * (Lx / k.ex2);
  c[1] = k.sc * (Ly / k.ey2);
  c[2] = k.sc * (Lz / k.ez2);
  if (loss) {
    const double l = sqrt((double)nx * nx + (double)ny * ny + (double)nz * nz + 1e-16);
    loss[0] += (l - 1.0) * (l - 1.0);
    loss[1] += (double)Lx * Lx + (double)Ly * Ly + (double)Lz * Lz;
    loss[2] += 1.0;
  }
}

// V_R bits of the vertices (x, y, z0 - 1 .. z0 + 32) of one grid column as bits 0..33 of a word
// pair (vertices outside the interior read 0).
__device__ __forceinline__ uint64_t column_window(const StencilArgs& a, const uint32_t* __restrict__ bm, int x, int y,
                                                  int z0) {
  if (x < 1 || x > a.g.rx - 2 || y < 1 || y > a.g.ry - 2) return 0ull;
  const int64_t b = (int64_t)lin3(a.g, x, y, z0) - 1;  // bit of vertex z0 - 1 (may precede the column)
  const int64_t w0 = b >> 5;
  const int s = (int)(b & 31);
  const uint32_t u0 = (w0 >= 0 && w0 < a.nwords) ? __ldg(bm + w0) : 0u;
  const uint32_t u1 = (w0 + 1 < a.nwords) ? __ldg(bm + w0 + 1) : 0u;
  const uint32_t u2 = (s > 0 && w0 + 2 < a.nwords) ? __ldg(bm + w0 + 2) : 0u;
  uint64_t v = ((uint64_t)u1 << 32 | u0) >> s;
  if (s > 0) v |= (uint64_t)u2 << (64 - s);
  // keep interior z only: z = z0 - 1 + k in [1, rz - 2]
  const int klo = max(0, 2 - z0), khi = min(33, a.g.rz - 1 - z0);
  if (khi < klo) return 0ull;
  const uint64_t keep = ((khi >= 63 ? ~0ull : ((1ull << (khi + 1)) - 1ull))) & ~((1ull << klo) - 1ull);
  return v & keep;
}

// Does tile t own a vertex of the filtered V_R set? A lane per column, two tiles a warp (its own voxels, no
// halo).
__global__ void __launch_bounds__(256) k_tile_flags(StencilArgs a, int ntiles, uint8_t* __restrict__ flags) {
  static_assert(TX * TY == 16, "half a warp a tile");
  const bool relax_on = a.relax_r > 0.0f && a.counts[1] > 0;
  const uint32_t* bm = a.fb + (relax_on ? a.nwords : 0);
  const int lane = threadIdx.x & 31, q = lane & 15;
  for (int t0 = 2 * (blockIdx.x * 8 + (threadIdx.x >> 5)); t0 < ntiles; t0 += 16 * gridDim.x) {
    const int t = t0 + (lane >> 4);
    bool hit = false;
    if (t < ntiles) {
      int x0, y0, z0;
      tile_origin(a, t, x0, y0, z0);
      const int x = x0 + q / TY, y = y0 + q % TY, z1 = min(z0 + TZ, a.g.rz) - 1;
      if (x < a.g.rx && y < a.g.ry) {
        const int b0 = lin3(a.g, x, y, z0), b1 = lin3(a.g, x, y, z1);
        for (int w = b0 >> 5; w <= (b1 >> 5); ++w) {  // 32 bits: at most two words
          uint32_t m = 0xffffffffu;
          if (w == (b0 >> 5)) m &= 0xffffffffu << (b0 & 31);
          if (w == (b1 >> 5)) m &= 0xffffffffu >> (31 - (b1 & 31));
          hit |= (__ldg(bm + w) & m) != 0u;
        }
      }
    }
    const unsigned any = __ballot_sync(0xffffffffu, hit);
    if (q == 0 && t < ntiles) flags[t] = (any >> (lane & 16) & 0xffffu) ? 1 : 0;
  }
}

// Fused eikonal + curvature gradient in gather form over 32x4x4 tiles. Block b of B owns tiles b, b + B,
// b + 2B, ...; its threads test kRegThreads of them at once against the flags of the 3x3x3 tiles around each
// (a tile's outputs need the vertices of its halo). A warp then takes every eighth tile that needs it: the
// V_R windows of the halo's columns, a compact list of their active vertices, each vertex's terms evaluated
// once (SDF through L1) and added to the tile's sums in ordered passes. A round of eight tiles lasts as long as its
// most crowded one, so the most crowded may wait for the whole block, which keeps the terms in slots and lets each
// output sum its neighbours' in a fixed order (round_limit). An output gets one addition a launch; per-cluster loss
// partials (fixed assignment and order) for k_reg_finalize. Bound by the chain of one tile (loads, ~150 instructions
// a vertex, passes): V_R is a thin band of few, unevenly filled tiles in a training step, and what a batch's samples
// touch without a band.
constexpr int kRegThreads = 256;
constexpr int kRegWarps = kRegThreads / 32;
constexpr int kHaloVerts = MX * MY * (TZ + 2);
// Costs of a tile of v vertices, in the same unit (~5 ns with every block busy): kWarpCost * v by a warp, kBlockCost + v
// by the block. With 8 full tiles a round both ways are equal at kBlockCost = 1224; 1060, 1240, 1400, 1600:
// 256^3 and 8,192 rays 38.2, 37.9, 37.4, 36.9 us; 64^3 and 2,048 rays 12.1, 12.2, 12.2, 13.1; 512^3 with every vertex
// active 5.11, 4.27, 4.26, 4.26 ms. All tiles by warps, 55, 33 us and 5.00 ms; by the block from 152 vertices on 39, 12 us
// and 5.06 ms, but 3.16 ms instead of 1.69 where 30% of 512^3 vertices are active anywhere.
constexpr int kWarpCost = 16, kBlockCost = 1400;

struct TileColumns {
  uint64_t win[MX * MY];  // bits of the columns' vertices z0 - 1 .. z0 + 32
  int off[MX * MY + 1];   // first slot of a column
};

// A tile's windows and slots, by one warp. Returns how many vertices are active.
__device__ __forceinline__ int tile_columns(const StencilArgs& a, const uint32_t* bm, int x0, int y0, int z0,
                                            TileColumns& tc, int lane) {
  // the halo's corner columns touch no output
  const bool corner = (lane / MY == 0 || lane / MY == MX - 1) && (lane % MY == 0 || lane % MY == MY - 1);
  const uint64_t w0 = corner ? 0ull : column_window(a, bm, x0 - 1 + lane / MY, y0 - 1 + lane % MY, z0);
  const uint64_t w1 = lane < MX * MY - 33 ? column_window(a, bm, x0 - 1 + (lane + 32) / MY, y0 - 1 + (lane + 32) % MY, z0) : 0ull;
  const int c0 = __popcll(w0), c1 = __popcll(w1);
  int inc = c0, inc1 = c1;  // columns 0..31, then 32..35
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o), v1 = __shfl_up_sync(0xffffffffu, inc1, o);
    if (lane >= o) {
      inc += v;
      inc1 += v1;
    }
  }
  const int first = __shfl_sync(0xffffffffu, inc, 31), total = first + __shfl_sync(0xffffffffu, inc1, 31);
  tc.win[lane] = w0;
  tc.off[lane] = inc - c0;
  if (lane < MX * MY - 32) {
    tc.win[lane + 32] = w1;
    tc.off[lane + 32] = first + inc1 - c1;
  }
  __syncwarp();
  return total;
}

// The most vertices that a tile of this round may have for a warp, v[w] being those of warp w's tile: the limit with the
// smallest sum of the longest warp and of what is left to the block, one tile after the other. By one warp.
__device__ __forceinline__ int round_limit(const int* v, int lane) {
  const int limit = lane < kRegWarps ? v[lane] : 0;
  int cost = kWarpCost * limit;
#pragma unroll
  for (int w = 0; w < kRegWarps; ++w) cost += v[w] > limit ? kBlockCost + v[w] : 0;
  const int best = __reduce_min_sync(0xffffffffu, cost);
  return __reduce_max_sync(0xffffffffu, cost == best ? limit : 0);
}

// A tile by one warp: 32 vertices at a time, their 7 terms added into the outputs' sums in 7
// ordered passes (two vertices never share a target within a pass), then the sums to the gradient. acc
// holds zeros.
__device__ __forceinline__ void tile_by_warp(const StencilArgs& a, const StencilConsts& k, int x0, int y0, int z0,
                                             const TileColumns& tc, int total, float* acc, uint16_t* list, int lane,
                                             double* loss) {
  for (int c = lane; c < MX * MY; c += 32) {
    int pos = tc.off[c];
    for (uint64_t m = tc.win[c]; m; m &= m - 1) list[pos++] = (uint16_t)(c * (TZ + 2) + __ffsll((long long)m) - 1);
  }
  __syncwarp();
  for (int s = lane; s - lane < total; s += 32) {  // whole warps
    const bool mine = s < total;
    float e[3] = {0.0f, 0.0f, 0.0f}, c[3] = {0.0f, 0.0f, 0.0f};
    int ox = -9, oy = 0, oz = 0;
    if (mine) {
      const int code = list[s], col = code / (TZ + 2), kb = code - (TZ + 2) * col;
      ox = col / MY - 1;
      oy = col % MY - 1;
      oz = kb - 1;
      const bool owned = (unsigned)ox < TX && (unsigned)oy < TY && (unsigned)oz < TZ;
      vertex_terms(a, k, x0 + ox, y0 + oy, z0 + oz, e, c, owned ? loss : nullptr);
    }
#pragma unroll
    for (int p = 0; p < 7; ++p) {
      const int ax = p == 1 ? 1 : (p == 2 ? -1 : 0), ay = p == 3 ? 1 : (p == 4 ? -1 : 0);
      const int az = p == 5 ? 1 : (p == 6 ? -1 : 0), q = p ? (p - 1) >> 1 : 0;
      const float term = p == 0 ? -2.0f * (c[0] + c[1] + c[2]) : (p & 1) ? e[q] + c[q] : c[q] - e[q];
      if ((unsigned)(ox + ax) < TX && (unsigned)(oy + ay) < TY && (unsigned)(oz + az) < TZ)
        acc[((ox + ax) * TY + oy + ay) * TZ + oz + az] += term;
      __syncwarp();
    }
  }
#pragma unroll 4
  for (int o = lane; o < TX * TY * TZ; o += 32) {
    const float v = acc[o];
    if (v != 0.0f) {
      atomicAdd(a.gg + lin3(a.g, x0 + o / (TY * TZ), y0 + o / TZ % TY, z0 + lane), v);  // its only one: no load to wait for
    }
  }
  __syncwarp();
}

// A tile by the whole block: terms into slots, then every output sums its neighbours'. term: [6][kHaloVerts].
__device__ __forceinline__ void tile_by_block(const StencilArgs& a, const StencilConsts& k, int x0, int y0, int z0,
                                              const TileColumns& tc, int total, float* term, uint16_t* list, int warp,
                                              int lane, double* loss) {
  constexpr int kWarps = kRegWarps, cap = kHaloVerts;
  for (int c = warp; c < MX * MY; c += kWarps) {
    const uint64_t w = tc.win[c];
    if (w == 0ull) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int kb = lane + 32 * h;
      if (kb < TZ + 2 && (w >> kb & 1ull)) list[tc.off[c] + __popcll(w & ((1ull << kb) - 1ull))] = (uint16_t)(c * (TZ + 2) + kb);
    }
  }
  __syncthreads();
  for (int s = 32 * warp + lane; s < total; s += 32 * kWarps) {
    const int code = list[s], col = code / (TZ + 2), kb = code - (TZ + 2) * col, cx = col / MY, cy = col % MY;
    const bool owned = cx >= 1 && cx <= TX && cy >= 1 && cy <= TY && kb >= 1 && kb <= TZ;
    float e[3], c[3];
    vertex_terms(a, k, x0 - 1 + cx, y0 - 1 + cy, z0 - 1 + kb, e, c, owned ? loss : nullptr);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      term[q * cap + s] = e[q];
      term[(3 + q) * cap + s] = c[q];
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int o = warp; o < TX * TY; o += kWarps) {  // lane = z
    const int col = (o / TY + 1) * MY + o % TY + 1;
    const uint64_t near[5] = {tc.win[col], tc.win[col - MY], tc.win[col + MY], tc.win[col - 1], tc.win[col + 1]};
    if ((near[0] | near[1] | near[2] | near[3] | near[4]) == 0ull) continue;
    const int first[5] = {tc.off[col], tc.off[col - MY], tc.off[col + MY], tc.off[col - 1], tc.off[col + 1]};
    auto slot = [&](int c, int b) {  // of vertex b of column near[c], or -1
      return (near[c] >> b & 1ull) ? first[c] + __popcll(near[c] & ((1ull << b) - 1ull)) : -1;
    };
    const int kb = lane + 1;
    float v = 0.0f;
    bool any = false;
    int q = slot(0, kb);
    if (q >= 0) {
      v = -2.0f * (term[3 * cap + q] + term[4 * cap + q] + term[5 * cap + q]);
      any = true;
    }
#pragma unroll
    for (int d = 0; d < 6; ++d) {  // the neighbour below adds e + c, the one above c - e
      const int ax = d >> 1;
      q = ax < 2 ? slot(1 + d, kb) : slot(0, (d & 1) ? kb + 1 : kb - 1);
      if (q >= 0) {
        v += (d & 1) ? term[(3 + ax) * cap + q] - term[ax * cap + q] : term[ax * cap + q] + term[(3 + ax) * cap + q];
        any = true;
      }
    }
    if (any) atomicAdd(a.gg + lin3(a.g, x0 + o / TY, y0 + o % TY, z0 + lane), v);  // its only one: no load to wait for
  }
  __syncthreads();  // the columns, the list and the terms are read
}

__global__ void __launch_bounds__(kRegThreads, 4) k_reg_stencil(StencilArgs a, const uint8_t* __restrict__ flags,
                                                             double* __restrict__ partials, int ntiles) {
  // the block's slots and their list, or the warps' sums and lists
  constexpr int kSums = kRegWarps * TX * TY * TZ, kSlots = 6 * kHaloVerts;
  __shared__ float term[kSums + kRegWarps * kHaloVerts / 2];
  static_assert(kSlots + kHaloVerts / 2 <= kSums + kRegWarps * kHaloVerts / 2 && kHaloVerts % 2 == 0, "slots and list");
  uint16_t* list = reinterpret_cast<uint16_t*>(term + kSlots);
  __shared__ TileColumns cols[kRegWarps];
  __shared__ int queue[kRegThreads], verts[kRegWarps];  // tiles to do; vertices of the warps' tiles
  __shared__ int qcount[kRegWarps];
  __shared__ double red[3][kRegWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool relax_on = a.relax_r > 0.0f && a.counts[1] > 0;
  const uint32_t* bm = a.fb + (relax_on ? a.nwords : 0);
  // |V_R| after the filters: counts[3] (relax) / counts[2] (no relax); the filtered bitmaps
  // already carry the band, so the band count is the one to use
  const unsigned long long nv = relax_on ? a.counts[3] : a.counts[2];
  StencilConsts k;
  k.inv_nv = nv > 0 ? 2.0f / (float)nv : 0.0f;
  k.dx = 2.0f * a.g.eps[0];
  k.dy = 2.0f * a.g.eps[1];
  k.dz = 2.0f * a.g.eps[2];
  k.ex2 = a.g.eps[0] * a.g.eps[0];
  k.ey2 = a.g.eps[1] * a.g.eps[1];
  k.ez2 = a.g.eps[2] * a.g.eps[2];
  k.sc = k.inv_nv * a.w_curv;
  k.w_eik = a.w_eik;
  double loss[3] = {0.0, 0.0, 0.0};
  const int nblk = gridDim.x;
  for (int64_t base = blockIdx.x; base < ntiles; base += (int64_t)nblk * kRegThreads) {
    const int64_t tl = base + (int64_t)tid * nblk;
    bool need = false;
    if (tl < ntiles) {
      const int t = (int)tl, tz = t % a.tiles_z, ty = (t / a.tiles_z) % a.tiles_y, tx = t / (a.tiles_z * a.tiles_y);
      for (int dx = -1; dx <= 1; ++dx)
        for (int dy = -1; dy <= 1; ++dy)
          for (int dz = -1; dz <= 1; ++dz) {
            const int nx = tx + dx, ny = ty + dy, nz = tz + dz;
            if (nx < 0 || nx >= a.tiles_x || ny < 0 || ny >= a.tiles_y || nz < 0 || nz >= a.tiles_z) continue;
            need |= __ldg(flags + ((int64_t)nx * a.tiles_y + ny) * a.tiles_z + nz) != 0;
          }
    }
    const unsigned votes = __ballot_sync(0xffffffffu, need);
    if (lane == 0) qcount[warp] = __popc(votes);
    __syncthreads();
    int at = __popc(votes & ((1u << lane) - 1u)), todo = 0;
#pragma unroll
    for (int w = 0; w < kRegWarps; ++w) {
      if (w < warp) at += qcount[w];
      todo += qcount[w];
    }
    if (need) queue[at] = (int)tl;
    __syncthreads();
    for (int n0 = 0; n0 < todo; n0 += kRegWarps) {  // a tile a warp, then the most crowded ones of them
      const int n = n0 + warp;
      int x0, y0, z0, total = 0;
      if (n < todo) {
        tile_origin(a, queue[n], x0, y0, z0);
        total = tile_columns(a, bm, x0, y0, z0, cols[warp], lane);
      }
      if (lane == 0) verts[warp] = total;
      __syncthreads();
      const int limit = round_limit(verts, lane);
      if (total > 0 && total <= limit) {
        float* acc = term + TX * TY * TZ * warp;
        for (int o = lane; o < TX * TY * TZ; o += 32) acc[o] = 0.0f;
        __syncwarp();
        tile_by_warp(a, k, x0, y0, z0, cols[warp], total, acc,
                     reinterpret_cast<uint16_t*>(term + kSums) + kHaloVerts * warp, lane, loss);
      }
      __syncthreads();
#pragma unroll 1
      for (int w = 0; w < kRegWarps; ++w) {
        if (verts[w] <= limit) continue;
        tile_origin(a, queue[n0 + w], x0, y0, z0);
        tile_by_block(a, k, x0, y0, z0, cols[w], verts[w], term, list, warp, lane, loss);
      }
      __syncthreads();  // the columns and verts are read
    }
    __syncthreads();  // the queue is read
  }
  double le = warp_sum_d(loss[0]), lc = warp_sum_d(loss[1]), ln = warp_sum_d(loss[2]);
  if (lane == 0) {
    red[0][warp] = le;
    red[1][warp] = lc;
    red[2][warp] = ln;
  }
  // the cluster's blocks in order, by its first one: one partial a cluster
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  cl.sync();
  if (cl.block_rank() == 0 && tid < 3) {
    double sum = 0;
    for (unsigned b = 0; b < cl.num_blocks(); ++b) {
      const double* theirs = cl.map_shared_rank(&red[tid][0], b);
      for (int w = 0; w < kRegWarps; ++w) sum += theirs[w];
    }
    partials[3 * (blockIdx.x / cl.num_blocks()) + tid] = sum;
  }
  cl.sync();  // until it has read them
}

// Mean losses over interior vertices from the per-block partials, fixed reduction order; and
// |V_R| after the filters (relax sphere when it keeps any vertex, band) for n_active.
__global__ void __launch_bounds__(256) k_reg_finalize(const double* __restrict__ partials, int nblocks,
                                                      float* __restrict__ losses,
                                                      const unsigned long long* __restrict__ counts, int relax,
                                                      int band, long long* __restrict__ n_active) {
  __shared__ double red[3][8];
  double a = 0, b = 0, k = 0;
  for (int i = threadIdx.x; i < nblocks; i += blockDim.x) {
    a += partials[3 * i];
    b += partials[3 * i + 1];
    k += partials[3 * i + 2];
  }
  a = warp_sum_d(a);
  b = warp_sum_d(b);
  k = warp_sum_d(k);
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = a;
    red[1][threadIdx.x >> 5] = b;
    red[2][threadIdx.x >> 5] = k;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a = b = k = 0;
    for (int w = 0; w < 8; ++w) {
      a += red[0][w];
      b += red[1][w];
      k += red[2][w];
    }
    if (losses) {
      losses[0] = k > 0 ? (float)(a / k) : 0.0f;
      losses[1] = k > 0 ? (float)(b / k) : 0.0f;
    }
    if (n_active) {
      const bool relax_on = relax && counts[1] > 0;
      *n_active = (long long)(band ? (relax_on ? counts[3] : counts[2]) : (relax_on ? counts[1] : counts[0]));
    }
  }
}

static int check_reg(const int32_t res[3]) {
  VX_REQUIRE(res && res[0] >= 3 && res[1] >= 3 && res[2] >= 3, "grid resolution must be >= 3 per axis");
  VX_REQUIRE((int64_t)res[0] * res[1] * res[2] < (int64_t(1) << 31), "grid has 2^31 or more voxels");
  return VX_OK;
}

static Grid grid_eps(const int32_t res[3], const float eps[3]) {
  const float lo[3] = {0, 0, 0}, hi[3] = {1, 1, 1};
  Grid g = make_grid(res, lo, hi);
  for (int a = 0; a < 3; ++a) g.eps[a] = eps[a];
  set_fd(g);
  return g;
}

}  // namespace vx

using namespace vx;

extern "C" {

int vx_reg_list_blocks(int64_t n_verts) { return (int)grid_for(n_verts, 256, 4); }

int vx_eikonal_grad(const float* grid, const int32_t res[3], const int64_t* verts, int64_t n_verts, float* grad_grid,
                    const float eps[3], float weight, double* partials, int n_partials, unsigned int* counter,
                    float* losses, void* stream) {
  if (int s = check_reg(res)) return s;
  VX_REQUIRE(n_verts >= 0, "n_verts < 0");
  if (n_verts == 0) return VX_OK;
  VX_REQUIRE(grid && verts && eps && partials && counter, "null pointer");
  const int blocks = vx_reg_list_blocks(n_verts);
  VX_REQUIRE(n_partials >= 3 * blocks, "partials buffer too small (%d < %d)", n_partials, 3 * blocks);
  RegOut o{partials, counter, losses};
  k_eikonal_list<<<blocks, 256, 0, (cudaStream_t)stream>>>(grid, grid_eps(res, eps), verts, n_verts, grad_grid,
                                                            weight, o);
  count_launches(1);
  return check_launch("eikonal_grad");
}

int vx_curvature_grad(const float* grid, const int32_t res[3], const int64_t* verts, int64_t n_verts,
                      float* grad_grid, const float eps[3], float weight, double* partials, int n_partials,
                      unsigned int* counter, float* losses, void* stream) {
  if (int s = check_reg(res)) return s;
  VX_REQUIRE(n_verts >= 0, "n_verts < 0");
  if (n_verts == 0) return VX_OK;
  VX_REQUIRE(grid && verts && eps && partials && counter, "null pointer");
  const int blocks = vx_reg_list_blocks(n_verts);
  VX_REQUIRE(n_partials >= 3 * blocks, "partials buffer too small (%d < %d)", n_partials, 3 * blocks);
  RegOut o{partials, counter, losses};
  k_curvature_list<<<blocks, 256, 0, (cudaStream_t)stream>>>(grid, grid_eps(res, eps), verts, n_verts, grad_grid,
                                                              weight, o);
  count_launches(1);
  return check_launch("curvature_grad");
}

static int64_t stencil_tiles(const int32_t res[3]) {
  return (int64_t)((res[2] + TZ - 1) / TZ) * ((res[1] + TY - 1) / TY) * ((res[0] + TX - 1) / TX);
}

// Blocks that share one of the nb loss partials: up to 4 blocks a SM, as many as are resident, a tile each on small
// grids.
static unsigned stencil_cluster(int64_t nb) {
  unsigned c = 8;
  while (c > 1 && nb * c > (int64_t)kSMs * 4) c /= 2;
  return c;
}

int64_t vx_reg_stencil_blocks(const int32_t res[3]) {
  const int64_t t = (stencil_tiles(res) + 7) / 8;  // up to 8 blocks share a partial (stencil_cluster)
  const int64_t cap = (int64_t)kSMs * 4;
  return t < cap ? t : cap;
}

int64_t vx_reg_stencil_workspace(const int32_t res[3]) {
  // 3 loss doubles per block, then one flag byte per tile
  return 3 * vx_reg_stencil_blocks(res) + (stencil_tiles(res) + 7) / 8;
}

int vx_reg_stencil(const float* grid, const uint32_t* bitmap, const int32_t res[3], const float xyz_min[3],
                   const float xyz_max[3], float relax_radius, float band, const unsigned long long* counts,
                   float w_eik, float w_curv, float* grad_grid, double* partials, int64_t n_partials,
                   unsigned int* counter, float* losses, int64_t* n_active, void* stream) {
  if (int s = check_reg(res)) return s;
  VX_REQUIRE(grid && bitmap && counts && grad_grid && partials && xyz_min && xyz_max, "null pointer");
  const int64_t nb = vx_reg_stencil_blocks(res);
  const int64_t need = vx_reg_stencil_workspace(res);
  VX_REQUIRE(n_partials >= need, "workspace too small (%lld < %lld doubles)", (long long)n_partials,
             (long long)need);
  StencilArgs a;
  a.f = grid;
  a.fb = bitmap;
  a.nwords = ((int64_t)res[0] * res[1] * res[2] + 31) / 32;
  a.g = make_grid(res, xyz_min, xyz_max);
  a.counts = counts;
  a.relax_r = relax_radius;
  a.w_eik = w_eik;
  a.w_curv = w_curv;
  a.gg = grad_grid;
  a.tiles_z = (res[2] + TZ - 1) / TZ;
  a.tiles_y = (res[1] + TY - 1) / TY;
  a.tiles_x = (res[0] + TX - 1) / TX;
  (void)counter;
  const int64_t ntiles = stencil_tiles(res);
  uint8_t* flags = reinterpret_cast<uint8_t*>(partials + 3 * nb);
  cudaStream_t st = (cudaStream_t)stream;
  k_tile_flags<<<grid_for(ntiles, 16), 256, 0, st>>>(a, (int)ntiles, flags);
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = stencil_cluster(nb);
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nb * attr.val.clusterDim.x);
  cfg.blockDim = dim3(kRegThreads);
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_reg_stencil, a, static_cast<const uint8_t*>(flags), partials, (int)ntiles);
  if (e != cudaSuccess) return set_error(VX_ERR_CUDA, "reg_stencil: %s", cudaGetErrorString(e));
  if (losses || n_active)
    k_reg_finalize<<<1, 256, 0, st>>>(partials, (int)nb, losses, counts, relax_radius > 0.0f ? 1 : 0,
                                      band > 0.0f ? 1 : 0, reinterpret_cast<long long*>(n_active));
  count_launches(losses || n_active ? 3 : 2);
  return check_launch("reg_stencil");
}

}  // extern "C"
