// Appearance hand-off: multiresolution hash encoding (models/radiance_hash.py:71-166),
// degree-4 spherical harmonics of the view direction (models/embedder.py:55-87) and the
// copy of the Eq.7 normal, written as one row per sample of the radiance MLP input
// ([hash 32 | SH 16 | normal 3], models/radiance_mlp.py:94-98).
//
// Four threads per sample, a quarter of the levels each: the 8 corner features of a level are
// gathers from the (L, 2^19, 2) table (64 MiB at the default size, L2-resident). The adjoint takes a
// thread per level and run of samples and scatters with float2 and float4 atomics (sm_90+).
// Hash indices are computed in uint32 arithmetic: the low log2(T) bits of
// x*1 ^ y*2654435761 ^ z*805459861 equal the reference's int64 value modulo 2^log2(T).
#include "hashgrid.cuh"

namespace vx {

// A block takes 256 / kGroups rows, kGroups threads each: thread group g encodes levels [g * lpt, (g + 1) * lpt), builds
// its share of the four SH quarters and one group copies the normal; the rows meet in shared memory and leave with
// consecutive lanes on consecutive columns. Bound by the table's sector requests (L1 to L2). 200,003 points,
// 11 of 16 levels open, with the SH of as many directions: 111 us with a thread a row (4-byte stores a row
// apart, levels one after the other), 70 us with four. Four threads need levels to share: app_groups.
__host__ __device__ inline int app_columns(const HashArgs& a) {
  return (a.table ? 2 * a.L : 0) + (a.sh_col >= 0 ? 16 : 0) + (a.nrm_col >= 0 ? 3 : 0) + (a.pad_col >= 0 ? 1 : 0);
}

// Threads a row. One thread writes its row itself, which pays up to two levels: 300,000 points of one level 13.9 us by four
// threads, 6.5 by one, of two levels 17.1 and 11.1, of three 26.0 and 25.0; 15,000 points of three 4.5 and 5.4.
inline int app_groups(const HashArgs& a) { return a.table && a.L <= 2 ? 1 : 4; }

template <int kGroups>
__global__ void __launch_bounds__(256) k_appearance_fwd(HashArgs a) {
  constexpr int kAppRows = 256 / kGroups, kWarps = 8 / kGroups;  // rows of a block, warps of a group
  extern __shared__ float srow[];  // [kAppRows][pitch]
  const uint32_t mask = (1u << a.log2T) - 1u;
  const size_t T = (size_t)1 << a.log2T;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = w / kWarps;
  const int ls = 32 * (w % kWarps) + lane;  // this thread's row in the block
  const int ncol = app_columns(a), pitch = ncol | 1, lpt = (a.L + kGroups - 1) / kGroups;
  constexpr bool kDirect = kGroups == 1;  // a thread's row goes straight to its columns
  const int sh0 = kDirect ? a.sh_col : a.table ? 2 * a.L : 0, nrm0 = kDirect ? a.nrm_col : sh0 + (a.sh_col >= 0 ? 16 : 0);
  const int pad0 = kDirect ? a.pad_col : nrm0 + (a.nrm_col >= 0 ? 3 : 0);
  const int width = ncol >= 32 ? 32 : 1 << (32 - __clz(max(ncol - 1, 1)));  // lanes of a row on the way out
  for (int64_t base = (int64_t)blockIdx.x * kAppRows; base < a.P; base += (int64_t)gridDim.x * kAppRows) {
    const int64_t i = base + ls;
    float* mine = kDirect ? a.out + i * a.ld : srow + ls * pitch;
    if (i < a.P) {
      if (a.table) {
        float x[3];
        sample_pos(a, i, x);
        const int l1 = min((g + 1) * lpt, a.L);
#pragma unroll 4
        for (int l = g * lpt; l < l1; ++l) {
          const float lw = a.lw[l];
          float f0 = 0.0f, f1 = 0.0f;
          if (lw != 0.0f) {
            LevelCell c;
            level_cell(x, a.res[l], mask, c);
            gather_level(reinterpret_cast<const float2*>(a.table) + (size_t)l * T, c, f0, f1);
            if (lw < 1.0f) {
              f0 *= lw;
              f1 *= lw;
            }
          }
          mine[2 * l] = f0;
          mine[2 * l + 1] = f1;
        }
      }
      if (a.sh_col >= 0) {
        float dx, dy, dz;
        if (a.dirs) {
          dx = a.dirs[i * a.dir_ss];
          dy = a.dirs[i * a.dir_ss + 1];
          dz = a.dirs[i * a.dir_ss + 2];
        } else {
          const int64_t r = i / a.S;
          dx = __ldg(a.rays_d + 3 * r);
          dy = __ldg(a.rays_d + 3 * r + 1);
          dz = __ldg(a.rays_d + 3 * r + 2);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k % kGroups != g) continue;
          const float4 v = sh_chunk(dx, dy, dz, k);
          mine[sh0 + 4 * k] = v.x;
          mine[sh0 + 4 * k + 1] = v.y;
          mine[sh0 + 4 * k + 2] = v.z;
          mine[sh0 + 4 * k + 3] = v.w;
        }
      }
      if (a.nrm_col >= 0 && g == 1 % kGroups) {
        mine[nrm0] = a.normals[3 * i];
        mine[nrm0 + 1] = a.normals[3 * i + 1];
        mine[nrm0 + 2] = a.normals[3 * i + 2];
      }
      if (a.pad_col >= 0 && g == 2 % kGroups) mine[pad0] = 0.0f;
    }
    if (kDirect) continue;
    __syncthreads();
    const int nrows = (int)(a.P - base < kAppRows ? a.P - base : kAppRows);
    for (int c = lane & (width - 1); c < ncol; c += width) {
      int to = c;  // the value's column; of parts laid over one another the last stays
      bool gone = false;
      const bool pad = a.pad_col >= 0, nrm = a.nrm_col >= 0, sh = a.sh_col >= 0;
      if (pad && c >= pad0) {
        to = a.pad_col;
      } else if (nrm && c >= nrm0) {
        to = a.nrm_col + c - nrm0;
        gone = pad && to == a.pad_col;
      } else {
        if (sh && c >= sh0) to = a.sh_col + c - sh0;
        gone = (pad && to == a.pad_col) || (nrm && to >= a.nrm_col && to < a.nrm_col + 3) ||
               (c < sh0 && sh && to >= a.sh_col && to < a.sh_col + 16);
      }
      if (!gone)
        for (int r = (32 * w + lane) / width; r < nrows; r += 256 / width) a.out[(base + r) * a.ld + to] = srow[r * pitch + c];
    }
    __syncthreads();
  }
}

// Adjoint of the hash encoding: thread (l, seg) scatters level l of kRun consecutive samples. While they stay
// in one cell of the level its eight corner gradients add up in registers; they go out by float4 atomics for
// the x-pairs of even cells and float2 ones otherwise when the cell changes and at the end (one copy of
// that code: unrolled over the samples it outgrew the instruction cache). What bounds it: the atomics, ~250 G
// vector reductions a second into the L2-resident table. 1 M samples of a training step 128 us with every
// sample's corners sent, 106, 89, 83 and 94 us with runs of 2, 4, 8 and 12; 2,048 rays 41 -> 29 us.

__device__ __forceinline__ void flush_cell(float2* __restrict__ tab, int cx, int cy, int cz, uint32_t mask, float2 (&acc)[8]) {
  uint32_t h[8];
#pragma unroll
  for (int k = 0; k < 8; ++k)
    h[k] = hash3((uint32_t)(cx + (k >> 2)), (uint32_t)(cy + ((k >> 1) & 1)), (uint32_t)(cz + (k & 1)), mask);
  if ((cx & 1) == 0) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool odd = h[k] & 1u;
      const float2 a = odd ? acc[k + 4] : acc[k], b = odd ? acc[k] : acc[k + 4];
      atomicAdd(reinterpret_cast<float4*>(tab) + (h[k] >> 1), make_float4(a.x, a.y, b.x, b.y));
    }
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) atomicAdd(tab + h[k], acc[k]);
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = make_float2(0.0f, 0.0f);
}

template <int kRun>
__global__ void __launch_bounds__(256) k_hash_bwd(HashArgs a) {
  const uint32_t mask = (1u << a.log2T) - 1u;
  const int l = threadIdx.x;
  const float lw = a.lw[l], fr = (float)a.res[l];
  if (lw == 0.0f) return;
  float2* tab = reinterpret_cast<float2*>(a.table_grad) + ((size_t)l << a.log2T);
  const int64_t nseg = (a.P + kRun - 1) / kRun;
  for (int64_t seg = blockIdx.x * (int64_t)blockDim.y + threadIdx.y; seg < nseg; seg += (int64_t)gridDim.x * blockDim.y) {
    const int64_t i0 = seg * kRun;
    float2 g[kRun];
#pragma unroll
    for (int u = 0; u < kRun; ++u) {
      g[u] = make_float2(0.0f, 0.0f);
      if (i0 + u < a.P) {
        const float* p = a.d_out + (i0 + u) * a.ld_d + 2 * l;
        g[u] = make_float2(__ldg(p), __ldg(p + 1));
      }
    }
    int cx = -1, cy = 0, cz = 0;
    float2 acc[8];
    if constexpr (kRun == 1) {  // the position's loads beside the gradient's, no loop
      float x[3];
      sample_pos(a, i0, x);
      if (g[0].x == 0.0f && g[0].y == 0.0f) continue;
      const float g0 = lw < 1.0f ? g[0].x * lw : g[0].x, g1 = lw < 1.0f ? g[0].y * lw : g[0].y;
      const float sx = x[0] * fr, sy = x[1] * fr, sz = x[2] * fr;
      cx = (int)floorf(sx);
      cy = (int)floorf(sy);
      cz = (int)floorf(sz);
      const float dx = sx - (float)cx, dy = sy - (float)cy, dz = sz - (float)cz;
      const float ox = 1.0f - dx, oy = 1.0f - dy, oz = 1.0f - dz;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float w = ((k & 4) ? dx : ox) * ((k & 2) ? dy : oy) * ((k & 1) ? dz : oz);
        acc[k] = make_float2(w * g0, w * g1);
      }
      flush_cell(tab, cx, cy, cz, mask, acc);
      continue;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = make_float2(0.0f, 0.0f);
#pragma unroll 1
    for (int u = 0;; ++u) {
      float g0 = g[0].x, g1 = g[0].y;
#pragma unroll
      for (int k = 0; k + 1 < kRun; ++k) g[k] = g[k + 1];
      if (u < kRun && g0 == 0.0f && g1 == 0.0f) continue;
      float sx = 0.0f, sy = 0.0f, sz = 0.0f;
      int nx = -1, ny = 0, nz = 0;
      if (u < kRun) {
        float x[3];
        sample_pos(a, i0 + u, x);
        sx = x[0] * fr;
        sy = x[1] * fr;
        sz = x[2] * fr;
        nx = (int)floorf(sx);
        ny = (int)floorf(sy);
        nz = (int)floorf(sz);
      }
      if (nx != cx || ny != cy || nz != cz) {
        if (cx >= 0) flush_cell(tab, cx, cy, cz, mask, acc);
        cx = nx;
        cy = ny;
        cz = nz;
      }
      if (u == kRun) break;
      if (lw < 1.0f) {
        g0 *= lw;
        g1 *= lw;
      }
      const float dx = sx - (float)nx, dy = sy - (float)ny, dz = sz - (float)nz;
      const float ox = 1.0f - dx, oy = 1.0f - dy, oz = 1.0f - dz;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float w = ((k & 4) ? dx : ox) * ((k & 2) ? dy : oy) * ((k & 1) ? dz : oz);
        acc[k].x = fmaf(w, g0, acc[k].x);
        acc[k].y = fmaf(w, g1, acc[k].y);
      }
    }
  }
}

}  // namespace vx

using namespace vx;

extern "C" {

int vx_appearance_forward(const float* table, int n_levels, int log2_size, int n_features, const int32_t* level_res,
                          const float* level_weights, const float* pts_norm, const float* rays_o, const float* rays_d,
                          const float* mid, int n_samples, const float xyz_min[3], const float xyz_max[3],
                          int64_t n_points, float* out, int64_t ld, int sh_col, const float* dirs,
                          int64_t dir_stride, int normal_col, const float* normals, int pad_col, void* stream) {
  HashArgs a{};
  if (table) {
    if (int s = fill_hash(a, table, n_levels, log2_size, n_features, level_res, level_weights)) return s;
  } else {
    a.table = nullptr;
    a.L = 0;
  }
  VX_REQUIRE(n_points >= 0, "n_points < 0");
  if (n_points == 0) return VX_OK;
  VX_REQUIRE(out, "out is null");
  VX_REQUIRE(!table || pts_norm || (rays_o && rays_d && mid && n_samples >= 1 && xyz_min && xyz_max),
             "need normalised points or rays + midpoints + bounds");
  VX_REQUIRE(!table || ld >= 2 * n_levels, "row stride smaller than the hash feature width");
  VX_REQUIRE(sh_col < 0 || (sh_col + 16 <= ld && (dirs || rays_d)), "bad SH column or missing directions");
  VX_REQUIRE(normal_col < 0 || (normal_col + 3 <= ld && normals), "bad normal column or missing normals");
  VX_REQUIRE(pad_col < ld, "bad pad column");
  fill_positions(a, pts_norm, rays_o, rays_d, mid, n_samples, pts_norm ? nullptr : xyz_min, xyz_max);
  a.P = n_points;
  a.out = out;
  a.ld = ld;
  a.sh_col = sh_col;
  a.dirs = dirs;
  a.dir_ss = dir_stride;
  a.nrm_col = normal_col;
  a.normals = normals;
  a.pad_col = pad_col;
  const int rows = 256 / app_groups(a);  // of a block
  const size_t smem = rows == 256 ? 0 : (size_t)rows * (app_columns(a) | 1) * sizeof(float);  // at most 22 KB
  const unsigned blocks = grid_for((n_points + rows - 1) / rows * 256, 256, 32);
  if (app_groups(a) == 1)
    k_appearance_fwd<1><<<blocks, 256, smem, (cudaStream_t)stream>>>(a);
  else
    k_appearance_fwd<4><<<blocks, 256, smem, (cudaStream_t)stream>>>(a);
  count_launches(1);
  return check_launch("appearance_forward");
}

int vx_hash_encode_backward(float* table_grad, int n_levels, int log2_size, int n_features, const int32_t* level_res,
                            const float* level_weights, const float* pts_norm, const float* rays_o,
                            const float* rays_d, const float* mid, int n_samples, const float xyz_min[3],
                            const float xyz_max[3], int64_t n_points, const float* d_out, int64_t ld_d,
                            void* stream) {
  HashArgs a{};
  if (int s = fill_hash(a, nullptr, n_levels, log2_size, n_features, level_res, level_weights)) return s;
  VX_REQUIRE(n_points >= 0, "n_points < 0");
  if (n_points == 0) return VX_OK;
  VX_REQUIRE(table_grad && d_out, "null pointer");
  VX_REQUIRE(pts_norm || (rays_o && rays_d && mid && n_samples >= 1 && xyz_min && xyz_max),
             "need normalised points or rays + midpoints + bounds");
  VX_REQUIRE(ld_d >= 2 * n_levels, "gradient row stride smaller than the hash feature width");
  fill_positions(a, pts_norm, rays_o, rays_d, mid, n_samples, pts_norm ? nullptr : xyz_min, xyz_max);
  a.table_grad = table_grad;
  a.P = n_points;
  a.d_out = d_out;
  a.ld_d = ld_d;
  // Consecutive samples of a ray share cells; a caller's own points and rays of few samples hardly do and take one sample
  // a thread (100,000 points of 4 levels 18.6 us in runs of 1, 20.2 of 2, 21.1 of 4; 300,000 of 16 levels 153 us all
  // three). Few samples of rays need the threads too: below 2^17 samples x levels (6,400 samples, 8 levels 4.8, 4.8, 6.6 us;
  // 16 levels 7.3, 7.1, 6.9). With a training step's gradients, most of them 0, runs of 8 and of 4 cross near 2^18 samples
  // (80 and 128 a ray: 102,400 27.6 us in runs of 4, 29.7 of 8; 163,840 35.9, 36.9; 262,144 43.1, 43.0; 384,000 54.3, 52.3;
  // 1,048,576 106.5, 99.3).
  const bool shared = !pts_norm && n_samples >= 8 && n_points * n_levels >= (int64_t(1) << 17);
  const int run = !shared ? 1 : n_points < (int64_t(1) << 18) ? 4 : 8;
  auto kern = run == 1 ? k_hash_bwd<1> : run == 4 ? k_hash_bwd<4> : k_hash_bwd<8>;
  const dim3 threads(n_levels, 256 / n_levels);
  kern<<<grid_for((n_points + run - 1) / run, (int)threads.y, 32), threads, 0, (cudaStream_t)stream>>>(a);
  count_launches(1);
  return check_launch("hash_encode_backward");
}

}  // extern "C"
