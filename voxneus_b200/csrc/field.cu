// SDF-grid field queries: trilinear SDF (S2), Eq.7 interpolated gradients and normals
// (S3/S8), their adjoints, the reference-compatible gradient_interp pair, and the lattice
// query of the large-grid workload.
//
// One thread per point, grid-stride loops over a grid sized to the 148 SMs. The 32-value
// Eq.7 stencil is read through the read-only path; a 256^3 grid (64 MiB) is L2-resident,
// so neighbouring samples of a ray hit L1/L2.
#include "common.cuh"

namespace vx {

__global__ void __launch_bounds__(256) k_gradient_interp_fwd(const float* __restrict__ f, Grid g,
                                                             const float* __restrict__ coords, int64_t n,
                                                             float* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    Eq7 e;
    eq7_setup_grid_coords(g, coords[3 * i], coords[3 * i + 1], coords[3 * i + 2], e);
    float w[8], gr[3];
    eq7_weights(e, w);
    eq7_gradient(f, g, e, w, gr);
    out[3 * i] = gr[0];
    out[3 * i + 1] = gr[1];
    out[3 * i + 2] = gr[2];
  }
}

__global__ void __launch_bounds__(256) k_gradient_interp_bwd(const float* __restrict__ dout,
                                                             const float* __restrict__ coords, int64_t n, Grid g,
                                                             float* __restrict__ gg) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    Eq7 e;
    eq7_setup_grid_coords(g, coords[3 * i], coords[3 * i + 1], coords[3 * i + 2], e);
    float w[8];
    eq7_weights(e, w);
    const float dg[3] = {dout[3 * i], dout[3 * i + 1], dout[3 * i + 2]};
    eq7_scatter(gg, g, e, w, dg);
  }
}

// sdf / grad / normal / corners / weights for world points; every output optional.
__global__ void __launch_bounds__(256) k_field_query(const float* __restrict__ f, Grid g,
                                                     const float* __restrict__ xyz, int64_t n,
                                                     float* __restrict__ sdf, float* __restrict__ grad,
                                                     float* __restrict__ normal, int64_t* __restrict__ corners,
                                                     float* __restrict__ weights) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float px = xyz[3 * i], py = xyz[3 * i + 1], pz = xyz[3 * i + 2];
    if (sdf && !(grad || normal)) sdf[i] = query_sdf(f, g, px, py, pz);
    if (grad || normal || corners || weights) {
      Eq7 e;
      eq7_setup(g, px, py, pz, e);
      float w[8];
      eq7_weights(e, w);
      if (grad || normal) {
        float c[8], gr[3], nn[3], len;  // the cell's corner values, shared by the SDF and the gradient
        eq7_load_block(f, g, e, c);
        if (sdf) sdf[i] = query_sdf_block(f, g, px, py, pz, e, c);
        eq7_gradient_block(f, g, e, w, c, gr);
        if (grad) {
          grad[3 * i] = gr[0];
          grad[3 * i + 1] = gr[1];
          grad[3 * i + 2] = gr[2];
        }
        if (normal) {
          normalize_eps(gr, nn, len);
          normal[3 * i] = nn[0];
          normal[3 * i + 1] = nn[1];
          normal[3 * i + 2] = nn[2];
        }
      }
      if (corners) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          int64_t* c = corners + (i * 8 + k) * 3;
          c[0] = (k & 4) ? e.x1 : e.x0;
          c[1] = (k & 2) ? e.y1 : e.y0;
          c[2] = (k & 1) ? e.z1 : e.z0;
        }
      }
      if (weights) {
#pragma unroll
        for (int k = 0; k < 8; ++k) weights[i * 8 + k] = w[k];
      }
    }
  }
}

// Adjoint of k_field_query with respect to the grid: d_sdf (n), d_grad (n,3), d_normal (n,3),
// each optional.
__global__ void __launch_bounds__(256, 4) k_field_query_bwd(const float* __restrict__ f, Grid g,
                                                         const float* __restrict__ xyz, int64_t n,
                                                         const float* __restrict__ d_sdf,
                                                         const float* __restrict__ d_grad,
                                                         const float* __restrict__ d_normal,
                                                         float* __restrict__ gg) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float px = xyz[3 * i], py = xyz[3 * i + 1], pz = xyz[3 * i + 2];
    if (d_sdf) {
      Tri t;
      gs_setup(g, px, py, pz, t);
      gs_scatter(gg, g, t, d_sdf[i]);
    }
    if (d_grad || d_normal) {
      Eq7 e;
      eq7_setup(g, px, py, pz, e);
      float w[8];
      eq7_weights(e, w);
      float dg[3] = {0.0f, 0.0f, 0.0f};
      if (d_normal) {
        float c[8], gr[3], nn[3], len;
        eq7_load_block(f, g, e, c);
        if (eq7_interior(g, e))  // 300,007 points: 93 -> 84 us for the two adjoints of a query
          eq7_gradient_interior(f + lin3(g, e.x0, e.y0, e.z0), g.ry * g.rz, g.rz, g, w, c, gr);
        else
          eq7_gradient_block(f, g, e, w, c, gr);
        normalize_eps(gr, nn, len);
        const float dn[3] = {d_normal[3 * i], d_normal[3 * i + 1], d_normal[3 * i + 2]};
        normalize_eps_bwd(gr, len, dn, dg);
      }
      if (d_grad) {
        dg[0] += d_grad[3 * i];
        dg[1] += d_grad[3 * i + 1];
        dg[2] += d_grad[3 * i + 2];
      }
      eq7_scatter(gg, g, e, w, dg);
    }
  }
}

// Lattice value: ATen's linspace split (start + step*i on the first half, end - step*(n-1-i)
// on the second), evaluated without FMA.
__device__ __forceinline__ float lattice_coord(float lo, float hi, int n, int i) {
  if (n <= 1) return lo;
  const float step = (hi - lo) / (float)(n - 1);
  if (i < n / 2) return __fadd_rn(lo, __fmul_rn(step, (float)i));
  return __fsub_rn(hi, __fmul_rn(step, (float)(n - 1 - i)));
}

// One lattice point against the grid in global memory.
__device__ __forceinline__ void lattice_point(const float* __restrict__ f, const Grid& g, float px, float py, float pz,
                                              int64_t i, float* __restrict__ sdf, float* __restrict__ normal) {
  if (!normal) {
    if (sdf) sdf[i] = query_sdf(f, g, px, py, pz);
    return;
  }
  Eq7 e;
  eq7_setup(g, px, py, pz, e);
  float c[8], w[8], gr[3], nn[3], len;
  eq7_load_block(f, g, e, c);
  if (sdf) sdf[i] = query_sdf_block(f, g, px, py, pz, e, c);
  eq7_weights(e, w);
  if (__all_sync(__activemask(), eq7_interior(g, e)))  // lanes apart would take both ways
    eq7_gradient_interior(f + lin3(g, e.x0, e.y0, e.z0), g.ry * g.rz, g.rz, g, w, c, gr);
  else
    eq7_gradient_block(f, g, e, w, c, gr);
  normalize_eps(gr, nn, len);
  normal[3 * i] = nn[0];
  normal[3 * i + 1] = nn[1];
  normal[3 * i + 2] = nn[2];
}

__global__ void __launch_bounds__(256, 4) k_field_lattice(const float* __restrict__ f, Grid g, int nx, int ny, int nz,
                                                       float lx, float ly, float lz, float hx, float hy, float hz,
                                                       float* __restrict__ sdf, float* __restrict__ normal) {
  const int64_t total = (int64_t)nx * ny * nz;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int k = (int)(i % nz);
    const int64_t r = i / nz;
    const int j = (int)(r % ny);
    const int ii = (int)(r / ny);
    lattice_point(f, g, lattice_coord(lx, hx, nx, ii), lattice_coord(ly, hy, ny, j), lattice_coord(lz, hz, nz, k), i, sdf,
                  normal);
  }
}

// SDF and normals of a lattice whose spacing is below ~1.7 voxels, in bricks of 8 x 8 x 32 points: the
// brick's voxels (its cells and their face neighbours, at most 16 x 16 x 56) are read once into shared
// memory with coalesced rows and every point's 32 stencil values come from there, where the plain kernel
// reads them through L1 (32 requests a point, each of up to 5 lines). What depends on one axis only (the
// coordinate's cell and weights, three IEEE divisions each) is evaluated once per brick and axis index.
// Points at the grid's border, or whose two cells differ by rounding, take the plain path. What bounds
// it: shared-memory loads (32 a point, about two wavefronts each at 1.6 voxels a point) and issue.
// 320^3 points of a 512^3 grid: 1138 us (plain, a division per difference) -> 784 us (plain) -> 543 us.
constexpr int kBx = 8, kBy = 8, kBz = 32;     // points of a brick
constexpr int kVx = 16, kVy = 16, kVz = 60;   // voxels of its region, at most (rows start on 16 bytes)
constexpr int kBrickThreads = 256;

struct AxisPoint {
  float p;       // coordinate
  int e0;        // Eq.7 cell
  float d;       // Eq.7 offset in the cell
  float lo, hi;  // grid_sample weights of the lower and upper corner
  int in;        // both cells the same, and interior
};

struct Inv2Eps {
  float v[3];  // 1 / (2 eps), the interior differences' reciprocal
  __device__ float operator[](int a) const { return v[a]; }
};

__global__ void __launch_bounds__(kBrickThreads, 3)
    k_field_lattice_brick(const float* __restrict__ f, Grid g, int nx, int ny, int nz, float lx, float ly, float lz,
                          float hx, float hy, float hz, int by_n, int bz_n, int vec, Inv2Eps i2e,
                          float* __restrict__ sdf, float* __restrict__ normal) {
  extern __shared__ __align__(16) float vox[];
  __shared__ AxisPoint ax[kBx + kBy + kBz];
  __shared__ int lo_s[3], hi_s[3];  // the brick's cells (monotone up to rounding: taken over all points)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bz = (blockIdx.x % bz_n) * kBz, by = (blockIdx.x / bz_n % by_n) * kBy, bx = (blockIdx.x / bz_n / by_n) * kBx;
  if (tid < 3) {
    lo_s[tid] = INT32_MAX;
    hi_s[tid] = 0;
  }
  __syncthreads();
  if (tid < kBx + kBy + kBz) {
    const int a = tid < kBx ? 0 : (tid < kBx + kBy ? 1 : 2);
    const int n = a == 0 ? nx : (a == 1 ? ny : nz), R = gdim(g, a);
    const int i = a == 0 ? bx + tid : (a == 1 ? by + tid - kBx : bz + tid - kBx - kBy);
    const float lo = a == 0 ? lx : (a == 1 ? ly : lz), hi = a == 0 ? hx : (a == 1 ? hy : hz);
    const float glo = a == 0 ? g.lo[0] : (a == 1 ? g.lo[1] : g.lo[2]);
    const float den = a == 0 ? g.den[0] : (a == 1 ? g.den[1] : g.den[2]);
    const float inv = a == 0 ? g.inv_den[0] : (a == 1 ? g.inv_den[1] : g.inv_den[2]);
    const float top = a == 0 ? g.hi_clamp[0] : (a == 1 ? g.hi_clamp[1] : g.hi_clamp[2]);
    AxisPoint q;
    q.p = lattice_coord(lo, hi, n, min(i, n - 1));
    const float c = gs_coord(q.p, glo, den, inv, R);
    const int gi = (int)floorf(c);
    q.lo = (float)(gi + 1) - c;
    q.hi = c - (float)gi;
    const float t = fminf(fmaxf(eq7_coord(q.p, glo, den, inv, R), 0.0f), top);
    q.e0 = min(max((int)floorf(t), 0), R - 1);
    q.d = t - (float)q.e0;
    q.in = (unsigned)(q.e0 - 1) < (unsigned)(R - 3) && gi == q.e0;
    ax[tid] = q;
    atomicMin(lo_s + a, q.e0);
    atomicMax(hi_s + a, q.e0);
  }
  __syncthreads();
  // its region: the cells, their upper corners and one voxel around
  const int x_lo = max(lo_s[0] - 1, 0), y_lo = max(lo_s[1] - 1, 0), z_lo = max(lo_s[2] - 1, 0) & (vec ? ~3 : ~0);
  const int mx = min(hi_s[0] + 2, g.rx - 1) - x_lo + 1, my = min(hi_s[1] + 2, g.ry - 1) - y_lo + 1;
  const int mz = min(hi_s[2] + 2, g.rz - 1) - z_lo + 1;
  const bool fits = mx <= kVx && my <= kVy && mz <= kVz;
  if (fits) {  // asynchronous copies, all of a thread's in flight together
    const float* src = f + lin3(g, x_lo, y_lo, z_lo);
    if (vec) {  // grid rows of whole float4: 16 lanes a row (the row's last chunk may run past the region)
      const int y = tid >> 4, c4 = 4 * (tid & 15);
      if (y < my && c4 < mz)
        for (int x = 0; x < mx; ++x) {
          float* d = vox + (x * kVy + y) * kVz + c4;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(d)),
                       "l"(src + (x * g.ry + y) * g.rz + c4)
                       : "memory");
        }
    } else {
      for (int r = warp; r < mx * kVy; r += kBrickThreads / 32) {
        const int x = r / kVy, y = r % kVy;
        for (int z = lane; y < my && z < mz; z += 32) {
          float* d = vox + r * kVz + z;
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(d)),
                       "l"(src + (x * g.ry + y) * g.rz + z)
                       : "memory");
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  __syncthreads();
  // warp = the row's y, lane = its z (both fixed); x in the loop
  const AxisPoint qy = ax[kBx + warp], qz = ax[kBx + kBy + lane];
  if (by + warp >= ny || bz + lane >= nz) return;
  const bool yz_in = fits && qy.in && qz.in;
  const float oy = 1.0f - qy.d, oz = 1.0f - qz.d;
  const float zy[4] = {qz.lo * qy.lo, qz.hi * qy.lo, qz.lo * qy.hi, qz.hi * qy.hi};  // grid_sample's order
  const float* p0 = vox + (qy.e0 - y_lo) * kVz + (qz.e0 - z_lo);
  int64_t i = ((int64_t)bx * ny + by + warp) * nz + bz + lane;
  const int64_t step = (int64_t)ny * nz;
  const int xn = min(kBx, nx - bx);
#pragma unroll 1
  for (int xi = 0; xi < xn; ++xi, i += step) {
    const AxisPoint qx = ax[xi];
    if (!(yz_in && qx.in)) {
      lattice_point(f, g, qx.p, qy.p, qz.p, i, sdf, normal);
      continue;
    }
    const float* p = p0 + (qx.e0 - x_lo) * (kVy * kVz);
    float c[8], w[8], gr[3];
#pragma unroll
    for (int k = 0; k < 8; ++k) c[k] = p[((k & 4) ? kVy * kVz : 0) + ((k & 2) ? kVz : 0) + (k & 1)];
    if (sdf) {  // as gs_setup and query_sdf_block
      float acc = 0.0f;
#pragma unroll
      for (int k = 0; k < 8; ++k) acc = fmaf(c[k], zy[k & 3] * ((k & 4) ? qx.hi : qx.lo), acc);
      sdf[i] = acc;
    }
    const float ox = 1.0f - qx.d;
#pragma unroll
    for (int k = 0; k < 8; ++k) w[k] = ((k & 4) ? qx.d : ox) * ((k & 2) ? qy.d : oy) * ((k & 1) ? qz.d : oz);
    eq7_blend_interior(p, kVy * kVz, kVz, w, c, gr);
#pragma unroll
    for (int a = 0; a < 3; ++a) gr[a] *= i2e[a];
    const float inv = 1.0f / (norm3(gr[0], gr[1], gr[2]) + 1e-8f);
    normal[3 * i] = gr[0] * inv;
    normal[3 * i + 1] = gr[1] * inv;
    normal[3 * i + 2] = gr[2] * inv;
  }
}

// Corners and weights at grid-index coordinates (geometry/coordinates.py:55-124).
__global__ void __launch_bounds__(256) k_corners_weights(Grid g, const float* __restrict__ coords, int64_t n,
                                                         int64_t* __restrict__ corners, float* __restrict__ weights) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    Eq7 e;
    eq7_setup_grid_coords(g, coords[3 * i], coords[3 * i + 1], coords[3 * i + 2], e);
    float w[8];
    eq7_weights(e, w);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (corners) {
        int64_t* c = corners + (i * 8 + k) * 3;
        c[0] = (k & 4) ? e.x1 : e.x0;
        c[1] = (k & 2) ? e.y1 : e.y0;
        c[2] = (k & 1) ? e.z1 : e.z0;
      }
      if (weights) weights[i * 8 + k] = w[k];
    }
  }
}

static Grid grid_from_eps(const int32_t res[3], const float eps[3]) {
  const float lo[3] = {0.f, 0.f, 0.f}, hi[3] = {1.f, 1.f, 1.f};
  Grid g = make_grid(res, lo, hi);
  for (int a = 0; a < 3; ++a) g.eps[a] = eps[a];
  set_fd(g);
  return g;
}

}  // namespace vx

using namespace vx;

extern "C" {

int vx_gradient_interp_forward(const float* grid, const int32_t res[3], const float* coords, int64_t n,
                               const float eps[3], float* out_grad, void* stream) {
  if (int s = check_grid(res)) return s;
  VX_REQUIRE(n >= 0, "n < 0");
  if (n == 0) return VX_OK;
  VX_REQUIRE(grid && coords && out_grad && eps, "null pointer");
  Grid g = grid_from_eps(res, eps);
  k_gradient_interp_fwd<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(grid, g, coords, n, out_grad);
  count_launches(1);
  return check_launch("gradient_interp_forward");
}

int vx_gradient_interp_backward(const float* grad_out, const float* coords, int64_t n, float* grad_grid,
                                const int32_t res[3], const float eps[3], void* stream) {
  if (int s = check_grid(res)) return s;
  VX_REQUIRE(n >= 0, "n < 0");
  if (n == 0) return VX_OK;
  VX_REQUIRE(grad_out && coords && grad_grid && eps, "null pointer");
  Grid g = grid_from_eps(res, eps);
  k_gradient_interp_bwd<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(grad_out, coords, n, g, grad_grid);
  count_launches(1);
  return check_launch("gradient_interp_backward");
}

int vx_field_query(const float* grid, const int32_t res[3], const float xyz_min[3], const float xyz_max[3],
                   const float* xyz, int64_t n, float* sdf, float* grad, float* normal, int64_t* corners,
                   float* weights, void* stream) {
  if (int s = check_grid(res)) return s;
  VX_REQUIRE(n >= 0, "n < 0");
  if (n == 0) return VX_OK;
  VX_REQUIRE(grid && xyz && xyz_min && xyz_max, "null pointer");
  Grid g = make_grid(res, xyz_min, xyz_max);
  k_field_query<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(grid, g, xyz, n, sdf, grad, normal, corners,
                                                                      weights);
  count_launches(1);
  return check_launch("field_query");
}

int vx_field_query_backward(const float* grid, const int32_t res[3], const float xyz_min[3], const float xyz_max[3],
                            const float* xyz, int64_t n, const float* d_sdf, const float* d_grad,
                            const float* d_normal, float* grad_grid, void* stream) {
  if (int s = check_grid(res)) return s;
  VX_REQUIRE(n >= 0, "n < 0");
  if (n == 0 || (!d_sdf && !d_grad && !d_normal)) return VX_OK;
  VX_REQUIRE(grid && xyz && grad_grid && xyz_min && xyz_max, "null pointer");
  Grid g = make_grid(res, xyz_min, xyz_max);
  k_field_query_bwd<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(grid, g, xyz, n, d_sdf, d_grad, d_normal,
                                                                          grad_grid);
  count_launches(1);
  return check_launch("field_query_backward");
}

int vx_field_query_lattice(const float* grid, const int32_t res[3], const float xyz_min[3], const float xyz_max[3],
                           const int32_t lattice[3], const float lat_min[3], const float lat_max[3], float* sdf,
                           float* normal, void* stream) {
  if (int s = check_grid(res)) return s;
  VX_REQUIRE(lattice && lat_min && lat_max, "null pointer");
  VX_REQUIRE(lattice[0] > 0 && lattice[1] > 0 && lattice[2] > 0, "lattice size must be positive");
  VX_REQUIRE(grid && xyz_min && xyz_max, "null pointer");
  Grid g = make_grid(res, xyz_min, xyz_max);
  const int64_t total = (int64_t)lattice[0] * lattice[1] * lattice[2];
  // Bricks where a brick's voxels fit their region: (points - 1) * spacing rounded up, 1 and 3 more voxels an
  // axis (a brick that still does not fit takes the plain path). Wider lattices share few voxels between
  // points: at 3.2 voxels a point a brick would read 8 voxels a point more than the stencil's 32.
  // A brick at the grid's border answers its border points one after the other, which is all that a small lattice
  // waits for, and lanes past the lattice idle. In cells with whole stencils only, bricks are faster from 2^18 points on
  // (48^3 of 64^3 5.0 us plain, 6.3 in bricks; 64^3 8.7, 6.6); over the whole grid from ~3 M on (130^3 of 128^3 64.0, 69.9;
  // 160^3 117, 99), if most of the lanes have such points (400 x 400 x 20 of 16^3, 41% of them: 121, 183 us).
  const int bn[3] = {kBx, kBy, kBz}, vn[3] = {kVx, kVy, kVz};
  bool brick = normal != nullptr;
  double inner = 1.0, used = 1.0;  // fraction of the points with whole stencils, of the bricks' lanes with points
  for (int a = 0; a < 3; ++a) {
    const double s = lattice[a] > 1 ? fabs((double)lat_max[a] - lat_min[a]) / (lattice[a] - 1) / g.eps[a] : 0.0;
    brick = brick && res[a] >= 4 && res[a] <= 4096 && floor(s * (bn[a] - 1)) + 5.0 + (a == 2 ? 3.0 : 0.0) <= vn[a];
    const double c0 = ((double)(lat_min[a] < lat_max[a] ? lat_min[a] : lat_max[a]) - xyz_min[a]) / g.eps[a];
    const double c1 = c0 + s * (lattice[a] - 1), in = fmin(c1, res[a] - 2.0) - fmax(c0, 1.0);
    inner *= in < 0.0 ? 0.0 : c1 > c0 ? in / (c1 - c0) : 1.0;
    used *= (double)lattice[a] / ((lattice[a] + bn[a] - 1) / bn[a] * bn[a]);
  }
  brick = brick && (inner == 1.0 ? total >= (1 << 18) : total >= (3 << 20) && inner * used >= 0.6);
  if (brick) {
    const int64_t bx = (lattice[0] + kBx - 1) / kBx, by = (lattice[1] + kBy - 1) / kBy, bz = (lattice[2] + kBz - 1) / kBz;
    const int vec = res[2] % 4 == 0 && (reinterpret_cast<uintptr_t>(grid) & 15) == 0;
    const Inv2Eps i2e{{1.0f / (2.0f * g.eps[0]), 1.0f / (2.0f * g.eps[1]), 1.0f / (2.0f * g.eps[2])}};
    const size_t smem = (size_t)kVx * kVy * kVz * sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(k_field_lattice_brick, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return set_error(VX_ERR_CUDA, "field_query_lattice: %s", cudaGetErrorString(e));
    if (bx * by * bz <= INT32_MAX) {
      k_field_lattice_brick<<<(unsigned)(bx * by * bz), kBrickThreads, smem, (cudaStream_t)stream>>>(
          grid, g, lattice[0], lattice[1], lattice[2], lat_min[0], lat_min[1], lat_min[2], lat_max[0], lat_max[1],
          lat_max[2], (int)by, (int)bz, vec, i2e, sdf, normal);
      count_launches(1);
      return check_launch("field_query_lattice");
    }
  }
  k_field_lattice<<<grid_for(total, 256), 256, 0, (cudaStream_t)stream>>>(
      grid, g, lattice[0], lattice[1], lattice[2], lat_min[0], lat_min[1], lat_min[2], lat_max[0], lat_max[1],
      lat_max[2], sdf, normal);
  count_launches(1);
  return check_launch("field_query_lattice");
}

int vx_corners_weights(const float* coords, int64_t n, const int32_t res[3], int64_t* corners, float* weights,
                       void* stream) {
  if (int s = check_grid(res)) return s;
  VX_REQUIRE(n >= 0, "n < 0");
  if (n == 0) return VX_OK;
  VX_REQUIRE(coords && (corners || weights), "null pointer");
  const float eps[3] = {1.f, 1.f, 1.f};
  Grid g = grid_from_eps(res, eps);
  k_corners_weights<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(g, coords, n, corners, weights);
  count_launches(1);
  return check_launch("corners_weights");
}

}  // extern "C"
