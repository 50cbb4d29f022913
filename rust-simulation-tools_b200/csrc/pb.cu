// Poisson-Boltzmann engine on the GPU in FP64.  Set-up, plain SOR and the
// energy follow the reference's arithmetic with unfused multiply-adds (built
// with -fmad=false); the multigrid cycles take its steps with explicit fused
// ones, which round less often:
//   pb_grid.rs   auto_grid, map_charges, spatial hash, SAS test, flood fill
//                from the boundary, SES by distance threshold, face
//                dielectrics from exact chord intervals, kappa-bar^2 map
//   pb_solver.rs Debye-Hueckel boundary, red-black SOR, residual, full-
//                weighting restriction, trilinear prolongation, injection
//                coarsening, V-cycle, convergence / divergence logic, energy
//   pb_energy.rs solvated and reference solves, two-level focusing
//
// Set-up work that is O(atoms) -- the spatial hash and the trilinear charge
// spreading in atom order -- is done on the host; everything that touches
// the grid runs in the kernels below.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <unordered_map>

#include "common.cuh"
#include "frame_plain.hpp"
#include "pb.cuh"

namespace rstg {

static const double kFourPiEc = 4.0 * kPi * 332.0522;  // pb_solver.rs:155

// ---------------------------------------------------------------------------
// host helpers
// ---------------------------------------------------------------------------
static void bbox(const std::vector<double>& x, double* mn, double* mx) {
  for (int d = 0; d < 3; d++) {
    mn[d] = std::numeric_limits<double>::max();
    mx[d] = std::numeric_limits<double>::lowest();
  }
  for (size_t a = 0; a < x.size() / 3; a++)
    for (int d = 0; d < 3; d++) {
      if (x[3 * a + d] < mn[d]) mn[d] = x[3 * a + d];
      if (x[3 * a + d] > mx[d]) mx[d] = x[3 * a + d];
    }
}

PbGeom pb_auto_grid(const std::vector<double>& x, double h, double buffer) {
  double mn[3], mx[3];
  bbox(x, mn, mx);
  PbGeom g;
  int dims[3];
  double org[3];
  for (int d = 0; d < 3; d++) {
    double ext = mx[d] - mn[d] + 2.0 * buffer;
    size_t n = (size_t)std::ceil(ext / h) + 1;
    n = (n % 2 == 0) ? n + 1 : n;
    if (n > 4096) throw Error(RSTG_ERR_INVALID, "PB grid dimension exceeds 4096 points");
    dims[d] = (int)n;
    double gext = (double)(n - 1) * h;
    org[d] = 0.5 * (mn[d] + mx[d]) - 0.5 * gext;
  }
  g.nx = dims[0];
  g.ny = dims[1];
  g.nz = dims[2];
  g.ox = org[0];
  g.oy = org[1];
  g.oz = org[2];
  g.h = h;
  return g;
}

PbGeom pb_coarse_grid(const std::vector<double>& x, double h, double fill, int64_t fs) {
  double mn[3], mx[3];
  bbox(x, mn, mx);
  double ch = h * (double)fs;
  PbGeom g;
  int dims[3];
  double org[3];
  for (int d = 0; d < 3; d++) {
    double ext = (mx[d] - mn[d]) * fill;
    size_t n = (size_t)std::ceil(ext / ch) + 1;
    n = (n % 2 == 0) ? n + 1 : n;
    if (n > 4096) throw Error(RSTG_ERR_INVALID, "PB coarse grid dimension exceeds 4096 points");
    dims[d] = (int)n;
    org[d] = 0.5 * (mn[d] + mx[d]) - 0.5 * ((double)(n - 1) * ch);
  }
  g.nx = dims[0];
  g.ny = dims[1];
  g.nz = dims[2];
  g.ox = org[0];
  g.oy = org[1];
  g.oz = org[2];
  g.h = ch;
  return g;
}

double pb_omega(int nx, int ny, int nz) {
  double r = (std::cos(kPi / (double)nx) + std::cos(kPi / (double)ny) + std::cos(kPi / (double)nz)) / 3.0;
  return 2.0 / (1.0 + std::sqrt(1.0 - r * r));
}

static double spectral_radius(int nx, int ny, int nz) {
  return (std::cos(kPi / (double)nx) + std::cos(kPi / (double)ny) + std::cos(kPi / (double)nz)) / 3.0;
}

PbHash pb_build_hash(const std::vector<double>& x, double max_eff) {
  PbHash H;
  size_t n = x.size() / 3;
  if (n == 0) return H;
  double cs = std::max(max_eff, 0.1);
  H.inv = 1.0 / cs;
  double mn[3], mx[3];
  bbox(x, mn, mx);
  H.ox = mn[0] - max_eff;
  H.oy = mn[1] - max_eff;
  H.oz = mn[2] - max_eff;
  H.gx = (int)((size_t)std::ceil((mx[0] - H.ox) * H.inv) + 1);
  H.gy = (int)((size_t)std::ceil((mx[1] - H.oy) * H.inv) + 1);
  H.gz = (int)((size_t)std::ceil((mx[2] - H.oz) * H.inv) + 1);
  size_t nc = (size_t)H.gx * H.gy * H.gz;
  if (nc > (size_t)1 << 28) throw Error(RSTG_ERR_INVALID, "spatial hash too large");
  std::vector<int32_t> cell(n), cnt(nc + 1, 0);
  for (size_t a = 0; a < n; a++) {
    size_t cx = (size_t)((x[3 * a] - H.ox) * H.inv), cy = (size_t)((x[3 * a + 1] - H.oy) * H.inv),
           cz = (size_t)((x[3 * a + 2] - H.oz) * H.inv);
    cell[a] = (int32_t)(cx + (size_t)H.gx * (cy + (size_t)H.gy * cz));
    cnt[cell[a] + 1]++;
  }
  for (size_t c = 0; c < nc; c++) cnt[c + 1] += cnt[c];
  H.start = cnt;
  H.atoms.assign(n, 0);
  std::vector<int32_t> cur(cnt.begin(), cnt.end() - 1);
  for (size_t a = 0; a < n; a++) H.atoms[cur[cell[a]]++] = (int32_t)a;  // atom order within a cell
  return H;
}

// Trilinear charge spreading (pb_grid.rs:220-292) summed in atom order; the
// result is sparse (8 points per atom) and scattered on the device.
static void spread_charges(const PbGeom& g, const std::vector<double>& x, const std::vector<double>& q,
                           std::vector<int64_t>& idx, std::vector<double>& val) {
  idx.clear();
  val.clear();
  long nx = g.nx, ny = g.ny, nz = g.nz;
  double org[3] = {g.ox, g.oy, g.oz};
  // open-addressing table: grid index -> position in idx/val (first-touch order)
  size_t cap = 64;
  while (cap < 16 * q.size() + 16) cap <<= 1;
  std::vector<int64_t> key(cap, -1);
  std::vector<int32_t> pos(cap, 0);
  idx.reserve(8 * q.size());
  val.reserve(8 * q.size());
  for (size_t a = 0; a < q.size(); a++) {
    double fc[3];
    for (int d = 0; d < 3; d++) fc[d] = (x[3 * a + d] - org[d]) / g.h;
    long ix = (long)std::floor(fc[0]), iy = (long)std::floor(fc[1]), iz = (long)std::floor(fc[2]);
    if (ix < 0 || ix >= nx - 1 || iy < 0 || iy >= ny - 1 || iz < 0 || iz >= nz - 1) continue;
    double dx = fc[0] - (double)ix, dy = fc[1] - (double)iy, dz = fc[2] - (double)iz;
    double vol = g.h * g.h * g.h;
    double qd = q[a] / vol;
    double wx[2] = {1.0 - dx, dx}, wy[2] = {1.0 - dy, dy}, wz[2] = {1.0 - dz, dz};
    for (int a0 = 0; a0 < 2; a0++)
      for (int a1 = 0; a1 < 2; a1++)
        for (int a2 = 0; a2 < 2; a2++) {
          int64_t k = (ix + a0) + nx * ((iy + a1) + ny * (iz + a2));
          double v = qd * wx[a0] * wy[a1] * wz[a2];
          size_t h = (size_t)((uint64_t)k * 0x9E3779B97F4A7C15ull >> 20) & (cap - 1);
          while (key[h] != -1 && key[h] != k) h = (h + 1) & (cap - 1);
          if (key[h] == -1) {  // grid point first touched: 0.0 + v (pb_grid.rs:280-288)
            key[h] = k;
            pos[h] = (int32_t)val.size();
            idx.push_back(k);
            val.push_back(0.0 + v);
          } else {
            val[pos[h]] += v;
          }
        }
  }
}

// ---------------------------------------------------------------------------
// device: grid set-up
// ---------------------------------------------------------------------------
struct HashDev {
  double inv, ox, oy, oz;
  int gx, gy, gz;
  const int* start;
  const int* atoms;
};

struct GeomDev {
  int nx, ny, nz;
  double h, ox, oy, oz;
};

__device__ __forceinline__ void grid_point(const GeomDev& g, int ix, int iy, int iz, double* p) {
  p[0] = g.ox + (double)ix * g.h;
  p[1] = g.oy + (double)iy * g.h;
  p[2] = g.oz + (double)iz * g.h;
}

__device__ bool hash_inside(const HashDev& H, const double* p, const double* __restrict__ xyz,
                            const double* __restrict__ radii, double probe) {
  if (H.gx == 0) return false;
  long cx = (long)((p[0] - H.ox) * H.inv), cy = (long)((p[1] - H.oy) * H.inv), cz = (long)((p[2] - H.oz) * H.inv);
  for (long dz = -1; dz <= 1; dz++) {
    long jz = cz + dz;
    if (jz < 0 || jz >= H.gz) continue;
    for (long dy = -1; dy <= 1; dy++) {
      long jy = cy + dy;
      if (jy < 0 || jy >= H.gy) continue;
      for (long dx = -1; dx <= 1; dx++) {
        long jx = cx + dx;
        if (jx < 0 || jx >= H.gx) continue;
        long c = jx + (long)H.gx * (jy + (long)H.gy * jz);
        for (int k = H.start[c]; k < H.start[c + 1]; k++) {
          int a = H.atoms[k];
          double ddx = p[0] - xyz[3 * a], ddy = p[1] - xyz[3 * a + 1], ddz = p[2] - xyz[3 * a + 2];
          double d2 = ddx * ddx + ddy * ddy + ddz * ddz;
          double th = radii[a] + probe;
          if (d2 < th * th) return true;
        }
      }
    }
  }
  return false;
}

__global__ void k_inside(GeomDev g, HashDev H, const double* __restrict__ xyz, const double* __restrict__ radii,
                         double probe, uint8_t* __restrict__ out) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long n = (long long)g.nx * g.ny * g.nz;
  if (idx >= n) return;
  int iz = (int)(idx / ((long long)g.nx * g.ny)), iy = (int)((idx / g.nx) % g.ny), ix = (int)(idx % g.nx);
  double p[3];
  grid_point(g, ix, iy, iz, p);
  out[idx] = hash_inside(H, p, xyz, radii, probe) ? 1 : 0;
}

__global__ void k_kappa(GeomDev g, HashDev H, const double* __restrict__ xyz, const double* __restrict__ radii,
                        double ion, double kbs, double* __restrict__ out) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long n = (long long)g.nx * g.ny * g.nz;
  if (idx >= n) return;
  int iz = (int)(idx / ((long long)g.nx * g.ny)), iy = (int)((idx / g.nx) % g.ny), ix = (int)(idx % g.nx);
  double p[3];
  grid_point(g, ix, iy, iz, p);
  out[idx] = hash_inside(H, p, xyz, radii, ion) ? 0.0 : kbs;
}

__global__ void k_flood_seed(GeomDev g, const uint8_t* __restrict__ sas, uint8_t* __restrict__ ext) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long n = (long long)g.nx * g.ny * g.nz;
  if (idx >= n) return;
  int iz = (int)(idx / ((long long)g.nx * g.ny)), iy = (int)((idx / g.nx) % g.ny), ix = (int)(idx % g.nx);
  bool bd = ix == 0 || ix == g.nx - 1 || iy == 0 || iy == g.ny - 1 || iz == 0 || iz == g.nz - 1;
  ext[idx] = (bd && !sas[idx]) ? 1 : 0;
}

// One propagation pass of the connected exterior (pb_grid.rs:621-686) over
// 8^3 tiles: inside a tile the front advances until it stops, across tiles
// through repeated launches until no point changes.  The fixed point is the
// set of outside-SAS points 6-connected to an outside-SAS boundary point,
// whatever the visiting order.  With act_in, only tiles marked there run; a
// tile that grew marks itself and its six face neighbours in act_out.
__global__ void k_flood(GeomDev g, const uint8_t* __restrict__ sas, uint8_t* __restrict__ ext, int* changed,
                        const uint8_t* __restrict__ act_in, uint8_t* __restrict__ act_out) {
  __shared__ uint8_t se[10][10][10], ss[10][10][10];
  int tile = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  if (act_in && !act_in[tile]) return;
  int tx = threadIdx.x, ty = threadIdx.y, tz = threadIdx.z;
  int bx = blockIdx.x * 8, by = blockIdx.y * 8, bz = blockIdx.z * 8;
  int t = tx + 8 * (ty + 8 * tz);
  for (int k = t; k < 1000; k += 512) {
    int hx = k % 10, hy = (k / 10) % 10, hz = k / 100;
    int gx = bx + hx - 1, gy = by + hy - 1, gz = bz + hz - 1;
    bool in = gx >= 0 && gx < g.nx && gy >= 0 && gy < g.ny && gz >= 0 && gz < g.nz;
    long long gi = in ? gx + (long long)g.nx * (gy + (long long)g.ny * gz) : 0;
    se[hz][hy][hx] = in ? ext[gi] : 0;
    ss[hz][hy][hx] = in ? sas[gi] : 1;
  }
  __syncthreads();
  int ix = bx + tx, iy = by + ty, iz = bz + tz;
  bool mine = ix < g.nx && iy < g.ny && iz < g.nz;
  bool grew = false;
  for (int it = 0; it < 512; it++) {
    int c = 0;
    if (mine && !ss[tz + 1][ty + 1][tx + 1] && !se[tz + 1][ty + 1][tx + 1]) {
      if (se[tz + 1][ty + 1][tx] | se[tz + 1][ty + 1][tx + 2] | se[tz + 1][ty][tx + 1] | se[tz + 1][ty + 2][tx + 1] |
          se[tz][ty + 1][tx + 1] | se[tz + 2][ty + 1][tx + 1])
        c = 1;
    }
    __syncthreads();
    if (c) {
      se[tz + 1][ty + 1][tx + 1] = 1;
      grew = true;
    }
    if (!__syncthreads_or(c)) break;
  }
  if (grew) ext[ix + (long long)g.nx * (iy + (long long)g.ny * iz)] = 1;
  if (__syncthreads_or(grew) && t == 0) {
    atomicExch(changed, 1);
    if (act_out) {
      int X = blockIdx.x, Y = blockIdx.y, Z = blockIdx.z, NX = gridDim.x, NY = gridDim.y, NZ = gridDim.z;
      act_out[tile] = 1;
      if (X > 0) act_out[tile - 1] = 1;
      if (X + 1 < NX) act_out[tile + 1] = 1;
      if (Y > 0) act_out[tile - NX] = 1;
      if (Y + 1 < NY) act_out[tile + NX] = 1;
      if (Z > 0) act_out[tile - NX * NY] = 1;
      if (Z + 1 < NZ) act_out[tile + NX * NY] = 1;
    }
  }
}

// SES classification (pb_grid.rs:688-707): a point is outside the SES when a
// connected-exterior point lies within squared index distance thr; the
// squared Euclidean distance transform there is an exact integer, so testing
// the integer offsets of the ball gives the same answer.
__global__ void k_ses(GeomDev g, const uint8_t* __restrict__ ext, const int4* __restrict__ offs, int noffs,
                      uint8_t* __restrict__ inside) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long n = (long long)g.nx * g.ny * g.nz;
  if (idx >= n) return;
  int iz = (int)(idx / ((long long)g.nx * g.ny)), iy = (int)((idx / g.nx) % g.ny), ix = (int)(idx % g.nx);
  bool out = false;
  for (int k = 0; k < noffs && !out; k++) {
    int4 o = offs[k];
    int x = ix + o.x, y = iy + o.y, z = iz + o.z;
    if (x < 0 || x >= g.nx || y < 0 || y >= g.ny || z < 0 || z >= g.nz) continue;
    out = ext[x + (long long)g.nx * (y + (long long)g.ny * z)] != 0;
  }
  inside[idx] = out ? 0 : 1;
}

constexpr int kMaxIntervals = 64;

// fraction_inside_along_axis (pb_grid.rs:717-801) with probe 0, candidate
// atoms from a hash whose cells are at least max radius + h wide.
__device__ double edge_fraction(const HashDev& H, const double* __restrict__ xyz, const double* __restrict__ radii,
                                double lo, double hi, double p1, double p2, int axis, const double* pt, int* ovf) {
  double len = hi - lo;
  if (len <= 0.0) return 0.0;
  int a1 = axis == 0 ? 1 : 0, a2 = axis == 2 ? 1 : 2;
  double ilo_[kMaxIntervals], ihi_[kMaxIntervals];
  int m = 0;
  long cx = (long)((pt[0] - H.ox) * H.inv), cy = (long)((pt[1] - H.oy) * H.inv), cz = (long)((pt[2] - H.oz) * H.inv);
  for (long dz = -1; dz <= 1; dz++) {
    long jz = cz + dz;
    if (jz < 0 || jz >= H.gz) continue;
    for (long dy = -1; dy <= 1; dy++) {
      long jy = cy + dy;
      if (jy < 0 || jy >= H.gy) continue;
      for (long dx = -1; dx <= 1; dx++) {
        long jx = cx + dx;
        if (jx < 0 || jx >= H.gx) continue;
        long c = jx + (long)H.gx * (jy + (long)H.gy * jz);
        for (int k = H.start[c]; k < H.start[c + 1]; k++) {
          int a = H.atoms[k];
          double R = radii[a] + 0.0;
          double d1 = p1 - xyz[3 * a + a1], d2 = p2 - xyz[3 * a + a2];
          double rs = R * R - d1 * d1 - d2 * d2;
          if (rs <= 0.0) continue;
          double rho = sqrt(rs);
          double ca = xyz[3 * a + axis];
          double l = fmax(ca - rho, lo), u = fmin(ca + rho, hi);
          if (l < u) {
            if (m == kMaxIntervals) {
              atomicExch(ovf, 1);
              continue;
            }
            int p = m++;  // insertion by start
            while (p > 0 && ilo_[p - 1] > l) {
              ilo_[p] = ilo_[p - 1];
              ihi_[p] = ihi_[p - 1];
              p--;
            }
            ilo_[p] = l;
            ihi_[p] = u;
          }
        }
      }
    }
  }
  if (m == 0) return 0.0;
  double total = 0.0, clo = ilo_[0], chi = ihi_[0];
  for (int k = 1; k < m; k++) {
    if (ilo_[k] <= chi) {
      chi = fmax(chi, ihi_[k]);
    } else {
      total += chi - clo;
      clo = ilo_[k];
      chi = ihi_[k];
    }
  }
  total += chi - clo;
  return fmin(1.0, fmax(0.0, total / len));
}

__device__ __forceinline__ double harmonic(double f, double ein, double eout) {  // pb_grid.rs:809-817
  if (f <= 0.0) return eout;
  if (f >= 1.0) return ein;
  return 1.0 / (f / ein + (1.0 - f) / eout);
}

__global__ void k_eps(GeomDev g, const uint8_t* __restrict__ inside, HashDev H, const double* __restrict__ xyz,
                      const double* __restrict__ radii, double ein, double eout, double* __restrict__ ex,
                      double* __restrict__ ey, double* __restrict__ ez, int* ovf) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long n = (long long)g.nx * g.ny * g.nz;
  if (idx >= n) return;
  int iz = (int)(idx / ((long long)g.nx * g.ny)), iy = (int)((idx / g.nx) % g.ny), ix = (int)(idx % g.nx);
  bool a = inside[idx];
  double p[3];
  grid_point(g, ix, iy, iz, p);
  double vx = eout, vy = eout, vz = eout;
  if (ix + 1 < g.nx) {
    bool b = inside[idx + 1];
    vx = a == b ? (a ? ein : eout)
                : harmonic(edge_fraction(H, xyz, radii, p[0], p[0] + g.h, p[1], p[2], 0, p, ovf), ein, eout);
  }
  if (iy + 1 < g.ny) {
    bool b = inside[idx + g.nx];
    vy = a == b ? (a ? ein : eout)
                : harmonic(edge_fraction(H, xyz, radii, p[1], p[1] + g.h, p[0], p[2], 1, p, ovf), ein, eout);
  }
  if (iz + 1 < g.nz) {
    bool b = inside[idx + (long long)g.nx * g.ny];
    vz = a == b ? (a ? ein : eout)
                : harmonic(edge_fraction(H, xyz, radii, p[2], p[2] + g.h, p[0], p[1], 2, p, ovf), ein, eout);
  }
  ex[idx] = vx;
  ey[idx] = vy;
  ez[idx] = vz;
}

__global__ void k_fill(double* __restrict__ a, long long n, double v) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = v;
}

__global__ void k_scatter(const long long* __restrict__ idx, const double* __restrict__ val, int m,
                          double* __restrict__ out) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m) out[idx[k]] = val[k];
}

// Boundary points of a grid enumerated face by face: the two z faces, the
// two y faces of the interior z planes, the two x faces of the interior
// rows.  Grids one or two points thick name some points twice (the same
// value is written twice).
__device__ __forceinline__ bool boundary_point(const GeomDev& g, long long k, int& ix, int& iy, int& iz) {
  long long nxy = (long long)g.nx * g.ny;
  int nzi = max(g.nz - 2, 0), nyi = max(g.ny - 2, 0);
  if (k < 2 * nxy) {
    iz = k < nxy ? 0 : g.nz - 1;
    long long r = k % nxy;
    ix = (int)(r % g.nx);
    iy = (int)(r / g.nx);
    return true;
  }
  k -= 2 * nxy;
  long long nyf = (long long)g.nx * nzi;
  if (k < 2 * nyf) {
    iy = k < nyf ? 0 : g.ny - 1;
    long long r = k % nyf;
    ix = (int)(r % g.nx);
    iz = 1 + (int)(r / g.nx);
    return true;
  }
  k -= 2 * nyf;
  long long nxf = (long long)nyi * nzi;
  if (k < 2 * nxf) {
    ix = k < nxf ? 0 : g.nx - 1;
    long long r = k % nxf;
    iy = 1 + (int)(r % nyi);
    iz = 1 + (int)(r / nyi);
    return true;
  }
  return false;
}

static long long boundary_count(const PbGeom& g) {
  long long nzi = std::max(g.nz - 2, 0), nyi = std::max(g.ny - 2, 0);
  return 2LL * g.nx * g.ny + 2LL * g.nx * nzi + 2LL * nyi * nzi;
}

// set_dh_boundary, pb_solver.rs:68-93: atoms summed in order per boundary
// point (pb_solver.rs:31-60 visits every point of a grid that is one or two
// points thick; those points are all boundary points).
__global__ void k_dh(GeomDev g, long long nbnd, const double* __restrict__ xyz, const double* __restrict__ q, int na,
                     double kap, double eout, double* __restrict__ phi) {
  __shared__ double sx[256], sy[256], sz[256], sq[256];
  long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int ix = 0, iy = 0, iz = 0;
  bool valid = k < nbnd && boundary_point(g, k, ix, iy, iz);
  double p[3];
  grid_point(g, ix, iy, iz, p);
  double s = 0.0;
  const double conv = 332.0522;
  for (int a0 = 0; a0 < na; a0 += 256) {
    int a = a0 + threadIdx.x;
    if (a < na) {
      sx[threadIdx.x] = xyz[3 * a];
      sy[threadIdx.x] = xyz[3 * a + 1];
      sz[threadIdx.x] = xyz[3 * a + 2];
      sq[threadIdx.x] = q[a];
    }
    __syncthreads();
    int m = min(256, na - a0);
    if (valid)
      for (int j = 0; j < m; j++) {
        double dx = p[0] - sx[j], dy = p[1] - sy[j], dz = p[2] - sz[j];
        double r = sqrt(dx * dx + dy * dy + dz * dz);
        if (r > 1e-10) s += conv * sq[j] * exp(-kap * r) / (eout * r);
      }
    __syncthreads();
  }
  if (valid) phi[ix + (long long)g.nx * (iy + (long long)g.ny * iz)] = s;
}

// Focusing boundary: fine boundary values interpolated from the coarse
// potential (pb_solver.rs:100-114, pb_grid.rs:142-182).
__global__ void k_interp_boundary(GeomDev f, GeomDev c, const double* __restrict__ cphi, double* __restrict__ phi) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)f.nx * f.ny * f.nz) return;
  int iz = (int)(idx / ((long long)f.nx * f.ny)), iy = (int)((idx / f.nx) % f.ny), ix = (int)(idx % f.nx);
  if (!(ix == 0 || ix == f.nx - 1 || iy == 0 || iy == f.ny - 1 || iz == 0 || iz == f.nz - 1)) return;
  double p[3];
  grid_point(f, ix, iy, iz, p);
  double fc[3] = {(p[0] - c.ox) / c.h, (p[1] - c.oy) / c.h, (p[2] - c.oz) / c.h};
  long cx = (long)floor(fc[0]), cy = (long)floor(fc[1]), cz = (long)floor(fc[2]);
  double v = 0.0;
  if (!(cx < 0 || cx >= c.nx - 1 || cy < 0 || cy >= c.ny - 1 || cz < 0 || cz >= c.nz - 1)) {
    double dx = fc[0] - (double)cx, dy = fc[1] - (double)cy, dz = fc[2] - (double)cz;
    auto at = [&](long x, long y, long z) { return cphi[x + (long)c.nx * (y + (long)c.ny * z)]; };
    double c00 = at(cx, cy, cz) * (1.0 - dx) + at(cx + 1, cy, cz) * dx;
    double c10 = at(cx, cy + 1, cz) * (1.0 - dx) + at(cx + 1, cy + 1, cz) * dx;
    double c01 = at(cx, cy, cz + 1) * (1.0 - dx) + at(cx + 1, cy, cz + 1) * dx;
    double c11 = at(cx, cy + 1, cz + 1) * (1.0 - dx) + at(cx + 1, cy + 1, cz + 1) * dx;
    double c0 = c00 * (1.0 - dy) + c10 * dy, c1 = c01 * (1.0 - dy) + c11 * dy;
    v = c0 * (1.0 - dz) + c1 * dz;
  }
  phi[idx] = v;
}

// ---------------------------------------------------------------------------
// device: multigrid (pb_solver.rs)
// ---------------------------------------------------------------------------
struct LevelDev {
  int nx, ny, nz;
  double ihx, ihy, ihz;
  const double *ex, *ey, *ez, *k2;
};

__device__ __forceinline__ void stencil(const LevelDev& L, const double* __restrict__ phi, long long idx,
                                        double& ns, double& dg) {
  long long sy = L.nx, sz = (long long)L.nx * L.ny;
  double exp_ = L.ex[idx], exm = L.ex[idx - 1], eyp = L.ey[idx], eym = L.ey[idx - sy], ezp = L.ez[idx],
         ezm = L.ez[idx - sz];
  ns = (exp_ * phi[idx + 1] + exm * phi[idx - 1]) * L.ihx + (eyp * phi[idx + sy] + eym * phi[idx - sy]) * L.ihy +
       (ezp * phi[idx + sz] + ezm * phi[idx - sz]) * L.ihz;
  dg = (exp_ + exm) * L.ihx + (eyp + eym) * L.ihy + (ezp + ezm) * L.ihz + L.k2[idx];
}

// one colour of a red-black SOR sweep (pb_solver.rs:250-317) with per-block
// sums of (phi_GS - phi)^2 for the plain-SOR convergence test
__global__ void k_rb(LevelDev L, double* __restrict__ phi, const double* __restrict__ rho, double omega,
                     double rhs_scale, int color, double* __restrict__ rms_part) {
  __shared__ double sh[32];
  int iy = blockIdx.y + 1, iz = blockIdx.z + 1;
  int x0 = 1 + ((1 + iy + iz + color) & 1);
  int ix = x0 + 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  double r2 = 0.0;
  if (ix < L.nx - 1) {
    long long idx = ix + (long long)L.nx * (iy + (long long)L.ny * iz);
    double ns, dg;
    stencil(L, phi, idx, ns, dg);
    double rhs = rhs_scale * rho[idx];
    double gs = (ns + rhs) / dg;
    double old = phi[idx];
    double res = gs - old;
    r2 = res * res;
    phi[idx] = old + omega * (gs - old);
  }
  double s = block_sum(r2, sh);
  if (threadIdx.x == 0) rms_part[blockIdx.x + gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z)] = s;
}

__global__ void k_residual(LevelDev L, const double* __restrict__ phi, const double* __restrict__ rho,
                           double rhs_scale, double* __restrict__ sq_part) {
  __shared__ double sh[32];
  int ix = 1 + blockIdx.x * blockDim.x + threadIdx.x, iy = blockIdx.y + 1, iz = blockIdx.z + 1;
  double r2 = 0.0;
  if (ix < L.nx - 1) {
    long long idx = ix + (long long)L.nx * (iy + (long long)L.ny * iz);
    double ns, dg;
    stencil(L, phi, idx, ns, dg);
    double r = rhs_scale * rho[idx] + ns - dg * phi[idx];
    r2 = r * r;
  }
  double s = block_sum(r2, sh);
  if (threadIdx.x == 0) sq_part[blockIdx.x + gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z)] = s;
}

// Injection coarsening of the maps src[k] into dst[k], k = blockIdx.y.
struct Coarsen {
  const double* src[8];
  double* dst[8];
};
__global__ void k_coarsen(Coarsen m, int fnx, int fny, int fnz, int cnx, int cny, int cnz) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)cnx * cny * cnz) return;
  int cz = (int)(i / ((long long)cnx * cny)), cy = (int)((i / cnx) % cny), cx = (int)(i % cnx);
  int fx = min(2 * cx, fnx - 1), fy = min(2 * cy, fny - 1), fz = min(2 * cz, fnz - 1);
  m.dst[blockIdx.y][i] = m.src[blockIdx.y][fx + (long long)fnx * (fy + (long long)fny * fz)];
}

// Coarse face dielectric of the relative-residual mode: two fine faces in
// series along the face's axis (harmonic mean; equal values copied), the
// 3 x 3 neighbouring lines across it in parallel (weights 1-2-1 per
// transverse direction, renormalised at the grid edge).
__global__ void k_coarsen_face(const double* __restrict__ f, int fnx, int fny, int fnz, double* __restrict__ c,
                               int cnx, int cny, int cnz, int axis) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)cnx * cny * cnz) return;
  int cz = (int)(i / ((long long)cnx * cny)), cy = (int)((i / cnx) % cny), cx = (int)(i % cnx);
  const int n[3] = {fnx, fny, fnz};
  const int b[3] = {min(2 * cx, fnx - 1), min(2 * cy, fny - 1), min(2 * cz, fnz - 1)};
  const int t1 = axis == 0 ? 1 : 0, t2 = axis == 2 ? 1 : 2;
  double sum = 0.0, ws = 0.0, first = 0.0;
  bool same = true, any = false;
  for (int u = -1; u <= 1; u++)
    for (int v = -1; v <= 1; v++) {
      int p[3] = {b[0], b[1], b[2]};
      p[t1] += u;
      p[t2] += v;
      if (p[t1] < 0 || p[t1] >= n[t1] || p[t2] < 0 || p[t2] >= n[t2]) continue;
      int q[3] = {p[0], p[1], p[2]};
      q[axis] = min(p[axis] + 1, n[axis] - 1);
      const double e0 = f[p[0] + (long long)fnx * (p[1] + (long long)fny * p[2])];
      const double e1 = f[q[0] + (long long)fnx * (q[1] + (long long)fny * q[2])];
      if (!any) first = e0;
      any = true;
      same = same && e0 == first && e1 == first;
      const double w = (u == 0 ? 2.0 : 1.0) * (v == 0 ? 2.0 : 1.0);
      sum += w * (e0 == e1 ? e0 : 2.0 / (1.0 / e0 + 1.0 / e1));
      ws += w;
    }
  c[i] = same ? first : sum / ws;
}

// ---------------------------------------------------------------------------
// Multigrid cycles (pb_solver.rs:1015-1167) of one or two solves on one grid
// in one cooperative launch: `blocks` blocks a solve, a barrier among them
// where one launch after another stood, and the stopping rule on the device.
//
// A cycle of a 77 x 67 x 67 grid moves 20 MB through L2, a microsecond or two a
// pass; what it costs is the way from one dependent pass to the next.  As 71
// launches and a host synchronisation a cycle of one solve took 395 us; here
// one of both solves side by side takes 195 us: a barrier 1.5 us, a sweep of
// level 0 2.8 (5.5 with the reference's 28 operations and a division a point in
// place of multiply-adds on codes), of level 1 1.0, the block's levels
// together 60.  Energy of 132 atoms with focusing: 34.0 ms as launches, 9.0.
// One block does the levels that fit its shared memory, from lb down, with a
// block barrier a pass.
// ---------------------------------------------------------------------------
constexpr int kMgThreads = 640, kMgLevels = 10;  // 1,024 threads have too few registers (the energy below: 9.8 ms)
constexpr unsigned kMgSpin = 1u << 23;  // polls of a barrier before it gives up (some seconds)

// Counter over n0 x n1 x n2 cells in steps of a block's threads: (d0, d1, d2)
// is that step in mixed radix.  Each block takes one run of `per` cells, so
// that every SM has the same share and a row's neighbours meet in L1.
struct MgWalk {
  unsigned n0, n1, n2, d0, d1, d2, per;
};
struct MgGeo {
  int nx, ny, nz;
  double ih, om;
  MgWalk half, in, all, pairs;  // points of one colour (an upper bound a row), interior, every point, pairs along x
};
// Coefficients of a point.  Most have one dielectric on all six faces: those
// are named by a code (1, + 2 the second value, + 4 ions, + 8 no charge) and
// take their coefficients from a table of four, so that a sweep reads the
// potential and a byte; the others (code 0) read their faces and `di`, omega
// over the diagonal.  (Lists of the others, to do them with full warps, were no
// faster: one more dependent read a pass.)
struct MgPtr {
  const double *ex, *ey, *ez, *k2;
  double *rhs, *phi, *res, *di;  // rhs of level 0 is the charge density, never written
  uint8_t* code;
};
struct MgState {
  double r0, best, prev, r;
  int growing, cycles, status, pad;  // status: 0 running, 1 converged, 2 diverging, 3 out of cycles, 4 a barrier gave up
};
struct MgArgs {
  MgGeo g[kMgLevels + 1];
  MgPtr p[2][kMgLevels + 1];
  int nlev, lb, blocks, quota, maxv, rel;  // lb > nlev: no level fits shared memory
  double tol, rs, val[2][2], kb[2];  // the two dielectrics and kappa-bar^2 of a solve
  unsigned* bar;  // 32 words a solve
  MgState* st;
  double* part;
};

__device__ __forceinline__ bool mg_barrier(unsigned* ctr, unsigned target) {
  __syncthreads();
  int ok = 1;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
    unsigned v;
    for (unsigned k = 0;; k++) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
      if ((int)(v - target) >= 0) break;
      if (k == kMgSpin) {
        ok = 0;
        break;
      }
    }
  }
  return __syncthreads_and(ok);
}

// First cell of this thread in the walks of the two finest levels' sweeps,
// worked out once: a division costs as much as the rest of a point.
struct MgStart {
  unsigned a, bc;
};
__device__ __forceinline__ MgStart mg_start(const MgWalk& w, unsigned blk) {
  const unsigned t = blk * w.per + threadIdx.x, q = t / w.n0, c = q / w.n1;
  return MgStart{t - q * w.n0, (q - c * w.n1) | c << 16};  // at most 4,096 cells a dimension
}

template <typename Fn>
__device__ __forceinline__ void mg_walk(const MgWalk& w, unsigned blk, const MgStart& at, Fn fn) {
  const unsigned lo = blk * w.per, hi = min(lo + w.per, w.n0 * w.n1 * w.n2);
  unsigned a = at.a, b = at.bc & 0xffffu, c = at.bc >> 16;
  for (unsigned t = lo + threadIdx.x; t < hi; t += kMgThreads) {
    fn(a, b, c);
    a += w.d0;
    b += w.d1;
    c += w.d2;
    if (a >= w.n0) {
      a -= w.n0;
      b++;
    }
    if (b >= w.n1) {
      b -= w.n1;
      c++;
    }
  }
}
template <typename Fn>
__device__ __forceinline__ void mg_walk(const MgWalk& w, unsigned blk, Fn fn) {
  mg_walk(w, blk, mg_start(w, blk), fn);
}

// Codes and `di` of one level, of a solve each blockIdx.y.
struct MgCodes {
  MgPtr p[2];
  double val[2][2], kb[2];
};
__global__ void k_mg_codes(const __grid_constant__ MgCodes A, int nx, int ny, int nz, double ih, double om, int top) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x, sy = nx, sz = (unsigned)nx * ny;
  const unsigned z = i / sz, y = (i - z * sz) / sy, x = i - z * sz - y * sy;
  const int j = blockIdx.y;
  const MgPtr& p = A.p[j];
  const bool inner = x - 1 < (unsigned)nx - 2 && y - 1 < (unsigned)ny - 2 && z - 1 < (unsigned)nz - 2;
  unsigned code = 0;
  if (inner) {
    const double a = p.ex[i], b = p.ex[i - 1], c = p.ey[i], d = p.ey[i - sy], e = p.ez[i], f = p.ez[i - sz], k = p.k2[i];
    p.di[i] = om / (ih * ((a + b) + (c + d) + (e + f)) + k);
    const bool same = a == b && a == c && a == d && a == e && a == f;
    const int v = a == A.val[j][0] ? 0 : a == A.val[j][1] ? 1 : -1;
    if (same && v >= 0 && (k == 0.0 || k == A.kb[j]))
      code = 1 + 2 * v + (k != 0.0 ? 4 : 0) + (top && p.rhs[i] == 0.0 ? 8 : 0);
  }
  if (z < (unsigned)nz) p.code[i] = (uint8_t)code;
}

// Table of a level's plain points: face term, omega over the diagonal, diagonal.
struct MgTab {
  double v, di, dg;
};
__device__ __forceinline__ MgTab mg_tab(const MgGeo& g, double val, double k) {
  MgTab t;
  t.v = val * g.ih;
  t.dg = fma(6.0, t.v, k);
  t.di = g.om / t.dg;
  return t;
}

// A point and its neighbours, read before its code is known.
struct MgNear {
  double f, xp, xm, yp, ym, zp, zm;
};
__device__ __forceinline__ MgNear mg_near(const double* f, unsigned sy, unsigned sz) {
  return MgNear{f[0], f[1], f[-1], f[sy], f[-(int)sy], f[sz], f[-(int)sz]};
}
__device__ __forceinline__ double mg_six(const MgNear& n) { return ((n.xp + n.xm) + (n.yp + n.ym)) + (n.zp + n.zm); }
// The six neighbours' terms of a point with faces of its own, and its diagonal.
__device__ __forceinline__ double mg_faces(const MgGeo& g, const MgPtr& p, unsigned i, const MgNear& n, unsigned sy,
                                           unsigned sz) {
  double u = __ldg(p.ex + i) * n.xp, v = __ldg(p.ex + i - 1) * n.xm;
  u = fma(__ldg(p.ey + i), n.yp, u);
  v = fma(__ldg(p.ey + i - sy), n.ym, v);
  u = fma(__ldg(p.ez + i), n.zp, u);
  v = fma(__ldg(p.ez + i - sz), n.zm, v);
  return g.ih * (u + v);
}
__device__ __forceinline__ double mg_diag(const MgGeo& g, const MgPtr& p, unsigned i, unsigned sy, unsigned sz) {
  return fma(g.ih, (__ldg(p.ex + i) + __ldg(p.ex + i - 1)) + (__ldg(p.ey + i) + __ldg(p.ey + i - sy)) +
                       (__ldg(p.ez + i) + __ldg(p.ez + i - sz)),
             __ldg(p.k2 + i));
}

// phi + omega (phi_GS - phi) of one point (pb_solver.rs:250-317); b: its right-hand side
__device__ __forceinline__ double mg_update(const MgGeo& g, const MgPtr& p, const MgTab* tab, unsigned code, unsigned i,
                                            const MgNear& n, double b, unsigned sy, unsigned sz) {
  const double old = (1.0 - g.om) * n.f;
  if (code & 1) {
    const MgTab& t = tab[(code >> 1) & 3];
    return fma(t.di, fma(t.v, mg_six(n), b), old);
  }
  return fma(__ldg(p.di + i), mg_faces(g, p, i, n, sy, sz) + b, old);
}
__device__ __forceinline__ double mg_defect(const MgGeo& g, const MgPtr& p, const MgTab* tab, unsigned code, unsigned i,
                                            const MgNear& n, double b, unsigned sy, unsigned sz) {
  if (code & 1) {
    const MgTab& t = tab[(code >> 1) & 3];
    return fma(-t.dg, n.f, fma(t.v, mg_six(n), b));
  }
  return fma(-mg_diag(g, p, i, sy, sz), n.f, mg_faces(g, p, i, n, sy, sz) + b);
}
// right-hand side of a point; on level 0 most have no charge
template <bool kTop>
__device__ __forceinline__ double mg_rhs(const MgPtr& p, unsigned code, unsigned i, double rs) {
  if (!kTop) return p.rhs[i];
  return code & 8 ? 0.0 : rs * p.rhs[i];
}

// one colour of a sweep
template <bool kTop>
__device__ __forceinline__ void mg_sweep(const MgGeo& g, const MgPtr& p, const MgTab* tab, double rs, int colour,
                                         unsigned blk, const MgStart& at) {
  const unsigned sy = g.nx, sz = (unsigned)g.nx * g.ny;
  mg_walk(g.half, blk, at, [&](unsigned a, unsigned b, unsigned c) {
    const unsigned x = 1 + ((1 + b + c + colour) & 1) + 2 * a;
    if (x >= (unsigned)g.nx - 1) return;
    const unsigned i = x + sy * (b + 1) + sz * (c + 1);
    const unsigned code = __ldg(p.code + i);
    const MgNear n = mg_near(p.phi + i, sy, sz);
    p.phi[i] = mg_update(g, p, tab, code, i, n, mg_rhs<kTop>(p, code, i, rs), sy, sz);
  });
}

// residual into res (whose boundary is never read), or the sum of its squares
template <bool kTop, bool kNorm>
__device__ __forceinline__ double mg_residual(const MgGeo& g, const MgPtr& p, const MgTab* tab, double rs, unsigned blk) {
  const unsigned sy = g.nx, sz = (unsigned)g.nx * g.ny;
  double sum = 0.0;
  mg_walk(g.in, blk, [&](unsigned a, unsigned b, unsigned c) {
    const unsigned i = a + 1 + sy * (b + 1) + sz * (c + 1);
    const unsigned code = __ldg(p.code + i);
    const MgNear n = mg_near(p.phi + i, sy, sz);
    const double r = mg_defect(g, p, tab, code, i, n, mg_rhs<kTop>(p, code, i, rs), sy, sz);
    if (kNorm)
      sum = fma(r, r, sum);
    else
      p.res[i] = r;
  });
  return sum;
}

// Full weighting of the fine residual at one inner coarse point: all 27 fine
// points lie inside the fine grid's boundary.  (A coarse boundary point's
// right-hand side is never read.)
__device__ __forceinline__ double mg_restrict(const MgGeo& f, const double* res, unsigned cx, unsigned cy, unsigned cz,
                                              double scale) {
  const int sy = f.nx, sz = f.nx * f.ny;
  const double* q = res + (2 * cx + sy * (2 * cy) + (unsigned)sz * (2 * cz));
  auto row = [&](int o) { return fma(2.0, q[o], q[o - 1] + q[o + 1]); };
  auto plane = [&](int o) { return fma(2.0, row(o), row(o - sy) + row(o + sy)); };
  return scale * 0.015625 * fma(2.0, plane(0), plane(-sz) + plane(sz));
}

// Trilinear coarse correction c at the fine points 2 px and 2 px + 1 of a row.
__device__ __forceinline__ void mg_prolong(const MgGeo& cg, const double* c, unsigned px, unsigned fy, unsigned fz,
                                           double* even, double* odd) {
  const int mx = cg.nx >= 2 ? cg.nx - 2 : 0, my = cg.ny >= 2 ? cg.ny - 2 : 0, mz = cg.nz >= 2 ? cg.nz - 2 : 0;
  const int x0 = min((int)px, mx), y0 = min((int)(fy >> 1), my), z0 = min((int)(fz >> 1), mz);
  const double dx = (double)((int)px - x0), dy = (double)(int)(fy - 2 * y0) * 0.5, dz = (double)(int)(fz - 2 * z0) * 0.5;
  const unsigned sy = cg.nx, sz = (unsigned)cg.nx * cg.ny;
  const double* q = c + (x0 + sy * y0 + sz * z0);
  auto lerp = [](double a, double b, double t) { return fma(t, b - a, a); };
  const double l = lerp(lerp(q[0], q[sy], dy), lerp(q[sz], q[sz + sy], dy), dz);
  const double r = lerp(lerp(q[1], q[sy + 1], dy), lerp(q[sz + 1], q[sz + sy + 1], dy), dz);
  *even = lerp(l, r, dx);
  *odd = lerp(l, r, dx + 0.5);
}
// that correction added to the row's points of e; skip: not on the boundary
__device__ __forceinline__ void mg_correct(const MgGeo& g, const MgGeo& cg, const double* c, double* e, unsigned px,
                                           unsigned y, unsigned z, bool skip) {
  const bool edge = y == 0 || z == 0 || y == (unsigned)g.ny - 1 || z == (unsigned)g.nz - 1;
  if (skip && edge) return;
  double a, b;
  mg_prolong(cg, c, px, y, z, &a, &b);
  const unsigned x = 2 * px;
  double* at = e + (x + g.nx * (y + g.ny * z));
  if (!skip || (x > 0 && x + 1 < (unsigned)g.nx)) at[0] += a;
  if (x + 1 < (unsigned)g.nx && (!skip || x + 2 < (unsigned)g.nx)) at[1] += b;
}

// Points of one colour for a thread of the block: a fixed pair of x and a y,
// walking along z, so that no division stands in the loop.
struct MgLine {
  int x0, y, z0, dz, pair, per, K;
};
__device__ __forceinline__ MgLine mg_line(const MgGeo& g) {
  MgLine l;
  l.K = (g.nx - 1) >> 1;
  l.per = l.K * (g.ny - 2);
  const int t = threadIdx.x;
  if (l.per <= kMgThreads) {
    l.dz = kMgThreads / l.per;
    const int q = t / l.per;
    l.pair = t - q * l.per;
    l.z0 = q < l.dz ? 1 + q : g.nz;
  } else {
    l.dz = 1;
    l.z0 = 1;
    l.pair = t;
  }
  l.y = 1 + l.pair / l.K;
  l.x0 = 1 + 2 * (l.pair % l.K);
  return l;
}
template <typename Fn>
__device__ __forceinline__ void mg_line_points(const MgGeo& g, const MgLine& l, int colour, Fn fn) {
  const int sy = g.nx, sz = g.nx * g.ny;
  int x0 = l.x0, y = l.y;
  for (int r = l.pair;;) {
    if (r < l.per)
      for (int z = l.z0; z <= g.nz - 2; z += l.dz) {
        const int x = x0 + ((1 + y + z + colour) & 1);
        if (x <= g.nx - 2) fn(x + sy * y + sz * z);
      }
    if (l.per <= kMgThreads || (r += kMgThreads) >= l.per) break;
    y = 1 + r / l.K;
    x0 = 1 + 2 * (r % l.K);
  }
}

// One colour of a sweep by one block, on shared memory.
__device__ __forceinline__ void mg_block_sweep(const MgGeo& g, const MgPtr& p, const MgTab* tab, const MgLine& l,
                                               double* e, const double* rhs, const uint8_t* code, int colour) {
  const int sy = g.nx, sz = g.nx * g.ny;
  mg_line_points(g, l, colour, [&](int i) {
    e[i] = mg_update(g, p, tab, code[i], i, mg_near(e + i, sy, sz), rhs[i], sy, sz);
  });
  __syncthreads();
}

// 50 sweeps of the coarsest level in shared memory.  With one point of each
// colour a thread their coefficients stay in registers, with omega over the
// diagonal multiplied in, so that a colour is four dependent multiply-adds;
// only the warps that own points take part (barrier 1).
__device__ __forceinline__ void mg_coarsest(const MgGeo& g, const MgPtr& p, const MgTab* tab, double* e,
                                            const double* rhs, const uint8_t* code) {
  if (g.nx < 3 || g.ny < 3 || g.nz < 3) return;
  const int sy = g.nx, sz = g.nx * g.ny, K = (g.nx - 1) >> 1, need = K * (g.ny - 2) * (g.nz - 2), t = threadIdx.x;
  if (need <= kMgThreads) {
    const int part = (need + 31) & ~31;
    if (t >= part) return;
    const int a = t % K, b = (t / K) % (g.ny - 2), c = t / (K * (g.ny - 2));
    double co[2][6], b0[2], val[2];
    int id[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int x = 1 + ((1 + b + c + k) & 1) + 2 * a;
      id[k] = t < need && x < g.nx - 1 ? x + sy * (b + 1) + sz * (c + 1) : 0;
      if (!id[k]) continue;
      const double di = p.di[id[k]], u = di * g.ih;
      co[k][0] = u * p.ex[id[k]];
      co[k][1] = u * p.ex[id[k] - 1];
      co[k][2] = u * p.ey[id[k]];
      co[k][3] = u * p.ey[id[k] - sy];
      co[k][4] = u * p.ez[id[k]];
      co[k][5] = u * p.ez[id[k] - sz];
      b0[k] = di * rhs[id[k]];
      val[k] = e[id[k]];
    }
    const double rest = 1.0 - g.om;
    for (int s = 0; s < 50; s++) {
#pragma unroll
      for (int k = 0; k < 2; k++) {
        if (id[k]) {
          const double* f = e + id[k];
          double u = fma(co[k][0], f[1], fma(rest, val[k], b0[k])), v = co[k][1] * f[-1];
          u = fma(co[k][2], f[sy], u);
          v = fma(co[k][3], f[-sy], v);
          u = fma(co[k][4], f[sz], u);
          v = fma(co[k][5], f[-sz], v);
          val[k] = u + v;
          e[id[k]] = val[k];
        }
        asm volatile("bar.sync 1, %0;" ::"r"(part) : "memory");
      }
    }
  } else {
    const MgLine l = mg_line(g);
    for (int s = 0; s < 100; s++) mg_block_sweep(g, p, tab, l, e, rhs, code, s & 1);
  }
}

// The cycle from level lb down, by one block: corrections, right-hand sides and
// codes of every level and one residual in shared memory, the faces of points
// that have their own through L1.  `load`: codes, once a launch.
__device__ void mg_bottom(const MgArgs& A, const MgGeo* G, const MgPtr* P, const MgTab (*tab)[4], double* sh,
                          bool load) {
  const int tid = threadIdx.x;
  auto points = [&](int l) { return G[l].nx * G[l].ny * G[l].nz; };
  int all = 0;
  for (int l = A.lb; l <= A.nlev; l++) all += points(l);
  auto first = [&](int l) {
    int o = 0;
    for (int q = A.lb; q < l; q++) o += points(q);
    return o;
  };
  double* const res = sh + 2 * all;
  uint8_t* const codes = reinterpret_cast<uint8_t*>(res + points(A.lb));
  if (load) {
    for (int l = A.lb, o = 0; l <= A.nlev; o += points(l), l++)
      for (int k = tid; k < points(l); k += kMgThreads) codes[o + k] = __ldg(P[l].code + k);
    return;
  }
  const int n = points(A.lb);
#pragma unroll 4
  for (int k = tid; k < n; k += kMgThreads) sh[all + k] = P[A.lb].rhs[k];
  for (int k = tid; k < all; k += kMgThreads) sh[k] = 0.0;
  __syncthreads();
  auto smooth = [&](int l) {
    const MgGeo& g = G[l];
    const MgLine ln = mg_line(g);
    double* e = sh + first(l);
    for (int s = 0; s < 6; s++)
      mg_block_sweep(g, P[l], tab[l], ln, e, e + all, codes + first(l), s & 1);
  };
  for (int l = A.lb; l < A.nlev; l++) {
    const MgGeo &g = G[l], &c = G[l + 1];
    smooth(l);
    double *e = sh + first(l), *ec = sh + first(l + 1);
    const uint8_t* cd = codes + first(l);
    const int sy = g.nx, sz = g.nx * g.ny;
    const MgLine ln = mg_line(g);
    for (int k = 0; k < 2; k++)
      mg_line_points(g, ln, k, [&](int i) {
        res[i] = mg_defect(g, P[l], tab[l], cd[i], i, mg_near(e + i, sy, sz), e[all + i], sy, sz);
      });
    __syncthreads();
    const int ix = c.nx - 2, iy = c.ny - 2;
    for (int k = tid; k < ix * iy * (c.nz - 2); k += kMgThreads) {
      const int q = k / ix, x = k - q * ix + 1, z = q / iy + 1, y = q - (z - 1) * iy + 1;
      ec[all + x + c.nx * (y + c.ny * z)] = mg_restrict(g, res, x, y, z, A.rel ? 1.0 : 0.25);
    }
    __syncthreads();
  }
  mg_coarsest(G[A.nlev], P[A.nlev], tab[A.nlev], sh + first(A.nlev), sh + first(A.nlev) + all, codes + first(A.nlev));
  __syncthreads();
  for (int l = A.nlev - 1; l >= A.lb; l--) {
    const MgGeo& g = G[l];
    const int np = (g.nx + 1) >> 1;
    for (int k = tid; k < np * g.ny * g.nz; k += kMgThreads) {
      const int q = k / np, z = q / g.ny;
      mg_correct(g, G[l + 1], sh + first(l + 1), sh + first(l), k - q * np, q - z * g.ny, z, A.rel);
    }
    __syncthreads();
    smooth(l);
  }
  for (int k = tid; k < points(A.lb); k += kMgThreads) P[A.lb].phi[k] = sh[k];
}

__global__ void __launch_bounds__(kMgThreads, 1) k_mg(const __grid_constant__ MgArgs A) {
  extern __shared__ __align__(16) double mg_sh[];
  __shared__ double red[32];
  __shared__ MgTab tab[kMgLevels + 1][4];
  __shared__ MgStart starts[2][kMgThreads];
  __shared__ MgGeo G[kMgLevels + 1];  // shared memory answers sooner than indexed parameters
  __shared__ MgPtr P[kMgLevels + 1];
  const int job = blockIdx.x / A.blocks, blk = blockIdx.x - job * A.blocks, tid = threadIdx.x;
  MgState S = A.st[job];
  if (S.status != 0) return;
  unsigned* const ctr = A.bar + 32 * job;
  if (tid < 4 * (A.nlev + 1))
    tab[tid >> 2][tid & 3] = mg_tab(A.g[tid >> 2], A.val[job][tid & 1], tid & 2 ? A.kb[job] : 0.0);
  if (tid <= A.nlev) {
    G[tid] = A.g[tid];
    P[tid] = A.p[job][tid];
  }
  __syncthreads();
  for (int l = 0; l < 2 && l < min(A.lb, A.nlev + 1); l++) starts[l][tid] = mg_start(G[l].half, blk);
  if (blk == 0 && A.lb <= A.nlev) mg_bottom(A, G, P, tab, mg_sh, true);
  __syncthreads();
  unsigned passes = 0;
  bool alive = true;
  auto barrier = [&] {
    if (alive) alive = mg_barrier(ctr, ++passes * (unsigned)A.blocks);
  };
  auto norm = [&] {  // RMS residual of level 0, the same bits in every block
    double s = block_sum(mg_residual<true, true>(G[0], P[0], tab[0], A.rs, blk), red);
    if (tid == 0) A.part[job * A.blocks + blk] = s;
    barrier();
    double v = 0.0;
    for (int k = tid; k < A.blocks; k += kMgThreads) v += __ldcg(A.part + job * A.blocks + k);
    v = block_sum(v, red);
    __syncthreads();
    if (tid == 0) red[0] = v;
    __syncthreads();
    v = red[0];
    __syncthreads();
    const double n = (double)(G[0].nx - 2) * (G[0].ny - 2) * (G[0].nz - 2);
    return sqrt(v / n);
  };
  auto smooth = [&](int l) {
    for (int s = 0; s < 6 && alive; s++) {
      if (l == 0)
        mg_sweep<true>(G[0], P[0], tab[0], A.rs, s & 1, blk, starts[0][tid]);
      else
        mg_sweep<false>(G[l], P[l], tab[l], 1.0, s & 1, blk, l == 1 ? starts[1][tid] : mg_start(G[l].half, blk));
      barrier();
    }
  };
  if (A.rel && S.cycles == 0) S.r0 = norm();
  const int split = min(A.lb, A.nlev);  // levels above it are swept by all blocks
  for (int cyc = 0; cyc < A.quota && alive && S.status == 0; cyc++) {
    for (int l = 0; l < split && alive; l++) {
      smooth(l);
      if (l == 0)
        mg_residual<true, false>(G[0], P[0], tab[0], A.rs, blk);
      else
        mg_residual<false, false>(G[l], P[l], tab[l], 1.0, blk);
      barrier();
      const MgGeo &f = G[l], &c = G[l + 1];
      mg_walk(c.all, blk, [&](unsigned x, unsigned y, unsigned z) {
        const unsigned i = x + c.nx * (y + c.ny * z);
        P[l + 1].phi[i] = 0.0;
        if (x - 1 < (unsigned)c.nx - 2 && y - 1 < (unsigned)c.ny - 2 && z - 1 < (unsigned)c.nz - 2)
          P[l + 1].rhs[i] = mg_restrict(f, P[l].res, x, y, z, A.rel ? 1.0 : 0.25);
      });
      barrier();
    }
    if (A.lb <= A.nlev) {
      if (blk == 0 && alive) mg_bottom(A, G, P, tab, mg_sh, false);
      barrier();
    } else if (G[A.nlev].nx >= 3 && G[A.nlev].ny >= 3 && G[A.nlev].nz >= 3) {
      for (int s = 0; s < 100 && alive; s++) {
        mg_sweep<false>(G[A.nlev], P[A.nlev], tab[A.nlev], 1.0, s & 1, blk, mg_start(G[A.nlev].half, blk));
        barrier();
      }
    }
    for (int l = split - 1; l >= 0 && alive; l--) {
      const MgGeo &f = G[l], &c = G[l + 1];
      mg_walk(f.pairs, blk, [&](unsigned px, unsigned y, unsigned z) {
        mg_correct(f, c, P[l + 1].phi, P[l].phi, px, y, z, A.rel);
      });
      barrier();
      smooth(l);
    }
    S.r = norm();
    S.cycles++;
    if (S.r < S.best) {
      S.best = S.r;
      S.growing = 0;
    } else {
      S.growing++;
    }
    if (!isfinite(S.r) || S.r > S.best * 1e4 || (S.growing >= 5 && S.r > S.prev)) {
      S.status = 2;
    } else {
      S.prev = S.r;
      if (A.rel ? S.r < A.tol * S.r0 : S.r < A.tol)
        S.status = 1;
      else if (S.cycles >= A.maxv)
        S.status = 3;
    }
  }
  if (!alive) S.status = 4;
  if (tid == 0 && (blk == 0 || !alive)) A.st[job] = S;
}

__global__ void k_sum_fixed(const double* __restrict__ in, long long n, double* __restrict__ out) {
  __shared__ double sh[32];
  double s = 0.0;
  for (long long i = threadIdx.x; i < n; i += blockDim.x) s += in[i];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) out[0] = s;
}

// Largest |v| into out (zeroed before): the bits of a non-negative double order
// as the value does, and those of a NaN above all (pb_energy.rs:188-194 checks
// finiteness).
__global__ void k_maxabs(const double* __restrict__ in, long long n, unsigned long long* __restrict__ out) {
  unsigned long long m = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    m = max(m, (unsigned long long)__double_as_longlong(fabs(in[i])));
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// compute_elec_energy, pb_solver.rs:1174-1186: trilinear phi at each atom,
// then 0.5 * sum in atom order.
__global__ void k_atom_phi(GeomDev g, const double* __restrict__ phi, const double* __restrict__ xyz,
                           const double* __restrict__ q, int na, double* __restrict__ out) {
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= na) return;
  double fc[3] = {(xyz[3 * a] - g.ox) / g.h, (xyz[3 * a + 1] - g.oy) / g.h, (xyz[3 * a + 2] - g.oz) / g.h};
  long cx = (long)floor(fc[0]), cy = (long)floor(fc[1]), cz = (long)floor(fc[2]);
  double v = 0.0;
  if (!(cx < 0 || cx >= g.nx - 1 || cy < 0 || cy >= g.ny - 1 || cz < 0 || cz >= g.nz - 1)) {
    double dx = fc[0] - (double)cx, dy = fc[1] - (double)cy, dz = fc[2] - (double)cz;
    auto at = [&](long x, long y, long z) { return phi[x + (long)g.nx * (y + (long)g.ny * z)]; };
    double c00 = at(cx, cy, cz) * (1.0 - dx) + at(cx + 1, cy, cz) * dx;
    double c10 = at(cx, cy + 1, cz) * (1.0 - dx) + at(cx + 1, cy + 1, cz) * dx;
    double c01 = at(cx, cy, cz + 1) * (1.0 - dx) + at(cx + 1, cy, cz + 1) * dx;
    double c11 = at(cx, cy + 1, cz + 1) * (1.0 - dx) + at(cx + 1, cy + 1, cz + 1) * dx;
    double c0 = c00 * (1.0 - dy) + c10 * dy, c1 = c01 * (1.0 - dy) + c11 * dy;
    v = c0 * (1.0 - dz) + c1 * dz;
  }
  out[a] = q[a] * v;
}

// One warp: the lanes load ahead, the additions keep atom order.
__global__ void k_seq_sum(const double* __restrict__ in, int n, double* __restrict__ out) {
  double e = 0.0;
  double v = (int)threadIdx.x < n ? in[threadIdx.x] : 0.0;
  for (int a = 0; a < n; a += 32) {
    const double cur = v;
    v = a + 32 + (int)threadIdx.x < n ? in[a + 32 + threadIdx.x] : 0.0;
    const int m = min(32, n - a);
    for (int k = 0; k < m; k++) e += __shfl_sync(0xffffffffu, cur, k);
  }
  if (threadIdx.x == 0) out[0] = 0.5 * e;
}

// ===========================================================================
// host orchestration
// ===========================================================================
static GeomDev gdev(const PbGeom& g) { return GeomDev{g.nx, g.ny, g.nz, g.h, g.ox, g.oy, g.oz}; }

struct HashBuf {
  HashDev d{};
  DevBuf start, atoms;
  HashBuf(const PbHash& H, cudaStream_t st) {
    d.inv = H.inv;
    d.ox = H.ox;
    d.oy = H.oy;
    d.oz = H.oz;
    d.gx = H.gx;
    d.gy = H.gy;
    d.gz = H.gz;
    start = DevBuf(std::max<size_t>(H.start.size(), 1) * 4, st);
    atoms = DevBuf(std::max<size_t>(H.atoms.size(), 1) * 4, st);
    if (!H.start.empty())
      RSTG_CUDA(cudaMemcpyAsync(start.p, H.start.data(), H.start.size() * 4, cudaMemcpyHostToDevice, st));
    if (!H.atoms.empty())
      RSTG_CUDA(cudaMemcpyAsync(atoms.p, H.atoms.data(), H.atoms.size() * 4, cudaMemcpyHostToDevice, st));
    d.start = start.as<int>();
    d.atoms = atoms.as<int>();
  }
};

static unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// Device maps of one grid; MapsView is the non-owning form the solver reads.
struct MapsView {
  PbGeom g;
  const double *rho, *ex, *ey, *ez, *k2;
  double val[2], kb;  // dielectric inside and outside, kappa-bar^2
};

struct Maps {
  PbGeom g;
  DevBuf rho, ex, ey, ez, k2;
};

// Charge map of a grid (sparse host spreading, device scatter) into a
// caller-owned array of g.n() doubles.
static void charge_into(Ctx* c, const PbGeom& g, const AtomsDev& A, double* rho) {
  cudaStream_t st = pb_stream(c);
  RSTG_CUDA(cudaMemsetAsync(rho, 0, g.n() * 8, st));
  std::vector<int64_t> idx;
  std::vector<double> val;
  spread_charges(g, A.hx, A.hq, idx, val);
  if (idx.empty()) return;
  DevBuf di(idx.size() * 8, st), dv(val.size() * 8, st);
  RSTG_CUDA(cudaMemcpyAsync(di.p, idx.data(), idx.size() * 8, cudaMemcpyHostToDevice, st));
  RSTG_CUDA(cudaMemcpyAsync(dv.p, val.data(), val.size() * 8, cudaMemcpyHostToDevice, st));
  k_scatter<<<nblk((long long)idx.size(), 256), 256, 0, st>>>(di.as<long long>(), dv.as<double>(), (int)idx.size(),
                                                              rho);
  launched(c);
  // no synchronisation: copies from pageable host memory are staged before
  // cudaMemcpyAsync returns, and the device buffers are freed in stream order
}

static void charge_map(Ctx* c, const PbGeom& g, const AtomsDev& A, DevBuf& rho) {
  rho = DevBuf(g.n() * 8, pb_stream(c));
  charge_into(c, g, A, rho.as<double>());
}

// assign_dielectrics (pb_grid.rs:827-940) and assign_kappa (pb_grid.rs:951-985)
static void dielectric_into(Ctx* c, const PbGeom& g, const AtomsDev& A, double probe, double ein, double eout,
                            double* ex, double* ey, double* ez) {
  cudaStream_t st = pb_stream(c);
  long long n = (long long)g.n();
  GeomDev gd = gdev(g);
  if (std::fabs(ein - eout) < std::numeric_limits<double>::epsilon()) {
    for (double* b : {ex, ey, ez}) k_fill<<<nblk(n, 256), 256, 0, st>>>(b, n, ein);
    launched(c, 3);
    return;
  }
  double max_eff = A.max_r + std::max(probe, 0.0);
  HashBuf hs(pb_build_hash(A.hx, max_eff), st);
  DevBuf inside(n, st);
  if (probe <= 0.0) {
    k_inside<<<nblk(n, 256), 256, 0, st>>>(gd, hs.d, A.xyz.as<double>(), A.r.as<double>(), 0.0, inside.as<uint8_t>());
    launched(c);
  } else {
    DevBuf sas(n, st), ext(n, st), flag(8, st);
    k_inside<<<nblk(n, 256), 256, 0, st>>>(gd, hs.d, A.xyz.as<double>(), A.r.as<double>(), probe, sas.as<uint8_t>());
    k_flood_seed<<<nblk(n, 256), 256, 0, st>>>(gd, sas.as<uint8_t>(), ext.as<uint8_t>());
    launched(c, 2);
    dim3 fb(8, 8, 8), fg(nblk(g.nx, 8), nblk(g.ny, 8), nblk(g.nz, 8));
    size_t ntile = (size_t)fg.x * fg.y * fg.z;
    DevBuf act(2 * ntile, st);
    uint8_t* act_a = act.as<uint8_t>();
    uint8_t* act_b = act_a + ntile;
    long long limit = (long long)g.nx + g.ny + g.nz + 64;
    bool done = false;
    int pass = 0;
    for (long long it = 0; it < limit * 8 && !done; it += 8) {
      RSTG_CUDA(cudaMemsetAsync(flag.p, 0, 4, st));
      for (int k = 0; k < 8; k++, pass++) {  // pass 0 visits every tile, later passes the marked ones
        uint8_t* in = pass == 0 ? nullptr : ((pass & 1) ? act_a : act_b);
        uint8_t* out = (pass & 1) ? act_b : act_a;
        RSTG_CUDA(cudaMemsetAsync(out, 0, ntile, st));
        k_flood<<<fg, fb, 0, st>>>(gd, sas.as<uint8_t>(), ext.as<uint8_t>(), flag.as<int>(), in, out);
      }
      launched(c, 8);
      int h = 0;
      RSTG_CUDA(cudaMemcpyAsync(&h, flag.p, 4, cudaMemcpyDeviceToHost, st));
      RSTG_CUDA(cudaStreamSynchronize(st));
      done = h == 0;
    }
    if (!done) throw Error(RSTG_ERR_INVALID, "PB exterior flood fill did not settle");
    double thr = (probe / g.h) * (probe / g.h);
    int R = (int)std::floor(std::sqrt(thr)) + 1;
    std::vector<int4> offs;
    for (int z = -R; z <= R; z++)
      for (int y = -R; y <= R; y++)
        for (int x = -R; x <= R; x++)
          if ((double)(x * x + y * y + z * z) <= thr) offs.push_back(make_int4(x, y, z, x * x + y * y + z * z));
    std::sort(offs.begin(), offs.end(), [](const int4& a, const int4& b) { return a.w < b.w; });
    DevBuf doff(offs.size() * sizeof(int4), st);
    RSTG_CUDA(cudaMemcpyAsync(doff.p, offs.data(), offs.size() * sizeof(int4), cudaMemcpyHostToDevice, st));
    k_ses<<<nblk(n, 256), 256, 0, st>>>(gd, ext.as<uint8_t>(), doff.as<int4>(), (int)offs.size(), inside.as<uint8_t>());
    launched(c);
  }
  HashBuf he(pb_build_hash(A.hx, A.max_r + g.h), st);
  DevBuf ovf(8, st);
  RSTG_CUDA(cudaMemsetAsync(ovf.p, 0, 4, st));
  k_eps<<<nblk(n, 128), 128, 0, st>>>(gd, inside.as<uint8_t>(), he.d, A.xyz.as<double>(), A.r.as<double>(), ein, eout,
                                      ex, ey, ez, ovf.as<int>());
  launched(c);
  int h = 0;
  RSTG_CUDA(cudaMemcpyAsync(&h, ovf.p, 4, cudaMemcpyDeviceToHost, st));
  RSTG_CUDA(cudaStreamSynchronize(st));
  if (h) throw Error(RSTG_ERR_INVALID, "more than 64 atom chords on one grid edge");
}

static void dielectric_maps(Ctx* c, Maps& M, const AtomsDev& A, double probe, double ein, double eout) {
  cudaStream_t st = pb_stream(c);
  long long n = (long long)M.g.n();
  M.ex = DevBuf(n * 8, st);
  M.ey = DevBuf(n * 8, st);
  M.ez = DevBuf(n * 8, st);
  dielectric_into(c, M.g, A, probe, ein, eout, M.ex.as<double>(), M.ey.as<double>(), M.ez.as<double>());
}

static void kappa_into(Ctx* c, const PbGeom& g, const AtomsDev& A, double ion, double kap, double eps_s, bool ionic,
                       double* k2) {
  cudaStream_t st = pb_stream(c);
  long long n = (long long)g.n();
  if (!ionic) {
    RSTG_CUDA(cudaMemsetAsync(k2, 0, n * 8, st));
    return;
  }
  double kbs = eps_s * kap * kap;
  HashBuf hk(pb_build_hash(A.hx, A.max_r + ion), st);
  k_kappa<<<nblk(n, 256), 256, 0, st>>>(gdev(g), hk.d, A.xyz.as<double>(), A.r.as<double>(), ion, kbs, k2);
  launched(c);
}

static void kappa_map(Ctx* c, Maps& M, const AtomsDev& A, double ion, double kap, double eps_s, bool ionic) {
  M.k2 = DevBuf(M.g.n() * 8, pb_stream(c));
  kappa_into(c, M.g, A, ion, kap, eps_s, ionic, M.k2.as<double>());
}

struct SolveOut {
  DevBuf phi;
  int64_t iterations = 0;
  double residual = 0.0;
  bool converged = false;
};

static LevelDev ldev(const PbGeom& g, const double* ex, const double* ey, const double* ez, const double* k2) {
  double ih = 1.0 / (g.h * g.h);
  return LevelDev{g.nx, g.ny, g.nz, ih, ih, ih, ex, ey, ez, k2};
}

// Sweeps and residual of plain SOR, one launch each.
struct Solver {
  Ctx* c;
  cudaStream_t st;
  MapsView M;
  DevBuf part, scal;
  Solver(Ctx* cc, const MapsView& m) : c(cc), st(pb_stream(cc)), M(m) {
    size_t parts = (size_t)nblk(m.g.nx, 128) * std::max(m.g.ny - 2, 1) * std::max(m.g.nz - 2, 1);
    part = DevBuf(std::max<size_t>(parts, 1) * 8, st);
    scal = DevBuf(64, st);
  }

  double smooth(const LevelDev& ld, double* phi, const double* rho, double omega, double rs) {
    dim3 grid(nblk((ld.nx - 1) / 2, 64), std::max(ld.ny - 2, 1), std::max(ld.nz - 2, 1));
    if (ld.nx < 3 || ld.ny < 3 || ld.nz < 3) return 0.0;
    for (int color = 0; color < 2; color++) {  // per-colour partial sums, accumulated in fixed order
      k_rb<<<grid, 64, 0, st>>>(ld, phi, rho, omega, rs, color, part.as<double>());
      k_sum_fixed<<<1, 1024, 0, st>>>(part.as<double>(), (long long)grid.x * grid.y * grid.z,
                                      scal.as<double>() + 1 + color);
      launched(c, 2);
    }
    double h[2];
    RSTG_CUDA(cudaMemcpyAsync(h, scal.as<double>() + 1, 16, cudaMemcpyDeviceToHost, st));
    RSTG_CUDA(cudaStreamSynchronize(st));
    long long cnt = 0;
    for (int color = 0; color < 2; color++)
      for (int iz = 1; iz < ld.nz - 1; iz++)
        for (int iy = 1; iy < ld.ny - 1; iy++) {
          int x0 = 1 + ((1 + iy + iz + color) & 1);
          if (x0 < ld.nx - 1) cnt += (ld.nx - 1 - x0 + 1) / 2;
        }
    return cnt > 0 ? std::sqrt((h[0] + h[1]) / (double)cnt) : 0.0;
  }

  double rms_residual(const LevelDev& ld, const double* phi, const double* rho, double rs) {
    const PbGeom& g = M.g;
    if (g.nx < 3 || g.ny < 3 || g.nz < 3) return 0.0;
    dim3 grid(nblk(g.nx - 2, 128), g.ny - 2, g.nz - 2);
    k_residual<<<grid, 128, 0, st>>>(ld, phi, rho, rs, part.as<double>());
    long long nb = (long long)grid.x * grid.y * grid.z;
    k_sum_fixed<<<1, 1024, 0, st>>>(part.as<double>(), nb, scal.as<double>());
    launched(c, 2);
    double s = 0.0;
    RSTG_CUDA(cudaMemcpyAsync(&s, scal.p, 8, cudaMemcpyDeviceToHost, st));
    RSTG_CUDA(cudaStreamSynchronize(st));
    double cnt = (double)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
    return std::sqrt(s / cnt);
  }
};

static void apply_bc(Ctx* c, const PbGeom& g, double* phi, const AtomsDev& A, const BcSpec& bc) {
  cudaStream_t st = pb_stream(c);
  long long n = (long long)g.n();
  if (bc.kind == 1) {
    long long nbnd = boundary_count(g);
    k_dh<<<nblk(nbnd, 256), 256, 0, st>>>(gdev(g), nbnd, A.xyz.as<double>(), A.q.as<double>(), A.n, bc.kappa, bc.eout,
                                          phi);
  } else {
    k_interp_boundary<<<nblk(n, 256), 256, 0, st>>>(gdev(g), gdev(*bc.cg), bc.cphi, phi);
  }
  launched(c);
}

// One solve: maps, boundary values and result.
struct MgTask {
  MapsView M;
  BcSpec bc;
  SolveOut R;
};

// k_mg on one or two tasks of the same grid.  rel: the relative-residual mode's
// consistent multigrid (Gauss-Seidel smoothing, restriction without the 0.25
// factor, series/parallel coarse dielectrics, corrections zero on the boundary)
// instead of the reference's (levels: pb_solver.rs:776-836).
static std::vector<MgState> run_mg(Ctx* c, std::vector<MgTask*>& T, int maxv, double tol, bool rel) {
  cudaStream_t st = pb_stream(c);
  const int jobs = (int)T.size();
  MgArgs A{};
  std::vector<PbGeom> G{T[0]->M.g};
  while (std::min(G.back().nx, std::min(G.back().ny, G.back().nz)) > 5) {
    PbGeom g = G.back();
    g.nx = (g.nx + 1) / 2;
    g.ny = (g.ny + 1) / 2;
    g.nz = (g.nz + 1) / 2;
    g.h *= 2.0;
    G.push_back(g);
  }
  A.nlev = (int)G.size() - 1;
  if (A.nlev > kMgLevels) throw Error(RSTG_ERR_NOMEM, "PB grid has too many multigrid levels");
  // shared memory of mg_bottom: corrections, right-hand sides and codes from lb down, the residual of lb
  constexpr size_t kBottom = 200 << 10;
  size_t below = 0, smem = 0;
  A.lb = A.nlev + 1;
  for (int l = A.nlev; l >= 1; l--) {
    below += G[l].n();
    const size_t need = (2 * below + G[l].n()) * 8 + below;
    if (need > kBottom) break;
    A.lb = l;
    smem = need;
  }
  // a solve gets as many blocks as its finest level has work for
  RSTG_CUDA(cudaFuncSetAttribute(k_mg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBottom));
  const long long half = (long long)((G[0].nx - 1) / 2) * (G[0].ny - 2) * (G[0].nz - 2);
  A.blocks = (int)std::max<long long>(1, std::min<long long>(c->prop.multiProcessorCount / jobs, nblk(half, kMgThreads)));
  auto walk = [&](unsigned n0, unsigned n1, unsigned n2) {
    const unsigned s = kMgThreads, per = nblk(nblk((long long)n0 * n1 * n2, A.blocks), 32) * 32;
    return MgWalk{n0, n1, n2, s % n0, s / n0 % n1, s / n0 / n1, per};
  };
  size_t total = 0, codes = 0;
  for (int l = 0; l <= A.nlev; l++) {
    const PbGeom& g = G[l];
    MgGeo& d = A.g[l];
    d.nx = g.nx;
    d.ny = g.ny;
    d.nz = g.nz;
    d.ih = 1.0 / (g.h * g.h);
    d.om = rel ? 1.0 : pb_omega(g.nx, g.ny, g.nz);
    if (g.nx >= 3 && g.ny >= 3 && g.nz >= 3) {
      d.half = walk((g.nx - 1) / 2, g.ny - 2, g.nz - 2);
      d.in = walk(g.nx - 2, g.ny - 2, g.nz - 2);
    }
    d.all = walk(g.nx, g.ny, g.nz);
    d.pairs = walk((g.nx + 1) / 2, g.ny, g.nz);
    total += g.n() * (1 + (l < A.nlev ? 1 : 0) + (l > 0 ? 6 : 0));
    codes += g.n();
  }
  A.quota = (int)std::max<long long>(1, (64ll << 20) / (long long)G[0].n());  // a launch of some ten milliseconds at most
  A.maxv = maxv;
  A.rel = rel;
  A.tol = tol;
  A.rs = kFourPiEc;
  std::vector<DevBuf> mem(jobs);
  for (int j = 0; j < jobs; j++) {
    const MapsView& M = T[j]->M;
    mem[j] = DevBuf(total * 8 + codes, st);
    double* at = mem[j].as<double>();
    for (int l = 0; l < A.nlev; l++) {
      A.p[j][l].res = at;
      at += G[l].n();
    }
    A.p[j][0].ex = M.ex;
    A.p[j][0].ey = M.ey;
    A.p[j][0].ez = M.ez;
    A.p[j][0].k2 = M.k2;
    A.p[j][0].rhs = const_cast<double*>(M.rho);
    A.p[j][0].phi = T[j]->R.phi.as<double>();
    for (int l = 1; l <= A.nlev; l++) {
      MgPtr& q = A.p[j][l];
      const double** maps[4] = {&q.ex, &q.ey, &q.ez, &q.k2};
      for (const double** m : maps) {
        *m = at;
        at += G[l].n();
      }
      q.rhs = at;
      q.phi = at + G[l].n();
      at += 2 * G[l].n();
    }
    uint8_t* code = reinterpret_cast<uint8_t*>(mem[j].as<double>() + total);
    for (int l = 0; l <= A.nlev; l++) {
      A.p[j][l].di = at;
      A.p[j][l].code = code;
      at += G[l].n();
      code += G[l].n();
    }
    A.val[j][0] = M.val[0];
    A.val[j][1] = M.val[1];
    A.kb[j] = M.kb;
  }
  for (int l = 1; l <= A.nlev; l++) {
    const PbGeom &f = G[l - 1], &g = G[l];
    Coarsen m{};
    int maps = 0;
    for (int j = 0; j < jobs; j++) {
      const double* src[4] = {A.p[j][l - 1].ex, A.p[j][l - 1].ey, A.p[j][l - 1].ez, A.p[j][l - 1].k2};
      const double* dst[4] = {A.p[j][l].ex, A.p[j][l].ey, A.p[j][l].ez, A.p[j][l].k2};
      for (int k = 0; k < 4; k++) {
        if (rel && k < 3) {
          k_coarsen_face<<<nblk(g.n(), 256), 256, 0, st>>>(src[k], f.nx, f.ny, f.nz, const_cast<double*>(dst[k]), g.nx,
                                                           g.ny, g.nz, k);
          launched(c);
          continue;
        }
        m.src[maps] = src[k];
        m.dst[maps++] = const_cast<double*>(dst[k]);
      }
    }
    k_coarsen<<<dim3(nblk(g.n(), 256), maps), 256, 0, st>>>(m, f.nx, f.ny, f.nz, g.nx, g.ny, g.nz);
    launched(c);
  }
  for (int l = 0; l <= A.nlev; l++) {
    MgCodes m{};
    for (int j = 0; j < jobs; j++) {
      m.p[j] = A.p[j][l];
      m.val[j][0] = A.val[j][0];
      m.val[j][1] = A.val[j][1];
      m.kb[j] = A.kb[j];
    }
    k_mg_codes<<<dim3(nblk(G[l].n(), 256), jobs), 256, 0, st>>>(m, G[l].nx, G[l].ny, G[l].nz, A.g[l].ih, A.g[l].om, l == 0);
    launched(c);
  }
  DevBuf bar(jobs * 128, st), state(jobs * sizeof(MgState), st), part((size_t)jobs * A.blocks * 8, st);
  A.bar = bar.as<unsigned>();
  A.st = state.as<MgState>();
  A.part = part.as<double>();
  std::vector<MgState> S(jobs);
  for (MgState& s : S) s.best = s.prev = std::numeric_limits<double>::max();
  RSTG_CUDA(cudaMemcpyAsync(state.p, S.data(), S.size() * sizeof(MgState), cudaMemcpyHostToDevice, st));
  void* args[] = {&A};
  for (bool running = true; running;) {
    RSTG_CUDA(cudaMemsetAsync(bar.p, 0, bar.bytes, st));
    RSTG_CUDA(cudaLaunchCooperativeKernel((const void*)k_mg, dim3(A.blocks * jobs), dim3(kMgThreads), args, smem, st));
    launched(c);
    RSTG_CUDA(cudaMemcpyAsync(S.data(), state.p, S.size() * sizeof(MgState), cudaMemcpyDeviceToHost, st));
    RSTG_CUDA(cudaStreamSynchronize(st));
    running = false;
    for (const MgState& s : S) {
      if (s.status == 4) throw Error(RSTG_ERR_CUDA, "PB multigrid: the blocks of a solve lost one another");
      running = running || s.status == 0;
    }
  }
  return S;
}

// solve_lpbe_multigrid (pb_solver.rs:1015-1167) with the plain SOR fallback
// (pb_solver.rs:373-447), for one or two tasks of the same grid.  rtol > 0:
// the relative-residual mode -- the consistent multigrid, stopping when the
// RMS residual falls below rtol times its initial value (SOR grids: the
// residual after each sweep); the reference's cycle cap and divergence rule stay.
static void solve_mg(Ctx* c, std::vector<MgTask*> tasks, const AtomsDev& A, double tol, int64_t maxit,
                     double rtol = 0.0) {
  cudaStream_t st = pb_stream(c);
  const PbGeom& g = tasks[0]->M.g;
  const long long n = (long long)g.n();
  const bool rel = rtol > 0.0;
  for (MgTask* t : tasks) {
    t->R.phi = DevBuf(n * 8, st);
    RSTG_CUDA(cudaMemsetAsync(t->R.phi.p, 0, n * 8, st));
    apply_bc(c, g, t->R.phi.as<double>(), A, t->bc);
  }
  auto sor = [&](MgTask& t, bool restart, double r0) {
    const MapsView& M = t.M;
    SolveOut& R = t.R;
    Solver S(c, M);
    const LevelDev top = ldev(g, M.ex, M.ey, M.ez, M.k2);
    if (restart && rel) r0 = S.rms_residual(top, R.phi.as<double>(), M.rho, kFourPiEc);
    if (restart) RSTG_CUDA(cudaMemsetAsync(R.phi.p, 0, n * 8, st));
    apply_bc(c, g, R.phi.as<double>(), A, t.bc);
    double rj = spectral_radius(g.nx, g.ny, g.nz), rs2 = rj * rj, om = 1.0;
    R.residual = std::numeric_limits<double>::max();
    R.converged = false;
    for (int64_t it = 0; it < maxit; it++) {
      double rms = S.smooth(top, R.phi.as<double>(), M.rho, om, kFourPiEc);
      if (rel) rms = S.rms_residual(top, R.phi.as<double>(), M.rho, kFourPiEc) / std::max(r0, 1e-300);
      R.residual = rms;
      R.iterations = it + 1;
      om = it == 0 ? 1.0 / (1.0 - rs2 / 2.0) : 1.0 / (1.0 - rs2 * om / 4.0);
      if (rms < (rel ? rtol : tol)) {
        R.converged = true;
        return;
      }
    }
  };
  if (std::min(g.nx, std::min(g.ny, g.nz)) <= 8) {
    for (MgTask* t : tasks) sor(*t, true, 0.0);
    return;
  }
  const int maxv = (int)std::min<int64_t>(std::max<int64_t>(maxit / 6, 1), 200);
  const std::vector<MgState> S = run_mg(c, tasks, maxv, rel ? rtol : tol, rel);
  for (size_t k = 0; k < tasks.size(); k++) {
    if (S[k].status == 2) {
      sor(*tasks[k], false, S[k].r0);
      continue;
    }
    tasks[k]->R.iterations = S[k].cycles;
    tasks[k]->R.residual = rel ? S[k].r / std::max(S[k].r0, 1e-300) : S[k].r;
    tasks[k]->R.converged = S[k].status == 1;
  }
}

static double elec_energy(Ctx* c, const PbGeom& g, const double* phi, const AtomsDev& A) {
  cudaStream_t st = pb_stream(c);
  if (A.n == 0) return 0.0;
  DevBuf v(A.n * 8, st), e(8, st);
  k_atom_phi<<<nblk(A.n, 128), 128, 0, st>>>(gdev(g), phi, A.xyz.as<double>(), A.q.as<double>(), A.n, v.as<double>());
  k_seq_sum<<<1, 32, 0, st>>>(v.as<double>(), A.n, e.as<double>());
  launched(c, 2);
  double h = 0.0;
  RSTG_CUDA(cudaMemcpyAsync(&h, e.p, 8, cudaMemcpyDeviceToHost, st));
  RSTG_CUDA(cudaStreamSynchronize(st));
  return h;
}

static double maxabs(Ctx* c, const DevBuf& phi, long long n) {
  DevBuf o(8, pb_stream(c));
  RSTG_CUDA(cudaMemsetAsync(o.p, 0, 8, pb_stream(c)));
  k_maxabs<<<(unsigned)std::min<long long>(nblk(n, 1024), 296), 1024, 0, pb_stream(c)>>>(phi.as<double>(), n,
                                                                                        o.as<unsigned long long>());
  launched(c);
  double h = 0.0;
  RSTG_CUDA(cudaMemcpyAsync(&h, o.p, 8, cudaMemcpyDeviceToHost, pb_stream(c)));
  RSTG_CUDA(cudaStreamSynchronize(pb_stream(c)));
  return h;
}

// A solve of the pair: solvated (ionic) or reference.
struct PbSide {
  double eout = 1.0;
  bool ionic = false;
  SolveOut* out = nullptr;
  double energy = 0.0;
};
// Grids of up to this many points have the two solves of a pair side by side:
// one alone leaves the GPU waiting at barriers (a pass over fewer points than
// this takes less than ten barriers), and the second set of maps and levels costs
// at most 140 MB.  Decided for the coarse and the fine grid apart: the
// coarse one can be the larger (fillratio / fscale set its size).
constexpr size_t kPairPoints = 2u << 20;

// pb_solve_with_focusing, pb_energy.rs:134-322, for the two sides of a pair
static void solve_focus(Ctx* c, const Maps& fine_rho, const PbGeom* cg, const AtomsDev& A, const rstg_pb_params& p,
                        double kap, PbSide (&side)[2], double rtol) {
  const double ein = p.solute_dielectric;
  BcSpec dh[2], bc[2];
  for (int k = 0; k < 2; k++) {
    dh[k].kind = 1;
    dh[k].kappa = side[k].ionic ? kap : 0.0;
    dh[k].eout = side[k].eout;
    bc[k] = dh[k];
  }
  // both solves on one grid; their maps are given back when they end
  auto solve = [&](const PbGeom& g, const double* rho, const BcSpec* b, double tol, SolveOut* const* out) {
    const int per = g.n() <= kPairPoints ? 2 : 1;
    for (int k0 = 0; k0 < 2; k0 += per) {
      Maps M[2];
      MgTask task[2];
      std::vector<MgTask*> list;
      for (int k = k0; k < k0 + per; k++) {
        M[k].g = g;
        dielectric_maps(c, M[k], A, p.probe_radius, ein, side[k].eout);
        kappa_map(c, M[k], A, p.ion_radius, kap, p.solvent_dielectric, side[k].ionic);
        task[k].M = MapsView{g, rho, M[k].ex.as<double>(), M[k].ey.as<double>(), M[k].ez.as<double>(),
                             M[k].k2.as<double>(), {ein, side[k].eout}, p.solvent_dielectric * kap * kap};
        task[k].bc = b[k];
        list.push_back(&task[k]);
      }
      solve_mg(c, list, A, tol, p.max_iterations, rtol);
      for (int k = k0; k < k0 + per; k++) *out[k] = std::move(task[k].R);
    }
  };
  SolveOut cr[2];
  if (cg) {
    DevBuf rho;
    charge_map(c, *cg, A, rho);
    SolveOut* const out[2] = {&cr[0], &cr[1]};
    solve(*cg, rho.as<double>(), dh, p.tolerance * 10.0, out);
    for (int k = 0; k < 2; k++) {
      const double mp = maxabs(c, cr[k].phi, (long long)cg->n());
      if (cr[k].converged && std::isfinite(mp) && mp < 1e10) {
        bc[k].kind = 2;
        bc[k].cg = cg;
        bc[k].cphi = cr[k].phi.as<double>();
      }
    }
  }
  SolveOut* const out[2] = {side[0].out, side[1].out};
  solve(fine_rho.g, fine_rho.rho.as<double>(), bc, p.tolerance, out);
  for (int k = 0; k < 2; k++) side[k].energy = elec_energy(c, fine_rho.g, side[k].out->phi.as<double>(), A);
}

void pb_grid_maps(Ctx* c, const std::vector<double>& x, const std::vector<double>& q, const std::vector<double>& radii,
                  const rstg_pb_params& p, double ein, double eout, bool ionic, int64_t* dims, double* origin,
                  double* charge, uint8_t* inside, double* ex, double* ey, double* ez, double* k2, double* bphi) {
  double s = p.salt_concentration;
  double kap = s <= 0.0 ? 0.0
                        : std::sqrt(8.0 * kPi * 332.0522 * 6.022e-4 * s / (p.solvent_dielectric * 0.00198688 * p.temperature));
  PbGeom g = pb_auto_grid(x, p.grid_spacing, p.grid_buffer);
  dims[0] = g.nx;
  dims[1] = g.ny;
  dims[2] = g.nz;
  origin[0] = g.ox;
  origin[1] = g.oy;
  origin[2] = g.oz;
  if (!charge) return;
  cudaStream_t st = pb_stream(c);
  AtomsDev A(x, q, radii, st);
  Maps M;
  M.g = g;
  charge_map(c, g, A, M.rho);
  dielectric_maps(c, M, A, p.probe_radius, ein, eout);
  kappa_map(c, M, A, p.ion_radius, kap, p.solvent_dielectric, ionic);
  long long n = (long long)g.n();
  DevBuf phi(n * 8, st), ins(n, st);
  RSTG_CUDA(cudaMemsetAsync(phi.p, 0, n * 8, st));
  BcSpec dh;
  dh.kappa = ionic ? kap : 0.0;
  dh.eout = eout;
  apply_bc(c, g, phi.as<double>(), A, dh);
  if (inside) {
    if (p.probe_radius > 0.0) {
      HashBuf hs(pb_build_hash(A.hx, A.max_r + p.probe_radius), st);
      DevBuf sas(n, st), ext(n, st), flag(8, st);
      GeomDev gd = gdev(g);
      k_inside<<<nblk(n, 256), 256, 0, st>>>(gd, hs.d, A.xyz.as<double>(), A.r.as<double>(), p.probe_radius,
                                             sas.as<uint8_t>());
      k_flood_seed<<<nblk(n, 256), 256, 0, st>>>(gd, sas.as<uint8_t>(), ext.as<uint8_t>());
      launched(c, 2);
      dim3 fb(8, 8, 8), fg(nblk(g.nx, 8), nblk(g.ny, 8), nblk(g.nz, 8));
      for (int guard = 0; guard < 100000; guard++) {
        RSTG_CUDA(cudaMemsetAsync(flag.p, 0, 4, st));
        k_flood<<<fg, fb, 0, st>>>(gd, sas.as<uint8_t>(), ext.as<uint8_t>(), flag.as<int>(), nullptr, nullptr);
        launched(c);
        int h = 0;
        RSTG_CUDA(cudaMemcpyAsync(&h, flag.p, 4, cudaMemcpyDeviceToHost, st));
        RSTG_CUDA(cudaStreamSynchronize(st));
        if (!h) break;
      }
      double thr = (p.probe_radius / g.h) * (p.probe_radius / g.h);
      int R = (int)std::floor(std::sqrt(thr)) + 1;
      std::vector<int4> offs;
      for (int z = -R; z <= R; z++)
        for (int y = -R; y <= R; y++)
          for (int xx = -R; xx <= R; xx++)
            if ((double)(xx * xx + y * y + z * z) <= thr) offs.push_back(make_int4(xx, y, z, 0));
      DevBuf doff(offs.size() * sizeof(int4), st);
      RSTG_CUDA(cudaMemcpyAsync(doff.p, offs.data(), offs.size() * sizeof(int4), cudaMemcpyHostToDevice, st));
      k_ses<<<nblk(n, 256), 256, 0, st>>>(gd, ext.as<uint8_t>(), doff.as<int4>(), (int)offs.size(), ins.as<uint8_t>());
      launched(c);
      RSTG_CUDA(cudaStreamSynchronize(st));
    } else {
      HashBuf hs(pb_build_hash(A.hx, A.max_r), st);
      k_inside<<<nblk(n, 256), 256, 0, st>>>(gdev(g), hs.d, A.xyz.as<double>(), A.r.as<double>(), 0.0,
                                             ins.as<uint8_t>());
      launched(c);
      RSTG_CUDA(cudaStreamSynchronize(st));
    }
    RSTG_CUDA(cudaMemcpyAsync(inside, ins.p, n, cudaMemcpyDeviceToHost, st));
  }
  RSTG_CUDA(cudaMemcpyAsync(charge, M.rho.p, n * 8, cudaMemcpyDeviceToHost, st));
  RSTG_CUDA(cudaMemcpyAsync(ex, M.ex.p, n * 8, cudaMemcpyDeviceToHost, st));
  RSTG_CUDA(cudaMemcpyAsync(ey, M.ey.p, n * 8, cudaMemcpyDeviceToHost, st));
  RSTG_CUDA(cudaMemcpyAsync(ez, M.ez.p, n * 8, cudaMemcpyDeviceToHost, st));
  RSTG_CUDA(cudaMemcpyAsync(k2, M.k2.p, n * 8, cudaMemcpyDeviceToHost, st));
  RSTG_CUDA(cudaMemcpyAsync(bphi, phi.p, n * 8, cudaMemcpyDeviceToHost, st));
  RSTG_CUDA(cudaStreamSynchronize(st));
}

double pb_energy_run(Ctx* c, const std::vector<double>& x, const std::vector<double>& q,
                     const std::vector<double>& radii, const rstg_pb_params& p, rstg_pb_diag* diag, double rtol) {
  if (!(p.grid_spacing > 0.0)) throw Error(RSTG_ERR_INVALID, "grid_spacing must be positive");
  if (q.empty()) return 0.0;
  double s = p.salt_concentration;
  double kap = s <= 0.0 ? 0.0
                        : std::sqrt(8.0 * kPi * 332.0522 * 6.022e-4 * s / (p.solvent_dielectric * 0.00198688 * p.temperature));
  AtomsDev A(x, q, radii, pb_stream(c));
  Maps fine;
  fine.g = pb_auto_grid(x, p.grid_spacing, p.grid_buffer);
  if (fine.g.n() > (size_t)600 * 600 * 600) throw Error(RSTG_ERR_NOMEM, "PB grid exceeds 600^3 points");
  PbGeom cg;
  bool focus = p.fillratio > 0.0 && p.fscale > 1;
  if (focus) cg = pb_coarse_grid(x, p.grid_spacing, p.fillratio, p.fscale);
  charge_map(c, fine.g, A, fine.rho);
  SolveOut rs, rr;
  PbSide sides[2];
  sides[0].eout = p.solvent_dielectric;
  sides[0].ionic = true;
  sides[0].out = &rs;
  sides[1].eout = p.solute_dielectric;
  sides[1].out = &rr;
  solve_focus(c, fine, focus ? &cg : nullptr, A, p, kap, sides, rtol);
  const double es = sides[0].energy, er = sides[1].energy;
  if (diag) {
    diag->iterations[0] = rs.iterations;
    diag->iterations[1] = rr.iterations;
    diag->residual[0] = rs.residual;
    diag->residual[1] = rr.residual;
    diag->converged[0] = rs.converged;
    diag->converged[1] = rr.converged;
    diag->dims[0] = fine.g.nx;
    diag->dims[1] = fine.g.ny;
    diag->dims[2] = fine.g.nz;
  }
  return es - er;
}

// ---------------------------------------------------------------------------
// entry points of the batched engine (pb_batch.cu)
// ---------------------------------------------------------------------------
static thread_local cudaStream_t t_pb_stream = nullptr;
cudaStream_t pb_stream(Ctx* c) { return t_pb_stream ? t_pb_stream : c->stream; }
PbStreamScope::PbStreamScope(cudaStream_t s) : prev(t_pb_stream) { t_pb_stream = s; }
PbStreamScope::~PbStreamScope() { t_pb_stream = prev; }

double pb_kappa(const rstg_pb_params& p) {  // pb_energy.rs:337-345
  double s = p.salt_concentration;
  return s <= 0.0 ? 0.0
                  : std::sqrt(8.0 * kPi * 332.0522 * 6.022e-4 * s / (p.solvent_dielectric * 0.00198688 * p.temperature));
}

void pb_maps_into(Ctx* c, const PbGeom& g, const AtomsDev& A, const rstg_pb_params& p, double ein, double eout,
                  double kap, bool ionic, double* rho, double* ex, double* ey, double* ez, double* k2) {
  if (rho) charge_into(c, g, A, rho);
  if (ex) dielectric_into(c, g, A, p.probe_radius, ein, eout, ex, ey, ez);
  if (k2) kappa_into(c, g, A, p.ion_radius, kap, p.solvent_dielectric, ionic, k2);
}

void pb_boundary(Ctx* c, const PbGeom& g, double* phi, const AtomsDev& A, const BcSpec& bc) { apply_bc(c, g, phi, A, bc); }

}  // namespace rstg
