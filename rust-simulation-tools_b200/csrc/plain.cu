// Plain FP64 kernels.  Built with -fmad=false: an a*b+c is two rounded operations,
// as in the reference's Rust f64 code, except where a fused one is written out (the
// far series of the Born integrals).  Pair energies take one reciprocal root where
// the reference has a root and divisions; SASA point tests run in FP32 and are
// decided by the reference's FP64 expression near the threshold.
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "f32x2.cuh"
#include "plain.cuh"

namespace rstg {

static constexpr int kWarpsPerBlock = 8;
static constexpr int kSasaThreads = 128;
static constexpr int kSasaMaxNeighbors = 2048;
static constexpr int kSasaPlanes = 256;  // neighbours that the packed point tests hold

std::vector<double> fibonacci_sphere(int64_t n) {
  std::vector<double> v;
  if (n <= 0) return v;
  if (n == 1) return {0.0, 1.0, 0.0};
  double phi = kPi * (3.0 - std::sqrt(5.0));
  for (int64_t i = 0; i < n; i++) {
    double y = 1.0 - ((double)i / (double)(n - 1)) * 2.0;
    double r = std::sqrt(1.0 - y * y);
    double th = phi * (double)i;
    v.push_back(std::cos(th) * r);
    v.push_back(y);
    v.push_back(std::sin(th) * r);
  }
  return v;
}

DevTopo DevTopo::upload(const Topology& t, int parts, const double* coords, cudaStream_t st) {
  DevTopo d;
  const int64_t n = t.n_atoms;
  d.n = n;
  d.nt = std::max<int64_t>(t.n_types, 1);
  d.scee = t.scee;
  d.scnb = t.scnb;
  for (double r : t.radii) d.max_radius = std::max(d.max_radius, r);
  std::vector<char> host;
  std::vector<std::pair<DevView*, size_t>> at;
  auto room = [&](DevView& v, size_t bytes) {  // 16-byte aligned (vector loads), never empty
    const size_t o = host.size();
    at.push_back({&v, o});
    host.resize(o + std::max<size_t>((bytes + 15) & ~(size_t)15, 16));
    return host.data() + o;
  };
  auto put = [&](DevView& v, const void* src, size_t bytes) {
    char* p = room(v, bytes);
    if (bytes) memcpy(p, src, bytes);
  };
  host.reserve((size_t)n * (parts & kMm ? 220 : 56) + 65536);
  if (coords) put(d.xyz, coords, n * 24);
  put(d.rad, t.radii.data(), n * 8);
  if (parts & (kGb | kMm)) put(d.q, t.charges_amber.data(), n * 8);
  if (parts & kGb) put(d.scr, t.screen.data(), n * 8);
  if (parts & kMm) {
    int32_t* ty = (int32_t*)room(d.type, n * 4);
    for (int64_t i = 0; i < n; i++) ty[i] = t.n_types > 0 ? (int32_t)t.type_idx[i] : 0;  // (without types the tables hold one zero)
    // dense LJ tables from NONBONDED_PARM_INDEX (lj_ab, mm_energy.rs:152-161)
    const int64_t nt = d.nt;
    for (DevView* v : {&d.ljA, &d.ljB}) {
      double* L = (double*)room(*v, nt * nt * 8);
      const std::vector<double>& src = v == &d.ljA ? t.lj_a : t.lj_b;
      for (int64_t k = 0; k < nt * nt; k++) L[k] = 0.0;
      for (int64_t a = 0; a < t.n_types; a++)
        for (int64_t b = 0; b < t.n_types; b++) {
          const int64_t idx = t.nb_index[t.n_types * a + b];
          if (idx >= 1) L[a * nt + b] = src[idx - 1];
        }
    }
    PairWindows w = PairWindows::build(t);
    put(d.win, w.win.data(), w.win.size() * 8);
    put(d.farp, w.far_ptr.data(), w.far_ptr.size() * 4);
    put(d.far, w.far.data(), w.far.size() * 4);
    d.nb = t.bond_i.size();
    d.na = t.ang_i.size();
    d.nd = t.dih_i.size();
    int32_t* ix = (int32_t*)room(d.bidx, d.nb * 8);
    for (int64_t k = 0; k < d.nb; k++) {
      ix[2 * k] = (int32_t)t.bond_i[k];
      ix[2 * k + 1] = (int32_t)t.bond_j[k];
    }
    double* pr = (double*)room(d.bpar, d.nb * 16);
    for (int64_t k = 0; k < d.nb; k++) {
      pr[2 * k] = t.bond_k[t.bond_t[k]];
      pr[2 * k + 1] = t.bond_req[t.bond_t[k]];
    }
    ix = (int32_t*)room(d.aidx, d.na * 12);
    for (int64_t k = 0; k < d.na; k++) {
      ix[3 * k] = (int32_t)t.ang_i[k];
      ix[3 * k + 1] = (int32_t)t.ang_j[k];
      ix[3 * k + 2] = (int32_t)t.ang_k[k];
    }
    pr = (double*)room(d.apar, d.na * 16);
    for (int64_t k = 0; k < d.na; k++) {
      pr[2 * k] = t.angle_k[t.ang_t[k]];
      pr[2 * k + 1] = t.angle_teq[t.ang_t[k]];
    }
    ix = (int32_t*)room(d.didx, d.nd * 16);
    for (int64_t k = 0; k < d.nd; k++) {
      ix[4 * k] = (int32_t)t.dih_i[k];
      ix[4 * k + 1] = (int32_t)t.dih_j[k];
      ix[4 * k + 2] = (int32_t)t.dih_k[k];
      ix[4 * k + 3] = (int32_t)t.dih_l[k];
    }
    pr = (double*)room(d.dpar, d.nd * 24);
    for (int64_t k = 0; k < d.nd; k++) {
      pr[3 * k] = t.dih_pk[t.dih_t[k]];
      pr[3 * k + 1] = t.dih_pn[t.dih_t[k]];
      pr[3 * k + 2] = t.dih_phase[t.dih_t[k]];
    }
  }
  d.mem = DevBuf(host.size(), st);
  RSTG_CUDA(cudaMemcpyAsync(d.mem.p, host.data(), host.size(), cudaMemcpyHostToDevice, st));
  for (auto& a : at) a.first->p = (char*)d.mem.p + a.second;
  return d;
}

// ---------------------------------------------------------------------------
// Born radii, gb_energy.rs:144-258: one warp per atom i, lanes stride j.  Bound
// by FP64 issue: the closed form costs a square root, a logarithm and two
// divisions a pair, the far series (nearly every pair) one division and
// fourteen multiply-adds.  5,050 atoms: 320 us with the closed form
// throughout, 146 here.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double hct_term64(double r2, double rho_i, double sj) {
  const double r = sqrt(r2);
  if (r == 0.0) return 0.0;
  if (rho_i >= r + sj) return 0.0;
  const double u = r + sj, d = fabs(r - sj), l = (rho_i > d) ? rho_i : d;
  // one division for 1/l and 1/u, one for 1/r
  const double inv = 1.0 / (l * u), l_inv = u * inv, u_inv = l * inv, r_inv = 1.0 / r;
  const double contrib = 0.5 * (l_inv - u_inv + 0.25 * (u_inv * u_inv - l_inv * l_inv) * (r - sj * sj * r_inv) +
                                0.5 * log(l * u_inv) * r_inv);
  if (rho_i < sj - r) return contrib + 2.0 * (1.0 / rho_i - l_inv);
  return contrib;
}

// The same integral where 0 <= s <= r / 4 and 0 <= rho_i <= r - s, r neither 0
// nor infinite: (1/r) sum_k k/(2k+1) x^(2k+1), x = s/r, in powers of
// y = s^2 / r^2 <= 1/16.  Fourteen terms leave at most 2.2e-17 of the first, and
// the series has none of the closed form's cancellation.
__device__ __forceinline__ double hct_series64(double r2, double sj) {
  const double u = 1.0 / r2, s2 = sj * sj, y = s2 * u;
  double p = 14.0 / 29.0;
#pragma unroll
  for (int m = 12; m >= 0; m--) p = fma(p, y, (double)(m + 1) / (double)(2 * m + 3));
  return (s2 * sj * u) * (u * p);
}

__device__ __forceinline__ double radius_from_psi64(double psi, double rho_i, double radius_i, int model,
                                                    double rgbmax) {
  double alpha = 1.0, beta = 0.0, gamma = 0.0;
  if (model == 1) {
    alpha = 0.8;
    gamma = 2.909125;
  } else if (model == 2) {
    alpha = 1.0;
    beta = 0.8;
    gamma = 4.85;
  }
  double R;
  if (model == 0) {
    double inv_r = 1.0 / rho_i - psi;
    R = inv_r > 0.0 ? 1.0 / inv_r : rgbmax;
  } else {
    double pr = psi * rho_i, p2 = pr * pr, p3 = p2 * pr;
    double tv = tanh(alpha * pr - beta * p2 + gamma * p3);
    double inv_r = 1.0 / rho_i - tv / radius_i;
    R = inv_r > 0.0 ? 1.0 / inv_r : rgbmax;
  }
  if (R > rgbmax) R = rgbmax;
  return R;
}

__global__ void k_born_radii_plain(int n, const double* __restrict__ xyz, const double* __restrict__ rad,
                                   const double* __restrict__ scr, double offset, double cut2, int model,
                                   double rgbmax, double* __restrict__ R) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= n) return;
  int i = warp;
  double xi = xyz[3 * i], yi = xyz[3 * i + 1], zi = xyz[3 * i + 2];
  double rho_i = rad[i] - offset, psi = 0.0;
  // the pairs of a strip of 1024 columns outside the series' domain are marked
  // and evaluated after it, each lane over its own
  for (int j0 = lane; j0 < n; j0 += 1024) {
    unsigned near = 0u;
    for (int t = 0, j = j0; t < 32 && j < n; t++, j += 32) {
      if (j == i) continue;
      const double dx = xi - xyz[3 * j], dy = yi - xyz[3 * j + 1], dz = zi - xyz[3 * j + 2];
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (r2 > cut2) continue;
      const double sj = scr[j] * (rad[j] - offset), rs = rho_i + sj;
      if (rho_i >= 0.0 && sj >= 0.0 && ordinary(r2) && 16.0 * (sj * sj) <= r2 && rs * rs <= r2)
        psi += hct_series64(r2, sj);
      else
        near |= 1u << t;
    }
    while (near) {
      const int j = j0 + 32 * (__ffs(near) - 1);
      near &= near - 1;
      const double dx = xi - xyz[3 * j], dy = yi - xyz[3 * j + 1], dz = zi - xyz[3 * j + 2];
      psi += hct_term64(dx * dx + dy * dy + dz * dz, rho_i, scr[j] * (rad[j] - offset));
    }
  }
  psi = warp_sum(psi);
  if (lane == 0) R[i] = radius_from_psi64(psi, rho_i, rad[i], model, rgbmax);
}

void plain_born_radii(Ctx* c, cudaStream_t st, const DevTopo& t, const double* d_xyz, const rstg_gb_params& p, double* d_R) {
  if (t.n == 0) return;
  int threads = 32 * kWarpsPerBlock;
  int blocks = (int)((t.n + kWarpsPerBlock - 1) / kWarpsPerBlock);
  k_born_radii_plain<<<blocks, threads, 0, st>>>((int)t.n, d_xyz, t.rad.as<double>(), t.scr.as<double>(),
                                                         p.offset, p.cutoff * p.cutoff, p.model, p.rgbmax, d_R);
  launched(c);
}

// ---------------------------------------------------------------------------
// GB energy from radii, gb_energy.rs:283-355.  Block b handles rows b and
// n-1-b (balanced triangle); per-block partials are summed in fixed order.
// (A warp per row pair left a 2,030-atom energy 127 blocks of long serial
// loops: 63 us, 21 here.)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double gb_pair64(double qi, double qj, double r2, double Ri, double Rj, const GbConst& k) {
  const double rr = Ri * Rj, f2 = r2 + rr * exp(-r2 / (4.0 * rr)), fi = rsqrt(f2);
  if (k.no_salt) return k.diel_ns * qi * qj * fi;
  const double f = ordinary(f2) ? f2 * fi : f2;  // 0 and infinity stay what they are
  return -0.5 * qi * qj * (k.inv_ein - exp(-kKScale * k.kappa * f) * k.inv_eout) * fi;
}
__device__ __forceinline__ double gb_self64(double qi, double Ri, const GbConst& k) {
  if (k.no_salt) return k.diel_ns * qi * qi / Ri;
  return -0.5 * qi * qi * (k.inv_ein - exp(-kKScale * k.kappa * Ri) * k.inv_eout) / Ri;
}

__global__ void k_gb_plain(int n, const double* __restrict__ xyz, const double* __restrict__ q,
                           const double* __restrict__ R, GbConst k, double* __restrict__ part) {
  __shared__ double sh[32];
  const int nw = (n + 1) / 2;
  double acc = 0.0;
  for (int side = 0; side < 2; side++) {
    const int i = side == 0 ? (int)blockIdx.x : n - 1 - (int)blockIdx.x;
    if ((int)blockIdx.x >= nw || (side == 1 && i == (int)blockIdx.x)) break;
    const double xi = xyz[3 * i], yi = xyz[3 * i + 1], zi = xyz[3 * i + 2], qi = q[i], Ri = R[i];
    if (threadIdx.x == 0) acc += gb_self64(qi, Ri, k);
    for (int j = i + 1 + threadIdx.x; j < n; j += blockDim.x) {
      const double dx = xi - xyz[3 * j], dy = yi - xyz[3 * j + 1], dz = zi - xyz[3 * j + 2];
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (r2 > k.cut2) continue;
      acc += 2.0 * gb_pair64(qi, q[j], r2, Ri, R[j], k);
    }
  }
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

GbConst gb_const(const rstg_gb_params& p) {
  GbConst k;
  double s = p.salt_concentration;
  k.kappa = s <= 0.0 ? 0.0
                     : std::sqrt(8.0 * kPi * 332.0522 * 6.022e-4 * s / (p.solvent_dielectric * 0.00198688 * p.temperature));
  k.inv_ein = 1.0 / p.solute_dielectric;
  k.inv_eout = 1.0 / p.solvent_dielectric;
  k.diel_ns = -0.5 * (k.inv_ein - k.inv_eout);
  k.no_salt = k.kappa <= 0.0;
  k.cut2 = p.cutoff * p.cutoff;
  return k;
}

void plain_gb_energy(Ctx* c, cudaStream_t st, const DevTopo& t, const double* d_xyz, const rstg_gb_params& p, const double* d_R,
                     double* d_out) {
  if (t.n == 0) {
    RSTG_CUDA(cudaMemsetAsync(d_out, 0, 8, st));
    return;
  }
  int64_t nw = (t.n + 1) / 2;
  DevBuf part(nw * 8, st);
  k_gb_plain<<<(unsigned)nw, kRowThreads, 0, st>>>((int)t.n, d_xyz, t.q.as<double>(), d_R, gb_const(p),
                                                 part.as<double>());
  launched(c);
  sum_columns(c, st, part.as<double>(), nw, 1, d_out);
}

// ---------------------------------------------------------------------------
// MM energy, mm_energy.rs:179-267: bonded terms one thread each, non-bonded
// over i<j with each pair's class from PairWindows (1-4 tested first).
// ---------------------------------------------------------------------------
// Class of the pair i < j (mm_energy.rs:230-252: 1-4 first, then exclusion):
// 0 excluded, 1 full, 2 scaled 1-4.  The 64 atoms after i have a bit each,
// pairs farther along the chain stand in a short list.
__device__ __forceinline__ int pair_class(ulonglong2 win, const int* __restrict__ far, int f0, int f1, int i, int j) {
  const int d = j - i - 1;
  if (d < 64) return ((win.y >> d) & 1ull) ? 2 : (((win.x >> d) & 1ull) ? 0 : 1);
  int cls = 1;
  for (int k = f0; k < f1; k++)
    if (far[2 * k] == j) cls = far[2 * k + 1];
  return cls;
}

// MM pair terms, mm_energy.rs:230-267: blocks over row pairs as k_gb_plain,
// one reciprocal root a pair in place of a square root and three divisions.
// 2,030 atoms: 105 us with a warp per row pair, 19 here.
__global__ void __launch_bounds__(kRowThreads)
    k_nb_plain(int n, const double* __restrict__ xyz, const double* __restrict__ q, const int* __restrict__ type, int nt,
               const double* __restrict__ A, const double* __restrict__ B, const ulonglong2* __restrict__ win,
               const int* __restrict__ farp, const int* __restrict__ far, double scee, double scnb,
               double* __restrict__ part) {
  __shared__ double sh[32];
  double vdw = 0, elec = 0, v14 = 0, e14 = 0;
  for (int side = 0; side < 2; side++) {
    const int i = side == 0 ? (int)blockIdx.x : n - 1 - (int)blockIdx.x;
    if (side == 1 && i == (int)blockIdx.x) break;
    const double xi = xyz[3 * i], yi = xyz[3 * i + 1], zi = xyz[3 * i + 2], qi = q[i];
    const int ti = type[i] * nt, f0 = farp[i], f1 = farp[i + 1];
    const ulonglong2 w = win[i];
    for (int j = i + 1 + threadIdx.x; j < n; j += blockDim.x) {
      const int cls = pair_class(w, far, f0, f1, i, j);
      if (!cls) continue;
      const double dx = xi - xyz[3 * j], dy = yi - xyz[3 * j + 1], dz = zi - xyz[3 * j + 2];
      const double r2 = dx * dx + dy * dy + dz * dz, ri = rsqrt(r2), i2 = ri * ri, i6 = i2 * i2 * i2;
      const double a = A[ti + type[j]], b = B[ti + type[j]], v = a * (i6 * i6) - b * i6, e = qi * q[j] * ri;
      if (cls == 2) {
        v14 += v / scnb;
        e14 += e / scee;
      } else {
        vdw += v;
        elec += e;
      }
    }
  }
  vdw = block_sum(vdw, sh);
  elec = block_sum(elec, sh);
  v14 = block_sum(v14, sh);
  e14 = block_sum(e14, sh);
  if (threadIdx.x == 0) {
    part[4 * blockIdx.x] = vdw;
    part[4 * blockIdx.x + 1] = elec;
    part[4 * blockIdx.x + 2] = v14;
    part[4 * blockIdx.x + 3] = e14;
  }
}

__device__ __forceinline__ void cross3(const double* a, const double* b, double* o) {
  o[0] = a[1] * b[2] - a[2] * b[1];
  o[1] = a[2] * b[0] - a[0] * b[2];
  o[2] = a[0] * b[1] - a[1] * b[0];
}

// Bonded terms, mm_energy.rs:97-149,187-212; part[blk][3].
__global__ void k_bonded_plain(const double* __restrict__ x, int nb, const int* __restrict__ bi,
                               const double* __restrict__ bp, int na, const int* __restrict__ ai,
                               const double* __restrict__ ap, int nd, const int* __restrict__ di,
                               const double* __restrict__ dp, double* __restrict__ part) {
  __shared__ double sh[32];
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  double eb = 0, ea = 0, ed = 0;
  if (t < nb) {
    int i = bi[2 * t], j = bi[2 * t + 1];
    double dx = x[3 * i] - x[3 * j], dy = x[3 * i + 1] - x[3 * j + 1], dz = x[3 * i + 2] - x[3 * j + 2];
    double r = sqrt(dx * dx + dy * dy + dz * dz), k = bp[2 * t], req = bp[2 * t + 1];
    eb = k * (r - req) * (r - req);
  }
  if (t < na) {
    int i = ai[3 * t], j = ai[3 * t + 1], k = ai[3 * t + 2];
    double ba[3] = {x[3 * i] - x[3 * j], x[3 * i + 1] - x[3 * j + 1], x[3 * i + 2] - x[3 * j + 2]};
    double bc[3] = {x[3 * k] - x[3 * j], x[3 * k + 1] - x[3 * j + 1], x[3 * k + 2] - x[3 * j + 2]};
    double dot = ba[0] * bc[0] + ba[1] * bc[1] + ba[2] * bc[2];
    double m1 = sqrt(ba[0] * ba[0] + ba[1] * ba[1] + ba[2] * ba[2]);
    double m2 = sqrt(bc[0] * bc[0] + bc[1] * bc[1] + bc[2] * bc[2]);
    double cs = fmin(1.0, fmax(-1.0, dot / (m1 * m2)));
    double th = acos(cs), ka = ap[2 * t], teq = ap[2 * t + 1];
    ea = ka * (th - teq) * (th - teq);
  }
  if (t < nd) {
    int a = di[4 * t], b = di[4 * t + 1], c = di[4 * t + 2], d = di[4 * t + 3];
    double b1[3] = {x[3 * b] - x[3 * a], x[3 * b + 1] - x[3 * a + 1], x[3 * b + 2] - x[3 * a + 2]};
    double b2[3] = {x[3 * c] - x[3 * b], x[3 * c + 1] - x[3 * b + 1], x[3 * c + 2] - x[3 * b + 2]};
    double b3[3] = {x[3 * d] - x[3 * c], x[3 * d + 1] - x[3 * c + 1], x[3 * d + 2] - x[3 * c + 2]};
    double n1[3], n2[3], m1[3], u[3] = {0, 0, 0};
    cross3(b1, b2, n1);
    cross3(b2, b3, n2);
    double len = sqrt(b2[0] * b2[0] + b2[1] * b2[1] + b2[2] * b2[2]);
    if (!(len < 1e-20)) {
      u[0] = b2[0] / len;
      u[1] = b2[1] / len;
      u[2] = b2[2] / len;
    }
    cross3(n1, u, m1);
    double xx = n1[0] * n2[0] + n1[1] * n2[1] + n1[2] * n2[2];
    double yy = m1[0] * n2[0] + m1[1] * n2[1] + m1[2] * n2[2];
    double phi = atan2(-yy, xx);
    ed = dp[3 * t] * (1.0 + cos(dp[3 * t + 1] * phi - dp[3 * t + 2]));
  }
  eb = block_sum(eb, sh);
  ea = block_sum(ea, sh);
  ed = block_sum(ed, sh);
  if (threadIdx.x == 0) {
    part[3 * blockIdx.x] = eb;
    part[3 * blockIdx.x + 1] = ea;
    part[3 * blockIdx.x + 2] = ed;
  }
}

void plain_mm_energy(Ctx* c, cudaStream_t st, const DevTopo& t, const double* d_xyz, double* d_out) {
  RSTG_CUDA(cudaMemsetAsync(d_out, 0, 7 * 8, st));
  int64_t m = std::max(t.nb, std::max(t.na, t.nd));
  if (m > 0) {
    int blocks = (int)((m + 255) / 256);
    DevBuf part(blocks * 3 * 8, st);
    k_bonded_plain<<<blocks, 256, 0, st>>>(d_xyz, (int)t.nb, t.bidx.as<int>(), t.bpar.as<double>(),
                                                   (int)t.na, t.aidx.as<int>(), t.apar.as<double>(), (int)t.nd,
                                                   t.didx.as<int>(), t.dpar.as<double>(), part.as<double>());
    launched(c);
    sum_columns(c, st, part.as<double>(), blocks, 3, d_out);
  }
  if (t.n >= 2) {
    int64_t nw = (t.n + 1) / 2;
    DevBuf part(nw * 4 * 8, st);
    k_nb_plain<<<(unsigned)nw, kRowThreads, 0, st>>>(
        (int)t.n, d_xyz, t.q.as<double>(), t.type.as<int>(), (int)t.nt, t.ljA.as<double>(), t.ljB.as<double>(),
        t.win.as<ulonglong2>(), t.farp.as<int>(), t.far.as<int>(), t.scee, t.scnb, part.as<double>());
    launched(c);
    sum_columns(c, st, part.as<double>(), nw, 4, d_out + 3);
  }
}

// ---------------------------------------------------------------------------
// SASA, core/src/sasa.rs:228-289: one block per atom.  Neighbours are the
// atoms within r_i + probe + max(r) + probe (the reference's KD-tree query
// radius, inclusive).  A point er s lies inside neighbour j's expanded sphere
// where g = s . 2 er v - (er^2 + |v|^2 - ro^2) > 0 (v the vector to j, ro its
// expanded radius); g is evaluated in FP32 from FP64 differences, two
// neighbours per packed instruction and two points per lane, with the
// neighbours that bury most first, and a point whose largest g lies within
// `band` of 0 is decided by the reference's exact FP64 expression, so counts
// match bit for bit.  Atoms with more than kSasaPlanes touching neighbours take
// that expression throughout.  Bound by FP64 issue of the neighbour search and
// FP32 issue of the tests; 5,050 atoms, 960 points: 303 us with FP64 tests,
// 79 here.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

__global__ void __launch_bounds__(kSasaThreads)
    k_sasa_plain(int n, const double* __restrict__ xyz, const double* __restrict__ rad, double probe, double max_ext,
                 int npts, const double* __restrict__ sphere, double* __restrict__ per_atom,
                 int* __restrict__ overflow) {
  constexpr int kBins = 8;
  __shared__ int nb[kSasaMaxNeighbors];
  __shared__ __align__(16) float wx[kSasaPlanes + 4], wy[kSasaPlanes + 4], wz[kSasaPlanes + 4], wc[kSasaPlanes + 4];
  __shared__ int val[kSasaPlanes + 4], hist[kBins + 1];
  __shared__ int cnt, touch;
  __shared__ int wsum[kSasaThreads / 32];
  const int i = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) cnt = touch = 0;
  if (threadIdx.x <= kBins) hist[threadIdx.x] = 0;
  __syncthreads();
  const double xi = xyz[3 * i], yi = xyz[3 * i + 1], zi = xyz[3 * i + 2];
  const double er = rad[i] + probe, search = er + max_ext, s2 = search * search;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    if (j == i) continue;
    double dx = xyz[3 * j] - xi, dy = xyz[3 * j + 1] - yi, dz = xyz[3 * j + 2] - zi;
    if (dx * dx + dy * dy + dz * dz <= s2) {
      int k = atomicAdd(&cnt, 1);
      if (k < kSasaMaxNeighbors) nb[k] = j;
    }
  }
  __syncthreads();
  int m = cnt;
  if (m > kSasaMaxNeighbors) {
    if (threadIdx.x == 0) atomicExch(overflow, 1);
    m = kSasaMaxNeighbors;
  }
  // ten times the FP32 error of g, whose terms are at most about (er + max_ext)^2
  const float band = fmaxf(2e-4f, (float)(4e-6 * s2)), erf = (float)er;
  // plane of neighbour j and its class: the cosine of the buried cap's edge in eighths; -1: out of reach
  struct Plane {
    float x, y, z, c;
    int cls;
  };
  auto plane = [&](int j) {
    Plane p;
    const float vx = (float)(xyz[3 * j] - xi), vy = (float)(xyz[3 * j + 1] - yi), vz = (float)(xyz[3 * j + 2] - zi);
    const float ro = (float)(rad[j] + probe), d2 = fmaf(vx, vx, fmaf(vy, vy, vz * vz)), d = sqrtf(d2);
    p.c = fmaf(ro, ro, -(erf * erf)) - d2;
    p.x = 2.f * erf * vx;
    p.y = 2.f * erf * vy;
    p.z = 2.f * erf * vz;
    const float t = -p.c * 4.f / fmaxf(erf * d, 1e-12f);
    p.cls = d > (fabsf(erf) + fabsf(ro)) * 1.001f + 1e-3f ? -1 : min(max((int)t, 0), kBins - 1);
    return p;
  };
  int place[2] = {0, 0};
  Plane keep[2];
  const bool packed_m = m <= 2 * kSasaThreads;  // two candidates a thread
  if (packed_m) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int k = h * kSasaThreads + threadIdx.x;
      keep[h].cls = -1;
      if (k < m) {
        keep[h] = plane(nb[k]);
        if (keep[h].cls >= 0) {
          place[h] = atomicAdd(&hist[keep[h].cls], 1);
          atomicAdd(&touch, 1);
        }
      }
    }
  }
  __syncthreads();
  const int t4 = (touch + 3) & ~3;
  const bool packed = packed_m && touch <= kSasaPlanes;
  if (packed) {
    if (threadIdx.x == 0) {
      int at = 0;
      for (int b = 0; b < kBins; b++) {
        const int c = hist[b];
        hist[b] = at;
        at += c;
      }
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; h++)
      if (keep[h].cls >= 0) {
        const int q = hist[keep[h].cls] + place[h];
        val[q] = nb[h * kSasaThreads + threadIdx.x];
        wx[q] = keep[h].x;
        wy[q] = keep[h].y;
        wz[q] = keep[h].z;
        wc[q] = keep[h].c;
      }
    if (threadIdx.x < t4 - touch) {  // padding: never buries
      const int q = touch + threadIdx.x;
      wx[q] = wy[q] = wz[q] = 0.f;
      wc[q] = -3e38f;
      val[q] = i;
    }
    __syncthreads();
  }
  // the reference's test of point p against neighbour j
  auto outside = [&](int p, int j) {
    double tx = xi + sphere[3 * p] * er, ty = yi + sphere[3 * p + 1] * er, tz = zi + sphere[3 * p + 2] * er;
    double oer = rad[j] + probe;
    double dx = tx - xyz[3 * j], dy = ty - xyz[3 * j + 1], dz = tz - xyz[3 * j + 2];
    double d2 = dx * dx + dy * dy + dz * dz;
    return d2 > oer * oer;
  };
  int acc = 0;
  if (packed) {
    for (int p0 = 64 * w; p0 < npts; p0 += 64 * (kSasaThreads / 32)) {
      const int pi[2] = {p0 + lane, p0 + 32 + lane};
      float sx[2], sy[2], sz[2], mg[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const bool v = pi[h] < npts;
        sx[h] = v ? (float)sphere[3 * pi[h]] : 0.f;
        sy[h] = v ? (float)sphere[3 * pi[h] + 1] : 0.f;
        sz[h] = v ? (float)sphere[3 * pi[h] + 2] : 0.f;
        mg[h] = v ? -3e38f : 3e38f;
      }
      const f2 px = dup2(sx[0]), py = dup2(sy[0]), pz = dup2(sz[0]), qx = dup2(sx[1]), qy = dup2(sy[1]), qz = dup2(sz[1]);
#pragma unroll 1
      for (int k = 0; k < t4; k += 4) {
        const ulonglong2 x = *(const ulonglong2*)(wx + k), y = *(const ulonglong2*)(wy + k), z = *(const ulonglong2*)(wz + k),
                         c = *(const ulonglong2*)(wc + k);
        float u, v;
        un2(fma2(px, x.x, fma2(py, y.x, fma2(pz, z.x, c.x))), u, v);
        mg[0] = max3(mg[0], u, v);
        un2(fma2(qx, x.x, fma2(qy, y.x, fma2(qz, z.x, c.x))), u, v);
        mg[1] = max3(mg[1], u, v);
        un2(fma2(px, x.y, fma2(py, y.y, fma2(pz, z.y, c.y))), u, v);
        mg[0] = max3(mg[0], u, v);
        un2(fma2(qx, x.y, fma2(qy, y.y, fma2(qz, z.y, c.y))), u, v);
        mg[1] = max3(mg[1], u, v);
        if (__all_sync(0xffffffffu, fminf(mg[0], mg[1]) > band)) break;
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        if (pi[h] >= npts || mg[h] > band) continue;
        bool ok = true;
        if (mg[h] >= -band)
          for (int k = 0; k < touch && ok; k++) {
            const float g = fmaf(sx[h], wx[k], fmaf(sy[h], wy[k], fmaf(sz[h], wz[k], wc[k])));
            if (g >= -2.f * band) ok = outside(pi[h], val[k]);
          }
        acc += ok ? 1 : 0;
      }
    }
  } else {
    for (int p = threadIdx.x; p < npts; p += blockDim.x) {
      bool ok = true;
      for (int k = 0; k < m && ok; k++) ok = outside(p, nb[k]);
      acc += ok ? 1 : 0;
    }
  }
  acc = warp_sumi(acc);
  if (lane == 0) wsum[w] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    int total = 0;
    for (int h = 0; h < (int)(blockDim.x >> 5); h++) total += wsum[h];
    double frac = (double)total / (double)npts;
    double area = 4.0 * kPi * (er * er);
    per_atom[i] = frac * area;
  }
}

void plain_sasa(Ctx* c, cudaStream_t st, const DevTopo& t, const double* d_xyz, double probe, int64_t n_points,
                const double* d_sphere, double* d_per_atom, double* d_total, int* d_overflow) {
  if (t.n == 0) {
    RSTG_CUDA(cudaMemsetAsync(d_total, 0, 8, st));
    return;
  }
  k_sasa_plain<<<(unsigned)t.n, kSasaThreads, 0, st>>>((int)t.n, d_xyz, t.rad.as<double>(), probe,
                                                               t.max_radius + probe, (int)n_points, d_sphere,
                                                               d_per_atom, d_overflow);
  launched(c);
  sum_columns(c, st, d_per_atom, t.n, 1, d_total);
}

// ---------------------------------------------------------------------------
// Decomposition pair loop, decomposition.rs:240-283.  A block of eight warps
// takes 32 receptor atoms, the lanes; the warps share the ligand.  Each pair is
// evaluated once for its row sums and its column's sum over the block's rows
// (colpart [block][nL][2], added in block order by k_colpart).  5,000 x 50
// atoms: a row kernel and a column kernel of seven blocks took 430 us,
// 17 here.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    k_decomp(const double* __restrict__ xyz, const double* __restrict__ q, const int* __restrict__ type, int nt,
             const double* __restrict__ A, const double* __restrict__ B, const ulonglong2* __restrict__ win,
             const int* __restrict__ farp, const int* __restrict__ far, double scee, double scnb,
             const int* __restrict__ rec, int nR, const int* __restrict__ lig, int nL, double* __restrict__ rows,
             double* __restrict__ colpart) {
  __shared__ double acc[8][2][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, a = blockIdx.x * 32 + lane;
  const bool live = a < nR;
  const int ra = rec[min(a, nR - 1)], ta = type[ra] * nt;
  const double xa = xyz[3 * ra], ya = xyz[3 * ra + 1], za = xyz[3 * ra + 2], qa = q[ra];
  const ulonglong2 wa = win[ra];
  const int a0 = farp[ra], a1 = farp[ra + 1];
  double sv = 0.0, se = 0.0;
  for (int b = w; b < nL; b += 8) {
    const int lb = lig[b];
    const double dx = xa - xyz[3 * lb], dy = ya - xyz[3 * lb + 1], dz = za - xyz[3 * lb + 2];
    const double r2 = dx * dx + dy * dy + dz * dz;
    double v = 0.0, e = 0.0;
    int cls = 0;
    if (live && !(r2 < 1e-20))  // r < 1e-10 is skipped; an atom in both lists pairs with itself at r = 0
      cls = ra < lb ? pair_class(wa, far, a0, a1, ra, lb) : pair_class(win[lb], far, farp[lb], farp[lb + 1], lb, ra);
    if (cls) {
      const double ri = rsqrt(r2), i2 = ri * ri, i6 = i2 * i2 * i2;
      v = (A[ta + type[lb]] * i6 - B[ta + type[lb]]) * i6;
      e = qa * q[lb] * ri;
      if (cls == 2) {
        v /= scnb;
        e /= scee;
      }
    }
    sv += v;
    se += e;
    v = warp_sum(v);
    e = warp_sum(e);
    if (lane == 0) {
      colpart[2 * ((long long)blockIdx.x * nL + b)] = v;
      colpart[2 * ((long long)blockIdx.x * nL + b) + 1] = e;
    }
  }
  acc[w][0][lane] = sv;
  acc[w][1][lane] = se;
  __syncthreads();
  if (threadIdx.x < 64) {
    double t = 0.0;
    for (int h = 0; h < 8; h++) t += acc[h][w][lane];
    if (live) rows[2 * a + w] = t;
  }
}

__global__ void k_colpart(const double* __restrict__ in, int blocks, int cols, double* __restrict__ out) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (c >= cols) return;
  double s = 0.0;
  for (int b = lane; b < blocks; b += 32) s += in[(long long)b * cols + c];
  s = warp_sum(s);
  if (lane == 0) out[c] = s;
}

void plain_decomp_pairs(Ctx* c, cudaStream_t st, const DevTopo& C, const double* d_xyz, const int* d_rec, int nR, const int* d_lig,
                        int nL, double* d_rows, double* d_cols) {
  if (nR <= 0 || nL <= 0) {
    if (nR > 0) RSTG_CUDA(cudaMemsetAsync(d_rows, 0, (size_t)nR * 16, st));
    if (nL > 0) RSTG_CUDA(cudaMemsetAsync(d_cols, 0, (size_t)nL * 16, st));
    return;
  }
  const int blocks = (nR + 31) / 32;
  DevBuf part((size_t)blocks * nL * 16, st);
  k_decomp<<<blocks, 256, 0, st>>>(d_xyz, C.q.as<double>(), C.type.as<int>(), (int)C.nt, C.ljA.as<double>(),
                                          C.ljB.as<double>(), C.win.as<ulonglong2>(), C.farp.as<int>(), C.far.as<int>(),
                                          C.scee, C.scnb, d_rec, nR, d_lig, nL, d_rows, part.as<double>());
  k_colpart<<<(2 * nL + 7) / 8, 256, 0, st>>>(part.as<double>(), blocks, 2 * nL, d_cols);
  launched(c, 2);
}

// ---------------------------------------------------------------------------
// Deterministic column sums (one block per column, fixed thread order).
// ---------------------------------------------------------------------------
__global__ void k_sum_columns(const double* __restrict__ in, long long rows, int cols, double* __restrict__ out) {
  __shared__ double sh[32];
  int c = blockIdx.x;
  double s = 0.0;
  for (long long r = threadIdx.x; r < rows; r += blockDim.x) s += in[r * cols + c];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) out[c] = s;
}

void sum_columns(Ctx* c, cudaStream_t st, const double* d_in, int64_t rows, int cols, double* d_out) {
  k_sum_columns<<<cols, 512, 0, st>>>(d_in, rows, cols, d_out);
  launched(c);
}

}  // namespace rstg
