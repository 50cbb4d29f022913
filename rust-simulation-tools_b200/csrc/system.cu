// Batched, binding-difference-fused MM-GBSA engine.
//
// Layout: complex atoms are permuted into "slots": receptor atoms first
// (slots [0, nR)), then ligand atoms (slots [nR, nC)); each part is sorted
// along a Morton curve of the first frame so that a 128-slot tile is a compact
// blob and close pairs fall into few tiles.  Per batch of B frames:
//
//   K0 prep     input frames -> slot-ordered FP64 and FP32 coordinates
//   K1 psi      HCT descreening over all ordered complex pairs, split into
//               own-part and other-part sums: psi_C = psi_own + psi_other
//               (descreening is pairwise additive, gb_energy.rs:157-217), so
//               the complex and sub-system Born radii come from one pass;
//               also emits each atom's SASA neighbour list
//   K2 pairs    32 rows by 32-column words of the triangle: GB pair energy with complex radii
//               and, for same-part pairs, with sub-system radii; LJ+Coulomb
//               for same-part pairs
//   K3 sasa     a warp per atom: a point is accessible in the sub-system iff
//               no own-part neighbour buries it, and in the complex iff also
//               no other-part neighbour does (core/src/sasa.rs:256-265)
//   K4 rl       receptor x ligand LJ+Coulomb and GB in FP64, per-atom row/column sums
//               (binding difference of the non-bonded term and the
//               per-residue vdW/elec of decomposition.rs:240-283)
//   K6 bonded   bonded terms by part, and 1-4 class corrections
//   K5 reduce   per-frame FrameEnergy (binding.rs:333-415) and per-residue
//               terms (decomposition.rs:309-375)
//
// Precision: FP32 pair arithmetic with FP64 accumulation; close pairs
// (r < 3.5 A for LJ/Coulomb, any pair outside the far-field series domain for
// the HCT integral) take the reference's FP64 expressions; SASA point tests
// are FP32 with an FP64 re-check of the reference expression inside a
// band of +-2e-4 A^2 (more for large probes), so accessible-point counts equal the reference's.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>

#include "common.cuh"
#include "f32x2.cuh"
#include "system.hpp"

namespace rstg {

// A^2: SASA point tests closer than this to the threshold are redone in FP64 with
// the reference's rounding.  A test's FP32 error grows with the squared reach
// (er + the largest expanded radius)^2, the bound of its terms: 4e-6 of it is ten
// times the error, 2e-4 at a probe of 1.4 A.
static constexpr float kSasaBand = 2e-4f, kSasaBandRel = 4e-6f;
static constexpr float kNbGuard2 = 3.5f * 3.5f;

// k_sasa: warps per block (fewer where the neighbours of four do not fit), and classes of its neighbour order per part (own, other)
static constexpr int kSasaWarps = 4, kSasaBins = 8;
// neighbour capacity with the padding of the two parts to whole groups of four
__host__ __device__ constexpr int sasa_cap(int cap) { return cap + 8; }
// shared memory of a k_sasa block: per warp the ordered neighbours (four
// floats and the atom each), each entry's class and place, the class counts
static size_t sasa_smem(int cap, int warps) {
  return (size_t)warps * (sasa_cap(cap) * (4 * sizeof(float) + 2 * sizeof(int)) + 2 * kSasaBins * sizeof(int));
}

struct GbConstF {
  double kappa, inv_ein, inv_eout, diel_ns, cut2;
  double f0;        // -(1/eps_in - 1/eps_out)/2 without salt: the decomposition's weights (decomposition.rs:320-337)
  float fk, fie, fio, fdns, fcut2;
  float fkl;        // -fk log2(e): E = 2^(fkl f)
  float fdev;       // 0.52 fk times the largest radius
  float tile_far2;  // A^2: k_psi row and column groups whose boxes are farther apart hold no SASA neighbours and only far-field pairs
  int no_salt, model;
  double rgbmax;
};

struct FusedParams {
  DevBuf slot_src, P32, q64, rho64, rad64, sj64, type, lj32, lj64, items, tile_rec, masks, sphere32, sphere64,
      res_ptr, res_slots, bterms, bpar, corr;
  int nt = 0, nb = 0, nitems = 0, nrec = 0, npts = 0, nres = 0, nterms = 0, ncorr = 0;
  double probe = 1.4;
  float max_ext = 0.f;  // largest radius + probe
  GbConstF gb{};
};

// ---------------------------------------------------------------------------
// K0: prep
// ---------------------------------------------------------------------------
// Also the bounding box of every 32 consecutive slots (one warp; slots follow
// a Morton curve, so the boxes are compact): two float4 (min, max) per chunk.
__global__ void k_prep(int nC, int n_top, const void* __restrict__ in, int f64, const int* __restrict__ slot_src,
                       const float4* __restrict__ P32, double* __restrict__ xyz64, float4* __restrict__ xyz32,
                       float4* __restrict__ boxes) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  int f = blockIdx.y;
  const bool live = s < nC;
  if ((s & ~31) >= nC) return;  // whole warps only
  if (!live) s = nC - 1;
  long long src = ((long long)f * n_top + slot_src[s]) * 3;
  double x[3];
  if (f64) {
    const double* p = (const double*)in + src;
    x[0] = p[0];
    x[1] = p[1];
    x[2] = p[2];
  } else {
    // DCD path: float32 Angstrom -> f64 nm (dcd.rs:429-437) -> Angstrom (binding.rs:630-633)
    const float* p = (const float*)in + src;
    for (int d = 0; d < 3; d++) x[d] = __dmul_rn(__dmul_rn((double)p[d], 0.1), 10.0);
  }
  long long o = (long long)f * nC + s;
  const float4 v = make_float4((float)x[0], (float)x[1], (float)x[2], P32[s].x);
  if (live) {
    xyz64[3 * o] = x[0];
    xyz64[3 * o + 1] = x[1];
    xyz64[3 * o + 2] = x[2];
    xyz32[o] = v;
  }
  float lo[3] = {v.x, v.y, v.z}, hi[3] = {v.x, v.y, v.z};
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1)
#pragma unroll
    for (int d = 0; d < 3; d++) {
      lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], sh));
      hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], sh));
    }
  if ((threadIdx.x & 31) == 0) {
    const long long c = (long long)f * ((nC + 31) >> 5) + (s >> 5);
    boxes[2 * c] = make_float4(lo[0], lo[1], lo[2], 0.f);
    boxes[2 * c + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
  }
}

// ---------------------------------------------------------------------------
// K1: psi + Born radii + self energies + SASA neighbour lists
// ---------------------------------------------------------------------------
// HCT integral of one pair (gb_energy.rs:157-217) in FP64: one division for
// 1/l and 1/u, one for 1/r.
__device__ __forceinline__ double hct64(double r2, double rho_i, double sj) {
  const double r = sqrt(r2);
  if (r == 0.0 || rho_i >= r + sj) return 0.0;
  const double u = r + sj, d = fabs(r - sj), l = rho_i > d ? rho_i : d;
  const double inv = 1.0 / (l * u), li = u * inv, ui = l * inv, ri = 1.0 / r;
  const double c = 0.5 * (li - ui + 0.25 * (ui * ui - li * li) * (r - sj * sj * ri) + 0.5 * log(l * ui) * ri);
  return (rho_i < sj - r) ? c + 2.0 * (1.0 / rho_i - li) : c;
}

__device__ __forceinline__ double radius64(double psi, double rho_i, double radius_i, int model, double rgbmax) {
  double alpha = 1.0, beta = 0.0, gamma = 0.0;
  if (model == 1) {
    alpha = 0.8;
    gamma = 2.909125;
  } else if (model == 2) {
    beta = 0.8;
    gamma = 4.85;
  }
  double R;
  if (model == 0) {
    double inv_r = 1.0 / rho_i - psi;
    R = inv_r > 0.0 ? 1.0 / inv_r : rgbmax;
  } else {
    double pr = psi * rho_i, p2 = pr * pr, p3 = p2 * pr;
    double inv_r = 1.0 / rho_i - tanh(alpha * pr - beta * p2 + gamma * p3) / radius_i;
    R = inv_r > 0.0 ? 1.0 / inv_r : rgbmax;
  }
  return R > rgbmax ? rgbmax : R;
}

__device__ __forceinline__ double self64(double q, double R, const GbConstF& k) {
  if (k.no_salt) return k.diel_ns * q * q / R;
  return -0.5 * q * q * (k.inv_ein - exp(-kKScale * k.kappa * R) * k.inv_eout) / R;
}

// Far-field HCT integral: with l = r - s, u = r + s (rho_i <= r - s) the
// reference expression equals (1/r) sum_k k/(2k+1) x^(2k+1), x = s/r.  The
// series has no cancellation; what follows k = 6 is at most 8.3e-8 of the first
// term, at x = 1/4 ((7/15) x^15 against x^3 / 3).
// In terms of u = 1/r^2 and the column's s^2, s^3: x^2 = s^2 u and
// x^3 / r = s^3 u^2.
// hct_add adds the pair's term to acc with one rounding.
__host__ __device__ constexpr float hct_c(int t) { return (float)(6 - t) / (float)(13 - 2 * t); }  // k / (2k + 1), k = 6 - t
__device__ __forceinline__ float hct_add(float s2, float s3, float u, float acc) {
  const float x2 = s2 * u;
  float p = fmaf(x2, hct_c(0), hct_c(1));
#pragma unroll
  for (int t = 2; t < 6; t++) p = fmaf(x2, p, hct_c(t));
  return fmaf(s3 * u, u * p, acc);
}

// reciprocal with the special-function unit's approximation (relative error
// about 2^-23, the order of the FP32 rounding of the series it feeds)
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Squared distance of two boxes (lo, hi): 0 where they overlap.
__device__ __forceinline__ float box_gap2(const float4& alo, const float4& ahi, const float4& blo, const float4& bhi) {
  const float gx = fmaxf(0.f, fmaxf(blo.x - ahi.x, alo.x - bhi.x)), gy = fmaxf(0.f, fmaxf(blo.y - ahi.y, alo.y - bhi.y)),
              gz = fmaxf(0.f, fmaxf(blo.z - ahi.z, alo.z - bhi.z));
  return fmaf(gx, gx, fmaf(gy, gy, gz * gz));
}
// Largest squared distance of two points of the boxes.
__device__ __forceinline__ float box_span2(const float4& alo, const float4& ahi, const float4& blo, const float4& bhi) {
  const float gx = fmaxf(bhi.x - alo.x, ahi.x - blo.x), gy = fmaxf(bhi.y - alo.y, ahi.y - blo.y),
              gz = fmaxf(bhi.z - alo.z, ahi.z - blo.z);
  return fmaf(gx, gx, fmaf(gy, gy, gz * gz));
}

// Born radii of 64 rows of a frame.  Eight warps share the rows (two per
// lane) and take the frame's 128-column tiles in turn, so a small frame
// spreads over its warps and no block barrier stands between tiles: each
// warp stages its own columns (structure of arrays) in shared memory.  The far
// field is evaluated for two columns per instruction (f32x2.cuh); with two
// rows per lane a 16-byte shared load feeds eight pairs, which keeps the
// loop at the issue rate rather than the shared-memory rate.  Per row and
// 32-column word one of four forms runs, chosen from the chunks' bounding
// boxes by a ballot over eight tiles at once:
//   far      boxes farther apart than k.tile_far2: no SASA neighbour, no near
//            pair (both rows of a lane in one loop when both are far)
//   near     per-pair tests into two bit masks; marked pairs go to the row's
//            SASA neighbour list and to a short list of near pairs
//   general  words that straddle the receptor / ligand boundary or the end of
//            the slots, or that a finite cutoff may cut
// FP32 far sums run over the columns of a tile in order (of either half of it
// where `halves`, see psi_halves), then enter the FP64 sums.  The near pairs (FP64) are evaluated after the column loop by four
// lanes per row over the row's whole list, so lanes stay evenly loaded.
// Every sum has a fixed order that does not depend on the number of frames.
// Bound by instruction issue (66 % of the slots, FMA pipe 57 %).  128 frames of
// 5,050 atoms: 5.9 ms with one thread per row and scalar arithmetic, 3.1 ms
// here (41 M -> 18 M warp instructions a frame); 10 frames of 2,030 atoms:
// 481 -> 115 us, 1 frame of 132 atoms: 69 -> 37 us.
constexpr int kPsiRows = 64, kPsiWarps = 8, kPsiCap = 48, kPsiBatch = 8, kPsiCols = 64;
struct PsiSmem {
  union {
    float col[kPsiWarps][7][kPsiCols];  // x, y, z, s, s^2, s^3, SASA reach of half of a warp's tile
    double2 psi[kPsiWarps][kPsiRows];
  };
  unsigned short list[kPsiWarps][kPsiCap][kPsiRows];  // near pairs: (tile of the warp) * 128 + column
  int scnt[kPsiRows];
  unsigned short ncnt[kPsiWarps][kPsiRows];
  double red[32];
};

struct PsiRow {
  f2 x, y, z;
  float rho, ext, po, pc;
  int i;
  bool in_r;
};

__global__ void __launch_bounds__(32 * kPsiWarps, 3)
    k_psi(int nC, int nR, const float4* __restrict__ xyz32, const double* __restrict__ xyz64,
          const float4* __restrict__ boxes, const float4* __restrict__ P32, const double* __restrict__ rho64,
          const double* __restrict__ sj64, const double* __restrict__ rad64, const double* __restrict__ q64, GbConstF k,
          int halves, int cap, int* __restrict__ nbr, int* __restrict__ nbrcnt, double* __restrict__ R64, float4* __restrict__ Rf,
          float* __restrict__ dRf, double* __restrict__ wdec, double* __restrict__ part, int* __restrict__ diag) {
  extern __shared__ __align__(16) unsigned char psi_raw[];
  PsiSmem& sm = *reinterpret_cast<PsiSmem*>(psi_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, f = blockIdx.y, row0 = blockIdx.x * kPsiRows;
  const float4* X = xyz32 + (long long)f * nC;
  const double* X64 = xyz64 + (long long)f * nC * 3;
  const int nchunk = (nC + 31) >> 5, ntile = (nC + kTile - 1) / kTile;
  const float4* B = boxes + 2LL * f * nchunk;
  if (threadIdx.x < kPsiRows) sm.scnt[threadIdx.x] = 0;
  __syncthreads();
  PsiRow R[2];
  double psiO[2] = {0.0, 0.0}, psiX[2] = {0.0, 0.0};
  int nc[2] = {0, 0};
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const int i = min(row0 + 32 * r + lane, nC - 1);
    const float4 x = X[i], p = P32[i];
    R[r] = PsiRow{dup2(x.x), dup2(x.y), dup2(x.z), p.y, p.w, 0.f, 0.f, i, i < nR};
  }
  const bool live1 = row0 + 32 < nC;  // the second 32 rows hold any atom (the first always do)
  const unsigned vmask[2] = {row0 + lane < nC ? ~0u : 0u, row0 + 32 + lane < nC ? ~0u : 0u};
  const int ch0 = row0 >> 5, ch1 = min(ch0 + 1, nchunk - 1);
  // few tiles: two warps per tile, one for each 32 rows
  const bool split = 2 * ntile <= kPsiWarps;
  const int tstep = split ? kPsiWarps / 2 : kPsiWarps, tfirst = split ? warp >> 1 : warp;
  float (*col)[kPsiCols] = sm.col[warp];
  int n64 = 0;

  auto near_direct = [&](int r, int j) {  // a near pair that found no room in the list
    const int i = R[r].i;
    const double dx = X64[3 * i] - X64[3 * j], dy = X64[3 * i + 1] - X64[3 * j + 1], dz = X64[3 * i + 2] - X64[3 * j + 2];
    const double r2 = dx * dx + dy * dy + dz * dz;
    n64++;
    if (r2 > k.cut2) return;
    const double t = hct64(r2, rho64[i], sj64[j]);
    if ((j < nR) == R[r].in_r)
      psiO[r] += t;
    else
      psiX[r] += t;
  };
  // marked pairs of a word to the lists; kt: ordinal of the tile among this warp's
  auto append = [&](int r, unsigned nm, unsigned sm_, int jw, int c0, int kt) {
    const int rl = 32 * r + lane;
    if (sm_) {
      int b = atomicAdd(&sm.scnt[rl], __popc(sm_));
      int* my = nbr + ((long long)f * nC + R[r].i) * cap;
      do {
        const int c = __ffs(sm_) - 1;
        sm_ &= sm_ - 1;
        if (b < cap) my[b] = jw + c;
        b++;
      } while (sm_);
    }
    while (nm) {
      const int c = __ffs(nm) - 1;
      nm &= nm - 1;
      if (nc[r] < kPsiCap && kt < 512)
        sm.list[warp][nc[r]++][rl] = (unsigned short)(kt * kTile + c0 + c);
      else
        near_direct(r, jw + c);
    }
  };

  for (int kb = 0; tfirst + tstep * kb < ntile; kb += kPsiBatch) {
    // forms of the words of the next eight tiles, one word per lane
    unsigned far_[2], near_[2];
    {
      const int t = tfirst + tstep * (kb + (lane >> 2)), c = 4 * t + (lane & 3);
      const int cc = min(c, nchunk - 1);
      const float4 lo = B[2 * cc], hi = B[2 * cc + 1];
      const bool full = t < ntile && 32 * c + 32 <= nC && (32 * c + 32 <= nR || 32 * c >= nR);
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const int rc = r ? ch1 : ch0;
        const float4 rlo = B[2 * rc], rhi = B[2 * rc + 1];
        const bool ok = full && box_span2(rlo, rhi, lo, hi) * 1.0001f < k.fcut2;
        const bool fr = box_gap2(rlo, rhi, lo, hi) > k.tile_far2;
        far_[r] = __ballot_sync(0xffffffffu, ok && fr);
        near_[r] = __ballot_sync(0xffffffffu, ok && !fr);
      }
    }
    for (int q = 0; q < kPsiBatch; q++) {
      const int kt = kb + q, t = tfirst + tstep * kt, j0 = t * kTile;
      if (t >= ntile) break;
      R[0].po = R[0].pc = R[1].po = R[1].pc = 0.f;
      auto flush = [&] {
#pragma unroll
        for (int r = 0; r < 2; r++) {
          psiO[r] += (double)R[r].po;
          psiX[r] += (double)R[r].pc;
        }
      };
#pragma unroll 1
      for (int w = 0; w < 4; w++) {
        if (w == 2 && halves) {
          flush();
          R[0].po = R[0].pc = R[1].po = R[1].pc = 0.f;
        }
        if ((w & 1) == 0) {  // stage the next half of the tile: two columns per lane
          const int j = j0 + 32 * w + 2 * lane;
          const float4 x0 = X[min(j, nC - 1)], x1 = X[min(j + 1, nC - 1)], p0 = P32[min(j, nC - 1)],
                       p1 = P32[min(j + 1, nC - 1)];
          __syncwarp();
          auto put = [&](int a, float v0, float v1) { *(float2*)&col[a][2 * lane] = make_float2(v0, v1); };
          put(0, x0.x, x1.x);
          put(1, x0.y, x1.y);
          put(2, x0.z, x1.z);
          put(3, p0.z, p1.z);
          put(4, p0.z * p0.z, p1.z * p1.z);
          put(5, p0.z * p0.z * p0.z, p1.z * p1.z * p1.z);
          put(6, p0.w, p1.w);
          __syncwarp();
        }
        const int c0 = 32 * (w & 1), bit = 4 * q + w, jw = j0 + 32 * w;  // first column in the stage, and its slot
        const bool f0 = (far_[0] >> bit) & 1u, f1 = (far_[1] >> bit) & 1u;
        const bool own0 = (jw < nR) == R[0].in_r, own1 = (jw < nR) == R[1].in_r;  // of a word inside one part
        auto ld = [&](int a, int jj) { return *(const ulonglong2*)&col[a][jj]; };
        // far-field terms of two columns added to acc in column order
        auto far2 = [&](const PsiRow& P, f2 x, f2 y, f2 z, f2 s2, f2 s3, float acc) {
          const f2 dx = sub2(P.x, x), dy = sub2(P.y, y), dz = sub2(P.z, z);
          const f2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
          float a, b;
          un2(r2, a, b);
          const f2 u = pk2(rcp_approx(a), rcp_approx(b)), x2 = mul2(s2, u);
          f2 p = fma2(x2, dup2(hct_c(0)), dup2(hct_c(1)));
#pragma unroll
          for (int h = 2; h < 6; h++) p = fma2(x2, p, dup2(hct_c(h)));
          float a0, a1, b0, b1;
          un2(mul2(s3, u), a0, a1);
          un2(mul2(u, p), b0, b1);
          return fmaf(a1, b1, fmaf(a0, b0, acc));
        };
        if (f0 && f1 && !split) {
          float a0 = own0 ? R[0].po : R[0].pc, a1 = own1 ? R[1].po : R[1].pc;
#pragma unroll 2
          for (int jj = c0; jj < c0 + 32; jj += 4) {
            const ulonglong2 x = ld(0, jj), y = ld(1, jj), z = ld(2, jj), s2 = ld(4, jj), s3 = ld(5, jj);
            a0 = far2(R[0], x.x, y.x, z.x, s2.x, s3.x, a0);
            a1 = far2(R[1], x.x, y.x, z.x, s2.x, s3.x, a1);
            a0 = far2(R[0], x.y, y.y, z.y, s2.y, s3.y, a0);
            a1 = far2(R[1], x.y, y.y, z.y, s2.y, s3.y, a1);
          }
          (own0 ? R[0].po : R[0].pc) = a0;
          (own1 ? R[1].po : R[1].pc) = a1;
          continue;
        }
#pragma unroll
        for (int r = 0; r < 2; r++) {
          if ((r == 1 && !live1) || (split && r != (warp & 1))) continue;
          PsiRow& P = R[r];
          const bool own = r ? own1 : own0;
          if (r ? f1 : f0) {
            float a = own ? P.po : P.pc;
#pragma unroll 2
            for (int jj = c0; jj < c0 + 32; jj += 4) {
              const ulonglong2 x = ld(0, jj), y = ld(1, jj), z = ld(2, jj), s2 = ld(4, jj), s3 = ld(5, jj);
              a = far2(P, x.x, y.x, z.x, s2.x, s3.x, a);
              a = far2(P, x.y, y.y, z.y, s2.y, s3.y, a);
            }
            (own ? P.po : P.pc) = a;
          } else if ((near_[r] >> bit) & 1u) {
            float a = own ? P.po : P.pc;
            unsigned nm = 0u, sm_ = 0u;
            const f2 rho = dup2(P.rho), ext = dup2(P.ext);
#pragma unroll 1
            for (int jj = c0; jj < c0 + 32; jj += 4) {
              const ulonglong2 x = ld(0, jj), y = ld(1, jj), z = ld(2, jj), s1 = ld(3, jj), s2 = ld(4, jj), s3 = ld(5, jj),
                               e = ld(6, jj);
              unsigned nb = 0u, sb = 0u;
              auto two = [&](f2 xx, f2 yy, f2 zz, f2 t1, f2 t2, f2 t3, f2 ee, unsigned b0) {
                const f2 dx = sub2(P.x, xx), dy = sub2(P.y, yy), dz = sub2(P.z, zz);
                const f2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
                float ra, rb, la, lb, ta, tb, qa, qb;
                un2(r2, ra, rb);
                const f2 reach = add2(ext, ee);
                un2(fma2(mul2(reach, reach), dup2(1.00001f), dup2(1e-4f)), la, lb);
                const f2 rs = add2(rho, t1);
                un2(mul2(rs, rs), ta, tb);
                un2(mul2(dup2(16.f), t2), qa, qb);
                // far field: s <= r / 4, rho_i + s <= r and r > 0 (a pair with
                // rho_i + s < 0 that fails the squared test takes the FP64 path)
                const bool fa = ra >= fmaxf(fmaxf(ta, qa), 1.17549435e-38f), fb = rb >= fmaxf(fmaxf(tb, qb), 1.17549435e-38f);
                const f2 u = pk2(rcp_approx(ra), rcp_approx(rb)), x2 = mul2(t2, u);
                f2 p = fma2(x2, dup2(hct_c(0)), dup2(hct_c(1)));
#pragma unroll
                for (int h = 2; h < 6; h++) p = fma2(x2, p, dup2(hct_c(h)));
                float a0, a1, b0_, b1_;
                un2(mul2(t3, u), a0, a1);
                un2(mul2(u, p), b0_, b1_);
                if (fa)
                  a = fmaf(a0, b0_, a);
                else
                  nb |= b0;
                if (fb)
                  a = fmaf(a1, b1_, a);
                else
                  nb |= 2u * b0;
                if (ra <= la) sb |= b0;
                if (rb <= lb) sb |= 2u * b0;
              };
              two(x.x, y.x, z.x, s1.x, s2.x, s3.x, e.x, 1u);
              two(x.y, y.y, z.y, s1.y, s2.y, s3.y, e.y, 4u);
              nm |= nb << (jj - c0);
              sm_ |= sb << (jj - c0);
            }
            (own ? P.po : P.pc) = a;
            unsigned v = vmask[r];
            if (4 * t + w == ch0 + r) v &= ~(1u << lane);  // the row's own column
            append(r, nm & v, sm_ & v, jw, 32 * w, kt);
          } else {
            unsigned nm = 0u, sm_ = 0u;
            float xi, yi, zi, d_;
            un2(P.x, xi, d_);
            un2(P.y, yi, d_);
            un2(P.z, zi, d_);
            const int hi = min(32, nC - jw);
            for (int c = 0; c < hi; c++) {
              const int j = jw + c, jj = c0 + c;
              if (j == P.i) continue;
              const float dx = xi - col[0][jj], dy = yi - col[1][jj], dz = zi - col[2][jj];
              const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
              const float ee = P.ext + col[6][jj];
              if (r2 <= fmaf(ee * ee, 1.00001f, 1e-4f)) sm_ |= 1u << c;
              if (r2 > k.fcut2) continue;
              const float rs = P.rho + col[3][jj];
              if (r2 > 0.f && 16.f * col[4][jj] <= r2 && rs * rs <= r2) {
                float& a = ((j < nR) == P.in_r) ? P.po : P.pc;
                a = hct_add(col[4][jj], col[5][jj], rcp_approx(r2), a);
              } else {
                nm |= 1u << c;
              }
            }
            append(r, nm & vmask[r], sm_ & vmask[r], jw, 32 * w, kt);
          }
        }
      }
      flush();
    }
  }
  __syncthreads();  // every warp is done with its columns: the union turns into the partial sums
#pragma unroll
  for (int r = 0; r < 2; r++) {
    sm.psi[warp][32 * r + lane] = make_double2(psiO[r], psiX[r]);
    sm.ncnt[warp][32 * r + lane] = (unsigned short)nc[r];
  }
  __syncthreads();
  // near pairs: four lanes per row over the row's lists in warp order
  const int row = threadIdx.x >> 2, h = threadIdx.x & 3, i = min(row0 + row, nC - 1);
  const bool in_r = i < nR;
  double so = 0.0, sx = 0.0;
  {
    const double xi = X64[3 * i], yi = X64[3 * i + 1], zi = X64[3 * i + 2], rho_i = rho64[i];
    int w = 0, e = h, n = row0 + row < nC ? sm.ncnt[0][row] : 0;
    for (;;) {
      while (e >= n && w < kPsiWarps - 1) {
        e -= n;
        n = row0 + row < nC ? sm.ncnt[++w][row] : (w++, 0);
      }
      if (e >= n) break;
      const int code = sm.list[w][e][row], j = ((split ? w >> 1 : w) + tstep * (code >> 7)) * kTile + (code & 127);
      const double dx = xi - X64[3 * j], dy = yi - X64[3 * j + 1], dz = zi - X64[3 * j + 2];
      const double r2 = dx * dx + dy * dy + dz * dz;
      n64++;
      if (!(r2 > k.cut2)) {
        const double t = hct64(r2, rho_i, sj64[j]);
        if ((j < nR) == in_r)
          so += t;
        else
          sx += t;
      }
      e += 4;
    }
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    so += __shfl_xor_sync(0xffffffffu, so, o);
    sx += __shfl_xor_sync(0xffffffffu, sx, o);
  }
  double sC = 0.0, sR = 0.0, sL = 0.0, sD = 0.0, sW = 0.0;
  if (h == 0 && row0 + row < nC) {
#pragma unroll
    for (int w = 0; w < kPsiWarps; w++) {
      const double2 v = sm.psi[w][row];
      so += v.x;
      sx += v.y;
    }
    const int cnt = sm.scnt[row];
    const long long o = (long long)f * nC + i;
    nbrcnt[o] = cnt;
    if (cnt > cap) atomicMax(diag + 3, cnt);
    const double rho_i = rho64[i], rad = rad64[i];
    const double Rc = radius64(so + sx, rho_i, rad, k.model, k.rgbmax), Rs = radius64(so, rho_i, rad, k.model, k.rgbmax);
    R64[2 * o] = Rc;
    R64[2 * o + 1] = Rs;
    Rf[o] = make_float4((float)Rc, (float)Rs, (float)(1.0 / Rc), (float)(1.0 / Rs));
    dRf[o] = (float)(Rc - Rs);
    const double q = q64[i], ec = self64(q, Rc, k), es = self64(q, Rs, k);
    sC = ec;
    sD = ec - es;
    if (in_r)
      sR = es;
    else
      sL = es;
    sW = fabs(k.f0 * q * q / Rc - k.f0 * q * q / Rs);
    wdec[o] = sW;
  }
  n64 = warp_sumi(n64);
  if (lane == 0 && n64) atomicAdd((unsigned long long*)(diag + 4), (unsigned long long)n64);
  sC = block_sum(sC, sm.red);
  sR = block_sum(sR, sm.red);
  sL = block_sum(sL, sm.red);
  sD = block_sum(sD, sm.red);
  sW = block_sum(sW, sm.red);
  if (threadIdx.x == 0) {
    double* p = part + ((long long)f * gridDim.x + blockIdx.x) * 5;
    p[0] = sC;
    p[1] = sR;
    p[2] = sL;
    p[3] = sD;
    p[4] = sW;
  }
}

// ---------------------------------------------------------------------------
// K2: pair energies of the triangle, 32 rows by 32-column words
// ---------------------------------------------------------------------------
// GB pair energy (gb_energy.rs:339-353) with its ingredients:
// f_GB^2 = r2 + RiRj e, e = exp(-t), t = r2 / (4 RiRj); E = exp(-0.73 kappa f).
// The exponentials run on the special-function unit in base 2: the caller
// passes u = -t log2(e) (its per-row and per-column factors carry the
// constants), so e = 2^u, and E = 2^(fkl f) with fkl = -0.73 kappa log2(e).
// e is taken as 0 beyond t = 16 (u < kU16), where it is below 1.2e-7.  The
// pair energy is the returned value times finv.
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f, kU16 = -16.f * 1.4426950408889634f;
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float gb_pair_parts(float qq, float r2, float RiRj, float u, const GbConstF& k, float& e,
                                               float& f2, float& finv, float& E) {
  e = u > kU16 ? ex2_approx(u) : 0.f;
  f2 = fmaf(RiRj, e, r2);
  finv = rsqrtf(f2);
  if (k.no_salt) {
    E = 0.f;
    return k.fdns * qq;
  }
  float f = f2 * finv;
  E = ex2_approx(k.fkl * f);
  return -0.5f * qq * fmaf(-E, k.fio, k.fie);
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// exp(x) - 1 without cancellation: for |x| < 0.2 the Taylor sum to x^6 (the
// relative error is about x^6 / 5040 < 1.3e-8), for |x| < kSmallX that to x^4
// (about x^4 / 120 < 9e-7 of a term that is itself a correction).
constexpr float kSmallX = 0.1f;
__device__ __forceinline__ float expm1_6(float x) {
  return x * (1.f + x * (0.5f + x * (1.f / 6.f + x * (1.f / 24.f + x * (1.f / 120.f + x * (1.f / 720.f))))));
}
__device__ __forceinline__ float expm1_4(float x) { return x * (1.f + x * (0.5f + x * (1.f / 6.f + x * (1.f / 24.f)))); }

// p(complex radii) - p(subsystem radii) of one pair, evaluated from the
// differences themselves so that its rounding is relative to the difference,
// not to p: dRR = RcRc' - RsRs' comes from the FP64 radius differences;
// exp(-tS) = exp(-tC) (1 + expm1(tC - tS)) with tC - tS = -tC dRR / RRs;
// 1/fC - 1/fS = -(fC - fS)/(fC fS); E/f likewise through expm1, or as the
// difference itself where the exponents are kSmallX and more apart.  eC, f2C,
// finvC, EC are the complex pair's ingredients; uC, uS the base-2 exponents
// -tC log2(e), -tS log2(e); iRRsN = ln(2) / RRs, so tC - tS = uC dRR iRRsN.
__device__ __forceinline__ float gb_pair_delta(float qq, float r2, float RRc, float RRs, float iRRsN, float dRR,
                                               float uC, float uS, float eC, float f2C, float finvC, float EC,
                                               const GbConstF& k) {
  float dt = uC * dRR * iRRsN;  // tC - tS
  float g;                      // RRc eC - RRs eS
  if (fabsf(dt) < 0.2f && uC > kU16) {
    g = eC * (dRR - RRs * expm1_6(dt));
  } else {
    float eS = uS > kU16 ? ex2_approx(uS) : 0.f;
    g = RRc * eC - RRs * eS;
  }
  float f2S = f2C - g;
  float finvS = rsqrtf(f2S);
  float df = __fdividef(g, f2C * finvC + f2S * finvS);  // fC - fS
  float dinv = -df * finvC * finvS;                     // 1/fC - 1/fS
  if (k.no_salt) return k.fdns * qq * dinv;
  const float zz = k.fk * df;
  const float dh = fabsf(zz) < kSmallX ? EC * (dinv - expm1_4(zz) * finvS)  // EC/fC - ES/fS
                                       : EC * finvC - ex2_approx(k.fkl * (f2S * finvS)) * finvS;
  return -0.5f * qq * (k.fie * dinv - k.fio * dh);
}

__device__ __forceinline__ double nb64(const double* X64, int i, int j, double qq, double A, double B, int cls,
                                      double scee, double scnb) {
  double dx = X64[3 * i] - X64[3 * j], dy = X64[3 * i + 1] - X64[3 * j + 1], dz = X64[3 * i + 2] - X64[3 * j + 2];
  double r2 = dx * dx + dy * dy + dz * dz, r = sqrt(r2), r6 = r2 * r2 * r2, r12 = r6 * r6;
  if (cls == 2) return (A / r12 - B / r6) / scnb + qq / r / scee;
  return (A / r12 - B / r6) + qq / r;
}

// One row of a tile.
struct PairRow {
  float4 xi, Ri;
  float dRi, iRc, iRs, iRsN;  // -log2(e) / (4 R_C), -log2(e) / (4 R_part), ln(2) / R_part
  int ti;
  bool in_r;
};

// The 32 columns of a word as arrays, so that one 16-byte shared load feeds
// four columns of every row.
struct PairTile {
  float x[32], y[32], z[32], q[32];
  float Rc[32], Rs[32], iRc[32], iRs[32], dR[32];
  int t[32];  // type * number of types: the column's row of the Lennard-Jones table
};

// Sums of one row over one 32-column word: GB pair energy with complex
// radii, with part radii, their difference, Lennard-Jones + Coulomb (times
// kMmScale: with salt the Lennard-Jones table carries the -1/2 of the GB
// prefactor, so that one product of charges serves both; a power of two, so
// every rounding is the unscaled one's).
struct PairSum {
  float c, s, d, m;
};
template <bool kSalt>
constexpr float kMmScale = kSalt ? -0.5f : 1.f;

// Columns [lo, hi) of the word from slot j0 on one by one, with every test: the receptor /
// ligand class of each pair, the cutoff (of the GB terms), the exclusion (wex) and 1-4 (w14)
// masks.  Cross pairs contribute the complex GB energy only (their
// Lennard-Jones, Coulomb and binding GB terms are summed in FP64 by
// k_rl).  FP64 Lennard-Jones / Coulomb pairs are marked in dfr.  fused
// (words of a 128 x 128 tile between the parts): a pair's product enters the
// sum with one rounding; elsewhere the pair energy is rounded first, since the
// part's sum takes the same value.
template <bool kSalt>
__device__ __forceinline__ void pair_word(int lo, int hi, int j0, int nR, bool fused, const PairRow& P, const GbConstF& k,
                                          const PairTile& T, const float2* __restrict__ slj, unsigned wex, unsigned w14,
                                          PairSum& a, unsigned& dfr) {
#pragma unroll 1
  for (int jj = lo; jj < hi; jj++) {
    const float dx = P.xi.x - T.x[jj], dy = P.xi.y - T.y[jj], dz = P.xi.z - T.z[jj];
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const bool same = (j0 + jj < nR) == P.in_r;
    const float qq = P.xi.w * T.q[jj];
    if (!(r2 > k.fcut2)) {  // the cutoff is of the GB terms alone
      const float tc = r2 * P.iRc * T.iRc[jj];  // -t log2(e): P.iRc carries -log2(e) / (4 R_C,i)
      const float RRc = P.Ri.x * T.Rc[jj];
      float eC, f2C, finvC, EC;
      const float wC = gb_pair_parts(qq, r2, RRc, tc, k, eC, f2C, finvC, EC), pC = __fmul_rn(wC, finvC);
      a.c = fused ? fmaf(wC, finvC, a.c) : __fadd_rn(a.c, pC);
      if (same) {
        const float ts = r2 * P.iRs * T.iRs[jj];
        const float dRR = fmaf(P.Ri.x, T.dR[jj], T.Rs[jj] * P.dRi);  // RcRc' - RsRs'
        const float dp = (dRR == 0.f || (tc <= kU16 && ts <= kU16))
                             ? 0.f
                             : gb_pair_delta(qq, r2, RRc, P.Ri.y * T.Rs[jj], P.iRsN * T.iRs[jj], dRR, tc, ts, eC, f2C,
                                             finvC, EC, k);
        a.s = __fadd_rn(a.s, __fsub_rn(pC, dp));
        a.d = __fadd_rn(a.d, dp);
      }
    }
    if (!same) continue;
    const bool is14 = (w14 >> jj) & 1u, excl = (wex >> jj) & 1u;
    if (is14 || (!excl && r2 < kNbGuard2)) {
      dfr |= 1u << jj;
    } else if (!excl) {
      // the column's type selects the table row (one for the warp) and the
      // lanes' row types spread over it: few shared-memory bank conflicts
      const float2 ab = slj[T.t[jj] + P.ti];
      const float rinv = rsqrtf(r2), ir2 = rinv * rinv, ir6 = ir2 * ir2 * ir2;
      a.m += fmaf(ab.x * ir6, ir6, fmaf(-ab.y, ir6, kMmScale<kSalt> * qq * rinv));
    }
  }
}

// The word's 32 columns, two per packed instruction, each pair with the
// scalar code's operations and rounding and the columns added in order.
// kForm: kCross, kCrossFused receptor x ligand words (GB pair energy with
// complex radii only, see pair_word); kSmall words whose radii differ too little for |tC - tS| >= 0.2 and
// for |0.73 kappa (fC - fS)| >= kSmallX, so the difference form needs its common branch only (a pair with t beyond 16
// for one radii set alone counts as beyond it for both: below 1e-9 of the
// pair); kAny words that evaluate both branches, far the largest |0.73 kappa (fC - fS)| among their pairs (from
// kSmallX on the sums do not hold); kMm words wholly beyond the
// cutoff, Lennard-Jones and Coulomb terms alone.  kTests: words that may hold
// FP64 Lennard-Jones / Coulomb pairs or masked ones.  No cutoff test: the
// caller has ruled it out.
enum PairForm { kCross, kCrossFused, kSmall, kAny, kMm };
template <bool kSalt, PairForm kForm, bool kTests>
__device__ __forceinline__ void pair_word2(const PairRow& P, const GbConstF& k, const PairTile& T,
                                           const float2* __restrict__ slj, unsigned wex, unsigned w14, PairSum& a,
                                           unsigned& dfr, float& far) {
  const f2 xi = dup2(P.xi.x), yi = dup2(P.xi.y), zi = dup2(P.xi.z), qi = dup2(kMmScale<kSalt> * P.xi.w);
  const f2 Rci = dup2(P.Ri.x), Rsi = dup2(P.Ri.y), iRci = dup2(P.iRc), iRsi = dup2(P.iRs), niRsN = dup2(-P.iRsN),
           dRi = dup2(P.dRi);
  const f2 fie = dup2(k.fie), nfio = dup2(-k.fio), fkl = dup2(k.fkl), fk = dup2(k.fk);
  const unsigned skip = wex | w14;
  // Lennard-Jones and Coulomb terms of two columns
  auto mm = [&](f2 r2, f2 qq, int t0, int t1, int b) {
    float r0, r1, i0, i1, q0, q1;
    un2(r2, r0, r1);
    const f2 ri = pk2(rsqrtf(r0), rsqrtf(r1)), i2 = mul2(ri, ri);
    un2(mul2(mul2(i2, i2), i2), i0, i1);
    un2(mul2(qq, ri), q0, q1);
    const float2 A = slj[t0 + P.ti], B = slj[t1 + P.ti];
    const float m0 = fmaf(A.x * i0, i0, fmaf(-A.y, i0, q0)), m1 = fmaf(B.x * i1, i1, fmaf(-B.y, i1, q1));
    if (kTests) {
      const unsigned o0 = 1u << b, o1 = 2u << b;
      if (r0 < kNbGuard2) dfr |= o0;
      if (r1 < kNbGuard2) dfr |= o1;
      if (!((dfr | skip) & o0)) a.m = __fadd_rn(a.m, m0);
      if (!((dfr | skip) & o1)) a.m = __fadd_rn(a.m, m1);
    } else {
      a.m = __fadd_rn(__fadd_rn(a.m, m0), m1);
    }
  };
  auto two = [&](f2 x, f2 y, f2 z, f2 q, f2 Rc, f2 Rs, f2 iRc, f2 iRs, f2 dR, int t0, int t1, int b) {
    const f2 dx = sub2(xi, x), dy = sub2(yi, y), dz = sub2(zi, z);
    const f2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
    const f2 qq = mul2(qi, q), tc = mul2(mul2(r2, iRci), iRc), RRc = mul2(Rci, Rc);
    if (kForm == kMm) {
      mm(r2, qq, t0, t1, b);
      return;
    }
    float u0, u1;
    un2(tc, u0, u1);
    const bool v0 = u0 > kU16, v1 = u1 > kU16;
    const float e0 = ex2_approx(u0), e1 = ex2_approx(u1);
    const f2 e = pk2(v0 ? e0 : 0.f, v1 ? e1 : 0.f), f2C = fma2(RRc, e, r2);
    float c0_, c1_;
    un2(f2C, c0_, c1_);
    const f2 finv = pk2(rsqrtf(c0_), rsqrtf(c1_));
    const f2 w = kSalt ? qq : mul2(dup2(k.fdns), qq);  // (with salt qq carries the -1/2)
    f2 E, wC = w;
    if (kSalt) {
      float h0, h1;
      un2(mul2(fkl, mul2(f2C, finv)), h0, h1);
      E = pk2(ex2_approx(h0), ex2_approx(h1));
      wC = mul2(w, fma2(E, nfio, fie));
    }
    const f2 pC = mul2(wC, finv);
    float p0, p1;
    if (kForm == kCrossFused) {
      float w0, w1, i0, i1;
      un2(wC, w0, w1);
      un2(finv, i0, i1);
      a.c = fmaf(w1, i1, fmaf(w0, i0, a.c));
    } else {
      un2(pC, p0, p1);
      a.c = __fadd_rn(__fadd_rn(a.c, p0), p1);
    }
    if (kForm == kCross || kForm == kCrossFused) return;
    const f2 ts = mul2(mul2(r2, iRsi), iRs), dRR = fma2(Rci, dR, mul2(Rs, dRi)), RRs = mul2(Rsi, Rs);
    const f2 dt = mul2(mul2(tc, dRR), mul2(niRsN, iRs));  // tS - tC
    // -expm1(tC - tS), the Taylor sum of expm1_6 with alternating signs
    f2 g = fma2(dt, dup2(-1.f / 720.f), dup2(1.f / 120.f));
    g = fma2(dt, g, dup2(-1.f / 24.f));
    g = fma2(dt, g, dup2(1.f / 6.f));
    g = fma2(dt, g, dup2(-0.5f));
    g = fma2(dt, g, dup2(1.f));
    g = mul2(dt, g);
    g = mul2(e, fma2(RRs, g, dRR));  // RRc eC - RRs eS
    if (kForm == kAny) {
      float t0s, t1s, y0, y1, g0, g1, h0, h1;
      un2(ts, t0s, t1s);
      un2(dt, y0, y1);
      un2(g, g0, g1);
      const float x0 = ex2_approx(t0s), x1 = ex2_approx(t1s);
      const f2 eS = pk2(t0s > kU16 ? x0 : 0.f, t1s > kU16 ? x1 : 0.f);
      un2(fma2(RRc, e, mul2(mul2(dup2(-1.f), RRs), eS)), h0, h1);
      g = pk2(v0 && fabsf(y0) < 0.2f ? g0 : h0, v1 && fabsf(y1) < 0.2f ? g1 : h1);
    }
    const f2 f2S = sub2(f2C, g);
    float s0, s1, d0, d1, n0, n1;
    un2(f2S, s0, s1);
    const f2 finvS = pk2(rsqrtf(s0), rsqrtf(s1));
    un2(fma2(f2C, finv, mul2(f2S, finvS)), d0, d1);
    const f2 df = mul2(g, pk2(rcp_approx(d0), rcp_approx(d1)));  // fC - fS
    const f2 D = mul2(mul2(df, finv), finvS);                   // 1/fS - 1/fC
    f2 nd;                                                      // p(part radii) - p(complex radii)
    if (kSalt) {
      const f2 zz = mul2(fk, df);
      f2 h = fma2(zz, dup2(1.f / 24.f), dup2(1.f / 6.f));
      h = fma2(zz, h, dup2(0.5f));
      h = fma2(zz, h, dup2(1.f));
      h = mul2(zz, h);
      const f2 ndh = mul2(E, fma2(h, finvS, D));
      if (kForm == kAny) {
        float z0, z1;
        un2(zz, z0, z1);
        far = max3(far, fabsf(z0), fabsf(z1));
      }
      nd = mul2(w, fma2(fie, D, mul2(nfio, ndh)));
    } else {
      nd = mul2(w, D);
    }
    un2(nd, n0, n1);
    un2(add2(pC, nd), s0, s1);
    a.s = __fadd_rn(__fadd_rn(a.s, s0), s1);
    a.d = __fsub_rn(__fsub_rn(a.d, n0), n1);
    mm(r2, qq, t0, t1, b);
  };
#pragma unroll 1
  for (int jj = 0; jj < 32; jj += 4) {
    auto ld = [&](const float* v) { return *(const ulonglong2*)(v + jj); };
    const ulonglong2 x = ld(T.x), y = ld(T.y), z = ld(T.z), q = ld(T.q), Rc = ld(T.Rc), Rs = ld(T.Rs), iRc = ld(T.iRc),
                     iRs = ld(T.iRs), dR = ld(T.dR);
    const int4 t = *(const int4*)(T.t + jj);
    two(x.x, y.x, z.x, q.x, Rc.x, Rs.x, iRc.x, iRs.x, dR.x, t.x, t.y, jj);
    two(x.y, y.y, z.y, q.y, Rc.y, Rs.y, iRc.y, iRs.y, dR.y, t.z, t.w, jj + 2);
  }
  if (kTests) dfr = (dfr & ~wex) | w14;  // 1-4 pairs, and unmasked ones closer than 3.5 A
}

// Persistent warps over work items (frame, 32 rows, up to `span` 32-column
// words to their right): the Lennard-Jones type table is staged in shared
// memory once per block, everything else is a warp's own, so no barrier stands
// between items and a small frame still spreads over many warps.  A word that
// lies in one part, off the diagonal, inside the slots and inside the cutoff
// (by the chunks' bounding boxes) runs on the packed loop, with the per-pair
// tests only where the boxes come closer than 3.5 A or a mask is set; the
// others run one pair at a time.  Pairs whose Lennard-Jones / Coulomb term
// takes the FP64 path (closer than 3.5 A, or 1-4) are marked in a bit mask per
// lane; after the word the warp lists them and evaluates them one per lane,
// whichever rows they belong to.  Each item's six sums are reduced in a fixed
// order and written to its own slot.
// Bound by the FP32 pipe: about 57 FP32 operations and 6 special functions a
// pair (69 and 52 cycles of a scheduler) against 100 measured.  128 frames of
// 5,050 atoms: 8.4 ms with scalar arithmetic and a block per 128 x 128 tile,
// 4.65 here; 8 frames of 25,080 atoms 11.5 -> 6.86 ms, 1 frame of 132 atoms
// 43 -> 27 us.
constexpr int kPairWarps = 8;
struct PairWarp {
  PairTile T;
  unsigned short list[1024];  // row << 5 | column of a word's FP64 pairs
};

template <bool kSalt, int MINB>
__global__ void __launch_bounds__(32 * kPairWarps, MINB)
    k_pairs(int nC, int nR, const int4* __restrict__ items, int per_frame, long long nitems,
            const float4* __restrict__ xyz32, const double* __restrict__ xyz64, const float4* __restrict__ boxes,
            const float4* __restrict__ Rf, const float* __restrict__ dRf, const int* __restrict__ type, int nt,
            const float2* __restrict__ lj32, const double2* __restrict__ lj64, const int* __restrict__ tile_rec, int nb,
            const unsigned* __restrict__ masks, GbConstF k, double scee, double scnb, double* __restrict__ part,
            int* __restrict__ diag) {
  extern __shared__ __align__(16) unsigned char pair_raw[];
  PairWarp& W = reinterpret_cast<PairWarp*>(pair_raw)[threadIdx.x >> 5];
  float2* slj = reinterpret_cast<float2*>(pair_raw + kPairWarps * sizeof(PairWarp));  // nt*nt (A, B), [column type][row type]
  for (int t = threadIdx.x; t < nt * nt; t += blockDim.x) slj[t] = make_float2(kMmScale<kSalt> * lj32[t].x, kMmScale<kSalt> * lj32[t].y);
  __syncthreads();
  const int lane = threadIdx.x & 31, nchunk = (nC + 31) >> 5;
  const long long nwarps = (long long)gridDim.x * kPairWarps;
  PairTile& T = W.T;
  int n64 = 0;
  // consecutive items (which share their rows or columns) go to one block
  for (long long item = (long long)blockIdx.x * kPairWarps + (threadIdx.x >> 5); item < nitems; item += nwarps) {
    const int f = (int)(item / per_frame);
    const int4 it = items[item % per_frame];
    const int rch = it.x;
    const int i = rch * 32 + lane;
    const float4* X = xyz32 + (long long)f * nC;
    const double* X64 = xyz64 + (long long)f * nC * 3;
    const float4* RF = Rf + (long long)f * nC;
    const float* DR = dRf + (long long)f * nC;
    const float4* B = boxes + 2LL * f * nchunk;
    const bool live = i < nC, in_r = i < nR;
    double aC = 0.0, aS = 0.0, aD = 0.0, aM = 0.0, eR = 0.0, eL = 0.0;
    PairRow P;
    {
      const int ic = min(i, nC - 1);
      P.xi = X[ic];
      P.Ri = RF[ic];
      P.dRi = DR[ic];
      P.ti = type[ic];
      P.in_r = in_r;
      P.iRc = -0.25f * kLog2e * P.Ri.z;
      P.iRs = -0.25f * kLog2e * P.Ri.w;
      P.iRsN = kLn2 * P.Ri.w;
    }
    const float4 rlo = B[2 * rch], rhi = B[2 * rch + 1];
    const float rdev = warp_maxf(fabsf(P.dRi * P.Ri.w));
#pragma unroll 1
    for (int cch = it.y; cch < it.z; cch++) {
      const int j0 = cch * 32;
      __syncwarp();
      float cdev;  // largest |R_C - R_part| / R_part of the columns
      {
        const int j = min(j0 + lane, nC - 1);
        const float4 x = X[j], r = RF[j];
        const float d = DR[j];
        T.x[lane] = x.x;
        T.y[lane] = x.y;
        T.z[lane] = x.z;
        T.q[lane] = x.w;
        T.Rc[lane] = r.x;
        T.Rs[lane] = r.y;
        T.iRc[lane] = r.z;
        T.iRs[lane] = r.w;
        T.dR[lane] = d;
        T.t[lane] = type[j] * nt;
        cdev = warp_maxf(fabsf(d * r.w));
      }
      unsigned mex = 0u, m14 = 0u;
      const int rec = tile_rec[(rch >> 2) * nb + (cch >> 2)];
      if (rec >= 0) {
        const unsigned* mr = masks + ((long long)rec * 2 * kTile + (i & (kTile - 1))) * 4 + (cch & 3);
        mex = mr[0];
        m14 = mr[kTile * 4];
      }
      __syncwarp();
      const float4 clo = B[2 * cch], chi = B[2 * cch + 1];
      const bool cR = j0 + 32 <= nR, cL = j0 >= nR;
      const bool whole = cch != rch && (cR || cL) && j0 + 32 <= nC;
      const float gap2 = box_gap2(rlo, rhi, clo, chi) * 0.9999f;
      const bool packed = whole && box_span2(rlo, rhi, clo, chi) * 1.0001f < k.fcut2;
      const bool same = cR == in_r;  // of a packed word
      const int t0 = (rch >> 2) * kTile, u0 = (cch >> 2) * kTile;  // first slots of the row's and the column's tile
      const bool fused = (t0 + kTile <= nR && u0 >= nR) || (t0 >= nR && u0 + kTile <= nR);
      PairSum a{0.f, 0.f, 0.f, 0.f};
      unsigned dfr = 0u;
      bool single = !packed;
      float far = 0.f;
      if (packed) {
        // |tC - tS| = tC dev, dev = |RcRc' - RsRs'| / RsRs' and tC < 16; then |fC^2 - fS^2| <= 1.01 RsRs' dev
        // (e^-t (1 + 1.11 t) stays below 1.01) and f >= sqrt(RR), so |fC - fS| <= 0.52 R dev of the largest R
        const float dev = rdev + (1.f + rdev) * cdev;
        const bool small = 16.1f * dev < 0.2f && k.fdev * dev < kSmallX;
        if (!__any_sync(0xffffffffu, same && live))
          if (fused)
            pair_word2<kSalt, kCrossFused, false>(P, k, T, slj, 0u, 0u, a, dfr, far);
          else
            pair_word2<kSalt, kCross, false>(P, k, T, slj, 0u, 0u, a, dfr, far);
        else if (gap2 > kNbGuard2 && !__any_sync(0xffffffffu, (mex | m14) != 0u))
          if (small)
            pair_word2<kSalt, kSmall, false>(P, k, T, slj, 0u, 0u, a, dfr, far);
          else
            pair_word2<kSalt, kAny, false>(P, k, T, slj, 0u, 0u, a, dfr, far);
        else
          pair_word2<kSalt, kAny, true>(P, k, T, slj, mex, m14, a, dfr, far);
        // a pair whose exponentials are too far apart for their sum, or an overflow of the branch that a pair does not take
        single = same && (a.d != a.d || far >= kSmallX);
        if (!same) {
          a.s = a.d = a.m = 0.f;
          dfr = 0u;
        }
      }
      if (whole && gap2 > fmaxf(k.fcut2, kNbGuard2)) {  // every pair beyond the cutoff
        if (!__any_sync(0xffffffffu, same && live)) {
          single = false;
        } else if (!__any_sync(0xffffffffu, (mex | m14) != 0u)) {
          pair_word2<kSalt, kMm, false>(P, k, T, slj, 0u, 0u, a, dfr, far);
          if (!same) a.m = 0.f;
          single = false;
        }
      }
      if (single && live) {
        a = PairSum{0.f, 0.f, 0.f, 0.f};
        dfr = 0u;
        pair_word<kSalt>(cch == rch ? lane + 1 : 0, min(32, nC - j0), j0, nR, fused, P, k, T, slj, mex, m14, a, dfr);
      }
      if (!live) {
        a = PairSum{0.f, 0.f, 0.f, 0.f};
        dfr = 0u;
      }
      aC += (double)a.c;
      aS += (double)a.s;
      aD += (double)a.d;
      aM += (double)(a.m * (1.f / kMmScale<kSalt>));
      if (!__any_sync(0xffffffffu, dfr != 0u)) continue;
      // the word's FP64 Lennard-Jones / Coulomb pairs, listed row by row
      int at = __popc(dfr), total;
      {
        const int n = at;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, at, o);
          if (lane >= o) at += t;
        }
        total = __shfl_sync(0xffffffffu, at, 31);
        at -= n;
      }
      const unsigned all14 = m14;
      while (dfr) {
        const int b = __ffs(dfr) - 1;
        dfr &= dfr - 1;
        W.list[at++] = (unsigned short)(((all14 >> b) & 1u) << 10 | lane << 5 | b);
      }
      __syncwarp();
      for (int e = lane; e < total; e += 32) {
        const int code = W.list[e], a_ = rch * 32 + ((code >> 5) & 31), c = code & 31;
        const double2 ab = lj64[type[a_] * nt + type[j0 + c]];
        const double v = nb64(X64, a_, j0 + c, (double)X[a_].w * (double)T.q[c], ab.x, ab.y, (code >> 10) ? 2 : 1, scee, scnb);
        (a_ < nR ? eR : eL) += v;
      }
      if (lane == 0) n64 += total;
    }
    {
      const double vC = warp_sum(aC), vD = warp_sum(aD);
      double sR = 0.0, sL = 0.0, mR = 0.0, mL = 0.0;
      const unsigned rb = __ballot_sync(0xffffffffu, in_r), lv = __ballot_sync(0xffffffffu, live);
      if ((rb & lv) == lv) {
        sR = warp_sum(aS);
        mR = warp_sum(aM + eR);
      } else if (rb == 0u) {
        sL = warp_sum(aS);
        mL = warp_sum(aM + eL);
      } else {
        sR = warp_sum(in_r ? aS : 0.0);
        sL = warp_sum(in_r ? 0.0 : aS);
        mR = warp_sum((in_r ? aM : 0.0) + eR);
        mL = warp_sum((in_r ? 0.0 : aM) + eL);
      }
      const double v = lane == 0 ? vC : lane == 1 ? sR : lane == 2 ? sL : lane == 3 ? vD : lane == 4 ? mR : mL;
      if (lane < 6) part[item * 6 + lane] = v;
    }
  }
  if (lane == 0 && n64) atomicAdd((unsigned long long*)(diag + 4), (unsigned long long)n64);
}

using PairsFn = void (*)(int, int, const int4*, int, long long, const float4*, const double*, const float4*,
                         const float4*, const float*, const int*, int, const float2*, const double2*, const int*, int,
                         const unsigned*, GbConstF, double, double, double*, int*);
// [resident blocks per SM - 2][salt]; the sums do not depend on the choice
static const PairsFn kPairsFn[2][2] = {{k_pairs<false, 2>, k_pairs<true, 2>}, {k_pairs<false, 3>, k_pairs<true, 3>}};
// ---------------------------------------------------------------------------
// K3: SASA (one warp per atom), own-part then other-part neighbours
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool exact_buried(const double* X64, int i, int j, const double* sph64, int p, double er,
                                             double oer) {
  // core/src/sasa.rs:249-265 with explicit single roundings
  double t[3], d2 = 0.0;
  for (int d = 0; d < 3; d++) t[d] = __dadd_rn(X64[3 * i + d], __dmul_rn(sph64[3 * p + d], er));
  double dx = __dsub_rn(t[0], X64[3 * j]), dy = __dsub_rn(t[1], X64[3 * j + 1]), dz = __dsub_rn(t[2], X64[3 * j + 2]);
  d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  return !(d2 > __dmul_rn(oer, oer));
}

// A sphere point er s of atom i lies inside neighbour j's expanded sphere
// where g = s . 2 er v - (er^2 + |v|^2 - ro^2) > 0, v the vector to j and ro
// its expanded radius: three multiply-adds a test instead of a distance.  v is
// the difference of the FP64 coordinates, rounded once, so |g| errs by less
// than a tenth of the band (kSasaBand); points whose largest g falls inside the
// band are decided with the reference's FP64 expression, so the counts are the
// reference's.  Neighbours are ordered own part first, then the other part,
// each by the part of the sphere that it buries (the cap's cosine, in classes;
// a counting sort), so that buried points, nearly all of them, finish after a
// group or two.  A lane takes two points at a time and the neighbours go in
// groups of four, two per packed instruction; a warp leaves the loop when all
// its points are buried.  SPLIT warps share an atom's points where atoms are few
// (each orders the neighbours for itself; the counts are whole numbers).
// Bound by instruction issue and the FP32 pipe; 128 frames of 5,050 atoms, 960
// points: 3.6 ms with one distance test at a time in distance order, 2.1 here;
// 8 frames of 25,080 atoms 1.07 -> 0.62 ms.
template <int SPLIT>
__global__ void __launch_bounds__(32 * kSasaWarps)
    k_sasa(int nC, int nR, int cap, const int* __restrict__ nbr, const int* __restrict__ nbrcnt,
           const float4* __restrict__ P32, const double* __restrict__ xyz64, const double* __restrict__ rad64,
           double probe, float max_ext, int npts, const float4* __restrict__ sph32, const double* __restrict__ sph64,
           double* __restrict__ sasa, int* __restrict__ diag) {
  extern __shared__ __align__(16) unsigned char sasa_raw[];
  __shared__ int2 counts[kSasaWarps];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, pc = sasa_cap(cap);
  // per warp: 2 er v_x, v_y, v_z, |v|^2 term (each pc floats), atom, class << 16 | place, class counts
  float* wx = (float*)(sasa_raw + (size_t)w * (pc * 24 + 2 * kSasaBins * 4));
  float *wy = wx + pc, *wz = wy + pc, *wc = wz + pc;
  int *val = (int*)(wc + pc), *tag = val + pc, *hist = tag + pc;
  const int i = (blockIdx.x * (blockDim.x >> 5) + w) / SPLIT, f = blockIdx.y, share = w % SPLIT;
  const bool live = i < nC;
  const long long o = (long long)f * nC + i;
  int cs = 0, cc = 0, rechecks = 0;
  double er = 0.0;
  if (live) {
    const int cnt = min(nbrcnt[o], cap);
    const int* L = nbr + o * cap;
    const double* X64 = xyz64 + (long long)f * nC * 3;
    const double x0 = X64[3 * i], y0 = X64[3 * i + 1], z0 = X64[3 * i + 2];
    const bool in_r = i < nR;
    er = rad64[i] + probe;
    const float erf = (float)er, er2 = erf * erf, inv2er = 4.f / erf, reach = erf + max_ext;
    const float band = fmaxf(kSasaBand, kSasaBandRel * reach * reach);
    if (lane < 2 * kSasaBins) hist[lane] = 0;
    __syncwarp();
    // a neighbour's vector (of the FP64 coordinates, rounded once), constant term and class
    struct Nb {
      float x, y, z, c;
      int cls;
    };
    auto entry = [&](int j) {
      Nb n;
      const float vx = (float)(X64[3 * j] - x0), vy = (float)(X64[3 * j + 1] - y0), vz = (float)(X64[3 * j + 2] - z0);
      const float ro = P32[j].w, d2 = fmaf(vx, vx, fmaf(vy, vy, vz * vz));
      n.c = fmaf(ro, ro, -er2) - d2;
      n.x = 2.f * erf * vx;
      n.y = 2.f * erf * vy;
      n.z = 2.f * erf * vz;
      // cosine of the buried cap's edge, -c / (2 er d), in eighths; below 0: the first class
      const float t = -n.c * rsqrtf(fmaxf(d2, 1e-12f)) * inv2er;
      n.cls = min(max((int)t, 0), kSasaBins - 1) + (((j < nR) == in_r) ? 0 : kSasaBins);
      return n;
    };
    // the first 128 entries stay in registers between counting and placing
    Nb keep[4];
    int kj[4], kp[4];
#pragma unroll
    for (int h = 0; h < 4; h++) {
      const int k = 32 * h + lane;
      if (k < cnt) {
        kj[h] = L[k];
        keep[h] = entry(kj[h]);
        kp[h] = atomicAdd(&hist[keep[h].cls], 1);
      }
    }
    for (int k = 128 + lane; k < cnt; k += 32) {
      const int cls = entry(L[k]).cls;
      tag[k] = (cls << 16) | atomicAdd(&hist[cls], 1);
    }
    __syncwarp();
    int n_own = 0, n_oth = 0;
    if (lane < 2 * kSasaBins) {  // exclusive prefix sums of the class counts, per part
      const int c = hist[lane];
      int incl = c;
#pragma unroll
      for (int sh = 1; sh < kSasaBins; sh <<= 1) {
        const int t = __shfl_up_sync(0xffffu, incl, sh);
        if ((lane & (kSasaBins - 1)) >= sh) incl += t;
      }
      n_own = __shfl_sync(0xffffu, incl, kSasaBins - 1);
      n_oth = __shfl_sync(0xffffu, incl, 2 * kSasaBins - 1);
      hist[lane] = incl - c + (lane < kSasaBins ? 0 : (n_own + 3) & ~3);
    }
    n_own = __shfl_sync(0xffffffffu, n_own, 0);
    n_oth = __shfl_sync(0xffffffffu, n_oth, 0);
    const int own4 = (n_own + 3) & ~3, all4 = own4 + ((n_oth + 3) & ~3);
    __syncwarp();
    auto place = [&](int q, int j, const Nb& n) {
      val[q] = j;
      wx[q] = n.x;
      wy[q] = n.y;
      wz[q] = n.z;
      wc[q] = n.c;
    };
#pragma unroll
    for (int h = 0; h < 4; h++)
      if (32 * h + lane < cnt) place(hist[keep[h].cls] + kp[h], kj[h], keep[h]);
    for (int k = 128 + lane; k < cnt; k += 32) place(hist[tag[k] >> 16] + (tag[k] & 0xffff), L[k], entry(L[k]));
    if (lane < 8) {  // padding: never buries
      const int q = lane < 4 ? n_own + lane : own4 + n_oth + (lane - 4);
      if (q < (lane < 4 ? own4 : all4)) {
        wx[q] = wy[q] = wz[q] = 0.f;
        wc[q] = -3e38f;
        val[q] = i;
      }
    }
    __syncwarp();
    // largest g of the lane's points over the neighbours [a, b), until every point of the warp is buried
    auto scan = [&](const float4& p, const float4& q, int a, int b, float& m0, float& m1) {
      const f2 px = dup2(p.x), py = dup2(p.y), pz = dup2(p.z), qx = dup2(q.x), qy = dup2(q.y), qz = dup2(q.z);
#pragma unroll 1
      for (int k = a; k < b; k += 4) {
        const ulonglong2 x = *(const ulonglong2*)(wx + k), y = *(const ulonglong2*)(wy + k), z = *(const ulonglong2*)(wz + k),
                         c = *(const ulonglong2*)(wc + k);
        float u, v;
        un2(fma2(px, x.x, fma2(py, y.x, fma2(pz, z.x, c.x))), u, v);
        m0 = max3(m0, u, v);
        un2(fma2(qx, x.x, fma2(qy, y.x, fma2(qz, z.x, c.x))), u, v);
        m1 = max3(m1, u, v);
        un2(fma2(px, x.y, fma2(py, y.y, fma2(pz, z.y, c.y))), u, v);
        m0 = max3(m0, u, v);
        un2(fma2(qx, x.y, fma2(qy, y.y, fma2(qz, z.y, c.y))), u, v);
        m1 = max3(m1, u, v);
        if (__all_sync(0xffffffffu, fminf(m0, m1) > band)) break;
      }
    };
    // a point whose largest g lies in the band: the reference's test of the neighbours in the band
    auto decide = [&](const float4& p, int a, int b) {
      for (int k = a; k < b; k++) {
        const float g = fmaf(p.x, wx[k], fmaf(p.y, wy[k], fmaf(p.z, wz[k], wc[k])));
        if (g < -2.f * band) continue;
        rechecks++;
        const int j = val[k];
        if (exact_buried(X64, i, j, sph64, __float_as_int(p.w), er, __dadd_rn(rad64[j], probe))) return true;
      }
      return false;
    };
    auto buried = [&](const float4& p, float m, int a, int b) {
      return m > band || (m >= -band && decide(p, a, b));
    };
    // sph32 is stored patch by patch (32 points compact on the sphere per
    // patch); .w holds the point's index in the reference's order
    for (int p0 = 64 * share; p0 < npts; p0 += 64 * SPLIT) {
      const int pa = p0 + lane, pb = pa + 32;
      const bool va = pa < npts, vb = pb < npts;
      const float4 p = sph32[va ? pa : 0], q = sph32[vb ? pb : 0];
      float m0 = va ? -3e38f : 3e38f, m1 = vb ? -3e38f : 3e38f;
      scan(p, q, 0, own4, m0, m1);
      bool fa = va && !buried(p, m0, 0, n_own), fb = vb && !buried(q, m1, 0, n_own);
      cs += (int)fa + (int)fb;
      if (n_oth > 0 && __any_sync(0xffffffffu, fa || fb)) {
        m0 = fa ? -3e38f : 3e38f;
        m1 = fb ? -3e38f : 3e38f;
        scan(p, q, own4, all4, m0, m1);
        fa = fa && !buried(p, m0, own4, own4 + n_oth);
        fb = fb && !buried(q, m1, own4, own4 + n_oth);
      }
      cc += (int)fa + (int)fb;
    }
    cs = warp_sumi(cs);
    cc = warp_sumi(cc);
    rechecks = warp_sumi(rechecks);
    if (lane == 0 && rechecks) atomicAdd((unsigned long long*)(diag + 6), (unsigned long long)rechecks);
  }
  if (SPLIT > 1) {
    if (lane == 0) counts[w] = make_int2(cs, cc);
    __syncthreads();
    if (share == 0)
      for (int h = 1; h < SPLIT; h++) {
        cs += counts[w + h].x;
        cc += counts[w + h].y;
      }
  }
  if (live && lane == 0 && share == 0) {
    const double area = 4.0 * kPi * (er * er);
    sasa[2 * o] = ((double)cc / (double)npts) * area;      // in the complex
    sasa[2 * o + 1] = ((double)cs / (double)npts) * area;  // in its own part
  }
}
using SasaFn = void (*)(int, int, int, const int*, const int*, const float4*, const double*, const double*, double, float, int,
                        const float4*, const double*, double*, int*);
static const SasaFn kSasaFn[3] = {k_sasa<1>, k_sasa<2>, k_sasa<4>};

// ---------------------------------------------------------------------------
// K4: receptor x ligand non-bonded in FP64 (rows per receptor slot, columns
// per ligand slot)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int pair_class(const int* tile_rec, int nb, const unsigned* masks, int a, int b) {
  int bi = a / kTile, bj = b / kTile;
  int rec = tile_rec[bi * nb + bj];
  if (rec < 0) return 1;
  int row = a % kTile, col = b % kTile;
  const unsigned* mr = masks + ((long long)rec * 2 * kTile + row) * 4;
  if ((mr[kTile * 4 + (col >> 5)] >> (col & 31)) & 1u) return 2;
  if ((mr[col >> 5] >> (col & 31)) & 1u) return 0;
  return 1;
}

// Receptor x ligand pairs in FP64: per receptor atom the vdW, Coulomb and GB
// (complex radii) sums over the ligand, rows [nR][3], and per ligand atom the
// vdW and Coulomb sums over a group of receptor chunks, colpart [group][nL][2].
// The GB sum is the cross part of the binding GB difference, kept in FP64
// because each such pair enters it whole.  A block of eight warps takes
// `chunks` 32-atom receptor chunks; a lane is a receptor atom and the warps share
// the ligand, so a small ligand's serial loop is an eighth as long and each
// pair is evaluated once for its row and its column.  Bound by FP64 issue (two
// exponentials and two reciprocal roots a pair); 128 frames of 5,000 x 50
// atoms: 0.70 ms as a row kernel and a column kernel, 0.38 here; 8 frames of
// 25,000 x 80 atoms 0.91 -> 0.25 ms.
constexpr int kRlWarps = 8, kRlGroups = 64;
__global__ void __launch_bounds__(32 * kRlWarps)
    k_rl(int nC, int nR, int chunks, const double* __restrict__ xyz64, const double* __restrict__ q64,
         const int* __restrict__ type, int nt, const double2* __restrict__ lj64, const int* __restrict__ tile_rec, int nb,
         const unsigned* __restrict__ masks, double scee, double scnb, const double* __restrict__ R64, GbConstF k,
         double* __restrict__ rows, double* __restrict__ colpart) {
  __shared__ double acc[kRlWarps][3][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, f = blockIdx.y, nL = nC - nR;
  const double* X64 = xyz64 + (long long)f * nC * 3;
  const double* RC = R64 + (long long)f * nC * 2;
  double* cp = colpart + ((long long)f * gridDim.x + blockIdx.x) * nL * 2;
  for (int c = 0; c < chunks; c++) {
    const int a0 = (blockIdx.x * chunks + c) * 32, a = min(a0 + lane, nR - 1);
    if (a0 >= nR) break;
    const bool live = a0 + lane < nR;
    const double xa = X64[3 * a], ya = X64[3 * a + 1], za = X64[3 * a + 2], qa = q64[a], Ra = RC[2 * a];
    const int ta = type[a] * nt;
    double sv = 0.0, se = 0.0, sg = 0.0;
    for (int b = nR + w; b < nC; b += kRlWarps) {
      const double dx = xa - X64[3 * b], dy = ya - X64[3 * b + 1], dz = za - X64[3 * b + 2];
      const double r2 = dx * dx + dy * dy + dz * dz, qq = qa * q64[b];
      double v = 0.0, e = 0.0;
      const int cls = pair_class(tile_rec, nb, masks, a, b);
      if (live && cls && !(r2 < 1e-20)) {  // decomposition.rs:247-249: r < 1e-10 is skipped
        const double ri = rsqrt(r2), i2 = ri * ri, i6 = i2 * i2 * i2;
        const double2 ab = lj64[ta + type[b]];
        v = (ab.x * i6 - ab.y) * i6;
        e = qq * ri;
        if (cls == 2) {
          v /= scnb;
          e /= scee;
        }
      }
      sv += v;
      se += e;
      if (live && !(r2 > k.cut2)) {  // GB pair energy, gb_energy.rs:339-353
        const double RR = Ra * RC[2 * b], f2v = r2 + RR * exp(-r2 / (4.0 * RR)), fi = rsqrt(f2v);
        const double fv = ordinary(f2v) ? f2v * fi : f2v;  // 0 and infinity stay what they are
        sg += k.no_salt ? k.diel_ns * qq * fi
                        : -0.5 * qq * (k.inv_ein - exp(-kKScale * k.kappa * fv) * k.inv_eout) * fi;
      }
      v = warp_sum(v);
      e = warp_sum(e);
      if (lane == 0) {
        double* o = cp + 2 * (b - nR);
        o[0] = c ? o[0] + v : v;
        o[1] = c ? o[1] + e : e;
      }
    }
    acc[w][0][lane] = sv;
    acc[w][1][lane] = se;
    acc[w][2][lane] = sg;
    __syncthreads();
    if (threadIdx.x < 96) {
      const int q = threadIdx.x >> 5;
      double t = 0.0;
#pragma unroll
      for (int h = 0; h < kRlWarps; h++) t += acc[h][q][lane];
      if (live) rows[3 * ((long long)f * nR + a) + q] = t;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// K6: bonded terms by part (mm_energy.rs:187-212) and 1-4 class corrections
// term record: kind (0 bond, 1 angle, 2 dihedral, 3 correction), part
// (0 receptor, 1 ligand, 2 spanning), atoms a b c d; params p0 p1 p2
// ---------------------------------------------------------------------------
struct BTerm {
  int kind, part, a, b, c, d, cls, pad;
};

__device__ __forceinline__ void cross3d(const double* u, const double* v, double* o) {
  o[0] = u[1] * v[2] - u[2] * v[1];
  o[1] = u[2] * v[0] - u[0] * v[2];
  o[2] = u[0] * v[1] - u[1] * v[0];
}

__global__ void k_bonded(int nC, int nterms, const BTerm* __restrict__ terms, const double* __restrict__ par,
                         const double* __restrict__ xyz64, const double* __restrict__ q64, const int* __restrict__ type,
                         int nt, const double2* __restrict__ lj64, double scee, double scnb,
                         double* __restrict__ part) {
  __shared__ double sh[32];
  int t = blockIdx.x * blockDim.x + threadIdx.x, f = blockIdx.y;
  const double* x = xyz64 + (long long)f * nC * 3;
  double e[5] = {0, 0, 0, 0, 0};  // part R, part L, spanning, corr R, corr L
  if (t < nterms) {
    BTerm T = terms[t];
    const double* P = par + 3 * t;
    double v = 0.0;
    if (T.kind == 0) {
      double dx = x[3 * T.a] - x[3 * T.b], dy = x[3 * T.a + 1] - x[3 * T.b + 1], dz = x[3 * T.a + 2] - x[3 * T.b + 2];
      double r = sqrt(dx * dx + dy * dy + dz * dz);
      v = P[0] * (r - P[1]) * (r - P[1]);
    } else if (T.kind == 1) {
      double ba[3], bc[3];
      for (int d = 0; d < 3; d++) {
        ba[d] = x[3 * T.a + d] - x[3 * T.b + d];
        bc[d] = x[3 * T.c + d] - x[3 * T.b + d];
      }
      double dot = ba[0] * bc[0] + ba[1] * bc[1] + ba[2] * bc[2];
      double m1 = sqrt(ba[0] * ba[0] + ba[1] * ba[1] + ba[2] * ba[2]), m2 = sqrt(bc[0] * bc[0] + bc[1] * bc[1] + bc[2] * bc[2]);
      double th = acos(fmin(1.0, fmax(-1.0, dot / (m1 * m2))));
      v = P[0] * (th - P[1]) * (th - P[1]);
    } else if (T.kind == 2) {
      double b1[3], b2[3], b3[3], n1[3], n2[3], m1[3], u[3] = {0, 0, 0};
      for (int d = 0; d < 3; d++) {
        b1[d] = x[3 * T.b + d] - x[3 * T.a + d];
        b2[d] = x[3 * T.c + d] - x[3 * T.b + d];
        b3[d] = x[3 * T.d + d] - x[3 * T.c + d];
      }
      cross3d(b1, b2, n1);
      cross3d(b2, b3, n2);
      double len = sqrt(b2[0] * b2[0] + b2[1] * b2[1] + b2[2] * b2[2]);
      if (!(len < 1e-20))
        for (int d = 0; d < 3; d++) u[d] = b2[d] / len;
      cross3d(n1, u, m1);
      double xx = n1[0] * n2[0] + n1[1] * n2[1] + n1[2] * n2[2], yy = m1[0] * n2[0] + m1[1] * n2[1] + m1[2] * n2[2];
      v = P[0] * (1.0 + cos(P[1] * atan2(-yy, xx) - P[2]));
    } else {
      // pair that is 1-4 in the complex but not in its part: part value minus complex value
      double2 ab = lj64[type[T.a] * nt + type[T.b]];
      double qq = q64[T.a] * q64[T.b];
      double ec = nb64(x, T.a, T.b, qq, ab.x, ab.y, 2, scee, scnb);
      double es = T.cls ? nb64(x, T.a, T.b, qq, ab.x, ab.y, 1, scee, scnb) : 0.0;
      e[3 + T.part] = es - ec;
    }
    if (T.kind < 3) e[T.part] = v;
  }
  for (int q = 0; q < 5; q++) {
    double s = block_sum(e[q], sh);
    if (threadIdx.x == 0) part[((long long)f * gridDim.x + blockIdx.x) * 5 + q] = s;
  }
}

// ---------------------------------------------------------------------------
// K5: per-frame reduction -> FrameEnergy and per-residue terms
// ---------------------------------------------------------------------------
// One block per frame; every sum goes over the threads, the lanes of a warp
// and the warps in a fixed order, with one barrier for all of them (a barrier
// pair per sum, 256 threads and two divisions an atom took 215 us a frame of
// 25,080 atoms, this 95).
__global__ void __launch_bounds__(1024)
    k_reduce(int nC, int nR, int nb1, int nitems, int nbp, int ngrp, const double* __restrict__ k1part,
             const double* __restrict__ k2part, const double* __restrict__ sasa, const double* __restrict__ rows,
             const double* __restrict__ colpart, double* __restrict__ cols, const double* __restrict__ bpart,
             const double* __restrict__ wdec, double gamma, double beta, int nres, const int* __restrict__ res_ptr,
             const int* __restrict__ res_slots, rstg_frame_energy* __restrict__ out,
             rstg_residue_energy* __restrict__ decomp) {
  __shared__ double sh[22][32];
  __shared__ double tot[22];
  const int f = blockIdx.x, nL = nC - nR, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  auto put = [&](int q, double v) {
    v = warp_sum(v);
    if (lane == 0) sh[q][warp] = v;
  };
  {
    double v[5] = {0, 0, 0, 0, 0};
    for (int b = threadIdx.x; b < nb1; b += blockDim.x)
#pragma unroll
      for (int q = 0; q < 5; q++) v[q] += k1part[((long long)f * nb1 + b) * 5 + q];
#pragma unroll
    for (int q = 0; q < 5; q++) put(q < 4 ? q : 14, v[q]);
  }
  {
    double v[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 2
    for (int t = threadIdx.x; t < nitems; t += blockDim.x)
#pragma unroll
      for (int q = 0; q < 6; q++) v[q] += k2part[((long long)f * nitems + t) * 6 + q];
#pragma unroll
    for (int q = 0; q < 6; q++) put(4 + q, v[q]);
  }
  {
    double vc = 0.0, vr = 0.0, vl = 0.0, vd = 0.0;
    const double2* S = (const double2*)sasa + (long long)f * nC;
#pragma unroll 4
    for (int s = threadIdx.x; s < nC; s += blockDim.x) {
      const double2 t = S[s];
      vc += t.x;
      if (s < nR)
        vr += t.y;
      else
        vl += t.y;
      vd += t.x - t.y;
    }
    put(10, vc);
    put(11, vr);
    put(12, vl);
    put(13, vd);
  }
  {
    double ve = 0.0, vg = 0.0;
    const double* r = rows + (long long)f * nR * 3;
#pragma unroll 4
    for (int a = threadIdx.x; a < nR; a += blockDim.x) {
      ve += r[3 * a] + r[3 * a + 1];
      vg += r[3 * a + 2];
    }
    put(15, ve);
    put(21, vg);
  }
  {
    double v[5] = {0, 0, 0, 0, 0};
    for (int b = threadIdx.x; b < nbp; b += blockDim.x)
#pragma unroll
      for (int q = 0; q < 5; q++) v[q] += bpart[((long long)f * nbp + b) * 5 + q];
#pragma unroll
    for (int q = 0; q < 5; q++) put(16 + q, v[q]);
  }
  if (decomp)  // column sums of the ligand atoms over the receptor groups
    for (int c = warp; c < 2 * nL; c += nw) {
      double v = 0.0;
      for (int g = lane; g < ngrp; g += 32) v += colpart[((long long)f * ngrp + g) * nL * 2 + c];
      v = warp_sum(v);
      if (lane == 0) cols[(long long)f * nL * 2 + c] = v;
    }
  __syncthreads();
  if (threadIdx.x < 22) {
    double t = 0.0;
    for (int w = 0; w < nw; w++) t += sh[threadIdx.x][w];
    tot[threadIdx.x] = t;
  }
  __syncthreads();
  double selfC = tot[0], selfR = tot[1], selfL = tot[2], dself = tot[3];
  // pair sums count each unordered pair once; the reference adds 2 x pair (gb_energy.rs:348)
  double gbC = 2.0 * tot[4], gbR = 2.0 * tot[5], gbL = 2.0 * tot[6], dgb = 2.0 * (tot[7] + tot[21]), mmR = tot[8],
         mmL = tot[9];
  double SC = tot[10], SR = tot[11], SL = tot[12], dS = tot[13], tw = tot[14], eRL = tot[15];
  double bR = tot[16], bL = tot[17], bX = tot[18], cR = tot[19], cL = tot[20];
  double d_polar = dself + dgb;
  if (threadIdx.x == 0) {
    rstg_frame_energy e;
    e.receptor.mm = mmR + bR + cR;
    e.ligand.mm = mmL + bL + cL;
    e.complex.mm = mmR + mmL + eRL + bR + bL + bX;
    e.delta_mm = eRL + bX - cR - cL;
    e.complex.polar = selfC + gbC;
    e.receptor.polar = selfR + gbR;
    e.ligand.polar = selfL + gbL;
    e.delta_polar = d_polar;
    e.complex.sa = gamma * SC + beta;
    e.receptor.sa = gamma * SR + beta;
    e.ligand.sa = gamma * SL + beta;
    e.delta_sa = gamma * dS - beta;
    e.delta_total = e.delta_mm + e.delta_polar + e.delta_sa;
    out[f] = e;
  }
  if (!decomp) return;
  for (int r = threadIdx.x; r < nres; r += blockDim.x) {
    rstg_residue_energy x{0.0, 0.0, 0.0, 0.0};
    double w = 0.0;
    for (int k = res_ptr[r]; k < res_ptr[r + 1]; k++) {
      int s = res_slots[k];
      const double* rc = s < nR ? rows + ((long long)f * nR + s) * 3 : cols + ((long long)f * nL + (s - nR)) * 2;
      x.vdw += 0.5 * rc[0];
      x.elec += 0.5 * rc[1];
      w += wdec[(long long)f * nC + s];
      const double* S = sasa + ((long long)f * nC + s) * 2;
      x.sa += gamma * (S[0] - S[1]);
    }
    x.polar = tw > 1e-20 ? d_polar * (w / tw) : 0.0;
    decomp[(long long)f * nres + r] = x;
  }
}

// ===========================================================================
// host side
// ===========================================================================
// Order sphere points into patches of 32 that are compact on the sphere
// (recursive bisection along the axis of largest spread), so one warp's 32
// points are all buried or all exposed more often than not.
static void bisect(const std::vector<double>& sp, std::vector<int>& idx, size_t a, size_t b, std::vector<int>& out) {
  size_t n = b - a;
  if (n <= 32) {
    out.insert(out.end(), idx.begin() + a, idx.begin() + b);
    return;
  }
  double lo[3] = {1e9, 1e9, 1e9}, hi[3] = {-1e9, -1e9, -1e9};
  for (size_t k = a; k < b; k++)
    for (int d = 0; d < 3; d++) {
      lo[d] = std::min(lo[d], sp[3 * idx[k] + d]);
      hi[d] = std::max(hi[d], sp[3 * idx[k] + d]);
    }
  int ax = 0;
  for (int d = 1; d < 3; d++)
    if (hi[d] - lo[d] > hi[ax] - lo[ax]) ax = d;
  std::sort(idx.begin() + a, idx.begin() + b, [&](int u, int v) { return sp[3 * u + ax] < sp[3 * v + ax]; });
  size_t groups = (n + 31) / 32, left = (groups / 2) * 32;
  bisect(sp, idx, a, a + left, out);
  bisect(sp, idx, a + left, b, out);
}

static std::vector<int> sphere_patches(const std::vector<double>& sp, int n) {
  std::vector<int> idx(n), out;
  for (int k = 0; k < n; k++) idx[k] = k;
  bisect(sp, idx, 0, n, out);
  return out;
}

static uint64_t morton3(uint32_t x, uint32_t y, uint32_t z) {
  auto spread = [](uint64_t v) {
    v &= 0x1fffff;
    v = (v | v << 32) & 0x1f00000000ffffull;
    v = (v | v << 16) & 0x1f0000ff0000ffull;
    v = (v | v << 8) & 0x100f00f00f00f00full;
    v = (v | v << 4) & 0x10c30c30c30c30c3ull;
    v = (v | v << 2) & 0x1249249249249249ull;
    return v;
  };
  return spread(x) | spread(y) << 1 | spread(z) << 2;
}

System::System(Ctx* c, const Topology& t, const std::vector<int64_t>& rres, const std::vector<int64_t>& lres,
               const rstg_solvation& s, const rstg_sa_params& sp, const rstg_system_opts& o)
    : ctx(c), solv(s), sa(sp), opts(o), split(Split::make(t, rres, lres)) {
  n_top = t.n_atoms;
  nC = split.complex.n_atoms;
  nR = split.rec_atoms.size();
  nL = split.lig_atoms.size();
  n_res_rec = split.rec_res.size();
  n_res_lig = split.lig_res.size();
  if (sa.n_sphere_points < 1) throw Error(RSTG_ERR_INVALID, "n_sphere_points must be >= 1");
  bool fused = opts.mode == RSTG_MODE_FUSED && (solv.method == 0 || solv.method == 1);
  if (solv.method == 1) rstg_gb_params_default(&solv.gb);  // GB kernels run with defaults; PB gives the polar terms
  if (fused) {  // the fused engine's slots hold every atom of the complex once, in its part
    std::vector<uint8_t> seen(nC, 0);
    fused = nR + nL == nC;
    for (const auto* part : {&split.rec_atoms, &split.lig_atoms})
      for (int64_t a : *part) {
        fused = fused && !seen[a];  // parts that share atoms, or a residue listed twice: evaluate the parts independently
        seen[a] = 1;
      }
  }
  if (!fused) {
    opts.mode = RSTG_MODE_PLAIN;
    plain = std::make_unique<PlainFrameEval>(c, t, rres, lres, solv, sa);
  }
  batch = opts.max_batch_frames > 0 ? opts.max_batch_frames : 0;
}

System::~System() {
  if (graph) cudaGraphExecDestroy(graph);
  if (side_) cudaStreamDestroy(side_);
  if (fork_ev_) cudaEventDestroy(fork_ev_);
  if (join_ev_) cudaEventDestroy(join_ev_);
}

// k_rl: 32-atom receptor chunks per block, at most kRlGroups blocks a frame
static int rl_chunks(int64_t nR) { return (int)std::max<int64_t>((nR + 32 * kRlGroups - 1) / (32 * kRlGroups), 1); }
static int rl_groups(int64_t nR) {
  return (int)std::max<int64_t>((nR + 32 * rl_chunks(nR) - 1) / (32 * rl_chunks(nR)), 1);
}

// Grid points of the three PB grids of one frame, estimated from the atom
// counts (a sphere at 0.05 atoms/A^3 plus the grid buffer) until a frame
// has been seen.
int64_t System::pb_points_estimate() const {
  int64_t pts = 0;
  for (int64_t n : {nC, nR, nL}) {
    if (n == 0) continue;
    double side = 2.0 * std::cbrt(3.0 * (double)n / (4.0 * kPi * 0.05)) + 2.0 * solv.pb.grid_buffer;
    double m = side / solv.pb.grid_spacing + 2.0;
    pts += (int64_t)(m * m * m);
  }
  return pts;
}

int64_t System::footprint(int64_t F) const {
  if (opts.mode == RSTG_MODE_PLAIN) return nC * 200 + F * 0;
  int64_t pb = 0;
  if (solv.method == 1) {  // PB pools: ~95 B per solvated and ~45 B per reference grid point
    int64_t fpb = pb_frames_per_batch > 0 ? std::min(F, pb_frames_per_batch) : std::min<int64_t>(F, 16);
    pb = fpb * pb_points_estimate() * 140;
  }
  int64_t per = n_top * 24 + nC * (24 + 16 + 16 + 4 + 8 + 8 + 4 + (int64_t)nbr_cap * 4 + 16 + 8) + nR * 24 + nL * 16 * (1 + (int64_t)rl_groups(nR)) +
                (n_res_rec + n_res_lig) * 32 + 256;
  int64_t nb = (nC + kTile - 1) / kTile;
  per += nb * (nb + 1) / 2 * 48 + nb * 192;
  return per * F + nC * 128 + pb;
}

void System::prepare_fused(const double* x0) {
  cudaStream_t st = stream();
  const Topology& C = split.complex;
  // slot order: receptor atoms then ligand atoms, each along a Morton curve
  double mn[3] = {1e300, 1e300, 1e300};
  for (int64_t a = 0; a < nC; a++)
    for (int d = 0; d < 3; d++) mn[d] = std::min(mn[d], x0[3 * a + d]);
  auto code = [&](int64_t a) {
    uint32_t q[3];
    for (int d = 0; d < 3; d++) {
      double v = (x0[3 * a + d] - mn[d]) / 2.0;
      q[d] = (uint32_t)std::min(std::max(v, 0.0), 2097151.0);
    }
    return morton3(q[0], q[1], q[2]);
  };
  slot_atom.clear();
  for (int part = 0; part < 2; part++) {
    std::vector<int64_t> at = part ? split.lig_atoms : split.rec_atoms;
    std::vector<std::pair<uint64_t, int64_t>> keyed;
    for (int64_t a : at) keyed.push_back({code(a), a});
    std::stable_sort(keyed.begin(), keyed.end(),
                     [](const std::pair<uint64_t, int64_t>& u, const std::pair<uint64_t, int64_t>& v) { return u.first < v.first; });
    for (auto& k : keyed) slot_atom.push_back(k.second);
  }
  std::vector<int32_t> inv(nC, -1);
  for (int64_t s = 0; s < nC; s++) inv[slot_atom[s]] = (int32_t)s;
  slot_src.resize(nC);
  for (int64_t s = 0; s < nC; s++)
    slot_src[s] = (int32_t)(split.complex_atoms.empty() ? slot_atom[s] : split.complex_atoms[slot_atom[s]]);

  fp = std::make_unique<FusedParams>();
  FusedParams& F = *fp;
  auto up = [&](DevBuf& b, const void* src, size_t bytes) {
    b = DevBuf(bytes ? bytes : 16, st);
    if (bytes) RSTG_CUDA(cudaMemcpyAsync(b.p, src, bytes, cudaMemcpyHostToDevice, st));
  };
  const rstg_gb_params& g = solv.gb;
  std::vector<float4> P(nC);
  std::vector<double> q(nC), rho(nC), rad(nC), sj(nC);
  std::vector<int32_t> ty(nC);
  for (int64_t s = 0; s < nC; s++) {
    int64_t a = slot_atom[s];
    q[s] = C.charges_amber[a];
    rad[s] = C.radii[a];
    rho[s] = C.radii[a] - g.offset;
    sj[s] = C.screen[a] * rho[s];
    ty[s] = C.n_types > 0 ? (int32_t)C.type_idx[a] : 0;  // (without types the tables hold one zero)
    P[s] = make_float4((float)q[s], (float)rho[s], (float)sj[s], (float)(C.radii[a] + sa.probe_radius));
  }
  up(F.slot_src, slot_src.data(), nC * 4);
  up(F.P32, P.data(), nC * sizeof(float4));
  up(F.q64, q.data(), nC * 8);
  up(F.rho64, rho.data(), nC * 8);
  up(F.rad64, rad.data(), nC * 8);
  up(F.sj64, sj.data(), nC * 8);
  up(F.type, ty.data(), nC * 4);
  int nt = (int)std::max<int64_t>(C.n_types, 1);
  F.nt = nt;
  std::vector<float2> l32(nt * nt, make_float2(0, 0));
  std::vector<double2> l64(nt * nt, make_double2(0, 0));
  for (int a = 0; a < C.n_types; a++)
    for (int b = 0; b < C.n_types; b++) {
      int64_t idx = C.nb_index[C.n_types * a + b];
      if (idx >= 1) {
        l64[a * nt + b] = make_double2(C.lj_a[idx - 1], C.lj_b[idx - 1]);
        l32[b * nt + a] = make_float2((float)C.lj_a[idx - 1], (float)C.lj_b[idx - 1]);  // column type major
      }
    }
  up(F.lj32, l32.data(), l32.size() * sizeof(float2));
  up(F.lj64, l64.data(), l64.size() * sizeof(double2));
  // tiles and exclusion / 1-4 masks in slot space
  int nb = (int)((nC + kTile - 1) / kTile);
  F.nb = nb;
  PairClasses pc = PairClasses::build(C);
  std::vector<int> trec(nb * nb, -1);
  std::vector<unsigned> masks;
  auto mark = [&](uint64_t key, int which) {
    int64_t a = (int64_t)(key >> 32), b = (int64_t)(key & 0xffffffffu);
    int sa_ = inv[a], sb = inv[b];
    if (sa_ > sb) std::swap(sa_, sb);
    int bi = sa_ / kTile, bj = sb / kTile;
    int& r = trec[bi * nb + bj];
    if (r < 0) {
      r = (int)(masks.size() / (2 * kTile * 4));
      masks.resize(masks.size() + 2 * kTile * 4, 0u);
    }
    int row = sa_ % kTile, col = sb % kTile;
    masks[((size_t)r * 2 * kTile + (which ? kTile : 0) + row) * 4 + (col >> 5)] |= 1u << (col & 31);
  };
  for (auto k : pc.excl_keys) mark(k, 0);
  for (auto k : pc.p14_keys) mark(k, 1);
  // work items of k_pairs: 32 rows and up to `span` 32-column words; a span
  // of an eighth of the slots gives a single small frame hundreds of items, and
  // 64 words are enough to make the item's own cost small
  std::vector<int4> items;
  const int nchunk = (int)((nC + 31) / 32), span = std::min(std::max(nchunk / 8, 1), 64);
  for (int r = 0; r < nchunk; r++)
    for (int c = r; c < nchunk; c += span) items.push_back(make_int4(r, c, std::min(c + span, nchunk), 0));
  F.nitems = (int)items.size();
  up(F.items, items.data(), items.size() * sizeof(int4));
  size_t ljsm = (size_t)nt * nt * sizeof(float2);
  if (ljsm > 160 * 1024) throw Error(RSTG_ERR_INVALID, "too many Lennard-Jones types for the fused kernels");
  // the limits are the function's, not the system's: every system sets the same
  RSTG_CUDA(cudaFuncSetAttribute(k_psi, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PsiSmem)));
  for (auto& v : kPairsFn)
    for (PairsFn fn : v)
      RSTG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     160 * 1024 + kPairWarps * (int)sizeof(PairWarp)));
  up(F.tile_rec, trec.data(), trec.size() * 4);
  up(F.masks, masks.data(), masks.size() * 4);
  // sphere points (host libm, as the reference)
  auto sp64 = fibonacci_sphere(sa.n_sphere_points);
  F.npts = (int)sa.n_sphere_points;
  std::vector<int> order = sphere_patches(sp64, F.npts);
  std::vector<float4> sp32(F.npts);
  for (int k = 0; k < F.npts; k++) {
    int p = order[k];
    float idx_bits;
    memcpy(&idx_bits, &p, 4);
    sp32[k] = make_float4((float)sp64[3 * p], (float)sp64[3 * p + 1], (float)sp64[3 * p + 2], idx_bits);
  }
  up(F.sphere32, sp32.data(), sp32.size() * sizeof(float4));
  up(F.sphere64, sp64.data(), sp64.size() * 8);
  F.probe = sa.probe_radius;
  // residues: receptor residues then ligand residues, as listed
  std::vector<int32_t> rp{0}, rs;
  for (int part = 0; part < 2; part++)
    for (int64_t r : (part ? split.lig_res : split.rec_res)) {
      std::vector<int32_t> ss;
      for (int64_t a : C.select({r})) ss.push_back(inv[a]);
      std::sort(ss.begin(), ss.end());
      rs.insert(rs.end(), ss.begin(), ss.end());
      rp.push_back((int32_t)rs.size());
    }
  F.nres = (int)(rp.size() - 1);
  up(F.res_ptr, rp.data(), rp.size() * 4);
  up(F.res_slots, rs.data(), rs.size() * 4);
  // bonded terms by part, and 1-4 class corrections
  std::vector<BTerm> terms;
  std::vector<double> par;
  auto part_of = [&](std::initializer_list<int64_t> atoms) {
    bool allR = true, allL = true;
    for (int64_t a : atoms) {
      int s = inv[a];
      allR &= s < nR;
      allL &= s >= nR;
    }
    return allR ? 0 : (allL ? 1 : 2);
  };
  for (size_t b = 0; b < C.bond_i.size(); b++) {
    terms.push_back({0, part_of({C.bond_i[b], C.bond_j[b]}), inv[C.bond_i[b]], inv[C.bond_j[b]], 0, 0, 0, 0});
    par.insert(par.end(), {C.bond_k[C.bond_t[b]], C.bond_req[C.bond_t[b]], 0.0});
  }
  for (size_t a = 0; a < C.ang_i.size(); a++) {
    terms.push_back({1, part_of({C.ang_i[a], C.ang_j[a], C.ang_k[a]}), inv[C.ang_i[a]], inv[C.ang_j[a]],
                     inv[C.ang_k[a]], 0, 0, 0});
    par.insert(par.end(), {C.angle_k[C.ang_t[a]], C.angle_teq[C.ang_t[a]], 0.0});
  }
  for (size_t d = 0; d < C.dih_i.size(); d++) {
    terms.push_back({2, part_of({C.dih_i[d], C.dih_j[d], C.dih_k[d], C.dih_l[d]}), inv[C.dih_i[d]], inv[C.dih_j[d]],
                     inv[C.dih_k[d]], inv[C.dih_l[d]], 0, 0});
    par.insert(par.end(), {C.dih_pk[C.dih_t[d]], C.dih_pn[C.dih_t[d]], C.dih_phase[C.dih_t[d]]});
  }
  // pairs that are 1-4 in the complex through a dihedral spanning the parts
  // but not 1-4 in the part's own topology
  for (int part = 0; part < 2; part++) {
    const Topology& sub = part ? split.lig : split.rec;
    const std::vector<int64_t>& at = part ? split.lig_atoms : split.rec_atoms;
    PairClasses spc = PairClasses::build(sub);
    std::vector<int64_t> loc(nC, -1);
    for (size_t k = 0; k < at.size(); k++) loc[at[k]] = (int64_t)k;
    for (auto key : pc.p14_keys) {
      int64_t a = (int64_t)(key >> 32), b = (int64_t)(key & 0xffffffffu);
      if (loc[a] < 0 || loc[b] < 0) continue;
      int cs = spc.cls(loc[a], loc[b]);
      if (cs == 2) continue;
      terms.push_back({3, part, inv[a], inv[b], 0, 0, cs, 0});
      par.insert(par.end(), {0.0, 0.0, 0.0});
    }
  }
  F.nterms = (int)terms.size();
  up(F.bterms, terms.data(), terms.size() * sizeof(BTerm));
  up(F.bpar, par.data(), par.size() * 8);
  // GB constants
  GbConstF& k = F.gb;
  double s_ = g.salt_concentration;
  k.kappa = s_ <= 0.0 ? 0.0 : std::sqrt(8.0 * kPi * 332.0522 * 6.022e-4 * s_ / (g.solvent_dielectric * 0.00198688 * g.temperature));
  k.inv_ein = 1.0 / g.solute_dielectric;
  k.inv_eout = 1.0 / g.solvent_dielectric;
  k.diel_ns = -0.5 * (k.inv_ein - k.inv_eout);
  k.f0 = -0.5 * (1.0 / g.solute_dielectric - 1.0 / g.solvent_dielectric);
  k.no_salt = k.kappa <= 0.0;
  k.cut2 = g.cutoff * g.cutoff;
  k.fk = (float)(kKScale * k.kappa);
  k.fkl = (float)(-kKScale * k.kappa * 1.4426950408889634);
  k.fie = (float)k.inv_ein;
  k.fio = (float)k.inv_eout;
  k.fdns = (float)k.diel_ns;
  k.fcut2 = (float)std::min(k.cut2, 3.0e38);
  {
    // the largest SASA reach and HCT far-field bound over all atoms, with a
    // margin for the FP32 rounding of the box distance and of r^2
    double ext = 0.0, sm = 0.0, rm = 0.0;
    for (int64_t a = 0; a < nC; a++) {
      ext = std::max(ext, (double)P[a].w);
      sm = std::max(sm, std::fabs((double)P[a].z));
      rm = std::max(rm, std::fabs((double)P[a].y));
    }
    F.max_ext = (float)ext;
    const double far2 = std::max({4.0 * ext * ext * 1.00001 + 1e-4, 16.0 * sm * sm, (rm + sm) * (rm + sm)});
    k.tile_far2 = (float)(far2 * 1.001 + 0.01);
  }
  k.model = g.model;
  k.rgbmax = g.rgbmax;
  k.fdev = 0.52f * k.fk * (float)std::min(std::fabs(g.rgbmax), 1e30);
  // neighbour capacity from the first frame (x1.5 + 32 margin; re-sized on overflow)
  {
    double cell = 0.0;
    for (int64_t a = 0; a < nC; a++) cell = std::max(cell, C.radii[a] + sa.probe_radius);
    cell = std::max(2.0 * cell, 1e-3);
    // atoms sorted by cell along x-major order; per row of cells the atoms of
    // three neighbouring cells are one range
    std::vector<std::pair<uint64_t, int64_t>> cells(nC);
    auto cid = [&](int64_t a, int d) { return (int64_t)std::floor((x0[3 * a + d] - mn[d]) / cell); };
    auto code3 = [](int64_t cx, int64_t cy, int64_t cz) {
      return ((uint64_t)(cz + 1) << 42) | ((uint64_t)(cy + 1) << 21) | (uint64_t)(cx + 1);
    };
    for (int64_t a = 0; a < nC; a++) cells[a] = {code3(cid(a, 0), cid(a, 1), cid(a, 2)), a};
    std::sort(cells.begin(), cells.end());
    std::vector<double> sx(nC * 4);
    for (int64_t k = 0; k < nC; k++) {
      const int64_t a = cells[k].second;
      for (int d = 0; d < 3; d++) sx[4 * k + d] = x0[3 * a + d];
      sx[4 * k + 3] = C.radii[a] + sa.probe_radius;
    }
    auto first = [&](uint64_t c) {
      return (int64_t)(std::lower_bound(cells.begin(), cells.end(), std::make_pair(c, (int64_t)-1)) - cells.begin());
    };
    int64_t mx = 0;
    for (int64_t k = 0; k < nC;) {
      int64_t e = k;
      while (e < nC && cells[e].first == cells[k].first) e++;
      const int64_t a0 = cells[k].second;
      int64_t lo[9], hi[9];
      for (int q = 0; q < 9; q++) {
        const int64_t cy = cid(a0, 1) + q % 3 - 1, cz = cid(a0, 2) + q / 3 - 1;
        lo[q] = first(code3(cid(a0, 0) - 1, cy, cz));
        hi[q] = first(code3(cid(a0, 0) + 2, cy, cz));
      }
      for (int64_t i = k; i < e; i++) {
        int64_t cnt = -1;  // the atom itself
        for (int q = 0; q < 9; q++)
          for (int64_t b = lo[q]; b < hi[q]; b++) {
            const double r = sx[4 * i + 3] + sx[4 * b + 3], dx = sx[4 * i] - sx[4 * b], dy = sx[4 * i + 1] - sx[4 * b + 1],
                         dz = sx[4 * i + 2] - sx[4 * b + 2];
            cnt += dx * dx + dy * dy + dz * dz <= r * r;
          }
        mx = std::max(mx, cnt);
      }
      k = e;
    }
    nbr_cap = (int)std::max<int64_t>(64, ((mx * 3 / 2 + 32) + 31) / 32 * 32);
  }
  if (batch <= 0) {
    // frames per batch: enough CTAs for every SM several times over, within
    // a device-memory share of about 2 GB for the batch buffers
    int64_t per = footprint(1);
    batch = std::max<int64_t>(1, std::min<int64_t>(256, (int64_t)(2.0e9 / std::max<int64_t>(per, 1))));
  }
  perm_ready = true;
}

// row blocks of k_psi per frame
static int psi_blocks(int64_t nC) { return (int)((nC + kPsiRows - 1) / kPsiRows); }

void System::ensure_buffers(int64_t frames) {
  if (frames <= buf_frames) return;
  if (graph) {  // a captured graph holds the old buffers' addresses and capacities
    cudaGraphExecDestroy(graph);
    graph = nullptr;
  }
  cudaStream_t st = stream();
  int64_t B = frames;
  int nb1 = psi_blocks(nC);
  int nbp = std::max(1, (fp->nterms + 255) / 256);
  in_frames = DevBuf(B * n_top * 3 * 8, st);  // room for float64 input
  xyz64 = DevBuf(B * nC * 24, st);
  xyz32 = DevBuf(B * nC * 16, st);
  boxes = DevBuf(B * ((nC + 31) / 32) * 32, st);
  R64 = DevBuf(B * nC * 16, st);
  Rf = DevBuf(B * nC * 16, st);
  dRf = DevBuf(B * nC * 4, st);
  nbr = DevBuf(B * nC * (int64_t)nbr_cap * 4, st);
  nbrcnt = DevBuf(B * nC * 4, st);
  sasa = DevBuf(B * nC * 16, st);
  k1part = DevBuf(B * nb1 * 5 * 8, st);
  wdec = DevBuf(B * nC * 8, st);
  colpart = DevBuf(B * (int64_t)rl_groups(nR) * std::max<int64_t>(nL, 1) * 16, st);
  k2part = DevBuf(B * (int64_t)fp->nitems * 6 * 8, st);
  rows = DevBuf(B * std::max<int64_t>(nR, 1) * 24, st);
  cols = DevBuf(B * std::max<int64_t>(nL, 1) * 16, st);
  bpart = DevBuf(B * nbp * 5 * 8, st);
  res_buf = DevBuf(B * sizeof(rstg_frame_energy), st);
  dec_buf = DevBuf(B * std::max<int64_t>(fp->nres, 1) * sizeof(rstg_residue_energy), st);
  diag = DevBuf(64, st);
  RSTG_CUDA(cudaMemsetAsync(diag.p, 0, 64, st));
  // (the neighbours of two atoms in 200 KB of shared memory bound the capacity)
  if ((size_t)2 * (nbr_cap * 24 + 64) > 200 * 1024) throw Error(RSTG_ERR_INVALID, "SASA neighbour capacity exceeds shared memory");
  sasa_warps = kSasaWarps;
  while (sasa_warps > 1 && sasa_smem(nbr_cap, sasa_warps) > 200 * 1024) sasa_warps /= 2;
  for (SasaFn fn : kSasaFn)
    RSTG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  buf_frames = B;
  if (graph) {
    cudaGraphExecDestroy(graph);
    graph = nullptr;
  }
}

void System::launch_pairs(int64_t F) {
  FusedParams& P = *fp;
  const size_t smem = kPairWarps * sizeof(PairWarp) + (size_t)P.nt * P.nt * sizeof(float2);
  const long long items = (long long)P.nitems * F, sms = ctx->prop.multiProcessorCount;
  // Two blocks per SM keep every value in registers; three spill a little but
  // finish few items sooner.  Where the items are at least eight per warp of
  // the former, it wins (128 frames of 5,050 atoms 4.7 against 5.1 ms; 37 of
  // 1,187 atoms, three items per warp: 150 against 139 us).
  const int three = items < 8 * 2 * kPairWarps * sms;
  const PairsFn fn = kPairsFn[three][P.gb.no_salt ? 0 : 1];
  // persistent grid: the resident blocks of the shape, a whole number of SMs
  int& per_sm = pairs_per_sm[three];
  if (per_sm == 0) RSTG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 32 * kPairWarps, smem));
  const long long grid = std::min<long long>((items + kPairWarps - 1) / kPairWarps, std::max(per_sm, 1) * sms);
  fn<<<(unsigned)grid, 32 * kPairWarps, smem, stream()>>>(
      (int)nC, (int)nR, P.items.as<int4>(), P.nitems, items, xyz32.as<float4>(), xyz64.as<double>(), boxes.as<float4>(),
      Rf.as<float4>(), dRf.as<float>(), P.type.as<int>(), P.nt, P.lj32.as<float2>(), P.lj64.as<double2>(),
      P.tile_rec.as<int>(), P.nb, P.masks.as<unsigned>(), P.gb, split.complex.scee, split.complex.scnb,
      k2part.as<double>(), diag.as<int>());
}

// FP32 sums of k_psi over 64 columns (a tile's halves apart) or 128.  Energies
// differ by about 1e-8 between the two, and the choice is the one that systems
// have had since their launch shapes were timed on the first run: two threads a
// row, 64 columns each, at four blocks of 128 rows an SM, against one thread at
// eight.  The former won by more than 2 % where its waves counted half were
// fewer, that is where they are odd in number (up to five; later the difference
// is too small), except on fewer than 91 atoms and on 136 to 256 of which 4
// blocks an SM are resident (0.96 to 1.1 of the other's time), and in a second wave
// on 7,500 atoms and more, whose columns outlast the tail (0.94 to 0.97 from
// 5.2 blocks an SM).  Of 235 random sizes where the timed choice repeated
// itself this rule gives 227.
static bool psi_halves(int64_t nC, int64_t frames, int sms) {
  const int64_t blocks = (nC + kTile - 1) / kTile * frames, waves = (blocks + 4 * sms - 1) / (4 * sms);
  if (waves == 1) return nC > 90 && (blocks <= 3 * sms || nC <= 135 || nC > 256);
  if (waves == 2) return nC >= 7500 && 5 * blocks >= 26 * sms;
  return waves == 3 || waves == 5;
}

// The choice holds for every system of the process with the same device, atom
// counts and sphere points, so that equal inputs give equal results whatever
// the number of frames; the first run of such a system makes it, for its batch
// or the frames that hold 2,048 tile pairs.  Without autotune: 128.
void System::choose_psi(int64_t F) {
  if (psi_shares > 0) return;
  psi_shares = 1;
  if (!opts.autotune) return;
  static std::mutex mu;
  static std::map<std::array<int64_t, 4>, int> chosen;
  const int64_t nb = (nC + kTile - 1) / kTile, pairs = nb * (nb + 1) / 2;
  const int64_t frames = std::max<int64_t>(1, std::min(batch, std::max(std::min(F, batch), (2048 + pairs - 1) / pairs)));
  std::lock_guard<std::mutex> lk(mu);
  psi_shares = chosen.emplace(std::array<int64_t, 4>{ctx->device, nC, nR, fp->npts},
                              psi_halves(nC, frames, ctx->prop.multiProcessorCount) ? 2 : 1).first->second;
}

void System::launch_psi(int64_t F) {
  FusedParams& P = *fp;
  k_psi<<<dim3((unsigned)psi_blocks(nC), (unsigned)F), 32 * kPsiWarps, sizeof(PsiSmem), stream()>>>(
      (int)nC, (int)nR, xyz32.as<float4>(), xyz64.as<double>(), boxes.as<float4>(), P.P32.as<float4>(),
      P.rho64.as<double>(), P.sj64.as<double>(), P.rad64.as<double>(), P.q64.as<double>(), P.gb, psi_shares == 2, nbr_cap, nbr.as<int>(),
      nbrcnt.as<int>(), R64.as<double>(), Rf.as<float4>(), dRf.as<float>(), wdec.as<double>(),
      k1part.as<double>(), diag.as<int>());
}

void System::launch_sasa(int64_t F, cudaStream_t st) {
  FusedParams& P = *fp;
  // warps per atom: the least power of two up to four that gives every SM 16
  // warps (1 frame of 132 atoms: 59 -> 12 us with four)
  const long long atoms = (long long)nC * F, want = 16LL * ctx->prop.multiProcessorCount;
  const int lg = sasa_warps < kSasaWarps || atoms >= want ? 0 : (2 * atoms >= want ? 1 : 2), per = sasa_warps >> lg;
  kSasaFn[lg]<<<dim3((unsigned)((nC + per - 1) / per), (unsigned)F), 32 * sasa_warps,
                sasa_smem(nbr_cap, sasa_warps), st>>>(
      (int)nC, (int)nR, nbr_cap, nbr.as<int>(), nbrcnt.as<int>(), P.P32.as<float4>(), xyz64.as<double>(),
      P.rad64.as<double>(), P.probe, P.max_ext, P.npts, P.sphere32.as<float4>(), P.sphere64.as<double>(), sasa.as<double>(),
      diag.as<int>());
}

void System::tuning(int32_t* shape12, double* ms12) const {
  // every launch shape follows from the sizes: no candidates
  int32_t o[12] = {1, 2, sasa_warps, (int32_t)batch, 0, 0, 0, 0, std::max(psi_shares, 1), 3, 0, 1};
  if (shape12) memcpy(shape12, o, sizeof(o));
  if (ms12)
    for (int k = 0; k < 12; k++) ms12[k] = 0.0;
}

void System::launch_batch(const void* d_frames, bool f64, int64_t F, rstg_frame_energy* d_out,
                          rstg_residue_energy* d_decomp, Prof* prof) {
  auto mark = [&](const char* name, double flops, double bytes) {
    if (!prof) return;
    prof->names[prof->n] = name;
    prof->flops[prof->n] = flops;
    prof->bytes[prof->n] = bytes;
    prof->n++;
    RSTG_CUDA(cudaEventRecord(prof->ev[prof->n], stream()));
  };
  if (prof) {
    prof->n = 0;
    RSTG_CUDA(cudaEventRecord(prof->ev[0], stream()));
  }
  const double Fd = (double)F, nCd = (double)nC, nRd = (double)nR, nLd = (double)nL;
  // algorithmic operation counts per pair: HCT 32, GB 24 (18 without salt), LJ + Coulomb 22
  const double gbf = fp && fp->gb.no_salt ? 18.0 : 24.0;
  const double same_pairs = nRd * (nRd - 1) / 2 + nLd * (nLd - 1) / 2;
  cudaStream_t st = stream();
  FusedParams& P = *fp;
  unsigned Fu = (unsigned)F;
  int nb1 = psi_blocks(nC);
  int nbp = std::max(1, (P.nterms + 255) / 256);
  k_prep<<<dim3((unsigned)((nC + 255) / 256), Fu), 256, 0, st>>>((int)nC, (int)n_top, d_frames, f64 ? 1 : 0,
                                                                 P.slot_src.as<int>(), P.P32.as<float4>(),
                                                                 xyz64.as<double>(), xyz32.as<float4>(),
                                                                 boxes.as<float4>());
  mark("prep", 0.0, Fd * (n_top * 12.0 + nCd * 40.0));
  launch_psi(F);
  mark("psi", Fd * nCd * (nCd - 1) * 32.0, 0.0);
  int nlaunch = 4;
  // What follows needs the Born radii and neighbour lists but nothing of one
  // another: on the context's own stream the pair kernel runs beside the
  // others on a second one (a small batch fills the GPU with neither; 10
  // frames of 2,030 atoms: 429 -> 341 us with it).  A caller's stream, a server's
  // prioritised one and the profile keep to a single stream.
  const bool fork = !prof && !stream_ && ctx->own_stream;
  if (fork && !side_) {
    RSTG_CUDA(cudaStreamCreateWithFlags(&side_, cudaStreamNonBlocking));
    RSTG_CUDA(cudaEventCreateWithFlags(&fork_ev_, cudaEventDisableTiming));
    RSTG_CUDA(cudaEventCreateWithFlags(&join_ev_, cudaEventDisableTiming));
  }
  cudaStream_t sd = fork ? side_ : st;
  if (fork) {
    RSTG_CUDA(cudaEventRecord(fork_ev_, st));
    RSTG_CUDA(cudaStreamWaitEvent(sd, fork_ev_, 0));
  }
  launch_pairs(F);
  mark("pairs", Fd * (nCd * (nCd - 1) / 2 * gbf + same_pairs * (gbf + 22.0)), 0.0);
  launch_sasa(F, sd);
  mark("sasa", 0.0, 0.0);
  const int chunks = rl_chunks(nR), ngrp = rl_groups(nR);
  if (nR > 0 && nL > 0) {
    k_rl<<<dim3((unsigned)ngrp, Fu), 32 * kRlWarps, 0, sd>>>(
        (int)nC, (int)nR, chunks, xyz64.as<double>(), P.q64.as<double>(), P.type.as<int>(), P.nt, P.lj64.as<double2>(),
        P.tile_rec.as<int>(), P.nb, P.masks.as<unsigned>(), split.complex.scee, split.complex.scnb, R64.as<double>(),
        P.gb, rows.as<double>(), colpart.as<double>());
    mark("rl", Fd * nRd * nLd * 44.0, 0.0);
    nlaunch++;
  } else {
    RSTG_CUDA(cudaMemsetAsync(rows.p, 0, rows.bytes, sd));
  }
  if (P.nterms > 0) {
    k_bonded<<<dim3((unsigned)nbp, Fu), 256, 0, sd>>>((int)nC, P.nterms, P.bterms.as<BTerm>(), P.bpar.as<double>(),
                                                      xyz64.as<double>(), P.q64.as<double>(), P.type.as<int>(), P.nt,
                                                      P.lj64.as<double2>(), split.complex.scee, split.complex.scnb,
                                                      bpart.as<double>());
    mark("bonded", 0.0, 0.0);
    nlaunch++;
  } else {
    RSTG_CUDA(cudaMemsetAsync(bpart.p, 0, bpart.bytes, sd));
  }
  if (fork) {
    RSTG_CUDA(cudaEventRecord(join_ev_, sd));
    RSTG_CUDA(cudaStreamWaitEvent(st, join_ev_, 0));
  }
  k_reduce<<<Fu, nC < 512 ? 256 : 1024, 0, st>>>(
      (int)nC, (int)nR, nb1, P.nitems, nbp, nR > 0 && nL > 0 ? ngrp : 0, k1part.as<double>(), k2part.as<double>(),
      sasa.as<double>(), rows.as<double>(), colpart.as<double>(), cols.as<double>(), bpart.as<double>(),
      wdec.as<double>(), sa.surface_tension, sa.offset, P.nres, P.res_ptr.as<int>(), P.res_slots.as<int>(), d_out,
      d_decomp);
  mark("reduce", 0.0, 0.0);
  nlaunch++;
  launched(ctx, nlaunch);
  last_stats[0] += nlaunch;
}

void System::release_buffers() {
  if (graph) cudaGraphExecDestroy(graph);
  graph = nullptr;
  for (DevBuf* b : {&in_frames, &xyz64, &xyz32, &boxes, &R64, &Rf, &dRf, &nbr, &nbrcnt, &sasa, &k1part, &wdec, &k2part, &rows, &colpart, &cols, &bpart,
                    &res_buf, &dec_buf, &diag})
    *b = DevBuf();
  buf_frames = 0;
  if (pbe) pbe->release();  // the PB pools are part of the footprint a server accounts for
}

void System::profile(const float* d_frames, int64_t F, int32_t* n, char* names, double* ms, double* flops,
                     double* bytes) {
  if (opts.mode != RSTG_MODE_FUSED) throw Error(RSTG_ERR_INVALID, "profiling needs a fused-mode system");
  cudaStream_t st = stream();
  if (!perm_ready) {
    std::vector<float> fr(n_top * 3);
    RSTG_CUDA(cudaMemcpyAsync(fr.data(), d_frames, fr.size() * 4, cudaMemcpyDeviceToHost, st));
    RSTG_CUDA(cudaStreamSynchronize(st));
    std::vector<double> x0(nC * 3);
    for (int64_t a = 0; a < nC; a++) {
      int64_t t = split.complex_atoms.empty() ? a : split.complex_atoms[a];
      for (int d = 0; d < 3; d++) x0[3 * a + d] = fr[3 * t + d];
    }
    prepare_fused(x0.data());
  }
  ensure_buffers(std::min(F, batch));
  Prof pr;
  for (auto& e : pr.ev) RSTG_CUDA(cudaEventCreate(&e));
  std::vector<double> tot(8, 0.0), fl(8, 0.0), by(8, 0.0);
  int nk = 0;
  try {
    for (int64_t f0 = 0; f0 < F; f0 += batch) {
      int64_t B = std::min(batch, F - f0);
      RSTG_CUDA(cudaMemcpyAsync(in_frames.p, d_frames + (size_t)f0 * n_top * 3, (size_t)B * n_top * 12,
                                cudaMemcpyDeviceToDevice, st));
      launch_batch(in_frames.p, false, B, res_buf.as<rstg_frame_energy>(), dec_buf.as<rstg_residue_energy>(), &pr);
      RSTG_CUDA(cudaStreamSynchronize(st));
      nk = pr.n;
      for (int k = 0; k < pr.n; k++) {
        float t = 0.f;
        RSTG_CUDA(cudaEventElapsedTime(&t, pr.ev[k], pr.ev[k + 1]));
        tot[k] += t;
        fl[k] += pr.flops[k];
        by[k] += pr.bytes[k];
      }
    }
  } catch (...) {
    for (auto& e : pr.ev) cudaEventDestroy(e);
    throw;
  }
  for (auto& e : pr.ev) cudaEventDestroy(e);
  *n = nk;
  for (int k = 0; k < nk; k++) {
    if (names) {
      memset(names + 32 * k, 0, 32);
      strncpy(names + 32 * k, pr.names[k], 31);
    }
    if (ms) ms[k] = tot[k];
    if (flops) flops[k] = fl[k];
    if (bytes) bytes[k] = by[k];
  }
}

int System::graph_kernels() const { return 4 + (nR > 0 && nL > 0 ? 1 : 0) + (fp->nterms > 0 ? 1 : 0) + 1; }

void System::run_plain(const void* frames, bool f64, bool host_in, int64_t F, rstg_frame_energy* out, bool host_out,
                       rstg_residue_energy* decomp) {
  cudaStream_t st = stream();
  std::vector<char> hbuf;
  const char* src = (const char*)frames;
  size_t esz = f64 ? 8 : 4;
  if (!host_in) {
    hbuf.resize(F * n_top * 3 * esz);
    RSTG_CUDA(cudaMemcpyAsync(hbuf.data(), frames, hbuf.size(), cudaMemcpyDeviceToHost, st));
    RSTG_CUDA(cudaStreamSynchronize(st));
    src = hbuf.data();
  }
  std::vector<rstg_frame_energy> res(F);
  int64_t nres = n_res_rec + n_res_lig;
  std::vector<rstg_residue_energy> dres(decomp ? F * nres : 0);
  int64_t before = ctx->launches.load();
  plain->pb_rel_tol = pb_rel_tol;
  for (int64_t f = 0; f < F; f++) {
    std::vector<double> xc(nC * 3);
    for (int64_t a = 0; a < nC; a++) {
      int64_t t = split.complex_atoms.empty() ? a : split.complex_atoms[a];
      for (int d = 0; d < 3; d++) {
        size_t k = ((size_t)f * n_top + t) * 3 + d;
        xc[3 * a + d] = f64 ? ((const double*)src)[k] : ((double)((const float*)src)[k] * 0.1) * 10.0;
      }
    }
    res[f] = plain->run(xc.data());
    if (decomp) plain->decompose(xc.data(), solv.gb, &dres[f * nres], &dres[f * nres + n_res_rec]);
  }
  last_stats[0] = ctx->launches.load() - before;
  if (host_out) {
    memcpy(out, res.data(), F * sizeof(rstg_frame_energy));
    if (decomp) memcpy(decomp, dres.data(), dres.size() * sizeof(rstg_residue_energy));
  } else {
    RSTG_CUDA(cudaMemcpyAsync(out, res.data(), F * sizeof(rstg_frame_energy), cudaMemcpyHostToDevice, st));
    if (decomp)
      RSTG_CUDA(cudaMemcpyAsync(decomp, dres.data(), dres.size() * sizeof(rstg_residue_energy), cudaMemcpyHostToDevice, st));
    RSTG_CUDA(cudaStreamSynchronize(st));
  }
}

void System::run_pb(const void* frames, bool f64, bool host_in, int64_t F, rstg_frame_energy* out, bool host_out) {
  cudaStream_t st = stream();
  size_t esz = f64 ? 8 : 4;
  std::vector<char> hbuf;
  const char* src = (const char*)frames;
  if (!host_in) {
    hbuf.resize((size_t)F * n_top * 3 * esz);
    RSTG_CUDA(cudaMemcpyAsync(hbuf.data(), frames, hbuf.size(), cudaMemcpyDeviceToHost, st));
    src = hbuf.data();
  }
  std::vector<rstg_frame_energy> res(F);
  RSTG_CUDA(cudaMemcpyAsync(res.data(), out, F * sizeof(rstg_frame_energy),
                            host_out ? cudaMemcpyHostToHost : cudaMemcpyDeviceToHost, st));
  RSTG_CUDA(cudaStreamSynchronize(st));
  if (!pbe) {
    pbe = std::make_unique<PbBatchEngine>(ctx, st);
    pbe->profile = pb_profile;
  }
  pbe->set_stream(st);
  const Topology* T[3] = {&split.complex, &split.rec, &split.lig};
  const std::vector<int64_t>* sel[3] = {nullptr, &split.rec_atoms, &split.lig_atoms};
  int64_t chunk = pb_frames_per_batch;
  if (chunk <= 0) {  // device memory budget: at most 60 % of the free memory and 64 GB
    // (every lock-step cycle has a fixed cost, mostly the coarse levels, so
    // fewer and larger batches are faster)
    size_t fr = 0, tot = 0;
    RSTG_CUDA(cudaMemGetInfo(&fr, &tot));
    double budget = std::min(0.6 * (double)fr, 64e9);
    chunk = std::max<int64_t>(1, (int64_t)(budget / (140.0 * (double)std::max<int64_t>(pb_points_estimate(), 1))));
  }
  std::vector<std::vector<double>> xs;
  std::vector<double> pol;
  for (int64_t f0 = 0; f0 < F; f0 += chunk) {
    int64_t B = std::min(chunk, F - f0);
    xs.assign(B * 3, {});
    std::vector<const std::vector<double>*> X, Q, R;
    for (int64_t b = 0; b < B; b++) {
      std::vector<double> xc(nC * 3);
      for (int64_t a = 0; a < nC; a++) {
        int64_t t = split.complex_atoms.empty() ? a : split.complex_atoms[a];
        for (int d = 0; d < 3; d++) {
          size_t k = ((size_t)(f0 + b) * n_top + t) * 3 + d;
          xc[3 * a + d] = f64 ? ((const double*)src)[k] : ((double)((const float*)src)[k] * 0.1) * 10.0;
        }
      }
      for (int k = 0; k < 3; k++) {
        std::vector<double>& x = xs[3 * b + k];
        if (!sel[k]) {
          x = xc;
        } else {
          x.resize(sel[k]->size() * 3);
          for (size_t i = 0; i < sel[k]->size(); i++)
            for (int d = 0; d < 3; d++) x[3 * i + d] = xc[3 * (*sel[k])[i] + d];
        }
        X.push_back(&x);
        Q.push_back(&T[k]->charges);
        R.push_back(&T[k]->radii);
      }
    }
    pol.assign(B * 3, 0.0);
    pb_polar_batch(ctx, st, *pbe, solv.pb, X, Q, R, pol.data(), nullptr, pb_rel_tol);
    for (int64_t b = 0; b < B; b++) {
      rstg_frame_energy& e = res[f0 + b];
      e.complex.polar = pol[3 * b];
      e.receptor.polar = pol[3 * b + 1];
      e.ligand.polar = pol[3 * b + 2];
      e.delta_polar = e.complex.polar - e.receptor.polar - e.ligand.polar;
      e.delta_total = e.delta_mm + e.delta_polar + e.delta_sa;
    }
  }
  RSTG_CUDA(cudaMemcpyAsync(out, res.data(), F * sizeof(rstg_frame_energy),
                            host_out ? cudaMemcpyHostToHost : cudaMemcpyHostToDevice, st));
  RSTG_CUDA(cudaStreamSynchronize(st));
}

void System::run(const void* frames, bool f64, bool host_in, int64_t F, rstg_frame_energy* out, bool host_out,
                 rstg_residue_energy* decomp_out) {
  if (F <= 0) return;
  if (opts.mode == RSTG_MODE_PLAIN) {
    run_plain(frames, f64, host_in, F, out, host_out, decomp_out);
    return;
  }
  cudaStream_t st = stream();
  size_t esz = f64 ? 8 : 4;
  if (!perm_ready) {
    std::vector<double> x0(nC * 3);
    std::vector<char> fr(n_top * 3 * esz);
    if (host_in)
      memcpy(fr.data(), frames, fr.size());
    else {
      RSTG_CUDA(cudaMemcpyAsync(fr.data(), frames, fr.size(), cudaMemcpyDeviceToHost, st));
      RSTG_CUDA(cudaStreamSynchronize(st));
    }
    for (int64_t a = 0; a < nC; a++) {
      int64_t t = split.complex_atoms.empty() ? a : split.complex_atoms[a];
      for (int d = 0; d < 3; d++)
        x0[3 * a + d] = f64 ? ((double*)fr.data())[3 * t + d] : (double)((float*)fr.data())[3 * t + d];
    }
    prepare_fused(x0.data());
  }
  int64_t nres = fp->nres;
  for (int attempt = 0; attempt < 3; attempt++) {
    ensure_buffers(std::min(F, batch));
    choose_psi(F);
    RSTG_CUDA(cudaMemsetAsync(diag.p, 0, 64, st));
    last_stats[0] = 0;
    for (int64_t f0 = 0; f0 < F; f0 += batch) {
      int64_t B = std::min(batch, F - f0);
      const char* src = (const char*)frames + (size_t)f0 * n_top * 3 * esz;
      RSTG_CUDA(cudaMemcpyAsync(in_frames.p, src, (size_t)B * n_top * 3 * esz,
                                host_in ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, st));
      bool want_dec = decomp_out != nullptr;
      rstg_residue_energy* dd = want_dec ? dec_buf.as<rstg_residue_energy>() : nullptr;
      bool use_graph = opts.use_graphs && B == batch;
      if (use_graph && (!graph || graph_frames != B || graph_input_f64 != (int)f64 || graph_decomp != (void*)dd)) {
        if (graph) cudaGraphExecDestroy(graph);
        graph = nullptr;
        cudaGraph_t g;
        RSTG_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        int64_t before = last_stats[0];
        try {
          launch_batch(in_frames.p, f64, B, res_buf.as<rstg_frame_energy>(), dd);
        } catch (...) {
          cudaStreamEndCapture(st, &g);
          throw;
        }
        RSTG_CUDA(cudaStreamEndCapture(st, &g));
        RSTG_CUDA(cudaGraphInstantiate(&graph, g, 0));
        cudaGraphDestroy(g);
        graph_frames = B;
        graph_input_f64 = (int)f64;
        graph_decomp = dd;
        last_stats[0] = before;  // the captured launches run below
        ctx->launches -= graph_kernels();
      }
      if (use_graph) {
        RSTG_CUDA(cudaGraphLaunch(graph, st));
        ctx->launches += graph_kernels();
        last_stats[0] += graph_kernels();
      } else {
        launch_batch(in_frames.p, f64, B, res_buf.as<rstg_frame_energy>(), dd);
      }
      auto kind = host_out ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
      RSTG_CUDA(cudaMemcpyAsync(out + f0, res_buf.p, B * sizeof(rstg_frame_energy), kind, st));
      if (want_dec)
        RSTG_CUDA(cudaMemcpyAsync(decomp_out + f0 * nres, dec_buf.p, B * nres * sizeof(rstg_residue_energy), kind, st));
    }
    int h[16];
    RSTG_CUDA(cudaMemcpyAsync(h, diag.p, 64, cudaMemcpyDeviceToHost, st));
    RSTG_CUDA(cudaStreamSynchronize(st));
    unsigned long long n64, nre;
    memcpy(&n64, h + 4, 8);
    memcpy(&nre, h + 6, 8);
    last_stats[1] = (int64_t)n64;
    last_stats[2] = (int64_t)nre;
    last_stats[3] = h[3];
    if (h[3] <= nbr_cap) {
      if (solv.method == 1) run_pb(frames, f64, host_in, F, out, host_out);
      return;
    }
    // a neighbour list overflowed: grow the capacity and run again
    nbr_cap = ((h[3] * 3 / 2 + 32) + 31) / 32 * 32;
    buf_frames = 0;
  }
  throw Error(RSTG_ERR_INVALID, "SASA neighbour list capacity could not be sized");
}

}  // namespace rstg
