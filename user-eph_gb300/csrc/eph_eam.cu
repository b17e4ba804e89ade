// The engine's pair force for standalone runs: eam/alloy (a LAMMPS setfl
// file; E = sum_i F_a(rho_i) + 1/2 sum_{i != j} phi_ab(r_ij), rho_i = sum_j
// f_b(r_ij)), evaluated on the GPU from the fix's own spatial bins each step
// before post_force, as LAMMPS's Verlet computes the pair force between
// initial_integrate and post_force.  No reference counterpart: the reference
// fix receives the pair force from LAMMPS (Tests/MD_Run/run.lmp uses
// pair_style eam/alloy with Ni.eam); this gives the standalone driver the
// same physics.  Tables: cubic Hermite per interval (host hermite_table).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "eph_candidates.cuh"
#include "eph_ctx_impl.hpp"
#include "eph_df64.cuh"
#include "eph_df_pair.cuh"

using namespace ephgb;

struct EamDevice {
  Eam host;
  DevBuf<D4> F, f, z2r;  // [element][nrho], [element][nr], [pair][nr]
  // f and z2r as double-floats for the df64 pair sums (FAST mode with
  // EPH_PAIRS_DF64): two float4 per interval, hi and lo parts
  DevBuf<float4> fd, zd;
  DevBuf<float2> fpd;  // F'(rho_i) / dr as a double-float, gathered per pair
  DevBuf<double> fp, energy, esum;
  DevBuf<unsigned> pj;    // pair list, [kcap][n]
  DevBuf<int> ns, ns_in;  // pairs per atom; with kept lists, those at the front of its rows
  int kcap = 0;
  int map[65] = {0};      // LAMMPS type -> setfl element
  double rc2_band = 0.0;  // FP32 candidate threshold
};

namespace {

constexpr unsigned FULL = 0xffffffffu;

struct EamParams {
  const D4 *F, *f, *z2r;
  const float4 *fd, *zd;
  int nel, nrho, nr;
  double inv_drho, inv_dr, rho_max, rc2;
  float rc2_band;
  float inv_dr_hi, inv_dr_lo, rc2_hi, rc2_lo;  // 1/dr and rc^2 as double-floats
  int map[65];
  int one;  // the one element of every type, or -1
};

// value and d/d(index) of a Hermite table at x (in units of the knot spacing)
__device__ __forceinline__ void herm(const D4 *__restrict__ t, int n, double x, double &v, double &dv) {
  int m = x > 0.0 ? (int)x : 0;  // below the table: its first interval
  if (m > n - 2) m = n - 2;
  double p = x - (double)m;
  if (p > 1.0) p = 1.0;
  const D4 c = t[m];
  v = fma(p, fma(p, fma(p, c.w, c.z), c.y), c.x);
  dv = fma(p, fma(3.0 * p, c.w, 2.0 * c.z), c.y);
}

// e = x_j (periodic image of the pair code) - x_i
__device__ __forceinline__ void image_vector(const StepParams &P, const D4 &xi, const D4 &xj, unsigned code,
                                             double &ex, double &ey, double &ez) {
  double cx = xj.x, cy = xj.y, cz = xj.z;
  if (code != CODE_NOSHIFT) {
    const int mx = (int)(code % 3u) - 1, my = (int)((code / 3u) % 3u) - 1, mz = (int)(code / 9u) - 1;
    if (mx) cx = xj.x + (mx > 0 ? P.prd[0] : -P.prd[0]);
    if (my) cy = xj.y + (my > 0 ? P.prd[1] : -P.prd[1]);
    if (mz) cz = xj.z + (mz > 0 ? P.prd[2] : -P.prd[2]);
  }
  ex = cx - xi.x;
  ey = cy - xi.y;
  ez = cz - xi.z;
}

// Pass 1 of the EAM density sweeps: atom i's candidates in the 27 bins
// around it (FP32/integer work, warp-uniform loop bounds), stored by cset as
// neighbour index | periodic-image code << 27; returns their count
template <class Set>
__device__ __forceinline__ int eam_candidates(const StepParams &P, const EamParams &E, int i, bool valid, int4 Bi,
                                              float4 oi, const int *__restrict__ bin_count,
                                              const BinEntry *__restrict__ bins, int kcap, unsigned *__restrict__ err,
                                              Set cset) {
  int nc = 0;
  for (int dz = -1; dz <= 1; ++dz) {
    const int Tz = Bi.z + dz, tz = Tz < 0 ? Tz + P.nb[2] : (Tz >= P.nb[2] ? Tz - P.nb[2] : Tz);
    const int kz = Tz < 0 ? -1 : (Tz >= P.nb[2] ? 1 : 0);
    const float bz = (float)dz * P.wf[2] - oi.z;
    for (int dy = -1; dy <= 1; ++dy) {
      const int Ty = Bi.y + dy, ty = Ty < 0 ? Ty + P.nb[1] : (Ty >= P.nb[1] ? Ty - P.nb[1] : Ty);
      const int ky = Ty < 0 ? -1 : (Ty >= P.nb[1] ? 1 : 0);
      const float by = (float)dy * P.wf[1] - oi.y;
      for (int dx = -1; dx <= 1; ++dx) {
        const int Tx = Bi.x + dx, tx = Tx < 0 ? Tx + P.nb[0] : (Tx >= P.nb[0] ? Tx - P.nb[0] : Tx);
        const int kx = Tx < 0 ? -1 : (Tx >= P.nb[0] ? 1 : 0);
        const float bx = (float)dx * P.wf[0] - oi.x;
        const int flat = tx + P.nb[0] * (ty + P.nb[1] * tz);
        int cnt = 0;
        if (valid) {
          cnt = bin_count[flat];
          cnt = cnt < P.bcap ? cnt : P.bcap;
        }
        const int cmax = __reduce_max_sync(FULL, cnt);
        const BinEntry *be = bins + (size_t)flat * P.bcap;
        for (int s = 0; s < cmax; ++s) {
          if (s >= cnt) continue;
          const BinEntry b = be[s];
          const unsigned j = b.idx & IDX_MASK;
          const float fx = bx + b.ox, fy = by + b.oy, fz = bz + b.oz;
          if (j == (unsigned)i || fx * fx + fy * fy + fz * fz >= E.rc2_band) continue;
          const unsigned wc = b.idx >> IDX_BITS;
          const int mx = kx - ((int)(wc % 3u) - 1), my = ky - ((int)((wc / 3u) % 3u) - 1),
                    mz = kz - ((int)(wc / 9u) - 1);
          if (mx < -1 || mx > 1 || my < -1 || my > 1 || mz < -1 || mz > 1) {
            atomicOr(err, ERR_DRIFT);
          } else if (nc >= kcap) {
            atomicOr(err, ERR_PAIR_OVERFLOW);
          } else {
            cset(nc++, j | ((unsigned)((mx + 1) + 3 * (my + 1) + 9 * (mz + 1)) << IDX_BITS));
          }
        }
      }
    }
  }
  return nc;
}

// rho_i = sum_j f_b(r_ij) over the 27 bins around atom i (bin edge >= the
// cutoff), the pairs within the cutoff written to the EAM pair list
// (u32: neighbour index | periodic-image code << 27, row k of atom i at
// k * n + i), then F_a(rho_i) and F'_a(rho_i) (beyond the table F continues
// linearly with the slope at its end).  Two passes as in the fix's density
// sweep: FP32/integer candidates (warp-uniform loop bounds) kept in shared
// memory with the overflow in the list rows, then the FP64 pass over the
// candidates in lockstep.
__global__ void __launch_bounds__(128)
    k_eam_density(StepParams P, EamParams E, const D4 *__restrict__ x, const int *__restrict__ type,
                  const int *__restrict__ bin_count, const BinEntry *__restrict__ bins,
                  const int4 *__restrict__ atom_bin, const float4 *__restrict__ atom_off,
                  unsigned *__restrict__ epj, int *__restrict__ ens, int kcap, double *__restrict__ fp,
                  double *__restrict__ energy, unsigned *__restrict__ err) {
  __shared__ unsigned s_cand[CAND_SMEM * 128];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int t = threadIdx.x, nt = blockDim.x;
  const bool valid = i < P.n;
  auto cget = [&](int k) -> unsigned { return k < CAND_SMEM ? s_cand[k * nt + t] : epj[(size_t)k * P.n + i]; };
  auto cset = [&](int k, unsigned u) {
    if (k < CAND_SMEM)
      s_cand[k * nt + t] = u;
    else
      epj[(size_t)k * P.n + i] = u;
  };
  const D4 xi = valid ? x[i] : D4{0.0, 0.0, 0.0, 0.0};
  int4 Bi = make_int4(0, 0, 0, 0);
  float4 oi = make_float4(0.f, 0.f, 0.f, 0.f);
  if (valid) {
    Bi = atom_bin[i];
    oi = atom_off[i];
  }
  const int nc = eam_candidates(P, E, i, valid, Bi, oi, bin_count, bins, kcap, err, cset);
  __syncwarp();
  double rho = 0.0;
  int ns = 0;
  const int nmax = __reduce_max_sync(FULL, nc);
  for (int k = 0; k < nmax; ++k) {
    if (k >= nc) continue;
    const unsigned u = cget(k);
    const unsigned j = u & IDX_MASK;
    double ex, ey, ez;
    image_vector(P, xi, x[j], u >> IDX_BITS, ex, ey, ez);
    const double r2 = fma(ez, ez, fma(ey, ey, ex * ex));
    if (r2 < E.rc2) {
      epj[(size_t)ns * P.n + i] = u;  // ns <= k: the candidate there is consumed
      ++ns;
      double v, dv;
      herm(E.f + (size_t)E.map[type[j]] * E.nr, E.nr, sqrt(r2) * E.inv_dr, v, dv);
      rho += v;
    }
  }
  if (!valid) return;
  ens[i] = ns;
  const int a = E.map[type[i]];
  double F, dF;
  herm(E.F + (size_t)a * E.nrho, E.nrho, rho * E.inv_drho, F, dF);
  dF *= E.inv_drho;
  if (rho > E.rho_max) F += dF * (rho - E.rho_max);
  fp[i] = dF;
  energy[i] = F;
}

// f_i = sum_j [F'_a(rho_i) f_b'(r) + F'_b(rho_j) f_a'(r) + phi_ab'(r)] e / r over
// the EAM pair list, added to the external force (if any); energy[i] +=
// 1/2 sum_j phi_ab(r)
__global__ void __launch_bounds__(128)
    k_eam_force(StepParams P, EamParams E, const D4 *__restrict__ x, const int *__restrict__ type,
                const unsigned *__restrict__ epj, const int *__restrict__ ens, const double *__restrict__ fp,
                const D4 *__restrict__ fext, D4 *__restrict__ f, double *__restrict__ energy) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  const D4 xi = x[i];
  const int a = E.map[type[i]];
  const double fpi = fp[i];
  double fx = 0.0, fy = 0.0, fz = 0.0, ep = 0.0;
  const int ns = ens[i];
  for (int k = 0; k < ns; ++k) {
    const unsigned u = epj[(size_t)k * P.n + i];
    const unsigned j = u & IDX_MASK;
    double ex, ey, ez;
    image_vector(P, xi, x[j], u >> IDX_BITS, ex, ey, ez);
    const double r2 = fma(ez, ez, fma(ey, ey, ex * ex));
    const double rinv = rsqrt(r2), r = r2 * rinv, q = r * E.inv_dr;
    const int b = E.map[type[j]];
    double fb, dfb, fa, dfa, z, dz;
    herm(E.f + (size_t)b * E.nr, E.nr, q, fb, dfb);
    dfa = dfb;
    if (a != b) herm(E.f + (size_t)a * E.nr, E.nr, q, fa, dfa);
    const int hi = a > b ? a : b, lo = a > b ? b : a;
    herm(E.z2r + (size_t)(hi * (hi + 1) / 2 + lo) * E.nr, E.nr, q, z, dz);
    const double phi = z * rinv;
    const double dphi = fma(dz, E.inv_dr, -phi) * rinv;
    const double dEdr = fma(fpi * E.inv_dr, dfb, fma(fp[j] * E.inv_dr, dfa, dphi));
    const double s = dEdr * rinv;
    fx = fma(s, ex, fx);
    fy = fma(s, ey, fy);
    fz = fma(s, ez, fz);
    ep = fma(0.5, phi, ep);
  }
  D4 out{fx, fy, fz, 0.0};
  if (fext) {
    const D4 g = fext[i];
    out.x += g.x;
    out.y += g.y;
    out.z += g.z;
  }
  f[i] = out;
  energy[i] += ep;
}

// ---------------------------------------------- df64 pair sums (FAST mode)

// The interval m of a Hermite table of n knots at q >= 0 (knot units) and the
// offset p in it: m from the FP32 part of q settled by the sign of the
// double-float remainder, with herm()'s clamps (at most the last interval, p
// at most 1)
__device__ __forceinline__ void herm_place(int n, df64::df q, int &m, df64::df &p) {
  using namespace df64;
  const df one{1.0f, 0.0f};
  const float kr = floor_estimate(q.hi);
  m = floor_estimate_int(kr);
  float th, te;
  two_sum(q.hi, -kr, th, te);
  p = make(th, te + q.lo);
  if (!(p.hi >= 0.0f && p.hi < 1.0f) || (unsigned)m > (unsigned)(n - 2)) {  // rarely: at a knot or past the table
    if (lt(p, df{0.0f, 0.0f})) {
      m -= 1;
      p = add(p, one);
    } else if (!lt(p, one)) {
      m += 1;
      p = sub(p, one);
    }
    if (m > n - 2) {
      p = add(p, df{(float)(m - (n - 2)), 0.0f});
      m = n - 2;
      if (!lt(p, one)) p = one;
    }
    if (m < 0) m = 0;
  }
}

// value of the table at (m, p)
__device__ __forceinline__ df64::df herm_value(const float4 *__restrict__ t, int m, df64::df p) {
  using namespace df64;
  float4 hi, lo;
  load_row(t + 2 * (size_t)m, hi, lo);
  return horner(df{hi.x, lo.x}, df{hi.y, lo.y}, df{hi.z, lo.z}, df{hi.w, lo.w}, p);
}

// value and derivative per knot unit: Horner's scheme and, from its partial
// sums, Horner's scheme of the derivative (synthetic division)
__device__ __forceinline__ void herm_both(const float4 *__restrict__ t, int m, df64::df p, df64::df &v, df64::df &dv) {
  using namespace df64;
  float4 hi, lo;
  load_row(t + 2 * (size_t)m, hi, lo);
  const df b3{hi.w, lo.w};
  const df b2 = fma(p, b3, df{hi.z, lo.z});
  const df b1 = fma(p, b2, df{hi.y, lo.y});
  v = fma(p, b1, df{hi.x, lo.x});
  dv = fma(p, fma(p, b3, b2), b1);
}

// resident blocks of 128 threads per SM the df64 sweeps are compiled for (GB300,
// both sweeps at 256,000 atoms with 7 + 6 / 8 + 7 / 10 + 8 blocks: 655 / 645 / 671 us)
#ifndef EPH_EAM_DENSITY_BLOCKS
#define EPH_EAM_DENSITY_BLOCKS 8
#endif
#ifndef EPH_EAM_FORCE_BLOCKS
#define EPH_EAM_FORCE_BLOCKS 7
#endif

// rho_i = sum_j f_b(r_ij) with the pair arithmetic in double-float and LANES
// lanes per atom: the candidates from the bins of the step or the kept lists
// (pair_candidates), e from the fixed-point positions, r^2, the cut-off test,
// the in-cut-off pairs to the EAM pair list (row k at k * n + i), r and f_b(r)
// in df64, rho_i in blocked sums; F and F' per atom in FP64; F' / dr also as a
// double-float for k_eam_force_df.  ONE: every type is the same setfl element.
// What bounds it: the candidates.  The 27 bins of 6.5 A hold 675 of them per
// atom, of which 78-85 are pairs; the bins' search took two thirds of the
// instructions (73,000 a warp), the kept lists leave 121 per atom.
// GB300, 256,000 atoms: 989 us -> 273 (kept lists); where the bins are searched
// every step, 16,384 atoms took both sweeps 536 us, now 100 (8 lanes).
template <bool ONE, int LANES, bool LIST>
__global__ void __launch_bounds__(128, EPH_EAM_DENSITY_BLOCKS)
    k_eam_density_df(StepParams P, EamParams E, CandidateArgs C, const int *__restrict__ type, int *__restrict__ ens,
                     int *__restrict__ ens_in, double *__restrict__ fp, float2 *__restrict__ fpd, double *__restrict__ energy) {
  using namespace df64;
  constexpr int CAP = LIST ? 0 : (LANES == 1 ? CAND_SMEM : CAND_SMEM * LANES - 1);
  __shared__ unsigned s_cand[CAP ? CAND_SMEM * 128 : 1];
  const int t = threadIdx.x, a = t / LANES, g = t % LANES;
  const int i = blockIdx.x * (128 / LANES) + a;
  const bool valid = i < P.n;
  const size_t n = (size_t)P.n;
  auto at = [&](int k) -> unsigned & { return s_cand[LANES == 1 ? k * 128 + t : a * CAP + k]; };
  long long xi[3] = {0, 0, 0};
  if (valid) own_fixed(C.rec, i, xi);
  const unsigned *tail;
  unsigned step;
  int first;
  const int nc = pair_candidates<LANES, LIST, LIST, CAP>(P, C, i, g, valid, at, tail, step, first);
  __syncwarp();
  const df rc2{E.rc2_hi, E.rc2_lo}, inv_dr{E.inv_dr_hi, E.inv_dr_lo};
  bsum rs = bsum_zero();
  int ns = 0, far = 0;
  const int nmax = __reduce_max_sync(FULL, nc);
  auto cand = [&](int k) -> unsigned {
    if (k >= nc) return CODE_NOSHIFT << IDX_BITS;  // atom 0, not counted
    return k < CAP ? at(k) : tail[(size_t)k * step];
  };
  unsigned u = cand(g), u2 = cand(g + LANES);
  int4 ra, rb;
  load_record(C.rec + 4 * (size_t)(u & IDX_MASK), ra, rb);
  for (int k = g, m = 0; k - g < nmax; k += LANES, ++m) {
    const unsigned uc = u;
    const int4 ca = ra, cb = rb;
    u = u2;
    u2 = cand(k + 2 * LANES);
    load_record(C.rec + 4 * (size_t)(u & IDX_MASK), ra, rb);
    long long ef[3];
    pair_fixed(P, ca, cb, uc >> IDX_BITS, xi, ef);
    const df ex = fixed_df(ef[0], P.fix_hi, P.fix_lo), ey = fixed_df(ef[1], P.fix_hi, P.fix_lo),
             ez = fixed_df(ef[2], P.fix_hi, P.fix_lo);
    const df r2 = dot3(ex, ey, ez, ex, ey, ez);
    bool in = k < nc && lt(r2, rc2);
    if (LIST) in = in && (k >= first || cb.w == 0);  // a moved atom in a kept list is out of reach
    const unsigned who = __ballot_sync(FULL, in);
    if (who != 0u) {  // else the lists' shell, together at their ends
      // the pair's row: from the front, in lane order; with kept lists the pairs
      // the fix's density sweep does not need go to the row's back
      const bool out = LIST && in && !(r2.hi < P.rc2_band);
      int slot = ns, back = far;
      if (LANES > 1) {
        const unsigned lane = t & 31, below = (1u << lane) - 1u;
        const unsigned group = ((1u << LANES) - 1u) << (lane & ~(LANES - 1));
        const unsigned outs = LIST ? __ballot_sync(FULL, out) & group : 0u, ins = who & group & ~outs;
        slot += __popc(ins & below);
        ns += __popc(ins);
        if (LIST) {
          back += __popc(outs & below);
          far += __popc(outs);
        }
      } else {
        ns += in && !out;
        far += out;
      }
      if (in) {
        const int row = out ? C.kcap - 1 - back : slot;
        // with kept lists no candidate waits in these rows; else row <= k, and the
        // candidate there is consumed
        if (ns + far <= C.kcap) C.pj[(size_t)row * n + i] = uc;
        else atomicOr(C.err, ERR_PAIR_OVERFLOW);
        const df r = mul(r2, rsqrt(r2, rsqrt_estimate(r2.hi)));
        int mk;
        df p;
        herm_place(E.nr, mul(r, inv_dr), mk, p);
        const int b = ONE ? E.one : E.map[type[uc & IDX_MASK]];
        acc_add(rs.blk, herm_value(E.fd + 2 * (size_t)b * E.nr, mk, p));
      }
    }
    if ((m & 7) == 7) bsum_fold(rs);  // at most 8 terms to a block, skipped iterations or not
  }
  double rho = to_double(bsum_value(rs));
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) rho += __shfl_xor_sync(FULL, rho, o);
  if (!valid || g != 0) return;
  // more pairs than rows (the step ends in an error): some rows between those
  // counted were never written, so none are read
  if (ns + far > C.kcap) ns = far = 0;
  ens[i] = ns + far;
  if (LIST) ens_in[i] = ns;
  const int el = ONE ? E.one : E.map[type[i]];
  double F, dF;
  herm(E.F + (size_t)el * E.nrho, E.nrho, rho * E.inv_drho, F, dF);
  dF *= E.inv_drho;
  if (rho > E.rho_max) F += dF * (rho - E.rho_max);
  fp[i] = dF;
  const df gd = from_double(dF * E.inv_dr);
  fpd[i] = make_float2(gd.hi, gd.lo);
  energy[i] = F;
}

// k_eam_force with the pair arithmetic in double-float and LANES lanes per
// atom: per pair 1/r (a Newton step on the FP32 estimate), r = r^2 / r and a
// residual step (the steep tables need r to the last bits), the
// Hermite tables f_b, f_a and z2r = r phi at one interval and offset, dE/dr and
// (dE/dr / r) e in df64, the force and 1/2 sum phi in blocked sums.  Bound by
// FP32 issue: ~700 instructions per pair before (an interval and a scaled
// derivative per table, square root and reciprocal apart), ~430 now.
// GB300, 256,000 atoms: 596 -> 366 us (361 without the residual step).
template <bool ONE, int LANES>
__global__ void __launch_bounds__(128, EPH_EAM_FORCE_BLOCKS)
    k_eam_force_df(StepParams P, EamParams E, const int *__restrict__ type, const unsigned *__restrict__ epj,
                   const int *__restrict__ ens, const int *__restrict__ ens_in, int kcap,
                   const float2 *__restrict__ fpd, const D4 *__restrict__ fext, D4 *__restrict__ f,
                   double *__restrict__ energy, const int4 *__restrict__ rec) {
  using namespace df64;
  const int t = threadIdx.x, g = t % LANES;
  const int i = blockIdx.x * (128 / LANES) + t / LANES;
  const bool valid = i < P.n;
  if (LANES == 1 && !valid) return;
  long long xi[3] = {0, 0, 0};
  int el = ONE ? E.one : 0, ns = 0, front = 0;
  df fpi{0.0f, 0.0f};
  if (valid) {
    own_fixed(rec, i, xi);
    if (!ONE) el = E.map[type[i]];
    const float2 gi = fpd[i];
    fpi = df{gi.x, gi.y};
    ns = front = ens[i];
    if (ens_in) front = ens_in[i];  // the others from the row's back
  }
  const df inv_dr{E.inv_dr_hi, E.inv_dr_lo};
  bsum s[4] = {bsum_zero(), bsum_zero(), bsum_zero(), bsum_zero()};
  const size_t n = (size_t)P.n;
  auto pair = [&](int k) -> unsigned {
    if (k >= ns) return CODE_NOSHIFT << IDX_BITS;
    return epj[(size_t)(k < front ? k : kcap - 1 - (k - front)) * n + i];
  };
  unsigned u = pair(g), u2 = pair(g + LANES);
  int4 ra, rb;
  load_record(rec + 4 * (size_t)(u & IDX_MASK), ra, rb);
  float2 gn = fpd[u & IDX_MASK];
  for (int k = g, m = 0; k < ns; k += LANES, ++m) {
    const unsigned uc = u;
    const int4 ca = ra, cb = rb;
    const float2 gj = gn;
    u = u2;
    u2 = pair(k + 2 * LANES);
    load_record(rec + 4 * (size_t)(u & IDX_MASK), ra, rb);
    gn = fpd[u & IDX_MASK];
    long long ef[3];
    pair_fixed(P, ca, cb, uc >> IDX_BITS, xi, ef);
    const df ex = fixed_df(ef[0], P.fix_hi, P.fix_lo), ey = fixed_df(ef[1], P.fix_hi, P.fix_lo),
             ez = fixed_df(ef[2], P.fix_hi, P.fix_lo);
    const df r2 = dot3(ex, ey, ez, ex, ey, ez);
    const float y = rsqrt_estimate(r2.hi);
    const df rinv = rsqrt(r2, y);
    int mk;
    df p;
    herm_place(E.nr, mul(sqrt_near(r2, mul(r2, rinv), y), inv_dr), mk, p);
    const int b = ONE ? el : E.map[type[uc & IDX_MASK]];
    df fb, dfb, z, dz;
    herm_both(E.fd + 2 * (size_t)b * E.nr, mk, p, fb, dfb);
    const int hi = el > b ? el : b, lo = el > b ? b : el;
    herm_both(E.zd + 2 * (size_t)(hi * (hi + 1) / 2 + lo) * E.nr, mk, p, z, dz);
    // F'_a(rho_i) f_b' + F'_b(rho_j) f_a'
    df emb;
    if (ONE || el == b) {
      emb = mul(add(fpi, df{gj.x, gj.y}), dfb);
    } else {
      df fa, dfa;
      herm_both(E.fd + 2 * (size_t)el * E.nr, mk, p, fa, dfa);
      emb = add(mul(fpi, dfb), mul(df{gj.x, gj.y}, dfa));
    }
    const df phi = mul(z, rinv);
    const df dphi = mul(fma(dz, inv_dr, neg(phi)), rinv);
    const df sc = mul(add(emb, dphi), rinv);
    acc_fma(s[0].blk, sc, ex);
    acc_fma(s[1].blk, sc, ey);
    acc_fma(s[2].blk, sc, ez);
    acc_add(s[3].blk, df{0.5f * phi.hi, 0.5f * phi.lo});
    if ((m & 7) == 7) {
#pragma unroll
      for (int q = 0; q < 4; ++q) bsum_fold(s[q]);
    }
  }
  double w[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    w[q] = to_double(bsum_value(s[q]));
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) w[q] += __shfl_xor_sync(FULL, w[q], o);
  }
  if (!valid || g != 0) return;
  D4 out{w[0], w[1], w[2], 0.0};
  if (fext) {
    const D4 e = fext[i];
    out.x += e.x;
    out.y += e.y;
    out.z += e.z;
  }
  f[i] = out;
  energy[i] += w[3];
}

// sum of the per-atom energies in a fixed order: ENERGY_BLOCKS partial sums,
// then theirs (one block over all atoms took 478 us at 256,000 atoms, GB300)
constexpr int ENERGY_BLOCKS = 256;
__global__ void k_eam_energy_sum(const double *__restrict__ e, int n, double *__restrict__ out) {
  __shared__ double s[256];
  double acc = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) acc += e[i];
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) s[threadIdx.x] += s[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = s[0];
}

EamParams eam_params(const eph_ctx *c) {
  const EamDevice *d = c->eam;
  EamParams E;
  E.F = d->F.p;
  E.f = d->f.p;
  E.z2r = d->z2r.p;
  E.nel = d->host.nel;
  E.nrho = (int)d->host.nrho;
  E.nr = (int)d->host.nr;
  E.inv_drho = 1.0 / d->host.drho;
  E.inv_dr = 1.0 / d->host.dr;
  E.rho_max = d->host.drho * (double)(d->host.nrho - 1);
  E.rc2 = d->host.rc * d->host.rc;
  E.rc2_band = (float)d->rc2_band;
  E.fd = d->fd.p;
  E.zd = d->zd.p;
  const df64::df idr = df64::from_double(E.inv_dr), rc2 = df64::from_double(E.rc2);
  E.inv_dr_hi = idr.hi;
  E.inv_dr_lo = idr.lo;
  E.rc2_hi = rc2.hi;
  E.rc2_lo = rc2.lo;
  std::memcpy(E.map, d->map, sizeof(E.map));
  E.one = d->map[1];
  for (int t = 2; t <= c->ntypes; ++t)
    if (d->map[t] != E.one) E.one = -1;
  return E;
}

// The Hermite tables in FP64 (D4 {c0, c1, c2, c3} per interval) and, with
// df not NULL, as double-floats (float4 hi parts, float4 lo parts per
// interval; each coefficient the nearest float plus the nearest float to
// the rest)
int upload_table(eph_ctx *c, DevBuf<D4> &dst, const std::vector<std::vector<double>> &tabs,
                 DevBuf<float4> *dfo = nullptr) {
  std::vector<double> all;
  for (const auto &t : tabs) {
    std::vector<double> coef;
    hermite_table(t, coef);
    all.insert(all.end(), coef.begin(), coef.end());
  }
  CUDA_TRY(c, dst.alloc(all.size() / 4));
  CUDA_TRY(c, ctxi::upload(c, dst.p, all.data(), all.size() * sizeof(double)));
  std::vector<float> split;
  if (dfo) {
    split.resize(2 * all.size());
    for (size_t m = 0; m < all.size() / 4; ++m)
      for (int k = 0; k < 4; ++k) {
        const df64::df v = df64::from_double(all[4 * m + k]);
        split[8 * m + k] = v.hi;
        split[8 * m + 4 + k] = v.lo;
      }
    CUDA_TRY(c, dfo->alloc(all.size() / 2));
    CUDA_TRY(c, ctxi::upload(c, dfo->p, split.data(), split.size() * sizeof(float)));
  }
  CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  return EPH_OK;
}

// Lanes per atom of the df64 EAM sweeps (measured on GB300, both sweeps, us
// with 2 / 4 / 8 / 16 lanes: 2,048 atoms 212 / 117 / 71 / 49, 6,912 atoms 218 /
// 126 / 83 / 68, 16,384 atoms 122 / 80 / 66 / 76, 32,000 atoms 143 / 115 / 114 /
// 125, 131,072 atoms 364 / 351 / 362 / 417, 256,000 atoms 649 / 642 / 671 / 789,
// 500,000 atoms 1,173 / 1,210 / 1,280 / 1,518; one lane 1,219 there)
int eam_lanes(const eph_ctx *c) {
  return c->n <= 10000 ? 16 : (c->n <= 32000 ? 8 : (c->n <= 360000 ? 4 : 2));
}

template <bool ONE, int LANES>
void launch_eam_df(eph_ctx *c, const EamParams &E, const CandidateArgs &C, const D4 *fext) {
  EamDevice *d = c->eam;
  const int nb = nblocks((long)c->n * LANES);
  if (c->reuse)
    k_eam_density_df<ONE, LANES, true><<<nb, BLOCK, 0, c->stream>>>(c->P, E, C, c->type.p, d->ns.p, d->ns_in.p,
                                                                    d->fp.p, d->fpd.p,
                                                                    d->energy.p);
  else
    k_eam_density_df<ONE, LANES, false><<<nb, BLOCK, 0, c->stream>>>(c->P, E, C, c->type.p, d->ns.p, nullptr, d->fp.p,
                                                                     d->fpd.p, d->energy.p);
  k_eam_force_df<ONE, LANES><<<nb, BLOCK, 0, c->stream>>>(c->P, E, c->type.p, d->pj.p, d->ns.p,
                                                          c->reuse ? d->ns_in.p : nullptr, d->kcap, d->fpd.p, fext,
                                                          c->f.p, d->energy.p, c->dfrec.p);
}

}  // namespace

namespace ephgb {
namespace ctxi {

double eam_cutoff(const eph_ctx *c) { return c->eam ? c->eam->host.rc : 0.0; }

int eam_rows(const eph_ctx *c) { return c->eam ? c->eam->kcap : 0; }

void eam_free(eph_ctx *c) {
  delete c->eam;
  c->eam = nullptr;
}

int eam_resize(eph_ctx *c) {
  EamDevice *d = c->eam;
  if (!d || d->fp.n == (size_t)c->n) return EPH_OK;
  const size_t N = (size_t)c->n;
  CUDA_TRY(c, d->fp.alloc(N));
  CUDA_TRY(c, d->energy.alloc(N));
  CUDA_TRY(c, d->ns.alloc(N));
  CUDA_TRY(c, d->ns_in.alloc(N));
  CUDA_TRY(c, d->fpd.alloc(N));
  CUDA_TRY(c, cudaMemsetAsync(d->energy.p, 0, sizeof(double) * N, c->stream));
  // pair rows from the number density: twice the cut-off sphere, plus slack
  const double dens = (double)c->n / (c->prd[0] * c->prd[1] * c->prd[2]);
  const double rc = d->host.rc;
  d->kcap = ((int)std::ceil(2.0 * dens * 4.18879020478639 * rc * rc * rc + 32.0) + 7) / 8 * 8;
  CUDA_TRY(c, d->pj.alloc((size_t)d->kcap * N));
  return EPH_OK;
}

bool eam_pair_list(const eph_ctx *c, const unsigned **pj, const int **ns, const int **inner) {
  const EamDevice *d = c->eam;
  if (!d || !d->pj.p || !d->ns.p || d->ns.n < (size_t)c->n) return false;
  // every pair within the fix's FP32 candidate threshold must be in the list
  // (within the EAM cut-off, by the FP64 test), with room for FP32 rounding
  if (!((double)c->P.rc2_band * (1.0 + 1e-5) < d->host.rc * d->host.rc)) return false;
  *pj = d->pj.p;
  *ns = d->ns.p;
  *inner = c->reuse ? d->ns_in.p : nullptr;
  return true;
}

int launch_eam(eph_ctx *c) {
  EamDevice *d = c->eam;
  const EamParams E = eam_params(c);
  const int nb = nblocks(c->n);
  if (d->fp.n < (size_t)c->n) return fail(c, EPH_ERR_STATE, "pair force buffers not sized for the atoms");
  PhaseScope ps(c, EPH_PHASE_PAIR);
  ps.launched(2);
  const D4 *fext = c->have_fext ? c->fext.p : nullptr;
  if (c->mode == EPH_MODE_FAST && c->pair_arith == EPH_PAIRS_DF64) {
    CandidateArgs C{};
    C.bin_count = c->bin_count.p;
    C.bins = c->bins.p;
    C.atom_bin = c->atom_bin.p;
    C.atom_off = c->atom_off.p;
    C.rec = c->dfrec.p;
    C.x = c->x.p;
    C.err = c->d_err.p;
    C.pj = d->pj.p;
    C.kcap = d->kcap;
    C.band = E.rc2_band;
    C.cl = c->cl.p;
    C.cl_n = c->cl_n.p;
    C.state = c->state.p;
    C.rb = c->rb.p;
    C.flist = c->flist.p;
    C.fpos = c->fpos.p;
    C.far2 = far_cutoff2(c, E.rc2);
    C.xref = c->xref.p;
    C.moved = c->mcand.p;
    C.mcap = c->mcap;
    const int lanes = eam_lanes(c);
    if (E.one >= 0) {
      if (lanes == 2) launch_eam_df<true, 2>(c, E, C, fext);
      else if (lanes == 4) launch_eam_df<true, 4>(c, E, C, fext);
      else if (lanes == 8) launch_eam_df<true, 8>(c, E, C, fext);
      else launch_eam_df<true, 16>(c, E, C, fext);
    } else {
      if (lanes == 2) launch_eam_df<false, 2>(c, E, C, fext);
      else if (lanes == 4) launch_eam_df<false, 4>(c, E, C, fext);
      else if (lanes == 8) launch_eam_df<false, 8>(c, E, C, fext);
      else launch_eam_df<false, 16>(c, E, C, fext);
    }
  } else {
    k_eam_density<<<nb, BLOCK, 0, c->stream>>>(c->P, E, c->x.p, c->type.p, c->bin_count.p, c->bins.p,
                                                c->atom_bin.p, c->atom_off.p, d->pj.p, d->ns.p, d->kcap, d->fp.p,
                                                d->energy.p, c->d_err.p);
    k_eam_force<<<nb, BLOCK, 0, c->stream>>>(c->P, E, c->x.p, c->type.p, d->pj.p, d->ns.p, d->fp.p, fext, c->f.p,
                                              d->energy.p);
  }
  CUDA_TRY(c, cudaGetLastError());
  c->eam_list_fresh = true;  // this step's pairs: the fix's density sweep may read them
  return EPH_OK;
}

}  // namespace ctxi
}  // namespace ephgb

extern "C" {

int eph_set_pair_eam(eph_ctx *c, const char *path, int ntypes, const char *const *elements) {
  if (!c || !path || !elements) return EPH_ERR_ARG;
  if (c->n > 0) return ctxi::fail(c, EPH_ERR_STATE, "set the pair force before the atoms (eph_set_atoms)");
  if (ntypes != c->ntypes) return ctxi::fail(c, EPH_ERR_ARG, "one setfl element name per atom type");
  EamDevice *d = new (std::nothrow) EamDevice();
  if (!d) return EPH_ERR_ARG;
  std::string e = d->host.load(path);
  if (!e.empty()) {
    delete d;
    return ctxi::fail(c, EPH_ERR_FILE, e);
  }
  for (int t = 1; t <= ntypes; ++t) {
    int m = -1;
    for (int k = 0; k < d->host.nel; ++k)
      if (d->host.names[k] == elements[t - 1]) m = k;
    if (m < 0) {
      delete d;
      return ctxi::fail(c, EPH_ERR_ARG, std::string("element ") + elements[t - 1] + " not in the setfl file");
    }
    d->map[t] = m;
  }
  ctxi::eam_free(c);
  ctxi::drop_list(c);  // a larger radius: configured with the atoms
  c->eam = d;
  int r;
  CUDA_TRY(c, cudaSetDevice(c->device));
  if ((r = upload_table(c, d->F, d->host.F)) || (r = upload_table(c, d->f, d->host.f, &d->fd)) ||
      (r = upload_table(c, d->z2r, d->host.z2r, &d->zd)))
    return r;
  CUDA_TRY(c, d->esum.alloc(1 + ENERGY_BLOCKS));
  d->rc2_band = d->host.rc * d->host.rc * (1.0 + 1e-4);
  // the bins must hold every pair within the larger of the two cutoffs (all
  // of their geometry: the FP64, FP32 and double-float bin edges)
  if ((r = ctxi::set_bin_geometry(c, std::max(c->beta.r_cutoff, d->host.rc))))
    return ctxi::fail(c, EPH_ERR_ARG, "box edge shorter than three EAM cutoffs");
  c->bin_count.free();
  c->bcap = 0;
  ctxi::drop_graph(c);
  c->buf_gen += 1;
  return EPH_OK;
}

int eph_pair_energy(eph_ctx *c, double *E) {
  if (!c || !E) return EPH_ERR_ARG;
  *E = 0.0;
  if (!c->eam || !c->eam->energy.p) return EPH_OK;
  double *part = c->eam->esum.p + 1;
  k_eam_energy_sum<<<ENERGY_BLOCKS, 256, 0, c->stream>>>(c->eam->energy.p, c->n, part);
  k_eam_energy_sum<<<1, 256, 0, c->stream>>>(part, ENERGY_BLOCKS, c->eam->esum.p);
  CUDA_TRY(c, cudaMemcpyAsync(E, c->eam->esum.p, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  return ctxi::check_device(c);
}

}  // extern "C"
