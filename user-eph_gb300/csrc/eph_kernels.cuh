// sm_103a kernels of the fix-eph hot path.
//
// One to 32 lanes per atom by size, one thread per atom for what is done once
// per atom.  The FP64 pipe of GB300 issues about two instructions per clock per
// SM, so the kernels with FP64 pair terms are bound by FP64 instruction issue,
// not by HBM (those with df64 terms: see k_density_df): the design removes FP64 work
// (in-cutoff pairs compacted per step so the warps sweep them in lockstep,
// pair geometry and rho(r^2) cached once per step, alpha/beta per atom once)
// and keeps integer/FP32 work (binning, candidate tests, sorting) off the
// FP64 pipe.
//
// This translation unit is compiled with -fmad=false: in EXACT mode every
// product and sum rounds separately, in the reference's order, so forces and
// densities equal the reference's bit for bit; FAST mode writes its FMAs
// explicitly.
#pragma once

#include "eph_candidates.cuh"
#include "eph_device.cuh"
#include "eph_df64.cuh"
#include "eph_softfp.cuh"
#include "eph_df_pair.cuh"

namespace ephgb {

// ------------------------------------------------------------- integrator

// The half kick and drift of FixEPH::initial_integrate (fix_eph.cpp:305-328)
// for one atom of the group
template <bool FAST>
__device__ __forceinline__ void kick_drift(const StepParams &P, double dtfm, const D4 &fi, D4 &xi, D4 &vi) {
  if (FAST) {
    vi.x = fma(dtfm, fi.x, vi.x);
    vi.y = fma(dtfm, fi.y, vi.y);
    vi.z = fma(dtfm, fi.z, vi.z);
    xi.x = fma(P.dtv, vi.x, xi.x);
    xi.y = fma(P.dtv, vi.y, xi.y);
    xi.z = fma(P.dtv, vi.z, xi.z);
  } else {
    vi.x += dtfm * fi.x;
    vi.y += dtfm * fi.y;
    vi.z += dtfm * fi.z;
    xi.x += P.dtv * vi.x;
    xi.y += P.dtv * vi.y;
    xi.z += P.dtv * vi.z;
  }
}

// The half kick of FixEPH::final_integrate (fix_eph.cpp:330-348)
template <bool FAST>
__device__ __forceinline__ void kick(double dtfm, const D4 &fi, D4 &vi) {
  if (FAST) {
    vi.x = fma(dtfm, fi.x, vi.x);
    vi.y = fma(dtfm, fi.y, vi.y);
    vi.z = fma(dtfm, fi.z, vi.z);
  } else {
    vi.x += dtfm * fi.x;
    vi.y += dtfm * fi.y;
    vi.z += dtfm * fi.z;
  }
}

// FixEPH::initial_integrate (fix_eph.cpp:305-328) and the engine's rebuild
// test (an atom moved more than skin/2 since the last wrap).  With `clear`, also
// the engine's force of the step to come: the external one, or zero (a
// memset or copy of its own before).
template <bool FAST>
__global__ void k_initial_integrate(StepParams P, D4 *__restrict__ x, D4 *__restrict__ v, D4 *__restrict__ f,
                                    const int *__restrict__ type, const int *__restrict__ mask,
                                    const D4 *__restrict__ xhold, int check_wrap, int *__restrict__ wrapflag,
                                    int clear, const D4 *__restrict__ fext) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool moved = false;
  if (i < P.n) {
    D4 xi = x[i];
    if (!(P.flags & 0x08) && (mask[i] & P.groupbit)) {
      D4 vi = v[i];
      kick_drift<FAST>(P, P.dtfm[type[i]], f[i], xi, vi);
      v[i] = vi;
      x[i] = xi;
    }
    if (clear) f[i] = fext ? fext[i] : D4{0.0, 0.0, 0.0, 0.0};
    if (check_wrap) {
      const D4 h = xhold[i];
      const double dx = xi.x - h.x, dy = xi.y - h.y, dz = xi.z - h.z;
      moved = dx * dx + dy * dy + dz * dz > P.triggersq;
    }
  }
  if (__any_sync(0xffffffffu, moved) && (threadIdx.x & 31) == 0) atomicOr(wrapflag, 1);
}

// FixEPH::final_integrate (fix_eph.cpp:330-348)
template <bool FAST>
__global__ void k_final_integrate(StepParams P, D4 *__restrict__ v, const D4 *__restrict__ f,
                                  const int *__restrict__ type, const int *__restrict__ mask) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.n || (P.flags & 0x08) || !(mask[i] & P.groupbit)) return;
  D4 vi = v[i];
  kick<FAST>(P.dtfm[type[i]], f[i], vi);
  v[i] = vi;
}

// The hooks with the engine's host arrays (eph_initial_integrate_host,
// eph_final_integrate_host), one chunk of `count` atoms per launch (the
// pointers start at the chunk): the staged host rows (n x 3 doubles) go into
// the D4 records (x.w, the element, kept), the hook's arithmetic runs, and
// the rows the engine reads back are written to staging for the
// device->host copies -- the work of k_pack3, the hook's kernel and
// k_unpack3 in one pass.
template <bool FAST>
__global__ void k_initial_host(StepParams P, int count, const double *__restrict__ sx, const double *__restrict__ sv,
                               D4 *__restrict__ x, D4 *__restrict__ v, const D4 *__restrict__ f,
                               const int *__restrict__ type, const int *__restrict__ mask, double *__restrict__ ox,
                               double *__restrict__ ov) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const size_t r = 3 * (size_t)i;
  D4 xi = x[i];
  xi.x = sx[r];
  xi.y = sx[r + 1];
  xi.z = sx[r + 2];
  D4 vi = v[i];
  vi.x = sv[r];
  vi.y = sv[r + 1];
  vi.z = sv[r + 2];
  if (!(P.flags & 0x08) && (mask[i] & P.groupbit)) kick_drift<FAST>(P, P.dtfm[type[i]], f[i], xi, vi);
  x[i] = xi;
  v[i] = vi;
  ox[r] = xi.x;
  ox[r + 1] = xi.y;
  ox[r + 2] = xi.z;
  ov[r] = vi.x;
  ov[r + 1] = vi.y;
  ov[r + 2] = vi.z;
}

template <bool FAST>
__global__ void k_final_host(StepParams P, int count, const double *__restrict__ sf, D4 *__restrict__ f,
                             D4 *__restrict__ v, const int *__restrict__ type, const int *__restrict__ mask,
                             double *__restrict__ ov) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const size_t r = 3 * (size_t)i;
  D4 fi = f[i];
  fi.x = sf[r];
  fi.y = sf[r + 1];
  fi.z = sf[r + 2];
  f[i] = fi;
  D4 vi = v[i];
  if (!(P.flags & 0x08) && (mask[i] & P.groupbit)) {
    kick<FAST>(P.dtfm[type[i]], fi, vi);
    v[i] = vi;
  }
  ov[r] = vi.x;
  ov[r + 1] = vi.y;
  ov[r + 2] = vi.z;
}

// ------------------------------------------------------------------ binning

// LAMMPS Domain::pbc for an orthogonal box: a position into [lo, hi)
__device__ __forceinline__ void wrap_into_box(const StepParams &P, D4 &xi) {
  double *c[3] = {&xi.x, &xi.y, &xi.z};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double q = *c[k];
    if (q < P.lo[k]) q += P.prd[k];
    if (q >= P.hi[k]) {
      q -= P.prd[k];
      q = q > P.lo[k] ? q : P.lo[k];
    }
    *c[k] = q;
  }
}

// Wrap positions into [lo, hi) when the engine rebuilds, then drop every
// atom into its spatial bin.  A bin edge is at least the cutoff (with list
// reuse: the list radius), so all pairs inside it are found in the 27 bins
// around an atom.  Bins keep unwrapped coordinates: an atom that drifted up
// to one bin outside the box carries a wrap code and the offset from its own
// (unwrapped) bin corner.
// With a gate (candidate-list reuse): nothing unless *gate (a build step),
// no wrap (k_list_check did it), and the positions are kept in xref.
// With rec (the df64 pair sums), also the atom's record for them (df_record).
__global__ void k_bin(StepParams P, D4 *__restrict__ x, D4 *__restrict__ xhold, const int *__restrict__ wrapflag,
                      int *__restrict__ bin_count, BinEntry *__restrict__ bins, int4 *__restrict__ atom_bin,
                      float4 *__restrict__ atom_off, unsigned *__restrict__ err,
                      unsigned long long *__restrict__ counters, int bump_step, const int *__restrict__ gate = nullptr,
                      D4 *__restrict__ xref = nullptr, int4 *__restrict__ rec = nullptr,
                      const D4 *__restrict__ v = nullptr) {
  if (gate && !*gate) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && bump_step) *P.step += 1ull;  // read by the density sweep that follows
  if (i >= P.n) return;
  D4 xi = x[i];
  if (!gate && *wrapflag) {
    wrap_into_box(P, xi);
    x[i] = xi;
    xhold[i] = xi;
    if (i == 0) atomicAdd(&counters[CNT_WRAP], 1ull);
  }
  if (xref) xref[i] = xi;
  const double p[3] = {xi.x, xi.y, xi.z};
  int B[3], t[3], wc[3];
  float o[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double s = p[k] - P.lo[k];
    int b = (int)floor(s * P.inv_w[k]);
    if (b < -1 || b > P.nb[k]) {
      atomicOr(err, ERR_DRIFT);
      b = b < -1 ? -1 : P.nb[k];
    }
    B[k] = b;
    t[k] = b < 0 ? b + P.nb[k] : (b >= P.nb[k] ? b - P.nb[k] : b);
    wc[k] = (b - t[k]) / P.nb[k];
    o[k] = (float)(s - (double)b * P.w[k]);
  }
  const int flat = t[0] + P.nb[0] * (t[1] + P.nb[1] * t[2]);
  const unsigned code = (unsigned)((wc[0] + 1) + 3 * (wc[1] + 1) + 9 * (wc[2] + 1));
  const int slot = atomicAdd(&bin_count[flat], 1);
  if (slot < P.bcap) {
    BinEntry be;
    be.idx = (unsigned)i | (code << IDX_BITS);
    be.ox = o[0];
    be.oy = o[1];
    be.oz = o[2];
    bins[(size_t)flat * P.bcap + slot] = be;
  } else {
    atomicOr(err, ERR_BIN_OVERFLOW);
  }
  atom_bin[i] = make_int4(B[0], B[1], B[2], flat);
  atom_off[i] = make_float4(o[0], o[1], o[2], 0.f);
  if (rec) {
    const int none[3] = {0, 0, 0};
    df_record(P, i, xi, none, false, v[i], rec);
  }
}

// -------------------------------------------------------- density sweep

// Sorts every bin's entries by atom index with one warp per bin, for bins of
// at most 32 R entries: lane l holds entries l, l + 32, ..., each entry's place
// is the number of entries with a smaller atom index (indices are distinct),
// found by broadcasting every entry's key across the warp; all loads happen
// before any store.
constexpr int SORT_WARP_MAX = 128;
template <int R>
__global__ void k_bin_sort_warp(int nbins, int bcap, const int *__restrict__ bin_count, BinEntry *__restrict__ bins,
                                const int *__restrict__ gate = nullptr) {
  if (gate && !*gate) return;
  const long w = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= nbins) return;  // whole warps leave together
  int cnt = bin_count[w];
  cnt = cnt < bcap ? cnt : bcap;
  BinEntry *e = bins + (size_t)w * bcap;
  BinEntry b[R];
  unsigned key[R];
  int place[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    b[r] = BinEntry{};
    if (lane + 32 * r < cnt) b[r] = e[lane + 32 * r];
    key[r] = lane + 32 * r < cnt ? (b[r].idx & IDX_MASK) : 0xffffffffu;
    place[r] = 0;
  }
  const int most = cnt < 32 ? cnt : 32;
  for (int s = 0; s < most; ++s) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const unsigned k = __shfl_sync(0xffffffffu, key[r], s);
#pragma unroll
      for (int q = 0; q < R; ++q) place[q] += k < key[q];
    }
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (lane + 32 * r < cnt) e[place[r]] = b[r];
}

// The same with one thread per bin (a handful of entries each), so the candidate order below is fixed run to run.
__global__ void k_bin_sort(int nbins, int bcap, const int *__restrict__ bin_count, BinEntry *__restrict__ bins,
                           const int *__restrict__ gate = nullptr) {
  if (gate && !*gate) return;
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbins) return;
  int cnt = bin_count[b];
  cnt = cnt < bcap ? cnt : bcap;
  BinEntry *e = bins + (size_t)b * bcap;
  for (int k = 1; k < cnt; ++k) {
    const BinEntry v = e[k];
    const unsigned key = v.idx & IDX_MASK;
    int p = k;
    while (p > 0 && (e[p - 1].idx & IDX_MASK) > key) {
      e[p] = e[p - 1];
      --p;
    }
    e[p] = v;
  }
}

// One in-cutoff pair (i, j) of the density sweep: rho_j(r^2) into rho_i, the
// pair cache row at `slot`, and with FUSE_W the sums of M_i and S_i.
template <bool MULTI, bool FUSE_W>
__device__ __forceinline__ void density_pair(const StepParams &P, int ei, unsigned u, int ej, double ex, double ey,
                                             double ez, double r2, size_t slot, unsigned *__restrict__ pj,
                                             D4 *__restrict__ pe, double2 *__restrict__ pg,
                                             const D4 *__restrict__ v, unsigned *__restrict__ err, double &rho,
                                             double &mxx, double &mxy, double &mxz, double &myy, double &myz,
                                             double &mzz, double &Sx, double &Sy, double &Sz) {
  const double rji = spline_eval<true>(P.tab_rho_r_sq + (size_t)ej * P.n_rho, P.inv_dr_sq, P.n_rho, r2, err);
  double rij = rji;
  if (MULTI && ej != ei)
    rij = spline_eval<true>(P.tab_rho_r_sq + (size_t)ei * P.n_rho, P.inv_dr_sq, P.n_rho, r2, err);
  // with M_i summed (FUSE_W) rho_i is its trace, sum_j H_ij r^2
  // (density_epilogue): one FP64 add per pair less
  if (!FUSE_W) rho += rji;
  pj[slot] = u;
  const double inv_r2 = recip_nr(r2);
  const double H = rji * inv_r2;
  const double hx = H * ex, hy = H * ey, hz = H * ez;
  if (FUSE_W && !MULTI) {
    // one element: H_ij = H_ji, and the force sweep takes the pair's
    // H e from here instead of multiplying by H per pair
    pe[slot] = D4{ex, ey, ez, hx};
    pg[slot] = make_double2(hy, hz);
  } else {
    pe[slot] = D4{ex, ey, ez, H};
    if (MULTI) pg[slot] = make_double2(rij * inv_r2, 0.0);
  }
  if (FUSE_W) {
    const D4 vj = v[u & IDX_MASK];
    mxx = fma(hx, ex, mxx);
    mxy = fma(hx, ey, mxy);
    mxz = fma(hx, ez, mxz);
    myy = fma(hy, ey, myy);
    myz = fma(hy, ez, myz);
    mzz = fma(hz, ez, mzz);
    const double d = dot3_fma(ex, ey, ez, vj.x, vj.y, vj.z);
    Sx = fma(d, hx, Sx);
    Sy = fma(d, hy, Sy);
    Sz = fma(d, hz, Sz);
  }
}

// e = x_j (periodic image of the pair code) - x_i, as the engine's ghost
// atoms give it: (x_j + image shift) - x_i
__device__ __forceinline__ void density_vector(const StepParams &P, const D4 &xi, const D4 &xj, unsigned code,
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

// atom i's deviates of this step: the device generator's or those given
__device__ __forceinline__ void atom_deviates(const StepParams &P, int i, const D4 *__restrict__ xi_given, int xi_mode,
                                              double *xi3) {
  if (xi_mode == 0) {
    gaussian3(P.seed, *P.step, (unsigned)i, xi3);
  } else {
    const D4 g = xi_given[i];
    xi3[0] = g.x;
    xi3[1] = g.y;
    xi3[2] = g.z;
  }
}

// what an atom's epilogue needs that does not depend on its pairs, where
// another warp of the block made it meanwhile
struct ReadyAtom {
  double xi[3], Te;
  int cell;
};

// The end of the density sweep for atom i (its pairs summed): alpha, beta,
// the deviates, its grid cell and T_e, and the per-atom records.
// With DFG (the df64 force sweep follows) the gathered records go to G as
// double-floats, 64 B per atom of which 48 are used: {W hi, X_x hi}, {W lo,
// X_x lo}, {X_y hi, X_z hi, X_y lo, X_z lo} (W = a_i w_i, X = a_i xi_i); an atom the
// reference skips as a neighbour (rho <= 0 or outside the group) is marked
// by a NaN in its first word.
template <bool FAST, bool FUSE_W, bool DFG = false>
__device__ __forceinline__ void density_epilogue(
    const StepParams &P, int i, bool active, const D4 &xi, int ei, double rho, int ns, double mxx, double mxy,
    double mxz, double myy, double myz, double mzz, double Sx, double Sy, double Sz,
    const D4 *__restrict__ xi_given, int xi_mode, const double *__restrict__ T_e, int *__restrict__ nshort,
    D4 *__restrict__ A, D4 *__restrict__ Bw, double *__restrict__ rho_out, double *__restrict__ beta_out,
    int *__restrict__ cell, double *__restrict__ Te_i, unsigned *__restrict__ err,
    unsigned long long *__restrict__ counters, const D4 *__restrict__ v, D4 *__restrict__ Mm,
    D4 *__restrict__ G, const ReadyAtom *ready = nullptr) {
  nshort[i] = ns;
  // FAST with M_i: rho_i = trace M_i = sum_j rho_j(r^2) / r^2 * r^2, within
  // the reciprocal's error (~6e-14) of the sum of rho_j(r^2)
  if (FAST && FUSE_W) rho = mxx + myy + mzz;
  // per-atom quantities
  double alpha = 0.0, beta = 0.0, xi3[3] = {0.0, 0.0, 0.0};
  if (active) {
    if (rho > P.rho_cutoff) {  // eph_beta.h:174-197
      atomicAdd(&counters[CNT_RHO_CUTOFF], 1ull);
    } else {
      beta = spline_eval<FAST>(P.tab_beta + (size_t)ei * P.n_beta, P.inv_drho, P.n_beta, rho, err);
      if (rho > 0) alpha = spline_eval<FAST>(P.tab_alpha + (size_t)ei * P.n_beta, P.inv_drho, P.n_beta, rho, err);
    }
    if (FAST && rho > 0) alpha = alpha / rho;
    if (P.flags & 0x02) {
      if (ready) {
        xi3[0] = ready->xi[0];
        xi3[1] = ready->xi[1];
        xi3[2] = ready->xi[2];
      } else {
        atom_deviates(P, i, xi_given, xi_mode, xi3);
      }
    }
    const int c = ready ? ready->cell : (int)grid_index(P, xi.x, xi.y, xi.z);
    cell[i] = c;
    Te_i[i] = ready ? ready->Te : T_e[c];
  }
  A[i] = D4{rho, alpha, xi3[0], xi3[1]};
  if (FUSE_W) {
    // w_i = a_i (M_i v_i - S_i), a_i = alpha_i/rho_i; k_friction_w's rule: w
    // stays 0 unless rho_i > 0.  For k_forces_m: M_i, and the records
    // G_i = {a_i w_i, a_i xi_i, rho_i} that the neighbours gather.
    double wx = 0.0, wy = 0.0, wz = 0.0;
    if (active && pos_double(rho)) {
      const D4 vi = v[i];
      wx = alpha * (fma(mxx, vi.x, fma(mxy, vi.y, mxz * vi.z)) - Sx);
      wy = alpha * (fma(mxy, vi.x, fma(myy, vi.y, myz * vi.z)) - Sy);
      wz = alpha * (fma(mxz, vi.x, fma(myz, vi.y, mzz * vi.z)) - Sz);
    }
    Bw[i] = D4{xi3[2], wx, wy, wz};
    Mm[i] = D4{mxx, mxy, mxz, myy};
    Mm[(size_t)P.n + i] = D4{myz, mzz, 0.0, 0.0};
    if (DFG) {
      const df64::df W[3] = {df64::from_double(alpha * wx), df64::from_double(alpha * wy),
                             df64::from_double(alpha * wz)};
      const df64::df X[3] = {df64::from_double(alpha * xi3[0]), df64::from_double(alpha * xi3[1]),
                             df64::from_double(alpha * xi3[2])};
      const bool live = active && pos_double(rho);
      float4 *g = reinterpret_cast<float4 *>(G) + 4 * (size_t)i;
      g[0] = make_float4(live ? W[0].hi : __int_as_float(0x7fc00000), W[1].hi, W[2].hi, X[0].hi);
      g[1] = make_float4(W[0].lo, W[1].lo, W[2].lo, X[0].lo);
      g[2] = make_float4(X[1].hi, X[2].hi, X[1].lo, X[2].lo);
    } else {
      G[2 * (size_t)i] = D4{alpha * wx, alpha * wy, alpha * wz, alpha * xi3[0]};
      G[2 * (size_t)i + 1] = D4{alpha * xi3[1], alpha * xi3[2], active ? rho : 0.0, 0.0};
    }
  } else {
    Bw[i] = D4{xi3[2], 0.0, 0.0, 0.0};
  }
  rho_out[i] = rho;
  beta_out[i] = beta;
}

// calculate_environment (fix_eph.cpp:431-466) plus everything per atom the
// later sweeps need.  One thread per atom, warps kept converged: a warp FP64
// instruction costs the same whether 1 or 32 lanes are active, so the FP64
// work must run in lockstep.
//   pass 1 (FP32/integer): candidates from the 27 bins around the atom with an
//     FP32 distance test padded by 1e-4 of rc^2, kept in shared memory in the
//     fixed bin-stencil order of index-sorted bins (EXACT: k_density_exact, in
//     ascending neighbour index, the order of the reference's list)
//   pass 2 (FP64): the exact test r^2 < rc^2 with e = (x_j + image) - x_i, the
//     density sum, and the pair cache of the in-cutoff pairs
// Pair cache row k of atom i sits at k*n + i (coalesced across the warp):
//   pj: neighbour index | image code << 27
//   pe: e_ij and (EXACT) r^2 or (FAST) rho_j(r^2)/r^2
//   pg: (EXACT) rho_j(r^2), rho_i(r^2); (FAST, several elements) rho_i(r^2)/r^2
// A[i] = {rho_i, alpha_i (EXACT) | alpha_i/rho_i (FAST), xi_x, xi_y}
// Bw[i] = {xi_z, w_i} (w written by the friction sweep, or here with FUSE_W)
// Candidates: the first CAND_SMEM rows of an atom live in shared memory
// ([CAND_SMEM][blockDim]), further ones in the atom's own rows of pj (read
// back before pass 2 overwrites them: pair slot <= candidate slot).
// FUSE_W (FAST mode, one lane per atom): the friction pre-vector of stage 1
// in the same pass — it needs only this atom's density, so its sums ride
// along with rho and the separate sweep over the pair cache is saved:
// M_i = sum_j H_ij e e^T and S_i = sum_j H_ij (e.v_j) e (H_ij = rho_j(r^2)/r^2),
// then w_i = (alpha_i / rho_i) (M_i v_i - S_i).  It also leaves M_i and the
// records G_i = {a_i w_i, a_i xi_i, rho_i} for k_forces_m.
template <bool MULTI, bool FUSE_W = false>
__global__ void __launch_bounds__(128) k_density(
    StepParams P, const D4 *__restrict__ x, const int *__restrict__ mask, const int *__restrict__ bin_count,
    const BinEntry *__restrict__ bins, const int4 *__restrict__ atom_bin, const float4 *__restrict__ atom_off,
    const D4 *__restrict__ xi_given, int xi_mode, const double *__restrict__ T_e, unsigned *__restrict__ pj,
    D4 *__restrict__ pe, double2 *__restrict__ pg, int *__restrict__ nshort, D4 *__restrict__ A,
    D4 *__restrict__ Bw, double *__restrict__ rho_out, double *__restrict__ beta_out, int *__restrict__ cell,
    double *__restrict__ Te_i, int *__restrict__ wrapflag, unsigned *__restrict__ err,
    unsigned long long *__restrict__ counters, const D4 *__restrict__ v = nullptr, D4 *__restrict__ Mm = nullptr,
    D4 *__restrict__ G = nullptr) {
  __shared__ unsigned s_cand[CAND_SMEM * 128];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int t = threadIdx.x, nt = blockDim.x;
  if (i == 0) *wrapflag = 0;  // the binning kernel has read it
  const bool valid = i < P.n;
  const bool active = valid && (mask[i] & P.groupbit) != 0;
  auto cget = [&](int k) -> unsigned { return k < CAND_SMEM ? s_cand[k * nt + t] : pj[(size_t)k * P.n + i]; };
  auto cset = [&](int k, unsigned u) {
    if (k < CAND_SMEM)
      s_cand[k * nt + t] = u;
    else
      pj[(size_t)k * P.n + i] = u;
  };
  D4 xi = D4{0.0, 0.0, 0.0, 0.0};
  if (valid) xi = x[i];
  const int ei = (int)xi.w;
  double rho = 0.0;
  int ns = 0, nc = 0;
  // pass 1: candidates, FP32/integer work only, warp-uniform loop bounds
  {
    int4 Bi = make_int4(0, 0, 0, 0);
    float4 oi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (active) {
      Bi = atom_bin[i];
      oi = atom_off[i];
    }
    nc = collect_candidates(P, i, active, Bi, oi, bin_count, bins, err, cset, P.rc2_band, P.kcap);
  }
  __syncwarp();
  // pass 2: exact FP64 test, density and pair cache, in lockstep
  // FUSE_W: M_i = sum_j H_ij e e^T over all pairs and S_i = sum_j H_ij (e.v_j) e
  double Sx = 0.0, Sy = 0.0, Sz = 0.0;
  double mxx = 0.0, mxy = 0.0, mxz = 0.0, myy = 0.0, myz = 0.0, mzz = 0.0;
  const int nmax = __reduce_max_sync(0xffffffffu, nc);
  for (int k = 0; k < nmax; ++k) {
    if (k < nc) {
      const unsigned u = cget(k);
      const D4 xj = x[u & IDX_MASK];
      double ex, ey, ez;
      density_vector(P, xi, xj, u >> IDX_BITS, ex, ey, ez);
      const double r2 = dot3_fma(ex, ey, ez, ex, ey, ez);
      if (below(r2, P.rc2)) {  // r2 >= 0
        density_pair<MULTI, FUSE_W>(P, ei, u, (int)xj.w, ex, ey, ez, r2, (size_t)ns * P.n + i, pj, pe, pg,
                                          v, err, rho, mxx, mxy, mxz, myy, myz, mzz, Sx, Sy, Sz);
        ++ns;
      }
    }
  }
  if (!valid) return;
  density_epilogue<true, FUSE_W>(P, i, active, xi, ei, rho, ns, mxx, mxy, mxz, myy, myz, mzz, Sx, Sy, Sz, xi_given,
                                 xi_mode, T_e, nshort, A, Bw, rho_out, beta_out, cell, Te_i, err, counters, v, Mm, G);
}

// The density sweep of EXACT mode, L lanes per atom: the lanes search
// the 27 bins together, sort the atom's candidates by neighbour index (each
// counts the smaller ones of its own, then writes them to their places), test
// and cache the pairs, compacted in that order; one thread per atom, in the
// block's first threads, then adds the densities in the same order and
// finishes the atom.  Candidate k is kept in shared memory for k < EXD_CAP;
// further ones wait in the atom's rows of pj, and in order in the first word
// of its rows of pe: row k is read, in step, before the pair rows up to k are
// written.
// Latency and issue bind it (FP64 pipe half busy).  One lane per atom inserted
// each candidate into its place through shared memory, a serial chain.
// GB300, us per step: 2,048 atoms 377 -> 31, 62,500 atoms 424 -> 205.
constexpr int EXD_THREADS = 256;
constexpr int EXD_CAP = 72;  // a row stride of 8 banks: the lanes of 4 atoms in distinct banks
template <bool MULTI, int L>
__global__ void __launch_bounds__(EXD_THREADS, 4) k_density_exact(
    StepParams P, const D4 *__restrict__ x, const int *__restrict__ mask, const int *__restrict__ bin_count,
    const BinEntry *__restrict__ bins, const int4 *__restrict__ atom_bin, const float4 *__restrict__ atom_off,
    const D4 *__restrict__ xi_given, int xi_mode, const double *__restrict__ T_e, unsigned *__restrict__ pj,
    D4 *__restrict__ pe, double2 *__restrict__ pg, int *__restrict__ nshort, D4 *__restrict__ A,
    D4 *__restrict__ Bw, double *__restrict__ rho_out, double *__restrict__ beta_out, int *__restrict__ cell,
    double *__restrict__ Te_i, int *__restrict__ wrapflag, unsigned *__restrict__ err,
    unsigned long long *__restrict__ counters) {
  constexpr int NA = EXD_THREADS / L, CAP = EXD_CAP;
  __shared__ unsigned s_found[NA * CAP], s_sorted[NA * CAP];
  __shared__ int s_ns[NA];
  const int t = threadIdx.x, a = t / L, g = t & (L - 1), lane = t & 31;
  const int i = blockIdx.x * NA + a;
  if (blockIdx.x == 0 && t == 0) *wrapflag = 0;  // the binning kernel has read it
  const bool active = i < P.n && (mask[i] & P.groupbit) != 0;
  unsigned *found = s_found + a * CAP, *sorted = s_sorted + a * CAP;
  auto place = [&](int k) -> unsigned & { return k < CAP ? found[k] : pj[(size_t)k * P.n + i]; };
  auto in_order = [&](int k) -> unsigned & {
    return k < CAP ? sorted[k] : *reinterpret_cast<unsigned *>(pe + (size_t)k * P.n + i);
  };
  int nc = 0;
  {
    int4 Bi = make_int4(0, 0, 0, 0);
    float4 oi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (active) {
      Bi = atom_bin[i];
      oi = atom_off[i];
    }
    auto set = [&](int k, unsigned u) { place(k) = u; };
    shared_candidates<L>(P, i, active, Bi, oi, bin_count, bins, err, nc, P.kcap, set, P.rc2_band);
  }
  __syncwarp();
  const int nmax = __reduce_max_sync(0xffffffffu, nc);
  // an atom's candidates are distinct atoms: a box has at least three bins
  // along every axis
  for (int m = g; m - g < nmax; m += 4 * L) {
    unsigned u[4], key[4];
    int rank[4] = {0, 0, 0, 0};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      u[q] = m + q * L < nc ? place(m + q * L) : 0u;
      key[q] = u[q] & IDX_MASK;
    }
    for (int k = 0; k < nc; ++k) {
      const unsigned other = place(k) & IDX_MASK;
#pragma unroll
      for (int q = 0; q < 4; ++q) rank[q] += other < key[q] ? 1 : 0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (m + q * L < nc) in_order(rank[q]) = u[q];
  }
  __syncwarp();
  D4 xi = D4{0.0, 0.0, 0.0, 0.0};
  if (active) xi = x[i];
  const int ei = (int)xi.w;
  int ns = 0;
  for (int k = g; k - g < nmax; k += L) {
    bool in = false;
    unsigned u = 0;
    D4 xj = D4{0.0, 0.0, 0.0, 0.0};
    double ex = 0.0, ey = 0.0, ez = 0.0, r2 = 0.0;
    if (k < nc) {
      u = in_order(k);
      xj = x[u & IDX_MASK];
      density_vector(P, xi, xj, u >> IDX_BITS, ex, ey, ez);
      r2 = dot3(ex, ey, ez, ex, ey, ez);
      in = below(r2, P.rc2);  // r2 >= 0
    }
    const unsigned who = (__ballot_sync(0xffffffffu, in) >> (lane & ~(L - 1))) & ((1u << L) - 1u);
    if (in) {
      const size_t slot = (size_t)(ns + __popc(who & ((1u << g) - 1u))) * P.n + i;
      const int ej = (int)xj.w;
      const double rji = spline_eval<false>(P.tab_rho_r_sq + (size_t)ej * P.n_rho, P.inv_dr_sq, P.n_rho, r2, err);
      double rij = rji;
      if (MULTI && ej != ei)
        rij = spline_eval<false>(P.tab_rho_r_sq + (size_t)ei * P.n_rho, P.inv_dr_sq, P.n_rho, r2, err);
      pj[slot] = u;
      pe[slot] = D4{ex, ey, ez, r2};
      pg[slot] = make_double2(rji, rij);
    }
    ns += __popc(who);
  }
  if (g == 0) s_ns[a] = ns;
  __syncthreads();
  if (t >= NA) return;
  const int o = blockIdx.x * NA + t;
  if (o >= P.n) return;
  ns = s_ns[t];
  double rho = 0.0;
#pragma unroll 8
  for (int k = 0; k < ns; ++k) rho += pg[(size_t)k * P.n + o].x;
  const D4 xo = x[o];
  density_epilogue<false, false>(P, o, (mask[o] & P.groupbit) != 0, xo, (int)xo.w, rho, ns, 0.0, 0.0, 0.0, 0.0, 0.0,
                                 0.0, 0.0, 0.0, 0.0, xi_given, xi_mode, T_e, nshort, A, Bw, rho_out, beta_out, cell,
                                 Te_i, err, counters, nullptr, nullptr, nullptr);
}

// ------------------------------------------- FAST pair sweeps in df64

// resident blocks of 128 threads per SM the df64 sweeps are compiled for
// (their register budget: 65,536 / (128 x blocks)); measured on GB300 at
// 2,048,000 atoms: density 6 / 7 / 8 blocks 1.44 / 1.36 / 1.69 ms (8 spills),
// forces 8 / 9 blocks 0.86 / 0.80 ms
#ifndef EPH_DF_DENSITY_BLOCKS
#define EPH_DF_DENSITY_BLOCKS 7
#endif
#ifndef EPH_DF_FORCES_BLOCKS
#define EPH_DF_FORCES_BLOCKS 9
#endif

// The FAST density sweep with TPA lanes per atom for small systems (FP64 pair
// terms), where one lane per atom leaves the SMs a few warps each.  The
// lanes search the 27 bins together and leave the atom's pairs -- the
// candidates sure to be inside the cut-off by their FP32 distance, and those
// within its error of the cut-off that pass the FP64 test -- in one list in
// shared memory, whose entry k is row k of the pair cache; then lane g sums
// rows g, g + TPA, ....  Meanwhile the block's last warps draw the atoms'
// deviates and find their grid cells; the lanes' sums meet in shared memory
// and one thread per atom, in the block's first threads, finishes the atom.
// Sums in a fixed order (the same every run), within rounding of the one-lane
// sweep.
// FP64 issue and latency bound it: a warp FP64 instruction takes 16 cycles of
// the SM's pipe however few lanes are active, so what counts is full warps
// and short chains.  GB300, us per launch at 4,000 atoms: 90 with the lanes'
// own candidates (half the iterations idle, an extra pass for the exact
// test) and everything per atom on every eighth lane; 33 now (16 lanes).
constexpr int tpa_threads(int tpa) { return 128 + (128 / tpa + 31) / 32 * 32; }
template <bool MULTI, bool FUSE_W, int TPA>
__global__ void __launch_bounds__(tpa_threads(TPA)) k_density_tpa(
    StepParams P, const D4 *__restrict__ x, const int *__restrict__ mask, const int *__restrict__ bin_count,
    const BinEntry *__restrict__ bins, const int4 *__restrict__ atom_bin, const float4 *__restrict__ atom_off,
    const D4 *__restrict__ xi_given, int xi_mode, const double *__restrict__ T_e, unsigned *__restrict__ pj,
    D4 *__restrict__ pe, double2 *__restrict__ pg, int *__restrict__ nshort, D4 *__restrict__ A,
    D4 *__restrict__ Bw, double *__restrict__ rho_out, double *__restrict__ beta_out, int *__restrict__ cell,
    double *__restrict__ Te_i, int *__restrict__ wrapflag, unsigned *__restrict__ err,
    unsigned long long *__restrict__ counters, const D4 *__restrict__ v, D4 *__restrict__ Mm,
    D4 *__restrict__ G, const unsigned *__restrict__ elist, const int *__restrict__ ens,
    const int4 *__restrict__ rec) {
  constexpr int NA = 128 / TPA;  // atoms per block
  constexpr int NSUM = FUSE_W ? 9 : 1;
  __shared__ __align__(16) unsigned s_cand[NA * (KMAX + 1)];
  __shared__ double s_sum[NSUM * 128];
  double *s_tot = reinterpret_cast<double *>(s_cand);  // [NSUM][NA], once the lists are read
  __shared__ ReadyAtom s_ready[NA];
  __shared__ int s_ns[NA];
  const int t = threadIdx.x, a = t / TPA, g = t % TPA;
  if (blockIdx.x == 0 && t == 0) *wrapflag = 0;  // the binning kernel has read it
  if (t >= 128) {  // the last warps: what does not depend on the pairs
    const int r = t - 128, o = blockIdx.x * NA + r;
    if (r < NA && o < P.n && (mask[o] & P.groupbit)) {
      ReadyAtom w{{0.0, 0.0, 0.0}, 0.0, 0};
      const D4 xo = x[o];
      w.cell = (int)grid_index(P, xo.x, xo.y, xo.z);
      w.Te = T_e[w.cell];
      if (P.flags & 0x02) atom_deviates(P, o, xi_given, xi_mode, w.xi);
      s_ready[r] = w;
    }
    __syncthreads();
    __syncthreads();
    return;
  }
  const int i = blockIdx.x * NA + a;
  const bool valid = i < P.n;
  const bool active = valid && (mask[i] & P.groupbit) != 0;
  unsigned *list = s_cand + a * (KMAX + 1);
  D4 xi = D4{0.0, 0.0, 0.0, 0.0};
  if (valid) xi = x[i];
  const int ei = (int)xi.w;
  int ns = 0;
  {
    int4 Bi = make_int4(0, 0, 0, 0);
    float4 oi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (active) {
      Bi = atom_bin[i];
      oi = atom_off[i];
    }
    const float sure = (float)(P.rc2 * (1.0 - 1e-4));
    auto set = [&](int k, unsigned u) { list[k] = u; };
    auto inside = [&](unsigned u, float r2) {
      if (r2 < sure) return true;
      double ex, ey, ez;
      density_vector(P, xi, x[u & IDX_MASK], u >> IDX_BITS, ex, ey, ez);
      return below(dot3_fma(ex, ey, ez, ex, ey, ez), P.rc2);
    };
    if (elist) {  // the engine's EAM pair list of this step
      long long xf[3] = {0, 0, 0};
      if (valid) own_fixed(rec, i, xf);
      list_candidates<TPA>(P, i, active, xf, elist, ens, rec, err, ns, P.kcap, set, P.rc2_band, inside);
    } else {
      shared_candidates<TPA>(P, i, active, Bi, oi, bin_count, bins, err, ns, P.kcap, set, P.rc2_band, nullptr, -1.f,
                             inside);
    }
  }
  __syncwarp();
  double rho = 0.0, Sx = 0.0, Sy = 0.0, Sz = 0.0;
  double mxx = 0.0, mxy = 0.0, mxz = 0.0, myy = 0.0, myz = 0.0, mzz = 0.0;
  unsigned u_next = g < ns ? list[g] : 0u;
  D4 x_next = xi;
  if (g < ns) x_next = x[u_next & IDX_MASK];
  for (int k = g; k < ns; k += TPA) {
    const unsigned u = u_next;
    const D4 xj = x_next;
    if (k + TPA < ns) {  // the next neighbour's position while this pair is summed
      u_next = list[k + TPA];
      x_next = x[u_next & IDX_MASK];
    }
    double ex, ey, ez;
    density_vector(P, xi, xj, u >> IDX_BITS, ex, ey, ez);
    const double r2 = dot3_fma(ex, ey, ez, ex, ey, ez);
    density_pair<MULTI, FUSE_W>(P, ei, u, (int)xj.w, ex, ey, ez, r2, (size_t)k * P.n + i, pj, pe, pg, v, err,
                                      rho, mxx, mxy, mxz, myy, myz, mzz, Sx, Sy, Sz);
  }
  // sum q of the atom's lane l at q * 128 + l * NA + (atom): the finishing
  // threads read neighbouring words
  const int at = g * NA + a;
  if (FUSE_W) {
    const double m[9] = {mxx, mxy, mxz, myy, myz, mzz, Sx, Sy, Sz};
#pragma unroll
    for (int q = 0; q < NSUM; ++q) s_sum[q * 128 + at] = m[q];
  } else {
    s_sum[at] = rho;
  }
  if (g == 0) s_ns[a] = ns;
  __syncthreads();
  for (int q = t; q < NSUM * NA; q += 128) {  // sum q / NA of atom q % NA
    const double *w = s_sum + q / NA * 128 + q % NA;
    double sum = w[0];
#pragma unroll
    for (int l = 1; l < TPA; ++l) sum += w[l * NA];
    s_tot[q] = sum;
  }
  __syncthreads();
  const int o = blockIdx.x * NA + t;
  if (t >= NA || o >= P.n) return;
  double m[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) m[q] = q < NSUM ? s_tot[q * NA + t] : 0.0;
  const D4 xo = x[o];
  density_epilogue<true, FUSE_W>(P, o, (mask[o] & P.groupbit) != 0, xo, (int)xo.w, m[0], s_ns[t], m[0], m[1], m[2],
                                 m[3], m[4], m[5], m[6], m[7], m[8], xi_given, xi_mode, T_e, nshort, A, Bw, rho_out,
                                 beta_out, cell, Te_i, err, counters, v, Mm, G, s_ready + t);
}

// ------------------------------------------------ candidate-list reuse

// FAST mode, one lane per atom.  The candidates of atom i within r_list =
// r_cutoff + s (s the list skin) are kept from a build step on: while atoms
// i and j both moved less than s/2 since the build, |x_i - x_j| < r_cutoff
// implies that j is in i's list.  Atoms that moved farther ("moved", at most
// LIST_FMAX of them) are handled every step instead: they and every atom
// within r_cutoff + s/2 of one of them search the bins of the build afresh
// (the df64 sweeps: see pair_candidates), leave moved atoms' bin entries out
// and take the moved atoms as extra candidates.  More moved atoms, or a request from the host,
// make the step a build step.  Decisions live on the device (rb[0] build
// requested, rb[1] moved atoms this step, rb[2] this step builds, rb[3] the lists
// are of the group's atoms only, which a step with a pair force makes anew), so a
// captured step replays them.  Lists hold atom indices; the periodic image of
// a pair is the minimum image of the current positions, decided in FP32 (the
// box is at least three list radii wide, so it is the image within the
// cutoff), and e = (x_j +- L) - x_i rounds as the engine's ghost atoms give
// it.

// First kernel of a step with list reuse: the engine's wrap (as k_bin does
// it), then each atom's displacement since the list build; moved atoms get
// state 2 and join the list of moved atoms (state 0 otherwise).  With RECORDS
// (the df64 sweeps), also every atom's record for them and whether it moved.
// The boxes added to a record's position are those of the image next to the
// position at the build (so the image codes of the lists' entries stay what
// they were), or, for an atom that moved, of the image in the box (the codes
// of the searches around it are found there).  With RECORDS the displacement's
// images and square are FP32 work, against a threshold lowered by their error
// (an atom may count as moved a hair early, never late): three differences
// and the velocities' split are all that is left in FP64.  FP64 issue bound it before (83%
// of that pipe), memory does now: GB300, 2,048,000 atoms: 169 -> 76 us.
template <bool RECORDS>
__global__ void k_list_check(StepParams P, D4 *__restrict__ x, D4 *__restrict__ xhold,
                             const int *__restrict__ wrapflag, const D4 *__restrict__ xref, int *__restrict__ state,
                             int *__restrict__ rb, int *__restrict__ flist, unsigned long long *__restrict__ counters,
                             int4 *__restrict__ rec, const D4 *__restrict__ v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *P.step += 1ull;  // read by the density sweep that follows
  bool moved = false;
  if (i < P.n) {
    D4 xi = x[i];
    if (*wrapflag) {
      wrap_into_box(P, xi);
      x[i] = xi;
      xhold[i] = xi;
      if (i == 0) atomicAdd(&counters[CNT_WRAP], 1ull);
    }
    const D4 r = xref[i];
    if (RECORDS) {
      const double now[3] = {xi.x, xi.y, xi.z}, d[3] = {xi.x - r.x, xi.y - r.y, xi.z - r.z};
      long long f[3];
      int image[3];
      float r2 = 0.0f;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        f[k] = to_fixed_coord(now[k], P.fix_q);
        const float df = float_bits(d[k]), half = P.half_prdf[k];
        image[k] = df > half ? -1 : (df < -half ? 1 : 0);
        const float e = df + (float)(2 * image[k]) * half;
        r2 += e * e;
      }
      moved = !(r2 < P.lslow2_band);
      if (moved) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          double q;
          image[k] = wrap_image(P, k, now[k], q);
        }
      }
      df_record_fixed(P, i, f, (int)trunc_index(xi.w), image, moved, v[i], rec);
    } else {
      const double dx = min_image(xi.x - r.x, P.prd[0], P.half_prd[0]),
                   dy = min_image(xi.y - r.y, P.prd[1], P.half_prd[1]),
                   dz = min_image(xi.z - r.z, P.prd[2], P.half_prd[2]);
      moved = dx * dx + dy * dy + dz * dz >= P.lslow2;
    }
    state[i] = moved ? 2 : 0;
  }
  // one atomic per warp (after a long run without a build most atoms move)
  const unsigned mv = __ballot_sync(0xffffffffu, moved);
  if (mv) {
    const int lane = threadIdx.x & 31, lead = __ffs(mv) - 1;
    int base = 0;
    if (lane == lead) base = atomicAdd(&rb[1], __popc(mv));
    base = __shfl_sync(0xffffffffu, base, lead);
    const int k = base + __popc(mv & ((1u << lane) - 1u));
    if (moved && k < LIST_FMAX) flist[k] = i;
  }
}

// One warp: build or not, and the moved atoms in index order (they were
// appended in any order; the order of the extra candidates must not change
// from run to run).
__global__ void k_list_decide(int *__restrict__ rb, int *__restrict__ flist,
                              unsigned long long *__restrict__ counters, bool pair_force) {
  const int lane = threadIdx.x;
  const int cnt = rb[1];
  const bool build = rb[0] != 0 || (pair_force && rb[3] != 0) || cnt > LIST_FMAX;
  if (!build && cnt > 1) {
    const int v = lane < cnt ? flist[lane] : 0x7fffffff;
    int rank = 0;
    for (int s = 0; s < 32; ++s) rank += __shfl_sync(0xffffffffu, v, s) < v;
    __syncwarp();
    if (lane < cnt) flist[rank] = v;
  }
  if (lane == 0) {
    rb[2] = build ? 1 : 0;
    rb[0] = 0;
    if (build) {
      rb[3] = 0;
      atomicAdd(&counters[CNT_BUILD], 1ull);
    }
  }
}

// On a build step: clears the bins.  Otherwise block b: moved atom flist[b]
// flags (state |= 1) every atom whose position at the build lies within
// r_cutoff + s/2 of its current position -- the only unmoved atoms it can now
// be within r_cutoff of -- and leaves its position wrapped into the box, which
// those atoms compare with.  One thread wraps (a division per axis: FP64 issue,
// 16 cycles for each warp that would repeat it).
__global__ void __launch_bounds__(512) k_list_mark(StepParams P, const D4 *__restrict__ x, const int *__restrict__ rb,
                                                   const int *__restrict__ flist, int *__restrict__ bin_count,
                                                   int nbins, const BinEntry *__restrict__ bins,
                                                   int *__restrict__ state, D4 *__restrict__ fpos) {
  if (rb[2]) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < nbins) bin_count[q] = 0;
    return;
  }
  if ((int)blockIdx.x >= rb[1]) return;
  __shared__ int4 s_B;
  __shared__ float4 s_o;
  if (threadIdx.x == 0) {
    double wrapped[3];
    int4 B;
    float4 o;
    current_bin(P, x[flist[blockIdx.x]], B, o, wrapped);
    fpos[blockIdx.x] = D4{wrapped[0], wrapped[1], wrapped[2], 0.0};
    s_B = B;
    s_o = o;
  }
  __syncthreads();
  const int4 B = s_B;
  const float4 o = s_o;
  const int per = 27 * P.bcap;
  for (int q = threadIdx.x; q < per; q += blockDim.x) {
    const int slot = q % P.bcap, b = q / P.bcap;
    const int dx = b % 3 - 1, dy = (b / 3) % 3 - 1, dz = b / 9 - 1;
    const int Tx = B.x + dx, Ty = B.y + dy, Tz = B.z + dz;
    const int tx = Tx < 0 ? Tx + P.nb[0] : (Tx >= P.nb[0] ? Tx - P.nb[0] : Tx);
    const int ty = Ty < 0 ? Ty + P.nb[1] : (Ty >= P.nb[1] ? Ty - P.nb[1] : Ty);
    const int tz = Tz < 0 ? Tz + P.nb[2] : (Tz >= P.nb[2] ? Tz - P.nb[2] : Tz);
    const int flat = tx + P.nb[0] * (ty + P.nb[1] * tz);
    const int cnt = min(bin_count[flat], P.bcap);
    if (slot >= cnt) continue;
    const BinEntry e = bins[(size_t)flat * P.bcap + slot];
    const float ex = ((float)dx * P.wf[0] - o.x) + e.ox;
    const float ey = ((float)dy * P.wf[1] - o.y) + e.oy;
    const float ez = ((float)dz * P.wf[2] - o.z) + e.oz;
    if (ex * ex + ey * ey + ez * ez < P.rmark2_band) atomicOr(&state[e.idx & IDX_MASK], 1);
  }
}

// k_density (FAST, stage 1 and M_i folded in) over the kept candidate lists:
// on a build step pass 1 searches the bins within r_list for every atom and
// writes the lists (rows k * n + i of cl, counts in cl_n); otherwise an atom
// reads its list, except the atoms flagged by k_list_check / k_list_mark,
// which search the bins of the build afresh (their candidates in shared
// memory, spilling into their pj rows as in k_density) and add the moved
// atoms.  Pass 2 and the epilogue are k_density's.
// (128 threads a block; 64 registers as k_density has: with
// __launch_bounds__(128) ptxas settled on 56 and spilled)
template <bool MULTI>
__global__ void __maxnreg__(64) k_density_list(
    StepParams P, const D4 *__restrict__ x, const int *__restrict__ mask, const int *__restrict__ bin_count,
    const BinEntry *__restrict__ bins, const int4 *__restrict__ atom_bin, const float4 *__restrict__ atom_off,
    const D4 *__restrict__ xi_given, int xi_mode, const double *__restrict__ T_e, unsigned *__restrict__ pj,
    D4 *__restrict__ pe, double2 *__restrict__ pg, int *__restrict__ nshort, D4 *__restrict__ A,
    D4 *__restrict__ Bw, double *__restrict__ rho_out, double *__restrict__ beta_out, int *__restrict__ cell,
    double *__restrict__ Te_i, int *__restrict__ wrapflag, unsigned *__restrict__ err,
    unsigned long long *__restrict__ counters, const D4 *__restrict__ v, D4 *__restrict__ Mm, D4 *__restrict__ G,
    unsigned *__restrict__ cl, int *__restrict__ cl_n, const int *__restrict__ state, const int *__restrict__ rb,
    const int *__restrict__ flist) {
  __shared__ unsigned s_cand[CAND_SMEM * 128];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int t = threadIdx.x, nt = blockDim.x;
  if (i == 0) *wrapflag = 0;  // k_list_check has read it
  const bool valid = i < P.n;
  const bool active = valid && (mask[i] & P.groupbit) != 0;
  const size_t n = (size_t)P.n;
  auto sset = [&](int k, unsigned u) {
    if (k < CAND_SMEM)
      s_cand[k * nt + t] = u;
    else
      pj[(size_t)k * n + i] = u;
  };
  // build steps: the list rows, their first CAND_SMEM also in shared memory
  auto lset = [&](int k, unsigned u) {
    if (k < CAND_SMEM) s_cand[k * nt + t] = u;
    cl[(size_t)k * n + i] = u;
  };
  D4 xi = D4{0.0, 0.0, 0.0, 0.0};
  if (valid) xi = x[i];
  const int ei = (int)xi.w;
  const bool build = rb[2] != 0;
  int nc = 0;
  bool fresh = false;
  if (build) {
    int4 Bi = make_int4(0, 0, 0, 0);
    float4 oi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (active) {
      Bi = atom_bin[i];
      oi = atom_off[i];
    }
    // the candidates inside the cut-off first, the shell out to r_list after
    // them: the shell's pairs mostly fail the exact test, and at the end of
    // the lists whole warps skip them
    nc = collect_candidates(P, i, active, Bi, oi, bin_count, bins, err, lset, P.rc2_band, P.lcap);
    nc = collect_candidates(P, i, active, Bi, oi, bin_count, bins, err, lset, P.rl2_band, P.lcap,
                                  nullptr, P.rc2_band, nc);
    if (valid) cl_n[i] = nc;
  } else {
    const int st = active ? state[i] : 0;
    fresh = st != 0;
    if (__any_sync(0xffffffffu, fresh)) {
      int4 Bi = make_int4(0, 0, 0, 0);
      float4 oi = make_float4(0.f, 0.f, 0.f, 0.f);
      if (fresh) {
        if (st & 2) {
          current_bin(P, xi, Bi, oi);
        } else {
          Bi = atom_bin[i];
          oi = atom_off[i];
        }
      }
      nc = collect_candidates<true>(P, i, fresh, Bi, oi, bin_count, bins, err, sset, P.rl2_band, P.kcap,
                                          state);
      // the moved atoms near enough (a widened test; pass 2 decides)
      const int nf = rb[1];  // <= LIST_FMAX on a step without a build
      for (int q = 0; q < nf; ++q) {
        const int f = flist[q];
        if (fresh && f != i) {
          const D4 xf = x[f];
          const double dx = min_image(xf.x - xi.x, P.prd[0], P.half_prd[0]);
          const double dy = min_image(xf.y - xi.y, P.prd[1], P.half_prd[1]);
          const double dz = min_image(xf.z - xi.z, P.prd[2], P.half_prd[2]);
          if (dx * dx + dy * dy + dz * dz < P.rc2 * (1.0 + 1e-4)) {
            if (nc < P.kcap)
              sset(nc++, (unsigned)f | (CODE_NOSHIFT << IDX_BITS));
            else
              atomicOr(err, ERR_PAIR_OVERFLOW);
          }
        }
      }
    }
    if (active && !fresh) {
      // the list's head into shared memory: independent loads up front
      // instead of one DRAM round trip in front of every pair
      nc = cl_n[i];
      const int nh = nc < CAND_SMEM ? nc : CAND_SMEM;
#pragma unroll 8
      for (int k = 0; k < nh; ++k) s_cand[k * nt + t] = __ldcs(cl + (size_t)k * n + i);  // read once a step
    }
  }
  __syncwarp();
  // candidate k: shared memory, then the list rows (or, for an atom that
  // searched afresh, its pj rows)
  const unsigned *__restrict__ tail = fresh ? pj : cl;
  double rho = 0.0, Sx = 0.0, Sy = 0.0, Sz = 0.0;
  double mxx = 0.0, mxy = 0.0, mxz = 0.0, myy = 0.0, myz = 0.0, mzz = 0.0;
  int ns = 0;
  // pass 2: the image of each candidate from FP32 copies of the positions
  // (integer and FP32 work), then k_density's FP64 work per pair
  const float xif = float_bits(xi.x), yif = float_bits(xi.y), zif = float_bits(xi.z);
  const int nmax = __reduce_max_sync(0xffffffffu, nc);
  for (int k = 0; k < nmax; ++k) {
    if (k < nc) {
      const unsigned j = (k < CAND_SMEM ? s_cand[k * nt + t] : __ldcs(tail + (size_t)k * n + i)) & IDX_MASK;
      const D4 xj = x[j];
      const unsigned code = image_code(P, xif, yif, zif, xj);
      double ex, ey, ez;
      density_vector(P, xi, xj, code, ex, ey, ez);
      const double r2 = dot3_fma(ex, ey, ez, ex, ey, ez);
      if (below(r2, P.rc2)) {
        if (ns < P.kcap)
          density_pair<MULTI, true>(P, ei, j | (code << IDX_BITS), (int)xj.w, ex, ey, ez, r2,
                                          (size_t)ns * n + i, pj, pe, pg, v, err, rho, mxx, mxy, mxz, myy, myz, mzz,
                                          Sx, Sy, Sz);
        else
          atomicOr(err, ERR_PAIR_OVERFLOW);
        ++ns;
      }
    }
  }
  if (!valid) return;
  density_epilogue<true, true>(P, i, active, xi, ei, rho, ns < P.kcap ? ns : P.kcap, mxx, mxy, mxz, myy, myz, mzz, Sx, Sy, Sz, xi_given,
                               xi_mode, T_e, nshort, A, Bw, rho_out, beta_out, cell, Te_i, err, counters, v, Mm, G);
}

// ------------------------------------------- FAST density sweep in df64
//
// calculate_environment (fix_eph.cpp:431-466), stage 1 and M_i in one pass
// (the FAST density sweep of k_density<MULTI, true>) with every
// per-pair operation in df64 on the FP32 pipe and LANES lanes per atom.
//   pass 1 gathers the atom's candidates into shared memory (its lanes share
//     one list): DF_BINS searches the 27 bins of the step, DF_EAM takes them
//     from the EAM engine's pair list, DF_LIST keeps lists (pair_candidates);
//   pass 2 forms e from the fixed-point positions (pair_fixed, fixed_df), r^2,
//     the cut-off test, rho_j(r^2) (spline_rho_df), H = rho_j(r^2) / r^2 and the
//     sums of M_i and S_i (blocked df64 sums: 8 products, then a Dekker
//     addition into the totals in shared memory), lane g taking candidates g,
//     g + LANES, ...; a candidate outside the cut-off is evaluated at r^2 = 1
//     with H forced to 0, so its terms add exact zeros and it writes no pair;
//   the epilogue (density_epilogue, FP64) runs on one thread per atom in the
//     block's first warps, whatever LANES is.
// Pair cache (row k of atom i at k*n + i): pj = neighbour | image code << 27,
// pe = {e hi, H_ji hi}, {the lo parts} (H_ji = rho_i(r^2) / r^2, the weight
// of the neighbour's term in the force sweep): 36 B per pair.  H e, which the
// cache used to hold too (52 B), costs the force sweep two multiplications.
//
// What bounds it on GB300, in the order it was taken away (2,048,000 atoms,
// kept lists, ms per launch): 1.98 at the start, with the L1 at 68 % of its
// wavefront rate (every 16-byte load of a scattered record touches a line per
// lane), 500 instructions per candidate and little L1 left beside the
// candidates in shared memory.  Fixed-point positions whose image the list
// keeps (no bins to unpack, no image test) and 36 B instead of 52 B per cached
// pair: 420 instructions, but 2.03 until the loads changed; 256-bit loads of
// record halves and table rows: 1.84; lists read from global memory two
// candidates ahead, so that the L1 keeps the table and records: 1.47; the
// division-free grid cell: 1.44; 7 blocks per SM, which the totals' place in
// shared memory allows: 1.36 (1.375 since moved atoms test what they find).  Now
// the issue slots, the L1 and (in the epilogues) the FP64 pipe are each 60-65 % busy.  Cooperative asynchronous
// copies of whole records to shared memory took 1.69 and were not kept.
enum : int { DF_BINS = 0, DF_LIST = 1, DF_EAM = 2 };

// what the sweep reads and writes besides the step constants
struct DensityArgs {
  CandidateArgs C;
  const int *mask;
  const D4 *v, *xi_given;
  int xi_mode;
  const double *T_e;
  float4 *pe;
  int *nshort;
  D4 *A, *Bw;
  double *rho, *beta;
  int *cell;
  double *Te_i;
  int *wrapflag;
  unsigned long long *counters;
  D4 *Mm, *G;
  // DF_EAM
  const unsigned *elist;
  const int *ens, *ens_in;
};

template <bool MULTI, int LANES, int SRC>
__global__ void __launch_bounds__(128, EPH_DF_DENSITY_BLOCKS) k_density_df(StepParams P, DensityArgs D) {
  using namespace df64;
  constexpr int NA = 128 / LANES;                    // atoms per block
  // The bin search keeps its candidates in shared memory: candidate k of atom
  // a at k * 128 + t with one lane per atom, else in the atom's own run of an
  // odd length (its lanes read neighbouring words).  Lists are read row by
  // row from global memory, two candidates ahead: what shared memory they
  // would take is L1 that the spline table and the records need.
  constexpr int CAP = SRC != DF_BINS ? 0 : (LANES == 1 ? CAND_SMEM : CAND_SMEM * LANES - 1);
  __shared__ unsigned s_cand[CAP ? CAND_SMEM * 128 : 1];
  __shared__ float2 s_tot[9 * 128];
  const int t = threadIdx.x, a = t / LANES, g = t % LANES;
  const int i = blockIdx.x * NA + a;
  if (i == 0 && g == 0) *D.wrapflag = 0;  // the kernels before have read it
  const bool valid = i < P.n;
  const bool active = valid && (D.mask[i] & P.groupbit) != 0;
  const size_t n = (size_t)P.n;
  auto at = [&](int k) -> unsigned & { return s_cand[LANES == 1 ? k * 128 + t : a * CAP + k]; };
  unsigned *__restrict__ pj = D.C.pj;
#pragma unroll
  for (int q = 0; q < 9; ++q) s_tot[q * 128 + t] = make_float2(0.f, 0.f);
  int nc = 0;
  int first = 0;
  const unsigned *tail = pj + i;
  if (SRC == DF_EAM && D.ens_in) {  // the list has them apart
    tail = D.elist + i;
    nc = active ? D.ens_in[i] : 0;
  } else if (SRC == DF_EAM) {
    auto set = [&](int k, unsigned u) { pj[(size_t)k * n + i] = u; };
    long long xi[3] = {0, 0, 0};
    if (valid) own_fixed(D.C.rec, i, xi);
    list_candidates<LANES>(P, i, active, xi, D.elist, D.ens, D.C.rec, D.C.err, nc, P.kcap, set, P.rc2_band);
  } else {
    unsigned step;  // n: a moved atom's candidates wait in its rows of pj
    nc = pair_candidates<LANES, SRC == DF_LIST, false, CAP>(P, D.C, i, g, active, at, tail, step, first);
  }
  __syncwarp();
  // after the candidates: their searches need the registers
  long long xi[3] = {0, 0, 0};
  int ei = 0;
  if (valid) {
    int4 ra, rb;
    load_record(D.C.rec + 4 * (size_t)i, ra, rb);
    xi[0] = ((long long)ra.y << 32) | (unsigned)ra.x;
    xi[1] = ((long long)ra.w << 32) | (unsigned)ra.z;
    xi[2] = ((long long)rb.y << 32) | (unsigned)rb.x;
    ei = rb.z;
  }
  // pass 2; the next candidate's position is loaded while this one is summed,
  // each half of a record in one 256-bit load (load_row)
  acc sm[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) sm[q] = acc_zero();
  const df rc2{P.rc2_hi, P.rc2_lo};
  const int nmax = __reduce_max_sync(0xffffffffu, nc);
  int ns = 0;
  auto cand = [&](int k) -> unsigned {
    if (k >= nc) return CODE_NOSHIFT << IDX_BITS;  // atom 0, not counted
    return k < CAP ? at(k) : tail[(size_t)k * n];
  };
  unsigned u = cand(g), u2 = cand(g + LANES);
  int4 ra, rb;
  load_record(D.C.rec + 4 * (size_t)(u & IDX_MASK), ra, rb);
  for (int k = g, m = 0; k - g < nmax; k += LANES, ++m) {
    const unsigned uc = u;
    const int4 ca = ra, cb = rb;
    int4 V0, V1;
    load_record(D.C.rec + 4 * (size_t)(uc & IDX_MASK) + 2, V0, V1);
    u = u2;
    u2 = cand(k + 2 * LANES);
    load_record(D.C.rec + 4 * (size_t)(u & IDX_MASK), ra, rb);
    long long ef[3];
    pair_fixed(P, ca, cb, uc >> IDX_BITS, xi, ef);
    const df ex = fixed_df(ef[0], P.fix_hi, P.fix_lo), ey = fixed_df(ef[1], P.fix_hi, P.fix_lo),
             ez = fixed_df(ef[2], P.fix_hi, P.fix_lo);
    df r2 = dot3(ex, ey, ez, ex, ey, ez);
    // a moved atom in a kept list is out of the cut-off of every atom that
    // reads its list (it may even be outside the integers' range)
    bool in = k < nc && lt(r2, rc2);
    if (SRC == DF_LIST) in = in && (k >= first || cb.w == 0);
    // the shell beyond the cut-off sits at the end of the lists: where no
    // lane of the warp has a pair inside, the iteration would add only zeros
    const unsigned who = __ballot_sync(0xffffffffu, in);
    if (who != 0u) {
      if (!in) r2 = df{1.0f, 0.0f};
      const int ej = cb.z;
      const df rji = spline_rho_df(P, ej, r2, D.C.err);
      const df inv = recip(r2, rcp_estimate(r2.hi));
      df H = mul(rji, inv);
      if (!in) H = df{0.0f, 0.0f};
      const df hx = mul(H, ex), hy = mul(H, ey), hz = mul(H, ez);
      int slot = ns;
      if (LANES > 1) {  // the atom's pairs in lane order
        const int lane = t & 31;
        const unsigned mine = who & (((1u << LANES) - 1u) << (lane & ~(LANES - 1)));
        slot += __popc(mine & ((1u << lane) - 1u));
        ns += __popc(mine);
      } else {
        ns += in;
      }
      if (in) {
        if (slot < P.kcap) {
          const size_t row = (size_t)slot * n + i;
          pj[row] = uc;
          df Hji = H;
          if (MULTI && ej != ei) Hji = mul(spline_rho_df(P, ei, r2, D.C.err), inv);
          store_row(D.pe + 2 * row, make_float4(ex.hi, ey.hi, ez.hi, Hji.hi),
                    make_float4(ex.lo, ey.lo, ez.lo, Hji.lo));
        } else {
          atomicOr(D.C.err, ERR_PAIR_OVERFLOW);
        }
      }
      acc_fma(sm[0], hx, ex);
      acc_fma(sm[1], hx, ey);
      acc_fma(sm[2], hx, ez);
      acc_fma(sm[3], hy, ey);
      acc_fma(sm[4], hy, ez);
      acc_fma(sm[5], hz, ez);
      const df d = dot3(ex, ey, ez, df{__int_as_float(V0.x), __int_as_float(V1.x)},
                        df{__int_as_float(V0.y), __int_as_float(V1.y)}, df{__int_as_float(V0.z), __int_as_float(V1.z)});
      acc_fma(sm[6], d, hx);
      acc_fma(sm[7], d, hy);
      acc_fma(sm[8], d, hz);
    }
    if ((m & 7) == 7) {
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        const float2 w = s_tot[q * 128 + t];
        const df sum = add(df{w.x, w.y}, acc_value(sm[q]));
        s_tot[q * 128 + t] = make_float2(sum.hi, sum.lo);
        sm[q] = acc_zero();
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    const float2 w = s_tot[q * 128 + t];
    const df sum = add(df{w.x, w.y}, acc_value(sm[q]));
    s_tot[q * 128 + t] = make_float2(sum.hi, sum.lo);
  }
  // one thread per atom: thread t of the first NA finishes atom blockIdx.x * NA + t
  int o = i, ns_o = ns;
  if (LANES > 1) {
    __shared__ int s_ns[NA];
    if (g == 0) s_ns[a] = ns;
    __syncthreads();
    if (t >= NA) return;
    o = blockIdx.x * NA + t;
    ns_o = s_ns[t];
  }
  if (o >= P.n) return;
  double mq[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    const float2 *w = s_tot + q * 128 + (LANES > 1 ? t * LANES : t);
    double sum = to_double(df{w[0].x, w[0].y});
#pragma unroll
    for (int l = 1; l < LANES; ++l) sum += to_double(df{w[l].x, w[l].y});
    mq[q] = sum;
  }
  const D4 xo = D.C.x[o];
  const bool act = LANES > 1 ? (D.mask[o] & P.groupbit) != 0 : active;
  density_epilogue<true, true, true>(P, o, act, xo, LANES > 1 ? (int)xo.w : ei, 0.0, ns_o < P.kcap ? ns_o : P.kcap,
                                     mq[0], mq[1], mq[2], mq[3], mq[4], mq[5], mq[6], mq[7], mq[8], D.xi_given,
                                     D.xi_mode, D.T_e, D.nshort, D.A, D.Bw, D.rho, D.beta, D.cell, D.Te_i, D.C.err,
                                     D.counters, D.v, D.Mm, D.G);
}

// -------------------------------------------------------- friction sweep 1

// The EXACT sweeps over the pairs: several lanes of a warp per atom make the
// terms of as many pairs at once, and the sums still run one pair after the
// other in ascending neighbour index, as the reference's do: the terms of a
// chunk go through shared memory, where each of an atom's first lanes adds
// one component's.  A pair that does not count leaves -0.0, which changes no
// sum.  (One lane per atom left the SMs few warps with chains of FP64
// latency, and everything else waiting for it.)
constexpr int EX_THREADS = 128;
constexpr int EX_ROW = EX_THREADS + 1;  // row of one component: distinct banks for the adding lanes

// dot3 with its products on the integer units
__device__ __forceinline__ double soft_dot3(const D4 &e, double x, double y, double z) {
  return soft::mul(e.x, x) + soft::mul(e.y, y) + soft::mul(e.z, z);
}

// force_prl stage 1 (fix_eph.cpp:699-741) in the reference's expression order
// (EXACT mode; FAST mode folds it into the density sweep):
// w_i = sum_j p_ij [(e.v_i) - (e.v_j)] e,  p_ij = alpha_i rho_j(r^2) / (rho_i r^2)
// FP64 issue binds it: what a pair leaves to the FP64 pipe is 12 operations,
// the quotient and ten of the 13 products run on the integer units.  GB300, us
// per step at 62,500 atoms: 186 with one lane per atom and the hardware's
// operations; 145 with the quotients here; 127 with four lanes; 82 with the
// products.
template <int L>
__global__ void __launch_bounds__(EX_THREADS) k_friction_w(StepParams P, const int *__restrict__ mask,
                                                            const D4 *__restrict__ v, const unsigned *__restrict__ pj,
                                                            const D4 *__restrict__ pe, const double2 *__restrict__ pg,
                                                            const int *__restrict__ nshort, const D4 *__restrict__ A,
                                                            D4 *__restrict__ Bw) {
  __shared__ double s_term[3 * EX_ROW];
  const int t = threadIdx.x, g = t & (L - 1), i = blockIdx.x * (EX_THREADS / L) + t / L;
  D4 Ai{0.0, 0.0, 0.0, 0.0}, vi{0.0, 0.0, 0.0, 0.0};
  int ns = 0;
  if (i < P.n && (mask[i] & P.groupbit)) {
    Ai = A[i];
    if (pos_double(Ai.x)) {  // otherwise Bw[i].yzw stays 0
      vi = v[i];
      ns = nshort[i];
    }
  }
  constexpr int OWN = (3 + L - 1) / L;  // components g, g + L, ...
  double w[OWN];
#pragma unroll
  for (int c = 0; c < OWN; ++c) w[c] = 0.0;
  const int nmax = __reduce_max_sync(0xffffffffu, ns);
  for (int k = g; k - g < nmax; k += L) {
    double tx = -0.0, ty = -0.0, tz = -0.0;
    if (k < ns) {
      const size_t slot = (size_t)k * P.n + i;
      const unsigned j = pj[slot] & IDX_MASK;
      const D4 e = pe[slot];
      const D4 vj = v[j];
      const double rji = pg[slot].x;
      const double prescaler = soft::div(soft::mul(Ai.y, rji), soft::divisor(soft::mul(Ai.x, e.w)));
      const double var1 = soft::mul(prescaler, dot3(e.x, e.y, e.z, vi.x, vi.y, vi.z));
      const double var2 = soft::mul(prescaler, soft_dot3(e, vj.x, vj.y, vj.z));
      const double dvar = var1 - var2;
      tx = soft::mul(dvar, e.x);
      ty = soft::mul(dvar, e.y);
      tz = soft::mul(dvar, e.z);
    }
    s_term[t] = tx;
    s_term[EX_ROW + t] = ty;
    s_term[2 * EX_ROW + t] = tz;
    __syncwarp();
#pragma unroll
    for (int c = 0; c < OWN; ++c) {
      const int q = g + c * L;
      if (q < 3) {
        const double *term = s_term + q * EX_ROW + (t - g);
#pragma unroll
        for (int m = 0; m < L; ++m) w[c] += term[m];
      }
    }
    __syncwarp();
  }
  if (ns == 0) return;
#pragma unroll
  for (int c = 0; c < OWN; ++c)
    if (g + c * L < 3) reinterpret_cast<double *>(Bw + i)[1 + g + c * L] = w[c];
}

// ------------------------------------------------ friction + random sweep

// The end of post_force for atom i: the coloured-noise memory of
// eph/coloured/exp (fix_eph_coloured_exp.cpp:562-568, :619-625), f_EPH and
// f_RNG, and their addition to the engine's force unless NOFRICTION /
// NORANDOM keep them out (fix_eph.cpp:892-906).
template <bool FRIC, bool RAND>
__device__ __forceinline__ void store_forces(const StepParams &P, int i, bool live, double fex, double fey,
                                             double fez, double frx, double fry, double frz, D4 *__restrict__ f,
                                             D4 *__restrict__ f_eph, D4 *__restrict__ f_rng, D4 *__restrict__ f_dis,
                                             D4 *__restrict__ f_sto) {
  if (P.coloured && live) {
    if (FRIC) {
      D4 d = f_dis[i];
      d.x = d.x * (1. - P.zeta) + P.zeta * fex;
      d.y = d.y * (1. - P.zeta) + P.zeta * fey;
      d.z = d.z * (1. - P.zeta) + P.zeta * fez;
      f_dis[i] = d;
      fex = d.x;
      fey = d.y;
      fez = d.z;
    }
    if (RAND) {
      D4 d = f_sto[i];
      d.x = d.x * (1. - P.zeta) + P.zeta * frx;
      d.y = d.y * (1. - P.zeta) + P.zeta * fry;
      d.z = d.z * (1. - P.zeta) + P.zeta * frz;
      f_sto[i] = d;
      frx = d.x;
      fry = d.y;
      frz = d.z;
    }
  }
  f_eph[i] = D4{fex, fey, fez, 0.0};
  f_rng[i] = D4{frx, fry, frz, 0.0};
  D4 fi = f[i];
  if (FRIC && !(P.flags & 0x10)) {
    fi.x += fex;
    fi.y += fey;
    fi.z += fez;
  }
  if (RAND && !(P.flags & 0x20)) {
    fi.x += frx;
    fi.y += fry;
    fi.z += frz;
  }
  f[i] = fi;
}

// force_prl stages 2 and 3 (fix_eph.cpp:748-836) in one pass over the pairs,
// then the force update of post_force (fix_eph.cpp:892-906), FAST mode:
//   f_EPH_i -= sum_j [a_i rho_j(r^2) (e.w_i)/(rho_i r^2) - a_j rho_i(r^2) (e.w_j)/(rho_j r^2)] e
//   f_RNG_i  = eta sqrt(T_e(x_i)) sum_j [same with xi] e
template <bool MULTI, bool FRIC, bool RAND>
__global__ void __launch_bounds__(128) k_forces(StepParams P, const int *__restrict__ mask,
                                                const unsigned *__restrict__ pj, const D4 *__restrict__ pe,
                                                const double2 *__restrict__ pg, const int *__restrict__ nshort,
                                                const D4 *__restrict__ A, const D4 *__restrict__ Bw,
                                                const double *__restrict__ Te_i, D4 *__restrict__ f,
                                                D4 *__restrict__ f_eph, D4 *__restrict__ f_rng,
                                                D4 *__restrict__ f_dis, D4 *__restrict__ f_sto) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  double fex = 0.0, fey = 0.0, fez = 0.0, frx = 0.0, fry = 0.0, frz = 0.0;
  const D4 Ai = A[i];
  const bool live = (mask[i] & P.groupbit) && pos_double(Ai.x);
  if (live) {
    const D4 Bi = Bw[i];
    const double xix = Ai.z, xiy = Ai.w, xiz = Bi.x;
    const int ns = nshort[i];
    for (int k = 0; k < ns; ++k) {
      const size_t slot = (size_t)k * P.n + i;
      const unsigned j = pj[slot] & IDX_MASK;
      const D4 Aj = A[j];
      if (!pos_double(Aj.x)) continue;
      const D4 e = pe[slot];
      // one element has no pg rows (the buffer is not allocated)
      const double2 g = MULTI ? pg[slot] : make_double2(0.0, 0.0);
      const D4 Bj = Bw[j];
      const double a = Ai.y * e.w;                  // alpha_i/rho_i * rho_j(r^2)/r^2
      const double b = Aj.y * (MULTI ? g.x : e.w);  // alpha_j/rho_j * rho_i(r^2)/r^2
      if (FRIC) {
        const double di = dot3_fma(e.x, e.y, e.z, Bi.y, Bi.z, Bi.w);
        const double dj = dot3_fma(e.x, e.y, e.z, Bj.y, Bj.z, Bj.w);
        const double dvar = fma(a, di, -(b * dj));
        fex = fma(-dvar, e.x, fex);
        fey = fma(-dvar, e.y, fey);
        fez = fma(-dvar, e.z, fez);
      }
      if (RAND) {
        const double di = dot3_fma(e.x, e.y, e.z, xix, xiy, xiz);
        const double dj = dot3_fma(e.x, e.y, e.z, Aj.z, Aj.w, Bj.x);
        const double dvar = fma(a, di, -(b * dj));
        frx = fma(dvar, e.x, frx);
        fry = fma(dvar, e.y, fry);
        frz = fma(dvar, e.z, frz);
      }
    }
    if (RAND) {
      const double var = P.eta * sqrt(Te_i[i]);
      frx *= var;
      fry *= var;
      frz *= var;
    }
  }
  store_forces<FRIC, RAND>(P, i, live, fex, fey, fez, frx, fry, frz, f, f_eph, f_rng, f_dis, f_sto);
}

// The same in the reference's expression order (EXACT mode).  FP64 issue
// and integer issue bind it: per pair 32 operations stay on the FP64 pipe (the
// four scalar products and the sums; with these products on the integer units
// too it took 240), beside two divisors, four quotients and ten products on
// the integer units.  GB300, us per step at 62,500 atoms: 459 with one lane
// per atom and the hardware's operations; 277 with the quotients here; 226 with
// four lanes and the products.
template <bool MULTI, bool FRIC, bool RAND, int L>
__global__ void __launch_bounds__(EX_THREADS) k_forces_exact(StepParams P, const int *__restrict__ mask,
                                                              const unsigned *__restrict__ pj,
                                                              const D4 *__restrict__ pe,
                                                              const double2 *__restrict__ pg,
                                                              const int *__restrict__ nshort,
                                                              const D4 *__restrict__ A, const D4 *__restrict__ Bw,
                                                              const double *__restrict__ Te_i, D4 *__restrict__ f,
                                                              D4 *__restrict__ f_eph, D4 *__restrict__ f_rng,
                                                              D4 *__restrict__ f_dis, D4 *__restrict__ f_sto) {
  constexpr int NA = EX_THREADS / L;
  __shared__ double s_term[6 * EX_ROW];
  const int t = threadIdx.x, g = t & (L - 1), i = blockIdx.x * NA + t / L;
  D4 Ai{0.0, 0.0, 0.0, 0.0}, Bi{0.0, 0.0, 0.0, 0.0};
  int ns = 0;
  if (i < P.n && (mask[i] & P.groupbit)) {
    Ai = A[i];
    if (pos_double(Ai.x)) {
      Bi = Bw[i];
      ns = nshort[i];
    }
  }
  // components g, g + L, ... of friction x, y, z, random x, y, z
  constexpr int OWN = (6 + L - 1) / L;
  double sum[OWN];
#pragma unroll
  for (int c = 0; c < OWN; ++c) sum[c] = 0.0;
  const int nmax = FRIC || RAND ? __reduce_max_sync(0xffffffffu, ns) : 0;
  for (int k = g; k - g < nmax; k += L) {
    double term[6] = {-0.0, -0.0, -0.0, -0.0, -0.0, -0.0};
    if (k < ns) {
      const size_t slot = (size_t)k * P.n + i;
      const unsigned j = pj[slot] & IDX_MASK;
      const D4 Aj = A[j];
      if (pos_double(Aj.x)) {
        const D4 e = pe[slot];
        const double2 q = pg[slot];
        const D4 Bj = Bw[j];
        const double ai = soft::mul(Ai.y, q.x);                  // alpha_i * rho_j(r^2)
        const double aj = soft::mul(Aj.y, MULTI ? q.y : q.x);  // alpha_j * rho_i(r^2)
        const soft::Divisor den_i = soft::divisor(soft::mul(Ai.x, e.w)), den_j = soft::divisor(soft::mul(Aj.x, e.w));
        if (FRIC) {
          const double var1 = soft::div(ai * dot3(e.x, e.y, e.z, Bi.y, Bi.z, Bi.w), den_i);
          const double var2 = soft::div(aj * dot3(e.x, e.y, e.z, Bj.y, Bj.z, Bj.w), den_j);
          const double dvar = var1 - var2;
          term[0] = -soft::mul(dvar, e.x);
          term[1] = -soft::mul(dvar, e.y);
          term[2] = -soft::mul(dvar, e.z);
        }
        if (RAND) {
          const double var1 = soft::div(ai * dot3(e.x, e.y, e.z, Ai.z, Ai.w, Bi.x), den_i);
          const double var2 = soft::div(aj * dot3(e.x, e.y, e.z, Aj.z, Aj.w, Bj.x), den_j);
          const double dvar = var1 - var2;
          term[3] = soft::mul(dvar, e.x);
          term[4] = soft::mul(dvar, e.y);
          term[5] = soft::mul(dvar, e.z);
        }
      }
    }
#pragma unroll
    for (int q = FRIC ? 0 : 3; q < (RAND ? 6 : 3); ++q) s_term[q * EX_ROW + t] = term[q];
    __syncwarp();
#pragma unroll
    for (int c = 0; c < OWN; ++c) {
      const int q = g + c * L;
      if (q >= (FRIC ? 0 : 3) && q < (RAND ? 6 : 3)) {
        const double *p = s_term + q * EX_ROW + (t - g);
#pragma unroll
        for (int m = 0; m < L; ++m) sum[c] += p[m];
      }
    }
    __syncwarp();
  }
  // a thread per atom finishes, in the block's first threads
  __syncthreads();
#pragma unroll
  for (int c = 0; c < OWN; ++c)
    if (g + c * L < 6) s_term[(g + c * L) * EX_ROW + t / L] = sum[c];
  __syncthreads();
  if (t >= NA) return;
  const int o = blockIdx.x * NA + t;
  if (o >= P.n) return;
  double r[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) r[q] = s_term[q * EX_ROW + t];
  const bool live = (mask[o] & P.groupbit) && pos_double(A[o].x);
  if (RAND && live) {
    const double var = P.eta * sqrt(Te_i[o]);
    r[3] *= var;
    r[4] *= var;
    r[5] *= var;
  }
  store_forces<FRIC, RAND>(P, o, live, r[0], r[1], r[2], r[3], r[4], r[5], f, f_eph, f_rng, f_dis, f_sto);
}

// Stages 2 and 3 in FAST mode after k_density<.., true> (same sums as
// k_forces, split into the atom's own part and the neighbours' part); TPA
// lanes per atom take rows g, g + TPA, ... of the neighbours' part and
// their sums meet in shared memory, where one thread per atom finishes.  With W_i = a_i w_i, X_i = a_i xi_i (a_i = alpha_i/rho_i)
// and M_i = sum_j H_ij e e^T over all of the atom's pairs:
//   f_EPH_i = -M_i W_i + sum_{j live} H_ji (e.W_j) e + sum_{j not live} H_ij (e.W_i) e
//   f_RNG_i = eta sqrt(T_e) [M_i X_i - sum_{j live} H_ji (e.X_j) e - sum_{j not live} H_ij (e.X_i) e]
// ("live": rho_j > 0, the reference's test; the last sums take back the
// pairs it skips).  Per pair 14 FP64 instructions instead of 24.  A skipped
// pair is the same term with the atom's own record and H_ij, so it takes its
// turn in the loop (with part of the atoms outside the group every atom has
// some: a second pass over the pairs for them, by one lane per atom, made the
// sweep of 9,724 atoms, a fifth of them outside, 53 us instead of 23 on
// GB300, and that of 32,000 atoms in df64 187 instead of 35).
template <bool MULTI, bool RAND, int TPA = 1>
__global__ void __launch_bounds__(128) k_forces_m(StepParams P, const unsigned *__restrict__ pj,
                                                  const D4 *__restrict__ pe, const double2 *__restrict__ pg,
                                                  const int *__restrict__ nshort, const D4 *__restrict__ Mm,
                                                  const D4 *__restrict__ G, const double *__restrict__ Te_i,
                                                  D4 *__restrict__ f, D4 *__restrict__ f_eph, D4 *__restrict__ f_rng,
                                                  D4 *__restrict__ f_dis, D4 *__restrict__ f_sto) {
  const long gt = (long)blockIdx.x * blockDim.x + threadIdx.x;
  int i = (int)(gt / TPA);
  const int g = (int)(gt % TPA);
  if (TPA == 1 && i >= P.n) return;  // with TPA > 1 every lane joins the sums
  double fex = 0.0, fey = 0.0, fez = 0.0, frx = 0.0, fry = 0.0, frz = 0.0;
  bool live = false;
  int ns = 0;
  if (i < P.n) {
    live = pos_double(G[2 * (size_t)i + 1].z);  // rho_i > 0 (0 outside the group)
    if (live) ns = nshort[i];
  }
  unsigned j_next = g < ns ? pj[(size_t)g * P.n + i] & IDX_MASK : 0u;
  for (int k = g; k < ns; k += TPA) {
    const size_t slot = (size_t)k * P.n + i;
    const unsigned j = j_next;
    if (k + TPA < ns) j_next = pj[slot + (size_t)TPA * P.n] & IDX_MASK;
    const D4 e = pe[slot];
    D4 Gj1 = G[2 * (size_t)j], Gj2 = G[2 * (size_t)j + 1];
    const bool skip = !pos_double(Gj2.z);
    if (skip) {  // a pair the reference skips: its share of M_i comes back out
      Gj1 = G[2 * (size_t)i];
      Gj2 = G[2 * (size_t)i + 1];
    }
    if (MULTI) {
      const double Hji = skip ? e.w : pg[slot].x;  // rho_i(r^2)/r^2 (H_ij)
      const double sw = Hji * dot3_fma(e.x, e.y, e.z, Gj1.x, Gj1.y, Gj1.z);
      fex = fma(sw, e.x, fex);
      fey = fma(sw, e.y, fey);
      fez = fma(sw, e.z, fez);
      if (RAND) {
        const double sx = Hji * dot3_fma(e.x, e.y, e.z, Gj1.w, Gj2.x, Gj2.y);
        frx = fma(sx, e.x, frx);
        fry = fma(sx, e.y, fry);
        frz = fma(sx, e.z, frz);
      }
    } else {  // the pair's H e: {e.w, pg.x, pg.y}
      const double2 h = pg[slot];
      const double sw = dot3_fma(e.x, e.y, e.z, Gj1.x, Gj1.y, Gj1.z);
      fex = fma(sw, e.w, fex);
      fey = fma(sw, h.x, fey);
      fez = fma(sw, h.y, fez);
      if (RAND) {
        const double sx = dot3_fma(e.x, e.y, e.z, Gj1.w, Gj2.x, Gj2.y);
        frx = fma(sx, e.w, frx);
        fry = fma(sx, h.x, fry);
        frz = fma(sx, h.y, frz);
      }
    }
  }
  if (TPA > 1) {
    // the lanes' sums meet in shared memory; the block's first threads finish
    // an atom each
    constexpr int NA = 128 / TPA, NSUM = RAND ? 6 : 3;
    __shared__ double s_sum[NSUM * 128], s_tot[NSUM * NA];
    const int t = threadIdx.x, at = g * NA + t / TPA;
    s_sum[at] = fex;
    s_sum[128 + at] = fey;
    s_sum[256 + at] = fez;
    if (RAND) {
      s_sum[(NSUM - 3) * 128 + at] = frx;
      s_sum[(NSUM - 2) * 128 + at] = fry;
      s_sum[(NSUM - 1) * 128 + at] = frz;
    }
    __syncthreads();
    for (int q = t; q < NSUM * NA; q += 128) {
      const double *w = s_sum + q / NA * 128 + q % NA;
      double sum = w[0];
#pragma unroll
      for (int l = 1; l < TPA; ++l) sum += w[l * NA];
      s_tot[q] = sum;
    }
    __syncthreads();
    i = blockIdx.x * NA + t;
    if (t >= NA || i >= P.n) return;
    fex = s_tot[t];
    fey = s_tot[NA + t];
    fez = s_tot[2 * NA + t];
    if (RAND) {
      frx = s_tot[(NSUM - 3) * NA + t];
      fry = s_tot[(NSUM - 2) * NA + t];
      frz = s_tot[(NSUM - 1) * NA + t];
    }
    live = pos_double(G[2 * (size_t)i + 1].z);
  }
  if (live) {
    const D4 Gi1 = G[2 * (size_t)i], Gi2 = G[2 * (size_t)i + 1];
    const D4 M1 = Mm[i], M2 = Mm[(size_t)P.n + i];  // {xx, xy, xz, yy}, {yz, zz}
    fex -= fma(M1.x, Gi1.x, fma(M1.y, Gi1.y, M1.z * Gi1.z));
    fey -= fma(M1.y, Gi1.x, fma(M1.w, Gi1.y, M2.x * Gi1.z));
    fez -= fma(M1.z, Gi1.x, fma(M2.x, Gi1.y, M2.y * Gi1.z));
    if (RAND) {
      const double var = P.eta * sqrt(Te_i[i]);
      frx = var * (fma(M1.x, Gi1.w, fma(M1.y, Gi2.x, M1.z * Gi2.y)) - frx);
      fry = var * (fma(M1.y, Gi1.w, fma(M1.w, Gi2.x, M2.x * Gi2.y)) - fry);
      frz = var * (fma(M1.z, Gi1.w, fma(M2.x, Gi2.x, M2.y * Gi2.y)) - frz);
    }
  }
  store_forces<true, RAND>(P, i, live, fex, fey, fez, frx, fry, frz, f, f_eph, f_rng, f_dis, f_sto);
}

// k_forces_m over the df64 pair cache and records of k_density_df: per pair
// H_ji (e.W_j) e and H_ji (e.X_j) e in df64 with blocked sums; the per-atom
// part (-M_i W_i, the pairs the reference skips, eta sqrt(T_e), the force
// update) in FP64 as k_forces_m does it, with W_i = a_i w_i and X_i = a_i xi_i
// formed from A and Bw exactly as the FP64 records are.  A neighbour the
// reference skips (rho_j <= 0 or outside the group) carries a NaN in its
// record's first word.
// It streams the pair cache (36 B per pair) and gathers a 48 B record per pair
// from L2; on GB300 the latency of those loads bounds it, so the totals live
// in shared memory (56 registers, 9 blocks per SM) and the next neighbour's
// index is loaded one pair ahead.  2,048,000 atoms: 1.18 ms with 52 B per pair
// and 16-byte loads; 1.10 with 36 B; 0.84 with 256-bit loads and 8 blocks; 0.80
// with the skipped pairs in the loop and 9.
template <bool MULTI, bool RAND, int TPA = 1>
__global__ void __launch_bounds__(128, EPH_DF_FORCES_BLOCKS)
    k_forces_df(StepParams P, const unsigned *__restrict__ pj, const float4 *__restrict__ pe,
                const int *__restrict__ nshort, const D4 *__restrict__ Mm, const float4 *__restrict__ Gf,
                const D4 *__restrict__ A, const D4 *__restrict__ Bw, const double *__restrict__ Te_i,
                D4 *__restrict__ f, D4 *__restrict__ f_eph, D4 *__restrict__ f_rng, D4 *__restrict__ f_dis,
                D4 *__restrict__ f_sto, const int4 *__restrict__ rec, unsigned *__restrict__ err) {
  using namespace df64;
  __shared__ float2 s_tot[6 * 128];  // the sums' totals; the blocks of 8 are in registers
  const int t = threadIdx.x;
  const long gt = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int i = (int)(gt / TPA), g = (int)(gt % TPA);
  if (TPA == 1 && i >= P.n) return;  // with TPA > 1 every lane joins the butterfly
  constexpr int NS = RAND ? 6 : 3;
  acc sm[NS];
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    sm[q] = acc_zero();
    s_tot[q * 128 + t] = make_float2(0.f, 0.f);
  }
  bool live = false;
  int ns = 0, skipped = 0;
  if (i < P.n) {
    const float g0 = Gf[4 * (size_t)i].x;
    live = g0 == g0;  // not NaN: rho_i > 0 and in the group
    if (live) ns = nshort[i];
  }
  auto fold = [&]() {
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const float2 w = s_tot[q * 128 + t];
      const df sum = add(df{w.x, w.y}, acc_value(sm[q]));
      s_tot[q * 128 + t] = make_float2(sum.hi, sum.lo);
      sm[q] = acc_zero();
    }
  };
  int m = 0;
  unsigned jn = g < ns ? pj[(size_t)g * P.n + i] & IDX_MASK : 0u;
  for (int k = g; k < ns; k += TPA, ++m) {
    const size_t slot = (size_t)k * P.n + i;
    const unsigned j = jn;
    if (k + TPA < ns) jn = pj[slot + (size_t)TPA * P.n] & IDX_MASK;
    float4 a, b, G0, G1, G2;
    load_row(Gf + 4 * (size_t)j, G0, G1);
    load_row_once(pe + 2 * slot, a, b);
    if (RAND) G2 = Gf[4 * (size_t)j + 2];
    const df ex{a.x, b.x}, ey{a.y, b.y}, ez{a.z, b.z};
    df H{a.w, b.w};  // H_ji
    if (G0.x != G0.x) {  // a pair the reference skips: its share of M_i comes back out
      ++skipped;
      load_row(Gf + 4 * (size_t)i, G0, G1);
      if (RAND) G2 = Gf[4 * (size_t)i + 2];
      if (MULTI) {  // H_ij: the cached H_ji with one element
        const int ej = rec[4 * (size_t)j + 1].z;
        if (ej != rec[4 * (size_t)i + 1].z) {
          const df r2 = dot3(ex, ey, ez, ex, ey, ez);
          H = mul(spline_rho_df(P, ej, r2, err), recip(r2, rcp_estimate(r2.hi)));
        }
      }
    }
    const df sw = mul(H, dot3(ex, ey, ez, df{G0.x, G1.x}, df{G0.y, G1.y}, df{G0.z, G1.z}));
    acc_fma(sm[0], sw, ex);
    acc_fma(sm[1], sw, ey);
    acc_fma(sm[2], sw, ez);
    if (RAND) {
      const df sx = mul(H, dot3(ex, ey, ez, df{G0.w, G1.w}, df{G2.x, G2.z}, df{G2.y, G2.w}));
      acc_fma(sm[NS - 3], sx, ex);
      acc_fma(sm[NS - 2], sx, ey);
      acc_fma(sm[NS - 1], sx, ez);
    }
    if ((m & 7) == 7) fold();
  }
  fold();
  // More than half of the pairs skipped: -M_i W_i and what comes back out nearly
  // cancel, so the live pairs (the fewer ones) are summed alone, both terms of
  // each.  All lanes of an atom decide alike.
#pragma unroll
  for (int o = TPA / 2; o > 0; o >>= 1) skipped += __shfl_xor_sync(0xffffffffu, skipped, o);
  const bool direct = 2 * skipped > ns;
  if (direct) {
#pragma unroll
    for (int q = 0; q < NS; ++q) s_tot[q * 128 + t] = make_float2(0.f, 0.f);
    m = 0;
    for (int k = g; k < ns; k += TPA) {
      const size_t slot = (size_t)k * P.n + i;
      const unsigned j = pj[slot] & IDX_MASK;
      float4 a, b, G0, G1, O0, O1;
      load_row(Gf + 4 * (size_t)j, G0, G1);
      if (G0.x != G0.x) continue;
      load_row(Gf + 4 * (size_t)i, O0, O1);
      load_row(pe + 2 * slot, a, b);
      const df ex{a.x, b.x}, ey{a.y, b.y}, ez{a.z, b.z}, Hji{a.w, b.w};
      df Hij = Hji;
      if (MULTI) {
        const int ej = rec[4 * (size_t)j + 1].z;
        if (ej != rec[4 * (size_t)i + 1].z) {
          const df r2 = dot3(ex, ey, ez, ex, ey, ez);
          Hij = mul(spline_rho_df(P, ej, r2, err), recip(r2, rcp_estimate(r2.hi)));
        }
      }
      const df sw = sub(mul(Hji, dot3(ex, ey, ez, df{G0.x, G1.x}, df{G0.y, G1.y}, df{G0.z, G1.z})),
                        mul(Hij, dot3(ex, ey, ez, df{O0.x, O1.x}, df{O0.y, O1.y}, df{O0.z, O1.z})));
      acc_fma(sm[0], sw, ex);
      acc_fma(sm[1], sw, ey);
      acc_fma(sm[2], sw, ez);
      if (RAND) {
        const float4 G2 = Gf[4 * (size_t)j + 2], O2 = Gf[4 * (size_t)i + 2];
        const df sx = sub(mul(Hji, dot3(ex, ey, ez, df{G0.w, G1.w}, df{G2.x, G2.z}, df{G2.y, G2.w})),
                          mul(Hij, dot3(ex, ey, ez, df{O0.w, O1.w}, df{O2.x, O2.z}, df{O2.y, O2.w})));
        acc_fma(sm[NS - 3], sx, ex);
        acc_fma(sm[NS - 2], sx, ey);
        acc_fma(sm[NS - 1], sx, ez);
      }
      if ((++m & 7) == 0) fold();
    }
    fold();
  }
  double tot[6];
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    const float2 w = s_tot[q * 128 + t];
    tot[q] = to_double(df{w.x, w.y});
  }
  double fex = tot[0], fey = tot[1], fez = tot[2];
  double frx = 0.0, fry = 0.0, frz = 0.0;
  if (RAND) {
    frx = tot[3];
    fry = tot[4];
    frz = tot[5];
  }
  if (TPA > 1) {
#pragma unroll
    for (int o = TPA / 2; o > 0; o >>= 1) {
      fex += __shfl_xor_sync(0xffffffffu, fex, o);
      fey += __shfl_xor_sync(0xffffffffu, fey, o);
      fez += __shfl_xor_sync(0xffffffffu, fez, o);
      if (RAND) {
        frx += __shfl_xor_sync(0xffffffffu, frx, o);
        fry += __shfl_xor_sync(0xffffffffu, fry, o);
        frz += __shfl_xor_sync(0xffffffffu, frz, o);
      }
    }
    if (i >= P.n || g != 0) return;
  }
  if (live) {
    const D4 Ai = A[i], Bi = Bw[i];
    const double a = Ai.y;  // alpha_i / rho_i
    const double Wx = a * Bi.y, Wy = a * Bi.z, Wz = a * Bi.w;
    const double Xx = a * Ai.z, Xy = a * Ai.w, Xz = a * Bi.x;
    D4 M1 = Mm[i], M2 = Mm[(size_t)P.n + i];  // {xx, xy, xz, yy}, {yz, zz}
    if (direct) M1 = M2 = D4{0.0, 0.0, 0.0, 0.0};
    fex -= fma(M1.x, Wx, fma(M1.y, Wy, M1.z * Wz));
    fey -= fma(M1.y, Wx, fma(M1.w, Wy, M2.x * Wz));
    fez -= fma(M1.z, Wx, fma(M2.x, Wy, M2.y * Wz));
    if (RAND) {
      const double var = P.eta * sqrt(Te_i[i]);
      frx = var * (fma(M1.x, Xx, fma(M1.y, Xy, M1.z * Xz)) - frx);
      fry = var * (fma(M1.y, Xx, fma(M1.w, Xy, M2.x * Xz)) - fry);
      frz = var * (fma(M1.z, Xx, fma(M2.x, Xy, M2.y * Xz)) - frz);
    }
  }
  store_forces<true, RAND>(P, i, live, fex, fey, fez, frx, fry, frz, f, f_eph, f_rng, f_dis, f_sto);
}

// ------------------------------------- pair sweeps, several lanes per atom

// FAST mode with TPA lanes per atom (TPA = 2, 4, 8): lane g of an atom takes
// rows g, g + TPA, ...; the lanes' sums are combined by a butterfly over the
// TPA neighbouring lanes.  Small systems (tens of thousands of atoms) leave
// the SMs with a few warps each and the one-lane sweeps wait on their loads;
// TPA times more warps hide that.  The order of the sums depends on TPA
// (results within rounding of the one-lane sweeps, the same every run).
template <bool MULTI, bool FRIC, bool RAND, int TPA>
__global__ void __launch_bounds__(128) k_forces_tpa(StepParams P, const int *__restrict__ mask,
                                                     const unsigned *__restrict__ pj, const D4 *__restrict__ pe,
                                                     const double2 *__restrict__ pg, const int *__restrict__ nshort,
                                                     const D4 *__restrict__ A, const D4 *__restrict__ Bw,
                                                     const double *__restrict__ Te_i, D4 *__restrict__ f,
                                                     D4 *__restrict__ f_eph, D4 *__restrict__ f_rng,
                                                     D4 *__restrict__ f_dis, D4 *__restrict__ f_sto) {
  const int gt = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = gt / TPA, g = gt % TPA;
  double fex = 0.0, fey = 0.0, fez = 0.0, frx = 0.0, fry = 0.0, frz = 0.0;
  D4 Ai{0.0, 0.0, 0.0, 0.0};
  bool live = false;
  if (i < P.n) {
    Ai = A[i];
    live = (mask[i] & P.groupbit) && pos_double(Ai.x);
  }
  if (live) {
    const D4 Bi = Bw[i];
    const double xix = Ai.z, xiy = Ai.w, xiz = Bi.x;
    const int ns = nshort[i];
    for (int k = g; k < ns; k += TPA) {
      const size_t slot = (size_t)k * P.n + i;
      const unsigned j = pj[slot] & IDX_MASK;
      const D4 Aj = A[j];
      if (!pos_double(Aj.x)) continue;
      const D4 e = pe[slot];
      const D4 Bj = Bw[j];
      const double a = Ai.y * e.w;
      const double b = Aj.y * (MULTI ? pg[slot].x : e.w);
      if (FRIC) {
        const double di = dot3_fma(e.x, e.y, e.z, Bi.y, Bi.z, Bi.w);
        const double dj = dot3_fma(e.x, e.y, e.z, Bj.y, Bj.z, Bj.w);
        const double dvar = fma(a, di, -(b * dj));
        fex = fma(-dvar, e.x, fex);
        fey = fma(-dvar, e.y, fey);
        fez = fma(-dvar, e.z, fez);
      }
      if (RAND) {
        const double di = dot3_fma(e.x, e.y, e.z, xix, xiy, xiz);
        const double dj = dot3_fma(e.x, e.y, e.z, Aj.z, Aj.w, Bj.x);
        const double dvar = fma(a, di, -(b * dj));
        frx = fma(dvar, e.x, frx);
        fry = fma(dvar, e.y, fry);
        frz = fma(dvar, e.z, frz);
      }
    }
  }
#pragma unroll
  for (int o = TPA / 2; o > 0; o >>= 1) {
    if (FRIC) {
      fex += __shfl_xor_sync(0xffffffffu, fex, o);
      fey += __shfl_xor_sync(0xffffffffu, fey, o);
      fez += __shfl_xor_sync(0xffffffffu, fez, o);
    }
    if (RAND) {
      frx += __shfl_xor_sync(0xffffffffu, frx, o);
      fry += __shfl_xor_sync(0xffffffffu, fry, o);
      frz += __shfl_xor_sync(0xffffffffu, frz, o);
    }
  }
  if (i >= P.n || g != 0) return;
  if (live && RAND) {
    const double var = P.eta * sqrt(Te_i[i]);
    frx *= var;
    fry *= var;
    frz *= var;
  }
  store_forces<FRIC, RAND>(P, i, live, fex, fey, fez, frx, fry, frz, f, f_eph, f_rng, f_dis, f_sto);
}

// --------------------------------------------------------- model 1 (TTM)

// force_ttm (fix_eph.cpp:468-503): a local Langevin thermostat with the
// site's beta(rho_i): f_EPH = -beta v_i, f_RNG = eta alpha(rho_i) sqrt(T_e) xi_i;
// then the force update of post_force (:892-906).
template <bool FAST, bool FRIC, bool RAND>
__global__ void k_forces_ttm(StepParams P, const int *__restrict__ mask, const D4 *__restrict__ x,
                             const D4 *__restrict__ v,
                             const D4 *__restrict__ A, const D4 *__restrict__ Bw, const double *__restrict__ rho,
                             const double *__restrict__ beta, const double *__restrict__ Te_i, D4 *__restrict__ f,
                             D4 *__restrict__ f_eph, D4 *__restrict__ f_rng, unsigned *__restrict__ err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  D4 fe = D4{0.0, 0.0, 0.0, 0.0}, fr = D4{0.0, 0.0, 0.0, 0.0};
  if (mask[i] & P.groupbit) {
    if (FRIC) {
      const double var = -beta[i];
      const D4 vi = v[i];
      fe = D4{var * vi.x, var * vi.y, var * vi.z, 0.0};
    }
    if (RAND) {
      const double r = rho[i];
      double alpha = 0.0;
      if (!(r > P.rho_cutoff)) {  // eph_beta.h:188-197
        const int e = (int)x[i].w;
        alpha = spline_eval<FAST>(P.tab_alpha + (size_t)e * P.n_beta, P.inv_drho, P.n_beta, r, err);
      }
      const double var = P.eta * alpha * sqrt(Te_i[i]);
      fr = D4{var * A[i].z, var * A[i].w, var * Bw[i].x, 0.0};
    }
  }
  f_eph[i] = fe;
  f_rng[i] = fr;
  D4 fi = f[i];
  if (FRIC && !(P.flags & 0x10)) {
    fi.x += fe.x;
    fi.y += fe.y;
    fi.z += fe.z;
  }
  if (RAND && !(P.flags & 0x20)) {
    fi.x += fr.x;
    fi.y += fr.y;
    fi.z += fr.z;
  }
  f[i] = fi;
}

// ------------------------------------------------------- energy deposition

// end_of_step deposition (fix_eph.cpp:364-390, eph_fdm.h:172-179): per atom
// dE = -f.v dt for the friction and the random force, dT_e[cell] += dE/(dV dt).
// The grid sums are exact: every term becomes a 128-bit fixed-point integer
// (2^-64 units) and integer addition is order-free, so the grid and the
// energy total are the same whatever order the atoms arrive in; the block
// totals of the energy go to `part`, and the last block to leave its own
// (`left` counts them, and is 0 again afterwards) adds them up and adds the
// step's exchange to Ee (fix_eph.cpp:402-404): integers, so the sum does not
// depend on which block that is.
// KICK: final_integrate in the same pass (0: not here, 1: EXACT, 2: FAST).
// (A launch of its own for each of the two took 3.7 and 3.3 us more of a step of
// 110 us at 4,000 atoms on GB300.)
// The quotients and half of the products run on the integer units (the same
// bits): FP64 issue bound it (83% of that pipe), GB300, 2,048,000 atoms: 137 ->
// 78 us.
template <bool FRIC, bool RAND, bool GRID, int KICK>
__global__ void __launch_bounds__(256) k_deposit(StepParams P, const int *__restrict__ mask,
                                                 D4 *__restrict__ v, const D4 *__restrict__ f_eph,
                                                 const D4 *__restrict__ f_rng, const int *__restrict__ cell,
                                                 U128 *__restrict__ acc, U128 *__restrict__ part,
                                                 unsigned *__restrict__ err, const D4 *__restrict__ f,
                                                 const int *__restrict__ type, unsigned *__restrict__ left,
                                                 double *__restrict__ E_local, double *__restrict__ Ee) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  U128 e{0ull, 0ull};
  if (i < P.n && (mask[i] & P.groupbit)) {
    D4 vi = v[i];
    if (KICK && !(P.flags & 0x08)) {
      kick<KICK == 2>(P.dtfm[type[i]], f[i], vi);
      v[i] = vi;
    }
    U128 g{0ull, 0ull};
    const soft::Divisor prescale = soft::divisor(P.prescale);
    if (FRIC) {
      const D4 fe = f_eph[i];
      double dE = 0.0;
      dE -= soft::mul(fe.x * vi.x, P.dt);
      dE -= soft::mul(fe.y * vi.y, P.dt);
      dE -= soft::mul(fe.z * vi.z, P.dt);
      e = add128(e, to_fixed(dE, err));
      if (GRID) g = add128(g, to_fixed(soft::div(dE, prescale), err));
    }
    if (RAND) {
      const D4 fr = f_rng[i];
      double dE = 0.0;
      dE -= soft::mul(fr.x * vi.x, P.dt);
      dE -= soft::mul(fr.y * vi.y, P.dt);
      dE -= soft::mul(fr.z * vi.z, P.dt);
      e = add128(e, to_fixed(dE, err));
      if (GRID) g = add128(g, to_fixed(soft::div(dE, prescale), err));
    }
    if (GRID && (g.lo | g.hi)) atomic_add128(acc + cell[i], g);
  }
  // block total of the energy, integer adds
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) e = add128(e, shfl_down128(e, d));
  __shared__ U128 warp_tot[8];
  if ((threadIdx.x & 31) == 0) warp_tot[threadIdx.x >> 5] = e;
  __syncthreads();
  __shared__ bool s_last;
  if (threadIdx.x == 0) {
    U128 t{0ull, 0ull};
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = add128(t, warp_tot[w]);
    part[blockIdx.x] = t;
    __threadfence();
    s_last = atomicAdd(left, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  e = U128{0ull, 0ull};
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
    const ulonglong2 t = __ldcg(reinterpret_cast<const ulonglong2 *>(part + b));
    e = add128(e, U128{t.x, t.y});
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) e = add128(e, shfl_down128(e, d));
  if ((threadIdx.x & 31) == 0) warp_tot[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    U128 t{0ull, 0ull};
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = add128(t, warp_tot[w]);
    const double step = from_fixed(t);
    *E_local = step;
    *Ee += step;
    *left = 0u;
  }
}

// ------------------------------------------------------------- FDM solve
// eph_fdm.h:280-287: C_e and kappa_e of the T-dependent cells from T, before
// the stability test; the prescaler rho_e C_e follows.
__global__ void k_fdm_tdyn_params(long ncells, TdynTables t, const double *__restrict__ T, double *__restrict__ C,
                                  double *__restrict__ kappa, double *__restrict__ rhoC, unsigned *__restrict__ err) {
  const long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= ncells || !t.tdyn[r]) return;
  const double c = spline_eval<false>(t.C_T, t.inv_dT, t.n, T[r], err);
  C[r] = c;
  kappa[r] = spline_eval<false>(t.K_T, t.inv_dT, t.n, T[r], err);
  rhoC[r] = t.rho[r] * c;
}

// c_min, rho_min, kappa_max of the stability rule (eph_fdm.h:290-300): cell 0
// whatever its flag, then every cell that is not CONSTANT_VALUE.  One block.
__global__ void k_fdm_bounds(long ncells, const double *__restrict__ C, const double *__restrict__ rho,
                             const double *__restrict__ kappa, const signed char *__restrict__ flag,
                             double *__restrict__ out) {
  double c_min = C[0], r_min = rho[0], k_max = kappa[0];
  for (long i = 1 + threadIdx.x; i < ncells; i += blockDim.x)
    if (flag[i] != 0) {
      c_min = fmin(c_min, C[i]);
      r_min = fmin(r_min, rho[i]);
      k_max = fmax(k_max, kappa[i]);
    }
  __shared__ double s[3][256];
  s[0][threadIdx.x] = c_min;
  s[1][threadIdx.x] = r_min;
  s[2][threadIdx.x] = k_max;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) {
      s[0][threadIdx.x] = fmin(s[0][threadIdx.x], s[0][threadIdx.x + h]);
      s[1][threadIdx.x] = fmin(s[1][threadIdx.x], s[1][threadIdx.x + h]);
      s[2][threadIdx.x] = fmax(s[2][threadIdx.x], s[2][threadIdx.x + h]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = s[0][0];
    out[1] = s[1][0];
    out[2] = s[2][0];
  }
}

// T of cell r after one substep of EPH_FDM::solve (eph_fdm.h:315-396) with
// the reference's expression order: the variable-kappa 7-point stencil with
// periodic wrap and ZERO_DERIVATIVE walls, then T += (ddT + dT + S)/(rho_e C_e)
// dt' on DYNAMIC cells and the clamp at T = 0.  FAST: ih2 = 1/h^2 per axis and
// irhoC = 1/(rho_e C_e) per cell come precomputed (the same correctly rounded
// quotients as 1.0 / x here).
template <bool FAST>
__device__ __forceinline__ double fdm_cell(long r, long nx, long ny, long nz, double dx, double dy, double dz,
                                           double inner_dt, const double *__restrict__ T,
                                           const double *__restrict__ kappa, const double *__restrict__ rhoC,
                                           const double *__restrict__ S, const signed char *__restrict__ flag,
                                           double dTr, unsigned long long *__restrict__ counters,
                                           const TdynTables &td, double3 ih2, const double *__restrict__ irhoC) {
  const long i = r % nx, j = (r / nx) % ny, k = r / (nx * ny);
  const double Tr = T[r];
  double ddT = 0.0;
  if (flag[r] != 2) {
    long p, q;
    const long pr[3] = {(i > 0) ? r - 1 : r + (nx - 1), (j > 0) ? r - nx : r + (ny - 1) * nx,
                        (k > 0) ? r - nx * ny : r + (nz - 1) * nx * ny};
    const long qr[3] = {(i < nx - 1) ? r + 1 : r - (nx - 1), (j < ny - 1) ? r + nx : r - (ny - 1) * nx,
                        (k < nz - 1) ? r + nx * ny : r - (nz - 1) * nx * ny};
    const double h[3] = {dx, dy, dz};
    const double ih2s[3] = {ih2.x, ih2.y, ih2.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      p = pr[a];
      q = qr[a];
      if (flag[q] == 2) q = r;
      else if (flag[p] == 2) p = r;
      const double Tq = T[q], Tp = T[p];
      if (FAST) {  // reciprocals instead of the reference's divisions (within 1e-15 of them)
        const double ih2v = ih2s[a];
        ddT = fma((kappa[q] - kappa[p]) * (Tq - Tp), 0.25 * ih2v, ddT);
        ddT = fma(kappa[r] * ih2v, Tq + Tp - 2.0 * Tr, ddT);
      } else {
        const soft::Divisor hd = soft::divisor(h[a]);
        ddT += soft::div(soft::div((kappa[q] - kappa[p]) * (Tq - Tp), hd), hd) * 0.25;
        ddT += kappa[r] * soft::div(soft::div(Tq + Tp - 2.0 * Tr, hd), hd);
      }
    }
  }
  double t = Tr;
  if (FAST && flag[r] == 1 && !(td.tdyn && td.tdyn[r] == 1)) {
    t = fma((ddT + dTr + S[r]) * inner_dt, irhoC[r], t);
  } else if (flag[r] == 1) {
    if (td.tdyn && td.tdyn[r] == 1) {  // eph_fdm.h:378-382: through E_e(T)
      double E = linear_eval(td, t);
      E += (ddT + dTr + S[r]) / td.rho[r] * inner_dt;
      t = linear_reverse(td, E);
    } else {
      t += soft::div(ddT + dTr + S[r], soft::divisor(rhoC[r])) * inner_dt;
    }
  }
  if (t < 0.0) {
    t = 0.0;
    atomicAdd(&counters[CNT_T_CLAMP], 1ull);
  }
  return t;
}

// One substep over the grid, one thread per cell: reads T, writes Tout.  The
// first substep turns the fixed-point deposits into dT and clears them.
// Launched as a programmatic dependent of the kernel before it (its launch
// overlaps that kernel's tail): waits for that kernel's results before
// touching memory.
template <bool FAST>
__global__ void k_fdm_substep(long nx, long ny, long nz, double dx, double dy, double dz, double inner_dt,
                              const double *__restrict__ T, double *__restrict__ Tout,
                              const double *__restrict__ kappa, const double *__restrict__ rhoC,
                              const double *__restrict__ S, const signed char *__restrict__ flag,
                              double *__restrict__ dT, U128 *__restrict__ acc, int first,
                              unsigned long long *__restrict__ counters, TdynTables td, double3 ih2,
                              const double *__restrict__ irhoC) {
  griddep_wait();
  const long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long ntotal = nx * ny * nz;
  if (r >= ntotal) return;
  double dTr;
  if (first) {
    U128 a = acc[r];
    dTr = from_fixed(a);
    dT[r] = dTr;
    acc[r] = U128{0ull, 0ull};
  } else {
    dTr = dT[r];
  }
  Tout[r] = fdm_cell<FAST>(r, nx, ny, nz, dx, dy, dz, inner_dt, T, kappa, rhoC, S, flag, dTr, counters, td,
                                  ih2, irhoC);
}

// ------------------------------------------------ FAST grid substeps
//
// A FAST substep is T' = T + sum over the six neighbours c_m (T_m - T) +
// c_s (dT + S): with the spacings, kappa, rho_e C_e and the substep length
// fixed between steps, everything of the stencil but the temperatures is a
// coefficient.  FP64 issue binds these kernels (2 lanes per SM and clock), so
// what counts is FP64 instructions per cell and substep: 31 in
// fdm_cell<true>, 14 from per-cell coefficients (k_fdm_coef, built when the
// grid or the time step changes), 12 on a uniform grid (the fix's words, no
// grid file), whose four coefficients are the same for every cell.  They are
// read from device memory, so captured steps follow a change of the grid's
// constants as they follow a change of the per-cell arrays.
struct FdmFast {
  int nx, ny, nz, nc;
  // uniform grid: kappa dt' / (rho_e C_e h^2) per axis and dt' / (rho_e C_e)
  const double *uni;
  // per cell otherwise: 6 x nc weights (-x, +x, -y, +y, -z, +z; -0.0 where the
  // stencil leaves a neighbour out), the source weight (-0.0 where the cell does
  // not change) and the constant source c_s S
  const double *coef, *src_w, *src0;
};

// the weight of what is left out: not merely multiplied by zero, since a wall's T
// may be infinite or NaN.  By the high word: k_fdm_coef leaves no other weight
// with this one (negative and below 2^-1042).
__device__ __forceinline__ bool left_out(double w) { return __double2hiint(w) == (int)0x80000000; }
__device__ __forceinline__ double not_left_out(double w) { return left_out(w) ? 0.0 : w; }

// the neighbours of cell r in the order -x, +x, -y, +y, -z, +z (periodic)
__device__ __forceinline__ void fdm_neighbours(const FdmFast &F, int r, int *m) {
  const int nxy = F.nx * F.ny;
  const int row = r / F.nx, i = r - row * F.nx, k = row / F.ny, j = row - k * F.ny;
  m[0] = i > 0 ? r - 1 : r + (F.nx - 1);
  m[1] = i < F.nx - 1 ? r + 1 : r - (F.nx - 1);
  m[2] = j > 0 ? r - F.nx : r + (nxy - F.nx);
  m[3] = j < F.ny - 1 ? r + F.nx : r - (nxy - F.nx);
  m[4] = k > 0 ? r - nxy : r + (F.nz - 1) * nxy;
  m[5] = k < F.nz - 1 ? r + nxy : r - (F.nz - 1) * nxy;
}

// T of a cell after one substep from its own T, its neighbours' and its
// source term `src` (c_s dT on a uniform grid, c_s (dT + S) otherwise); w: the
// uniform grid's three coefficients or the cell's six weights; fixed: T stays
template <bool UNIFORM>
__device__ __forceinline__ double fdm_next(double T, const double *Tm, const double *w, double src, bool fixed,
                                           unsigned long long *__restrict__ counters) {
  double d;
  if (UNIFORM) {
    d = fma(w[0], fma(-2.0, T, Tm[0] + Tm[1]), src);
    d = fma(w[1], fma(-2.0, T, Tm[2] + Tm[3]), d);
    d = fma(w[2], fma(-2.0, T, Tm[4] + Tm[5]), d);
  } else {
    d = src;
#pragma unroll
    for (int q = 0; q < 6; ++q) d = fma(w[q], Tm[q] - T, d);
  }
  if (UNIFORM || !fixed) T += d;
  if (neg_double(T)) {
    T = 0.0;
    atomicAdd(&counters[CNT_T_CLAMP], 1ull);
  }
  return T;
}

// the weights of cell r, its source weight and constant source
template <bool UNIFORM>
__device__ __forceinline__ void fdm_weights(const FdmFast &F, int r, double *w, double &sw, double &s0) {
  if (UNIFORM) {
#pragma unroll
    for (int q = 0; q < 3; ++q) w[q] = F.uni[q];
    sw = F.uni[3];
    s0 = 0.0;
  } else {
#pragma unroll
    for (int q = 0; q < 6; ++q) w[q] = F.coef[(size_t)q * F.nc + r];
    sw = F.src_w[r];
    s0 = F.src0[r];
  }
}

// The coefficients of FdmFast per cell (eph_fdm.h:322-387: a wall neighbour is
// replaced by the cell itself; only DYNAMIC cells change)
__global__ void k_fdm_coef(FdmFast F, double3 ih2, double inner_dt, const double *__restrict__ kappa,
                           const double *__restrict__ irhoC, const double *__restrict__ S,
                           const signed char *__restrict__ flag, double *__restrict__ coef,
                           double *__restrict__ src_w, double *__restrict__ src0) {
  const int r = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (r >= F.nc) return;
  int m[6];
  fdm_neighbours(F, r, m);
  const bool dyn = flag[r] == 1;
  const double c = dyn ? inner_dt * irhoC[r] : 0.0, kr = kappa[r];
  const double ih[3] = {ih2.x, ih2.y, ih2.z};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int p = m[2 * a], q = m[2 * a + 1];
    const bool wq = flag[q] == 2, wp = !wq && flag[p] == 2;
    if (wq) q = r;
    if (wp) p = r;
    const double d = 0.25 * (kappa[q] - kappa[p]), s = c * ih[a];
    coef[(size_t)(2 * a) * F.nc + r] = wp ? -0.0 : not_left_out(s * (kr - d));
    coef[(size_t)(2 * a + 1) * F.nc + r] = wq ? -0.0 : not_left_out(s * (kr + d));
  }
  src_w[r] = dyn ? not_left_out(c) : -0.0;
  src0[r] = dyn ? c * S[r] : 0.0;
}

// One substep over the grid, one thread per cell (k_fdm_substep's contract:
// the first substep turns the deposits into dT and clears them).  Measured on
// GB300 (us per substep, uniform): 64^3 cells 22 -> 10.5 (FP64 issue: 5 us),
// 26^3 cells 6.5 -> 2.2.
template <bool UNIFORM>
__global__ void __launch_bounds__(128)
    k_fdm_fast(FdmFast F, const double *__restrict__ T, double *__restrict__ Tout, double *__restrict__ dT,
               U128 *__restrict__ acc, int first, unsigned long long *__restrict__ counters) {
  griddep_launch();
  const int r = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  int m[6];
  double w[6], sw, s0;
  if (r < F.nc) {
    fdm_neighbours(F, r, m);
    fdm_weights<UNIFORM>(F, r, w, sw, s0);
    if (!UNIFORM)
#pragma unroll
      for (int q = 0; q < 6; ++q) m[q] = left_out(w[q]) ? r : m[q];
  }
  griddep_wait();
  if (r >= F.nc) return;
  double dTr;
  if (first) {
    dTr = from_fixed(acc[r]);
    dT[r] = dTr;
    acc[r] = U128{0ull, 0ull};
  } else {
    dTr = dT[r];
  }
  double Tm[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) Tm[q] = T[m[q]];
  Tout[r] = fdm_next<UNIFORM>(T[r], Tm, w, fma(sw, dTr, s0), left_out(sw), counters);
}

// All substeps of a small grid in one launch of one thread-block cluster
// (cluster size = grid size, chosen at launch), block b holding cells
// [b * blockDim, (b + 1) * blockDim), one per thread: the temperatures live in
// two shared-memory buffers per block and neighbours are read from the
// owning block's buffer through distributed shared memory, so a substep is
// one cluster barrier, six such reads and the FP64 chain.  The hardware
// barrier is reached the same number of times by every thread (the loop
// bound is a launch argument).  As many SMs as a cluster may have: with few
// cells per SM the FP64 chain of a substep is short.
// Measured on GB300 (us per step): 10^3 cells, 17 substeps 55 -> 19; 16^3
// cells, 11 substeps 56 (11 launches) -> 18.
constexpr int FDM_CLUSTER_CELLS = 384;  // cells per block at most
template <bool UNIFORM>
__global__ void __launch_bounds__(FDM_CLUSTER_CELLS)
    k_fdm_cluster_fast(FdmFast F, unsigned nsub, double *__restrict__ T0, double *__restrict__ rec,
                       double *__restrict__ dT, U128 *__restrict__ acc, unsigned long long *__restrict__ counters) {
  extern __shared__ double s_T[];  // [2][blockDim]
  const int t = (int)threadIdx.x, nt = (int)blockDim.x;
  const int r = (int)blockIdx.x * nt + t;
  const bool mine = r < F.nc;
  double T = 0.0, src = 0.0, w[6];
  unsigned at[6];  // shared::cluster addresses of the neighbours in buffer 0
  bool fixed = false;
  if (mine) {
    int m[6];
    fdm_neighbours(F, r, m);
    double sw, s0;
    fdm_weights<UNIFORM>(F, r, w, sw, s0);
    fixed = left_out(sw);
    if (!UNIFORM)
#pragma unroll
      for (int q = 0; q < 6; ++q) m[q] = left_out(w[q]) ? r : m[q];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const int owner = m[q] / nt;
      const unsigned local = (unsigned)__cvta_generic_to_shared(s_T + (m[q] - owner * nt));
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at[q]) : "r"(local), "r"(owner));
    }
    T = T0[r];
    s_T[t] = T;
    const double dTr = from_fixed(acc[r]);
    dT[r] = dTr;
    acc[r] = U128{0ull, 0ull};
    src = fma(sw, dTr, s0);
  }
  unsigned cur = 0;  // byte offset of the buffer being read
  const unsigned half = (unsigned)(nt * sizeof(double));
  for (unsigned s = 0; s < nsub; ++s) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (mine) {
      double Tm[6];
#pragma unroll
      for (int q = 0; q < 6; ++q)
        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(Tm[q]) : "r"(at[q] + cur) : "memory");
      T = fdm_next<UNIFORM>(T, Tm, w, src, fixed, counters);
      s_T[(cur ? 0 : nt) + t] = T;
      if (rec) rec[(size_t)s * (size_t)F.nc + r] = T;
    }
    cur = half - cur;
  }
  if (mine) T0[r] = T;
  // no block leaves while another may still read its buffers
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The EXACT substeps of a small grid the same way, in fdm_cell's expressions
// (no cell with a temperature-dependent C_e).  The quotients' latency binds it:
// 13 per cell and substep, of which three follow one another.  GB300, us per
// step: 8^3 cells 116 -> 33, 20^3 cells 134 -> 73.
constexpr int FDM_EXACT_CELLS = 512;  // cells per block at most
__global__ void __launch_bounds__(FDM_EXACT_CELLS)
    k_fdm_cluster_exact(FdmFast F, double3 h, double inner_dt, unsigned nsub, double *__restrict__ T0,
                        double *__restrict__ rec, const double *__restrict__ kappa, const double *__restrict__ rhoC,
                        const double *__restrict__ S, const signed char *__restrict__ flag, double *__restrict__ dT,
                        U128 *__restrict__ acc, unsigned long long *__restrict__ counters) {
  extern __shared__ double s_T[];  // [2][blockDim]
  const int t = (int)threadIdx.x, nt = (int)blockDim.x;
  const int r = (int)blockIdx.x * nt + t;
  const bool mine = r < F.nc;
  const soft::Divisor hd[3] = {soft::divisor(h.x), soft::divisor(h.y), soft::divisor(h.z)};
  soft::Divisor rc = hd[0];
  double T = 0.0, dTr = 0.0, Sr = 0.0, kr = 0.0, kd[3] = {0.0, 0.0, 0.0};
  int fl = 0;
  unsigned at[6];
  if (mine) {
    int m[6];
    fdm_neighbours(F, r, m);
    fl = flag[r];
    kr = kappa[r];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      int &p = m[2 * a], &q = m[2 * a + 1];
      if (flag[q] == 2) q = r;
      else if (flag[p] == 2) p = r;
      kd[a] = kappa[q] - kappa[p];
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const int owner = m[q] / nt;
      const unsigned local = (unsigned)__cvta_generic_to_shared(s_T + (m[q] - owner * nt));
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at[q]) : "r"(local), "r"(owner));
    }
    T = T0[r];
    s_T[t] = T;
    rc = soft::divisor(rhoC[r]);
    Sr = S[r];
    dTr = from_fixed(acc[r]);
    dT[r] = dTr;
    acc[r] = U128{0ull, 0ull};
  }
  unsigned cur = 0;
  const unsigned half = (unsigned)(nt * sizeof(double));
  for (unsigned s = 0; s < nsub; ++s) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (mine) {
      double Tm[6];
#pragma unroll
      for (int q = 0; q < 6; ++q)
        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(Tm[q]) : "r"(at[q] + cur) : "memory");
      double ddT = 0.0;
      if (fl != 2) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const double Tp = Tm[2 * a], Tq = Tm[2 * a + 1];
          ddT += soft::div(soft::div(kd[a] * (Tq - Tp), hd[a]), hd[a]) * 0.25;
          ddT += kr * soft::div(soft::div(Tq + Tp - 2.0 * T, hd[a]), hd[a]);
        }
      }
      if (fl == 1) T += soft::div(ddT + dTr + Sr, rc) * inner_dt;
      if (T < 0.0) {
        T = 0.0;
        atomicAdd(&counters[CNT_T_CLAMP], 1ull);
      }
      s_T[(cur ? 0 : nt) + t] = T;
      if (rec) rec[(size_t)s * (size_t)F.nc + r] = T;
    }
    cur = half - cur;
  }
  if (mine) T0[r] = T;
  // no block leaves while another may still read its buffers
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Exact sum of the grid temperatures (EPH_FDM::get_T_total, eph_fdm.h:189-196).
__global__ void k_grid_sum(const double *__restrict__ T, long ncells, U128 *__restrict__ out,
                           unsigned *__restrict__ err) {
  U128 t{0ull, 0ull};
  for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x; r < ncells; r += (long)gridDim.x * blockDim.x)
    t = add128(t, to_fixed(T[r], err));
  for (int d = 16; d > 0; d >>= 1) t = add128(t, shfl_down128(t, d));
  if ((threadIdx.x & 31) == 0 && (t.lo | t.hi)) atomic_add128(out, t);
}

__global__ void k_from_fixed(const U128 *__restrict__ in, double *__restrict__ out) { *out = from_fixed(*in); }

// ------------------------------------------------------------ layout moves

// engine layout (n x 3) <-> padded device layout; w is kept
__global__ void k_pack3(int n, const double *__restrict__ src, D4 *__restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  D4 d = dst[i];
  d.x = src[3 * (size_t)i + 0];
  d.y = src[3 * (size_t)i + 1];
  d.z = src[3 * (size_t)i + 2];
  dst[i] = d;
}

__global__ void k_unpack3(int n, const D4 *__restrict__ src, double *__restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const D4 s = src[i];
  dst[3 * (size_t)i + 0] = s.x;
  dst[3 * (size_t)i + 1] = s.y;
  dst[3 * (size_t)i + 2] = s.z;
}

// per-atom array of the fix (fix_eph.cpp:406-428): rho, beta(rho), f_EPH, f_RNG
__global__ void k_peratom(int n, int groupbit, const int *__restrict__ mask, const double *__restrict__ rho,
                          const double *__restrict__ beta, const D4 *__restrict__ f_eph,
                          const D4 *__restrict__ f_rng, double *__restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double *o = out + 8 * (size_t)i;
  if (mask[i] & groupbit) {
    const D4 a = f_eph[i], b = f_rng[i];
    o[0] = rho[i];
    o[1] = beta[i];
    o[2] = a.x;
    o[3] = a.y;
    o[4] = a.z;
    o[5] = b.x;
    o[6] = b.y;
    o[7] = b.z;
  } else {
    for (int k = 0; k < 8; ++k) o[k] = 0.0;
  }
}

// rho and w in the engine layout
__global__ void k_get_w(int n, const D4 *__restrict__ Bw, double *__restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const D4 b = Bw[i];
  dst[3 * (size_t)i + 0] = b.y;
  dst[3 * (size_t)i + 1] = b.z;
  dst[3 * (size_t)i + 2] = b.w;
}

// the deviates the last post_force used (A.z, A.w, Bw.x)
__global__ void k_get_xi(int n, const D4 *__restrict__ A, const D4 *__restrict__ Bw, double *__restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  dst[3 * (size_t)i + 0] = A[i].z;
  dst[3 * (size_t)i + 1] = A[i].w;
  dst[3 * (size_t)i + 2] = Bw[i].x;
}

__global__ void k_set_elem(int n, const int *__restrict__ type, const int *__restrict__ type_map,
                           D4 *__restrict__ x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  x[i].w = (double)type_map[type[i]];
}

}  // namespace ephgb
