// Candidates of a pair sweep: the bin search over the 27 bins around an atom
// (one or several lanes per atom), the kept lists with their moved atoms, and
// the EAM engine's pair list.  Device functions shared by the fix's sweeps
// (eph_kernels.cuh) and the EAM sweeps (eph_eam.cu).
#pragma once

#include "eph_device.cuh"
#include "eph_df_pair.cuh"

namespace ephgb {

__device__ __forceinline__ double min_image(double d, double L, double h) {
  return d > h ? d - L : (d < -h ? d + L : d);
}

// The 3x3x3 image code of x_j seen from x_i: the image of x_j within half a
// box of x_i on every axis, decided in FP32 (the box is at least three list
// radii wide, so a pair within the list radius is far from the threshold).
// The pair vector then comes from density_vector, the rounding of the bin
// search path.
__device__ __forceinline__ unsigned image_code(const StepParams &P, float xi, float yi, float zi, const D4 &xj) {
  const float dx = float_bits(xj.x) - xi, dy = float_bits(xj.y) - yi, dz = float_bits(xj.z) - zi;
  const int mx = dx > P.half_prdf[0] ? -1 : (dx < -P.half_prdf[0] ? 1 : 0);
  const int my = dy > P.half_prdf[1] ? -1 : (dy < -P.half_prdf[1] ? 1 : 0);
  const int mz = dz > P.half_prdf[2] ? -1 : (dz < -P.half_prdf[2] ? 1 : 0);
  return (unsigned)((mx + 1) + 3 * (my + 1) + 9 * (mz + 1));
}

// The boxes that bring coordinate p of axis k into [lo, lo + L), and its offset
// there
__device__ __forceinline__ int wrap_image(const StepParams &P, int k, double p, double &q) {
  q = p - P.lo[k];
  const double turns = floor(q / P.prd[k]);
  q -= turns * P.prd[k];
  int image = -(int)turns;
  if (q >= P.prd[k]) {
    q -= P.prd[k];
    --image;
  }
  if (q < 0.0) q = 0.0;
  return image;
}

// The bin and FP32 offset of a position wrapped into the box (an atom whose
// bins entry is stale: it moved since the build), and the wrapped position
__device__ __forceinline__ void current_bin(const StepParams &P, const D4 &xi, int4 &B, float4 &o,
                                            double *wrapped = nullptr) {
  const double p[3] = {xi.x, xi.y, xi.z};
  int b[3];
  float of[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double q;
    const int image = wrap_image(P, k, p[k], q);
    if (wrapped) wrapped[k] = p[k] + image * P.prd[k];
    int bb = (int)floor(q * P.inv_w[k]);
    bb = bb < 0 ? 0 : (bb >= P.nb[k] ? P.nb[k] - 1 : bb);
    b[k] = bb;
    of[k] = (float)(q - (double)bb * P.w[k]);
  }
  B = make_int4(b[0], b[1], b[2], b[0] + P.nb[0] * (b[1] + P.nb[1] * b[2]));
  o = make_float4(of[0], of[1], of[2], 0.f);
}

// Append u to the candidate list of the lane's atom where `take`: with one
// lane per atom after the lane's own nc entries; with LANES lanes, which share
// the atom's list and all call this together, in lane order (nc, the list's
// length, stays the same on the atom's lanes).  At most cap entries.
template <int LANES, class Set>
__device__ __forceinline__ void append_candidate(bool take, unsigned u, int &nc, int cap, Set cset,
                                                 unsigned *__restrict__ err) {
  int pos = nc;
  if (LANES == 1) {
    if (take && nc < cap) ++nc;
  } else {
    const int lane = threadIdx.x & 31;
    const unsigned mine = (LANES == 32 ? 0xffffffffu : ((1u << LANES) - 1u) << (lane & ~(LANES - 1)));
    const unsigned who = __ballot_sync(0xffffffffu, take) & mine;
    pos += __popc(who & ((1u << lane) - 1u));
    nc += __popc(who);
    nc = nc < cap ? nc : cap;
  }
  if (take) {
    if (pos < cap) cset(pos, u);
    else atomicOr(err, ERR_PAIR_OVERFLOW);
  }
}

// Candidates of atom i in the bin at stencil offset (dx, dy, dz) from its
// own: the entries whose FP32 distance passes the widened cut-off, appended
// through cset in bin order while nc < cap.  Contains a warp-wide max: every lane of the
// warp calls it the same number of times (look = false for a lane with
// nothing to search).  r2band is the FP32 threshold (the cutoff's, or the
// candidate list's); with SKIP, entries of atoms flagged as moved (skip[j] &
// 2) are left out.
template <bool SKIP = false, class Set>
__device__ __forceinline__ void bin_candidates(const StepParams &P, int i, bool look, int4 Bi, float4 oi, int dx,
                                               int dy, int dz, const int *__restrict__ bin_count,
                                               const BinEntry *__restrict__ bins, unsigned *__restrict__ err,
                                               int &nc, int cap, Set cset, float r2band,
                                               const int *__restrict__ skip = nullptr, float r2lo = -1.f) {
  const int Tz = Bi.z + dz, tz = Tz < 0 ? Tz + P.nb[2] : (Tz >= P.nb[2] ? Tz - P.nb[2] : Tz);
  const int kz = Tz < 0 ? -1 : (Tz >= P.nb[2] ? 1 : 0);
  const float bz = (float)dz * P.wf[2] - oi.z;
  const int Ty = Bi.y + dy, ty = Ty < 0 ? Ty + P.nb[1] : (Ty >= P.nb[1] ? Ty - P.nb[1] : Ty);
  const int ky = Ty < 0 ? -1 : (Ty >= P.nb[1] ? 1 : 0);
  const float by = (float)dy * P.wf[1] - oi.y;
  const int Tx = Bi.x + dx, tx = Tx < 0 ? Tx + P.nb[0] : (Tx >= P.nb[0] ? Tx - P.nb[0] : Tx);
  const int kx = Tx < 0 ? -1 : (Tx >= P.nb[0] ? 1 : 0);
  const float bx = (float)dx * P.wf[0] - oi.x;
  const int flat = tx + P.nb[0] * (ty + P.nb[1] * tz);
  int cnt = 0;
  if (look) {
    cnt = bin_count[flat];
    cnt = cnt < P.bcap ? cnt : P.bcap;
  }
  const int cmax = __reduce_max_sync(0xffffffffu, cnt);
  const BinEntry *be = bins + (size_t)flat * P.bcap;
  for (int s = 0; s < cmax; ++s) {
    if (s < cnt) {
      const BinEntry b = be[s];
      const unsigned j = b.idx & IDX_MASK;
      const float ex = bx + b.ox, ey = by + b.oy, ez = bz + b.oz;
      const float r2 = ex * ex + ey * ey + ez * ez;
      if (j != (unsigned)i && r2 < r2band && r2 >= r2lo && !(SKIP && (skip[j] & 2))) {
        const unsigned wc = b.idx >> IDX_BITS;
        const int mx = kx - ((int)(wc % 3u) - 1), my = ky - ((int)((wc / 3u) % 3u) - 1),
                  mz = kz - ((int)(wc / 9u) - 1);
        if (mx < -1 || mx > 1 || my < -1 || my > 1 || mz < -1 || mz > 1) {
          atomicOr(err, ERR_DRIFT);
        } else if (nc >= cap) {
          atomicOr(err, ERR_PAIR_OVERFLOW);
        } else {
          const unsigned u = j | ((unsigned)((mx + 1) + 3 * (my + 1) + 9 * (mz + 1)) << IDX_BITS);
          cset(nc++, u);
        }
      }
    }
  }
}

// bin_candidates over all 27 bins with LANES lanes per atom: lane g
// takes bins g, g + LANES, ... of the stencil and the lanes append to the
// atom's one list what `keep` does not refuse (a candidate and its FP32 r^2).
// Every lane of the warp calls it.
struct KeepAll {
  __device__ bool operator()(unsigned, float) const { return true; }
};
template <int LANES, bool SKIP = false, class Set, class Keep = KeepAll>
__device__ __forceinline__ void shared_candidates(const StepParams &P, int i, bool active, int4 Bi, float4 oi,
                                                  const int *__restrict__ bin_count,
                                                  const BinEntry *__restrict__ bins, unsigned *__restrict__ err,
                                                  int &nc, int cap, Set cset, float r2band,
                                                  const int *__restrict__ skip = nullptr, float r2lo = -1.f,
                                                  Keep keep = Keep()) {
  constexpr int CHUNK = 4;
  const int g = (int)threadIdx.x & (LANES - 1);
  for (int m = 0; m < (27 + LANES - 1) / LANES; ++m) {
    const int b = g + m * LANES;
    const bool look = active && b < 27;
    const int bb = b < 27 ? b : 13, dx = bb % 3 - 1, dy = (bb / 3) % 3 - 1, dz = bb / 9 - 1;
    const int Tz = Bi.z + dz, tz = Tz < 0 ? Tz + P.nb[2] : (Tz >= P.nb[2] ? Tz - P.nb[2] : Tz);
    const int Ty = Bi.y + dy, ty = Ty < 0 ? Ty + P.nb[1] : (Ty >= P.nb[1] ? Ty - P.nb[1] : Ty);
    const int Tx = Bi.x + dx, tx = Tx < 0 ? Tx + P.nb[0] : (Tx >= P.nb[0] ? Tx - P.nb[0] : Tx);
    const int kz = Tz < 0 ? -1 : (Tz >= P.nb[2] ? 1 : 0), ky = Ty < 0 ? -1 : (Ty >= P.nb[1] ? 1 : 0),
              kx = Tx < 0 ? -1 : (Tx >= P.nb[0] ? 1 : 0);
    const float bx = (float)dx * P.wf[0] - oi.x, by = (float)dy * P.wf[1] - oi.y, bz = (float)dz * P.wf[2] - oi.z;
    const int flat = tx + P.nb[0] * (ty + P.nb[1] * tz);
    const BinEntry *be = bins + (size_t)flat * P.bcap;
    // entries CHUNK at a time, the first ones beside the count (slots past it
    // are read, not used): one memory latency per chunk instead of per entry
    BinEntry e[CHUNK];
#pragma unroll
    for (int c = 0; c < CHUNK; ++c) e[c] = be[c < P.bcap ? c : 0];
    int cnt = 0;
    if (look) {
      cnt = bin_count[flat];
      cnt = cnt < P.bcap ? cnt : P.bcap;
    }
    const int cmax = __reduce_max_sync(0xffffffffu, cnt);
    for (int s0 = 0; s0 < cmax; s0 += CHUNK) {
      if (s0) {
#pragma unroll
        for (int c = 0; c < CHUNK; ++c)
          if (s0 + c < cnt) e[c] = be[s0 + c];
      }
#pragma unroll
      for (int c = 0; c < CHUNK; ++c) {
        bool take = false;
        unsigned u = 0;
        if (s0 + c < cnt) {
          const unsigned j = e[c].idx & IDX_MASK;
          const float ex = bx + e[c].ox, ey = by + e[c].oy, ez = bz + e[c].oz;
          const float r2 = ex * ex + ey * ey + ez * ez;
          if (j != (unsigned)i && r2 < r2band && r2 >= r2lo && !(SKIP && (skip[j] & 2))) {
            const unsigned wc = e[c].idx >> IDX_BITS;
            const int mx = kx - ((int)(wc % 3u) - 1), my = ky - ((int)((wc / 3u) % 3u) - 1),
                      mz = kz - ((int)(wc / 9u) - 1);
            take = mx >= -1 && mx <= 1 && my >= -1 && my <= 1 && mz >= -1 && mz <= 1;
            if (!take) atomicOr(err, ERR_DRIFT);
            u = j | ((unsigned)((mx + 1) + 3 * (my + 1) + 9 * (mz + 1)) << IDX_BITS);
            take = take && keep(u, r2);
          }
        }
        append_candidate<LANES>(take, u, nc, cap, cset, err);
      }
    }
  }
}

// Pass 1 of the density sweep for atom i: the candidates of the 27 bins
// around its own within the FP32 thresholds r2lo <= r^2 < r2band, appended
// after the first nc0 (at most cap in all).  Returns their number.
template <bool SKIP = false, class Set>
__device__ __forceinline__ int collect_candidates(const StepParams &P, int i, bool active, int4 Bi, float4 oi,
                                                  const int *__restrict__ bin_count,
                                                  const BinEntry *__restrict__ bins, unsigned *__restrict__ err,
                                                  Set cset, float r2band, int cap,
                                                  const int *__restrict__ skip = nullptr, float r2lo = -1.f,
                                                  int nc0 = 0) {
  int nc = nc0;
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx)
        bin_candidates<SKIP>(P, i, active, Bi, oi, dx, dy, dz, bin_count, bins, err, nc, cap, cset,
                                   r2band, skip, r2lo);
  return nc;
}

// the FP32 r^2 of candidate u from position xi, by the high words of the
// fixed-point positions of this step
__device__ __forceinline__ float pair_r2(const StepParams &P, const int4 *__restrict__ rec, unsigned u,
                                         const long long *xi) {
  long long e[3];
  int4 ra, rb;
  load_record(rec + 4 * (size_t)(u & IDX_MASK), ra, rb);
  pair_fixed(P, ra, rb, u >> IDX_BITS, xi, e);
  const float ex = (float)(int)(e[0] >> 32) * P.fix_hi, ey = (float)(int)(e[1] >> 32) * P.fix_hi,
              ez = (float)(int)(e[2] >> 32) * P.fix_hi;
  return ex * ex + ey * ey + ez * ez;
}

// Pass 1 from the standalone engine's EAM pair list of this step
// (k_eam_density's rows: every pair within the EAM cut-off, which exceeds
// r2band): its entries within the FP32 threshold r2band, from the high words
// of the fixed-point positions -- the candidates of the bin search, without
// scanning the bins.  Lane g of the atom's LANES takes entries g, g + LANES,
// ....
template <int LANES, class Set, class Keep = KeepAll>
__device__ __forceinline__ void list_candidates(const StepParams &P, int i, bool active, const long long *xi,
                                                const unsigned *__restrict__ elist, const int *__restrict__ ens,
                                                const int4 *__restrict__ rec, unsigned *__restrict__ err, int &nc,
                                                int cap, Set cset, float r2band, Keep keep = Keep()) {
  const int g = (int)threadIdx.x & (LANES - 1);
  const int ne = active ? ens[i] : 0;
  const int nmax = __reduce_max_sync(0xffffffffu, ne);
  for (int k = g; k - g < nmax; k += LANES) {
    bool take = false;
    unsigned u = 0;
    if (k < ne) {
      u = elist[(size_t)k * P.n + i];
      const float r2 = pair_r2(P, rec, u, xi);
      take = r2 < r2band && keep(u, r2);
    }
    append_candidate<LANES>(take, u, nc, cap, cset, err);
  }
}

// what the candidate search reads
struct CandidateArgs {
  const int *bin_count;
  const BinEntry *bins;
  const int4 *atom_bin;
  const float4 *atom_off;
  const int4 *rec;
  const D4 *x;
  unsigned *err;
  // rows of the sweep's own pair list (kcap of them), which also hold the
  // candidates that have no room in shared memory (and a moved atom's, without
  // `moved`): a row is written only after the candidate there is read
  unsigned *pj;
  int kcap;
  float band;  // FP32 threshold of the cut-off
  // kept lists
  unsigned *cl;
  int *cl_n;
  const int *state, *rb, *flist;
  const D4 *xref;
  int *partial;    // set by a build that leaves the atoms outside the group without lists of this build (or null)
  const D4 *fpos;  // the moved atoms' positions wrapped into the box
  float far2;      // the moved atoms' widened cut-off (far_cutoff2)
  // candidates of the moved atoms, mcap each (all that their bins can hold, and
  // every moved atom), for a sweep that keeps other pairs in their rows of pj
  unsigned *moved;
  int mcap;
};

// The candidates of atom i from the bins of this step or the kept lists,
// LANES lanes to an atom (g: the lane's number); none where it is not active.
// `at(k)`, k < CAP, is the
// shared-memory place of candidate k; further ones go to the atom's rows of
// pj, or stay in the list (`tail`: where number 0 would be; number k is k `step`
// on, which is n but for a moved atom's with MOVED_ROWS).  Of the candidates
// before number `first` those flagged as moved do not count: a list's entries
// for them are of the build.
// Kept lists: build steps search the bins within r_list and write the lists;
// atoms that moved (k_list_check) search the bins of the build, atoms near one
// (k_list_mark) take their list, and both then add the moved atoms.  What a moved
// atom finds is tested with the positions of this step, so that it needs no more
// rows than a search of this step's bins; it waits in the atom's rows of pj, or
// with MOVED_ROWS in rows of its own (C.moved), where the sweep writes pairs to
// the far end of pj's rows: nothing would keep those off candidates not read
// yet, and with half the box empty, rows for half the neighbours, they were lost.
// A cascade's few hundred such atoms sit in a few
// warps, whose latency is the sweep's tail: searching bin after bin with the
// one lane, for both kinds, made the sweep 215 us at 131,072 atoms of two
// elements on GB300; 154 now, as without moved atoms.
// Every lane of the warp calls it.
template <int LANES, bool LIST, bool MOVED_ROWS, int CAP, class At>
__device__ __forceinline__ int pair_candidates(const StepParams &P, const CandidateArgs &C, int i, int g, bool active, At at,
                                               const unsigned *&tail, unsigned &step, int &first) {
  const size_t n = (size_t)P.n;
  int nc = 0;
  first = 0;
  step = (unsigned)P.n;
  tail = C.pj + i;
  auto set = [&](int k, unsigned u) {
    if (k < CAP) at(k) = u;
    else C.pj[(size_t)k * n + i] = u;
  };
  if (!LIST) {
    int4 Bi = make_int4(0, 0, 0, 0);
    float4 oi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (active) {
      Bi = C.atom_bin[i];
      oi = C.atom_off[i];
    }
    if (LANES == 1)
      nc = collect_candidates(P, i, active, Bi, oi, C.bin_count, C.bins, C.err, set, C.band, C.kcap);
    else
      shared_candidates<LANES>(P, i, active, Bi, oi, C.bin_count, C.bins, C.err, nc, C.kcap, set, C.band);
    return nc;
  }
  if (C.rb[2] != 0) {  // a build step
    int4 Bi = make_int4(0, 0, 0, 0);
    float4 oi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (active) {
      Bi = C.atom_bin[i];
      oi = C.atom_off[i];
    }
    auto lset = [&](int k, unsigned u) {
      if (k < CAP) at(k) = u;
      C.cl[(size_t)k * n + i] = u;
    };
    // the candidates inside the cut-off first, the shell out to r_list after
    // them: the shell's pairs mostly fail the exact test, and at the end of
    // the lists whole warps skip them
    if (LANES == 1) {
      nc = collect_candidates(P, i, active, Bi, oi, C.bin_count, C.bins, C.err, lset, C.band, P.lcap);
      nc = collect_candidates(P, i, active, Bi, oi, C.bin_count, C.bins, C.err, lset, P.rl2_band, P.lcap,
                              nullptr, C.band, nc);
    } else {
      shared_candidates<LANES>(P, i, active, Bi, oi, C.bin_count, C.bins, C.err, nc, P.lcap, lset, C.band);
      shared_candidates<LANES>(P, i, active, Bi, oi, C.bin_count, C.bins, C.err, nc, P.lcap, lset, P.rl2_band, nullptr,
                               C.band);
    }
    tail = C.cl + i;
    // an atom that is not active keeps the list that another sweep made
    if (active && g == 0) C.cl_n[i] = nc;
    if (C.partial && i == 0 && g == 0) *C.partial = 1;
    return nc;
  }
  const int st = active ? C.state[i] : 0;
  const bool near = st != 0;
  if (__any_sync(0xffffffffu, near)) {
    int4 Bi = make_int4(0, 0, 0, 0);
    float4 oi = make_float4(0.f, 0.f, 0.f, 0.f);
    double base[3] = {0.0, 0.0, 0.0};  // the position in the record
    if (near) {
      const D4 x = C.x[i];
      if (st & 2) {
        current_bin(P, x, Bi, oi, base);
      } else {
        const D4 r = C.xref[i];
        base[0] = r.x + min_image(x.x - r.x, P.prd[0], P.half_prd[0]);
        base[1] = r.y + min_image(x.y - r.y, P.prd[1], P.half_prd[1]);
        base[2] = r.z + min_image(x.z - r.z, P.prd[2], P.half_prd[2]);
      }
    }
    // an atom that moved searches the bins of the build, the whole warp for one
    // such atom after the other
    const int nf = C.rb[1];  // <= LIST_FMAX on a step without a build
    int room = C.kcap;
    unsigned *rows = C.pj + i;
    for (unsigned todo = __ballot_sync(0xffffffffu, (st & 2) != 0 && g == 0); todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      const int is = __shfl_sync(0xffffffffu, i, src);
      const int4 Bs = make_int4(__shfl_sync(0xffffffffu, Bi.x, src), __shfl_sync(0xffffffffu, Bi.y, src),
                                __shfl_sync(0xffffffffu, Bi.z, src), 0);
      const float4 os = make_float4(__shfl_sync(0xffffffffu, oi.x, src), __shfl_sync(0xffffffffu, oi.y, src),
                                    __shfl_sync(0xffffffffu, oi.z, src), 0.f);
      int found = 0;
      unsigned *own = C.pj + is;
      if (MOVED_ROWS) {  // the moved atoms' order in flist
        const int lane = (int)threadIdx.x & 31;
        own = C.moved + (size_t)(__ffs(__ballot_sync(0xffffffffu, lane < nf && C.flist[lane] == is)) - 1) * C.mcap;
      }
      const size_t next = MOVED_ROWS ? 1 : n;
      const int most = MOVED_ROWS ? C.mcap : C.kcap;
      long long xs[3];
      own_fixed(C.rec, is, xs);
      auto row = [&](int k, unsigned u) { own[(size_t)k * next] = u; };
      auto near_now = [&](unsigned u, float) { return pair_r2(P, C.rec, u, xs) < C.band; };
      shared_candidates<32, true>(P, is, true, Bs, os, C.bin_count, C.bins, C.err, found, most, row, P.rl2_band,
                                  C.state, -1.f, near_now);
      if (i == is) {
        nc = found;
        if (MOVED_ROWS) {
          rows = own;
          step = 1;
          room = most;
        }
      }
    }
    // one that did not, but is near one that did, has the unmoved ones in its
    // list, whose rows past the end take the moved ones
    if (st == 1) {
      nc = first = C.cl_n[i];
      rows = C.cl + i;
      room = P.lcap;
    }
    tail = rows;
    const size_t next = MOVED_ROWS ? step : n;
    auto add = [&](int k, unsigned u) { rows[(size_t)k * next] = u; };
    // the moved atoms near enough (a widened FP32 test; the exact one decides),
    // their image next to the position above; the atom's lanes take turns
    for (int q = g; q - g < nf; q += LANES) {
      bool take = false;
      unsigned u = 0;
      if (near && q < nf) {
        const int f = C.flist[q];
        const D4 w = C.fpos[q];
        const double d[3] = {w.x - base[0], w.y - base[1], w.z - base[2]};
        float r2 = 0.0f;
        unsigned code = 0, place = 1;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float df = float_bits(d[k]), half = P.half_prdf[k];
          const int m = df > half ? -1 : (df < -half ? 1 : 0);
          const float c = df + (float)(2 * m) * half;
          r2 += c * c;
          code += (unsigned)(m + 1) * place;
          place *= 3u;
        }
        take = f != i && r2 < C.far2;
        u = (unsigned)f | (code << IDX_BITS);
      }
      append_candidate<LANES>(take, u, nc, room, add, C.err);
    }
  }
  if (!near) {
    tail = C.cl + i;
    nc = active ? C.cl_n[i] : 0;
    first = nc;
  }
  return nc;
}

}  // namespace ephgb
