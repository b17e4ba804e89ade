// Pair helpers of the df64 sweeps, shared by the forward sweeps
// (eph_kernels.cuh) and the reverse sweeps of the adjoint (eph_adjoint.cu):
// the rho(r^2) spline of the local-form df64 tables and a pair's
// displacement from double-float coordinates.
#pragma once

#include "eph_device.cuh"
#include "eph_df64.cuh"

namespace ephgb {

// A 32-byte row {hi parts, lo parts} in one 256-bit load: rows of different
// lanes lie in different lines, and each 16-byte half loaded by itself costs
// the L1 as many wavefronts as the whole row.
__device__ __forceinline__ void load_row(const float4 *__restrict__ row, float4 &hi, float4 &lo) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(hi.x), "=f"(hi.y), "=f"(hi.z), "=f"(hi.w), "=f"(lo.x), "=f"(lo.y), "=f"(lo.z), "=f"(lo.w)
      : "l"(row));
}

// the same for a row that other kernels write and that is read once a step
__device__ __forceinline__ void load_row_once(const float4 *row, float4 &hi, float4 &lo) {
  asm volatile("ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(hi.x), "=f"(hi.y), "=f"(hi.z), "=f"(hi.w), "=f"(lo.x), "=f"(lo.y), "=f"(lo.z), "=f"(lo.w)
               : "l"(row));
}
__device__ __forceinline__ void store_row(float4 *row, float4 hi, float4 lo) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(row), "f"(hi.x), "f"(hi.y), "f"(hi.z),
               "f"(hi.w), "f"(lo.x), "f"(lo.y), "f"(lo.z), "f"(lo.w)
               : "memory");
}

__device__ __forceinline__ void load_record(const int4 *__restrict__ half, int4 &a, int4 &b) {
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
      : "l"(half));
}

// rho_e(x) of element e at x = r^2 from the local-form df64 table: knot
// k = floor(x / dx) from the FP32 quotient, moved by one where the df64
// offset t = x - k dx falls outside [0, dx) (so the interval is that of the
// df64 x, not of its FP32 part), then y = a' + t (b' + t (c' + t d')).  The
// local form was expanded from the reference's absolute-form cubic on the
// host (the same polynomial), so the value is the reference's spline to
// ~1e-14 without the cancellation of evaluating the absolute form at large x.
__device__ __forceinline__ df64::df spline_rho_df(const StepParams &P, int e, df64::df x, unsigned *err) {
  using namespace df64;
  // floor(x / dx) from the FP32 quotient without a conversion instruction
  // (floor_estimate; off by one at most, settled by the sign of t below)
  const float q = x.hi * P.inv_dxr_f;
  const float kr = floor_estimate(q);
  int k = floor_estimate_int(kr);
  float p, pe;
  two_prod(kr, P.dxr_hi, p, pe);
  pe = fmaf(kr, P.dxr_lo, pe);
  float th, te;
  two_sum(x.hi, -p, th, te);
  df t = make(th, (te + x.lo) - pe);
  const df dx = df{P.dxr_hi, P.dxr_lo};
  // rarely: x within an FP32 rounding of a knot (one test and a branch around
  // both corrections; k past the table only there or beyond it)
  if (!(t.hi >= 0.0f && t.hi < P.dxr_hi) || (unsigned)k >= (unsigned)P.n_rho) {
    if (t.hi < 0.0f) {
      k -= 1;
      t = add(t, dx);
    } else if (!(t.hi < P.dxr_hi)) {
      k += 1;
      t = sub(t, dx);
    }
    if (k < 0 || k >= P.n_rho) {
      atomicOr(err, ERR_SPLINE_RANGE);
      k = k < 0 ? 0 : P.n_rho - 1;
    }
  }
  float4 hi, lo;
  load_row(P.tab_rho_df + 2 * ((size_t)e * P.n_rho + k), hi, lo);
  return horner(df{hi.x, lo.x}, df{hi.y, lo.y}, df{hi.z, lo.z}, df{hi.w, lo.w}, t);
}

// The same spline's value and derivative d rho / d x at x, and its knot k
// (the interval whose coefficients the value comes from)
__device__ __forceinline__ void spline_rho_df_vd(const StepParams &P, int e, df64::df x, df64::df &val,
                                                 df64::df &der, int &k) {
  using namespace df64;
  const float q = x.hi * P.inv_dxr_f;
  const float kr = floor_estimate(q);
  k = floor_estimate_int(kr);
  float p, pe;
  two_prod(kr, P.dxr_hi, p, pe);
  pe = fmaf(kr, P.dxr_lo, pe);
  float th, te;
  two_sum(x.hi, -p, th, te);
  df t = make(th, (te + x.lo) - pe);
  const df dx = df{P.dxr_hi, P.dxr_lo};
  if (t.hi < 0.0f) {
    k -= 1;
    t = add(t, dx);
  } else if (!(t.hi < P.dxr_hi)) {
    k += 1;
    t = sub(t, dx);
  }
  k = k < 0 ? 0 : (k >= P.n_rho ? P.n_rho - 1 : k);
  float4 hi, lo;
  load_row(P.tab_rho_df + 2 * ((size_t)e * P.n_rho + k), hi, lo);
  const df a0{hi.x, lo.x}, a1{hi.y, lo.y}, a2{hi.z, lo.z}, a3{hi.w, lo.w};
  val = horner(a0, a1, a2, a3, t);
  // d/dt of a' + b' t + c' t^2 + d' t^3
  der = fma(t, fma(t, mul(df{3.0f, 0.0f}, a3), mul(df{2.0f, 0.0f}, a2)), a1);
}

// displacement component d w + (o_j - o_i) of a pair from double-float coordinates
__device__ __forceinline__ df64::df pair_disp(int d, float ojh, float ojl, float oih, float oil, float wh,
                                              float wl) {
  using namespace df64;
  float s, se;
  two_sum(ojh, -oih, s, se);
  const float dw = (float)d * wh;  // exact: d is -1, 0 or 1
  float s2, se2;
  two_sum(s, dw, s2, se2);
  return make(s2, ((ojl - oil) + se) + (se2 + (float)d * wl));
}

// ------------------------------------------ fixed-point pair displacements
//
// Positions of the df64 pair sums are 64-bit fixed point, 2^-P.fix_q A, kept
// modulo 2^64: an FP64 coordinate converts exactly (its last bit is far above
// the unit), the difference of two neighbours' is two integer additions and
// exact (any pair within the bins' radius is below a quarter of the range, so
// the wrap-around of the integers does not matter), and a periodic image is
// the box edge added, only for pairs across the boundary.  The difference
// splits into the double-float hi + lo by three conversions: 9 instructions
// per axis, with an error of one rounding of lo (2^-48 of the displacement).

// a coordinate (or box edge) in the fixed-point unit, modulo 2^64
__host__ __device__ __forceinline__ long long to_fixed_coord(double v, int q) {
#if defined(__CUDA_ARCH__)
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
#else
  union {
    double d;
    unsigned long long u;
  } w;
  w.d = v;
  const unsigned long long b = w.u;
#endif
  const int e = (int)((b >> 52) & 0x7ffu);
  if (e == 0) return 0;
  const unsigned long long m = (b & ((1ull << 52) - 1ull)) | (1ull << 52);
  const int sh = e - 1075 + q;
  unsigned long long r = 0;
  if (sh >= 0) r = sh < 64 ? m << sh : 0ull;
  else if (sh > -55) r = (m + (1ull << (-sh - 1))) >> -sh;  // half away from zero
  return (long long)((b >> 63) ? ~r + 1ull : r);
}

// a difference of fixed-point coordinates in A: hi the nearest float of its
// top 32 bits, lo the rest (fix_hi = 2^(32 - q), fix_lo = 2^(8 - q))
__device__ __forceinline__ df64::df fixed_df(long long e, float fix_hi, float fix_lo) {
  const int h = (int)(e >> 32);
  const float hf = __int2float_rn(h);
  const int r = h - __float2int_rn(hf);
  const int l = (int)__funnelshift_r((unsigned)e, (unsigned)r, 8);  // r 2^24 + the next 24 bits
  return df64::df{hf * fix_hi, __int2float_rn(l) * fix_lo};
}

// the record's fixed-point position (df_record: {x lo, x hi, y lo, y hi}, {z lo,
// z hi, element, moved}) plus the image of `code`, minus xi
__device__ __forceinline__ void pair_fixed(const StepParams &P, int4 a, int4 b, unsigned code, const long long *xi,
                                           long long *e) {
  e[0] = (((long long)a.y << 32) | (unsigned)a.x) - xi[0];
  e[1] = (((long long)a.w << 32) | (unsigned)a.z) - xi[1];
  e[2] = (((long long)b.y << 32) | (unsigned)b.x) - xi[2];
  if (code != CODE_NOSHIFT) {
    const int mx = (int)(code % 3u) - 1, my = (int)((code / 3u) % 3u) - 1, mz = (int)(code / 9u) - 1;
    e[0] += mx < 0 ? -P.fix_prd[0] : (mx > 0 ? P.fix_prd[0] : 0ll);
    e[1] += my < 0 ? -P.fix_prd[1] : (my > 0 ? P.fix_prd[1] : 0ll);
    e[2] += mz < 0 ? -P.fix_prd[2] : (mz > 0 ? P.fix_prd[2] : 0ll);
  }
}

// atom i's fixed-point position from its record
__device__ __forceinline__ void own_fixed(const int4 *__restrict__ rec, int i, long long *xf) {
  int4 a, b;
  load_record(rec + 4 * (size_t)i, a, b);
  xf[0] = ((long long)a.y << 32) | (unsigned)a.x;
  xf[1] = ((long long)a.w << 32) | (unsigned)a.z;
  xf[2] = ((long long)b.y << 32) | (unsigned)b.x;
}

// The record of atom i for the df64 pair sums, one 64-byte line half: {x lo,
// x hi, y lo, y hi}, {z lo, z hi, element, moved}, velocity hi parts, velocity
// lo parts.  Position in fixed point plus `image` boxes.
__device__ __forceinline__ void df_record_fixed(const StepParams &P, int i, const long long *at, int element,
                                                const int *image, bool moved, const D4 &v, int4 *__restrict__ rec) {
  long long f[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) f[k] = at[k] + (long long)image[k] * P.fix_prd[k];
  const df64::df vx = df64::from_double(v.x), vy = df64::from_double(v.y), vz = df64::from_double(v.z);
  int4 *r = rec + 4 * (size_t)i;
  r[0] = make_int4((int)f[0], (int)(f[0] >> 32), (int)f[1], (int)(f[1] >> 32));
  r[1] = make_int4((int)f[2], (int)(f[2] >> 32), element, moved ? 1 : 0);
  r[2] = make_int4(__float_as_int(vx.hi), __float_as_int(vy.hi), __float_as_int(vz.hi), 0);
  r[3] = make_int4(__float_as_int(vx.lo), __float_as_int(vy.lo), __float_as_int(vz.lo), 0);
}

__device__ __forceinline__ void df_record(const StepParams &P, int i, const D4 &x, const int *image, bool moved,
                                          const D4 &v, int4 *__restrict__ rec) {
  const long long f[3] = {to_fixed_coord(x.x, P.fix_q), to_fixed_coord(x.y, P.fix_q), to_fixed_coord(x.z, P.fix_q)};
  df_record_fixed(P, i, f, (int)trunc_index(x.w), image, moved, v, rec);
}

}  // namespace ephgb
