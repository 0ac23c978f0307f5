// plain_f64.cu -- FP64 kernels with the reference's arithmetic (sm_100a).
//
// Compiled with -fmad=false: every multiply and add rounds on its own, as in
// pyFTLE's numpy / numba / generic-x86-64 C++ code, so HOLD-mode positions
// are bit-exact with the reference and BLEND-mode positions bit-exact with
// the CPU oracle.  Division and sqrt are IEEE (CUDA's FP64 defaults).
//
// Reference operations restated here (paths inside pyFTLE):
//   physical -> index  grid_interp.py:76-81, 163-168   ((x - min) / delta)
//   bilinear           GridInterp.cpp:93-142           (operand order :136-137)
//   trilinear          GridInterp.cpp:15-91            (lerp x, then y, then z)
//   Euler / AB2 / RK4  integrate.py:16-109, 177-342
//   Jacobian           cauchy_green.py:15-76, 79-153
//   CG, lambda, FTLE   ftle.py:9-233
#include <math.h>

#include "common.cuh"

namespace ftle {

// ---------------------------------------------------------------------------
// cell location and interpolation (bit-exact with the reference)
// ---------------------------------------------------------------------------

// The cell of a point: the record of its lower corner, byte steps to the next node along
// each axis, in-cell fractions.
template <int DIM>
struct Cell64 {
  const char *p;
  long long d[DIM];
  double f[DIM];
};

// v / spacing for any dividend and spacing, as IEEE division rounds it: the reciprocal form of
// grid_coords on mantissas in [1, 2) (man_* from the host), scaled afterwards in two factors.
// Zeros, infinities and NaN keep their class and sign.
__device__ __forceinline__ double div_scaled(double v, const GridK &g, int a) {
  const double sign = g.spacing[a] < 0.0 ? -1.0 : 1.0;
  if (v == 0.0 || !(fabs(v) <= 1.7976931348623157e308)) return v * sign;
  int e = -1023;
  if (fabs(v) < 2.2250738585072014e-308) {  // subnormal
    v *= 0x1p60;
    e -= 60;
  }
  const int hw = __double2hiint(v);
  e += (hw >> 20) & 0x7ff;
  const double m = __hiloint2double((hw & 0x800fffff) | 0x3ff00000, __double2loint(v));
  const double q0 = fma(m, g.man_hi[a], m * g.man_lo[a]);
  const double q = fma(fma(-q0, g.man[a], m), g.man_hi[a], q0);
  e -= g.man_exp[a];
  e = e < -1200 ? -1200 : (e > 1200 ? 1200 : e);
  const int half = e >> 1;  // two factors inside the exponent range
  return q * __hiloint2double((1023 + half) << 20, 0) *
         __hiloint2double((1023 + e - half) << 20, 0);
}

// (x - origin) / spacing per axis as IEEE division rounds it, by multiplication.  With
// 1/s = hi + lo (hi = RN(1/s), both from the host) q0 = RN(a hi + RN(a lo)) is within half
// an ulp plus 2^-53 ulp of a/s, r = a - q0 s is exact in an FMA, and the last FMA's
// argument q0 + r hi differs from a/s by less than the distance of any quotient of two
// 53-bit numbers from a rounding boundary, so it rounds as a/s does.  That needs s and a
// away from the ends of the exponent range: below div_min (the host's; every dividend where a
// spacing is extreme) a dividend, zeros among them, takes div_scaled.  Infinities, NaN and
// dividends that overflow come out not finite, which locate64 rejects as it does the quotient.
// (4 instructions instead of ~12 and a subroutine's registers; see window_f64_kernel.)
template <int DIM>
__device__ __forceinline__ void grid_coords(const GridK &g, const double *x, double *p) {
  unsigned least = 0x7fffffffu;
#pragma unroll
  for (int a = 0; a < DIM; ++a) {
    const double v = x[a] - g.origin[a];
    least = min(least, (unsigned)__double2hiint(v) & 0x7fffffffu);
    const double q0 = fma(v, g.rcp_hi[a], v * g.rcp_lo[a]);
    p[a] = fma(fma(-q0, g.spacing[a], v), g.rcp_hi[a], q0);
  }
  if (least < g.div_min) {
#pragma unroll
    for (int a = 0; a < DIM; ++a) p[a] = div_scaled(x[a] - g.origin[a], g, a);
  }
}

// Node stride of each axis in the meshgrid-"xy" order (2D j*nx + i, 3D (j*nx + i)*nz + k).
template <int DIM>
__device__ __forceinline__ long long node_stride(const GridK &g, int a) {
  if constexpr (DIM == 2) return a == 0 ? 1 : g.n[0];
  return a == 0 ? g.n[2] : (a == 1 ? (long long)g.n[0] * g.n[2] : 1);
}

// GridInterp.cpp's floor and "x0 >= 0 && x0+1 < n" test, equal for every finite p, which
// also rejects NaN / inf (the reference rejects them through the INT_MIN its float->int
// conversion returns).  Periodic grids wrap the cell instead.  Adding 1.5 * 2^52 rounding
// down leaves floor(p) in the low word and 0x43380000 (plus its sign) in the high word for
// |p| < 2^31: two FP64 additions in place of three conversions on the quarter-rate unit.
// RB: bytes of a node's record at `base`.
template <int DIM, int RB>
__device__ __forceinline__ bool locate64(const GridK &g, const void *base, const double *x,
                                         Cell64<DIM> &c) {
  constexpr double kMagic = 6755399441055744.0;
  double p[DIM];
  grid_coords<DIM>(g, x, p);
  bool ok = true;
  long long node = 0;
#pragma unroll
  for (int a = 0; a < DIM; ++a) {
    const double t = __dadd_rd(p[a], kMagic);
    c.f[a] = p[a] - (t - kMagic);
    int q = __double2loint(t);
    const int n = g.n[a];
    const long long stride = node_stride<DIM>(g, a);
    c.d[a] = stride * RB;
    if (g.periodic) {
      ok = ok && __double2hiint(t) == 0x43380000 + (q >> 31) &&
           (unsigned)(q + 999999999) <= 1999999998u;
      if ((unsigned)q >= (unsigned)n) {  // usually within one period of the grid
        q += q < 0 ? n : -n;
        if ((unsigned)q >= (unsigned)n) q = wrap_index(q, n);
      }
      if (q + 1 == n) c.d[a] = -(long long)(n - 1) * stride * RB;
    } else {
      ok = ok && __double2hiint(t) == 0x43380000 && (unsigned)q < (unsigned)(n - 1);
    }
    node += q * stride;
  }
  c.p = static_cast<const char *>(base) + node * RB;
  return ok;
}

// Corner records in the reference's operand order:
//   2D v00 v10 v01 v11;  3D x0y0z0 x1y0z0 x0y0z1 x1y0z1 x0y1z0 x1y1z0 x0y1z1 x1y1z1
template <int DIM>
__device__ __forceinline__ void corners(const Cell64<DIM> &c, const char **r) {
  constexpr int kSecond = DIM == 2 ? 1 : 2;  // the axis that moves second
  r[0] = c.p;
  r[1] = r[0] + c.d[0];
  r[2] = r[0] + c.d[kSecond];
  r[3] = r[1] + c.d[kSecond];
  if constexpr (DIM == 3) {
#pragma unroll
    for (int q = 0; q < 4; ++q) r[4 + q] = r[q] + c.d[1];
  }
}

__device__ __forceinline__ double bilinear(double v00, double v10, double v01, double v11,
                                           double xd, double yd) {
  return v00 * (1.0 - xd) * (1.0 - yd) + v10 * xd * (1.0 - yd) + v01 * (1.0 - xd) * yd +
         v11 * xd * yd;
}

__device__ __forceinline__ double trilinear(const double *v, double xd, double yd, double zd) {
  const double c00 = v[0] * (1.0 - xd) + v[1] * xd;
  const double c01 = v[2] * (1.0 - xd) + v[3] * xd;
  const double c10 = v[4] * (1.0 - xd) + v[5] * xd;
  const double c11 = v[6] * (1.0 - xd) + v[7] * xd;
  const double c0 = c00 * (1.0 - yd) + c10 * yd;
  const double c1 = c01 * (1.0 - yd) + c11 * yd;
  return c0 * (1.0 - zd) + c1 * zd;
}

template <int DIM>
__device__ __forceinline__ double interp_corners(const double *v, const double *f) {
  if constexpr (DIM == 2)
    return bilinear(v[0], v[1], v[2], v[3], f[0], f[1]);
  else
    return trilinear(v, f[0], f[1], f[2]);
}

// Velocity from one reference-layout (dim, nodes) snapshot.
template <int DIM>
__device__ __forceinline__ void velocity_planar(const GridK &g, const double *__restrict__ snap,
                                                const double *x, double *u) {
  Cell64<DIM> c;
  if (!locate64<DIM, 8>(g, snap, x, c)) {
#pragma unroll
    for (int a = 0; a < DIM; ++a) u[a] = 0.0;
    return;
  }
  const char *r[1 << DIM];
  corners<DIM>(c, r);
#pragma unroll
  for (int comp = 0; comp < DIM; ++comp) {
    double v[1 << DIM];
#pragma unroll
    for (int q = 0; q < (1 << DIM); ++q)
      v[q] = __ldg(reinterpret_cast<const double *>(r[q] + comp * g.nodes * 8));
    u[comp] = interp_corners<DIM>(v, c.f);
  }
}

// ---------------------------------------------------------------------------
// packed FP64 snapshot records: record (s, node) = [snapshot s | successor]
// ---------------------------------------------------------------------------

// The (time-blended) corner values a thread interpolated last.  RK4's third stage has the
// time of the second and, a fraction of a cell away, nearly always its cell; so have the
// first stage of a step and the last of the step before where t + h rounds to the next t.
// Such a stage takes the values from here: the same bits, without the loads and the blend.
template <int DIM>
struct Corners64 {
  const char *p = nullptr;  // record of the lower corner in its snapshot
  double alpha;
  double v[DIM][1 << DIM];
};

// HOLD: only the first half is read.  2D record = 4 doubles, 3D = 6 doubles
// (48 bytes, so every record is 16-byte aligned).
template <int DIM, bool BLEND, bool TRY>
__device__ __forceinline__ void velocity_packed(const GridK &g, const double *__restrict__ rec,
                                                double alpha, const double *x, double *u,
                                                Corners64<DIM> &last) {
  Cell64<DIM> c;
  if (!locate64<DIM, 16 * DIM>(g, rec, x, c)) {
#pragma unroll
    for (int a = 0; a < DIM; ++a) u[a] = 0.0;
    return;
  }
  if (!TRY || c.p != last.p || (BLEND && alpha != last.alpha)) {
    last.p = c.p;
    last.alpha = alpha;
    const char *rp[1 << DIM];
    corners<DIM>(c, rp);
    const double oma = 1.0 - alpha;
#pragma unroll
    for (int q = 0; q < (1 << DIM); ++q) {
      const double *r = reinterpret_cast<const double *>(rp[q]);
      const double2 a = __ldg(reinterpret_cast<const double2 *>(r));
      if constexpr (DIM == 2) {
        if constexpr (BLEND) {
          const double2 b = __ldg(reinterpret_cast<const double2 *>(r) + 1);
          last.v[0][q] = a.x * oma + b.x * alpha;
          last.v[1][q] = a.y * oma + b.y * alpha;
        } else {
          last.v[0][q] = a.x;
          last.v[1][q] = a.y;
        }
      } else {
        if constexpr (BLEND) {
          const double2 m = __ldg(reinterpret_cast<const double2 *>(r) + 1);
          const double2 b = __ldg(reinterpret_cast<const double2 *>(r) + 2);
          last.v[0][q] = a.x * oma + m.y * alpha;
          last.v[1][q] = a.y * oma + b.x * alpha;
          last.v[2][q] = m.x * oma + b.y * alpha;
        } else {
          last.v[0][q] = a.x;
          last.v[1][q] = a.y;
          last.v[2][q] = __ldg(r + 2);
        }
      }
    }
  }
#pragma unroll
  for (int comp = 0; comp < DIM; ++comp) u[comp] = interp_corners<DIM>(last.v[comp], c.f);
}

// The same velocity from the snapshots as the caller has them, (S, dim, nodes): the successor's
// corners are read and blended in the records' order, so the bits are those of packed records.
template <int DIM, bool BLEND>
__device__ __forceinline__ void velocity_source(const WinK &w, int s, double alpha,
                                                const double *x, double *u) {
  const GridK &g = w.g;
  const long long set = g.nodes * DIM;
  Cell64<DIM> c;
  if (!locate64<DIM, 8>(g, static_cast<const double *>(w.snaps) + s * set, x, c)) {
#pragma unroll
    for (int a = 0; a < DIM; ++a) u[a] = 0.0;
    return;
  }
  const int next = s + 1 < w.num_snaps ? s + 1 : (w.periodic_time ? 0 : w.num_snaps - 1);
  const long long to_next = (next - s) * set * 8;
  const double oma = 1.0 - alpha;
  const char *r[1 << DIM];
  corners<DIM>(c, r);
#pragma unroll
  for (int comp = 0; comp < DIM; ++comp) {
    double v[1 << DIM];
#pragma unroll
    for (int q = 0; q < (1 << DIM); ++q) {
      const char *p = r[q] + comp * g.nodes * 8;
      v[q] = __ldg(reinterpret_cast<const double *>(p));
      if constexpr (BLEND)
        v[q] = v[q] * oma + __ldg(reinterpret_cast<const double *>(p + to_next)) * alpha;
    }
    u[comp] = interp_corners<DIM>(v, c.f);
  }
}

// ---------------------------------------------------------------------------
// time lookup (BLEND)
// ---------------------------------------------------------------------------

// Snapshot record and blend weight at time t (record s pairs s with its successor).
__device__ __forceinline__ void time_pair(const WinK &w, double t, int &s0, double &alpha) {
  double tau = (t - w.snap_t0) / w.snap_dt;
  const int S = w.num_snaps;
  if (w.periodic_time) {
    tau = tau - (double)S * floor(tau / (double)S);
    int s = (int)floor(tau);
    s = s >= S ? S - 1 : (s < 0 ? 0 : s);
    s0 = s;
    alpha = tau - (double)s;
  } else if (!(tau > 0.0)) {
    s0 = 0;
    alpha = 0.0;
  } else if (tau >= (double)(S - 1)) {
    s0 = S - 2;
    alpha = 1.0;
  } else {
    const int s = (int)floor(tau);
    s0 = s;
    alpha = tau - (double)s;
  }
}

// The time lookups of a run of steps, shared by the lanes of a warp: lane PTS*k + c holds
// point c (t, t + h/2, t + h) of step first + k, so a lookup and its two divisions run once
// per 10 RK4 steps (32 Euler / AB2 steps) instead of once per particle and stage; a stage
// takes its pair from the lane that holds it.
template <int MODE, int INTEG>
struct StepTimes {
  static constexpr int kPoints = INTEG == FTLE_RK4 ? 3 : 1;
  static constexpr int kSteps = 32 / kPoints;
  int s = 0;
  double alpha = 0.0;
  __device__ __forceinline__ void load(const WinK &w, int first) {
    if constexpr (MODE == FTLE_BLEND) {
      const int lane = threadIdx.x & 31, c = lane % kPoints;
      const double t = w.t0 + (double)(first + lane / kPoints) * w.h;
      time_pair(w, c == 0 ? t : (c == 1 ? t + 0.5 * w.h : t + w.h), s, alpha);
    }
  }
};

// Velocity at point c of the k-th step of `times` (step number `step`).
template <int DIM, bool TRY, bool SOURCE, int MODE, int INTEG>
__device__ __forceinline__ void field(const WinK &w, const StepTimes<MODE, INTEG> &times, int k,
                                      int step, int c, const double *x, double *u,
                                      Corners64<DIM> &last) {
  const double *recs = static_cast<const double *>(w.snaps);
  const long long rec_set = w.g.nodes * (2 * DIM);
  if constexpr (MODE == FTLE_HOLD) {
    int s = w.first_snapshot + step;
    if (w.periodic_time) s %= w.num_snaps;
    if constexpr (SOURCE)
      velocity_source<DIM, false>(w, s, 0.0, x, u);
    else
      velocity_packed<DIM, false, TRY>(w.g, recs + s * rec_set, 0.0, x, u, last);
  } else {
    const int lane = k * times.kPoints + c;
    const int s = __shfl_sync(0xffffffffu, times.s, lane);
    const double alpha = __shfl_sync(0xffffffffu, times.alpha, lane);
    if constexpr (SOURCE)
      velocity_source<DIM, true>(w, s, alpha, x, u);
    else
      velocity_packed<DIM, true, TRY>(w.g, recs + s * rec_set, alpha, x, u, last);
  }
}

// One particle through the whole window (integrate.py restated step by step).  All lanes of
// a warp take part (the time lookups are shared).  SOURCE: w.snaps are the snapshots as the
// caller has them, not records.
template <int DIM, int MODE, int INTEG, bool SOURCE = false>
__device__ __forceinline__ void advect(const WinK &w, double *x) {
  const double h = w.h;
  double vprev[DIM];
  StepTimes<MODE, INTEG> times;
  Corners64<DIM> last;
  for (int first = 0; first < w.num_steps; first += times.kSteps) {
    times.load(w, first);
    const int run = min(times.kSteps, w.num_steps - first);
    for (int k = 0; k < run; ++k) {
      const int i = first + k;
      if constexpr (INTEG == FTLE_EULER) {
        double v[DIM];
        field<DIM, false, SOURCE>(w, times, k, i, 0, x, v, last);
#pragma unroll
        for (int a = 0; a < DIM; ++a) x[a] = x[a] + h * v[a];
      } else if constexpr (INTEG == FTLE_AB2) {
        double v[DIM];
        field<DIM, false, SOURCE>(w, times, k, i, 0, x, v, last);
        if (i == 0) {
#pragma unroll
          for (int a = 0; a < DIM; ++a) x[a] = x[a] + h * v[a];
        } else {
#pragma unroll
          for (int a = 0; a < DIM; ++a) x[a] = x[a] + h * (1.5 * v[a] - 0.5 * vprev[a]);
        }
#pragma unroll
        for (int a = 0; a < DIM; ++a) vprev[a] = v[a];
      } else {
        const double hh = 0.5 * h;
        // stages 1 and 3 try the previous stage's corners in BLEND; in HOLD, where only the
        // loads would be saved, the test cost more than they did (2D 4 %, 3D 5 % slower)
        constexpr bool kTry = MODE == FTLE_BLEND;
        double kv[DIM], acc[DIM], tmp[DIM];
        field<DIM, kTry, SOURCE>(w, times, k, i, 0, x, kv, last);
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
          acc[a] = kv[a];
          tmp[a] = x[a] + hh * kv[a];
        }
        field<DIM, false, SOURCE>(w, times, k, i, 1, tmp, kv, last);
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
          acc[a] = acc[a] + 2.0 * kv[a];
          tmp[a] = x[a] + hh * kv[a];
        }
        field<DIM, kTry, SOURCE>(w, times, k, i, 1, tmp, kv, last);
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
          acc[a] = acc[a] + 2.0 * kv[a];
          tmp[a] = x[a] + h * kv[a];
        }
        field<DIM, false, SOURCE>(w, times, k, i, 2, tmp, kv, last);
        const double h6 = h / 6.0;
#pragma unroll
        for (int a = 0; a < DIM; ++a) x[a] = x[a] + h6 * (acc[a] + kv[a]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// FTLE epilogue
// ---------------------------------------------------------------------------

// ftle.py:122-163 on C = F^T F (ftle.py:62-67).
__device__ __forceinline__ double lambda_max_2x2(double F00, double F01, double F10, double F11) {
  const double A = F00 * F00 + F10 * F10;
  const double B = F00 * F01 + F10 * F11;
  const double C = F01 * F00 + F11 * F10;
  const double D = F01 * F01 + F11 * F11;
  const double trace = A + D;
  const double det = A * D - B * C;
  const double l1 = 0.5 * (trace + sqrt(trace * trace - 4.0 * det));
  const double l2 = 0.5 * (trace - sqrt(trace * trace - 4.0 * det));
  return (l2 > l1) ? l2 : l1;
}

// C = F F^T (ftle.py:96) then lambda_max (the reference takes max(np.linalg.eigvals(C)),
// ftle.py:118-119).
__device__ __forceinline__ double lambda_max_3x3(const double J[3][3]) {
  double C[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int k = 0; k < 3; ++k)
      C[i][k] = J[i][0] * J[k][0] + J[i][1] * J[k][1] + J[i][2] * J[k][2];
  return lmax3_sym(C[0][0], C[0][1], C[0][2], C[1][1], C[1][2], C[2][2]);
}

__device__ __forceinline__ double ftle_value(double lambda, double map_period) {
  return (1.0 / map_period) * log(sqrt(lambda));
}

// Role pairs of the Jacobian columns: (right, left), (top, bottom), (front, back).
__device__ __forceinline__ int plus_role(int j) { return j == 0 ? 1 : 2 * j; }
__device__ __forceinline__ int minus_role(int j) { return j == 0 ? 0 : 2 * j + 1; }

// FTLE of one group from its K final positions P[role][a] and initial diagonal
// separations id[j] (right-left x, top-bottom y, front-back z).
template <int DIM>
__device__ __forceinline__ double group_ftle(const double (*P)[DIM], const double *id,
                                             double map_period) {
  double J[DIM][DIM];
#pragma unroll
  for (int i = 0; i < DIM; ++i)
#pragma unroll
    for (int j = 0; j < DIM; ++j) J[i][j] = (P[plus_role(j)][i] - P[minus_role(j)][i]) / id[j];
  if constexpr (DIM == 2)
    return ftle_value(lambda_max_2x2(J[0][0], J[0][1], J[1][0], J[1][1]), map_period);
  else
    return ftle_value(lambda_max_3x3(J), map_period);
}

// ---------------------------------------------------------------------------
// fused window kernel: one thread per particle, G groups per block
// ---------------------------------------------------------------------------
// Groups per block and blocks per SM (the register budget).  The kernel is bound by the
// latency of its FP64 chains and by L1 data wavefronts, so the budget is the largest that
// does not spill: 3D BLEND holds 24 blended corner values, 128 registers at 15 warps per SM
// (5 blocks of 96 threads; 6 blocks at 96 registers spill and run 1.15x slower), 2D BLEND
// 64 registers at 32 warps (72 at 28 1.06x, unbounded 1.22x slower), 3D HOLD 80 at 24 warps,
// 2D HOLD 48 at 40 warps (RK4; the one-stage integrators 64).  Blocks of 96 / 128 threads
// also spread small windows over more SMs.
// Measured against division by IEEE `/`, conversions for floor, `%` for every periodic wrap,
// a time lookup per thread and stage and no reuse of corners: ABC 128^3, 262,080 groups, 100
// RK4 steps BLEND 16.11 -> 9.44 ms; turbulence 512^2, 131,072 groups, 80 steps BLEND 1.63 ->
// 0.97 ms; gyre 512 x 256, 80,000 groups, 51 steps HOLD 0.423 -> 0.336 ms.
template <int DIM, int MODE>
constexpr int kGroups = DIM == 2 ? 32 : (MODE == FTLE_BLEND ? 16 : 32);
template <int DIM, int MODE, int INTEG>
constexpr int kBlocksPerSM = DIM == 2
                                 ? (MODE == FTLE_HOLD && INTEG == FTLE_RK4 ? 10 : 8)
                                 : (MODE == FTLE_BLEND ? 5 : 4);

template <int DIM, int MODE, int INTEG>
__global__ void __launch_bounds__(2 * DIM * kGroups<DIM, MODE>, kBlocksPerSM<DIM, MODE, INTEG>)
    window_f64_kernel(const WinK w) {
  constexpr int G = kGroups<DIM, MODE>;
  constexpr int K = 2 * DIM;
  const int tid = threadIdx.x;
  // role-minor: a warp holds every neighbour of a few groups, whose gathers mostly read
  // the same cell's records, so a load touches a few lines instead of 32 (a warp of one
  // role over 32 groups ran 1.36x slower in 3D BLEND, 1.24x in 2D HOLD); the
  // per-particle arithmetic is the same either way
  const int role = tid % K, gl = tid / K;
  const long long g = (long long)blockIdx.x * G + gl;
  // threads past the last group advect a point at 0: a warp's lanes share time lookups
  const bool active = g < w.N;
  const long long row = (long long)role * w.N + g;
  double x[DIM], x0[DIM];
#pragma unroll
  for (int a = 0; a < DIM; ++a) x[a] = x0[a] = active ? w.positions[row * DIM + a] : 0.0;
  advect<DIM, MODE, INTEG>(w, x);
  if (active && !w.keep_positions) {
#pragma unroll
    for (int a = 0; a < DIM; ++a) w.positions[row * DIM + a] = x[a];
  }
  if (w.ftle != nullptr) {  // uniform across the block
    __shared__ double sx[K][G][DIM];
    __shared__ double sx0[K][G][DIM];
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
      sx[role][gl][a] = x[a];
      sx0[role][gl][a] = x0[a];
    }
    __syncthreads();
    if (tid < G) {
      const long long gg = (long long)blockIdx.x * G + tid;
      if (gg < w.N) {
        double P[K][DIM];
        double id[DIM];
#pragma unroll
        for (int r = 0; r < K; ++r)
#pragma unroll
          for (int a = 0; a < DIM; ++a) P[r][a] = sx[r][tid][a];
#pragma unroll
        for (int j = 0; j < DIM; ++j) id[j] = sx0[plus_role(j)][tid][j] - sx0[minus_role(j)][tid][j];
        w.ftle[gg] = group_ftle<DIM>(P, id, w.map_period);
      }
    }
  }
}

// FTLE of every stride-th group of a window, straight from the snapshots as the caller has
// them: the sample that judges a 16-bit window.  One thread per particle, one warp (3D: three)
// per block, so that a sample spreads over the SMs.  While it fits them it is one FP64 chain long
// (1,311 groups of a 512^2 window, 80 steps: 0.17 ms on 164 of the chip's 592 schedulers), which
// is why the caller runs it beside the window itself.  Beyond that the planes' scattered 8-byte
// gathers cost more than records would, in 3D above all.  Alone, ms, against writing the records
// and a window over them (which take twice the series' memory):
//   2D, 80 steps: 1,311 groups 0.17, 0.24;   20,972 0.33, 0.33;   167,773 2.1, 1.3
//   3D, 200 steps: 1,250 groups 1.5, 1.6;   20,972 4.1, 2.7;   167,773 43.9, 14.1
template <int DIM>
constexpr int kSampleGroups = DIM == 2 ? 8 : 16;

template <int DIM, int MODE, int INTEG>
__global__ void __launch_bounds__(2 * DIM * kSampleGroups<DIM>)
    sample_f64_kernel(const WinK w, long long stride, long long samples) {
  constexpr int G = kSampleGroups<DIM>;
  constexpr int K = 2 * DIM;
  __shared__ double sx[K][G][DIM];
  __shared__ double sx0[K][G][DIM];
  const int role = threadIdx.x % K, gl = threadIdx.x / K;
  const long long i = (long long)blockIdx.x * G + gl;
  // threads past the last group repeat it: a warp's lanes share time lookups
  const long long row = (long long)role * w.N + min(i, samples - 1) * stride;
  double x[DIM];
#pragma unroll
  for (int a = 0; a < DIM; ++a) {
    x[a] = w.positions[row * DIM + a];
    sx0[role][gl][a] = x[a];
  }
  advect<DIM, MODE, INTEG, true>(w, x);
#pragma unroll
  for (int a = 0; a < DIM; ++a) sx[role][gl][a] = x[a];
  __syncthreads();
  const long long out = (long long)blockIdx.x * G + threadIdx.x;
  if (threadIdx.x < G && out < samples) {
    double P[K][DIM], id[DIM];
#pragma unroll
    for (int r = 0; r < K; ++r)
#pragma unroll
      for (int a = 0; a < DIM; ++a) P[r][a] = sx[r][threadIdx.x][a];
#pragma unroll
    for (int j = 0; j < DIM; ++j)
      id[j] = sx0[plus_role(j)][threadIdx.x][j] - sx0[minus_role(j)][threadIdx.x][j];
    w.ftle[out] = group_ftle<DIM>(P, id, w.map_period);
  }
}

// Sums of squares of (field[i * stride] - sample[i]) and sample[i], one pair per block.
constexpr int kNormThreads = 256;

__global__ void __launch_bounds__(kNormThreads)
    sample_norms_kernel(const double *__restrict__ field, const double *__restrict__ sample,
                        long long stride, long long samples, double2 *sums) {
  double2 s = make_double2(0.0, 0.0);
  for (long long i = blockIdx.x * (long long)kNormThreads + threadIdx.x; i < samples;
       i += (long long)gridDim.x * kNormThreads) {
    const double r = sample[i], d = field[i * stride] - r;
    s.x += d * d;
    s.y += r * r;
  }
  __shared__ double2 part[kNormThreads];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int half = kNormThreads / 2; half > 0; half >>= 1) {
    if (threadIdx.x < half) {
      part[threadIdx.x].x += part[threadIdx.x + half].x;
      part[threadIdx.x].y += part[threadIdx.x + half].y;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = part[0];
}

// ---------------------------------------------------------------------------
// closed-form velocity fields (the "analytical" interpolator on the device)
// ---------------------------------------------------------------------------

struct FlowK {
  int kind;
  double p[8];
};

// Double gyre, in the operand order of pyFTLE's example velocity_fn:
//   f = eps sin(wt) x^2 + (1 - 2 eps sin(wt)) x,  u = -pi A sin(pi f) cos(pi y),
//   v = pi A cos(pi f) sin(pi y) df/dx.
// Time-periodic ABC: A(t) = A + a sin(w t), u = A(t) sin z + C cos y,
//   v = B sin x + A(t) cos z, w = C sin y + B cos x.
// `s` is sin(w t) of the evaluation's time.  Each angle's sine and cosine share one range
// reduction (sincos).  (Against separate calls and a sine of time per thread: double gyre,
// 45,150 groups, 4 fields of 51 RK4 steps 2.05 -> 1.35 ms a pass; ABC, 125,000 groups, 2 fields
// 4.69 -> 2.90 ms.  sincospi(f) is 10 % faster in 2D, but not the reference's sin(pi * f): its
// FTLE differs by 1.4e-13.)
template <int DIM>
__device__ __forceinline__ void flow_velocity(const FlowK &f, double s, const double *x,
                                              double *u) {
  if constexpr (DIM == 2) {
    const double A = f.p[0], eps = f.p[1];
    const double xx = x[0], yy = x[1];
    const double ff = eps * s * (xx * xx) + (1.0 - 2.0 * eps * s) * xx;
    const double dfdx = 2.0 * eps * s * xx + (1.0 - 2.0 * eps * s);
    const double pi = 3.141592653589793;
    double sf, cf, sy, cy;
    sincos(pi * ff, &sf, &cf);
    sincos(pi * yy, &sy, &cy);
    u[0] = -pi * A * sf * cy;
    u[1] = pi * A * cf * sy * dfdx;
  } else {
    const double At = f.p[0] + f.p[3] * s;
    const double B = f.p[1], C = f.p[2];
    double sn[3], cs[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) sincos(x[a], &sn[a], &cs[a]);
    u[0] = At * sn[2] + C * cs[1];
    u[1] = B * sn[0] + At * cs[2];
    u[2] = C * sn[1] + B * cs[0];
  }
}

// sin(w t) at the points of a run of steps, shared by the lanes of a warp as StepTimes.
template <int INTEG>
struct StepSines {
  static constexpr int kPoints = INTEG == FTLE_RK4 ? 3 : 1;
  static constexpr int kSteps = 32 / kPoints;
  double value;
  __device__ __forceinline__ void load(double omega, double t0, double h, int freeze, int first) {
    const int lane = threadIdx.x & 31, c = lane % kPoints;
    const double t = t0 + (double)(first + lane / kPoints) * h;
    value = sin(omega * (freeze ? 0.0 : (c == 0 ? t : (c == 1 ? t + 0.5 * h : t + h))));
  }
  __device__ __forceinline__ double at(int k, int c) const {
    return __shfl_sync(0xffffffffu, value, k * kPoints + c);
  }
};

// All lanes of a warp take part (the sines of time are shared).
template <int DIM, int INTEG>
__device__ __forceinline__ void advect_analytic(const FlowK &f, double t0, double h, int steps,
                                                int freeze, double *x) {
  double vprev[DIM];
  StepSines<INTEG> sines;
  for (int first = 0; first < steps; first += sines.kSteps) {
    sines.load(f.p[DIM == 2 ? 2 : 4], t0, h, freeze, first);
    const int run = min(sines.kSteps, steps - first);
    for (int i = 0; i < run; ++i) {
      if constexpr (INTEG == FTLE_EULER || INTEG == FTLE_AB2) {
        double v[DIM];
        flow_velocity<DIM>(f, sines.at(i, 0), x, v);
        if (INTEG == FTLE_EULER || first + i == 0) {
#pragma unroll
          for (int a = 0; a < DIM; ++a) x[a] = x[a] + h * v[a];
        } else {
#pragma unroll
          for (int a = 0; a < DIM; ++a) x[a] = x[a] + h * (1.5 * v[a] - 0.5 * vprev[a]);
        }
#pragma unroll
        for (int a = 0; a < DIM; ++a) vprev[a] = v[a];
      } else {
        const double hh = 0.5 * h;
        const double sh = sines.at(i, 1);
        double k[DIM], acc[DIM], tmp[DIM];
        flow_velocity<DIM>(f, sines.at(i, 0), x, k);
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
          acc[a] = k[a];
          tmp[a] = x[a] + hh * k[a];
        }
        flow_velocity<DIM>(f, sh, tmp, k);
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
          acc[a] = acc[a] + 2.0 * k[a];
          tmp[a] = x[a] + hh * k[a];
        }
        flow_velocity<DIM>(f, sh, tmp, k);
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
          acc[a] = acc[a] + 2.0 * k[a];
          tmp[a] = x[a] + h * k[a];
        }
        flow_velocity<DIM>(f, sines.at(i, 2), tmp, k);
        const double h6 = h / 6.0;
#pragma unroll
        for (int a = 0; a < DIM; ++a) x[a] = x[a] + h6 * (acc[a] + k[a]);
      }
    }
  }
}

// Bound by the FP64 work of the trigonometry.
template <int DIM, int INTEG, int G>
__global__ void __launch_bounds__(2 * DIM * G)
    analytic_window_kernel(const FlowK f, double t0, double h, int steps, int freeze,
                           double *positions, long long N, double map_period, double *ftle) {
  constexpr int K = 2 * DIM;
  const int tid = threadIdx.x;
  const int role = tid / G, gl = tid % G;
  const long long g = (long long)blockIdx.x * G + gl;
  // threads past the last group advect a point at 0: a warp's lanes share the sines of time
  const bool active = g < N;
  const long long row = (long long)role * N + g;
  double x[DIM], x0[DIM];
#pragma unroll
  for (int a = 0; a < DIM; ++a) x[a] = x0[a] = active ? positions[row * DIM + a] : 0.0;
  advect_analytic<DIM, INTEG>(f, t0, h, steps, freeze, x);
  if (active) {
#pragma unroll
    for (int a = 0; a < DIM; ++a) positions[row * DIM + a] = x[a];
  }
  if (ftle != nullptr) {
    __shared__ double sx[K][G][DIM];
    __shared__ double sx0[K][G][DIM];
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
      sx[role][gl][a] = x[a];
      sx0[role][gl][a] = x0[a];
    }
    __syncthreads();
    if (tid < G) {
      const long long gg = (long long)blockIdx.x * G + tid;
      if (gg < N) {
        double P[K][DIM];
        double id[DIM];
#pragma unroll
        for (int r = 0; r < K; ++r)
#pragma unroll
          for (int a = 0; a < DIM; ++a) P[r][a] = sx[r][tid][a];
#pragma unroll
        for (int j = 0; j < DIM; ++j)
          id[j] = sx0[plus_role(j)][tid][j] - sx0[minus_role(j)][tid][j];
        ftle[gg] = group_ftle<DIM>(P, id, map_period);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// per-step kernels (compatibility path of the Integrator / Interpolator API)
// ---------------------------------------------------------------------------

__global__ void interp2d_kernel(const double *__restrict__ v, int nx, int ny,
                                const double *__restrict__ pts, long long n, double *out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double px = pts[i * 2 + 0], py = pts[i * 2 + 1];
    double c = 0.0;
    if (px >= 0.0 && px < (double)(nx - 1) && py >= 0.0 && py < (double)(ny - 1)) {
      const int x0 = (int)floor(px), y0 = (int)floor(py);
      const double xd = px - (double)x0, yd = py - (double)y0;
      const long long b = (long long)x0 * ny + y0;
      c = bilinear(__ldg(v + b), __ldg(v + b + ny), __ldg(v + b + 1), __ldg(v + b + ny + 1), xd,
                   yd);
    }
    out[i] = c;
  }
}

__global__ void interp3d_kernel(const double *__restrict__ v, int X, int Y, int Z,
                                const double *__restrict__ pts, long long n, double *out) {
  const long long YZ = (long long)Y * Z;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double px = pts[i * 3 + 0], py = pts[i * 3 + 1], pz = pts[i * 3 + 2];
    double c = 0.0;
    if (px >= 0.0 && px < (double)(X - 1) && py >= 0.0 && py < (double)(Y - 1) && pz >= 0.0 &&
        pz < (double)(Z - 1)) {
      const int x0 = (int)floor(px), y0 = (int)floor(py), z0 = (int)floor(pz);
      const double xd = px - (double)x0, yd = py - (double)y0, zd = pz - (double)z0;
      const long long b = (long long)x0 * YZ + (long long)y0 * Z + z0;
      double vv[8];
      vv[0] = __ldg(v + b);                // x0y0z0
      vv[1] = __ldg(v + b + YZ);           // x1y0z0
      vv[2] = __ldg(v + b + 1);            // x0y0z1
      vv[3] = __ldg(v + b + YZ + 1);       // x1y0z1
      vv[4] = __ldg(v + b + Z);            // x0y1z0
      vv[5] = __ldg(v + b + YZ + Z);       // x1y1z0
      vv[6] = __ldg(v + b + Z + 1);        // x0y1z1
      vv[7] = __ldg(v + b + YZ + Z + 1);   // x1y1z1
      c = trilinear(vv, xd, yd, zd);
    }
    out[i] = c;
  }
}

template <int DIM>
__global__ void grid_interpolate_kernel(const GridK g, const double *__restrict__ snap,
                                        const double *__restrict__ pts, long long m,
                                        double *out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < m;
       i += (long long)gridDim.x * blockDim.x) {
    double x[DIM], u[DIM];
#pragma unroll
    for (int a = 0; a < DIM; ++a) x[a] = pts[i * DIM + a];
    velocity_planar<DIM>(g, snap, x, u);
#pragma unroll
    for (int a = 0; a < DIM; ++a) out[i * DIM + a] = u[a];
  }
}

template <int DIM, int INTEG>
__global__ void grid_step_kernel(const GridK g, const double *__restrict__ snap, double h,
                                 double *pos, long long m, double *hist, int hist_valid) {
  // RK4 with m = K*N (role-blocked neighbour groups): work item j takes role j mod K of
  // group j / K, so a warp holds every neighbour of a few groups and their four stages'
  // gathers share cells (3D 2.95x, 2D 1.31x faster); each particle is still advected
  // once, by the same arithmetic.  Euler / AB2 evaluate once per step and are bound by
  // streaming positions (and history), which that order makes strided (3D 1.5x slower),
  // so they keep the particle order.
  constexpr int K = 2 * DIM;
  const long long ng = (INTEG == FTLE_RK4 && m % K == 0) ? m / K : 0;
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < m;
       j += (long long)gridDim.x * blockDim.x) {
    const long long i = ng ? (j % K) * ng + j / K : j;
    double x[DIM];
#pragma unroll
    for (int a = 0; a < DIM; ++a) x[a] = pos[i * DIM + a];
    if constexpr (INTEG == FTLE_EULER) {
      double v[DIM];
      velocity_planar<DIM>(g, snap, x, v);
#pragma unroll
      for (int a = 0; a < DIM; ++a) x[a] = x[a] + h * v[a];
    } else if constexpr (INTEG == FTLE_AB2) {
      double v[DIM];
      velocity_planar<DIM>(g, snap, x, v);
#pragma unroll
      for (int a = 0; a < DIM; ++a) {
        if (hist_valid)
          x[a] = x[a] + h * (1.5 * v[a] - 0.5 * hist[i * DIM + a]);
        else
          x[a] = x[a] + h * v[a];
        hist[i * DIM + a] = v[a];
      }
    } else {
      const double hh = 0.5 * h;
      double k[DIM], acc[DIM], tmp[DIM];
      velocity_planar<DIM>(g, snap, x, k);
#pragma unroll
      for (int a = 0; a < DIM; ++a) {
        acc[a] = k[a];
        tmp[a] = x[a] + hh * k[a];
      }
      velocity_planar<DIM>(g, snap, tmp, k);
#pragma unroll
      for (int a = 0; a < DIM; ++a) {
        acc[a] = acc[a] + 2.0 * k[a];
        tmp[a] = x[a] + hh * k[a];
      }
      velocity_planar<DIM>(g, snap, tmp, k);
#pragma unroll
      for (int a = 0; a < DIM; ++a) {
        acc[a] = acc[a] + 2.0 * k[a];
        tmp[a] = x[a] + h * k[a];
      }
      velocity_planar<DIM>(g, snap, tmp, k);
      const double h6 = h / 6.0;
#pragma unroll
      for (int a = 0; a < DIM; ++a) x[a] = x[a] + h6 * (acc[a] + k[a]);
    }
#pragma unroll
    for (int a = 0; a < DIM; ++a) pos[i * DIM + a] = x[a];
  }
}

__global__ void axpy_kernel(double *out, const double *x, double a, const double *k, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    out[i] = x[i] + a * k[i];
}

__global__ void ab2_kernel(double *x, double h, const double *v, const double *vp, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    x[i] = x[i] + h * (1.5 * v[i] - 0.5 * vp[i]);
}

__global__ void rk4_kernel(double *x, double h6, const double *k1, const double *k2,
                           const double *k3, const double *k4, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    x[i] = x[i] + h6 * (((k1[i] + 2.0 * k2[i]) + 2.0 * k3[i]) + k4[i]);
}

// ---------------------------------------------------------------------------
// FTLE building blocks
// ---------------------------------------------------------------------------

// A warp's 32 consecutive items of W doubles, moved through shared memory: a thread's own W
// doubles lie W*8 bytes from its neighbour's, so reading or writing them directly touches
// every sector W times.  (3D, 600,001 groups: Jacobian, whose inputs move the same way, 40.6 ->
// 27.9 us, 6.2 TB/s; C 29.6 -> 11.7 us; lambda_max 38.3 -> 11.8 us and FTLE 41.7 -> 15.4 us,
// both also by lmax3_sym's closed form in place of rotations.)
constexpr int kTileWarps = 4;
template <int W>
struct WarpTile {
  static constexpr int kPitch = W | 1;  // odd: no bank conflicts
  double v[32 * kPitch];
  static __device__ __forceinline__ int slot(int e) { return e / W * kPitch + e % W; }
  // all lanes: items [first, first + count) of `src` -> the lanes' own W values
  __device__ __forceinline__ void load(const double *__restrict__ src, long long first, int count,
                                       int lane, double *own) {
    __syncwarp();
#pragma unroll
    for (int j = 0; j < W; ++j) {
      const int e = 32 * j + lane;
      if (e < count * W) v[slot(e)] = __ldg(src + first * W + e);
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < W; ++j) own[j] = v[lane * kPitch + j];
  }
  __device__ __forceinline__ void store(double *dst, long long first, int count, int lane,
                                        const double *own) {
    __syncwarp();
#pragma unroll
    for (int j = 0; j < W; ++j) v[lane * kPitch + j] = own[j];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < W; ++j) {
      const int e = 32 * j + lane;
      if (e < count * W) dst[first * W + e] = v[slot(e)];
    }
  }
};

// Runs body(first item, items, lane, tile) for every 32 items of n.
template <int W, typename Body>
__device__ __forceinline__ void for_warp_tiles(long long n, const Body &body) {
  __shared__ WarpTile<W> tiles[kTileWarps];
  const int lane = threadIdx.x & 31;
  WarpTile<W> &tile = tiles[threadIdx.x >> 5];
  const long long step = (long long)gridDim.x * kTileWarps * 32;
  for (long long first = ((long long)blockIdx.x * kTileWarps + (threadIdx.x >> 5)) * 32; first < n;
       first += step)
    body(first, (int)min(32ll, n - first), lane, tile);
}

template <int DIM>
__global__ void __launch_bounds__(32 * kTileWarps)
    jacobian_kernel(const double *__restrict__ pos, const double *__restrict__ idl, long long N,
                    double *J) {
  constexpr int K = 2 * DIM;
  __shared__ double tiles[kTileWarps][K][32 * DIM];  // a warp's rows of every role
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto &tile = tiles[warp];
  WarpTile<DIM * DIM> &out = *reinterpret_cast<WarpTile<DIM * DIM> *>(&tile[0][0]);
  static_assert(sizeof(out) <= sizeof(tile), "the output tile takes the input tiles' place");
  const long long step = (long long)gridDim.x * kTileWarps * 32;
  for (long long first = ((long long)blockIdx.x * kTileWarps + warp) * 32; first < N;
       first += step) {
    const int count = (int)min(32ll, N - first);
    double v[K][DIM], id[DIM], own[DIM * DIM];
#pragma unroll
    for (int r = 0; r < K; ++r)
#pragma unroll
      for (int j = 0; j < DIM; ++j)
        v[r][j] = __ldg(pos + ((long long)r * N + first) * DIM + min(32 * j + lane, count * DIM - 1));
    const long long g = first + min(lane, count - 1);
#pragma unroll
    for (int j = 0; j < DIM; ++j) id[j] = __ldg(idl + ((long long)j * N + g) * DIM + j);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < K; ++r)
#pragma unroll
      for (int j = 0; j < DIM; ++j) tile[r][32 * j + lane] = v[r][j];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < DIM; ++i)
#pragma unroll
      for (int j = 0; j < DIM; ++j)
        own[i * DIM + j] =
            (tile[plus_role(j)][lane * DIM + i] - tile[minus_role(j)][lane * DIM + i]) / id[j];
    out.store(J, first, count, lane, own);
  }
}

template <int DIM>
__global__ void cauchy_green_kernel(const double *__restrict__ J, long long n, double *C) {
  for_warp_tiles<DIM * DIM>(n, [&](long long first, int count, int lane, auto &tile) {
    double F[DIM * DIM], c[DIM * DIM];
    tile.load(J, first, count, lane, F);
    if constexpr (DIM == 2) {  // C = F^T F, ftle.py:62-67
      c[0] = F[0] * F[0] + F[2] * F[2];
      c[1] = F[0] * F[1] + F[2] * F[3];
      c[2] = F[1] * F[0] + F[3] * F[2];
      c[3] = F[1] * F[1] + F[3] * F[3];
    } else {  // C = F F^T, ftle.py:96
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k)
          c[i * 3 + k] = F[i * 3 + 0] * F[k * 3 + 0] + F[i * 3 + 1] * F[k * 3 + 1] +
                         F[i * 3 + 2] * F[k * 3 + 2];
    }
    tile.store(C, first, count, lane, c);
  });
}

template <int DIM>
__global__ void max_eigenvalue_kernel(const double *__restrict__ C, long long n, double *out) {
  for_warp_tiles<DIM * DIM>(n, [&](long long first, int count, int lane, auto &tile) {
    double c[DIM * DIM];
    tile.load(C, first, count, lane, c);
    if (lane >= count) return;
    if constexpr (DIM == 2) {  // ftle.py:146-161 on (A, B, C, D)
      const double trace = c[0] + c[3];
      const double det = c[0] * c[3] - c[1] * c[2];
      const double l1 = 0.5 * (trace + sqrt(trace * trace - 4.0 * det));
      const double l2 = 0.5 * (trace - sqrt(trace * trace - 4.0 * det));
      out[first + lane] = (l2 > l1) ? l2 : l1;
    } else {  // symmetric part (exact for a symmetric C)
      out[first + lane] = lmax3_sym(c[0], 0.5 * (c[1] + c[3]), 0.5 * (c[2] + c[6]), c[4],
                                    0.5 * (c[5] + c[7]), c[8]);
    }
  });
}

template <int DIM>
__global__ void ftle_from_jacobian_kernel(const double *__restrict__ J, long long n,
                                          double map_period, double *out) {
  for_warp_tiles<DIM * DIM>(n, [&](long long first, int count, int lane, auto &tile) {
    double F[DIM * DIM];
    tile.load(J, first, count, lane, F);
    if (lane >= count) return;
    if constexpr (DIM == 2) {
      out[first + lane] = ftle_value(lambda_max_2x2(F[0], F[1], F[2], F[3]), map_period);
    } else {
      double M[3][3];
#pragma unroll
      for (int i = 0; i < 9; ++i) M[i / 3][i % 3] = F[i];
      out[first + lane] = ftle_value(lambda_max_3x3(M), map_period);
    }
  });
}

// Initial separations (DIM planes of N x DIM, right-left, top-bottom (, front-back)) and the
// centroid, summed in role order, of every group: every role's rows are one contiguous block,
// so thread e takes element e of each.
template <int DIM>
__global__ void group_init_kernel(const double *__restrict__ pos, long long N, double *deltas,
                                  double *centroid) {
  const long long n = N * DIM;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    double x[2 * DIM];
#pragma unroll
    for (int r = 0; r < 2 * DIM; ++r) x[r] = __ldg(pos + r * n + e);
#pragma unroll
    for (int j = 0; j < DIM; ++j) deltas[j * n + e] = x[plus_role(j)] - x[minus_role(j)];
    double s = x[0];
#pragma unroll
    for (int r = 1; r < 2 * DIM; ++r) s = s + x[r];
    centroid[e] = s / (double)(2 * DIM);
  }
}

template <int DIM>
__global__ void ftle_from_positions_kernel(const double *__restrict__ pos,
                                           const double *__restrict__ idl, long long N,
                                           double map_period, double *out) {
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < N;
       g += (long long)gridDim.x * blockDim.x) {
    double P[2 * DIM][DIM];
    double id[DIM];
#pragma unroll
    for (int r = 0; r < 2 * DIM; ++r)
#pragma unroll
      for (int a = 0; a < DIM; ++a) P[r][a] = pos[((long long)r * N + g) * DIM + a];
#pragma unroll
    for (int j = 0; j < DIM; ++j) id[j] = idl[((long long)j * N + g) * DIM + j];
    out[g] = group_ftle<DIM>(P, id, map_period);
  }
}

// ---------------------------------------------------------------------------
// FP64 snapshot packing: (S, dim, nodes) -> records (S, nodes, 2*dim)
// ---------------------------------------------------------------------------
// One thread per node and run of R snapshots, as pack16_kernel.  A warp's 32 records of a
// snapshot are one contiguous piece of the destination: they go through the warp's shared
// memory so that every store covers whole sectors (8-byte stores at the record stride kept
// the load-store unit busy: gyre 512 x 256 x 101, 202 us; now 96 us, 6.6 TB/s).
template <int DIM, int R>
__global__ void __launch_bounds__(256)
    pack_f64_kernel(const double *__restrict__ src, long long nodes, int S, int periodic_time,
                    double *dst) {
  __shared__ double2 stage[8][32 * DIM];
  const int lane = threadIdx.x & 31;
  const long long p0 = blockIdx.x * 256ll + (threadIdx.x & ~31);  // the warp's first node
  if (p0 >= nodes) return;
  const long long p = min(p0 + lane, nodes - 1);
  const int count = (int)min(32ll, nodes - p0) * DIM;  // 16-byte pieces of the warp's records
  double2 *buf = stage[threadIdx.x >> 5];
  for (int run = blockIdx.y; run * R < S; run += gridDim.y) {
    const int s0 = run * R;
    double v[R + 1][DIM];
#pragma unroll
    for (int r = 0; r <= R; ++r) {
      const int s = s0 + r < S ? s0 + r : (periodic_time ? 0 : S - 1);
#pragma unroll
      for (int c = 0; c < DIM; ++c) v[r][c] = __ldg(src + ((long long)s * DIM + c) * nodes + p);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (s0 + r >= S) break;
      double rec[2 * DIM];
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        rec[c] = v[r][c];
        rec[DIM + c] = v[r + 1][c];
      }
#pragma unroll
      for (int j = 0; j < DIM; ++j) buf[lane * DIM + j] = make_double2(rec[2 * j], rec[2 * j + 1]);
      __syncwarp();
      double2 *out = reinterpret_cast<double2 *>(dst) + ((long long)(s0 + r) * nodes + p0) * DIM;
#pragma unroll
      for (int j = 0; j < DIM; ++j)
        if (lane + 32 * j < count) out[lane + 32 * j] = buf[lane + 32 * j];
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------------------
// host entry points
// ---------------------------------------------------------------------------

template <int DIM, int MODE, int INTEG>
static void launch_window(const WinK &w, cudaStream_t st) {
  constexpr int G = kGroups<DIM, MODE>;
  const long long blocks = (w.N + G - 1) / G;
  window_f64_kernel<DIM, MODE, INTEG><<<(unsigned)blocks, 2 * DIM * G, 0, st>>>(w);
}

template <int DIM, int MODE, int INTEG>
static void launch_sample(const WinK &w, long long stride, long long samples, cudaStream_t st) {
  constexpr int G = kSampleGroups<DIM>;
  sample_f64_kernel<DIM, MODE, INTEG>
      <<<(unsigned)((samples + G - 1) / G), 2 * DIM * G, 0, st>>>(w, stride, samples);
}

template <int DIM, int MODE>
static void launch_sample_i(const WinK &w, int integ, long long stride, long long samples,
                            cudaStream_t st) {
  if (integ == FTLE_EULER)
    launch_sample<DIM, MODE, FTLE_EULER>(w, stride, samples, st);
  else if (integ == FTLE_AB2)
    launch_sample<DIM, MODE, FTLE_AB2>(w, stride, samples, st);
  else
    launch_sample<DIM, MODE, FTLE_RK4>(w, stride, samples, st);
}

template <int DIM, int MODE>
static void launch_window_i(const WinK &w, int integ, cudaStream_t st) {
  if (integ == FTLE_EULER)
    launch_window<DIM, MODE, FTLE_EULER>(w, st);
  else if (integ == FTLE_AB2)
    launch_window<DIM, MODE, FTLE_AB2>(w, st);
  else
    launch_window<DIM, MODE, FTLE_RK4>(w, st);
}

}  // namespace ftle

using namespace ftle;

extern "C" {

int ftle_window_run_f64(const ftle_window *w, void *stream) {
  WinK k;
  int rc = window_to_kernel(w, &k);
  if (rc) return rc;
  if (w->storage != FTLE_F64) return fail_invalid("ftle_window_run_f64 needs FTLE_F64 storage");
  if (k.N == 0) return FTLE_OK;
  cudaStream_t st = as_stream(stream);
  const int dim = w->grid.dim;
  if (dim == 2) {
    if (w->time_mode == FTLE_HOLD)
      launch_window_i<2, FTLE_HOLD>(k, w->integrator, st);
    else
      launch_window_i<2, FTLE_BLEND>(k, w->integrator, st);
  } else {
    if (w->time_mode == FTLE_HOLD)
      launch_window_i<3, FTLE_HOLD>(k, w->integrator, st);
    else
      launch_window_i<3, FTLE_BLEND>(k, w->integrator, st);
  }
  return check_launch("window_f64_kernel");
}

int ftle_window_sample_f64(const ftle_window *w, const double *source, const double *seeds,
                           int64_t stride, double *sample, void *stream) {
  WinK k;
  int rc = window_to_kernel(w, &k);
  if (rc) return rc;
  if (stride < 1) return fail_invalid("stride must be >= 1");
  const int64_t samples = (k.N + stride - 1) / stride;
  if (samples == 0) return FTLE_OK;
  if (!source || !seeds || !sample) return fail_invalid("null pointer");
  if (!(k.map_period > 0.0) && !(k.map_period < 0.0))
    return fail_invalid("map_period must be non-zero");
  k.snaps = source;
  k.positions = const_cast<double *>(seeds);
  k.ftle = sample;
  cudaStream_t st = as_stream(stream);
  if (w->grid.dim == 2) {
    if (w->time_mode == FTLE_HOLD)
      launch_sample_i<2, FTLE_HOLD>(k, w->integrator, stride, samples, st);
    else
      launch_sample_i<2, FTLE_BLEND>(k, w->integrator, stride, samples, st);
  } else {
    if (w->time_mode == FTLE_HOLD)
      launch_sample_i<3, FTLE_HOLD>(k, w->integrator, stride, samples, st);
    else
      launch_sample_i<3, FTLE_BLEND>(k, w->integrator, stride, samples, st);
  }
  return check_launch("sample_f64_kernel");
}

int ftle_sample_norms(const double *field, const double *sample, int64_t num_groups,
                      int64_t stride, double *sums, int32_t blocks, void *stream) {
  if (stride < 1) return fail_invalid("stride must be >= 1");
  if (blocks < 1 || num_groups < 0) return fail_invalid("sizes must be positive");
  if (!sums || (num_groups > 0 && (!field || !sample))) return fail_invalid("null pointer");
  if (reinterpret_cast<uintptr_t>(sums) % 16 != 0)
    return fail_invalid("sums must be 16-byte aligned");
  sample_norms_kernel<<<(unsigned)blocks, kNormThreads, 0, as_stream(stream)>>>(
      field, sample, stride, (num_groups + stride - 1) / stride,
      reinterpret_cast<double2 *>(sums));
  return check_launch("sample_norms_kernel");
}

int ftle_interp2d_vec_inplace(const double *v, int32_t nx, int32_t ny, const double *points,
                              int64_t n, double *out, void *stream) {
  if (n < 0) return fail_invalid("n must be >= 0");
  if (n == 0) return FTLE_OK;
  if (!v || !points || !out) return fail_invalid("null pointer");
  if (nx < 1 || ny < 1) return fail_invalid("v must be 2D with positive extents");
  interp2d_kernel<<<grid_blocks(n, 256), 256, 0, as_stream(stream)>>>(v, nx, ny, points, n, out);
  return check_launch("interp2d_kernel");
}

int ftle_interp3d_vec_inplace(const double *v, int32_t X, int32_t Y, int32_t Z,
                              const double *points, int64_t n, double *out, void *stream) {
  if (n < 0) return fail_invalid("n must be >= 0");
  if (n == 0) return FTLE_OK;
  if (!v || !points || !out) return fail_invalid("null pointer");
  if (X < 1 || Y < 1 || Z < 1) return fail_invalid("v must be 3D with positive extents");
  interp3d_kernel<<<grid_blocks(n, 256), 256, 0, as_stream(stream)>>>(v, X, Y, Z, points, n,
                                                                       out);
  return check_launch("interp3d_kernel");
}

int ftle_grid_interpolate(const ftle_grid *grid, const double *snapshot, const double *points,
                          int64_t m, double *out, void *stream) {
  GridK g;
  int rc = grid_from_abi(grid, &g);
  if (rc) return rc;
  if (m < 0) return fail_invalid("m must be >= 0");
  if (m == 0) return FTLE_OK;
  if (!snapshot || !points || !out) return fail_invalid("null pointer");
  cudaStream_t st = as_stream(stream);
  if (grid->dim == 2)
    grid_interpolate_kernel<2><<<grid_blocks(m, 256), 256, 0, st>>>(g, snapshot, points, m, out);
  else
    grid_interpolate_kernel<3><<<grid_blocks(m, 256), 256, 0, st>>>(g, snapshot, points, m, out);
  return check_launch("grid_interpolate_kernel");
}

int ftle_grid_step(const ftle_grid *grid, const double *snapshot, int32_t integrator, double h,
                   double *positions, int64_t m, double *history, int32_t history_valid,
                   void *stream) {
  GridK g;
  int rc = grid_from_abi(grid, &g);
  if (rc) return rc;
  if (m < 0) return fail_invalid("m must be >= 0");
  if (integrator < FTLE_EULER || integrator > FTLE_RK4)
    return fail_invalid("unknown integrator %d", integrator);
  if (integrator == FTLE_AB2 && !history && m > 0) return fail_invalid("AB2 needs a history buffer");
  if (m == 0) return FTLE_OK;
  if (!snapshot || !positions) return fail_invalid("null pointer");
  cudaStream_t st = as_stream(stream);
  const unsigned b = grid_blocks(m, 128);
#define STEP(D, I) grid_step_kernel<D, I><<<b, 128, 0, st>>>(g, snapshot, h, positions, m, history, history_valid)
  if (grid->dim == 2) {
    if (integrator == FTLE_EULER) STEP(2, FTLE_EULER);
    else if (integrator == FTLE_AB2) STEP(2, FTLE_AB2);
    else STEP(2, FTLE_RK4);
  } else {
    if (integrator == FTLE_EULER) STEP(3, FTLE_EULER);
    else if (integrator == FTLE_AB2) STEP(3, FTLE_AB2);
    else STEP(3, FTLE_RK4);
  }
#undef STEP
  return check_launch("grid_step_kernel");
}

int ftle_axpy(double *out, const double *x, double a, const double *k, int64_t n, void *stream) {
  if (n < 0) return fail_invalid("n must be >= 0");
  if (n == 0) return FTLE_OK;
  if (!out || !x || !k) return fail_invalid("null pointer");
  axpy_kernel<<<grid_blocks(n, 256), 256, 0, as_stream(stream)>>>(out, x, a, k, n);
  return check_launch("axpy_kernel");
}

int ftle_ab2_update(double *x, double h, const double *v, const double *v_prev, int64_t n,
                    void *stream) {
  if (n < 0) return fail_invalid("n must be >= 0");
  if (n == 0) return FTLE_OK;
  if (!x || !v || !v_prev) return fail_invalid("null pointer");
  ab2_kernel<<<grid_blocks(n, 256), 256, 0, as_stream(stream)>>>(x, h, v, v_prev, n);
  return check_launch("ab2_kernel");
}

int ftle_rk4_update(double *x, double h, const double *k1, const double *k2, const double *k3,
                    const double *k4, int64_t n, void *stream) {
  if (n < 0) return fail_invalid("n must be >= 0");
  if (n == 0) return FTLE_OK;
  if (!x || !k1 || !k2 || !k3 || !k4) return fail_invalid("null pointer");
  rk4_kernel<<<grid_blocks(n, 256), 256, 0, as_stream(stream)>>>(x, h / 6.0, k1, k2, k3, k4, n);
  return check_launch("rk4_kernel");
}

#define DIM_DISPATCH(dim, KERNEL, THREADS, ...)                    \
  do {                                                             \
    if ((dim) == 2)                                                \
      KERNEL<2><<<b, THREADS, 0, as_stream(stream)>>>(__VA_ARGS__); \
    else                                                           \
      KERNEL<3><<<b, THREADS, 0, as_stream(stream)>>>(__VA_ARGS__); \
  } while (0)
constexpr int kTileThreads = 32 * kTileWarps;

int ftle_group_init(int32_t dim, const double *positions, int64_t num_groups, double *deltas,
                    double *centroid, void *stream) {
  if (dim != 2 && dim != 3) return fail_invalid("dim must be 2 or 3");
  if (num_groups < 0) return fail_invalid("num_groups must be >= 0");
  if (num_groups == 0) return FTLE_OK;
  if (!positions || !deltas || !centroid) return fail_invalid("null pointer");
  const unsigned b = grid_blocks(num_groups * dim, 256);
  DIM_DISPATCH(dim, group_init_kernel, 256, positions, num_groups, deltas, centroid);
  return check_launch("group_init_kernel");
}

int ftle_flow_map_jacobian(int32_t dim, const double *positions, const double *initial_deltas,
                           int64_t num_groups, double *jacobian, void *stream) {
  if (dim != 2 && dim != 3) return fail_invalid("dim must be 2 or 3");
  if (num_groups < 0) return fail_invalid("num_groups must be >= 0");
  if (num_groups == 0) return FTLE_OK;
  if (!positions || !initial_deltas || !jacobian) return fail_invalid("null pointer");
  const unsigned b = grid_blocks(num_groups, kTileThreads);
  DIM_DISPATCH(dim, jacobian_kernel, kTileThreads, positions, initial_deltas, num_groups, jacobian);
  return check_launch("jacobian_kernel");
}

int ftle_cauchy_green(int32_t dim, const double *jacobian, int64_t n, double *cauchy_green,
                      void *stream) {
  if (dim != 2 && dim != 3) return fail_invalid("dim must be 2 or 3");
  if (n < 0) return fail_invalid("n must be >= 0");
  if (n == 0) return FTLE_OK;
  if (!jacobian || !cauchy_green) return fail_invalid("null pointer");
  const unsigned b = grid_blocks(n, kTileThreads);
  DIM_DISPATCH(dim, cauchy_green_kernel, kTileThreads, jacobian, n, cauchy_green);
  return check_launch("cauchy_green_kernel");
}

int ftle_max_eigenvalue(int32_t dim, const double *cauchy_green, int64_t n, double *out,
                        void *stream) {
  if (dim != 2 && dim != 3) return fail_invalid("dim must be 2 or 3");
  if (n < 0) return fail_invalid("n must be >= 0");
  if (n == 0) return FTLE_OK;
  if (!cauchy_green || !out) return fail_invalid("null pointer");
  const unsigned b = grid_blocks(n, kTileThreads);
  DIM_DISPATCH(dim, max_eigenvalue_kernel, kTileThreads, cauchy_green, n, out);
  return check_launch("max_eigenvalue_kernel");
}

int ftle_from_jacobian(int32_t dim, const double *jacobian, int64_t n, double map_period,
                       double *out, void *stream) {
  if (dim != 2 && dim != 3) return fail_invalid("dim must be 2 or 3");
  if (n < 0) return fail_invalid("n must be >= 0");
  if (!(map_period != 0.0)) return fail_invalid("map_period must be non-zero");
  if (n == 0) return FTLE_OK;
  if (!jacobian || !out) return fail_invalid("null pointer");
  const unsigned b = grid_blocks(n, kTileThreads);
  DIM_DISPATCH(dim, ftle_from_jacobian_kernel, kTileThreads, jacobian, n, map_period, out);
  return check_launch("ftle_from_jacobian_kernel");
}

int ftle_from_positions(int32_t dim, const double *positions, const double *initial_deltas,
                        int64_t num_groups, double map_period, double *out, void *stream) {
  if (dim != 2 && dim != 3) return fail_invalid("dim must be 2 or 3");
  if (num_groups < 0) return fail_invalid("num_groups must be >= 0");
  if (!(map_period != 0.0)) return fail_invalid("map_period must be non-zero");
  if (num_groups == 0) return FTLE_OK;
  if (!positions || !initial_deltas || !out) return fail_invalid("null pointer");
  const unsigned b = grid_blocks(num_groups, 256);
  DIM_DISPATCH(dim, ftle_from_positions_kernel, 256, positions, initial_deltas, num_groups,
               map_period, out);
  return check_launch("ftle_from_positions_kernel");
}

int ftle_analytic_window_run(const ftle_flow *flow, int32_t integrator, double t0, double h,
                             int32_t num_steps, int32_t freeze_time, double *positions,
                             int64_t num_groups, double map_period, double *ftle, void *stream) {
  if (!flow) return fail_invalid("flow descriptor is NULL");
  int dim;
  if (flow->kind == FTLE_FLOW_DOUBLE_GYRE)
    dim = 2;
  else if (flow->kind == FTLE_FLOW_ABC)
    dim = 3;
  else
    return fail_invalid("unknown flow kind %d", flow->kind);
  if (integrator < FTLE_EULER || integrator > FTLE_RK4)
    return fail_invalid("unknown integrator %d", integrator);
  if (num_steps < 0 || num_groups < 0) return fail_invalid("sizes must be >= 0");
  if (ftle && !(map_period > 0.0) && !(map_period < 0.0))
    return fail_invalid("map_period must be non-zero");
  if (num_groups == 0) return FTLE_OK;
  if (!positions) return fail_invalid("positions are required");
  FlowK f;
  f.kind = flow->kind;
  for (int i = 0; i < 8; ++i) f.p[i] = flow->params[i];
  cudaStream_t st = as_stream(stream);
#define AN(D, I, G)                                                                       \
  analytic_window_kernel<D, I, G><<<(unsigned)((num_groups + G - 1) / G), 2 * D * G, 0, st>>>( \
      f, t0, h, num_steps, freeze_time, positions, num_groups, map_period, ftle)
  if (dim == 2) {
    if (integrator == FTLE_EULER) AN(2, FTLE_EULER, 64);
    else if (integrator == FTLE_AB2) AN(2, FTLE_AB2, 64);
    else AN(2, FTLE_RK4, 64);
  } else {
    if (integrator == FTLE_EULER) AN(3, FTLE_EULER, 32);
    else if (integrator == FTLE_AB2) AN(3, FTLE_AB2, 32);
    else AN(3, FTLE_RK4, 32);
  }
#undef AN
  return check_launch("analytic_window_kernel");
}

}  // extern "C"

namespace ftle {

int pack_snapshots_f64(int32_t dim, int64_t nodes, int32_t num_snapshots, int32_t periodic_time,
                       const double *src, double *dst, void *stream) {
  cudaStream_t st = as_stream(stream);
#define PACK(D, R)                                                                     \
  pack_f64_kernel<D, R><<<pack_grid(nodes, num_snapshots, R), 256, 0, st>>>(src, nodes, \
      num_snapshots, periodic_time, dst)
  // runs of snapshots pay in 3D (128^3 x 16: none 460 us, runs of 8 417, of 4 384); in 2D the
  // second read of a value comes from L2 and single snapshots are a little faster (512 x 256
  // x 40: 39.7 us against 42.7 with runs of 8)
  if (dim == 2)
    PACK(2, 1);
  else if (num_snapshots >= 2)
    PACK(3, 4);
  else
    PACK(3, 1);
#undef PACK
  return check_launch("pack_f64_kernel");
}

}  // namespace ftle

