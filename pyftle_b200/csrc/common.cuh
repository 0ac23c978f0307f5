// common.cuh -- shared host/device helpers of the FTLE engine (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "pyftle_b200.h"

namespace ftle {

// ---------------------------------------------------------------------------
// host-side error plumbing (no exceptions cross the C ABI)
// ---------------------------------------------------------------------------
void set_error(const char *fmt, ...);
int fail_invalid(const char *fmt, ...);
int check_launch(const char *what);

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

constexpr int kNumSMs = 148;  // B200

// Grid constants passed by value to kernels.
struct GridK {
  int n[3];
  double origin[3];
  double spacing[3];
  int periodic;
  long long nodes;
  // for the FP64 path's correctly rounded division by the spacing (plain_f64.cu)
  double rcp_hi[3], rcp_lo[3];             // 1/spacing as RN(1/s) and the rest of it
  unsigned div_min;                        // high word of the least |x - origin| it covers
  double man[3], man_hi[3], man_lo[3];     // spacing / 2^man_exp in +-[1, 2), its reciprocal
  int man_exp[3];
};

int grid_from_abi(const ftle_grid *g, GridK *out);

// Window constants passed by value to the window kernels.
struct WinK {
  GridK g;
  const void *snaps;  // packed records (layout depends on the storage type)
  int num_snaps, periodic_time, first_snapshot, num_steps;
  double snap_t0, snap_dt, t0, h, map_period;
  double *positions;
  long long N;
  double *ftle;
  int keep_positions;  // FTLE_KEEP_POSITIONS: do not write final positions
};

// Validates an ftle_window and converts it to kernel constants.
int window_to_kernel(const ftle_window *w, WinK *k);

int pack_snapshots_f64(int32_t dim, int64_t nodes, int32_t num_snapshots, int32_t periodic_time,
                       const double *src, double *dst, void *stream);
int pack_snapshots_16(int32_t dim, int64_t nodes, int32_t num_snapshots, int32_t periodic_time,
                      const double *src, int32_t storage, void *dst, void *stream);

// Blocks for a grid-stride launch over n work items.
inline unsigned grid_blocks(int64_t n, int threads, int per_sm = 8) {
  int64_t b = (n + threads - 1) / threads;
  int64_t cap = (int64_t)kNumSMs * per_sm * 8;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (unsigned)b;
}

// Grid of a packing kernel: blocks of 256 nodes x runs of `run` snapshots per thread.  A run
// reads (and encodes) its values once plus a successor, a single snapshot twice; long runs
// take registers and leave a longer tail.
inline dim3 pack_grid(int64_t nodes, int32_t num_snapshots, int run) {
  const int64_t runs = (num_snapshots + run - 1) / run;
  return dim3((unsigned)((nodes + 255) / 256), (unsigned)(runs < 65535 ? runs : 65535));
}

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------

// Wrap a cell index into [0, n) for periodic grids.
__device__ __forceinline__ int wrap_index(int q, int n) {
  int r = q % n;
  return r < 0 ? r + n : r;
}

// Largest eigenvalue of a symmetric 3x3 matrix (FP64).  With q = tr A / 3 and B = A - q I the
// eigenvalues of B solve x^3 - c1 x = det B.  The root on det B's side is the isolated one
// (its distance from the others is at least sqrt(3) times the root mean square): an FP32
// start and two Newton steps give it to rounding.  On the positive side it is the largest;
// on the negative side (x the smallest) the other two are -x/2 +- d, and d^2 is half the
// squared norm of B + x/2 I - 3/2 x P with P = adj(B - x I) / tr adj the projector on x's
// eigenvector, which stays accurate when the two coincide.  B is scaled by a power of two.
// Relative error 0.5-0.9e-16 (root mean square, 3e-16 at most) over random, stretched, graded,
// nearly isotropic and nearly degenerate C = F F^T, where cyclic Jacobi rotations have 0.6-1.4e-16
// (5e-16); 0.2e-16 where C is all but diagonal, which rotations leave exact.  About a tenth of
// their operations.
static __device__ __noinline__ double lmax3_sym(double a00, double a01, double a02, double a11,
                                                double a12, double a22) {
  const double off = fabs(a01) + fabs(a02) + fabs(a12);
  if (off <= 1e-300 || off < 1e-18 * (fabs(a00) + fabs(a11) + fabs(a22))) {
    double mx = a00;
    if (a11 > mx) mx = a11;
    if (a22 > mx) mx = a22;
    return mx;
  }
  const double tr = a00 + a11 + a22;
  const double q = tr * (1.0 / 3.0);
  double b0 = a00 - q, b1 = a11 - q, b2 = a22 - q;
  // what rounding left of B's trace: next to a multiple of I it is as large as B
  const double t = (b0 + b1 + b2) * (1.0 / 3.0);
  b0 -= t, b1 -= t, b2 -= t;
  int e = ((__double2hiint(fabs(b0) + fabs(b1) + fabs(b2) + off) >> 20) & 0x7ff) - 1023;
  e = e > 1022 ? 1022 : e;
  const double down = __hiloint2double((1023 - e) << 20, 0);
  b0 *= down, b1 *= down, b2 *= down;
  a01 *= down, a02 *= down, a12 *= down;
  const double c1 =
      fma(0.5, fma(b0, b0, fma(b1, b1, b2 * b2)), fma(a01, a01, fma(a02, a02, a12 * a12)));
  const double det = fma(b0, fma(b1, b2, -(a12 * a12)),
                         fma(a01, fma(a12, a02, -(a01 * b2)), a02 * fma(a01, a12, -(b1 * a02))));
  // y^3 - 3y = rho in [0, 2] for y = |x| / sqrt(c1 / 3)
  const float ip = rsqrtf((float)c1 * (1.0f / 3.0f));
  const float rho = fminf(fabsf((float)det) * ip * ip * ip, 2.0f);
  float y = fmaf(fmaf(-0.016346f, rho, 1.0f / 6.0f), rho, 1.7320508f);
#pragma unroll
  for (int i = 0; i < 2; ++i)
    y -= __fdividef(fmaf(y, fmaf(y, y, -3.0f), -rho), fmaf(3.0f * y, y, -3.0f));
  double x = (double)__fdividef(y, ip);
  if (det < 0.0) x = -x;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double f = fma(x, fma(x, x, -c1), -det);
    x = fma(-f, (double)__frcp_rn((float)fma(3.0 * x, x, -c1)), x);
  }
  double m = x;
  if (det < 0.0) {
    const double r0 = b0 - x, r1 = b1 - x, r2 = b2 - x;
    const double d00 = fma(r1, r2, -(a12 * a12)), d11 = fma(r0, r2, -(a02 * a02));
    const double d22 = fma(r0, r1, -(a01 * a01));
    const double s = -1.5 * x / (d00 + d11 + d22), h = 0.5 * x;
    const double e0 = fma(s, d00, b0 + h), e1 = fma(s, d11, b1 + h), e2 = fma(s, d22, b2 + h);
    const double f0 = fma(s, fma(a02, a12, -(a01 * r2)), a01);
    const double f1 = fma(s, fma(a01, a12, -(a02 * r1)), a02);
    const double f2 = fma(s, fma(a01, a02, -(a12 * r0)), a12);
    m = sqrt(fma(0.5, fma(e0, e0, fma(e1, e1, e2 * e2)), fma(f0, f0, fma(f1, f1, f2 * f2)))) - h;
  }
  return q + fma(m, __hiloint2double((1023 + e) << 20, 0), t);
}

}  // namespace ftle
