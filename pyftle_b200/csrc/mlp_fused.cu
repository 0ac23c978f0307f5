// mlp_fused.cu -- fused surrogate inference: seeds -> FTLE in one persistent kernel.
//
// Network: F Fourier frequencies (2F features of (x0, t0)), `depth` hidden layers of `hid`
// SiLU units, DIM outputs (the displacement / out_scale); 2D and 3D, hid a multiple of 64 up
// to 384.  The FTLE of the surrogate flow map x0 -> x0 + s*y(x0) needs y and its Jacobian, so
// every seed carries 1 + DIM rows through the network: the primal activations and the
// forward-mode tangents d/dx0, ... (the tangent of a SiLU layer is the pre-activation tangent
// times silu'(z) of the primal row).
//
// Tile = 128 tensor-core rows, 32 seeds.  TMEM lane quadrant q (rows 32q..32q+31) holds 8
// seeds as [8 primal | 8 d/dx | 8 d/dy | 8 d/dz] (in 2D the last 8 rows are zero): the fragment
// loads then put all rows of a seed into one thread.  The tile's activations stay in shared
// memory as the next layer's A operand.
//
// Warp roles:
//   * a producer warp streams the packed weights (64-wide K chunks, already in the 128-byte-swizzled
//     layout) by 1D bulk copies into a ring;
//   * an MMA warp issues the tcgen05.mma chains (M = 128, N = hid or its half, K = 16) of a
//     layer once the layer's input is complete;
//   * 4 P epilogue warps: warp w reads TMEM lane quadrant w%4 and the (w/4)-th part of every
//     64 columns, applies bias, SiLU and the tangent rule and writes the BF16 A operand of the next layer
//     in place; at the output layer the first part's warps form F = I + s*J, C = F^T F and the
//     FTLE in FP64 (as ftle_mlp_jacobian_ftle).  They also compute the next tile's features.
// A layer's MMAs and its epilogue depend on each other.  They overlap by 64-column chunk: the
// MMAs of a chunk start when its columns are written (up to hid = 256 into the other of two
// accumulators; above, one fits and its first half has to be read), the next tile's features
// are made under the output layer's MMAs, and a tile's FP64 tail under the next one's layer 1.
// Up to hid = 128 two CTAs of P = 2 share an SM (262,144 seeds, 4 x 128 in 2D: 316 us, one CTA
// of P = 4 476 us); above, one of P = 4.  Bound by shared memory: an MMA of N = 256 reads 12 KB
// in its 131 clocks, beside the weights' arrival and the epilogue's stores.
// 1M seeds, 4 x 256 in 2D: 3.63 ms with a SiLU in every lane and silu'(z) shuffled to the
// tangent rows, 2.44 ms now; 262,144 seeds, 4 x 384 in 3D: 2.65 ms on the layered kernels,
// 1.23 ms.  What mattered on the way: counting ring positions instead of dividing (a 64-bit
// division per chunk cost more than its MMAs) and suspending waits (polling warps took the
// operand reads' shared-memory cycles, 2.89 -> 2.70 ms).
// Every wait is bounded; on timeout the kernel flags the error word, stops all roles, waits
// (bounded) for its copies and MMAs in flight, frees TMEM, returns.
#include <cuda_bf16.h>

#include "common.cuh"
#include "umma.cuh"

namespace ftle {
namespace mlp {

// Rows (N) of a weight chunk, of kChunkK columns: one instruction's N, at most 256.
__host__ __device__ __forceinline__ int weight_rows(int hid) { return hid <= 256 ? hid : hid / 2; }
constexpr int kSeeds = 8;      // seeds per TMEM lane quadrant
constexpr int kTile = 4 * kSeeds;
constexpr int kTwoCtaHid = 128; // two CTAs share an SM up to this width
constexpr int kOutRows = 16;    // output rows evaluated (the first DIM are used)
constexpr int kMaxDepth = 8;
constexpr int kMaxStages = 8;
constexpr int kMaxChunks = 6;   // 384 / 64
constexpr int kAChunkBytes = 128 * kChunkK * 2;  // 16 KB: 128 rows x 64 columns of A

struct FieldArgs {
  const double *points;  // n rows of ld doubles: the seed, and its start time where ld > DIM
  int ld;
  long long n;
  double t0;             // start time where the rows hold none
  int hid, depth, freqs;
  const unsigned char *wpack;
  const float *bias[kMaxDepth + 1];
  const float4 *freq;    // (kx, ky, kt, phase); 3D two per frequency, (kx, ky, kz, kt), (phase, ...)
  double out_scale;
  double inv_T;
  double *ftle;          // n, may be null
  double *end_pos;       // n x DIM, may be null
  int *err;
  int stages;            // weight ring
};

// Bytes of the packed weights: every layer's chunks, the output's 16 x hid.
__host__ __device__ inline long long packed_bytes(int hid, int depth, int feats) {
  return 2ll * hid * (feats + (long long)(depth - 1) * hid + kOutRows);
}
inline size_t field_smem(int hid, int depth, int feats, int dim, int stages) {
  return (size_t)((hid + feats) / kChunkK) * kAChunkBytes + (size_t)stages * weight_rows(hid) * kChunkK * 2 +
         (size_t)(depth * hid + kOutRows) * 4 + (size_t)(feats / 2) * 16 * (dim - 1) + 1024;
}

struct FieldShared {
  unsigned long long full_bar[kMaxStages];
  unsigned long long empty_bar[kMaxStages];
  unsigned long long acc_full[2];
  unsigned long long f_ready;               // layer 0's operand (features)
  unsigned long long out_read;              // the output accumulator
  unsigned long long a_ready[kMaxChunks];   // 64-column chunk of a hidden layer's output
  unsigned long long drain_bar;
  uint32_t tmem_slot;
  int abort_flag;
};

__device__ __forceinline__ bool aborted(const FieldShared &S) {
  return *reinterpret_cast<const volatile int *>(&S.abort_flag) != 0;
}
__device__ __forceinline__ void flag_abort(const FieldArgs &a, FieldShared &S) {
  *reinterpret_cast<volatile int *>(&S.abort_flag) = 1;
  atomicExch(a.err, 1);
}

// Position in the weight ring (kept by counting: a division per chunk costs more than its MMAs).
struct RingPos {
  int slot = 0, turns = 0, stages;
  uint32_t phase = 0;
  __device__ explicit RingPos(int n) : stages(n) {}
  __device__ __forceinline__ void next() {
    if (++slot == stages) {
      slot = 0;
      phase ^= 1u;
      ++turns;
    }
  }
};

__device__ void field_producer(const FieldArgs &a, FieldShared &S, uint32_t sW, long long tiles) {
  const int rows = weight_rows(a.hid);
  const int per = (2 * a.freqs + (a.depth - 1) * a.hid) / kChunkK * (a.hid / rows) + 1;
  const uint32_t slot = (uint32_t)(rows * kChunkK * 2), last = (uint32_t)a.hid * kOutRows * 2;
  RingPos r(a.stages);
  bool ok = true;
  for (long long t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
    const unsigned char *src = a.wpack;
    for (int i = 0; i < per; ++i, r.next()) {
      const uint32_t bytes = i + 1 < per ? slot : last;
      ok = mbar_wait(smem_u32(&S.empty_bar[r.slot]), r.phase ^ 1u) && !aborted(S);
      if (!ok) break;
      mbar_expect_tx(smem_u32(&S.full_bar[r.slot]), bytes);
      bulk_g2s(sW + r.slot * slot, src, bytes, smem_u32(&S.full_bar[r.slot]));
      src += bytes;
    }
  }
  if (!ok) flag_abort(a, S);
  // copies in flight land before the CTA exits: slots below the position in this turn of the
  // ring, the others in the one before
  for (int k = 0; k < a.stages; ++k)
    if (k < r.slot || r.turns > 0)
      mbar_wait(smem_u32(&S.full_bar[k]), k < r.slot ? r.phase : r.phase ^ 1u);
}

// TMEM columns between the two accumulators, 0 where only one fits.
__device__ __forceinline__ uint32_t acc_stride(int hid) { return hid <= 256 ? (uint32_t)hid : 0u; }

// One thread issues every MMA, so its instructions per chunk are the tensor core's pace: the
// descriptors advance by constants.
__device__ void field_mma(const FieldArgs &a, FieldShared &S, uint32_t sA, uint32_t sF, uint32_t sW,
                          uint32_t tmem, long long tiles) {
  const int nh = weight_rows(a.hid), halves = a.hid / nh;
  const uint32_t idesc = idesc_bf16(128, nh), idesc_out = idesc_bf16(128, kOutRows);
  const uint32_t stride = acc_stride(a.hid);
  const int chunks = a.hid / kChunkK, depth = a.depth, feat_chunks = 2 * a.freqs / kChunkK;
  // descriptor address fields count 16 bytes
  const uint64_t a0 = smem_desc_sw128(sA, 16, 1024), f0 = smem_desc_sw128(sF, 16, 1024),
                 w0 = smem_desc_sw128(sW, 16, 1024);
  const uint32_t slot16 = (uint32_t)(nh * kChunkK * 2) >> 4;
  RingPos r(a.stages);
  uint32_t layer = 0, ready = 0, tile = 0;  // ready: hidden outputs consumed
  bool ok = true;
  auto input = [&](int c) { return mbar_wait(smem_u32(&S.a_ready[c]), ready & 1u); };
  for (long long t = blockIdx.x; ok && t < tiles; t += gridDim.x, ++tile) {
    for (int l = 0; ok && l <= depth; ++l, ++layer) {
      const uint32_t acc = tmem + (layer & 1u) * stride;
      if (l == 0) {
        // with two accumulators layer 0's is free (the output layer's input, complete by then,
        // came from it); the last tile's outputs have to be read before layer 1, which implies
        // it: every warp reads them before its part of layer 0.  With one accumulator they
        // have to be read here.
        ok = mbar_wait(smem_u32(&S.f_ready), tile & 1u) &&
             (stride != 0 || tile == 0 || mbar_wait(smem_u32(&S.out_read), (tile - 1) & 1u));
      } else if (l == depth) {
        for (int c = 0; ok && c < chunks; ++c) ok = input(c);  // the whole input
      }
      ok = ok && !aborted(S);
      if (l < depth) {
        const int nk = l == 0 ? feat_chunks : chunks;
        for (int h = 0; ok && h < halves; ++h) {
          uint64_t ad = l == 0 ? f0 : a0;
          for (int c = 0; ok && c < nk; ++c, ad += kAChunkBytes >> 4, r.next()) {
            if (l > 0 && h == 0) {
              // this chunk of the input; with one accumulator the first half's columns have
              // to be read as well, which the input chunks of the same columns imply
              if (stride == 0 && c == 0)
                for (int k = 1; ok && k < (chunks + 1) / 2; ++k) ok = input(k);
              ok = ok && input(c);
            }
            ok = ok && mbar_wait(smem_u32(&S.full_bar[r.slot]), r.phase);
            if (!ok) break;
            fence_after_sync();
            const uint64_t wd = w0 + (uint32_t)r.slot * slot16;
#pragma unroll
            for (int kk = 0; kk < kChunkK / 16; ++kk)
              umma(acc + (uint32_t)(h * nh), ad + 2 * kk, wd + 2 * kk, idesc, (c | kk) ? 1u : 0u);
            umma_commit(smem_u32(&S.empty_bar[r.slot]));
          }
        }
      } else if (ok) {
        ok = mbar_wait(smem_u32(&S.full_bar[r.slot]), r.phase);
        if (ok) {
          fence_after_sync();
          uint64_t wd = w0 + (uint32_t)r.slot * slot16, ad = a0;
          for (int c = 0; c < chunks; ++c, ad += kAChunkBytes >> 4, wd += kOutRows * kChunkK * 2 >> 4)
#pragma unroll
            for (int kk = 0; kk < kChunkK / 16; ++kk)
              umma(acc, ad + 2 * kk, wd + 2 * kk, idesc_out, (c | kk) ? 1u : 0u);
          umma_commit(smem_u32(&S.empty_bar[r.slot]));
          r.next();
        }
      }
      if (l > 0) ++ready;
      if (ok) umma_commit(smem_u32(&S.acc_full[layer & 1u]));
    }
  }
  if (!ok) flag_abort(a, S);
  // MMAs in flight complete before the CTA exits
  umma_commit(smem_u32(&S.drain_bar));
  mbar_wait(smem_u32(&S.drain_bar), 0);
}

// ---- epilogue warps -------------------------------------------------------------------
// W columns [c, c + W) of a hidden layer: bias, SiLU, tangent rule, BF16 A operand of the next
// layer.  The 16x256b TMEM loads give thread t rows t/4 and t/4 + 8 of a 16-row half and
// columns 2(t%4), 2(t%4)+1 of every 8: with 8 rows per role that is all roles of one seed in
// one thread, so a SiLU is evaluated once per seed and column, silu'(z) stays in its thread,
// and a warp's 4-byte stores are free of bank conflicts.  Pairs of columns go through the
// packed FP32 instructions, which round like sigmoidf_ and dsilu_from.
template <int W>
struct Fragment {  // [8-column block][primal, d/dx pairs], [...][d/dy, d/dz pairs]
  uint32_t p[W / 2], q[W / 2];
  __device__ __forceinline__ void start(uint32_t taddr) {
    tmem_ld16x256_start(taddr, p);
    tmem_ld16x256_start(taddr + (16u << 16), q);
  }
  __device__ __forceinline__ void wait() {
    tmem_wait(p);
    tmem_wait(q);
  }
};

template <int DIM, int W>
__device__ __forceinline__ void hidden_part(const Fragment<W> &f, const float *bias, int lane,
                                            unsigned char *sA, int quad, int c) {
  const int s = lane >> 2;  // the seed: row 8 role + s of the quadrant
  unsigned char *out = sA + (c >> 6) * kAChunkBytes + quad * 4096 + s * 128 + (lane & 3) * 4;
  const float2 half = make_float2(0.5f, 0.5f), one = make_float2(1.0f, 1.0f),
               neg = make_float2(-1.0f, -1.0f);
  auto pair = [](const uint32_t *r) { return make_float2(__uint_as_float(r[0]), __uint_as_float(r[1])); };
  auto put = [&](int role, int i, float2 v) {
    *reinterpret_cast<__nv_bfloat162 *>(out + role * 1024 + (((((c & 63) >> 3) + i) ^ s) << 4)) =
        __floats2bfloat162_rn(v.x, v.y);
  };
#pragma unroll
  for (int i = 0; i < W / 8; ++i) {
    const float2 z = __fadd2_rn(pair(f.p + 4 * i),
                                *reinterpret_cast<const float2 *>(bias + 8 * i + 2 * (lane & 3)));
    const float2 u = __fmul2_rn(half, z);
    const float2 sg = __ffma2_rn(half, make_float2(tanh_approx(u.x), tanh_approx(u.y)), half);
    const float2 h = __fmul2_rn(z, sg);
    const float2 d = __ffma2_rn(h, __ffma2_rn(sg, neg, one), sg);
    put(0, i, h);
    put(1, i, __fmul2_rn(pair(f.p + 4 * i + 2), d));
    put(2, i, __fmul2_rn(pair(f.q + 4 * i), d));
    if constexpr (DIM == 3) put(3, i, __fmul2_rn(pair(f.q + 4 * i + 2), d));
  }
}

// Layer 0's operand of tile t: features and their tangents, two frequencies at a time.
template <int DIM, int P>
__device__ __forceinline__ void field_features(const FieldArgs &a, FieldShared &S, unsigned char *sF,
                                               const float4 *sfreq, long long t, int warp, int lane) {
  constexpr int kRoles = DIM + 1;
  const int F = a.freqs;
  for (int e = warp * 32 + lane; e < kTile * (F / 2); e += 128 * P) {
    const int st = e / (F / 2), f = 2 * (e - st * (F / 2));
    const int q = st / kSeeds, s = st - q * kSeeds;
    const long long g = t * kTile + st;
    __nv_bfloat16 vals[kRoles][2][2];  // [role][sin | cos][frequency]
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float sn = 0.f, cs = 0.f, kk[3];
      const float4 k = sfreq[(f + i) * (DIM - 1)];
      kk[0] = k.x, kk[1] = k.y, kk[2] = k.z;
      if (g < a.n) {
        const double *pt = a.points + g * a.ld;
        const double tt = a.ld > DIM ? pt[DIM] : a.t0;
        // the phase is formed and reduced in FP64, as in the feature kernels of training
        double ph;
        if constexpr (DIM == 2)
          ph = (double)k.x * pt[0] + (double)k.y * pt[1] + (double)k.z * tt + (double)k.w;
        else
          ph = (double)k.x * pt[0] + (double)k.y * pt[1] + (double)k.z * pt[2] +
               (double)k.w * tt + (double)sfreq[2 * (f + i) + 1].x;
        const double two_pi = 6.283185307179586;
        sincosf((float)(ph - two_pi * floor(ph / two_pi)), &sn, &cs);
      }
      vals[0][0][i] = __float2bfloat16_rn(sn);
      vals[0][1][i] = __float2bfloat16_rn(cs);
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        vals[1 + d][0][i] = __float2bfloat16_rn(kk[d] * cs);
        vals[1 + d][1][i] = __float2bfloat16_rn(-kk[d] * sn);
      }
    }
#pragma unroll
    for (int rr = 0; rr < kRoles; ++rr)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int r = 32 * q + rr * kSeeds + s, c = j * F + f;
        *reinterpret_cast<__nv_bfloat162 *>(sF + (c >> 6) * kAChunkBytes + sw128_off(r, c & 63)) =
            __nv_bfloat162(vals[rr][j][0], vals[rr][j][1]);
      }
  }
  fence_before_sync();
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(&S.f_ready));
}

template <int DIM, int P>
__device__ void field_epilogue(const FieldArgs &a, FieldShared &S, unsigned char *sA,
                               unsigned char *sF, const float *sbias, const float4 *sfreq, uint32_t tmem,
                               long long tiles, int warp, int lane) {
  const int quad = warp & 3, part = warp >> 2;
  const bool primal = lane < kSeeds;
  const int sl = lane & (kSeeds - 1);
  const uint32_t stride = acc_stride(a.hid);
  constexpr int W = kChunkK / P;  // this warp's columns of a 64-column chunk
  // the outputs of the last tile, j[r][d] = dy_r / dx_d, of seed g (in the first part's primal
  // lanes), and their FP64 fields
  float y[DIM] = {}, j[DIM][DIM] = {};
  long long g = a.n;
  auto finish = [&]() {
    if (primal && g < a.n) {
      const double s = a.out_scale;
      if (a.ftle) {
        double lam;
        if constexpr (DIM == 2) {
          const double fa = 1.0 + s * (double)j[0][0], fb = s * (double)j[0][1];
          const double fc = s * (double)j[1][0], fd = 1.0 + s * (double)j[1][1];
          const double c11 = fa * fa + fc * fc, c12 = fa * fb + fc * fd;
          const double c22 = fb * fb + fd * fd;
          const double tr = 0.5 * (c11 + c22), df = 0.5 * (c11 - c22);
          lam = tr + sqrt(df * df + c12 * c12);
        } else {
          double Fm[3][3], C[3][3];
#pragma unroll
          for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int d = 0; d < 3; ++d) Fm[r][d] = (r == d ? 1.0 : 0.0) + s * (double)j[r][d];
#pragma unroll
          for (int u = 0; u < 3; ++u)
#pragma unroll
            for (int v = 0; v < 3; ++v)
              C[u][v] = Fm[0][u] * Fm[0][v] + Fm[1][u] * Fm[1][v] + Fm[2][u] * Fm[2][v];
          lam = lmax3_sym(C[0][0], C[0][1], C[0][2], C[1][1], C[1][2], C[2][2]);
        }
        a.ftle[g] = log(sqrt(lam)) * a.inv_T;
      }
      if (a.end_pos) {
        const float *b = sbias + a.depth * a.hid;
#pragma unroll
        for (int r = 0; r < DIM; ++r)
          a.end_pos[DIM * g + r] = a.points[a.ld * g + r] + s * (double)(y[r] + b[r]);
      }
    }
    g = a.n;
  };
  uint32_t layer = 0;
  field_features<DIM, P>(a, S, sF, sfreq, blockIdx.x, warp, lane);
  for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
    for (int l = 0; l <= a.depth; ++l, ++layer) {
      // the next tile's features while the output layer's MMAs run, so that its layer 0
      // follows them at once
      if (l == a.depth && t + gridDim.x < tiles)
        field_features<DIM, P>(a, S, sF, sfreq, t + gridDim.x, warp, lane);
      const bool ok = mbar_wait(smem_u32(&S.acc_full[layer & 1u]), (layer >> 1) & 1u);
      if (__any_sync(0xFFFFFFFFu, !ok || aborted(S))) {  // warp-uniform exit
        if (lane == 0) flag_abort(a, S);
        return;
      }
      fence_after_sync();
      const uint32_t trow = tmem + ((uint32_t)(32 * quad) << 16) + (layer & 1u) * stride;
      if (l < a.depth) {
        // all warps work on one 64-column chunk after the other: the next layer's MMAs of a
        // chunk start as soon as it is complete
        const float *b = sbias + l * a.hid;
        Fragment<W> f0, f1;
        auto chunk = [&](const Fragment<W> &f, int k) {
          const int c = kChunkK * k + W * part;
          hidden_part<DIM, W>(f, b + c, lane, sA, quad, c);
          fence_before_sync();
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&S.a_ready[k]));
        };
        const uint32_t tcol = trow + (uint32_t)(W * part);
        const int chunks = a.hid / kChunkK;
        f0.start(tcol);
        for (int k = 0; k < chunks; k += 2) {
          f0.wait();
          if (k + 1 < chunks) f1.start(tcol + (uint32_t)(kChunkK * (k + 1)));
          chunk(f0, k);
          if (k + 1 < chunks) {
            f1.wait();
            if (k + 2 < chunks) f0.start(tcol + (uint32_t)(kChunkK * (k + 2)));
            chunk(f1, k + 1);
          }
        }
        if (l == 0) finish();  // the last tile's fields, while layer 1's MMAs run
      } else {
        if (part == 0) {
          uint32_t rr[16];
          tmem_ld16_start(trow, rr);
          tmem_wait16(rr);
          fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&S.out_read));
#pragma unroll
          for (int r = 0; r < DIM; ++r) {
            y[r] = __uint_as_float(rr[r]);
#pragma unroll
            for (int d = 0; d < DIM; ++d)
              j[r][d] = __shfl_sync(0xFFFFFFFFu, y[r], sl + (1 + d) * kSeeds);
          }
          g = t * kTile + quad * kSeeds + lane;
        }
      }
    }
  }
  finish();
}

template <int DIM, int P>
__global__ void __launch_bounds__(64 + 128 * P, P == 2 ? 2 : 1) surrogate_field_kernel(FieldArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) FieldShared S;
  constexpr int kThreads = 64 + 128 * P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long tiles = (a.n + kTile - 1) / kTile;
  const int feats = 2 * a.freqs;
  const int achunks = (a.hid + feats) / kChunkK;  // hidden operand, then the features'
  uint32_t cols = 32;  // TMEM is allocated in powers of two
  while (cols < (uint32_t)a.hid + acc_stride(a.hid)) cols *= 2;
  // [A | features | weight ring | frequencies | biases]
  unsigned char *base = smem + ((1024u - (smem_u32(smem) & 1023u)) & 1023u);
  unsigned char *sA = base, *sF = base + a.hid / kChunkK * kAChunkBytes;
  const uint32_t sW = smem_u32(base) + achunks * kAChunkBytes;
  float4 *sfreq = reinterpret_cast<float4 *>(base + achunks * kAChunkBytes +
                                             (size_t)a.stages * weight_rows(a.hid) * kChunkK * 2);
  float *sbias = reinterpret_cast<float *>(sfreq + a.freqs * (DIM - 1));

  if (warp == 0) tmem_alloc(smem_u32(&S.tmem_slot), cols);
  if (tid == 32) {
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(smem_u32(&S.full_bar[s]), 1);
      mbar_init(smem_u32(&S.empty_bar[s]), 1);
    }
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&S.acc_full[i]), 1);
    mbar_init(smem_u32(&S.f_ready), 4 * P);
    mbar_init(smem_u32(&S.out_read), 4);
    for (int i = 0; i < kMaxChunks; ++i) mbar_init(smem_u32(&S.a_ready[i]), 4 * P);
    mbar_init(smem_u32(&S.drain_bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    S.abort_flag = 0;
  }
  if constexpr (DIM == 2) {  // the fourth row block of each quadrant is zero throughout
    for (int i = tid; i < achunks * 4 * 64; i += kThreads)
      *reinterpret_cast<uint4 *>(sA + (i >> 8) * kAChunkBytes + ((i >> 6) & 3) * 4096 + 3072 +
                                 (i & 63) * 16) = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async_smem();
  }
  for (int i = tid; i < a.depth * a.hid; i += kThreads) sbias[i] = a.bias[i / a.hid][i % a.hid];
  for (int i = tid; i < kOutRows; i += kThreads) sbias[a.depth * a.hid + i] = a.bias[a.depth][i];
  for (int i = tid; i < a.freqs * (DIM - 1); i += kThreads) sfreq[i] = a.freq[i];
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = S.tmem_slot;

  if (warp < 4 * P) {
    field_epilogue<DIM, P>(a, S, sA, sF, sbias, sfreq, tmem, tiles, warp, lane);
  } else if (warp == 4 * P) {
    if (lane == 0) field_producer(a, S, sW, tiles);
  } else {
    if (lane == 0) field_mma(a, S, smem_u32(sA), smem_u32(sF), sW, tmem, tiles);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, cols);
}

// Packs the BF16 weight matrices (row-major out x in: hid x feats, depth - 1 of hid x hid, the
// first 16 rows of the output layer) into the chunk images; a thread moves 8 values along K.
struct PackArgs {
  const __nv_bfloat16 *w[kMaxDepth + 1];
  int hid, depth, feats;
};
__global__ void surrogate_pack_kernel(const PackArgs a, unsigned char *__restrict__ out) {
  const long long total = packed_bytes(a.hid, a.depth, a.feats) / 16;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    // layer l's image starts after hid * (its predecessors' K) values
    long long q = e * 8;
    int l = 0, K = a.feats;
    while (l < a.depth && q >= (long long)a.hid * K) {
      q -= (long long)a.hid * K;
      ++l;
      K = a.hid;
    }
    // chunks of `rows` x 64, the rows' halves outermost; a row is 8 pieces of 16 bytes, swizzled
    const int rows = l < a.depth ? weight_rows(a.hid) : kOutRows, nk = K / kChunkK;
    const int chunk = (int)(q / (rows * kChunkK)), p = (int)(q - (long long)chunk * rows * kChunkK) / 8;
    const int r = chunk / nk * rows + (p >> 3);
    const int k = chunk % nk * kChunkK + (((p & 7) ^ (p >> 3 & 7)) << 3);
    const __nv_bfloat16 *src = a.w[l] + (long long)r * K + k;
    __align__(16) __nv_bfloat16 v[8];
    if (reinterpret_cast<uintptr_t>(src) % 16 == 0) {
      *reinterpret_cast<uint4 *>(v) = *reinterpret_cast<const uint4 *>(src);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = src[i];
    }
    *reinterpret_cast<uint4 *>(out + e * 16) = *reinterpret_cast<const uint4 *>(v);
  }
}

}  // namespace mlp
}  // namespace ftle

using namespace ftle;
using namespace ftle::mlp;

namespace {

// Dynamic shared memory a block may take: two CTAs per SM up to hid = kTwoCtaHid.
constexpr size_t field_room(bool two_ctas) { return two_ctas ? 112 * 1024 : 224 * 1024; }

// Ring slots that fit beside the activations, 0 if the shape is not one of the kernel's.
int field_stages(int dim, int hid, int depth, int freqs) {
  if ((dim != 2 && dim != 3) || hid < 64 || hid > 384 || hid % 64 || depth < 1 ||
      depth > kMaxDepth || freqs < 32 || freqs % 32 || freqs > 64)
    return 0;
  const size_t room = field_room(hid <= kTwoCtaHid);
  const size_t fixed = field_smem(hid, depth, 2 * freqs, dim, 0);
  if (fixed > room) return 0;
  const size_t fit = (room - fixed) / ((size_t)weight_rows(hid) * kChunkK * 2);
  return fit < 2 ? 0 : (int)(fit < kMaxStages ? fit : kMaxStages);
}

int launch_pack(const PackArgs &p, void *packed, void *stream) {
  const long long pieces = packed_bytes(p.hid, p.depth, p.feats) / 16;
  surrogate_pack_kernel<<<grid_blocks(pieces, 128), 128, 0, as_stream(stream)>>>(
      p, static_cast<unsigned char *>(packed));
  return check_launch("surrogate_pack_kernel");
}

template <int DIM, int P>
void launch_field(const FieldArgs &a, cudaStream_t st) {
  const long long tiles = (a.n + kTile - 1) / kTile;
  const long long cap = (long long)kNumSMs * (P == 2 ? 2 : 1);
  const size_t smem = field_smem(a.hid, a.depth, 2 * a.freqs, DIM, a.stages);
  // the limit is the instance's, the same on every call: one of this shape's size would be
  // lowered by another thread's smaller network before this launch
  cudaFuncSetAttribute(surrogate_field_kernel<DIM, P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)field_room(P == 2));
  surrogate_field_kernel<DIM, P><<<(unsigned)(tiles < cap ? tiles : cap), 64 + 128 * P, smem, st>>>(a);
}

int run_field(FieldArgs &a, int dim, void *stream) {
  a.stages = field_stages(dim, a.hid, a.depth, a.freqs);
  if (!a.stages) return fail_invalid("the fused kernel does not take this network's shape");
  if (reinterpret_cast<uintptr_t>(a.wpack) % 16 || reinterpret_cast<uintptr_t>(a.freq) % 16)
    return fail_invalid("packed weights and freq must be 16-byte aligned");
  cudaStream_t st = as_stream(stream);
  if (dim == 2) {
    if (a.hid <= kTwoCtaHid) launch_field<2, 2>(a, st);
    else launch_field<2, 4>(a, st);
  } else {
    if (a.hid <= kTwoCtaHid) launch_field<3, 2>(a, st);
    else launch_field<3, 4>(a, st);
  }
  return check_launch("surrogate_field_kernel");
}

constexpr int kFixedHid = 256, kFixedDepth = 4, kFixedFreq = 32;  // the 2D entry points' network

}  // namespace

extern "C" {

int64_t ftle_surrogate_packed_bytes(void) {
  return packed_bytes(kFixedHid, kFixedDepth, 2 * kFixedFreq);
}

int ftle_surrogate_pack(const void *w0, const void *w1, const void *w2, const void *w3,
                        const void *w4, void *packed, void *stream) {
  if (!w0 || !w1 || !w2 || !w3 || !w4 || !packed) return fail_invalid("null pointer");
  if (reinterpret_cast<uintptr_t>(packed) % 16) return fail_invalid("packed must be 16-byte aligned");
  PackArgs p{};
  const void *w[5] = {w0, w1, w2, w3, w4};
  for (int l = 0; l < 5; ++l) p.w[l] = static_cast<const __nv_bfloat16 *>(w[l]);
  p.hid = kFixedHid;
  p.depth = kFixedDepth;
  p.feats = 2 * kFixedFreq;
  return launch_pack(p, packed, stream);
}

int ftle_surrogate_ftle(const double *points, int64_t n, double t0, const void *packed,
                        const float *bias, const float *freq, double out_scale, double T,
                        double *ftle, double *end_positions, int32_t *error_word, void *stream) {
  if (n < 0) return fail_invalid("n must be >= 0");
  if (n == 0) return FTLE_OK;
  if (!points || !packed || !bias || !freq || !error_word) return fail_invalid("null pointer");
  if (!ftle && !end_positions) return fail_invalid("nothing to compute");
  if (T == 0.0) return fail_invalid("T must be non-zero");
  FieldArgs a{};
  a.points = points;
  a.ld = 2;
  a.n = n;
  a.t0 = t0;
  a.hid = kFixedHid;
  a.depth = kFixedDepth;
  a.freqs = kFixedFreq;
  a.wpack = static_cast<const unsigned char *>(packed);
  for (int l = 0; l <= kFixedDepth; ++l) a.bias[l] = bias + l * kFixedHid;
  a.freq = reinterpret_cast<const float4 *>(freq);
  a.out_scale = out_scale;
  a.inv_T = 1.0 / fabs(T);
  a.ftle = ftle;
  a.end_pos = end_positions;
  a.err = error_word;
  return run_field(a, 2, stream);
}

int64_t ftle_mlp_field_bytes(int32_t dim, int32_t hidden, int32_t depth, int32_t num_freq) {
  return field_stages(dim, hidden, depth, num_freq) ? packed_bytes(hidden, depth, 2 * num_freq) : -1;
}

// Layer l's weights (out x in) and biases follow each other in the flat parameters; the output
// layer's rows are padded to 64.
static int64_t layer_offset(int l, int hid, int feats) {
  return l == 0 ? 0 : (int64_t)hid * (feats + 1) + (int64_t)(l - 1) * hid * (hid + 1);
}

int ftle_mlp_field_pack(int32_t dim, int32_t hidden, int32_t depth, int32_t num_freq,
                        const void *w_bf16, void *packed, void *stream) {
  if (!field_stages(dim, hidden, depth, num_freq))
    return fail_invalid("the fused kernel does not take this network's shape");
  if (!w_bf16 || !packed) return fail_invalid("null pointer");
  if (reinterpret_cast<uintptr_t>(packed) % 16) return fail_invalid("packed must be 16-byte aligned");
  PackArgs p{};
  p.hid = hidden;
  p.depth = depth;
  p.feats = 2 * num_freq;
  for (int l = 0; l <= depth; ++l)
    p.w[l] = static_cast<const __nv_bfloat16 *>(w_bf16) + layer_offset(l, hidden, p.feats);
  return launch_pack(p, packed, stream);
}

int ftle_mlp_field(int32_t dim, int32_t hidden, int32_t depth, int32_t num_freq,
                   const double *points, int64_t n, const void *packed, const float *w,
                   const float *freq, double out_scale, double T, double *ftle,
                   int32_t *error_word, void *stream) {
  if (n < 0) return fail_invalid("n must be >= 0");
  if (n == 0) return FTLE_OK;
  if (!points || !packed || !w || !freq || !ftle || !error_word) return fail_invalid("null pointer");
  if (T == 0.0) return fail_invalid("T must be non-zero");
  if (!field_stages(dim, hidden, depth, num_freq))
    return fail_invalid("the fused kernel does not take this network's shape");
  FieldArgs a{};
  a.points = points;
  a.ld = dim + 1;
  a.n = n;
  a.hid = hidden;
  a.depth = depth;
  a.freqs = num_freq;
  a.wpack = static_cast<const unsigned char *>(packed);
  for (int l = 0; l <= depth; ++l)
    a.bias[l] = w + layer_offset(l, hidden, 2 * num_freq) +
                (int64_t)(l < depth ? hidden : 64) * (l == 0 ? 2 * num_freq : hidden);
  a.freq = reinterpret_cast<const float4 *>(freq);
  a.out_scale = out_scale;
  a.inv_T = 1.0 / fabs(T);
  a.ftle = ftle;
  a.err = error_word;
  return run_field(a, dim, stream);
}

}  // extern "C"
