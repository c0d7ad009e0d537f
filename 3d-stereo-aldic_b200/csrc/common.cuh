// Shared device helpers for the ALDIC B200 kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define ALDIC_NAN __longlong_as_double(0x7ff8000000000000LL)

namespace aldic {

// ---------------------------------------------------------------------------------
// Local 4x4 B-spline stencil of ba_interp2_spline.cpp:235-331 in separable form.
// The reference evaluates A = BC*Q*BC^T and sum a_ij tr^i tc^j; since the stencil is the
// outer product of one cubic basis per axis, the same value is
//   sum_r w_r(tr) * sum_c w_c(tc) * Q[r][c]
// with w(t) = [(-33t + 57t^2 - 24t^3), (56 - 3t - 117t^2 + 64t^3),
//              (45t + 75t^2 - 64t^3),  (-9t - 15t^2 + 24t^3)] / 56,
// the rows of BC = B*C (B the cubic B-spline basis, C the truncated prefilter inverse
// [71 -19 5 -1; ...]/56).  The weights sum to 1 and w(0) = [0 1 0 0].
// ---------------------------------------------------------------------------------
__device__ __forceinline__ void bspline_weights(float t, float w[4]) {
  const float k = 1.0f / 56.0f;
  w[0] = k * (t * fmaf(t, fmaf(t, -24.0f, 57.0f), -33.0f));
  w[1] = k * fmaf(t, fmaf(t, fmaf(t, 64.0f, -117.0f), -3.0f), 56.0f);
  w[2] = k * (t * fmaf(t, fmaf(t, -64.0f, 75.0f), 45.0f));
  w[3] = k * (t * fmaf(t, fmaf(t, 24.0f, -15.0f), -9.0f));
}

// Interpolate the column-major M-row image `img` with tap 0 at 0-based (r0, c0), all 16
// taps in bounds, fractions tr (dim 1) and tc (dim 2).
__device__ __forceinline__ float stencil16(const float* __restrict__ img, int M, int r0, int c0, float tr, float tc) {
  float wr[4], wc[4];
  bspline_weights(tr, wr);
  bspline_weights(tc, wc);
  const float* p = img + (size_t)r0 + (size_t)c0 * M;
  float acc = 0.f;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float* q = p + (size_t)c * M;
    float col = wr[0] * __ldg(q);
    col = fmaf(wr[1], __ldg(q + 1), col);
    col = fmaf(wr[2], __ldg(q + 2), col);
    col = fmaf(wr[3], __ldg(q + 3), col);
    acc = fmaf(wc[c], col, acc);
  }
  return acc;
}

// The same stencil in FP64 arranged as the reference's double path computes it
// (ba_interp2_spline.cpp:235-331): per row i of the integer matrix K = 56 BC (up to sign and
// scale), T_ij = K_j . (K_i . Q), and the value sum_ij s_ij T_ij tr^i tc^j, where each
// scale s_ij is a float-literal constant of the reference rounded to float before it is
// promoted (3/56, 1/7, 9/3136, 3/392, 1/49; ba_interp2_spline.cpp:310-325).  It tracks the
// reference MEX to ~1e-13 and serves the FP64 re-solve of subsets whose FP32 convergence
// decision was too close to call.  All 16 taps in bounds.
__device__ __forceinline__ double stencil16_ref64(const float* __restrict__ img, int M, int r0, int c0, double tr,
                                                  double tc) {
  // The scales depend on (i, j) only through the classes {0}, {1, 2}, {3} of each index, so the
  // four powers of tr are combined once per class of j (R0, R1, R3) and column.
  const double s356 = (double)(3.0f / 56.0f), s17 = (double)(1.0f / 7.0f);
  const double s9 = (double)((1.0f / 3136.0f) * 9.0f), s3392 = (double)(3.0f / 392.0f);
  const double s149 = (double)(1.0f / 49.0f);
  const float* p = img + (size_t)r0 + (size_t)c0 * M;
  const double tr2 = tr * tr, tr3 = tr2 * tr, tc2 = tc * tc, tc3 = tc2 * tc;
  double R0 = 0.0, R1[4], R3[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const double q0 = __ldg(p + (size_t)c * M), q1 = __ldg(p + (size_t)c * M + 1);
    const double q2 = __ldg(p + (size_t)c * M + 2), q3 = __ldg(p + (size_t)c * M + 3);
    const double k1 = ((11 * q0 + q1) + -15 * q2) + 3 * q3, k2 = ((19 * q0 + -39 * q1) + 25 * q2) + -5 * q3;
    const double k3 = ((-3 * q0 + 8 * q1) + -8 * q2) + 3 * q3;
    const double e12 = fma(k2, tr2, -(k1 * tr)), e3 = k3 * tr3;
    if (c == 1) R0 = fma(s17, e3, fma(s356, e12, q1));
    R1[c] = fma(s3392, e3, fma(s9, e12, s356 * q1));
    R3[c] = fma(s149, e3, fma(s3392, e12, s17 * q1));
  }
  const double j1 = ((11 * R1[0] + R1[1]) + -15 * R1[2]) + 3 * R1[3];
  const double j2 = ((19 * R1[0] + -39 * R1[1]) + 25 * R1[2]) + -5 * R1[3];
  const double j3 = ((-3 * R3[0] + 8 * R3[1]) + -8 * R3[2]) + 3 * R3[3];
  return fma(j3, tc3, fma(j2, tc2, fma(-j1, tc, R0)));
}

// Clamped version for arbitrary points (the MEX clamps taps to the image edge,
// ba_interp2_spline.cpp:60-66).
__device__ __forceinline__ float stencil16_clamped(const float* __restrict__ img, int M, int N, int r0, int c0, float tr,
                                                   float tc) {
  float wr[4], wc[4];
  bspline_weights(tr, wr);
  bspline_weights(tc, wc);
  float acc = 0.f;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int cc = min(max(c0 + c, 0), N - 1);
    float col = 0.f;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int rr = min(max(r0 + r, 0), M - 1);
      col = fmaf(wr[r], __ldg(img + (size_t)rr + (size_t)cc * M), col);
    }
    acc = fmaf(wc[c], col, acc);
  }
  return acc;
}

// ---------------------------------------------------------------------------------
// Packed FP32 pairs (sm_100 .f32x2 instructions): one instruction, two lanes of IEEE
// round-to-nearest results, each identical to the scalar operation.
// ---------------------------------------------------------------------------------
// The host forms (same IEEE results lane by lane) serve host-side checks of the
// functions built on them.
__host__ __device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
#ifndef __CUDA_ARCH__
  return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
#else
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
#endif
}

__host__ __device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
#ifndef __CUDA_ARCH__
  return make_float2(a.x * b.x, a.y * b.y);
#else
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
#endif
}

__host__ __device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
#ifndef __CUDA_ARCH__
  return make_float2(a.x + b.x, a.y + b.y);
#else
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
#endif
}

__host__ __device__ __forceinline__ float2 fsub2(float2 a, float2 b) {
#ifndef __CUDA_ARCH__
  return make_float2(a.x - b.x, a.y - b.y);
#else
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "sub.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
#endif
}

// ---------------------------------------------------------------------------------
// Reductions
// ---------------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum of one double per thread over the block, returned to every thread (fixed order: warp
// shuffles, then the warp totals in warp order).  red holds blockDim.x / 32 doubles; the
// leading barrier lets the same red serve call after call.
__device__ __forceinline__ double block_sum_all(double v, double* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double s = 0.0;
  for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += red[k];
  return s;
}

// Block-wide sums of K doubles per thread; result in out[0..K) (shared), visible to all
// threads after return.  scratch must hold (NT/32)*K doubles.
template <int K, int NT>
__device__ __forceinline__ void block_sum(double (&v)[K], double* scratch, double* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double s = warp_sum(v[k]);
    if (lane == 0) scratch[warp * K + k] = s;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double s = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) s += scratch[w * K + threadIdx.x];
    out[threadIdx.x] = s;
  }
  __syncthreads();
}

// Block-wide sums for a runtime number of warps (scratch holds nwarps*K doubles).
template <int K>
__device__ __forceinline__ void block_sum_dyn(double (&v)[K], double* scratch, double* out, int nwarps) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double s = warp_sum(v[k]);
    if (lane == 0) scratch[warp * K + k] = s;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double s = 0;
    for (int w = 0; w < nwarps; ++w) s += scratch[w * K + threadIdx.x];
    out[threadIdx.x] = s;
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------------
// Bit columns: a mask of up to 128 rows as two 64-bit words per column (word 2 c + r / 64, bit
// r % 64).  The flood fills of the solvers run on them: one warp, lanes = columns; a fill along a
// column is six doubling steps on the words, a fill across columns five doubling steps of warp
// shuffles, alternated until nothing changes (a few rounds for the regions met, where a sweep
// over pixels needs as many rounds as the region is wide).
// ---------------------------------------------------------------------------------
__device__ __forceinline__ bool bit_at(const uint64_t* m, int r, int c) { return (m[2 * c + (r >> 6)] >> (r & 63)) & 1; }

// m = on(r, c) over rows x cols (rows <= 128); all nt threads of the block call it.
template <class On>
__device__ __forceinline__ void build_bits(uint64_t* m, int rows, int cols, int nt, On on) {
  const int lane = threadIdx.x & 31;
  for (int c = threadIdx.x >> 5; c < cols; c += nt >> 5) {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int r = 32 * k + lane;
      w[k] = 32 * k < rows ? __ballot_sync(0xffffffffu, r < rows && on(r, c)) : 0u;
    }
    if (lane < 2) m[2 * c + lane] = lane ? (uint64_t)w[3] << 32 | w[2] : (uint64_t)w[1] << 32 | w[0];
  }
}

// Whether every bit of rows x cols is set (uniform over the block).
__device__ __forceinline__ bool bits_full(const uint64_t* m, int rows, int cols) {
  int full = 1;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    const uint64_t lo = rows >= 64 ? ~0ull : (1ull << rows) - 1;
    const uint64_t hi = rows <= 64 ? 0ull : rows >= 128 ? ~0ull : (1ull << (rows - 64)) - 1;
    full &= m[2 * c] == lo && m[2 * c + 1] == hi;
  }
  return __syncthreads_and(full);
}

// Both words of a column filled along it from the set bits of r through the bits of on.
__device__ __forceinline__ void fill_column(uint64_t (&r)[2], const uint64_t (&on)[2]) {
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      uint64_t u = r[k], p = on[k], d = u, q = p;
#pragma unroll
      for (int s = 1; s < 64; s <<= 1) {
        u |= p & (u << s);
        p &= p << s;
        d |= q & (d >> s);
        q &= q >> s;
      }
      r[k] = u | d;
    }
    if (pass == 0) {  // across the word boundary, then once more within the words
      const uint64_t up = (r[0] >> 63) & on[1], dn = (r[1] << 63) & on[0];
      if (!((up & ~r[1]) | (dn & ~r[0]))) return;
      r[1] |= up;
      r[0] |= dn;
    }
  }
}

// bwselect: the connected component of the set bits of on (rows x cols, rows <= 128, cols <= 128)
// that contains the 0-based seed (sr, sc), 4- or 8-connected, into lab.  All threads of the
// block call it; a barrier before (on written) is the caller's, the one after is here.
__device__ inline void flood_bits(const uint64_t* on, uint64_t* lab, int rows, int cols, int sr, int sc, int conn) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const bool seed_ok = sr >= 0 && sr < rows && sc >= 0 && sc < cols && bit_at(on, sr, sc);
    const int groups = (cols + 31) / 32;  // columns 32 j + lane
    for (int c = lane; c < cols; c += 32) {
      lab[2 * c] = seed_ok && c == sc && sr < 64 ? 1ull << sr : 0ull;
      lab[2 * c + 1] = seed_ok && c == sc && sr >= 64 ? 1ull << (sr - 64) : 0ull;
    }
    __syncwarp();
    // every productive round sets at least one bit, so rows cols rounds bound the loop
    for (int round = 0; seed_ok && round < rows * cols; ++round) {
      uint64_t changed = 0;
      for (int j = 0; j < groups; ++j) {
        const int c = 32 * j + lane;
        const bool in = c < cols;
        uint64_t o[2] = {in ? on[2 * c] : 0ull, in ? on[2 * c + 1] : 0ull};
        uint64_t r[2] = {in ? lab[2 * c] : 0ull, in ? lab[2 * c + 1] : 0ull};
        const uint64_t r0 = r[0], r1 = r[1];
        // from the neighbouring columns (8-connected: their rows one up and down as well)
#pragma unroll
        for (int k = -1; k <= 1; k += 2) {
          const int cn = c + k;
          if (in && cn >= 0 && cn < cols) {
            uint64_t a0 = lab[2 * cn], a1 = lab[2 * cn + 1];
            if (conn == 8) {
              const uint64_t b0 = a0 | a0 << 1 | a0 >> 1 | a1 << 63, b1 = a1 | a1 << 1 | a1 >> 1 | a0 >> 63;
              a0 = b0;
              a1 = b1;
            }
            r[0] |= a0 & o[0];
            r[1] |= a1 & o[1];
          }
        }
        fill_column(r, o);
        // along the rows through the 32 columns of the group
        uint64_t p[2] = {o[0], o[1]}, q[2] = {o[0], o[1]}, d[2] = {r[0], r[1]};
#pragma unroll
        for (int s = 1; s < 32; s <<= 1)
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            if (k == 1 && rows <= 64) continue;
            const uint64_t ru = __shfl_up_sync(0xffffffffu, r[k], s), pu = __shfl_up_sync(0xffffffffu, p[k], s);
            const uint64_t rd = __shfl_down_sync(0xffffffffu, d[k], s), pd = __shfl_down_sync(0xffffffffu, q[k], s);
            r[k] |= lane >= s ? p[k] & ru : 0ull;
            p[k] &= lane >= s ? pu : 0ull;
            d[k] |= lane + s < 32 ? q[k] & rd : 0ull;
            q[k] &= lane + s < 32 ? pd : 0ull;
          }
        r[0] |= d[0];
        r[1] |= d[1];
        changed |= (r[0] ^ r0) | (r[1] ^ r1);
        __syncwarp();
        if (in) {
          lab[2 * c] = r[0];
          lab[2 * c + 1] = r[1];
        }
        __syncwarp();
      }
      if (!__any_sync(0xffffffffu, changed != 0)) break;
    }
  }
  __syncthreads();
}

// MATLAB round(): half away from zero.
__device__ __forceinline__ double mround(double x) { return round(x); }

// Inverse-compositional update P <- P o dP^-1 (func/funICGN.m:289-307).  Returns false
// when det(dP) == 0.
__device__ __forceinline__ bool compose_inverse(double P[6], const double d[6]) {
  const double det = (1 + d[0]) * (1 + d[3]) - d[1] * d[2];
  if (!(det != 0)) return false;
  const double t1 = (-d[0] - d[0] * d[3] + d[1] * d[2]) / det;
  const double t2 = -d[1] / det;
  const double t3 = -d[2] / det;
  const double t4 = (-d[3] - d[0] * d[3] + d[1] * d[2]) / det;
  const double t5 = (-d[4] - d[3] * d[4] + d[2] * d[5]) / det;
  const double t6 = (-d[5] - d[0] * d[5] + d[1] * d[4]) / det;
  const double a00 = 1 + P[0], a01 = P[2], a02 = P[4];
  const double a10 = P[1], a11 = 1 + P[3], a12 = P[5];
  const double n00 = a00 * (1 + t1) + a01 * t2;
  const double n10 = a10 * (1 + t1) + a11 * t2;
  const double n01 = a00 * t3 + a01 * (1 + t4);
  const double n11 = a10 * t3 + a11 * (1 + t4);
  const double n02 = a00 * t5 + a01 * t6 + a02;
  const double n12 = a10 * t5 + a11 * t6 + a12;
  P[0] = n00 - 1;
  P[1] = n10;
  P[2] = n01;
  P[3] = n11 - 1;
  P[4] = n02;
  P[5] = n12;
  return true;
}

// compose_inverse with one reciprocal of the determinant instead of six divisions (the FP64
// results differ in their last bits).
__device__ __forceinline__ bool compose_inverse_rcp(double P[6], const double d[6]) {
  const double det = (1 + d[0]) * (1 + d[3]) - d[1] * d[2];
  if (!(det != 0)) return false;
  const double id = 1.0 / det;
  const double t1 = (-d[0] - d[0] * d[3] + d[1] * d[2]) * id;
  const double t2 = -d[1] * id;
  const double t3 = -d[2] * id;
  const double t4 = (-d[3] - d[0] * d[3] + d[1] * d[2]) * id;
  const double t5 = (-d[4] - d[3] * d[4] + d[2] * d[5]) * id;
  const double t6 = (-d[5] - d[0] * d[5] + d[1] * d[4]) * id;
  const double a00 = 1 + P[0], a01 = P[2], a02 = P[4];
  const double a10 = P[1], a11 = 1 + P[3], a12 = P[5];
  P[0] = a00 * (1 + t1) + a01 * t2 - 1;
  P[1] = a10 * (1 + t1) + a11 * t2;
  P[2] = a00 * t3 + a01 * (1 + t4);
  P[3] = a10 * t3 + a11 * (1 + t4) - 1;
  P[4] = a00 * t5 + a01 * t6 + a02;
  P[5] = a10 * t5 + a11 * t6 + a12;
  return true;
}

// x = A^-1 b for an n x n (n <= 6) column-major system, Gaussian elimination with
// partial pivoting in FP64 (mldivide's general path; a zero pivot yields Inf/NaN).
__device__ inline void solve_small(int n, const double* Ain, const double* bin, double* x) {
  double A[36], b[6];
  for (int i = 0; i < n * n; ++i) A[i] = Ain[i];
  for (int i = 0; i < n; ++i) b[i] = bin[i];
  for (int k = 0; k < n; ++k) {
    int piv = k;
    double best = fabs(A[k + k * n]);
    for (int i = k + 1; i < n; ++i)
      if (fabs(A[i + k * n]) > best) {
        best = fabs(A[i + k * n]);
        piv = i;
      }
    if (piv != k) {
      for (int j = 0; j < n; ++j) {
        const double t = A[k + j * n];
        A[k + j * n] = A[piv + j * n];
        A[piv + j * n] = t;
      }
      const double t = b[k];
      b[k] = b[piv];
      b[piv] = t;
    }
    for (int i = k + 1; i < n; ++i) {
      const double l = A[i + k * n] / A[k + k * n];
      for (int j = k; j < n; ++j) A[i + j * n] -= l * A[k + j * n];
      b[i] -= l * b[k];
    }
  }
  for (int i = n - 1; i >= 0; --i) {
    double s = b[i];
    for (int j = i + 1; j < n; ++j) s -= A[i + j * n] * x[j];
    x[i] = s / A[i + i * n];
  }
}

}  // namespace aldic
