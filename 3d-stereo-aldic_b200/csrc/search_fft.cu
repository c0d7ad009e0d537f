// Whole-field integer search, the correlation of a subset as a product of spectra: the
// numerators of all shifts of a subset (func/funIntegerSearch.m:100-203, normxcorr2) are
//     C = IFFT(conj(FFT(T)) FFT(D)),
// T the centred template and D the zero-padded cut-out window, in a 2-D real transform of
// L x L >= (na + w - 1)^2 held in the shared memory of one CTA.  The shifts at both ends wrap
// onto rows and columns of D that are zero, so the ring of partial windows needs no table.
//
// An FP32 transform is off by a few ulp of |T| |D| at every shift, where a sum over the window
// off by that of |T| |D in the window|.  So the maximum found here counts only where no
// other shift comes within the error bound of both (kFftErr); the remaining subsets, and those
// with values that are not finite, go to a list that the direct kernel works through.
//
// Work per subset and why it is taken: a direct sum costs na nb (w+1)^2 products (34 M at
// radius 70 and window 41), the shared products of a tile 187 na nb = 3.8 M, the transforms about
// 2.4 M operations.  40 000 subsets of that shape: 15.5 ms with the tile kernel, 8.2 ms so; 2088 of
// window 33 at radius 20 705 us with the direct kernel, 255 us so (whole searches).  Bound by issue
// slots (46 % used) and the latencies between the passes' barriers: one CTA of 12 warps fills an
// SM's shared memory at L = 192.
#include "search_common.cuh"
#include "search_fft.cuh"

#include <algorithm>
#include <type_traits>

namespace aldic {

namespace {

// Bound of a numerator's error over |T| |D|, in units of u = 2^-24, from the roundings of the passes
// (first order; Higham, Accuracy and Stability of Numerical Algorithms, chapter 24).  A layer of complex
// additions adds u in the 2-norm, a product with a rounded root 3 u (2 u by FMAs, Jeannerod et al. 2017,
// and the root's own), a radix-3 step 5 u, a radix-5 step 8 u.  So one dimension of 16 B values costs
// F = 7 + 3 + b with b = 5 (B = 3), 2, 8, 9, 6, 13, 12, 10 (B = 12), and
//   D, two rows a transform:                  2 F + 1
//   T, rows:                                  F + 1
//      columns, n = W1 / B rows summed:       (8 + n / 4) sqrt(n) <= 48, then 3 + b
//   the product:                              2
//   the inverse, whose every output is at most the sum of |spectrum| / L^2 <= |T| |D| times the
//   roundings on a path; two rows share one:  F + 2 (F + 1)
//   T to FP32, 1 / (|T| L^2), 1 / sqrt:       7
// An error of a spectrum in the 2-norm reaches a numerator at most times the other factor's norm
// (Cauchy-Schwarz).  The sums are 136 (L = 64) to 192 (L = 144); 256 covers them with the second order.
// Measured errors are far smaller (up to 3.4 u on plane waves and ramps); the bound is what makes the
// choice of the maximum certain, and costs nothing on speckles, whose peaks stand clear of it.
constexpr float kFftErr = 256.f * 5.9604645e-8f;

// cos and sin of 2 pi k / 720: the roots of every radix below.
struct Roots {
  float c[720], s[720];
};
constexpr double taylor(double x, bool cosine) {  // |x| <= pi / 4
  double t = cosine ? 1.0 : x, r = t;
  for (int i = cosine ? 1 : 2; i < 30; i += 2) {
    t *= -x * x / (double)(i * (i + 1));
    r += t;
  }
  return r;
}
constexpr Roots make_roots() {
  Roots r{};
  for (int k = 0; k < 720; ++k) {
    // quadrant q and offset in [-pi/4, pi/4]
    const int q = (k + 90) / 180;
    const double x = (k - 180 * q) * (6.283185307179586476925 / 720.0);
    const double c = taylor(x, true), s = taylor(x, false);
    const double cc = q % 4 == 0 ? c : q % 4 == 1 ? -s : q % 4 == 2 ? -c : s;
    const double ss = q % 4 == 0 ? s : q % 4 == 1 ? c : q % 4 == 2 ? -s : -c;
    r.c[k] = (float)cc;
    r.s[k] = (float)ss;
  }
  return r;
}
constexpr Roots kRoots = make_roots();

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return fadd2(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return fsub2(a, b); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {  // a conj(b)
  return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
}
template <bool INV>
__device__ __forceinline__ float2 twiddle(float2 a, float2 t) {
  return INV ? cmulc(a, t) : cmul(a, t);
}
// a exp(-2 pi i K / N) (its conjugate with INV), the root as immediate operands
template <bool INV, int N, int K0>
__device__ __forceinline__ float2 root(float2 a) {
  constexpr int K = K0 % N;
  if constexpr (K == 0) {
    return a;
  } else if constexpr (2 * K == N) {
    return make_float2(-a.x, -a.y);
  } else if constexpr (4 * K == N) {
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
  } else if constexpr (4 * K == 3 * N) {
    return INV ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
  } else {
    constexpr float c = kRoots.c[K * (720 / N)], s = INV ? kRoots.s[K * (720 / N)] : -kRoots.s[K * (720 / N)];
    return make_float2(fmaf(a.x, c, -s * a.y), fmaf(a.x, s, c * a.y));
  }
}

template <int I, int E, class F>
__device__ __forceinline__ void unrolled(F&& f) {
  if constexpr (I < E) {
    f(std::integral_constant<int, I>{});
    unrolled<I + 1, E>(f);
  }
}

// In-place DFT of N values in registers, natural order in and out.
template <int N, bool INV>
__device__ __forceinline__ void dft(float2 (&v)[N]) {
  if constexpr (N == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (N == 3) {
    const float h = INV ? 0.86602540378443865f : -0.86602540378443865f;
    const float2 s = cadd(v[1], v[2]), d = csub(v[1], v[2]);
    const float2 m = make_float2(fmaf(-0.5f, s.x, v[0].x), fmaf(-0.5f, s.y, v[0].y));
    v[0] = cadd(v[0], s);
    v[1] = make_float2(fmaf(-h, d.y, m.x), fmaf(h, d.x, m.y));
    v[2] = make_float2(fmaf(h, d.y, m.x), fmaf(-h, d.x, m.y));
  } else if constexpr (N == 4) {
    const float2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = csub(v[1], v[3]);
    const float2 e = INV ? make_float2(-d.y, d.x) : make_float2(d.y, -d.x);
    v[0] = cadd(a, c);
    v[1] = cadd(b, e);
    v[2] = csub(a, c);
    v[3] = csub(b, e);
  } else if constexpr (N == 5) {
    const float c1 = 0.30901699437494742f, c2 = -0.80901699437494742f;
    const float s1 = INV ? 0.95105651629515357f : -0.95105651629515357f;
    const float s2 = INV ? 0.58778525229247313f : -0.58778525229247313f;
    const float2 p1 = cadd(v[1], v[4]), m1 = csub(v[1], v[4]), p2 = cadd(v[2], v[3]), m2 = csub(v[2], v[3]);
    const float2 a = make_float2(fmaf(c1, p1.x, fmaf(c2, p2.x, v[0].x)), fmaf(c1, p1.y, fmaf(c2, p2.y, v[0].y)));
    const float2 b = make_float2(fmaf(c2, p1.x, fmaf(c1, p2.x, v[0].x)), fmaf(c2, p1.y, fmaf(c1, p2.y, v[0].y)));
    const float2 c = make_float2(fmaf(s1, m1.x, s2 * m2.x), fmaf(s1, m1.y, s2 * m2.y));
    const float2 d = make_float2(fmaf(s2, m1.x, -s1 * m2.x), fmaf(s2, m1.y, -s1 * m2.y));
    v[0] = cadd(v[0], cadd(p1, p2));
    v[1] = make_float2(a.x - c.y, a.y + c.x);
    v[4] = make_float2(a.x + c.y, a.y - c.x);
    v[2] = make_float2(b.x - d.y, b.y + d.x);
    v[3] = make_float2(b.x + d.y, b.y - d.x);
  } else {
    constexpr int N1 = N % 4 == 0 ? 4 : N % 3 == 0 ? 3 : 2, N2 = N / N1;
    float2 y[N1][N2];
    unrolled<0, N2>([&](auto n2) {
      float2 c[N1];
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1) c[n1] = v[N2 * n1 + n2];
      dft<N1, INV>(c);
      unrolled<0, N1>([&](auto k1) { y[k1][n2] = root<INV, N, decltype(n2)::value * decltype(k1)::value>(c[k1]); });
    });
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
      dft<N2, INV>(y[k1]);
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) v[k1 + N1 * k2] = y[k1][k2];
    }
  }
}

// A transform of L = 16 B values: 16-point DFTs of the elements a B + b (a = 0 .. 15), twiddled,
// then B-point DFTs over b give the elements k1 + 16 k2.
template <int L>
struct FftShape {
  static constexpr int B = L / 16, NU = L / 2 + 1;
  // threads and CTAs an SM: measured over both for every size (40 000 subsets at L = 192: 512 threads
  // of 128 registers 9.48, 480 8.98, 384 of 168 8.18 ms; L = 80: 256 threads twice 1.13, 192 three
  // times 0.99 ms)
  static constexpr int NT = L >= 160 ? 384 : L == 144 ? 320 : L >= 96 ? 256 : L == 80 ? 192 : L == 64 ? 160 : 128;
  static constexpr int MINB = L >= 160 ? 1 : L >= 96 ? 2 : L == 80 ? 3 : L == 64 ? 4 : 6;
  static_assert(L % 16 == 0 && L <= 192, "16 B with B <= 12");
};

constexpr int kCand = 32;  // shifts whose order may be decided in FP64 before a subset goes to the list
// FP64 values no further apart count as equal, and the first shift wins: the integral images' rounding
// (45 ulp of the prefix sum of g^2) moves a value by 1e-11 on 2048 x 2048.
constexpr double kSame = 1e-10;

// Value of one shift in FP64, by a warp (in every lane).
__device__ __noinline__ double shift_value(const SearchArgs& a, SubsetGeom s, int aa, int bb, SubsetPrm P) {
  const int W1 = a.winsize + 1, lane = threadIdx.x & 31;
  const int i0 = max(0, 1 - aa), i1 = min(W1, s.dr1 - s.dr0 + 2 - aa);  // the window's rows and columns inside D
  const int j0 = max(0, 1 - bb), j1 = min(W1, s.dc1 - s.dc0 + 2 - bb);
  const float* f = a.f + (s.ii - 1 + i0) + (size_t)(s.jj - 1 + j0) * a.M;
  const float* g = a.g + (s.dr0 - 1 + aa + i0) + (size_t)(s.dc0 - 1 + bb + j0) * a.M;
  const int R = i1 - i0, n = R * (j1 - j0), di = 32 % R, step = di + 32 / R * a.M;
  int i = lane % R, k = i + lane / R * a.M;
  double num = 0.0;
#pragma unroll 8  // loads in flight
  for (int p = lane; p < n; p += 32) {
    num += ((double)__ldg(f + k) - P.fm) * (double)__ldg(g + k);
    i += di;
    k += step;
    if (i >= R) {
      i -= R;
      k += a.M - R;
    }
  }
  return ncc_at(a, s, aa, bb, warp_sum(num), P.denT, P.tolz);
}

}  // namespace

// Two rows of a real image share one complex transform, whose intermediate of L values lies in the
// place of the two half spectra (2 NU values) that it becomes, rotated by b + p / 8 so that the
// writes of 16 pairs p and the reads of 16 k1 both fall into different banks.
template <int L>
__device__ __forceinline__ void rows_first(float2 (&v)[16], float2* o, int p, int b, const float2* tw) {
  dft<16, false>(v);
  const int r = b + (p >> 3);
  o += b * 16;
  o[r & 15] = v[0];
#pragma unroll
  for (int k = 1; k < 16; ++k) o[(k + r) & 15] = cmul(v[k], tw[b * k]);
}

// The B-point part at k1 and 16 - k1 (k1 = 0 .. 8) of every pair, and both rows' half spectra (times
// 2).  Every thread of the block calls it; the pairs lie one after the other from S on.
template <int L, int NT>
__device__ __forceinline__ void rows_second(float2* S, int npairs) {
  constexpr int B = L / 16, NU = L / 2 + 1;
#pragma unroll 1
  for (int p0 = 0; p0 < npairs; p0 += NT / 9) {
    const int p = p0 + threadIdx.x / 9, k1 = threadIdx.x % 9;
    const bool on = threadIdx.x < NT / 9 * 9 && p < npairs;
    float2 X[B], Y[B];
    float2* const o = S + p * 2 * NU;
    if (on) {
#pragma unroll
      for (int b = 0; b < B; ++b) {
        X[b] = o[b * 16 + ((k1 + b + (p >> 3)) & 15)];
        Y[b] = o[b * 16 + ((16 - k1 + b + (p >> 3)) & 15)];
      }
      dft<B, false>(X);
      dft<B, false>(Y);
      if (k1 == 0) {  // the partner of 16 k2 is 16 (B - k2)
#pragma unroll
        for (int k = 0; k < B; ++k) Y[k] = X[(k + 1) % B];
      }
    }
    __syncthreads();
    if (on) {
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) {
        const int k = k1 + 16 * k2;
        const bool low = 2 * k <= L;
        const float2 z = low ? X[k2] : Y[B - 1 - k2], y = low ? Y[B - 1 - k2] : X[k2];
        const int u = low ? k : L - k;
        o[u] = make_float2(z.x + y.x, z.y - y.y);
        o[NU + u] = make_float2(z.y + y.y, y.x - z.x);
      }
    }
  }
}

template <int L>
__device__ __forceinline__ void fill_twiddles(float2* tw, int nt) {  // exp(-2 pi i k / L)
  for (int k = threadIdx.x; k < L; k += nt) {
    double sn, cs;
    sincospi(2.0 * k / L, &sn, &cs);
    tw[k] = make_float2((float)cs, (float)-sn);
  }
}

// Half spectra over the columns of every row of g, for each grid column jb + blockIdx.y (its cut-out
// columns, zero elsewhere): rows[(column, image row)][NU].  A row serves every subset of its grid
// column that it is cut out for (18 of them at radius 70 and step 10).
constexpr int kRowPairs = 32, kRowThreads = 288;  // 9 threads a pair in the second part
template <int L>
__global__ void __launch_bounds__(kRowThreads) fft_rows_kernel(SearchArgs a, int jb, float2* __restrict__ rows) {
  constexpr int B = L / 16, NU = L / 2 + 1;
  extern __shared__ __align__(16) float2 S[];
  float2* const tw = S + 2 * kRowPairs * NU;
  fill_twiddles<L>(tw, kRowThreads);
  const AxisGeom g = axis_geom(a.gy0 + (jb + (int)blockIdx.y) * a.step, a.winsize, a.s0, a.s1, a.N, a.gy1);
  if (!g.ok) return;
  __syncthreads();
  const int x0 = blockIdx.x * 2 * kRowPairs;
#pragma unroll 1
  for (int it = threadIdx.x; it < kRowPairs * B; it += kRowThreads) {
    const int p = it % kRowPairs, b = it / kRowPairs, x = x0 + 2 * p;
    float2 v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int c = g.d0 - 1 + b + k * B;
      const bool okc = c >= g.d0 && c <= g.d1;
      const float* q = a.g + (long long)c * a.M + x;
      v[k].x = okc && x < a.M ? __ldg(q) : 0.f;
      v[k].y = okc && x + 1 < a.M ? __ldg(q + 1) : 0.f;
    }
    rows_first<L>(v, S + p * 2 * NU, p, b, tw);
  }
  __syncthreads();
  rows_second<L, kRowThreads>(S, kRowPairs);
  __syncthreads();
  const int nr = min(2 * kRowPairs, a.M - x0);
  float2* const out = rows + ((long long)blockIdx.y * a.M + x0) * NU;
  for (int k = threadIdx.x; k < nr * NU; k += kRowThreads) out[k] = S[k];
}

// One CTA per subset of the grid columns jb .. jb + nj - 1.  S holds the rows x of D and, after
// them, those of T as half spectra over the columns (NU values a row; lanes run along a row, so the
// accesses of the column passes are conflict-free).
template <int L>
__global__ void __launch_bounds__(FftShape<L>::NT, FftShape<L>::MINB)
    ncc_fft_kernel(const __grid_constant__ SearchArgs a, int jb, int nj, const float2* __restrict__ rows, const float* __restrict__ map,
                   const SubsetPrm* __restrict__ prm, const float2* __restrict__ ringv, int* __restrict__ best,
                   int* __restrict__ flist, int* __restrict__ fcount) {
  using Sh = FftShape<L>;
  constexpr int B = Sh::B, NU = Sh::NU, NT = Sh::NT;
  extern __shared__ __align__(16) float2 S[];
  __shared__ float s_lo[NT / 32];
  __shared__ double s_val[kCand];
  __shared__ int s_ncand, s_cand[kCand];
  const int tid = threadIdx.x, lane = tid & 31;
  const int W1 = a.winsize + 1, NPT = (W1 + 1) / 2, nda = a.s0 + a.s1 + 3;
  float2* const FT = S + L * NU;         // rows of T
  float2* const tw = FT + 2 * NPT * NU;  // exp(-2 pi i k / L)
  const long long n = (long long)a.nx * (jb + nj);
  const int NW = a.N - W1 + 1;
  fill_twiddles<L>(tw, NT);
  __syncthreads();
  for (long long t = (long long)a.nx * jb + blockIdx.x; t < n; t += gridDim.x) {
    const SubsetPrm P = prm[t];
    if (!P.valid) continue;
    const SubsetGeom s = subset_geom(a, t);
    // ---- columns of D, 16-point part, and rows of T ----
    const float2* const rb = rows + ((long long)(t / a.nx - jb) * a.M + s.dr0 - 1) * NU;
    const int xlast = s.dr1 - s.dr0 + 1;
    const float fmh = (float)P.fm, fml = (float)(P.fm - (double)fmh);
#pragma unroll 1
    for (int it0 = tid; it0 < (NU + NPT) * B; it0 += NT) {
      float2 v[16];
      if (it0 >= NU * B) {  // rows of T
        const int it = it0 - NU * B, p = it % NPT, b = it / NPT;
        const float* fp = a.f + (s.ii - 1 + 2 * p) + (long long)(s.jj - 1 + b) * a.M;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const bool okc = b + k * B < W1;
          v[k].x = okc ? (__ldg(fp + (long long)k * B * a.M) - fmh) - fml : 0.f;
          v[k].y = okc && 2 * p + 1 < W1 ? (__ldg(fp + (long long)k * B * a.M + 1) - fmh) - fml : 0.f;
        }
        rows_first<L>(v, FT + p * 2 * NU, p, b, tw);
        continue;
      }
      const int u = it0 % NU, b = it0 / NU;
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const int x = k * B + b;
        v[k] = x >= 1 && x <= xlast ? __ldg(rb + x * NU + u) : make_float2(0.f, 0.f);
      }
      dft<16, false>(v);
      float2* const c = S + b * NU + u;
      c[0] = v[0];
#pragma unroll
      for (int k = 1; k < 16; ++k) c[k * B * NU] = cmul(v[k], tw[b * k]);
    }
    __syncthreads();
    rows_second<L, NT>(FT, NPT);
    __syncthreads();
    // ---- columns: T at k1 = q and q + 8 (its few rows summed directly), the rest of D's
    // transform, the product and the B-point part of the inverse ----
#pragma unroll 1
    for (int it = tid; it < NU * 8; it += NT) {
      const int u = it % NU, q = it / NU;
      // sums over a = 4 g .. 4 g + 3 of T's rows a B + b, g apart by W_16^(4 q g)
      float2 F1[B], F2[B];
      const float2 w1 = tw[q * B], w2 = tw[2 * q * B % L], w3 = tw[3 * q * B % L];
      const auto group = [&](int i, float2& e, float2& o) {
        const float2* const r = FT + i * NU + u;
        float2 f[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) f[k] = i + k * B < W1 ? r[k * B * NU] : make_float2(0.f, 0.f);
        e = cadd(f[0], cmul(f[2], w2));
        o = cadd(cmul(f[1], w1), cmul(f[3], w3));
      };
#pragma unroll
      for (int b = 0; b < B; ++b) {
        float2 e, o;
        group(b, e, o);
        F1[b] = cadd(e, o);
        F2[b] = csub(e, o);
        if (b % 3 == 2) asm volatile("" ::: "memory");  // bounds the loads in flight, and with them the registers
      }
#pragma unroll 1
      for (int g = 1; 4 * g * B < W1; ++g) {
        const float2 wg = tw[4 * q * g * B % L];
#pragma unroll
        for (int b = 0; b < B; ++b) {
          float2 e, o;
          group(4 * g * B + b, e, o);
          F1[b] = cadd(F1[b], cmul(cadd(e, o), wg));
          F2[b] = cadd(F2[b], cmul(csub(e, o), wg));
          if (b % 3 == 2) asm volatile("" ::: "memory");
        }
      }
#pragma unroll
      for (int b = 0; b < B; ++b) {
        F1[b] = cmul(F1[b], tw[b * q]);
        F2[b] = cmul(F2[b], tw[b * (q + 8)]);
      }
      dft<B, false>(F1);
      dft<B, false>(F2);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float2* const c = S + (q + 8 * h) * B * NU + u;
        float2 G[B];
#pragma unroll
        for (int b = 0; b < B; ++b) G[b] = c[b * NU];
        dft<B, false>(G);
#pragma unroll
        for (int b = 0; b < B; ++b) G[b] = cmulc(G[b], h ? F2[b] : F1[b]);
        dft<B, true>(G);
#pragma unroll
        for (int b = 0; b < B; ++b) c[b * NU] = G[b];
      }
    }
    __syncthreads();
    // ---- columns, 16-point part of the inverse ----
#pragma unroll 1
    for (int it = tid; it < NU * B; it += NT) {
      const int u = it % NU, b = it / NU;
      float2* const c = S + b * NU + u;
      float2 v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = k == 0 ? c[0] : cmulc(c[k * B * NU], tw[b * k]);
      dft<16, true>(v);
#pragma unroll
      for (int k = 0; k < 16; ++k)
        if (k * B + b <= s.na) c[k * B * NU] = v[k];
    }
    __syncthreads();
    // ---- rows of the crop, two at a time ----
    const int NPO = (s.na + 1) / 2;
#pragma unroll 1
    for (int p0 = 0; p0 < NPO; p0 += NT / B) {
      const int p = p0 + tid / B, b = tid % B;
      const bool on = tid < NT / B * B && p < NPO;
      float2* const o = S + p * 2 * NU;
      float2 v[16];
      if (on) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const int f = k * B + b;
          const bool low = 2 * f <= L;
          const int u = low ? f : L - f;
          const float2 c0 = o[u], c1 = o[NU + u];
          v[k] = low ? make_float2(c0.x - c1.y, c0.y + c1.x) : make_float2(c0.x + c1.y, c1.x - c0.y);
        }
        dft<16, true>(v);
      }
      __syncthreads();
      if (on) {
#pragma unroll
        for (int k = 0; k < 16; ++k) o[b * 16 + ((k + b + (p >> 3)) & 15)] = k == 0 ? v[k] : cmulc(v[k], tw[b * k]);
      }
    }
    __syncthreads();
    // ---- the last part, the normalised values and the running maximum ----
    const float inv = (float)(1.0 / P.denT) * (0.25f / ((float)L * (float)L));
    const float err = kFftErr * P.gnorm;
    const float2* const rv = ringv + t * 4 * nda;
    // largest lower bound of this thread's shifts, its item with the largest upper bound, and the
    // largest upper bound of its other items
    float lo = -INFINITY, hi = -INFINITY, hi2 = -INFINITY;
    int ihi = 0;
#pragma unroll 1
    for (int it = tid; it < NPO * 16; it += NT) {
      const int n1 = it & 15, p = it >> 4;
      // 1 / sqrt of the variance sums of both rows' shifts (NaN outside the crop, which no maximum
      // takes; 0 for a flat window), fetched ahead of the transform.  Where the sum is near the
      // zero threshold the bounds lie so far apart that the shift is a candidate.
      float rs[2][B];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int aa = 2 * p + h;
        const bool ra = aa == 0 || aa == s.na - 1;
        const float2* const rrow = rv + (aa == 0 ? 0 : nda);
        const float* const mrow = map + (long long)(s.ii - 2 - s.L + aa) * NW + (s.jj - 2 - s.U);
#pragma unroll
        for (int k = 0; k < B; ++k) {
          const int bb = n1 + 16 * k;
          rs[h][k] = NAN;
          if (aa < s.na && bb < s.nb) {
            const bool rb = bb == 0 || bb == s.nb - 1;
            rs[h][k] = __ldg(ra ? &rrow[bb].y : rb ? &rv[(bb == 0 ? 2 : 3) * nda + aa].y : mrow + bb);
          }
        }
      }
      float2 v[B];
      float2* const o = S + p * 2 * NU;
#pragma unroll
      for (int b = 0; b < B; ++b) v[b] = o[b * 16 + ((n1 + b + (p >> 3)) & 15)];
      dft<B, true>(v);
      float ih = -INFINITY;
#pragma unroll
      for (int k = 0; k < B; ++k) {
        const float c0 = v[k].x * inv * rs[0][k], c1 = v[k].y * inv * rs[1][k];
        const float2 h = make_float2(fmaf(err, rs[0][k], c0), fmaf(err, rs[1][k], c1));
        lo = fmaxf(lo, fmaxf(fmaf(-err, rs[0][k], c0), fmaf(-err, rs[1][k], c1)));
        ih = fmaxf(ih, fmaxf(h.x, h.y));
        o[k * 16 + ((n1 + k + (p >> 3)) & 15)] = h;
      }
      hi2 = fmaxf(hi2, fminf(hi, ih));
      if (ih > hi) ihi = it;
      hi = fmaxf(hi, ih);
    }
    float m = lo;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    if (lane == 0) s_lo[tid >> 5] = m;
    if (tid == 0) s_ncand = 0;
    __syncthreads();
    m = s_lo[0];
#pragma unroll
    for (int k = 1; k < NT / 32; ++k) m = fmaxf(m, s_lo[k]);
    // ---- the shifts that may be the maximum: mostly one ----
    if (hi >= m && m > -INFINITY) {
#pragma unroll 1
      for (int it = hi2 >= m ? tid : ihi; it < NPO * 16; it += NT) {
        const int n1 = it & 15, p = it >> 4;
        float2 h[B];
#pragma unroll
        for (int k = 0; k < B; ++k) h[k] = S[p * 2 * NU + k * 16 + ((n1 + k + (p >> 3)) & 15)];
#pragma unroll
        for (int k = 0; k < B; ++k) {
          if (!(fmaxf(h[k].x, h[k].y) >= m)) continue;
          const int lin = 2 * p + (n1 + 16 * k) * s.na, c = atomicAdd(&s_ncand, (h[k].x >= m) + (h[k].y >= m));
          if (c < kCand) s_cand[c] = lin + (h[k].x >= m ? 0 : 1);
          if (h[k].x >= m && h[k].y >= m && c + 1 < kCand) s_cand[c + 1] = lin + 1;
        }
        if (hi2 < m) break;
      }
    }
    __syncthreads();
    const int nc = s_ncand;
    if (nc > 1 && nc <= kCand) {  // close ones: their values in FP64, a warp each
      for (int c = tid >> 5; c < nc; c += NT / 32) {
        const int lin = s_cand[c];
        const double v = shift_value(a, s, lin % s.na, lin / s.na, P);
        if (lane == 0) s_val[c] = v;
      }
      __syncthreads();
    }
    if (tid == 0) {
      int w = 0;
      if (nc > 1 && nc <= kCand) {
        double top = s_val[0];
        for (int c = 1; c < nc; ++c) top = fmax(top, s_val[c]);
        w = -1;
        for (int c = 0; c < nc; ++c)
          if (s_val[c] >= top - kSame && (w < 0 || s_cand[c] < s_cand[w])) w = c;
      }
      // above 1: a variance sum that is all cancellation
      const bool sure = P.gnorm < 1e15f && P.denT < 1e15 && m < 1.00001f && nc > 0 && nc <= kCand && w >= 0;
      best[t] = sure ? s_cand[w] : -1;
      if (!sure) flist[atomicAdd(fcount, 1)] = (int)t;
    }
  }
}

namespace {

constexpr int kFftL[] = {48, 64, 80, 96, 128, 144, 160, 192};

constexpr size_t kRowBytes = 64 << 20;  // of row spectra at a time: they stay in L2 between their two kernels

size_t fft_smem(int L, int W1) { return ((size_t)(L + (W1 + 1) / 2 * 2) * (L / 2 + 1) + L) * sizeof(float2); }
size_t row_bytes(int L, int M) { return (size_t)M * (L / 2 + 1) * sizeof(float2); }
int row_columns(int L, int M, int ny) {  // grid columns at a time
  const size_t c = kRowBytes / row_bytes(L, M);
  return (int)std::max<size_t>(1, std::min<size_t>(c, (size_t)ny));
}

template <int L>
int launch_fft(const SearchArgs& a, const SearchTables& t, cudaStream_t st) {
  const size_t smem = fft_smem(L, a.winsize + 1);
  constexpr size_t rsmem = ((size_t)2 * kRowPairs * (L / 2 + 1) + L) * sizeof(float2);
  auto kern = ncc_fft_kernel<L>;
  int dev = 0, sms = 148, per = 1;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaFuncSetAttribute(fft_rows_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rsmem) != cudaSuccess ||
      cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, FftShape<L>::NT, smem) != cudaSuccess || per < 1)
    return -1;
  const int cols = row_columns(L, a.M, a.ny), nbatch = (a.ny + cols - 1) / cols, step = (a.ny + nbatch - 1) / nbatch;
  int launches = 0;
  for (int jb = 0; jb < a.ny; jb += step) {
    const int nj = std::min(step, a.ny - jb);
    fft_rows_kernel<L><<<dim3((a.M + 2 * kRowPairs - 1) / (2 * kRowPairs), nj), kRowThreads, rsmem, st>>>(a, jb, (float2*)t.rows);
    const unsigned grid = (unsigned)std::min<long long>((long long)a.nx * nj, (long long)sms * per);
    kern<<<grid, FftShape<L>::NT, smem, st>>>(a, jb, nj, (const float2*)t.rows, t.map, t.prm, t.ringv,
                                                 t.best, t.flist, a.left);
    launches += 2;
  }
  return launches;
}

}  // namespace

// Transform size of a search, 0 where none fits.
static int transform_size(int winsize, int s0, int s1) {
  const int need = s0 + s1 + 3 + winsize - 1;
  for (int L : kFftL)
    if (L >= need) return fft_smem(L, winsize + 1) <= 225 * 1024 ? L : 0;
  return 0;
}

// The transform size that a call of implementation 0 takes, 0 for the other kernels.  The transforms' time goes with
// n L^2, the tiles' with the waves of tiles and their products and shifts, the direct kernel's with
// its shifts and template rounded up to its blocks; the factors (us) are fits to the measured times
// of the three over windows of 21 to 49, steps of 8 to 32 and radii of 4 to 70, 55 us being what
// the tables of the transforms' way cost at least (direct / transforms: 100 subsets at window 41 and
// radius 5 97 / 108 us, 2088 at window 33 and radius 20 705 / 255 us; tile / transforms: 9604 at
// window 41, step 10 and radius 20 682 / 802 us, radius 35 1576 / 1106 us).
static int transform_for(const SearchArgs& a) {
  const int W1 = a.winsize + 1, nda = a.s0 + a.s1 + 3;
  const int L = transform_size(a.winsize, a.s0, a.s1);
  if (a.impl != 0 || a.list || !L || a.M < W1 || a.N < W1 || !search_direct_available(a.winsize))
    return 0;
  const double n = (double)a.nx * a.ny, fft = n * L * L * 5.5e-6, tile = search_tile_us(a);
  if (tile >= 0) return fft < tile ? L : 0;
  const double direct = n * (0.015 + (double)((nda + 31) / 32 * 32) * round_up16(nda) * W1 * round_up8(W1) * 8e-8);
  return 55 + fft < direct ? L : 0;
}

static size_t transform_bytes(const SearchArgs& a, int L) {
  return search_tables_bytes(a, row_bytes(L, a.M) * row_columns(L, a.M, a.ny));
}

size_t search_choose(SearchArgs& a) {
  a.fft = transform_for(a);
  if (a.fft) return transform_bytes(a, a.fft);
  return a.list || a.impl == 2 ? 0 : search_tile_bytes(a);
}

int launch_search_fft(const SearchArgs& a, cudaStream_t st) {
  const int L = a.fft;
  if (!L || !a.scratch || transform_bytes(a, L) > a.scratch_bytes) return -1;
  SearchTables t;
  const int launches = launch_search_tables(a, row_bytes(L, a.M) * row_columns(L, a.M, a.ny), &t, st);
  if (cudaMemsetAsync(a.left, 0, sizeof(int), st) != cudaSuccess) return -1;
  if (a.ev_start) cudaEventRecord(a.ev_start, st);
  int l = -1;
  switch (L) {
    case 48: l = launch_fft<48>(a, t, st); break;
    case 64: l = launch_fft<64>(a, t, st); break;
    case 80: l = launch_fft<80>(a, t, st); break;
    case 96: l = launch_fft<96>(a, t, st); break;
    case 128: l = launch_fft<128>(a, t, st); break;
    case 144: l = launch_fft<144>(a, t, st); break;
    case 160: l = launch_fft<160>(a, t, st); break;
    case 192: l = launch_fft<192>(a, t, st); break;
  }
  if (l < 0) return -1;
  SearchArgs d = a;  // the subsets left to direct sums
  d.ev_start = d.ev_stop = nullptr;
  d.dlist = t.flist;
  d.dcount = a.left;
  const int ld = launch_search_direct(d, st);
  if (ld < 0) return -1;
  if (a.ev_stop) cudaEventRecord(a.ev_stop, st);
  launch_search_refit(a, t, st);
  return launches + l + ld + 1;
}

}  // namespace aldic
