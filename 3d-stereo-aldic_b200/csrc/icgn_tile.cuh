// The 6-DOF solve of nominal-window subsets without a mask region.  Included by icgn.cu after its
// shared helpers.
//
// A group of NW warps solves one subset without a block barrier.  Lane l of the group takes the
// window's pixels l, l + 32 NW, ... (column-major order) in packed FP32 pairs with Kahan
// compensation; the lanes' sums are added in FP64 and every thread runs the same FP64
// Gauss-Newton control.
//
// Read through L1, the 16 taps of a pixel bound the kernel: a warp's 32 pixels wrap over two
// window columns, so each gather touches three cache lines (L1 two thirds busy at half the issue
// rate).  Here the window's footprint is copied once per subset into shared memory, by
// asynchronous copies that overlap the set-up sums, and each tap is one shared-memory wavefront:
// the column pitch is W1 plus a multiple of 32 floats, so 32 consecutive window pixels lie in 32
// different banks wherever the wrap falls.  The buffers of a CTA's two groups share each
// column (rows of group 0, then of group 1), which fills the pitch.
#pragma once

namespace aldic {

constexpr int kTileGroups = 2;  // subset groups per CTA

struct TileGeom {
  int rows, cols;  // of a group's buffer (deformed-image pixels); 0: the taps are read from the image
  int pitch;       // floats between columns, both groups' rows within
};

// Packed FP32 pairs kept in one 64-bit register.
typedef unsigned long long f32x2_t;
__device__ __forceinline__ f32x2_t pk(float x, float y) {
  f32x2_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ void upk(f32x2_t v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ f32x2_t pfma(f32x2_t a, f32x2_t b, f32x2_t c) {
  f32x2_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2_t pmul(f32x2_t a, f32x2_t b) {
  f32x2_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2_t padd(f32x2_t a, f32x2_t b) {
  f32x2_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2_t psub(f32x2_t a, f32x2_t b) {
  f32x2_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// Kahan-compensated accumulation (Kahan 1965), the compensation kept with the opposite sign:
// the running total is s + k.  The caller forms y = x + k, fused into the term's own
// operation (y = fma(a, b, k) for a product term), then
//   t = s + y;  k = (s - t) + y;  s = t
// (each operation rounded on its own, never contracted or reassociated).  The error of the total is
// bounded by ~2 ulp of sum |x|, independent of the number of terms.
__device__ __forceinline__ void pkahan(f32x2_t& s, f32x2_t& k, f32x2_t y) {
  const f32x2_t t = padd(s, y);
  k = padd(psub(s, t), y);
  s = t;
}
// bspline_weights of common.cuh for a pair of points
__device__ __forceinline__ void pweights(f32x2_t t, f32x2_t w[4]) {
  const f32x2_t k = pk(1.0f / 56.0f, 1.0f / 56.0f);
  w[0] = pmul(k, pmul(t, pfma(t, pfma(t, pk(-24.0f, -24.0f), pk(57.0f, 57.0f)), pk(-33.0f, -33.0f))));
  w[1] = pmul(k, pfma(t, pfma(t, pfma(t, pk(64.0f, 64.0f), pk(-117.0f, -117.0f)), pk(-3.0f, -3.0f)), pk(56.0f, 56.0f)));
  w[2] = pmul(k, pmul(t, pfma(t, pfma(t, pk(-64.0f, -64.0f), pk(75.0f, 75.0f)), pk(45.0f, 45.0f))));
  w[3] = pmul(k, pmul(t, pfma(t, pfma(t, pk(24.0f, 24.0f), pk(-15.0f, -15.0f)), pk(-9.0f, -9.0f))));
}
extern __shared__ __align__(16) float s_tile[];

// Tap source: the image, or the CTA's shared-memory buffer (byte offsets).
template <bool SMEM>
struct Taps {
  using Ptr = typename std::conditional<SMEM, uint32_t, const float*>::type;
  static __device__ __forceinline__ float ld(uint32_t a) {
    return *reinterpret_cast<const float*>(reinterpret_cast<const char*>(s_tile) + a);
  }
  static __device__ __forceinline__ float ld(const float* a) { return __ldg(a); }
  static __device__ __forceinline__ uint32_t at(uint32_t a, int e) { return a + 4u * (uint32_t)e; }
  static __device__ __forceinline__ const float* at(const float* a, int e) { return a + e; }
};
// stencil16 of common.cuh at two tap-0 positions
template <bool SMEM>
__device__ __forceinline__ f32x2_t pstencil(typename Taps<SMEM>::Ptr qa, typename Taps<SMEM>::Ptr qb, int pitch,
                                            f32x2_t tr, f32x2_t tc) {
  using T = Taps<SMEM>;
  f32x2_t wr[4], wc[4];
  pweights(tr, wr);
  pweights(tc, wc);
  // taps by scalar FMAs on the weights' halves: pairing the loaded taps costs more moves than the
  // packed form saves issue slots
  float ra[4], rb[4], ca[4], cb[4], aa = 0.f, ab = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    upk(wr[k], ra[k], rb[k]);
    upk(wc[k], ca[k], cb[k]);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float va = ra[0] * T::ld(qa), vb = rb[0] * T::ld(qb);
#pragma unroll
    for (int r = 1; r < 4; ++r) {
      va = fmaf(ra[r], T::ld(T::at(qa, r)), va);
      vb = fmaf(rb[r], T::ld(T::at(qb, r)), vb);
    }
    aa = fmaf(ca[c], va, aa);
    ab = fmaf(cb[c], vb, ab);
    qa = T::at(qa, pitch);
    qb = T::at(qb, pitch);
  }
  return pk(aa, ab);
}
// stencil16 of common.cuh
template <bool SMEM>
__device__ __forceinline__ float stencil_at(typename Taps<SMEM>::Ptr q, int pitch, float tr, float tc) {
  using T = Taps<SMEM>;
  float wr[4], wc[4];
  bspline_weights(tr, wr);
  bspline_weights(tc, wc);
  float acc = 0.f;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float col = wr[0] * T::ld(q);
#pragma unroll
    for (int r = 1; r < 4; ++r) col = fmaf(wr[r], T::ld(T::at(q, r)), col);
    acc = fmaf(wc[c], col, acc);
    q = T::at(q, pitch);
  }
  return acc;
}

// floor() of a packed pair of window coordinates (|l| < 2^22) by one round-down addition:
// t = floor(l) + 1.5 2^23 exactly, so t's bits less kFloorBits are the integer and t - 1.5 2^23
// is the float.
constexpr float kFloorMagic = 12582912.0f;
constexpr uint32_t kFloorBits = 0x4B400000u;
__device__ __forceinline__ f32x2_t pfloor_magic(f32x2_t l, f32x2_t magic) {
  f32x2_t d;
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(d) : "l"(l), "l"(magic));
  return d;
}

// Sums of 32 doubles per lane over the warp: returns, in lane l, the sum of v[l] (halving
// exchanges: 31 shuffled doubles instead of 160).
__device__ __forceinline__ double warp_sum_transposed32(double (&v)[32], int lane) {
#pragma unroll
  for (int h = 16; h > 0; h >>= 1) {
    const bool up = lane & h;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double keep = up ? v[i + h] : v[i], send = up ? v[i] : v[i + h];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
    }
  }
  return v[0];
}

// Sums of 8 doubles per lane over the warp, left in every lane.
__device__ __forceinline__ void warp_sum8(double (&v)[8], int lane) {
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const int h = 4 >> s, m = 16 >> s;
    const bool up = lane & m;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double keep = up ? v[i + h] : v[i], send = up ? v[i] : v[i + h];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
    }
  }
  double t = v[0];
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  t += __shfl_xor_sync(0xffffffffu, t, 1);
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __shfl_sync(0xffffffffu, t, i * 4);
}

// Copy rows [r0, r0 + rows) x columns [c0, c0 + cols) of the deformed image into the group's
// buffer by 4-byte asynchronous copies (no alignment rule); entries outside the image become 0
// (no tap of an accepted warp reads them).  Every thread of the group calls it, and tile_wait()
// before the buffer is read.
template <int NW>
__device__ __forceinline__ void tile_issue(const FrameDev& fr, uint32_t tile, const TileGeom& geo, int r0, int c0,
                                           int gt) {
  constexpr int GT = 32 * NW;
  const int qb = GT / geo.rows, rb = GT % geo.rows;
  int r = gt % geo.rows, c = gt / geo.rows;
  const uint32_t base = smem_u32(s_tile) + tile;
  while (c < geo.cols) {
    const int ir = r0 + r, ic = c0 + c;
    const bool in = (unsigned)ir < (unsigned)fr.M && (unsigned)ic < (unsigned)fr.N;
    const float* src = fr.def + (in ? (size_t)ir + (size_t)ic * fr.M : 0);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(base + 4u * (uint32_t)(r + c * geo.pitch)),
                 "l"(src), "r"(in ? 4 : 0)
                 : "memory");
    r += rb;
    c += qb;
    if (r >= geo.rows) {
      r -= geo.rows;
      c += 1;
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int NW>
__device__ __forceinline__ void tile_wait(int bar) {
  asm volatile("cp.async.wait_all;" ::: "memory");
  group_bar<NW>(bar);
}

// warped_oob: the extremes of the affine warp over the window are at its corners, where the
// products have their absolute values; the roundings are those of the corners.
__device__ __forceinline__ bool window_oob(const FrameDev& fr, const double P[6], double x0, double y0, double h) {
  const double cu = x0 + P[4], cv = y0 + P[5];
  const double eu = fma(fabs(1 + P[0]), h, fabs(P[2]) * h), ev = fma(fabs(P[1]), h, fabs(1 + P[3]) * h);
  return !(cu - eu >= 3 && cu + eu <= fr.M - 2 && cv - ev >= 3 && cv + ev <= fr.N - 2);
}

// The FP32 warp coefficients of an iteration and the image row / column of tap 0 of the window
// centre (prep_coeffs).
struct WarpF {
  float p0, p1, p2, p3, f5, f6;
  int br, bc;
};
__device__ __forceinline__ WarpF warp_coeffs(const double P[6], double x0, double y0) {
  const double n5 = mround(P[4]), n6 = mround(P[5]);
  return WarpF{(float)P[0],        (float)P[1],        (float)P[2],         (float)P[3],
               (float)(P[4] - n5), (float)(P[5] - n6), (int)(x0 + n5) - 2, (int)(y0 + n6) - 2};
}

// Image rows and columns that the window's taps can touch (0-based, one of margin each side).
__device__ __forceinline__ void tile_footprint(const WarpF& w, int half, int& rlo, int& rhi, int& clo, int& chi) {
  const float h = (float)half;
  const float ex = fmaf(fabsf(1.f + w.p0), h, fabsf(w.p2) * h), ey = fmaf(fabsf(1.f + w.p3), h, fabsf(w.p1) * h);
  rlo = w.br + (int)floorf(w.f5 - ex) - 1;
  rhi = w.br + (int)floorf(w.f5 + ex) + 4;
  clo = w.bc + (int)floorf(w.f6 - ey) - 1;
  chi = w.bc + (int)floorf(w.f6 + ey) + 4;
}

// The per-lane sums of one iteration: c[0..5] sum J g, c[6] sum g, c[7] sum g^2 (selected pixels),
// fg sum f g; n selected pixels and nz exact zeros (QUAD; uniform windows count all).
struct PixelSums {
  double c[8], fg;
  int n, nz;
};

// SMEM: taps from the group's buffer at byte offset tile (its first image row tr0, column tc0),
// else from the image.
template <int GT, bool QUAD, bool FG, bool SMEM>
__device__ __forceinline__ void pixel_sums(const FrameDev& fr, const WarpF& w, uint32_t tile, int tpitch, int tr0,
                                           int tc0, int r0, int c0, int crop, int W1, int gt, PixelSums& out) {
  const int half = W1 / 2, npx = W1 * W1, gM = fr.M - 6;
  f32x2_t C[6], K[6], S = 0, KS = 0, S2 = 0, KS2 = 0, fg = 0;
#pragma unroll
  for (int k = 0; k < 6; ++k) C[k] = K[k] = 0;
  const f32x2_t pp0 = pk(w.p0, w.p0), pp1 = pk(w.p1, w.p1), pp2 = pk(w.p2, w.p2), pp3 = pk(w.p3, w.p3);
  const f32x2_t ff5 = pk(w.f5, w.f5), ff6 = pk(w.f6, w.f6), magic = pk(kFloorMagic, kFloorMagic);
  int n = 0, nz = 0;
  // the pair's window offsets, stepped as floats with the wrap at the window's last row
  int aa = gt % W1, bb = gt / W1;
  int ab = aa + GT % W1, bbb = bb + GT / W1;
  if (ab >= W1) {
    ab -= W1;
    bbb += 1;
  }
  float dxa = (float)(aa - half), dxb = (float)(ab - half), dya = (float)(bb - half), dyb = (float)(bbb - half);
  const float fhalf = (float)half, fW1 = (float)W1, sx = (float)((2 * GT) % W1), sy = (float)((2 * GT) / W1);
  const int kstep = (2 * GT) % W1 + (2 * GT) / W1 * gM, kwrap = gM - W1;
  const int fstep = (2 * GT) % W1 + (2 * GT) / W1 * fr.M, fwrap = fr.M - W1;
  int ka = (r0 + aa - crop) + (c0 + bb - crop) * gM, kb = (r0 + ab - crop) + (c0 + bbb - crop) * gM;
  int fa = (r0 + aa) + (c0 + bb) * fr.M, fb = (r0 + ab) + (c0 + bbb) * fr.M;
  // tap 0's element from the bits of the two round-down sums
  const int pitch = SMEM ? tpitch : fr.M;
  const int base = SMEM ? (w.br - tr0) + (w.bc - tc0) * pitch : w.br + w.bc * pitch;
  using T = Taps<SMEM>;
  typename T::Ptr img;
  if constexpr (SMEM)
    img = tile;
  else
    img = fr.def;
  const uint32_t upitch = (uint32_t)pitch, ibase = (uint32_t)base - kFloorBits - kFloorBits * upitch;
  int p = gt;
  float gxa = 0.f, gxb = 0.f, gya = 0.f, gyb = 0.f;
  if (p + GT < npx) {
    gxa = __ldg(fr.gx + ka);
    gxb = __ldg(fr.gx + kb);
    gya = __ldg(fr.gy + ka);
    gyb = __ldg(fr.gy + kb);
  }
#pragma unroll 1
  for (; p + GT < npx; p += 2 * GT) {
    const f32x2_t dx = pk(dxa, dxb), dy = pk(dya, dyb), gx = pk(gxa, gxb), gy = pk(gya, gyb);
    f32x2_t f = 0;
    if (FG) f = pk(__ldg(fr.ref + fa), __ldg(fr.ref + fb));
    const f32x2_t lx = padd(dx, pfma(pp0, dx, pfma(pp2, dy, ff5)));
    const f32x2_t ly = padd(dy, pfma(pp3, dy, pfma(pp1, dx, ff6)));
    const f32x2_t mx = pfloor_magic(lx, magic), my = pfloor_magic(ly, magic);
    float mxa, mxb, mya, myb;
    upk(mx, mxa, mxb);
    upk(my, mya, myb);
    const int ia = (int)(__float_as_uint(mxa) + __float_as_uint(mya) * upitch + ibase);
    const int ib = (int)(__float_as_uint(mxb) + __float_as_uint(myb) * upitch + ibase);
    // the next pair, its gradients in flight while this one is summed
    dxa += sx;
    dxb += sx;
    dya += sy;
    dyb += sy;
    ka += kstep;
    kb += kstep;
    if (FG) {
      fa += fstep;
      fb += fstep;
    }
    if (dxa > fhalf) {
      dxa -= fW1;
      dya += 1.f;
      ka += kwrap;
      if (FG) fa += fwrap;
    }
    if (dxb > fhalf) {
      dxb -= fW1;
      dyb += 1.f;
      kb += kwrap;
      if (FG) fb += fwrap;
    }
    if (p + 3 * GT < npx) {
      gxa = __ldg(fr.gx + ka);
      gxb = __ldg(fr.gx + kb);
      gya = __ldg(fr.gy + ka);
      gyb = __ldg(fr.gy + kb);
    }
    const f32x2_t g = pstencil<SMEM>(T::at(img, ia), T::at(img, ib), pitch, psub(lx, psub(mx, magic)), psub(ly, psub(my, magic)));
    const f32x2_t ag = pmul(gx, g), bg = pmul(gy, g);
    pkahan(C[0], K[0], pfma(ag, dx, K[0]));
    pkahan(C[1], K[1], pfma(bg, dx, K[1]));
    pkahan(C[2], K[2], pfma(ag, dy, K[2]));
    pkahan(C[3], K[3], pfma(bg, dy, K[3]));
    pkahan(C[4], K[4], padd(ag, K[4]));
    pkahan(C[5], K[5], padd(bg, K[5]));
    if (!QUAD) {
      pkahan(S, KS, padd(g, KS));
      pkahan(S2, KS2, pfma(g, g, KS2));
    } else {
      // S holds (sum g, sum g^2) of the selected pixels, one pixel after the other
      float ga, gb;
      upk(g, ga, gb);
      if (fabsf(ga) > 1e-10f && fabsf(gb) > 1e-10f) {
        pkahan(S, KS, pfma(pk(ga, ga), pk(1.f, ga), KS));
        pkahan(S, KS, pfma(pk(gb, gb), pk(1.f, gb), KS));
        n += 2;
      } else {
        if (fabsf(ga) > 1e-10f) {
          pkahan(S, KS, pfma(pk(ga, ga), pk(1.f, ga), KS));
          n += 1;
        }
        if (fabsf(gb) > 1e-10f) {
          pkahan(S, KS, pfma(pk(gb, gb), pk(1.f, gb), KS));
          n += 1;
        }
        nz += (ga == 0.f) + (gb == 0.f);
      }
    }
    if (FG) fg = pfma(f, g, fg);
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    float cx, cy, kx, ky;
    upk(C[k], cx, cy);
    upk(K[k], kx, ky);
    out.c[k] = ((double)cx + (double)kx) + ((double)cy + (double)ky);
  }
  {
    float sx_, sy_, kx, ky;
    upk(S, sx_, sy_);
    upk(KS, kx, ky);
    if (QUAD) {
      out.c[6] = (double)sx_ + (double)kx;
      out.c[7] = (double)sy_ + (double)ky;
    } else {
      float tx, ty, ux, uy;
      upk(S2, tx, ty);
      upk(KS2, ux, uy);
      out.c[6] = ((double)sx_ + (double)kx) + ((double)sy_ + (double)ky);
      out.c[7] = ((double)tx + (double)ux) + ((double)ty + (double)uy);
    }
    float x, y;
    upk(fg, x, y);
    out.fg = (double)x + (double)y;
  }
  if (p < npx) {  // the last, unpaired pixel
    const float lx = dxa + fmaf(w.p0, dxa, fmaf(w.p2, dya, w.f5));
    const float ly = dya + fmaf(w.p3, dya, fmaf(w.p1, dxa, w.f6));
    const float ix = floorf(lx), iy = floorf(ly);
    const float g = stencil_at<SMEM>(T::at(img, base + (int)ix + (int)iy * pitch), pitch, lx - ix, ly - iy);
    const float ag = __ldg(fr.gx + ka) * g, bg = __ldg(fr.gy + ka) * g;
    out.c[0] += (double)(ag * dxa);
    out.c[1] += (double)(bg * dxa);
    out.c[2] += (double)(ag * dya);
    out.c[3] += (double)(bg * dya);
    out.c[4] += (double)ag;
    out.c[5] += (double)bg;
    if (!QUAD || fabsf(g) > 1e-10f) {
      out.c[6] += (double)g;
      out.c[7] += (double)g * (double)g;
      n += 1;
    }
    if (QUAD && g == 0.f) nz += 1;
    if (FG) out.fg += (double)__ldg(fr.ref + fa) * (double)g;
  }
  out.n = n;
  out.nz = nz;
}

template <int NW, bool SLOW, bool QUAD, bool FG>
__global__ void __launch_bounds__(32 * NW * kTileGroups, 8 / NW) icgn_tile_kernel(IcgnArgs a, TileGeom geo) {
  constexpr int NG = kTileGroups, GT = 32 * NW;
  struct __align__(16) Group {
    double inv[36];    // H^-1, row-major
    double h[22];      // packed upper triangle by rows
    double A[6], B[6];
    double sums[34];   // set-up sums
    double aug[72], fac[6];
    double red[NW == 1 ? 2 : NW * 34];
    int qi;
  };
  __shared__ Group s_group[NG];
  const int lane = threadIdx.x & 31, grp = threadIdx.x / GT, gw = (threadIdx.x % GT) >> 5;
  const int gt = threadIdx.x % GT, bar = 1 + grp;
  Group& s = s_group[grp];
  const uint32_t tile = 4u * (uint32_t)(grp * geo.rows);  // byte offset of the group's buffer
  const FrameDev& fr = a.fr;
  const bool epi = !QUAD && FG && a.variant == 2;
  const int count = a.qcount[SLOW ? 1 : 0];
  const int gM = fr.M - 6;
  int* next = a.qcount + (SLOW ? 3 : 2);
  while (true) {
    // the group's next queue entry (dynamic: slow subsets do not pile up on one group)
    int qi = 0;
    if (gt == 0) qi = atomicAdd(next, 1);
    if (NW == 1) {
      qi = __shfl_sync(0xffffffffu, qi, 0);
    } else {
      if (gt == 0) s.qi = qi;
      group_bar<NW>(bar);
      qi = s.qi;
    }
    if (qi >= count) break;
    int* q = a.queue + 3 * ((SLOW ? a.n : 0) + qi);
    if (SLOW && q[2] != kSlowSubset) {
      group_bar<NW>(bar);
      continue;
    }
    const long long t = q[0];
    const int W1 = q[1] + 1, npx = W1 * W1, half = W1 / 2;
    double x0 = a.coords[t], y0 = a.coords[a.n + t];
    if (QUAD) {
      x0 = mround(x0);
      y0 = mround(y0);
    }
    const int r0 = (int)x0 - half - 1, c0 = (int)y0 - half - 1;
    double P[6] = {0.0, 0.0, 0.0, 0.0, epi ? 0.0 : a.U0[2 * t], epi ? 0.0 : a.U0[2 * t + 1]};
    if (a.F0 && !epi)
      for (int k = 0; k < 4; ++k) P[k] = a.F0[4 * t + k];  // a gradient initial guess (learned)
    double normInit = 0.0;
    int step = 0;
    if (SLOW && a.carry) {  // continue from where the warp pass stopped: P, the first norm, the step
      const double* cs = a.carry + 8 * t;
#pragma unroll
      for (int k = 0; k < 6; ++k) P[k] = cs[k];
      normInit = cs[6];
      step = (int)cs[7];
    }
    // the buffer around the first iteration's footprint, in flight during the set-up sums
    int tr0 = 0, tc0 = 0;
    bool tile_ok = false, pending = false;
    bool oob = window_oob(fr, P, x0, y0, half);
    if (!oob) {
      int rlo, rhi, clo, chi;
      tile_footprint(warp_coeffs(P, x0, y0), half, rlo, rhi, clo, chi);
      if (rhi - rlo < geo.rows && chi - clo < geo.cols) {
        tr0 = rlo - (geo.rows - 1 - (rhi - rlo)) / 2;
        tc0 = clo - (geo.cols - 1 - (chi - clo)) / 2;
        tile_issue<NW>(fr, tile, geo, tr0, tc0, gt);
        pending = true;
      }
    }
    // ---- set-up sums in FP64: with a = f_x^2, b = f_x f_y, c = f_y^2 the 21 entries of H are the
    //      18 sums of a, b, c times {dx dx, dx dy, dy dy, dx, dy, 1}; sum J f, sum J, f statistics
    {
      double v[32], fab = 0.0;
      int n = 0;
#pragma unroll
      for (int k = 0; k < 32; ++k) v[k] = 0.0;
      int aa = gt % W1, bb = gt / W1;
      const int q_nt = GT / W1, r_nt = GT % W1;
      float dxf = (float)(aa - half), dyf = (float)(bb - half);
      const float fhalf = (float)half, fW1 = (float)W1, sx = (float)r_nt, sy = (float)q_nt;
      int k = (r0 + aa) + (c0 + bb) * fr.M, kg = (r0 + aa - a.crop) + (c0 + bb - a.crop) * gM;
      const int kstep = r_nt + q_nt * fr.M, kwrap = fr.M - W1, gstep = r_nt + q_nt * gM, gwrap = gM - W1;
      float ff = 0.f, fx = 0.f, fy = 0.f;
      if (gt < npx) {
        ff = __ldg(fr.ref + k);
        fx = __ldg(fr.gx + kg);
        fy = __ldg(fr.gy + kg);
      }
#pragma unroll 2
      for (int p = gt; p < npx; p += GT) {
        const double f = ff, gx = fx, gy = fy, dx = dxf, dy = dyf;
        const bool sel = !QUAD || fabsf(ff) > 1e-10f;
        dxf += sx;
        dyf += sy;
        k += kstep;
        kg += gstep;
        if (dxf > fhalf) {
          dxf -= fW1;
          dyf += 1.f;
          k += kwrap;
          kg += gwrap;
        }
        if (p + GT < npx) {
          ff = __ldg(fr.ref + k);
          fx = __ldg(fr.gx + kg);
          fy = __ldg(fr.gy + kg);
        }
        const double m[3] = {gx * gx, gx * gy, gy * gy};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double mx = m[i] * dx, my = m[i] * dy;
          v[6 * i] = fma(mx, dx, v[6 * i]);
          v[6 * i + 1] = fma(mx, dy, v[6 * i + 1]);
          v[6 * i + 2] = fma(my, dy, v[6 * i + 2]);
          v[6 * i + 3] += mx;
          v[6 * i + 4] += my;
          v[6 * i + 5] += m[i];
        }
        const double gf = gx * f, hf = gy * f;
        v[18] = fma(gf, dx, v[18]);  // sum J f, in the order of J
        v[19] = fma(hf, dx, v[19]);
        v[20] = fma(gf, dy, v[20]);
        v[21] = fma(hf, dy, v[21]);
        v[22] += gf;
        v[23] += hf;
        v[24] = fma(gx, dx, v[24]);  // sum J
        v[25] = fma(gy, dx, v[25]);
        v[26] = fma(gx, dy, v[26]);
        v[27] = fma(gy, dy, v[27]);
        v[28] += gx;
        v[29] += gy;
        if (sel) {
          v[30] += f;
          v[31] = fma(f, f, v[31]);
          n += 1;
        }
        fab += fabs(f);
      }
      const double mine = warp_sum_transposed32(v, lane);
      fab = warp_sum(fab);
      n = __reduce_add_sync(0xffffffffu, n);
      if (NW == 1) {
        s.sums[lane] = mine;
        if (lane == 0) {
          s.sums[32] = fab;
          s.sums[33] = (double)n;
        }
      } else {
        s.red[gw * 34 + lane] = mine;
        if (lane == 0) {
          s.red[gw * 34 + 32] = fab;
          s.red[gw * 34 + 33] = (double)n;
        }
        group_bar<NW>(bar);
        for (int e = gt; e < 34; e += GT) {
          double t_ = s.red[e];
#pragma unroll
          for (int u = 1; u < NW; ++u) t_ += s.red[u * 34 + e];
          s.sums[e] = t_;
        }
      }
    }
    group_bar<NW>(bar);
    const double nf = s.sums[33], sabsf = s.sums[32];
    double meanf = ALDIC_NAN, bf = ALDIC_NAN;
    if (nf > 0) {
      meanf = s.sums[30] / nf;
      bf = sqrt(fmax(s.sums[31] - s.sums[30] * s.sums[30] / nf, 0.0));
    }
    if (gw == 0) {
      if (lane < 6) {
        s.B[lane] = s.sums[24 + lane];
        s.A[lane] = (s.sums[18 + lane] - meanf * s.sums[24 + lane]) / bf;
      }
      if (lane < 21) {
        // packed entry (i, j) of J = (f_x dx, f_y dx, f_x dy, f_y dy, f_x, f_y): the product's
        // gradient part (0 f_x^2, 1 f_x f_y, 2 f_y^2) and offset part (0 dx dx, 1 dx dy, 2 dy dy,
        // 3 dx, 4 dy, 5 one)
        int i = 0, e = lane;
        while (e >= 6 - i) {
          e -= 6 - i;
          ++i;
        }
        const int j = i + e, part = (i & 1) + (j & 1), oi = i >> 1, oj = j >> 1;  // 0 dx, 1 dy, 2 one
        const int off = oj == 2 ? 3 + oi : oi + oj;
        s.h[lane] = s.sums[6 * part + off];
      }
      __syncwarp();
      invert6_warp(s.h, s.aug, s.fac, s.inv, lane);
    }
    group_bar<NW>(bar);
    // ---- Gauss-Newton iterations (control replicated in every thread) ----
    const double trH = s.h[0] + s.h[6] + s.h[11] + s.h[15] + s.h[18] + s.h[20];
    const double inpx = 1.0 / (double)npx;
    double normNew = 1.0, normAbs = 1.0, znssd = ALDIC_NAN, iInit = 1.0 / normInit;
    int status = 0, requeue = -1;
    while (step <= a.max_iter && normNew > a.tol && normAbs > a.tol) {
      if (!SLOW && step >= a.warp_cap) {
        requeue = (a.slow_fp64 && !epi) ? kToFp64 : kSlowSubset;
        break;
      }
      step += 1;
      if (oob) {
        normNew = 1e6;
        break;
      }
      const WarpF w = warp_coeffs(P, x0, y0);
      int rlo, rhi, clo, chi;
      tile_footprint(w, half, rlo, rhi, clo, chi);
      if (pending) {
        tile_wait<NW>(bar);
        pending = false;
        tile_ok = true;
      }
      if (!(tile_ok && rlo >= tr0 && rhi < tr0 + geo.rows && clo >= tc0 && chi < tc0 + geo.cols)) {
        tile_ok = rhi - rlo < geo.rows && chi - clo < geo.cols;
        if (tile_ok) {  // the warp moved out of the buffer: load the one around it
          group_bar<NW>(bar);
          tr0 = rlo - (geo.rows - 1 - (rhi - rlo)) / 2;
          tc0 = clo - (geo.cols - 1 - (chi - clo)) / 2;
          tile_issue<NW>(fr, tile, geo, tr0, tc0, gt);
          tile_wait<NW>(bar);
        }
      }
      PixelSums ps;
      if (tile_ok)
        pixel_sums<GT, QUAD, FG, true>(fr, w, tile, geo.pitch, tr0, tc0, r0, c0, a.crop, W1, gt, ps);
      else  // a footprint larger than the buffer (a large deformation)
        pixel_sums<GT, QUAD, FG, false>(fr, w, tile, geo.pitch, tr0, tc0, r0, c0, a.crop, W1, gt, ps);
      warp_sum8(ps.c, lane);
      if (FG) ps.fg = warp_sum(ps.fg);
      int n = QUAD ? __reduce_add_sync(0xffffffffu, ps.n) : 0;
      int nz = QUAD ? __any_sync(0xffffffffu, ps.nz) : 0;
      if (NW > 1) {
        if (lane == 0) {
#pragma unroll
          for (int k = 0; k < 8; ++k) s.red[gw * 34 + k] = ps.c[k];
          s.red[gw * 34 + 8] = ps.fg;
          s.red[gw * 34 + 9] = (double)n;
          s.red[gw * 34 + 10] = (double)nz;
        }
        group_bar<NW>(bar);
        double tot[11];
#pragma unroll
        for (int k = 0; k < 11; ++k) {
          tot[k] = s.red[k];
#pragma unroll
          for (int u = 1; u < NW; ++u) tot[k] += s.red[u * 34 + k];
        }
        group_bar<NW>(bar);
#pragma unroll
        for (int k = 0; k < 8; ++k) ps.c[k] = tot[k];
        ps.fg = tot[8];
        n = (int)tot[9];
        nz = tot[10] > 0;
      }
      if (QUAD && nz) {  // exact zero in g: the g-region flood fill is needed
        requeue = 0;
        break;
      }
      if (!QUAD) n = npx;
      // mean and norm of g over the selected pixels
      double meang = ALDIC_NAN, ibg = ALDIC_NAN, in_ = inpx;
      if (n > 0) {
        if (n != npx) in_ = 1.0 / (double)n;
        meang = ps.c[6] * in_;
        ibg = 1.0 / sqrt(fmax(ps.c[7] - ps.c[6] * meang, 0.0));
      }
      if (FG) znssd = 2.0 - 2.0 * (ps.fg - meanf * ps.c[6]) / bf * ibg;
      double b[6], nn = 0.0;
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        b[k] = bf * (s.A[k] - (ps.c[k] - meang * s.B[k]) * ibg);
        nn += b[k] * b[k];
      }
      normAbs = sqrt(nn);
      if (step == 1) {
        normInit = normAbs;
        iInit = 1.0 / normInit;
      }
      normNew = normInit > a.tol ? normAbs * iInit : 0.0;
      if (!epi && a.band > 0) {
        const double sig = step * a.noise * 5.9604644775390625e-08 * (bf * ibg) * sqrt(fmax(trH * ps.c[7] * in_, 0.0));
        const double lim = a.band * a.tol + sig;
        if (!(fabs(normAbs - a.tol) > lim) ||
            (normInit > a.tol && !(fabs(normNew - a.tol) > fma(sig, iInit, a.band * a.tol)))) {
          requeue = kToFp64;  // the FP64 pass re-solves this subset from its initial guess
          break;
        }
      }
      if (!(normNew < a.tol || normAbs < a.tol)) {
        double dP[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          double acc = 0;
#pragma unroll
          for (int j = 0; j < 6; j += 2) {
            const double2 r = *reinterpret_cast<const double2*>(&s.inv[6 * i + j]);
            acc = fma(r.x, b[j], acc);
            acc = fma(r.y, b[j + 1], acc);
          }
          dP[i] = -acc;
        }
        if (!compose_inverse_rcp(P, dP)) {
          step = a.max_iter + 1000;
          status = 1;
        } else if (epi) {
          P[4] = 0.0;
          P[5] = 0.0;
        }
        oob = window_oob(fr, P, x0, y0, half);
      }
    }
    // a copy never waited for must land before the next subset's goes into the buffer
    if (pending) asm volatile("cp.async.wait_all;" ::: "memory");
    if (gt == 0) {
      if (requeue == kToFp64) {
        push_fp64(a, t, W1 - 1, 0);  // unmasked, at the window this pass solved
        if (SLOW) q[2] = kMovedSubset;
      } else if (requeue >= 0) {
        if (requeue == kSlowSubset && a.carry) {
          double* cs = a.carry + 8 * t;
#pragma unroll
          for (int k = 0; k < 6; ++k) cs[k] = P[k];
          cs[6] = normInit;
          cs[7] = (double)step;
        }
        // hand this subset to a later pass (they run after this kernel): a queue-0 subset is
        // appended to queue 1 (at most one entry each), a queue-1 subset is re-flagged in place
        if (SLOW) {
          q[2] = requeue;
        } else {
          const int pos = atomicAdd(&a.qcount[1], 1);
          int* q1 = a.queue + 3 * ((long long)a.n + pos);
          q1[0] = (int)t;
          q1[1] = W1 - 1;
          q1[2] = requeue;
        }
      } else {
        if (status == 1) step -= 1000;
        if (!(normNew < a.tol || normAbs < a.tol)) step = a.max_iter + 1;
        if (isnan(normNew)) step = a.max_iter + 1;
        if (QUAD && sabsf < 1e-6) step = a.max_iter + 3;
        if (epi) {
          a.znssd[t] = znssd;
          if (a.conv) a.conv[t] = step;
        } else {
          a.conv[t] = step;
          a.U[2 * t] = P[4];
          a.U[2 * t + 1] = P[5];
          for (int k = 0; k < 4; ++k) a.F[4 * t + k] = P[k];
          if (FG) a.zncc[t] = 1.0 - 0.5 * znssd;
          if (a.H)
            for (int k = 0; k < 21; ++k) a.H[t + a.n * k] = s.h[k];
        }
      }
    }
    group_bar<NW>(bar);
  }
}

// The buffers of a CTA for windows of W1 x W1 pixels.  A column holds at least W1 + 9 rows of both
// groups: the footprint of a small warp is W1 + 6, the rest is room for the warp to move and stretch
// before the buffer is loaded again.
constexpr int kSmBytes = 227 * 1024, kCtaBytes = 5 * 1024;  // per CTA: static and reserved shared memory
inline int tile_pitch(int W1) { return W1 + (kTileGroups * (W1 + 9) - W1 + 31) / 32 * 32; }
// CTAs an SM whose buffers fit its shared memory.
inline int tile_ctas(int W1) {
  const int fit = kSmBytes / (tile_pitch(W1) * (int)sizeof(float) * (W1 + 9) + kCtaBytes);
  return fit < 8 ? fit : 8;
}
// As many columns as fit without one CTA less per SM.
inline TileGeom tile_geometry(int W1) {
  TileGeom g;
  g.pitch = tile_pitch(W1);
  g.rows = g.pitch / kTileGroups;
  g.cols = (kSmBytes / tile_ctas(W1) - kCtaBytes) / (g.pitch * (int)sizeof(float));
  if (g.cols > W1 + 16) g.cols = W1 + 16;
  return g;
}
// Whether n windows are staged.  With 4 to 6 CTAs an SM (windows of 47 to 69) the pass has too few warps
// when there are more subsets than run at once, and reading the image is faster (20 000 subsets at 2048 x
// 2048, staged / from the image: window 45, 8 CTAs, 1217 / 1351 us; 49, 6 CTAs, 1698 / 1518; 61, 4 CTAs,
// 2606 / 2116); of fewer subsets a warp's own time counts (window 61: 300 subsets 209 / 242 us, 1184, the
// last that run at once, 238 / 281, 1500 417 / 357).
inline bool tile_staged(int W1, long long n, int sms) {
  const int ctas = tile_ctas(W1);
  return ctas >= 7 || (ctas >= 4 && n <= (long long)kTileGroups * ctas * sms);
}

template <int NW, bool SLOW>
inline int launch_icgn_tile(const IcgnArgs& a, const TileGeom& g, int sms, cudaStream_t st) {
  const bool quad = a.variant == 1, fg = a.variant == 2 || a.zncc != nullptr;
  auto k = quad ? (fg ? icgn_tile_kernel<NW, SLOW, true, true> : icgn_tile_kernel<NW, SLOW, true, false>)
                : (fg ? icgn_tile_kernel<NW, SLOW, false, true> : icgn_tile_kernel<NW, SLOW, false, false>);
  const int threads = 32 * NW * kTileGroups;
  const size_t smem = (size_t)g.pitch * g.cols * sizeof(float);
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem);
  long long grid = (long long)sms * (per_sm < 1 ? 1 : per_sm);
  const long long need = (a.n + kTileGroups - 1) / kTileGroups;
  if (grid > need) grid = need;
  k<<<(unsigned)grid, threads, smem, st>>>(a, g);
  return 1;
}

}  // namespace aldic
