// ALDIC's global step, Subpb2Quadtree (func_quadtree/Subpb2Quadtree.m), on the device.
//
// On a quadtree mesh of 8-node elements (corners 1-4; mid-side "hanging" nodes 5-8 where a
// neighbour is refined, 0 where absent) the step minimises, in the finite-element space,
//   sum over elements and Gauss points of |J| w ((beta + alpha) |grad Uhat|^2
//       - 2 beta grad(N_a) . F_a Uhat_a + mu |Uhat - U|^2 + alpha grad(N) U terms)
// i.e. it solves A Uhat = b with (:149-204)
//   A_e = sum_g |J| w ((beta + alpha) DN' DN + mu N' N),
//   b_e = sum_g |J| w (beta diag(DN' F_rows') + mu N' N U_e + alpha DN' DN U_e),
// where the F rows of an x dof of node a are (F11_a, F12_a) and of a y dof (F21_a, F22_a), and
// v, W are 0 (:40-41: 0 * vdual, 0 * udual).  Both DN' DN and N' N couple x dofs with x dofs
// and y with y by the same numbers, so A_e = K_e (x) I_2 with one 8 x 8 K_e per element, and
// the x and y systems share one matrix.
//
// Layout: K_e row-major per element (64 doubles), b_e per element as (x, y) per local node
// (16 doubles); node -> (element, slot) adjacency lists built on the host, so every product
// and right-hand side is a gather in a fixed order (deterministic, no atomics).  The free
// nodes (all nodes of the elements but the first of unique(elementsFEM), :234-238, less
// the dirichlet nodes) are solved by Jacobi-preconditioned conjugate gradients on the
// interleaved 2 n vector; the dirichlet nodes hold U (:271-273) and enter the right-hand
// side through the same gather.  The reference solves the free block directly (:276).
#include <algorithm>
#include <cstdio>
#include <vector>

#include "common.cuh"
#include "kernels.h"

namespace aldic {

// Gauss points and weights of :60-77 (orders 4 and 5 with the file's rounded constants).
struct GaussRule {
  int np;
  double pt[5];
  double wt[5];
};

__host__ __device__ inline GaussRule gauss_rule(int order) {
  GaussRule g{};
  if (order == 2) {
    g.np = 2;
    g.pt[0] = -1.0 / sqrt(3.0);
    g.pt[1] = 1.0 / sqrt(3.0);
    g.wt[0] = g.wt[1] = 1.0;
  } else if (order == 3) {
    g.np = 3;
    g.pt[0] = 0.0;
    g.pt[1] = sqrt(3.0 / 5.0);
    g.pt[2] = -sqrt(3.0 / 5.0);
    g.wt[0] = 8.0 / 9.0;
    g.wt[1] = g.wt[2] = 5.0 / 9.0;
  } else if (order == 4) {
    g.np = 4;
    g.pt[0] = 0.339981;
    g.pt[1] = -0.339981;
    g.pt[2] = 0.861136;
    g.pt[3] = -0.861136;
    g.wt[0] = g.wt[1] = 0.652145;
    g.wt[2] = g.wt[3] = 0.347855;
  } else {
    g.np = 5;
    g.pt[0] = 0.0;
    g.pt[1] = 0.538469;
    g.pt[2] = -0.538469;
    g.pt[3] = 0.90618;
    g.pt[4] = -0.90618;
    g.wt[0] = 0.568889;
    g.wt[1] = g.wt[2] = 0.478629;
    g.wt[3] = g.wt[4] = 0.236927;
  }
  return g;
}

__host__ __device__ inline double sgn(double x) { return (double)((x > 0.0) - (x < 0.0)); }

// Shape functions and their (ksi, eta) derivatives (:138-148 and funDN*, :343-396): the
// corner functions less half of the two adjacent mid-side ones; d5..d8 switch the mid-side
// nodes (right, top, left, bottom edge) on; sign(0) = 0 as MATLAB's.
__host__ __device__ inline void quadtree_shape(double ksi, double eta, const double d[4], double N[8],
                                               double dk[8], double de[8]) {
  const double aks = fabs(ksi), aet = fabs(eta);
  N[4] = d[0] * 0.5 * (1.0 + ksi) * (1.0 - aet);
  N[5] = d[1] * 0.5 * (1.0 + eta) * (1.0 - aks);
  N[6] = d[2] * 0.5 * (1.0 - ksi) * (1.0 - aet);
  N[7] = d[3] * 0.5 * (1.0 - eta) * (1.0 - aks);
  N[0] = (1.0 - ksi) * (1.0 - eta) * 0.25 - 0.5 * (N[6] + N[7]);
  N[1] = (1.0 + ksi) * (1.0 - eta) * 0.25 - 0.5 * (N[7] + N[4]);
  N[2] = (1.0 + ksi) * (1.0 + eta) * 0.25 - 0.5 * (N[4] + N[5]);
  N[3] = (1.0 - ksi) * (1.0 + eta) * 0.25 - 0.5 * (N[5] + N[6]);
  dk[4] = d[0] * 0.5 * (1.0 - aet);
  de[4] = d[0] * 0.5 * (1.0 + ksi) * sgn(-eta);
  dk[5] = d[1] * 0.5 * (1.0 + eta) * sgn(-ksi);
  de[5] = d[1] * 0.5 * (1.0 - aks);
  dk[6] = d[2] * 0.5 * (-1.0) * (1.0 - aet);
  de[6] = d[2] * 0.5 * (1.0 - ksi) * sgn(-eta);
  dk[7] = d[3] * 0.5 * (1.0 - eta) * sgn(-ksi);
  de[7] = d[3] * 0.5 * (-1.0) * (1.0 - aks);
  dk[0] = -0.25 * (1.0 - eta) - 0.5 * (dk[6] + dk[7]);
  de[0] = -0.25 * (1.0 - ksi) - 0.5 * (de[6] + de[7]);
  dk[1] = 0.25 * (1.0 - eta) - 0.5 * (dk[7] + dk[4]);
  de[1] = -0.25 * (1.0 + ksi) - 0.5 * (de[7] + de[4]);
  dk[2] = 0.25 * (1.0 + eta) - 0.5 * (dk[4] + dk[5]);
  de[2] = 0.25 * (1.0 + ksi) - 0.5 * (de[4] + de[5]);
  dk[3] = -0.25 * (1.0 + eta) - 0.5 * (dk[5] + dk[6]);
  de[3] = 0.25 * (1.0 - ksi) - 0.5 * (de[5] + de[6]);
}

// Row a of K_e and the (x, y) right-hand side of local node a of one element.  xy: the 8
// nodes' coordinates (0 at absent mid-side nodes, as the reference), ue: their (x, y)
// displacements U (0 when absent), fa: node a's (F11, F21, F12, F22).
__host__ __device__ inline void subpb2_element_row(int a, const double xy[16], const double d[4], const double ue[16],
                                                   const double fa[4], int order, double beta, double mu,
                                                   double alpha, double krow[8], double brow[2]) {
  const GaussRule g = gauss_rule(order);
  for (int b = 0; b < 8; ++b) krow[b] = 0.0;
  brow[0] = brow[1] = 0.0;
  for (int je = 0; je < g.np; ++je)    // ndgrid order: ksi runs fastest
    for (int ik = 0; ik < g.np; ++ik) {
      const double ksi = g.pt[ik], eta = g.pt[je], w = g.wt[ik] * g.wt[je];
      double N[8], dk[8], de[8];
      quadtree_shape(ksi, eta, d, N, dk, de);
      double j11 = 0.0, j12 = 0.0, j21 = 0.0, j22 = 0.0;
      for (int k = 0; k < 8; ++k) {
        j11 += dk[k] * xy[2 * k];
        j12 += dk[k] * xy[2 * k + 1];
        j21 += de[k] * xy[2 * k];
        j22 += de[k] * xy[2 * k + 1];
      }
      const double jac = j11 * j22 - j12 * j21;
      const double i11 = j22 / jac, i12 = -j12 / jac, i21 = -j21 / jac, i22 = j11 / jac;
      const double jw = jac * w;
      const double dxa = i11 * dk[a] + i12 * de[a], dya = i21 * dk[a] + i22 * de[a];
      double mux = 0.0, muy = 0.0, alx = 0.0, aly = 0.0;
      for (int b = 0; b < 8; ++b) {
        const double dxb = i11 * dk[b] + i12 * de[b], dyb = i21 * dk[b] + i22 * de[b];
        const double gg = dxa * dxb + dya * dyb, nn = N[a] * N[b];
        krow[b] += jw * ((beta + alpha) * gg + mu * nn);
        mux += nn * ue[2 * b];
        muy += nn * ue[2 * b + 1];
        alx += gg * ue[2 * b];
        aly += gg * ue[2 * b + 1];
      }
      brow[0] += jw * (beta * (dxa * fa[0] + dya * fa[2]) + mu * mux + alpha * alx);
      brow[1] += jw * (beta * (dxa * fa[1] + dya * fa[3]) + mu * muy + alpha * aly);
    }
}

// One thread per (element, local node): K_e row and b_e entries; rows of absent nodes are 0.
// elem: n_el x 8 column-major, 1-based node numbers (0 = no mid-side node); coords n x 2
// column-major; U 2n interleaved; F 4n (F11 F21 F12 F22 per node).
__global__ void subpb2_element_kernel(int n_el, const int* __restrict__ elem, const double* __restrict__ coords,
                                      long long n, const double* __restrict__ U, const double* __restrict__ F,
                                      int order, double beta, double mu, double alpha, double* __restrict__ Ke,
                                      double* __restrict__ be) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= 8LL * n_el) return;
  const int e = (int)(t >> 3), a = (int)(t & 7);
  double* kr = Ke + (long long)e * 64 + a * 8;
  double* br = be + (long long)e * 16 + a * 2;
  int id[8];
  for (int k = 0; k < 8; ++k) id[k] = elem[e + (long long)k * n_el];
  if (id[a] == 0) {
    for (int b = 0; b < 8; ++b) kr[b] = 0.0;
    br[0] = br[1] = 0.0;
    return;
  }
  double xy[16], ue[16], d[4], fa[4];
  for (int k = 0; k < 8; ++k) {
    const long long g = id[k] - 1;
    const bool on = id[k] != 0;
    xy[2 * k] = on ? coords[g] : 0.0;
    xy[2 * k + 1] = on ? coords[g + n] : 0.0;
    ue[2 * k] = on ? U[2 * g] : 0.0;
    ue[2 * k + 1] = on ? U[2 * g + 1] : 0.0;
  }
  for (int k = 0; k < 4; ++k) d[k] = id[4 + k] != 0 ? 1.0 : 0.0;
  const long long ga = id[a] - 1;
  for (int k = 0; k < 4; ++k) fa[k] = F[4 * ga + k];
  double krow[8], brow[2];
  subpb2_element_row(a, xy, d, ue, fa, order, beta, mu, alpha, krow, brow);
  for (int b = 0; b < 8; ++b) kr[b] = krow[b];
  br[0] = brow[0];
  br[1] = brow[1];
}

// (K x) at node i for both components: the node's (element, slot) entries, each a row of
// that element's K_e against the element's nodes.  x is 2n interleaved.
__host__ __device__ inline void subpb2_gather_row(long long i, const int* adj_ptr, const int* adj, const int* elem,
                                                  int n_el, const double* Ke, const double* x, double& yx,
                                                  double& yy) {
  yx = 0.0;
  yy = 0.0;
  for (int q = adj_ptr[i]; q < adj_ptr[i + 1]; ++q) {
    const int e = adj[q] >> 3, s = adj[q] & 7;
    const double* kr = Ke + (long long)e * 64 + s * 8;
    for (int b = 0; b < 8; ++b) {
      const int nb = elem[e + (long long)b * n_el];
      if (nb == 0) continue;
      yx += kr[b] * x[2 * (long long)(nb - 1)];
      yy += kr[b] * x[2 * (long long)(nb - 1) + 1];
    }
  }
}

// State of the solve, one set for the interleaved 2 n system.
struct Subpb2Scalars {
  double rz, rr0, beta;
  int it, done, ok, timeout;
  unsigned int arrived;  // grid barrier: CTAs arrived since the launch
};

namespace {

constexpr int kCgThreads = 128;
constexpr int kEll = 32;          // entries of a matrix row; a node with more neighbours gathers from K_e
constexpr int kEllOverflow = 255;
constexpr int kAsmThreads = 64;
constexpr long long kBarrierSpins = 20000000LL;  // some seconds of polling

}  // namespace

// Per node: the rows of the assembled matrix (column numbers and values, one row per thread in
// column-major ELL arrays of n rows, so that consecutive threads read consecutive entries), the
// right-hand side (into r), the Jacobi diagonal and the start x = U at dirichlet nodes, 0
// elsewhere.  free_[i]: 1 free, 2 dirichlet, 0 neither (only free rows are kept).
__global__ void __launch_bounds__(kAsmThreads) subpb2_assemble_kernel(
    long long n, const int* __restrict__ adj_ptr, const int* __restrict__ adj, const int* __restrict__ elem, int n_el,
    const double* __restrict__ Ke, const double* __restrict__ be, const unsigned char* __restrict__ free_,
    const double* __restrict__ U, double* __restrict__ r, double* __restrict__ D, double* __restrict__ x,
    int* __restrict__ col, double* __restrict__ val, unsigned char* __restrict__ cnt) {
  __shared__ int sc[kEll][kAsmThreads];
  __shared__ double sv[kEll][kAsmThreads];
  const int t = threadIdx.x;
  const long long i = blockIdx.x * (long long)kAsmThreads + t;
  if (i >= n) return;
  const int kind = free_[i];
  double bx = 0.0, by = 0.0, dg = 0.0;
  int m = 0;
  if (kind == 1)
    for (int q = adj_ptr[i]; q < adj_ptr[i + 1]; ++q) {
      const int e = adj[q] >> 3, s = adj[q] & 7;
      const double* kr = Ke + (long long)e * 64 + s * 8;
      bx += be[(long long)e * 16 + 2 * s];
      by += be[(long long)e * 16 + 2 * s + 1];
      dg += kr[s];
      for (int b = 0; b < 8; ++b) {
        const int nb = elem[e + (long long)b * n_el] - 1;
        if (nb < 0 || m == kEllOverflow) continue;
        int k = 0;
        while (k < m && sc[k][t] != nb) ++k;
        if (k < m) {
          sv[k][t] += kr[b];
        } else if (m < kEll) {
          sc[m][t] = nb;
          sv[m][t] = kr[b];
          ++m;
        } else {
          m = kEllOverflow;
        }
      }
    }
  cnt[i] = (unsigned char)m;
  if (m != kEllOverflow)
    for (int k = 0; k < m; ++k) {
      col[k * n + i] = sc[k][t];
      val[k * n + i] = sv[k][t];
    }
  r[2 * i] = bx;
  r[2 * i + 1] = by;
  D[i] = dg;
  x[2 * i] = kind == 2 ? U[2 * i] : 0.0;
  x[2 * i + 1] = kind == 2 ? U[2 * i + 1] : 0.0;
}

namespace {

// Grid barrier that exchanges two sums: every CTA stores its partials of v0, v1, arrives at one
// counter, and after the barrier adds all CTAs' partials in CTA order, so all get the same bits.
// (Flag slots that carry the values and are polled by every CTA were slower: 3.5 us against
// 1.2 us for the counter on 139 CTAs.)  Partials alternate between two sets: a CTA is at most one
// barrier ahead of one that still reads.  False after a time-out of the wait, which ends every CTA
// at this or its next barrier.  Every thread calls it; writes before it are visible to all CTAs
// after it (cooperative launch).
__device__ __forceinline__ bool grid_exchange(double2* parts, unsigned int& epoch, Subpb2Scalars* sc, double& v0,
                                              double& v1, double* red) {
  ++epoch;
  double2* set = parts + (size_t)gridDim.x * (epoch & 1);
  v0 = warp_sum(v0);
  v1 = warp_sum(v1);
  const int wid = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[2 * wid] = v0;
    red[2 * wid + 1] = v1;
  }
  __syncthreads();
  int late = 0;
  if (threadIdx.x == 0) {
    double2 v = make_double2(red[0], red[1]);
#pragma unroll
    for (int k = 1; k < kCgThreads / 32; ++k) {
      v.x += red[2 * k];
      v.y += red[2 * k + 1];
    }
    __stcg(set + blockIdx.x, v);
    __threadfence();  // this CTA's writes (ordered by the barrier above) before its arrival
    atomicAdd(&sc->arrived, 1u);
    const unsigned int target = epoch * gridDim.x;
    long long spins = 0;
    unsigned int seen;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&sc->arrived) : "memory");
    } while (seen < target && ++spins < kBarrierSpins);
    late = seen < target;
    if (late) atomicExch(&sc->timeout, 1);
  }
  late = __syncthreads_or(late);
  double s0 = 0.0, s1 = 0.0;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += kCgThreads) {
    const double2 v = __ldcg(set + k);
    s0 += v.x;
    s1 += v.y;
  }
  s0 = warp_sum(s0);
  s1 = warp_sum(s1);
  if ((threadIdx.x & 31) == 0) {
    red[2 * wid] = s0;
    red[2 * wid + 1] = s1;
  }
  __syncthreads();
  v0 = v1 = 0.0;
#pragma unroll
  for (int k = 0; k < kCgThreads / 32; ++k) {
    v0 += red[2 * k];
    v1 += red[2 * k + 1];
  }
  __syncthreads();  // red is free again
  return !late;
}

}  // namespace

// The whole Jacobi-preconditioned conjugate-gradient solve (or its next `iters` iterations) in one
// cooperative launch.  Per iteration two grid barriers: after q = K p (with the sum p q) and after
// the update of x, r, z (with the sums r z and r r).  The new direction p = z + beta p_old is
// formed where it is read, by the node and by its neighbours, and kept in the other of two
// buffers, which saves a third barrier.  ONE: a thread has one node and keeps its x, r, D and the
// first kEllRegs entries of its matrix row in registers.
//
// What bounds it: the latency of the barriers and gathers (17 757 nodes: the matrix and the
// vectors are 5 MB in L2).  Five launches an iteration and a host read-back every 16 took 872 us
// a solve of 30 iterations; one launch with every row read from L2 436 us; this form 275 us (185 us in the kernel).
constexpr int kEllRegs = 12;

template <bool ONE>
__global__ void __launch_bounds__(kCgThreads) subpb2_cg_kernel(
    int start, int iters, long long n, const int* __restrict__ adj_ptr, const int* __restrict__ adj,
    const int* __restrict__ elem, int n_el, const double* __restrict__ Ke, const unsigned char* __restrict__ free_,
    const int* __restrict__ col, const double* __restrict__ val, const unsigned char* __restrict__ cnt,
    const double* __restrict__ D, double* __restrict__ x, double2* __restrict__ r, double2* __restrict__ z,
    double2* __restrict__ p0, double2* __restrict__ p1, double2* __restrict__ q, double2* __restrict__ parts,
    double tol2, int maxit, Subpb2Scalars* sc) {
  __shared__ double red[2 * (kCgThreads / 32)];
  const long long stride = (long long)gridDim.x * kCgThreads, first = blockIdx.x * (long long)kCgThreads + threadIdx.x;
  unsigned int epoch = 0;
  double rz, rr0, beta = 0.0;
  int it = 0;
  if (start) {  // r = b - K x, z = r / D on the free nodes
    double srz = 0.0, srr = 0.0;
    for (long long i = first; i < n; i += stride) {
      double2 ri = make_double2(0.0, 0.0), zi = ri;
      if (free_[i] == 1) {
        double kx = 0.0, ky = 0.0;
        const int m = cnt[i];
        if (m == kEllOverflow)
          subpb2_gather_row(i, adj_ptr, adj, elem, n_el, Ke, x, kx, ky);
        else
          for (int k = 0; k < m; ++k) {
            const long long c = col[k * n + i];
            const double a = val[k * n + i];
            kx = fma(a, x[2 * c], kx);
            ky = fma(a, x[2 * c + 1], ky);
          }
        ri = make_double2(r[i].x - kx, r[i].y - ky);
        zi = make_double2(ri.x / D[i], ri.y / D[i]);
      }
      r[i] = ri;
      z[i] = zi;
      p0[i] = p1[i] = q[i] = make_double2(0.0, 0.0);
      srz += ri.x * zi.x + ri.y * zi.y;
      srr += ri.x * ri.x + ri.y * ri.y;
    }
    if (!grid_exchange(parts, epoch, sc, srz, srr, red)) return;
    rz = srz;
    rr0 = srr;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      sc->rr0 = rr0;
      sc->rz = rz;
      sc->it = 0;
      sc->ok = 1;
      sc->done = rr0 == 0.0;
    }
    if (rr0 == 0.0) return;
  } else {  // the last launch's state
    rz = sc->rz;
    rr0 = sc->rr0;
    it = sc->it;
    beta = sc->beta;
  }
  // ONE: the thread's node in registers
  const long long i1 = first;
  const bool mine = ONE && i1 < n && free_[i1] == 1;
  const int m1 = mine ? cnt[i1] : 0;
  int c1[kEllRegs];
  double a1[kEllRegs], x1x = 0.0, x1y = 0.0, d1 = 1.0;
  double2 r1 = make_double2(0.0, 0.0), z1 = r1, pa = r1;
#pragma unroll
  for (int k = 0; k < kEllRegs; ++k) {
    const bool on = mine && m1 != kEllOverflow && k < m1;
    c1[k] = on ? col[k * n + i1] : (mine ? (int)i1 : 0);
    a1[k] = on ? val[k * n + i1] : 0.0;
  }
  if (mine) {
    x1x = x[2 * i1];
    x1y = x[2 * i1 + 1];
    d1 = D[i1];
    r1 = r[i1];
    z1 = z[i1];
    pa = (it & 1 ? p1 : p0)[i1];
  }
  for (int k_ = 0; k_ < iters; ++k_) {
    // q = K p with p = z + beta p_old
    double2* po = it & 1 ? p1 : p0;
    double2* pn = it & 1 ? p0 : p1;
    double pq = 0.0, unused = 0.0;
    double2 q1 = make_double2(0.0, 0.0);
    for (long long i = first; i < n; i += stride) {
      if (free_[i] != 1) continue;
      const int m = ONE ? m1 : cnt[i];
      const double2 zi = ONE ? z1 : z[i], pi = ONE ? pa : po[i];
      const double2 pv = make_double2(fma(beta, pi.x, zi.x), fma(beta, pi.y, zi.y));
      double qx = 0.0, qy = 0.0;
      if (m == kEllOverflow) {
        for (int a = adj_ptr[i]; a < adj_ptr[i + 1]; ++a) {
          const int e = adj[a] >> 3;
          const double* kr = Ke + (long long)e * 64 + (adj[a] & 7) * 8;
          for (int b = 0; b < 8; ++b) {
            const long long nb = elem[e + (long long)b * n_el] - 1;
            if (nb < 0) continue;
            const double2 zn = __ldcg(z + nb), pp = __ldcg(po + nb);
            qx += kr[b] * fma(beta, pp.x, zn.x);
            qy += kr[b] * fma(beta, pp.y, zn.y);
          }
        }
      } else {
        if constexpr (ONE) {
          double2 zn[kEllRegs], pp[kEllRegs];
#pragma unroll
          for (int k = 0; k < kEllRegs; ++k) {  // entries past the row's end are the node's own, times 0
            zn[k] = __ldcg(z + c1[k]);
            pp[k] = __ldcg(po + c1[k]);
          }
#pragma unroll
          for (int k = 0; k < kEllRegs; ++k) {
            qx = fma(a1[k], fma(beta, pp[k].x, zn[k].x), qx);
            qy = fma(a1[k], fma(beta, pp[k].y, zn[k].y), qy);
          }
        }
#pragma unroll 4
        for (int k = ONE ? kEllRegs : 0; k < m; ++k) {
          const int c = col[k * n + i];
          const double a = val[k * n + i];
          const double2 zn = __ldcg(z + c), pp = __ldcg(po + c);
          qx = fma(a, fma(beta, pp.x, zn.x), qx);
          qy = fma(a, fma(beta, pp.y, zn.y), qy);
        }
      }
      pn[i] = pv;
      if (ONE) {
        pa = pv;
        q1 = make_double2(qx, qy);
      } else {
        q[i] = make_double2(qx, qy);
      }
      pq += pv.x * qx + pv.y * qy;
    }
    if (!grid_exchange(parts, epoch, sc, pq, unused, red)) return;
    if (!(pq > 0.0)) {  // no descent direction left: stop with what x holds
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        sc->done = 1;
        sc->ok = 0;
      }
      break;
    }
    // x += alpha p, r -= alpha q, z = r / D on the free nodes
    const double al = rz / pq;
    double srz = 0.0, srr = 0.0;
    for (long long i = first; i < n; i += stride) {
      if (free_[i] != 1) continue;
      const double2 pv = ONE ? pa : pn[i], qv = ONE ? q1 : q[i];
      double2 rv = ONE ? r1 : r[i];
      const double d = ONE ? d1 : D[i];
      rv = make_double2(fma(-al, qv.x, rv.x), fma(-al, qv.y, rv.y));
      const double2 zv = make_double2(rv.x / d, rv.y / d);
      if (ONE) {
        x1x = fma(al, pv.x, x1x);
        x1y = fma(al, pv.y, x1y);
        r1 = rv;
        z1 = zv;
      } else {
        x[2 * i] = fma(al, pv.x, x[2 * i]);  // the caller's array: 8-byte aligned
        x[2 * i + 1] = fma(al, pv.y, x[2 * i + 1]);
        r[i] = rv;
      }
      z[i] = zv;
      srz += rv.x * zv.x + rv.y * zv.y;
      srr += rv.x * rv.x + rv.y * rv.y;
    }
    if (!grid_exchange(parts, epoch, sc, srz, srr, red)) return;
    beta = srz / rz;
    rz = srz;
    ++it;
    const bool conv = srr <= tol2 * rr0, last = it >= maxit;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      sc->rz = rz;
      sc->beta = beta;
      sc->it = it;
      if (conv || last) sc->done = 1;
      if (last && !conv) sc->ok = 0;
    }
    if (conv || last) break;
  }
  if (mine) {
    x[2 * i1] = x1x;
    x[2 * i1 + 1] = x1y;
    r[i1] = r1;
  }
}

// CTAs that the two forms of the solve may have, all resident at once.  One node a thread: 3 an SM (168
// registers), short barriers.  Several: as many as fit (7 an SM at 72 registers), for the loads in flight
// (3 / 7 an SM, a solve of 38 iterations: 90 000 nodes 802 / 734 us, 490 000 3.87 / 2.62 ms, 1.68 M 13.2 /
// 8.0 ms; five launches an iteration took 12.6 ms there).
static void cg_limits(long long* one, long long* many) {
  int dev = 0, sms = 148, per_one = 1, per_many = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_one, subpb2_cg_kernel<true>, kCgThreads, 0);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_many, subpb2_cg_kernel<false>, kCgThreads, 0);
  *one = (long long)sms * std::max(1, std::min(per_one, 3));
  *many = (long long)sms * std::max(1, per_many);
}

int subpb2_cg_blocks(long long n) {
  long long one, many;
  cg_limits(&one, &many);
  const long long need = (n + kCgThreads - 1) / kCgThreads;
  return (int)std::max(1LL, std::min(need, need <= one ? one : many));
}

int subpb2_mesh_tables(long long n, long long n_el, const int* E, long long n_dir, const int* dir,
                       std::vector<int>& ptr, std::vector<int>& adj, std::vector<unsigned char>& kind, char* msg,
                       size_t msg_len) {
  std::vector<int> cnt((size_t)n + 1, 0), ids;
  ids.reserve((size_t)n_el * 8);
  for (long long e = 0; e < n_el; ++e)
    for (int k = 0; k < 8; ++k) {
      const int id = E[(size_t)e + (size_t)k * n_el];
      if (id < 0 || id > n || (k < 4 && id == 0)) {
        std::snprintf(msg, msg_len, "element %lld node %d: %d (corners 1..n, mid-side 0..n)", e + 1, k + 1, id);
        return 1;
      }
      ids.push_back(id);
      if (id) ++cnt[(size_t)id];
    }
  ptr.assign((size_t)n + 1, 0);
  for (long long i = 0; i < n; ++i) ptr[(size_t)i + 1] = ptr[(size_t)i] + cnt[(size_t)i + 1];
  adj.assign((size_t)ptr[(size_t)n], 0);
  std::vector<int> pos(ptr.begin(), ptr.end() - 1);
  for (long long e = 0; e < n_el; ++e)
    for (int k = 0; k < 8; ++k) {
      const int id = E[(size_t)e + (size_t)k * n_el];
      if (id) adj[(size_t)pos[(size_t)id - 1]++] = (int)(e * 8 + k);
    }
  // involved: unique(elementsFEM(:, 1:8)) less its first entry (:234-238: the reference
  // drops the 0 that absent mid-side nodes leave there); then the dirichlet nodes
  std::sort(ids.begin(), ids.end());
  ids.erase(std::unique(ids.begin(), ids.end()), ids.end());
  kind.assign((size_t)n, 0);
  for (size_t k = 1; k < ids.size(); ++k) kind[(size_t)ids[k] - 1] = 1;
  for (long long k = 0; k < n_dir; ++k) {
    const int d = dir[k];
    if (d < 1 || d > n) {
      std::snprintf(msg, msg_len, "dirichlet node %d outside 1..%lld", d, n);
      return 1;
    }
    kind[(size_t)d - 1] = 2;
  }
  return 0;
}

size_t subpb2_scalars_bytes() { return sizeof(Subpb2Scalars); }

size_t subpb2_ell_bytes(long long n) { return (size_t)n * kEll * (sizeof(int) + sizeof(double)) + (size_t)n + 512; }

void subpb2_read_status(const void* host_copy, int* it, int* done, int* ok, int* timeout) {
  const Subpb2Scalars* s = (const Subpb2Scalars*)host_copy;
  *it = s->it;
  *done = s->done;
  *ok = s->ok;
  *timeout = s->timeout;
}

namespace {
struct Ell {
  double* val;
  int* col;
  unsigned char* cnt;
};
Ell ell_parts(void* base, long long n) {
  Ell e;
  e.val = (double*)base;
  e.col = (int*)(e.val + (size_t)n * kEll);
  e.cnt = (unsigned char*)(e.col + (size_t)n * kEll);
  return e;
}
}  // namespace

int launch_subpb2_setup(int n_el, const int* elem, const double* coords, long long n, const double* U,
                        const double* F, int order, double beta, double mu, double alpha, const int* adj_ptr,
                        const int* adj, const unsigned char* free_, double* Ke, double* be, void* ell, double* D,
                        double* x, double* r, cudaStream_t st) {
  const long long rows = 8LL * n_el;
  subpb2_element_kernel<<<(unsigned)((rows + 127) / 128), 128, 0, st>>>(n_el, elem, coords, n, U, F, order, beta, mu,
                                                                        alpha, Ke, be);
  const Ell e = ell_parts(ell, n);
  subpb2_assemble_kernel<<<(unsigned)((n + kAsmThreads - 1) / kAsmThreads), kAsmThreads, 0, st>>>(
      n, adj_ptr, adj, elem, n_el, Ke, be, free_, U, r, D, x, e.col, e.val, e.cnt);
  return 2;
}

size_t subpb2_parts_bytes(int blocks) { return (size_t)blocks * 2 * sizeof(double2); }

int launch_subpb2_cg(bool start, int iters, int blocks, long long n, const int* adj_ptr, const int* adj,
                     const int* elem, int n_el, const double* Ke, const unsigned char* free_, void* ell,
                     const double* D, double* x, double* r, double* z, double* p0, double* p1, double* q, void* parts,
                     double tol2, int maxit, Subpb2Scalars* sc, cudaStream_t st) {
  const Ell e = ell_parts(ell, n);
  if (start)
    cudaMemsetAsync(sc, 0, sizeof(Subpb2Scalars), st);
  else
    cudaMemsetAsync(&sc->arrived, 0, sizeof(unsigned int), st);  // barriers count from 1 in every launch
  int s = start ? 1 : 0;
  const int *col = e.col;
  const double *val = e.val;
  const unsigned char* cnt = e.cnt;
  void* args[] = {&s, &iters, &n, &adj_ptr, &adj, &elem, &n_el, &Ke, &free_, &col, &val, &cnt, &D, &x, &r, &z, &p0,
                  &p1, &q, &parts, &tol2, &maxit, &sc};
  long long one, many;
  cg_limits(&one, &many);
  const void* k = blocks <= one && n <= blocks * (long long)kCgThreads ? (const void*)subpb2_cg_kernel<true>
                                                                       : (const void*)subpb2_cg_kernel<false>;
  cudaLaunchCooperativeKernel(k, dim3((unsigned)blocks), dim3(kCgThreads), args, 0, st);
  return 1;
}

}  // namespace aldic
