// akb_rve.cu -- batched periodic RVE solves (the micro problems of FE^2).
//
// FP32 RVEs of up to 16^3 cells (but 14^3, whose planes divide by neither 2 x 2
// nor 4 x 2; of 16^3 fewer than kManyInstances) are relaxed by a cluster of CTAs
// each: k_rve_cluster, below. All others by k_rve and k_rve_indexed:
// one CTA relaxes one RVE with its whole state on chip: the fluctuation w,
// the velocity and the force of the n^3 periodic nodes (component-major),
// the inverse fictitious mass, the voxel materials and the voxel shape
// gradients live in shared memory (n = 16 in FP32: 170 KB), so an iteration
// reads and writes no global memory. Elements are visited in 8 colours
// (voxel parity in x, y, z; n even keeps them periodic-consistent): voxels
// of one colour share no node, so each thread adds its element's force to
// its 8 corners without atomics and the sum over the 8 colours is in a fixed
// order (deterministic).
//
// Per iteration (leapfrog dynamic relaxation, mass-proportional damping c):
//   f = -sum_e sum_q w_q P(H + grad w) grad N_a     (voxel force, 8 Gauss pts)
//   v = ((1 - c dt / 2) v + dt f / m) / (1 + c dt / 2);  w += dt v
// with m the lumped mass of density lambda + 2 mu (unit P-wave speed in every
// voxel), dt = factor h s_min(F) / c_J (s_min the smallest singular value of
// F, c_J the P-wave speed raised by compression, ln J < 0) and
// c = factor 2 (2 pi / L) min sqrt(mu / (lambda + 2 mu)) (critical damping of
// the lowest shear mode). Strain concentrates in the soft phase beyond what
// F shows, so an attempt whose residual turns non-finite or explodes is
// restarted from its initial state with a 0.6x time step (at most 3 times).
// The homogenised stress is sum w_q P / L^3.
#include <algorithm>
#include <cmath>
#include <memory>
#include <mutex>
#include <type_traits>
#include <vector>

#include "../../include/akb_fe2.h"
#include "akb_fastmath.cuh"

struct akb_rve {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool owns_stream = false;
  int mode = AKB_MODE_FP32_BULK;
  int n = 0, nmat = 0;
  double L = 1.0;
  int max_it = 2000, check = 10;
  double tol = 1e-4, tsf = 0.6, dampf = 0.6;
  double lam[8] = {0}, mu[8] = {0};
  int kind[8] = {0};
  double vf[8] = {0};
  uint8_t* d_vmat = nullptr;
  void* d_inv_mass = nullptr;  // float or double per mode
  size_t smem = 0;
  int clusters = 0;  // clusters of k_rve_cluster the device runs at once (0: not this way)
};

namespace akb {
namespace {

constexpr int kRveThreads = 256;  // 2 voxels per thread and colour at n = 16; no register spills
constexpr double kDivergence = 1e4;     // relative residual taken as divergence
constexpr double kRestartFactor = 0.6;  // time-step factor of each restart
constexpr int kMaxRestarts = 3;

struct RveArgs {
  int n, nn, nmat, max_it, check;
  int write_fluct;  // write the relaxed fluctuation back
  double L, h, tol, tsf, dampf;
  double lam[8], mu[8];
  int kind[8];
  const uint8_t* vmat;
  const void* inv_mass;
};

__host__ __device__ inline int corner_x(int a) { return ((a & 3) == 1 || (a & 3) == 2) ? 1 : 0; }
__host__ __device__ inline int corner_y(int a) { return (a >> 1) & 1; }
__host__ __device__ inline int corner_z(int a) { return a >> 2; }

// Shared-memory position of node (or voxel) (x, y, z): grouped by parity
// class (x, y, z mod 2), then (x/2, y/2, z/2) lexicographic. A voxel colour
// reaches each of its corners in one parity class, and its threads' voxels
// are consecutive in that class, so the gathers and scatters of a warp hit
// consecutive words (no bank conflicts).
__device__ inline int pidx(int x, int y, int z, int n) {
  const int hn = n >> 1;
  return ((x & 1) | ((y & 1) << 1) | ((z & 1) << 2)) * (hn * hn * hn) + (x >> 1) +
         hn * ((y >> 1) + hn * (z >> 1));
}

__device__ inline double det3d(const double* m) {
  return m[0] * (m[4] * m[8] - m[5] * m[7]) - m[1] * (m[3] * m[8] - m[5] * m[6]) +
         m[2] * (m[3] * m[7] - m[4] * m[6]);
}

// Smallest eigenvalue of a symmetric 3x3 matrix (trigonometric solution of
// the characteristic cubic, O. K. Smith, Comm. ACM 4(4):168, 1961).
__device__ double smallest_eigenvalue(const double* A) {
  const double p1 = A[1] * A[1] + A[2] * A[2] + A[5] * A[5];
  const double q = (A[0] + A[4] + A[8]) / 3.0;
  const double p2 = (A[0] - q) * (A[0] - q) + (A[4] - q) * (A[4] - q) +
                    (A[8] - q) * (A[8] - q) + 2.0 * p1;
  if (p2 <= 0.0) return q;
  const double p = sqrt(p2 / 6.0);
  double Bm[9];
  for (int k = 0; k < 9; ++k) Bm[k] = (A[k] - (k % 4 == 0 ? q : 0.0)) / p;
  double r = det3d(Bm) / 2.0;
  r = fmin(1.0, fmax(-1.0, r));
  const double phi = acos(r) / 3.0;
  return q + 2.0 * p * cos(phi + 2.0 * M_PI / 3.0);
}

template <typename S>
struct RveSmem {
  S *u, *v, *f, *im, *B;
  uint8_t* mat;
  double* red;  // 16 warps x 9
  double* par;  // dt, c, fscale, r
};

template <typename S>
__host__ __device__ inline size_t rve_smem_bytes(int nn) {
  size_t b = 9 * (size_t)nn * sizeof(S) + (size_t)nn * sizeof(S) + 192 * sizeof(S);
  b = (b + (size_t)nn + 15) & ~size_t(15);
  return b + (16 * 9 + 8) * sizeof(double);
}

template <typename S>
__device__ inline RveSmem<S> carve(unsigned char* smem, int nn) {
  RveSmem<S> s;
  S* p = reinterpret_cast<S*>(smem);
  s.u = p;
  s.v = p + 3 * nn;
  s.f = p + 6 * nn;
  s.im = p + 9 * nn;
  s.B = p + 10 * nn;
  s.mat = reinterpret_cast<uint8_t*>(p + 10 * nn + 192);
  size_t off = ((size_t)(10 * nn + 192) * sizeof(S) + (size_t)nn + 15) & ~size_t(15);
  s.red = reinterpret_cast<double*>(smem + off);
  s.par = s.red + 16 * 9;
  return s;
}

// First Piola-Kirchhoff stress of a voxel point (row-major, g = grad u):
// neo-Hookean P = mu (F - F^-T) + lambda ln J F^-T (the reference's F S with
// S = mu (I - C^-1) + lambda ln J C^-1, since F C^-1 = F^-T), written without
// O(1) terms that cancel at small strain: with t = tr g, I2 = (t^2 - tr g^2)/2,
//   J - 1 = t + I2 + det g,  adj(F) = (1 + t + I2) I - (1 + t) g + g^2,
//   F - F^-T = g + (det(g) I + (1 + t) g^T - (g^T)^2) / J,  F^-T = adj(F)^T / J,
//   ln J = log1p(J - 1);
// or small-strain elastic sigma.
template <typename S>
__device__ inline void voxel_stress(const MatParams& mp, const S* g, S* P) {
  const S lam = S(mp.lambda), mu = S(mp.mu);
  if (mp.kind != AKB_MATERIAL_NEOHOOKEAN) {
    const S tr = g[0] + g[4] + g[8];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) P[i * 3 + j] = mu * (g[i * 3 + j] + g[j * 3 + i]) + (i == j ? lam * tr : S(0));
    return;
  }
  S gg[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      gg[i * 3 + j] = g[i * 3] * g[j] + g[i * 3 + 1] * g[3 + j] + g[i * 3 + 2] * g[6 + j];
  const S t = g[0] + g[4] + g[8];
  const S I2 = S(0.5) * (t * t - (gg[0] + gg[4] + gg[8]));
  const S dg = g[0] * (g[4] * g[8] - g[5] * g[7]) - g[1] * (g[3] * g[8] - g[5] * g[6]) +
               g[2] * (g[3] * g[7] - g[4] * g[6]);
  const S jm1 = t + I2 + dg;
  const S iJ = S(1) / (S(1) + jm1);
  const S a = mu * iJ, b = lam * log1p(jm1) * iJ, c = S(1) + t;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const S gt = g[j * 3 + i], ggt = gg[j * 3 + i];
      const S adjT = (i == j ? c + I2 : S(0)) - c * gt + ggt;
      const S dev = (i == j ? dg : S(0)) + c * gt - ggt;
      P[i * 3 + j] = mu * g[i * 3 + j] + a * dev + b * adjT;
    }
}

// The same in FP32 with every rounding spelled out (which product of a sum of
// products is fused is the compiler's choice otherwise, and differs from kernel
// to kernel): all kernels that relax FP32 RVEs agree bit for bit.
__device__ __forceinline__ void voxel_stress_f32(const MatParams& mp, const float* g, float* P) {
  const float lam = float(mp.lambda), mu = float(mp.mu);
  if (mp.kind != AKB_MATERIAL_NEOHOOKEAN) {
    const float lt = __fmul_rn(lam, g[0] + g[4] + g[8]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        P[i * 3 + j] = __fmaf_rn(mu, g[i * 3 + j] + g[j * 3 + i], i == j ? lt : 0.0f);
    return;
  }
  float gg[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const float x = __fmaf_rn(g[i * 3], g[j], __fmul_rn(g[i * 3 + 1], g[3 + j]));
      // (the last products of entries 3 and 4 are those of det g below)
      gg[i * 3 + j] = i == 1 && j < 2 ? __fadd_rn(x, __fmul_rn(g[i * 3 + 2], g[6 + j]))
                                      : __fmaf_rn(g[i * 3 + 2], g[6 + j], x);
    }
  const float t = g[0] + g[4] + g[8];
  const float I2 = 0.5f * __fmaf_rn(t, t, -(gg[0] + gg[4] + gg[8]));
  const float d0 = __fmaf_rn(g[4], g[8], -__fmul_rn(g[5], g[7]));
  const float d1 = __fmaf_rn(g[3], g[8], -__fmul_rn(g[5], g[6]));
  const float d2 = __fmaf_rn(-g[4], g[6], __fmul_rn(g[3], g[7]));
  const float dg = __fmaf_rn(g[2], d2, __fmaf_rn(g[0], d0, -__fmul_rn(g[1], d1)));
  const float jm1 = __fadd_rn(__fadd_rn(t, I2), dg);
  const float iJ = 1.0f / __fadd_rn(1.0f, jm1);
  const float a = __fmul_rn(mu, iJ), b = __fmul_rn(__fmul_rn(lam, log1pf(jm1)), iJ), c = 1.0f + t;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const float gt = g[j * 3 + i], ggt = gg[j * 3 + i];
      float adjT, dev;
      if (i == j) {
        adjT = __fadd_rn(__fmaf_rn(-c, gt, __fadd_rn(c, I2)), ggt);
        dev = __fadd_rn(__fmaf_rn(c, gt, dg), -ggt);
      } else {
        const float cg = __fmul_rn(c, gt);
        adjT = __fadd_rn(ggt, -cg);
        dev = __fadd_rn(cg, -ggt);
      }
      P[i * 3 + j] = __fmaf_rn(b, adjT, __fmaf_rn(mu, g[i * 3 + j], __fmul_rn(a, dev)));
    }
}

// Edge sums T_j[e] = sum_q W[q][j][e] w_q P[:, j] of a voxel from its edge
// differences D (see voxel_forces); PSUM adds sum_q w_q P to psum.
template <typename S, bool PSUM>
__device__ __forceinline__ void voxel_edge_sums(const S* B, const MatParams& mp,
                                                const S (&D)[3][4][3], S wq, S (&T)[3][4][3],
                                                double* psum) {
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int i = 0; i < 3; ++i) T[j][e][i] = 0;
#pragma unroll 1
  for (int q = 0; q < 8; ++q) {
    const S* Wq = B + q * 12;  // [direction][edge]
    S g[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        S c;
        if constexpr (sizeof(S) == 4) {
          c = __fmaf_rn(Wq[j * 4], D[j][0][i], __fmul_rn(Wq[j * 4 + 1], D[j][1][i]));
          c = __fmaf_rn(Wq[j * 4 + 2], D[j][2][i], c);
          c = __fmaf_rn(Wq[j * 4 + 3], D[j][3][i], c);
        } else {
          c = Wq[j * 4] * D[j][0][i];
#pragma unroll
          for (int e = 1; e < 4; ++e) c += Wq[j * 4 + e] * D[j][e][i];
        }
        g[i * 3 + j] = c;
      }
    S P[9];
    if constexpr (sizeof(S) == 4)
      voxel_stress_f32(mp, g, P);
    else
      voxel_stress<S>(mp, g, P);
#pragma unroll
    for (int k = 0; k < 9; ++k) P[k] *= wq;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          if constexpr (sizeof(S) == 4)
            T[j][e][i] = __fmaf_rn(Wq[j * 4 + e], P[i * 3 + j], T[j][e][i]);
          else
            T[j][e][i] += Wq[j * 4 + e] * P[i * 3 + j];
        }
    if (PSUM)
#pragma unroll
      for (int k = 0; k < 9; ++k) psum[k] += double(P[k]);
  }
}

// CTAs of the cluster that relaxes an FP32 RVE (k_rve_cluster)
constexpr int kClusterThreads = 512;
constexpr int kClusterVoxels = 1024;

// CTAs per RVE of n^3 cells, 0: not this way.
__host__ __device__ inline int cluster_of(int n) {
  for (int c = 1; c <= 4; c *= 2)
    if (n % c == 0 && (n / c) % 2 == 0 && (int64_t)n * n * n / c <= kClusterVoxels) return c;
  return 0;
}

// An RVE of 16^3 is relaxed by a cluster of four CTAs or, in large numbers, by
// one CTA (kManyInstances), and its stress must not tell which: one CTA adds the
// voxels' w P up as the four would. There a thread has a voxel of colour c and
// the one of colour c + 4 at the same place t in the colour, c = 0..3, t a
// quarter of the colour's places for each CTA; then come its warp, the CTA's 16
// warps and the CTAs. Here thread x has t = x and x + 256: eight sums.
template <typename S>
__host__ __device__ inline bool sums_by_quarters(int n) {
  return sizeof(S) == 4 && cluster_of(n) == 4;
}
constexpr int kQuarterSums = 8;

// f -= element forces of every voxel (8 colours); PSUM also adds
// sum_q w_q P (row-major) of this thread's voxels to psum (with `quarters`, to
// its eight sums there).
//
// The voxel is a cube, so its shape gradients factor along its 12 edges:
// with corners o = ox + 2 oy + 4 oz and s(b) = 2 b - 1,
//   dN_o/dx at Gauss point q = s(ox) (1 + s(oy) c_y)(1 + s(oz) c_z) / (4 h),
// so du/dx at q is sum over the 4 x-edges e = oy + 2 oz of
// W[q][x][e] (u(1, oy, oz) - u(0, oy, oz)) (and likewise along y, z), and the
// corner force sum_q w_q P grad N_o is s(ox) T_x[e_x(o)] + s(oy) T_y[e_y(o)]
// + s(oz) T_z[e_z(o)] with the edge sums T_j[e] = sum_q W[q][j][e] w_q P[:, j].
// Same arithmetic content as the shape-gradient form, half the operations.
template <typename S, bool PSUM>
__device__ void voxel_forces(const RveArgs& R, const RveSmem<S>& s, const S* hH,
                             const MatParams* mats, double* psum, bool quarters = false) {
  const int n = R.n, nn = R.nn, hn = n >> 1, nc = hn * hn * hn;
  const S wq = S(R.h * R.h * R.h / 8.0);
  for (int color = 0; color < 8; ++color) {
    for (int t = threadIdx.x; t < nc; t += blockDim.x) {
      const int ex = 2 * (t % hn) + (color & 1);
      const int ey = 2 * ((t / hn) % hn) + ((color >> 1) & 1);
      const int ez = 2 * (t / (hn * hn)) + (color >> 2);
      const int x1 = ex + 1 == n ? 0 : ex + 1, y1 = ey + 1 == n ? 0 : ey + 1,
                z1 = ez + 1 == n ? 0 : ez + 1;
      int nd[8];
#pragma unroll
      for (int o = 0; o < 8; ++o) nd[o] = pidx((o & 1) ? x1 : ex, (o & 2) ? y1 : ey, (o & 4) ? z1 : ez, n);
      S D[3][4][3];  // edge differences [direction][edge][component]
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        S uc[8];
#pragma unroll
        for (int o = 0; o < 8; ++o) uc[o] = s.u[i * nn + nd[o]];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          // total displacement along the edge: fluctuation + h H e_j (the
          // weights of a direction sum to 1/h, so sum_e W D = H + grad w)
          const int b0 = e & 1, b1 = e >> 1;
          D[0][e][i] = (uc[1 + 2 * b0 + 4 * b1] - uc[2 * b0 + 4 * b1]) + hH[i * 3 + 0];
          D[1][e][i] = (uc[b0 + 2 + 4 * b1] - uc[b0 + 4 * b1]) + hH[i * 3 + 1];
          D[2][e][i] = (uc[b0 + 2 * b1 + 4] - uc[b0 + 2 * b1]) + hH[i * 3 + 2];
        }
      }
      const MatParams& mp = mats[s.mat[pidx(ex, ey, ez, n)]];
      S T[3][4][3];
      double* to = psum;
      if constexpr (PSUM && sizeof(S) == 4)
        if (quarters) to += ((color & 3) * 2 + t / kRveThreads) * 9;
      voxel_edge_sums<S, PSUM>(s.B, mp, D, wq, T, to);
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        const int ox = o & 1, oy = (o >> 1) & 1, oz = o >> 2;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const S tx = T[0][oy + 2 * oz][i], ty = T[1][ox + 2 * oz][i], tz = T[2][ox + 2 * oy][i];
          const S fo = (ox ? tx : -tx) + (oy ? ty : -ty) + (oz ? tz : -tz);
          s.f[i * nn + nd[o]] -= fo;
        }
      }
    }
    __syncthreads();
  }
}

__device__ inline double warp_max(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ inline double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Time-step scale, damping and residual scale of an instance.
__device__ __noinline__ void instance_scales(const RveArgs& R, const double* Hd, double* par) {
  double F[9], C[9];
  for (int k = 0; k < 9; ++k) F[k] = Hd[k] + (k % 4 == 0 ? 1.0 : 0.0);
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double c = 0;
      for (int k = 0; k < 3; ++k) c += F[k * 3 + i] * F[k * 3 + j];
      C[i * 3 + j] = c;
    }
  const double J = det3d(F);
  const double smin = sqrt(fmax(smallest_eigenvalue(C), 0.0));
  const double stiff = J > 0 ? fmax(0.0, -log(J)) : 0.0;
  double c2 = 0.0, cs = 1e300, mumax = 0.0, hmax = 0.0;
  for (int m = 0; m < R.nmat; ++m) {
    const double m2 = R.lam[m] + 2.0 * R.mu[m];
    const double t = R.kind[m] == AKB_MATERIAL_NEOHOOKEAN ? (m2 + 2.0 * R.lam[m] * stiff) / m2 : 1.0;
    c2 = fmax(c2, t);
    cs = fmin(cs, sqrt(R.mu[m] / m2));
    mumax = fmax(mumax, R.mu[m]);
  }
  for (int k = 0; k < 9; ++k) hmax = fmax(hmax, fabs(Hd[k]));
  par[0] = R.h * smin / sqrt(c2);
  par[1] = R.dampf * 2.0 * (2.0 * M_PI / R.L) * cs;
  par[2] = R.h * R.h * mumax * fmax(hmax, 1e-6);
}

// Edge weight W[q][direction][edge] (see voxel_forces), t = 12 q + 4 direction + edge.
template <typename S>
__device__ inline S edge_weight(const RveArgs& R, int t) {
  const int q = t / 12, j = (t / 4) % 3, e = t % 4;
  const double gp = 1.0 / sqrt(3.0);
  const double c[3] = {(q & 1) ? gp : -gp, (q & 2) ? gp : -gp, (q & 4) ? gp : -gp};
  const int d1 = j == 0 ? 1 : 0, d2 = j == 2 ? 1 : 2;  // the two other directions
  const double s1 = 2.0 * (e & 1) - 1.0, s2 = 2.0 * (e >> 1) - 1.0;
  return S((1.0 + s1 * c[d1]) * (1.0 + s2 * c[d2]) / (4.0 * R.h));
}

__device__ inline MatParams instance_material(const RveArgs& R, int k) {
  MatParams mp{};
  mp.kind = R.kind[k];
  mp.finite = R.kind[k] == AKB_MATERIAL_NEOHOOKEAN;
  mp.lambda = R.lam[k];
  mp.mu = R.mu[k];
  mp.E = 1.0;
  return mp;
}

// One RVE instance, by the whole CTA: relaxation from the instance's
// fluctuation (or zero), homogenised stress, state written back.
template <typename S>
__device__ __forceinline__ void rve_instance(const RveArgs& R, int64_t inst,
                                             const double* __restrict__ grad_u, S* fluct,
                                             double* __restrict__ stress, int32_t* iterations,
                                             double* residual, double* internal_force) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int nn = R.nn, tid = threadIdx.x, bs = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nwarps = bs >> 5;
  RveSmem<S> s = carve<S>(smem, nn);
  __shared__ MatParams mats[8];

  // the constant tables
  const S* im_g = static_cast<const S*>(R.inv_mass);
  for (int k = tid; k < nn; k += bs) {
    const int q = pidx(k % R.n, (k / R.n) % R.n, k / (R.n * R.n), R.n);
    s.im[q] = im_g[k];
    s.mat[q] = R.vmat[k];
  }
  if (tid < 96) s.B[tid] = edge_weight<S>(R, tid);
  if (tid < R.nmat) mats[tid] = instance_material(R, tid);
  __shared__ S hH[9];  // h H, row-major
  double Hd[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Hd[i * 3 + j] = grad_u[inst * 9 + i + 3 * j];
  if (tid < 9) hH[tid] = S(R.h * Hd[tid]);
  if (tid == 0) {
    instance_scales(R, Hd, s.par);
  }
  __syncthreads();
  const double fscale = s.par[2];

  // Relaxation; an attempt whose residual turns non-finite or exceeds
  // kDivergence restarts from the initial state with a 0.6x time step.
  int total = 0, k = 0;
  double r = 0.0, tsf = R.tsf;
  for (int attempt = 0;; ++attempt, tsf *= kRestartFactor) {
    for (int idx = tid; idx < 3 * nn; idx += bs) {
      const int node = idx / 3, i = idx - 3 * node;
      const int q = pidx(node % R.n, (node / R.n) % R.n, node / (R.n * R.n), R.n);
      s.u[i * nn + q] = fluct ? fluct[inst * 3 * nn + idx] : S(0);
      s.v[idx] = 0;
    }
    const double dtd = tsf * s.par[0];
    const S dt = S(dtd);
    const S a1 = S(1.0 - 0.5 * s.par[1] * dtd), a2 = S(1.0 + 0.5 * s.par[1] * dtd);
    __syncthreads();
    bool diverged = false;
    for (k = 0;; ++k) {
      for (int idx = tid; idx < 3 * nn; idx += bs) s.f[idx] = 0;
      __syncthreads();
      voxel_forces<S, false>(R, s, hH, mats, nullptr);
      const bool last = k >= R.max_it;
      if (last || (R.check > 0 && k % R.check == 0)) {
        double lm = 0.0;
        for (int idx = tid; idx < 3 * nn; idx += bs) {
          const double x = double(s.f[idx]);
          lm = isfinite(x) ? fmax(lm, fabs(x)) : INFINITY;
        }
        lm = warp_max(lm);
        if (lane == 0) s.red[warp] = lm;
        __syncthreads();
        double m = 0.0;
        for (int w = 0; w < nwarps; ++w) m = fmax(m, s.red[w]);
        r = isfinite(m) ? m / fscale : INFINITY;
        __syncthreads();  // s.red is reused
        diverged = !(r <= kDivergence);
        if (last || diverged || (R.tol >= 0 && r <= R.tol)) break;
      }
      for (int idx = tid; idx < 3 * nn; idx += bs) {
        const int node = idx % nn;
        const S vv = (a1 * s.v[idx] + dt * s.f[idx] * s.im[node]) / a2;
        s.v[idx] = vv;
        s.u[idx] += dt * vv;
      }
      __syncthreads();
    }
    total += k;
    if (!diverged || attempt >= kMaxRestarts) break;
    __syncthreads();
  }

  // homogenised stress (and force) of the final state
  for (int idx = tid; idx < 3 * nn; idx += bs) s.f[idx] = 0;
  __syncthreads();
  const bool quarters = sums_by_quarters<S>(R.n);
  constexpr int kSums = sizeof(S) == 4 ? kQuarterSums : 1;
  double ps[kSums * 9];
#pragma unroll
  for (int q = 0; q < kSums * 9; ++q) ps[q] = 0.0;
  voxel_forces<S, true>(R, s, hH, mats, ps, quarters);
  // the warps' sums: of all voxels, or [colour mod 4][32 consecutive places] (the
  // velocities are done with)
  double* sums = quarters ? reinterpret_cast<double*>(s.v) : s.red;
#pragma unroll
  for (int j = 0; j < kSums; ++j) {
    if (j > 0 && !quarters) break;
    const int at = quarters ? (j >> 1) * 16 + (j & 1) * 8 + warp : warp;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const double x = warp_sum(ps[j * 9 + q]);
      if (lane == 0) sums[at * 9 + q] = x;
    }
  }
  __syncthreads();
  if (tid < 9) {
    double t = 0.0;
    if (quarters) {
      for (int z = 0; z < 4; ++z) {
        double tz = 0.0;
        for (int w = 0; w < 16; ++w) tz += sums[((w >> 2) * 16 + z * 4 + (w & 3)) * 9 + tid];
        t += tz;
      }
    } else {
      for (int w = 0; w < nwarps; ++w) t += sums[w * 9 + tid];
    }
    const int i = tid / 3, j = tid % 3;
    stress[inst * 9 + i + 3 * j] = t / (R.L * R.L * R.L);
  }
  if (tid == 0) {
    if (iterations) iterations[inst] = total;
    if (residual) residual[inst] = r;
  }
  for (int idx = tid; idx < 3 * nn; idx += bs) {
    const int node = idx / 3, i = idx - 3 * node;
    const int q = pidx(node % R.n, (node / R.n) % R.n, node / (R.n * R.n), R.n);
    if (fluct && R.write_fluct) fluct[inst * 3 * nn + idx] = s.u[i * nn + q];
    if (internal_force) internal_force[inst * 3 * nn + idx] = double(s.f[i * nn + q]);
  }
}

template <typename S>
__global__ void __launch_bounds__(kRveThreads, 1)
    k_rve(RveArgs R, int64_t nb, const double* __restrict__ grad_u, S* fluct,
          double* __restrict__ stress, int32_t* iterations, double* residual,
          double* internal_force) {
  const int64_t inst = blockIdx.x;
  if (inst >= nb) return;
  rve_instance<S>(R, inst, grad_u, fluct, stress, iterations, residual, internal_force);
}

// The instances index[0 .. min(*count, capacity)) of arrays over all points,
// the count read on the device (written by an earlier kernel on the same
// stream): CTAs stride over the list, so a short or empty list costs one
// small launch and no host round trip.
template <typename S>
__global__ void __launch_bounds__(kRveThreads, 1)
    k_rve_indexed(RveArgs R, int64_t capacity, const int32_t* __restrict__ index,
                  const int32_t* __restrict__ count, const double* __restrict__ grad_u, S* fluct,
                  double* __restrict__ stress, int32_t* iterations, double* residual) {
  const int64_t n = min((int64_t)*count, capacity);
  for (int64_t b = blockIdx.x; b < n; b += gridDim.x) {
    const int64_t inst = index[b];
    if (inst < 0 || inst >= capacity) continue;  // uniform over the CTA
    rve_instance<S>(R, inst, grad_u, fluct, stress, iterations, residual, nullptr);
    __syncthreads();  // shared state is reused by the next instance
  }
}

// ------------------------------------------------------- one RVE per cluster
// FP32 RVEs are relaxed by a cluster of C CTAs, each owning n / C planes of
// voxels and nodes (C = 1, 2 or 4: at most 1024 voxels a CTA). Bound by FP32
// issue, and for small batches by the slowest instance (of 512 random
// gradients it takes 1500-2200 updates against 260 on average), so an update
// has to be short as well as cheap. Two changes against one CTA per RVE:
//  - the corner forces of every voxel go to shared memory (96 bytes a voxel)
//    and each node then adds its 8 voxels' in colour order, the order in which
//    the coloured scatter added them (the same sums bit for bit), so that a
//    step is two cluster barriers instead of ten CTA barriers and all voxels
//    are computed at once: 16 warps of 128 registers instead of 8 of 227. The
//    edge differences, edge sums and stresses of a voxel do not fit 128: 324 to
//    340 bytes a thread are spilled (220 with one CTA), 548 to 576 (348) read back;
//  - the planes are spread over C SMs. A CTA reads the forces of the layer
//    below its first plane, and writes the displacements of that plane, in the
//    neighbour's shared memory.
//
// With four CTAs per RVE the layers' exchange costs a cluster 8 to 12 % of its
// rate against a whole RVE per SM (k_rve, the same bits), and what it gains is
// the time of the slowest instances at the end. From this many instances on,
// k_rve. Random gradients up to 0.3 (mean of five draws), ms by clusters and by
// k_rve: 512 74 and 100, 1024 137 and 154, 2048 272 and 289, 2560 334 and 334,
// 3072 398 and 376, 4096 531 and 505; of gradients up to 0.06, which all take
// about the same number of updates, 512 43 and 43, 1024 85 and 77, 2048 171 and 152.
// (Fewer CTAs per RVE are faster at any count: 4096 of 8^3 76 -> 28 ms.)
constexpr int64_t kManyInstances = 2560;
// Calls without updates (akb_rve_stress) have no slowest instance: four CTAs per
// RVE are faster only while few waves of clusters hold them all. 16^3, us by
// clusters and by k_rve: 20 states 98 and 196, 72 190 and 196, 100 236 and 204,
// 1000 1600 and 1130.
constexpr int kStressWaves = 2;

struct ClusterLayout {
  int u, v, im, B, F, mat, red, total;  // byte offsets
};
__host__ __device__ inline ClusterLayout cluster_layout(int n, int C) {
  const int nl = n * n * n / C, halo = C > 1 ? n * n : 0;
  ClusterLayout s;
  s.u = 0;
  s.v = s.u + 4 * 3 * (nl + halo);
  s.im = s.v + 4 * 3 * nl;
  s.B = s.im + 4 * nl;
  s.F = s.B + 4 * 96;
  s.mat = s.F + 4 * 24 * nl;
  s.red = (s.mat + nl + 15) & ~15;
  // 16 warps x 9, the CTAs' sums (4 x 9) and maxima (2 x 4), 3 scales
  s.total = s.red + 8 * (16 * 9 + 4 * 9 + 8 + 4);
  return s;
}

template <int C>
__device__ inline void cluster_sync() {
  if constexpr (C == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}
// The address of this CTA's shared-memory address a in CTA `rank` of the cluster.
__device__ inline uint32_t remote(uint32_t a, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ inline float ld_remote(uint32_t a) {
  float x;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(a) : "memory");
  return x;
}
__device__ inline void st_remote(uint32_t a, float x) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(x) : "memory");
}
__device__ inline void st_remote(uint32_t a, double x) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(x) : "memory");
}

// One instance, by the whole cluster.
template <int C>
__device__ __forceinline__ void rve_cluster_instance(const RveArgs& R, int rank, int64_t inst,
                                                     const double* __restrict__ grad_u, float* fluct,
                                                     double* __restrict__ stress,
                                                     int32_t* iterations, double* residual,
                                                     double* internal_force) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ MatParams mats[8];
  __shared__ float hH[9];
  const int n = R.n, nn = R.nn, hn = n >> 1, plane = n * n, nl = nn / C, Zs = n / C;
  const int z0 = rank * Zs, cls = nl >> 3, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const ClusterLayout lay = cluster_layout(n, C);
  float* u = reinterpret_cast<float*>(smem + lay.u);  // [3][nl + halo]
  float* v = reinterpret_cast<float*>(smem + lay.v);  // [3][nl]
  float* im = reinterpret_cast<float*>(smem + lay.im);
  float* B = reinterpret_cast<float*>(smem + lay.B);
  float* F = reinterpret_cast<float*>(smem + lay.F);  // [corner][component][nl]
  uint8_t* mat = smem + lay.mat;
  double* red = reinterpret_cast<double*>(smem + lay.red);
  double *csum = red + 16 * 9, *cmax = csum + 4 * 9, *par = cmax + 8;
  const int US = nl + (C > 1 ? plane : 0);
  const int below = (rank + C - 1) % C;
  // position of node (or voxel) (x, y, z0 + z): by parity class as pidx; the
  // plane above the CTA's (the next CTA's first) follows
  auto at = [&](int x, int y, int z) {
    if (C > 1 && z == Zs) return nl + ((x & 1) | ((y & 1) << 1)) * (hn * hn) + (x >> 1) + hn * (y >> 1);
    return ((x & 1) | ((y & 1) << 1) | ((z & 1) << 2)) * cls + (x >> 1) + hn * ((y >> 1) + hn * (z >> 1));
  };
  // this thread's voxels and nodes: positions tid + m kClusterThreads < nl, and
  // their (x, y, z), packed
  constexpr int kNodes = (kClusterVoxels + kClusterThreads - 1) / kClusterThreads;
  int xyz[kNodes];
#pragma unroll
  for (int m = 0; m < kNodes; ++m) {
    const int k = tid + m * kClusterThreads, c = k / cls, t = k - c * cls;
    xyz[m] = (2 * (t % hn) + (c & 1)) | (2 * ((t / hn) % hn) + ((c >> 1) & 1)) << 8 |
             (2 * (t / (hn * hn)) + (c >> 2)) << 16;
  }

  for (int k = tid; k < nl; k += kClusterThreads) {
    const int x = k % n, y = (k / n) % n, z = k / plane, g = k + z0 * plane;
    im[at(x, y, z)] = static_cast<const float*>(R.inv_mass)[g];
    mat[at(x, y, z)] = R.vmat[g];
  }
  if (tid < 96) B[tid] = edge_weight<float>(R, tid);
  if (tid < R.nmat) mats[tid] = instance_material(R, tid);
  double Hd[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Hd[i * 3 + j] = grad_u[inst * 9 + i + 3 * j];
  if (tid < 9) hH[tid] = float(R.h * grad_u[inst * 9 + tid / 3 + 3 * (tid % 3)]);
  if (tid == 0) instance_scales(R, Hd, par);
  __syncthreads();
  const double fscale = par[2];
  const float wq = float(R.h * R.h * R.h / 8.0);

  // corner forces of the CTA's voxels into F
  auto voxels = [&](auto psum_tag, double* psum) {
    constexpr bool PSUM = decltype(psum_tag)::value;
#pragma unroll 1
    for (int m = 0; m < kNodes; ++m) {
      const int k = tid + m * kClusterThreads;
      if (k >= nl) break;
      int pk = xyz[0];
#pragma unroll
      for (int j = 1; j < kNodes; ++j) pk = m == j ? xyz[j] : pk;
      const int ex = pk & 255, ey = (pk >> 8) & 255, ez = pk >> 16;
      const int x1 = ex + 1 == n ? 0 : ex + 1, y1 = ey + 1 == n ? 0 : ey + 1,
                z1 = C == 1 && ez + 1 == n ? 0 : ez + 1;
      int nd[8];
#pragma unroll
      for (int o = 0; o < 8; ++o) nd[o] = at((o & 1) ? x1 : ex, (o & 2) ? y1 : ey, (o & 4) ? z1 : ez);
      float D[3][4][3];  // edge differences [direction][edge][component]
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        float uc[8];
#pragma unroll
        for (int o = 0; o < 8; ++o) uc[o] = u[i * US + nd[o]];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int b0 = e & 1, b1 = e >> 1;
          D[0][e][i] = (uc[1 + 2 * b0 + 4 * b1] - uc[2 * b0 + 4 * b1]) + hH[i * 3 + 0];
          D[1][e][i] = (uc[b0 + 2 + 4 * b1] - uc[b0 + 4 * b1]) + hH[i * 3 + 1];
          D[2][e][i] = (uc[b0 + 2 * b1 + 4] - uc[b0 + 2 * b1]) + hH[i * 3 + 2];
        }
      }
      float T[3][4][3];
      voxel_edge_sums<float, PSUM>(B, mats[mat[k]], D, wq, T, psum);
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        const int ox = o & 1, oy = (o >> 1) & 1, oz = o >> 2;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const float tx = T[0][oy + 2 * oz][i], ty = T[1][ox + 2 * oz][i], tz = T[2][ox + 2 * oy][i];
          F[(o * 3 + i) * nl + k] = (ox ? tx : -tx) + (oy ? ty : -ty) + (oz ? tz : -tz);
        }
      }
    }
  };
  // the force of the CTA's node at position k: its voxels' in colour order
  const uint32_t F_below = C > 1 ? remote((uint32_t)__cvta_generic_to_shared(F), below) : 0;
  auto force = [&](int x, int y, int z, float* f) {
    f[0] = f[1] = f[2] = 0.0f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const bool hx = (x & 1) != (c & 1), hy = (y & 1) != ((c >> 1) & 1), hz = (z & 1) != (c >> 2);
      const int vx = hx ? (x == 0 ? n - 1 : x - 1) : x, vy = hy ? (y == 0 ? n - 1 : y - 1) : y;
      const int vz = hz ? (z == 0 ? Zs - 1 : z - 1) : z;
      const int o = (hx ? 1 : 0) + (hy ? 2 : 0) + (hz ? 4 : 0);
      const int w = o * 3 * nl + at(vx, vy, vz);
#pragma unroll
      for (int i = 0; i < 3; ++i)
        f[i] -= C > 1 && hz && z == 0 ? ld_remote(F_below + 4 * (w + i * nl)) : F[w + i * nl];
    }
  };

  int total = 0, k = 0;
  double r = 0.0, tsf = R.tsf;
  for (int attempt = 0;; ++attempt, tsf *= kRestartFactor) {
    for (int idx = tid; idx < 3 * US; idx += kClusterThreads) {
      const int node = idx / 3, i = idx - 3 * node;
      const int x = node % n, y = (node / n) % n, z = node / plane;
      const int64_t g = (int64_t)((z0 + z) % n) * plane + node % plane;
      u[i * US + at(x, y, z)] = fluct ? fluct[inst * 3 * nn + 3 * g + i] : 0.0f;
      if (z < Zs) v[idx] = 0.0f;
    }
    const double dtd = tsf * par[0];
    const float dt = float(dtd);
    const float a1 = float(1.0 - 0.5 * par[1] * dtd), a2 = float(1.0 + 0.5 * par[1] * dtd);
    __syncthreads();
    bool diverged = false;
    for (k = 0;; ++k) {
      voxels(std::false_type{}, nullptr);
      cluster_sync<C>();  // every corner force is written
      float f[kNodes][3];
#pragma unroll
      for (int m = 0; m < kNodes; ++m) {
        const int q = tid + m * kClusterThreads;
        if (q < nl) {
          force(xyz[m] & 255, (xyz[m] >> 8) & 255, xyz[m] >> 16, f[m]);
        }
      }
      const bool last = k >= R.max_it;
      if (last || (R.check > 0 && k % R.check == 0)) {
        double lm = 0.0;
#pragma unroll
        for (int m = 0; m < kNodes; ++m)
          if (tid + m * kClusterThreads < nl)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              const double x = double(f[m][i]);
              lm = isfinite(x) ? fmax(lm, fabs(x)) : INFINITY;
            }
        lm = warp_max(lm);
        if (lane == 0) red[warp] = lm;
        __syncthreads();
        if (tid < C) {
          double m = 0.0;
          for (int w = 0; w < kClusterThreads / 32; ++w) m = fmax(m, red[w]);
          if constexpr (C == 1)
            cmax[0] = m;
          else
            st_remote(remote((uint32_t)__cvta_generic_to_shared(cmax + rank), tid), m);
        }
        cluster_sync<C>();
        double m = 0.0;
        for (int w = 0; w < C; ++w) m = fmax(m, cmax[w]);
        r = isfinite(m) ? m / fscale : INFINITY;
        diverged = !(r <= kDivergence);
        if (last || diverged || (R.tol >= 0 && r <= R.tol)) break;
      }
#pragma unroll
      for (int m = 0; m < kNodes; ++m) {
        const int q = tid + m * kClusterThreads;
        if (q < nl) {
          const float imq = im[q];
          const int x = xyz[m] & 255, y = (xyz[m] >> 8) & 255, z = xyz[m] >> 16;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const float vv =
                __fmaf_rn(a1, v[i * nl + q], __fmul_rn(__fmul_rn(dt, f[m][i]), imq)) / a2;
            v[i * nl + q] = vv;
            const float un = __fmaf_rn(dt, vv, u[i * US + q]);
            u[i * US + q] = un;
            if (C > 1 && z == 0)  // the plane above the CTA below
              st_remote(remote((uint32_t)__cvta_generic_to_shared(u + i * US + at(x, y, Zs)), below), un);
          }
        }
      }
      cluster_sync<C>();  // every displacement is written
    }
    total += k;
    if (!diverged || attempt >= kMaxRestarts) break;
    cluster_sync<C>();
  }

  // homogenised stress (and force) of the final state
  double ps[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) ps[q] = 0.0;
  cluster_sync<C>();  // the forces of the last update are read
  voxels(std::true_type{}, ps);
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    const double x = warp_sum(ps[q]);
    if (lane == 0) red[warp * 9 + q] = x;
  }
  __syncthreads();
  if (tid < 9) {
    double t = 0.0;
    for (int w = 0; w < kClusterThreads / 32; ++w) t += red[w * 9 + tid];
    if constexpr (C == 1)
      csum[tid] = t;
    else
      st_remote(remote((uint32_t)__cvta_generic_to_shared(csum + rank * 9 + tid), 0), t);
  }
  cluster_sync<C>();
  if (rank == 0 && tid < 9) {
    double t = 0.0;
    for (int w = 0; w < C; ++w) t += csum[w * 9 + tid];
    const int i = tid / 3, j = tid % 3;
    stress[inst * 9 + i + 3 * j] = t / (R.L * R.L * R.L);
  }
  if (rank == 0 && tid == 0) {
    if (iterations) iterations[inst] = total;
    if (residual) residual[inst] = r;
  }
#pragma unroll
  for (int m = 0; m < kNodes; ++m) {
    const int q = tid + m * kClusterThreads;
    if (q >= nl) break;
    const int x = xyz[m] & 255, y = (xyz[m] >> 8) & 255, z = xyz[m] >> 16;
    const int64_t g = inst * 3 * nn + 3 * ((int64_t)(z0 + z) * plane + y * n + x);
    if (fluct && R.write_fluct)
#pragma unroll
      for (int i = 0; i < 3; ++i) fluct[g + i] = u[i * US + q];
    if (internal_force) {
      float f[3];
      force(x, y, z, f);
#pragma unroll
      for (int i = 0; i < 3; ++i) internal_force[g + i] = double(f[i]);
    }
  }
  cluster_sync<C>();  // no CTA leaves (or reuses its memory) while another reads it
}

__device__ inline int cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}

// The instances [0, nb), or with INDEXED index[0 .. min(*count, nb)), the count
// read on the device: clusters stride over them.
template <int C, bool INDEXED>
__global__ void __launch_bounds__(kClusterThreads, 1)
    k_rve_cluster(RveArgs R, int64_t nb, const int32_t* __restrict__ index,
                  const int32_t* __restrict__ count, const double* __restrict__ grad_u,
                  float* fluct, double* __restrict__ stress, int32_t* iterations, double* residual,
                  double* internal_force) {
  const int rank = C == 1 ? 0 : cluster_rank();
  grid_wait();  // whatever the stream did before has completed
  const int64_t n = INDEXED ? min((int64_t)*count, nb) : nb;
  for (int64_t b = blockIdx.x / C; b < n; b += gridDim.x / C) {
    const int64_t inst = INDEXED ? index[b] : b;
    if (inst < 0 || inst >= nb) continue;  // uniform over the cluster
    rve_cluster_instance<C>(R, rank, inst, grad_u, fluct, stress, iterations, residual,
                            internal_force);
  }
}

std::mutex g_rve_attr_mutex;

template <typename S>
cudaError_t raise_limit(size_t bytes) {
  std::lock_guard<std::mutex> lock(g_rve_attr_mutex);
  cudaFuncAttributes attr;
  cudaError_t e = cudaFuncGetAttributes(&attr, k_rve<S>);
  if (e != cudaSuccess) return e;
  if ((size_t)attr.maxDynamicSharedSizeBytes >= bytes) return cudaSuccess;
  e = cudaFuncSetAttribute(k_rve<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_rve_indexed<S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)bytes);
}

template <int C>
cudaLaunchConfig_t cluster_config(int n, int64_t clusters, cudaLaunchAttribute* at) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * C));
  cfg.blockDim = dim3(kClusterThreads);
  cfg.dynamicSmemBytes = cluster_layout(n, C).total;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = C;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// *resident: the clusters the device runs at once. It can be fewer than SMs / C:
// a cluster's CTAs sit in one GPC, whose SM count C need not divide.
template <int C>
cudaError_t configure_cluster(int n, int* resident) {
  std::lock_guard<std::mutex> lock(g_rve_attr_mutex);
  const int bytes = cluster_layout(n, C).total;
  const void* kernels[2] = {(const void*)k_rve_cluster<C, false>, (const void*)k_rve_cluster<C, true>};
  for (const void* k : kernels) {
    cudaFuncAttributes attr;
    cudaError_t e = cudaFuncGetAttributes(&attr, k);
    if (e == cudaSuccess && attr.maxDynamicSharedSizeBytes < bytes)
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = cluster_config<C>(n, 1, &at);
  return cudaOccupancyMaxActiveClusters(resident, k_rve_cluster<C, true>, &cfg);
}
cudaError_t configure_cluster(int n, int* resident) {
  switch (cluster_of(n)) {
  case 1: return configure_cluster<1>(n, resident);
  case 2: return configure_cluster<2>(n, resident);
  case 4: return configure_cluster<4>(n, resident);
  default: return cudaSuccess;
  }
}

// `clusters` clusters over nb instances (or the listed ones of them).
template <int C, bool INDEXED>
cudaError_t launch_cluster(const RveArgs& a, int64_t clusters, int64_t nb, const int32_t* index,
                           const int32_t* count, const double* grad_u, float* fluct, double* stress,
                           int32_t* iterations, double* residual, double* force, cudaStream_t s) {
  cudaLaunchAttribute at[2];
  cudaLaunchConfig_t cfg = cluster_config<C>(a.n, std::min<int64_t>(clusters, INT32_MAX / C), at);
  cfg.stream = s;
  // the launch itself overlaps the kernel before it: most lists are empty
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, k_rve_cluster<C, INDEXED>, a, nb, index, count, grad_u, fluct,
                            stress, iterations, residual, force);
}
template <bool INDEXED>
cudaError_t launch_cluster(int C, const RveArgs& a, int64_t clusters, int64_t nb,
                           const int32_t* index, const int32_t* count, const double* grad_u,
                           void* fluct, double* stress, int32_t* iterations, double* residual,
                           double* force, cudaStream_t s) {
  float* w = static_cast<float*>(fluct);
  switch (C) {
  case 1: return launch_cluster<1, INDEXED>(a, clusters, nb, index, count, grad_u, w, stress,
                                            iterations, residual, force, s);
  case 2: return launch_cluster<2, INDEXED>(a, clusters, nb, index, count, grad_u, w, stress,
                                            iterations, residual, force, s);
  default: return launch_cluster<4, INDEXED>(a, clusters, nb, index, count, grad_u, w, stress,
                                             iterations, residual, force, s);
  }
}

RveArgs args_of(const akb_rve* r, int max_it) {
  RveArgs a{};
  a.n = r->n;
  a.nn = r->n * r->n * r->n;
  a.nmat = r->nmat;
  a.max_it = max_it;
  a.write_fluct = max_it > 0;
  a.check = r->check;
  a.L = r->L;
  a.h = r->L / r->n;
  a.tol = r->tol;
  a.tsf = r->tsf;
  a.dampf = r->dampf;
  for (int m = 0; m < 8; ++m) {
    a.lam[m] = r->lam[m];
    a.mu[m] = r->mu[m];
    a.kind[m] = r->kind[m];
  }
  a.vmat = r->d_vmat;
  a.inv_mass = r->d_inv_mass;
  return a;
}

akb_status launch(akb_rve* r, int max_it, int64_t nb, const double* grad_u, void* fluct,
                  double* stress, int32_t* iterations, double* residual, double* force,
                  void* stream) {
  if (!r) return fail(AKB_ERR_INVALID_ARGUMENT, "null RVE");
  if (nb < 0 || (nb > 0 && (!grad_u || !stress)))
    return fail(AKB_ERR_INVALID_ARGUMENT, "grad_u and stress are required");
  if (nb > INT32_MAX) return fail(AKB_ERR_UNSUPPORTED, "more than 2^31 RVEs in one call");
  if (nb == 0) return AKB_OK;
  AKB_CUDA_TRY(cudaSetDevice(r->device));
  cudaStream_t s = stream ? (cudaStream_t)stream : r->stream;
  const RveArgs a = args_of(r, max_it);
  if (r->mode == AKB_MODE_FP64)
    k_rve<double><<<(unsigned)nb, kRveThreads, r->smem, s>>>(
        a, nb, grad_u, static_cast<double*>(fluct), stress, iterations, residual, force);
  else if (const int C = cluster_of(r->n);
           C && (C < 4 || nb < (max_it ? kManyInstances : kStressWaves * r->clusters + 1)))
    AKB_CUDA_TRY(launch_cluster<false>(C, a, nb, nb, nullptr, nullptr, grad_u, fluct, stress,
                                       iterations, residual, force, s));
  else
    k_rve<float><<<(unsigned)nb, kRveThreads, r->smem, s>>>(
        a, nb, grad_u, static_cast<float*>(fluct), stress, iterations, residual, force);
  AKB_CUDA_TRY(cudaGetLastError());
  return AKB_OK;
}

}  // namespace
}  // namespace akb

using namespace akb;

extern "C" {

akb_status akb_rve_create(const akb_rve_desc* desc, const akb_rve_options* options,
                          akb_rve** out) {
  if (!out) return fail(AKB_ERR_INVALID_ARGUMENT, "null output handle");
  *out = nullptr;
  if (!desc || !desc->voxel_material || !desc->materials)
    return fail(AKB_ERR_INVALID_ARGUMENT, "RVE description, voxels and materials are required");
  const int n = desc->cells;
  if (n < 2 || n > 64 || (n & 1)) return fail(AKB_ERR_INVALID_ARGUMENT, "cells must be even, 2..64");
  if (desc->nb_materials < 1 || desc->nb_materials > 8)
    return fail(AKB_ERR_INVALID_ARGUMENT, "1..8 materials");
  if (!(desc->length > 0)) return fail(AKB_ERR_INVALID_ARGUMENT, "length must be positive");
  akb_rve_options opt{AKB_MODE_FP32_BULK, 0, nullptr, 0, 0, 0.0, 0.0, 0.0};
  if (options) opt = *options;
  if (opt.precision_mode != AKB_MODE_FP32_BULK && opt.precision_mode != AKB_MODE_FP64)
    return fail(AKB_ERR_UNSUPPORTED, "RVE precision: AKB_MODE_FP32_BULK or AKB_MODE_FP64");
  auto r = std::make_unique<akb_rve>();
  r->mode = opt.precision_mode;
  r->n = n;
  r->nmat = desc->nb_materials;
  r->L = desc->length;
  r->max_it = opt.max_iterations > 0 ? opt.max_iterations : 2000;
  r->check = opt.check_interval > 0 ? opt.check_interval : 10;
  r->tol = opt.tolerance != 0.0 ? opt.tolerance : 1e-4;
  r->tsf = opt.time_step_factor > 0 ? opt.time_step_factor : 0.6;
  r->dampf = opt.damping_factor > 0 ? opt.damping_factor : 0.6;
  for (int m = 0; m < r->nmat; ++m) {
    const akb_material_desc& md = desc->materials[m];
    if (md.kind != AKB_MATERIAL_ELASTIC && md.kind != AKB_MATERIAL_NEOHOOKEAN)
      return fail(AKB_ERR_UNSUPPORTED, "RVE materials: elastic or neo-Hookean");
    if (!(md.E > 0) || !(md.nu > -1.0 && md.nu < 0.5))
      return fail(AKB_ERR_INVALID_ARGUMENT, "RVE material needs E > 0, -1 < nu < 0.5");
    r->kind[m] = md.kind;
    r->lam[m] = md.nu * md.E / ((1 + md.nu) * (1 - 2 * md.nu));
    r->mu[m] = md.E / (2 * (1 + md.nu));
  }
  const int64_t nn = (int64_t)n * n * n;
  for (int64_t e = 0; e < nn; ++e)
    if (desc->voxel_material[e] >= r->nmat)
      return fail(AKB_ERR_INVALID_ARGUMENT, "voxel material index out of range");
  r->smem = r->mode == AKB_MODE_FP64 ? rve_smem_bytes<double>((int)nn) : rve_smem_bytes<float>((int)nn);
  if (r->smem > 227 * 1024)
    return fail(AKB_ERR_UNSUPPORTED, "RVE does not fit in one SM's shared memory (use FP32 or fewer cells)");
  // lumped fictitious mass: density lambda + 2 mu, h^3/8 per voxel corner
  const double h = r->L / n;
  std::vector<double> mass(nn, 0.0);
  for (int ez = 0; ez < n; ++ez)
    for (int ey = 0; ey < n; ++ey)
      for (int ex = 0; ex < n; ++ex) {
        const int m = desc->voxel_material[ex + n * (ey + n * ez)];
        r->vf[m] += 1.0 / (double)nn;
        for (int a = 0; a < 8; ++a) {
          const int x = (ex + corner_x(a)) % n, y = (ey + corner_y(a)) % n, z = (ez + corner_z(a)) % n;
          mass[x + n * (y + n * z)] += (r->lam[m] + 2.0 * r->mu[m]) * h * h * h / 8.0;
        }
      }
  r->device = opt.device;
  AKB_CUDA_TRY(cudaSetDevice(r->device));
  if (opt.stream) {
    r->stream = (cudaStream_t)opt.stream;
  } else {
    AKB_CUDA_TRY(cudaStreamCreateWithFlags(&r->stream, cudaStreamNonBlocking));
    r->owns_stream = true;
  }
  AKB_CUDA_TRY(cudaMalloc((void**)&r->d_vmat, nn));
  AKB_CUDA_TRY(cudaMemcpy(r->d_vmat, desc->voxel_material, nn, cudaMemcpyHostToDevice));
  if (r->mode == AKB_MODE_FP64) {
    std::vector<double> im(nn);
    for (int64_t k = 0; k < nn; ++k) im[k] = 1.0 / mass[k];
    AKB_CUDA_TRY(cudaMalloc(&r->d_inv_mass, nn * sizeof(double)));
    AKB_CUDA_TRY(cudaMemcpy(r->d_inv_mass, im.data(), nn * sizeof(double), cudaMemcpyHostToDevice));
    AKB_CUDA_TRY(raise_limit<double>(r->smem));
  } else {
    std::vector<float> im(nn);
    for (int64_t k = 0; k < nn; ++k) im[k] = (float)(1.0 / mass[k]);
    AKB_CUDA_TRY(cudaMalloc(&r->d_inv_mass, nn * sizeof(float)));
    AKB_CUDA_TRY(cudaMemcpy(r->d_inv_mass, im.data(), nn * sizeof(float), cudaMemcpyHostToDevice));
    AKB_CUDA_TRY(raise_limit<float>(r->smem));
    AKB_CUDA_TRY(configure_cluster(n, &r->clusters));
  }
  *out = r.release();
  return AKB_OK;
}

akb_status akb_rve_destroy(akb_rve* r) {
  if (!r) return AKB_OK;
  cudaSetDevice(r->device);
  cudaStreamSynchronize(r->stream);
  cudaFree(r->d_vmat);
  cudaFree(r->d_inv_mass);
  if (r->owns_stream) cudaStreamDestroy(r->stream);
  delete r;
  return AKB_OK;
}

akb_status akb_rve_get_info(const akb_rve* r, akb_rve_info* info) {
  if (!r || !info) return fail(AKB_ERR_INVALID_ARGUMENT, "null argument");
  info->cells = r->n;
  info->precision_mode = r->mode;
  info->nb_nodes = (int64_t)r->n * r->n * r->n;
  for (int m = 0; m < 8; ++m) info->volume_fraction[m] = r->vf[m];
  info->shared_bytes = (int64_t)r->smem;
  return AKB_OK;
}

akb_status akb_rve_solve(akb_rve* r, int64_t nb, const double* grad_u, void* fluctuation,
                         double* stress, int32_t* iterations, double* residual, void* stream) {
  if (!r) return fail(AKB_ERR_INVALID_ARGUMENT, "null RVE");
  return launch(r, r->max_it, nb, grad_u, fluctuation, stress, iterations, residual, nullptr,
                stream);
}

akb_status akb_rve_solve_indexed(akb_rve* r, int64_t capacity, const int32_t* index,
                                 const int32_t* count, const double* grad_u, void* fluctuation,
                                 double* stress, int32_t* iterations, double* residual,
                                 void* stream) {
  if (!r) return fail(AKB_ERR_INVALID_ARGUMENT, "null RVE");
  if (capacity < 0 || (capacity > 0 && (!index || !count || !grad_u || !stress)))
    return fail(AKB_ERR_INVALID_ARGUMENT, "index, count, grad_u and stress are required");
  if (capacity > INT32_MAX) return fail(AKB_ERR_UNSUPPORTED, "more than 2^31 RVEs in one call");
  if (capacity == 0) return AKB_OK;
  AKB_CUDA_TRY(cudaSetDevice(r->device));
  cudaStream_t s = stream ? (cudaStream_t)stream : r->stream;
  int sms = 0;
  AKB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device));
  const unsigned grid = (unsigned)std::min<int64_t>(capacity, std::max(sms, 1));
  const RveArgs a = args_of(r, r->max_it);
  if (r->mode == AKB_MODE_FP64)
    k_rve_indexed<double><<<grid, kRveThreads, r->smem, s>>>(
        a, capacity, index, count, grad_u, static_cast<double*>(fluctuation), stress, iterations,
        residual);
  else if (const int C = cluster_of(r->n))
    // no more clusters than run at once: the rest would start when one of these
    // has worked off its whole share (37 clusters of four where fewer fit: 32768
    // listed 16^3 RVEs 7388 ms, the resident ones 4349; an empty list in a macro
    // step of 32^3 cells 228 -> 226 us). Long lists stay with the clusters: the
    // host does not know the length, and a second, mostly empty launch of
    // k_rve_indexed costs every macro step 1.5 to 2.5 us. Strong gradients, as
    // they leave a surrogate's envelope: 4096 listed 571 ms by clusters, 582 by
    // k_rve_indexed, 16384 2199 and 2183; equal small ones 340 and 325, 1358 and 1275.
    AKB_CUDA_TRY(launch_cluster<true>(C, a, std::min<int64_t>(capacity, std::max(r->clusters, 1)),
                                      capacity, index, count, grad_u, fluctuation, stress,
                                      iterations, residual, nullptr, s));
  else
    k_rve_indexed<float><<<grid, kRveThreads, r->smem, s>>>(
        a, capacity, index, count, grad_u, static_cast<float*>(fluctuation), stress, iterations,
        residual);
  AKB_CUDA_TRY(cudaGetLastError());
  return AKB_OK;
}

akb_status akb_rve_stress(akb_rve* r, int64_t nb, const double* grad_u, const void* fluctuation,
                          double* stress, double* internal_force, void* stream) {
  if (!r) return fail(AKB_ERR_INVALID_ARGUMENT, "null RVE");
  if (!fluctuation) return fail(AKB_ERR_INVALID_ARGUMENT, "fluctuation is required");
  // zero updates: the state is only read
  return launch(r, 0, nb, grad_u, const_cast<void*>(fluctuation), stress, nullptr, nullptr,
                internal_force, stream);
}

}  // extern "C"
