// Total Lagrangian operators: material tangent (materialTangentMatrix,
// src/nonlinear.jl:2083-2268), initial-stress (geometric) stiffness
// (initialStressMatrix, :2417-2595) and internal force (internalForceVector,
// :2738-2910), with the hyperelastic laws in closed form (the reference
// differentiates psi with Tensors.jl, ext/LowLevelFEMTensorsExt.jl:9-60).
//
// A CTA works on one element (k_tl_matrix) or on several small ones at once
// (k_tl_packed, k_tl_force).  Phase A (threads over integration points):
// Jacobian inverse, weight, interpolated F (or S, C), law -> PK2 stress S and
// 6x6 Voigt tangent D, all kept in shared memory.  Phase B (per point):
// physical gradients g, B(F) (6x3 per node) and T = w D B staged for all
// nodes, then every thread accumulates the 3x3 blocks of its node pairs
// (upper triangle; in k_tl_matrix in tiles of PPT per thread so the
// accumulators stay in registers).  Blocks go to the same pair buffer and
// element-ordered gather as the linear operators.
// Arithmetic contract: identical, operation by operation, to the oracle's
// TL restatement (intrinsics only; ln by the atanh series of the oracle).
#include "common.cuh"

#include <algorithm>

namespace {

constexpr int TL_THREADS = 128;
constexpr int TLP_THREADS = 384;  // most threads of k_tl_packed: hex27's 378 node pairs
// per-point record: wq, invJ[9], F or S [9], D[36], S[9] (tangent); an odd
// stride, so that the threads of the point phase write to different banks
constexpr int QD = 65;
// k_tl_matrix's stride: with 65 doubles a hex125 element takes 116 KB instead of
// 115, and one CTA fits on an SM instead of two (216 elements 75 instead of 60
// ms); its point phase is a small part.  The limits on an element's size are
// those of this stride.
constexpr int QM = 64;
constexpr int QF = 19;  // the internal force's record: wq, invJ[9], P[9]
// TL_FORCE: F in, first Piola-Kirchhoff stress out (internal force)
enum { TL_KMAT = 0, TL_KGEO_S = 1, TL_KGEO_C = 2, TL_KTAN = 3, TL_FORCE = 4 };

struct TLArgs {
  const double *xyz;
  const int32_t *conn;
  const int32_t *emat;
  int64_t nel;
  int npe, nip, npairs;
  const double *w, *N, *dN;
  const double *T;  // elementwise nodal tensors, 9*npe per element
  int law;
  double prm[36];
  double *out;      // pair blocks (matrices) or element vectors (force)
  unsigned *status;
};

__device__ __constant__ int VI[6] = {0, 1, 2, 1, 0, 0};
__device__ __constant__ int VJ[6] = {0, 1, 2, 2, 2, 1};

__device__ double tl_ln(double x) {
  int e;
  double m = frexp(x, &e);
  if (m < 0.70710678118654752440) {
    m = __dmul_rn(m, 2.0);
    e = e - 1;
  }
  double s = __ddiv_rn(__dsub_rn(m, 1.0), __dadd_rn(m, 1.0));
  double s2 = __dmul_rn(s, s);
  double p = __ddiv_rn(1.0, 25.0);
  for (int k = 11; k >= 0; --k) p = __fma_rn(p, s2, __ddiv_rn(1.0, __dadd_rn(__dmul_rn(2.0, (double)k), 1.0)));
  return __fma_rn((double)e, 0.69314718055994530942, __dmul_rn(2.0, __dmul_rn(s, p)));
}

// S (3x3) and, WITH_D, D (6x6 row-major) from C; false if det C <= 0.
template <bool WITH_D>
__device__ bool tl_law(int law, const double *prm, const double C[3][3], double S[3][3], double *D) {
  if (law == LLF_LAW_CONSTANT_C) {
    if constexpr (WITH_D)
      for (int a = 0; a < 6; ++a)
        for (int b = 0; b < 6; ++b) D[a * 6 + b] = prm[b * 6 + a];
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) S[i][j] = 0.0;
    return true;
  }
  const double mu = prm[0], lam = prm[1];
  if (law == LLF_LAW_SVK) {
    double E[3][3];
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) E[i][j] = __dmul_rn(0.5, __dsub_rn(C[i][j], i == j ? 1.0 : 0.0));
    double trE = __dadd_rn(__dadd_rn(E[0][0], E[1][1]), E[2][2]);
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) S[i][j] = __fma_rn(lam, i == j ? trE : 0.0, __dmul_rn(__dmul_rn(2.0, mu), E[i][j]));
    if constexpr (WITH_D)
      for (int a = 0; a < 6; ++a)
        for (int b = 0; b < 6; ++b) {
          int I = VI[a], J = VJ[a], K = VI[b], L = VJ[b];
          double v = __dmul_rn(lam, (I == J && K == L) ? 1.0 : 0.0);
          v = __dadd_rn(v, __dmul_rn(mu, __dadd_rn((I == K && J == L) ? 1.0 : 0.0, (I == L && J == K) ? 1.0 : 0.0)));
          D[a * 6 + b] = v;
        }
    return true;
  }
  double c00 = __dsub_rn(__dmul_rn(C[1][1], C[2][2]), __dmul_rn(C[1][2], C[2][1]));
  double c01 = -__dsub_rn(__dmul_rn(C[1][0], C[2][2]), __dmul_rn(C[1][2], C[2][0]));
  double c02 = __dsub_rn(__dmul_rn(C[1][0], C[2][1]), __dmul_rn(C[1][1], C[2][0]));
  double c10 = -__dsub_rn(__dmul_rn(C[0][1], C[2][2]), __dmul_rn(C[0][2], C[2][1]));
  double c11 = __dsub_rn(__dmul_rn(C[0][0], C[2][2]), __dmul_rn(C[0][2], C[2][0]));
  double c12 = -__dsub_rn(__dmul_rn(C[0][0], C[2][1]), __dmul_rn(C[0][1], C[2][0]));
  double c20 = __dsub_rn(__dmul_rn(C[0][1], C[1][2]), __dmul_rn(C[0][2], C[1][1]));
  double c21 = -__dsub_rn(__dmul_rn(C[0][0], C[1][2]), __dmul_rn(C[0][2], C[1][0]));
  double c22 = __dsub_rn(__dmul_rn(C[0][0], C[1][1]), __dmul_rn(C[0][1], C[1][0]));
  double det = __dadd_rn(__dadd_rn(__dmul_rn(C[0][0], c00), __dmul_rn(C[0][1], c01)), __dmul_rn(C[0][2], c02));
  if (!(det > 0.0)) return false;
  double r = __drcp_rn(det);
  double Ci[3][3] = {{__dmul_rn(c00, r), __dmul_rn(c10, r), __dmul_rn(c20, r)},
                     {__dmul_rn(c01, r), __dmul_rn(c11, r), __dmul_rn(c21, r)},
                     {__dmul_rn(c02, r), __dmul_rn(c12, r), __dmul_rn(c22, r)}};
  double lnJ = __dmul_rn(0.5, tl_ln(det));
  double t = __dmul_rn(lam, lnJ);
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j)
      S[i][j] = __fma_rn(t, Ci[i][j], __dmul_rn(mu, __dsub_rn(i == j ? 1.0 : 0.0, Ci[i][j])));
  // C = F^T F is symmetric bit for bit (its products commute), so C^-1 and D
  // are too: the upper triangle of D, mirrored
  if constexpr (WITH_D) {
    const double m2 = __dsub_rn(mu, t);
#pragma unroll
    for (int a = 0; a < 6; ++a)
#pragma unroll
      for (int b = a; b < 6; ++b) {
        constexpr int WI[6] = {0, 1, 2, 1, 0, 0}, WJ[6] = {0, 1, 2, 2, 2, 1};
        const int I = WI[a], J = WJ[a], K = WI[b], L = WJ[b];
        const double sym = __dadd_rn(__dmul_rn(Ci[I][K], Ci[J][L]), __dmul_rn(Ci[I][L], Ci[J][K]));
        const double v = __fma_rn(lam, __dmul_rn(Ci[I][J], Ci[K][L]), __dmul_rn(m2, sym));
        D[a * 6 + b] = v;
        D[b * 6 + a] = v;
      }
  }
  return true;
}

__device__ __forceinline__ int pair_off(int a, int npe) { return a * npe - (a * (a - 1)) / 2; }
__device__ __forceinline__ void pair_dec(int pi, int npe, int &a, int &b) {
  int lo = 0, hi = npe - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (pair_off(mid, npe) <= pi) lo = mid; else hi = mid - 1;
  }
  a = lo;
  b = a + (pi - pair_off(a, npe));
}

// Phase A for one point: wq, invJ, and the tensors the mode needs.
// Layout of rec: [0] wq, [1..9] invJ, [10..18] F (KMAT, KTAN), S (KGEO) or
// P (FORCE), [19..54] D, [55..63] S (KTAN).
template <int mode>
__device__ __forceinline__ void tl_point(const TLArgs &A, int q, const double *sX, const double *sT, double *rec) {
  const int npe = A.npe;
  const double *dNq = A.dN + (size_t)q * npe * 3;
  double J[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) J[i][j] = 0.0;
  for (int a = 0; a < npe; ++a) {  // nine independent chains, each in node order
    double d[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) d[j] = __ldg(dNq + a * 3 + j);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) J[i][j] = __fma_rn(sX[a * 3 + i], d[j], J[i][j]);
  }
  double c00 = __dsub_rn(__dmul_rn(J[1][1], J[2][2]), __dmul_rn(J[1][2], J[2][1]));
  double c01 = -__dsub_rn(__dmul_rn(J[1][0], J[2][2]), __dmul_rn(J[1][2], J[2][0]));
  double c02 = __dsub_rn(__dmul_rn(J[1][0], J[2][1]), __dmul_rn(J[1][1], J[2][0]));
  double c10 = -__dsub_rn(__dmul_rn(J[0][1], J[2][2]), __dmul_rn(J[0][2], J[2][1]));
  double c11 = __dsub_rn(__dmul_rn(J[0][0], J[2][2]), __dmul_rn(J[0][2], J[2][0]));
  double c12 = -__dsub_rn(__dmul_rn(J[0][0], J[2][1]), __dmul_rn(J[0][1], J[2][0]));
  double c20 = __dsub_rn(__dmul_rn(J[0][1], J[1][2]), __dmul_rn(J[0][2], J[1][1]));
  double c21 = -__dsub_rn(__dmul_rn(J[0][0], J[1][2]), __dmul_rn(J[0][2], J[1][0]));
  double c22 = __dsub_rn(__dmul_rn(J[0][0], J[1][1]), __dmul_rn(J[0][1], J[1][0]));
  double det = __dadd_rn(__dadd_rn(__dmul_rn(J[0][0], c00), __dmul_rn(J[0][1], c01)), __dmul_rn(J[0][2], c02));
  if (!(det > 0.0)) atomicOr(A.status, ST_BAD_JACOBIAN);
  double r = __drcp_rn(det);
  rec[0] = __dmul_rn(det, __ldg(A.w + q));
  rec[1] = __dmul_rn(c00, r); rec[2] = __dmul_rn(c10, r); rec[3] = __dmul_rn(c20, r);
  rec[4] = __dmul_rn(c01, r); rec[5] = __dmul_rn(c11, r); rec[6] = __dmul_rn(c21, r);
  rec[7] = __dmul_rn(c02, r); rec[8] = __dmul_rn(c12, r); rec[9] = __dmul_rn(c22, r);
  // interpolated nodal tensor (column-major per node)
  const double *Nq = A.N + (size_t)q * npe;
  double Tq[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Tq[i][j] = 0.0;
  for (int a = 0; a < npe; ++a) {
    const double na = __ldg(Nq + a);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) Tq[i][j] = __fma_rn(na, sT[9 * a + 3 * j + i], Tq[i][j]);
  }
  if (mode == TL_KGEO_S) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) rec[10 + 3 * i + j] = Tq[i][j];
    return;
  }
  double C[3][3];
  if (mode != TL_KGEO_C) {
#pragma unroll
    for (int I = 0; I < 3; ++I)
#pragma unroll
      for (int J2 = 0; J2 < 3; ++J2) {
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) acc = __fma_rn(Tq[k][I], Tq[k][J2], acc);
        C[I][J2] = acc;
      }
  } else {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) C[i][j] = Tq[i][j];
  }
  constexpr bool with_d = mode == TL_KMAT || mode == TL_KTAN;
  if (with_d)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) rec[10 + 3 * i + j] = Tq[i][j];  // F
  double S[3][3];
  if (!tl_law<with_d>(A.law, A.prm, C, S, rec + 19)) {
    atomicOr(A.status, ST_NONFINITE);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) S[i][j] = 0.0;
  }
  if (mode == TL_FORCE) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int J2 = 0; J2 < 3; ++J2) {
        double s = 0.0;
#pragma unroll
        for (int K = 0; K < 3; ++K) s = __fma_rn(Tq[i][K], S[K][J2], s);
        rec[10 + 3 * i + J2] = s;  // P
      }
  }
  if (mode == TL_KGEO_C || mode == TL_KTAN) {
    constexpr int at = mode == TL_KTAN ? 55 : 10;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) rec[at + 3 * i + j] = S[i][j];
  }
}

template <int MODE>
__global__ void __launch_bounds__(TL_THREADS) k_tl_matrix(TLArgs A) {
  extern __shared__ double sm[];
  constexpr int PPT = 4;                   // node pairs per thread of a tile
  const int npe = A.npe, nip = A.nip;
  double *sX = sm;                         // npe*3
  double *sT = sX + npe * 3;               // npe*9
  double *qd = sT + npe * 9;               // nip*QM
  double *sG = qd + (size_t)nip * QM;      // npe*3
  double *sB = sG + npe * 3;               // npe*18
  double *sTb = sB + npe * 18;             // npe*18 (KMAT)
  constexpr bool MAT = (MODE == TL_KMAT || MODE == TL_KTAN);
  constexpr int BS = MAT ? 9 : 1;
  for (int64_t e = blockIdx.x; e < A.nel; e += gridDim.x) {
    if (A.emat && A.emat[e] < 0) continue;
    for (int t = threadIdx.x; t < npe * 3; t += blockDim.x)
      sX[t] = A.xyz[(size_t)A.conn[e * npe + t / 3] * 3 + t % 3];
    for (int t = threadIdx.x; t < npe * 9; t += blockDim.x) sT[t] = A.T[(size_t)e * npe * 9 + t];
    __syncthreads();
    for (int q = threadIdx.x; q < nip; q += blockDim.x) tl_point<MODE>(A, q, sX, sT, qd + (size_t)q * QM);
    __syncthreads();
    double *Ke = A.out + (size_t)e * npe * npe * BS;  // [column node][row node][block]
    const int tile = blockDim.x * PPT;
    for (int p0 = 0; p0 < A.npairs; p0 += tile) {
      double acc[PPT][BS];
#pragma unroll
      for (int k = 0; k < PPT; ++k)
#pragma unroll
        for (int m = 0; m < BS; ++m) acc[k][m] = 0.0;
      for (int q = 0; q < nip; ++q) {
        const double *rec = qd + (size_t)q * QM;
        // physical gradients of all nodes at q
        for (int t = threadIdx.x; t < npe * 3; t += blockDim.x) {
          int a = t / 3, i = t % 3;
          const double *d = A.dN + ((size_t)q * npe + a) * 3;
          double s = 0.0;
          for (int j = 0; j < 3; ++j) s = __fma_rn(rec[1 + 3 * j + i], __ldg(d + j), s);
          sG[t] = s;
        }
        __syncthreads();
        if (MAT) {
          // B(F) per node (src/nonlinear.jl:2219-2242)
          for (int t = threadIdx.x; t < npe * 3; t += blockDim.x) {
            int b = t / 3, j = t % 3;
            const double *F = rec + 10;  // F[j][k] at 10 + 3j + k
            double v1 = F[3 * j + 0], v2 = F[3 * j + 1], v3 = F[3 * j + 2];
            const double *g = sG + 3 * b;
            double *Bb = sB + b * 18;
            Bb[0 * 3 + j] = __dmul_rn(v1, g[0]);
            Bb[1 * 3 + j] = __dmul_rn(v2, g[1]);
            Bb[2 * 3 + j] = __dmul_rn(v3, g[2]);
            Bb[3 * 3 + j] = __dadd_rn(__dmul_rn(v2, g[2]), __dmul_rn(v3, g[1]));
            Bb[4 * 3 + j] = __dadd_rn(__dmul_rn(v1, g[2]), __dmul_rn(v3, g[0]));
            Bb[5 * 3 + j] = __dadd_rn(__dmul_rn(v1, g[1]), __dmul_rn(v2, g[0]));
          }
          __syncthreads();
          const double *D = rec + 19;
          const double wq = rec[0];
          for (int t = threadIdx.x; t < npe * 18; t += blockDim.x) {
            int b = t / 18, I = (t % 18) / 3, j = t % 3;
            double s = 0.0;
            for (int J2 = 0; J2 < 6; ++J2) s = __fma_rn(D[I * 6 + J2], sB[b * 18 + J2 * 3 + j], s);
            sTb[t] = __dmul_rn(s, wq);
          }
          __syncthreads();
        }
#pragma unroll
        for (int k = 0; k < PPT; ++k) {
          const int pi = p0 + k * blockDim.x + threadIdx.x;
          if (pi >= A.npairs) continue;
          int a, b;
          pair_dec(pi, npe, a, b);
          if (MAT) {
            const double *Ba = sB + a * 18, *Tb = sTb + b * 18;
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
              for (int j = 0; j < 3; ++j) {
                if (a == b && j < i) continue;
                double s = acc[k][i * 3 + j];
#pragma unroll
                for (int I = 0; I < 6; ++I) s = __fma_rn(Ba[I * 3 + i], Tb[I * 3 + j], s);
                acc[k][i * 3 + j] = s;
              }
            if (MODE == TL_KTAN) {  // consistent tangent: geometric part from the same S
              const double *S = rec + 55, *ga = sG + 3 * a, *gb = sG + 3 * b;
              double tv[3];
#pragma unroll
              for (int I = 0; I < 3; ++I) {
                double s = 0.0;
#pragma unroll
                for (int J2 = 0; J2 < 3; ++J2) s = __fma_rn(S[3 * I + J2], gb[J2], s);
                tv[I] = s;
              }
              double v = 0.0;
#pragma unroll
              for (int I = 0; I < 3; ++I) v = __fma_rn(ga[I], tv[I], v);
#pragma unroll
              for (int i = 0; i < 3; ++i) acc[k][i * 3 + i] = __fma_rn(v, rec[0], acc[k][i * 3 + i]);
            }
          } else {
            const double *S = rec + 10, *ga = sG + 3 * a, *gb = sG + 3 * b;
            double tv[3];
#pragma unroll
            for (int I = 0; I < 3; ++I) {
              double s = 0.0;
#pragma unroll
              for (int J2 = 0; J2 < 3; ++J2) s = __fma_rn(S[3 * I + J2], gb[J2], s);
              tv[I] = s;
            }
            double v = 0.0;
#pragma unroll
            for (int I = 0; I < 3; ++I) v = __fma_rn(ga[I], tv[I], v);
            acc[k][0] = __fma_rn(v, rec[0], acc[k][0]);
          }
        }
        __syncthreads();
      }
#pragma unroll
      for (int k = 0; k < PPT; ++k) {
        const int pi = p0 + k * blockDim.x + threadIdx.x;
        if (pi >= A.npairs) continue;
        int a, b;
        pair_dec(pi, npe, a, b);
        double *ab = Ke + ((size_t)b * npe + a) * BS;   // block (a,b)
        double *ba = Ke + ((size_t)a * npe + b) * BS;   // mirror (b,a)
        if (MAT) {
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              const double v = (a == b && j < i) ? acc[k][j * 3 + i] : acc[k][i * 3 + j];
              ab[i * 3 + j] = v;
              if (a != b) ba[j * 3 + i] = v;
            }
        } else {
          ab[0] = acc[k][0];
          if (a != b) ba[0] = acc[k][0];
        }
      }
    }
    __syncthreads();
  }
}

// The same element matrices for elements of up to 384 node pairs, E of them
// per CTA (e0 .. e0+E-1), so that the lanes of every phase are filled: the
// FP64 pipe, which bounds this kernel, is spent per warp instruction, however
// few lanes take part.  One element per 128-thread CTA used 36 lanes of hex8's
// pair loop and 8 of its point phase.  Phases: the points of all elements,
// then the physical gradients at all points, then per point B(F) (with
// T = w D B and S g, which depend on one node only, staged once per node
// instead of once per pair) and the node pairs, one per thread.  hex8,
// 29,760 elements: 4.14 -> 1.71 ms (31,000 FP64 lane operations per element
// at 608 G/s take 1.5 ms).
// Shared memory (doubles): sX [E npe 3] | qd [E nip QD] | sG [E nip npe 3] |
// stage [E npe 39], which starts as sT [E npe 9].
template <int MODE>
__global__ void __launch_bounds__(TLP_THREADS, 2) k_tl_packed(TLArgs A, int E) {
  extern __shared__ double sm[];
  const int npe = A.npe, nip = A.nip;
  constexpr bool MAT = (MODE == TL_KMAT || MODE == TL_KTAN);
  constexpr int BS = MAT ? 9 : 1;
  double *sX = sm;
  double *qd = sX + (size_t)E * npe * 3;
  double *sG = qd + (size_t)E * nip * QD;
  double *sS = sG + (size_t)E * nip * npe * 3;   // S g  [E npe 3]
  double *sB = sS + (size_t)E * npe * 3;         // B    [E npe 18]
  double *sTb = sB + (size_t)E * npe * 18;       // w D B [E npe 18]
  double *sT = sS;
  // this thread's node pair
  const int el = threadIdx.x / A.npairs;
  int a = 0, b = 0;
  if (el < E) pair_dec(threadIdx.x - el * A.npairs, npe, a, b);
  for (int64_t e0 = (int64_t)blockIdx.x * E; e0 < A.nel; e0 += (int64_t)gridDim.x * E) {
    const int ne = (int)(A.nel - e0 < E ? A.nel - e0 : E);
    for (int t = threadIdx.x; t < ne * npe * 3; t += blockDim.x)
      sX[t] = A.xyz[(size_t)A.conn[e0 * npe + t / 3] * 3 + t % 3];
    for (int t = threadIdx.x; t < ne * npe * 9; t += blockDim.x) sT[t] = A.T[(size_t)e0 * npe * 9 + t];
    __syncthreads();
    for (int t = threadIdx.x; t < ne * nip; t += blockDim.x) {
      const int k = t / nip;
      if (A.emat && A.emat[e0 + k] < 0) continue;
      tl_point<MODE>(A, t - k * nip, sX + (size_t)k * npe * 3, sT + (size_t)k * npe * 9, qd + (size_t)t * QD);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < ne * nip * npe; t += blockDim.x) {
      const int p = t / npe, q = p % nip;   // point of the CTA, of its element
      const double *inv = qd + (size_t)p * QD + 1, *d = A.dN + ((size_t)q * npe + (t - p * npe)) * 3;
      const double d0 = __ldg(d), d1 = __ldg(d + 1), d2 = __ldg(d + 2);
#pragma unroll
      for (int i = 0; i < 3; ++i)
        sG[(size_t)t * 3 + i] = __fma_rn(inv[6 + i], d2, __fma_rn(inv[3 + i], d1, __fma_rn(inv[i], d0, 0.0)));
    }
    const bool live = el < ne && !(A.emat && A.emat[e0 + el] < 0);
    double acc[BS];
#pragma unroll
    for (int m = 0; m < BS; ++m) acc[m] = 0.0;
    for (int q = 0; q < nip; ++q) {
      __syncthreads();   // the gradients (q = 0), the pairs' reads of the last point
      for (int t = threadIdx.x; t < ne * npe * 3; t += blockDim.x) {
        const int n = t / 3, j = t - 3 * n, k = n / npe;   // node of the CTA, component, element
        const double *rec = qd + ((size_t)k * nip + q) * QD;
        const double *g = sG + (((size_t)k * nip + q) * npe + (n - k * npe)) * 3;
        const double g0 = g[0], g1 = g[1], g2 = g[2];
        if (MAT) {  // column j of B(F) (src/nonlinear.jl:2219-2242) and of w D B
          const double *F = rec + 10 + 3 * j, *D = rec + 19;
          const double v1 = F[0], v2 = F[1], v3 = F[2];
          double Bc[6];
          Bc[0] = __dmul_rn(v1, g0);
          Bc[1] = __dmul_rn(v2, g1);
          Bc[2] = __dmul_rn(v3, g2);
          Bc[3] = __dadd_rn(__dmul_rn(v2, g2), __dmul_rn(v3, g1));
          Bc[4] = __dadd_rn(__dmul_rn(v1, g2), __dmul_rn(v3, g0));
          Bc[5] = __dadd_rn(__dmul_rn(v1, g1), __dmul_rn(v2, g0));
          const double wq = rec[0];
#pragma unroll
          for (int I = 0; I < 6; ++I) {
            double s = 0.0;
#pragma unroll
            for (int J2 = 0; J2 < 6; ++J2) s = __fma_rn(D[I * 6 + J2], Bc[J2], s);
            sB[(size_t)n * 18 + I * 3 + j] = Bc[I];
            sTb[(size_t)n * 18 + I * 3 + j] = __dmul_rn(s, wq);
          }
        }
        if (MODE != TL_KMAT) {  // row j of S g
          const double *S = rec + (MODE == TL_KTAN ? 55 : 10) + 3 * j;
          sS[(size_t)n * 3 + j] = __fma_rn(S[2], g2, __fma_rn(S[1], g1, __fma_rn(S[0], g0, 0.0)));
        }
      }
      __syncthreads();
      if (live) {
        const size_t na = (size_t)el * npe + a, nb = (size_t)el * npe + b;
        if (MAT) {
          const double *Ba = sB + na * 18, *Tb = sTb + nb * 18;
#pragma unroll
          for (int I = 0; I < 6; ++I) {
            double x[3], y[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              x[i] = Ba[I * 3 + i];
              y[i] = Tb[I * 3 + i];
            }
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
              for (int j = 0; j < 3; ++j) acc[i * 3 + j] = __fma_rn(x[i], y[j], acc[i * 3 + j]);
          }
        }
        if (MODE != TL_KMAT) {  // geometric part
          const double *ga = sG + (((size_t)el * nip + q) * npe + a) * 3, *tv = sS + nb * 3;
          const double wq = qd[((size_t)el * nip + q) * QD];
          const double v = __fma_rn(ga[2], tv[2], __fma_rn(ga[1], tv[1], __fma_rn(ga[0], tv[0], 0.0)));
          if (MAT) {
#pragma unroll
            for (int i = 0; i < 3; ++i) acc[i * 3 + i] = __fma_rn(v, wq, acc[i * 3 + i]);
          } else {
            acc[0] = __fma_rn(v, wq, acc[0]);
          }
        }
      }
    }
    if (live) {
      double *Ke = A.out + (size_t)(e0 + el) * npe * npe * BS;  // [column node][row node][block]
      double *ab = Ke + ((size_t)b * npe + a) * BS;   // block (a,b)
      double *ba = Ke + ((size_t)a * npe + b) * BS;   // mirror (b,a)
      if (MAT) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const double v = (a == b && j < i) ? acc[j * 3 + i] : acc[i * 3 + j];
            ab[i * 3 + j] = v;
            if (a != b) ba[j * 3 + i] = v;
          }
      } else {
        ab[0] = acc[0];
        if (a != b) ba[0] = acc[0];
      }
    }
    __syncthreads();
  }
}

// Internal force: element vectors fe[e][a][i], E elements per CTA (the
// points of small elements fill whole warps: hex8 took 8 lanes of 128 one
// element at a time).  A point's record holds only w, J^-1 and P, and a
// thread makes NC components of a node: all three, so that the node's physical
// gradient is formed once per point (hex8, 29,760 elements: 1.49 -> 0.25 ms;
// hex125, 576 elements: 1.46 -> 0.68 ms), or one on meshes of few CTAs, where
// its longest chain is what counts.
template <int MODE, int NC>  // TL_FORCE: T = F with law, TL_KGEO_S: T = P
__global__ void __launch_bounds__(TL_THREADS) k_tl_force(TLArgs A, int E) {
  extern __shared__ double sm[];
  const int npe = A.npe, nip = A.nip;
  double *sX = sm;
  double *sT = sX + (size_t)E * npe * 3;
  double *qd = sT + (size_t)E * npe * 9;
  for (int64_t e0 = (int64_t)blockIdx.x * E; e0 < A.nel; e0 += (int64_t)gridDim.x * E) {
    const int ne = (int)(A.nel - e0 < E ? A.nel - e0 : E);
    for (int t = threadIdx.x; t < ne * npe * 3; t += blockDim.x)
      sX[t] = A.xyz[(size_t)A.conn[e0 * npe + t / 3] * 3 + t % 3];
    for (int t = threadIdx.x; t < ne * npe * 9; t += blockDim.x) sT[t] = A.T[(size_t)e0 * npe * 9 + t];
    __syncthreads();
    for (int t = threadIdx.x; t < ne * nip; t += blockDim.x) {
      const int k = t / nip;
      tl_point<MODE>(A, t - k * nip, sX + (size_t)k * npe * 3, sT + (size_t)k * npe * 9, qd + (size_t)t * QF);
    }
    __syncthreads();
    constexpr int NT = 3 / NC;   // threads per node
    for (int t = threadIdx.x; t < ne * npe * NT; t += blockDim.x) {
      const int n = t / NT, k = n / npe, a = n - k * npe, i0 = t - n * NT;
      double fe[NC] = {};
      for (int q = 0; q < nip; ++q) {
        const double *rec = qd + ((size_t)k * nip + q) * QF;
        const double *d = A.dN + ((size_t)q * npe + a) * 3;
        const double d0 = __ldg(d), d1 = __ldg(d + 1), d2 = __ldg(d + 2);
        double g[3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
          g[c] = __fma_rn(rec[7 + c], d2, __fma_rn(rec[4 + c], d1, __fma_rn(rec[1 + c], d0, 0.0)));
#pragma unroll
        for (int i = 0; i < NC; ++i) {
          const double *P = rec + 10 + 3 * (i0 + i);
          const double v = __fma_rn(P[2], g[2], __fma_rn(P[1], g[1], __fma_rn(P[0], g[0], 0.0)));
          fe[i] = __fma_rn(v, rec[0], fe[i]);
        }
      }
#pragma unroll
      for (int i = 0; i < NC; ++i) A.out[((size_t)e0 * npe + n) * 3 + i0 + i] = fe[i];
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------ tensor-core form
// Consistent tangent on the 5th-generation tensor cores (tcgen05), for
// high-order elements where the element contraction is dense.  Per point q
// the tangent is [B_q; G_q]^T diag(w D_q, w S_q (x) I) [B_q; G_q], with B_q
// the 6 x 3npe matrix B(F) and G_q the 9 x 3npe displacement-gradient
// operator, so the whole element matrix is one GEMM over K = 15 rows per
// point.  One CTA computes 128 columns x 192 rows of one element matrix:
//   - the point data (F, w D, w S, physical gradients; FP64 as in the FP64
//     form, rounded to FP32) come from k_tl_points_tc, two points per
//     k-block, fetched by cp.async.bulk two k-blocks ahead;
//   - per k-block of 2 points (2 x 15 K values, padded to 32) eight warps form
//     the weighted operands [D B; S G] of the tile's columns, a thread per
//     column and point, and write them to tensor memory (tcgen05.st: the M
//     operand), while the other eight form [B; G] of the tile's rows in shared
//     memory (the N operand, K-major core matrices of 8 rows x 16 bytes).
//     Both are split into TF32 hi and lo parts;
//   - one thread issues tcgen05.mma kind::tf32 (M 128, N 192, K 8) for the
//     three split products hi*hi + hi*lo + lo*hi into an FP32 accumulator in
//     tensor memory and commits to an mbarrier;
//   - the epilogue reads the accumulator with tcgen05.ld and writes the
//     element matrix (FP32) in the gather's layout.
// Two CTAs per SM (256 columns of tensor memory each): one builds while the
// other's products run.
// Bound by the tensor cores' TF32 rate (1.03 TFLOP of split products for 576
// hex125: 1.1 ms) and what of the build their two CTAs leave uncovered.
// Forming both operands in shared memory, one CTA per SM and two stages, was
// bound by the build: 2.30 ms; with the M operand, the dearer of the two, in
// tensor memory it is 128 columns a thread each instead of 192, without
// shared-memory traffic on either side, and the build hides: 1.50 ms.  A
// separate product for the geometric part (K 6 + 3 instead of 15) took 1.40 ms
// but sums the same terms in another order.
// Every mbarrier wait is bounded (2 s): a timeout sets ST_TIMEOUT, the CTA
// skips its epilogue and releases its tensor memory.
constexpr int TC_M = 128, TC_N = 192, TC_KB = 32, TC_PTS = 2, TC_THREADS = 512;
constexpr int TC_TILE = TC_N * TC_KB;   // floats of the N operand's tile (hi or lo)
constexpr int TC_COL_HI = TC_N, TC_COL_LO = TC_N + TC_KB, TC_COLS = 256;   // tensor memory: accumulator | M operand
static_assert(TC_THREADS == 2 * TC_M * TC_PTS, "half the threads: one per column and point");

struct TcArgs {
  const float *pd;     // nel * nip * tc_pstride(npe) packed point data (k_tl_points_tc)
  const int32_t *emat;
  int64_t nel;
  int npe, nip, n, nstrip, nhalf;
  float *Kf;           // nel * npe * cs
  int64_t cs;
  unsigned *status;
};

__device__ __forceinline__ uint32_t tc_saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, K-major, no swizzle: core matrices of
// 8 rows x 16 bytes, LBO = distance of K-adjacent core matrices (128 B),
// SBO = distance of 8-row groups (TC_KB / 4 core matrices of 128 B).
__device__ __forceinline__ uint64_t tc_desc(const float *p) {
  const uint64_t lbo = 128, sbo = (TC_KB / 4) * 128;
  return (uint64_t)((tc_saddr(p) & 0x3FFFF) >> 4) | ((lbo >> 4) << 16) | ((sbo >> 4) << 32) | ((uint64_t)1 << 46);
}

__device__ __forceinline__ int tc_off(int row, int k) {
  return ((row >> 3) * (TC_KB / 4) + (k >> 2)) * 32 + (row & 7) * 4 + (k & 3);
}

__device__ __forceinline__ float tc_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// The 16 K values of a row at a point: b[6], then g in the places of
// component ci of [G] (gradient index times 3 plus component), hi and lo parts.
__device__ __forceinline__ void tc_row16(const float (&b)[6], const float (&g)[3], int ci, float (&h)[16],
                                         float (&l)[16]) {
#pragma unroll
  for (int r = 0; r < 6; ++r) {
    h[r] = tc_tf32(b[r]);
    l[r] = b[r] - h[r];
  }
#pragma unroll
  for (int I = 0; I < 3; ++I) {
    const float gh = tc_tf32(g[I]), gl = g[I] - gh;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      h[6 + 3 * I + c] = c == ci ? gh : 0.f;
      l[6 + 3 * I + c] = c == ci ? gl : 0.f;
    }
  }
  h[15] = l[15] = 0.f;
}

// B(F) of a node with gradient g at component ci (F's row ci).
__device__ __forceinline__ void tc_brow(const float *F, int ci, const float (&g)[3], float (&b)[6]) {
  const float v1 = F[3 * ci], v2 = F[3 * ci + 1], v3 = F[3 * ci + 2];
  b[0] = v1 * g[0];
  b[1] = v2 * g[1];
  b[2] = v3 * g[2];
  b[3] = fmaf(v2, g[2], v3 * g[1]);
  b[4] = fmaf(v1, g[2], v3 * g[0]);
  b[5] = fmaf(v1, g[1], v2 * g[0]);
}

// 16 values of this thread's tensor-memory lane.
__device__ __forceinline__ void tc_st16(uint32_t addr, const float (&v)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(addr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
                 "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
                 "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])), "r"(__float_as_uint(v[8])),
                 "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
                 "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])),
                 "r"(__float_as_uint(v[15]))
               : "memory");
}

__device__ __forceinline__ uint64_t tc_now() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait on an mbarrier phase (2 s); false on timeout.
__device__ __forceinline__ bool tc_wait(uint64_t *bar, unsigned parity) {
  const uint64_t t0 = tc_now();
  for (;;) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(tc_saddr(bar)), "r"(parity) : "memory");
    if (ok) return true;
    if (tc_now() - t0 > 2000000000ull) return false;
  }
}

// Packed FP32 point data of the tensor-core form, one CTA per element: for
// every point q a run of tc_pstride(npe) floats (16-byte multiple)
//   [0,9) F | [12,48) w D | [48,57) w S | [60, 60+3 npe) grad N_a, 0 between
// computed in FP64 (the FP64 form's point record and gradients) and rounded.
constexpr int TP_D = 12, TP_S = 48, TP_G = 60;   // 16-byte aligned parts
__host__ __device__ __forceinline__ int tc_pstride(int npe) { return (TP_G + 3 * npe + 3) & ~3; }

__global__ void __launch_bounds__(TL_THREADS) k_tl_points_tc(TLArgs A, float *pd) {
  extern __shared__ double sm[];
  const int npe = A.npe, nip = A.nip, ps = tc_pstride(npe);
  double *sX = sm, *sT = sX + npe * 3, *rec = sT + npe * 9;  // rec: nip * QD
  for (int64_t e = blockIdx.x; e < A.nel; e += gridDim.x) {
    if (A.emat && A.emat[e] < 0) continue;
    for (int t = threadIdx.x; t < npe * 3; t += blockDim.x)
      sX[t] = A.xyz[(size_t)A.conn[e * npe + t / 3] * 3 + t % 3];
    for (int t = threadIdx.x; t < npe * 9; t += blockDim.x) sT[t] = A.T[(size_t)e * npe * 9 + t];
    __syncthreads();
    for (int q = threadIdx.x; q < nip; q += blockDim.x) tl_point<TL_KTAN>(A, q, sX, sT, rec + (size_t)q * QD);
    __syncthreads();
    float *out = pd + (size_t)e * nip * ps;
    for (int t = threadIdx.x; t < nip * ps; t += blockDim.x) {
      const int q = t / ps, f = t - q * ps;
      const double *r = rec + (size_t)q * QD;
      double v = 0.0;
      if (f < 9) v = r[10 + f];
      else if (f >= TP_D && f < TP_D + 36) v = __dmul_rn(r[0], r[19 + (f - TP_D)]);
      else if (f >= TP_S && f < TP_S + 9) v = __dmul_rn(r[0], r[55 + (f - TP_S)]);
      else if (f >= TP_G && f < TP_G + 3 * npe) {
        const int a = (f - TP_G) / 3, I = (f - TP_G) % 3;
        const double *d = A.dN + ((size_t)q * npe + a) * 3;
        double g = 0.0;
        for (int J = 0; J < 3; ++J) g = __fma_rn(r[1 + 3 * J + I], d[J], g);
        v = g;
      }
      out[t] = (float)v;
    }
    __syncthreads();
  }
}

__device__ __forceinline__ void tc_bulk(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc_saddr(bar)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(tc_saddr(dst)), "l"(src), "r"(bytes), "r"(tc_saddr(bar))
               : "memory");
}

// Shared memory: N operand hi, lo | 2 point-data buffers (TC_PTS points each,
// fetched by cp.async.bulk two k-blocks ahead) | mbarriers: products, point
// data x2 | tensor-memory address.
__global__ void __launch_bounds__(TC_THREADS, 2) k_tl_tangent_tc(TcArgs A) {
  extern __shared__ __align__(1024) float tsm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per_e = A.nstrip * A.nhalf;
  const int64_t e = blockIdx.x / per_e;
  const int rr = (int)(blockIdx.x - e * per_e);
  const int col0 = (rr / A.nhalf) * TC_M, row0 = (rr % A.nhalf) * TC_N;
  if (e >= A.nel || (A.emat && A.emat[e] < 0)) return;  // uniform across the CTA
  const int npe = A.npe, nip = A.nip, n = A.n, ps = tc_pstride(npe);
  float *Nhi = tsm, *Nlo = Nhi + TC_TILE;
  float *pbuf = tsm + 2 * TC_TILE;                       // 2 x TC_PTS * ps
  uint64_t *bar = (uint64_t *)(pbuf + 2 * TC_PTS * ps);  // 0 products, 1 and 2 point data
  uint32_t *tslot = (uint32_t *)(bar + 3);
  const float *pd = A.pd + (size_t)e * nip * ps;
  const int nkb = (nip + TC_PTS - 1) / TC_PTS;
  auto fetch = [&](int kb) {   // point data of k-block kb into buffer kb & 1
    const int q0 = kb * TC_PTS, np = nip - q0 < TC_PTS ? nip - q0 : TC_PTS;
    tc_bulk(pbuf + (kb & 1) * TC_PTS * ps, pd + (size_t)q0 * ps, (unsigned)(np * ps * sizeof(float)), bar + 1 + (kb & 1));
  };
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_saddr(tslot)),
                 "r"((uint32_t)TC_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int b = 0; b < 3; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_saddr(bar + b)), "r"(1u) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fetch(0);
    if (nkb > 1) fetch(1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(TC_N >> 3) << 17) |
                         ((uint32_t)(TC_M >> 4) << 24);
  bool ok = true;
  int fetched = nkb < 2 ? nkb : 2;  // point-data copies issued (k-blocks 0 .. fetched-1)
  for (int kb = 0; kb < nkb; ++kb) {
    const int q0 = kb * TC_PTS;
    const float *pb = pbuf + (kb & 1) * TC_PTS * ps;
    // the operands' values, formed while the products of k-block kb - 1 run;
    // they are split and stored once those are done
    bool w = tc_wait(bar + 1 + (kb & 1), (unsigned)(kb >> 1) & 1u);
    if (warp < TC_THREADS / 64) {
      // M operand: column col0 + 32 (warp % 4) + lane (the lanes of tensor
      // memory this warp may access) at point warp / 4, so w D and w S are
      // broadcasts
      const int ql = warp >> 2, gj = col0 + (warp & 3) * 32 + lane;
      float d[6], sg[3];
#pragma unroll
      for (int r = 0; r < 6; ++r) d[r] = 0.f;
#pragma unroll
      for (int I = 0; I < 3; ++I) sg[I] = 0.f;
      const int b = gj / 3, cj = gj - 3 * b;
      if (gj < n && q0 + ql < nip) {
        const float *P = pb + ql * ps;
        const float g[3] = {P[TP_G + 3 * b], P[TP_G + 3 * b + 1], P[TP_G + 3 * b + 2]};
        float Bv[6];
        tc_brow(P, cj, g, Bv);
        const float4 *wD = reinterpret_cast<const float4 *>(P + TP_D);
#pragma unroll
        for (int r = 0; r < 6; r += 2) {   // two rows of w D: three 16-byte words
          float t[12];
#pragma unroll
          for (int x = 0; x < 3; ++x) *reinterpret_cast<float4 *>(t + 4 * x) = wD[r * 6 / 4 + x];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            float acc = 0.f;
#pragma unroll
            for (int r2 = 0; r2 < 6; ++r2) acc = fmaf(t[6 * u + r2], Bv[r2], acc);
            d[r + u] = acc;
          }
        }
#pragma unroll
        for (int I = 0; I < 3; ++I)
#pragma unroll
          for (int J = 0; J < 3; ++J) sg[I] = fmaf(P[TP_S + 3 * I + J], g[J], sg[I]);
      }
      if (kb > 0) w = w && tc_wait(bar, (unsigned)(kb - 1) & 1u);
      if (__all_sync(0xffffffffu, w)) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float h[16], l[16];
        tc_row16(d, sg, cj, h, l);
        const uint32_t t0 = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(ql * 16);
        tc_st16(t0 + TC_COL_HI, h);
        tc_st16(t0 + TC_COL_LO, l);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      }
    } else {
      // N operand: the tile's rows (a warp's rows share the point)
      constexpr int ROUNDS = (TC_N * TC_PTS + TC_THREADS / 2 - 1) / (TC_THREADS / 2);
      float g[ROUNDS][3], Bv[ROUNDS][6];
#pragma unroll
      for (int k = 0; k < ROUNDS; ++k) {
        const int t = tid - TC_THREADS / 2 + k * (TC_THREADS / 2), ql = t / TC_N, gi = row0 + t - ql * TC_N;
#pragma unroll
        for (int r = 0; r < 6; ++r) Bv[k][r] = 0.f;
#pragma unroll
        for (int I = 0; I < 3; ++I) g[k][I] = 0.f;
        if (t < TC_N * TC_PTS && gi < n && q0 + ql < nip) {
          const float *P = pb + ql * ps;
          const int a = gi / 3;
#pragma unroll
          for (int I = 0; I < 3; ++I) g[k][I] = P[TP_G + 3 * a + I];
          tc_brow(P, gi - 3 * a, g[k], Bv[k]);
        }
      }
      if (kb > 0) w = w && tc_wait(bar, (unsigned)(kb - 1) & 1u);
      if (w) {
#pragma unroll
        for (int k = 0; k < ROUNDS; ++k) {
          const int t = tid - TC_THREADS / 2 + k * (TC_THREADS / 2), ql = t / TC_N, i = t - ql * TC_N;
          if (t >= TC_N * TC_PTS) break;
          float h[16], l[16];
          tc_row16(Bv[k], g[k], i % 3, h, l);   // row0 is a multiple of 3
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int o = tc_off(i, ql * 16 + 4 * c);
            *reinterpret_cast<float4 *>(Nhi + o) = make_float4(h[4 * c], h[4 * c + 1], h[4 * c + 2], h[4 * c + 3]);
            *reinterpret_cast<float4 *>(Nlo + o) = make_float4(l[4 * c], l[4 * c + 1], l[4 * c + 2], l[4 * c + 3]);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
    }
    if (!__syncthreads_and(w)) {
      ok = false;
      break;
    }
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int kk = 0; kk < TC_KB / 8; ++kk)
#pragma unroll
        for (int p = 0; p < 3; ++p) {   // hi hi, then the columns' lo, then the rows' lo
          const uint32_t Mx = tmem + (uint32_t)((p == 1 ? TC_COL_LO : TC_COL_HI) + kk * 8);
          const float *Nx = (p == 2 ? Nlo : Nhi) + kk * 64;
          const uint32_t acc = (kb | kk | p) != 0;
          asm volatile("{\n\t.reg .pred pa;\n\tsetp.ne.b32 pa, %4, 0;\n\t"
                       "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, pa;\n\t}"
                       ::"r"(tmem), "r"(Mx), "l"(tc_desc(Nx)), "r"(idesc), "r"(acc)
                       : "memory");
        }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_saddr(bar))
                   : "memory");
      if (kb + 2 < nkb) {   // every thread has read the point data of kb
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        fetch(kb + 2);
      }
    }
    if (kb + 2 < nkb) ++fetched;
  }
  // the last commit covers every earlier MMA of this thread
  const bool fin = ok ? tc_wait(bar, (unsigned)(nkb - 1) & 1u) : false;
  ok = __syncthreads_and(fin);
  if (!ok && tid == 0) atomicOr(A.status, ST_TIMEOUT);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok) {
    // warp w reads TMEM lanes 32 (w % 4) .. +31 and 48 of the 192 rows (16 nodes)
    constexpr int CW = TC_N / (TC_THREADS / 128);
    static_assert(CW % 3 == 0 && CW % 16 == 0, "whole nodes, 16 columns a load");
    const int lanes = (warp & 3) * 32, cbeg = (warp >> 2) * CW;
    const int gj = col0 + lanes + lane, b = gj / 3, cj = gj - 3 * b;
    uint32_t r[CW];
#pragma unroll
    for (int c0 = 0; c0 < CW; c0 += 16)
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                   : "=r"(r[c0]), "=r"(r[c0 + 1]), "=r"(r[c0 + 2]), "=r"(r[c0 + 3]), "=r"(r[c0 + 4]), "=r"(r[c0 + 5]),
                     "=r"(r[c0 + 6]), "=r"(r[c0 + 7]), "=r"(r[c0 + 8]), "=r"(r[c0 + 9]), "=r"(r[c0 + 10]),
                     "=r"(r[c0 + 11]), "=r"(r[c0 + 12]), "=r"(r[c0 + 13]), "=r"(r[c0 + 14]), "=r"(r[c0 + 15])
                   : "r"(tmem + ((uint32_t)lanes << 16) + (uint32_t)(cbeg + c0)));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (gj < n) {
      float *K = A.Kf + ((size_t)e * npe + b) * A.cs + cj;
      const int a0 = (row0 + cbeg) / 3;
#pragma unroll
      for (int u = 0; u < CW; ++u)
        if (a0 + u / 3 < npe) K[(a0 + u / 3) * kf_bstride(3, true, 4) + (u % 3) * 3] = __uint_as_float(r[u]);
    }
  } else {
    // drain this CTA's point-data copies (bounded) before it exits: copy k of
    // buffer k & 1 is that buffer's (k >> 1)-th phase
    for (int k = 0; k < fetched; ++k) tc_wait(bar + 1 + (k & 1), (unsigned)(k >> 1) & 1u);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TC_COLS) : "memory");
}

size_t tl_smem(int npe, int nip) {
  return sizeof(double) * ((size_t)npe * 12 + (size_t)nip * QM + (size_t)npe * 39);
}

int fill_args(llf_ctx *ctx, llf_mesh *mesh, const double *T, int law, const double *params,
              int nparams, TLArgs &a) {
  a.xyz = mesh->d_xyz;
  a.conn = mesh->d_conn;
  a.emat = mesh->d_emat;
  a.nel = mesh->nel;
  a.npe = mesh->npe;
  a.nip = mesh->nip;
  a.npairs = mesh->npe * (mesh->npe + 1) / 2;
  a.w = mesh->d_w;
  a.N = mesh->d_N;
  a.dN = mesh->d_dN;
  a.T = T;
  a.law = law;
  a.status = ctx->d_status;
  for (int i = 0; i < 36; ++i) a.prm[i] = 0.0;
  if (law == LLF_LAW_CONSTANT_C) {
    if (nparams != 36 || !params) return llf_fail(ctx, LLF_ERR_ARG, "constant tangent needs 36 parameters (6x6)");
  } else if (law == LLF_LAW_NEOHOOKE_COMP || law == LLF_LAW_SVK) {
    if (nparams < 2 || !params) return llf_fail(ctx, LLF_ERR_ARG, "law needs parameters (mu, lambda)");
  } else {
    return llf_fail(ctx, LLF_ERR_UNSUPPORTED, "unknown hyperelastic law");
  }
  for (int i = 0; i < nparams && i < 36; ++i) a.prm[i] = params[i];
  return LLF_OK;
}

// Elements per CTA of k_tl_packed: the count whose node pairs fill their
// warps best within TLP_THREADS threads and 110 KB of shared memory (two
// CTAs per SM), the larger one of equals; 0 when one element does not fit.  A
// mesh that would leave SMs idle puts fewer in a CTA (216 hex8: 94 us with ten
// in each of 22 CTAs).
int packed_elements(const TLArgs &a, size_t per_elem, int sms) {
  int best = 0;
  double fill = 0.0;
  for (int E = 1; E * a.npairs <= TLP_THREADS && E * per_elem <= 110 * 1024; ++E) {
    const double f = (double)(E * a.npairs) / ((E * a.npairs + 31) / 32 * 32);
    if (f >= fill) {
      fill = f;
      best = E;
    }
  }
  return (int)std::min<int64_t>(best, std::max<int64_t>(1, (a.nel + sms - 1) / sms));
}

template <int MODE>
int launch_matrix(llf_ctx *ctx, TLArgs a, size_t smem) {
  const char *name = MODE == TL_KMAT ? "k_tl_material" : (MODE == TL_KTAN ? "k_tl_tangent" : "k_tl_geometric");
  const size_t per_elem = sizeof(double) * ((size_t)a.npe * 3 + (size_t)a.nip * QD + (size_t)a.nip * a.npe * 3 +
                                            (size_t)a.npe * 39);
  if (const int E = packed_elements(a, per_elem, ctx->num_sms)) {
    auto fn = k_tl_packed<MODE>;
    const size_t sp = E * per_elem;
    const int threads = (E * a.npairs + 31) / 32 * 32;
    if (sp > 48 * 1024)
      LLF_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sp));
    int per_sm = 1;
    LLF_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, sp));
    const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)ctx->num_sms * std::max(per_sm, 1),
                                                                (a.nel + E - 1) / E));
    KernelScope ks(ctx, name);
    fn<<<(unsigned)grid, threads, sp, ctx->stream>>>(a, E);
    LLF_CUDA_TRY(ctx, cudaGetLastError());
    return LLF_OK;
  }
  auto fn = k_tl_matrix<MODE>;
  if (smem > 48 * 1024)
    LLF_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 1;
  LLF_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, TL_THREADS, smem));
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)ctx->num_sms * std::max(per_sm, 1), a.nel));
  KernelScope ks(ctx, name);
  fn<<<(unsigned)grid, TL_THREADS, smem, ctx->stream>>>(a);
  LLF_CUDA_TRY(ctx, cudaGetLastError());
  return LLF_OK;
}

int tl_matrix(llf_ctx *ctx, llf_mesh *mesh, llf_pattern *pat, int mode, const double *dT, int law,
              const double *params, int nparams, llf_matrix *m) {
  if (mesh->dim != 3 || pat->pdim != 3)
    return llf_fail(ctx, LLF_ERR_ARG, "Total Lagrangian operators need dim == 3 and pdim == 3");
  TLArgs a{};
  int rc = fill_args(ctx, mesh, dT, law, params, nparams, a);
  if (rc) return rc;
  size_t smem = tl_smem(mesh->npe, mesh->nip);
  if (smem > 200 * 1024) return llf_fail(ctx, LLF_ERR_LIMIT, "element too large for the TL kernels");
  const bool mat = (mode == TL_KMAT || mode == TL_KTAN);
  const int BS = mat ? 9 : 1;
  double *Kp = nullptr;
  int64_t *cnt = nullptr;
  LLF_CUDA_TRY(ctx, dalloc(ctx, &Kp, (size_t)mesh->nel * mesh->npe * mesh->npe * BS));
  LLF_CUDA_TRY(ctx, dalloc(ctx, &cnt, pat->ndof + 1));
  LLF_CUDA_TRY(ctx, cudaMemsetAsync(cnt, 0, sizeof(int64_t) * (pat->ndof + 1), ctx->stream));
  a.out = Kp;
  rc = (mode == TL_KMAT) ? launch_matrix<TL_KMAT>(ctx, a, smem)
       : (mode == TL_KTAN) ? launch_matrix<TL_KTAN>(ctx, a, smem)
       : (mode == TL_KGEO_S ? launch_matrix<TL_KGEO_S>(ctx, a, smem) : launch_matrix<TL_KGEO_C>(ctx, a, smem));
  if (rc == LLF_OK) {
    cudaError_t e = dalloc(ctx, &m->d_nz, pat->nnz);
    rc = (e == cudaSuccess) ? gather_full(ctx, pat, Kp, (int64_t)mesh->npe * BS, mat, m->d_nz, cnt)
                            : llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e));
  }
  dfree(ctx, Kp);
  if (rc == LLF_OK) rc = llf_check_status(ctx, mat ? "materialTangentMatrix" : "initialStressMatrix");
  if (rc == LLF_OK) rc = matrix_finalize(ctx, m, cnt);
  dfree(ctx, cnt);
  return rc;
}

}  // namespace

int tl_material_tangent_impl(llf_ctx *ctx, llf_mesh *mesh, llf_pattern *pat, const double *d_F,
                             int law, const double *params, int nparams, llf_matrix *m) {
  return tl_matrix(ctx, mesh, pat, TL_KMAT, d_F, law, params, nparams, m);
}

int tl_tangent_impl(llf_ctx *ctx, llf_mesh *mesh, llf_pattern *pat, const double *d_F, int law,
                    const double *params, int nparams, llf_matrix *m) {
  return tl_matrix(ctx, mesh, pat, TL_KTAN, d_F, law, params, nparams, m);
}

// Tensor-core form of the consistent tangent (k_tl_points_tc + k_tl_tangent_tc,
// then the FP32 element matrices summed in FP64 by the gather).
namespace {
// Exact symmetry of the tensor-core element matrices: the tiles above and
// below the diagonal round their FP32 sums differently, so block (b,a) is
// not quite block (a,b)^T.  Each mirrored pair of entries is replaced by
// their mean, so the gathered tangent is symmetric bit for bit (CG relies
// on it; unsymmetric rounding cost it about twice the iterations).  One
// thread per element and node pair a <= b, a block of 256 threads per
// 16 x 16 tile of node pairs: a warp holds four row nodes by eight column
// nodes, so its 48-byte blocks are runs of 192 bytes on one side of the
// diagonal and 384 on the other, each block moved as three 16-byte words.
// Bound by HBM (the element matrices read and written once): hex125, 576
// elements, 432 MB: 1.12 ms with a thread per pair in pair order and scalar
// accesses, 0.16 ms now.
constexpr int SYM_TILE = 16;
__global__ void __launch_bounds__(SYM_TILE * SYM_TILE)
k_tc_symmetrize(float *__restrict__ Kf, int npe, int64_t cs, int tiles, int tpe) {
  constexpr int BSTR = kf_bstride(3, true, 4);
  static_assert(BSTR == 12, "a block is three 16-byte words");
  const int64_t e = blockIdx.x / tpe;
  int p = (int)(blockIdx.x - e * tpe), ta = 0;
  while (p >= tiles - ta) {  // tile index -> (ta, tb >= ta), row by row
    p -= tiles - ta;
    ++ta;
  }
  const int t = threadIdx.x;
  const int a = ta * SYM_TILE + (t & 3) + 4 * ((t >> 5) & 3), b = (ta + p) * SYM_TILE + ((t >> 2) & 7) + 8 * (t >> 7);
  if (a > b || b >= npe) return;
  float4 *X = reinterpret_cast<float4 *>(Kf + ((size_t)e * npe + b) * cs + (size_t)a * BSTR);  // block (a, b)
  float4 *Y = reinterpret_cast<float4 *>(Kf + ((size_t)e * npe + a) * cs + (size_t)b * BSTR);  // block (b, a)
  float x[BSTR], y[BSTR];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    *reinterpret_cast<float4 *>(x + 4 * k) = X[k];
    *reinterpret_cast<float4 *>(y + 4 * k) = Y[k];
  }
#pragma unroll
  for (int ci = 0; ci < 3; ++ci)
#pragma unroll
    for (int cj = 0; cj < 3; ++cj) {
      if (a == b && cj <= ci) continue;
      const float m = (x[ci * 3 + cj] + y[cj * 3 + ci]) * 0.5f;
      x[ci * 3 + cj] = m;
      y[cj * 3 + ci] = m;
      if (a == b) x[cj * 3 + ci] = m;   // one block
    }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    X[k] = *reinterpret_cast<float4 *>(x + 4 * k);
    if (a != b) Y[k] = *reinterpret_cast<float4 *>(y + 4 * k);
  }
}
}  // namespace

int tl_tangent_tc_impl(llf_ctx *ctx, llf_mesh *mesh, llf_pattern *pat, const double *d_F, int law,
                       const double *params, int nparams, llf_matrix *m) {
  if (mesh->dim != 3 || pat->pdim != 3)
    return llf_fail(ctx, LLF_ERR_ARG, "Total Lagrangian operators need dim == 3 and pdim == 3");
  TLArgs a{};
  int rc = fill_args(ctx, mesh, d_F, law, params, nparams, a);
  if (rc) return rc;
  const int npe = mesh->npe, nip = mesh->nip, n = 3 * npe;
  cudaStream_t s = ctx->stream;
  float *pd = nullptr;
  float *Kf = nullptr;
  int64_t *cnt = nullptr;
  const int ps = tc_pstride(npe);
  const int64_t cs = kf_colstride(npe, kf_bstride(3, true, (int)sizeof(float)), (int)sizeof(float));
  LLF_CUDA_TRY(ctx, dalloc(ctx, &pd, (size_t)mesh->nel * nip * ps));
  LLF_CUDA_TRY(ctx, dalloc(ctx, &Kf, (size_t)mesh->nel * npe * cs));
  LLF_CUDA_TRY(ctx, dalloc(ctx, &cnt, pat->ndof + 1));
  LLF_CUDA_TRY(ctx, cudaMemsetAsync(cnt, 0, sizeof(int64_t) * (pat->ndof + 1), s));
  {
    const size_t smem = sizeof(double) * ((size_t)npe * 12 + (size_t)nip * QD);   // 203 KB at most
    if (sizeof(double) * ((size_t)npe * 12 + (size_t)nip * QM) > 200 * 1024)
      rc = llf_fail(ctx, LLF_ERR_LIMIT, "tensor-core tangent: element too large");
    if (rc == LLF_OK && smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(k_tl_points_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e));
    }
    if (rc == LLF_OK) {
      const unsigned grid = (unsigned)std::min<int64_t>(std::max<int64_t>(mesh->nel, 1), (int64_t)ctx->num_sms * 4);
      KernelScope ks(ctx, "k_tl_points_tc");
      k_tl_points_tc<<<grid, TL_THREADS, smem, s>>>(a, pd);
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e));
    }
  }
  TcArgs t{};
  t.pd = pd;
  t.emat = mesh->d_emat;
  t.nel = mesh->nel;
  t.npe = npe;
  t.nip = nip;
  t.n = n;
  t.nstrip = (n + TC_M - 1) / TC_M;
  t.nhalf = (n + TC_N - 1) / TC_N;
  t.Kf = Kf;
  t.cs = cs;
  t.status = ctx->d_status;
  // at least 80 KB, so that at most two CTAs, whose tensor memory fits, share an SM
  const size_t smem = std::max<size_t>(80 * 1024, sizeof(float) * (2 * TC_TILE + 2 * (size_t)TC_PTS * ps) +
                                                      3 * sizeof(uint64_t) + 16);
  if (rc == LLF_OK && smem > 220 * 1024) rc = llf_fail(ctx, LLF_ERR_LIMIT, "tensor-core tangent: element too large");
  const int64_t ctas = mesh->nel * t.nstrip * t.nhalf;
  if (rc == LLF_OK && ctas >= ((int64_t)1 << 31)) rc = llf_fail(ctx, LLF_ERR_LIMIT, "tensor-core tangent: too many tiles");
  if (rc == LLF_OK && ctas > 0) {
    cudaError_t e = cudaFuncSetAttribute(k_tl_tangent_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e));
    if (rc == LLF_OK) {
      KernelScope ks(ctx, "k_tl_tangent_tc");
      k_tl_tangent_tc<<<(unsigned)ctas, TC_THREADS, smem, s>>>(t);
      e = cudaGetLastError();
      if (e != cudaSuccess) rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e));
    }
  }
  if (rc == LLF_OK && mesh->nel > 0) {
    const int tiles = (npe + SYM_TILE - 1) / SYM_TILE, tpe = tiles * (tiles + 1) / 2;
    const int64_t per = ((int64_t)1 << 30) / tpe;   // elements per launch
    for (int64_t e0 = 0; e0 < mesh->nel; e0 += per) {
      KernelScope ks(ctx, "k_tc_symmetrize");
      k_tc_symmetrize<<<(unsigned)(std::min(per, mesh->nel - e0) * tpe), SYM_TILE * SYM_TILE, 0, s>>>(
          Kf + (size_t)e0 * npe * cs, npe, cs, tiles, tpe);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e));
  }
  if (rc == LLF_OK) {
    cudaError_t e = dalloc(ctx, &m->d_nz, pat->nnz);
    rc = (e == cudaSuccess) ? gather_full32(ctx, pat, Kf, cs, true, m->d_nz, cnt)
                            : llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e));
  }
  dfree(ctx, pd);
  dfree(ctx, Kf);
  if (rc == LLF_OK) rc = llf_check_status(ctx, "tangent (tensor-core form)");
  if (rc == LLF_OK) rc = matrix_finalize(ctx, m, cnt);
  dfree(ctx, cnt);
  return rc;
}

int tl_initial_stress_impl(llf_ctx *ctx, llf_mesh *mesh, llf_pattern *pat, const double *d_S,
                           const double *d_C, int law, const double *params, int nparams,
                           llf_matrix *m) {
  if (d_S) {
    double dummy[2] = {0.0, 0.0};
    return tl_matrix(ctx, mesh, pat, TL_KGEO_S, d_S, LLF_LAW_NEOHOOKE_COMP, dummy, 2, m);
  }
  return tl_matrix(ctx, mesh, pat, TL_KGEO_C, d_C, law, params, nparams, m);
}

int tl_internal_force_impl(llf_ctx *ctx, llf_mesh *mesh, const double *d_P, const double *d_F,
                           int law, const double *params, int nparams, double *d_f) {
  TLArgs a{};
  int rc;
  if (d_P) {
    double dummy[2] = {0.0, 0.0};
    rc = fill_args(ctx, mesh, d_P, LLF_LAW_NEOHOOKE_COMP, dummy, 2, a);
  } else {
    rc = fill_args(ctx, mesh, d_F, law, params, nparams, a);
  }
  if (rc) return rc;
  // elements per CTA: as many as fill the CTA's threads with points and nodes,
  // or, where that leaves at most two CTAs per SM, with points and node
  // components in one round (48 tet35: 152 and 115 us, 64 hex27 65 and 53, 216
  // hex8 35 and 28; with more CTAs the repeated gradients cost more than the
  // shorter chain saves: 512 hex27 65 and 82)
  const size_t per_elem = sizeof(double) * ((size_t)mesh->npe * 12 + (size_t)mesh->nip * QF);
  const int fit = (int)((100 * 1024) / per_elem);
  const int E1 = std::max(1, std::min(TL_THREADS / std::max(3 * mesh->npe, mesh->nip), fit));
  const bool few = 3 * mesh->npe <= TL_THREADS && (mesh->nel + E1 - 1) / E1 <= 2 * (int64_t)ctx->num_sms;
  const int E = few ? E1 : std::max(1, std::min(TL_THREADS / std::max(mesh->npe, mesh->nip), fit));
  const size_t smem = E * per_elem;
  if (smem > 200 * 1024) return llf_fail(ctx, LLF_ERR_LIMIT, "element too large for the TL kernels");
  double *fe = nullptr;
  LLF_CUDA_TRY(ctx, dalloc(ctx, &fe, (size_t)mesh->nel * mesh->npe * 3));
  a.out = fe;
  auto go = [&](auto fn) -> int {
    if (smem > 48 * 1024)
      LLF_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 1;
    LLF_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, TL_THREADS, smem));
    const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)ctx->num_sms * std::max(per_sm, 1),
                                                                (mesh->nel + E - 1) / E));
    KernelScope ks(ctx, "k_tl_force");
    fn<<<(unsigned)grid, TL_THREADS, smem, ctx->stream>>>(a, E);
    LLF_CUDA_TRY(ctx, cudaGetLastError());
    return LLF_OK;
  };
  if (few)
    rc = d_P ? go(k_tl_force<TL_KGEO_S, 1>) : go(k_tl_force<TL_FORCE, 1>);
  else
    rc = d_P ? go(k_tl_force<TL_KGEO_S, 3>) : go(k_tl_force<TL_FORCE, 3>);
  if (rc == LLF_OK) {
    LLF_CUDA_TRY(ctx, cudaMemsetAsync(d_f, 0, sizeof(double) * 3 * mesh->non, ctx->stream));
    rc = node_gather(ctx, mesh->d_conn, mesh->nel, mesh->npe, mesh->non, 3, fe, d_f);
  }
  dfree(ctx, fe);
  if (rc) return rc;
  return llf_check_status(ctx, "internalForceVector");
}
