// Element-operator assembly into the reference's CSC layout.
//
// Pipeline (one call of llf_assemble_*):
//   geometry      k_affine_geometry, once per mesh geometry (kept on the
//                 device mesh): which elements are affine images of the
//                 reference element (and which of those are axis-aligned
//                 bricks), with their J^-1 and det;
//   k_elem_packed elements of up to 384 node pairs: as many per CTA as fill
//                 its threads (one hex27, eight hex8), after k_affine_coeff
//                 has formed the affine ones' coefficients;
//   k_elem_affine conduction of tet35, mass of tet35 and hex64 on meshes whose
//                 elements are all affine (larger elements whose matrix and
//                 table fit in shared memory): one CTA per element at a time
//                 (persistent), the entries formed from the reference pair
//                 tables into a shared-memory image of the element matrix,
//                 which one bulk store writes out;
//   k_elem_fp64   other elements: one CTA per element at a time, element node
//                 coordinates gathered into shared memory, the reference
//                 shape gradients staged in shared memory for the CTA's
//                 lifetime (read from global memory for elements whose tables
//                 do not fit), Jacobian / inverse / physical gradients per
//                 integration point (the affine form for affine elements),
//                 then the upper-triangle node-pair blocks, each written
//                 twice (block and mirror).  All three leave the element
//                 matrix whole in the layout Kf[element][column node b][row
//                 node a][block];
//   k_colgather   (gather.cu) sums every entry over its elements in element
//                 order, the order SparseArrays.sparse combines the
//                 reference's triplets (src/linear.jl:314-323), and writes
//                 the column with its non-zero count, or, when the pattern
//                 kept the stored layout of an earlier assembly of the same
//                 operator and form, compacted straight into it (dropzeros!,
//                 every column's count checked);
//   finalize      otherwise dropzeros! (src/linear.jl:324): scan of the
//                 counts, then compaction into 1-based Int64 SparseMatrixCSC
//                 arrays, whose column starts the pattern keeps.
// Every floating-point operation of the FP64 form is an explicit IEEE
// intrinsic (__dmul_rn, __dadd_rn, __fma_rn, __drcp_rn), so no contraction
// or reassociation can move the result away from the CPU oracle's.
#include "common.cuh"
#include "affine.cuh"

#include <algorithm>

namespace {

constexpr int ELEM_THREADS = 128;

struct ElemArgs {
  const double *xyz;
  const int32_t *conn;
  const int32_t *emat;
  int64_t nel;
  int npe, nip, npairs;
  const double *w, *N, *dN;  // device tables
  const double *c1, *c2;     // per-material coefficients
  double *Kf;                // nel * npe * colstride (full element matrices)
  int64_t colstride;         // doubles per element-matrix column (16-byte multiple)
  double *scratch;           // per-CTA global scratch for G, S (large elements)
  int64_t scratch_stride;    // doubles per CTA
  unsigned *status;
  // affine-element form: per-element flag and invJ/det (k_affine_geometry;
  // aflag null = none), and per upper-triangle node pair in pair order the
  // symmetric [0,NS) and antisymmetric [6,6+NA) parts of R_ab, and Mref_ab
  const uint8_t *aflag;
  const double *ageo, *Rp, *Mp;
  int cta_cap;               // host side: CTAs per SM at most (0: as many as fit)
  bool all_affine, any_affine;  // host side: k_affine_geometry counted no non-affine element, met an affine one
};

__device__ __forceinline__ int pair_offset(int a, int npe) {
  return a * npe - (a * (a - 1)) / 2;
}
__device__ __forceinline__ void pair_decode(int pi, int npe, int &a, int &b) {
  int lo = 0, hi = npe - 1;
  while (lo < hi) {  // largest a with pair_offset(a) <= pi
    int mid = (lo + hi + 1) >> 1;
    if (pair_offset(mid, npe) <= pi) lo = mid; else hi = mid - 1;
  }
  a = lo;
  b = a + (pi - pair_offset(a, npe));
}

// Geometry at one point (contract of the oracle): returns det, fills inv
// (row-major invJ[i][j]).  dNq(a, j) is the reference gradient of node a.
template <int DIM, class Tab>
__device__ __forceinline__ double geom_point(const double *sX, Tab dNq, int npe, double *inv) {
  double J[3][3];
#pragma unroll
  for (int i = 0; i < DIM; ++i)
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      double acc = 0.0;
      for (int a = 0; a < npe; ++a) acc = __fma_rn(sX[a * DIM + i], dNq(a, j), acc);
      J[i][j] = acc;
    }
  return jac_inverse<DIM>(J, inv);
}

// Store block (a,b) (a <= b) of the element matrix and its mirror (b,a) in
// the column-major-by-node layout Kf[e][col node][row node][i*P+j].
template <int P, int BS>
__device__ __forceinline__ void store_pair(double *Ke, int64_t cs, int a, int b, const double *blk) {
  double *ab = Ke + (size_t)b * cs + (size_t)a * BS;  // rows of node a, columns of node b
#pragma unroll
  for (int k = 0; k < BS; ++k) ab[k] = blk[k];
  if (a != b) {
    double *ba = Ke + (size_t)a * cs + (size_t)b * BS;
    if (BS == 1) {
      ba[0] = blk[0];
    } else {
#pragma unroll
      for (int i = 0; i < P; ++i)
#pragma unroll
        for (int j = 0; j < P; ++j) ba[j * P + i] = blk[i * P + j];
    }
  }
}

// Node-pair blocks of an affine element (contract of the oracle): per pair
// the symmetric part S (NS values) and antisymmetric part A (NA values) of
// R_ab; elasticity Ksym = W S, Kanti = U A (a != b), heat (c1 trV) . S, mass
// (c1 det) Mref_ab.
// ALIGNED (axis-aligned elements, flag 2 of k_affine_geometry, whose
// coefficients affine_stage_aligned forms): elasticity through the
// collapsed Lame combination of the oracle's orc_element_aligned, 15 FP64
// operations per node pair in 3D instead of 51; heat leaves the mixed
// components, whose coefficients are exact zeros there, out of its fma
// chain (a left-out fma(+-0, s, acc) returns acc whenever acc is non-zero,
// so the value is the full chain's up to the sign of a zero result, and
// zeros are dropped from the stored CSC and add nothing to a non-zero sum).
// Rp, Mp: the pair tables in global memory (read through the read-only
// path) or, with TAB_SMEM, in shared memory.
template <bool TAB_SMEM>
__device__ __forceinline__ double ld_tab(const double *p) {
  if (TAB_SMEM) return *p;
  return __ldg(p);
}

template <int KIND, int DIM, int P, int BS, bool ALIGNED, bool TAB_SMEM = false>
__device__ __forceinline__ void affine_pairs(const ElemArgs &A, const double *sAff, double *Ke,
                                             const double *Rp, const double *Mp) {
  constexpr int NS = DIM == 3 ? 6 : 3, NA = DIM == 3 ? 3 : 1;
  const int npe = A.npe;
  if (KIND == KIND_MASS) {
    const double cm = sAff[AF_M];
    for (int pi = threadIdx.x; pi < A.npairs; pi += blockDim.x) {
      int a, b;
      pair_decode(pi, npe, a, b);
      double blk[BS];
      blk[0] = __dmul_rn(cm, ld_tab<TAB_SMEM>(Mp + pi));
      store_pair<P, BS>(Ke, A.colstride, a, b, blk);
    }
  } else if (KIND == KIND_HEAT) {
    double Q[NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) Q[n] = (!ALIGNED || n < DIM) ? sAff[AF_Q + n] : 0.0;
    for (int pi = threadIdx.x; pi < A.npairs; pi += blockDim.x) {
      int a, b;
      pair_decode(pi, npe, a, b);
      const double *sp = Rp + (size_t)pi * 9;
      double acc = 0.0;
#pragma unroll
      for (int n = 0; n < (ALIGNED ? DIM : NS); ++n) acc = __fma_rn(Q[n], ld_tab<TAB_SMEM>(sp + n), acc);
      double blk[BS];
      blk[0] = acc;
      store_pair<P, BS>(Ke, A.colstride, a, b, blk);
    }
  } else if (ALIGNED) {
    // axis-aligned elasticity (contract of the oracle's orc_element_aligned):
    // g = sum beta_n S_n, K_ii = fma(alpha_i, S_i, g), h = b_m A_m,
    // K_ij = fma(a_m, S_m, h), K_ji = fma(a_m, S_m, -h); a == b: a_m S_m
    double al[DIM], be[DIM], am[NA], bm[NA];
#pragma unroll
    for (int i = 0; i < DIM; ++i) {
      al[i] = sAff[AF_W + i];
      be[i] = sAff[AF_W + DIM + i];
    }
#pragma unroll
    for (int m = 0; m < NA; ++m) {
      am[m] = sAff[AF_W + 2 * DIM + m];
      bm[m] = sAff[AF_W + 2 * DIM + NA + m];
    }
    for (int pi = threadIdx.x; pi < A.npairs; pi += blockDim.x) {
      int a, b;
      pair_decode(pi, npe, a, b);
      const double *sp = Rp + (size_t)pi * 9;
      double sv[NS], av[NA];
#pragma unroll
      for (int n = 0; n < NS; ++n) sv[n] = ld_tab<TAB_SMEM>(sp + n);
#pragma unroll
      for (int n = 0; n < NA; ++n) av[n] = ld_tab<TAB_SMEM>(sp + 6 + n);
      double g = __dmul_rn(be[0], sv[0]);
#pragma unroll
      for (int n = 1; n < DIM; ++n) g = __fma_rn(be[n], sv[n], g);
      double blk[BS];
#pragma unroll
      for (int i = 0; i < DIM; ++i) blk[i * DIM + i] = __fma_rn(al[i], sv[i], g);
#pragma unroll
      for (int m = 0; m < NA; ++m) {
        const int i = sym_k<DIM>(DIM + m), j = sym_l<DIM>(DIM + m);
        if (a != b) {
          const double h = __dmul_rn(bm[m], av[m]);
          blk[i * DIM + j] = __fma_rn(am[m], sv[DIM + m], h);
          blk[j * DIM + i] = __fma_rn(am[m], sv[DIM + m], -h);
        } else {
          const double v = __dmul_rn(am[m], sv[DIM + m]);
          blk[i * DIM + j] = v;
          blk[j * DIM + i] = v;
        }
      }
      store_pair<P, BS>(Ke, A.colstride, a, b, blk);
    }
  } else {
    double W[NS * NS], U[NA * NA];
#pragma unroll
    for (int t = 0; t < NS * NS; ++t) W[t] = sAff[AF_W + t];
#pragma unroll
    for (int t = 0; t < NA * NA; ++t) U[t] = sAff[AF_U + t];
    for (int pi = threadIdx.x; pi < A.npairs; pi += blockDim.x) {
      int a, b;
      pair_decode(pi, npe, a, b);
      const double *sp = Rp + (size_t)pi * 9;
      double sv[NS], av[NA];
#pragma unroll
      for (int n = 0; n < NS; ++n) sv[n] = ld_tab<TAB_SMEM>(sp + n);
#pragma unroll
      for (int n = 0; n < NA; ++n) av[n] = ld_tab<TAB_SMEM>(sp + 6 + n);
      double ks[NS];
#pragma unroll
      for (int m = 0; m < NS; ++m) {
        double acc = 0.0;
#pragma unroll
        for (int n = 0; n < NS; ++n) acc = __fma_rn(W[m * NS + n], sv[n], acc);
        ks[m] = acc;
      }
      double blk[BS];
#pragma unroll
      for (int i = 0; i < DIM; ++i) blk[i * DIM + i] = ks[i];
      if (a != b) {
#pragma unroll
        for (int m = 0; m < NA; ++m) {
          double acc = 0.0;
#pragma unroll
          for (int n = 0; n < NA; ++n) acc = __fma_rn(U[m * NA + n], av[n], acc);
          const int i = sym_k<DIM>(DIM + m), j = sym_l<DIM>(DIM + m);
          blk[i * DIM + j] = __dadd_rn(ks[DIM + m], acc);
          blk[j * DIM + i] = __dsub_rn(ks[DIM + m], acc);
        }
      } else {
#pragma unroll
        for (int m = 0; m < NA; ++m) {
          const int i = sym_k<DIM>(DIM + m), j = sym_l<DIM>(DIM + m);
          blk[i * DIM + j] = ks[DIM + m];
          blk[j * DIM + i] = ks[DIM + m];
        }
      }
      store_pair<P, BS>(Ke, A.colstride, a, b, blk);
    }
  }
}

// Shared-memory layout of k_elem_fp64 (doubles):
//   [SMEM] sdN [nip*npe*DIM] | sw [nip] | sN [nip*npe] (mass) |
//   sX [npe*DIM] | sWd [nip] | sInv [nip*9] | sAff [32] | [SMEM] G, S (each nip*npe*gsw)
// Without SMEM the tables are read from global memory (stride 3) and G, S
// live in a per-CTA global scratch slot (L2 resident).
template <int KIND, int DIM, bool SMEM>
__global__ void __launch_bounds__(ELEM_THREADS)
k_elem_fp64(ElemArgs A) {
  extern __shared__ double smem[];
  const int npe = A.npe, nip = A.nip;
  constexpr int gsw = (KIND == KIND_MASS) ? 1 : DIM;
  double *sdN = smem;
  double *sw = sdN + (SMEM ? (size_t)nip * npe * DIM : 0);
  double *sN = sw + (SMEM ? nip : 0);
  double *sX = sN + ((SMEM && KIND == KIND_MASS) ? (size_t)nip * npe : 0);
  double *sWd = sX + (size_t)npe * DIM;
  double *sInv = sWd + nip;
  double *sAff = sInv + (size_t)nip * 9;  // affine-form scratch (AF_* offsets)
  double *G = SMEM ? (sAff + AFF_DOUBLES) : (A.scratch + (size_t)blockIdx.x * A.scratch_stride);
  double *S = G + (size_t)nip * npe * gsw;
  // table accessors
  const int tstride = SMEM ? DIM : 3;
  const double *tdN = SMEM ? sdN : A.dN;
  const double *tw = SMEM ? sw : A.w;
  const double *tN = SMEM ? sN : A.N;

  if (SMEM) {
    for (int t = threadIdx.x; t < nip * npe * DIM; t += blockDim.x) {
      int j = t % DIM, qa = t / DIM;
      sdN[t] = A.dN[(size_t)qa * 3 + j];
    }
    for (int t = threadIdx.x; t < nip; t += blockDim.x) sw[t] = A.w[t];
    if (KIND == KIND_MASS)
      for (int t = threadIdx.x; t < nip * npe; t += blockDim.x) sN[t] = A.N[t];
    __syncthreads();
  }

  constexpr int BS = (KIND == KIND_ELASTIC) ? DIM * DIM : 1;
  constexpr int P = (KIND == KIND_ELASTIC) ? DIM : 1;
  for (int64_t e = blockIdx.x; e < A.nel; e += gridDim.x) {
    const int mat = A.emat ? A.emat[e] : 0;
    if (mat < 0) continue;  // uniform across the CTA
    const double c1 = A.c1[mat];
    const double c2 = (KIND == KIND_ELASTIC) ? A.c2[mat] : 0.0;
    double *Ke = A.Kf + (size_t)e * npe * A.colstride;
    if (A.aflag && A.aflag[e]) {  // uniform across the CTA
      const bool aligned = A.aflag[e] == 2;   // uniform across the CTA
      if (threadIdx.x < 32) {
        if (aligned)
          affine_stage_aligned<DIM>(A.ageo + (size_t)e * 10, c1, c2, sAff, A.status, threadIdx.x);
        else
          affine_stage<DIM>(A.ageo + (size_t)e * 10, c1, c2, sAff, A.status, threadIdx.x);
      }
      __syncthreads();
      if (aligned)
        affine_pairs<KIND, DIM, P, BS, true>(A, sAff, Ke, A.Rp, A.Mp);
      else
        affine_pairs<KIND, DIM, P, BS, false>(A, sAff, Ke, A.Rp, A.Mp);
    } else {
      for (int t = threadIdx.x; t < npe * DIM; t += blockDim.x) {
        int a = t / DIM, i = t % DIM;
        sX[t] = A.xyz[(size_t)A.conn[e * npe + a] * 3 + i];
      }
      __syncthreads();
      for (int q = threadIdx.x; q < nip; q += blockDim.x) {
        double inv[9];
        const double *dq = tdN + (size_t)q * npe * tstride;
        double det = geom_point<DIM>(sX, [&](int a, int j) { return dq[a * tstride + j]; }, npe, inv);
        if (!(det > 0.0)) atomicOr(A.status, ST_BAD_JACOBIAN);
        sWd[q] = __dmul_rn(det, tw[q]);
#pragma unroll
        for (int k = 0; k < 9; ++k) sInv[q * 9 + k] = inv[k];
      }
      __syncthreads();
      if (KIND == KIND_MASS) {
        for (int t = threadIdx.x; t < nip * npe; t += blockDim.x) S[t] = __dmul_rn(sWd[t / npe], tN[t]);
      } else {
        for (int t = threadIdx.x; t < nip * npe; t += blockDim.x) {
          const int q = t / npe;
          const double *inv = sInv + q * 9;
          const double *d = tdN + (size_t)t * tstride;
          const double wd = sWd[q];
#pragma unroll
          for (int i = 0; i < DIM; ++i) {
            double acc = 0.0;
#pragma unroll
            for (int j = 0; j < DIM; ++j) acc = __fma_rn(inv[3 * j + i], d[j], acc);
            G[(size_t)t * DIM + i] = acc;
            S[(size_t)t * DIM + i] = __dmul_rn(wd, acc);
          }
        }
      }
      __syncthreads();

      for (int pi = threadIdx.x; pi < A.npairs; pi += blockDim.x) {
        int a, b;
        pair_decode(pi, npe, a, b);
        double blk[BS];
        if (KIND == KIND_ELASTIC) {
          double O[DIM][DIM];
#pragma unroll
          for (int i = 0; i < DIM; ++i)
#pragma unroll
            for (int j = 0; j < DIM; ++j) O[i][j] = 0.0;
          if (a != b) {
            for (int q = 0; q < nip; ++q) {
              const double *sa = S + ((size_t)q * npe + a) * DIM;
              const double *gb = G + ((size_t)q * npe + b) * DIM;
              double s_[DIM], g_[DIM];
#pragma unroll
              for (int i = 0; i < DIM; ++i) { s_[i] = sa[i]; g_[i] = gb[i]; }
#pragma unroll
              for (int i = 0; i < DIM; ++i)
#pragma unroll
                for (int j = 0; j < DIM; ++j) O[i][j] = __fma_rn(s_[i], g_[j], O[i][j]);
            }
          } else {
            for (int q = 0; q < nip; ++q) {
              const double *sa = S + ((size_t)q * npe + a) * DIM;
              const double *ga = G + ((size_t)q * npe + a) * DIM;
              double s_[DIM], g_[DIM];
#pragma unroll
              for (int i = 0; i < DIM; ++i) { s_[i] = sa[i]; g_[i] = ga[i]; }
#pragma unroll
              for (int i = 0; i < DIM; ++i)
#pragma unroll
                for (int j = i; j < DIM; ++j) O[i][j] = __fma_rn(s_[i], g_[j], O[i][j]);
            }
#pragma unroll
            for (int i = 0; i < DIM; ++i)
#pragma unroll
              for (int j = 0; j < i; ++j) O[i][j] = O[j][i];
          }
          double tr = __dadd_rn(O[0][0], O[1 % DIM][1 % DIM]);
          if (DIM == 3) tr = __dadd_rn(tr, O[2 % DIM][2 % DIM]);
#pragma unroll
          for (int i = 0; i < DIM; ++i)
#pragma unroll
            for (int j = 0; j < DIM; ++j) {
              double t = __fma_rn(c2, O[j][i], __dmul_rn(c1, O[i][j]));
              if (i == j) t = __fma_rn(c2, tr, t);
              blk[i * DIM + j] = t;
            }
        } else if (KIND == KIND_HEAT) {
          double acc = 0.0;
          for (int q = 0; q < nip; ++q) {
            const double *sa = S + ((size_t)q * npe + a) * DIM;
            const double *gb = G + ((size_t)q * npe + b) * DIM;
#pragma unroll
            for (int i = 0; i < DIM; ++i) acc = __fma_rn(sa[i], gb[i], acc);
          }
          blk[0] = __dmul_rn(c1, acc);
        } else {  // mass
          double acc = 0.0;
          for (int q = 0; q < nip; ++q)
            acc = __fma_rn(S[(size_t)q * npe + a], tN[(size_t)q * npe + b], acc);
          blk[0] = __dmul_rn(c1, acc);
        }
        store_pair<P, BS>(Ke, A.colstride, a, b, blk);
      }

    }
    __syncthreads();
  }
}

// Affine-element kernel with staged stores for conduction and mass in 3D, on
// meshes whose elements are all affine (k_affine_geometry counted no other):
// one CTA per element at a time (grid-stride, persistent).  The pair table (the parts of R_ab, or
// Mref_ab) is copied into shared memory once per CTA by a bulk copy
// (cp.async.bulk completing on an mbarrier; a bounded wait).  Each element
// matrix is built in a shared-memory image of its Kf run (the same layout,
// column padding included) and leaves with one bulk store (cp.async.bulk
// global <- shared), which drains while the CTA forms the next element's
// coefficients; the warp that forms them rotates from element to element.
// The arithmetic is affine_pairs', so Kf holds what k_elem_fp64 writes.
// Shared memory: image [npe * colstride] | table [tab_n, even] | sAff |
// mbarrier.
__device__ __forceinline__ uint32_t sh_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ uint64_t now_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait on an mbarrier phase (2 s); false on timeout.
__device__ __forceinline__ bool bar_wait(uint64_t *bar, unsigned parity) {
  const uint64_t t0 = now_ns();
  for (;;) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(sh_addr(bar)), "r"(parity) : "memory");
    if (ok) return true;
    if (now_ns() - t0 > 2000000000ull) return false;
  }
}

constexpr int AFFK_MAX_THREADS = 256;

template <int KIND>
__global__ void __launch_bounds__(AFFK_MAX_THREADS)
k_elem_affine(ElemArgs A, int tab_n) {
  extern __shared__ __align__(128) double smem_a[];
  static_assert(KIND != KIND_ELASTIC, "no elastic element beyond k_elem_packed's fits");
  const int64_t kelems = (int64_t)A.npe * A.colstride;
  const unsigned ke_bytes = (unsigned)(kelems * 8);
  double *sKe = smem_a;
  double *sTab = sKe + kelems;
  double *sAff = sTab + ((tab_n + 1) & ~1);
  uint64_t *bar = reinterpret_cast<uint64_t *>(sAff + AFF_DOUBLES);
  const double *gTab = KIND == KIND_MASS ? A.Mp : A.Rp;
  const unsigned tab_bytes = (unsigned)tab_n * 8u;
  if ((tab_bytes & 15u) == 0 && ((uintptr_t)gTab & 15u) == 0) {
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sh_addr(bar)), "r"(1u) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sh_addr(bar)), "r"(tab_bytes)
                   : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(sh_addr(sTab)), "l"(gTab), "r"(tab_bytes), "r"(sh_addr(bar))
                   : "memory");
    }
    const bool ok = bar_wait(bar, 0);
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) atomicOr(A.status, ST_TIMEOUT);
      return;
    }
  } else {
    for (int t = threadIdx.x; t < tab_n; t += blockDim.x) sTab[t] = gTab[t];
    __syncthreads();
  }
  const int nwarps = (int)(blockDim.x >> 5);
  unsigned iter = 0;
  for (int64_t e = blockIdx.x; e < A.nel; e += gridDim.x, ++iter) {
    const int mat = A.emat ? A.emat[e] : 0;
    if (mat < 0) continue;  // uniform across the CTA
    const double c1 = A.c1[mat];
    const bool aligned = A.aflag[e] == 2;
    if ((int)(threadIdx.x >> 5) == (int)((blockIdx.x + iter) % (unsigned)nwarps)) {
      const int lane = threadIdx.x & 31;
      if (aligned)
        affine_stage_aligned<3>(A.ageo + (size_t)e * 10, c1, 0.0, sAff, A.status, lane);
      else
        affine_stage<3>(A.ageo + (size_t)e * 10, c1, 0.0, sAff, A.status, lane);
    }
    // the previous element's store has read the image
    if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncthreads();
    if (aligned)
      affine_pairs<KIND, 3, 1, 1, true, true>(A, sAff, sKe, sTab, sTab);
    else
      affine_pairs<KIND, 3, 1, 1, false, true>(A, sAff, sKe, sTab, sTab);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
      double *Ke = A.Kf + (size_t)e * kelems;
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(Ke), "r"(sh_addr(sKe)),
                   "r"(ke_bytes)
                   : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
  }
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// One or more elements per CTA (E of them: elements e0 .. e0+E-1 at a time,
// persistent), one node pair per thread, for elements of at most PACK_PAIRS
// node pairs, affine or not.  The FP64 pipe bounds it and is spent per warp
// instruction, and a 128-thread CTA per element filled it badly: 36 of 64
// lanes for hex8's pairs (10 of 128 for tet4 and quad4), about 28
// instructions of one warp for the coefficients of an affine element, where
// its pairs take 6 (hex8 conduction) to 102 (tet10 elasticity), and by points
// 27 lanes of one warp with 240 dependent operations each for a hex27's
// Jacobians.  Here the coefficients come from k_affine_coeff, a thread per
// element (6 warp instructions each), the pairs of the E elements fill their
// warps, and a thread keeps its pair's table row in registers.  The E element
// matrices are formed in a shared-memory image of their Kf run and leave with
// one bulk store.  The next E elements' coefficients and coordinates are
// copied in meanwhile (cp.async, two buffers).  Elements that are not affine
// go through the points as in k_elem_fp64, all E at once, each entry of a
// Jacobian in its own thread.  The arithmetic is k_elem_fp64's.
// Measured, element kernel alone:
//   tet10 elasticity, 178,002 turned: 1.33 -> 0.90 + 0.07 ms of coefficients
//   (9.8 M pairs of 51 FP64 operations take 0.82 ms);
//   hex27 elasticity, 64,000 boxes: 1.06 (k_elem_affine) -> 0.94 + 0.01 ms;
//   hex27 elasticity, 4,522 curved: 1.41 (k_elem_fp64) -> 0.93 ms (operations
//   0.80 ms); tet20, 10,368 curved: 4.41 -> 2.86 ms;
//   hex8 conduction, 249,856 boxes: 0.283 -> 0.079 + 0.013 ms; hex27
//   conduction, 64,000: 0.212 -> 0.202 + 0.009 ms boxes, 0.382 -> 0.275 +
//   0.017 ms turned (without the two buffers 0.224 and 0.29).
// Shared memory (doubles): image [E kelems] | coefficients [2][E NC] |
// flags [2][E ints] | QUAD: X [2][E npe DIM] | det w [E nip] |
// J^-1 [E nip 9] | G, S [E nip npe gsw each].
constexpr int PACK_PAIRS = 384, PACK_THREADS = 384;
// coefficients of an affine element
template <int KIND, int DIM>
constexpr int AFF_PACK = KIND == KIND_MASS ? 1 : (KIND == KIND_HEAT ? (DIM == 3 ? 6 : 3) : (DIM == 3 ? 45 : 10));

// Coefficients of the affine elements, one thread each, by the operations of
// affine_coefficients / affine_stage_aligned: elasticity W [36] then U [9]
// (2D: 9 and 1), axis-aligned elasticity alpha, beta, a, b; conduction c1 trV
// [NS]; mass c1 det.  A block's run of coefficients is staged in shared memory
// and written whole: by element each store touched 32 sectors (tet10 elasticity,
// 178,002 turned elements: 0.094 -> 0.074 ms).
template <int KIND, int DIM>
__global__ void __launch_bounds__(128)
k_affine_coeff(const double *__restrict__ ageo, const uint8_t *__restrict__ aflag, const int32_t *__restrict__ emat,
               const double *__restrict__ mc1, const double *__restrict__ mc2, int64_t nel, double *__restrict__ coef,
               unsigned *status) {
  constexpr int NS = DIM == 3 ? 6 : 3, NA = DIM == 3 ? 3 : 1, NC = AFF_PACK<KIND, DIM>;
  __shared__ double sOut[128 * NC];
  for (int64_t e0 = (int64_t)blockIdx.x * 128; e0 < nel; e0 += (int64_t)gridDim.x * 128) {
    const int64_t e = e0 + threadIdx.x;
    const int mat = e >= nel ? -1 : (emat ? emat[e] : 0), flag = e < nel ? aflag[e] : 0;
    if (mat >= 0 && flag) {
      const double *inv = ageo + (size_t)e * 10;
      const double c1 = mc1[mat], c2 = KIND == KIND_ELASTIC ? mc2[mat] : 0.0, det = inv[9];
      double *out = sOut + threadIdx.x * NC;
      if (!(det > 0.0)) atomicOr(status, ST_BAD_JACOBIAN);
      const double cp = __dadd_rn(c1, c2), cm = __dsub_rn(c1, c2);
      if (KIND == KIND_MASS) {
        out[0] = __dmul_rn(c1, det);
      } else if (flag == 2) {
#pragma unroll
        for (int n = 0; n < (KIND == KIND_ELASTIC ? NS : DIM); ++n) {
          const int k = sym_k<DIM>(n), l = sym_l<DIM>(n);
          const double V = __dmul_rn(det, __dmul_rn(inv[k * 3 + k], inv[l * 3 + l]));
          if (KIND == KIND_HEAT) {
            out[n] = __dmul_rn(c1, V);
          } else if (n < DIM) {
            out[n] = __dmul_rn(cp, V);
            out[DIM + n] = __dmul_rn(c2, V);
          } else {
            out[DIM + n] = __dmul_rn(cp, V);
            out[DIM + NA + n] = __dmul_rn(cm, V);
          }
        }
      } else {
#pragma unroll
        for (int n = 0; n < NS; ++n) {
          const int k = sym_k<DIM>(n), l = sym_l<DIM>(n);
          double V[NS];
#pragma unroll
          for (int m = 0; m < NS; ++m) {
            const int i = sym_k<DIM>(m), j = sym_l<DIM>(m);
            V[m] = k == l ? __dmul_rn(det, __dmul_rn(inv[k * 3 + i], inv[k * 3 + j]))
                          : __dmul_rn(det, __fma_rn(inv[k * 3 + i], inv[l * 3 + j],
                                                    __dmul_rn(inv[l * 3 + i], inv[k * 3 + j])));
          }
          double tr = __dadd_rn(V[0], V[1]);
          if (DIM == 3) tr = __dadd_rn(tr, V[2]);
          if (KIND == KIND_HEAT) {
            out[n] = __dmul_rn(c1, tr);
          } else {
#pragma unroll
            for (int m = 0; m < NS; ++m) {
              const double v = __dmul_rn(cp, V[m]);
              out[m * NS + n] = m < DIM ? __fma_rn(c2, tr, v) : v;
            }
          }
        }
        if (KIND == KIND_ELASTIC) {
#pragma unroll
          for (int t = 0; t < NA * NA; ++t) {
            const int m = t / NA, n = t - m * NA;
            const int i = sym_k<DIM>(DIM + m), j = sym_l<DIM>(DIM + m);
            const int k = sym_k<DIM>(DIM + n), l = sym_l<DIM>(DIM + n);
            out[NS * NS + t] = __dmul_rn(cm, __dmul_rn(det, __fma_rn(inv[k * 3 + i], inv[l * 3 + j],
                                                                    -__dmul_rn(inv[l * 3 + i], inv[k * 3 + j]))));
          }
        }
      }
    }
    __syncthreads();
    const int n = (int)(nel - e0 < 128 ? nel - e0 : 128) * NC;
    for (int t = threadIdx.x; t < n; t += 128) coef[(size_t)e0 * NC + t] = sOut[t];
    __syncthreads();
  }
}

// 8-byte copy to shared memory, under way until the next cp.async wait
__device__ __forceinline__ void copy_async8(double *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sh_addr(dst)), "l"(src) : "memory");
}

template <int KIND, int DIM, bool QUAD>
__global__ void __launch_bounds__(PACK_THREADS, 2)
k_elem_packed(ElemArgs A, const double *__restrict__ coef, int E) {
  extern __shared__ __align__(128) double smem_p[];
  constexpr int NS = DIM == 3 ? 6 : 3, NA = DIM == 3 ? 3 : 1;
  constexpr int BS = (KIND == KIND_ELASTIC) ? DIM * DIM : 1;
  constexpr int P = (KIND == KIND_ELASTIC) ? DIM : 1;
  constexpr int gsw = (KIND == KIND_MASS) ? 1 : DIM;
  constexpr int NC = AFF_PACK<KIND, DIM>;
  const int npe = A.npe, nip = A.nip;
  const int64_t kelems = (int64_t)npe * A.colstride;
  double *sKe = smem_p, *sCo2 = sKe + E * kelems;
  int *sFlag2 = reinterpret_cast<int *>(sCo2 + 2 * (size_t)E * NC);   // -1 masked, 0 points, 1 affine, 2 aligned
  double *sX2 = sCo2 + 2 * (size_t)E * NC + E;
  double *sWd = sX2 + (QUAD ? 2 * (size_t)E * npe * DIM : 0), *sInv = sWd + (size_t)E * nip;
  double *G = sInv + (size_t)E * nip * 9, *S = G + (size_t)E * nip * npe * gsw;
  // this thread's node pair and its table row
  const int el = threadIdx.x / A.npairs, pi = threadIdx.x - el * A.npairs;
  int a = 0, b = 0;
  double sv[NS], av[NA];
  if (el < E) {
    pair_decode(pi, npe, a, b);
    if (A.aflag) {
      if (KIND == KIND_MASS) {
        sv[0] = A.Mp[pi];
      } else {
#pragma unroll
        for (int n = 0; n < NS; ++n) sv[n] = A.Rp[(size_t)pi * 9 + n];
#pragma unroll
        for (int n = 0; n < NA; ++n) av[n] = A.Rp[(size_t)pi * 9 + 6 + n];
      }
    }
  }
  // coefficients and coordinates of the elements from e0 on, under way into
  // buffer h while the elements before are computed
  auto fetch = [&](int64_t e0, int h) {
    const int ne = (int)(A.nel - e0 < E ? A.nel - e0 : E);
    if ((int)threadIdx.x < ne) {
      const int64_t e = e0 + threadIdx.x;
      sFlag2[h * E + threadIdx.x] = A.emat && A.emat[e] < 0 ? -1 : (A.aflag ? (int)A.aflag[e] : 0);
    }
    for (int t = threadIdx.x; coef && t < ne * NC; t += blockDim.x)
      copy_async8(sCo2 + (size_t)h * E * NC + t, coef + (size_t)e0 * NC + t);
    if (QUAD)
      for (int t = threadIdx.x; t < ne * npe * DIM; t += blockDim.x)
        copy_async8(sX2 + (size_t)h * E * npe * DIM + t, A.xyz + (size_t)A.conn[e0 * npe + t / DIM] * 3 + t % DIM);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int64_t step = (int64_t)gridDim.x * E;
  int h = 0;
  if ((int64_t)blockIdx.x * E < A.nel) fetch((int64_t)blockIdx.x * E, 0);
  for (int64_t e0 = (int64_t)blockIdx.x * E; e0 < A.nel; e0 += step, h ^= 1) {
    const int ne = (int)(A.nel - e0 < E ? A.nel - e0 : E);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // the previous elements' store has read the image
    if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncthreads();
    if (e0 + step < A.nel) fetch(e0 + step, h ^ 1);
    const int *sFlag = sFlag2 + h * E;
    const double *sX = sX2 + (size_t)h * E * npe * DIM, *sCo = sCo2 + (size_t)h * E * NC;
    if (QUAD) {
      // J of every point, one entry per thread (its fma chain over the nodes),
      // then the inverse, one point per thread, in place
      for (int t = threadIdx.x; t < ne * nip * DIM * DIM; t += blockDim.x) {
        const int p = t / (DIM * DIM), ij = t - p * DIM * DIM, k = p / nip, q = p - k * nip;
        if (sFlag[k] != 0) continue;
        const int i = ij / DIM, j = ij - i * DIM;
        const double *x = sX + (size_t)k * npe * DIM + i, *d = A.dN + (size_t)q * npe * 3 + j;
        double acc = 0.0;
        for (int n = 0; n < npe; ++n) acc = __fma_rn(x[n * DIM], __ldg(d + n * 3), acc);
        sInv[(size_t)p * 9 + 3 * i + j] = acc;
      }
      __syncthreads();
      for (int t = threadIdx.x; t < ne * nip; t += blockDim.x) {
        const int k = t / nip, q = t - k * nip;
        if (sFlag[k] != 0) continue;
        double J[3][3], inv[9];
#pragma unroll
        for (int i = 0; i < DIM; ++i)
#pragma unroll
          for (int j = 0; j < DIM; ++j) J[i][j] = sInv[(size_t)t * 9 + 3 * i + j];
        const double det = jac_inverse<DIM>(J, inv);
        if (!(det > 0.0)) atomicOr(A.status, ST_BAD_JACOBIAN);
        sWd[t] = __dmul_rn(det, __ldg(A.w + q));
#pragma unroll
        for (int n = 0; n < 9; ++n) sInv[(size_t)t * 9 + n] = inv[n];
      }
      __syncthreads();
      for (int t = threadIdx.x; t < ne * nip * npe; t += blockDim.x) {
        const int p = t / npe, k = p / nip, q = p - k * nip, n = t - p * npe;   // point, element, node
        if (sFlag[k] != 0) continue;
        const double wd = sWd[p];
        if (KIND == KIND_MASS) {
          S[t] = __dmul_rn(wd, __ldg(A.N + (size_t)q * npe + n));
        } else {
          const double *inv = sInv + (size_t)p * 9, *d = A.dN + ((size_t)q * npe + n) * 3;
#pragma unroll
          for (int i = 0; i < DIM; ++i) {
            double acc = 0.0;
#pragma unroll
            for (int j = 0; j < DIM; ++j) acc = __fma_rn(inv[3 * j + i], __ldg(d + j), acc);
            G[(size_t)t * DIM + i] = acc;
            S[(size_t)t * DIM + i] = __dmul_rn(wd, acc);
          }
        }
      }
      __syncthreads();
    }
    const int flag = el < ne ? sFlag[el] : -1;
    if (flag >= 0) {
      const double *C = sCo + (size_t)el * NC;
      double blk[BS];
      if (QUAD && flag == 0) {
        const size_t p0 = (size_t)el * nip * npe;
        if (KIND == KIND_ELASTIC) {
          const int64_t e = e0 + el;
          const int mat = A.emat ? A.emat[e] : 0;
          const double c1 = A.c1[mat], c2 = A.c2[mat];
          double O[DIM][DIM];
#pragma unroll
          for (int i = 0; i < DIM; ++i)
#pragma unroll
            for (int j = 0; j < DIM; ++j) O[i][j] = 0.0;
          for (int q = 0; q < nip; ++q) {
            const double *sa = S + (p0 + (size_t)q * npe + a) * DIM, *gb = G + (p0 + (size_t)q * npe + b) * DIM;
            double s_[DIM], g_[DIM];
#pragma unroll
            for (int i = 0; i < DIM; ++i) { s_[i] = sa[i]; g_[i] = gb[i]; }
#pragma unroll
            for (int i = 0; i < DIM; ++i)
#pragma unroll
              for (int j = 0; j < DIM; ++j) O[i][j] = __fma_rn(s_[i], g_[j], O[i][j]);
          }
          if (a == b) {   // the upper triangle, mirrored
#pragma unroll
            for (int i = 0; i < DIM; ++i)
#pragma unroll
              for (int j = 0; j < i; ++j) O[i][j] = O[j][i];
          }
          double tr = __dadd_rn(O[0][0], O[1 % DIM][1 % DIM]);
          if (DIM == 3) tr = __dadd_rn(tr, O[2 % DIM][2 % DIM]);
#pragma unroll
          for (int i = 0; i < DIM; ++i)
#pragma unroll
            for (int j = 0; j < DIM; ++j) {
              double t = __fma_rn(c2, O[j][i], __dmul_rn(c1, O[i][j]));
              if (i == j) t = __fma_rn(c2, tr, t);
              blk[i * DIM + j] = t;
            }
        } else {
          const double c1 = A.c1[A.emat ? A.emat[e0 + el] : 0];
          double acc = 0.0;
          for (int q = 0; q < nip; ++q) {
            if (KIND == KIND_HEAT) {
              const double *sa = S + (p0 + (size_t)q * npe + a) * DIM, *gb = G + (p0 + (size_t)q * npe + b) * DIM;
#pragma unroll
              for (int i = 0; i < DIM; ++i) acc = __fma_rn(sa[i], gb[i], acc);
            } else {
              acc = __fma_rn(S[p0 + (size_t)q * npe + a], __ldg(A.N + (size_t)q * npe + b), acc);
            }
          }
          blk[0] = __dmul_rn(c1, acc);
        }
      } else if (KIND == KIND_MASS) {
        blk[0] = __dmul_rn(C[0], sv[0]);
      } else if (KIND == KIND_HEAT) {
        double acc = 0.0;
#pragma unroll
        for (int n = 0; n < NS; ++n)
          if (n < DIM || flag == 1) acc = __fma_rn(C[n], sv[n], acc);
        blk[0] = acc;
      } else if (flag == 2) {
        double g = __dmul_rn(C[DIM], sv[0]);
#pragma unroll
        for (int n = 1; n < DIM; ++n) g = __fma_rn(C[DIM + n], sv[n], g);
#pragma unroll
        for (int i = 0; i < DIM; ++i) blk[i * DIM + i] = __fma_rn(C[i], sv[i], g);
#pragma unroll
        for (int m = 0; m < NA; ++m) {
          const int i = sym_k<DIM>(DIM + m), j = sym_l<DIM>(DIM + m);
          const double am = C[2 * DIM + m], s = sv[DIM + m];
          if (a != b) {
            const double h = __dmul_rn(C[2 * DIM + NA + m], av[m]);
            blk[i * DIM + j] = __fma_rn(am, s, h);
            blk[j * DIM + i] = __fma_rn(am, s, -h);
          } else {
            blk[i * DIM + j] = blk[j * DIM + i] = __dmul_rn(am, s);
          }
        }
      } else {
        double ks[NS];
#pragma unroll
        for (int m = 0; m < NS; ++m) {
          double acc = 0.0;
#pragma unroll
          for (int n = 0; n < NS; ++n) acc = __fma_rn(C[m * NS + n], sv[n], acc);
          ks[m] = acc;
        }
#pragma unroll
        for (int i = 0; i < DIM; ++i) blk[i * DIM + i] = ks[i];
#pragma unroll
        for (int m = 0; m < NA; ++m) {
          const int i = sym_k<DIM>(DIM + m), j = sym_l<DIM>(DIM + m);
          double acc = 0.0;
#pragma unroll
          for (int n = 0; n < NA; ++n) acc = __fma_rn(C[NS * NS + m * NA + n], av[n], acc);
          blk[i * DIM + j] = a != b ? __dadd_rn(ks[DIM + m], acc) : ks[DIM + m];
          blk[j * DIM + i] = a != b ? __dsub_rn(ks[DIM + m], acc) : ks[DIM + m];
        }
      }
      store_pair<P, BS>(sKe + (size_t)el * kelems, A.colstride, a, b, blk);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                   ::"l"(A.Kf + (size_t)e0 * kelems), "r"(sh_addr(sKe)), "r"((unsigned)(ne * kelems * 8))
                   : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
  }
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// Non-zero test on the bit pattern (integer pipe): every value but +-0.
__device__ __forceinline__ int nonzero_bits(double v) {
  return ((unsigned long long)__double_as_longlong(v) << 1) != 0ull;
}

// ---------------------------------------------------------------- dropzeros
// Structural entry count of every column (a matrix that keeps its pattern).
__global__ void k_count_struct(const int64_t *__restrict__ colptr, int64_t ndof, int64_t *__restrict__ cnt) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ndof; c += (int64_t)gridDim.x * blockDim.x)
    cnt[c] = colptr[c + 1] - colptr[c];
}

__global__ void k_count_nz(const double *__restrict__ nz, const int64_t *__restrict__ colptr,
                           int64_t ndof, int64_t *__restrict__ cnt) {
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int64_t c = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); c < ndof;
       c += (int64_t)gridDim.x * wpb) {
    int64_t s = colptr[c], e = colptr[c + 1];
    int n = 0;
    for (int64_t k = s + lane; k < e; k += 32) n += nonzero_bits(nz[k]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) n += __shfl_xor_sync(0xffffffffu, n, off);
    if (lane == 0) cnt[c] = n;
  }
}

// One warp per DoF column; four 32-entry chunks loaded (values and row
// nodes) before their ballots so that each warp keeps 2 KB in flight.
// rowval_s may be null (values only); keepbits (or null) receives one bit
// per structural entry, set when the entry is stored (the array must start
// zeroed; chunk boundaries do not fall on word boundaries, so the words are
// or-ed in).
template <int P, bool KEEP>
__global__ void k_compact(const double *__restrict__ nz, const int64_t *__restrict__ colptr,
                          const int64_t *__restrict__ nptr, const int32_t *__restrict__ nadj,
                          int64_t ndof, const int64_t *__restrict__ outptr,
                          int64_t *__restrict__ rowval_s, double *__restrict__ nzval_s,
                          unsigned *__restrict__ keepbits = nullptr) {
  constexpr int U = 4;
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int64_t c = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); c < ndof;
       c += (int64_t)gridDim.x * wpb) {
    const int64_t s = colptr[c];
    const int len = (int)(colptr[c + 1] - s);
    const int32_t *rn = nadj + nptr[c / P];
    int64_t o = outptr[c];
    for (int l0 = 0; l0 < len; l0 += 32 * U) {
      double v[U];
      int64_t row[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int l = l0 + u * 32 + lane;
        v[u] = l < len ? nz[s + l] : 0.0;
        row[u] = l < len ? (int64_t)P * rn[l / P] + l % P : 0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool keep = (l0 + u * 32 + lane < len) && (KEEP || nonzero_bits(v[u]));
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const int off = __popc(bal & ((1u << lane) - 1u));
          if (rowval_s) rowval_s[o + off] = row[u] + 1;
          nzval_s[o + off] = v[u];
        }
        if (keepbits && lane == 0 && bal) {
          const int64_t sidx = s + l0 + u * 32;
          const int sh = (int)(sidx & 31);
          atomicOr(keepbits + (sidx >> 5), bal << sh);
          if (sh) atomicOr(keepbits + (sidx >> 5) + 1, bal >> (32 - sh));
        }
        o += __popc(bal);
      }
    }
  }
}

// Number of differing 32-bit words of two arrays (device counter).
__global__ void k_words_differ(const unsigned *__restrict__ a, const unsigned *__restrict__ b, int64_t n,
                               unsigned long long *cnt) {
  unsigned long long c = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    c += a[i] != b[i];
  if (c) atomicAdd(cnt, c);
}

__global__ void k_colptr_1based(const int64_t *__restrict__ in, int64_t n,
                                int64_t *__restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = in[i] + 1;
}

// Row sums of a symmetric matrix = column sums in row order, from 0.0
// (sum(M, dims=2) walks columns in order; M[R,C] == M[C,R] bit for bit).
__global__ void k_lump(const double *__restrict__ nz, const int64_t *__restrict__ colptr,
                       int64_t ndof, double *__restrict__ diag) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ndof;
       c += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int64_t k = colptr[c]; k < colptr[c + 1]; ++k) acc = __dadd_rn(acc, nz[k]);
    diag[c] = acc;
  }
}

__global__ void k_diag_stored(const double *__restrict__ diag, int64_t ndof,
                              int64_t *__restrict__ cnt) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ndof;
       c += (int64_t)gridDim.x * blockDim.x)
    cnt[c] = nonzero_bits(diag[c]);
}

__global__ void k_diag_compact(const double *__restrict__ diag, int64_t ndof,
                               const int64_t *__restrict__ outptr,
                               int64_t *__restrict__ rowval_s, double *__restrict__ nzval_s) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ndof;
       c += (int64_t)gridDim.x * blockDim.x)
    if (nonzero_bits(diag[c])) {
      rowval_s[outptr[c]] = c + 1;
      nzval_s[outptr[c]] = diag[c];
    }
}

__global__ void k_axpby(double a, const double *__restrict__ x, double b,
                        const double *__restrict__ y, double *__restrict__ z, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    z[i] = __fma_rn(b, y[i], __dmul_rn(a, x[i]));
}

inline unsigned grid_1d(int64_t n, int threads, int sms) {
  int64_t b = (n + threads - 1) / threads;
  int64_t cap = (int64_t)sms * 16;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (unsigned)b;
}

template <int KIND, int DIM, bool SM>
int launch_elem(llf_ctx *ctx, const ElemArgs &a, size_t smem, unsigned grid) {
  auto fn = k_elem_fp64<KIND, DIM, SM>;
  if (smem > 48 * 1024)
    LLF_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem));
  KernelScope ks(ctx, "k_elem_fp64");
  fn<<<grid, ELEM_THREADS, smem, ctx->stream>>>(a);
  LLF_CUDA_TRY(ctx, cudaGetLastError());
  return LLF_OK;
}

// The staged affine kernel when every element is affine and two CTAs fit on
// an SM (with the conduction table, tet35's 630 node pairs do and hex64's 2080
// do not); *done = false otherwise.  Threads: the node pairs in as few rounds
// of at most 256 as possible, rounded up to whole warps (tet35: 3 rounds of
// 224).
template <int KIND>
int run_elem_affine(llf_ctx *ctx, const ElemArgs &a, bool *done) {
  *done = false;
  const int npairs = a.npairs;
  if (!a.all_affine || !a.aflag) return LLF_OK;
  const int tab_n = KIND == KIND_MASS ? npairs : npairs * 9;
  const size_t smem = sizeof(double) * ((size_t)a.npe * a.colstride + ((tab_n + 1) & ~1) + AFF_DOUBLES) + 16;
  if (smem > 110 * 1024) return LLF_OK;
  const int rounds = (npairs + AFFK_MAX_THREADS - 1) / AFFK_MAX_THREADS;
  const int threads = ((npairs + rounds - 1) / rounds + 31) / 32 * 32;
  auto fn = k_elem_affine<KIND>;
  if (smem > 48 * 1024)
    LLF_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  LLF_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem));
  if (per_sm < 1) return LLF_OK;
  if (a.cta_cap > 0 && per_sm > a.cta_cap) per_sm = a.cta_cap;
  int64_t grid = (int64_t)ctx->num_sms * per_sm;
  if (grid > a.nel) grid = a.nel;
  KernelScope ks(ctx, "k_elem_affine");
  fn<<<(unsigned)grid, threads, smem, ctx->stream>>>(a, tab_n);
  LLF_CUDA_TRY(ctx, cudaGetLastError());
  *done = true;
  return LLF_OK;
}

// Elements per CTA of k_elem_packed: as many as fill their warps best with
// node pairs, the larger count of equals, within PACK_THREADS threads and
// 108 KB of shared memory (two CTAs per SM); 0: one does not fit.
int packed_count(int npairs, size_t per_elem) {
  int best = 0;
  double fill = 0.0;
  for (int E = 1; E * npairs <= PACK_THREADS && E * per_elem <= 108 * 1024; ++E) {
    const double f = (double)(E * npairs) / ((E * npairs + 31) / 32 * 32);
    if (f >= fill) {
      fill = f;
      best = E;
    }
  }
  return best;
}

// k_elem_packed for elements of at most PACK_PAIRS node pairs; *done = false
// otherwise (from hex64's 2080 pairs on a thread has many pairs either way).  A
// mesh that would leave SMs idle puts fewer elements in a CTA.
template <int KIND, int DIM>
int run_elem_packed(llf_ctx *ctx, const ElemArgs &a, bool *done) {
  *done = false;
  const bool quad = !a.all_affine || !a.aflag;
  // The mass matrix by points has one operation per pair and point and little
  // shared memory; beyond 144 pairs an element per small CTA is as good on the
  // whole (ms there and here: 14,400 curved quad25 0.340 and 0.397, 27,000 hex27
  // 1.014 and 1.038, 10,368 tet20 0.595 and 0.556).
  if (a.npairs > (KIND == KIND_MASS && quad ? 144 : PACK_PAIRS)) return LLF_OK;
  const int gsw = (KIND == KIND_MASS) ? 1 : DIM;
  const size_t per_elem = sizeof(double) * ((size_t)a.npe * a.colstride + 2 * AFF_PACK<KIND, DIM> + 1 +
                                            (quad ? 2 * (size_t)a.npe * DIM + (size_t)a.nip * 10 +
                                                        2 * (size_t)a.nip * a.npe * gsw : 0));
  int E = packed_count(a.npairs, per_elem);
  if (E < 1) return LLF_OK;
  E = (int)std::min<int64_t>(E, (a.nel + ctx->num_sms - 1) / ctx->num_sms);
  double *coef = nullptr;
  if (a.aflag && a.any_affine) {
    LLF_CUDA_TRY(ctx, dalloc(ctx, &coef, (size_t)a.nel * AFF_PACK<KIND, DIM>));
    KernelScope ks(ctx, "k_affine_coeff");
    k_affine_coeff<KIND, DIM><<<grid_1d(a.nel, 128, ctx->num_sms), 128, 0, ctx->stream>>>(
        a.ageo, a.aflag, a.emat, a.c1, a.c2, a.nel, coef, a.status);
    LLF_CUDA_TRY(ctx, cudaGetLastError());
  }
  const size_t smem = E * per_elem;
  const int threads = (E * a.npairs + 31) / 32 * 32;
  auto launch = [&](auto fn) -> int {
    if (smem > 48 * 1024)
      LLF_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 1;
    LLF_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem));
    if (per_sm < 1) per_sm = 1;
    if (a.cta_cap > 0 && per_sm > a.cta_cap) per_sm = a.cta_cap;
    const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)ctx->num_sms * per_sm, (a.nel + E - 1) / E));
    KernelScope ks(ctx, "k_elem_packed");
    fn<<<(unsigned)grid, threads, smem, ctx->stream>>>(a, coef, E);
    LLF_CUDA_TRY(ctx, cudaGetLastError());
    return LLF_OK;
  };
  const int rc = quad ? launch(k_elem_packed<KIND, DIM, true>) : launch(k_elem_packed<KIND, DIM, false>);
  dfree(ctx, coef);
  *done = rc == LLF_OK;
  return rc;
}

template <int KIND, int DIM>
int run_elem(llf_ctx *ctx, ElemArgs a) {
  {
    bool done = false;
    int rc = run_elem_packed<KIND, DIM>(ctx, a, &done);
    if constexpr (KIND != KIND_ELASTIC && DIM == 3)
      if (rc == LLF_OK && !done) rc = run_elem_affine<KIND>(ctx, a, &done);
    if (rc != LLF_OK || done) return rc;
  }
  const int npe = a.npe, nip = a.nip;
  const int gsw = (KIND == KIND_MASS) ? 1 : DIM;
  const size_t tables = sizeof(double) * ((size_t)nip * npe * DIM + nip +
                                          (KIND == KIND_MASS ? (size_t)nip * npe : 0));
  const size_t local = sizeof(double) * ((size_t)npe * DIM + nip + (size_t)nip * 9 + AFF_DOUBLES);
  const size_t gs = sizeof(double) * 2 * (size_t)nip * npe * gsw;
  const bool in_smem = tables + local + gs <= 96 * 1024;
  const size_t smem = in_smem ? tables + local + gs : local;
  if (smem > 200 * 1024) return llf_fail(ctx, LLF_ERR_LIMIT, "element exceeds shared memory");
  // the dynamic shared-memory limit is raised before the occupancy query:
  // above 48 KB the query answers 0 for a kernel still at the default limit
  int per_sm = 0;
  if (in_smem) {
    if (smem > 48 * 1024)
      LLF_CUDA_TRY(ctx, cudaFuncSetAttribute(k_elem_fp64<KIND, DIM, true>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    LLF_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                          &per_sm, k_elem_fp64<KIND, DIM, true>, ELEM_THREADS, smem));
  } else {
    if (smem > 48 * 1024)
      LLF_CUDA_TRY(ctx, cudaFuncSetAttribute(k_elem_fp64<KIND, DIM, false>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    LLF_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                          &per_sm, k_elem_fp64<KIND, DIM, false>, ELEM_THREADS, smem));
  }
  if (per_sm < 1) per_sm = 1;
  if (a.cta_cap > 0 && per_sm > a.cta_cap) per_sm = a.cta_cap;
  int64_t grid = (int64_t)ctx->num_sms * per_sm;
  if (grid > a.nel) grid = a.nel > 0 ? a.nel : 1;
  double *scratch = nullptr;
  if (!in_smem) {
    a.scratch_stride = (int64_t)(gs / sizeof(double));
    LLF_CUDA_TRY(ctx, dalloc(ctx, &scratch, (size_t)grid * a.scratch_stride));
    a.scratch = scratch;
  }
  int rc = in_smem ? launch_elem<KIND, DIM, true>(ctx, a, smem, (unsigned)grid)
                   : launch_elem<KIND, DIM, false>(ctx, a, smem, (unsigned)grid);
  dfree(ctx, scratch);
  return rc;
}

}  // namespace

// ------------------------------------------------------------------ host
// Structural values from the stored values and the keep bits, one warp per
// DoF column, 64 entries at a time (a word pair of the bits); an entry that
// is not stored is +0.0.  Bound by HBM: nzval read, the structural values
// written.  hex27 40^3 (297.7 M entries): 0.91 ms; the binary search of
// every stored row in the column's node list that the bits replace took
// 2.55 ms.
__global__ void __launch_bounds__(256)
k_expand_nz(const int64_t *__restrict__ colptr, int64_t ndof, const int64_t *__restrict__ colptr_s,
            const double *__restrict__ nzval_s, const uint2 *__restrict__ keep, double *__restrict__ nz) {
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int64_t c = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); c < ndof; c += (int64_t)gridDim.x * wpb) {
    const int64_t s = colptr[c];
    const int len = (int)(colptr[c + 1] - s);
    const double *v = nzval_s + (colptr_s[c] - 1);
    const uint2 *kw = keep + keep_pos(s, c);
    const unsigned below = (1u << lane) - 1u;
#pragma unroll 4
    for (int l0 = 0; l0 < len; l0 += 64) {
      const uint2 w = kw[l0 >> 6];
      const int l = l0 + lane, nx = __popc(w.x);
      const double a = (w.x >> lane) & 1u ? v[__popc(w.x & below)] : 0.0;
      const double b = (w.y >> lane) & 1u ? v[nx + __popc(w.y & below)] : 0.0;
      if (l < len) nz[s + l] = a;
      if (l + 32 < len) nz[s + l + 32] = b;
      v += nx + __popc(w.y);
    }
  }
}

int matrix_ensure_nz(llf_ctx *ctx, const llf_matrix *cm) {
  llf_matrix *m = const_cast<llf_matrix *>(cm);
  if (m->d_nz || m->diagonal_only) return LLF_OK;
  if (!m->d_colptr_s || !m->d_keep)
    return llf_fail(ctx, LLF_ERR_STATE, "matrix has neither structural nor stored values");
  return matrix_expand_nz(ctx, m, &m->d_nz);
}

int matrix_expand_nz(llf_ctx *ctx, const llf_matrix *m, double **nz) {
  const llf_pattern *pat = m->pat;
  const int64_t n = pat->ndof;
  LLF_CUDA_TRY(ctx, dalloc(ctx, nz, pat->nnz > 0 ? pat->nnz : 1));
  KernelScope ks(ctx, "k_expand_nz");
  k_expand_nz<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 7) / 8, (int64_t)1 << 30)), 256, 0, ctx->stream>>>(
      pat->d_colptr, n, m->d_colptr_s, m->d_nzval_s, m->d_keep, *nz);
  LLF_CUDA_TRY(ctx, cudaGetLastError());
  return LLF_OK;
}

int matrix_finalize(llf_ctx *ctx, llf_matrix *m, int64_t *counts, int64_t **ptr0_out) {
  llf_pattern *pat = m->pat;
  const int64_t n = pat->ndof;
  cudaStream_t s = ctx->stream;
  int64_t *cnt = counts;
  const bool keep = m->keep_pattern && !m->diagonal_only;
  if (!cnt || m->diagonal_only || keep) {
    cnt = nullptr;
    LLF_CUDA_TRY(ctx, dalloc(ctx, &cnt, n + 1));
    LLF_CUDA_TRY(ctx, cudaMemsetAsync(cnt, 0, sizeof(int64_t) * (n + 1), s));
    if (keep) {
      KernelScope ks(ctx, "k_count_struct");
      k_count_struct<<<grid_1d(n, 256, ctx->num_sms), 256, 0, s>>>(pat->d_colptr, n, cnt);
    } else if (m->diagonal_only) {
      KernelScope ks(ctx, "k_diag_stored");
      k_diag_stored<<<grid_1d(n, 256, ctx->num_sms), 256, 0, s>>>(m->d_diag, n, cnt);
    } else {
      KernelScope ks(ctx, "k_count_nz");
      k_count_nz<<<grid_1d(n * 32, 256, ctx->num_sms), 256, 0, s>>>(m->d_nz, pat->d_colptr, n, cnt);
    }
    LLF_CUDA_TRY(ctx, cudaGetLastError());
  }
  int64_t *ptr0 = nullptr;
  LLF_CUDA_TRY(ctx, dalloc(ctx, &ptr0, n + 1));
  int64_t total = 0;
  {
    KernelScope ks(ctx, "scan");
    LLF_CUDA_TRY(ctx, exclusive_scan_i64(ctx, cnt, ptr0, n + 1, &total));
  }
  dfree(ctx, m->d_colptr_s);
  dfree(ctx, m->d_rowval_s);
  dfree(ctx, m->d_nzval_s);
  m->nnz_s = total;
  LLF_CUDA_TRY(ctx, dalloc(ctx, &m->d_colptr_s, n + 1));
  LLF_CUDA_TRY(ctx, dalloc(ctx, &m->d_rowval_s, total));
  LLF_CUDA_TRY(ctx, dalloc(ctx, &m->d_nzval_s, total));
  if (m->diagonal_only) {
    KernelScope ks(ctx, "k_diag_compact");
    k_diag_compact<<<grid_1d(n, 256, ctx->num_sms), 256, 0, s>>>(m->d_diag, n, ptr0,
                                                                 m->d_rowval_s, m->d_nzval_s);
  } else {
    unsigned g = grid_1d(n * 32, 256, ctx->num_sms);
    KernelScope ks(ctx, "k_compact");
    switch (pat->pdim) {
#define LLF_COMPACT(PP, KK) \
  k_compact<PP, KK><<<g, 256, 0, s>>>(m->d_nz, pat->d_colptr, pat->d_nptr, pat->d_nadj, n, ptr0, m->d_rowval_s, \
                                      m->d_nzval_s)
      case 1: if (keep) LLF_COMPACT(1, true); else LLF_COMPACT(1, false); break;
      case 2: if (keep) LLF_COMPACT(2, true); else LLF_COMPACT(2, false); break;
      case 3: if (keep) LLF_COMPACT(3, true); else LLF_COMPACT(3, false); break;
#undef LLF_COMPACT
      default: return llf_fail(ctx, LLF_ERR_UNSUPPORTED, "pdim must be 1, 2 or 3");
    }
  }
  LLF_CUDA_TRY(ctx, cudaGetLastError());
  {
    KernelScope ks(ctx, "k_colptr_1based");
    k_colptr_1based<<<grid_1d(n + 1, 256, ctx->num_sms), 256, 0, s>>>(ptr0, n + 1, m->d_colptr_s);
  }
  LLF_CUDA_TRY(ctx, cudaGetLastError());
  if (cnt != counts) dfree(ctx, cnt);
  if (ptr0_out) {
    *ptr0_out = ptr0;
  } else {
    dfree(ctx, ptr0);
  }
  return LLF_OK;
}

// ------------------------------------------------------- stored layouts
namespace {

llf_pattern::StoredLayout *layout_find(llf_pattern *pat, int kind, int form) {
  for (auto &l : pat->layouts)
    if (l.d_ptr0 && l.kind == kind && l.form == form) return &l;
  return nullptr;
}

// Keep ptr0 (ndof + 1, taken over) as the layout of (kind, form): in the
// slot of the same operator and form, else an empty one, else the least
// recently used.
void layout_store(llf_ctx *ctx, llf_pattern *pat, int kind, int form, int64_t *ptr0, int64_t total) {
  llf_pattern::StoredLayout *slot = layout_find(pat, kind, form);
  if (!slot)
    for (auto &l : pat->layouts)
      if (!l.d_ptr0) { slot = &l; break; }
  if (!slot) {
    slot = &pat->layouts[0];
    for (auto &l : pat->layouts)
      if (l.used < slot->used) slot = &l;
  }
  dfree(ctx, slot->d_ptr0);
  slot->kind = kind;
  slot->form = form;
  slot->total = total;
  slot->d_ptr0 = ptr0;
  slot->used = ++pat->layout_clock;
}

// Stored-layout reuse is on unless LLF_STORED_LAYOUT=0.
bool layout_reuse_enabled() {
  const char *v = getenv("LLF_STORED_LAYOUT");
  return !(v && v[0] == '0');
}

}  // namespace

void pattern_free_layouts(llf_ctx *ctx, llf_pattern *pat) {
  for (auto &l : pat->layouts) {
    dfree(ctx, l.d_ptr0);
    l = llf_pattern::StoredLayout{};
  }
}

int assemble_impl(llf_ctx *ctx, llf_mesh *mesh, llf_pattern *pat, int kind, int ptype,
                  const double *c1, const double *c2, int nmat, int form, int lumped,
                  llf_matrix *m, const double *init, GatherSink *sink) {
  (void)ptype;
  if (!pat->tune.from_tuner) tune_lookup(pat, kind, form);
  const int dim = mesh->dim;
  const int npe = mesh->npe;
  const int P = pat->pdim;
  const int BS = (kind == KIND_ELASTIC) ? P * P : 1;
  cudaStream_t s = ctx->stream;

  double *d_c1 = nullptr;   // c1, then c2
  int64_t *cnt = nullptr;
  LLF_CUDA_TRY(ctx, dalloc(ctx, &d_c1, 2 * (size_t)nmat));
  LLF_CUDA_TRY(ctx, dalloc(ctx, &cnt, pat->ndof + 1));
  std::vector<double> hc(c1, c1 + nmat);
  hc.insert(hc.end(), c2 ? c2 : c1, (c2 ? c2 : c1) + nmat);
  LLF_CUDA_TRY(ctx, cudaMemcpyAsync(d_c1, hc.data(), sizeof(double) * hc.size(), cudaMemcpyHostToDevice, s));
  const double *d_c2 = d_c1 + nmat;
  // the stored layout of the last assembly of this operator and form on
  // the pattern: the gather then writes the stored CSC itself, and the
  // structural values are left to matrix_ensure_nz
  const bool reuse = !sink && !init && !(kind == KIND_MASS && lumped) && !m->keep_pattern && layout_reuse_enabled();
  llf_pattern::StoredLayout *lay = reuse ? layout_find(pat, kind, form) : nullptr;
  StoredSpec spec;
  if (!lay) LLF_CUDA_TRY(ctx, cudaMemsetAsync(cnt, 0, sizeof(int64_t) * (pat->ndof + 1), s));
  if (lay) {
    LLF_CUDA_TRY(ctx, dalloc(ctx, &m->d_rowval_s, lay->total > 0 ? lay->total : 1));
    LLF_CUDA_TRY(ctx, dalloc(ctx, &m->d_nzval_s, lay->total > 0 ? lay->total : 1));
    spec.ptr0 = lay->d_ptr0;
    spec.rowval_s = m->d_rowval_s;
    spec.nzval_s = m->d_nzval_s;
    spec.mismatch = ctx->d_status + 1;
    LLF_CUDA_TRY(ctx, dalloc(ctx, &m->d_keep, keep_words(pat->nnz, pat->ndof)));
    spec.keep = m->d_keep;
    spec.nz_slot = &m->d_nz;
    spec.cnt_fallback = cnt;
    // the column pointers follow from the layout alone (recomputed if a
    // column's count turns out to differ)
    LLF_CUDA_TRY(ctx, dalloc(ctx, &m->d_colptr_s, pat->ndof + 1));
    {
      KernelScope ks(ctx, "k_colptr_1based");
      k_colptr_1based<<<grid_1d(pat->ndof + 1, 256, ctx->num_sms), 256, 0, s>>>(lay->d_ptr0, pat->ndof + 1,
                                                                               m->d_colptr_s);
    }
    LLF_CUDA_TRY(ctx, cudaGetLastError());
  } else if (!sink) {
    LLF_CUDA_TRY(ctx, dalloc(ctx, &m->d_nz, pat->nnz));
  }
  StoredSpec *sp = lay ? &spec : nullptr;
  int64_t *ptr0 = nullptr;   // the stored layout of this assembly, kept on the pattern
  // affine geometry of every element (built-in tables only), kept on the
  // mesh until its coordinates, connectivity, materials or tables change
  uint8_t *aflag = nullptr;
  double *ageo = nullptr;
  bool all_affine = false;
  if (mesh->d_Rp) {
    if (mesh->geo_cached != mesh->geo_version || mesh->geo_cached_tables != mesh->tables_version ||
        !mesh->d_aflag) {
      mesh->geo_cached = -1;
      if (!mesh->d_aflag) {
        LLF_CUDA_TRY(ctx, dalloc(ctx, &mesh->d_aflag, mesh->nel));
        LLF_CUDA_TRY(ctx, dalloc(ctx, &mesh->d_ageo, (size_t)mesh->nel * 10));
      }
      unsigned long long *nonaff = nullptr;   // elements in use that are not affine; whether one is
      LLF_CUDA_TRY(ctx, dalloc(ctx, &nonaff, 2));
      LLF_CUDA_TRY(ctx, cudaMemsetAsync(nonaff, 0, 2 * sizeof(unsigned long long), s));
      {
        KernelScope ks(ctx, "k_affine_geometry");
        const unsigned g = grid_1d(mesh->nel, 128, ctx->num_sms);
        if (dim == 3)
          k_affine_geometry<3><<<g, 128, 0, s>>>(mesh->d_xyz, mesh->d_conn, mesh->d_emat, mesh->nel, npe,
                                                 mesh->d_dN, mesh->d_nref, mesh->d_ageo, mesh->d_aflag, nonaff);
        else
          k_affine_geometry<2><<<g, 128, 0, s>>>(mesh->d_xyz, mesh->d_conn, mesh->d_emat, mesh->nel, npe,
                                                 mesh->d_dN, mesh->d_nref, mesh->d_ageo, mesh->d_aflag, nonaff);
        LLF_CUDA_TRY(ctx, cudaGetLastError());
      }
      unsigned long long h[2] = {1, 1};
      LLF_CUDA_TRY(ctx, cudaMemcpyAsync(h, nonaff, sizeof(h), cudaMemcpyDeviceToHost, s));
      LLF_CUDA_TRY(ctx, cudaStreamSynchronize(s));
      dfree(ctx, nonaff);
      mesh->geo_all_affine = h[0] == 0;
      mesh->geo_any_affine = h[1] != 0;
      mesh->geo_cached = mesh->geo_version;
      mesh->geo_cached_tables = mesh->tables_version;
    }
    aflag = mesh->d_aflag;
    ageo = mesh->d_ageo;
    all_affine = mesh->geo_all_affine;
  }
  int rc = LLF_OK;
  if (form == LLF_FP32Q) {
    rc = assemble_fp32_impl(ctx, mesh, pat, kind, d_c1, d_c2, aflag, ageo, m->d_nz, cnt, init, sink, sp, all_affine);
  } else {
    double *Kf = nullptr;
    const int64_t cs = kf_colstride(npe, BS, (int)sizeof(double));
    LLF_CUDA_TRY(ctx, dalloc(ctx, &Kf, (size_t)mesh->nel * npe * cs));
    ElemArgs a{};
    a.xyz = mesh->d_xyz;
    a.conn = mesh->d_conn;
    a.emat = mesh->d_emat;
    a.nel = mesh->nel;
    a.npe = npe;
    a.nip = mesh->nip;
    a.npairs = npe * (npe + 1) / 2;
    a.w = mesh->d_w;
    a.N = mesh->d_N;
    a.dN = mesh->d_dN;
    a.c1 = d_c1;
    a.c2 = d_c2;
    a.Kf = Kf;
    a.colstride = cs;
    a.status = ctx->d_status;
    a.aflag = aflag;
    a.ageo = ageo;
    a.Rp = mesh->d_Rp;
    a.Mp = mesh->d_Mp;
    a.cta_cap = pat->tune.elem_cap;
    a.all_affine = all_affine;
    a.any_affine = aflag && mesh->geo_any_affine;
    // element range [e0, e1): the element-indexed arrays are offset
    auto elems = [&](int64_t e0, int64_t e1) -> int {
      ElemArgs b = a;
      b.conn = a.conn + e0 * npe;
      b.emat = a.emat ? a.emat + e0 : nullptr;
      b.nel = e1 - e0;
      b.Kf = a.Kf + e0 * npe * cs;
      b.aflag = a.aflag ? a.aflag + e0 : nullptr;
      b.ageo = a.ageo ? a.ageo + e0 * 10 : nullptr;
      if (b.nel <= 0) return LLF_OK;
      if (dim == 3) {
        if (kind == KIND_ELASTIC) return run_elem<KIND_ELASTIC, 3>(ctx, b);
        if (kind == KIND_HEAT) return run_elem<KIND_HEAT, 3>(ctx, b);
        return run_elem<KIND_MASS, 3>(ctx, b);
      }
      if (kind == KIND_ELASTIC) return run_elem<KIND_ELASTIC, 2>(ctx, b);
      if (kind == KIND_HEAT) return run_elem<KIND_HEAT, 2>(ctx, b);
      return run_elem<KIND_MASS, 2>(ctx, b);
    };
    if (sink) {
      rc = sink->gather(ctx, pat, Kf, cs, kind == KIND_ELASTIC, elems);
    } else {
      rc = elems(0, mesh->nel);
      if (rc == LLF_OK) rc = gather_full(ctx, pat, Kf, cs, kind == KIND_ELASTIC, m->d_nz, cnt, init, sp);
    }
    dfree(ctx, Kf);
  }
  dfree(ctx, d_c1);
  if (rc == LLF_OK) rc = llf_check_status(ctx, "assembly", spec.status_read && !spec.fell_back);
  if (sink) {
    dfree(ctx, cnt);
    return rc;
  }
  if (rc == LLF_OK && kind == KIND_MASS && lumped) {
    m->diagonal_only = true;
    cudaError_t e = dalloc(ctx, &m->d_diag, pat->ndof);
    if (e != cudaSuccess) rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e));
    if (rc == LLF_OK) {
      KernelScope ks(ctx, "k_lump");
      k_lump<<<grid_1d(pat->ndof, 128, ctx->num_sms), 128, 0, s>>>(m->d_nz, pat->d_colptr,
                                                                   pat->ndof, m->d_diag);
    }
  }
  if (lay && rc == LLF_OK) {
    if (!spec.fell_back) {  // every column's count matched: the stored CSC is complete
      m->nnz_s = lay->total;
      lay->used = ++pat->layout_clock;
      dfree(ctx, cnt);
      return LLF_OK;
    }
    // a column's count differed: the gather ran again the usual way
    dfree(ctx, m->d_keep);
    dfree(ctx, m->d_rowval_s);
    dfree(ctx, m->d_nzval_s);
    rc = matrix_finalize(ctx, m, cnt, reuse ? &ptr0 : nullptr);
  } else {
    if (rc == LLF_OK)
      rc = matrix_finalize(ctx, m, (kind == KIND_MASS && lumped) ? nullptr : cnt, reuse ? &ptr0 : nullptr);
  }
  if (rc == LLF_OK && ptr0) layout_store(ctx, pat, kind, form, ptr0, m->nnz_s);
  dfree(ctx, cnt);
  return rc;
}

namespace {
// Structural values of a*X + b*D for a lumped (diagonal) D: off the
// diagonal a*x, on it fma(b, d, a*x) — the full-full formula with zeros off
// the diagonal of D.
__global__ void k_axpby_diag(double a, const double *__restrict__ x, double b, const double *__restrict__ d,
                             const int64_t *__restrict__ colptr, const int32_t *__restrict__ diagpos, int P,
                             int64_t ndof, double *__restrict__ z) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ndof; c += (int64_t)gridDim.x * blockDim.x) {
    const int64_t B = c / P;
    const int j = (int)(c - B * P);
    const int64_t k = colptr[c] + (int64_t)P * diagpos[B] + j;
    z[k] = __fma_rn(b, d[c], __dmul_rn(a, x[k]));
  }
}

__global__ void k_scale(double a, const double *__restrict__ x, double *__restrict__ z, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    z[i] = __dmul_rn(a, x[i]);
}
}  // namespace

int matrix_axpby_impl(llf_ctx *ctx, double a, const llf_matrix *A, double b,
                      const llf_matrix *B, llf_matrix *C) {
  if (!A->diagonal_only) {
    const int rc = matrix_ensure_nz(ctx, A);
    if (rc != LLF_OK) return rc;
  }
  if (!B->diagonal_only) {
    const int rc = matrix_ensure_nz(ctx, B);
    if (rc != LLF_OK) return rc;
  }
  if (A->pat != B->pat)
    return llf_fail(ctx, LLF_ERR_STATE, "axpby: matrices live on different patterns");
  C->pat = A->pat;
  if (A->diagonal_only && B->diagonal_only) {  // both lumped: a lumped result
    const int64_t n = A->pat->ndof;
    C->diagonal_only = true;
    LLF_CUDA_TRY(ctx, dalloc(ctx, &C->d_diag, n));
    k_axpby<<<grid_1d(n, 256, ctx->num_sms), 256, 0, ctx->stream>>>(a, A->d_diag, b, B->d_diag, C->d_diag, n);
    LLF_CUDA_TRY(ctx, cudaGetLastError());
    return matrix_finalize(ctx, C, nullptr);
  }
  if (A->diagonal_only || B->diagonal_only) {  // one lumped operand
    const llf_matrix *F = A->diagonal_only ? B : A, *D = A->diagonal_only ? A : B;
    const double af = A->diagonal_only ? b : a, bd = A->diagonal_only ? a : b;
    const llf_pattern *p = A->pat;
    LLF_CUDA_TRY(ctx, dalloc(ctx, &C->d_nz, p->nnz));
    k_scale<<<grid_1d(p->nnz, 256, ctx->num_sms), 256, 0, ctx->stream>>>(af, F->d_nz, C->d_nz, p->nnz);
    k_axpby_diag<<<grid_1d(p->ndof, 256, ctx->num_sms), 256, 0, ctx->stream>>>(
        af, F->d_nz, bd, D->d_diag, p->d_colptr, p->d_diagpos, p->pdim, p->ndof, C->d_nz);
    LLF_CUDA_TRY(ctx, cudaGetLastError());
    return matrix_finalize(ctx, C, nullptr);
  }
  int64_t n = A->pat->nnz;
  LLF_CUDA_TRY(ctx, dalloc(ctx, &C->d_nz, n));
  {
    KernelScope ks(ctx, "k_axpby");
    k_axpby<<<grid_1d(n, 256, ctx->num_sms), 256, 0, ctx->stream>>>(a, A->d_nz, b, B->d_nz,
                                                                    C->d_nz, n);
  }
  LLF_CUDA_TRY(ctx, cudaGetLastError());
  return matrix_finalize(ctx, C, nullptr);
}

// ---------------------------------------------------------------- to host
// Assembly straight into host SparseMatrixCSC arrays.  After the element
// kernel the columns are processed in NSLAB node slabs on the compute
// stream: gather (structural values and non-zero counts), scan of the
// counts continued from the previous slab's end (a device-side carry),
// compaction and the 1-based column pointers.  Each slab's end offset is
// copied to pinned host memory behind an event; the host waits for slab s
// only, then copies its compacted rows and values to the caller's arrays
// on a second stream while the GPU works on the slabs after it, so the
// device-to-host copy (the largest cost of the whole call) overlaps all but
// the first slab of the gather and compaction.  The result is the one
// llf_assemble_stiffness + llf_matrix_copy_csc give, bit for bit.
namespace {

__global__ void k_slab_carry(int64_t *__restrict__ outptr, int64_t n, int64_t *__restrict__ carry, int s,
                             const int64_t *__restrict__ slab_total) {
  const int64_t c0 = carry[s];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    outptr[i] += c0;
  if (blockIdx.x == 0 && threadIdx.x == 0) carry[s + 1] = c0 + *slab_total;
}

// d_max[k] = 1 + the largest element index in the lists of the nodes of
// slab k (B[k] <= node < B[k+1]); lists are sorted, so the last entry.
__global__ void k_slab_last_elem(const int64_t *__restrict__ n2e_ptr, const int2 *__restrict__ n2e, int64_t non,
                                 const int64_t *__restrict__ B, int nslab, int64_t *__restrict__ d_max) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < non; v += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = n2e_ptr[v + 1];
    if (e == n2e_ptr[v]) continue;
    int k = 0;
    while (k + 1 < nslab && v >= B[k + 1]) ++k;
    atomicMax((unsigned long long *)&d_max[k], (unsigned long long)(n2e[e - 1].x + 1));
  }
}

__global__ void k_colptr_last(const int64_t *__restrict__ carry, int s, int64_t *__restrict__ colptr_last) {
  *colptr_last = carry[s] + 1;
}

struct HostSlabSink : GatherSink {
  static constexpr int NSLAB = 16;
  int64_t capacity = 0;
  int64_t *h_colptr = nullptr, *h_rowval = nullptr;
  double *h_nzval = nullptr;
  unsigned *h_keep = nullptr;   // values-only form: keep bits instead of rowval
  int keep_changed = 1;         // values-only form: the bits differ from the last call's on the pattern
  int64_t nnz = 0;

  template <class T>
  int run(llf_ctx *ctx, llf_pattern *pat, const T *Kf, int64_t cs, bool blockval, const ElemLauncher &elems) {
    const int P = pat->pdim;
    const int64_t non = pat->mesh->non, ndof = pat->ndof;
    cudaStream_t s = ctx->stream;
    double *nz = nullptr, *nzval = nullptr;
    int64_t *cnt = nullptr, *outptr = nullptr, *rowval = nullptr, *colptr = nullptr, *carry = nullptr,
            *totals = nullptr, *h_end = nullptr;
    cudaStream_t cp = nullptr;
    cudaEvent_t ev[NSLAB] = {}, done[NSLAB] = {};
    int rc = LLF_OK;
    unsigned *keep = nullptr;
    const int64_t nwords = pat->nnz / 32 + 2;
    cudaError_t e = dalloc(ctx, &nz, pat->nnz);
    if (e == cudaSuccess && h_keep) e = dalloc(ctx, &keep, nwords);
    if (e == cudaSuccess && h_keep) e = cudaMemsetAsync(keep, 0, sizeof(unsigned) * nwords, s);
    if (e == cudaSuccess) e = dalloc(ctx, &cnt, ndof + 1);
    if (e == cudaSuccess) e = dalloc(ctx, &outptr, ndof + 1);
    if (e == cudaSuccess) e = dalloc(ctx, &colptr, ndof + 1);
    if (e == cudaSuccess && !h_keep) e = dalloc(ctx, &rowval, pat->nnz);
    if (e == cudaSuccess) e = dalloc(ctx, &nzval, pat->nnz);
    if (e == cudaSuccess) e = dalloc(ctx, &carry, NSLAB + 1);
    if (e == cudaSuccess) e = dalloc(ctx, &totals, NSLAB);
    if (e == cudaSuccess) e = cudaMemsetAsync(carry, 0, sizeof(int64_t) * (NSLAB + 1), s);
    if (e == cudaSuccess) e = cudaMallocHost((void **)&h_end, sizeof(int64_t) * (NSLAB + 1));
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&cp, cudaStreamNonBlocking);
    for (int k = 0; k < NSLAB && e == cudaSuccess; ++k) {
      e = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&done[k], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e));
    // 1. all slabs on the compute stream, each after the elements it needs
    int64_t B[NSLAB + 1];
    for (int k = 0; k <= NSLAB; ++k) B[k] = non * k / NSLAB;
    if (rc == LLF_OK) rc = slab_elements(ctx, pat, B);
    int64_t e_done = 0;
    for (int k = 0; k < NSLAB && rc == LLF_OK; ++k) {
      const int64_t B0 = B[k], nB = B[k + 1] - B[k], c0 = B0 * P, nc = nB * P;
      const int64_t e_need = pat->slab_elem_end[k];
      if (e_need > e_done) {
        rc = elems(e_done, e_need);
        if (rc != LLF_OK) break;
        e_done = e_need;
      }
      if (nB > 0) {
        rc = gather_slab(ctx, pat, Kf, cs, blockval, nz, cnt, B0, nB);
        if (rc != LLF_OK) break;
        {
          KernelScope ks(ctx, "scan");
          e = exclusive_scan_i64_dev(ctx, cnt + c0, outptr + c0, nc, totals + k);
        }
        if (e != cudaSuccess) { rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e)); break; }
      } else {
        cudaMemsetAsync(totals + k, 0, sizeof(int64_t), s);
      }
      k_slab_carry<<<grid_1d(std::max<int64_t>(nc, 1), 256, ctx->num_sms), 256, 0, s>>>(outptr + c0, nc, carry, k,
                                                                                       totals + k);
      if (nc > 0) {
        const unsigned g = grid_1d(nc * 32, 256, ctx->num_sms);
        KernelScope ks(ctx, "k_compact");
#define LLF_SLAB_COMPACT(PP) \
  k_compact<PP, false><<<g, 256, 0, s>>>(nz, pat->d_colptr + c0, pat->d_nptr + B0, pat->d_nadj, nc, outptr + c0, \
                                          rowval, nzval, keep)
        if (P == 1) LLF_SLAB_COMPACT(1); else if (P == 2) LLF_SLAB_COMPACT(2); else LLF_SLAB_COMPACT(3);
#undef LLF_SLAB_COMPACT
        k_colptr_1based<<<grid_1d(nc, 256, ctx->num_sms), 256, 0, s>>>(outptr + c0, nc, colptr + c0);
      }
      if (k == NSLAB - 1) k_colptr_last<<<1, 1, 0, s>>>(carry, NSLAB, colptr + ndof);
      cudaMemcpyAsync(h_end + k + 1, carry + k + 1, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
      cudaEventRecord(ev[k], s);
      e = cudaGetLastError();
      if (e != cudaSuccess) { rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e)); break; }
    }
    // 2. each slab to the host as soon as it is compacted
    h_end[0] = 0;
    for (int k = 0; k < NSLAB && rc == LLF_OK; ++k) {
      e = cudaEventSynchronize(ev[k]);
      if (e != cudaSuccess) { rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e)); break; }
      const int64_t o0 = h_end[k], o1 = h_end[k + 1];
      if (o1 > capacity) { rc = llf_fail(ctx, LLF_ERR_LIMIT, "llf_assemble_stiffness_csc: capacity too small"); break; }
      const int64_t c0 = B[k] * P, nc = (B[k + 1] - B[k]) * P + (k == NSLAB - 1 ? 1 : 0);
      e = cudaStreamWaitEvent(cp, ev[k], 0);
      if (e == cudaSuccess && nc > 0)
        e = cudaMemcpyAsync(h_colptr + c0, colptr + c0, sizeof(int64_t) * nc, cudaMemcpyDeviceToHost, cp);
      if (e == cudaSuccess && o1 > o0 && !h_keep)
        e = cudaMemcpyAsync(h_rowval + o0, rowval + o0, sizeof(int64_t) * (o1 - o0), cudaMemcpyDeviceToHost, cp);
      if (e == cudaSuccess && o1 > o0)
        e = cudaMemcpyAsync(h_nzval + o0, nzval + o0, sizeof(double) * (o1 - o0), cudaMemcpyDeviceToHost, cp);
      if (e == cudaSuccess) e = cudaEventRecord(done[k], cp);
      if (e != cudaSuccess) rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e));
    }
    // the keep bits once every slab is compacted (the words at slab edges
    // take bits from both neighbours)
    if (rc == LLF_OK && h_keep) {
      const int64_t nw = (pat->nnz + 31) / 32;
      unsigned long long *ndiff = nullptr;
      unsigned long long hdiff = 1;
      e = cudaMemcpyAsync(h_keep, keep, sizeof(unsigned) * nw, cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess && pat->d_keep_prev) {   // compare with the last call's bits on the device
        e = dalloc(ctx, &ndiff, 1);
        if (e == cudaSuccess) e = cudaMemsetAsync(ndiff, 0, sizeof(unsigned long long), s);
        if (e == cudaSuccess) {
          KernelScope ks(ctx, "k_words_differ");
          k_words_differ<<<grid_1d(nw, 256, ctx->num_sms), 256, 0, s>>>(keep, pat->d_keep_prev, nw, ndiff);
          e = cudaGetLastError();
        }
        if (e == cudaSuccess)
          e = cudaMemcpyAsync(&hdiff, ndiff, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s);
      }
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      dfree(ctx, ndiff);
      if (e != cudaSuccess) {
        rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e));
      } else {
        keep_changed = hdiff != 0;
        dfree(ctx, pat->d_keep_prev);   // this call's bits become the pattern's reference
        pat->d_keep_prev = keep;
        keep = nullptr;
      }
    }
    if (cp) {
      cudaError_t e2 = cudaStreamSynchronize(cp);
      if (rc == LLF_OK && e2 != cudaSuccess) rc = llf_fail(ctx, LLF_ERR_CUDA, cudaGetErrorString(e2));
    }
    // the buffers are freed on the compute stream after the copies that read them
    for (int k = 0; k < NSLAB; ++k)
      if (done[k]) cudaStreamWaitEvent(s, done[k], 0);
    if (rc == LLF_OK) nnz = h_end[NSLAB];
    dfree(ctx, nz);
    dfree(ctx, cnt);
    dfree(ctx, outptr);
    dfree(ctx, colptr);
    dfree(ctx, rowval);
    dfree(ctx, nzval);
    dfree(ctx, carry);
    dfree(ctx, totals);
    dfree(ctx, keep);
    cudaStreamSynchronize(s);
    for (int k = 0; k < NSLAB; ++k) {
      if (ev[k]) cudaEventDestroy(ev[k]);
      if (done[k]) cudaEventDestroy(done[k]);
    }
    if (cp) cudaStreamDestroy(cp);
    if (h_end) cudaFreeHost(h_end);
    return rc;
  }
  // pat->slab_elem_end for the node slabs B (once per pattern): prefix
  // maximum over the slabs of the last element in each node's list.
  static int slab_elements(llf_ctx *ctx, llf_pattern *pat, const int64_t *B) {
    if ((int)pat->slab_elem_end.size() == NSLAB) return LLF_OK;
    int64_t *d_B = nullptr, *d_max = nullptr;
    LLF_CUDA_TRY(ctx, dalloc(ctx, &d_B, NSLAB + 1));
    LLF_CUDA_TRY(ctx, dalloc(ctx, &d_max, NSLAB));
    LLF_CUDA_TRY(ctx, cudaMemcpyAsync(d_B, B, sizeof(int64_t) * (NSLAB + 1), cudaMemcpyHostToDevice, ctx->stream));
    LLF_CUDA_TRY(ctx, cudaMemsetAsync(d_max, 0, sizeof(int64_t) * NSLAB, ctx->stream));
    k_slab_last_elem<<<grid_1d(pat->mesh->non, 256, ctx->num_sms), 256, 0, ctx->stream>>>(
        pat->d_n2e_ptr, pat->d_n2e, pat->mesh->non, d_B, NSLAB, d_max);
    std::vector<int64_t> h(NSLAB);
    LLF_CUDA_TRY(ctx, cudaMemcpyAsync(h.data(), d_max, sizeof(int64_t) * NSLAB, cudaMemcpyDeviceToHost,
                                      ctx->stream));
    LLF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    dfree(ctx, d_B);
    dfree(ctx, d_max);
    for (int k = 1; k < NSLAB; ++k) h[k] = std::max(h[k], h[k - 1]);
    pat->slab_elem_end = h;
    return LLF_OK;
  }
  int gather(llf_ctx *ctx, llf_pattern *pat, const double *Kf, int64_t cs, bool blockval,
             const ElemLauncher &elems) override {
    return run<double>(ctx, pat, Kf, cs, blockval, elems);
  }
  int gather(llf_ctx *ctx, llf_pattern *pat, const float *Kf, int64_t cs, bool blockval,
             const ElemLauncher &elems) override {
    return run<float>(ctx, pat, Kf, cs, blockval, elems);
  }
};

}  // namespace

int assemble_to_host_impl(llf_ctx *ctx, llf_mesh *mesh, llf_pattern *pat, int kind, const double *c1,
                          const double *c2, int nmat, int form, int64_t capacity, int64_t *colptr,
                          int64_t *rowval, double *nzval, int64_t *nnz, unsigned *keep, int *keep_changed) {
  HostSlabSink sink;
  sink.capacity = capacity;
  sink.h_colptr = colptr;
  sink.h_rowval = rowval;
  sink.h_nzval = nzval;
  sink.h_keep = keep;
  if (keep_changed) *keep_changed = 1;
  llf_matrix scratch;
  scratch.pat = pat;
  int rc = assemble_impl(ctx, mesh, pat, kind, LLF_SOLID, c1, c2, nmat, form, 0, &scratch, nullptr, &sink);
  if (rc == LLF_OK) *nnz = sink.nnz;
  if (rc == LLF_OK && keep_changed) *keep_changed = sink.keep_changed;
  return rc;
}
