// Column-node gather: element matrices, whole in the layout Kf[element]
// [column node b][row node a][block], summed into the columns of a pattern.
//
// A column node B owns its element list (ascending), its row-node list and,
// from the pattern's element-to-column map, the row position of every local
// node of those elements.  Its elements are walked in ascending order, so
// each entry is the sum SparseArrays.sparse makes of the reference's triplets
// (src/linear.jl:314-323): the first value, then + each later one.  The sums
// live in shared memory, one plane per DoF column of B in the order the
// column is written out.
//
// What bounds it: per element column npe * P * P values are read once and
// added once.  GB300 spends its FP64 pipe (16 SM cycles) and its shared-memory
// and L1 wavefronts per warp instruction, however few lanes take part, so the
// G lanes of a column node take the values of an element column as one flat
// run (lane l: values l, l + G, ...): coalesced loads, and every lane adds.
// One lane per row node left 10 of 32 lanes busy for tet10 and 8 for hex8,
// and read a block of 72 bytes per lane (nine loads of 61 sectors each).
// G follows the length of the run (run_colgather): 32, or 16 or 8 lanes, two
// or four column nodes per warp, for runs that short.  Into a kept layout:
// tet10, 178,002 elements: 1.13 -> 0.55 ms; hex8 heat, 249,856 elements:
// 0.235 -> 0.112 ms; hex27, 64,000 elements (7.9 GB of traffic): 2.02 ->
// 1.89 ms, 4.2 TB/s, bound by latency at the 20 warps per SM that its two
// element columns in registers leave.  Fewer registers by a launch bound, by
// loading one element at a time, or by taking the nodes' pointers in batches
// with an L2 prefetch of the next node's columns were all slower (2.0 to 2.9
// ms).
//
// With FP64 values that are only moved, the values travel as their bit
// patterns (64-bit integers), so that moving, selecting and storing them
// takes no FP64 instruction.
#include "common.cuh"

#include <algorithm>
#include <vector>

namespace {

// Exact FP32 -> FP64 widening on the integer pipe (sign, exponent rebias,
// mantissa shift; subnormals normalised by their leading-zero count; Inf and
// NaN keep their payload): the precision form's gather widens every element
// value, and GB300's FP64 pipe is kept for the additions.
__device__ __forceinline__ double widen(unsigned long long b) { return __longlong_as_double((long long)b); }
__device__ __forceinline__ double widen(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned e = (u >> 23) & 0xffu, m = u & 0x7fffffu;
  if (e - 1u < 254u) {  // normal: in 32-bit halves, exponent + (1023 - 127), mantissa << 29
    const unsigned hi = (u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u);
    return __hiloint2double((int)hi, (int)(u << 29));
  }
  unsigned long long bits;
  if (e != 0u) {
    const unsigned long long ed = e == 0xffu ? 0x7ffull : (unsigned long long)(e + 896u);
    bits = (ed << 52) | ((unsigned long long)m << 29);
  } else if (m != 0u) {
    const int p = 31 - __clz((int)m);
    bits = ((unsigned long long)(p + 874) << 52) | (((unsigned long long)m << (52 - p)) & 0xfffffffffffffull);
  } else {
    bits = 0ull;
  }
  return __longlong_as_double((long long)(((unsigned long long)(u >> 31) << 63) | bits));
}
template <class T> struct GatherWord { using type = T; };
template <> struct GatherWord<double> { using type = unsigned long long; };
__device__ __forceinline__ unsigned long long value_bits(unsigned long long b) { return b; }
__device__ __forceinline__ unsigned long long value_bits(float f) {
  return (unsigned long long)__double_as_longlong(widen(f));
}

constexpr unsigned long long NEG_ZERO = 0x8000000000000000ull;  // the identity of IEEE addition

// Doubles of one column node's accumulator: P planes of an odd stride, so
// that the planes of one row position lie in different banks.
__host__ __device__ constexpr int plane_stride(int md, int P) { return (md * P) | 1; }

// T = double (FP64 form) or float (precision form); FP64 sums in element
// order in both.  BLOCKVAL: P x P blocks, entry (i,j) at i*P+j; otherwise one
// scalar per node pair, placed on the component diagonal.  NCH: most rounds
// of G lanes that an element column takes, whose values are prefetched one
// element ahead (longer ones: k_colgather_wide).
// first_marked: bit 15 of a map entry marks the first block of its row
// position; that block is stored and later ones are added, one FP64 addition
// per contribution after the first.  Otherwise, and with init (values to
// accumulate into), the accumulator starts from -0.0 or init and every block
// is added.  Without spec, the column is written to nz with its non-zero
// count; column (B,j) holds the entries (row node t, component i) at P*t + i.
// With spec.ptr0 it is compacted (dropzeros!) straight into the stored CSC at
// the layout of an earlier assembly: each DoF column's non-zeros go, in row
// order, to [ptr0[c], ptr0[c+1]) (writes stay inside that range) and its keep
// bits to spec.keep, and a column whose count differs sets *spec.mismatch.
template <int P, bool BLOCKVAL, class T, int G, int NCH>
__global__ void k_colgather(const int64_t *__restrict__ nptr, const int64_t *__restrict__ n2e_ptr,
                            const int2 *__restrict__ n2e, const uint16_t *__restrict__ pos,
                            const T *__restrict__ Kf, int64_t cs, int npe, int64_t non, int max_deg,
                            const double *__restrict__ init, double *__restrict__ nz,
                            int64_t *__restrict__ cnt, const int32_t *__restrict__ list,
                            const int32_t *__restrict__ nadj, StoredSpec spec, int first_marked) {
  extern __shared__ double cg_smem[];
  constexpr int NPW = 32 / G;                                    // column nodes per warp
  constexpr int VPN = BLOCKVAL ? P * P : P;                      // flat values per row node
  constexpr int BSTR = kf_bstride(P, BLOCKVAL, (int)sizeof(T));  // stored block stride
  using W = typename GatherWord<T>::type;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const int gl = lane & (G - 1), gi = lane / G;
  const int ps = plane_stride(max_deg, P);
  double *wacc = cg_smem + (size_t)wib * NPW * P * ps;
  double *acc = wacc + (size_t)gi * P * ps;
  unsigned long long *accb = reinterpret_cast<unsigned long long *>(acc);
  const int NV = npe * VPN;
  const bool store_first = first_marked && init == nullptr;
  const unsigned tmask = first_marked ? 0x7fffu : 0xffffu;
  const int nw = (int)non, wstride = (int)gridDim.x * wpb * NPW;  // node counts fit int32 (nadj holds int32 nodes)
  // where value f of an element column lies in memory and in the planes
  auto value_at = [](int f) { return BLOCKVAL ? (f / VPN) * BSTR + f % VPN : f / VPN; };
  auto plane_at = [&](int f, int t) {
    const int r = f % VPN;
    return BLOCKVAL ? (r % P) * ps + t * P + r / P : r * ps + t * P + r;
  };
  // add value f, v, of the row position in map entry raw
  auto put = [&](int f, unsigned raw, W v) {
    const int t = (int)(raw & tmask), at = plane_at(f, t);
    if (store_first && (raw & 0x8000u)) {
      accb[at] = value_bits(v);
      if (!BLOCKVAL)
#pragma unroll
        for (int j = 1; j < P; ++j) accb[((f % VPN + j) % P) * ps + t * P + f % VPN] = 0ull;
    } else {
      acc[at] = __dadd_rn(acc[at], widen(v));
      if (!BLOCKVAL && P > 1 && !store_first)
#pragma unroll
        for (int j = 1; j < P; ++j) {
          double *o = acc + ((f % VPN + j) % P) * ps + t * P + f % VPN;
          *o = __dadd_rn(*o, 0.0);
        }
    }
  };
  for (int w0 = ((int)blockIdx.x * wpb + wib) * NPW; w0 < nw; w0 += wstride) {
    const int w = w0 + gi;
    const bool act = NPW == 1 || w < nw;
    const int B = act ? (list ? __ldg(list + w) : w) : 0;  // column node (non: nodes of the list)
    const int64_t c0 = nptr[B], s = n2e_ptr[B];
    const int deg = act ? (int)(nptr[B + 1] - c0) : 0, nb = act ? (int)(n2e_ptr[B + 1] - s) : 0;
    int nbmax = nb;
#pragma unroll
    for (int off = G; off < 32; off <<= 1) nbmax = max(nbmax, __shfl_xor_sync(0xffffffffu, nbmax, off));
    if (!store_first) {
      const unsigned long long *src = reinterpret_cast<const unsigned long long *>(init) + (size_t)P * P * c0;
      for (int j = 0; j < P; ++j)
        for (int r = gl; r < P * deg; r += G) accb[j * ps + r] = init ? src[j * P * deg + r] : NEG_ZERO;
      __syncwarp();
    }
    {
      // VPN == 1: a lane's values have row nodes of their own; otherwise lane
      // a of the group holds the position of row node a (npe <= G)
      constexpr int NT = VPN == 1 ? NCH : 1;
      W cur[NCH], nxt[NCH];
      unsigned tc[NT], tn[NT];
      int2 el = make_int2(0, 0);   // elements k0 + gl of the list
#pragma unroll
      for (int m = 0; m < NT; ++m) tc[m] = tn[m] = 0xffffu;
      auto load = [&](int k, W *dst, unsigned *td) {
        if ((k & (G - 1)) == 0) el = k + gl < nb ? n2e[s + k + gl] : make_int2(0, 0);
        const int ex = __shfl_sync(0xffffffffu, el.x, k & (G - 1), G), ey = __shfl_sync(0xffffffffu, el.y, k & (G - 1), G);
        if (k < nb) {
          const W *col = reinterpret_cast<const W *>(Kf) + ((size_t)ex * npe + ey) * cs;
          const uint16_t *pk = pos + (s + k) * npe;
#pragma unroll
          for (int m = 0; m < NCH; ++m) {
            const int f = gl + m * G;
            if (f < NV) {
              dst[m] = col[value_at(f)];
              if (VPN == 1) td[m] = pk[f];
            }
          }
          if (VPN > 1 && gl < npe) td[0] = pk[gl];
        }
      };
      load(0, cur, tc);
      for (int k = 0; k < nbmax; ++k) {  // elements of B, ascending
        if (k + 1 < nbmax) load(k + 1, nxt, tn);
#pragma unroll
        for (int m = 0; m < NCH; ++m) {  // the values of one element hold distinct entries
          const int f = gl + m * G;
          const unsigned raw = VPN == 1 ? tc[m < NT ? m : 0] : __shfl_sync(0xffffffffu, tc[0], f / VPN, G);
          if (f < NV && k < nb && raw != 0xffffu) put(f, raw, cur[m]);
        }
        __syncwarp();
#pragma unroll
        for (int m = 0; m < NCH; ++m) cur[m] = nxt[m];
#pragma unroll
        for (int m = 0; m < NT; ++m) tc[m] = tn[m];
      }
    }
    // write-out, the warp over each of its column nodes: 64 entries at a time
#pragma unroll 1
    for (int n = 0; n < NPW; ++n) {
      if (NPW > 1 && w0 + n >= nw) break;   // warp-uniform
      const int Bn = NPW == 1 ? B : __shfl_sync(0xffffffffu, B, n * G);
      const int dn = NPW == 1 ? deg : __shfl_sync(0xffffffffu, deg, n * G);
      const int64_t cn = NPW == 1 ? c0 : nptr[Bn];
      const unsigned long long *ab = reinterpret_cast<const unsigned long long *>(wacc + (size_t)n * P * ps);
      const int len = P * dn;
      const unsigned below = (1u << lane) - 1u;
      if (spec.ptr0) {
        int64_t o[P], oend[P], kp[P];
        int run[P];
#pragma unroll
        for (int j = 0; j < P; ++j) {
          o[j] = spec.ptr0[(int64_t)P * Bn + j];
          oend[j] = spec.ptr0[(int64_t)P * Bn + j + 1];
          kp[j] = keep_pos((int64_t)P * P * cn + j * len, (int64_t)P * Bn + j);
          run[j] = 0;
        }
        for (int i0 = 0; i0 < len; i0 += 64) {
          const int ia = i0 + lane, ib = ia + 32;
          const int64_t ra = ia < len ? (int64_t)P * nadj[cn + ia / P] + ia % P + 1 : 0;
          const int64_t rb = ib < len ? (int64_t)P * nadj[cn + ib / P] + ib % P + 1 : 0;
#pragma unroll
          for (int j = 0; j < P; ++j) {
            const unsigned long long va = ia < len ? ab[j * ps + ia] : 0ull, vb = ib < len ? ab[j * ps + ib] : 0ull;
            const bool ka = (va << 1) != 0ull, kb = (vb << 1) != 0ull;   // every value but +-0
            const unsigned ba = __ballot_sync(0xffffffffu, ka), bb = __ballot_sync(0xffffffffu, kb);
            const int64_t ta = o[j] + run[j] + __popc(ba & below), tb = o[j] + run[j] + __popc(ba) + __popc(bb & below);
            if (ka && ta < oend[j]) {
              spec.rowval_s[ta] = ra;
              reinterpret_cast<unsigned long long *>(spec.nzval_s)[ta] = va;
            }
            if (kb && tb < oend[j]) {
              spec.rowval_s[tb] = rb;
              reinterpret_cast<unsigned long long *>(spec.nzval_s)[tb] = vb;
            }
            if (lane == 0) spec.keep[kp[j] + (i0 >> 6)] = make_uint2(ba, bb);
            run[j] += __popc(ba) + __popc(bb);
          }
        }
        bool differs = false;
#pragma unroll
        for (int j = 0; j < P; ++j) differs |= (int64_t)run[j] != oend[j] - o[j];
        if (lane == 0 && differs) atomicOr(spec.mismatch, 1u);
      } else {
#pragma unroll 1
        for (int j = 0; j < P; ++j) {
          unsigned long long *out = reinterpret_cast<unsigned long long *>(nz) + (size_t)P * P * cn + (size_t)j * len;
          int c = 0;
          for (int i0 = 0; i0 < len; i0 += 64) {
            const int ia = i0 + lane, ib = ia + 32;
            const unsigned long long va = ia < len ? ab[j * ps + ia] : 0ull, vb = ib < len ? ab[j * ps + ib] : 0ull;
            if (ia < len) out[ia] = va;
            if (ib < len) out[ib] = vb;
            c += __popc(__ballot_sync(0xffffffffu, (va << 1) != 0ull)) +
                 __popc(__ballot_sync(0xffffffffu, (vb << 1) != 0ull));
          }
          if (lane == 0 && cnt) cnt[(int64_t)P * Bn + j] = c;
        }
      }
    }
    __syncwarp();
  }
}

// The same gather with a CTA of NT threads per column node, for element
// columns longer than a warp takes in the rounds above: the accumulator of
// such a node (hex125: 18 to 53 KB) leaves room for few nodes on an SM, and a
// warp each left it with four warps.  The values of an element column (at most
// NT R) go over the CTA's threads, R each, loaded an element ahead, with a
// barrier between elements; a plane is written out by the
// warps w, w + P, ..., a part each.
// Bound by latency and the barriers.  Both degree classes, against a warp
// each: hex125 576 elements from FP32 matrices 0.98 -> 0.37 ms, 216 from FP64
// ones 0.53 -> 0.29; tet35, 3,072 turned 0.46 -> 0.30; hex64, 1,000 turned 0.305
// -> 0.301 and, from FP32, 0.34 -> 0.28 ms.  hex27 (243 values) stays with a
// warp each: 1.88 against 2.56 ms for 64,000 elements.
template <int P, bool BLOCKVAL, class T, int NT, int R>
__global__ void __launch_bounds__(NT, NT == 192 ? 5 : 0)
k_colgather_wide(const int64_t *__restrict__ nptr, const int64_t *__restrict__ n2e_ptr,
                 const int2 *__restrict__ n2e, const uint16_t *__restrict__ pos, const T *__restrict__ Kf, int64_t cs,
                 int npe, int64_t non, int max_deg, const double *__restrict__ init, double *__restrict__ nz,
                 int64_t *__restrict__ cnt, const int32_t *__restrict__ list, const int32_t *__restrict__ nadj,
                 StoredSpec spec, int first_marked) {
  extern __shared__ double cg_smem[];
  constexpr int VPN = BLOCKVAL ? P * P : P;
  constexpr int BSTR = kf_bstride(P, BLOCKVAL, (int)sizeof(T));
  constexpr int PARTS = NT / 32 / P;   // warps per plane of the write-out
  static_assert(PARTS >= 1, "a warp per plane");
  using W = typename GatherWord<T>::type;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ps = plane_stride(max_deg, P), NV = npe * VPN;
  double *acc = cg_smem;
  unsigned long long *accb = reinterpret_cast<unsigned long long *>(acc);
  const bool store_first = first_marked && init == nullptr;
  const unsigned tmask = first_marked ? 0x7fffu : 0xffffu;
  auto put = [&](int f, unsigned raw, W v) {   // k_colgather's
    const int t = (int)(raw & tmask), r = f % VPN;
    const int at = BLOCKVAL ? (r % P) * ps + t * P + r / P : r * ps + t * P + r;
    if (store_first && (raw & 0x8000u)) {
      accb[at] = value_bits(v);
      if (!BLOCKVAL)
#pragma unroll
        for (int j = 1; j < P; ++j) accb[((r + j) % P) * ps + t * P + r] = 0ull;
    } else {
      acc[at] = __dadd_rn(acc[at], widen(v));
      if (!BLOCKVAL && P > 1 && !store_first)
#pragma unroll
        for (int j = 1; j < P; ++j) {
          double *o = acc + ((r + j) % P) * ps + t * P + r;
          *o = __dadd_rn(*o, 0.0);
        }
    }
  };
  for (int w = blockIdx.x; w < (int)non; w += (int)gridDim.x) {
    const int B = list ? __ldg(list + w) : w;
    const int64_t c0 = nptr[B], s = n2e_ptr[B];
    const int deg = (int)(nptr[B + 1] - c0), nb = (int)(n2e_ptr[B + 1] - s), len = P * deg;
    if (!store_first) {
      const unsigned long long *src = reinterpret_cast<const unsigned long long *>(init) + (size_t)P * P * c0;
      for (int j = 0; j < P; ++j)
        for (int r = tid; r < len; r += NT) accb[j * ps + r] = init ? src[j * len + r] : NEG_ZERO;
      __syncthreads();
    }
    auto load = [&](int2 el, int k, W *v, unsigned *raw) {
      const W *col = reinterpret_cast<const W *>(Kf) + ((size_t)el.x * npe + el.y) * cs;
      const uint16_t *pk = pos + (s + k) * npe;
#pragma unroll
      for (int m = 0; m < R; ++m) {
        const int f = tid + m * NT;
        raw[m] = 0xffffu;
        if (f < NV) {
          raw[m] = pk[f / VPN];
          v[m] = col[BLOCKVAL ? (f / VPN) * BSTR + f % VPN : f / VPN];
        }
      }
    };
    W cur[R], nxt[R];
    unsigned rc[R], rn[R];
    int2 en = nb > 1 ? n2e[s + 1] : make_int2(0, 0);   // the next element of the list
    if (nb > 0) load(n2e[s], 0, cur, rc);
    for (int k = 0; k < nb; ++k) {   // elements of B, ascending
      const int2 e2 = k + 2 < nb ? n2e[s + k + 2] : make_int2(0, 0);
      if (k + 1 < nb) load(en, k + 1, nxt, rn);
#pragma unroll
      for (int m = 0; m < R; ++m)
        if (rc[m] != 0xffffu) put(tid + m * NT, rc[m], cur[m]);
#pragma unroll
      for (int m = 0; m < R; ++m) {
        cur[m] = nxt[m];
        rc[m] = rn[m];
      }
      en = e2;
      __syncthreads();   // an entry's sum goes by elements
    }
    const int j = warp % P, part = warp / P;
    if (part < PARTS) {
      const unsigned long long *ab = accb + (size_t)j * ps;
      const unsigned below = (1u << lane) - 1u;
      const int blocks = (len + 63) / 64, i0 = blocks * part / PARTS * 64, i1 = min(blocks * (part + 1) / PARTS * 64, len);
      int run = 0;   // non-zeros of the plane before the current 64 entries
      for (int i = lane; i < i0; i += 32) run += (ab[i] << 1) != 0ull;   // every value but +-0
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) run += __shfl_xor_sync(0xffffffffu, run, off);
      const int64_t c = (int64_t)P * B + j;
      const int64_t o = spec.ptr0 ? spec.ptr0[c] : 0, oend = spec.ptr0 ? spec.ptr0[c + 1] : 0;
      unsigned long long *out = reinterpret_cast<unsigned long long *>(nz) + (size_t)P * P * c0 + (size_t)j * len;
      for (int i = i0; i < i1; i += 64) {
        const int ia = i + lane, ib = ia + 32;
        const unsigned long long va = ia < len ? ab[ia] : 0ull, vb = ib < len ? ab[ib] : 0ull;
        const bool ka = (va << 1) != 0ull, kb = (vb << 1) != 0ull;
        const unsigned ba = __ballot_sync(0xffffffffu, ka), bb = __ballot_sync(0xffffffffu, kb);
        if (spec.ptr0) {
          const int64_t ta = o + run + __popc(ba & below), tb = o + run + __popc(ba) + __popc(bb & below);
          if (ka && ta < oend) {
            spec.rowval_s[ta] = (int64_t)P * nadj[c0 + ia / P] + ia % P + 1;
            reinterpret_cast<unsigned long long *>(spec.nzval_s)[ta] = va;
          }
          if (kb && tb < oend) {
            spec.rowval_s[tb] = (int64_t)P * nadj[c0 + ib / P] + ib % P + 1;
            reinterpret_cast<unsigned long long *>(spec.nzval_s)[tb] = vb;
          }
          if (lane == 0) spec.keep[keep_pos((int64_t)P * P * c0 + (int64_t)j * len, c) + (i >> 6)] = make_uint2(ba, bb);
        } else {
          if (ia < len) out[ia] = va;
          if (ib < len) out[ib] = vb;
        }
        run += __popc(ba) + __popc(bb);
      }
      if (part == PARTS - 1 && lane == 0) {   // run: the plane's count
        if (spec.ptr0) {
          if ((int64_t)run != oend - o) atomicOr(spec.mismatch, 1u);
        } else if (cnt) {
          cnt[c] = run;
        }
      }
    }
    __syncthreads();
  }
}

// The column nodes of the pattern in two degree classes, once per pattern:
// when at least 60 % of the nodes have a degree of at most 0.7 of the
// largest, those nodes form the low class (ascending), the rest follow.
// The low class then runs with a smaller accumulator and so with more warps
// per SM (hex27: degree <= 75 against 125 for 7/8 of the nodes).  Each
// column is summed the same way whichever launch takes it.
static int gather_split(llf_ctx *ctx, llf_pattern *pat) {
  if (pat->gather_split_done) return LLF_OK;
  pat->gather_split_done = true;
  const int64_t non = pat->mesh->non;
  const int thr = pat->tune.gather_thr;   // percent of the largest degree
  if (non < 1024 || pat->max_deg < 16 || thr <= 0) return LLF_OK;
  std::vector<int64_t> h(non + 1);
  LLF_CUDA_TRY(ctx, cudaMemcpyAsync(h.data(), pat->d_nptr, sizeof(int64_t) * (non + 1), cudaMemcpyDeviceToHost,
                                    ctx->stream));
  LLF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  std::vector<int64_t> hist(pat->max_deg + 1, 0);
  for (int64_t b = 0; b < non; ++b) hist[h[b + 1] - h[b]]++;
  int md_low = -1;
  int64_t acc = 0;
  for (int d = 0; d <= pat->max_deg; ++d) {
    acc += hist[d];
    if (acc >= (non * 6 + 9) / 10) { md_low = d; break; }
  }
  if (md_low < 1 || md_low * 100 > pat->max_deg * thr) return LLF_OK;
  std::vector<int32_t> order;
  order.reserve(non);
  for (int64_t b = 0; b < non; ++b)
    if (h[b + 1] - h[b] <= md_low) order.push_back((int32_t)b);
  const int64_t n_low = (int64_t)order.size();
  for (int64_t b = 0; b < non; ++b)
    if (h[b + 1] - h[b] > md_low) order.push_back((int32_t)b);
  LLF_CUDA_TRY(ctx, dalloc(ctx, &pat->d_gather_nodes, non));
  LLF_CUDA_TRY(ctx, cudaMemcpyAsync(pat->d_gather_nodes, order.data(), sizeof(int32_t) * non, cudaMemcpyHostToDevice,
                                    ctx->stream));
  LLF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  pat->gather_n_low = n_low;
  pat->gather_md_low = md_low;
  return LLF_OK;
}

// Marks, once per pattern, the first block of every row position in the
// pattern's element-to-column map: per column node B (a warp each), its
// elements in ascending order, and the first element whose block reaches a
// row position gets bit 15 of that map entry (positions fit 15 bits).  The
// gather then stores that block and adds the later ones without keeping
// per-position marks of its own.
__global__ void k_mark_first(const int64_t *__restrict__ nptr, const int64_t *__restrict__ n2e_ptr,
                             uint16_t *__restrict__ pos, int npe, int64_t non, int max_deg) {
  extern __shared__ unsigned char mf_has[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  unsigned char *has = mf_has + (size_t)wib * ((max_deg + 7) & ~7);
  for (int64_t B = (int64_t)blockIdx.x * wpb + wib; B < non; B += (int64_t)gridDim.x * wpb) {
    const int deg = (int)(nptr[B + 1] - nptr[B]);
    const int64_t s = n2e_ptr[B];
    const int nb = (int)(n2e_ptr[B + 1] - s);
    for (int t = lane; t < deg; t += 32) has[t] = 0;
    __syncwarp();
    for (int k = 0; k < nb; ++k) {
      for (int a = lane; a < npe; a += 32) {  // the lanes of one element hold distinct positions
        const unsigned raw = pos[(s + k) * npe + a];
        if (raw < 0x8000u && !has[raw]) {
          has[raw] = 1;
          pos[(s + k) * npe + a] = (uint16_t)(raw | 0x8000u);
        }
      }
      __syncwarp();
    }
  }
}

// launch(md, list, b0, count): the column nodes of the list, or [b0, b0 +
// count), with accumulators of md row positions; the pattern's two degree
// classes one after the other when all its nodes are asked for.
template <class F>
int gather_classes(llf_ctx *ctx, llf_pattern *pat, int64_t B0, int64_t nB, F launch) {
  const int md = pat->max_deg > 0 ? pat->max_deg : 1;
  if (B0 == 0 && nB == pat->mesh->non) {
    int rc = gather_split(ctx, pat);
    if (rc != LLF_OK) return rc;
    if (pat->d_gather_nodes) {
      rc = launch(pat->gather_md_low, pat->d_gather_nodes, (int64_t)0, pat->gather_n_low);
      if (rc == LLF_OK)
        rc = launch(md, pat->d_gather_nodes + pat->gather_n_low, (int64_t)0, pat->mesh->non - pat->gather_n_low);
      return rc;
    }
  }
  return launch(md, (const int32_t *)nullptr, B0, nB);
}

template <int P, bool BV, class T, int G, int NCH>
int launch_colgather(llf_ctx *ctx, llf_pattern *pat, const int64_t *n2e_ptr, const int2 *n2e, const uint16_t *pos,
                     int npe, const T *Kf, int64_t cs, const double *init, double *nz, int64_t *cnt, int64_t B0,
                     int64_t nB, const StoredSpec &sp, bool first_marked) {
  auto fn = k_colgather<P, BV, T, G, NCH>;
  constexpr int NPW = 32 / G;
  return gather_classes(ctx, pat, B0, nB, [&](int md, const int32_t *list, int64_t b0, int64_t count) -> int {
    if (count <= 0) return LLF_OK;
    const size_t per_warp = (size_t)NPW * P * plane_stride(md, P) * sizeof(double);
    int wpb = (int)std::min<size_t>(pat->tune.gather_wpb > 0 ? pat->tune.gather_wpb : 4, (200 * 1024) / per_warp);
    if (wpb < 1) wpb = 1;
    const size_t smem = (size_t)wpb * per_warp;
    if (smem > 200 * 1024)
      return llf_fail(ctx, LLF_ERR_LIMIT, "a column node has too many neighbours for the gather buffer");
    if (smem > 48 * 1024)
      LLF_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 1;
    LLF_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, wpb * 32, smem));
    const int64_t need = (count + wpb * NPW - 1) / (wpb * NPW);
    const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)ctx->num_sms * std::max(per_sm, 1), need));
    KernelScope ks(ctx, "k_colgather");
    fn<<<(unsigned)grid, wpb * 32, smem, ctx->stream>>>(pat->d_nptr + b0, n2e_ptr + b0, n2e, pos, Kf, cs, npe, count,
                                                        md, init, nz, cnt ? cnt + b0 * P : nullptr, list,
                                                        pat->d_nadj, sp, first_marked ? 1 : 0);
    LLF_CUDA_TRY(ctx, cudaGetLastError());
    return LLF_OK;
  });
}

template <int P, bool BV, class T, int NT, int R>
int launch_wide(llf_ctx *ctx, llf_pattern *pat, const int64_t *n2e_ptr, const int2 *n2e, const uint16_t *pos, int npe,
                const T *Kf, int64_t cs, const double *init, double *nz, int64_t *cnt, int64_t B0, int64_t nB,
                const StoredSpec &sp, bool first_marked) {
  auto fn = k_colgather_wide<P, BV, T, NT, R>;
  return gather_classes(ctx, pat, B0, nB, [&](int md, const int32_t *list, int64_t b0, int64_t count) -> int {
    if (count <= 0) return LLF_OK;
    const size_t smem = (size_t)P * plane_stride(md, P) * sizeof(double);
    if (smem > 200 * 1024)
      return llf_fail(ctx, LLF_ERR_LIMIT, "a column node has too many neighbours for the gather buffer");
    if (smem > 48 * 1024)
      LLF_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 1;
    LLF_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, NT, smem));
    const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)ctx->num_sms * std::max(per_sm, 1), count));
    KernelScope ks(ctx, "k_colgather_wide");
    fn<<<(unsigned)grid, NT, smem, ctx->stream>>>(pat->d_nptr + b0, n2e_ptr + b0, n2e, pos, Kf, cs, npe, count, md, init,
                                                  nz, cnt ? cnt + b0 * P : nullptr, list, pat->d_nadj, sp,
                                                  first_marked ? 1 : 0);
    LLF_CUDA_TRY(ctx, cudaGetLastError());
    return LLF_OK;
  });
}

// Gather over explicit node -> element lists and element-to-column map (the
// pattern's own, or those of another element set on the same nodes) of the
// column nodes [B0, B0 + nB): the node-indexed arrays are offset, the
// offsets they hold (into n2e, pos, nz) stay absolute.
template <int P, bool BV, class T>
int run_colgather(llf_ctx *ctx, llf_pattern *pat, const int64_t *n2e_ptr, const int2 *n2e, const uint16_t *pos,
                  int npe, const T *Kf, int64_t cs, const double *init, double *nz, int64_t *cnt, int64_t B0,
                  int64_t nB, const StoredSpec *spec) {
  const StoredSpec sp = spec ? *spec : StoredSpec{};
  if (nB < 0) nB = pat->mesh->non - B0;
  if (pat->conn_version != pat->mesh->conn_version)
    return llf_fail(ctx, LLF_ERR_STATE, "the mesh connectivity changed after the pattern was built; rebuild it");
  // the pattern's own map: each position's first block marked (once)
  bool first_marked = false;
  const int mdm = pat->max_deg > 0 ? pat->max_deg : 1;
  if (pos == pat->d_pos && mdm < 0x7fff) {
    if (!pat->pos_first) {
      const int mw = 4;
      const size_t msm = (size_t)mw * ((mdm + 7) & ~7);
      KernelScope ks(ctx, "k_mark_first");
      k_mark_first<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((pat->mesh->non + mw - 1) / mw,
                                                                    (int64_t)ctx->num_sms * 8)),
                     mw * 32, msm, ctx->stream>>>(pat->d_nptr, pat->d_n2e_ptr, pat->d_pos, npe, pat->mesh->non, mdm);
      LLF_CUDA_TRY(ctx, cudaGetLastError());
      pat->pos_first = true;
    }
    first_marked = true;
  }
  // lanes per column node and rounds of them: the whole element column in
  // one round of 8 or 16 lanes, else rounds of 32 (prefetched up to 8; a
  // group then needs a lane per row node unless every value has its own)
  constexpr int VPN = BV ? P * P : P;
  const int nv = npe * VPN, rounds = (nv + 31) / 32;
  const bool lanes = VPN == 1 || npe <= 32;
#define LLF_GATHER(G, N) \
  return launch_colgather<P, BV, T, G, N>(ctx, pat, n2e_ptr, n2e, pos, npe, Kf, cs, init, nz, cnt, B0, nB, sp, first_marked)
  if (nv <= 8) LLF_GATHER(8, 1);
  if (nv <= 16) LLF_GATHER(16, 1);
  if (rounds == 1) LLF_GATHER(32, 1);
  if (rounds <= 3 && lanes) LLF_GATHER(32, 3);
  // the longest columns are quad25's (100 values) with two components and
  // hex125's (125) with one, hex27's (243) with three: rounds that no column
  // needs still cost registers and predicates (quad25, 40,000 elements: 737 us
  // with eight rounds, 503 with four)
  constexpr int LONGEST = P <= 2 ? 4 : 8;
  if (rounds <= LONGEST && lanes) LLF_GATHER(32, LONGEST);
#undef LLF_GATHER
#define LLF_WIDE(NT, R) \
  return launch_wide<P, BV, T, NT, R>(ctx, pat, n2e_ptr, n2e, pos, npe, Kf, cs, init, nz, cnt, B0, nB, sp, first_marked)
  // longer: a CTA per column node, the rounds that use its threads and its
  // registers best (measured with 64 to 576 threads).  Each is instantiated for
  // the columns that come to it: with two components scalars of hex64 and
  // hex125 (128 and 250 values), with three scalars (tet35 105 to hex125 375)
  // and blocks (tet35 315, hex64 576, hex125 1125)
  if constexpr (P == 3 || (P == 2 && !BV))
    if (nv <= 160 * 2) LLF_WIDE(160, 2);
  if constexpr (P == 3)
    if (nv <= 192 * 3) LLF_WIDE(192, 3);
  if constexpr (P == 3 && BV)
    if (nv <= 288 * 4) LLF_WIDE(288, 4);
  return llf_fail(ctx, LLF_ERR_LIMIT, "an element has too many nodes for the gather");
#undef LLF_WIDE
}

template <class T>
int gather_full_t(llf_ctx *ctx, llf_pattern *pat, const int64_t *n2e_ptr, const int2 *n2e, const uint16_t *pos,
                  int npe, const T *Kf, int64_t cs, bool blockval, const double *init, double *nz, int64_t *cnt,
                  const StoredSpec *spec = nullptr, int64_t B0 = 0, int64_t nB = -1) {
  switch (pat->pdim * 2 + (blockval ? 1 : 0)) {
    case 2:   // one component: a block is a scalar
    case 3: return run_colgather<1, true, T>(ctx, pat, n2e_ptr, n2e, pos, npe, Kf, cs, init, nz, cnt, B0, nB, spec);
    case 4: return run_colgather<2, false, T>(ctx, pat, n2e_ptr, n2e, pos, npe, Kf, cs, init, nz, cnt, B0, nB, spec);
    case 5: return run_colgather<2, true, T>(ctx, pat, n2e_ptr, n2e, pos, npe, Kf, cs, init, nz, cnt, B0, nB, spec);
    case 6: return run_colgather<3, false, T>(ctx, pat, n2e_ptr, n2e, pos, npe, Kf, cs, init, nz, cnt, B0, nB, spec);
    case 7: return run_colgather<3, true, T>(ctx, pat, n2e_ptr, n2e, pos, npe, Kf, cs, init, nz, cnt, B0, nB, spec);
  }
  return llf_fail(ctx, LLF_ERR_UNSUPPORTED, "pdim must be 1, 2 or 3");
}

// The gather into a kept stored layout; if a column's count differs, the
// usual gather (structural values and counts) follows.
template <class T>
int gather_spec_t(llf_ctx *ctx, llf_pattern *pat, const T *Kf, int64_t cs, bool blockval, StoredSpec *spec) {
  int rc = gather_full_t<T>(ctx, pat, pat->d_n2e_ptr, pat->d_n2e, pat->d_pos, pat->mesh->npe, Kf, cs, blockval,
                            nullptr, nullptr, nullptr, spec);
  if (rc != LLF_OK) return rc;
  // the status of the whole assembly comes with the mismatch word: one copy
  // into pinned memory and one wait
  LLF_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_status, ctx->d_status, 2 * sizeof(unsigned), cudaMemcpyDeviceToHost,
                                    ctx->stream));
  LLF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  spec->status_read = true;
  if (ctx->h_status[1] == 0) return LLF_OK;
  spec->fell_back = true;
  LLF_CUDA_TRY(ctx, cudaMemsetAsync(spec->mismatch, 0, sizeof(unsigned), ctx->stream));
  LLF_CUDA_TRY(ctx, cudaMemsetAsync(spec->cnt_fallback, 0, sizeof(int64_t) * (pat->ndof + 1), ctx->stream));
  LLF_CUDA_TRY(ctx, dalloc(ctx, spec->nz_slot, pat->nnz));
  return gather_full_t<T>(ctx, pat, pat->d_n2e_ptr, pat->d_n2e, pat->d_pos, pat->mesh->npe, Kf, cs, blockval,
                          nullptr, *spec->nz_slot, spec->cnt_fallback);
}

}  // namespace

int gather_full(llf_ctx *ctx, llf_pattern *pat, const double *Kf, int64_t colstride, bool blockval,
                double *nz, int64_t *cnt, const double *init, StoredSpec *spec) {
  if (spec) return gather_spec_t<double>(ctx, pat, Kf, colstride, blockval, spec);
  return gather_full_t<double>(ctx, pat, pat->d_n2e_ptr, pat->d_n2e, pat->d_pos, pat->mesh->npe, Kf, colstride,
                               blockval, init, nz, cnt);
}
int gather_full32(llf_ctx *ctx, llf_pattern *pat, const float *Kf, int64_t colstride, bool blockval,
                  double *nz, int64_t *cnt, const double *init, StoredSpec *spec) {
  if (spec) return gather_spec_t<float>(ctx, pat, Kf, colstride, blockval, spec);
  return gather_full_t<float>(ctx, pat, pat->d_n2e_ptr, pat->d_n2e, pat->d_pos, pat->mesh->npe, Kf, colstride,
                              blockval, init, nz, cnt);
}
int gather_full_ext(llf_ctx *ctx, llf_pattern *pat, const int64_t *n2e_ptr, const int2 *n2e, const uint16_t *pos,
                    int npe, const double *Kf, int64_t colstride, bool blockval, double *nz, int64_t *cnt) {
  return gather_full_t<double>(ctx, pat, n2e_ptr, n2e, pos, npe, Kf, colstride, blockval, nullptr, nz, cnt);
}
int gather_slab(llf_ctx *ctx, llf_pattern *pat, const double *Kf, int64_t cs, bool blockval, double *nz, int64_t *cnt,
                int64_t B0, int64_t nB) {
  return gather_full_t<double>(ctx, pat, pat->d_n2e_ptr, pat->d_n2e, pat->d_pos, pat->mesh->npe, Kf, cs, blockval,
                               nullptr, nz, cnt, nullptr, B0, nB);
}
int gather_slab(llf_ctx *ctx, llf_pattern *pat, const float *Kf, int64_t cs, bool blockval, double *nz, int64_t *cnt,
                int64_t B0, int64_t nB) {
  return gather_full_t<float>(ctx, pat, pat->d_n2e_ptr, pat->d_n2e, pat->d_pos, pat->mesh->npe, Kf, cs, blockval,
                              nullptr, nz, cnt, nullptr, B0, nB);
}
