// Strided batched GEMM over any algebra on the CUDA cores (k_gemm_simt), and in
// Float64 on the FP64 matrix instructions (k_gemm_dmma).
//
// Replaces analyze_binary's permute -> reshape -> (batched) GEMM chain
// (src/einsum.jl:104-124, src/binaryrules.jl:46-61,94-141, src/utils.jl:162-177,
// ext/CUDAExt.jl:115-117,156-178) for the element types whose arithmetic the
// tensor cores do not have (Int64, Bool, tropical, FP64, ComplexF64), for
// ComplexF32 and FP32 products too small for them, and for the plain FP32
// comparison path.  Operands are read in place through per-group mode strides,
// so no permuted copy is ever materialised; the output permutation is absorbed
// in the epilogue's strides.
#include <cooperative_groups.h>
#include <string.h>
#include <algorithm>
#include "kernels.h"

namespace ome {

// Launch arguments of k_gemm_simt.  The mode groups carry invariant-divisor
// constants, so that an offset costs four integer instructions per mode
// instead of a 64-bit division (`wide`: a group's extent does not fit 31 bits
// and 64-bit divisions are used: div[i].d and .m are then the low and the high
// half of the mode's extent).
struct SimtGroup {
  int32_t n;
  FastDiv div[MAXG];
  int64_t s0[MAXG], s1[MAXG];      // strides in the two tensors that have the group
};
struct SimtArgs {
  const void* A;
  const void* B;
  void* C;
  int64_t M, N, K, L;
  SimtGroup m, n, k, l;            // m: A, C   n: B, C   k: A, B   l: A, B
  int64_t l_sc[MAXG];
  int32_t a_rowfast, b_rowfast;    // consecutive threads load consecutive rows (else consecutive k)
  int32_t wide;
  int32_t S;                       // K splits (1: the epilogue writes C)
  int64_t kchunk;                  // K per split
  int64_t tiles_m, tiles_n, units;
  int32_t cluster;                 // 1: a tile's splits form a cluster and add up in shared memory
  void* partial;                   // S > 1 without a cluster: [S][L][M][N]
  int64_t p_elems;                 // its capacity in elements (self-check)
  RangeFlag only_if;               // nothing is done unless this is set (word NULL: always done)
  Scalar sx, sy;
  int sy_zero, sx_one;
};
// set (5) when a split partial's offset falls outside the scratch (self-check)
__device__ int g_ome_bounds_simt = 0;

__device__ __forceinline__ int64_t simt_off(int64_t i, const SimtGroup& g, const int64_t* str, int wide) {
  if (g.n == 1) return i * str[0];
  int64_t off = 0;
  if (!wide) {
    uint32_t r = (uint32_t)i;
    for (int m = 0; m < g.n; ++m) {
      const uint32_t q = fast_div(r, g.div[m]);
      off += (int64_t)(r - q * g.div[m].d) * str[m];
      r = q;
    }
  } else {
    for (int m = 0; m < g.n; ++m) {
      const int64_t e = (int64_t)(g.div[m].d | (uint64_t)g.div[m].m << 32), q = i / e;
      off += (i - q * e) * str[m];
      i = q;
    }
  }
  return off;
}

// One multiply-add of a thread's accumulator.  Int64 keeps a 64-bit sum of
// the low words' products and a 32-bit sum of the cross products, joined once
// at the end: three integer multiply-adds per step instead of four and an add.
// Max-plus takes two steps at a time (one three-input maximum).
template <class A>
struct SimtMac {
  using T = typename A::T;
  using Acc = T;
  static constexpr int STEP = 1;
  static __device__ __forceinline__ Acc init() { return A::zero(); }
  static __device__ __forceinline__ void mac(Acc& c, T a, T b) { c = A::fma(a, b, c); }
  static __device__ __forceinline__ T value(const Acc& c) { return c; }
};
template <>
struct SimtMac<AlgI64> {
  using T = long long;
  struct Acc {
    unsigned long long lo;
    uint32_t hi;
  };
  static constexpr int STEP = 1;
  static __device__ __forceinline__ Acc init() { return Acc{0ull, 0u}; }
  static __device__ __forceinline__ void mac(Acc& c, T a, T b) {
    const uint32_t al = (uint32_t)a, bl = (uint32_t)b;
    const uint32_t ah = (uint32_t)((unsigned long long)a >> 32), bh = (uint32_t)((unsigned long long)b >> 32);
    c.lo += (unsigned long long)al * bl;
    c.hi += al * bh;
    c.hi += ah * bl;
  }
  static __device__ __forceinline__ T value(const Acc& c) { return (T)(c.lo + ((unsigned long long)c.hi << 32)); }
};
template <>
struct SimtMac<AlgTF32> {
  using T = float;
  using Acc = float;
  static constexpr int STEP = 2;
  static __device__ __forceinline__ Acc init() { return AlgTF32::zero(); }
  static __device__ __forceinline__ void mac2(Acc& c, T a0, T b0, T a1, T b1) {
    c = max3_nan(c, a0 + b0, a1 + b1);
  }
  static __device__ __forceinline__ void mac(Acc& c, T a, T b) { c = AlgTF32::fma(a, b, c); }
  static __device__ __forceinline__ T value(const Acc& c) { return c; }
};

// N consecutive elements of shared memory as the widest aligned loads.
template <class T, int N>
__device__ __forceinline__ void lds_run(const T* p, T (&v)[N]) {
  if constexpr ((sizeof(T) * N) % 16 == 0) {
    constexpr int W = (int)(sizeof(T) * N / 16);
    uint4 w[W];
    const uint4* q = reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = q[i];
    memcpy(v, w, sizeof(v));
  } else if constexpr ((sizeof(T) * N) % 8 == 0) {
    constexpr int W = (int)(sizeof(T) * N / 8);
    uint2 w[W];
    const uint2* q = reinterpret_cast<const uint2*>(p);
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = q[i];
    memcpy(v, w, sizeof(v));
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = p[i];
  }
}

// One element from global to shared memory, asynchronously where the element
// is a cp.async size.
template <class T>
__device__ __forceinline__ void cp_elem(T* dst, const T* src) {
  if constexpr (sizeof(T) == 4 || sizeof(T) == 8 || sizeof(T) == 16) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"((int)sizeof(T)) : "memory");
  } else {
    *dst = *src;
  }
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Tile configuration: BM x BN output tile, TM x TN per thread, BK per stage.
template <class T, int BM_, int BN_, int TM_, int TN_, int BK_, int MINB_>
struct SimtTile {
  static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, BK = BK_, MINB = MINB_;
  static constexpr int TX = BN / TN, TY = BM / TM, NT = TX * TY;
  static constexpr int STAGES = 4;
  // columns per thread come in runs of G = 8 bytes, TX * G apart: a warp's
  // reads of B are conflict-free and its stores to C fill whole sectors
  static constexpr int G = (int)(8 / sizeof(T)) < 1 ? 1 : ((int)(8 / sizeof(T)) < TN ? (int)(8 / sizeof(T)) : TN);
  static constexpr int PAD = sizeof(T) >= 16 ? 1 : (int)(16 / sizeof(T));
  static constexpr int PA = BM + PAD, PB = BN + PAD;
  static constexpr int STAGE = (PA + PB) * BK;
  static constexpr size_t TABLES = (2 * BM + 2 * BN + (STAGES + 1) * 2 * BK) * sizeof(int64_t);
  static constexpr size_t SMEM = TABLES + (size_t)STAGES * STAGE * sizeof(T) +
                                 (std::is_same<T, long long>::value ? 2 * (BM + BN) * BK : 0);
  static constexpr bool CLUSTER = BM * BN <= STAGES * STAGE;   // a tile fits the stages
};

// Unit u -> tile, K split and batch; a cluster's blocks are a tile's splits.
__device__ __forceinline__ void simt_unit(const SimtArgs& g, int64_t u, int64_t& tm, int64_t& tn, int64_t& spi,
                                          int64_t& l) {
  int64_t r = u;
  if (g.cluster) {
    spi = r % g.S;
    r /= g.S;
  }
  tm = r % g.tiles_m;
  r /= g.tiles_m;
  tn = r % g.tiles_n;
  r /= g.tiles_n;
  if (!g.cluster) {
    spi = r % g.S;
    r /= g.S;
  }
  l = r;
}

// A tile's partial sums, one per block of the cluster in `tile` ([BM][BN],
// type V), added in split order; each block finishes its share of the tile.
template <class A, class V, int BM, int BN, int NT>
__device__ __forceinline__ void simt_cluster_finish(const SimtArgs& g, V* tile, const int64_t* cm, const int64_t* cn,
                                                    int64_t lc, int64_t m0, int64_t n0, int rank, int tid) {
  using T = typename A::T;
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  cl.sync();
  const T sx = scalar_as<T>(g.sx), sy = scalar_as<T>(g.sy);
  T* Cp = static_cast<T*>(g.C);
  for (int e = rank * NT + tid; e < BM * BN; e += g.S * NT) {
    const int mi = e / BN, nj = e % BN;
    if (m0 + mi >= g.M || n0 + nj >= g.N) continue;
    V acc = *cl.map_shared_rank(tile + e, 0);
    for (int q = 1; q < g.S; ++q) {
      const V w = *cl.map_shared_rank(tile + e, q);
      if constexpr (std::is_same<V, T>::value) acc = A::add(acc, w);
      else acc = acc + w;
    }
    T* cp = Cp + lc + cm[mi] + cn[nj];
    *cp = epilogue<A>((T)acc, cp, sx, sy, g.sy_zero, g.sx_one);
  }
  cl.sync();   // the other blocks have read this one's sums
}

// One operand of a tile: where its rows and its split's k start.
template <class T>
struct SimtOperand {
  const T* base;            // batch l
  const int64_t* rowoff;    // offsets of the tile's rows (shared memory)
  int rows;                 // rows of the tile inside the extent
  int rowfast;              // consecutive threads take consecutive rows (else consecutive k)
  int uniform;              // the index a thread steps over is one mode of stride `step`
  int64_t step;
};

// ROWS x BK elements of one operand into a stage ([k][row], pitch P): rows
// beyond the extent and k beyond the split get the algebra's zero.  A thread
// keeps its place along the fast index and steps along the other one; where
// that one is a single mode, its addresses differ by a constant (one table
// look-up per stage: per-element look-ups took as many shared-memory
// wavefronts as the products themselves, 18 -> 21 TFLOP/s on F64 1681^3).
template <class A, int ROWS, int P, int BK, int NT>
__device__ __forceinline__ void simt_load(typename A::T* st, const SimtOperand<typename A::T>& o, const int64_t* koff,
                                          int kvalid, int tid) {
  using T = typename A::T;
  constexpr int R = ROWS * BK / NT;
  static_assert(ROWS * BK % NT == 0 && NT % ROWS == 0 && NT % BK == 0, "whole loads");
  if (o.rowfast) {
    const int row = tid % ROWS, k0 = tid / ROWS;
    constexpr int DK = NT / ROWS;
    const T* p = o.base + o.rowoff[row];
    const bool in = row < o.rows;
    if (o.uniform) {
      p += koff[k0];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int k = k0 + r * DK;
        if (in && k < kvalid) cp_elem(st + k * P + row, p + r * o.step);
        else st[k * P + row] = A::zero();
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int k = k0 + r * DK;
        if (in && k < kvalid) cp_elem(st + k * P + row, p + koff[k]);
        else st[k * P + row] = A::zero();
      }
    }
  } else {
    const int k = tid % BK, r0 = tid / BK;
    constexpr int DR = NT / BK;
    const T* p = o.base + koff[k];
    const bool in = k < kvalid;
    if (o.uniform) {
      p += o.rowoff[r0];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int row = r0 + r * DR;
        if (in && row < o.rows) cp_elem(st + k * P + row, p + r * o.step);
        else st[k * P + row] = A::zero();
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int row = r0 + r * DR;
        if (in && row < o.rows) cp_elem(st + k * P + row, p + o.rowoff[row]);
        else st[k * P + row] = A::zero();
      }
    }
  }
}
// Int64 stages of small values.  Every thread looks at the values that it
// brought into a stage (its own copies have landed) and writes their low bytes
// to `bytes` as words of four consecutive k ([k / 4][row]); returns whether
// they all lie in [-128, 127], so that those words stand for them.
template <int ROWS, int P, int BK, int NT>
__device__ __forceinline__ bool simt_bytes(const long long* st, unsigned char* bytes, int rowfast, int tid) {
  bool ok = true;
#pragma unroll
  for (int r = 0; r < ROWS * BK / NT; ++r) {
    const int row = rowfast ? tid % ROWS : tid / BK + r * (NT / BK);
    const int k = rowfast ? tid / ROWS + r * (NT / ROWS) : tid % BK;
    const long long v = st[k * P + row];
    ok = ok && (unsigned long long)(v + 128) < 256ull;
    bytes[((k >> 2) * ROWS + row) * 4 + (k & 3)] = (unsigned char)v;
  }
  return ok;
}
// The operand's description for tile rows from r0 (extent R, row group rg with
// strides rs, k strides ks).
template <class T, int ROWS, int BK, int NT>
__device__ __forceinline__ SimtOperand<T> simt_operand(const T* base, const int64_t* rowoff, int64_t left, int rowfast,
                                                       const SimtGroup& rg, const int64_t* rs, const SimtGroup& kg,
                                                       const int64_t* ks) {
  SimtOperand<T> o;
  o.base = base;
  o.rowoff = rowoff;
  o.rows = (int)min(left, (int64_t)ROWS);
  o.rowfast = rowfast;
  o.uniform = rowfast ? kg.n == 1 : rg.n == 1;
  o.step = rowfast ? ks[0] * (NT / ROWS) : rs[0] * (NT / BK);
  return o;
}

// C[m,n,l] = sx * sum_k A[m,k,l] B[k,n,l] (+ sy*C) over any algebra.  Bound by
// the algebra's instructions per multiply-add, then by shared-memory
// wavefronts: elements go to shared memory with cp.async through four stages,
// a thread holds TM x TN accumulators, and all offsets come from shared-memory
// tables filled once per tile (rows, columns) or stage (k).  Units are (tile,
// K split, batch).  Against 64 x 64 tiles that divided in 64 bits for every
// element: Int64 256 x 65536 x 256 2.15 ms -> 0.44 ms on values in [-128, 127]
// (four products per instruction) and 1.67 ms on others; max-plus
// 128 x 16384 x 32 0.93 ms -> 0.03 ms; ComplexF32 1024^3 307 -> 259 us.
template <class A, class C>
__global__ void __launch_bounds__(C::NT, C::MINB) k_gemm_simt(const __grid_constant__ SimtArgs g) {
  using T = typename A::T;
  using Mac = SimtMac<A>;
  constexpr int BM = C::BM, BN = C::BN, BK = C::BK, TM = C::TM, TN = C::TN, NT = C::NT, G = C::G, TX = C::TX;
  constexpr int PA = C::PA, PB = C::PB, ST = C::STAGES;
  constexpr bool I64 = std::is_same<A, AlgI64>::value;
  extern __shared__ __align__(16) unsigned char simt_raw[];
  int64_t* am = reinterpret_cast<int64_t*>(simt_raw);   // row offsets in A and C, column offsets in B and C
  int64_t* cm = am + BM;
  int64_t* bn = cm + BM;
  int64_t* cn = bn + BN;
  int64_t* kt = cn + BN;                                // [ST + 1][2][BK] k offsets in A and B
  T* sm = reinterpret_cast<T*>(kt + (ST + 1) * 2 * BK);
  unsigned char* bytes = reinterpret_cast<unsigned char*>(sm + ST * C::STAGE);   // Int64: [2] of A's, B's words
  const T* Ap = static_cast<const T*>(g.A);
  const T* Bp = static_cast<const T*>(g.B);
  T* Cp = static_cast<T*>(g.C);
  const T sx = scalar_as<T>(g.sx), sy = scalar_as<T>(g.sy);
  const int tid = threadIdx.x;
  const int tx = tid % TX, ty = tid / TX;
  griddep_launch_dependents();
  if (g.only_if.word) {
    griddep_wait();   // the kernels that set it
    if (!g.only_if.set()) return;
  }

  for (int64_t u = blockIdx.x; u < g.units; u += gridDim.x) {
    int64_t tm, tn, spi, l;
    simt_unit(g, u, tm, tn, spi, l);
    const int64_t m0 = tm * BM, n0 = tn * BN;
    const int64_t kbeg = spi * g.kchunk;
    const int64_t kend = min(g.K, kbeg + g.kchunk);
    const int nk = (int)((kend - kbeg + BK - 1) / BK);
    const T* Al = Ap + simt_off(l, g.l, g.l.s0, g.wide);
    const T* Bl = Bp + simt_off(l, g.l, g.l.s1, g.wide);
    for (int i = tid; i < BM; i += NT) {
      const bool in = m0 + i < g.M;
      am[i] = in ? simt_off(m0 + i, g.m, g.m.s0, g.wide) : -1;
      cm[i] = in ? simt_off(m0 + i, g.m, g.m.s1, g.wide) : -1;
    }
    for (int i = tid; i < BN; i += NT) {
      const bool in = n0 + i < g.N;
      bn[i] = in ? simt_off(n0 + i, g.n, g.n.s0, g.wide) : -1;
      cn[i] = in ? simt_off(n0 + i, g.n, g.n.s1, g.wide) : -1;
    }
    auto ktable = [&](int it, int t) {      // thread t of 2 * BK: the k offsets of stage `it`
      const int64_t k = kbeg + (int64_t)it * BK + (t % BK);
      if (k < kend) kt[(it % (ST + 1)) * 2 * BK + t] = simt_off(k, g.k, t < BK ? g.k.s0 : g.k.s1, g.wide);
    };
    for (int t = tid; t < ST * 2 * BK; t += NT) ktable(t / (2 * BK), t % (2 * BK));
    const SimtOperand<T> oa =
        simt_operand<T, BM, BK, NT>(Al, am, g.M - m0, g.a_rowfast, g.m, g.m.s0, g.k, g.k.s0);
    const SimtOperand<T> ob =
        simt_operand<T, BN, BK, NT>(Bl, bn, g.N - n0, g.b_rowfast, g.n, g.n.s0, g.k, g.k.s1);
    __syncthreads();
    auto issue = [&](int it) {
      if (it < nk) {
        T* st = sm + (it % ST) * C::STAGE;
        const int64_t* kq = kt + (it % (ST + 1)) * 2 * BK;
        const int kv = (int)min((int64_t)BK, kend - kbeg - (int64_t)it * BK);
        simt_load<A, BM, PA, BK, NT>(st, oa, kq, kv, tid);
        simt_load<A, BN, PB, BK, NT>(st + PA * BK, ob, kq + BK, kv, tid);
      }
      cp_commit();
    };
    typename Mac::Acc acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = Mac::init();
    // Int64: sums of the stages of small values
    int acc8[I64 ? TM : 1][I64 ? TN : 1] = {};
    int nsmall = 0;
    auto flush = [&]() {
      if constexpr (I64) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            acc[i][j].lo += (unsigned long long)(long long)acc8[i][j];
            acc8[i][j] = 0;
          }
      }
    };
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) issue(s);
    auto frag = [&](const T* st, int kk, T (&a)[TM], T (&b)[TN]) {
      lds_run(st + kk * PA + ty * TM, a);
      const T* bs = st + PA * BK + kk * PB + tx * G;
#pragma unroll
      for (int j = 0; j < TN / G; ++j) {
        T w[G];
        lds_run(bs + j * TX * G, w);
#pragma unroll
        for (int q = 0; q < G; ++q) b[j * G + q] = w[q];
      }
    };
    for (int it = 0; it < nk; ++it) {
      cp_wait<ST - 2>();
      const T* st = sm + (it % ST) * C::STAGE;
      bool small = false;
      unsigned char* sb = bytes + (it & 1) * (BM + BN) * BK;
      if constexpr (I64) {
        const bool own = simt_bytes<BM, PA, BK, NT>(st, sb, g.a_rowfast, tid);
        const bool own2 = simt_bytes<BN, PB, BK, NT>(st + PA * BK, sb + BM * BK, g.b_rowfast, tid);
        small = __syncthreads_and(own && own2);
      } else {
        __syncthreads();
      }
      issue(it + ST - 1);
      if (tid < 2 * BK) ktable(it + ST, tid);
      if constexpr (Mac::STEP == 2) {
#pragma unroll
        for (int kk = 0; kk < BK; kk += 2) {
          T a0[TM], b0[TN], a1[TM], b1[TN];
          frag(st, kk, a0, b0);
          frag(st, kk + 1, a1, b1);
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) Mac::mac2(acc[i][j], a0[i], b0[j], a1[i], b1[j]);
        }
      } else {
        if constexpr (I64) {
          if (small) {
            // four k per instruction, exact: |sum| <= 2^14 per k
            if (++nsmall == 16384 / BK * 4) {
              flush();
              nsmall = 1;
            }
#pragma unroll
            for (int q = 0; q < BK / 4; ++q) {
              int a4[TM], b4[TN];
              lds_run(reinterpret_cast<const int*>(sb) + q * BM + ty * TM, a4);
#pragma unroll
              for (int j = 0; j < TN; ++j)
                b4[j] = reinterpret_cast<const int*>(sb + BM * BK)[q * BN + (j / G) * TX * G + tx * G + j % G];
#pragma unroll
              for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc8[i][j] = __dp4a(a4[i], b4[j], acc8[i][j]);
            }
            continue;
          }
        }
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
          T a[TM], b[TN];
          frag(st, kk, a, b);
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) Mac::mac(acc[i][j], a[i], b[j]);
        }
      }
    }
    cp_wait<0>();
    if constexpr (I64) flush();
    const int64_t lc = simt_off(l, g.l, g.l_sc, g.wide);
    if (g.cluster) {
      __syncthreads();   // the stages are free
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j)
          sm[(ty * TM + i) * BN + (j / G) * TX * G + tx * G + j % G] = Mac::value(acc[i][j]);
      simt_cluster_finish<A, T, BM, BN, NT>(g, sm, cm, cn, lc, m0, n0, (int)spi, tid);
      return;
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int64_t m = m0 + ty * TM + i;
      if (m >= g.M) break;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int nj = (j / G) * TX * G + tx * G + j % G;
        const int64_t n = n0 + nj;
        if (n >= g.N) continue;
        const T v = Mac::value(acc[i][j]);
        if (g.S > 1) {
          const int64_t po = ((spi * g.L + l) * g.M + m) * g.N + n;
          if (po < g.p_elems) static_cast<T*>(g.partial)[po] = v;
          else atomicCAS(&g_ome_bounds_simt, 0, 5);
        } else {
          T* cp = Cp + lc + cm[ty * TM + i] + cn[nj];
          *cp = epilogue<A>(v, cp, sx, sy, g.sy_zero, g.sx_one);
        }
      }
    }
    __syncthreads();
  }
}

// Sum the S split partials of every output; αβ epilogue.  GR threads share an
// output (partial s goes to thread s mod GR, the GR sums are added in order),
// so that a few outputs with many partials do not become one serial chain.
template <class A, int GR>
__global__ void __launch_bounds__(256) k_simt_splitk_finish(const __grid_constant__ SimtArgs g) {
  using T = typename A::T;
  constexpr int OUT = 256 / GR;
  __shared__ T part[GR][OUT];
  griddep_wait();   // the partials of the GEMM
  if (g.only_if.word && !g.only_if.set()) return;
  const T* pp = static_cast<const T*>(g.partial);
  T* Cp = static_cast<T*>(g.C);
  const T sx = scalar_as<T>(g.sx), sy = scalar_as<T>(g.sy);
  const int64_t per = g.L * g.M * g.N;
  const int o = threadIdx.x % OUT, gr = threadIdx.x / OUT;
  for (int64_t i0 = (int64_t)blockIdx.x * OUT; i0 < per; i0 += (int64_t)gridDim.x * OUT) {
    const int64_t i = i0 + o;
    T acc = A::zero();
    if (i < per) {
#pragma unroll 8
      for (int s = gr; s < g.S; s += GR) acc = A::add(acc, pp[s * per + i]);
    }
    if constexpr (GR > 1) {
      part[gr][o] = acc;
      __syncthreads();
      if (gr == 0) {
#pragma unroll
        for (int q = 1; q < GR; ++q) acc = A::add(acc, part[q][o]);
      }
    }
    if (gr == 0 && i < per) {
      int64_t m, n, l;
      if (per < ((int64_t)1 << 32)) {
        const uint32_t nn = (uint32_t)g.N, mm = (uint32_t)g.M, r = (uint32_t)i / nn;
        n = (uint32_t)i - r * nn;
        l = r / mm;
        m = r - (uint32_t)l * mm;
      } else {
        const int64_t r = i / g.N;
        n = i - r * g.N;
        l = r / g.M;
        m = r - l * g.M;
      }
      T* cp = Cp + simt_off(l, g.l, g.l_sc, g.wide) + simt_off(m, g.m, g.m.s1, g.wide) +
              simt_off(n, g.n, g.n.s1, g.wide);
      *cp = epilogue<A>(acc, cp, sx, sy, g.sy_zero, g.sx_one);
    }
    if constexpr (GR > 1) __syncthreads();
  }
}

// Multiply-adds per clock and SM that each algebra's inner loop sustains
// (its instructions per multiply-add on the pipe that they use).
template <class A> struct SimtRate { static constexpr double v = 64; };            // F64, max-plus F32
template <> struct SimtRate<AlgF32> { static constexpr double v = 110; };
template <> struct SimtRate<AlgC32> { static constexpr double v = 28; };
template <> struct SimtRate<AlgC64> { static constexpr double v = 16; };
template <> struct SimtRate<AlgI64> { static constexpr double v = 15; };
template <> struct SimtRate<AlgBool> { static constexpr double v = 25; };
template <> struct SimtRate<AlgTF64> { static constexpr double v = 10; };

// Tile choice and K split, by an estimate in clocks: SMs work through
// ceil(units / SMs) tiles' multiply-adds at the algebra's rate times what
// the tile shape reaches of it, each round of resident blocks adds its
// start-up and epilogue latency, and a split adds its launch and the traffic
// of its partials.
struct SimtChoice {
  double clocks = 1e300;
  int cfg = 0;
  int64_t S = 1;
  bool cluster = false;
};

template <class A, class C>
static void simt_consider(SimtChoice& best, int cfg, double eff, int occ, double lat, const SimtArgs& g, int num_sms,
                          size_t ws_bytes) {
  const double tiles = (double)((g.M + C::BM - 1) / C::BM) * (double)((g.N + C::BN - 1) / C::BN) * (double)g.L;
  const double es = sizeof(typename A::T);
  const double out = (double)g.M * (double)g.N * (double)g.L;
  auto estimate = [&](int64_t S) {
    const int64_t kc = ((g.K + S - 1) / S + C::BK - 1) / C::BK * C::BK;
    const double units = tiles * (double)((g.K + kc - 1) / kc);
    const double per_sm = std::ceil(units / num_sms), rounds = std::ceil(units / ((double)num_sms * occ));
    // an SM with fewer resident blocks than `occ` does not reach the rate
    const double fill = std::min(1.0, 0.6 + 0.4 * std::min(per_sm, (double)occ) / occ);
    // a block's stages follow each other at no less than their latency (`lat`
    // clocks per k: the FP64 matrix instructions' dependent sums are the slower)
    const double work = per_sm * (double)kc * C::BM * C::BN / (SimtRate<A>::v * eff * fill);
    return std::max(work, rounds * (double)kc * lat) + rounds * 4000.0 + out * es / 3500.0;
  };
  const int64_t smax = std::min<int64_t>(128, std::max<int64_t>(1, g.K / 64));
  for (int64_t S = 1; S <= smax; S += S < 16 ? 1 : S / 8) {
    if (S > 1 && (double)S * out * es > (double)ws_bytes) break;
    const double clk = estimate(S) + (S > 1 ? 7000.0 + 2.0 * S * out * es / 3500.0 : 0.0);
    if (clk < best.clocks) best = SimtChoice{clk, cfg, S, false};
  }
  // two to eight splits as a cluster: no second launch, no partials in memory
  // (16 x 16 x 256 11.9 -> 7.1 us); with more than two blocks per SM the
  // clusters' placement costs more than that (300^3 in 8 splits 25 us, in 2 16)
  if (C::CLUSTER)
    for (int64_t S = 2; S <= 8 && S * C::BK <= g.K && tiles * S <= 2.0 * num_sms; S *= 2) {
      const double clk = estimate(S) + 2000.0;
      if (clk < best.clocks) best = SimtChoice{clk, cfg, S, true};
    }
}

// Tile counts and K split of a chosen configuration.
template <class C>
static void simt_plan(SimtArgs& g, const SimtChoice& ch, void* workspace) {
  const int64_t S = ch.S;
  g.cluster = ch.cluster;
  g.tiles_m = (g.M + C::BM - 1) / C::BM;
  g.tiles_n = (g.N + C::BN - 1) / C::BN;
  g.kchunk = S > 1 ? ((g.K + S - 1) / S + C::BK - 1) / C::BK * C::BK : g.K;
  // (a cluster keeps its size; its last splits may be empty)
  g.S = (int32_t)(ch.cluster ? S : S > 1 ? (g.K + g.kchunk - 1) / g.kchunk : 1);
  g.units = g.tiles_m * g.tiles_n * g.S * g.L;
  g.partial = workspace;
  g.p_elems = (int64_t)g.S * g.L * g.M * g.N;
}

template <class K>
static cudaError_t launch_simt_kernel(K* kernel, const SimtArgs& g, int threads, size_t smem, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min<int64_t>(g.units, 0x7fffffff));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  cfg.attrs = at;
  cfg.numAttrs = 0;
  if (g.cluster) {
    cudaLaunchAttribute& c = at[cfg.numAttrs++];
    c.id = cudaLaunchAttributeClusterDimension;
    c.val.clusterDim.x = (unsigned)g.S;
    c.val.clusterDim.y = c.val.clusterDim.z = 1;
  }
  if (g.only_if.word) {   // (it usually returns at once: its launch overlaps the kernel before)
    cudaLaunchAttribute& c = at[cfg.numAttrs++];
    c.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    c.val.programmaticStreamSerializationAllowed = 1;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, g);
  count_launch();
  return e;
}

template <class A>
static cudaError_t launch_simt_finish(const SimtArgs& g, int num_sms, cudaStream_t s) {
  const int64_t per = g.L * g.M * g.N;
  const bool shared = per < (int64_t)num_sms * 512 && g.S >= 8;
  const int64_t nb = std::min<int64_t>((per + 255) / 256 * (shared ? 8 : 1), (int64_t)num_sms * 16);
  cudaError_t e = shared ? launch_pdl(k_simt_splitk_finish<A, 8>, dim3((unsigned)nb), dim3(256), 0, s, g)
                         : launch_pdl(k_simt_splitk_finish<A, 1>, dim3((unsigned)nb), dim3(256), 0, s, g);
  count_launch();
  return e;
}

template <class A, class C>
static cudaError_t launch_simt_cfg(SimtArgs& g, const SimtChoice& ch, void* workspace, int num_sms, cudaStream_t s) {
  simt_plan<C>(g, ch, workspace);
  static std::atomic<unsigned long long> attr{0};
  cudaError_t e = set_smem_once(attr, k_gemm_simt<A, C>, (int)C::SMEM);
  if (e != cudaSuccess) return e;
  {
    KernelTimer kt(s, "k_gemm_simt");
    e = launch_simt_kernel(k_gemm_simt<A, C>, g, C::NT, C::SMEM, s);
  }
  return e != cudaSuccess || g.S == 1 || g.cluster ? e : launch_simt_finish<A>(g, num_sms, s);
}

// ---------------------------------------------------------------------------
// FP64 matrix instructions
// ---------------------------------------------------------------------------

// Tile configuration of k_gemm_dmma: WM x WN per warp; elements of type T are
// multiplied as W (double, or complex double).  With T = W the fragments are
// read from the stages; otherwise a stage is widened into one of two buffers.
template <class T, class W_, int BM_, int BN_, int WM_, int WN_, int BK_, int STAGES_, int MINB_>
struct DmmaTile {
  using W = W_;
  static constexpr bool WIDEN = !std::is_same<T, W>::value;
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, BK = BK_, STAGES = STAGES_, MINB = MINB_;
  static constexpr int NT = (BM / WM) * (BN / WN) * 32;
  static constexpr int PAD = 32 / (int)sizeof(W);     // fragment reads are conflict-free
  static constexpr int PA = BM + PAD, PB = BN + PAD;
  static constexpr int STAGE = (PA + PB) * BK;
  static constexpr size_t TABLES = (2 * BM + 2 * BN + (STAGES + 1) * 2 * BK) * sizeof(int64_t);
  static constexpr size_t SMEM = TABLES + (size_t)STAGES * STAGE * sizeof(T) +
                                 (WIDEN ? 2 * (size_t)STAGE * sizeof(W) : 0);
  static constexpr bool CLUSTER = BM * BN * sizeof(W) <= SMEM - TABLES;   // a tile fits the stages
};

// The elements that this thread brought into a stage, widened to double (its
// own copies have landed; the same places as simt_load's).
template <int ROWS, int P, int BK, int NT>
__device__ __forceinline__ void simt_widen(double* w, const float* st, int rowfast, int tid) {
#pragma unroll
  for (int r = 0; r < ROWS * BK / NT; ++r) {
    const int row = rowfast ? tid % ROWS : tid / BK + r * (NT / BK);
    const int k = rowfast ? tid / ROWS + r * (NT / ROWS) : tid % BK;
    w[k * P + row] = (double)st[k * P + row];
  }
}

// D += A B on a 16 x 4 by 4 x 8 block: lane (g, t) = (lane / 4, lane % 4) holds
// A(g, t), A(g + 8, t), B(t, g) and D(g, 2t), D(g, 2t + 1), D(g + 8, 2t), D(g + 8, 2t + 1).
__device__ __forceinline__ void dmma(double (&d)[4], const double (&a)[2], double b) {
  asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a[0]), "d"(a[1]), "d"(b));
}

// The same product in Float64 or ComplexF64 on the FP64 matrix instructions
// (four real products per complex one): a fragment serves eight lanes, so the
// shared-memory wavefronts per multiply-add are a third of k_gemm_simt's,
// which bound that one.  Float64 1681^3 (rows on 8-byte boundaries) 1200 ->
// 450 us, 21 TFLOP/s; 2368 x 2048 x 2048 25 TFLOP/s of the pipe's 37; the
// matrix pipe is 64% busy over the 1.6 waves of 1681^3, the rest is their last
// part and the fixed wait between dependent issues with at most 12 warps on an
// SM.
template <class A, class C>
__global__ void __launch_bounds__(C::NT, C::MINB) k_gemm_dmma(const __grid_constant__ SimtArgs g) {
  using T = typename A::T;
  using W = typename C::W;
  constexpr bool CPLX = sizeof(W) == 16;
  constexpr int P = CPLX ? 2 : 1;                   // real accumulators per output
  constexpr int BM = C::BM, BN = C::BN, BK = C::BK, NT = C::NT, ST = C::STAGES;
  constexpr int PA = C::PA, PB = C::PB, MI = C::WM / 16, NI = C::WN / 8;
  extern __shared__ __align__(16) unsigned char simt_raw[];
  int64_t* am = reinterpret_cast<int64_t*>(simt_raw);
  int64_t* cm = am + BM;
  int64_t* bn = cm + BM;
  int64_t* cn = bn + BN;
  int64_t* kt = cn + BN;
  T* sm = reinterpret_cast<T*>(kt + (ST + 1) * 2 * BK);
  W* wide = reinterpret_cast<W*>(sm + ST * C::STAGE);   // widened stages [2]
  const T* Ap = static_cast<const T*>(g.A);
  const T* Bp = static_cast<const T*>(g.B);
  T* Cp = static_cast<T*>(g.C);
  const T sx = scalar_as<T>(g.sx), sy = scalar_as<T>(g.sy);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp % (BM / C::WM) * C::WM, wn = warp / (BM / C::WM) * C::WN;
  const int gg = lane >> 2, tt = lane & 3;
  griddep_launch_dependents();

  for (int64_t u = blockIdx.x; u < g.units; u += gridDim.x) {
    int64_t tm, tn, spi, l;
    simt_unit(g, u, tm, tn, spi, l);
    const int64_t m0 = tm * BM, n0 = tn * BN;
    const int64_t kbeg = spi * g.kchunk;
    const int64_t kend = min(g.K, kbeg + g.kchunk);
    const int nk = (int)((kend - kbeg + BK - 1) / BK);
    const T* Al = Ap + simt_off(l, g.l, g.l.s0, g.wide);
    const T* Bl = Bp + simt_off(l, g.l, g.l.s1, g.wide);
    for (int i = tid; i < BM; i += NT) {
      const bool in = m0 + i < g.M;
      am[i] = in ? simt_off(m0 + i, g.m, g.m.s0, g.wide) : -1;
      cm[i] = in ? simt_off(m0 + i, g.m, g.m.s1, g.wide) : -1;
    }
    for (int i = tid; i < BN; i += NT) {
      const bool in = n0 + i < g.N;
      bn[i] = in ? simt_off(n0 + i, g.n, g.n.s0, g.wide) : -1;
      cn[i] = in ? simt_off(n0 + i, g.n, g.n.s1, g.wide) : -1;
    }
    auto ktable = [&](int it, int t) {
      const int64_t k = kbeg + (int64_t)it * BK + (t % BK);
      if (k < kend) kt[(it % (ST + 1)) * 2 * BK + t] = simt_off(k, g.k, t < BK ? g.k.s0 : g.k.s1, g.wide);
    };
    for (int t = tid; t < ST * 2 * BK; t += NT) ktable(t / (2 * BK), t % (2 * BK));
    const SimtOperand<T> oa =
        simt_operand<T, BM, BK, NT>(Al, am, g.M - m0, g.a_rowfast, g.m, g.m.s0, g.k, g.k.s0);
    const SimtOperand<T> ob =
        simt_operand<T, BN, BK, NT>(Bl, bn, g.N - n0, g.b_rowfast, g.n, g.n.s0, g.k, g.k.s1);
    __syncthreads();
    auto issue = [&](int it) {
      if (it < nk) {
        T* st = sm + (it % ST) * C::STAGE;
        const int64_t* kq = kt + (it % (ST + 1)) * 2 * BK;
        const int kv = (int)min((int64_t)BK, kend - kbeg - (int64_t)it * BK);
        simt_load<A, BM, PA, BK, NT>(st, oa, kq, kv, tid);
        simt_load<A, BN, PB, BK, NT>(st + PA * BK, ob, kq + BK, kv, tid);
      }
      cp_commit();
    };
    double acc[MI][NI][P][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j)
#pragma unroll
        for (int p = 0; p < P; ++p)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[i][j][p][q] = 0.0;
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) issue(s);
    for (int it = 0; it < nk; ++it) {
      cp_wait<ST - 2>();
      const W* ws;
      if constexpr (C::WIDEN) {
        W* wd = wide + (it & 1) * C::STAGE;
        const T* st = sm + (it % ST) * C::STAGE;
        simt_widen<BM, PA, BK, NT>(wd, st, g.a_rowfast, tid);
        simt_widen<BN, PB, BK, NT>(wd + PA * BK, st + PA * BK, g.b_rowfast, tid);
        ws = wd;
      } else {
        ws = sm + (it % ST) * C::STAGE;
      }
      __syncthreads();
      issue(it + ST - 1);
      if (tid < 2 * BK) ktable(it + ST, tid);
      const W* as = ws + tt * PA + wm + gg;
      const W* bs = ws + PA * BK + tt * PB + wn + gg;
#pragma unroll
      for (int kk = 0; kk < BK; kk += 4) {
        if constexpr (!CPLX) {
          double a[MI][2], b[NI];
#pragma unroll
          for (int i = 0; i < MI; ++i) {
            a[i][0] = as[kk * PA + 16 * i];
            a[i][1] = as[kk * PA + 16 * i + 8];
          }
#pragma unroll
          for (int j = 0; j < NI; ++j) b[j] = bs[kk * PB + 8 * j];
#pragma unroll
          for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NI; ++j) dmma(acc[i][j][0], a[i], b[j]);
        } else {
          // (re, im): re += ar br - ai bi, im += ar bi + ai br
          double ar[MI][2], ai[MI][2], br[NI], bi[NI];
#pragma unroll
          for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const double2 v = *reinterpret_cast<const double2*>(as + kk * PA + 16 * i + 8 * h);
              ar[i][h] = v.x;
              ai[i][h] = v.y;
            }
#pragma unroll
          for (int j = 0; j < NI; ++j) {
            const double2 v = *reinterpret_cast<const double2*>(bs + kk * PB + 8 * j);
            br[j] = v.x;
            bi[j] = v.y;
          }
#pragma unroll
          for (int i = 0; i < MI; ++i) {
#pragma unroll
            for (int j = 0; j < NI; ++j) {
              dmma(acc[i][j][0], ar[i], br[j]);
              dmma(acc[i][j][1], ar[i], bi[j]);
              dmma(acc[i][j][1], ai[i], br[j]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) ai[i][h] = -ai[i][h];
#pragma unroll
            for (int j = 0; j < NI; ++j) dmma(acc[i][j][0], ai[i], bi[j]);
          }
        }
      }
    }
    cp_wait<0>();
    const int64_t lc = simt_off(l, g.l, g.l_sc, g.wide);
    if (g.cluster) {
      __syncthreads();   // the stages are free
      W* tile = reinterpret_cast<W*>(sm);
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            W& t = tile[(wm + 16 * i + 8 * (q >> 1) + gg) * BN + wn + 8 * j + 2 * tt + (q & 1)];
            if constexpr (CPLX) t = W{acc[i][j][0][q], acc[i][j][P - 1][q]};
            else t = acc[i][j][0][q];
          }
      simt_cluster_finish<A, W, BM, BN, NT>(g, tile, cm, cn, lc, m0, n0, (int)spi, tid);
      return;
    }
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int mi = wm + 16 * i + 8 * h + gg;
        const int64_t m = m0 + mi;
        if (m >= g.M) continue;
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int nj = wn + 8 * j + 2 * tt + q;
            const int64_t n = n0 + nj;
            if (n >= g.N) continue;
            T v;
            if constexpr (CPLX) v = T{acc[i][j][0][2 * h + q], acc[i][j][P - 1][2 * h + q]};
            else v = (T)acc[i][j][0][2 * h + q];
            if (g.S > 1) {
              const int64_t po = ((spi * g.L + l) * g.M + m) * g.N + n;
              if (po < g.p_elems) static_cast<T*>(g.partial)[po] = v;
              else atomicCAS(&g_ome_bounds_simt, 0, 5);
            } else {
              T* cp = Cp + lc + cm[mi] + cn[nj];
              *cp = epilogue<A>(v, cp, sx, sy, g.sy_zero, g.sx_one);
            }
          }
      }
    __syncthreads();
  }
}

template <class A, class C>
static cudaError_t launch_dmma_cfg(SimtArgs& g, const SimtChoice& ch, void* workspace, int num_sms, cudaStream_t s) {
  simt_plan<C>(g, ch, workspace);
  static std::atomic<unsigned long long> attr{0};
  cudaError_t e = set_smem_once(attr, k_gemm_dmma<A, C>, (int)C::SMEM);
  if (e != cudaSuccess) return e;
  {
    KernelTimer kt(s, "k_gemm_dmma");
    e = launch_simt_kernel(k_gemm_dmma<A, C>, g, C::NT, C::SMEM, s);
  }
  return e != cudaSuccess || g.S == 1 || g.cluster ? e : launch_simt_finish<A>(g, num_sms, s);
}

static void simt_group(SimtGroup& o, int n, const int64_t* ext, const int64_t* s0, const int64_t* s1, int wide) {
  o.n = n;
  for (int i = 0; i < n; ++i) {
    o.div[i] = wide ? FastDiv{(uint32_t)ext[i], (uint32_t)(ext[i] >> 32), 0} : make_fastdiv((uint32_t)ext[i]);
    o.s0[i] = s0[i];
    o.s1[i] = s1[i];
  }
}

// k_gemm_simt's / k_gemm_dmma's arguments from a contraction.
static void simt_args(SimtArgs& g, const GemmArgs& q) {
  const int64_t lim = (int64_t)1 << 31;
  g.wide = q.M >= lim || q.N >= lim || q.K >= lim || q.L >= lim;
  g.C = q.C;
  g.K = q.K;
  g.L = q.L;
  // the tile's columns run along C's contiguous mode (coalesced stores): the
  // operands change places when that mode is among A's rows
  const bool swap = q.m_sc[0] == 1 || (q.n_sc[0] != 1 && std::llabs(q.m_sc[0]) < std::llabs(q.n_sc[0]));
  if (!swap) {
    g.A = q.A; g.B = q.B; g.M = q.M; g.N = q.N;
    simt_group(g.m, q.nm, q.m_ext, q.m_sa, q.m_sc, g.wide);
    simt_group(g.n, q.nn, q.n_ext, q.n_sb, q.n_sc, g.wide);
    simt_group(g.k, q.nk, q.k_ext, q.k_sa, q.k_sb, g.wide);
    simt_group(g.l, q.nl, q.l_ext, q.l_sa, q.l_sb, g.wide);
    g.a_rowfast = q.a_m_fast; g.b_rowfast = q.b_n_fast;
  } else {
    g.A = q.B; g.B = q.A; g.M = q.N; g.N = q.M;
    simt_group(g.m, q.nn, q.n_ext, q.n_sb, q.n_sc, g.wide);
    simt_group(g.n, q.nm, q.m_ext, q.m_sa, q.m_sc, g.wide);
    simt_group(g.k, q.nk, q.k_ext, q.k_sb, q.k_sa, g.wide);
    simt_group(g.l, q.nl, q.l_ext, q.l_sb, q.l_sa, g.wide);
    g.a_rowfast = q.b_n_fast; g.b_rowfast = q.a_m_fast;
  }
  for (int i = 0; i < q.nl; ++i) g.l_sc[i] = q.l_sc[i];
  g.sx = q.sx;
  g.sy = q.sy;
  g.sy_zero = q.sy_zero;
  g.sx_one = q.sx_one;
  g.only_if = RangeFlag{nullptr, 0};
}

// CUDA-core GEMM: tile shape and K split by the estimate above; split
// partials go to `workspace`.
template <class A>
static cudaError_t launch_gemm_simt_ws_t(const GemmArgs& q, void* workspace, size_t ws_bytes, int num_sms,
                                         cudaStream_t s, const RangeFlag* only_if) {
  using T = typename A::T;
  if (q.M == 0 || q.N == 0 || q.L == 0) return cudaSuccess;
  SimtArgs g;
  simt_args(g, q);
  if (only_if) g.only_if = *only_if;
  SimtChoice best;
  if constexpr (std::is_same<A, AlgF64>::value || std::is_same<A, AlgC64>::value) {
    // FP64 matrix instructions once both sides fill a few of their tiles: the
    // CUDA-core tiles reach 15.5 TFLOP/s on F64 1681^3, these 21.5 (24.8 on
    // 2368 x 2048 x 2048); below, the smaller CUDA-core tiles waste less
    if (g.M >= 128 && g.N >= 128) {
      constexpr bool Z = std::is_same<A, AlgC64>::value;
      using D1 = DmmaTile<T, T, 64, 64, 32, 32, Z ? 8 : 16, Z ? 3 : 4, Z ? 2 : 3>;
      using D2 = DmmaTile<T, T, 128, 64, Z ? 32 : 64, 32, Z ? 8 : 16, Z ? 3 : 4, Z ? 1 : 2>;
      simt_consider<A, D1>(best, 1, 0.8, Z ? 2 : 3, Z ? 500 : 200, g, num_sms, ws_bytes);
      simt_consider<A, D2>(best, 2, 0.9, 1, Z ? 500 : 300, g, num_sms, ws_bytes);
      if (best.cfg == 1) return launch_dmma_cfg<A, D1>(g, best, workspace, num_sms, s);
      if (best.cfg == 2) return launch_dmma_cfg<A, D2>(g, best, workspace, num_sms, s);
    }
  }
  using T1 = SimtTile<T, 32, 32, 4, 2, 16, 4>;
  using T2 = SimtTile<T, 64, 64, 4, 4, 16, sizeof(T) >= 16 ? 1 : 2>;
  simt_consider<A, T1>(best, 1, 0.35, 8, 40, g, num_sms, ws_bytes);
  simt_consider<A, T2>(best, 2, 0.7, sizeof(T) >= 16 ? 1 : 2, 40, g, num_sms, ws_bytes);
  if constexpr (sizeof(T) >= 16) {
    if (best.cfg == 1) return launch_simt_cfg<A, T1>(g, best, workspace, num_sms, s);
    return launch_simt_cfg<A, T2>(g, best, workspace, num_sms, s);
  } else {
    // 8 x 8 per thread where the accumulators fit 255 registers (Int64's are 12
    // bytes, the Float64 maximum keeps temporaries)
    constexpr int TN3 = std::is_same<A, AlgI64>::value || std::is_same<A, AlgTF64>::value ? 4 : 8;
    using T3 = SimtTile<T, 128, 16 * TN3, 8, TN3, 8, sizeof(T) <= 4 ? 2 : 1>;
    simt_consider<A, T3>(best, 3, 0.9, sizeof(T) <= 4 ? 2 : 1, 80, g, num_sms, ws_bytes);
    if (best.cfg == 1) return launch_simt_cfg<A, T1>(g, best, workspace, num_sms, s);
    if (best.cfg == 2) return launch_simt_cfg<A, T2>(g, best, workspace, num_sms, s);
    return launch_simt_cfg<A, T3>(g, best, workspace, num_sms, s);
  }
}

// Batched GEMM whose batch mode is the contiguous one in A, B and C (Julia
// column-major `bij,bjk->bik`: b fastest) with small M, N (<= 64).  A CTA of
// 256 threads owns 4 consecutive batches and an NS-column slab of N (64:
// all of it, for 4-byte types with N > 32; otherwise 32); K runs in chunks of 16 staged in shared memory
// (two buffers, the next chunk's global loads in registers while the current
// one is multiplied).  Staging loads walk the batch mode fastest (4 batches =
// 16 contiguous bytes for 4-byte types), so each element of A and B leaves
// L2 once per slab instead of once per register tile; each thread keeps
// 8 x NS/8 accumulators of one batch and reads its operands from shared
// memory as 16-byte broadcasts (B in runs of 4 columns, conflict-free).  The tile leaves through shared memory too,
// batch mode fastest.  Plain algebra arithmetic in K order.
template <int NS_> struct BsCfg {
  static constexpr int NB = 4, KC = 16, NS = NS_, MT = 64, NT = 256;
  static constexpr int TR = 8, TC = NS / 8;          // thread tile: rows x columns
  static constexpr int KSTEP = 64 / NS;              // B staging: k rows lk0, lk0 + KSTEP, ...
  // every offset the compute reads (8*tm, 4*tn, 32, the strides below) is a
  // multiple of 4 elements, so its runs are 16-byte aligned for 4-byte and
  // wider types
  static constexpr int A_B = KC * MT + 8;            // elements per batch in an A stage (padded)
  static constexpr int B_B = KC * NS + 8;            // elements per batch in a B stage
  static constexpr int STAGE = NB * (A_B + B_B);
  static constexpr int C_ROW = MT + 1;               // epilogue tile: [batch][n][m], padded rows
  static constexpr int C_B = NS * C_ROW + 8;
  static constexpr int ELEMS = 2 * STAGE > NB * C_B ? 2 * STAGE : NB * C_B;
};

template <class A, bool FULL, int NS_>
__global__ void __launch_bounds__(256, 1) k_gemm_bstage(const __grid_constant__ GemmArgs g) {
  using Cf = BsCfg<NS_>;
  constexpr int NB = Cf::NB, KC = Cf::KC, NS = Cf::NS, MT = Cf::MT, TR = Cf::TR, TC = Cf::TC;
  constexpr int KSTEP = Cf::KSTEP, A_B = Cf::A_B, B_B = Cf::B_B, STAGE = Cf::STAGE, C_ROW = Cf::C_ROW,
                C_B = Cf::C_B;
  using T = typename A::T;
  extern __shared__ __align__(16) unsigned char bs_raw[];
  T* sm = reinterpret_cast<T*>(bs_raw);
  const int t = threadIdx.x;
  const int64_t b0 = (int64_t)blockIdx.x * NB;
  const int n0 = blockIdx.y * NS;
  const int M = (int)g.M, N = (int)g.N, K = (int)g.K;
  const int sma = (int)g.m_sa[0], ska = (int)g.k_sa[0], snb = (int)g.n_sb[0], skb = (int)g.k_sb[0];
  // staging roles: batch lb of the group; A row lm (all 16 k of a chunk);
  // B column ln, k rows lk0 + KSTEP*q
  const int lb = t & 3, lm = t >> 2, ln = (t >> 2) % NS, lk0 = (t >> 2) / NS;
  const bool bok = FULL || b0 + lb < g.L;
  const T* ga = static_cast<const T*>(g.A);
  const T* gb = static_cast<const T*>(g.B);
  if (bok) {
    ga += mode_offset(b0 + lb, g.nl, g.l_ext, g.l_sa) + (int64_t)lm * sma;
    gb += mode_offset(b0 + lb, g.nl, g.l_ext, g.l_sb) + (int64_t)(n0 + ln) * snb + (int64_t)lk0 * skb;
  }
  const bool aok = bok && (FULL || lm < M), bnok = bok && (FULL || n0 + ln < N);
  T ra[KC], rb[KC / KSTEP];
  auto load = [&](int k0) {
#pragma unroll
    for (int q = 0; q < KC; ++q)
      ra[q] = aok && (FULL || k0 + q < K) ? ga[(int64_t)(k0 + q) * ska] : A::zero();
#pragma unroll
    for (int q = 0; q < KC / KSTEP; ++q)
      rb[q] = bnok && (FULL || k0 + lk0 + KSTEP * q < K) ? gb[(int64_t)(k0 + KSTEP * q) * skb] : A::zero();
  };
  auto store = [&](int st) {
    T* as = sm + st * STAGE + lb * A_B + lm;
    T* bsm = sm + st * STAGE + NB * A_B + lb * B_B + lk0 * NS + ln;
#pragma unroll
    for (int q = 0; q < KC; ++q) as[q * MT] = ra[q];
#pragma unroll
    for (int q = 0; q < KC / KSTEP; ++q) bsm[KSTEP * q * NS] = rb[q];
  };
  // 16-byte types (complex128) stage straight from global memory after the
  // multiply: the accumulators leave no registers for a prefetch
  constexpr bool PREF = sizeof(T) < 16;
  auto load_store = [&](int k0, int st) {
    T* as = sm + st * STAGE + lb * A_B + lm;
    T* bsm = sm + st * STAGE + NB * A_B + lb * B_B + lk0 * NS + ln;
#pragma unroll 4
    for (int q = 0; q < KC; ++q)
      as[q * MT] = aok && (FULL || k0 + q < K) ? ga[(int64_t)(k0 + q) * ska] : A::zero();
#pragma unroll 4
    for (int q = 0; q < KC / KSTEP; ++q)
      bsm[KSTEP * q * NS] =
          bnok && (FULL || k0 + lk0 + KSTEP * q < K) ? gb[(int64_t)(k0 + KSTEP * q) * skb] : A::zero();
  };
  // compute roles: batch cb, rows TR*tm.., columns 4*tn.. (and 32 + 4*tn..
  // for 8-column tiles: a warp's 16-byte reads of B stay in one 128-byte row
  // of banks)
  const int cb = t >> 6, tm = (t >> 3) & 7, tn = t & 7;
  T acc[TR][TC];
#pragma unroll
  for (int r = 0; r < TR; ++r)
#pragma unroll
    for (int c = 0; c < TC; ++c) acc[r][c] = A::zero();
  const int nchunks = (K + KC - 1) / KC;
  if (PREF) {
    load(0);
    store(0);
  } else {
    load_store(0, 0);
  }
  __syncthreads();
  for (int ch = 0; ch < nchunks; ++ch) {
    const int st = ch & 1;
    if (PREF && ch + 1 < nchunks) load((ch + 1) * KC);
    const T* as = sm + st * STAGE + cb * A_B + TR * tm;
    const T* bsm = sm + st * STAGE + NB * A_B + cb * B_B + 4 * tn;
#pragma unroll 2
    for (int kk = 0; kk < KC; ++kk) {
      T av[TR], bv[TC];
      lds_run(as + kk * MT, av);
#pragma unroll
      for (int h = 0; h < TC / 4; ++h) {
        T b4[4];
        lds_run(bsm + kk * NS + 32 * h, b4);
#pragma unroll
        for (int c = 0; c < 4; ++c) bv[4 * h + c] = b4[c];
      }
#pragma unroll
      for (int r = 0; r < TR; ++r)
#pragma unroll
        for (int c = 0; c < TC; ++c) acc[r][c] = A::add(acc[r][c], A::mul(av[r], bv[c]));
    }
    if (ch + 1 < nchunks) {
      if (PREF) store(st ^ 1);
      else load_store((ch + 1) * KC, st ^ 1);
    }
    __syncthreads();
  }
  // tile -> shared [batch][n][m] -> C with the batch mode fastest
  {
    T* cs = sm + cb * C_B + (4 * tn) * C_ROW + TR * tm;
#pragma unroll
    for (int c = 0; c < TC; ++c)
#pragma unroll
      for (int r = 0; r < TR; ++r) cs[((c >> 2) * 32 + (c & 3)) * C_ROW + r] = acc[r][c];
  }
  __syncthreads();
  if (!bok || !(FULL || lm < M)) return;
  const T sx = scalar_as<T>(g.sx), sy = scalar_as<T>(g.sy);
  T* cp = static_cast<T*>(g.C) + mode_offset(b0 + lb, g.nl, g.l_ext, g.l_sc) + (int64_t)lm * g.m_sc[0] +
          (int64_t)n0 * g.n_sc[0];
  const T* cs = sm + lb * C_B + lm;
  const int nn = FULL ? NS : min(NS, N - n0);
  for (int q = 0; q < nn; ++q) {
    T* yp = cp + (int64_t)q * g.n_sc[0];
    *yp = epilogue<A>(cs[q * C_ROW], yp, sx, sy, g.sy_zero, g.sx_one);
  }
}

bool gemm_bfast_applies(const GemmArgs& g) {
  auto small = [](int64_t ext, int64_t str) { return ext * (str < 0 ? -str : str) < ((int64_t)1 << 30); };
  return g.l_sa[0] == 1 && g.l_sb[0] == 1 && g.l_sc[0] == 1 && g.l_ext[0] >= 32 && g.M <= 64 && g.N <= 64 &&
         g.K <= 1024 && g.L >= 32 && (g.L + 31) / 32 <= 0x7fffffff && g.nm == 1 && g.nn == 1 && g.nk == 1 &&
         small(g.M, g.m_sa[0]) && small(g.M, g.m_sc[0]) && small(g.N, g.n_sb[0]) && small(g.N, g.n_sc[0]) &&
         small(g.K, g.k_sa[0]) && small(g.K, g.k_sb[0]);
}

template <class A, int NS>
static cudaError_t launch_gemm_bstage_t(const GemmArgs& g, cudaStream_t s) {
  using Cf = BsCfg<NS>;
  const size_t smem = (size_t)Cf::ELEMS * sizeof(typename A::T);
  static std::atomic<unsigned long long> attr_full{0}, attr_part{0};
  cudaError_t e = set_smem_once(attr_full, k_gemm_bstage<A, true, NS>, (int)smem);
  if (e == cudaSuccess) e = set_smem_once(attr_part, k_gemm_bstage<A, false, NS>, (int)smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((unsigned)((g.L + Cf::NB - 1) / Cf::NB), (unsigned)((g.N + NS - 1) / NS));
  const bool full = g.M == Cf::MT && g.N % NS == 0 && g.K % Cf::KC == 0 && g.L % Cf::NB == 0;
  if (full) k_gemm_bstage<A, true, NS><<<grid, Cf::NT, smem, s>>>(g);
  else k_gemm_bstage<A, false, NS><<<grid, Cf::NT, smem, s>>>(g);
  count_launch();
  return cudaGetLastError();
}

// 64-column slabs (8 x 8 thread tiles) for types of at most 4 bytes; wider
// types keep 8 x 4 tiles, whose accumulators already fill the registers
template <class A>
static cudaError_t launch_gemm_bstage(const GemmArgs& g, cudaStream_t s) {
  if constexpr (sizeof(typename A::T) <= 4) {
    if (g.N > 32) return launch_gemm_bstage_t<A, 64>(g, s);
  }
  return launch_gemm_bstage_t<A, 32>(g, s);
}

cudaError_t launch_gemm_bfast(ome_dtype dt, const GemmArgs& g, cudaStream_t s) {
  if (g.M == 0 || g.N == 0 || g.L == 0) return cudaSuccess;
  if (!gemm_bfast_applies(g)) return cudaErrorNotSupported;
  cudaError_t e = cudaErrorInvalidValue;
  KernelTimer kt(s, "k_gemm_bstage");
  OME_DISPATCH(dt, ALG, e = launch_gemm_bstage<ALG>(g, s));
  return e;
}

// Read and clear the split-partial self-check flag (0 = no violation).
int simt_bounds_flag() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_ome_bounds_simt, sizeof(int)) != cudaSuccess) return 0;
  if (v) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_ome_bounds_simt, &zero, sizeof(int));
  }
  return v;
}

cudaError_t launch_gemm_small_f32(const GemmArgs& q, void* workspace, size_t ws_bytes, int num_sms, cudaStream_t s) {
  if (q.M == 0 || q.N == 0 || q.L == 0) return cudaSuccess;
  SimtArgs g;
  simt_args(g, q);
  using E1 = DmmaTile<float, double, 32, 32, 16, 16, 32, 3, 4>;
  using E2 = DmmaTile<float, double, 64, 64, 32, 32, 16, 4, 3>;
  SimtChoice best;
  simt_consider<AlgF64, E1>(best, 1, 0.4, 4, 85, g, num_sms, ws_bytes);
  simt_consider<AlgF64, E2>(best, 2, 0.6, 3, 200, g, num_sms, ws_bytes);
  if (best.cfg == 1) return launch_dmma_cfg<AlgF32, E1>(g, best, workspace, num_sms, s);
  return launch_dmma_cfg<AlgF32, E2>(g, best, workspace, num_sms, s);
}

cudaError_t launch_gemm_simt_ws(ome_dtype dt, const GemmArgs& g, void* workspace, size_t ws_bytes, int num_sms,
                                cudaStream_t s, const RangeFlag* only_if) {
  cudaError_t e = cudaErrorInvalidValue;
  OME_DISPATCH(dt, ALG, e = launch_gemm_simt_ws_t<ALG>(g, workspace, ws_bytes, num_sms, s, only_if));
  return e;
}

}  // namespace ome
