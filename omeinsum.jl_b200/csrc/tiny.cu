// Programs of small contractions: the leaves' side of a contraction tree in
// one launch.
//
// Most nodes of a tensor network's tree are tiny (of the 99 contractions of a
// 3-regular bond-2 network with 100 vertices 91 take at most 2^14
// multiply-adds, 45 of them 32), and one launch each costs 2-3 us on the
// device and 5 us on the host for nanoseconds of work.  Here one cluster of
// sixteen blocks walks the nodes level by level (src/einsequence.jl:270-287
// evaluates the same nodes in post-order): the nodes of a level are spread
// over the cluster's warps, and a cluster barrier orders a level's results
// before the next level's reads.  The descriptors travel as kernel arguments.
// Bound by latency: about 2 us per level, ten levels for that network.
#include <cooperative_groups.h>
#include <string.h>
#include <type_traits>

#include "dispatch.h"

namespace ome {

namespace {

constexpr int TINY_CTAS = 16, TINY_THREADS = 512, TINY_LEVELS = 64;

template <int CAP>
struct TinyArgs {
  int32_t nlevels;
  uint16_t begin[TINY_LEVELS + 1];   // first node of each level
  uint32_t items[TINY_LEVELS];       // warp items of each level
  TinyNode nodes[CAP];
};
// 100 nodes are 30.8 KB of the 32764 bytes a launch's arguments may have
constexpr int TINY_CAP = 100, TINY_CAP_SMALL = 12;
static_assert(sizeof(TinyArgs<TINY_CAP>) <= 32764, "kernel arguments");

// Sums run in the type W: Float64 for Float32 elements, the element type
// otherwise.  A result is kept in W too, for the nodes of the program that read
// it: in a network of 160 vertices the roundings of the 144 small nodes to
// Float32 were most of the value's error.
template <class A> struct TinyWide { using W = A; };
template <> struct TinyWide<AlgF32> { using W = AlgF64; };
template <> struct TinyWide<AlgC32> { using W = AlgC64; };

template <class U, class T>
__device__ __forceinline__ U tiny_as(T v) {
  if constexpr (std::is_same<U, T>::value) return v;
  else if constexpr (std::is_arithmetic<T>::value) return (U)v;
  else return U{(decltype(U::re))v.re, (decltype(U::re))v.im};
}
template <class T>
__device__ __forceinline__ T tiny_conj(T v, bool yes) {
  if constexpr (!std::is_arithmetic<T>::value) {
    if (yes) v.im = -v.im;
  }
  return v;
}
// Values written by other blocks of the cluster: past the L1 cache.
template <class T>
__device__ __forceinline__ T tiny_ld(const T* p) {
  if constexpr (sizeof(T) == 16) {
    const float4 w = __ldcg(reinterpret_cast<const float4*>(p));
    T v;
    memcpy(&v, &w, 16);
    return v;
  } else if constexpr (sizeof(T) == 8) {
    const double w = __ldcg(reinterpret_cast<const double*>(p));
    T v;
    memcpy(&v, &w, 8);
    return v;
  } else {
    return __ldcg(p);
  }
}

// The lowest digit of r in a mixed radix whose first extent is `ext`; r is
// divided by it.
__device__ __forceinline__ int32_t tiny_digit(uint32_t& r, uint32_t ext) {
  const uint32_t e = ext & 0xffffff, sh = ext >> 24;
  const uint32_t q = sh < 31 ? r >> sh : r / e;
  const int32_t d = (int32_t)(r - q * e);
  r = q;
  return d;
}

template <class A, class WA, int CAP>
__global__ void __launch_bounds__(TINY_THREADS, 1) k_tiny(const __grid_constant__ TinyArgs<CAP> a) {
  using T = typename A::T;
  using W = typename WA::T;
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int lane = threadIdx.x & 31;
  const uint32_t warp = blockIdx.x * (TINY_THREADS / 32) + (threadIdx.x >> 5);
  for (int lev = 0; lev < a.nlevels; ++lev) {
    const int nb = a.begin[lev], ne = a.begin[lev + 1];
    for (uint32_t it = warp; it < a.items[lev]; it += TINY_CTAS * (TINY_THREADS / 32)) {
      int lo = nb, hi = ne - 1;   // the item's node
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (a.nodes[mid].item0 <= it) lo = mid;
        else hi = mid - 1;
      }
      const TinyNode& n = a.nodes[lo];
      const bool by_warp = n.flags & TINY_WARP;   // a warp per output, else a thread
      const uint32_t o = by_warp ? it - n.item0 : (it - n.item0) * 32 + lane;
      const bool in = o < n.n_out;
      int32_t yo = 0, o0 = 0, o1 = 0;
      uint32_t r = in ? o : 0;
      for (int m = 0; m < n.nout; ++m) {
        const TinyMode md = n.mode[m];
        const int32_t d = tiny_digit(r, md.ext);
        yo += d * md.sy;
        o0 += d * md.s0;
        o1 += d * md.s1;
      }
      constexpr bool WIDE = !std::is_same<T, W>::value;
      const bool w0 = WIDE && (n.flags & TINY_WIDE0), w1 = WIDE && (n.flags & TINY_WIDE1);
      const T* x0 = static_cast<const T*>(n.x0) + (w0 ? 0 : o0);
      const T* x1 = static_cast<const T*>(n.x1) + (w1 ? 0 : o1);
      const W* x0w = static_cast<const W*>(n.x0) + (w0 ? o0 : 0);
      const W* x1w = static_cast<const W*>(n.x1) + (w1 ? o1 : 0);
      const bool two = n.x1 != nullptr, c0 = n.flags & TINY_CONJ0, c1 = n.flags & TINY_CONJ1;
      W acc = WA::zero();
      const uint32_t step = by_warp ? 32u : 1u;
      // a single summed mode (the usual case) needs no decomposition
      const bool flat = n.ninner == 1;
      const int32_t f0 = flat ? n.mode[n.nout].s0 : 0, f1 = flat ? n.mode[n.nout].s1 : 0;
      constexpr int U = sizeof(W) <= 8 ? 8 : 4;
      // X0, X1: the operands' stored types (one loop per pair, so that a step's
      // loads are issued together: 8.8 against 15 us for the 16^3 chain)
      auto sum = [&](auto* p0, auto* p1) {
        for (uint32_t jb = by_warp ? lane : 0; jb < n.n_in; jb += U * step) {
          // U steps' loads, then their sums in order
          std::remove_cv_t<std::remove_reference_t<decltype(*p0)>> v0[U];
          std::remove_cv_t<std::remove_reference_t<decltype(*p1)>> v1[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            uint32_t j = jb + u * step;
            if (j < n.n_in) {
              int32_t i0 = (int32_t)j * f0, i1 = (int32_t)j * f1;
              if (!flat) {
                i0 = i1 = 0;
                for (int m = n.nout; m < n.nout + n.ninner; ++m) {
                  const TinyMode md = n.mode[m];
                  const int32_t d = tiny_digit(j, md.ext);
                  i0 += d * md.s0;
                  i1 += d * md.s1;
                }
              }
              v0[u] = tiny_ld(p0 + i0);
              if (two) v1[u] = tiny_ld(p1 + i1);
            }
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (jb + u * step < n.n_in) {
              W p = tiny_conj(tiny_as<W>(v0[u]), c0);
              if constexpr (std::is_same<WA, AlgF32>::value) {   // (as k_loop_thread adds a product)
                acc = two ? WA::fma(p, v1[u], acc) : WA::add(acc, p);
              } else {
                if (two) p = WA::mul(p, tiny_conj(tiny_as<W>(v1[u]), c1));
                acc = WA::add(acc, p);
              }
            }
        }
      };
      if constexpr (WIDE) {
        if (w0 && w1) sum(x0w, x1w);
        else if (w0) sum(x0w, x1);
        else if (w1) sum(x0, x1w);
        else sum(x0, x1);
      } else {
        sum(x0, x1);
      }
      if (by_warp)
        for (int d = 16; d > 0; d >>= 1) acc = WA::add(acc, shfl_down_any(acc, d));
      if (in && (!by_warp || lane == 0)) {
        acc = tiny_conj(acc, n.flags & TINY_CONJY);
        if (n.y) static_cast<T*>(n.y)[yo] = tiny_as<T>(acc);
        if (WIDE && n.yw) static_cast<W*>(n.yw)[yo] = acc;
      }
    }
    if (lev + 1 < a.nlevels) cl.sync();
  }
}

// Launch configuration; at: one attribute, filled here.
cudaLaunchConfig_t tiny_config(cudaLaunchAttribute* at, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(TINY_CTAS);
  cfg.blockDim = dim3(TINY_THREADS);
  cfg.stream = s;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = TINY_CTAS;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// Whether the current device can place a cluster of sixteen blocks, which has to
// be asked for (asked once per device and kernel).
template <class A, class WA, int CAP>
bool tiny_fits() {
  static std::atomic<unsigned long long> asked{0}, fits{0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(asked.load(std::memory_order_acquire) & bit)) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = tiny_config(at, nullptr);
    int n = 0;
    cudaError_t e = cudaFuncSetAttribute(k_tiny<A, WA, CAP>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, k_tiny<A, WA, CAP>, &cfg);
    if (e != cudaSuccess) cudaGetLastError();
    else if (n > 0) fits.fetch_or(bit, std::memory_order_relaxed);
    asked.fetch_or(bit, std::memory_order_release);
  }
  return fits.load(std::memory_order_relaxed) & bit;
}

template <class A, class WA, int CAP>
cudaError_t launch_tiny_t(const TinyNode* nodes, const int* level, int n, cudaStream_t s) {
  TinyArgs<CAP> a;
  a.nlevels = 0;
  a.begin[0] = 0;
  memcpy(a.nodes, nodes, sizeof(TinyNode) * n);
  uint32_t items = 0;
  for (int i = 0; i < n; ++i) {
    if (i > 0 && level[i] != level[i - 1]) {
      a.items[a.nlevels++] = items;
      a.begin[a.nlevels] = (uint16_t)i;
      items = 0;
    }
    a.nodes[i].item0 = items;
    items += a.nodes[i].flags & TINY_WARP ? a.nodes[i].n_out : (a.nodes[i].n_out + 31) / 32;
  }
  a.items[a.nlevels++] = items;
  a.begin[a.nlevels] = (uint16_t)n;
  cudaLaunchAttribute at[1];
  const cudaLaunchConfig_t cfg = tiny_config(at, s);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_tiny<A, WA, CAP>, a);
  count_launch();
  return e;
}

}  // namespace

bool tiny_available(ome_dtype dt, bool plain) {
  bool ok = false;
  if (plain && dt == OME_F32) {
    ok = tiny_fits<AlgF32, AlgF32, TINY_CAP_SMALL>() && tiny_fits<AlgF32, AlgF32, TINY_CAP>();
  } else {
    OME_DISPATCH(dt, ALG, (ok = tiny_fits<ALG, TinyWide<ALG>::W, TINY_CAP_SMALL>() &&
                                tiny_fits<ALG, TinyWide<ALG>::W, TINY_CAP>()));
  }
  return ok;
}

size_t tiny_wide_size(ome_dtype dt) {
  size_t r = 0;
  OME_DISPATCH(dt, ALG, r = sizeof(typename TinyWide<ALG>::W::T));
  return r;
}

bool tiny_node(TinyNode& n, int nin, const HView* xs, const HView& y) {
  if (nin < 1 || nin > 2) return false;
  memset(&n, 0, sizeof(n));
  HView u[2];
  for (int i = 0; i < nin; ++i)
    if (unique_view(xs[i], u[i]) != OME_OK) return false;
  Modes outer, inner;
  outer.nt = inner.nt = nin + 1;
  int64_t st[3];
  for (int d = 0; d < y.nd; ++d) {
    for (int e = 0; e < d; ++e)
      if (y.lab[e] == y.lab[d]) return false;
    st[0] = y.str[d];
    for (int i = 0; i < nin; ++i) {
      const int k = find_lab(u[i], y.lab[d]);
      st[1 + i] = k >= 0 ? u[i].str[k] : 0;
    }
    outer.add(y.ext[d], st);
  }
  for (int i = 0; i < nin; ++i)
    for (int d = 0; d < u[i].nd; ++d) {
      const int32_t l = u[i].lab[d];
      if (find_lab(y, l) >= 0 || (i == 1 && find_lab(u[0], l) >= 0)) continue;
      st[0] = 0;
      for (int j = 0; j < nin; ++j) {
        const int k = find_lab(u[j], l);
        st[1 + j] = k >= 0 ? u[j].str[k] : 0;
      }
      inner.add(u[i].ext[d], st);
    }
  const int64_t no = outer.total(), ni = inner.total();
  if (no < 1 || ni < 1 || no * ni > TINY_WORK) return false;
  outer.normalize(0);
  inner.normalize(1);
  if (outer.n + inner.n > TINY_MODES) return false;
  n.n_out = (uint32_t)no;
  n.n_in = (uint32_t)ni;
  n.nout = (uint8_t)outer.n;
  n.ninner = (uint8_t)inner.n;
  // a warp per output when the outputs alone would leave lanes idle
  if (ni > 16 && no * 32 <= TINY_WORK) n.flags |= TINY_WARP;
  auto put = [&](const Modes& m, int at) {
    for (int i = 0; i < m.n; ++i) {
      TinyMode& md = n.mode[at + i];
      uint32_t sh = 0;
      while (((int64_t)1 << sh) < m.ext[i]) ++sh;
      md.ext = (uint32_t)m.ext[i] | (((int64_t)1 << sh) == m.ext[i] ? sh : 31u) << 24;
      for (int t = 0; t <= nin; ++t) {
        // the whole reach of a mode in 32 bits
        const int64_t v = m.str[t][i];
        if (v * m.ext[i] > 0x3fffffff / TINY_MODES || v * m.ext[i] < -(0x3fffffff / TINY_MODES)) return false;
        (t == 0 ? md.sy : t == 1 ? md.s0 : md.s1) = (int32_t)v;
      }
    }
    return true;
  };
  return put(outer, 0) && put(inner, outer.n);
}

cudaError_t launch_tiny(ome_dtype dt, const TinyNode* nodes, const int* level, int n, bool plain, cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  for (int b = 0; b < n && e == cudaSuccess;) {
    // at most TINY_CAP nodes and TINY_LEVELS levels a launch
    int c = 0, nl = 0;
    while (b + c < n && c < TINY_CAP) {
      if (c == 0 || level[b + c] != level[b + c - 1]) {
        if (nl == TINY_LEVELS) break;
        ++nl;
      }
      ++c;
    }
    KernelTimer kt(s, "k_tiny");
    e = cudaErrorInvalidValue;
    if (plain && dt == OME_F32) {
      e = c <= TINY_CAP_SMALL ? launch_tiny_t<AlgF32, AlgF32, TINY_CAP_SMALL>(nodes + b, level + b, c, s)
                              : launch_tiny_t<AlgF32, AlgF32, TINY_CAP>(nodes + b, level + b, c, s);
    } else if (c <= TINY_CAP_SMALL) {
      OME_DISPATCH(dt, ALG, e = (launch_tiny_t<ALG, TinyWide<ALG>::W, TINY_CAP_SMALL>(nodes + b, level + b, c, s)));
    } else {
      OME_DISPATCH(dt, ALG, e = (launch_tiny_t<ALG, TinyWide<ALG>::W, TINY_CAP>(nodes + b, level + b, c, s)));
    }
    b += c;
  }
  return e;
}

}  // namespace ome
