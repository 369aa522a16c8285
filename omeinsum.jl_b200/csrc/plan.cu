// Contraction-tree plans: NestedEinsum / SlicedEinsum execution and
// cost_and_gradient on the device.
//
// Reference behaviour restated:
//  * post-order evaluation of a NestedEinsum (src/einsequence.jl:270-287;
//    GPU form ext/CUDAExt.jl:121-147); intermediates live in the context's
//    workspace at offsets planned from their lifetimes instead of per-node
//    allocations and unsafe_free! (active_free);
//  * SlicedEinsum (src/slicing.jl:104-137): slices in CartesianIndices order
//    over the sliced labels (first label fastest, :37-71); each slice's leaves
//    are strided VIEWS of the inputs (no take_slice copies, :78-85); the
//    cross-slice sum is accumulated in FP64 for F32/F64/C32 (the reference
//    accumulates in the eltype); other eltypes accumulate in place;
//  * cost_and_gradient (src/bp.jl:122-130): cached forward pass, then
//    einsum_grad per child (src/autodiff.jl:24-30: conj(dy) replaces the
//    child's input, the child's labels become the output, result conjugated).
#include <string.h>
#include <algorithm>
#include <cmath>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "dispatch.h"

using namespace ome;

namespace {

struct PNode {
  std::vector<int> args;           // >= 0 node, < 0 input (-r-1)
  std::vector<int32_t> iy;         // output labels
  std::vector<int32_t> iy_s;       // output labels without sliced labels
  int64_t numel_s = 1, numel = 1;  // output elements (sliced / full)
  size_t off_fwd = 0;              // workspace offset in sliced forward
  size_t off_keep = 0;             // offset of the forward value when all are kept
  size_t off_grad = 0;             // offset of the gradient buffer
  // offsets of the same in the tiny programs' wider type (tiny nodes only)
  size_t off_fwd_w = 0, off_keep_w = 0, off_grad_w = 0;
  bool grad_tiny = false;          // the gradient is written by the reverse program
  int parent = -1;
  bool tiny = false;               // (sliced sizes) the node and its whole subtree are small contractions
  bool tiny_full = false;          // the same with full sizes
};

// A step of a tiny program: contraction of up to two operands, each a node's
// value, a node's gradient or an input.
struct TinyStep {
  enum Kind { VALUE, GRAD, INPUT, INPUT_GRAD, OUTPUT };
  int nin = 0, level = 0;
  Kind kind[3];                    // operands, then the result
  int ref[3];
  uint8_t flags = 0;
};

// Its launch descriptors for one set of input strides.
struct TinyProgram {
  std::vector<int64_t> strides;    // the caller's (empty: column-major)
  bool strided = false, ok = false;
  std::vector<TinyNode> nodes;
  std::vector<int> level;
};

}  // namespace

struct ome_plan {
  ome_dtype dt;
  int prec;
  int ninputs;
  std::vector<std::vector<int32_t>> in_labels;
  std::vector<int> in_pos;         // where input t's strides start in a caller's stride list
  std::map<int32_t, int64_t> ext;
  std::vector<int32_t> sliced;
  int64_t nslices = 1;
  std::vector<PNode> nodes;
  bool acc64 = false;
  size_t acc_off = 0, tmp_off = 0;  // FP64 accumulator and root temporary (sliced)
  size_t dy_off = 0;                        // root cotangent buffer (gradient)
  size_t arena_bytes = 0, grad_arena = 0;  // planned buffers (forward / gradient)
  size_t fwd_bytes = 0, grad_bytes = 0;     // plus per-node dispatch scratch: the least it runs in
  size_t fwd_peak = 0, grad_peak = 0;       // with the buffers of the evaluation in Float64 (`wide`)
  size_t esize = 0;
  size_t wsize = 0;                // bytes of the wider type; 0 if it is the element type
  bool fixed_sums = false;         // sliced Float32: every node's sums as a call of its own computes them
  // steps of the tiny programs, levels ascending: forward on sliced and on
  // full sizes, reverse sweep; programs built for the last input strides seen
  // (several threads may evaluate one plan)
  std::vector<TinyStep> steps[5];
  std::shared_ptr<const TinyProgram> prog[5];
  std::mutex prog_mutex;
  std::vector<std::vector<char>> rev_tiny;   // [node][child]: the gradient step is in the reverse program
  // Small Float32 / ComplexF32 trees are evaluated in Float64 / ComplexF64: the
  // same tree planned in that type, and where its inputs, output, cotangent and
  // gradients lie at the start of the workspace.
  std::unique_ptr<ome_plan> wide;
  std::vector<size_t> wide_in, wide_dx;
  size_t wide_y = 0, wide_dy = 0, wide_base = 0;
};
// forward on sliced and on full sizes, reverse sweep, inputs to the wider type,
// gradients from it
enum { TINY_FWD = 0, TINY_FWD_FULL = 1, TINY_REV = 2, TINY_WIDEN = 3, TINY_NARROW = 4 };

namespace {

struct Interval {
  size_t off, size;
};

// First-fit offset allocator over live intervals (256-byte aligned).
struct Arena {
  std::vector<std::pair<size_t, size_t>> live;  // (off, size)
  size_t peak = 0;
  size_t alloc(size_t bytes) {
    bytes = (bytes + 255) & ~(size_t)255;
    if (bytes == 0) bytes = 256;
    std::sort(live.begin(), live.end());
    size_t off = 0;
    for (auto& p : live) {
      if (p.first >= off + bytes) break;
      off = std::max(off, p.first + p.second);
    }
    live.push_back({off, bytes});
    peak = std::max(peak, off + bytes);
    return off;
  }
  void release(size_t off) {
    for (size_t i = 0; i < live.size(); ++i)
      if (live[i].first == off) {
        live.erase(live.begin() + i);
        return;
      }
  }
};

bool contains(const std::vector<int32_t>& v, int32_t l) { return std::find(v.begin(), v.end(), l) != v.end(); }

// Column-major contiguous view with labels `labs`; labels in `drop` are
// fixed at index `fix` (their stride folded into the base offset) and removed.
HView make_view(const ome_plan* p, char* base, const std::vector<int32_t>& labs, const std::vector<int32_t>& drop,
                const std::vector<int64_t>& fix) {
  HView v;
  v.data = base;
  v.nd = 0;
  int64_t s = 1;
  int64_t off = 0;
  for (int32_t l : labs) {
    const int64_t e = p->ext.at(l);
    auto it = std::find(drop.begin(), drop.end(), l);
    if (it != drop.end()) {
      off += fix[it - drop.begin()] * s;
    } else {
      v.lab[v.nd] = l;
      v.ext[v.nd] = e;
      v.str[v.nd] = s;
      v.nd++;
    }
    s *= e;
  }
  v.data = base + off * (int64_t)p->esize;
  return v;
}

std::vector<int32_t> child_labels(const ome_plan* p, int ref, bool sliced) {
  if (ref >= 0) return sliced ? p->nodes[ref].iy_s : p->nodes[ref].iy;
  const auto& l = p->in_labels[-ref - 1];
  if (!sliced) return l;
  std::vector<int32_t> r;
  for (int32_t x : l)
    if (!contains(p->sliced, x)) r.push_back(x);
  return r;
}

// Memory order of intermediates.  An intermediate's label order is internal to
// the plan (only the root's is the caller's), so each binary node lays out its
// children for itself, as analyze_binary's canonical orders do
// (src/einsum.jl:139-185; OMEinsumContractionOrders' optimize_permute):
// x1 = [outer1 (output order), inner, batch (output order)],
// x2 = [inner, outer2 (output order), batch (output order)], with one inner
// order shared by both (a leaf child's, if either child is a leaf).  Mode
// groups of the strided GEMM then merge into one or a few modes.  Top-down:
// a parent's order is final before its children are arranged.
void canonical_orders(ome_plan* p) {
  const int nn = (int)p->nodes.size();
  for (int j = nn - 1; j >= 0; --j) {
    PNode& n = p->nodes[j];
    if (n.args.size() != 2) continue;
    const int r1 = n.args[0], r2 = n.args[1];
    const std::vector<int32_t> L1 = r1 >= 0 ? p->nodes[r1].iy : p->in_labels[-r1 - 1];
    const std::vector<int32_t> L2 = r2 >= 0 ? p->nodes[r2].iy : p->in_labels[-r2 - 1];
    const std::vector<int32_t>& y = n.iy;
    std::vector<int32_t> o1, o2, batch, inner, d1, d2;
    for (int32_t l : y) {
      const bool a = contains(L1, l), b = contains(L2, l);
      if (a && b) batch.push_back(l);
      else if (a) o1.push_back(l);
      else if (b) o2.push_back(l);
    }
    const std::vector<int32_t>& ref = (r1 < 0 || r2 >= 0) ? L1 : L2;  // a leaf's order if there is one
    for (int32_t l : ref)
      if (contains(L1, l) && contains(L2, l) && !contains(y, l)) inner.push_back(l);
    for (int32_t l : L1)
      if (!contains(L2, l) && !contains(y, l)) d1.push_back(l);
    for (int32_t l : L2)
      if (!contains(L1, l) && !contains(y, l)) d2.push_back(l);
    auto rebuild = [&](int r, const std::vector<std::vector<int32_t>>& parts) {
      std::vector<int32_t> v;
      for (auto& q : parts) v.insert(v.end(), q.begin(), q.end());
      PNode& c = p->nodes[r];
      if (v.size() != c.iy.size()) return;  // not a permutation of the child's labels: keep
      c.iy = v;
      c.iy_s.clear();
      for (int32_t l : v)
        if (!contains(p->sliced, l)) c.iy_s.push_back(l);
    };
    if (r1 >= 0) rebuild(r1, {o1, inner, batch, d1});
    if (r2 >= 0) rebuild(r2, {inner, o2, batch, d2});
  }
}

std::vector<int32_t> drop_sliced(const ome_plan* p, const std::vector<int32_t>& l, bool sliced) {
  if (!sliced) return l;
  std::vector<int32_t> r;
  for (int32_t x : l)
    if (!contains(p->sliced, x)) r.push_back(x);
  return r;
}

// Whether the contraction of operands `xs` into labels `y` is a tiny step:
// one or two operands, no repeated output label, no label summed in one of
// two operands only, at most TINY_WORK multiply-adds.
bool tiny_step(const ome_plan* p, const std::vector<std::vector<int32_t>>& xs, const std::vector<int32_t>& y) {
  if (xs.empty() || xs.size() > 2) return false;
  for (size_t i = 0; i < y.size(); ++i)
    for (size_t k = 0; k < i; ++k)
      if (y[i] == y[k]) return false;
  std::vector<int32_t> seen;
  double work = 1;
  auto visit = [&](int32_t l) {
    if (contains(seen, l)) return;
    seen.push_back(l);
    work *= (double)p->ext.at(l);
  };
  for (int32_t l : y) visit(l);
  for (size_t i = 0; i < xs.size(); ++i)
    for (int32_t l : xs[i]) {
      if (xs.size() == 2 && !contains(y, l) && !contains(xs[1 - i], l) && p->ext.at(l) != 1) return false;
      visit(l);
    }
  if (p->fixed_sums) {   // only what k_loop_thread evaluates
    double terms = 1, m = 1, n = 1;
    for (int32_t l : seen) {
      const double e = (double)p->ext.at(l);
      if (!contains(y, l)) terms *= e;
      else if (!contains(xs.back(), l)) m *= e;
      else if (!contains(xs[0], l)) n *= e;
    }
    if (terms > 16 || (xs.size() == 2 && m >= 16 && n >= 16 && terms >= 8)) return false;
  }
  return work >= 1 && work <= (double)TINY_WORK;
}

// The steps that run as tiny programs: forward, the nodes whose whole subtree
// is tiny; in the reverse sweep, the gradient steps below which all are tiny.
void plan_tiny(ome_plan* p) {
  const int nn = (int)p->nodes.size(), root = nn - 1;
  auto labels = [&](int r, bool sliced) {
    return drop_sliced(p, r >= 0 ? p->nodes[r].iy : p->in_labels[-r - 1], sliced);
  };
  std::vector<int> depth(nn);
  for (int full = 0; full < 2; ++full) {
    const bool sliced = !full;
    std::vector<int> order;
    for (int j = 0; j < (full || p->sliced.empty() ? nn : root); ++j) {
      PNode& n = p->nodes[j];
      bool t = true;
      int d = 0;
      std::vector<std::vector<int32_t>> xs;
      for (int r : n.args) {
        if (r >= 0) {
          t = t && (full ? p->nodes[r].tiny_full : p->nodes[r].tiny);
          d = std::max(d, depth[r] + 1);
        }
        xs.push_back(labels(r, sliced));
      }
      t = t && tiny_step(p, xs, labels(j, sliced));
      (full ? n.tiny_full : n.tiny) = t;
      depth[j] = d;
      if (t) order.push_back(j);
    }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return depth[a] < depth[b]; });
    for (int j : order) {
      TinyStep s;
      const PNode& n = p->nodes[j];
      s.nin = (int)n.args.size();
      s.level = depth[j];
      for (int a = 0; a < s.nin; ++a) {
        s.kind[a] = n.args[a] >= 0 ? TinyStep::VALUE : TinyStep::INPUT;
        s.ref[a] = n.args[a] >= 0 ? n.args[a] : -n.args[a] - 1;
      }
      s.kind[2] = j == root ? TinyStep::OUTPUT : TinyStep::VALUE;   // (the root last: all others are below it)
      s.ref[2] = j;
      p->steps[full ? TINY_FWD_FULL : TINY_FWD].push_back(s);
    }
    // one step alone gains nothing
    if (order.size() < 2) {
      p->steps[full ? TINY_FWD_FULL : TINY_FWD].clear();
      for (int j : order) (full ? p->nodes[j].tiny_full : p->nodes[j].tiny) = false;
    }
  }
  // reverse: below[j] = every gradient step of j's subtree (j's own included) is tiny
  const bool cplx = p->dt == OME_C32 || p->dt == OME_C64;
  std::vector<char> below(nn, 0);
  p->rev_tiny.resize(nn);
  for (int j = 0; j < nn; ++j) {
    const PNode& n = p->nodes[j];
    bool all = true;
    p->rev_tiny[j].assign(n.args.size(), 0);
    for (size_t i = 0; i < n.args.size(); ++i) {
      std::vector<std::vector<int32_t>> xs;
      for (size_t a = 0; a < n.args.size(); ++a) xs.push_back(a == i ? n.iy : labels(n.args[a], false));
      const int r = n.args[i];
      const bool t = tiny_step(p, xs, labels(r, false)) && (r < 0 || below[r]);
      p->rev_tiny[j][i] = t;
      all = all && t;
    }
    below[j] = all;
  }
  std::vector<int> lev(nn, 0);   // reverse level of a node's own steps
  for (int j = root; j >= 0; --j) {
    const PNode& n = p->nodes[j];
    for (size_t i = 0; i < n.args.size(); ++i) {
      if (!p->rev_tiny[j][i]) continue;
      TinyStep s;
      s.nin = (int)n.args.size();
      s.level = lev[j];
      for (int a = 0; a < s.nin; ++a) {
        const int r = n.args[a];
        s.kind[a] = a == (int)i ? TinyStep::GRAD : r >= 0 ? TinyStep::VALUE : TinyStep::INPUT;
        s.ref[a] = a == (int)i ? j : r >= 0 ? r : -r - 1;
      }
      const int r = n.args[i];
      s.kind[2] = r >= 0 ? TinyStep::GRAD : TinyStep::INPUT_GRAD;
      s.ref[2] = r >= 0 ? r : -r - 1;
      if (cplx) s.flags = TINY_CONJY | (i == 0 ? TINY_CONJ0 : TINY_CONJ1);
      if (r >= 0) {
        lev[r] = lev[j] + 1;
        p->nodes[r].grad_tiny = true;
      }
      p->steps[TINY_REV].push_back(s);
    }
  }
  std::stable_sort(p->steps[TINY_REV].begin(), p->steps[TINY_REV].end(),
                   [](const TinyStep& a, const TinyStep& b) { return a.level < b.level; });
}

// Multiply-adds of all nodes on full sizes.
double plan_work(const ome_plan* p) {
  double total = 0;
  for (const PNode& n : p->nodes) {
    std::vector<int32_t> seen;
    double w = 1;
    auto visit = [&](const std::vector<int32_t>& l) {
      for (int32_t x : l)
        if (!contains(seen, x)) {
          seen.push_back(x);
          w *= (double)p->ext.at(x);
        }
    };
    visit(n.iy);
    for (int r : n.args) visit(r >= 0 ? p->nodes[r].iy : p->in_labels[-r - 1]);
    total += w;
  }
  return total;
}

}  // namespace

extern "C" {

int ome_plan_create(ome_ctx* ctx, ome_dtype dtype, int32_t ninputs, const int32_t* input_nlabels,
                    const int32_t* input_labels, int32_t nnodes, const int32_t* node_nargs, const int32_t* node_args,
                    const int32_t* node_niy, const int32_t* node_iy, int32_t nlabels, const int32_t* label_ids,
                    const int64_t* label_extents, int32_t nsliced, const int32_t* sliced_labels, int32_t prec,
                    ome_plan** out) {
  (void)ctx;
  if (!out) return set_err(OME_INVALID_ARGUMENT, "out is NULL");
  *out = nullptr;
  if ((int)dtype < 0 || (int)dtype > OME_TROP_F64) return set_err(OME_INVALID_ARGUMENT, "unknown dtype");
  if (ninputs < 1 || nnodes < 1) return set_err(OME_INVALID_ARGUMENT, "empty tree");
  auto p = new ome_plan();
  p->dt = dtype;
  p->prec = prec;
  p->esize = dtype_size(dtype);
  p->fixed_sums = dtype == OME_F32 && nsliced > 0;
  p->wsize = p->fixed_sums || tiny_wide_size(dtype) == p->esize ? 0 : tiny_wide_size(dtype);
  p->ninputs = ninputs;
  for (int i = 0; i < nlabels; ++i) {
    if (label_extents[i] < 0) {
      delete p;
      return set_err(OME_INVALID_ARGUMENT, "negative extent for label %d", label_ids[i]);
    }
    p->ext[label_ids[i]] = label_extents[i];
  }
  int pos = 0;
  for (int t = 0; t < ninputs; ++t) {
    std::vector<int32_t> l(input_labels + pos, input_labels + pos + input_nlabels[t]);
    p->in_pos.push_back(pos);
    pos += input_nlabels[t];
    for (int32_t x : l)
      if (!p->ext.count(x)) {
        delete p;
        return set_err(OME_INVALID_ARGUMENT, "label %d of input %d has no extent", x, t);
      }
    p->in_labels.push_back(l);
  }
  for (int i = 0; i < nsliced; ++i) {
    if (!p->ext.count(sliced_labels[i])) {
      delete p;
      return set_err(OME_INVALID_ARGUMENT, "sliced label %d has no extent", sliced_labels[i]);
    }
    p->sliced.push_back(sliced_labels[i]);
    p->nslices *= p->ext[sliced_labels[i]];
  }
  std::vector<int> input_used(ninputs, 0);
  int apos = 0, ypos = 0;
  p->nodes.resize(nnodes);
  for (int j = 0; j < nnodes; ++j) {
    PNode& n = p->nodes[j];
    for (int a = 0; a < node_nargs[j]; ++a) {
      const int r = node_args[apos++];
      if (r >= 0) {
        if (r >= j || p->nodes[r].parent != -1) {
          delete p;
          return set_err(OME_INVALID_ARGUMENT, "node %d: child %d is not an earlier unused node", j, r);
        }
        p->nodes[r].parent = j;
      } else {
        const int t = -r - 1;
        if (t >= ninputs || input_used[t]) {
          delete p;
          return set_err(OME_INVALID_ARGUMENT, "node %d: bad or repeated input %d", j, t);
        }
        input_used[t] = 1;
      }
      n.args.push_back(r);
    }
    if (n.args.empty()) {
      delete p;
      return set_err(OME_INVALID_ARGUMENT, "node %d has no children", j);
    }
    for (int a = 0; a < node_niy[j]; ++a) {
      const int32_t l = node_iy[ypos++];
      if (!p->ext.count(l)) {
        delete p;
        return set_err(OME_INVALID_ARGUMENT, "output label %d of node %d has no extent", l, j);
      }
      n.iy.push_back(l);
      if (!contains(p->sliced, l)) n.iy_s.push_back(l);
    }
    for (int32_t l : n.iy) n.numel *= p->ext[l];
    for (int32_t l : n.iy_s) n.numel_s *= p->ext[l];
  }
  canonical_orders(p);
  for (int t = 0; t < ninputs; ++t)
    if (!input_used[t]) {
      delete p;
      return set_err(OME_INVALID_ARGUMENT, "input %d is not used by the tree", t);
    }
  for (int j = 0; j < nnodes - 1; ++j)
    if (p->nodes[j].parent < 0) {
      delete p;
      return set_err(OME_INVALID_ARGUMENT, "node %d is not reachable from the root", j);
    }
  plan_tiny(p);
  // forward arena (sliced shapes), liveness: a node's output dies when its
  // parent ran.  The tiny nodes run before all others, in any order among
  // themselves, so their buffers are reserved together.  The FP64 cross-slice accumulator lives through every slice,
  // so it is reserved first and never shared with a node buffer.
  const int root = nnodes - 1;
  const bool sliced = !p->sliced.empty();
  p->acc64 = sliced && (dtype == OME_F32 || dtype == OME_F64 || dtype == OME_C32);
  Arena ar;
  if (p->acc64) p->acc_off = ar.alloc((size_t)p->nodes[root].numel * (dtype == OME_C32 ? 16 : 8));
  for (int j = 0; j < root; ++j)
    if (p->nodes[j].tiny) p->nodes[j].off_fwd = ar.alloc((size_t)p->nodes[j].numel_s * p->esize);
  if (p->wsize) {   // (wide copies live through the program only)
    for (int j = 0; j < root; ++j)
      if (p->nodes[j].tiny) p->nodes[j].off_fwd_w = ar.alloc((size_t)p->nodes[j].numel_s * p->wsize);
    for (int j = 0; j < root; ++j)
      if (p->nodes[j].tiny) ar.release(p->nodes[j].off_fwd_w);
  }
  for (int j = 0; j < root; ++j)
    if (p->nodes[j].tiny)
      for (int r : p->nodes[j].args)
        if (r >= 0) ar.release(p->nodes[r].off_fwd);
  for (int j = 0; j < root; ++j) {
    PNode& n = p->nodes[j];
    if (n.tiny) continue;
    n.off_fwd = ar.alloc((size_t)n.numel_s * p->esize);
    for (int r : n.args)
      if (r >= 0) ar.release(p->nodes[r].off_fwd);
  }
  // the root's temporary is written after every other node of the slice ran
  // (its children are still live here, so it cannot overlap them)
  if (p->acc64) p->tmp_off = ar.alloc((size_t)p->nodes[root].numel_s * p->esize);
  p->arena_bytes = ar.peak;
  // per-node dispatch scratch: dangling-label reductions (bounded by the
  // children's sizes), split-reduction partials and GEMM workspace; sliced
  // sizes for the forward plan, full sizes for the (unsliced) gradient
  // FP32 binary nodes that the dispatcher sends to the packed-operand
  // tensor-core GEMM (M, N >= 256, K >= 512, >= 1 GFLOP; ComplexF32: M, N, K >=
  // 128, >= 1 GFLOP, through the real embedding) need their BF16
  // terms in the workspace: L * (M/128 + N/128 tiles) * K/32 k-steps * 24 KB,
  // plus split partials and offset tables (at most 2 GB here; a node that
  // needs more takes its terms from the context's overflow scratch)
  auto packed_gemm_bytes = [&](int j, bool use_sliced) -> size_t {
    const PNode& n = p->nodes[j];
    const bool c32 = dtype == OME_C32;
    if ((dtype != OME_F32 && !c32) || prec == OME_PREC_FP32 || n.args.size() != 2) return 0;
    auto labs = [&](int r) -> std::vector<int32_t> {
      std::vector<int32_t> v;
      if (r >= 0) {
        v = use_sliced ? p->nodes[r].iy_s : p->nodes[r].iy;
      } else {
        for (int32_t l : p->in_labels[-r - 1])
          if (!(use_sliced && contains(p->sliced, l))) v.push_back(l);
      }
      return v;
    };
    const std::vector<int32_t> a = labs(n.args[0]), b = labs(n.args[1]);
    const std::vector<int32_t>& y = use_sliced ? n.iy_s : n.iy;
    double M = 1, N = 1, K = 1, L = 1;
    std::vector<int32_t> seen;
    for (const auto* v : {&a, &b})
      for (int32_t l : *v) {
        if (contains(seen, l)) continue;
        seen.push_back(l);
        const bool ia = contains(a, l), ib = contains(b, l), iy = contains(y, l);
        const double e = (double)p->ext[l];
        if (ia && ib && iy) L *= e;
        else if (ia && ib) K *= e;
        else if (ia && iy) M *= e;
        else if (ib && iy) N *= e;
      }
    if (c32) {   // (the real embedding of the longer side)
      if (M < 128 || N < 128 || K < 128 || 8.0 * M * N * K * L < 1e9) return 0;
      const double longer = std::max(M, N);
      N = std::min(M, N);
      M = 2 * longer;
      K *= 2;
    } else if (M < 256 || N < 256 || K < 512 || 2.0 * M * N * K * L < 1e9) {
      return 0;
    }
    const double bytes = L * (std::ceil(M / 128) + std::ceil(N / 128)) * std::ceil(K / 32) * 3 * 8192 +
                         74.0 * 256 * 256 * 4 + (M + N) * 8 + 4096;
    return bytes <= (double)((size_t)2 << 30) ? (size_t)bytes : 0;
  };
  auto scratch_bound = [&](bool use_sliced) {
    size_t scratch = 0;
    for (int j = 0; j < nnodes; ++j) {
      size_t sj = 0;
      for (int r : p->nodes[j].args) {
        int64_t c = 1;
        if (r >= 0) {
          c = use_sliced ? p->nodes[r].numel_s : p->nodes[r].numel;
        } else {
          for (int32_t l : p->in_labels[-r - 1])
            if (!(use_sliced && contains(p->sliced, l))) c *= p->ext[l];
        }
        sj += ((size_t)c * p->esize + 255) & ~(size_t)255;
      }
      sj += packed_gemm_bytes(j, use_sliced);
      scratch = std::max(scratch, sj);
    }
    return scratch + ((size_t)64 << 20);
  };
  const size_t scratch = scratch_bound(true), scratch_grad = scratch_bound(false);
  p->fwd_bytes = ((p->arena_bytes + 255) & ~(size_t)255) + scratch;
  // gradient arena: all forward values kept (unsliced) plus one gradient each
  size_t g = 0;
  for (int j = 0; j < root; ++j) {
    PNode& n = p->nodes[j];
    n.off_keep = g;
    g += ((size_t)n.numel * p->esize + 255) & ~(size_t)255;
  }
  for (int j = 0; j < root; ++j) {
    PNode& n = p->nodes[j];
    n.off_grad = g;
    g += ((size_t)n.numel * p->esize + 255) & ~(size_t)255;
  }
  if (p->wsize)
    for (int j = 0; j < root; ++j) {
      PNode& n = p->nodes[j];
      const size_t b = ((size_t)n.numel * p->wsize + 255) & ~(size_t)255;
      if (n.tiny_full) {
        n.off_keep_w = g;
        g += b;
      }
      if (n.grad_tiny) {
        n.off_grad_w = g;
        g += b;
      }
    }
  p->dy_off = g;
  p->grad_arena = g + ((size_t)p->nodes[root].numel * p->esize + 511);
  p->grad_bytes = ((p->grad_arena + 255) & ~(size_t)255) + scratch_grad;
  p->fwd_peak = p->fwd_bytes;
  p->grad_peak = p->grad_bytes;
  // Trees of up to 2^32 multiply-adds in Float64: every value is then rounded to
  // 32 bits once, at the end, where the roundings of a hundred nodes are
  // amplified by the network's cancellations.  Over 12 sets of inputs each of 26
  // networks between 2^26 and 2^32, with and without gradients, Float32 nodes
  // leave 1e-7 .. 4e-5 and which of two evaluations is the nearer one is chance;
  // Float64 leaves 1e-8 .. 5e-8.  Up to 2^26 (8 us of the FP64 pipe) the launches
  // set the time; 2^29.8 value and gradients 1.00 -> 1.19 ms, 2^31.1 1.15 -> 1.67
  // and its value alone 0.22 -> 0.41; above, Float64 would be most of the time.
  // Below eight nodes the two conversions' launches would be felt.  The second
  // plan's buffers may take 1 GiB.
  if ((dtype == OME_F32 || dtype == OME_C32) && prec != OME_PREC_FP32 && !sliced && nnodes >= 8 &&
      plan_work(p) <= 0x1p32) {
    bool small = true;
    for (auto& l : p->in_labels) {
      double n = 1;
      for (int32_t x : l) n *= (double)p->ext[x];
      small = small && n >= 1 && n <= (double)TINY_WORK && l.size() <= TINY_MODES;
    }
    ome_plan* w = nullptr;
    const ome_dtype wt = dtype == OME_F32 ? OME_F64 : OME_C64;
    if (small && ome_plan_create(ctx, wt, ninputs, input_nlabels, input_labels, nnodes, node_nargs, node_args, node_niy,
                                 node_iy, nlabels, label_ids, label_extents, 0, nullptr, prec, &w) == OME_OK &&
        w->grad_bytes > (size_t)1 << 30) {
      delete w;
      w = nullptr;
    }
    if (w) {
      p->wide.reset(w);
      size_t at = 0;
      auto take = [&](int64_t n) {
        const size_t o = at;
        at += ((size_t)std::max<int64_t>(n, 1) * w->esize + 255) & ~(size_t)255;
        return o;
      };
      for (int grad = 0; grad < 2; ++grad)
        for (auto& l : p->in_labels) {
          int64_t n = 1;
          for (int32_t x : l) n *= p->ext[x];
          (grad ? p->wide_dx : p->wide_in).push_back(take(n));
        }
      p->wide_y = take(p->nodes[root].numel);
      p->wide_dy = take(p->nodes[root].numel);
      p->wide_base = at;
      p->fwd_peak = std::max(p->fwd_bytes, at + w->fwd_bytes);
      p->grad_peak = std::max(p->grad_bytes, at + w->grad_bytes);
      for (int which : {TINY_WIDEN, TINY_NARROW})
        for (int t = 0; t < ninputs; ++t) {
          TinyStep st;
          st.nin = 1;
          st.kind[0] = TinyStep::INPUT;
          st.kind[2] = TinyStep::INPUT_GRAD;
          st.ref[0] = st.ref[2] = t;
          p->steps[which].push_back(st);
        }
    }
  }
  *out = p;
  return OME_OK;
}

int ome_plan_destroy(ome_plan* plan) {
  delete plan;
  return OME_OK;
}

int ome_plan_peak_bytes(const ome_plan* plan, size_t* forward_bytes, size_t* grad_bytes) {
  if (!plan) return set_err(OME_INVALID_ARGUMENT, "plan is NULL");
  if (forward_bytes) *forward_bytes = plan->fwd_peak;
  if (grad_bytes) *grad_bytes = plan->grad_peak;
  return OME_OK;
}

int ome_plan_min_bytes(const ome_plan* plan, size_t* forward_bytes, size_t* grad_bytes) {
  if (!plan) return set_err(OME_INVALID_ARGUMENT, "plan is NULL");
  if (forward_bytes) *forward_bytes = plan->fwd_bytes;
  if (grad_bytes) *grad_bytes = plan->grad_bytes;
  return OME_OK;
}

}  // extern "C"

namespace {

// The caller's input tensors: data, and element strides of all inputs' modes
// one after the other (NULL: column-major contiguous).
struct Leaves {
  const void* const* data;
  const int64_t* str;
};

// View of input t; labels in `drop` are fixed at index `fix` as in make_view.
HView leaf_view(const ome_plan* p, const Leaves& in, int t, const std::vector<int32_t>& drop,
                const std::vector<int64_t>& fix) {
  const auto& labs = p->in_labels[t];
  if (!in.str) return make_view(p, (char*)in.data[t], labs, drop, fix);
  const int64_t* str = in.str + p->in_pos[t];
  HView v;
  v.nd = 0;
  int64_t off = 0;
  for (size_t d = 0; d < labs.size(); ++d) {
    auto it = std::find(drop.begin(), drop.end(), labs[d]);
    if (it != drop.end()) {
      off += fix[it - drop.begin()] * str[d];
    } else {
      v.lab[v.nd] = labs[d];
      v.ext[v.nd] = p->ext.at(labs[d]);
      v.str[v.nd] = str[d];
      v.nd++;
    }
  }
  v.data = (char*)in.data[t] + off * (int64_t)p->esize;
  return v;
}

// Run one node: inputs from children (workspace or leaf views), output view y.
int run_node(ome_ctx* ctx, ome_plan* p, cudaStream_t s, int j, const Leaves& inputs, bool sliced,
             const std::vector<int64_t>& fix, size_t (*off_of)(const PNode&), const HView& y, const Scalar& sx,
             const Scalar& sy, size_t scratch_base) {
  const PNode& n = p->nodes[j];
  HView xs[MAXIN];
  const int nin = (int)n.args.size();
  if (nin > MAXIN) return set_err(OME_UNSUPPORTED, "node %d has %d children (max %d)", j, nin, MAXIN);
  static const std::vector<int32_t> none;
  static const std::vector<int64_t> nofix;
  for (int a = 0; a < nin; ++a) {
    const int r = n.args[a];
    if (r >= 0) {
      xs[a] = make_view(p, ctx->ws + off_of(p->nodes[r]), sliced ? p->nodes[r].iy_s : p->nodes[r].iy, none, nofix);
    } else {
      xs[a] = leaf_view(p, inputs, -r - 1, sliced ? p->sliced : none, sliced ? fix : nofix);
    }
  }
  ctx->ws_top = scratch_base;
  return einsum_views(ctx, s, p->dt, nin, xs, y, sx, sy, p->prec, false);
}

size_t off_fwd_of(const PNode& n) { return n.off_fwd; }
size_t off_keep_of(const PNode& n) { return n.off_keep; }

// The descriptors of a tiny program for the caller's input strides, from the
// plan's cache or built now (pointers are set per launch).  Not ok: the nodes
// run one by one, as the strides do not fit or the device cannot place the
// program's cluster.
std::shared_ptr<const TinyProgram> tiny_program(ome_plan* p, int which, const Leaves& in) {
  static const auto unavailable = std::make_shared<const TinyProgram>();
  if (!tiny_available(p->dt, p->fixed_sums)) return unavailable;
  size_t ns = 0;
  for (auto& l : p->in_labels) ns += l.size();
  {
    std::lock_guard<std::mutex> lk(p->prog_mutex);
    const auto& c = p->prog[which];
    if (c && c->strided == (in.str != nullptr) &&
        (!in.str || std::equal(c->strides.begin(), c->strides.end(), in.str)))
      return c;
  }
  auto prog = std::make_shared<TinyProgram>();
  prog->strided = in.str != nullptr;
  if (in.str) prog->strides.assign(in.str, in.str + ns);
  prog->ok = true;
  const bool sliced = which == TINY_FWD;
  static const std::vector<int32_t> none;
  const std::vector<int64_t> fix(p->sliced.size(), 0);
  const std::vector<int32_t>& drop = sliced ? p->sliced : none;
  std::vector<const void*> null((size_t)p->ninputs, nullptr);
  const Leaves nowhere{null.data(), in.str};
  for (const TinyStep& st : p->steps[which]) {
    HView xs[2], y;
    if (which >= TINY_WIDEN) {   // a copy, mode by mode (the labels may repeat)
      xs[0] = which == TINY_WIDEN ? leaf_view(p, nowhere, st.ref[0], none, fix)
                                  : make_view(p, nullptr, p->in_labels[st.ref[0]], none, fix);
      y = make_view(p, nullptr, p->in_labels[st.ref[2]], none, fix);
      for (int d = 0; d < y.nd; ++d) xs[0].lab[d] = y.lab[d] = d;
    } else for (int a = 0; a < st.nin; ++a)
      xs[a] = st.kind[a] == TinyStep::INPUT
                  ? leaf_view(p, nowhere, st.ref[a], drop, fix)
                  : make_view(p, nullptr, sliced ? p->nodes[st.ref[a]].iy_s : p->nodes[st.ref[a]].iy, none, fix);
    if (which < TINY_WIDEN) y = st.kind[2] == TinyStep::INPUT_GRAD
            ? make_view(p, nullptr, p->in_labels[st.ref[2]], none, fix)
            : make_view(p, nullptr, sliced ? p->nodes[st.ref[2]].iy_s : p->nodes[st.ref[2]].iy, none, fix);
    TinyNode n;
    if (!tiny_node(n, st.nin, xs, y)) {
      prog->ok = false;
      break;
    }
    n.flags |= st.flags;
    prog->nodes.push_back(n);
    prog->level.push_back(st.level);
  }
  std::lock_guard<std::mutex> lk(p->prog_mutex);
  p->prog[which] = prog;
  return prog;
}

// Runs a tiny program; *done = false (nothing launched) if the input strides
// do not fit its descriptors.  y: where a tree that is tiny as a whole puts
// its value (NULL: the root is left out).  values_wide: the tiny nodes' values
// are there in the wider type too.
int run_tiny(ome_ctx* ctx, ome_plan* p, cudaStream_t s, int which, const Leaves& in, const std::vector<int64_t>& fix,
             char* y, char* dy_root, void* const* dxs, bool values_wide, bool* done) {
  *done = true;
  const auto& steps = p->steps[which];
  if (steps.empty()) return OME_OK;
  auto prog = tiny_program(p, which, in);
  *done = prog->ok;
  if (!prog->ok) return OME_OK;
  const bool keep = which != TINY_FWD;
  const int root = (int)p->nodes.size() - 1;
  // element offsets of the inputs at this slice
  std::vector<int64_t> off((size_t)p->ninputs, 0);
  if (which == TINY_FWD && !p->sliced.empty())
    for (int t = 0; t < p->ninputs; ++t) {
      int64_t st = 1;
      for (size_t d = 0; d < p->in_labels[t].size(); ++d) {
        const int32_t l = p->in_labels[t][d];
        auto it = std::find(p->sliced.begin(), p->sliced.end(), l);
        if (it != p->sliced.end())
          off[t] += fix[it - p->sliced.begin()] * (in.str ? in.str[p->in_pos[t] + (int)d] : st);
        st *= p->ext.at(l);
      }
    }
  auto at = [&](TinyStep::Kind k, int ref) -> char* {
    switch (k) {
      case TinyStep::VALUE: return ctx->ws + (keep ? p->nodes[ref].off_keep : p->nodes[ref].off_fwd);
      case TinyStep::GRAD: return ref == root ? dy_root : ctx->ws + p->nodes[ref].off_grad;
      case TinyStep::INPUT: return (char*)in.data[ref] + off[ref] * (int64_t)p->esize;
      case TinyStep::OUTPUT: return y;
      default: return (char*)dxs[ref];
    }
  };
  std::vector<TinyNode> nodes(prog->nodes);
  size_t count = steps.size();
  if (steps.back().kind[2] == TinyStep::OUTPUT && !y) --count;
  // the wider copy of a value or gradient (NULL: there is none)
  auto wide = [&](TinyStep::Kind k, int ref) -> char* {
    if (!p->wsize || (k != TinyStep::VALUE && k != TinyStep::GRAD) || ref == root) return nullptr;
    const PNode& n = p->nodes[ref];
    if (k == TinyStep::VALUE && values_wide && (keep ? n.tiny_full : n.tiny)) return ctx->ws + (keep ? n.off_keep_w : n.off_fwd_w);
    return k == TinyStep::GRAD && n.grad_tiny ? ctx->ws + n.off_grad_w : nullptr;
  };
  for (size_t i = 0; i < count; ++i) {
    const TinyStep& st = steps[i];
    TinyNode& n = nodes[i];
    for (int a = 0; a < st.nin; ++a) {
      char* w = wide(st.kind[a], st.ref[a]);
      (a == 0 ? n.x0 : n.x1) = w ? w : at(st.kind[a], st.ref[a]);
      if (w) n.flags |= a == 0 ? TINY_WIDE0 : TINY_WIDE1;
    }
    if (st.nin == 1) n.x1 = nullptr;
    n.y = at(st.kind[2], st.ref[2]);
    n.yw = wide(st.kind[2], st.ref[2]);
    // a value that only this program reads is kept in the wider type alone
    if (which == TINY_FWD && n.yw) {
      const int up = p->nodes[st.ref[2]].parent;
      if (up >= 0 && p->nodes[up].tiny && (up != root || count == steps.size())) n.y = nullptr;
    }
  }
  return cuda_err(launch_tiny(p->dt, nodes.data(), prog->level.data(), (int)count, p->fixed_sums, s), "tiny program");
}

// The forward values of every node but the root: the tiny program, then the
// other nodes in post-order.  y: the tree's output if its value goes there as
// it is; *rooted = true if the program has put it there.
int run_forward(ome_ctx* ctx, ome_plan* p, cudaStream_t s, int which, const Leaves& inputs,
                const std::vector<int64_t>& fix, size_t scratch, char* y, bool* rooted, bool* programmed) {
  const bool sliced = which == TINY_FWD && !p->sliced.empty(), keep = which != TINY_FWD;
  static const std::vector<int32_t> none;
  static const std::vector<int64_t> nofix;
  const Scalar one = scalar_one(p->dt), zero = scalar_zero(p->dt);
  const int root = (int)p->nodes.size() - 1;
  bool done = false;
  int rc = run_tiny(ctx, p, s, which, inputs, fix, y, nullptr, nullptr, true, &done);
  *programmed = done;
  if (rc) return rc;
  *rooted = done && y && !p->steps[which].empty() && p->steps[which].back().kind[2] == TinyStep::OUTPUT;
  auto one_node = [&](int j) {
    const PNode& n = p->nodes[j];
    HView v = make_view(p, ctx->ws + (keep ? n.off_keep : n.off_fwd), sliced ? n.iy_s : n.iy, none, nofix);
    return run_node(ctx, p, s, j, inputs, sliced, fix, keep ? off_keep_of : off_fwd_of, v, one, zero, scratch);
  };
  for (int pass = done ? 1 : 0; pass < 2; ++pass)
    for (int j = 0; j < root; ++j) {
      const bool tiny = keep ? p->nodes[j].tiny_full : p->nodes[j].tiny;
      if (tiny != (pass == 0)) continue;
      rc = one_node(j);
      if (rc) return rc;
    }
  return OME_OK;
}


// Slices [b, e) of the tree, each root result added at its sliced output
// positions: into the F64/C64 buffer `acc` for acc64 plans (the root goes to
// the temporary first), else straight into the plan-dtype output `acc` with
// root scale sx and sy = one (the caller initialised or prescaled it).
int run_slices(ome_ctx* ctx, ome_plan* p, cudaStream_t s, const Leaves& inputs, int64_t b, int64_t e,
               char* acc, const Scalar& sx) {
  const ome_dtype dt = p->dt;
  struct Fixed {   // (see run_binary)
    ome_ctx* c;
    Fixed(ome_ctx* ctx, bool on) : c(ctx) { c->fixed_sums = on; }
    ~Fixed() { c->fixed_sums = false; }
  } fixed(ctx, p->fixed_sums);
  const Scalar one = scalar_one(dt), zero = scalar_zero(dt);
  const int root = (int)p->nodes.size() - 1;
  const PNode& rn = p->nodes[root];
  const size_t scratch = (p->arena_bytes + 255) & ~(size_t)255;
  static const std::vector<int32_t> none;
  static const std::vector<int64_t> nofix;
  std::vector<int64_t> fix(p->sliced.size(), 0);
  for (int64_t sl = b; sl < e; ++sl) {
    int64_t r = sl;
    for (size_t i = 0; i < p->sliced.size(); ++i) {
      const int64_t ext = p->ext[p->sliced[i]];
      fix[i] = r % ext;
      r /= ext;
    }
    bool rooted, programmed;
    int rc = run_forward(ctx, p, s, TINY_FWD, inputs, fix, scratch, nullptr, &rooted, &programmed);
    if (rc) return rc;
    if (p->acc64) {
      HView tv = make_view(p, ctx->ws + p->tmp_off, rn.iy_s, none, nofix);
      rc = run_node(ctx, p, s, root, inputs, true, fix, off_fwd_of, tv, one, zero, scratch);
      if (rc) return rc;
      // acc[slice positions] += temp
      const size_t w = dt == OME_C32 ? 16 : 8;
      HView av = make_view(p, acc, rn.iy, p->sliced, fix);
      // the accumulator view has element size w: rescale its base offset
      const int64_t eoff = (av.data - acc) / (int64_t)p->esize;
      char* abase = acc + eoff * (int64_t)w;
      rc = cuda_err(launch_acc64_strided(dt, abase, tv.data, av.nd, av.ext, av.str, s), "acc64");
      if (rc) return rc;
    } else {
      HView yv = make_view(p, acc, rn.iy, p->sliced, fix);
      rc = run_node(ctx, p, s, root, inputs, true, fix, off_fwd_of, yv, sx, one, scratch);
      if (rc) return rc;
    }
  }
  return OME_OK;
}

// The context above the wide plan's buffers.
struct WideCtx {
  ome_ctx* outer;
  ome_ctx inner;
  WideCtx(ome_ctx* c, const ome_plan* p) : outer(c), inner(*c) {
    inner.ws += p->wide_base;
    inner.ws_bytes -= p->wide_base;
  }
  ~WideCtx() {   // the overflow scratch may have grown
    outer->ovf = inner.ovf;
    outer->ovf_bytes = inner.ovf_bytes;
  }
};

// The inputs in the wider type, at wide_in; *done = false if their strides do
// not fit a program.
int widen_inputs(ome_ctx* ctx, ome_plan* p, cudaStream_t s, const Leaves& in, std::vector<const void*>& out,
                 bool* done) {
  auto prog = tiny_program(p, TINY_WIDEN, in);
  *done = prog->ok;
  if (!prog->ok) return OME_OK;
  std::vector<TinyNode> nodes(prog->nodes);
  out.resize(p->ninputs);
  for (int t = 0; t < p->ninputs; ++t) {
    out[t] = ctx->ws + p->wide_in[t];
    nodes[t].x0 = in.data[t];
    nodes[t].yw = ctx->ws + p->wide_in[t];
  }
  return cuda_err(launch_tiny(p->dt, nodes.data(), prog->level.data(), (int)nodes.size(), false, s), "inputs to Float64");
}

}  // namespace

extern "C" {

int ome_plan_execute(ome_ctx* ctx, ome_plan* p, void* stream, const void* const* inputs, void* y, const void* sxp,
                     const void* syp) {
  return ome_plan_execute_strided(ctx, p, stream, inputs, nullptr, y, sxp, syp);
}

int ome_plan_execute_strided(ome_ctx* ctx, ome_plan* p, void* stream, const void* const* in_data,
                             const int64_t* in_strides, void* y, const void* sxp, const void* syp) {
  if (!ctx || !p || !in_data || !y || !sxp || !syp) return set_err(OME_INVALID_ARGUMENT, "NULL argument");
  const Leaves inputs{in_data, in_strides};
  if (ctx->ws_bytes < p->fwd_bytes)
    return set_err(OME_OUT_OF_MEMORY, "plan needs %zu workspace bytes, context has %zu", p->fwd_bytes, ctx->ws_bytes);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const ome_dtype dt = p->dt;
  const Scalar sx = scalar_from(dt, sxp), sy = scalar_from(dt, syp);
  if (p->wide && ctx->ws_bytes >= p->fwd_peak) {
    std::vector<const void*> win;
    bool done;
    int rc = widen_inputs(ctx, p, s, inputs, win, &done);
    if (rc) return rc;
    if (done) {
      const ome_dtype wt = p->wide->dt;
      const Scalar one = scalar_one(wt), zero = scalar_zero(wt);
      WideCtx wc(ctx, p);
      rc = ome_plan_execute(&wc.inner, p->wide.get(), stream, win.data(), ctx->ws + p->wide_y, one.b, zero.b);
      if (rc) return rc;
      return cuda_err(launch_acc64_store(dt, y, ctx->ws + p->wide_y, p->nodes.back().numel, sx, sy,
                                         scalar_is_zero(dt, sy), s), "output from Float64");
    }
  }
  const Scalar one = scalar_one(dt), zero = scalar_zero(dt);
  const int root = (int)p->nodes.size() - 1;
  const PNode& rn = p->nodes[root];
  const size_t scratch = (p->arena_bytes + 255) & ~(size_t)255;
  static const std::vector<int32_t> none;
  static const std::vector<int64_t> nofix;

  if (p->sliced.empty()) {
    bool rooted, programmed;
    const bool plain = scalar_is_one(dt, sx) && scalar_is_zero(dt, sy);
    int rc = run_forward(ctx, p, s, TINY_FWD, inputs, nofix, scratch, plain ? (char*)y : nullptr, &rooted, &programmed);
    if (rc || rooted) return rc;
    HView yv = make_view(p, (char*)y, rn.iy, none, nofix);
    return run_node(ctx, p, s, root, inputs, false, nofix, off_fwd_of, yv, sx, sy, scratch);
  }

  // sliced: y <- sy*y first unless accumulating in FP64
  HView yfull = make_view(p, (char*)y, rn.iy, none, nofix);
  if (p->acc64) {
    const size_t w = dt == OME_C32 ? 16 : 8;
    int rc = cuda_err(cudaMemsetAsync(ctx->ws + p->acc_off, 0, (size_t)rn.numel * w, s), "memset");
    if (rc) return rc;
  } else {
    const bool syz = scalar_is_zero(dt, sy);
    if (!(scalar_is_one(dt, sy))) {
      int rc = cuda_err(launch_scale(dt, y, yfull.nd, yfull.ext, yfull.str, sy, syz, ctx->num_sms, s), "scale");
      if (rc) return rc;
    }
  }
  int rc = run_slices(ctx, p, s, inputs, 0, p->nslices, p->acc64 ? ctx->ws + p->acc_off : (char*)y, sx);
  if (rc) return rc;
  if (p->acc64) {
    return cuda_err(launch_acc64_store(dt, y, ctx->ws + p->acc_off, rn.numel, sx, sy, scalar_is_zero(dt, sy), s),
                    "acc64 store");
  }
  return OME_OK;
}

int ome_plan_slice_count(const ome_plan* p, int64_t* nslices) {
  if (!p || !nslices) return set_err(OME_INVALID_ARGUMENT, "NULL argument");
  *nslices = p->nslices;
  return OME_OK;
}

int ome_plan_partial_info(const ome_plan* p, int* partial_dtype, size_t* partial_bytes, int* reduce_op) {
  if (!p) return set_err(OME_INVALID_ARGUMENT, "plan is NULL");
  const int root = (int)p->nodes.size() - 1;
  const int64_t n = p->nodes[root].numel;
  ome_dtype pd = p->dt;
  if (p->acc64) pd = p->dt == OME_C32 ? OME_C64 : OME_F64;
  if (partial_dtype) *partial_dtype = (int)pd;
  if (partial_bytes) *partial_bytes = (size_t)n * dtype_size(pd);
  if (reduce_op) *reduce_op = (p->dt == OME_BOOL || p->dt == OME_TROP_F32 || p->dt == OME_TROP_F64) ? 1 : 0;
  return OME_OK;
}

int ome_plan_execute_slices(ome_ctx* ctx, ome_plan* p, void* stream, const void* const* inputs,
                            int64_t slice_begin, int64_t slice_end, void* partial) {
  if (!ctx || !p || !inputs || !partial) return set_err(OME_INVALID_ARGUMENT, "NULL argument");
  if (slice_begin < 0 || slice_end < slice_begin || slice_end > p->nslices)
    return set_err(OME_INVALID_ARGUMENT, "slice range [%lld, %lld) outside [0, %lld)", (long long)slice_begin,
                   (long long)slice_end, (long long)p->nslices);
  if (ctx->ws_bytes < p->fwd_bytes)
    return set_err(OME_OUT_OF_MEMORY, "plan needs %zu workspace bytes, context has %zu", p->fwd_bytes, ctx->ws_bytes);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int root = (int)p->nodes.size() - 1;
  const PNode& rn = p->nodes[root];
  if (p->wide && slice_end > slice_begin)   // (unsliced: the one slice is the whole tree)
    return ome_plan_execute(ctx, p, stream, inputs, partial, scalar_one(p->dt).b, scalar_zero(p->dt).b);
  if (p->acc64) {
    const size_t w = p->dt == OME_C32 ? 16 : 8;
    int rc = cuda_err(cudaMemsetAsync(partial, 0, (size_t)rn.numel * w, s), "memset");
    if (rc) return rc;
  } else {
    static const std::vector<int32_t> none;
    static const std::vector<int64_t> nofix;
    HView pv = make_view(p, (char*)partial, rn.iy, none, nofix);
    int rc = cuda_err(launch_scale(p->dt, partial, pv.nd, pv.ext, pv.str, scalar_zero(p->dt), 1, ctx->num_sms, s),
                      "fill");
    if (rc) return rc;
  }
  return run_slices(ctx, p, s, Leaves{inputs, nullptr}, slice_begin, slice_end, (char*)partial, scalar_one(p->dt));
}

int ome_plan_finish(ome_ctx* ctx, ome_plan* p, void* stream, const void* partial, void* y, const void* sxp,
                    const void* syp) {
  if (!ctx || !p || !partial || !y || !sxp || !syp) return set_err(OME_INVALID_ARGUMENT, "NULL argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const ome_dtype dt = p->dt;
  const Scalar sx = scalar_from(dt, sxp), sy = scalar_from(dt, syp);
  const int root = (int)p->nodes.size() - 1;
  const PNode& rn = p->nodes[root];
  if (p->acc64)
    return cuda_err(launch_acc64_store(dt, y, partial, rn.numel, sx, sy, scalar_is_zero(dt, sy), s), "acc64 store");
  static const std::vector<int32_t> none;
  static const std::vector<int64_t> nofix;
  HView xv = make_view(p, (char*)partial, rn.iy, none, nofix);
  HView yv = make_view(p, (char*)y, rn.iy, none, nofix);
  ctx->ws_top = 0;
  return einsum_views(ctx, s, dt, 1, &xv, yv, sx, sy, p->prec, false);
}

}  // extern "C"

namespace ome {
cudaError_t launch_conj(ome_dtype dt, void* x, int64_t n, cudaStream_t s);
cudaError_t launch_fill_one(ome_dtype dt, void* x, int64_t n, cudaStream_t s);
ome_dtype plan_dtype(const ome_plan* p) { return p->dt; }
int plan_ninputs(const ome_plan* p) { return p->ninputs; }
}

extern "C" {

int ome_plan_gradient(ome_ctx* ctx, ome_plan* p, void* stream, const void* const* inputs, const void* dy, void* y,
                      void* const* dxs) {
  return ome_plan_gradient_strided(ctx, p, stream, inputs, nullptr, dy, y, dxs);
}

int ome_plan_gradient_strided(ome_ctx* ctx, ome_plan* p, void* stream, const void* const* in_data,
                              const int64_t* in_strides, const void* dy, void* y, void* const* dxs) {
  if (!ctx || !p || !in_data || !y || !dxs) return set_err(OME_INVALID_ARGUMENT, "NULL argument");
  const Leaves inputs{in_data, in_strides};
  if (ctx->ws_bytes < p->grad_bytes)
    return set_err(OME_OUT_OF_MEMORY, "gradient needs %zu workspace bytes, context has %zu", p->grad_bytes,
                   ctx->ws_bytes);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const ome_dtype dt = p->dt;
  const bool cplx = dt == OME_C32 || dt == OME_C64;
  const Scalar one = scalar_one(dt), zero = scalar_zero(dt);
  const int root = (int)p->nodes.size() - 1;
  const PNode& rn = p->nodes[root];
  if (p->wide && ctx->ws_bytes >= p->grad_peak) {
    std::vector<const void*> win;
    bool done;
    int rc = widen_inputs(ctx, p, s, inputs, win, &done);
    if (rc) return rc;
    if (done) {
      if (dy) {
        if (dt == OME_F32) rc = cuda_err(cudaMemsetAsync(ctx->ws + p->wide_dy, 0, (size_t)rn.numel * 8, s), "memset");
        else rc = cuda_err(cudaMemsetAsync(ctx->ws + p->wide_dy, 0, (size_t)rn.numel * 16, s), "memset");
        if (!rc) rc = cuda_err(launch_acc64(dt, ctx->ws + p->wide_dy, dy, rn.numel, s), "cotangent to Float64");
        if (rc) return rc;
      }
      std::vector<void*> wdx(p->ninputs);
      for (int t = 0; t < p->ninputs; ++t) wdx[t] = ctx->ws + p->wide_dx[t];
      WideCtx wc(ctx, p);
      rc = ome_plan_gradient(&wc.inner, p->wide.get(), stream, win.data(), dy ? ctx->ws + p->wide_dy : nullptr,
                             ctx->ws + p->wide_y, wdx.data());
      if (rc) return rc;
      auto prog = tiny_program(p, TINY_NARROW, Leaves{nullptr, nullptr});
      std::vector<TinyNode> nodes(prog->nodes);
      for (int t = 0; t < p->ninputs; ++t) {
        nodes[t].x0 = wdx[t];
        nodes[t].flags |= TINY_WIDE0;
        nodes[t].y = dxs[t];
      }
      rc = cuda_err(launch_tiny(dt, nodes.data(), prog->level.data(), (int)nodes.size(), false, s), "gradients from Float64");
      if (rc) return rc;
      return cuda_err(launch_acc64_store(dt, y, ctx->ws + p->wide_y, rn.numel, one, zero, 1, s), "output from Float64");
    }
  }
  static const std::vector<int32_t> none;
  static const std::vector<int64_t> nofix;
  const size_t scratch = (p->grad_arena + 255) & ~(size_t)255;
  // forward, every value kept
  bool rooted, programmed;
  int rc = run_forward(ctx, p, s, TINY_FWD_FULL, inputs, nofix, scratch, (char*)y, &rooted, &programmed);
  if (rc) return rc;
  HView yv = make_view(p, (char*)y, rn.iy, none, nofix);
  if (!rooted) rc = run_node(ctx, p, s, root, inputs, false, nofix, off_keep_of, yv, one, zero, scratch);
  if (rc) return rc;
  // root cotangent: ones (init_gradient, src/bp.jl:133-138) or the caller's dy
  char* dy_root;
  ctx->ws_top = scratch;
  dy_root = ctx->ws + p->dy_off;
  if (dy) {
    rc = cuda_err(cudaMemcpyAsync(dy_root, dy, (size_t)rn.numel * p->esize, cudaMemcpyDeviceToDevice, s), "copy dy");
    if (rc) return rc;
  } else {
    if (rn.numel != 1) return set_err(OME_INVALID_ARGUMENT, "The output must be a scalar! Or you need to feed the gradient manually.");
    rc = cuda_err(launch_fill_one(dt, dy_root, 1, s), "fill");
    if (rc) return rc;
  }
  const size_t scratch2 = ctx->ws_top;
  // reverse sweep: the steps above, then the tiny program of the steps below
  // (all in node order if its descriptors do not fit the input strides)
  bool tiny = !p->steps[TINY_REV].empty() && tiny_program(p, TINY_REV, inputs)->ok;
  for (int j = root; j >= 0; --j) {
    const PNode& n = p->nodes[j];
    char* gj = j == root ? dy_root : ctx->ws + n.off_grad;
    // conj(dy) in place (complex): gradients are conj(einsum(.., conj(dy), ..))
    const int nin = (int)n.args.size();
    for (int i = 0; i < nin; ++i) {
      if (tiny && p->rev_tiny[j][i]) continue;
      HView xs[MAXIN];
      for (int a = 0; a < nin; ++a) {
        const int r = n.args[a];
        if (a == i) {
          xs[a] = make_view(p, gj, n.iy, none, nofix);
        } else if (r >= 0) {
          xs[a] = make_view(p, ctx->ws + p->nodes[r].off_keep, p->nodes[r].iy, none, nofix);
        } else {
          xs[a] = leaf_view(p, inputs, -r - 1, none, nofix);
        }
      }
      const int r = n.args[i];
      char* dst = r >= 0 ? ctx->ws + p->nodes[r].off_grad : (char*)dxs[-r - 1];
      const std::vector<int32_t>& labs = r >= 0 ? p->nodes[r].iy : p->in_labels[-r - 1];
      const int64_t cnt = r >= 0 ? p->nodes[r].numel : [&] {
        int64_t c = 1;
        for (int32_t l : labs) c *= p->ext[l];
        return c;
      }();
      HView dv = make_view(p, dst, labs, none, nofix);
      if (cplx) {
        rc = cuda_err(launch_conj(dt, gj, j == root ? rn.numel : n.numel, s), "conj");
        if (rc) return rc;
      }
      ctx->ws_top = scratch2;
      rc = einsum_views(ctx, s, dt, nin, xs, dv, one, zero, p->prec, false);
      if (rc) return rc;
      if (cplx) {
        rc = cuda_err(launch_conj(dt, gj, j == root ? rn.numel : n.numel, s), "conj");
        if (rc) return rc;
        rc = cuda_err(launch_conj(dt, dst, cnt, s), "conj");
        if (rc) return rc;
      }
    }
  }
  if (tiny) return run_tiny(ctx, p, s, TINY_REV, inputs, nofix, nullptr, dy_root, dxs, programmed, &tiny);
  return OME_OK;
}

}  // extern "C"
