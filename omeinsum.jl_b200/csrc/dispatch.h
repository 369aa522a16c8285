// Host-side einsum dispatch shared by the single-call API and the plan
// executor: labelled strided views, diagonal (repeated-label) views, label
// classification and mode sorting/merging.
#pragma once
#include <algorithm>
#include <string>
#include <vector>
#include "kernels.h"

struct ome_ctx {
  int device;
  int num_sms;
  char* ws;          // device workspace (plan intermediates, scratch)
  size_t ws_bytes;
  size_t ws_top;     // bump pointer; reset by every top-level call
  char* ovf;         // operand scratch of packed GEMMs that do not fit the workspace
  size_t ovf_bytes;  // (grown on demand outside stream capture; freed with the context)
  bool fixed_sums;   // the nodes of a sliced Float32 tree are being evaluated (see run_binary)
};

namespace ome {

// A labelled strided tensor on the host side of the ABI.
struct HView {
  char* data = nullptr;
  int nd = 0;
  int64_t ext[MAXD];
  int64_t str[MAXD];
  int32_t lab[MAXD];
};

inline int find_lab(const HView& v, int32_t l) {
  for (int d = 0; d < v.nd; ++d)
    if (v.lab[d] == l) return d;
  return -1;
}

// Mode table: one row per label, one stride column per tensor.
struct Modes {
  int n = 0, nt = 0;
  int64_t ext[2 * MAXD];
  int64_t str[MAXIN + 1][2 * MAXD];

  void add(int64_t e, const int64_t* s) {
    ext[n] = e;
    for (int t = 0; t < nt; ++t) str[t][n] = s[t];
    n++;
  }
  int64_t total() const {
    int64_t p = 1;
    for (int i = 0; i < n; ++i) p *= ext[i];
    return p;
  }
  // Drop unit modes; stable sort by |stride of tensor key| (zero strides last);
  // merge neighbours whose strides are consistent in every tensor.
  void normalize(int key) {
    int w = 0;
    for (int i = 0; i < n; ++i) {
      if (ext[i] == 1) continue;
      ext[w] = ext[i];
      for (int t = 0; t < nt; ++t) str[t][w] = str[t][i];
      w++;
    }
    n = w;
    std::vector<int> idx(n);
    for (int i = 0; i < n; ++i) idx[i] = i;
    auto k = [&](int i) -> uint64_t {
      int64_t s = str[key][i];
      if (s == 0) return ~0ull;
      return (uint64_t)(s < 0 ? -s : s);
    };
    std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return k(a) < k(b); });
    int64_t e2[2 * MAXD], s2[MAXIN + 1][2 * MAXD];
    for (int i = 0; i < n; ++i) {
      e2[i] = ext[idx[i]];
      for (int t = 0; t < nt; ++t) s2[t][i] = str[t][idx[i]];
    }
    int m = 0;
    for (int i = 0; i < n; ++i) {
      if (m > 0) {
        bool ok = true;
        for (int t = 0; t < nt && ok; ++t) ok = s2[t][i] == str[t][m - 1] * ext[m - 1];
        if (ok) {
          ext[m - 1] *= e2[i];
          continue;
        }
      }
      ext[m] = e2[i];
      for (int t = 0; t < nt; ++t) str[t][m] = s2[t][i];
      m++;
    }
    n = m;
  }
};

int set_err(int code, const char* fmt, ...);
int cuda_err(cudaError_t e, const char* what);

int view_from_tensor(const ome_tensor& t, HView& v, const char* what);
// Repeated labels -> one dimension with the summed stride (diagonal view).
int unique_view(const HView& v, HView& u);

void* ws_alloc(ome_ctx* c, size_t bytes);

// y <- sy*y + sx*f(xs) for labelled views (any number of inputs).
// loop_only forces the generic index kernel.
int einsum_views(ome_ctx* ctx, cudaStream_t s, ome_dtype dt, int nin, const HView* xs,
                 const HView& y, const Scalar& sx, const Scalar& sy, int prec, bool loop_only);

// Scalar helpers in the algebra of dt.
bool scalar_is_zero(ome_dtype dt, const Scalar& v);
bool scalar_is_one(ome_dtype dt, const Scalar& v);
Scalar scalar_one(ome_dtype dt);
Scalar scalar_zero(ome_dtype dt);
Scalar scalar_from(ome_dtype dt, const void* p);

// A plan's element type and number of inputs (plan.cu).
ome_dtype plan_dtype(const ome_plan* p);
int plan_ninputs(const ome_plan* p);

}  // namespace ome
