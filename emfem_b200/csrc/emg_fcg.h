// Batched flexible CG in FP64 (emg_fcg.cu).
#pragma once

#include <cstdint>
#include <functional>
#include <map>
#include <utility>
#include <vector>

#include "emg_internal.h"
#include "emg_linalg.h"

namespace emg {

// one pinned host word (move-only)
struct PinnedWord {
  int *p = nullptr;
  PinnedWord() = default;
  PinnedWord(const PinnedWord &) = delete;
  PinnedWord &operator=(const PinnedWord &) = delete;
  PinnedWord(PinnedWord &&o) noexcept : p(o.p) { o.p = nullptr; }
  PinnedWord &operator=(PinnedWord &&o) noexcept {
    if (this != &o) {
      release();
      p = o.p;
      o.p = nullptr;
    }
    return *this;
  }
  ~PinnedWord() { release(); }
  void release() {
    if (p) cudaFreeHost(p);
    p = nullptr;
  }
};

// CUDA graphs of whole iterations, valid for one signature (every address and
// size they were captured with)
struct IterGraphs {
  std::vector<uint64_t> sig;
  bool warm = false;  // one iteration has run eagerly under this signature
  std::map<int, std::pair<cudaGraphExec_t, long>> exec;  // (head, directions) -> graph, kernels
  IterGraphs() = default;
  IterGraphs(const IterGraphs &) = delete;
  IterGraphs &operator=(const IterGraphs &) = delete;
  ~IterGraphs() { clear(); }
  void clear() {
    for (auto &kv : exec) cudaGraphExecDestroy(kv.second.first);
    exec.clear();
    warm = false;
  }
};

// What the preconditioner takes from the FCG besides r: an FP32 copy of the
// residual, and the first zero-guess smoothing step of its edge level
// (RestrictJ0 in either precision; y null: none)
struct FcgFeed {
  float *r32 = nullptr;
  RestrictJ0<float> jf{};
  RestrictJ0<double> jd{};
};

// batched FCG on B(w_c) with AMS, K real columns; returns per-column iteration
// counts; x starts at zero.  Columns converge independently to
// ||r_c|| <= rtol ||b_c|| (unpreconditioned norm, src/em_la.cc:120).
struct Fcg {
  static constexpr int kMaxDirs = 30;
  int K = 0;
  int mmax = 1;
  DBuf<double> r, z;
  std::vector<DBuf<double>> P, S;  // previous directions and B-products (ring)
  DBuf<double> acc;                // sums in progress: mmax K (z, S_j), K (p, s), K (p, r), K (r, r), K (b, b)
  DBuf<double> eta, alpha, bn;  // eta: (p, s) of the ring
  DBuf<double *> xslot;            // where the running solve's x lies (graphs outlive a solve)
  DBuf<int> act, itsd, status;     // per-column activity and iteration counts; active count, NaN flag
  DBuf<unsigned> count;            // blocks done per reducing kernel
  PinnedWord h_status;             // two words (see fcg_update_kernel)
  IterGraphs graphs;
  std::vector<int> its;
  long total_its = 0;
  int verbose = 0;
  int check_every = 1;     // iterations between host looks at the column status
  // zs: the preconditioner leaves z split as x + G phi in FP32 (zs->x, zs->phi
  // over the edges zs->edges) instead of writing z; the dot products and the
  // direction then form z on the fly
  struct ZSplit {
    const int *edges;
    const float *x, *phi;
  };
  // pc(r, z) applies the preconditioner, opB(p, s) the operator; n rows, Kc
  // columns (even).  sig: every address and version pc and opB depend on;
  // with it, each kind of iteration is captured once into a CUDA graph and
  // replayed (one launch instead of some 20 to 250); empty: no graphs.
  int solve(int n, int Kc, const std::function<void(const double *, double *)> &pc,
            const std::function<void(const double *, double *)> &opB, const double *b, double *x, double rtol,
            int maxit, cudaStream_t s, const FcgFeed &feed = FcgFeed{}, const ZSplit *zs = nullptr,
            const std::vector<uint64_t> &sig = {});
};

}  // namespace emg
