// Batched linear-algebra kernels, their launchers and the SpMM autotuner.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <sstream>
#include <vector>

#include "emg_linalg.h"

namespace emg {

// ---------------------------------------------------------------------------
// SpMM dispatch and autotuning
// ---------------------------------------------------------------------------
using SpmmFn = void (*)(const SpmmArgs &, cudaStream_t);

template <typename T, int K, int V, int NL>
constexpr bool spmm_legal() {
  return (K % V) == 0 && (K / V) * NL <= 32 && (32 % ((K / V) * NL)) == 0 && sizeof(T) * V <= 16;
}

template <typename T, int K, int V, int NL, bool PK = false, int MINB = 1, int U = 4, bool LATE = false>
void spmm_launch(const SpmmArgs &a, cudaStream_t s) {
  constexpr int G = NL * (K / V);
  constexpr int RPW = 32 / G;
  long warps = ((long)a.n + RPW - 1) / RPW;
  long threads = warps * 32;
  unsigned grid = (unsigned)((threads + 255) / 256);
  if (grid == 0) return;
  launch_chain(&spmm_kernel<T, K, V, NL, PK, MINB, U, LATE>, grid, 256, s, a.chained, a);
}

// register-capped row-split kernel (nl = 400 + NL packed records, 500 + NL
// index and value arrays): 4 blocks of 256 threads per SM; K >= 16 (packed
// records: FP32 only)
template <typename T, int K, int V, int NL, bool PK>
SpmmFn spmm_pick_capped() {
  if constexpr (spmm_legal<T, K, V, NL>() && (sizeof(T) == 4 || !PK) && K >= 16)
    return &spmm_launch<T, K, V, NL, PK, 4>;
  else return nullptr;
}

// nl = 800 + NL: 6 blocks per SM, 2 nonzeros per round, late epilogue loads;
// whole 16-byte vectors only
template <typename T, int K, int V, int NL>
SpmmFn spmm_pick_dense() {
  if constexpr (spmm_legal<T, K, V, NL>() && sizeof(T) * V == 16 && K >= 8)
    return &spmm_launch<T, K, V, NL, false, 6, 2, true>;
  else return nullptr;
}

// row-group kernel (spmm_rows_kernel): nl = -B selects it with B gathers in
// flight per lane
template <typename T, int K, int V, int B>
constexpr bool spmm_rows_legal() {
  return (K % V) == 0 && (K / V) <= 32 && (32 % (K / V)) == 0 && ((K / V) % B) == 0 && sizeof(T) * V <= 16;
}

template <typename T, int K, int V, int B>
void spmm_rows_launch(const SpmmArgs &a, cudaStream_t s) {
  constexpr int RPW = 32 / (K / V);
  long warps = ((long)a.n + RPW - 1) / RPW;
  unsigned grid = (unsigned)((warps * 32 + 255) / 256);
  if (grid == 0) return;
  launch_chain(&spmm_rows_kernel<T, K, V, B>, grid, 256, s, a.chained, a);
}

template <typename T, int K, int V, int B>
SpmmFn spmm_rows_pick() {
  if constexpr (spmm_rows_legal<T, K, V, B>()) return &spmm_rows_launch<T, K, V, B>;
  else return nullptr;
}

// software-pipelined kernel (spmm_pipe_kernel): nl = 200 + U (index and
// value arrays) or 300 + U (packed records, FP32 two-part operators only)
template <typename T, int K, int V, int U, bool PK>
void spmm_pipe_launch(const SpmmArgs &a, cudaStream_t s) {
  constexpr int RPW = 32 / (K / V);
  long warps = ((long)a.n + RPW - 1) / RPW;
  unsigned grid = (unsigned)((warps * 32 + 255) / 256);
  if (grid == 0) return;
  launch_chain(&spmm_pipe_kernel<T, K, V, U, PK>, grid, 256, s, a.chained, a);
}

template <typename T, int K, int V, int U, bool PK>
SpmmFn spmm_pipe_pick() {
  if constexpr (spmm_legal<T, K, V, 1>() && (!PK || sizeof(T) == 4)) return &spmm_pipe_launch<T, K, V, U, PK>;
  else return nullptr;
}

// chunked kernel (spmm_chunk_kernel): nl = 601 (one block per SM minimum),
// 604 (register-capped, 4 blocks per SM); FP32 two-part operators with the
// chunked layout only
template <typename T, int K, int V, int MINB>
void spmm_chunk_launch(const SpmmArgs &a, cudaStream_t s) {
  constexpr int RPW = 32 / (K / V);
  long warps = ((long)a.n + RPW - 1) / RPW;
  unsigned grid = (unsigned)((warps * 32 + 255) / 256);
  if (grid == 0) return;
  launch_chain(&spmm_chunk_kernel<K, V, MINB>, grid, 256, s, a.chained, a);
}

template <typename T, int K, int V, int MINB>
SpmmFn spmm_chunk_pick() {
  if constexpr (spmm_legal<T, K, V, 1>() && sizeof(T) == 4 && K >= 8) return &spmm_chunk_launch<T, K, V, MINB>;
  else return nullptr;
}

// packed-record variant (nl = 100 + NL): FP32 two-part operators only
template <typename T, int K, int V, int NL>
SpmmFn spmm_pick_packed() {
  if constexpr (spmm_legal<T, K, V, NL>() && sizeof(T) == 4) return &spmm_launch<T, K, V, NL, true>;
  else return nullptr;
}

template <typename T, int K, int V, int NL>
SpmmFn spmm_pick() {
  if constexpr (spmm_legal<T, K, V, NL>()) return &spmm_launch<T, K, V, NL>;
  else return nullptr;
}
template <typename T, int K, int V>
SpmmFn spmm_pick_nl(int nl) {
  switch (nl) {
  case -4: return spmm_rows_pick<T, K, V, 4>();
  case -8: return spmm_rows_pick<T, K, V, 8>();
  case 101: return spmm_pick_packed<T, K, V, 1>();
  case 102: return spmm_pick_packed<T, K, V, 2>();
  case 104: return spmm_pick_packed<T, K, V, 4>();
  case 601: return spmm_chunk_pick<T, K, V, 1>();
  case 604: return spmm_chunk_pick<T, K, V, 4>();
  case 801: return spmm_pick_dense<T, K, V, 1>();
  case 802: return spmm_pick_dense<T, K, V, 2>();
  case 401: return spmm_pick_capped<T, K, V, 1, true>();
  case 402: return spmm_pick_capped<T, K, V, 2, true>();
  case 501: return spmm_pick_capped<T, K, V, 1, false>();
  case 502: return spmm_pick_capped<T, K, V, 2, false>();
  case 204: return spmm_pipe_pick<T, K, V, 4, false>();
  case 208: return spmm_pipe_pick<T, K, V, 8, false>();
  case 304: return spmm_pipe_pick<T, K, V, 4, true>();
  case 308: return spmm_pipe_pick<T, K, V, 8, true>();
  case 1: return spmm_pick<T, K, V, 1>();
  case 2: return spmm_pick<T, K, V, 2>();
  case 4: return spmm_pick<T, K, V, 4>();
  case 8: return spmm_pick<T, K, V, 8>();
  case 16: return spmm_pick<T, K, V, 16>();
  case 32: return spmm_pick<T, K, V, 32>();
  }
  return nullptr;
}
template <typename T, int K>
SpmmFn spmm_pick_v(int v, int nl) {
  switch (v) {
  case 1: return spmm_pick_nl<T, K, 1>(nl);
  case 2: return spmm_pick_nl<T, K, 2>(nl);
  case 4: return spmm_pick_nl<T, K, 4>(nl);
  }
  return nullptr;
}
template <typename T>
SpmmFn spmm_fn(int K, int v, int nl) {
  switch (K) {
  case 1: return spmm_pick_v<T, 1>(v, nl);
  case 2: return spmm_pick_v<T, 2>(v, nl);
  case 4: return spmm_pick_v<T, 4>(v, nl);
  case 8: return spmm_pick_v<T, 8>(v, nl);
  case 16: return spmm_pick_v<T, 16>(v, nl);
  case 32: return spmm_pick_v<T, 32>(v, nl);
  case 64: return spmm_pick_v<T, 64>(v, nl);
  }
  return nullptr;
}

SpmmTuner &tuner() {
  static SpmmTuner t;
  return t;
}

bool SpmmTuner::find(const Key &k, Layout &l) {
  std::lock_guard<std::mutex> lock(mu);
  auto it = best.find(k);
  if (it == best.end()) return false;
  l = it->second;
  return true;
}

SpmmTuner::Layout SpmmTuner::add(const Key &k, const Layout &l) {
  std::lock_guard<std::mutex> lock(mu);
  return best.emplace(k, l).first->second;
}

std::string SpmmTuner::report() {
  std::lock_guard<std::mutex> lock(mu);
  std::ostringstream os;
  for (auto &kv : best)
    os << "T" << std::get<0>(kv.first) * 8 << " K" << std::get<1>(kv.first) << " nnz/row class "
       << std::get<2>(kv.first) << " rows class " << (std::get<3>(kv.first) >> 2) << ": V=" << kv.second.first
       << (std::get<3>(kv.first) & 1 ? " (packed records available)" : "")
       << (std::get<3>(kv.first) & 2 ? " (chunks available)" : "")
       << (kv.second.second < 0 ? " rows kernel B="
                                : (kv.second.second > 800   ? " 6 blocks/SM NL="
                                   : kv.second.second > 600 ? " chunked, min blocks/SM "
                                   : kv.second.second > 500 ? " register-capped NL="
                                   : kv.second.second > 400 ? " packed register-capped NL="
                                   : kv.second.second > 300 ? " packed pipelined U="
                                   : kv.second.second > 200 ? " pipelined U="
                                   : kv.second.second > 100 ? " packed NL="
                                                            : " NL="))
       << (kv.second.second > 100 ? kv.second.second % 100 : std::abs(kv.second.second)) << "; ";
  return os.str();
}

static int row_bucket(const SpmmArgs &a, long nnz) {
  double avg = a.n > 0 ? (double)nnz / a.n : 0;
  return avg < 6 ? 0 : (avg < 12 ? 1 : (avg < 24 ? 2 : 3));
}

// row-count class, a factor of two wide: the layout that is fastest at 29000 rows
// of 21 nonzeros (11.9 us, one lane per row) takes 9.0 us at 11000 of 25,
// where two lanes take 7.5
static int size_class(const SpmmArgs &a) {
  int c = 0;
  while ((a.n >> c) > 1) ++c;
  return c;
}

// Layout of an operator whose rows x column lanes leave most of the chip idle
// (a quarter of its threads): the widest vectors, and as many lanes per row
// as bring it down to one round of 4 nonzeros per lane, because there a step
// costs its dependent loads and not its bandwidth.  An operator of 240 rows
// with 30 nonzeros (K = 32) takes 6.5 us this way and 15.7 us with one lane
// per row, the layout that wins at 20000 rows.
constexpr long kLaneSlots = 148L * 512;

template <typename T>
static std::pair<int, int> spmm_default(int K, double avg) {
  int vmax = (int)(16 / sizeof(T));
  int v = 1;
  while (v * 2 <= vmax && K % (v * 2) == 0) v *= 2;
  int cl = K / v;
  while (cl > 32) { v *= 2; cl = K / v; }
  int nl = 1;
  while (nl * 2 * cl <= 32 && nl * 4 < avg) nl *= 2;
  return {v, nl};
}

template <typename T>
void spmm_nnz(int K, const SpmmArgs &a, long nnz, cudaStream_t s) {
  if (a.n <= 0) return;
  SpmmTuner &tn = tuner();
  int bucket = row_bucket(a, nnz);
  const bool packed = a.pk != nullptr && sizeof(T) == 4 && a.vm != nullptr;
  const bool chunked = a.ch != nullptr && a.crp != nullptr && sizeof(T) == 4 && a.vm != nullptr;
  auto key = std::make_tuple((int)sizeof(T), K, bucket, 4 * size_class(a) + (packed ? 1 : 0) + (chunked ? 2 : 0));
  SpmmTuner::Layout cfg = spmm_default<T>(K, (double)nnz / a.n);
  const bool fills = (long)a.n * (K / cfg.first) >= kLaneSlots;
  if (fills && !tn.find(key, cfg)) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    EMG_CUDA(cudaStreamIsCapturing(s, &cs));
    const bool idempotent = a.mode == SPMM_AX || a.mode == SPMM_RES || a.mode == SPMM_JAC || a.mode == SPMM_CHEB1 ||
                            a.mode == SPMM_AXJ0 || a.mode == SPMM_RESJ0;
    if (cs == cudaStreamCaptureStatusNone && idempotent) {
      cudaEvent_t e0, e1;
      EMG_CUDA(cudaEventCreate(&e0));
      EMG_CUDA(cudaEventCreate(&e1));
      // candidates: the row-split, row-group and packed-record kernels.  The
      // software-pipelined kernel (nl 200 + U / 300 + U) is left out: it won
      // the tuning call's mode by a hair on the MT topography edge matrix and
      // then ran 17% slower over the solver's mix of smoothing modes.
      std::vector<SpmmTuner::Layout> cand;
      for (int v : {1, 2, 4})
        for (int nl : {1, 2, 4, 8, 16, 32, -4, -8, 101, 102, 104, 401, 402, 501, 502, 601, 604, 801, 802}) {
          if (((nl > 100 && nl < 200) || (nl > 400 && nl < 500)) && !packed) continue;
          if (nl > 600 && nl < 700 && !chunked) continue;
          if (spmm_fn<T>(K, v, nl)) cand.push_back({v, nl});
        }
      // two interleaved passes, each candidate's best: one slow sample (a
      // clock step, a neighbour's burst) does not decide the layout
      std::vector<float> best_ms(cand.size(), 1e30f);
      for (int pass = 0; pass < 2; ++pass)
        for (size_t i = 0; i < cand.size(); ++i) {
          SpmmFn f = spmm_fn<T>(K, cand[i].first, cand[i].second);
          SpmmArgs ta = a;
          ta.chained = false;
          f(ta, s);  // warm-up
          EMG_CUDA(cudaEventRecord(e0, s));
          for (int r = 0; r < 3; ++r) f(ta, s);
          EMG_CUDA(cudaEventRecord(e1, s));
          EMG_CUDA(cudaEventSynchronize(e1));
          float ms = 0;
          EMG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
          best_ms[i] = std::min(best_ms[i], ms);
        }
      float bestms = 1e30f;
      for (size_t i = 0; i < cand.size(); ++i)
        if (best_ms[i] < bestms) {
          bestms = best_ms[i];
          cfg = cand[i];
        }
      EMG_CUDA(cudaEventDestroy(e0));
      EMG_CUDA(cudaEventDestroy(e1));
      cfg = tn.add(key, cfg);
    }
  }
  SpmmFn f = spmm_fn<T>(K, cfg.first, cfg.second);
  if (!f) fail(EMG_ERR_ARG, "unsupported block width K=%d", K);
  f(a, s);
  EMG_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// tiled SpMM: per-tile column lists, x rows staged in shared memory
// ---------------------------------------------------------------------------
bool build_tiled(int n, const std::vector<int> &rp, const std::vector<int> &ci, int umax_limit, int r_max,
                 TiledPattern &tp, cudaStream_t s) {
  int R = 0, umax = 0;
  std::vector<int> urp, ucol;
  std::vector<unsigned short> lci;
  if (!tile_rows(n, rp, ci, umax_limit, r_max, R, umax, urp, ucol, lci)) return false;
  tp.n = n;
  tp.R = R;
  tp.ntiles = (int)urp.size() - 1;
  tp.umax = umax;
  tp.urp.upload(urp, s);
  tp.ucol.upload(ucol, s);
  tp.lci.upload(lci, s);
  EMG_CUDA(cudaStreamSynchronize(s));  // host arrays go out of scope
  return true;
}

template <typename T, int K, int V>
static void tiled_launch(const SpmmArgs &a, const TiledPattern &tp, cudaStream_t s) {
  static bool attr = false;
  if (!attr) {
    EMG_CUDA(cudaFuncSetAttribute(spmm_tiled_kernel<T, K, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  227 * 1024));
    attr = true;
  }
  const size_t smem = (size_t)tp.umax * K * sizeof(T);
  if (smem > 227 * 1024) fail(EMG_ERR_ARG, "tile needs %zu bytes of shared memory", smem);
  spmm_tiled_kernel<T, K, V><<<tp.ntiles, 256, smem, s>>>(a, TiledArgs{tp.R, tp.urp.p, tp.ucol.p, tp.lci.p});
}

template <typename T>
void spmm_tiled(int K, const SpmmArgs &a, const TiledPattern &tp, cudaStream_t s) {
  if (a.n <= 0) return;
  if (a.n != tp.n) fail(EMG_ERR_STATE, "tiled pattern has %d rows, operator %d", tp.n, a.n);
  constexpr int V0 = (int)(16 / sizeof(T));
  switch (K) {
  case 1: tiled_launch<T, 1, 1>(a, tp, s); break;
  case 2: tiled_launch<T, 2, (V0 < 2 ? V0 : 2)>(a, tp, s); break;
  case 4: tiled_launch<T, 4, (V0 < 4 ? V0 : 4)>(a, tp, s); break;
  case 8: tiled_launch<T, 8, V0>(a, tp, s); break;
  case 16: tiled_launch<T, 16, V0>(a, tp, s); break;
  case 32: tiled_launch<T, 32, V0>(a, tp, s); break;
  case 64: tiled_launch<T, 64, V0>(a, tp, s); break;
  default: fail(EMG_ERR_ARG, "unsupported block width K=%d", K);
  }
  EMG_LAUNCH_CHECK();
}

template void spmm_tiled<float>(int, const SpmmArgs &, const TiledPattern &, cudaStream_t);
template void spmm_tiled<double>(int, const SpmmArgs &, const TiledPattern &, cudaStream_t);

template <typename T>
bool spmm_layout(int K, int v, int nl, const SpmmArgs &a, cudaStream_t s) {
  SpmmFn f = spmm_fn<T>(K, v, nl);
  if (!f) return false;
  const bool packed_variant = (nl > 100 && nl < 200) || (nl > 300 && nl < 400) || (nl > 400 && nl < 500);
  if (packed_variant && (a.pk == nullptr || a.vm == nullptr)) return false;
  if (nl > 600 && nl < 700 && (a.ch == nullptr || a.crp == nullptr || a.vm == nullptr)) return false;
  if (a.n > 0) f(a, s);
  EMG_LAUNCH_CHECK();
  return true;
}
template bool spmm_layout<float>(int, int, int, const SpmmArgs &, cudaStream_t);
template bool spmm_layout<double>(int, int, int, const SpmmArgs &, cudaStream_t);

__global__ void pack_records_kernel(long nnz, const int *__restrict__ ci, const float *__restrict__ vc,
                                    const float *__restrict__ vm, int4 *__restrict__ out) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k < nnz) out[k] = make_int4(ci[k], __float_as_int(vc[k]), __float_as_int(vm[k]), 0);
}

// thread per row: the row's nonzeros into whole chunks of 4 (spmm_chunk_kernel)
__global__ void chunk_records_kernel(int n, const int *__restrict__ rp, const int *__restrict__ ci,
                                     const float *__restrict__ vc, const float *__restrict__ vm,
                                     const int *__restrict__ crp, int4 *__restrict__ ch) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int k0 = rp[r], k1 = rp[r + 1], q0 = crp[r], q1 = crp[r + 1];
  int *out = reinterpret_cast<int *>(ch);
  for (int t = 0; t < 4 * (q1 - q0); ++t) {
    const int k = k0 + t;
    const bool ok = k < k1;
    const long base = 12L * (q0 + t / 4) + (t & 3);
    out[base] = ok ? ci[k] : r;
    out[base + 4] = ok ? __float_as_int(vc[k]) : 0;
    out[base + 8] = ok ? __float_as_int(vm[k]) : 0;
  }
}

long chunk_row_pointer(const std::vector<int> &rp, std::vector<int> &crp) {
  const int n = (int)rp.size() - 1;
  crp.assign(n + 1, 0);
  for (int r = 0; r < n; ++r) crp[r + 1] = crp[r] + (rp[r + 1] - rp[r] + 3) / 4;
  return n >= 0 ? crp[n] : 0;
}

void chunk_records(int n, const int *rp, const int *ci, const float *vc, const float *vm, const int *crp, int4 *ch,
                   cudaStream_t s) {
  if (n <= 0) return;
  chunk_records_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, rp, ci, vc, vm, crp, ch);
  EMG_LAUNCH_CHECK();
}

void pack_records(long nnz, const int *ci, const float *vc, const float *vm, int4 *out, cudaStream_t s) {
  if (nnz <= 0) return;
  pack_records_kernel<<<(unsigned)((nnz + 255) / 256), 256, 0, s>>>(nnz, ci, vc, vm, out);
  EMG_LAUNCH_CHECK();
}

template void spmm_nnz<float>(int, const SpmmArgs &, long, cudaStream_t);
template void spmm_nnz<double>(int, const SpmmArgs &, long, cudaStream_t);

double spmm_algo_bytes(long n, long nnz, int K, int elem, bool two_parts, int mode) {
  double b = (double)nnz * (4.0 + elem * (two_parts ? 2 : 1)) + (double)(n + 1) * 4.0;
  double vec = (double)n * K * elem;
  b += 2.0 * vec;  // x gathered once, y written once
  if (mode == SPMM_RES) b += vec;
  if (mode == SPMM_JAC) b += vec + (double)n * elem * (two_parts ? 2 : 1);
  if (mode == SPMM_ADD) b += vec;
  if (mode == SPMM_CHEB1) b += 3.0 * vec + (double)n * elem * (two_parts ? 2 : 1);   // b, x-row in; r, d out
  if (mode == SPMM_CHEB2) b += 2.0 * vec + (double)n * elem * (two_parts ? 2 : 1);   // r, y-row in
  if (mode == SPMM_CHEBK) b += 4.0 * vec + (double)n * elem * (two_parts ? 2 : 1);   // r, y in; r, d out
  if (mode == SPMM_RESJ0) b += vec;
  if (mode == SPMM_AXJ0 || mode == SPMM_RESJ0) b += 2.0 * vec + (double)n * elem * 2;                      // r, d out; fed diagonal
  return b;
}

// ---------------------------------------------------------------------------
// column reductions and vector updates
// ---------------------------------------------------------------------------
static unsigned red_grid(long total) {
  long g = (total + 255) / 256;
  return (unsigned)std::max(1L, std::min(g, 148L * 8));
}

// columns per vector load of a K-column block row
template <typename T>
static int vec_width(int K) {
  return (K & 3) == 0 && sizeof(T) == 4 ? 4 : ((K & 1) == 0 ? 2 : 1);
}

// y (and d when given) = w b / (l1c + w_c l1m): one thread per V columns of a
// row; the diagonals load before the wait (emg_pdl.cuh)
template <typename T, int V>
__global__ void __launch_bounds__(256) jacobi0_kernel(long total, int cl, const T *b, const T *__restrict__ l1c,
                                                      const T *__restrict__ l1m, const double *__restrict__ omega,
                                                      double w, T *y, T *d) {
  pdl_trigger();
  const long i = blockIdx.x * 256L + threadIdx.x;
  T dg[V];
  if (i < total) {
    const long row = i / cl;
    const int c0 = (int)(i - row * cl) * V;
    const T dc = __ldg(l1c + row), dm = l1m ? __ldg(l1m + row) : T(0);
#pragma unroll
    for (int q = 0; q < V; ++q) dg[q] = l1m ? dc + (T)__ldg(omega + c0 + q) * dm : dc;
  }
  pdl_wait();
  if (i >= total) return;
  T v[V];
  ldv<T, V>(b + i * V, v);
#pragma unroll
  for (int q = 0; q < V; ++q) v[q] = (T)w * v[q] / dg[q];
  stv<T, V>(y + i * V, v);
  if (d) stv<T, V>(d + i * V, v);
}

template <typename T>
void jacobi0(int n, int K, const T *b, const T *l1c, const T *l1m, const double *omega, double w, T *y, T *d,
             cudaStream_t s) {
  if (n <= 0) return;
  const int v = vec_width<T>(K), cl = K / v;
  const long total = (long)n * cl;
  const unsigned grid = (unsigned)((total + 255) / 256);
  if (v == 1) launch_chain(&jacobi0_kernel<T, 1>, grid, 256, s, true, total, cl, b, l1c, l1m, omega, w, y, d);
  else if (v == 2) launch_chain(&jacobi0_kernel<T, 2>, grid, 256, s, true, total, cl, b, l1c, l1m, omega, w, y, d);
  else if constexpr (sizeof(T) == 4)
    launch_chain(&jacobi0_kernel<T, 4>, grid, 256, s, true, total, cl, b, l1c, l1m, omega, w, y, d);
  EMG_LAUNCH_CHECK();
}

__global__ void cvt_d2f_kernel(long n, const double *__restrict__ a, float *__restrict__ b) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}
void cvt_d2f(long count, const double *a, float *b, cudaStream_t s) {
  if (!count) return;
  cvt_d2f_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(count, a, b);
  EMG_LAUNCH_CHECK();
}
template <typename T>
void fill_zero(long count, T *a, cudaStream_t s) {
  if (count) EMG_CUDA(cudaMemsetAsync(a, 0, count * sizeof(T), s));
}

// ---------------------------------------------------------------------------
// AMS transfers
// ---------------------------------------------------------------------------
// One vertex per CL x NL lanes: CL lanes own V columns each, NL lanes split the
// incident edges (about 14 per vertex), U of them per lane and round.  The
// incidence codes and tangents of the first round load before the wait; what
// remains of the chain is one round of gathers.  With y, the first smoothing
// step of the level this right-hand side feeds is taken as well: y = d =
// c1 b / (l1c + w_c l1m), one pass and one launch less per V-cycle.
template <typename T>
struct RestrictArgs {
  int nv, K, sp, cl, nl;
  const int *inc_rp, *inc;
  const T *tangent, *r_edge;
  T *r_vert;
  RestrictJ0<T> j0;
};

template <typename T, int V, int D>
__global__ void __launch_bounds__(256) ams_restrict_kernel(RestrictArgs<T> a) {
  constexpr int U = 4;
  pdl_trigger();
  const int K = a.K, g = a.cl * a.nl;
  const long t = (blockIdx.x * 256L + threadIdx.x) / g;
  const int sub = (int)(threadIdx.x % g), c0 = (sub % a.cl) * V, sl = sub / a.cl;
  const bool valid = t < a.nv;
  const int v = (int)t;
  int k0 = 0, ke = 0;
  if (valid) {
    k0 = __ldg(a.inc_rp + v) + sl;
    ke = __ldg(a.inc_rp + v + 1);
  }
  int e[U];
  T w[U][D];
  auto fetch = [&]() {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u * a.nl;
      const int code = k < ke ? __ldg(a.inc + k) : -1;
      e[u] = code >> 1;  // -1 past the end
      if (code >= 0) {
        if constexpr (D == 3) {
#pragma unroll
          for (int d = 0; d < 3; ++d) w[u][d] = __ldg(a.tangent + 3 * (long)e[u] + d);
        } else if (a.sp == 0) {
          w[u][0] = (code & 1) ? T(1) : T(-1);
        } else {
          w[u][0] = T(0.5) * __ldg(a.tangent + 3 * (long)e[u] + (a.sp - 1));
        }
      }
    }
  };
  fetch();
  pdl_wait();
  T acc[D][V];
#pragma unroll
  for (int d = 0; d < D; ++d)
#pragma unroll
    for (int i = 0; i < V; ++i) acc[d][i] = T(0);
  while (k0 < ke) {
    T r[U][V];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (e[u] >= 0) ldv<T, V>(a.r_edge + (long)e[u] * K + c0, r[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (e[u] >= 0)
#pragma unroll
        for (int i = 0; i < V; ++i)
#pragma unroll
          for (int d = 0; d < D; ++d) acc[d][i] += w[u][d] * (D == 3 ? T(0.5) * r[u][i] : r[u][i]);
    k0 += a.nl * U;
    if (k0 < ke) fetch();
  }
  for (int off = a.cl; off < g; off <<= 1)
#pragma unroll
    for (int d = 0; d < D; ++d)
#pragma unroll
      for (int i = 0; i < V; ++i) acc[d][i] += __shfl_xor_sync(0xffffffffu, acc[d][i], off);
  if (!valid || sl != 0) return;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const long row = (long)D * v + d, o = row * K + c0;
    stv<T, V>(a.r_vert + o, acc[d]);
    if (a.j0.y) {
      const T dc = __ldg(a.j0.l1c + row), dm = a.j0.l1m ? __ldg(a.j0.l1m + row) : T(0);
#pragma unroll
      for (int i = 0; i < V; ++i)
        acc[d][i] = (T)a.j0.c1 * acc[d][i] / (a.j0.l1m ? dc + (T)__ldg(a.j0.omega + c0 + i) * dm : dc);
      stv<T, V>(a.j0.y + o, acc[d]);
      if (a.j0.d) stv<T, V>(a.j0.d + o, acc[d]);
    }
  }
}

template <typename T>
void ams_restrict(int nv, int K, int sp, const int *inc_rp, const int *inc, const T *tangent, const T *r_edge,
                  T *r_vert, cudaStream_t s, const RestrictJ0<T> &j0) {
  if (nv <= 0) return;
  const int v = vec_width<T>(K), cl = K / v;
  // 4 lanes x 4 edges cover the usual vertex in one round
  int nl = 1;
  while (nl < 4 && cl * nl * 2 <= 32) nl *= 2;
  if (cl > 32 || (32 % cl) != 0) fail(EMG_ERR_ARG, "unsupported block width K=%d", K);
  RestrictArgs<T> a{nv, K, sp, cl, nl, inc_rp, inc, tangent, r_edge, r_vert, j0};
  const unsigned grid = (unsigned)(((long)nv * cl * nl + 255) / 256);
  auto run = [&](auto k1, auto k3) { launch_chain(sp == 4 ? k3 : k1, grid, 256, s, true, a); };
  if (v == 1) run(&ams_restrict_kernel<T, 1, 1>, &ams_restrict_kernel<T, 1, 3>);
  else if (v == 2) run(&ams_restrict_kernel<T, 2, 1>, &ams_restrict_kernel<T, 2, 3>);
  else if constexpr (sizeof(T) == 4) run(&ams_restrict_kernel<T, 4, 1>, &ams_restrict_kernel<T, 4, 3>);
  EMG_LAUNCH_CHECK();
}

// x += Q e: one thread per V columns of an edge; end points and tangent load
// before the wait
template <typename T, int V>
__global__ void __launch_bounds__(256) ams_prolong_kernel(int ne, int K, int cl, int sp, const int *__restrict__ edges,
                                                          const T *__restrict__ tangent, const T *ev, T *x) {
  pdl_trigger();
  const long t = blockIdx.x * 256L + threadIdx.x;
  const bool valid = t < (long)ne * cl;
  int2 vv = make_int2(0, 0);
  T tg[3] = {T(0), T(0), T(0)};
  long e = 0;
  if (valid) {
    e = t / cl;
    vv = __ldg(reinterpret_cast<const int2 *>(edges) + e);
    if (sp == 4) {
#pragma unroll
      for (int d = 0; d < 3; ++d) tg[d] = __ldg(tangent + 3 * e + d);
    } else if (sp > 0) {
      tg[0] = __ldg(tangent + 3 * e + (sp - 1));
    }
  }
  pdl_wait();
  if (!valid) return;
  const int c0 = (int)(t - e * cl) * V;
  T xv[V], val[V], a[V], b[V];
  ldv<T, V>(x + e * K + c0, xv);
  if (sp == 4) {  // vector space: rows 3 v + d
#pragma unroll
    for (int i = 0; i < V; ++i) val[i] = T(0);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      ldv<T, V>(ev + (3 * (long)vv.x + d) * K + c0, a);
      ldv<T, V>(ev + (3 * (long)vv.y + d) * K + c0, b);
#pragma unroll
      for (int i = 0; i < V; ++i) val[i] += tg[d] * (a[i] + b[i]);
    }
#pragma unroll
    for (int i = 0; i < V; ++i) val[i] *= T(0.5);
  } else {
    ldv<T, V>(ev + (long)vv.x * K + c0, a);
    ldv<T, V>(ev + (long)vv.y * K + c0, b);
#pragma unroll
    for (int i = 0; i < V; ++i) val[i] = sp == 0 ? b[i] - a[i] : T(0.5) * tg[0] * (a[i] + b[i]);
  }
#pragma unroll
  for (int i = 0; i < V; ++i) xv[i] += val[i];
  stv<T, V>(x + e * K + c0, xv);
}

template <typename T>
void ams_prolong_add(int ne, int K, int sp, const int *edges, const T *tangent, const T *e_vert, T *x_edge,
                     cudaStream_t s) {
  if (ne <= 0) return;
  const int v = vec_width<T>(K), cl = K / v;
  const unsigned grid = (unsigned)(((long)ne * cl + 255) / 256);
  if (v == 1) launch_chain(&ams_prolong_kernel<T, 1>, grid, 256, s, true, ne, K, cl, sp, edges, tangent, e_vert, x_edge);
  else if (v == 2)
    launch_chain(&ams_prolong_kernel<T, 2>, grid, 256, s, true, ne, K, cl, sp, edges, tangent, e_vert, x_edge);
  else if constexpr (sizeof(T) == 4)
    launch_chain(&ams_prolong_kernel<T, 4>, grid, 256, s, true, ne, K, cl, sp, edges, tangent, e_vert, x_edge);
  EMG_LAUNCH_CHECK();
}

// Dense coarsest solve: a warp per row and column pair, its lanes split the
// row of the inverse (coalesced; up to kPre of its elements per lane load
// before the wait), so a row is a handful of loads deep instead of nc.
template <typename T>
__global__ void __launch_bounds__(256) coarse_apply_kernel(int nc, int K, const double *__restrict__ inv,
                                                           const int *__restrict__ slot, const T *b, T *x) {
  constexpr int kPre = 8;
  pdl_trigger();
  const int lane = threadIdx.x & 31, kp = (K + 1) / 2;
  const int t = (int)((blockIdx.x * 256 + threadIdx.x) >> 5);
  if (t >= nc * kp) {
    pdl_wait();
    return;
  }
  const int r = t / kp, c0 = (t - r * kp) * 2;
  const bool pair = c0 + 1 < K;
  const int s0 = __ldg(slot + c0), s1 = pair ? __ldg(slot + c0 + 1) : s0;
  const double *row0 = inv + ((long)s0 * nc + r) * nc, *row1 = inv + ((long)s1 * nc + r) * nc;
  double pre[kPre];
#pragma unroll
  for (int q = 0; q < kPre; ++q) pre[q] = lane + 32 * q < nc ? __ldg(row0 + lane + 32 * q) : 0.0;
  pdl_wait();
  double a0 = 0, a1 = 0;
  auto add = [&](int j, double w0) {
    const double w1 = s1 == s0 ? w0 : __ldg(row1 + j);
    a0 += w0 * (double)b[(long)j * K + c0];
    if (pair) a1 += w1 * (double)b[(long)j * K + c0 + 1];
  };
#pragma unroll
  for (int q = 0; q < kPre; ++q)
    if (lane + 32 * q < nc) add(lane + 32 * q, pre[q]);
  for (int j = lane + 32 * kPre; j < nc; j += 32) add(j, __ldg(row0 + j));
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    a0 += __shfl_xor_sync(0xffffffffu, a0, off);
    a1 += __shfl_xor_sync(0xffffffffu, a1, off);
  }
  if (lane == 0) {
    x[(long)r * K + c0] = (T)a0;
    if (pair) x[(long)r * K + c0 + 1] = (T)a1;
  }
}

template <typename T>
void coarse_apply(int nc, int K, const double *inv, const int *col_slot, const T *b, T *x, cudaStream_t s) {
  if (nc <= 0) return;
  const long warps = (long)nc * ((K + 1) / 2);
  launch_chain(&coarse_apply_kernel<T>, (unsigned)((warps * 32 + 255) / 256), 256, s, true, nc, K, inv, col_slot, b, x);
  EMG_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// complex FP64 kernels of the outer FGMRES
// ---------------------------------------------------------------------------
// column frequencies as a kernel argument
struct Omegas {
  double w[32];
};

// y = A(w_c) x or b - A(w_c) x: CL = K / V lanes of V columns per row, NL lanes
// splitting its nonzeros, U nonzeros per lane and round; the index and value
// loads of a round go out before its gathers.  L1 is the busiest unit
// (64 % at K = 16, 357k rows, its data pipe 62 %; L2 20 %, DRAM 23 %): a
// warp-wide load that touches several rows costs a pass per row, so few lanes per
// row with two columns each share the three matrix loads of a nonzero best.
// Measured at K = 16, 1.81M rows: whole calls 806 -> 699 us; the kernel 685 us
// with V = 2 and 3 blocks per SM, 842 with V = 1, 789 with V = 4, 1111 with two
// rows per warp and split nonzeros.
template <int K, int V, int NL, int U, int MINB>
__global__ void __launch_bounds__(256, MINB) spmm_complex_kernel(int n, const int *__restrict__ rp,
                                                           const int *__restrict__ ci, const double *__restrict__ Cv,
                                                           const double *__restrict__ Mv,
                                                           const double *__restrict__ omega,
                                                           const __grid_constant__ Omegas by_value,
                                                           const double2 *__restrict__ x,
                                                           const double2 *__restrict__ b, double2 *__restrict__ y,
                                                           bool residual, bool conj_out) {
  constexpr int CL = K / V, G = CL * NL;
  const int lane = threadIdx.x & 31;
  const int row = (int)((blockIdx.x * 256L + threadIdx.x) / G);
  const int sub = lane % G;
  const int cl = sub % CL, sl = sub / CL;
  double w[V], ar[V], ai[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    w[i] = omega ? __ldg(omega + cl + i * CL) : by_value.w[cl + i * CL];
    ar[i] = ai[i] = 0;
  }
  const bool valid = row < n;
  if (valid) {
    const int ke = __ldg(rp + row + 1);
    for (int k0 = __ldg(rp + row) + sl; k0 < ke; k0 += NL * U) {
      int j[U];
      double a[U], m[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = k0 + u * NL;
        const bool ok = k < ke;
        j[u] = ok ? __ldg(ci + k) : -1;
        a[u] = ok ? __ldg(Cv + k) : 0.0;
        m[u] = ok ? __ldg(Mv + k) : 0.0;
      }
      double2 xv[U][V];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < V; ++i)
          xv[u][i] = j[u] >= 0 ? __ldg(x + (long)j[u] * K + cl + i * CL) : make_double2(0, 0);
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < V; ++i) {
          const double mw = w[i] * m[u];
          ar[i] = fma(a[u], xv[u][i].x, fma(-mw, xv[u][i].y, ar[i]));
          ai[i] = fma(a[u], xv[u][i].y, fma(mw, xv[u][i].x, ai[i]));
        }
    }
  }
#pragma unroll
  for (int off = CL; off < G; off <<= 1)
#pragma unroll
    for (int i = 0; i < V; ++i) {
      ar[i] += __shfl_xor_sync(0xffffffffu, ar[i], off);
      ai[i] += __shfl_xor_sync(0xffffffffu, ai[i], off);
    }
  if (!valid || sl != 0) return;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    if (conj_out) ai[i] = -ai[i];
    const long o = (long)row * K + cl + i * CL;
    if (residual) {
      const double2 bv = __ldg(b + o);
      ar[i] = bv.x - ar[i];
      ai[i] = bv.y - ai[i];
    }
    y[o] = make_double2(ar[i], ai[i]);
  }
}

template <int K, int V, int NL, int U, int MINB>
static void spmm_complex_k(int n, const int *rp, const int *ci, const double *Cv, const double *Mv,
                           const double *omega, const Omegas &om, const double *x, const double *b, double *y,
                           bool residual, bool conj_out, cudaStream_t s) {
  const unsigned grid = (unsigned)(((long)n * (K / V * NL) + 255) / 256);
  spmm_complex_kernel<K, V, NL, U, MINB><<<grid, 256, 0, s>>>(n, rp, ci, Cv, Mv, omega, om, (const double2 *)x,
                                                              (const double2 *)b, (double2 *)y, residual, conj_out);
  EMG_LAUNCH_CHECK();
}

static void spmm_complex_any(int n, int K, const int *rp, const int *ci, const double *Cv, const double *Mv,
                             const double *omega, const Omegas &om, const double *x, const double *b, double *y,
                             bool residual, bool conj_out, cudaStream_t s) {
  if (n <= 0) return;
  auto run = [&](auto f) { f(n, rp, ci, Cv, Mv, omega, om, x, b, y, residual, conj_out, s); };
  // narrow blocks split a row over lanes (16 nonzeros in one round); from 8
  // columns on a row's lanes are its columns
  switch (K) {
  case 1: return run(&spmm_complex_k<1, 1, 4, 4, 1>);
  case 2: return run(&spmm_complex_k<2, 1, 2, 4, 4>);
  case 4: return run(&spmm_complex_k<4, 1, 2, 4, 4>);
  case 8: return run(&spmm_complex_k<8, 1, 1, 4, 4>);
  case 16: return run(&spmm_complex_k<16, 2, 1, 4, 3>);
  case 32: return run(&spmm_complex_k<32, 2, 1, 4, 3>);
  }
  fail(EMG_ERR_ARG, "unsupported complex block width %d", K);
}

void spmm_complex(int n, int K, const int *rp, const int *ci, const double *Cv, const double *Mv,
                  const double *omega, const double *x, const double *b, double *y, bool residual, bool conj_out,
                  cudaStream_t s) {
  spmm_complex_any(n, K, rp, ci, Cv, Mv, omega, Omegas{}, x, b, y, residual, conj_out, s);
}

void spmm_complex_host(int n, int K, const int *rp, const int *ci, const double *Cv, const double *Mv,
                       const double *omega_host, const double *x, double *y, bool conj_out, cudaStream_t s) {
  Omegas om{};
  if (K < 1 || K > 32) fail(EMG_ERR_ARG, "unsupported complex block width %d", K);
  std::copy(omega_host, omega_host + K, om.w);
  spmm_complex_any(n, K, rp, ci, Cv, Mv, nullptr, om, x, nullptr, y, false, conj_out, s);
}

constexpr int MAXJ = 32;

__global__ void __launch_bounds__(256) cmultidot_kernel(long total, int K, int J, const double2 *__restrict__ V,
                                                        long stride, const double2 *__restrict__ w,
                                                        double *__restrict__ h) {
  double hr[MAXJ], hi[MAXJ];
#pragma unroll
  for (int j = 0; j < MAXJ; ++j) { hr[j] = 0; hi[j] = 0; }
  for (long i = blockIdx.x * 256L + threadIdx.x; i < total; i += (long)gridDim.x * 256) {
    double2 wv = w[i];
#pragma unroll
    for (int j = 0; j < MAXJ; ++j) {
      if (j < J) {
        double2 v = __ldg(V + j * stride + i);
        hr[j] = fma(v.x, wv.x, fma(v.y, wv.y, hr[j]));
        hi[j] = fma(v.x, wv.y, fma(-v.y, wv.x, hi[j]));
      }
    }
  }
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int j = 0; j < MAXJ; ++j) {
    if (j < J) {
      double a = hr[j], b = hi[j];
      for (int off = K; off < 32; off <<= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, off);
        b += __shfl_xor_sync(0xffffffffu, b, off);
      }
      if (lane < K) {
        atomicAdd(h + 2 * (j * K + lane), a);
        atomicAdd(h + 2 * (j * K + lane) + 1, b);
      }
    }
  }
}

void cmultidot(int n, int K, int J, const double *V, long stride, const double *w, double *h, double *partial,
               int partial_blocks, cudaStream_t s) {
  (void)partial;
  (void)partial_blocks;
  if (K > 32) fail(EMG_ERR_ARG, "complex block width above 32");
  EMG_CUDA(cudaMemsetAsync(h, 0, sizeof(double) * 2 * J * K, s));
  long total = (long)n * K;
  unsigned grid = (unsigned)std::max(1L, std::min((total + 255) / 256, 148L * 2));
  // at most MAXJ basis vectors per pass (their partial sums live in registers)
  for (int j0 = 0; j0 < J; j0 += MAXJ) {
    const int jc = std::min(MAXJ, J - j0);
    cmultidot_kernel<<<grid, 256, 0, s>>>(total, K, jc, (const double2 *)(V + (size_t)j0 * stride), stride / 2,
                                          (const double2 *)w, h + 2L * j0 * K);
    EMG_LAUNCH_CHECK();
  }
}

__global__ void __launch_bounds__(256) cgs_update_kernel(long total, int K, int J, const double2 *__restrict__ V,
                                                         long stride, const double *__restrict__ h,
                                                         double2 *__restrict__ w, double *__restrict__ hn) {
  __shared__ double sh[256];
  double acc = 0;
  const int c = threadIdx.x % K;
  for (long i = blockIdx.x * 256L + threadIdx.x; i < total; i += (long)gridDim.x * 256) {
    double2 wv = w[i];
    for (int j = 0; j < J; ++j) {
      double2 v = __ldg(V + j * stride + i);
      double a = h[2 * (j * K + c)], b = h[2 * (j * K + c) + 1];
      wv.x -= a * v.x - b * v.y;
      wv.y -= a * v.y + b * v.x;
    }
    w[i] = wv;
    acc += wv.x * wv.x + wv.y * wv.y;
  }
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int st = 128; st >= K; st >>= 1) {
    if ((int)threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if ((int)threadIdx.x < K) atomicAdd(hn + threadIdx.x, sh[threadIdx.x]);
}

void cgs_update(int n, int K, int J, const double *V, long stride, const double *h, double *w, double *hn,
                cudaStream_t s) {
  EMG_CUDA(cudaMemsetAsync(hn, 0, sizeof(double) * K, s));
  long total = (long)n * K;
  cgs_update_kernel<<<red_grid(total), 256, 0, s>>>(total, K, J, (const double2 *)V, stride / 2, h, (double2 *)w,
                                                    hn);
  EMG_LAUNCH_CHECK();
}

__global__ void cscale_kernel(long total, int K, const double2 *__restrict__ w, const double *__restrict__ sc,
                              double2 *__restrict__ v) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= total) return;
  double f = sc[i % K];
  f = f > 0 ? 1.0 / f : 0.0;
  double2 a = w[i];
  v[i] = make_double2(a.x * f, a.y * f);
}

void cscale(int n, int K, const double *w, const double *scale, double *v, cudaStream_t s) {
  long total = (long)n * K;
  cscale_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(total, K, (const double2 *)w, scale, (double2 *)v);
  EMG_LAUNCH_CHECK();
}

__global__ void cupdate_kernel(long total, int K, int J, const double2 *__restrict__ Z, long stride,
                               const double *__restrict__ y, double2 *__restrict__ x) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= total) return;
  int c = (int)(i % K);
  double2 xv = x[i];
  for (int j = 0; j < J; ++j) {
    double2 z = __ldg(Z + j * stride + i);
    double a = y[2 * (j * K + c)], b = y[2 * (j * K + c) + 1];
    xv.x += a * z.x - b * z.y;
    xv.y += a * z.y + b * z.x;
  }
  x[i] = xv;
}

void cupdate(int n, int K, int J, const double *Z, long stride, const double *y, double *x, cudaStream_t s) {
  long total = (long)n * K;
  cupdate_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(total, K, J, (const double2 *)Z, stride / 2, y,
                                                                 (double2 *)x);
  EMG_LAUNCH_CHECK();
}

__global__ void __launch_bounds__(256) cnorm2_kernel(long total, int K, const double2 *__restrict__ x,
                                                     double *__restrict__ out) {
  __shared__ double sh[256];
  double acc = 0;
  for (long i = blockIdx.x * 256L + threadIdx.x; i < total; i += (long)gridDim.x * 256) {
    double2 v = x[i];
    acc += v.x * v.x + v.y * v.y;
  }
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int st = 128; st >= K; st >>= 1) {
    if ((int)threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if ((int)threadIdx.x < K) atomicAdd(out + threadIdx.x, sh[threadIdx.x]);
}

void cnorm2(int n, int K, const double *x, double *out, cudaStream_t s) {
  long total = (long)n * K;
  cnorm2_kernel<<<red_grid(total), 256, 0, s>>>(total, K, (const double2 *)x, out);
  EMG_LAUNCH_CHECK();
}

// out[c] += || |b_c| + (|C| + w_c |Ms|) |x_c| ||^2 (|.| entrywise, complex
// moduli): the scale of the rounding error in a computed residual b - A x.
// One thread per (row, column); K divides 32, so lanes l and l + K of a warp
// hold the same column.
__global__ void __launch_bounds__(256) abs_bound_kernel(long total, int K, const int *__restrict__ rp,
                                                        const int *__restrict__ ci, const double *__restrict__ Cv,
                                                        const double *__restrict__ Mv,
                                                        const double *__restrict__ omega,
                                                        const double2 *__restrict__ x,
                                                        const double2 *__restrict__ b, double *__restrict__ out) {
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  double v = 0;
  if (t < total) {
    const long row = t / K;
    const int c = (int)(t - row * K);
    const double w = __ldg(omega + c);
    const double2 bv = __ldg(b + t);
    double acc = hypot(bv.x, bv.y);
    for (int k = __ldg(rp + row), ke = __ldg(rp + row + 1); k < ke; ++k) {
      const double2 xv = __ldg(x + (long)__ldg(ci + k) * K + c);
      acc += (fabs(__ldg(Cv + k)) + w * fabs(__ldg(Mv + k))) * hypot(xv.x, xv.y);
    }
    v = acc * acc;
  }
  for (int off = 16; off >= K; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  const int lane = threadIdx.x & 31;
  if (lane < K && v != 0.0) atomicAdd(out + lane, v);
}

void abs_bound2(int n, int K, const int *rp, const int *ci, const double *Cv, const double *Mv, const double *omega,
                const double *x, const double *b, double *out, cudaStream_t s) {
  if (K < 1 || K > 32 || (32 % K) != 0) fail(EMG_ERR_ARG, "abs_bound2: block width %d does not divide 32", K);
  const long total = (long)n * K;
  if (total == 0) return;
  abs_bound_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(total, K, rp, ci, Cv, Mv, omega,
                                                                   (const double2 *)x, (const double2 *)b, out);
  EMG_LAUNCH_CHECK();
}

// explicit instantiations
#define EMG_INST(T)                                                                                              \
  template void jacobi0<T>(int, int, const T *, const T *, const T *, const double *, double, T *, T *,          \
                           cudaStream_t);                                                                        \
  template void fill_zero<T>(long, T *, cudaStream_t);                                                           \
  template void ams_restrict<T>(int, int, int, const int *, const int *, const T *, const T *, T *, cudaStream_t, \
                                const RestrictJ0<T> &);                                                          \
  template void ams_prolong_add<T>(int, int, int, const int *, const T *, const T *, T *, cudaStream_t);          \
  template void coarse_apply<T>(int, int, const double *, const int *, const T *, T *, cudaStream_t);
EMG_INST(float)
EMG_INST(double)
#undef EMG_INST

}  // namespace emg
