// Batched flexible CG with truncation (Notay 2000), FP64 recurrences.
//
// An iteration is the preconditioner, the operator and four passes over the
// block vectors: the dots with the previous B-products, the new direction,
// the two dots of the step length, and the update.  There is no scalar
// kernel, memset or copy between the passes (there were 14 launches per
// iteration around the preconditioner; in a stream each costs the host 3.3 us,
// more than the GPU needs for it below 20000 rows): a thread keeps its two
// columns (16-byte loads) along its grid stride, so the pass that uses a sum
// forms the scalars of those columns from it, once per thread, and the update
// ends in its last block, which stores them, retires columns and clears the
// sums.  With a last block in every reducing pass instead, 64-bit divisions
// by the row width and 8 blocks per SM (dots / step length, us per pass):
// 6.1k rows, 16 columns 5.9 / 4.8 -> 1.9 / 1.7, 100k rows, 8 columns 11.5 /
// 8.5 -> 5.1 / 4.9, 150k rows, 32 columns 39 / 25 -> 14 / 17 (the last move 100
// and 115 MB, 15 and 18 us if all of it came from HBM; part is in L2).  The direction
// pays 1.8 us for its scalars at the smallest size.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "emg_fcg.h"

namespace emg {

namespace {

constexpr int kThreads = 256;

// blocks of a pass: 4 per SM where every block adds to the same sums and four
// pairs of a thread are in flight, 8 for the update (4 / 8: dots 14 / 24 us,
// update pass -9 us at 150k rows and 32 columns)
unsigned pass_grid(long pairs, int per_sm = 4) {
  return (unsigned)std::max(1L, std::min((pairs + kThreads - 1) / kThreads, 148L * per_sm));
}

// out[q * K + c] += the block's sum of v[q][c % 2] over the threads of column
// pair c / 2 (pair of thread t: t % hp, hp = K / 2 a power of two <= 32)
template <int Q>
__device__ __forceinline__ void column_sums(double (&v)[Q][2], int nq, int hp, double *out) {
  __shared__ double sh[kThreads / 32][Q][32][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < Q; ++q)
    for (int off = 16; off >= hp; off >>= 1) {
      v[q][0] += __shfl_xor_sync(0xffffffffu, v[q][0], off);
      v[q][1] += __shfl_xor_sync(0xffffffffu, v[q][1], off);
    }
  if (lane < hp)
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      sh[warp][q][lane][0] = v[q][0];
      sh[warp][q][lane][1] = v[q][1];
    }
  __syncthreads();
  const int K = 2 * hp;
  for (int t = threadIdx.x; t < nq * K; t += kThreads) {
    const int q = t / K, c = t - q * K;
    double a = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) a += sh[w][q][c >> 1][c & 1];
    atomicAdd(out + t, a);
  }
}

// true in every thread of the last block to arrive; the sums of all blocks
// are then visible to it
__device__ __forceinline__ bool last_block(unsigned *count) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(count, 1u) == gridDim.x - 1;
    if (last) *count = 0;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

__device__ __forceinline__ double take(double *p) {  // read a finished sum and clear it
  const double v = __ldcg(p);
  *p = 0.0;
  return v;
}

// the residual in every form the preconditioner wants it (columns c, c + 1 of
// row `row`; i2: their index as a pair)
__device__ __forceinline__ void feed_residual(const FcgFeed &f, long i2, long row, int c, double2 r) {
  if (f.r32) reinterpret_cast<float2 *>(f.r32)[i2] = make_float2((float)r.x, (float)r.y);
  if (f.jf.y) {
    const float dc = __ldg(f.jf.l1c + row), dm = f.jf.l1m ? __ldg(f.jf.l1m + row) : 0.f;
    const float d0 = f.jf.l1m ? dc + (float)__ldg(f.jf.omega + c) * dm : dc;
    const float d1 = f.jf.l1m ? dc + (float)__ldg(f.jf.omega + c + 1) * dm : dc;
    const float2 v = make_float2((float)f.jf.c1 * (float)r.x / d0, (float)f.jf.c1 * (float)r.y / d1);
    reinterpret_cast<float2 *>(f.jf.y)[i2] = v;
    if (f.jf.d) reinterpret_cast<float2 *>(f.jf.d)[i2] = v;
  }
  if (f.jd.y) {
    const double dc = __ldg(f.jd.l1c + row), dm = f.jd.l1m ? __ldg(f.jd.l1m + row) : 0.0;
    const double d0 = f.jd.l1m ? dc + __ldg(f.jd.omega + c) * dm : dc;
    const double d1 = f.jd.l1m ? dc + __ldg(f.jd.omega + c + 1) * dm : dc;
    const double2 v = make_double2(f.jd.c1 * r.x / d0, f.jd.c1 * r.y / d1);
    reinterpret_cast<double2 *>(f.jd.y)[i2] = v;
    if (f.jd.d) reinterpret_cast<double2 *>(f.jd.d)[i2] = v;
  }
}

// x = 0, r = b in every form, bn = ||b_c||^2; columns with b = 0 start inactive
__global__ void __launch_bounds__(kThreads) fcg_init_kernel(long pairs, int hp, const double2 *b, double2 *x,
                                                            double2 *r, FcgFeed feed, double *bn_acc, double *bn,
                                                            int *act, int *its, int *status, double **xslot,
                                                            unsigned *count) {
  double v[1][2] = {{0, 0}};
  for (long i = blockIdx.x * (long)kThreads + threadIdx.x; i < pairs; i += (long)gridDim.x * kThreads) {
    const double2 bv = b[i];
    x[i] = make_double2(0, 0);
    r[i] = bv;
    const long row = i / hp;
    feed_residual(feed, i, row, 2 * (int)(i - row * hp), bv);
    v[0][0] = fma(bv.x, bv.x, v[0][0]);
    v[0][1] = fma(bv.y, bv.y, v[0][1]);
  }
  column_sums<1>(v, 1, hp, bn_acc);
  if (!last_block(count)) return;
  for (int c = threadIdx.x; c < 2 * hp; c += kThreads) {
    const double s = take(bn_acc + c);
    bn[c] = s;
    act[c] = s > 0.0;
    its[c] = 0;
  }
  if (threadIdx.x == 0) {
    status[0] = status[1] = 0;
    *xslot = reinterpret_cast<double *>(x);
  }
}

struct Dirs {
  const double *p[Fcg::kMaxDirs];
};

// z of the pair i2: stored, or x + G phi formed from the FP32 AMS output.  The
// pairs per row are a power of two and come as its logarithm: the 64-bit
// division was most of the instructions of the pass
template <bool SPLIT>
__device__ __forceinline__ double2 z_at(long i2, int lhp, const double2 *z, const Fcg::ZSplit &zs) {
  if constexpr (!SPLIT) return z[i2];
  const long e = i2 >> lhp;
  const int hp = 1 << lhp, c2 = (int)i2 & (hp - 1);
  const int2 v = __ldg(reinterpret_cast<const int2 *>(zs.edges) + e);
  const float2 x = reinterpret_cast<const float2 *>(zs.x)[i2];
  const float2 a = reinterpret_cast<const float2 *>(zs.phi)[(long)v.x * hp + c2];
  const float2 b = reinterpret_cast<const float2 *>(zs.phi)[(long)v.y * hp + c2];
  return make_double2((double)x.x + ((double)b.x - (double)a.x), (double)x.y + ((double)b.y - (double)a.y));
}

// dots (z, S_j) of the NJ directions from j0 on
struct Slots {
  int s[Fcg::kMaxDirs];
};

template <bool SPLIT, int NJ, int U>
__global__ void __launch_bounds__(kThreads) fcg_dots_kernel(long pairs, int lhp, const double2 *z, Fcg::ZSplit zs,
                                                            int j0, Dirs S, double *acc) {
  pdl_trigger();
  pdl_wait();
  double v[NJ][2] = {};
  const long step = (long)gridDim.x * kThreads;
  long i = blockIdx.x * (long)kThreads + threadIdx.x;
  auto add = [&](const double2 &zv, const double2 &sv, int j) {
    v[j][0] = fma(zv.x, sv.x, v[j][0]);
    v[j][1] = fma(zv.y, sv.y, v[j][1]);
  };
  for (; i + (U - 1) * step < pairs; i += U * step) {  // U pairs in flight
    double2 zv[U], sv[U][NJ];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      zv[u] = z_at<SPLIT>(i + u * step, lhp, z, zs);
#pragma unroll
      for (int j = 0; j < NJ; ++j)
        sv[u][j] = reinterpret_cast<const double2 *>(S.p[j0 + j])[i + u * step];
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
        add(zv[u], sv[u][j], j);
  }
  for (; i < pairs; i += step) {
    const double2 zv = z_at<SPLIT>(i, lhp, z, zs);
#pragma unroll
    for (int j = 0; j < NJ; ++j)
      add(zv, reinterpret_cast<const double2 *>(S.p[j0 + j])[i], j);
  }
  column_sums<NJ>(v, NJ, 1 << lhp, acc + (j0 << (lhp + 1)));
}

// p = z - sum_j beta_j P_j over NJ directions from j0 on, beta_j = (z, S_j) /
// eta_j of the active columns (slot[j]: ring slot of j).  A quotient and not
// a product with a stored 1 / eta: eta below 2^-1024, of right-hand sides of
// norm 1e-152, has no finite reciprocal
template <bool SPLIT, int NJ>
__global__ void __launch_bounds__(kThreads) fcg_direction_kernel(long pairs, int lhp, const double2 *z,
                                                                 Fcg::ZSplit zs, int j0, Dirs P, Slots slot,
                                                                 const double2 *acc, const double2 *eta,
                                                                 const int2 *act, double2 *p) {
  pdl_trigger();
  const long i = blockIdx.x * (long)kThreads + threadIdx.x;
  const int c2 = (int)i & ((1 << lhp) - 1);
  pdl_wait();
  if (i >= pairs) return;
  double2 d[NJ + 1], e[NJ + 1], pj[NJ + 1];
  const int2 on = act[c2];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    d[j] = acc[((j0 + j) << lhp) + c2];
    e[j] = eta[(slot.s[j0 + j] << lhp) + c2];
    pj[j] = reinterpret_cast<const double2 *>(P.p[j0 + j])[i];
  }
  double2 v = z_at<SPLIT>(i, lhp, z, zs);
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    v.x -= (on.x && e[j].x != 0.0 ? d[j].x / e[j].x : 0.0) * pj[j].x;
    v.y -= (on.y && e[j].y != 0.0 ? d[j].y / e[j].y : 0.0) * pj[j].y;
  }
  p[i] = v;
}

// (p, s), (p, r)
__global__ void __launch_bounds__(kThreads) fcg_step_kernel(long pairs, int lhp, const double2 *p, const double2 *sv,
                                                            const double2 *r, double *acc) {
  pdl_trigger();
  pdl_wait();
  double v[2][2] = {{0, 0}, {0, 0}};
#pragma unroll 2
  for (long i = blockIdx.x * (long)kThreads + threadIdx.x; i < pairs; i += (long)gridDim.x * kThreads) {
    const double2 a = p[i], b = sv[i], q = r[i];
    v[0][0] = fma(a.x, b.x, v[0][0]);
    v[0][1] = fma(a.y, b.y, v[0][1]);
    v[1][0] = fma(a.x, q.x, v[1][0]);
    v[1][1] = fma(a.y, q.y, v[1][1]);
  }
  column_sums<2>(v, 2, 1 << lhp, acc);
}

// x += alpha p, r -= alpha s (in every form), alpha = (p, r) / (p, s) of the
// active columns from their sums.  The last block stores (p, s) and alpha, counts
// the iteration of every active column, retires the converged ones (||r_c||^2 <=
// rtol^2 ||b_c||^2), flags NaN/Inf and clears the sums (acc: the nacc of this
// iteration's passes, those of the step length at kstep): status[0] = active
// columns left, status[1] = 1 + a non-finite column (0: none)
__global__ void __launch_bounds__(kThreads) fcg_update_kernel(long pairs, int lhp, const double2 *p,
                                                              const double2 *sv, double *const *xslot, double2 *r,
                                                              FcgFeed feed, double *acc, int kstep, int nacc,
                                                              double *acc_rr, double *eta, double *alpha, double *bn,
                                                              double rtol2, int *act, int *its, int *status,
                                                              unsigned *count) {
  pdl_trigger();
  pdl_wait();
  const int hp = 1 << lhp, K = 2 * hp;
  double2 *x = reinterpret_cast<double2 *>(*xslot);
  double v[1][2] = {{0, 0}};
  const long i0 = blockIdx.x * (long)kThreads + threadIdx.x;
  const int c = 2 * ((int)i0 & (hp - 1));  // the stride is a multiple of hp
  const double ps0 = acc[kstep + c], ps1 = acc[kstep + c + 1];
  const double a0 = (act[c] && ps0 != 0.0) ? acc[kstep + K + c] / ps0 : 0.0;
  const double a1 = (act[c + 1] && ps1 != 0.0) ? acc[kstep + K + c + 1] / ps1 : 0.0;
  for (long i = i0; i < pairs; i += (long)gridDim.x * kThreads) {
    double2 xv = x[i], rv = r[i];
    const double2 pv = p[i], s = sv[i];
    xv.x += a0 * pv.x;
    xv.y += a1 * pv.y;
    rv.x -= a0 * s.x;
    rv.y -= a1 * s.y;
    x[i] = xv;
    r[i] = rv;
    feed_residual(feed, i, i >> lhp, c, rv);
    v[0][0] = fma(rv.x, rv.x, v[0][0]);
    v[0][1] = fma(rv.y, rv.y, v[0][1]);
  }
  column_sums<1>(v, 1, hp, acc_rr);
  if (!last_block(count)) return;
  __shared__ int left;
  if (threadIdx.x == 0) left = 0;
  if (threadIdx.x < hp) {  // blocks start on a row, so this thread's columns are c and c + 1
    eta[c] = ps0;
    eta[c + 1] = ps1;
    alpha[c] = a0;
    alpha[c + 1] = a1;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < nacc; k += kThreads) acc[k] = 0.0;
  for (int k = threadIdx.x; k < K; k += kThreads) {
    const double rn = take(acc_rr + k);
    if (!act[k]) continue;
    its[k]++;
    if (!isfinite(rn)) {
      atomicCAS(status + 1, 0, k + 1);
      act[k] = 0;
    } else if (rn <= rtol2 * bn[k]) {
      act[k] = 0;
    } else {
      atomicAdd(&left, 1);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) status[0] = left;
}

auto dots_of(bool split, int nj) {
  switch (nj) {
  case 1: return split ? &fcg_dots_kernel<true, 1, 4> : &fcg_dots_kernel<false, 1, 4>;
  case 2: return split ? &fcg_dots_kernel<true, 2, 4> : &fcg_dots_kernel<false, 2, 4>;
  case 3: return split ? &fcg_dots_kernel<true, 3, 2> : &fcg_dots_kernel<false, 3, 2>;
  default: return split ? &fcg_dots_kernel<true, 4, 2> : &fcg_dots_kernel<false, 4, 2>;
  }
}

auto direction_of(bool split, int nj) {
  switch (nj) {
  case 0: return split ? &fcg_direction_kernel<true, 0> : &fcg_direction_kernel<false, 0>;
  case 1: return split ? &fcg_direction_kernel<true, 1> : &fcg_direction_kernel<false, 1>;
  case 2: return split ? &fcg_direction_kernel<true, 2> : &fcg_direction_kernel<false, 2>;
  case 3: return split ? &fcg_direction_kernel<true, 3> : &fcg_direction_kernel<false, 3>;
  default: return split ? &fcg_direction_kernel<true, 4> : &fcg_direction_kernel<false, 4>;
  }
}

}  // namespace

int Fcg::solve(int n, int Kc, const std::function<void(const double *, double *)> &pc,
               const std::function<void(const double *, double *)> &opB, const double *b, double *x, double rtol,
               int maxit, cudaStream_t s, const FcgFeed &feed, const ZSplit *zs, const std::vector<uint64_t> &ext) {
  K = Kc;
  if (mmax < 1) mmax = 1;
  if (mmax > kMaxDirs) fail(EMG_ERR_ARG, "batched FCG keeps at most %d directions", kMaxDirs);
  const int hp = K / 2;
  if (K < 2 || K > 64 || (hp & (hp - 1)) != 0 || 2 * hp != K) fail(EMG_ERR_ARG, "batched FCG: unsupported width %d", K);
  const size_t N = (size_t)n * K;
  const long pairs = (long)n * hp;
  r.alloc(N);
  z.alloc(N);
  if ((int)P.size() != mmax || P[0].n != N) {
    P.clear();
    S.clear();
    P.resize(mmax);
    S.resize(mmax);
    for (int j = 0; j < mmax; ++j) {
      P[j].alloc(N);
      S[j].alloc(N);
    }
  }
  acc.alloc((size_t)(mmax + 4) * K);
  eta.alloc((size_t)mmax * K);
  alpha.alloc(K);
  bn.alloc(K);
  xslot.alloc(1);
  act.alloc(K);
  itsd.alloc(K);
  status.alloc(2);
  count.alloc(2);
  if (!h_status.p) EMG_CUDA(cudaMallocHost((void **)&h_status.p, 2 * sizeof(int)));
  const int lhp = K == 2 ? 0 : K == 4 ? 1 : K == 8 ? 2 : K == 16 ? 3 : K == 32 ? 4 : 5;
  const unsigned dir_grid = (unsigned)((pairs + kThreads - 1) / kThreads);
  const int kstep = mmax * K;  // where the sums of the step length lie
  double *acc_rr = acc.p + kstep + 2 * K, *acc_bb = acc_rr + K;
  // a solve that failed half way may have left sums behind
  acc.zero(s);
  count.zero(s);
  fcg_init_kernel<<<pass_grid(pairs), kThreads, 0, s>>>(pairs, hp, (const double2 *)b, (double2 *)x, (double2 *)r.p,
                                                        feed, acc_bb, bn.p, act.p, itsd.p, status.p, xslot.p,
                                                        count.p);
  EMG_LAUNCH_CHECK();
  std::vector<uint64_t> sig = ext;
  if (!sig.empty()) {
    auto add = [&](const void *p) { sig.push_back((uint64_t)p); };
    sig.push_back((uint64_t)n);
    sig.push_back(((uint64_t)K << 32) | (uint64_t)mmax);
    uint64_t rt;
    static_assert(sizeof(rt) == sizeof(rtol), "");
    std::memcpy(&rt, &rtol, sizeof(rt));
    sig.push_back(rt);
    add(r.p);
    add(z.p);
    for (int j = 0; j < mmax; ++j) {
      add(P[j].p);
      add(S[j].p);
    }
    for (const void *p : {(const void *)acc.p, (const void *)eta.p, (const void *)alpha.p,
                          (const void *)bn.p, (const void *)xslot.p, (const void *)act.p, (const void *)itsd.p,
                          (const void *)status.p, (const void *)count.p, (const void *)feed.r32,
                          (const void *)feed.jf.y, (const void *)feed.jf.d, (const void *)feed.jd.y,
                          (const void *)feed.jd.d, (const void *)(zs ? zs->x : nullptr),
                          (const void *)(zs ? zs->phi : nullptr)})
      add(p);
    if (graphs.sig != sig) {
      graphs.clear();
      graphs.sig = sig;
    }
  }
  const ZSplit z0 = zs ? *zs : ZSplit{nullptr, nullptr, nullptr};
  // one iteration with nprev previous directions, the new one into slot head
  auto iterate = [&](int head, int nprev) {
    pc(r.p, z.p);
    Dirs Sd{}, Pd{};
    Slots sl{};
    for (int j = 0; j < nprev; ++j) {  // oldest first
      sl.s[j] = (head - nprev + j + mmax) % mmax;
      Sd.p[j] = S[sl.s[j]].p;
      Pd.p[j] = P[sl.s[j]].p;
    }
    for (int j0 = 0; j0 < nprev; j0 += 4) {
      launch_chain(dots_of(zs != nullptr, std::min(4, nprev - j0)), pass_grid(pairs), kThreads, s, true, pairs, lhp,
                   (const double2 *)z.p, z0, j0, Sd, acc.p);
      EMG_LAUNCH_CHECK();
    }
    double *p = P[head].p, *sv = S[head].p;
    for (int j0 = 0; j0 == 0 || j0 < nprev; j0 += 4) {  // a later group goes on from p
      launch_chain(direction_of(zs && j0 == 0, std::min(4, nprev - j0)), dir_grid, kThreads, s, true, pairs, lhp,
                   (const double2 *)(j0 ? p : z.p), z0, j0, Pd, sl, (const double2 *)acc.p, (const double2 *)eta.p,
                   (const int2 *)act.p, (double2 *)p);
      EMG_LAUNCH_CHECK();
    }
    opB(p, sv);
    launch_chain(&fcg_step_kernel, pass_grid(pairs), kThreads, s, true, pairs, lhp, (const double2 *)p,
                 (const double2 *)sv, (const double2 *)r.p, acc.p + kstep);
    EMG_LAUNCH_CHECK();
    launch_chain(&fcg_update_kernel, pass_grid(pairs, 8), kThreads, s, true, pairs, lhp, (const double2 *)p,
                 (const double2 *)sv, xslot.p, (double2 *)r.p, feed, acc.p, kstep, kstep + 2 * K, acc_rr,
                 eta.p + (size_t)head * K, alpha.p, bn.p, rtol * rtol, act.p, itsd.p, status.p, count.p + 1);
    EMG_LAUNCH_CHECK();
  };
  auto run = [&](int head, int nprev) {
    if (sig.empty() || !graphs.warm) {
      iterate(head, nprev);  // the SpMM autotuner picks its layouts here
      graphs.warm = !sig.empty();
      return;
    }
    auto it = graphs.exec.find(head * (kMaxDirs + 1) + nprev);
    if (it == graphs.exec.end()) {
      cudaGraph_t g = nullptr;
      const long l0 = launch_count();
      EMG_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
      try {
        iterate(head, nprev);
      } catch (...) {
        cudaStreamEndCapture(s, &g);
        if (g) cudaGraphDestroy(g);
        throw;
      }
      EMG_CUDA(cudaStreamEndCapture(s, &g));
      cudaGraphExec_t ex;
      const cudaError_t e = cudaGraphInstantiate(&ex, g, 0);
      cudaGraphDestroy(g);
      EMG_CUDA(e);
      const long kernels = launch_count() - l0;
      add_launches(-kernels);  // counted when the graph is launched
      it = graphs.exec.emplace(head * (kMaxDirs + 1) + nprev, std::make_pair(ex, kernels)).first;
    }
    EMG_CUDA(cudaGraphLaunch(it->second.first, s));
    add_launches(it->second.second);
  };
  its.assign(K, 0);
  const int every = std::max(1, check_every);
  int nprev = 0, head = 0, it = 0;
  for (it = 0; it < maxit; ++it) {
    run(head, nprev);
    head = (head + 1) % mmax;
    nprev = std::min(nprev + 1, mmax);
    // the host looks at the column status only every `every` iterations (and
    // at the cap); columns that converged in between stay frozen (alpha = beta
    // = 0 keeps x and r)
    if (verbose || (it + 1) % every == 0 || it + 1 == maxit) {
      EMG_CUDA(cudaMemcpyAsync(h_status.p, status.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
      EMG_CUDA(cudaStreamSynchronize(s));
      if (verbose) {
        std::vector<double> ha(K);
        std::vector<int> hact(K);
        alpha.download(ha.data(), K, s);
        act.download(hact.data(), K, s);
        EMG_CUDA(cudaStreamSynchronize(s));
        fprintf(stderr, "fcg it %d:", it);
        for (int c = 0; c < K; ++c) fprintf(stderr, " [%d a=%.3e%s]", c, ha[c], hact[c] ? "" : " done");
        fprintf(stderr, "\n");
      }
      if (h_status.p[1])
        fail(EMG_DIVERGED_NANORINF, "inner FCG: NaN or Inf in the residual of column %d", h_status.p[1] - 1);
      if (h_status.p[0] == 0) {
        ++it;
        break;
      }
    }
  }
  itsd.download(its.data(), K, s);
  EMG_CUDA(cudaStreamSynchronize(s));
  long tot = 0;
  for (int c = 0; c < K; ++c) tot += its[c];
  total_its += tot;
  return it;
}

}  // namespace emg
