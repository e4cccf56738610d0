// Element-matrix generation and row-wise assembly into the CSR pattern.
//
// Replaces the tet loop of assemble_matrix (src/em_fwd.cc:343-392): one
// thread per matrix row evaluates the edge's row of the closed-form Whitney
// element matrices of the tets around it (the 4-point rule of em_fe.cc:82-128
// is exact for these integrands, so the closed form equals the reference up to
// rounding) and sums them in a shared tile of the row's slots.
//
// C is omega-independent and the mass part is stored without omega (Ms);
// the reference's M is omega * Ms (src/em_fwd.cc:336,365).

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <numeric>

#include "emg_internal.h"
#include "emg_kernels.cuh"

namespace emg {

// get_cell_attribute (src/em_fwd.cc:14-72) once per attribute.
void sigma_table(int aniso_form, int nrho, int ncol, const double *rho, std::vector<double> &out) {
  out.assign((size_t)nrho * 9, 0.0);
  for (int i = 0; i < nrho; ++i) {
    const double *r = rho + (size_t)i * ncol;
    double *s = &out[(size_t)i * 9];
    switch (aniso_form) {
    case EMG_ISOTROPIC: s[0] = s[4] = s[8] = 1.0 / r[0]; break;
    case EMG_VERTICAL: s[0] = s[4] = 1.0 / r[0]; s[8] = 1.0 / r[1]; break;
    case EMG_TRIAXIAL: s[0] = 1.0 / r[0]; s[4] = 1.0 / r[1]; s[8] = 1.0 / r[2]; break;
    case EMG_ARBITRARY: {
      // sigma = Rz Ry Rx diag(1/rho) Rx^T Ry^T Rz^T, angles in degrees
      double cx = std::cos(r[3] * DTOR), sx = std::sin(r[3] * DTOR);
      double cy = std::cos(r[4] * DTOR), sy = std::sin(r[4] * DTOR);
      double cz = std::cos(r[5] * DTOR), sz = std::sin(r[5] * DTOR);
      double X[9] = {1, 0, 0, 0, cx, sx, 0, -sx, cx};
      double Y[9] = {cy, 0, -sy, 0, 1, 0, sy, 0, cy};
      double Z[9] = {cz, sz, 0, -sz, cz, 0, 0, 0, 1};
      double ZY[9], R[9];
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
          double v = 0;
          for (int k = 0; k < 3; ++k) v += Z[a * 3 + k] * Y[k * 3 + b];
          ZY[a * 3 + b] = v;
        }
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
          double v = 0;
          for (int k = 0; k < 3; ++k) v += ZY[a * 3 + k] * X[k * 3 + b];
          R[a * 3 + b] = v;
        }
      double d[3] = {1.0 / r[0], 1.0 / r[1], 1.0 / r[2]};
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
          double v = 0;
          for (int k = 0; k < 3; ++k) v += R[a * 3 + k] * d[k] * R[b * 3 + k];
          s[a * 3 + b] = v;
        }
      break;
    }
    default: fail(EMG_ERR_USER, "Unsupported anisotropy form %d.", aniso_form);
    }
  }
}

static void build_incidence(Context &c, const std::vector<int> &e2t_rp);

// ---------------------------------------------------------------------------
// host: CSR pattern = make_sparsity_patterns (src/em_fwd.cc:191-246)
// row e: sorted unique edges sharing a tet with e (diagonal included)
// ---------------------------------------------------------------------------
void build_sparsity(Context &c) {
  const int ne = c.ne, nt = c.nt;
  std::vector<int> e2t_rp(ne + 1, 0), e2t;
  for (int t = 0; t < nt; ++t)
    for (int i = 0; i < 6; ++i) e2t_rp[c.h_t2e[6 * (size_t)t + i] + 1]++;
  for (int e = 0; e < ne; ++e) e2t_rp[e + 1] += e2t_rp[e];
  e2t.resize(e2t_rp[ne]);
  {
    std::vector<int> pos(e2t_rp.begin(), e2t_rp.end() - 1);
    for (int t = 0; t < nt; ++t)
      for (int i = 0; i < 6; ++i) e2t[pos[c.h_t2e[6 * (size_t)t + i]]++] = t;
  }
  std::vector<int> cnt(ne + 1, 0);
#pragma omp parallel
  {
    std::vector<int> buf;
#pragma omp for schedule(dynamic, 4096)
    for (int e = 0; e < ne; ++e) {
      buf.clear();
      for (int k = e2t_rp[e]; k < e2t_rp[e + 1]; ++k)
        for (int i = 0; i < 6; ++i) buf.push_back(c.h_t2e[6 * (size_t)e2t[k] + i]);
      std::sort(buf.begin(), buf.end());
      cnt[e + 1] = (int)(std::unique(buf.begin(), buf.end()) - buf.begin());
    }
  }
  c.h_rp.assign(ne + 1, 0);
  for (int e = 0; e < ne; ++e) c.h_rp[e + 1] = c.h_rp[e] + cnt[e + 1];
  c.nnz = c.h_rp[ne];
  c.h_ci.resize(c.nnz);
#pragma omp parallel
  {
    std::vector<int> buf;
#pragma omp for schedule(dynamic, 4096)
    for (int e = 0; e < ne; ++e) {
      buf.clear();
      for (int k = e2t_rp[e]; k < e2t_rp[e + 1]; ++k)
        for (int i = 0; i < 6; ++i) buf.push_back(c.h_t2e[6 * (size_t)e2t[k] + i]);
      std::sort(buf.begin(), buf.end());
      int u = (int)(std::unique(buf.begin(), buf.end()) - buf.begin());
      std::copy(buf.begin(), buf.begin() + u, c.h_ci.begin() + c.h_rp[e]);
    }
  }
  c.rp.upload(c.h_rp, c.stream);
  c.ci.upload(c.h_ci, c.stream);
  c.chunk_rp.release();
  build_incidence(c, e2t_rp);
}

// vertex adjacency (pattern of G^T B G and Pi^T B Pi) and vertex->edge incidence
void build_vertex_pattern(Context &c) {
  const int nv = c.nv, ne = c.ne;
  std::vector<int> deg(nv + 1, 0);
  for (int e = 0; e < ne; ++e) {
    deg[c.h_edges[2 * e] + 1]++;
    deg[c.h_edges[2 * e + 1] + 1]++;
  }
  std::vector<int> inc_rp(nv + 1, 0);
  for (int v = 0; v < nv; ++v) inc_rp[v + 1] = inc_rp[v] + deg[v + 1];
  std::vector<int> inc(inc_rp[nv]);
  {
    std::vector<int> pos(inc_rp.begin(), inc_rp.end() - 1);
    for (int e = 0; e < ne; ++e) {
      inc[pos[c.h_edges[2 * e]]++] = 2 * e + 0;
      inc[pos[c.h_edges[2 * e + 1]]++] = 2 * e + 1;
    }
  }
  c.h_vrp.assign(nv + 1, 0);
  for (int v = 0; v < nv; ++v) c.h_vrp[v + 1] = c.h_vrp[v] + 1 + (inc_rp[v + 1] - inc_rp[v]);
  c.h_vci.resize(c.h_vrp[nv]);
#pragma omp parallel for schedule(static)
  for (int v = 0; v < nv; ++v) {
    int *out = &c.h_vci[c.h_vrp[v]];
    int k = 0;
    out[k++] = v;
    for (int j = inc_rp[v]; j < inc_rp[v + 1]; ++j) {
      int e = inc[j] >> 1, ep = inc[j] & 1;
      out[k++] = c.h_edges[2 * e + (1 - ep)];
    }
    std::sort(out, out + k);
  }
  c.vrp.upload(c.h_vrp, c.stream);
  c.vci.upload(c.h_vci, c.stream);
  c.vinc_rp.upload(inc_rp, c.stream);
  c.vinc.upload(inc, c.stream);
}

// ---------------------------------------------------------------------------
// device kernels
// ---------------------------------------------------------------------------
__device__ __forceinline__ int find_col(const int *__restrict__ ci, int b, int e, int col) {
  // rows are short (<= ~40): binary search
  int lo = b, hi = e - 1;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (__ldg(ci + mid) < col) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Tets around each edge (in any order) and the interior faces 4 t + f of their
// lower tet, for estimate_face_kernel: a block's faces lie together
__global__ void __launch_bounds__(256) incidence_kernel(int nt, const int *__restrict__ t2e,
                                                        const int *__restrict__ nbr, const int *__restrict__ inc_rp,
                                                        int *__restrict__ cursor, int *__restrict__ inc,
                                                        int *__restrict__ n_faces, int *__restrict__ faces) {
  __shared__ int warp_sum[8], base;
  const int t = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned mine = 0;  // bit f: face f is listed here
  if (t < nt) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int e = __ldg(t2e + 6 * (long)t + k);
      inc[__ldg(inc_rp + e) + atomicAdd(cursor + e, 1)] = t;
    }
    const int4 nb = __ldg(reinterpret_cast<const int4 *>(nbr) + t);
    mine = (nb.x > t ? 1u : 0u) | (nb.y > t ? 2u : 0u) | (nb.z > t ? 4u : 0u) | (nb.w > t ? 8u : 0u);
  }
  const int n = __popc(mine);
  int upto = n;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, upto, off);
    if (lane >= off) upto += v;
  }
  if (lane == 31) warp_sum[warp] = upto;
  __syncthreads();
  if (threadIdx.x == 0) {
    int sum = 0;
    for (int w = 0; w < 8; ++w) {
      const int v = warp_sum[w];
      warp_sum[w] = sum;
      sum += v;
    }
    base = atomicAdd(n_faces, sum);
  }
  __syncthreads();
  int o = base + warp_sum[warp] + upto - n;
  for (int f = 0; f < 4; ++f)
    if ((mine >> f) & 1) faces[o++] = 4 * t + f;
}

// Device copies of the incidence (its row pointer comes from the pattern's
// host pass) and the face list.  One allocation holds them with the assembly
// records: below a megabyte cudaMalloc takes 350 us where it needs a new
// driver slab, above it always.
static void build_incidence(Context &c, const std::vector<int> &e2t_rp) {
  c.n_faces = 0;
  for (long i = 0; i < 4L * c.nt; ++i) c.n_faces += c.h_nbr[i] > i / 4;
  const size_t n6 = 6 * (size_t)c.nt;
  const size_t recs = std::max(n6, ((size_t)c.ne + 1) / 2);  // the cursors lie there first
  const size_t ints = n6 + (size_t)c.ne + 1 + (size_t)c.n_faces + 1;
  c.inc_mem.alloc(recs + (ints + 1) / 2);
  c.erec = c.inc_mem.p;
  c.einc = reinterpret_cast<int *>(c.erec + recs);
  c.einc_rp = c.einc + n6;
  c.faces = c.einc_rp + c.ne + 1;
  int *count = c.faces + c.n_faces, *cursor = reinterpret_cast<int *>(c.erec);
  EMG_CUDA(cudaMemcpyAsync(c.einc_rp, e2t_rp.data(), sizeof(int) * ((size_t)c.ne + 1), cudaMemcpyHostToDevice,
                           c.stream));
  EMG_CUDA(cudaMemsetAsync(cursor, 0, sizeof(int) * (size_t)c.ne, c.stream));
  EMG_CUDA(cudaMemsetAsync(count, 0, sizeof(int), c.stream));
  incidence_kernel<<<(unsigned)((c.nt + 255) / 256), 256, 0, c.stream>>>(c.nt, c.t2e.p, c.nbr.p, c.einc_rp, cursor,
                                                                         c.einc, count, c.faces);
  EMG_LAUNCH_CHECK();
}

// Record of an (edge, tet) incidence for assemble_edge_kernel:
//   einc[j]: the tet, with the edge's canonical index k in bits 28..30
//   erec[j]: per canonical edge l of the tet 9 bits, its position in the
//            row (511: search for it), and in bit 58 + l whether it is on the
//            boundary
constexpr int kTetBits = 28;
constexpr unsigned kSearch = 511;

// The tets of an edge in the order in which its row sums the diagonal: by place
// within 32 tets, the order a warp per 32 tets adds them in.  A diagonal that is
// rounded another way moves solutions in the air by some 1e-10, so the order
// is kept.
__device__ __forceinline__ unsigned sum_order(int t) { return ((unsigned)(t & 31) << (kTetBits - 5)) | (unsigned)(t >> 5); }

// heap sort of one edge's list (5 tets as a rule, hundreds in a fan)
__device__ void sort_tets(int *a, int n) {
  auto sift = [&](int root, int end) {
    const int v = a[root];
    for (;;) {
      int child = 2 * root + 1;
      if (child >= end) break;
      if (child + 1 < end && sum_order(a[child + 1]) > sum_order(a[child])) ++child;
      if (sum_order(a[child]) <= sum_order(v)) break;
      a[root] = a[child];
      root = child;
    }
    a[root] = v;
  };
  for (int i = n / 2 - 1; i >= 0; --i) sift(i, n);
  for (int end = n - 1; end > 0; --end) {
    const int v = a[0];
    a[0] = a[end];
    a[end] = v;
    sift(0, end);
  }
}

__global__ void edge_records_kernel(int ne, const int *__restrict__ inc_rp, int *__restrict__ inc,
                                    const int *__restrict__ cedge, const unsigned char *__restrict__ ebdr,
                                    const int *__restrict__ rp, const int *__restrict__ ci,
                                    unsigned long long *__restrict__ rec) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const int kb = __ldg(rp + e), ke = __ldg(rp + e + 1);
  const int j0 = __ldg(inc_rp + e), j1 = __ldg(inc_rp + e + 1);
  sort_tets(inc + j0, j1 - j0);
  for (int j = j0; j < j1; ++j) {
    const int t = inc[j];
    unsigned long long r = 0;
    int k = 0;
    for (int l = 0; l < 6; ++l) {
      const int g = __ldg(cedge + 6 * (long)t + l);
      if (g == e) k = l;
      const int pos = find_col(ci, kb, ke, g) - kb;
      r |= (unsigned long long)(pos < (int)kSearch ? (unsigned)pos : kSearch) << (9 * l);
      if (__ldg(ebdr + g)) r |= 1ull << (58 + l);
    }
    rec[j] = r;
    inc[j] = t | (k << kTetBits);
  }
}

// whether a tet touches a boundary edge (ctx->bdr_cells, src/em_fwd.cc:377-388)
__global__ void bdr_cell_kernel(int nt, const int *__restrict__ cedge, const unsigned char *__restrict__ ebdr,
                                unsigned char *__restrict__ bdr_cell) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  bool any = false;
#pragma unroll
  for (int k = 0; k < 6; ++k) any |= __ldg(ebdr + __ldg(cedge + 6 * (long)t + k)) != 0;
  bdr_cell[t] = any ? 1 : 0;
}

// vslot[t*16 + p*4 + q] = slot of (ctet[t][p], ctet[t][q]) in the vertex pattern
__global__ void vslot_map_kernel(int nt, const int *__restrict__ tets, const int *__restrict__ rp,
                                 const int *__restrict__ ci, int *__restrict__ slot) {
  long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long)nt * 16) return;
  int t = (int)(idx / 16), ent = (int)(idx % 16);
  int row = __ldg(tets + 4 * (long)t + ent / 4), col = __ldg(tets + 4 * (long)t + ent % 4);
  slot[idx] = find_col(ci, __ldg(rp + row), __ldg(rp + row + 1), col);
}

void build_slot_maps(Context &c) {
  if (c.nt >= (1 << kTetBits)) fail(EMG_ERR_ARG, "mesh of %d tets", c.nt);
  edge_records_kernel<<<(unsigned)((c.ne + 127) / 128), 128, 0, c.stream>>>(c.ne, c.einc_rp, c.einc, c.cedge.p,
                                                                            c.ebdr.p, c.rp.p, c.ci.p, c.erec);
  EMG_LAUNCH_CHECK();
  c.bdr_cell.alloc(c.nt);
  bdr_cell_kernel<<<(unsigned)((c.nt + 255) / 256), 256, 0, c.stream>>>(c.nt, c.cedge.p, c.ebdr.p, c.bdr_cell.p);
  EMG_LAUNCH_CHECK();
  c.vslot.alloc((size_t)c.nt * 16);
  long n16 = (long)c.nt * 16;
  vslot_map_kernel<<<(unsigned)((n16 + 255) / 256), 256, 0, c.stream>>>(c.nt, c.ctet.p, c.vrp.p, c.vci.p, c.vslot.p);
  EMG_LAUNCH_CHECK();
}

// canonical tets: sorted vertex ids, canonical global edges, sort parity
__global__ void canonicalize_kernel(int nt, const int *__restrict__ tets, const int *__restrict__ t2e,
                                    const int *__restrict__ edges, int *__restrict__ ctet,
                                    int *__restrict__ cedge, signed char *__restrict__ cpar,
                                    int *__restrict__ bad) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  int v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __ldg(tets + 4 * (long)t + i);
  int par = 1;
  // sorting network on 4 keys, counting swaps for the parity
#define EMG_CSWAP(a, b) if (v[a] > v[b]) { int tmp_ = v[a]; v[a] = v[b]; v[b] = tmp_; par = -par; }
  EMG_CSWAP(0, 1) EMG_CSWAP(2, 3) EMG_CSWAP(0, 2) EMG_CSWAP(1, 3) EMG_CSWAP(1, 2)
#undef EMG_CSWAP
#pragma unroll
  for (int i = 0; i < 4; ++i) ctet[4 * (long)t + i] = v[i];
  cpar[t] = (signed char)par;
  int le[6], la[6], lb[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    le[i] = __ldg(t2e + 6 * (long)t + i);
    la[i] = __ldg(edges + 2 * (long)le[i]);
    lb[i] = __ldg(edges + 2 * (long)le[i] + 1);
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    int a = v[kEdgeP(k)], b = v[kEdgeQ(k)];
    int ge = -1;
#pragma unroll
    for (int i = 0; i < 6; ++i)
      if (la[i] == a && lb[i] == b) ge = le[i];
    if (ge < 0) atomicExch(bad, t + 1);
    cedge[6 * (long)t + k] = ge < 0 ? 0 : ge;
  }
}

void canonicalize(Context &c) {
  c.ctet.alloc((size_t)c.nt * 4);
  c.cedge.alloc((size_t)c.nt * 6);
  c.cpar.alloc((size_t)c.nt);
  DBuf<int> bad(1);
  bad.zero(c.stream);
  canonicalize_kernel<<<(unsigned)((c.nt + 255) / 256), 256, 0, c.stream>>>(c.nt, c.tets.p, c.t2e.p, c.edges.p,
                                                                            c.ctet.p, c.cedge.p, c.cpar.p, bad.p);
  EMG_LAUNCH_CHECK();
  int hb = 0;
  bad.download(&hb, 1, c.stream);
  EMG_CUDA(cudaStreamSynchronize(c.stream));
  if (hb) fail(EMG_ERR_USER, "tet %d: tet2edgelist does not match tetrahedronlist/edgelist", hb - 1);
}

struct ElemIn {
  const double *pts;
  const int *ctet, *cedge, *attr;
  const signed char *cpar;
  const unsigned char *ebdr;
  const double *sig;
};

// S_ab = grad l_a . sigma grad l_b (packed, a <= b)
__device__ __forceinline__ void grad_products(const ElemIn &in, int t, const TetGeom &g, double S[10]) {
  const double *sg = in.sig + 9 * (long)__ldg(in.attr + t);
  double s[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) s[k] = __ldg(sg + k);
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = p; q < 4; ++q) {
      double sq0 = s[0] * g.gr[q][0] + s[1] * g.gr[q][1] + s[2] * g.gr[q][2];
      double sq1 = s[3] * g.gr[q][0] + s[4] * g.gr[q][1] + s[5] * g.gr[q][2];
      double sq2 = s[6] * g.gr[q][0] + s[7] * g.gr[q][1] + s[8] * g.gr[q][2];
      S[sym_idx(p, q)] = g.gr[p][0] * sq0 + g.gr[p][1] * sq1 + g.gr[p][2] * sq2;
    }
}

// curl of the edge function l_a grad l_b - l_b grad l_a; the roundings are
// spelled out because an edge must give the same number as a row and as a column
__device__ __forceinline__ void edge_curl(const double ga[3], const double gb[3], double cu[3]) {
  cu[0] = 2.0 * fma(ga[1], gb[2], -__dmul_rn(ga[2], gb[1]));
  cu[1] = 2.0 * fma(ga[2], gb[0], -__dmul_rn(ga[0], gb[2]));
  cu[2] = 2.0 * fma(ga[0], gb[1], -__dmul_rn(ga[1], gb[0]));
}

__device__ __forceinline__ double pick3(int i, double a, double b, double c) { return i == 0 ? a : (i == 1 ? b : c); }

// Element matrices of tet t in canonical order: c (curl-curl / mu) and ms
// (mass without omega), boundary rows/columns zeroed as
// src/em_fwd.cc:377-388.  Returns whether the tet touches a boundary edge.
//   c_kl  = V/mu curl(phi_k).curl(phi_l),  curl(phi_k) = 2 grad l_p x grad l_q
//   ms_kl = V/20 [(1+d_pr) S_qs - (1+d_ps) S_qr - (1+d_qr) S_ps + (1+d_qs) S_pr]
// for k=(p,q), l=(r,s), S_ab = grad l_a . sigma grad l_b (int l_a l_b = V(1+d_ab)/20).
__device__ __forceinline__ bool element_matrices(const ElemIn &in, int t, double c[36], double ms[36],
                                                 TetGeom &g) {
  load_tet_geom(in.pts, in.ctet, in.cedge, in.cpar, t, g);
  double S[10];
  grad_products(in, t, g, S);
  double cu[6][3];
#pragma unroll
  for (int k = 0; k < 6; ++k) edge_curl(g.gr[kEdgeP(k)], g.gr[kEdgeQ(k)], cu[k]);
  const double vc = g.vol / MU, vm = g.vol / 20.0;
  bool bd[6];
  bool any = false;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    bd[k] = __ldg(in.ebdr + g.ge[k]) != 0;
    any |= bd[k];
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
#pragma unroll
    for (int l = 0; l <= k; ++l) {
      const int p = kEdgeP(k), q = kEdgeQ(k), r = kEdgeP(l), u = kEdgeQ(l);
      double ckl = vc * (cu[k][0] * cu[l][0] + cu[k][1] * cu[l][1] + cu[k][2] * cu[l][2]);
      double mkl = vm * ((1.0 + (p == r)) * S[sym_idx(q, u)] - (1.0 + (p == u)) * S[sym_idx(q, r)] -
                         (1.0 + (q == r)) * S[sym_idx(p, u)] + (1.0 + (q == u)) * S[sym_idx(p, r)]);
      if (bd[k] || bd[l]) {
        if (k != l) ckl = 0.0;
        mkl = 0.0;
      }
      c[k * 6 + l] = ckl;
      c[l * 6 + k] = ckl;
      ms[k * 6 + l] = mkl;
      ms[l * 6 + k] = mkl;
    }
  }
  return any;
}

// One thread per matrix row: the edge's row of the element matrices of each
// incident tet, summed in the row's slots of a shared tile and written once.
// A pair of edges meets in at most two tets (one per side of their common
// face), only the diagonal in more, so the tet-wise scatter that this
// replaces spent 72 FP64 atomics per tet on entries with one or two terms and
// was bound by them.  The row-wise sum recomputes a tet's geometry for each of
// its six edges instead, needs no atomics, no cleared arrays and no 36-entry
// slot map per tet, and always sums in the same order.
// Every row evaluates its entries as element_matrices does, from the sorted
// vertices and with the higher edge's operands first: entry (e, f) is the same
// number as (f, e), and the operator the one that the nodal spaces and G^T B
// are built from.  (In the air w sigma Ms is 1e-10 of C: rows that each
// started from their own edge moved solutions by 4e-10.)
// Bound: L1 at 68 % (the gathers of a tet's data, each a pass per lane, and the
// tile's read-modify-writes; C and Ms of a slot lie together for those) and
// latency, with 18 warps active per SM.  600k tets: 320 us scattered, 206 now; rows that differed from their
// mirror took 193, 6 blocks per SM instead of 5 (8 bytes spilled) 205.
constexpr int ASM_ROWS = 128;
constexpr int ASM_SLOTS = ASM_ROWS * 18;  // a tile holds rows of 18 slots on average (36.9 KB)

__global__ void __launch_bounds__(ASM_ROWS) assemble_edge_kernel(ElemIn in, int ne, const int *__restrict__ inc_rp,
                                                               const int *__restrict__ inc,
                                                               const unsigned long long *__restrict__ rec,
                                                               const int *__restrict__ rp, const int *__restrict__ ci,
                                                               double *__restrict__ Cv, double *__restrict__ Mv) {
  __shared__ double2 tile[ASM_SLOTS];  // (C, Ms) of a slot
  const int r0 = blockIdx.x * ASM_ROWS, r1 = min(ne, r0 + ASM_ROWS), e = r0 + (int)threadIdx.x;
  const int s0 = __ldg(rp + r0), ns = __ldg(rp + r1) - s0;
  const bool tiled = ns <= ASM_SLOTS;
  for (int i = threadIdx.x; i < ns; i += ASM_ROWS) {
    if (tiled) tile[i] = make_double2(0.0, 0.0);
    else Cv[s0 + i] = Mv[s0 + i] = 0.0;
  }
  __syncthreads();
  if (e < ne) {
    const int kb = __ldg(rp + e), ke = __ldg(rp + e + 1);
    const int j1 = __ldg(inc_rp + e + 1);
    for (int j = __ldg(inc_rp + e); j < j1; ++j) {
      const int tk = __ldg(inc + j), t = tk & ((1 << kTetBits) - 1), k = tk >> kTetBits;
      const unsigned long long rc6 = __ldg(rec + j);
      const int p = kEdgeP(k), q = kEdgeQ(k);
      TetGeom g;
      load_tet_geom(in.pts, in.ctet, in.cedge, in.cpar, t, g);
      double gp[3], gq[3], cu[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        gp[d] = pick3(p, g.gr[0][d], g.gr[1][d], g.gr[2][d]);
        gq[d] = pick3(q - 1, g.gr[1][d], g.gr[2][d], g.gr[3][d]);
      }
      edge_curl(gp, gq, cu);
      double Sp[4], Sq[4];  // S_px and S_qx
      {
        double S[10];
        grad_products(in, t, g, S);
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          Sp[x] = pick3(p, S[sym_idx(0, x)], S[sym_idx(1, x)], S[sym_idx(2, x)]);
          Sq[x] = pick3(q - 1, S[sym_idx(1, x)], S[sym_idx(2, x)], S[sym_idx(3, x)]);
        }
      }
      const double vc = g.vol / MU, vm = g.vol / 20.0;
      const bool row_bdr = (rc6 >> (58 + k)) & 1;
#pragma unroll
      for (int l = 0; l < 6; ++l) {
        const int r = kEdgeP(l), u = kEdgeQ(l);
        double cr[3];
        edge_curl(g.gr[r], g.gr[u], cr);
        double ckl = vc * (cu[0] * cr[0] + cu[1] * cr[1] + cu[2] * cr[2]);
        // the middle terms in the order of (higher edge, lower edge)
        const double qr = (q == r ? 2.0 : 1.0) * Sp[u], pu = (p == u ? 2.0 : 1.0) * Sq[r];
        double mkl = vm * ((p == r ? 2.0 : 1.0) * Sq[u] - (k >= l ? pu : qr) - (k >= l ? qr : pu) +
                           (q == u ? 2.0 : 1.0) * Sp[r]);
        if (row_bdr || ((rc6 >> (58 + l)) & 1)) {
          if (k != l) ckl = 0.0;
          mkl = 0.0;
        }
        int pos = (int)((rc6 >> (9 * l)) & kSearch);
        if (pos == (int)kSearch) pos = find_col(ci, kb, ke, __ldg(in.cedge + 6 * (long)t + l)) - kb;
        if (tiled) {
          double2 &s2 = tile[kb - s0 + pos];
          s2 = make_double2(s2.x + ckl, s2.y + mkl);
        } else {
          Cv[kb + pos] += ckl;
          Mv[kb + pos] += mkl;
        }
      }
    }
  }
  if (!tiled) return;
  __syncthreads();
  for (int i = threadIdx.x; i < ns; i += ASM_ROWS) {
    const double2 s2 = tile[i];
    Cv[s0 + i] = s2.x;
    Mv[s0 + i] = s2.y;
  }
}

ElemIn elem_in(Context &c) {
  return ElemIn{c.pts.p, c.ctet.p, c.cedge.p, c.attr.p, c.cpar.p, c.ebdr.p, c.sigma_tab.p};
}

void assemble_edge(Context &c) {
  c.Cv.alloc(c.nnz);
  c.Msv.alloc(c.nnz);
  assemble_edge_kernel<<<(unsigned)((c.ne + ASM_ROWS - 1) / ASM_ROWS), ASM_ROWS, 0, c.stream>>>(
      elem_in(c), c.ne, c.einc_rp, c.einc, c.erec, c.rp.p, c.ci.p, c.Cv.p, c.Msv.p);
  EMG_LAUNCH_CHECK();
}

// Nodal subspace operators Q^T K Q for Q = G_e (gradient: -1 at the lower,
// +1 at the higher vertex, src/em_la.cc:254-270) and Pi_{x,y,z},e (0.5 t_e[d]
// at both endpoints, t_e = x(v1) - x(v0): the Nedelec interpolation AMS
// builds from G and the vertex coordinates), K = c and ms.  Summing element
// contributions equals G^T B G etc. of the assembled B because the boundary
// zeroing is element-local.
struct NodalOut {
  double *v[8];
};

__global__ void __launch_bounds__(128) assemble_nodal_kernel(ElemIn in, int nt, const int *__restrict__ vslot,
                                                              NodalOut out) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  double c[36], m[36];
  TetGeom g;
  const bool touches_bdr = element_matrices(in, t, c, m, g);
  int vs[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) vs[k] = __ldg(vslot + 16 * (long)t + k);
#pragma unroll
  for (int sp = 0; sp < 4; ++sp) {
    double Q[6][4];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int a = kEdgeP(k), b = kEdgeQ(k);
#pragma unroll
      for (int p = 0; p < 4; ++p) Q[k][p] = 0.0;
      if (sp == 0) {
        Q[k][a] = -1.0;
        Q[k][b] = 1.0;
      } else {
        double w = 0.5 * (g.x[b][sp - 1] - g.x[a][sp - 1]);
        Q[k][a] = w;
        Q[k][b] = w;
      }
    }
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      // curl(grad) = 0: G_e^T c G_e vanishes exactly unless boundary zeroing
      // broke the element matrix; skipping it keeps rounding noise (~1e-16
      // |C|) out of the gradient space, where w sigma_air Ms is ~1e-10 |C|
      if (sp == 0 && part == 0 && !touches_bdr) continue;
      const double *K = part == 0 ? c : m;
      double KQ[6][4];
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          double v = 0;
#pragma unroll
          for (int j = 0; j < 6; ++j) v += K[i * 6 + j] * Q[j][q];
          KQ[i][q] = v;
        }
      double *o = out.v[sp * 2 + part];
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          double v = 0;
#pragma unroll
          for (int i = 0; i < 6; ++i) v += Q[i][p] * KQ[i][q];
          atomicAdd(o + vs[p * 4 + q], v);
        }
    }
  }
}

void assemble_nodal_device(Context &c, DBuf<double> &buf) {
  long vnnz = c.h_vrp[c.nv];
  buf.alloc((size_t)vnnz * 8);
  buf.zero(c.stream);
  NodalOut o;
  for (int k = 0; k < 8; ++k) o.v[k] = buf.p + (size_t)k * vnnz;
  assemble_nodal_kernel<<<(unsigned)((c.nt + 127) / 128), 128, 0, c.stream>>>(elem_in(c), c.nt, c.vslot.p, o);
  EMG_LAUNCH_CHECK();
}

void assemble_nodal(Context &c, HCsr out[4]) {
  long vnnz = c.h_vrp[c.nv];
  DBuf<double> buf;
  assemble_nodal_device(c, buf);
  // each part straight into its operator (no staging copy of all eight)
  for (int sp = 0; sp < 4; ++sp) {
    out[sp].n = out[sp].m = c.nv;
    out[sp].rp = c.h_vrp;
    out[sp].ci = c.h_vci;
    out[sp].vc.resize(vnnz);
    out[sp].vm.resize(vnnz);
    buf.download_at(out[sp].vc.data(), (size_t)(2 * sp) * vnnz, vnnz, c.stream);
    buf.download_at(out[sp].vm.data(), (size_t)(2 * sp + 1) * vnnz, vnnz, c.stream);
  }
  EMG_CUDA(cudaStreamSynchronize(c.stream));
}

// The vector nodal space of AMS (hypre's Pi space, cycle character '2'):
// Pi = [Pi_x Pi_y Pi_z] interpolates a vertex vector field (3 values per
// vertex) onto the edges, and Pi^T K Pi couples the three components.  The
// nine 4x4 element blocks Q_d1^T K Q_d2 are summed into nine vertex-pattern
// arrays per value part; the host interleaves them as row 3 v + d1, column
// 3 u + d2.
struct PiOut {
  double *v[18];  // (d1 * 3 + d2) * 2 + part
};

__global__ void __launch_bounds__(128) assemble_pivec_kernel(ElemIn in, int nt, const int *__restrict__ vslot,
                                                              PiOut out) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  double c[36], m[36];
  TetGeom g;
  element_matrices(in, t, c, m, g);
  int vs[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) vs[k] = __ldg(vslot + 16 * (long)t + k);
  // w[k][d]: Pi_d weight of edge k at both of its endpoints
  double w[6][3];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const int a = kEdgeP(k), b = kEdgeQ(k);
#pragma unroll
    for (int d = 0; d < 3; ++d) w[k][d] = 0.5 * (g.x[b][d] - g.x[a][d]);
  }
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    const double *K = part == 0 ? c : m;
#pragma unroll 1
    for (int d2 = 0; d2 < 3; ++d2) {
      // KQ = K Q_d2 (6 x 4)
      double KQ[6][4];
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) KQ[i][q] = 0.0;
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        const int a = kEdgeP(j), b = kEdgeQ(j);
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          const double v = K[i * 6 + j] * w[j][d2];
          KQ[i][a] += v;
          KQ[i][b] += v;
        }
      }
#pragma unroll 1
      for (int d1 = 0; d1 < 3; ++d1) {
        double B[4][4];
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
          for (int q = 0; q < 4; ++q) B[p][q] = 0.0;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          const int a = kEdgeP(i), b = kEdgeQ(i);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const double v = w[i][d1] * KQ[i][q];
            B[a][q] += v;
            B[b][q] += v;
          }
        }
        double *o = out.v[(d1 * 3 + d2) * 2 + part];
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
          for (int q = 0; q < 4; ++q) atomicAdd(o + vs[p * 4 + q], B[p][q]);
      }
    }
  }
}

void assemble_pi_vector(Context &c, HCsr &out, bool coupled) {
  const long vnnz = c.h_vrp[c.nv];
  DBuf<double> buf((size_t)vnnz * 18);
  buf.zero(c.stream);
  PiOut o;
  for (int k = 0; k < 18; ++k) o.v[k] = buf.p + (size_t)k * vnnz;
  assemble_pivec_kernel<<<(unsigned)((c.nt + 127) / 128), 128, 0, c.stream>>>(elem_in(c), c.nt, c.vslot.p, o);
  EMG_LAUNCH_CHECK();
  std::vector<double> h((size_t)vnnz * 18);
  buf.download(h.data(), h.size(), c.stream);
  EMG_CUDA(cudaStreamSynchronize(c.stream));
  const int nv = c.nv;
  out.n = out.m = 3 * nv;
  out.rp.assign(3 * (size_t)nv + 1, 0);
  const int nb = coupled ? 3 : 1;  // column blocks per row: all three components, or its own
  for (int v = 0; v < nv; ++v)
    for (int d = 0; d < 3; ++d) out.rp[3 * v + d + 1] = nb * (c.h_vrp[v + 1] - c.h_vrp[v]);
  for (int i = 0; i < 3 * nv; ++i) out.rp[i + 1] += out.rp[i];
  out.ci.resize(out.rp[3 * nv]);
  out.vc.resize(out.rp[3 * nv]);
  out.vm.resize(out.rp[3 * nv]);
#pragma omp parallel for schedule(static)
  for (int v = 0; v < nv; ++v)
    for (int d1 = 0; d1 < 3; ++d1) {
      long p = out.rp[3 * v + d1];
      for (int k = c.h_vrp[v]; k < c.h_vrp[v + 1]; ++k)
        for (int d2 = 0; d2 < 3; ++d2) {
          if (!coupled && d2 != d1) continue;
          out.ci[p] = 3 * c.h_vci[k] + d2;
          out.vc[p] = h[(size_t)((d1 * 3 + d2) * 2) * vnnz + k];
          out.vm[p] = h[(size_t)((d1 * 3 + d2) * 2 + 1) * vnnz + k];
          ++p;
        }
    }
}

// ---------------------------------------------------------------------------
// G^T B as a vertex x edge operator.  The gradient-space residual of AMS,
// G^T (b - B x), is formed as G^T b - (G^T B) x: G^T C vanishes exactly on
// every element without a boundary edge (curl grad = 0), so the product keeps
// no trace of the curl-curl scale that swamps w sigma Ms in the air when
// B x is evaluated in FP32.
// ---------------------------------------------------------------------------
void build_gtb_pattern(Context &c) {
  c.tiles.clear();
  const int nv = c.nv, nt = c.nt;
  std::vector<int> v2t_rp(nv + 1, 0), v2t;
  for (int t = 0; t < nt; ++t)
    for (int i = 0; i < 4; ++i) v2t_rp[c.h_tets[4 * (size_t)t + i] + 1]++;
  for (int v = 0; v < nv; ++v) v2t_rp[v + 1] += v2t_rp[v];
  v2t.resize(v2t_rp[nv]);
  {
    std::vector<int> pos(v2t_rp.begin(), v2t_rp.end() - 1);
    for (int t = 0; t < nt; ++t)
      for (int i = 0; i < 4; ++i) v2t[pos[c.h_tets[4 * (size_t)t + i]]++] = t;
  }
  std::vector<int> cnt(nv + 1, 0);
#pragma omp parallel
  {
    std::vector<int> buf;
#pragma omp for schedule(dynamic, 4096)
    for (int v = 0; v < nv; ++v) {
      buf.clear();
      for (int k = v2t_rp[v]; k < v2t_rp[v + 1]; ++k)
        for (int i = 0; i < 6; ++i) buf.push_back(c.h_t2e[6 * (size_t)v2t[k] + i]);
      std::sort(buf.begin(), buf.end());
      cnt[v + 1] = (int)(std::unique(buf.begin(), buf.end()) - buf.begin());
    }
  }
  c.h_grp.assign(nv + 1, 0);
  for (int v = 0; v < nv; ++v) c.h_grp[v + 1] = c.h_grp[v] + cnt[v + 1];
  c.h_gci.resize(c.h_grp[nv]);
#pragma omp parallel
  {
    std::vector<int> buf;
#pragma omp for schedule(dynamic, 4096)
    for (int v = 0; v < nv; ++v) {
      buf.clear();
      for (int k = v2t_rp[v]; k < v2t_rp[v + 1]; ++k)
        for (int i = 0; i < 6; ++i) buf.push_back(c.h_t2e[6 * (size_t)v2t[k] + i]);
      std::sort(buf.begin(), buf.end());
      int u = (int)(std::unique(buf.begin(), buf.end()) - buf.begin());
      std::copy(buf.begin(), buf.begin() + u, c.h_gci.begin() + c.h_grp[v]);
    }
  }
  c.grp.upload(c.h_grp, c.stream);
  c.gci.upload(c.h_gci, c.stream);
}

// gslot[t*24 + p*6 + k] = slot of (ctet[t][p], cedge[t][k]) in the G^T B pattern
__global__ void gslot_map_kernel(int nt, const int *__restrict__ ctet, const int *__restrict__ cedge,
                                 const int *__restrict__ rp, const int *__restrict__ ci, int *__restrict__ slot) {
  long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (idx >= (long)nt * 24) return;
  int t = (int)(idx / 24), ent = (int)(idx % 24);
  int row = __ldg(ctet + 4 * (long)t + ent / 6), col = __ldg(cedge + 6 * (long)t + ent % 6);
  slot[idx] = find_col(ci, __ldg(rp + row), __ldg(rp + row + 1), col);
}

__global__ void __launch_bounds__(128) assemble_gtb_kernel(ElemIn in, int nt, const int *__restrict__ gslot,
                                                            double *__restrict__ gc, double *__restrict__ gm) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  double c[36], m[36];
  TetGeom g;
  const bool touches_bdr = element_matrices(in, t, c, m, g);
  // (G_e^T K)[p][k] = sum over local edges j=(a,b): (-1 if p==a, +1 if p==b) K[j][k]
#pragma unroll
  for (int p = 0; p < 4; ++p) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      double vm = 0, vc = 0;
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        const double sgn = (kEdgeP(j) == p) ? -1.0 : ((kEdgeQ(j) == p) ? 1.0 : 0.0);
        if (sgn != 0.0) {
          vm += sgn * m[j * 6 + k];
          vc += sgn * c[j * 6 + k];
        }
      }
      const int sl = __ldg(gslot + 24 * (long)t + p * 6 + k);
      atomicAdd(gm + sl, vm);
      if (touches_bdr) atomicAdd(gc + sl, vc);
    }
  }
}

void assemble_gtb(Context &c, DBuf<double> &gc, DBuf<double> &gm) {
  if (c.h_grp.empty()) build_gtb_pattern(c);
  if (!c.gslot.p) {
    c.gslot.alloc((size_t)c.nt * 24);
    long n24 = (long)c.nt * 24;
    gslot_map_kernel<<<(unsigned)((n24 + 255) / 256), 256, 0, c.stream>>>(c.nt, c.ctet.p, c.cedge.p, c.grp.p, c.gci.p,
                                                                          c.gslot.p);
    EMG_LAUNCH_CHECK();
  }
  long nnz = c.h_grp[c.nv];
  gc.alloc(nnz);
  gm.alloc(nnz);
  gc.zero(c.stream);
  gm.zero(c.stream);
  assemble_gtb_kernel<<<(unsigned)((c.nt + 127) / 128), 128, 0, c.stream>>>(elem_in(c), c.nt, c.gslot.p, gc.p, gm.p);
  EMG_LAUNCH_CHECK();
}

}  // namespace emg
