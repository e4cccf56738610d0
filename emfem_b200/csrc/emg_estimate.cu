// Goal-oriented error indicator and RHS lifting kernels.
//
// estimate_error (src/em_fwd.cc:1102-1180): per tet the volume residual
//   sum_q |i w sigma e(q)|^2 jxw * R_t^2          (integrate_over_cell, :1005-1043)
// plus, per interior face, the normal-current and tangential-curl jumps
//   (sum_q |((sigma e) - (sigma_n e_n)).n|^2 jxw + |(curl e - curl e_n) x n|^2 jxw) R_f / 2
// (integrate_over_face, :1045-1100), credited in full to both tets.  A face is
// evaluated once, by the tet with the lower index and from its side, exactly
// as the reference's face_errors(t, f) >= 0 test arranges in its ascending tet
// loop; boundary faces contribute 0.  R_t, R_f are circumradii
// (src/em_mesh.h:232-274); the face rule is the reference's 3-point rule whose
// weights sum to 6x the face area (em_fe.cc:46-80).  Solutions are complex
// interleaved per edge.

#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <vector>

#include "emg_internal.h"
#include "emg_kernels.cuh"

namespace emg {

struct EstIn {
  const double *pts;
  const int *ctet, *cedge, *attr, *tets, *nbr, *non;
  const signed char *cpar;
  const double *sig;
  int nsol;
  const double2 *sol[3];
  double omega;
};

__device__ __forceinline__ void load_sigma(const EstIn &in, int t, double s[9]) {
  const double *sg = in.sig + 9 * (long)__ldg(in.attr + t);
#pragma unroll
  for (int k = 0; k < 9; ++k) s[k] = __ldg(sg + k);
}

__device__ __forceinline__ double dist3(const double *a, const double *b) {
  double dx = a[0] - b[0], dy = a[1] - b[1], dz = a[2] - b[2];
  return sqrt(dx * dx + dy * dy + dz * dz);
}

__device__ __forceinline__ void cmad(double2 &a, double f, double2 u) {  // a += f u
  a.x = fma(f, u.x, a.x);
  a.y = fma(f, u.y, a.y);
}

// One side of a face: the tet's vertices in the order a < b < c of the face's
// global ids, then the opposite vertex o.
struct FaceSide {
  double g[4][3];  // barycentric gradients
  double h[4];     // g_i . (sigma^T n): normal current of the unit gradient
  double m[4];     // g_i . n
  int eo[3];       // edges (a, o), (b, o), (c, o)
  double so[3];    // +1 where the edge runs towards o
};

// canonical edge joining sorted positions i < j
__device__ __forceinline__ int edge_of(int i, int j) { return i == 0 ? j - 1 : (i == 1 ? j + 1 : 5); }
__device__ __forceinline__ int at4(const int4 &v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }

// gradients of tet t seen from its face opposite sorted position p; x: the
// vertices (a, b, c, o); returns the determinant of the ordered tet
__device__ __forceinline__ double face_side(const EstIn &in, int t, const int4 &v, int p, double x[4][3], FaceSide &f) {
  const int q[4] = {p == 0 ? 1 : 0, p <= 1 ? 2 : 1, p <= 2 ? 3 : 2, p};
  const int vo = at4(v, p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int vi = at4(v, q[i]);
#pragma unroll
    for (int d = 0; d < 3; ++d) x[i][d] = __ldg(in.pts + 3 * (long)vi + d);
    if (i < 3) {
      f.eo[i] = __ldg(in.cedge + 6 * (long)t + edge_of(min(q[i], p), max(q[i], p)));
      f.so[i] = vi < vo ? 1.0 : -1.0;
    }
  }
  double e1[3], e2[3], e3[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    e1[d] = x[1][d] - x[0][d];
    e2[d] = x[2][d] - x[0][d];
    e3[d] = x[3][d] - x[0][d];
  }
  const double c23[3] = {e2[1] * e3[2] - e2[2] * e3[1], e2[2] * e3[0] - e2[0] * e3[2], e2[0] * e3[1] - e2[1] * e3[0]};
  const double c31[3] = {e3[1] * e1[2] - e3[2] * e1[1], e3[2] * e1[0] - e3[0] * e1[2], e3[0] * e1[1] - e3[1] * e1[0]};
  const double c12[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
  const double det = e1[0] * c23[0] + e1[1] * c23[1] + e1[2] * c23[2], inv = 1.0 / det;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    f.g[1][d] = c23[d] * inv;
    f.g[2][d] = c31[d] * inv;
    f.g[3][d] = c12[d] * inv;
    f.g[0][d] = -(f.g[1][d] + f.g[2][d] + f.g[3][d]);
  }
  return det;
}

__device__ __forceinline__ void face_weights(const EstIn &in, int t, const double n[3], FaceSide &f) {
  double s[9];
  load_sigma(in, t, s);
  double sn[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) sn[d] = s[d] * n[0] + s[3 + d] * n[1] + s[6 + d] * n[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f.h[i] = f.g[i][0] * sn[0] + f.g[i][1] * sn[1] + f.g[i][2] * sn[2];
    f.m[i] = f.g[i][0] * n[0] + f.g[i][1] * n[1] + f.g[i][2] * n[2];
  }
}

// Adds sign times the side's normal current at the face's three vertices to j
// and its curl x n to c, from the face's edge values (ab, ac, bc) and the
// three to the opposite vertex.  At vertex a only the edges that end there
// count: phi_(p,q) = l_p grad l_q - l_q grad l_p; and (g_p x g_q) x n =
// g_q (g_p . n) - g_p (g_q . n).
__device__ __forceinline__ void face_terms(const FaceSide &f, const double2 uf[3], const double2 uo[3], double sign,
                                           double2 j[3], double2 c[3]) {
  double2 v[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
  auto edge = [&](int p, int q, double2 u, double s) {
    if (p < 3) cmad(j[p], sign * s * f.h[q], u);
    if (q < 3) cmad(j[q], -sign * s * f.h[p], u);
    cmad(v[q], s * f.m[p], u);
    cmad(v[p], -s * f.m[q], u);
  };
  edge(0, 1, uf[0], 1.0);
  edge(0, 2, uf[1], 1.0);
  edge(1, 2, uf[2], 1.0);
#pragma unroll
  for (int i = 0; i < 3; ++i) edge(i, 3, uo[i], f.so[i]);
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int i = 0; i < 4; ++i) cmad(c[d], 2.0 * sign * f.g[i][d], v[i]);
}

// One thread per interior face (faces[i] = 4 t + f with t the lower tet): both
// tets' jumps, written to fe[(s*T + t)*4 + f] of both (integrate_over_face).
// The normal current is linear on the face, so its values at the three
// vertices give it at the quadrature points (1/2 of the vertex they are near
// plus 1/6 of all three), and the edges of the face belong to both tets: the
// kernel needs no quadrature points, no basis functions and 9 edge values.
// Bound: latency (194 registers leave 7.5 warps per SM; L1 30 %, FP64 22 %);
// nothing spills (it evaluated both fields at three points, spilled 1.1 KB per
// thread, and half its threads, one per (tet, face), left at once).
__global__ void __launch_bounds__(128) estimate_face_kernel(EstIn in, int nt, int nfaces,
                                                            const int *__restrict__ faces, double *__restrict__ fe) {
  const int i = blockIdx.x * 128 + threadIdx.x;
  if (i >= nfaces) return;
  const int id = __ldg(faces + i), t = id >> 2;
  const int n = __ldg(in.nbr + id), non = __ldg(in.non + id);
  const int4 vt = __ldg(reinterpret_cast<const int4 *>(in.ctet) + t);
  const int4 vn = __ldg(reinterpret_cast<const int4 *>(in.ctet) + n);
  const int ot = __ldg(in.tets + id), on = __ldg(in.tets + 4 * (long)n + non);
  const int p = ot == vt.x ? 0 : (ot == vt.y ? 1 : (ot == vt.z ? 2 : 3));
  const int pn = on == vn.x ? 0 : (on == vn.y ? 1 : (on == vn.z ? 2 : 3));
  FaceSide a, b;
  double nrm[3], jxw, fd;
  {
    double x[4][3];
    const double det = face_side(in, t, vt, p, x, a);
    // outward normal -grad(l_o)/|grad(l_o)| and the reference's face weight
    const double gl = sqrt(a.g[3][0] * a.g[3][0] + a.g[3][1] * a.g[3][1] + a.g[3][2] * a.g[3][2]);
#pragma unroll
    for (int d = 0; d < 3; ++d) nrm[d] = -a.g[3][d] / gl;
    jxw = gl * fabs(det);
    // circumradius of the face (src/em_mesh.h:256-274)
    const double la = dist3(x[1], x[2]), lb = dist3(x[0], x[2]), lc = dist3(x[0], x[1]);
    const double area = 0.25 * sqrt((la + lb + lc) * (lb + lc - la) * (lc + la - lb) * (la + lb - lc));
    fd = la * lb * lc / (4.0 * area);
    face_side(in, n, vn, pn, x, b);
  }
  face_weights(in, t, nrm, a);
  face_weights(in, n, nrm, b);
  const int qa = p == 0 ? 1 : 0, qb = p <= 1 ? 2 : 1, qc = p <= 2 ? 3 : 2;
  const int ef[3] = {__ldg(in.cedge + 6 * (long)t + edge_of(qa, qb)), __ldg(in.cedge + 6 * (long)t + edge_of(qa, qc)),
                     __ldg(in.cedge + 6 * (long)t + edge_of(qb, qc))};
#pragma unroll 1
  for (int s = 0; s < in.nsol; ++s) {
    const double2 *u = in.sol[s];
    const double2 uf[3] = {__ldg(u + ef[0]), __ldg(u + ef[1]), __ldg(u + ef[2])};
    const double2 ua[3] = {__ldg(u + a.eo[0]), __ldg(u + a.eo[1]), __ldg(u + a.eo[2])};
    const double2 ub[3] = {__ldg(u + b.eo[0]), __ldg(u + b.eo[1]), __ldg(u + b.eo[2])};
    double2 j[3] = {{0, 0}, {0, 0}, {0, 0}}, c[3] = {{0, 0}, {0, 0}, {0, 0}};
    face_terms(a, uf, ua, 1.0, j, c);
    face_terms(b, uf, ub, -1.0, j, c);
    const double tx = (j[0].x + j[1].x + j[2].x) / 6.0, ty = (j[0].y + j[1].y + j[2].y) / 6.0;
    double v = 0;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double jr = 0.5 * j[q].x + tx, ji = 0.5 * j[q].y + ty;
      v += jr * jr + ji * ji + 3.0 * (c[q].x * c[q].x + c[q].y * c[q].y);
    }
    v *= jxw * fd / 2.0;
    fe[((long)s * nt + t) * 4 + (id & 3)] = v;
    fe[((long)s * nt + n) * 4 + non] = v;
  }
}

// eta[s][t] = volume term (integrate_over_cell) + the four face terms in the
// reference's order, then the primal x dual combination sqrt(eta_p * eta_d)
// (src/em_fwd.cc:1172-1177).  The field at a quadrature point is B times the
// sum of its values at the four vertices plus (A - B) times the value at the
// vertex the point is near.
__global__ void __launch_bounds__(128) estimate_cell_kernel(EstIn in, int nt, const double *__restrict__ fe,
                                                            double *__restrict__ eta, double *__restrict__ err) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  TetGeom g;
  load_tet_geom(in.pts, in.ctet, in.cedge, in.cpar, t, g);
  double sg[9];
  load_sigma(in, t, sg);
  // circumradius of the tet (src/em_mesh.h:232-254)
  double diam;
  {
    double a = dist3(g.x[1], g.x[2]), b = dist3(g.x[0], g.x[2]), c = dist3(g.x[0], g.x[1]);
    double aa = dist3(g.x[0], g.x[3]), bb = dist3(g.x[1], g.x[3]), cc = dist3(g.x[2], g.x[3]);
    double la = a * aa, lb = b * bb, lc = c * cc;
    double sh = 0.5 * (la + lb + lc);
    diam = sqrt(sh * (sh - la) * (sh - lb) * (sh - lc)) / (6.0 * g.vol);
  }
  const double A = 0.585410196624969, B = 0.138196601125011;
  const double w = in.omega * in.omega * (g.vol * 6.0 / 24.0) * diam * diam;  // omega^2 det(J)/24 R^2
  const int4 nb = __ldg(reinterpret_cast<const int4 *>(in.nbr) + t);
  double es[3] = {0, 0, 0};
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    if (s >= in.nsol) break;
    // sigma e at the four vertices: the edges that end there
    double2 y[4][3], sum[3] = {{0, 0}, {0, 0}, {0, 0}};
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int d = 0; d < 3; ++d) y[p][d] = make_double2(0, 0);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int p = kEdgeP(k), q = kEdgeQ(k);
      const double2 u = __ldg(in.sol[s] + g.ge[k]);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        cmad(y[p][d], g.gr[q][d], u);
        cmad(y[q][d], -g.gr[p][d], u);
      }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      double2 z[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        z[d] = make_double2(0, 0);
#pragma unroll
        for (int c = 0; c < 3; ++c) cmad(z[d], sg[3 * d + c], y[p][c]);
        sum[d].x += z[d].x;
        sum[d].y += z[d].y;
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) y[p][d] = z[d];
    }
    double v = 0;
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double re = fma(A - B, y[p][d].x, B * sum[d].x), im = fma(A - B, y[p][d].y, B * sum[d].y);
        v += re * re + im * im;
      }
    v *= w;
    const long o = ((long)s * nt + t) * 4;
    if (nb.x >= 0) v += fe[o];
    if (nb.y >= 0) v += fe[o + 1];
    if (nb.z >= 0) v += fe[o + 2];
    if (nb.w >= 0) v += fe[o + 3];
    eta[(long)s * nt + t] = v;
    es[s] = v;
  }
  if (!err) return;
  const double dual = in.nsol == 3 ? es[2] : es[1];
#pragma unroll
  for (int s = 0; s < 2; ++s)
    if (s < in.nsol - 1) err[(long)s * nt + t] = sqrt(es[s] * dual);
}

void launch_estimate(Context &c, double omega, int nsol, const double *const *sol_dev, double *eta_dev,
                     double *err_dev, double *scratch_fe) {
  EstIn in;
  in.pts = c.pts.p;
  in.ctet = c.ctet.p;
  in.cedge = c.cedge.p;
  in.attr = c.attr.p;
  in.tets = c.tets.p;
  in.nbr = c.nbr.p;
  in.non = c.non.p;
  in.cpar = c.cpar.p;
  in.sig = c.sigma_tab.p;
  in.nsol = nsol;
  for (int s = 0; s < 3; ++s) in.sol[s] = s < nsol ? (const double2 *)sol_dev[s] : nullptr;
  in.omega = omega;
  if (c.n_faces > 0) {
    estimate_face_kernel<<<(unsigned)((c.n_faces + 127) / 128), 128, 0, c.stream>>>(in, c.nt, c.n_faces, c.faces,
                                                                                    scratch_fe);
    EMG_LAUNCH_CHECK();
  }
  estimate_cell_kernel<<<(unsigned)((c.nt + 127) / 128), 128, 0, c.stream>>>(in, c.nt, scratch_fe, eta_dev, err_dev);
  EMG_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// MT boundary lifting (assemble_rhs_mt, src/em_fwd.cc:516-572) for k boundary
// value sets at once: bv[e*k + j] (complex) holds the Dirichlet value of
// boundary edge e for column j; out s (complex interleaved, n x k).
// ---------------------------------------------------------------------------
struct LiftIn {
  const double *pts;
  const int *ctet, *cedge, *attr;
  const signed char *cpar;
  const unsigned char *ebdr, *bdr_cell;
  const double *sig;
};

__global__ void __launch_bounds__(128) rhs_mt_kernel(LiftIn in, int nt, int k, const double *__restrict__ omega,
                                                     const double2 *__restrict__ bv, const int *__restrict__ brank,
                                                     double *__restrict__ s) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt || !__ldg(in.bdr_cell + t)) return;
  TetGeom g;
  load_tet_geom(in.pts, in.ctet, in.cedge, in.cpar, t, g);
  const double *sgp = in.sig + 9 * (long)__ldg(in.attr + t);
  double sg[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) sg[q] = __ldg(sgp + q);
  double S[10];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = p; q < 4; ++q) {
      double a0 = sg[0] * g.gr[q][0] + sg[1] * g.gr[q][1] + sg[2] * g.gr[q][2];
      double a1 = sg[3] * g.gr[q][0] + sg[4] * g.gr[q][1] + sg[5] * g.gr[q][2];
      double a2 = sg[6] * g.gr[q][0] + sg[7] * g.gr[q][1] + sg[8] * g.gr[q][2];
      S[sym_idx(p, q)] = g.gr[p][0] * a0 + g.gr[p][1] * a1 + g.gr[p][2] * a2;
    }
  double cu[6][3];
#pragma unroll
  for (int e = 0; e < 6; ++e) {
    const int a = kEdgeP(e), b = kEdgeQ(e);
    cu[e][0] = 2.0 * (g.gr[a][1] * g.gr[b][2] - g.gr[a][2] * g.gr[b][1]);
    cu[e][1] = 2.0 * (g.gr[a][2] * g.gr[b][0] - g.gr[a][0] * g.gr[b][2]);
    cu[e][2] = 2.0 * (g.gr[a][0] * g.gr[b][1] - g.gr[a][1] * g.gr[b][0]);
  }
  bool bd[6];
#pragma unroll
  for (int e = 0; e < 6; ++e) bd[e] = __ldg(in.ebdr + g.ge[e]) != 0;
  const double vc = g.vol / MU, vm = g.vol / 20.0;
  for (int j = 0; j < k; ++j) {
    const double w = __ldg(omega + j);
    double br[6] = {0, 0, 0, 0, 0, 0}, bi[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      if (!bd[i]) continue;
      double2 v = __ldg(bv + (long)__ldg(brank + g.ge[i]) * k + j);
      double cii = vc * (cu[i][0] * cu[i][0] + cu[i][1] * cu[i][1] + cu[i][2] * cu[i][2]);
      br[i] += v.x * cii;
      bi[i] += -v.y * cii;
#pragma unroll
      for (int l = 0; l < 6; ++l) {
        if (bd[l]) continue;
        const int p = kEdgeP(l), q = kEdgeQ(l), r = kEdgeP(i), u = kEdgeQ(i);
        double cli = vc * (cu[l][0] * cu[i][0] + cu[l][1] * cu[i][1] + cu[l][2] * cu[i][2]);
        double mli = w * vm *
                     ((1.0 + (p == r)) * S[sym_idx(q, u)] - (1.0 + (p == u)) * S[sym_idx(q, r)] -
                      (1.0 + (q == r)) * S[sym_idx(p, u)] + (1.0 + (q == u)) * S[sym_idx(p, r)]);
        br[l] -= cli * v.x;
        bi[l] += mli * v.x;
        br[l] += mli * v.y;
        bi[l] += cli * v.y;
      }
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      atomicAdd(s + 2 * ((long)g.ge[i] * k + j), br[i]);
      atomicAdd(s + 2 * ((long)g.ge[i] * k + j) + 1, bi[i]);
    }
  }
}

void launch_rhs_mt(Context &c, int k, const double *omega_dev, const double *bv_dev, const int *brank_dev,
                   double *s_dev) {
  LiftIn in{c.pts.p, c.ctet.p, c.cedge.p, c.attr.p, c.cpar.p, c.ebdr.p, c.bdr_cell.p, c.sigma_tab.p};
  EMG_CUDA(cudaMemsetAsync(s_dev, 0, sizeof(double) * 2 * (size_t)c.ne * k, c.stream));
  rhs_mt_kernel<<<(unsigned)((c.nt + 127) / 128), 128, 0, c.stream>>>(in, c.nt, k, omega_dev, (const double2 *)bv_dev,
                                                                      brank_dev, s_dev);
  EMG_LAUNCH_CHECK();
}

}  // namespace emg

// ---------------------------------------------------------------------------
// Error estimate without any device allocation.
//
// emg_estimate_error obtains its per-tet and per-face scratch from the
// context's workspace, which the library allocates with cudaMalloc on first
// use.  Some callers cannot allow an allocation at that point -- a host
// application whose memory manager owns all device memory and forbids
// allocations once a run has started, or a caller that must not synchronise
// the device the way cudaMalloc/cudaFree can.  For them this variant keeps
// the scratch in a fixed file-scope device array and writes its results into
// device buffers the caller owns.
// ---------------------------------------------------------------------------
namespace {

constexpr int kNoAllocMaxTets = 131072;  // largest mesh the fixed scratch serves
constexpr int kNoAllocMaxSol = 3;        // MT: XY, YX and the dual solution

// face terms (n_sol x T x 4): 12.6 MB, held on every GPU that loads the library
// until the process exits
__device__ __align__(256) double g_estimate_scratch[kNoAllocMaxSol * kNoAllocMaxTets * 4];

}  // namespace

namespace emg {
// In host code g_estimate_scratch only names a host-side stand-in; the device
// address is looked up once per device, with that device current.  Device
// contexts call this when they are created, which also loads this file's
// module on that device, so emg_estimate_error_noalloc itself never loads a
// module or allocates.
double *noalloc_scratch_address(int device) {
  static std::mutex mu;
  static std::map<int, double *> addr;
  std::lock_guard<std::mutex> lock(mu);
  auto it = addr.find(device);
  if (it != addr.end()) return it->second;
  double *p = nullptr;
  emg::check_cuda(cudaGetSymbolAddress((void **)&p, g_estimate_scratch), "cudaGetSymbolAddress(g_estimate_scratch)",
                  __FILE__, __LINE__);
  addr[device] = p;
  return p;
}
}  // namespace emg

extern "C" int emg_estimate_error_noalloc(emg_context *ctx, int fidx, int tidx, double *err_dev, double *eta_dev) {
  using namespace emg;
  try {
    if (!ctx || !err_dev || !eta_dev) fail(EMG_ERR_ARG, "null argument");
    Context &c = *ctx;
    if (c.device < 0) fail(EMG_ERR_STATE, "host-only context has no device");
    if (!c.have_ls || c.nrho <= 0) fail(EMG_ERR_STATE, "estimate_error before create_linear_system");
    if (fidx < 0 || fidx >= (int)c.freqs.size()) fail(EMG_ERR_ARG, "frequency index out of range");
    if (c.nt > kNoAllocMaxTets)
      fail(EMG_ERR_ARG, "emg_estimate_error_noalloc serves meshes of at most %d tets (this one has %d); "
           "use emg_estimate_error", kNoAllocMaxTets, c.nt);
    const int slots3[3] = {EMG_SOL_MT_XY, EMG_SOL_MT_YX, EMG_SOL_DUAL};
    const int slots2[2] = {EMG_SOL_CSEM, EMG_SOL_DUAL};
    const int nsol = tidx < 0 ? 3 : 2;
    const double *sp[3];
    for (int s = 0; s < nsol; ++s) {
      auto it = c.sol.find(tidx < 0 ? slots3[s] : slots2[s]);
      if (it == c.sol.end() || it->second.n != (size_t)c.ne * 2) fail(EMG_ERR_STATE, "solution slot not created");
      sp[s] = it->second.p;
    }
    check_cuda(cudaSetDevice(c.device), "cudaSetDevice", __FILE__, __LINE__);
    double *scratch = noalloc_scratch_address(c.device);
    // every face entry is written before it is read, so nothing left in the
    // array by an earlier call needs clearing
    launch_estimate(c, 2 * PI * c.freqs[fidx], nsol, sp, eta_dev, err_dev, scratch);
    check_cuda(cudaStreamSynchronize(c.stream), "cudaStreamSynchronize", __FILE__, __LINE__);
  } catch (const Error &e) {
    set_last_error(e.what());
    return e.code;
  } catch (const std::exception &e) {
    set_last_error(e.what());
    return EMG_ERR_USER;
  }
  return EMG_OK;
}
