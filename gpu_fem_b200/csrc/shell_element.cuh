// Linear MITC4 shell element in explicit strain-displacement form.
//
// The reference evaluates the element with A2D forward/reverse sweeps per
// (element, quadrature point, Jacobian column)
// (include/shell/elem_group.h:98-303). Every map on that path is linear in
// the DOFs, so this file writes the same strains as E_q = B_q u with the
// 9 x 24 matrix B_q built entry by entry from per-element tables that are
// computed once:
//   membrane/shear rows  e0ty = (Xd^-1 T)^T gty (Xd^-1 T) from the MITC tying
//                        strains (include/shell/physics.h:94-209,
//                        include/shell/basis.h:314-502)
//   bending rows         u1x = T^T (u1d Xd^-1 T + u0d XdinvzT)
//                        (include/shell/basis.h:452-493)
//   drilling row         nodal drill strains interpolated to the point
//                        (include/shell/shell_utils.h:42-105)
// with the strain vector of LinearShellStrainCore
// (include/shell/a2d/a2dshellstrain.h:13-30) and the isotropic ABD stress of
// IsotropicShellStressCore (include/shell/a2d/a2disotropicshellstress.h:12-51).
// Then K_e = sum_q w_q detXd_q B_q^T D B_q and R_e = K_e u_e, which is the
// Hessian / gradient of the energy U = 1/2 sum_q w_q detXd_q E.S
// (include/shell/physics.h:19-37).
//
// Everything here is __host__ __device__ so the same code can be compiled
// for the CPU when checking the algebra.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define GF_HD __host__ __device__ __forceinline__
#else
#define GF_HD inline
#endif

namespace gf {

constexpr double kRt3 = 0.577350269189626;    // include/shell/quadrature.h:9
constexpr double kShear = 5.0 / 6.0;          // include/shell/data.h:11
constexpr double kDrill = 10.0;               // include/shell/data.h:12

// Material entry; per-element thickness is stored separately.
struct Material {
  double E, nu, tOffset;
  double refAxis[3];
  int has_ref_axis;
  int pad;
  // plane-stress stiffness (E / (1 - nu^2) times 1 and nu) and shear modulus,
  // a2disotropicshellstress.h:12-51
  double C0, C1, C5;
};
inline void material_constants(Material& m) {
  const double D = m.E / (1.0 - m.nu * m.nu);
  m.C0 = D;
  m.C1 = m.nu * D;
  m.C5 = m.E / 2.0 / (1.0 + m.nu);
}

// Node sign pattern of the tensor-product basis: node a sits at
// (xi_a, eta_a) = (-1 + 2 (a % 2), -1 + 2 (a / 2))  (basis.h:138-142).
GF_HD double node_xi(int a) { return (a & 1) ? 1.0 : -1.0; }
GF_HD double node_eta(int a) { return (a & 2) ? 1.0 : -1.0; }

// Bilinear shape function and its parametric derivatives at (xi, eta).
GF_HD void shape(int a, double xi, double eta, double& N, double& Nx, double& Ne) {
  const double sa = node_xi(a), ta = node_eta(a);
  const double fx = 0.5 * (1.0 + sa * xi), fe = 0.5 * (1.0 + ta * eta);
  N = fx * fe;
  Nx = 0.5 * sa * fe;
  Ne = 0.5 * ta * fx;
}

GF_HD void cross3(const double* a, const double* b, double* c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}
GF_HD double dot3(const double* a, const double* b) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

// Interpolated value and gradients of a 3-vector nodal field f[4][3].
GF_HD void interp3(const double* f, double xi, double eta, double* v, double* dxi,
                   double* deta) {
  for (int k = 0; k < 3; k++) v[k] = dxi[k] = deta[k] = 0.0;
  for (int a = 0; a < 4; a++) {
    double N, Nx, Ne;
    shape(a, xi, eta, N, Nx, Ne);
    for (int k = 0; k < 3; k++) {
      v[k] += N * f[3 * a + k];
      dxi[k] += Nx * f[3 * a + k];
      deta[k] += Ne * f[3 * a + k];
    }
  }
}

// 3x3 inverse (row-major) and determinant.
GF_HD double inv3(const double* A, double* B) {
  const double c0 = A[4] * A[8] - A[5] * A[7];
  const double c1 = A[3] * A[8] - A[5] * A[6];
  const double c2 = A[3] * A[7] - A[4] * A[6];
  const double det = A[0] * c0 - A[1] * c1 + A[2] * c2;
  const double id = 1.0 / det;
  B[0] = c0 * id;
  B[1] = -(A[1] * A[8] - A[2] * A[7]) * id;
  B[2] = (A[1] * A[5] - A[2] * A[4]) * id;
  B[3] = -c1 * id;
  B[4] = (A[0] * A[8] - A[2] * A[6]) * id;
  B[5] = -(A[0] * A[5] - A[2] * A[3]) * id;
  B[6] = c2 * id;
  B[7] = -(A[0] * A[7] - A[1] * A[6]) * id;
  B[8] = (A[0] * A[4] - A[1] * A[3]) * id;
  return det;
}
GF_HD void mm3(const double* A, const double* B, double* C) {
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++)
      C[3 * i + j] = A[3 * i] * B[j] + A[3 * i + 1] * B[3 + j] + A[3 * i + 2] * B[6 + j];
}

// ShellComputeTransform (include/shell/shell_utils.h:4-40): columns
// (t1, n x t1, n) with t1 = refAxis or dX/dxi projected off the normal.
GF_HD void shell_transform(const Material& m, const double* Xxi, const double* n0, double* T) {
  const double nn = sqrt(dot3(n0, n0));
  const double nh[3] = {n0[0] / nn, n0[1] / nn, n0[2] / nn};
  double t1[3];
  for (int i = 0; i < 3; i++) t1[i] = m.has_ref_axis ? m.refAxis[i] : Xxi[i];
  const double d = dot3(nh, t1);
  double tmp[3];
  for (int i = 0; i < 3; i++) tmp[i] = t1[i] - d * nh[i];
  const double tn = sqrt(dot3(tmp, tmp));
  const double t1h[3] = {tmp[0] / tn, tmp[1] / tn, tmp[2] / tn};
  double t2h[3];
  cross3(nh, t1h, t2h);
  for (int i = 0; i < 3; i++) {
    T[3 * i] = t1h[i];
    T[3 * i + 1] = t2h[i];
    T[3 * i + 2] = nh[i];
  }
}

GF_HD void quad_point(int q, double& xi, double& eta) {
  xi = (q & 1) ? kRt3 : -kRt3;
  eta = (q & 2) ? kRt3 : -kRt3;
}

// Element data from which every entry of the four B_q follows with a few
// multiplications. One element of a chunk; the assembled K_e overlays it once
// its strains have been used (kKeStride doubles a row).
constexpr int kKeStride = 26;  // padded rows: mirrored columns land in different banks
struct ElemData {
  // per DOF column l = 6a + c, independent of the quadrature point: tying
  // strains g11, g22, g12, g23, g13 of the column (before the interpolation
  // along the edges), the two factors of its director (or unit) vector
  // against the columns of T, an unused entry, and its nodal drill strains
  double tab[24][12];
  double M[4][5][6];   // E0, E1, E2, E6, E7 from (g11, g22, g12, g23, g13)
  double R[4][2][4][2];  // bending: (u1d Xd^-1 T + u0d XdinvzT) of [q][translation/rotation][node]
  double T[4][6];      // first two columns of the shell frame, [q][2 c + i]
  double scale[4];     // detXd * weight
  // sources of the tables
  double AA[4][10];    // Xd^-1 T (rows 0, 1) and XdinvzT (rows 0, 1, 2), first two columns
  double Tn[4][6];     // nodal frames, first two columns
  double XT[4][4];     // nodal Xd^-1 T, rows 0, 1, first two columns
  double tc[4][3];     // nodal T[:,0] x T[:,1]
  double fn[12];       // unit node normals (ShellComputeNodeNormals, basis.h:292-311)
  double X[12];
  double pad[10];      // elements start in different banks
};
static_assert(sizeof(ElemData) >= sizeof(double) * 24 * kKeStride, "K_e overlays ElemData");

GF_HD void elem_normal(const double* X, int n, double* fn) {
  double v[3], xi[3], eta[3], c[3];
  interp3(X, node_xi(n), node_eta(n), v, xi, eta);
  cross3(xi, eta, c);
  const double nrm = sqrt(dot3(c, c));
  for (int k = 0; k < 3; k++) fn[k] = (1.0 / nrm) * c[k];
}

// Frame of a point: Xd = [Xxi Xeta n0] with the interpolated node normals n0
// (at a node: its own), its inverse and determinant, the shell frame T and
// A = Xd^-1 T.
struct PointFrame {
  double T[9], A[9], Xdi[9], nxi[3], neta[3], det;
};
GF_HD void point_frame(const double* X, const double* fn, const Material& m, double xi, double eta,
                       PointFrame& f) {
  double xv[3], Xxi[3], Xeta[3], n0[3], Xd[9];
  interp3(X, xi, eta, xv, Xxi, Xeta);
  interp3(fn, xi, eta, n0, f.nxi, f.neta);
  for (int i = 0; i < 3; i++) {
    Xd[3 * i] = Xxi[i];
    Xd[3 * i + 1] = Xeta[i];
    Xd[3 * i + 2] = n0[i];
  }
  shell_transform(m, Xxi, n0, f.T);
  f.det = inv3(Xd, f.Xdi);
  mm3(f.Xdi, f.T, f.A);
}
// XdinvzT = -Xd^-1 Xdz Xd^-1 T, first two columns (Xdz = [n_xi n_eta 0])
GF_HD void point_bending(const PointFrame& f, double (*Az)[2]) {
  for (int i = 0; i < 3; i++) {
    const double d0 =
        f.Xdi[3 * i] * f.nxi[0] + f.Xdi[3 * i + 1] * f.nxi[1] + f.Xdi[3 * i + 2] * f.nxi[2];
    const double d1 =
        f.Xdi[3 * i] * f.neta[0] + f.Xdi[3 * i + 1] * f.neta[1] + f.Xdi[3 * i + 2] * f.neta[2];
    for (int j = 0; j < 2; j++) Az[i][j] = -(d0 * f.A[j] + d1 * f.A[3 + j]);
  }
}
// E0, E1, E2, E6, E7 from the packed tying strains (g11, g22, g12, g23, g13):
// e_ab = sum_ij A_ia G_ij A_jb, g33 = 0
GF_HD void tying_rows(const double* A, double (*M)[5]) {
  const int pa[5] = {0, 1, 0, 1, 0}, pb[5] = {0, 1, 1, 2, 2};
  for (int k = 0; k < 5; k++) {
    const int a = pa[k], b = pb[k];
    const double w = k < 2 ? 1.0 : 2.0;
    M[k][0] = w * (A[a] * A[b]);
    M[k][1] = w * (A[3 + a] * A[3 + b]);
    M[k][2] = w * (A[a] * A[3 + b] + A[3 + a] * A[b]);
    M[k][3] = w * (A[3 + a] * A[6 + b] + A[6 + a] * A[3 + b]);
    M[k][4] = w * (A[a] * A[6 + b] + A[6 + a] * A[b]);
  }
}

// Point pt of an element: nodes 0..3 (drill strain, shell_utils.h:42-105),
// then the quadrature points 4..7.
GF_HD void elem_point(ElemData& g, const Material& m, int pt) {
  double xi, eta;
  const int q = pt & 3;
  if (pt < 4) {
    xi = node_xi(q);
    eta = node_eta(q);
  } else {
    quad_point(q, xi, eta);
  }
  PointFrame f;
  point_frame(g.X, g.fn, m, xi, eta, f);
  double* T = pt < 4 ? g.Tn[q] : g.T[q];
  for (int c = 0; c < 3; c++) {
    T[2 * c] = f.T[3 * c];
    T[2 * c + 1] = f.T[3 * c + 1];
  }
  if (pt < 4) {
    g.XT[q][0] = f.A[0];
    g.XT[q][1] = f.A[1];
    g.XT[q][2] = f.A[3];
    g.XT[q][3] = f.A[4];
    const double t0[3] = {f.T[0], f.T[3], f.T[6]}, t1[3] = {f.T[1], f.T[4], f.T[7]};
    cross3(t0, t1, g.tc[q]);
    return;
  }
  double Az[3][2], M[5][5];
  point_bending(f, Az);
  for (int j = 0; j < 2; j++) {
    g.AA[q][j] = f.A[j];
    g.AA[q][2 + j] = f.A[3 + j];
    for (int i = 0; i < 3; i++) g.AA[q][4 + 2 * i + j] = Az[i][j];
  }
  g.scale[q] = f.det;  // quadrature weight is 1 (quadrature.h:13-17)
  tying_rows(f.A, M);
  for (int k = 0; k < 5; k++) {
    for (int z = 0; z < 5; z++) g.M[q][k][z] = M[k][z];
    g.M[q][k][5] = 0.0;
  }
}

// Table of DOF column l = 6a + c (MITC tying strain sensitivities,
// physics.h:94-209, and nodal drill strains, shell_utils.h:42-105). A node's
// shape functions vanish on the edges it does not lie on, so each tying
// strain of a column comes from the one point of its node's edge.
GF_HD void elem_column(ElemData& g, int l) {
  const int a = l / 6, c = l % 6, ia = a & 1, ja = a >> 1;
  const double sa = node_xi(a), ta = node_eta(a);
  const double* f = &g.fn[3 * a];
  const double *X0 = &g.X[6 * ja], *X1 = X0 + 3;           // the node's edge along xi
  const double *Y0 = &g.X[3 * ia], *Y1 = Y0 + 6;           // ... along eta
  double* t = g.tab[l];
  t[7] = 0.0;
  if (c < 3) {
    t[0] = 0.5 * sa * (0.5 * (X1[c] - X0[c]));
    t[1] = 0.5 * ta * (0.5 * (Y1[c] - Y0[c]));
    // centre tangents, summed over the nodes in order like every interpolation
    const double Xc = 0.25 * (((g.X[3 + c] - g.X[c]) - g.X[6 + c]) + g.X[9 + c]);
    const double Yc = 0.25 * (((-g.X[c] - g.X[3 + c]) + g.X[6 + c]) + g.X[9 + c]);
    t[2] = 0.5 * (0.25 * sa * Yc + 0.25 * ta * Xc);
    t[3] = 0.25 * ta * (0.5 * (g.fn[3 * ia + c] + g.fn[3 * ia + 6 + c]));
    t[4] = 0.25 * sa * (0.5 * (g.fn[6 * ja + c] + g.fn[6 * ja + 3 + c]));
    t[5] = 1.0;
    t[6] = 0.0;
    for (int n = 0; n < 4; n++) {
      const double Nx = (n >> 1) == ja ? 0.5 * sa : 0.0, Ne = (n & 1) == ia ? 0.5 * ta : 0.0;
      const double s0 = Nx * g.XT[n][0] + Ne * g.XT[n][2];
      const double s1 = Nx * g.XT[n][1] + Ne * g.XT[n][3];
      t[8 + n] = 0.5 * (g.Tn[n][2 * c + 1] * s0 - g.Tn[n][2 * c] * s1);
    }
  } else {
    // X . (e_k x f) = (f x X)_k: director sensitivity (director.h:98-107)
    const int k = c - 3, k1 = k == 2 ? 0 : k + 1, k2 = k == 0 ? 2 : k - 1;
    t[0] = t[1] = t[2] = 0.0;
    t[3] = 0.125 * (f[k1] * (Y1[k2] - Y0[k2]) - f[k2] * (Y1[k1] - Y0[k1]));
    t[4] = 0.125 * (f[k1] * (X1[k2] - X0[k2]) - f[k2] * (X1[k1] - X0[k1]));
    t[5] = f[k1];
    t[6] = f[k2];
    for (int n = 0; n < 4; n++) t[8 + n] = n == a ? -g.tc[a][k] : 0.0;
  }
}
// entry R[q][rot][a]: bending factors of node a's translations / rotations
// (basis.h:452-493)
GF_HD void elem_bending(ElemData& g, int q, int rot, int a) {
  double xi, eta, N, Nx, Ne;
  quad_point(q, xi, eta);
  shape(a, xi, eta, N, Nx, Ne);
  const double* A = g.AA[q];
  for (int j = 0; j < 2; j++)
    g.R[q][rot][a][j] =
        rot ? Nx * A[j] + Ne * A[2 + j] + N * A[8 + j] : Nx * A[4 + j] + Ne * A[6 + j];
}

// What a thread keeps of column l at quadrature point q: the interpolated
// tying strains g[5] and the bending and drill strains.
struct ColumnAt {
  double g[5], e3, e4, e5, e8;
};
GF_HD ColumnAt column_at(const ElemData& d, int l, int q) {
  const int a = l / 6, c = l % 6;
  double xi, eta;
  quad_point(q, xi, eta);
  const double na = 0.5 * (1.0 + node_xi(a) * xi), nb = 0.5 * (1.0 + node_eta(a) * eta);
  const double* t = d.tab[l];
  ColumnAt o;
  // interpTyingStrain (basis.h:314-368)
  o.g[0] = nb * t[0];
  o.g[1] = na * t[1];
  o.g[2] = t[2];
  o.g[3] = na * t[3];
  o.g[4] = nb * t[4];
  // w = T^T (e_c) for translations, T^T (e_k x f) = (f x T)_k for rotations
  const int k = c - 3;
  const int i1 = c < 3 ? c : (k == 0 ? 2 : k - 1), i2 = c < 3 ? c : (k == 2 ? 0 : k + 1);
  const double* T = d.T[q];
  const double w0 = t[5] * T[2 * i1] - t[6] * T[2 * i2];
  const double w1 = t[5] * T[2 * i1 + 1] - t[6] * T[2 * i2 + 1];
  const double* r = d.R[q][c < 3 ? 0 : 1][a];
  o.e3 = w0 * r[0];
  o.e4 = w1 * r[1];
  o.e5 = w0 * r[1] + w1 * r[0];
  const double x0 = 0.5 * (1.0 - xi), x1 = 0.5 * (1.0 + xi);
  const double y0 = 0.5 * (1.0 - eta), y1 = 0.5 * (1.0 + eta);
  o.e8 = x0 * y0 * t[8] + x1 * y0 * t[9] + x0 * y1 * t[10] + x1 * y1 * t[11];
  return o;
}
// row k (E0, E1, E2, E6, E7) of the membrane / transverse shear strains
GF_HD double tying_row(const ElemData& d, int q, int k, const double* g) {
  const double* m = d.M[q][k];
  return m[0] * g[0] + m[1] * g[1] + m[2] * g[2] + m[3] * g[3] + m[4] * g[4];
}

// Isotropic shell stiffnesses at a point, times the point's weight
// (a2disotropicshellstress.h:12-51): S = D E with the membrane-bending
// blocks a, b, d times (c0, c1; c1, c0) and c5, shear s, drill r.
struct Stiffness {
  double a0, a1, a5, b0, b1, b5, d0, d1, d5, s, r;
};
GF_HD Stiffness stiffness(const Material& m, double t, double w) {
  const double C0 = m.C0, C1 = m.C1, C5 = m.C5;
  const double to = m.tOffset;
  const double a = w * t, b = -w * t * t * to, d = w * (t * t * t / 12.0 + t * t * t * to * to);
  Stiffness o;
  o.a0 = a * C0, o.a1 = a * C1, o.a5 = a * C5;
  o.b0 = b * C0, o.b1 = b * C1, o.b5 = b * C5;
  o.d0 = d * C0, o.d1 = d * C1, o.d5 = d * C5;
  const double As = kShear * t * C5;
  o.s = w * As;
  o.r = w * kDrill * As;
  return o;
}

}  // namespace gf
