// Test-only host build of the device pair code (csrc/td_device.cuh compiled by a
// plain C++ compiler), so the kernels' arithmetic can be checked against the
// oracle on a machine without a GPU.  Not part of the library.
#include <cmath>
#include <cstdint>
#include "td_device.cuh"
using namespace cad;
extern "C" int host_td_inf(const double* X, const double* Y, const double* Z, int64_t M, const double* P1,
                           const double* P2, const double* P3, int64_t N, const double* Dss, const double* Dds,
                           const double* Dn, double nu, int disp, int strain, int hs, double* so, double* dout) {
  const int64_t MN = M * N;
  static TriDev t;  // ~13 KB; one record at a time
  for (int64_t j = 0; j < N; ++j) {
    double a[3] = {P1[j], P1[j + N], P1[j + 2 * N]}, b[3] = {P2[j], P2[j + N], P2[j + 2 * N]},
           c[3] = {P3[j], P3[j + N], P3[j + 2 * N]};
    build_triangle(a, b, c, Dss[j], Dds[j], Dn[j], nu, hs != 0, t);
    for (int64_t i = 0; i < M; ++i) {
      if (strain) {
        double E[3][6];
        if (hs) pair_strain<true>(t, X[i], Y[i], Z[i], E); else pair_strain<false>(t, X[i], Y[i], Z[i], E);
        for (int m = 0; m < 3; ++m) for (int k = 0; k < 6; ++k) so[(6 * m + k) * MN + i + M * j] = E[m][k];
      }
      if (disp) {
        double U[3][3];
        if (hs) pair_disp<true>(t, X[i], Y[i], Z[i], U); else pair_disp<false>(t, X[i], Y[i], Z[i], U);
        for (int m = 0; m < 3; ++m) for (int k = 0; k < 3; ++k) dout[(3 * m + k) * MN + i + M * j] = U[m][k];
      }
    }
  }
  return 0;
}

// The shared-edge half-space paths on the host, laid out as the kernels do.
// side_code: 3 per triangle, +-(edge + 1); edge_pts: 6 per edge (PA, PB).
// Influence fields: per-edge strain and displacement maps at every point,
// G[(e Q + q) M + i], read by pair_strain_full (full: the maps hold the whole
// strain) or pair_strain_edges (meshes with a horizontal triangle: the
// correction only), and by pair_disp_edges.
extern "C" int host_td_inf_edges(const double* X, const double* Y, const double* Z, int64_t M, const double* P1,
                                 const double* P2, const double* P3, int64_t N, const double* Dss, const double* Dds,
                                 const double* Dn, double nu, const int* side_code, const double* edge_pts, int64_t E,
                                 int full, double* so, double* dout) {
  const int64_t MN = M * N, Q = 27;
  double* G = new double[(size_t)(E * Q * M)];
  static FscSide s;
  for (int64_t e = 0; e < E; ++e) {
    build_side_geom(edge_pts + 6 * e, edge_pts + 6 * e + 3, nu, s);
    for (int64_t i = 0; i < M; ++i) {
      double Gm[3][6] = {}, Gu[3][3] = {};
      if (full) side_strain_map<true>(s, X[i], Y[i], Z[i], Gm);
      else if (s.skip == 0.0) side_strain_map<false>(s, X[i], Y[i], Z[i], Gm);
      if (s.skip == 0.0) fsc_disp_map(s, X[i], Y[i], Z[i], Gu);
      for (int q = 0; q < 18; ++q) G[(e * Q + q) * M + i] = Gm[q / 6][q % 6];
      for (int q = 0; q < 9; ++q) G[(e * Q + 18 + q) * M + i] = Gu[q / 3][q % 3];
    }
  }
  static TriDev t;
  for (int64_t j = 0; j < N; ++j) {
    double a[3] = {P1[j], P1[j + N], P1[j + 2 * N]}, b[3] = {P2[j], P2[j + N], P2[j + 2 * N]},
           c[3] = {P3[j], P3[j + N], P3[j + 2 * N]};
    build_triangle(a, b, c, Dss[j], Dds[j], Dn[j], nu, true, t);
    for (int64_t i = 0; i < M; ++i) {
      double Es[3][6], U[3][3];
      if (full) pair_strain_full(t, X[i], Y[i], Z[i], G + i, M, Q * M, side_code + 3 * j, Es);
      else pair_strain_edges(t, X[i], Y[i], Z[i], G + i, M, Q * M, side_code + 3 * j, Es);
      pair_disp_edges(t, X[i], Y[i], Z[i], G + 18 * M + i, M, Q * M, side_code + 3 * j, U);
      for (int m = 0; m < 3; ++m) for (int k = 0; k < 6; ++k) so[(6 * m + k) * MN + i + M * j] = Es[m][k];
      for (int m = 0; m < 3; ++m) for (int k = 0; k < 3; ++k) dout[(3 * m + k) * MN + i + M * j] = U[m][k];
    }
  }
  delete[] G;
  return 0;
}

// Tractions on the points' elements (dirs: normal, strike and dip of each, 9 x M)
// from per-edge maps of the whole strain: trac[(3 m + r) MN + i + M j].
extern "C" int host_td_trac_edges(const double* X, const double* Y, const double* Z, int64_t M, const double* P1,
                                  const double* P2, const double* P3, int64_t N, const double* Dss, const double* Dds,
                                  const double* Dn, double nu, double lam, double G2, const double* dirs,
                                  const int* side_code, const double* edge_pts, int64_t E, double* trac) {
  const int64_t MN = M * N;
  double* G = new double[(size_t)(E * 9 * M)];
  static FscSide s;
  for (int64_t e = 0; e < E; ++e) {
    build_side_geom(edge_pts + 6 * e, edge_pts + 6 * e + 3, nu, s);
    for (int64_t i = 0; i < M; ++i) {
      double d[3][3], W[3][3];
      for (int v = 0; v < 3; ++v) for (int c = 0; c < 3; ++c) d[v][c] = dirs[i + (3 * v + c) * M];
      side_traction_map(s, X[i], Y[i], Z[i], lam, G2, d[0], d[1], d[2], W);
      for (int q = 0; q < 9; ++q) G[(e * 9 + q) * M + i] = W[q / 3][q % 3];
    }
  }
  static TriDev t;
  for (int64_t j = 0; j < N; ++j) {
    double a[3] = {P1[j], P1[j + N], P1[j + 2 * N]}, b[3] = {P2[j], P2[j + N], P2[j + 2 * N]},
           c[3] = {P3[j], P3[j + N], P3[j + 2 * N]};
    build_triangle(a, b, c, Dss[j], Dds[j], Dn[j], nu, true, t, false);
    for (int64_t i = 0; i < M; ++i) {
      double S[9];
      sum_side_maps<9>(G + i, M, 9 * M, side_code + 3 * j, S);
      const bool nan = pair_on_side(t, X[i], Y[i], Z[i]);
      const double* axes[3] = {t.real.Vn, t.real.Vs, t.real.Vd};
      const double slip[3] = {t.Dn, t.Dss, t.Dds};
      for (int m = 0; m < 3; ++m)
        for (int r = 0; r < 3; ++r)
          trac[(3 * m + r) * MN + i + M * j] =
              nan ? qnan<double>()
                  : slip[m] * (axes[m][0] * S[r] + axes[m][1] * S[3 + r] + axes[m][2] * S[6 + r]);
    }
  }
  delete[] G;
  return 0;
}

// Net Burgers vector of the sides on edge e (tris[ptr[e] .. ptr[e + 1]) =
// +-(triangle + 1)), those without slip left out.
static void net_burgers(const TriDev* T, const int* ptr, const int* tris, int64_t e, double B[3]) {
  B[0] = B[1] = B[2] = 0.0;
  for (int k = ptr[e]; k < ptr[e + 1]; ++k) {
    const int cc = tris[k];
    const TriDev& t = T[(cc > 0 ? cc : -cc) - 1];
    const double sg = cc > 0 ? 1.0 : -1.0;
    const double slip[3] = {t.Dn, t.Dss, t.Dds};
    if (slip[0] == 0.0 && slip[1] == 0.0 && slip[2] == 0.0) continue;
    const double* axes[3] = {t.real.Vn, t.real.Vs, t.real.Vd};
    for (int m = 0; m < 3; ++m)
      for (int q = 0; q < 3; ++q) B[q] = add_rn(B[q], sg * mul_rn(axes[m][q], slip[m]));
  }
}

// Sums: each edge once for the net Burgers vector of the sides on it.  full
// (half space): all but the solid angles come from the edges (side_sum_full),
// and the triangles add those (pair_angle); otherwise the edges add the
// correction and the triangles their real + image terms.  hs = 0: the full
// space's segments (segment_sum) and solid angles.  so: 6 x M, dout: 3 x M.
extern "C" int host_td_sum_edges(const double* X, const double* Y, const double* Z, int64_t M, const double* P1,
                                 const double* P2, const double* P3, int64_t N, const double* Dss, const double* Dds,
                                 const double* Dn, double nu, const int* edge_ptr, const int* edge_tris,
                                 const double* edge_pts, int64_t E, int hs, int full, double* so, double* dout) {
  TriDev* T = new TriDev[(size_t)N];
  for (int64_t j = 0; j < N; ++j) {
    double a[3] = {P1[j], P1[j + N], P1[j + 2 * N]}, b[3] = {P2[j], P2[j + N], P2[j + 2 * N]},
           c[3] = {P3[j], P3[j + N], P3[j + 2 * N]};
    build_triangle(a, b, c, Dss[j], Dds[j], Dn[j], nu, hs != 0, T[j], !full);
  }
  FscSide* S = new FscSide[(size_t)E];
  SegRec* R = new SegRec[(size_t)E];
  for (int64_t e = 0; e < E; ++e) {
    double B[3];
    net_burgers(T, edge_ptr, edge_tris, e, B);
    if (hs) build_side_burgers(edge_pts + 6 * e, edge_pts + 6 * e + 3, B, nu, S[e]);
    else build_segment(edge_pts + 6 * e, edge_pts + 6 * e + 3, B, 0.5 * kInv4Pi / (1.0 - nu), R[e]);
  }
  for (int64_t i = 0; i < M; ++i) {
    double Es[6] = {}, Us[3] = {};
    if (full || !hs) {
      for (int64_t j = 0; j < N; ++j) {
        if (hs) pair_angle<true, true>(T[j], X[i], Y[i], Z[i], Es, Us);
        else pair_angle<false, true>(T[j], X[i], Y[i], Z[i], Es, Us);
      }
      for (int64_t e = 0; e < E; ++e) {
        if (!hs) { if (R[e].slips != 0.0) segment_sum<true, true>(R[e], X[i], Y[i], Z[i], Es, Us); }
        else if (S[e].skip != 2.0) side_sum_full<true>(S[e], X[i], Y[i], Z[i], Es, Us);
      }
      for (int k = 0; k < 6; ++k) so[k * M + i] = Es[k];
      for (int k = 0; k < 3; ++k) dout[k * M + i] = Us[k];
      continue;
    }
    for (int64_t j = 0; j < N; ++j) {
      double E6[3][6], U3[3][3];
      pair_strain_fs_image(T[j], X[i], Y[i], Z[i], E6);
      pair_disp_fs_image(T[j], X[i], Y[i], Z[i], U3);
      for (int k = 0; k < 6; ++k) Es[k] += (E6[0][k] + E6[1][k]) + E6[2][k];
      for (int k = 0; k < 3; ++k) Us[k] += (U3[0][k] + U3[1][k]) + U3[2][k];
    }
    double Ee[3][6] = {}, Ue[3][3] = {};
    for (int64_t e = 0; e < E; ++e)
      if (S[e].skip == 0.0) { fsc_strain(S[e], X[i], Y[i], Z[i], 0.0, 0.0, 1.0, Ee); fsc_disp(S[e], X[i], Y[i], Z[i], 0.0, 0.0, 1.0, Ue); }
    for (int k = 0; k < 6; ++k) so[k * M + i] = Es[k] + Ee[0][k];
    for (int k = 0; k < 3; ++k) dout[k * M + i] = Us[k] + Ue[0][k];
  }
  delete[] R;
  delete[] S;
  delete[] T;
  return 0;
}
