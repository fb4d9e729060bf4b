// swe_precompute.cu -- host-side validation and static geometry of one mesh.
//
// Everything the reference recomputes on each call from the nodes' plan
// positions alone (Domain::Norm / Tang / L / Area, src/Bathymetry.cpp:10-90) is
// evaluated here once, with the reference's operation order and without FMA
// contraction (-ffp-contract=off on the host compiler), so the device kernels
// see the same bits the CPU restatement computes on the fly.  What depends on
// the bathymetry too is computed on the device (swe_bed.cu).
#include <algorithm>
#include <cmath>
#include <string>
#include <thread>
#include <vector>

#include "swe_engine.cuh"

namespace swe {

void HostImage::resize(int C_, int E_, int N_, int I_) {
  C = C_; E = E_; N = N_; I = I_;
  cnode.assign(3 * (size_t)C, 0); cnbr.assign(3 * (size_t)C, -1); cedge.assign(3 * (size_t)C, 0);
  cinst.assign(C, 0); cown.assign(C, 0);
  area.assign(C, 0); cek.assign(3 * (size_t)C, 0);
  cnxc.assign(3 * (size_t)C, 0); cnyc.assign(3 * (size_t)C, 0);
  srec.assign(3 * (size_t)C, SlotRec{}); cslot.assign(3 * (size_t)C, int2{0, -1});
  erec.assign(E, EdgeRec{}); eidx.assign(E, int4{0, -1, 0, -1});
  eown.assign(E, 0); enb.assign(E, -1); eslotl.assign(E, 0); eslotr.assign(E, -1); einst.assign(E, 0);
  enx.assign(E, 0); eny.assign(E, 0); etx.assign(E, 0); ety.assign(E, 0); elmin.assign(E, 0);
  enode.assign(E, int2{0, 0}); nxy.assign(N, double2{0., 0.});
  nptr.assign((size_t)N + 1, 0); ncell.assign(3 * (size_t)C, 0);
  inst_cell_begin.assign(I, 0); inst_cfl.assign(I, 0); inst_cor.assign(I, 0);
}

namespace {

struct Geo {
  const HostInstance& h;
  const double* P(int64_t n) const { return h.geom.data() + 3 * n; }
  // src/Bathymetry.cpp:24-27
  void T(int64_t t, double out[3]) const {
    const int64_t* tp = h.cn.data() + 3 * t;
    const double k = 1. / 3.;
    for (int r = 0; r < 3; ++r) out[r] = P(tp[0])[r] * k + P(tp[1])[r] * k + P(tp[2])[r] * k;
  }
  // src/Bathymetry.cpp:82-85, src/PointOperations.cpp:4-6
  double L(int64_t e) const {
    const double* a = P(h.en[2 * e]);
    const double* b = P(h.en[2 * e + 1]);
    return sqrt((a[0] - b[0]) * (a[0] - b[0]) + (a[1] - b[1]) * (a[1] - b[1]));
  }
  // src/Bathymetry.cpp:87-90, src/PointOperations.cpp:8-14
  double Area(int64_t t) const {
    const int64_t* tp = h.cn.data() + 3 * t;
    const double *a = P(tp[0]), *b = P(tp[1]), *c = P(tp[2]);
    double ba0 = b[0] - a[0], ba1 = b[1] - a[1];
    double ca0 = c[0] - a[0], ca1 = c[1] - a[1];
    return 0.5 * fabs(ba0 * ca1 - ca0 * ba1);
  }
  // src/Bathymetry.cpp:69-76
  void Tang(int64_t e, int64_t t, double out[2]) const {
    const double* p0 = P(h.en[2 * e]);
    const double* p1 = P(h.en[2 * e + 1]);
    double l = L(e);
    double tan0 = (p1[0] - p0[0]) / l, tan1 = (p1[1] - p0[1]) / l;
    double tt[3];
    T(t, tt);
    double d0 = tt[0] - p0[0], d1 = tt[1] - p0[1];
    if (d0 * tan1 - tan0 * d1 > 0.) {
      tan0 = -tan0;
      tan1 = -tan1;
    }
    out[0] = tan0;
    out[1] = tan1;
  }
  // src/Bathymetry.cpp:78-80
  void Norm(int64_t e, int64_t t, double out[2]) const {
    double tg[2];
    Tang(e, t, tg);
    out[0] = tg[1];
    out[1] = -tg[0];
  }
};

}  // namespace

std::string validate_instance(const HostInstance& h) {
  const int64_t C = h.C, E = h.E, N = h.N;
  if (C <= 0 || E <= 0 || N <= 0) return "mesh must have cells, edges and nodes";
  if (C > (1ll << 29) || E > (1ll << 30) || N > (1ll << 30)) return "mesh too large for int32 device indexing";
  for (int64_t e = 0; e < E; ++e) {
    int64_t a = h.en[2 * e], b = h.en[2 * e + 1];
    if (a < 0 || a >= N || b < 0 || b >= N || a == b) return "edge_nodes[" + std::to_string(e) + "] out of range";
    int64_t o = h.ec[2 * e], n = h.ec[2 * e + 1];
    if (o < 0 || o >= C) return "edge_cells[" + std::to_string(e) + "][0] out of range";
    if (n >= C) return "edge_cells[" + std::to_string(e) + "][1] out of range";
    if (n < -1)
      return "edge_cells[" + std::to_string(e) + "][1] = " + std::to_string(n) +
             ": only the solid-wall code -1 is implemented (Boundaries::SOLID_WALL)";
    if (n == o) return "edge_cells[" + std::to_string(e) + "] joins a cell to itself";
  }
  for (int64_t i = 0; i < C; ++i) {
    for (int k = 0; k < 3; ++k) {
      int64_t nd = h.cn[3 * i + k];
      if (nd < 0 || nd >= N) return "cell_nodes[" + std::to_string(i) + "] out of range";
      int64_t e = h.ce[3 * i + k];
      if (e < 0 || e >= E) return "cell_edges[" + std::to_string(i) + "] out of range";
      int64_t o = h.ec[2 * e], n = h.ec[2 * e + 1];
      int64_t nb = h.ct[3 * i + k];
      if (o == i) {
        if (nb != n) return "cell_neighbours[" + std::to_string(i) + "] disagrees with edge_cells";
      } else if (n == i) {
        if (nb != o) return "cell_neighbours[" + std::to_string(i) + "] disagrees with edge_cells";
      } else {
        return "cell " + std::to_string(i) + " lists edge " + std::to_string(e) + " that does not touch it";
      }
    }
    if (h.ce[3 * i] == h.ce[3 * i + 1] || h.ce[3 * i] == h.ce[3 * i + 2] || h.ce[3 * i + 1] == h.ce[3 * i + 2])
      return "cell " + std::to_string(i) + " lists an edge twice";
  }
  for (size_t q = 0; q < h.geom.size(); ++q)
    if (!std::isfinite(h.geom[q])) return "non-finite geometry";
  Geo g{h};
  for (int64_t i = 0; i < C; ++i)
    if (!(g.Area(i) > 0.)) return "cell " + std::to_string(i) + " has zero area";
  return "";
}

void precompute_instance(const HostInstance& h, int inst, int64_t c0, int64_t e0, int64_t n0, HostImage& img) {
  const int64_t C = h.C, E = h.E, N = h.N, Ct = img.C;
  Geo g{h};
  img.inst_cell_begin[inst] = (int)c0;
  img.inst_cfl[inst] = h.cfl;
  img.inst_cor[inst] = h.cor;
  for (int64_t n = 0; n < N; ++n) img.nxy[n0 + n] = double2{h.geom[3 * n], h.geom[3 * n + 1]};
  // the cells around each node, a CSR over this instance's nodes whose
  // entries start at 3 c0 (each cell has three nodes): PartWet2 gathers its
  // lowest node's maximum over them (src/MUSCLObject.cpp:138-140)
  {
    std::vector<int64_t> at((size_t)N + 1, 0);
    for (int64_t i = 0; i < 3 * C; ++i) at[h.cn[i] + 1]++;
    for (int64_t n = 0; n < N; ++n) at[n + 1] += at[n];
    for (int64_t n = 0; n <= N; ++n) img.nptr[n0 + n] = (int)(3 * c0 + at[n]);
    for (int64_t i = 0; i < C; ++i)
      for (int k = 0; k < 3; ++k) img.ncell[3 * c0 + at[h.cn[3 * i + k]]++] = (int)(((c0 + i) << 2) | k);
  }

  auto cell_range = [&](int64_t lo, int64_t hi) {
    for (int64_t i = lo; i < hi; ++i) {
      const int64_t gi = c0 + i;
      const int64_t* ip = h.cn.data() + 3 * i;
      const int64_t* ie = h.ce.data() + 3 * i;
      const int64_t* it = h.ct.data() + 3 * i;
      img.cinst[gi] = inst;
      unsigned char own = 0;
      for (int k = 0; k < 3; ++k) {
        img.cnode[k * Ct + gi] = (int)(n0 + ip[k]);
        img.cnbr[k * Ct + gi] = it[k] < 0 ? -1 : (int)(c0 + it[k]);
        img.cedge[k * Ct + gi] = (int)(e0 + ie[k]);
        if (h.ec[2 * ie[k]] == i) own |= (unsigned char)(1u << k);
      }
      img.cown[gi] = own;
      const double area = g.Area(i);
      img.area[gi] = area;
      const double i_area = 1. / area;
      for (int k = 0; k < 3; ++k) {
        img.cek[k * Ct + gi] = i_area * g.L(ie[k]);  // src/TimeDisc.cpp:17,28
        double nrm[2];
        g.Norm(ie[k], i, nrm);  // src/TimeDisc.cpp:35
        // n c: the pressure term's geometry factor (src/TimeDisc.cpp:35 evaluates
        // n(e, i) * c first), kept whole so the update multiplies once
        img.cnxc[k * Ct + gi] = nrm[0] * img.cek[k * Ct + gi];
        img.cnyc[k * Ct + gi] = nrm[1] * img.cek[k * Ct + gi];
        img.srec[k * Ct + gi] = SlotRec{img.cek[k * Ct + gi], 0., img.cnxc[k * Ct + gi], img.cnyc[k * Ct + gi]};
        img.cslot[k * Ct + gi] = int2{img.cedge[k * Ct + gi], img.cnbr[k * Ct + gi]};
      }
    }
  };

  auto edge_range = [&](int64_t lo, int64_t hi) {
    for (int64_t e = lo; e < hi; ++e) {
      const int64_t ge = e0 + e;
      int64_t o = h.ec[2 * e], n = h.ec[2 * e + 1];
      img.einst[ge] = inst;
      img.eown[ge] = (int)(c0 + o);
      img.enb[ge] = n < 0 ? -1 : (int)(c0 + n);
      int ko = 0, kn = 0;
      for (int k = 0; k < 3; ++k) {
        if (h.ce[3 * o + k] == e) ko = k;
        if (n >= 0 && h.ce[3 * n + k] == e) kn = k;
      }
      img.eslotl[ge] = (int)(ko * Ct + c0 + o);
      img.eslotr[ge] = n < 0 ? -1 : (int)(kn * Ct + c0 + n);
      double nrm[2], tg[2];
      g.Norm(e, o, nrm);
      g.Tang(e, o, tg);
      img.enode[ge] = int2{(int)(n0 + h.en[2 * e]), (int)(n0 + h.en[2 * e + 1])};
      img.enx[ge] = nrm[0];
      img.eny[ge] = nrm[1];
      img.etx[ge] = tg[0];
      img.ety[ge] = tg[1];
      if (n >= 0) {
        double L = g.L(e);
        double dl = 2. * g.Area(o) / L;  // include/Fluxes.h:43-44, 86-87
        double dr = 2. * g.Area(n) / L;
        img.elmin[ge] = smin(dl, dr);
      } else {
        img.elmin[ge] = 0.;
      }
      img.erec[ge] = EdgeRec{img.enx[ge], img.eny[ge], img.etx[ge], img.ety[ge], 0., img.elmin[ge]};
      img.eidx[ge] = int4{img.eown[ge], img.enb[ge], img.eslotl[ge], img.eslotr[ge]};
    }
  };

  unsigned nt = std::max(1u, std::min(32u, std::thread::hardware_concurrency()));
  if (C + E < 20000) nt = 1;
  std::vector<std::thread> th;
  for (unsigned t = 0; t < nt; ++t) {
    int64_t clo = C * t / nt, chi = C * (t + 1) / nt;
    int64_t elo = E * t / nt, ehi = E * (t + 1) / nt;
    th.emplace_back([=, &cell_range, &edge_range] {
      cell_range(clo, chi);
      edge_range(elo, ehi);
    });
  }
  for (auto& x : th) x.join();
}

}  // namespace swe
