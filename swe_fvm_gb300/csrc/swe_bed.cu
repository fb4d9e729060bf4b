// swe_bed.cu -- the mesh records that depend on the node bathymetry, computed
// on the device.
//
// Everything MUSCLObject's reconstructions (src/MUSCLObject.cpp:31-191) and
// Domain's bathymetry (src/Bathymetry.cpp:10-90) need of the bed is evaluated
// here with the reference's operation order (no FMA contraction, the exact
// division of swe_fp64.cuh), so the records have the bits the CPU restatement
// computes on the fly.
//
// A context computes them at creation and again for every new bed (an
// inversion writes one per iteration).  On the host they were 1.3 KB a cell of
// single-core arithmetic and pageable upload: a new bed for 32,000 cells in six
// instances took 12 ms, now 0.35 ms with its upload.  The kernel is bound by the FP64
// pipe (some 60 operations per fully-wet plane, eight planes a cell); one thread
// per cell and plane, plus one for the cell's other records, keeps the chains
// short and small meshes spread over the SMs.
#include <cuda_runtime.h>

#include "swe_engine.cuh"

namespace swe {
namespace {

struct P3 {
  double v[3];
  __device__ double operator[](int r) const { return v[r]; }
};

__device__ __forceinline__ P3 node(const DevMesh& m, int id) {
  const int n = gidx(m, id, m.N);
  const double2 p = m.nxy[n];
  return P3{{p.x, p.y, m.nz[n]}};
}
// src/Bathymetry.cpp:24-27
__device__ __forceinline__ P3 centroid(const P3& a, const P3& b, const P3& c) {
  const double k = 1. / 3.;
  P3 t;
#pragma unroll
  for (int r = 0; r < 3; ++r) t.v[r] = a[r] * k + b[r] * k + c[r] * k;
  return t;
}
// edge centre = midpoint of the edge's nodes (Domain::E is a stub in the reference)
__device__ __forceinline__ P3 midpoint_of(const DevMesh& m, int e) {
  const int2 n = m.enode[gidx(m, e, m.E)];
  const P3 a = node(m, n.x), b = node(m, n.y);
  P3 t;
#pragma unroll
  for (int r = 0; r < 3; ++r) t.v[r] = (a[r] + b[r]) * 0.5;
  return t;
}

// Least double x for which the non-decreasing predicate holds (+inf: none), by
// galloping and halving over the ordered bit patterns from the guess x0.
template <class F>
__device__ double least(double x0, F holds) {
  const double inf = __longlong_as_double(0x7FF0000000000000ll);
  if (!(x0 == x0)) return inf;
  // k(x) monotone, consecutive doubles consecutive (both zeros at 0)
  auto at = [](long long k) { return __longlong_as_double(k < 0 ? (long long)(0x8000000000000000ull - (unsigned long long)k) : k); };
  const long long top = 0x7FF0000000000000ll;
  long long k = __double_as_longlong(x0);
  if (k < 0) k = -(k & 0x7FFFFFFFFFFFFFFFll);
  long long lo, hi, step = 1;  // fails at lo, holds at hi
  if (holds(at(k))) {
    hi = k;
    lo = k - step;
    while (lo > -top && holds(at(lo))) {
      hi = lo;
      step <<= 1;
      lo = (lo < -top + step) ? -top : lo - step;
    }
    if (lo <= -top) return at(hi);  // cannot happen: -inf is never wet
  } else {
    lo = k;
    hi = k + step;
    while (hi < top && !holds(at(hi))) {
      lo = hi;
      step <<= 1;
      hi = (hi > top - step) ? top : hi + step;
    }
    if (hi >= top) return inf;
  }
  while (hi - lo > 1) {
    const long long mid = lo + (hi - lo) / 2;
    if (holds(at(mid))) hi = mid;
    else lo = mid;
  }
  return at(hi);
}

// Fully-wet cell plane for one wet / part-wet neighbour combination
// (src/MUSCLObject.cpp:38-84); bit k of mask set = neighbour k partially wet.
__device__ void plane_record(const DevMesh& m, int i, int mask, double* rec, double* recv) {
  const int C = m.C;
  P3 P[3], E[3], Q[3];
  bool boundary = false;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    P[k] = node(m, m.cnode[k * C + i]);
    E[k] = midpoint_of(m, m.cedge[k * C + i]);
    if (m.cnbr[k * C + i] < 0) boundary = true;
  }
  if (boundary) {  // never fully wet
#pragma unroll
    for (int q = 0; q < kComboStride; ++q) rec[q] = 0.;
#pragma unroll
    for (int q = 0; q < kComboVStride; ++q) recv[q] = 0.;
    return;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int j = gidx(m, m.cnbr[k * C + i], C);
    if (mask >> k & 1) Q[k] = E[k];
    else Q[k] = centroid(node(m, m.cnode[j]), node(m, m.cnode[C + j]), node(m, m.cnode[2 * C + j]));
  }
  const P3 t = centroid(P[0], P[1], P[2]);
  double g0, g1;
  plane_gradient(Q[0][0], Q[0][1], Q[0][2], Q[1][0], Q[1][1], Q[1][2], Q[2][0], Q[2][1], Q[2][2], &g0, &g1);
  const double third = 1. / 3.;
  const double diag = 1. - third;
  rec[0] = g0;
  rec[1] = g1;
  double level = 0.;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double dx[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const double m0 = (k == 0) ? diag : -third;
      const double m1 = (k == 1) ? diag : -third;
      const double m2 = (k == 2) ? diag : -third;
      dx[r] = P[0][r] * m0 + P[1][r] * m1 + P[2][r] * m2;
    }
    // positivity of the vertex, is_wet((off + w) - z): its rounded sums are
    // non-decreasing in w, so it holds from one level on, kept in place of the
    // offset (the reconstruction then compares instead of adding six times)
    const double off = g0 * dx[0] + g1 * dx[1], z = P[k][2];
    const double from = least((z + kWetDepth) - off, [&](double w) { return is_wet((off + w) - z); });
    level = k == 0 ? from : smax(level, from);
    rec[3 + k] = g0 * (E[k][0] - t[0]) + g1 * (E[k][1] - t[1]);  // edge-centre offsets
    recv[k] = g0 * (P[k][0] - t[0]) + g1 * (P[k][1] - t[1]);     // vertex offsets
  }
  rec[2] = level;
}

// Scalars, dry plane, PartWet1 and PartWet2 records of cell i.
__device__ void cell_record(const DevMesh& m, const BedArrays& o, int i) {
  const int C = m.C;
  P3 P[3], E[3];
  bool boundary = false;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    P[k] = node(m, m.cnode[k * C + i]);
    E[k] = midpoint_of(m, m.cedge[k * C + i]);
    if (m.cnbr[k * C + i] < 0) boundary = true;  // src/TriangMesh.cpp:18-23
  }
  const P3 t = centroid(P[0], P[1], P[2]);
  const double bc = t[2];
  o.bc[i] = bc;
  const double wet = least(bc + kWetDepth, [&](double w) { return is_wet(w - bc); });
  // src/MUSCLObject.cpp:17-25 (maxCoeff of the node z)
  double mx = P[0][2];
  if (dlt(mx, P[1][2])) mx = P[1][2];
  if (dlt(mx, P[2][2])) mx = P[2][2];
  o.thr[i] = make_double2(wet, boundary ? __longlong_as_double(0x7FF0000000000000ll) : mx);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    o.zn[k * C + i] = P[k][2];
    o.ze[k * C + i] = E[k][2];
    o.srec[k * C + i].ze = E[k][2];
  }
  // dry cell: ReconstructDryCell + UpdateInterfaceValues (src/MUSCLObject.cpp:
  // 31-36, include/MUSCLObject.h:26-33, src/Assigners.cpp:8-20)
  double sx, sy;
  plane_gradient(P[0][0], P[0][1], P[0][2], P[1][0], P[1][1], P[1][2], P[2][0], P[2][1], P[2][2], &sx, &sy);
  double* dr = o.dry + (size_t)i * kDryStride;
  bool wet_slots = false;  // (a plane through the bed: only by rounding)
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double a = bc + (sx * (P[k][0] - t[0]) + sy * (P[k][1] - t[1]));
    dr[k] = dge0(a - P[k][2]) ? a : P[k][2];
    const double e = bc + (sx * (E[k][0] - t[0]) + sy * (E[k][1] - t[1]));
    const double at = dge0(e - E[k][2]) ? e : E[k][2];
    dr[3 + k] = is_wet(at - E[k][2]) ? at : E[k][2];
    wet_slots = wet_slots || is_wet(at - E[k][2]);
  }
  dr[6] = sx;
  dr[7] = sy;
  o.cown[i] = (unsigned char)((o.cown[i] & 7u) | (wet_slots ? 8u : 0u));
  // PartWet1 (src/MUSCLObject.cpp:86-112)
  {
    double b13 = P[0][2], b23 = P[0][2];
#pragma unroll
    for (int k = 1; k < 3; ++k) {
      if (dlt(b13, P[k][2])) b13 = P[k][2];
      if (dlt(P[k][2], b23)) b23 = P[k][2];
    }
    const double b12 = 3. * bc - b23 - b13;
    double* p = o.pw1 + (size_t)i * kPw1Stride;
    p[0] = b13;
    p[1] = b23;
    p[2] = b12;
    p[3] = b12 + SWE_DIV((1. / 3.) * (b13 - b12) * (b13 - b12), b13 - b23);  // b_delimiter
    p[4] = -3. * b13;                                                        // cubic b
    p[5] = 3. * (b12 * b13 + b13 * b23 - b12 * b23);                         // cubic c
    p[6] = b13 - b23;
    p[7] = b12 - b23;
    p[8] = b13 - b12;
    p[9] = b12 * (b12 + b23);
    p[10] = b23 * b23 * b13;
    p[11] = 0.;
  }
  // PartWet2 (src/MUSCLObject.cpp:114-191): vertices sorted by z
  {
    int s[3] = {0, 1, 2};
    auto z = [&](int k) { return k == 0 ? P[0][2] : k == 1 ? P[1][2] : P[2][2]; };
    auto order = [&](int& a, int& b) {
      if (dlt(z(b), z(a))) {
        const int q = a;
        a = b;
        b = q;
      }
    };
    order(s[0], s[1]);
    order(s[1], s[2]);
    order(s[0], s[1]);
    Pw2Rec& q = o.pw2[i];
    double lowest[2] = {0., 0.}, zs[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const P3 v = s[k] == 0 ? P[0] : s[k] == 1 ? P[1] : P[2];
      if (k == 0) {
        lowest[0] = v[0];
        lowest[1] = v[1];
      }
#pragma unroll
      for (int r = 0; r < 3; ++r) q.p[k][r] = v[r];
      zs[k] = v[2];
      q.sk[k] = s[k];
    }
    const double b23 = zs[0], b12 = zs[1], b13 = zs[2], d13 = b13 - b23;
    q.flat = dltc(d13, kTol) ? 1 : 0;
    q.ratio_b = SWE_DIV(b12 - b23, d13);
    q.hd2f = 2. * b13 - b12 - b23;
    q.d13 = d13;
    q.beta = SWE_DIV(b13 - b12, d13);
    q.tp0x = t[0] - lowest[0];
    q.tp0y = t[1] - lowest[1];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      q.dnode[k][0] = P[k][0] - t[0];
      q.dnode[k][1] = P[k][1] - t[1];
      q.dedge[k][0] = E[k][0] - t[0];
      q.dedge[k][1] = E[k][1] - t[1];
    }
    q.lo = m.cnode[s[0] * C + i];
    q.pad = 0;
  }
}

__global__ void __launch_bounds__(128) k_bed_cells(DevMesh m, BedArrays o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m.C) return;
  const int part = blockIdx.y;
  if (part < 8) plane_record(m, i, part, o.combo + combo_off(m.C, i, part), o.combov + combov_off(m.C, i, part));
  else cell_record(m, o, i);
}

__global__ void __launch_bounds__(256) k_bed_edges(DevMesh m, BedArrays o) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m.E) return;
  const int2 n = m.enode[e];
  const double z = (m.nz[gidx(m, n.x, m.N)] + m.nz[gidx(m, n.y, m.N)]) * 0.5;
  o.ezm[e] = z;
  o.erec[e].b = z;
}

}  // namespace

cudaError_t Engine::compute_bed(const double* nz_host) {
  const cudaError_t pending = cudaPeekAtLastError();
  cudaError_t e = cudaMemcpyAsync(bed_.nz, nz_host, mesh_.N * sizeof(double), cudaMemcpyHostToDevice, stream_);
  if (e != cudaSuccess) return e;
  k_bed_cells<<<dim3((mesh_.C + 127) / 128, 9), 128, 0, stream_>>>(mesh_, bed_);
  k_bed_edges<<<(mesh_.E + 255) / 256, 256, 0, stream_>>>(mesh_, bed_);
  launches_ += 2;
  return launch_error(pending);
}

}  // namespace swe
