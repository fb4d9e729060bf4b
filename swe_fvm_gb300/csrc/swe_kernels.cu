// swe_kernels.cu -- sm_103a kernels of one Runge-Kutta stage and the engine
// that sequences them.
//
// A stage (src/Solvers.cpp:5-59) is seven kernels over the concatenated cells
// and edges of every instance:
//   k_recon1  all cells    SpaceDisc::ComputeInterfaceValues pass 1
//                          (src/SpaceDisc.cpp:37-45), listing the partially
//                          wet cells (in a step the update before lists them)
//   k_partwet1 part-wet    their pass-1 level, on a second stream beside it
//   k_recon2  part-wet     pass 2 (src/SpaceDisc.cpp:47-51), gathering the
//                          node maximum it reads from the pass-1 values of
//                          the node's cells (order-independent)
//   k_flux    all edges    SpaceDisc::ComputeFluxes (src/SpaceDisc.cpp:54-74)
//                          with the flux plugin and the CFL min-reduction,
//                          except the edges of partially-wet cells
//   k_flux_pw those edges  on a second stream, after k_recon2
//   k_drain   all cells    TimeDisc::ComputeDrainingDt (src/TimeDisc.cpp:43-66),
//                          once per cell instead of 4x per RHS
//   k_update  all cells    TimeDisc::RHS + ConsAssigner (src/TimeDisc.cpp:3-41,
//                          src/Assigners.cpp:28-44), an edge-to-cell gather
// Every read of a stage comes from the start-of-stage state, so results do not
// depend on the cell order or on scheduling; the only atomics (CFL minimum,
// part-wet list append) are exact min/append operations.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cstdio>
#include <cstring>
#include <limits>
#include <map>
#include <mutex>
#include <string>
#include <type_traits>

#include "swe_engine.cuh"

namespace swe {

Scheme scheme_table(int scheme) {
  Scheme s{};
  s.s[0] = Stage{true, 0., 0., 1.};
  if (scheme == 0) {
    s.n = 1;
  } else if (scheme == 1) {
    s.n = 2;
    s.s[1] = Stage{false, 0.5, 0.5, 0.5};
  } else {
    s.n = 3;
    s.s[1] = Stage{false, 0.75, 0.25, 0.25};
    s.s[2] = Stage{false, 1. / 3., 2. / 3., 2. / 3.};
  }
  return s;
}

namespace {

constexpr double kInf = __builtin_huge_val();

// Meshes and batches from this many cells up (two warps per scheduler) form the
// products of the flux and update kernels on the integer pipe (Products).
// GB300's FP64 pipe holds a warp instruction for 64 cycles; an integer product
// takes about 26 issue slots of other pipes, so with both at work the kernels
// issue FP64 for the additions only: 1M-cell dam break, k_flux 180 -> 141 us,
// k_update 147 -> 99 us, step 773 -> 617 us; 250k-cell coast 339 -> 292 us.  With
// fewer warps the integer product is the longer chain (148 against 74 cycles):
// 44,402 cells 139 -> 137 us, 25,088 134.7 -> 135.4 us, 12,482 132 -> 135 us a step.
constexpr int64_t kSoftCells = 40000;

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// start moving the cache line of p towards this SM's L1 (no register, no wait)
__device__ __forceinline__ void prefetch_l1(const void* p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// two 16-byte loads of a 32-byte record through the read-only path
__device__ __forceinline__ void ldg_pair(const void* p, double2* a, double2* b) {
  const double2* q = (const double2*)p;
  *a = __ldg(q);
  *b = __ldg(q + 1);
}

// ------------------------------------------------------------ interface write
// UpdateInterfaceValues for one edge slot (src/SpaceDisc.cpp:24-29): AtPoint
// value (w, u, v) already dry-checked, through PrimAssigner with the edge
// bathymetry, plus the source gradient and Coriolis term.
// Source gradient plus the Coriolis term, (gx, gy) + cor (-v, u).  COR0 (cor
// is +-0 for every instance): x + (+-0) is x unless x is itself a zero, and
// then -0 only if both are -0, so the same bits come from integer operations.
// (A non-finite velocity would give NaN through the arithmetic; its state is
// already non-finite and reported by the update kernel.)
__device__ __forceinline__ double add_zero_product(double x, double c, double v) {
  const unsigned long long ux = (unsigned long long)dbits(x);
  if ((ux << 1) != 0ull) return x;
  const unsigned long long uc = (unsigned long long)dbits(c);
  const unsigned long long uv = (unsigned long long)dbits(v);
  return dfrom((long long)(ux & (uc ^ uv) & 0x8000000000000000ull));
}

// How a reconstruction writes a slot.  What the step's own kernels read is the
// depth (kLean): h = w - b where wet, else 0.  The slot's velocity is the
// cell's, zeroed or desingularised by that depth (slot_velocity), and the
// source gradient is one per cell.  The full form (kSlots, with or without
// Coriolis) adds the reference's interface values and source slots, for the
// getters and the adjoint: 120 B a cell more, which is why the step leaves them.
enum : int { kLean = 0, kSlotsCor0 = 1, kSlotsCor = 2 };

template <int FORM>
__device__ __forceinline__ void write_slot(const DevWork& wk, int slot, double h, double be, double w, double u, double v,
                                           double gx, double gy, double cor) {
  wk.eh[slot] = is_wet(h) ? h : 0.;  // h = w - be
  if (FORM == kLean) return;
  double ow, ou, ov;
  prim_assign(be, w, u, v, &ow, &ou, &ov);
  wk.ew[slot] = ow;
  wk.eu[slot] = ou;
  wk.ev[slot] = ov;
  double sx = gx, sy = gy;
  if (FORM == kSlotsCor0) {
    const double nov = dfrom(dbits(ov) ^ (long long)0x8000000000000000ull);
    sx = add_zero_product(gx, cor, nov);
    sy = add_zero_product(gy, cor, ou);
  } else {
    sx += cor * (-ov);
    sy += cor * ou;
  }
  wk.sx[slot] = sx;
  wk.sy[slot] = sy;
}

// The velocity at a slot of depth h (eh) in a cell with velocity (u, v), as
// UpdateInterfaceValues assigns it (src/Assigners.cpp:8-20): zero where the
// slot or the whole cell is dry, desingularised where it is thin.
__device__ __forceinline__ void slot_velocity(double h, bool dry_cell, double* u, double* v) {
  if (dry_cell || !is_wet(h)) {
    *u = 0.;
    *v = 0.;
  } else if (dltc(h, kEta1)) {
    const double s = SWE_DIV(kSqrt2 * h, SWE_SQRT(h * h + kEta2));
    *u *= s;
    *v *= s;
  }
}

// 0 - x: -x, but +0 for either zero
__device__ __forceinline__ double zero_minus(double x) {
  const unsigned long long u = ubits(x);
  return ufrom((u << 1) == 0ull ? 0ull : u ^ 0x8000000000000000ull);
}

// 0 x: a zero of x's sign (NaN where x is not finite)
__device__ __forceinline__ double zero_times(double x) {
  const unsigned long long u = ubits(x);
  return ufrom((~u & 0x7FF0000000000000ull) == 0ull ? 0x7FF8000000000000ull : u & 0x8000000000000000ull);
}

// MUSCL::AtPoint with a w-only plane (include/MUSCLObject.h:26-33): the value
// at a point whose offset term is `off` and whose bathymetry is z.
__device__ __forceinline__ bool at_point_wet(double w0, double off, double z, double* wout) {
  double a = w0 + off;
  if (dge0(a - z)) {
    *wout = a;
    return true;
  }
  *wout = z;
  return false;
}

// Pass-1 AtPoint value of cell c at its local node kn, from what pass 1 left:
// the class byte (dry / partially wet / fully wet, combination mask, plane
// kept), the PartWet1 level of a partially-wet cell and the state.  (a - z >= 0
// is a >= z: the sign of a difference is exact.)
__device__ __forceinline__ double pass1_value(const DevMesh& m, const DevWork& wk, const double* __restrict__ W,
                                              int c, int kn) {
  const int C = m.C;
  const unsigned cl = wk.cls[c];
  const unsigned type = cl & 3u;
  const double z = m.zn[kn * C + c];
  // level (the PartWet1 level is a flat plane's), and the kept plane's offset
  const double* from = type == 0u ? m.dry + (size_t)c * kDryStride + kn : type == 1u ? wk.pwrec + c : W + c;
  double val = *from;
  if (type == 2u && (cl & 32u)) val = val + m.combov[combov_off(C, c, (int)((cl >> 2) & 7u)) + kn];
  return type == 0u || dle(z, val) ? val : z;
}

// The node maximum m_max_wp of node nd (src/MUSCLObject.cpp:13-36): the
// largest pass-1 AtPoint value of the cells around it, starting from the
// node's bathymetry (every AtPoint value is >= it).  A maximum is exact and
// order-free, so gathering it where it is needed gives the value the
// reference's accumulation over its cell loop gives.  LANES = 8: the whole warp
// calls, and each group of 8 lanes shares its node's cells.
template <int LANES>
__device__ __forceinline__ unsigned long long node_max_key(const DevMesh& m, const DevWork& wk,
                                                           const double* __restrict__ W, int nd) {
  unsigned long long key = order_key(m.nz[nd]);
  const int q0 = m.nptr[nd], q1 = m.nptr[nd + 1];
  if (LANES > 1) {
    for (int q = q0 + (int)(threadIdx.x & (LANES - 1)); q < q1; q += LANES) {
      const int c = m.ncell[gidx(wk, q, 3 * m.C)];
      const unsigned long long k = order_key(pass1_value(m, wk, W, gidx(wk, c >> 2, m.C), c & 3));
      key = k > key ? k : key;
    }
    __syncwarp();
#pragma unroll
    for (int off = LANES / 2; off; off >>= 1) {
      const unsigned long long o = __shfl_xor_sync(0xFFFFFFFFu, key, off, LANES);
      key = o > key ? o : key;
    }
    return key;
  }
  // the first 8 cells (a triangulation node has about 6) with their loads
  // issued together, the rest one by one
  constexpr int kV = 8;
  int cq[kV];
#pragma unroll
  for (int j = 0; j < kV; ++j) cq[j] = q0 + j < q1 ? m.ncell[gidx(wk, q0 + j, 3 * m.C)] : -1;
#pragma unroll
  for (int j = 0; j < kV; ++j) {
    if (cq[j] >= 0) {
      const unsigned long long k = order_key(pass1_value(m, wk, W, gidx(wk, cq[j] >> 2, m.C), cq[j] & 3));
      key = k > key ? k : key;
    }
  }
  for (int q = q0 + kV; q < q1; ++q) {
    const int c = m.ncell[gidx(wk, q, 3 * m.C)];
    const unsigned long long k = order_key(pass1_value(m, wk, W, gidx(wk, c >> 2, m.C), c & 3));
    key = k > key ? k : key;
  }
  return key;
}

// PartWet1 level (src/MUSCLObject.cpp:86-112).  LANES = 8: the whole warp calls,
// a cell to each group of 8 lanes.
template <int LANES>
__device__ __forceinline__ double partwet1_level(const double* __restrict__ p, double w, double h) {
  const double b13 = p[0], b23 = p[1], bdel = p[3];
  const bool above_all = dle(b13, w), cube = !above_all && dle(w, bdel), bisect = !above_all && !cube;
  double level = w;
  if (cube) level = b23 + cbrt_rn(3. * h * p[6] * p[7]);
  if (LANES > 1 ? __any_sync(0xFFFFFFFFu, bisect) : bisect) {
    const double cc = p[6] * (3. * h * p[8] - p[9]) - p[10];
    const double root = LANES > 1 ? bisection_group<false>(cc, p[5], p[4], p[2], b13, bisect)
                                  : bisection(cc, p[5], p[4], p[2], b13);
    if (bisect) level = root;
  }
  return level;
}

// Appends the lanes' partially-wet cells to the list, one atomic a warp (every
// lane of the warp calls).
__device__ __forceinline__ void append_listed(const DevWork& wk, int C, bool part, int i) {
  const unsigned bal = __ballot_sync(0xffffffffu, part);
  if (bal) {
    const int leader = __ffs(bal) - 1;
    int base = 0;
    if (lane_id() == leader) base = atomicAdd(wk.pwcount, __popc(bal));
    base = __shfl_sync(0xffffffffu, base, leader);
    const int slot = base + __popc(bal & ((1u << lane_id()) - 1u));
    if (part && slot < C) wk.pwlist[slot] = i;
  }
}

// A partially-wet cell whose level stands above its highest vertex (in practice
// every wet cell along a wall) keeps that level, flat, in both passes
// (src/MUSCLObject.cpp:96-97, 124): pass 1 finishes it, marks its class byte, and
// only the others are listed.  Walls have most of the partially-wet cells of most
// meshes (the 25,000-cell coast lists 601 of 1033, an all-wet basin none of its
// rim: 20k-cell inversion iteration 12.1 -> 11.6 ms).  From kSoftCells cells on
// they are listed all the same: there their edges, walls among them, cost k_flux
// more than k_flux_pw, which runs beside it (32 basins of 218,000 cells 250 -> 257
// us a step, 1M-cell dam break 608 -> 615).
constexpr unsigned kFinished = 64u;
__device__ __forceinline__ bool listed_class(unsigned cls) { return (cls & (3u | kFinished)) == 1u; }
__device__ __forceinline__ bool above_all(const DevMesh& m, int i, double w) {
  return dlt(m.pw1[(size_t)i * kPw1Stride], w);
}

// Whether cell i with level w is partially wet (neither dry nor fully wet,
// src/MUSCLObject.cpp:13-29) and to be listed; finish: but for those cells.
__device__ __forceinline__ bool to_list(const DevMesh& m, int i, double w, bool finish) {
  const double2 t = __ldg(m.thr + i);
  return !dlt(w, t.x) && !dlt(t.y, w) && !(finish && above_all(m, i, w));
}

// The partially-wet cells of a state that no update left (a new state or bed).
__global__ void __launch_bounds__(256) k_list_partwet(DevMesh m, DevWork wk, const double* __restrict__ W,
                                                      bool finish) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  append_listed(wk, m.C, i < m.C && to_list(m, i, W[i], finish), i);
}

// ---------------------------------------------------------------- kernels
// Pass 1 but for the partly wet cells' levels (k_partwet1, beside it).  Bound by
// its gathers.  append: list the partially-wet cells that are left to it (a step's
// are listed by the update before it).  finish: see kFinished.
// The wet test and the plane's positivity are comparisons with levels kept in
// the mesh (DevMesh::thr, record entry 2) where the rounded sums would cost
// seven FP64 operations; 6 are left in a fully-wet cell of 18.
template <bool BATCH, int FORM>
__global__ void __launch_bounds__(256, 5) k_recon1(DevMesh m, DevWork wk, const double* __restrict__ W,
                                                const double* __restrict__ U, const double* __restrict__ V,
                                                int latch_mode, bool append, bool finish) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool part = false;
  unsigned char cls = 0;  // dry unless set below
  if (i < m.C) {
    const int inst = BATCH ? m.cinst[i] : 0;
    if (latch_mode != 3 && i == (BATCH ? m.inst_cell_begin[inst] : 0)) {
      if (latch_mode == 1) {  // dt = TimeDisc::CFLdt() of the previous flux pass
        double dt = m.inst_cfl[inst] * order_val(wk.r[inst]);
        wk.dt[inst] = dt;
        wk.tsum[inst] += dt;
      } else if (latch_mode == 2) {
        double dt = wk.fixed_dt[BATCH ? inst : 0];
        wk.dt[inst] = dt;
        wk.tsum[inst] += dt;
      }
      wk.r[inst] = order_key(1.0);  // src/SpaceDisc.cpp:56
    }
    const int C = m.C;
    // the combination record of the all-fully-wet neighbourhood (mask 0) is
    // the one nearly every fully-wet cell reads: start its line towards L1
    // now, before the loads that decide the class and the mask
    prefetch_l1(m.combo + combo_off(C, i, 0));
    const double cor = FORM == kSlotsCor ? m.inst_cor[inst] : FORM == kSlotsCor0 ? m.inst_cor[inst] : 0.;
    const double w = W[i];
    const double u = FORM == kLean ? 0. : U[i], v = FORM == kLean ? 0. : V[i];
    double gx = 0., gy = 0.;
    const double2 level = __ldg(m.thr + i);
    if (dlt(w, level.x)) {
      // ReconstructDryCell: every value is a mesh constant
      const double* dr = m.dry + (size_t)i * kDryStride;
      gx = dr[6];
      gy = dr[7];
      const bool wet_slots = (m.cown[i] & 8u) != 0u;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int slot = k * C + i;
        // (a dry cell's own slots are dry but for rounding, which the mesh record tells)
        const double be = FORM != kLean || wet_slots ? m.ze[slot] : 0.;
        const double h = wet_slots ? dr[3 + k] - be : 0.;
        write_slot<FORM>(wk, slot, h, be, FORM == kLean ? 0. : dr[3 + k], 0., 0., gx, gy, cor);
      }
    } else if (!dlt(level.y, w) && !(finish && above_all(m, i, w))) {
      // partially wet: listed for k_partwet1 and k_recon2
      part = true;
      cls = 1;
    } else {
      // ReconstructFullWetCell (src/MUSCLObject.cpp:38-84); or flat, a
      // partially-wet cell that is finished here
      const bool flat = !dlt(level.y, w);
      int mask = 0;
      bool first_order = flat;
      double wn[3] = {w, w, w};
#pragma unroll
      for (int k = 0; k < 3 && !flat; ++k) {
        const int nb = gidx(wk, m.cnbr[k * C + i], C);  // never a wall: fully-wet cells are interior
        const double wj = W[nb];
        wn[k] = wj;
        const double2 tj = __ldg(m.thr + nb);
        if (dlt(tj.y, wj)) {
          // fully-wet neighbour: plane point at its centroid
        } else if (dlt(wj, tj.x)) {
          first_order = true;
        } else {
          mask |= 1 << k;  // partially-wet neighbour: plane point at the edge centre
        }
      }
      cls = (unsigned char)(flat ? 1u | kFinished : 2u | ((unsigned)mask << 2));
      if (flat) wk.pwrec[i] = w;
      double at[3] = {w, w, w};  // the plane's level at the edge centres
      if (!first_order) {
        const double2* rec = (const double2*)(m.combo + combo_off(C, i, mask));
        const double2 g = __ldg(rec), p = __ldg(rec + 1), q = __ldg(rec + 2);
        if (dle(p.x, w)) {  // positive at the three vertices
          // binary TVD limiter on the w row (rows u, v of df are zero)
          const double vek[3] = {w + p.y, w + q.x, w + q.y};
          bool tvd = true;
#pragma unroll
          for (int k = 0; k < 3; ++k)
            if (!(dle(smin(w, wn[k]), vek[k]) && dle(vek[k], smax(w, wn[k])))) tvd = false;
          if (tvd) {
            cls |= 32;  // combination plane kept
            gx = g.x;
            gy = g.y;
#pragma unroll
            for (int k = 0; k < 3; ++k) at[k] = vek[k];
          } else {
            gx = zero_times(g.x);  // diag(TVD) * df keeps the sign of zero
            gy = zero_times(g.y);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int slot = k * C + i;
        // AtPoint below the bed gives (b, 0, 0), and so does a slot that is not
        // wet: one rule for both
        const double be = m.ze[slot], h = at[k] - be;
        const bool above = dge0(h);
        write_slot<FORM>(wk, slot, h, be, above ? at[k] : be, above ? u : 0., above ? v : 0., gx, gy, cor);
      }
    }
    if (!part) {
      wk.gx[i] = gx;
      wk.gy[i] = gy;
    }
    wk.cls[i] = cls;
  }
  if (append) append_listed(wk, m.C, part, i);
}

// Every node maximum (the reference's m_max_wp after pass 1), for the
// interface-value entry points that return them; the step itself gathers
// only the nodes PartWet2 reads (k_recon2).
__global__ void k_node_max_all(DevMesh m, DevWork wk, const double* __restrict__ W) {
  const int nd = blockIdx.x * blockDim.x + threadIdx.x;
  if (nd < m.N) wk.maxwp[nd] = node_max_key<1>(m, wk, W, nd);
}

// The partly wet cells' work is one long chain a cell (PartWet1's cube root or
// bisection, then the node maximum's gather, PartWet2's roots or bisection and a
// plane solve), and few cells have it: the kernels last as long as the chain.
// With up to kGroupCells listed, 8 lanes share a cell: they gather the node's
// cells together, take three steps of a bisection for one evaluation and a slot
// each.  Longer lists fill the SMs with one lane a cell (8 lanes issue about
// half of each cell's instructions each).  SSPRK2 step with 8 lanes, with one:
// 8192-cell Thacker bowl (200 listed) 120, 126 us; 25k-cell coast (2900) 134,
// 140 us; 250k-cell coast (14000) 306, 286 us.
constexpr int kGroupCells = 8000;

// Calls work.template operator()<LANES>(cell, own) for the listed cells: with 8
// lanes a cell the warp goes through its four cells together (a group past the
// end repeats the last cell and owns nothing).
template <class F>
__device__ __forceinline__ void for_listed(const DevMesh& m, const DevWork& wk, F&& work) {
  const int n = min(*wk.pwcount, m.C);
  const int t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  if (n <= kGroupCells) {
    for (int q0 = (t >> 5) * 4; q0 < n; q0 += (nt >> 5) * 4) {
      const int q = q0 + ((t >> 3) & 3);
      work(std::integral_constant<int, 8>{}, gidx(wk, wk.pwlist[min(q, n - 1)], m.C), q < n);
    }
  } else {
    for (int q = t; q < n; q += nt) work(std::integral_constant<int, 1>{}, gidx(wk, wk.pwlist[q], m.C), true);
  }
}

// PartWet1 level of the listed cells.
__global__ void __launch_bounds__(128) k_partwet1(DevMesh m, DevWork wk, const double* __restrict__ W) {
  for_listed(m, wk, [&](auto lanes, int i, bool own) {
    constexpr int L = decltype(lanes)::value;
    const double w = W[i];
    const double level = partwet1_level<L>(m.pw1 + (size_t)i * kPw1Stride, w, w - m.bc[i]);
    if (own && (threadIdx.x & (L - 1)) == 0) wk.pwrec[i] = level;
  });
}

// ReconstructPartWetCell2 (src/MUSCLObject.cpp:114-191) of cell i by LANES lanes
// (the whole warp calls where that is 8).
template <bool BATCH, int FORM, int LANES>
__device__ __forceinline__ void partwet2_cell(const DevMesh& m, const DevWork& wk, const double* __restrict__ W,
                                              const double* __restrict__ U, const double* __restrict__ V, int i,
                                              bool own) {
  const int C = m.C;
  const int lane = (int)(threadIdx.x & (LANES - 1));
  auto any = [](bool p) { return LANES > 1 ? __any_sync(0xFFFFFFFFu, p) != 0 : p; };
  const int inst = BATCH ? m.cinst[i] : 0;
  const double cor = FORM == kLean ? 0. : m.inst_cor[inst];
  const double w = W[i];
  const double u = FORM == kLean ? 0. : U[i], v = FORM == kLean ? 0. : V[i];
  const Pw2Rec& r = m.pw2[i];
  const double b23 = r.p[0][2], b12 = r.p[1][2], b13 = r.p[2][2];
  double w0 = wk.pwrec[i];  // PartWet1 fallback level
  double gx = 0., gy = 0.;
  bool plane = !(dlt(b13, w) || r.flat);
  if (any(plane)) {
    // the node maximum of the lowest node, gathered from its cells' pass-1
    // values; kept in maxwp for the adjoint's reverse of this cell
    const int lo = gidx(wk, r.lo, m.N);
    const unsigned long long key = node_max_key<LANES>(m, wk, W, lo);
    if (own && plane && lane == 0) wk.maxwp[lo] = key;
    const double w23 = order_val(key);
    const double h23 = w23 - b23;
    const double ratio_b = r.ratio_b;
    const double h_delim1 = 1. / 3. * h23 * ratio_b;
    const double h_delim2 = SWE_DIV(1. / 3. * h23 * r.hd2f, r.d13);
    const double hi = w - m.bc[i];
    const double ratio_h = SWE_DIV(hi, h23);
    // columns of the reference's `points` after all its writes: point 0 is
    // the lowest vertex with its bathymetry (see the restatement's notes)
    double p1x = r.p[1][0], p1y = r.p[1][1], p1z = b12;
    double p2x = r.p[2][0], p2y = r.p[2][1], p2z = b13;
    const bool one = plane && dle(hi, h_delim1), three = plane && !one && dle(h_delim2, hi);
    const bool two = plane && !one && !three;  // vertices wet
    if (one) {
      const double k2 = SWE_SQRT(SWE_DIV(3. * ratio_h, ratio_b));
      const double k3 = SWE_SQRT(3. * ratio_h * ratio_b);
      const double j2 = 1. - k2, j3 = 1. - k3;
      p1x = k2 * p1x + j2 * r.p[0][0];
      p1y = k2 * p1y + j2 * r.p[0][1];
      p1z = k2 * p1z + j2 * r.p[0][2];
      p2x = k3 * p2x + j3 * r.p[0][0];
      p2y = k3 * p2y + j3 * r.p[0][1];
      p2z = k3 * p2z + j3 * r.p[0][2];
    }
    if (three) p2z += 1.5 * (hi - h_delim2);
    if (any(two)) {
      const double alpha = 3. * ratio_h;
      const double beta = r.beta;
      const double cd = SWE_DIV(1. + beta - alpha, beta * beta), cc = SWE_DIV(alpha - 3., beta);
      const double k1 = 1. - (LANES > 1 ? bisection_group<true>(cd, cc, 0., 0., 1., two) : bisection01(cd, cc));
      if (two) {
        const double j1 = 1. - k1;
        p2x = k1 * p2x + j1 * r.p[1][0];
        p2y = k1 * p2y + j1 * r.p[1][1];
        p2z = k1 * b13 + j1 * b12;
        if (dltc(k1, kTol)) plane = false;
      }
    }
    if (plane) {
      plane_gradient(r.p[0][0], r.p[0][1], r.p[0][2], p1x, p1y, p1z, p2x, p2y, p2z, &gx, &gy);
      w0 = w23 + (gx * r.tp0x + gy * r.tp0y);
    }
  }
#pragma unroll
  for (int k0 = 0; k0 < (LANES > 1 ? 1 : 3); ++k0) {
    const int k = LANES > 1 ? lane : k0;
    if (own && k < 3) {
      const int slot = k * C + i;
      const double be = m.ze[slot];
      const double off = plane ? (gx * r.dedge[k][0] + gy * r.dedge[k][1]) : 0.;
      const double at = w0 + off, h = at - be;
      const bool over = dge0(h);
      write_slot<FORM>(wk, slot, h, be, over ? at : be, over ? u : 0., over ? v : 0., gx, gy, cor);
    }
  }
  if (own && lane == 0) {
    wk.gx[i] = gx;
    wk.gy[i] = gy;
  }
}

template <bool BATCH, int FORM>
__global__ void __launch_bounds__(128) k_recon2(DevMesh m, DevWork wk, const double* __restrict__ W,
                                                const double* __restrict__ U, const double* __restrict__ V) {
  for_listed(m, wk, [&](auto lanes, int i, bool own) {
    partwet2_cell<BATCH, FORM, decltype(lanes)::value>(m, wk, W, U, V, i, own);
  });
}

// SpaceDisc::ComputeFluxes with flux plugin FLUX and the CFL min-reduction.
// The flux of edge e (src/SpaceDisc.cpp:54-74) into f0..f2; *lw receives its
// length-to-wavespeed ratio or stays +inf.  SLOTS: from the full interface
// values (swe_compute_fluxes), else from the depths and the cells' velocities.
// Returns false where a product left the integer routine's range (nothing of
// use is stored then; the caller evaluates the edge again with SOFT = false).
template <class FLUX, bool TAPE, bool SOFT, bool SLOTS>
__device__ __forceinline__ bool flux_edge(const DevMesh& m, const DevWork& wk, const double* __restrict__ W,
                                          const double* __restrict__ U, const double* __restrict__ V, int e, int inst,
                                          double* lw) {
  Products<SOFT> prod;
  const int4 ix = __ldg(m.eidx + e);  // (owner, neighbour, owner's slot, neighbour's slot)
  const int o = gidx(wk, ix.x, m.C);
  const int nb = ix.y;
  double F[3];
  const double2* gr = (const double2*)(m.erec + e);
  const double2 n2 = __ldg(gr);
  const double nx = n2.x, ny = n2.y;
  if (nb < 0) {
    // solid wall: ElemFlux with the owner's cell-average depth (src/SpaceDisc.cpp:66-69)
    elem_flux(nx, ny, W[o] - m.bc[o], 0., 0., F);
  } else {
    const double2 t2 = __ldg(gr + 1), bl = __ldg(gr + 2);
    EdgeGeom g;
    g.nx = nx; g.ny = ny;
    g.tx = t2.x; g.ty = t2.y;
    g.b = bl.x;
    g.lmin = bl.y;
    const int sl = gidx(wk, ix.z, 3 * m.C), sr = gidx(wk, ix.w, 3 * m.C);
    DepthState L, R;
    if (SLOTS) {
      L = depth_state(SideState{wk.ew[sl], wk.eu[sl], wk.ev[sl]}, g.b);
      R = depth_state(SideState{wk.ew[sr], wk.eu[sr], wk.ev[sr]}, g.b);
    } else {
      const int n = gidx(wk, nb, m.C);
      L = DepthState{wk.eh[sl], U[o], V[o]};
      R = DepthState{wk.eh[sr], U[n], V[n]};
      slot_velocity(L.h, (wk.cls[o] & 3u) == 0u, &L.u, &L.v);
      slot_velocity(R.h, (wk.cls[n] & 3u) == 0u, &R.u, &R.v);
    }
    const double cor = m.inst_cor[inst];
    // the minimum so far (a stale one is only larger)
    const int cap = (int)((__ldcg(wk.r + inst) >> 32) & 0x7FFFFFFFull);
    if (TAPE) FLUX::eval_depth(prod, g, L, R, cor, cap, lw, F, EdgeTape{wk.ftape, m.E, e});
    else FLUX::eval_depth(prod, g, L, R, cor, cap, lw, F, NoTape{});
  }
  wk.f0[e] = F[0];
  wk.f1[e] = F[1];
  wk.f2[e] = F[2];
  return !prod.other;
}

// MODE 0: every edge, from the full interface values.  MODE 1: the edges none
// of whose cells is listed (the others wait for PartWet2 and go through k_flux_pw).
// TAPE: also store the intermediates the adjoint's reverse reads (wk.ftape).
// Register caps (the second __launch_bounds__ argument: blocks of 256 threads
// per SM) measured on the 1M-cell dam break, CUDA events, same bits: k_flux at
// 64 registers 0.211 -> 0.199 ms per launch, k_recon1 at 48 registers
// 0.091 -> 0.087 ms; more resident warps hide the gathers better than the
// few spilled registers cost.
template <class FLUX, bool BATCH, int MODE, bool TAPE, bool SOFT>
__global__ void __launch_bounds__(256, 4) k_flux(DevMesh m, DevWork wk, const double* __restrict__ W,
                                                 const double* __restrict__ U, const double* __restrict__ V) {
  __shared__ unsigned long long s_min[32];
  __shared__ int s_inst[32];
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  double lw = kInf;
  int inst = 0;
  if (e < m.E) {
    if (BATCH) inst = m.einst[e];
    bool mine = true;
    if (MODE == 1) {
      const int nb = m.enb[e];
      mine = !(listed_class(wk.cls[gidx(wk, m.eown[e], m.C)]) || (nb >= 0 && listed_class(wk.cls[gidx(wk, nb, m.C)])));
    }
    if (mine && !flux_edge<FLUX, TAPE, SOFT, MODE == 0>(m, wk, W, U, V, e, inst, &lw)) {
      lw = kInf;
      flux_edge<FLUX, TAPE, false, MODE == 0>(m, wk, W, U, V, e, inst, &lw);
    }
  }
  // min-reduction of the length-to-wavespeed ratio on order-preserving integer
  // keys (exact): warp, block, one atomicMin per block and instance
  const unsigned long long kNone = ~0ull;
  unsigned long long key = (dbits(lw) == dbits(kInf)) ? kNone : order_key(lw);
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const int inst0 = __shfl_sync(0xffffffffu, inst, 0);
  const bool warp_uniform = __all_sync(0xffffffffu, inst == inst0);
  if (warp_uniform) {
#pragma unroll
    for (int off = 16; off; off >>= 1) {
      const unsigned long long o = __shfl_xor_sync(0xffffffffu, key, off);
      key = o < key ? o : key;
    }
    if (lane == 0) {
      s_min[warp] = key;
      s_inst[warp] = inst0;
    }
  } else {
    if (key != kNone) atomicMin(wk.r + inst, key);
    if (lane == 0) {
      s_min[warp] = kNone;
      s_inst[warp] = -1;
    }
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    unsigned long long v = lane < nw ? s_min[lane] : kNone;
    int vi = lane < nw ? s_inst[lane] : s_inst[0];
    const int vi0 = __shfl_sync(0xffffffffu, vi, 0);
    const bool uni = __all_sync(0xffffffffu, vi == vi0 || v == kNone);
    if (uni) {
#pragma unroll
      for (int off = 16; off; off >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, off);
        v = o < v ? o : v;
      }
      if (lane == 0 && v != kNone) atomicMin(wk.r + vi0, v);
    } else if (v != kNone && vi >= 0) {
      atomicMin(wk.r + vi, v);
    }
  }
}

// The fluxes of the edges next to the stage's partially-wet cells (after
// PartWet2): listed cell i takes its local edge k unless the edge's owner is
// partially wet too and is not i, so that each edge is evaluated once.
template <class FLUX, bool BATCH, bool TAPE>
__global__ void __launch_bounds__(128) k_flux_pw(DevMesh m, DevWork wk, const double* __restrict__ W,
                                                 const double* __restrict__ U, const double* __restrict__ V) {
  const int C = m.C;
  const int n = 3 * min(*wk.pwcount, C);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int q = t / 3, k = t - 3 * q;
    const int i = gidx(wk, wk.pwlist[q], C);
    const int e = gidx(wk, m.cedge[k * C + i], m.E);
    const int o = gidx(wk, m.eown[e], C);
    if ((listed_class(wk.cls[o]) ? o : m.enb[e]) != i) continue;
    const int inst = BATCH ? m.einst[e] : 0;
    double lw = kInf;
    flux_edge<FLUX, TAPE, false, false>(m, wk, W, U, V, e, inst, &lw);
    if (dbits(lw) != dbits(kInf)) atomicMin(wk.r + inst, order_key(lw));
  }
}

// TimeDisc::ComputeDrainingDt once per cell; also empties the part-wet list
// for the next reconstruction.  The update only takes minima with the stage's
// dt, so a cell that plainly outlasts it (A h > 2 dt sum, dt_scale = 2 max(1, c)
// times the step's dt) keeps +inf and no quotient.
template <bool BATCH>
__global__ void __launch_bounds__(256) k_drain(DevMesh m, DevWork wk, const double* __restrict__ W, double dt_scale) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *wk.pwcount = 0;
  if (i >= m.C) return;
  const double h = W[i] - m.bc[i];
  double d;
  if (!is_wet(h)) {
    d = 0.;
  } else {
    const unsigned own = m.cown[i];
    double out[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double f = wk.f0[gidx(wk, m.cedge[k * m.C + i], m.E)];
      out[k] = smax(0., ((own >> k) & 1u) ? f : SWE_NEG(f));
    }
    const double sum = out[0] + out[1] + out[2];  // 0 + out[0] is out[0]
    d = kInf;
    if (dgtc(sum, kTol)) {
      const double vol = m.area[i] * h;
      if (!dlt(sum * (dt_scale * wk.dt[BATCH ? m.cinst[i] : 0]), vol)) d = SWE_DIV(vol, sum);
    }
  }
  wk.drain[i] = d;
}

// TimeDisc::RHS + the Shu-Osher combination + ConsAssigner.
// The output may be the same array as Wp or W0 (in-place stages): each thread
// reads its own cell before writing it, so no pointer here is __restrict__.
// STORE_N also writes the state before ConsAssigner to nst [3][C] (for the
// adjoint's segment recompute).
// HALF: a stage with a = b = c = 1/2 (SSPRK2's second), whose products with
// the coefficients are exact halvings.
// COR0: no instance has a Coriolis term.  SOFT: part of the products on the
// integer pipe.
//
// Bound by the FP64 pipe: 64-70 operations a cell of 73-79 before the slots
// held depths, the source products q g were formed once per cell and the first
// terms were negated instead of subtracted from zero.
// update_cell: (h, hu, hv) of cell i after the stage; false where a product left
// the integer routine's range.
template <bool BATCH, bool HALF, bool COR0, bool SOFT>
__device__ __forceinline__ bool update_cell(const DevMesh& m, const DevWork& wk, int i, const double* Wp,
                                            const double* Up, const double* Vp, const double* W0, const double* U0,
                                            const double* V0, const Stage& st, double* n) {
  Products<SOFT> prod;
  const int C = m.C;
  const int inst = BATCH ? m.cinst[i] : 0;
  const double dt = HALF ? SWE_HALF(wk.dt[inst]) : (st.first ? wk.dt[inst] : st.c * wk.dt[inst]);
  const unsigned own = m.cown[i];
  const double dti = wk.drain[i];
  // source terms: q times the gradient plus cor (-v, u) at a slot; the same for
  // the three slots unless one is dry or thin
  const double q = dt * (1. / 3.);
  const double gx = wk.gx[i], gy = wk.gy[i];
  const double up = Up[i], vp = Vp[i];
  const bool dry_cell = (wk.cls[i] & 3u) == 0u;
  const double cor = COR0 ? 0. : m.inst_cor[inst];
  double qsx, qsy;
  if (COR0) {
    qsx = prod.mul(q, gx);
    qsy = prod.mul(q, gy);
  } else {
    qsx = q * (gx + cor * (-vp));
    qsy = q * (gy + cor * up);
  }
  double r0 = 0., r1 = 0., r2 = 0.;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int slot = k * C + i;
    const int2 en = __ldg(m.cslot + slot);  // (edge, neighbour)
    double2 ce, nc;                         // (L/A, edge-centre z), (n_x L/A, n_y L/A)
    ldg_pair(m.srec + slot, &ce, &nc);
    const int e = gidx(wk, en.x, m.E);
    // sgn = +1 for the edge's owner, else -1: products with it are sign changes
    const bool out = (own >> k) & 1u;
    const double F0 = wk.f0[e], F1 = wk.f1[e], F2 = wk.f2[e];
    const int nb = en.y;
    const double dtik = nb < 0 ? kInf : wk.drain[gidx(wk, nb, C)];
    const double dtk = (out ? dgt0(F0) : dlt(F0, 0.)) ? smin(dt, dti) : smin(dt, dtik);  // sgn F0 > 0
    const double h_ek = wk.eh[slot];
    const double s = prod.mul(out ? dtk : SWE_NEG(dtk), ce.x);
    const double a0 = prod.mul(s, F0), a1 = prod.mul(s, F1), a2 = prod.mul(s, F2);
    if (k == 0) {
      r0 = zero_minus(a0);
      r1 = zero_minus(a1);
      r2 = zero_minus(a2);
    } else {
      r0 -= a0;
      r1 -= a1;
      r2 -= a2;
    }
    double qx = qsx, qy = qsy;
    if (COR0) {
      // a zero of g takes the sign of g + cor (-v, u) with cor = +-0
      if (((ubits(gx) << 1) == 0ull) || ((ubits(gy) << 1) == 0ull)) {
        const double c0 = m.inst_cor[inst];
        double u = up, v = vp;
        if (dry_cell || !is_wet(h_ek)) u = v = 0.;
        if ((ubits(gx) << 1) == 0ull) qx = add_zero_product(gx, c0, SWE_NEG(v));
        if ((ubits(gy) << 1) == 0ull) qy = add_zero_product(gy, c0, u);
      }
    } else if (dry_cell || dltc(h_ek, kEta1)) {
      double u = up, v = vp;
      slot_velocity(h_ek, dry_cell, &u, &v);
      qx = q * (gx + cor * (-v));
      qy = q * (gy + cor * u);
    }
    r1 -= prod.mul(qx, h_ek);
    r2 -= prod.mul(qy, h_ek);
    const double p = prod.mul(SWE_HALF(h_ek), h_ek);  // 0.5 h h
    r1 += prod.mul(dtk, prod.mul(nc.x, p));  // (n_x c) p
    r2 += prod.mul(dtk, prod.mul(nc.y, p));
  }
  const double b = m.bc[i];
  const double h0 = W0[i] - b;
  const double c00 = h0, c01 = prod.mul(h0, U0[i]), c02 = prod.mul(h0, V0[i]);
  if (st.first && !HALF) {
    n[0] = c00 + r0;
    n[1] = c01 + r1;
    n[2] = c02 + r2;
  } else {
    const double hp = Wp[i] - b;
    const double c10 = hp, c11 = prod.mul(hp, up), c12 = prod.mul(hp, vp);
    if (HALF) {
      n[0] = SWE_HALF(c00) + SWE_HALF(c10) + r0;
      n[1] = SWE_HALF(c01) + SWE_HALF(c11) + r1;
      n[2] = SWE_HALF(c02) + SWE_HALF(c12) + r2;
    } else {
      n[0] = st.a * c00 + st.b * c10 + r0;
      n[1] = st.a * c01 + st.b * c11 + r1;
      n[2] = st.a * c02 + st.b * c12 + r2;
    }
  }
  return !prod.other;
}

template <bool BATCH, bool STORE_N, bool HALF, bool COR0, bool SOFT>
__global__ void __launch_bounds__(256, 5) k_update(DevMesh m, DevWork wk, const double* Wp, const double* Up,
                                                const double* Vp, const double* W0, const double* U0,
                                                const double* V0, double* Wo, double* Uo, double* Vo, Stage st,
                                                double* nst = nullptr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m.C) return;
  if (!STORE_N) prefetch_l1(m.thr + i);  // for the class of the new state, at the end
  double n[3];
  if (!update_cell<BATCH, HALF, COR0, SOFT>(m, wk, i, Wp, Up, Vp, W0, U0, V0, st, n))
    update_cell<BATCH, HALF, COR0, false>(m, wk, i, Wp, Up, Vp, W0, U0, V0, st, n);
  const double b = m.bc[i];
  if (STORE_N) {
    nst[i] = n[0];
    nst[m.C + i] = n[1];
    nst[2 * m.C + i] = n[2];
  }
  double ow, ou, ov;
  cons_assign(b, n[0], n[1], n[2], &ow, &ou, &ov);
  Wo[i] = ow;
  Uo[i] = ou;
  Vo[i] = ov;
  // non-finite check on the exponent bits (integer pipe)
  const unsigned long long xw = (unsigned long long)dbits(ow) >> 52,
                           xu = (unsigned long long)dbits(ou) >> 52,
                           xv = (unsigned long long)dbits(ov) >> 52;
  if (((xw & 0x7FFull) == 0x7FFull) || ((xu & 0x7FFull) == 0x7FFull) || ((xv & 0x7FFull) == 0x7FFull))
    atomicOr(wk.err, kErrNonFinite);
  // list the next stage's partially-wet cells, so that their PartWet1 runs beside
  // its k_recon1 instead of after it (a plain append: one over the warp's lanes
  // kept registers across the whole kernel, 99 -> 110 us on a million cells)
  if (!STORE_N && to_list(m, i, ow, !SOFT)) {
    const int slot = atomicAdd(wk.pwcount, 1);
    if (slot < m.C) wk.pwlist[slot] = i;
  }
}

__global__ void k_init_nodes(DevMesh m, DevWork wk, bool list) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m.N) wk.maxwp[i] = order_key(m.nz[i]);
  if (list && i == 0) *wk.pwcount = 0;
}

inline int nblocks(int64_t n, int b) { return (int)((n + b - 1) / b); }

}  // namespace

// ------------------------------------------------------------------ engine
template <class T>
T* Engine::dalloc(size_t n) {
  T* p = nullptr;
  if (n == 0) n = 1;
  const cudaError_t e = device_alloc(&p, n);
  if (e != cudaSuccess) {
    alloc_error_ = e;
    return nullptr;
  }
  allocs_.push_back(p);
  bytes_ += n * sizeof(T);
  return p;
}
template int* Engine::dalloc<int>(size_t);
template double* Engine::dalloc<double>(size_t);

void Engine::set_stream(cudaStream_t s) {
  cudaStream_t next = s ? s : own_stream_;
  if (next == stream_) return;
  cudaEvent_t ev = nullptr;
  if (stream_ && cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) == cudaSuccess) {
    if (cudaEventRecord(ev, stream_) == cudaSuccess) cudaStreamWaitEvent(next, ev, 0);
    cudaEventDestroy(ev);  // released once the wait is satisfied
  } else if (stream_) {
    cudaStreamSynchronize(stream_);
  }
  stream_ = next;
}

Engine::~Engine() {
  // nothing of this engine may still run on its own streams when its memory
  // goes (a caller's stream is synchronised by swe_destroy)
  if (own_stream_) cudaStreamSynchronize(own_stream_);
  if (side_) cudaStreamSynchronize(side_);
  if (adj_) adjoint_state_delete(adj_);
  for (auto& row : graphs_)
    for (auto& g : row)
      if (g) cudaGraphExecDestroy(g);
  for (void* p : allocs_) cudaFree(p);
  if (h_word) cudaFreeHost(h_word);
  if (own_stream_) cudaStreamDestroy(own_stream_);
  if (side_) cudaStreamDestroy(side_);
  if (ev_fork_) cudaEventDestroy(ev_fork_);
  if (ev_pass1_) cudaEventDestroy(ev_pass1_);
  if (ev_join_) cudaEventDestroy(ev_join_);
}

// The side stream's blocks go first wherever an SM has room: its kernels are short
// and the stage waits for their chain.
static int side_priority() {
  int least = 0, greatest = 0;
  return cudaDeviceGetStreamPriorityRange(&least, &greatest) == cudaSuccess ? greatest : 0;
}

std::string Engine::init(std::vector<HostInstance>&& inst, int flux, int ws, int block, int* st, bool batched) {
  *st = 0;
  flux_ = flux;
  ws_ = ws;
  if (block > 0) blk_[0] = blk_[1] = blk_[2] = block;
  batched_ = batched;
  const int I = (int)inst.size();
  int64_t C = 0, E = 0, N = 0;
  cell_off.assign(I + 1, 0);
  edge_off.assign(I + 1, 0);
  node_off.assign(I + 1, 0);
  for (int q = 0; q < I; ++q) {
    std::string err = validate_instance(inst[q]);
    if (!err.empty()) {
      *st = 2;
      return (I > 1 ? "instance " + std::to_string(q) + ": " : std::string()) + err;
    }
    cell_off[q] = C;
    edge_off[q] = E;
    node_off[q] = N;
    C += inst[q].C;
    E += inst[q].E;
    N += inst[q].N;
  }
  cell_off[I] = C;
  edge_off[I] = E;
  node_off[I] = N;
  soft_ = C >= kSoftCells;
  cor0_ = true;
  for (const auto& q : inst) cor0_ = cor0_ && q.cor == 0.;
  if (3 * C > (1ll << 31) - 1 || E > (1ll << 31) - 1 || N > (1ll << 31) - 1) {
    *st = 1;
    return "total mesh too large for int32 device indexing";
  }
  HostImage img;
  img.resize((int)C, (int)E, (int)N, I);
  for (int q = 0; q < I; ++q) precompute_instance(inst[q], q, cell_off[q], edge_off[q], node_off[q], img);

  auto up = [&](auto& vec, auto*& dst) -> bool {
    using T = typename std::remove_reference<decltype(vec)>::type::value_type;
    T* d = dalloc<T>(vec.size());
    if (!d) return false;
    if (cudaMemcpy(d, vec.data(), vec.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) return false;
    dst = d;
    return true;
  };
  DevMesh& M = mesh_;
  M.C = (int)C; M.E = (int)E; M.N = (int)N; M.I = I;
  bool ok = true;
  const int *p_cnode, *p_cnbr, *p_cedge, *p_cinst, *p_eown, *p_enb, *p_esl, *p_esr, *p_einst, *p_icb;
  const double *p_area, *p_cek, *p_cnxc, *p_cnyc, *p_enx, *p_eny, *p_etx, *p_ety, *p_elmin, *p_cfl, *p_cor;
  const int2 *p_cslot, *p_enode;
  const double2* p_nxy;
  const int4* p_eidx;
  ok = ok && up(img.cnode, p_cnode) && up(img.cnbr, p_cnbr) && up(img.cedge, p_cedge) && up(img.cinst, p_cinst);
  ok = ok && up(img.cown, bed_.cown) && up(img.area, p_area);
  ok = ok && up(img.cek, p_cek) && up(img.cnxc, p_cnxc) && up(img.cnyc, p_cnyc);
  ok = ok && up(img.eown, p_eown) && up(img.enb, p_enb) && up(img.eslotl, p_esl) && up(img.eslotr, p_esr);
  ok = ok && up(img.einst, p_einst) && up(img.enx, p_enx) && up(img.eny, p_eny) && up(img.etx, p_etx);
  ok = ok && up(img.ety, p_ety) && up(img.elmin, p_elmin) && up(img.enode, p_enode) && up(img.nxy, p_nxy);
  ok = ok && up(img.inst_cell_begin, p_icb) && up(img.inst_cfl, p_cfl) && up(img.inst_cor, p_cor);
  ok = ok && up(img.srec, bed_.srec) && up(img.cslot, p_cslot) && up(img.erec, bed_.erec) && up(img.eidx, p_eidx);
  const int *p_nptr, *p_ncell;
  ok = ok && up(img.nptr, p_nptr) && up(img.ncell, p_ncell);
  bed_.bc = dalloc<double>(C); bed_.thr = dalloc<double2>(C);
  bed_.zn = dalloc<double>(3 * C); bed_.ze = dalloc<double>(3 * C);
  bed_.dry = dalloc<double>(kDryStride * C); bed_.combo = dalloc<double>(8 * kComboStride * C);
  bed_.combov = dalloc<double>(8 * kComboVStride * C);
  bed_.pw1 = dalloc<double>(kPw1Stride * C); bed_.pw2 = dalloc<Pw2Rec>(C);
  bed_.ezm = dalloc<double>(E); bed_.nz = dalloc<double>(N);
  ok = ok && bed_.bc && bed_.thr && bed_.combov && bed_.zn && bed_.ze && bed_.dry && bed_.combo && bed_.pw1 && bed_.pw2 &&
       bed_.ezm && bed_.nz;
  if (!ok) {
    *st = 6;
    return std::string("device allocation or upload failed: ") +
           cudaGetErrorString(alloc_error_ != cudaSuccess ? alloc_error_ : cudaGetLastError());
  }
  M.cnode = p_cnode; M.cnbr = p_cnbr; M.cedge = p_cedge; M.cinst = p_cinst; M.cown = bed_.cown;
  M.bc = bed_.bc; M.thr = bed_.thr; M.combov = bed_.combov; M.area = p_area; M.zn = bed_.zn; M.ze = bed_.ze; M.cek = p_cek;
  M.cnxc = p_cnxc; M.cnyc = p_cnyc; M.dry = bed_.dry; M.combo = bed_.combo; M.pw1 = bed_.pw1; M.pw2 = bed_.pw2;
  M.eown = p_eown; M.enb = p_enb; M.eslotl = p_esl; M.eslotr = p_esr; M.einst = p_einst;
  M.enx = p_enx; M.eny = p_eny; M.etx = p_etx; M.ety = p_ety; M.ezm = bed_.ezm; M.elmin = p_elmin;
  M.enode = p_enode; M.nxy = p_nxy; M.nz = bed_.nz; M.inst_cell_begin = p_icb; M.inst_cfl = p_cfl; M.inst_cor = p_cor;
  M.srec = bed_.srec; M.cslot = p_cslot; M.erec = bed_.erec; M.eidx = p_eidx;
  M.nptr = p_nptr; M.ncell = p_ncell;

  DevWork& Wk = work_;
  // What lives inside one stage or one call shares an allocation, in which the
  // field getters lay out their rows: they need no memory of their own.
  const size_t part = ((size_t)C + 31) / 32 * 32;  // 256-byte steps
  d_rows = dalloc<double>(std::max({10 * part, 6 * (size_t)E, (size_t)N}));
  if (d_rows) {
    Wk.eh = d_rows; Wk.gx = d_rows + 3 * part; Wk.gy = d_rows + 4 * part;
    Wk.drain = d_rows + 5 * part; Wk.pwrec = d_rows + 6 * part; d_io = d_rows + 7 * part;
  }
  Wk.ew = dalloc<double>(3 * C); Wk.eu = dalloc<double>(3 * C); Wk.ev = dalloc<double>(3 * C);
  Wk.sx = dalloc<double>(3 * C); Wk.sy = dalloc<double>(3 * C);
  Wk.f0 = dalloc<double>(E); Wk.f1 = dalloc<double>(E); Wk.f2 = dalloc<double>(E);
  Wk.maxwp = dalloc<unsigned long long>(N);
  Wk.pwlist = dalloc<int>(C);
  Wk.pwcount = dalloc<int>(1);
  Wk.cls = dalloc<unsigned char>(C);
  Wk.ftape = nullptr;
  Wk.r = dalloc<unsigned long long>(I);
  Wk.dt = dalloc<double>(I);
  Wk.tsum = dalloc<double>(I);
  d_fixed_dt = dalloc<double>(I);  // per instance
  Wk.fixed_dt = d_fixed_dt;
  Wk.err = dalloc<unsigned>(1);
  M.err = Wk.err;
  for (int q = 0; q < 6; ++q) state_[q] = dalloc<double>(C);
  d_ioflag = dalloc<unsigned>(1);
  if (!d_rows || !Wk.ew || !Wk.eu || !Wk.ev || !Wk.sx || !Wk.sy || !Wk.f0 || !Wk.f1 || !Wk.f2 || !Wk.maxwp ||
      !Wk.pwlist || !Wk.pwcount || !Wk.cls || !Wk.r || !Wk.dt || !Wk.tsum || !d_fixed_dt || !Wk.err ||
      !state_[5] || !d_ioflag) {
    *st = 6;
    return "device allocation failed";
  }
  if (cudaMallocHost(&h_word, sizeof(*h_word)) != cudaSuccess) {
    *st = 6;
    return "pinned allocation failed";
  }
  cudaMemset(Wk.eh, 0, 3 * C * sizeof(double));
  cudaMemset(Wk.gx, 0, C * sizeof(double));
  cudaMemset(Wk.gy, 0, C * sizeof(double));
  cudaMemset(Wk.ew, 0, 3 * C * sizeof(double));
  cudaMemset(Wk.eu, 0, 3 * C * sizeof(double));
  cudaMemset(Wk.ev, 0, 3 * C * sizeof(double));
  cudaMemset(Wk.sx, 0, 3 * C * sizeof(double));
  cudaMemset(Wk.sy, 0, 3 * C * sizeof(double));
  cudaMemset(Wk.f0, 0, E * sizeof(double));
  cudaMemset(Wk.f1, 0, E * sizeof(double));
  cudaMemset(Wk.f2, 0, E * sizeof(double));
  cudaMemset(Wk.pwcount, 0, sizeof(int));
  cudaMemset(Wk.pwlist, 0, C * sizeof(int));  // every entry a valid cell id from the start
  cudaMemset(Wk.dt, 0, I * sizeof(double));
  cudaMemset(Wk.tsum, 0, I * sizeof(double));
  cudaMemset(Wk.err, 0, sizeof(unsigned));
  std::vector<unsigned long long> one(I, order_key(1.0));
  cudaMemcpy(Wk.r, one.data(), I * sizeof(unsigned long long), cudaMemcpyHostToDevice);
  if (cudaStreamCreateWithFlags(&own_stream_, cudaStreamNonBlocking) != cudaSuccess ||
      cudaStreamCreateWithPriority(&side_, cudaStreamNonBlocking, side_priority()) != cudaSuccess ||
      cudaEventCreateWithFlags(&ev_fork_, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&ev_pass1_, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&ev_join_, cudaEventDisableTiming) != cudaSuccess) {
    *st = 5;
    return "stream creation failed";
  }
  stream_ = own_stream_;
  host = std::move(inst);
  const std::vector<double> nz = host_nz();
  cudaError_t ce = compute_bed(nz.data());
  k_init_nodes<<<nblocks(N, 256), 256, 0, stream_>>>(M, Wk, true);
  ++launches_;
  if (ce == cudaSuccess) ce = cudaGetLastError();
  const cudaError_t cs = cudaStreamSynchronize(stream_);  // also on failure: the copy reads nz
  if (ce == cudaSuccess) ce = cs;
  if (ce != cudaSuccess) {
    *st = 5;
    return std::string("CUDA error during set-up: ") + cudaGetErrorString(ce);
  }
  return "";
}

cudaError_t Engine::reset_pass(bool list) {
  k_init_nodes<<<nblocks(std::max(mesh_.N, 1), 256), 256, 0, stream_>>>(mesh_, work_, list);
  launches_ += 1;
  return cudaGetLastError();
}

void Engine::launch_recon1(const double* W, const double* U, const double* V, int latch_mode, bool slots,
                           List list) {
  const int b = blk_[0], g = nblocks(mesh_.C, b);
  const bool append = list != kNoList, finish = list != kEveryPartWet && !soft_;
  const int form = !slots ? kLean : cor0_ ? kSlotsCor0 : kSlotsCor;
  switch (form + (batched_ ? 3 : 0)) {
    case 0: k_recon1<false, kLean><<<g, b, 0, stream_>>>(mesh_, work_, W, U, V, latch_mode, append, finish); break;
    case 1: k_recon1<false, kSlotsCor0><<<g, b, 0, stream_>>>(mesh_, work_, W, U, V, latch_mode, append, finish); break;
    case 2: k_recon1<false, kSlotsCor><<<g, b, 0, stream_>>>(mesh_, work_, W, U, V, latch_mode, append, finish); break;
    case 3: k_recon1<true, kLean><<<g, b, 0, stream_>>>(mesh_, work_, W, U, V, latch_mode, append, finish); break;
    case 4: k_recon1<true, kSlotsCor0><<<g, b, 0, stream_>>>(mesh_, work_, W, U, V, latch_mode, append, finish); break;
    default: k_recon1<true, kSlotsCor><<<g, b, 0, stream_>>>(mesh_, work_, W, U, V, latch_mode, append, finish); break;
  }
  ++launches_;
}

// Blocks of the kernels over the listed cells (128 threads): one lane a cell for
// every cell, or 8 for kGroupCells of them, at most one full device.
int Engine::listed_blocks() const {
  const int b = 128;
  return std::min(std::max(nblocks(mesh_.C, b), nblocks(8ll * std::min(mesh_.C, kGroupCells), b)), 6 * 152);
}

void Engine::launch_partwet1(const double* W, cudaStream_t s) {
  k_partwet1<<<listed_blocks(), 128, 0, s>>>(mesh_, work_, W);
  ++launches_;
}

cudaError_t Engine::list_partwet(const double* W) {
  const cudaError_t pending = cudaPeekAtLastError();
  cudaError_t e = cudaMemsetAsync(work_.pwcount, 0, sizeof(int), stream_);
  if (e != cudaSuccess) return e;
  k_list_partwet<<<nblocks(mesh_.C, 256), 256, 0, stream_>>>(mesh_, work_, W, !soft_);
  ++launches_;
  return launch_error(pending);
}

cudaError_t Engine::ensure_list() {
  if (list_valid_ && !captured_) return cudaSuccess;
  return list_partwet(state(0, 0));
}

// The flags of steps of n stages that were accepted: the last update listed the
// new state's cells, and steps of several stages leave the full interface values
// to refresh_slots.  (A refused one leaves both as they are, or unlisted.)
void Engine::note_steps(int n) {
  list_valid_ = true;
  slots_stale_ = n > 1 && !captured_;
}

void Engine::launch_recon2(const double* W, const double* U, const double* V, cudaStream_t s, bool slots) {
  const int b = 128, g = listed_blocks();
  const int form = !slots ? kLean : cor0_ ? kSlotsCor0 : kSlotsCor;
  switch (form + (batched_ ? 3 : 0)) {
    case 0: k_recon2<false, kLean><<<g, b, 0, s>>>(mesh_, work_, W, U, V); break;
    case 1: k_recon2<false, kSlotsCor0><<<g, b, 0, s>>>(mesh_, work_, W, U, V); break;
    case 2: k_recon2<false, kSlotsCor><<<g, b, 0, s>>>(mesh_, work_, W, U, V); break;
    case 3: k_recon2<true, kLean><<<g, b, 0, s>>>(mesh_, work_, W, U, V); break;
    case 4: k_recon2<true, kSlotsCor0><<<g, b, 0, s>>>(mesh_, work_, W, U, V); break;
    default: k_recon2<true, kSlotsCor><<<g, b, 0, s>>>(mesh_, work_, W, U, V); break;
  }
  ++launches_;
}

bool Engine::note_capture() {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream_, &st) != cudaSuccess) cudaGetLastError();
  const bool now = st == cudaStreamCaptureStatusActive;
  captured_ = captured_ || now;
  return now;
}

cudaError_t Engine::keep_input() {
  cudaError_t e = cudaSuccess;
  for (int c = 0; c < 3 && e == cudaSuccess; ++c)
    e = cudaMemcpyAsync(state(1, c), state(0, c), mesh_.C * sizeof(double), cudaMemcpyDeviceToDevice, stream_);
  return e;
}

cudaError_t Engine::interface_values(const double* W, const double* U, const double* V, List list) {
  const bool now = W == state(0, 0) && note_capture();
  if (W == state(0, 0) && captured_) {
    cudaError_t e = keep_input();
    if (e != cudaSuccess) return e;
  }
  launch_recon1(W, U, V, 0, true, list);
  launch_partwet1(W, stream_);
  launch_recon2(W, U, V, stream_, true);
  k_node_max_all<<<nblocks(std::max(mesh_.N, 1), 256), 256, 0, stream_>>>(mesh_, work_, W);
  ++launches_;
  slots_stale_ = slots_stale_ && now;  // recorded only: nothing has run
  list_valid_ = W == state(0, 0) && list == kStepList;
  return cudaGetLastError();
}

cudaError_t Engine::refresh_slots() {
  const bool now = note_capture();
  if (!slots_stale_) return cudaSuccess;
  const cudaError_t pending = cudaPeekAtLastError();
  // the last stage read buffer 1; the CFL ratio of its flux pass stays
  cudaError_t e = cudaMemsetAsync(work_.pwcount, 0, sizeof(int), stream_);
  if (e != cudaSuccess) return e;
  launch_recon1(state(1, 0), state(1, 1), state(1, 2), 3, true, kStepList);
  launch_partwet1(state(1, 0), stream_);
  launch_recon2(state(1, 0), state(1, 1), state(1, 2), stream_, true);
  slots_stale_ = now;
  list_valid_ = false;  // it is that buffer's now
  return launch_error(pending);
}

// The plugin of (flux, wave speed), given to f as a type.
template <class F>
static void with_plugin(int flux, int ws, F&& f) {
  switch (flux * 3 + ws) {
    case 0: f(HLL<Rusanov>{}); break;
    case 1: f(HLL<Davis>{}); break;
    case 2: f(HLL<Einfeldt>{}); break;
    case 3: f(HLLC<Rusanov>{}); break;
    case 4: f(HLLC<Davis>{}); break;
    default: f(HLLC<Einfeldt>{}); break;
  }
}

template <class FLUX, bool BATCH>
static void launch_stage_flux(bool tape, bool soft, int g, int b, cudaStream_t s, const DevMesh& m, const DevWork& w,
                              const double* const* in) {
  switch ((tape ? 2 : 0) | (soft ? 1 : 0)) {
    case 0: k_flux<FLUX, BATCH, 1, false, false><<<g, b, 0, s>>>(m, w, in[0], in[1], in[2]); break;
    case 1: k_flux<FLUX, BATCH, 1, false, true><<<g, b, 0, s>>>(m, w, in[0], in[1], in[2]); break;
    case 2: k_flux<FLUX, BATCH, 1, true, false><<<g, b, 0, s>>>(m, w, in[0], in[1], in[2]); break;
    default: k_flux<FLUX, BATCH, 1, true, true><<<g, b, 0, s>>>(m, w, in[0], in[1], in[2]); break;
  }
}

cudaError_t Engine::fluxes(const double* W) {
  const int b = blk_[1], g = nblocks(mesh_.E, b);
  with_plugin(flux_, ws_, [&](auto plugin) {
    typedef decltype(plugin) P;
    if (batched_) k_flux<P, true, 0, false, false><<<g, b, 0, stream_>>>(mesh_, work_, W, nullptr, nullptr);
    else k_flux<P, false, 0, false, false><<<g, b, 0, stream_>>>(mesh_, work_, W, nullptr, nullptr);
  });
  launches_ += 1;
  return cudaGetLastError();
}

cudaError_t Engine::stage_fluxes(const double* const* in) {
  const int b = blk_[1], g = nblocks(mesh_.E, b);
  const bool tape = work_.ftape != nullptr;
  with_plugin(flux_, ws_, [&](auto plugin) {
    typedef decltype(plugin) P;
    if (batched_) launch_stage_flux<P, true>(tape, soft_, g, b, stream_, mesh_, work_, in);
    else launch_stage_flux<P, false>(tape, soft_, g, b, stream_, mesh_, work_, in);
  });
  launches_ += 1;
  return cudaGetLastError();
}

void Engine::stage_fluxes_pw(const double* const* in, cudaStream_t s) {
  const int g = std::max(1, std::min((3 * (int)mesh_.C + 127) / 128, 152 * 8));
  const bool tape = work_.ftape != nullptr;
  with_plugin(flux_, ws_, [&](auto plugin) {
    typedef decltype(plugin) P;
    if (batched_ && tape) k_flux_pw<P, true, true><<<g, 128, 0, s>>>(mesh_, work_, in[0], in[1], in[2]);
    else if (batched_) k_flux_pw<P, true, false><<<g, 128, 0, s>>>(mesh_, work_, in[0], in[1], in[2]);
    else if (tape) k_flux_pw<P, false, true><<<g, 128, 0, s>>>(mesh_, work_, in[0], in[1], in[2]);
    else k_flux_pw<P, false, false><<<g, 128, 0, s>>>(mesh_, work_, in[0], in[1], in[2]);
  });
  launches_ += 1;
}

cudaError_t Engine::launch_stage(const Stage& st, const double* const* in, const double* const* u0,
                                 double* const* out, bool first_stage_of_step, int latch_mode, bool full, cudaEvent_t* ev) {
  const int b = blk_[2];
  const int lm = first_stage_of_step ? latch_mode : 0;
  // a last stage that overwrites its own input (Euler) leaves the full interface
  // values now: refresh_slots could not make them later.  Inner stages in buffer 1
  // (SSPRK3's second) take this form too, although the next one replaces the values.
  const bool slots = full || in[0] == out[0];
  // (the input's partially-wet cells are listed: by the update before, or ensure_list)
  if (ev) {
    // per-kernel timing: the kernels one after another
    cudaEventRecord(ev[0], stream_);
    launch_recon1(in[0], in[1], in[2], lm, slots, kNoList);
    cudaEventRecord(ev[1], stream_);
    launch_partwet1(in[0], stream_);
    launch_recon2(in[0], in[1], in[2], stream_, slots);
    cudaEventRecord(ev[2], stream_);
    stage_fluxes_pw(in, stream_);
    cudaError_t e = stage_fluxes(in);
    if (e != cudaSuccess) return e;
    cudaEventRecord(ev[3], stream_);
  } else {
    // on the side stream: PartWet1 beside pass 1, then PartWet2 and the fluxes
    // next to partially-wet cells beside the other edges' fluxes
    cudaEventRecord(ev_fork_, stream_);
    cudaStreamWaitEvent(side_, ev_fork_, 0);
    launch_partwet1(in[0], side_);
    launch_recon1(in[0], in[1], in[2], lm, slots, kNoList);
    cudaEventRecord(ev_pass1_, stream_);
    cudaStreamWaitEvent(side_, ev_pass1_, 0);
    launch_recon2(in[0], in[1], in[2], side_, slots);
    stage_fluxes_pw(in, side_);
    cudaEventRecord(ev_join_, side_);
    cudaError_t e = stage_fluxes(in);
    if (e != cudaSuccess) return e;
    cudaStreamWaitEvent(stream_, ev_join_, 0);
  }
  const double dt_scale = 2. * std::max(1., st.first ? 1. : st.c);
  if (batched_) k_drain<true><<<nblocks(mesh_.C, b), b, 0, stream_>>>(mesh_, work_, in[0], dt_scale);
  else k_drain<false><<<nblocks(mesh_.C, b), b, 0, stream_>>>(mesh_, work_, in[0], dt_scale);
  if (ev) cudaEventRecord(ev[4], stream_);
  ++launches_;
  launch_update(st, in, u0, out, nullptr);
  if (ev) cudaEventRecord(ev[5], stream_);
  return cudaGetLastError();
}

template <bool BATCH, bool STORE_N, bool HALF>
static void update_kernel(int g, int b, cudaStream_t s, bool cor0, bool soft, const DevMesh& m, const DevWork& w,
                          const Stage& st, const double* const* in, const double* const* u0, double* const* out,
                          double* nst) {
#define SWE_UPDATE(COR0, SOFT)                                                                             \
  k_update<BATCH, STORE_N, HALF, COR0, SOFT><<<g, b, 0, s>>>(m, w, in[0], in[1], in[2], u0[0], u0[1], u0[2], \
                                                             out[0], out[1], out[2], st, nst)
  if (cor0 && soft) SWE_UPDATE(true, true);
  else if (cor0) SWE_UPDATE(true, false);
  else if (soft) SWE_UPDATE(false, true);
  else SWE_UPDATE(false, false);
#undef SWE_UPDATE
}

void Engine::launch_update(const Stage& st, const double* const* in, const double* const* u0, double* const* out,
                           double* nst) {
  const int b = blk_[2], g = nblocks(mesh_.C, b);
  const bool half = !st.first && st.a == 0.5 && st.b == 0.5 && st.c == 0.5;
  auto run = [&](auto kernel) { kernel(g, b, stream_, cor0_, soft_, mesh_, work_, st, in, u0, out, nst); };
  switch ((batched_ ? 4 : 0) | (nst ? 2 : 0) | (half ? 1 : 0)) {
    case 0: run(update_kernel<false, false, false>); break;
    case 1: run(update_kernel<false, false, true>); break;
    case 2: run(update_kernel<false, true, false>); break;
    case 3: run(update_kernel<false, true, true>); break;
    case 4: run(update_kernel<true, false, false>); break;
    case 5: run(update_kernel<true, false, true>); break;
    case 6: run(update_kernel<true, true, false>); break;
    default: run(update_kernel<true, true, true>); break;
  }
  ++launches_;
}

cudaError_t Engine::step_timed(int scheme, int latch_mode, double* acc) {
  const Scheme sc = scheme_of(scheme);
  double* S0[3] = {state(0, 0), state(0, 1), state(0, 2)};
  double* S1[3] = {state(1, 0), state(1, 1), state(1, 2)};
  cudaEvent_t ev[kMaxStages][6];
  for (auto& row : ev)
    for (auto& x : row) cudaEventCreate(&x);
  cudaError_t e = ensure_list();
  if (e == cudaSuccess && captured_ && sc.n == 1) e = keep_input();
  for (int s = 0; s < sc.n && e == cudaSuccess; ++s) {
    const bool last = (s == sc.n - 1);
    const double* const* in = (s == 0) ? S0 : S1;
    double* const* out = last ? S0 : S1;
    e = launch_stage(sc.s[s], in, S0, out, s == 0, latch_mode, captured_, ev[s]);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream_);
  if (e != cudaSuccess) list_valid_ = false;
  if (e == cudaSuccess) {
    note_steps(sc.n);
    for (int s = 0; s < sc.n; ++s)
      for (int k = 0; k < 5; ++k) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ev[s][k], ev[s][k + 1]);
        acc[k] += ms;
      }
    float tot = 0.f;
    cudaEventElapsedTime(&tot, ev[0][0], ev[sc.n - 1][5]);
    acc[5] += tot;
  }
  for (auto& row : ev)
    for (auto& x : row) cudaEventDestroy(x);
  return e;
}

void Engine::set_custom_scheme(const Scheme& sc) {
  custom_ = sc;
  for (auto& g : graphs_[kCustomScheme])
    if (g) {
      cudaGraphExecDestroy(g);
      g = nullptr;
    }
}

void Engine::set_blocks(const int blocks[3]) {
  bool same = true;
  for (int q = 0; q < 3; ++q) same = same && blk_[q] == blocks[q];
  if (same) return;
  for (int q = 0; q < 3; ++q) blk_[q] = blocks[q];
  for (auto& row : graphs_)
    for (auto& g : row)
      if (g) {
        cudaGraphExecDestroy(g);
        g = nullptr;
      }
}

namespace {
std::mutex g_tune_mu;
std::map<std::array<int, 7>, std::array<int, 3>> g_tune_cache;
}  // namespace

cudaError_t Engine::snapshot(double* buf, bool restore) {
  const int64_t C = mesh_.C;
  cudaError_t r = cudaSuccess;
  for (int c = 0; c < 3 && r == cudaSuccess; ++c)
    r = restore ? cudaMemcpyAsync(state(0, c), buf + c * C, C * sizeof(double), cudaMemcpyDeviceToDevice, stream_)
                : cudaMemcpyAsync(buf + c * C, state(0, c), C * sizeof(double), cudaMemcpyDeviceToDevice, stream_);
  if (restore) {
    state_changed();
    if (r == cudaSuccess) r = cudaMemsetAsync(work_.tsum, 0, mesh_.I * sizeof(double), stream_);
    if (r == cudaSuccess) r = cudaMemsetAsync(work_.dt, 0, mesh_.I * sizeof(double), stream_);
    if (r == cudaSuccess) r = cudaMemsetAsync(work_.err, 0, sizeof(unsigned), stream_);
  }
  return r;
}

cudaError_t Engine::autotune_blocks(int scheme) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int lg = 0;
  while ((1ll << (lg + 1)) <= (int64_t)mesh_.C) ++lg;
  const std::array<int, 7> key = {dev, flux_, ws_, batched_ ? 1 : 0, cor0_ ? 1 : 0, scheme, lg};
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tune_cache.find(key);
    if (it != g_tune_cache.end()) {
      set_blocks(it->second.data());
      return cudaSuccess;
    }
  }
  double* save = nullptr;
  e = device_alloc(&save, 3 * (size_t)mesh_.C);
  if (e != cudaSuccess) return e;
  static const int kCand[3] = {64, 128, 256};
  const double inf = std::numeric_limits<double>::infinity();
  double t[3][3] = {{inf, inf, inf}, {inf, inf, inf}, {inf, inf, inf}};  // [group][candidate]
  e = snapshot(save, false);
  for (int ci = 0; ci < 3 && e == cudaSuccess; ++ci) {
    const int b3[3] = {kCand[ci], kCand[ci], kCand[ci]};
    set_blocks(b3);
    for (int rep = 0; rep < 4 && e == cudaSuccess; ++rep) {  // rep 0 warms up
      double acc[6] = {0., 0., 0., 0., 0., 0.};
      e = snapshot(save, true);
      if (e == cudaSuccess) e = step_timed(scheme, 1, acc);
      if (e != cudaSuccess || rep == 0) continue;
      t[0][ci] = std::min(t[0][ci], acc[0] + acc[1]);
      t[1][ci] = std::min(t[1][ci], acc[2]);
      t[2][ci] = std::min(t[2][ci], acc[3] + acc[4]);
    }
  }
  int best[3] = {256, 256, 256};
  if (e == cudaSuccess)
    for (int g = 0; g < 3; ++g) {
      int k = 2;  // ties keep the largest block
      for (int ci = 1; ci >= 0; --ci)
        if (t[g][ci] < t[g][k]) k = ci;
      best[g] = kCand[k];
    }
  set_blocks(best);
  // back to the state before tuning
  cudaError_t e2 = snapshot(save, true);
  if (e2 == cudaSuccess) e2 = cudaStreamSynchronize(stream_);
  cudaFree(save);
  if (e == cudaSuccess) e = e2;
  if (e == cudaSuccess) {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune_cache[key] = {best[0], best[1], best[2]};
  }
  return e;
}

cudaError_t Engine::time_steps(int scheme, int n, float* ms) {
  double* save = nullptr;
  cudaError_t e = device_alloc(&save, 3 * (size_t)mesh_.C);
  if (e != cudaSuccess) return e;
  cudaEvent_t a = nullptr, b = nullptr;
  e = snapshot(save, false);
  if (e == cudaSuccess) e = cudaEventCreate(&a);
  if (e == cudaSuccess) e = cudaEventCreate(&b);
  if (e == cudaSuccess) e = run_graph(scheme, 1, 1);
  if (e == cudaSuccess) e = cudaEventRecord(a, stream_);
  if (e == cudaSuccess) e = run_graph(scheme, 1, n);
  if (e == cudaSuccess) e = cudaEventRecord(b, stream_);
  if (e == cudaSuccess) e = cudaEventSynchronize(b);
  if (e == cudaSuccess) {
    e = cudaEventElapsedTime(ms, a, b);
    *ms /= (float)n;
  }
  cudaError_t e2 = snapshot(save, true);
  if (e2 == cudaSuccess) e2 = cudaStreamSynchronize(stream_);
  if (a) cudaEventDestroy(a);
  if (b) cudaEventDestroy(b);
  cudaFree(save);
  return e == cudaSuccess ? e2 : e;
}

std::string Engine::set_layouts(std::vector<Layout>&& lay) {
  layouts = std::move(lay);
  bool any = false;
  for (const Layout& L : layouts) any = any || !L.identity();
  if (!any) return "";
  std::vector<int> from((size_t)mesh_.C);
  for (size_t q = 0; q < layouts.size(); ++q) {
    const int64_t c0 = cell_off[q], n = cell_off[q + 1] - c0;
    for (int64_t j = 0; j < n; ++j) from[c0 + j] = layouts[q].identity() ? (int)j : (int)layouts[q].cell_from[j];
  }
  std::vector<int> to((size_t)mesh_.C);
  for (size_t q = 0; q < layouts.size(); ++q) {
    const int64_t c0 = cell_off[q], n = cell_off[q + 1] - c0;
    for (int64_t j = 0; j < n; ++j) to[c0 + from[c0 + j]] = (int)(c0 + j);
  }
  d_cell_from = dalloc<int>(from.size());
  d_cell_to = dalloc<int>(to.size());
  if (!d_cell_from || !d_cell_to) return "device allocation failed";
  if (cudaMemcpy(d_cell_from, from.data(), from.size() * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(d_cell_to, to.data(), to.size() * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess)
    return std::string("uploading the cell layout: ") + cudaGetErrorString(cudaGetLastError());
  if (batched_) return "";
  // a context's field getters renumber edges and nodes too
  auto ints = [](const std::vector<int64_t>& v) { return std::vector<int>(v.begin(), v.end()); };
  std::string e = upload_map(ints(layouts[0].edge_from), &d_edge_caller);
  if (e.empty()) e = upload_map(ints(layouts[0].node_from), &d_node_caller);
  d_cell_caller = d_cell_from;
  return e;
}

std::string Engine::upload_map(const std::vector<int>& h, int** d) {
  int* p = dalloc<int>(h.size());
  if (!p) return "device allocation failed";
  const cudaError_t e = consume(cudaMemcpy(p, h.data(), h.size() * sizeof(int), cudaMemcpyHostToDevice));
  if (e != cudaSuccess) return std::string("uploading the caller order: ") + cudaGetErrorString(e);
  *d = p;
  return "";
}

std::string Engine::set_bathymetry(const std::vector<const double*>& z) {
  if (z.size() != host.size()) return "one bathymetry pointer per instance is required";
  for (size_t q = 0; q < host.size(); ++q) {
    if (!z[q]) continue;
    const HostInstance& h = host[q];
    const Layout* L = q < layouts.size() ? &layouts[q] : nullptr;
    for (int64_t p = 0; p < h.N; ++p)
      if (!std::isfinite(z[q][(L && !L->identity()) ? L->node_from[p] : p])) return "bathymetry has a non-finite value";
  }
  // the interface values stay those of the last reconstruction: left to a getter,
  // they would be made of its input and the new bed.  (A batch has no call that
  // reads them.)  Three kernels, within the runs' spread (1 %) of an iteration of
  // a 20k-cell gauge inversion, 11.7 ms.
  if (!batched_) {
    const cudaError_t es = refresh_slots();
    if (es != cudaSuccess) return std::string("interface values of the old bed: ") + cudaGetErrorString(es);
  }
  for (size_t q = 0; q < host.size(); ++q) {
    if (!z[q]) continue;
    HostInstance& h = host[q];
    const Layout* L = q < layouts.size() ? &layouts[q] : nullptr;
    for (int64_t p = 0; p < h.N; ++p) h.geom[3 * p + 2] = z[q][(L && !L->identity()) ? L->node_from[p] : p];
  }
  state_changed();
  const std::vector<double> nz = host_nz();
  cudaError_t e = compute_bed(nz.data());
  // the adjoint's tape and plane tables belong to the old bed
  if (adj_ && e == cudaSuccess) e = adjoint_state_new_bed(adj_, mesh_, stream_);
  // nz must outlive the asynchronous copy
  const cudaError_t es = cudaStreamSynchronize(stream_);
  if (e == cudaSuccess) e = es;
  return e == cudaSuccess ? "" : std::string("recomputing the mesh records: ") + cudaGetErrorString(e);
}

std::vector<double> Engine::host_nz() const {
  std::vector<double> nz((size_t)mesh_.N);
  for (size_t q = 0; q < host.size(); ++q)
    for (int64_t p = 0; p < host[q].N; ++p) nz[node_off[q] + p] = host[q].geom[3 * p + 2];
  return nz;
}

cudaError_t Engine::update_only(const Stage& st, const double* const* in, const double* const* u0,
                                double* const* out, double* nst) {
  launch_update(st, in, u0, out, nst);
  return cudaGetLastError();
}

cudaError_t Engine::step(int scheme, int latch_mode) {
  const Scheme sc = scheme_of(scheme);
  double* S0[3] = {state(0, 0), state(0, 1), state(0, 2)};
  double* S1[3] = {state(1, 0), state(1, 1), state(1, 2)};
  if (captured_ && sc.n == 1) {
    cudaError_t e = keep_input();
    if (e != cudaSuccess) return e;
  }
  for (int s = 0; s < sc.n; ++s) {
    const bool last = (s == sc.n - 1);
    const double* const* in = (s == 0) ? S0 : S1;
    double* const* out = last ? S0 : S1;
    cudaError_t e = launch_stage(sc.s[s], in, S0, out, s == 0, latch_mode, captured_);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t Engine::run_graph(int scheme, int latch_mode, int64_t n) {
  if (n <= 0) return cudaSuccess;
  const cudaError_t el = ensure_list();
  if (el != cudaSuccess) return el;
  if (captured_ && !graphs_slots_) {
    // the graphs of before leave no interface values; dropped here, as a call
    // that frees something would break off the caller's capture
    for (auto& row : graphs_)
      for (auto& g : row)
        if (g) {
          cudaGraphExecDestroy(g);
          g = nullptr;
        }
    graphs_slots_ = true;
  }
  cudaGraphExec_t& ge = graphs_[scheme][latch_mode];
  const int64_t per_step = launches_;
  if (!ge) {
    // capture on a private stream so that any caller stream (even the legacy
    // default one) can replay the graph
    cudaStream_t cap;
    if (cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking) != cudaSuccess) return cudaGetLastError();
    cudaStream_t saved = stream_;
    stream_ = cap;
    cudaGraph_t g;
    cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) {
      stream_ = saved;
      cudaStreamDestroy(cap);
      return e;
    }
    e = step(scheme, latch_mode);
    cudaError_t e2 = cudaStreamEndCapture(cap, &g);
    stream_ = saved;
    cudaStreamDestroy(cap);
    if (e != cudaSuccess) return e;
    if (e2 != cudaSuccess) return e2;
    e = cudaGraphInstantiate(&ge, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
      ge = nullptr;
      return e;
    }
    launches_ = per_step;  // capture launched nothing
  }
  const int64_t kernels_per_step = 7 * scheme_of(scheme).n;
  for (int64_t s = 0; s < n; ++s) {
    cudaError_t e = cudaGraphLaunch(ge, stream_);
    if (e != cudaSuccess) {
      list_valid_ = false;  // refused (a stream that is being captured): no listing ran
      return consume(e);
    }
    if (s == 0) note_steps(scheme_of(scheme).n);
  }
  launches_ += kernels_per_step * n;
  return cudaSuccess;
}

}  // namespace swe
