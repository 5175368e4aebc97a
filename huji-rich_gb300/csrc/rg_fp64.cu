// rg_fp64.cu -- plain-FP64 kernels of the hydro hot path for sm_103a.
//
// Compiled with --fmad=false: every multiply and add rounds separately, in
// the reference's order, so results are bit-identical to the reference's
// FP64 path (IEEE division and square root are exact-rounded on the device
// as on the host).  Each device function cites the reference code it
// restates (paths relative to the RICH source root).
//
// Passes of one step (hdsim::TimeAdvance, hdsim2d.cpp:149-241, fixed mesh):
//   k_cfl        per cell: SimpleCFL bound, block min, last block writes dt (the
//                first step only: each update forms the next one's)
//   k_slopes     per cell and component: LinearGaussImproved slope + limiter (order 2)
//   k_faces      per face: reconstruction to the face, HLLC in the face frame,
//                rotation back, optional dt*area scaling
//   k_update     per cell: ascending-face CSR gather of the face fluxes
//                (SimpleExtensiveUpdater order, no atomics) + SimpleCellUpdater
// Geometry-only terms are computed once per mesh upload (k_geom_*).
#include <math.h>

#include "rg_launch.cuh"
#include "rg_adjoint.cuh"
#include "rg_face.cuh"
#include "rg_fp64.cuh"
#include "rg_hllc.cuh"
#include "rg_lgi.cuh"

namespace rg {
namespace {

constexpr int kBlock = 256;

// ---------------------------------------------------------------- geometry

// Per face: physical_geometry.cpp:8-11 calcArea, Edge.cpp:83-86 Parallel,
// spatial_reconstruction.cpp:3-6 CalcCentroid, the flux-frame normal of
// simple_flux_calculator.cpp:91-93 (order 1) or modular_flux_calculator.cpp:12-22
// with simple_flux_calculator.cpp:27-31 (order 2).
__global__ void __launch_bounds__(kBlock) k_geom_faces(GeomArgs a) {
  chain_wait();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.mesh.e || mesh_rejected(a.mesh)) return;
  const int2 fc = a.mesh.face_cells[e];
  const dbl4 v = a.mesh.face_vertices[e];
  const double ax = v.x - v.z, ay = v.y - v.w;
  const double area = root(ax * ax + ay * ay);
  a.area[e] = area;
  const double2 p = make_double2(v.z - v.x, v.w - v.y);
  a.par[e] = p;
  const double2 mid = make_double2((v.x + v.z) * 0.5, (v.y + v.w) * 0.5);
  double2 n;
  if (a.order == 1) {
    const double2 x0 = a.mesh.points[fc.x], x1 = a.mesh.points[fc.y];
    n = make_double2(x1.x - x0.x, x1.y - x0.y);
  } else {
    double2 w;
    if (fc.x >= 0 && fc.x < a.mesh.n) {
      const double2 x0 = a.mesh.points[fc.x];
      w = make_double2(v.x - x0.x, v.y - x0.y);
    } else {
      const double2 x1 = a.mesh.points[fc.y];
      w = make_double2(x1.x - v.x, x1.y - v.y);
    }
    const double sp = w.x * p.x + w.y * p.y;
    const double pp = p.x * p.x + p.y * p.y;
    n = make_double2(w.x - quot(p.x * sp, pp), w.y - quot(p.y * sp, pp));
  }
  a.nrm[e] = n;
  a.nabs[e] = root(n.x * n.x + n.y * n.y);
  const double2 c0 = a.mesh.cms[fc.x], c1 = a.mesh.cms[fc.y];
  a.dm0[e] = make_double2(mid.x - c0.x, mid.y - c0.y);
  a.dm1[e] = make_double2(mid.x - c1.x, mid.y - c1.y);
  // |x1 - x0| (VoronoiMesh::CalcFaceVelocity's |rR - rL|) and the per-face
  // halves of calc_naive_slope (LinearGaussImproved.cpp:85-88): r_ij =
  // normalize(x_other - x_cell)*length and c_ij = centroid - 0.5*(cm_other +
  // cm_cell).  The second cell's r_ij is exactly -r_ij (x_a - x_b = -(x_b -
  // x_a), and rounding is sign-symmetric) and its c_ij the same (the sum
  // commutes), so each face computes them once.
  const double2 x0 = a.mesh.points[fc.x], x1 = a.mesh.points[fc.y];
  const double ddx = x1.x - x0.x, ddy = x1.y - x0.y;
  const double dab = root(ddx * ddx + ddy * ddy);
  a.dab[e] = dab;
  // Edge::GetLength = |second - first| = |first - second| = area
  a.rij[e] = make_double2(quot(ddx, dab) * area, quot(ddy, dab) * area);
  a.cij[e] = make_double2(mid.x - (c1.x + c0.x) * 0.5, mid.y - (c1.y + c0.y) * 0.5);
}

// Per cell: VoronoiMesh.cpp:410-413 GetWidth; the CSR neighbour words; the
// state-independent half of calc_naive_slope (LinearGaussImproved.cpp:67-126:
// matrix, determinant check, inverse, 0.5*r_ij) or of GetBoundarySlope (:401-417).
__global__ void __launch_bounds__(kBlock) k_geom_cells(GeomArgs a) {
  chain_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const MeshDev& m = a.mesh;
  if (t >= m.n || mesh_rejected(m)) return;
  const int i = a.cell_order ? a.cell_order[t] : t;
  a.width[i] = root(quot(m.volume[i], kPi));
  const int b = m.cell_off[i], nn = m.cell_off[i + 1] - b;
  // k_cell_order has set the boundary-slope flag (a face between a point and
  // its own mirror image); one pass over the faces writes the neighbour words
  // and the flag's half of the slope
  if (a.cflags[i] & kCellBoundarySlope) {
    const double2 cci = m.cms[i];
    double sxsy = 0, sy2 = 0, sx2 = 0;
    for (int k = 0; k < nn; ++k) {
      const int e = m.cell_faces[b + k];
      const int2 fc = m.face_cells[e];
      const bool first = fc.x == i;
      a.dmf[b + k] = dm_screen((first ? a.dm0 : a.dm1)[e]);
      const int other = first ? fc.y : fc.x;
      const bool mirror = orig_of(m, fc.x) == orig_of(m, fc.y);
      a.nbr[b + k] = static_cast<uint32_t>(other) | (mirror ? kNbrMirror : 0u) | (first ? kNbrFirst : 0u);
      const double2 co = m.cms[other];
      const double dx = co.x - cci.x, dy = co.y - cci.y;
      a.hr[b + k] = make_double2(dx, dy);
      sxsy += dy * dx;
      sx2 += dx * dx;
      sy2 += dy * dy;
    }
    a.minv[i] = make_dbl4(sxsy, sx2, sy2, sxsy * sxsy - sx2 * sy2);
    return;
  }
  if (nn > kMaxNaiveNeighbours) {
    record_error(a.status, 0, RG_ERR_TOO_MANY_NEIGHBORS, 2, i, nn);
    a.minv[i] = make_dbl4(0, 0, 0, 0);
    for (int k = 0; k < nn; ++k) {
      const int e = m.cell_faces[b + k];
      const int2 fc = m.face_cells[e];
      const bool first = fc.x == i;
      a.nbr[b + k] = static_cast<uint32_t>(first ? fc.y : fc.x) | (first ? kNbrFirst : 0u);
      a.dmf[b + k] = dm_screen((first ? a.dm0 : a.dm1)[e]);
    }
    return;
  }
  // no neighbour of this cell is a mirror image of it
  double m0 = 0, m1 = 0, m2 = 0, m3 = 0;
  for (int k = 0; k < nn; ++k) {
    const int e = m.cell_faces[b + k];
    const int2 fc = m.face_cells[e];
    const bool first = fc.x == i;
    a.nbr[b + k] = static_cast<uint32_t>(first ? fc.y : fc.x) | (first ? kNbrFirst : 0u);
    a.dmf[b + k] = dm_screen((first ? a.dm0 : a.dm1)[e]);
    const double2 r = a.rij[e], c = a.cij[e];
    // -r_ij for the second cell: a sign flip of the bit pattern
    const uint64_t flip = first ? 0u : 0x8000000000000000ull;
    const double rx = conv_double_bits(conv_dbits(r.x) ^ flip), ry = conv_double_bits(conv_dbits(r.y) ^ flip);
    m0 -= c.x * rx;
    m1 -= c.y * rx;
    m2 -= c.x * ry;
    m3 -= c.y * ry;
    a.hr[b + k] = make_double2(rx * 0.5, ry * 0.5);
  }
  const double vol = m.volume[i];
  m0 += vol;
  m3 += vol;
  const double det = m0 * m3 - m1 * m2;
  if (fabs(det) < 1e-10 * vol * vol) record_error(a.status, 0, RG_ERR_SINGULAR_MATRIX, 2, i, det);
  const double di = quot(1.0, det);
  a.minv[i] = make_dbl4(m3 * di, -m1 * di, -m2 * di, m0 * di);
}

// Per ghost: which cell it copies and, for rigid walls, the unit normal of
// RigidWallGenerator.cpp:5-15 (ghost minus real point, divided by its length).
__global__ void __launch_bounds__(kBlock) k_geom_ghosts(GeomArgs a) {
  chain_wait();
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const MeshDev& m = a.mesh;
  if (g >= m.g || mesh_rejected(m)) return;
  const int e = m.ghost_face[g];
  if (a.ghost_kind == RG_GHOST_PERIODIC || e < 0) {
    a.ghost_real[g] = m.ghost_source[g];
    a.ghost_unit[g] = make_double2(0, 0);
    return;
  }
  const int2 fc = m.face_cells[e];
  const bool ghost_first = fc.x >= m.n;
  a.ghost_real[g] = ghost_first ? fc.y : fc.x;
  const double2 x0 = m.points[fc.x], x1 = m.points[fc.y];
  const double2 nr = ghost_first ? make_double2(x0.x - x1.x, x0.y - x1.y)
                                 : make_double2(x1.x - x0.x, x1.y - x0.y);
  const double ab = root(nr.x * nr.x + nr.y * nr.y);
  a.ghost_unit[g] = make_double2(quot(nr.x, ab), quot(nr.y, ab));
}

// Per tile of kOrderTile cells: the order in which the per-cell FP64 kernels
// (device geometry, the per-cell geometry pass, slopes, update) take them, by
// (boundary-slope flag, neighbour count) and then by index.  Their per-cell
// loops run over a cell's neighbours, so a warp whose cells have equal counts
// runs no lane idle; every cell is still computed by one thread from the same
// inputs, so the results do not depend on the order.  The flag is
// LinearGaussImproved's (a face between a point and its own mirror image),
// taken from the topology and stored as the cell's flag for the per-cell
// geometry pass; runs after the index validation.
__global__ void __launch_bounds__(kOrderTile) k_cell_order(MeshDev m, int* order, int* cflags) {
  chain_wait();
  constexpr int kKeys = 128, kWarps = kOrderTile / 32;
  // count[w][k]: cells of warp w with key k, then their offset within key k
  __shared__ int count[kWarps][kKeys];
  __shared__ int start[kKeys];
  if (mesh_rejected(m)) return;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int base = blockIdx.x * kOrderTile, i = base + t, n = m.n;
  for (int j = t; j < kWarps * kKeys; j += kOrderTile) count[j / kKeys][j % kKeys] = 0;
  const bool live = i < n;
  int k = 0;
  if (live) {
    const int b = m.cell_off[i], nn = m.cell_off[i + 1] - b;
    bool mirror = false;
    for (int j = 0; j < nn; ++j) {
      const int2 fc = m.face_cells[m.cell_faces[b + j]];
      mirror |= orig_of(m, fc.x) == orig_of(m, fc.y);
    }
    k = (nn < 0 ? 0 : (nn > 63 ? 63 : nn)) | (mirror ? 64 : 0);
    cflags[i] = mirror ? kCellBoundarySlope : 0;
  }
  __syncthreads();
  // rank within the warp among equal keys (lanes in ascending order)
  const unsigned act = __ballot_sync(0xffffffffu, live);
  int before = 0;
  if (live) {
    const unsigned peers = __match_any_sync(act, k);
    before = __popc(peers & ((1u << lane) - 1u));
    if (lane == __ffs(peers) - 1) count[w][k] = __popc(peers);
  }
  __syncthreads();
  // per key: offsets of the warps (ascending), then the key's total
  if (t < kKeys) {
    int sum = 0;
    for (int ww = 0; ww < kWarps; ++ww) {
      const int c = count[ww][t];
      count[ww][t] = sum;
      sum += c;
    }
    start[t] = sum;
  }
  __syncthreads();
  if (t == 0) {
    int sum = 0;
    for (int kk = 0; kk < kKeys; ++kk) {
      const int c = start[kk];
      start[kk] = sum;
      sum += c;
    }
  }
  __syncthreads();
  if (live) order[base + start[k] + count[w][k] + before] = i;
}

// Index validation of an uploaded mesh, before any kernel indexes with it.
// Every read is bounds-checked against the array sizes; the first bad entry
// (smallest key: faces, then ghosts, then cells) is recorded.  Phase 0 keys:
// index = array position, value = the offending entry.
__global__ void __launch_bounds__(kBlock) k_validate(MeshDev m, DevStatus* st) {
  chain_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int np = m.n + m.g;
  if (t < m.e) {
    const int2 fc = m.face_cells[t];
    if (fc.x < 0 || fc.x >= np || fc.y < 0 || fc.y >= np || fc.x == fc.y || (fc.x >= m.n && fc.y >= m.n))
      record_error(st, 0, RG_ERR_INVALID_ARGUMENT, 0, t, fc.x);
  }
  if (t < m.g) {
    const int src = m.ghost_source[t], gf = m.ghost_face[t];
    bool bad = src < 0 || src >= m.n || gf < -1 || gf >= m.e;
    if (!bad && gf >= 0) {
      const int2 fc = m.face_cells[gf];
      bad = fc.x != m.n + t && fc.y != m.n + t;
    }
    if (bad) record_error(st, 0, RG_ERR_INVALID_ARGUMENT, 0, (1ll << 40) + t, gf);
  }
  if (t < m.n) {
    const int b = m.cell_off[t], e1 = m.cell_off[t + 1];
    bool bad = (t == 0 && b != 0) || b < 0 || e1 < b || e1 > m.m || e1 - b > (1 << 20);
    const int lo = b < 0 ? 0 : b, hi = e1 > m.m ? m.m : e1;
    int prev = -1;
    for (int k = lo; k < hi && !bad; ++k) {
      const int f = m.cell_faces[k];
      if (f < 0 || f >= m.e || f <= prev) {
        bad = true;
      } else {
        const int2 fc = m.face_cells[f];
        bad = fc.x != t && fc.y != t;
      }
      prev = f;
    }
    if (bad) record_error(st, 0, RG_ERR_INVALID_ARGUMENT, 0, (2ll << 40) + t, b);
  }
}

// ---------------------------------------------------------------- per step

// Cell i's SimpleCFL bound (simple_cfl.cpp:28-47) with state c: the bit pattern
// of 1 / max_e((cs + |v - w_e|) / R), which orders as an integer.  fmax over
// faces of (cs + sqrt(q_e)) / R equals (cs + sqrt(max q_e)) / R exactly: sqrt, +
// and / are correctly rounded, hence monotone, so the maximum commutes with
// them.  NaN terms are skipped as fmax skips them.
template <bool kBatch>
static __device__ __noinline__ unsigned long long cfl_bound_bits(const StepArgs& a, int i, Cell c) {
  const MeshDev& m = a.mesh;
  const double cs = root(quot(gamma_at<kBatch>(a, i) * c.p, c.d));
  double q = 0;
  bool any = false;
  const int b = m.cell_off[i], e1 = m.cell_off[i + 1];
  if (a.ev_zero) {
    // every face at rest: each term is vx^2 + vy^2 (v - 0 == v)
    const double qq = c.vx * c.vx + c.vy * c.vy;
    if (e1 > b && !isnan(qq)) {
      q = fmax(q, qq);
      any = true;
    }
  } else {
    for (int k = b; k < e1; ++k) {
      const double2 w = reinterpret_cast<const double2*>(a.ev)[m.cell_faces[k]];
      const double dx = c.vx - w.x, dy = c.vy - w.y;
      const double qq = dx * dx + dy * dy;
      if (!isnan(qq)) {
        q = fmax(q, qq);
        any = true;
      }
    }
  }
  const double res = any ? fmax(0.0, quot(cs + root(q), a.geom.width[i])) : 0.0;
  return static_cast<unsigned long long>(__double_as_longlong(quot(1.0, res)));
}

// FP32 bounds lo <= max_e((cs + |v - w_e|) / R) <= hi of that rate.  The
// truncations to 24 bits leave each difference v - w_e within
// 2^-23 (|v| + |w_e|) and a rounding; cs, the root and the quotient carry a few
// 2^-24 each.  hi is infinite (and lo 0) where an operand is outside the normal
// floats, a value is not finite or the rate is below 1e-30 (a width above 2^126,
// by which the approximate quotient is 0, among them).
template <bool kBatch>
__device__ __forceinline__ void cfl_estimate(const StepArgs& a, int i, const Cell& c, float& lo, float& hi) {
  const MeshDev& m = a.mesh;
  bool ok = true;
  const float d = trunc32(c.d, ok), p = trunc32(c.p, ok), vx = trunc32_any(c.vx, ok), vy = trunc32_any(c.vy, ok);
  const float g = trunc32(gamma_at<kBatch>(a, i), ok), r = trunc32(a.geom.width[i], ok);
  const float cs = sqrtf(__fdividef(g * p, d));
  const int b = m.cell_off[i], e1 = m.cell_off[i + 1];
  float q = 0.0f, w1 = 0.0f;
  if (a.ev_zero) {
    q = fmaf(vx, vx, vy * vy);
  } else {
    for (int k = b; k < e1; ++k) {
      const double2 w = reinterpret_cast<const double2*>(a.ev)[m.cell_faces[k]];
      const float wx = trunc32_any(w.x, ok), wy = trunc32_any(w.y, ok);
      const float dx = vx - wx, dy = vy - wy;
      q = fmaxf(q, fmaf(dx, dx, dy * dy));
      w1 = fmaxf(w1, fabsf(wx) + fabsf(wy));
    }
  }
  const float err = 3e-7f * (fabsf(vx) + fabsf(vy) + w1) + 1e-18f;
  const float v = sqrtf(q);
  lo = __fdividef(0.99999f * cs + fmaxf(0.99999f * v - err, 0.0f), r) * 0.99999f;
  hi = __fdividef(1.00001f * cs + 1.00001f * v + err, r) * 1.00001f;
  if (!(ok && e1 > b && hi > 1e-30f && hi < 1e30f && cs > 1e-15f && r > 0.0f)) {
    lo = 0.0f;
    hi = 3e38f;
  }
}

// The smallest exact bound of the block's cells, on the threads whose cell can
// hold it (the others return +inf): every thread of the block calls this, with
// live = false where it has no cell.  Only a cell whose estimate reaches the
// block's largest lower estimate is formed exactly: its quotients, roots and
// per-face FP64 differences are a third of the update kernel's work.
template <bool kBatch>
__device__ __forceinline__ unsigned long long cfl_block_bits(const StepArgs& a, bool live, int i, const Cell& c) {
  __shared__ unsigned best;
  float lo = 0.0f, hi = -1.0f;
  if (threadIdx.x == 0) best = 0u;
  if (live) cfl_estimate<kBatch>(a, i, c, lo, hi);
  __syncthreads();
  const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(lo));
  if ((threadIdx.x & 31) == 0) atomicMax(&best, top);
  __syncthreads();
  const bool need = live && hi >= __uint_as_float(best);
  __syncthreads();  // best is reused by the next call
  return need ? cfl_bound_bits<kBatch>(a, i, c) : kInfBits;
}

// simple_cfl.cpp:58-71 + lazy_list.hpp:185-191 (min over the cells, times cfl)
template <bool kBatch>
__global__ void __launch_bounds__(kMaxBlock) k_cfl(StepArgs a) {
  chain_wait();
  const MeshDev& m = a.mesh;
  unsigned long long bits = kInfBits;
  // the trip count is uniform across a block (base is per block)
  for (int base = blockIdx.x * blockDim.x; base < m.n; base += gridDim.x * blockDim.x) {
    const int t = base + threadIdx.x;
    if (kBatch) {
      // per-problem minimum; the update kernel turns it into the problem's dt
      const unsigned long long xb = t < m.n ? cfl_bound_bits<kBatch>(a, t, load_cell(a.cells, t)) : kInfBits;
      problem_min(a.dtmin_p, t < m.n ? a.cell_problem[t] : -1, xb);
    } else {
      const bool live = t < m.n;
      const unsigned long long xb = cfl_block_bits<kBatch>(a, live, t, live ? load_cell(a.cells, t) : Cell{1, 1, 0, 0});
      bits = xb < bits ? xb : bits;
    }
  }
  if (kBatch) return;
  grid_min_times(a.status, bits, a.cfl, &a.status->dt, nullptr, a.dt_trace);
}

// LinearGaussImproved.cpp:425-494 calc_slope of one component of one cell:
// lane q of a quad forms component q of {d, p, vx, vy}.  The four components
// share the geometry and the shock decision only, so a warp takes eight cells
// and each lane's chain of dependent operations is a quarter of a cell's; the
// FP64 operations of a lane are the Green-Gauss sums (8 per neighbour), which
// the reference's order of additions fixes, plus the limiter's surviving
// candidates (rg_lgi.cuh).  `quad`: the quad's lanes in the warp (all four run
// with the same cell).  Bound by the FP64 unit (62 % of its issue slots at 512^2).
// Events around the launch in Sedov's first steps, with one thread per cell and
// every candidate in FP64 (5,960 instructions in one chain): 489 us at 512^2, 159
// us at 256^2, 103 us at 96 x 101 cells; now 172, 62 and 25 us.
template <bool kBatch, bool kTrace>
__device__ __forceinline__ void slopes_lane(const StepArgs& a, int i, int q, unsigned quad, SlopeTrace* trace) {
  const MeshDev& m = a.mesh;
  const double c = a.cells[4 * static_cast<size_t>(i) + q];
  const int b = m.cell_off[i], nn = m.cell_off[i + 1] - b;
  const bool boundary = a.geom.cflags[i] & kCellBoundarySlope;
  const HydroComp load{a, q};
  double sx, sy;
  LaneNeighbours nb;
  const bool fits = nn <= kFit;
  if (fits) {
    lane_load(a, b, nn, load, nb);
    lane_slope(a, i, b, nn, boundary, c, nb, sx, sy);
  } else {
    lane_slope_any(a, i, b, nn, boundary, c, load, sx, sy);
  }
  double psi = 1.0, dphi_at = 0.0;
  int code = kTraceNone;
  const double nsx = sx, nsy = sy;
  if (a.slf) {
    // :136-157 is_shock / PressureRatio.  cond1 is
    // (div v)*width < -delta_v*cs: false whenever the left side is >= 0,
    // otherwise screened in FP32 against |left| vs delta_v*cs.
    const double lhs = (quad_value(quad, sx, 2) + quad_value(quad, sy, 3)) * a.geom.width[i];
    const double2 dp = reinterpret_cast<const double2*>(a.cells)[2 * static_cast<size_t>(i)];
    bool shock = false;
    if (lt(lhs, 0.0)) {
      const double gp = gamma_at<kBatch>(a, i) * dp.y;
      bool decided = false;
      if (fp32_safe(lhs) && fp32_safe(gp) && fp32_safe(dp.x)) {
        const float rhs_f = narrow(a.delta_v) * sqrtf(narrow(gp) / narrow(dp.x));
        const float l_f = -narrow(lhs);
        if (l_f > rhs_f * 1.000002f) {
          shock = true;
          decided = true;
        } else if (l_f < rhs_f * 0.999998f) {
          decided = true;
        }
      }
      if (!decided) shock = lhs < (-a.delta_v) * root(quot(gp, dp.x));
    }
    if (!shock && nn == 0) shock = 1.0 < a.delta_p;  // PressureRatio of no neighbours is 1
    if (!shock) {
      // PressureRatio < delta_p  <=>  some neighbour's ratio < delta_p: the
      // quad's lanes take every fourth neighbour each
      bool dp_ok = true;
      const float dp_f = trunc32(a.delta_p, dp_ok), pc_f = trunc32(dp.y, dp_ok);
      for (int k = q; k < nn && !shock; k += 4) {
        const int p = static_cast<int>(a.geom.nbr[b + k] & kNbrIdMask);
        const double np_ = a.cells[4 * static_cast<size_t>(copied_cell(a, p)) + 1];
        const bool lower = lt(np_, dp.y);
        const double num = lower ? np_ : dp.y;
        const double den = lower ? dp.y : np_;
        // num / den against delta_p by a product: three truncations and one
        // rounding are within 4e-7 of it (pressures are positive here: 1e-30
        // keeps the product a normal float)
        bool ok = dp_ok;
        const float np_f = trunc32(np_, ok);
        if (ok && fminf(np_f, pc_f) > 1e-30f && dp_f > 1e-6f) {
          const float nf = fminf(np_f, pc_f), df = fmaxf(np_f, pc_f) * dp_f;
          if (nf < df * 0.999999f) {
            shock = true;
            break;
          }
          if (nf > df * 1.000001f) continue;
        }
        shock = lt(quot(num, den), a.delta_p);
      }
      shock = __any_sync(quad, shock);
    }
    if (a.shock && q == 0) a.shock[i] = shock ? 1 : 0;
    const bool velocity = q >= 2;  // :268-283 the velocities' dead band takes |1e-9*q|
    if (fits)
      lane_limit<kTrace>(a, b, nn, c, sx, sy, shock, velocity, false, nb, load, psi, dphi_at, code);
    else
      lane_limit_any<kTrace>(a, b, nn, c, sx, sy, shock, velocity, false, load, psi, dphi_at, code);
    if (conv_dbits(psi) != kOneBits) {
      sx *= psi;
      sy *= psi;
    }
  }
  double* o = a.slopes + 8 * static_cast<size_t>(i) + q;
  o[0] = sx;
  o[4] = sy;
  if (kTrace) {
    SlopeTrace& tr = trace[i];
    tr.naive[q] = nsx;
    tr.naive[4 + q] = nsy;
    tr.psi[q] = psi;
    tr.dphi[q] = dphi_at;
    tr.code[q] = code;
  }
}

// Four lanes per cell (an item).  The plain build holds 64 registers (two
// resident blocks of kMaxBlock): bound by the FP64 unit's latency and issue, the
// slopes gain from every warp (512^2: 172 us; 179 us in 80 registers, 211 us
// with no cap).  kMinBlocks > 0: builds for blocks of up to kCappedBlock threads
// with kMinBlocks resident per SM (launch-shape variants 2 and 3)
template <bool kBatch, int kMinBlocks = 0, bool kTrace = false>
__global__ void __launch_bounds__(kMinBlocks ? kCappedBlock : kMaxBlock, kMinBlocks ? kMinBlocks : 2)
    k_slopes(StepArgs a, SlopeTrace* trace) {
  chain_wait();
  take_next_dt(a);
  const int* order = a.geom.cell_order;
  const int q = threadIdx.x & 3;
  const unsigned quad = 0xfu << (threadIdx.x & 28);
  for (long long t = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 2; t < a.mesh.n;
       t += (gridDim.x * static_cast<long long>(blockDim.x)) >> 2)
    slopes_lane<kBatch, kTrace>(a, order ? order[t] : static_cast<int>(t), q, quad, trace);
}

// ---------------------------------------------------------------- faces

// simple_flux_calculator.cpp:9-15 convert_to_primitive (ideal_gas.cpp:13-16, 40-44)
__device__ __forceinline__ Prim to_prim(double g, const Cell& c) {
  return Prim{c.d, c.p, c.vx, c.vy, quot(quot(c.p, c.d), g - 1), root(quot(g * c.p, c.d))};
}

// simple_flux_calculator.cpp:130-165 rotate / Hllc / rotate_back
__device__ __forceinline__ bool solve_face(Prim l, Prim r, double velocity, double2 n, double na, double2 p,
                                           double pa, Cons& out, const StepArgs& a, int face) {
  const double lx = quot(l.vx * n.x + l.vy * n.y, na), ly = quot(l.vx * p.x + l.vy * p.y, pa);
  const double rx = quot(r.vx * n.x + r.vy * n.y, na), ry = quot(r.vx * p.x + r.vy * p.y, pa);
  l.vx = lx;
  l.vy = ly;
  r.vx = rx;
  r.vy = ry;
  Cons c;
  if (!hllc(l, r, velocity, c, a.status, a.step, face)) return false;
  out.m = c.m;
  out.mx = quot(n.x * c.mx, na) + quot(p.x * c.my, pa);
  out.my = quot(n.y * c.mx, na) + quot(p.y * c.my, pa);
  out.en = c.en;
  return true;
}

// rotate / LagrangianHLLC / rotate_back (LagrangianFlux, condition_action_sequence_2.cpp:284-290)
__device__ __forceinline__ bool solve_face_lagrangian(Prim l, Prim r, double velocity, bool massflux, double2 n,
                                                      double na, double2 p, double pa, Cons& out, double& energy,
                                                      const StepArgs& a, int face) {
  const double lx = quot(l.vx * n.x + l.vy * n.y, na), ly = quot(l.vx * p.x + l.vy * p.y, pa);
  const double rx = quot(r.vx * n.x + r.vy * n.y, na), ry = quot(r.vx * p.x + r.vy * p.y, pa);
  l.vx = lx;
  l.vy = ly;
  r.vx = rx;
  r.vy = ry;
  Cons c;
  if (!lagrangian_hllc(l, r, velocity, massflux, c, energy, a.status, a.step, face)) return false;
  out.m = c.m;
  out.mx = quot(n.x * c.mx, na) + quot(p.x * c.my, pa);
  out.my = quot(n.y * c.mx, na) + quot(p.y * c.my, pa);
  out.en = c.en;
  return true;
}

// simple_flux_calculator.cpp:130-165 rotate / Hllc / rotate_back between the
// states l and r of face e with velocity w; false where an operand is outside
// the integer forms' range (the face then goes to its *_exact form).
template <bool kBatch>
__device__ __forceinline__ bool solve_face_fast(const StepArgs& a, int e, double g, const Cell& l, const Cell& r,
                                                double2 w, Cons& out) {
  FaceOps o;
  const double2 n = a.geom.nrm[e], p = a.geom.par[e];
  const Divisor dn = o.by(a.geom.nabs[e]), dp = o.by(a.geom.area[e]);
  double speed = 0.0;
  bool moving = false;
  if (!a.ev_zero && !(is_zero(w.x) && is_zero(w.y))) {
    speed = o.div(n.x * w.x + n.y * w.y, dn);
    moving = !is_zero(speed);
  }
  const FaceSide ls{l.d, l.p, o.div(l.vx * n.x + l.vy * n.y, dn)};
  const FaceSide rs{r.d, r.p, o.div(r.vx * n.x + r.vy * n.y, dn)};
  Cons f;
  bool left;
  const Divisor gm1 = kBatch ? o.by(g - 1) : a.gm1;
  o.ok = o.ok && gm1.ok;
  hllc_face(
      o, ls, rs, g, gm1, moving, speed,
      [&](bool lft) {
        const double vx = lft ? l.vx : r.vx, vy = lft ? l.vy : r.vy;
        return o.div(vx * p.x + vy * p.y, dp);
      },
      f, left);
  out.m = f.m;
  out.mx = o.div(o.mul(n.x, f.mx), dn) + o.div(o.mul(p.x, f.my), dp);
  out.my = o.div(o.mul(n.y, f.mx), dn) + o.div(o.mul(p.y, f.my), dp);
  out.en = f.en;
  return o.ok;
}

template <bool kBatch>
__device__ __forceinline__ void write_flux(const StepArgs& a, int e, int real_side, const Cons& c, bool scaled,
                                           double area) {
  if (scaled) {
    const double s = scaled_dt<kBatch>(a, real_side) * area;  // simple_extensive_updater.cpp:26-27
    store4(a.fluxes, e, c.m * s, c.en * s, c.mx * s, c.my * s);
  } else {
    store4(a.fluxes, e, c.m, c.en, c.mx, c.my);
  }
}

// simple_flux_calculator.cpp:17-25 reflect (Reflect, geometry.cpp:117-120);
// keeps the source's energy and sound speed.
__device__ __forceinline__ Prim reflect(Prim q, double2 axis, double aa) {
  const double s = 2 * (q.vx * axis.x + q.vy * axis.y);
  const double pp = aa * aa;
  const double tx = quot(axis.x * s, pp), ty = quot(axis.y * s, pp);
  q.vx = tx - q.vx;
  q.vy = ty - q.vy;
  return q;
}

// The face states of LinearGaussImproved (:570-590 real sides, :596-634 ghost sides).
__device__ __forceinline__ void lgi_states(const StepArgs& a, int e, int2 fc, Cell side[2]) {
  const MeshDev& m = a.mesh;
  const int ids[2] = {fc.x, fc.y};
  const double2 dms[2] = {a.geom.dm0[e], a.geom.dm1[e]};
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int pid = ids[s];
    Cell c = point_state(a, pid);
    int sid = pid;
    bool zero = false;
    if (pid >= m.n) {
      if (a.ghost_kind == RG_GHOST_PERIODIC)
        sid = m.ghost_source[pid - m.n];  // PeriodicGhostGenerator.cpp:19-24
      else
        zero = true;  // RigidWallGenerator.cpp:39-54: zero gradient
    }
    Cell gx{0, 0, 0, 0}, gy{0, 0, 0, 0};
    if (!zero) {
      const double2* sp = reinterpret_cast<const double2*>(a.slopes) + 4 * sid;
      const double2 s0 = sp[0], s1 = sp[1], s2 = sp[2], s3 = sp[3];
      gx = Cell{s0.x, s0.y, s1.x, s1.y};
      gy = Cell{s2.x, s2.y, s3.x, s3.y};
    }
    const MulFactor fx = mul_factor(dms[s].x), fy = mul_factor(dms[s].y);
    c.d += mul_rn(fx, dms[s].x, gx.d);
    c.p += mul_rn(fx, dms[s].x, gx.p);
    c.vx += mul_rn(fx, dms[s].x, gx.vx);
    c.vy += mul_rn(fx, dms[s].x, gx.vy);
    c.d += mul_rn(fy, dms[s].y, gy.d);
    c.p += mul_rn(fy, dms[s].y, gy.p);
    c.vx += mul_rn(fy, dms[s].y, gy.vx);
    c.vy += mul_rn(fy, dms[s].y, gy.vy);
    side[s] = c;
  }
}
__device__ __forceinline__ double2 face_velocity(const StepArgs& a, int e) {
  return a.ev_zero ? make_double2(0.0, 0.0) : reinterpret_cast<const double2*>(a.ev)[e];
}
// The cell states of SimpleFluxCalculator (simple_flux_calculator.cpp:80-126):
// a self-mirror ghost is its neighbour's reflection, any other its source.
__device__ __forceinline__ void pcm_states(const StepArgs& a, int e, int2 fc, Cell side[2]) {
  const MeshDev& m = a.mesh;
  const int oa = orig_of(m, fc.x), ob = orig_of(m, fc.y);
  side[0] = load_cell(a.cells, oa);
  side[1] = load_cell(a.cells, ob);
  if (oa == ob && (fc.x >= m.n || fc.y >= m.n)) {
    // both sides hold the real cell's state
    const Prim q = reflect(Prim{side[0].d, side[0].p, side[0].vx, side[0].vy, 0.0, 0.0}, a.geom.par[e], a.geom.area[e]);
    if (fc.x < m.n) {
      side[1].vx = q.vx;
      side[1].vy = q.vy;
    } else {
      side[0].vx = q.vx;
      side[0].vy = q.vy;
    }
  }
}

// Face e by hllc() itself: operands outside solve_face_fast's range, and its
// failures (recorded here).
template <bool kScaled, bool kBatch, bool kLgi>
static __device__ __noinline__ void face_exact(const StepArgs& a, int e) {
  const int2 fc = a.mesh.face_cells[e];
  Cell side[2];
  if (kLgi)
    lgi_states(a, e, fc, side);
  else
    pcm_states(a, e, fc, side);
  const double2 w = face_velocity(a, e);
  const double2 n = a.geom.nrm[e], p = a.geom.par[e];
  const double na = a.geom.nabs[e], pa = a.geom.area[e];
  // a face at rest has speed +-0 (the sign only reaches signs of zeros)
  const double speed = (w.x == 0.0 && w.y == 0.0) ? 0.0 : quot(n.x * w.x + n.y * w.y, na);
  const int real_side = fc.x < a.mesh.n ? fc.x : fc.y;
  const double g = gamma_at<kBatch>(a, real_side);
  Cons c;
  if (!solve_face(to_prim(g, side[0]), to_prim(g, side[1]), speed, n, na, p, pa, c, a, e)) return;
  if (a.mflux) a.mflux[e] = c.m;
  write_flux<kBatch>(a, e, real_side, c, kScaled, a.geom.xarea[e]);
}

// ModularFluxCalculator (modular_flux_calculator.cpp:39-71, kLgi) or
// SimpleFluxCalculator (simple_flux_calculator.cpp:216-244) for one face.
template <bool kScaled, bool kBatch, bool kLgi>
__device__ __forceinline__ void k_faces_item(const StepArgs& a, int e) {
  const int2 fc = a.mesh.face_cells[e];
  Cell side[2];
  if (kLgi)
    lgi_states(a, e, fc, side);
  else
    pcm_states(a, e, fc, side);
  const int real_side = fc.x < a.mesh.n ? fc.x : fc.y;
  Cons c;
  if (!solve_face_fast<kBatch>(a, e, gamma_at<kBatch>(a, real_side), side[0], side[1], face_velocity(a, e), c)) {
    face_exact<kScaled, kBatch, kLgi>(a, e);
    return;
  }
  if (a.mflux) a.mflux[e] = c.m;
  write_flux<kBatch>(a, e, real_side, c, kScaled, a.geom.xarea[e]);
}

// One thread per face.  Bound by the FP64 unit (85 FP64 instructions per warp,
// the integer pipes a third busy beside it) and by its 4,500 instructions of
// code: blocks of 512 run it in step and miss the instruction cache less.  64
// registers (two such blocks per SM) spill 300 bytes and still gain.  512^2
// (786,430 faces, RoundCells face velocities) 205 -> 141 us, 256^2 66 -> 45 us.
template <bool kScaled, bool kBatch, bool kLgi>
__global__ void __launch_bounds__(kMaxBlock, 2) k_faces(StepArgs a) {
  chain_wait();
  if (!kLgi) take_next_dt(a);
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < a.mesh.e; e += gridDim.x * blockDim.x)
    k_faces_item<kScaled, kBatch, kLgi>(a, e);
}

// ---------------------------------------------------------------- condition/action fluxes

// geometry.cpp normalize: v/abs(v)
__device__ __forceinline__ double2 normalize2(double x, double y) {
  const double ab = root(x * x + y * y);
  return make_double2(quot(x, ab), quot(y, ab));
}
// simple_flux_calculator.cpp:27-31 remove_parallel_component, then normalize
__device__ __forceinline__ double2 wall_normal(double wx, double wy, double2 p) {
  const double s = wx * p.x + wy * p.y, pp = p.x * p.x + p.y * p.y;
  return normalize2(wx - quot(p.x * s, pp), wy - quot(p.y * s, pp));
}
__device__ __forceinline__ bool has_sticker(const StepArgs& a, int p, int bit) {
  return a.stickers != nullptr && ((a.stickers[orig_of(a.mesh, p)] >> bit) & 1u) != 0;
}

// One face of ConditionActionSequence (condition_action_sequence.cpp:17-61)
// or ConditionActionSequence2 (condition_action_sequence_2.cpp:40-127): the
// first rule of sequence 0, else of sequence 1, whose condition holds picks
// the action; cell states are the cells' own records (a periodic ghost reads
// its source cell), face states LinearGaussImproved's (order 2).
template <bool kScaled>
__device__ __forceinline__ void k_faces_cas_item(const StepArgs& a, int e) {
  const MeshDev& m = a.mesh;
  const int2 fc = m.face_cells[e];
  int chosen = -1;
  bool aux = false;
  for (int pass = 0; pass < 2 && chosen < 0; ++pass) {
    for (int k = 0; k < a.n_rules && chosen < 0; ++k) {
      if (a.rules[k][0] != pass) continue;
      const int cond = a.rules[k][1];
      bool applies = false, ax = false;
      if (cond == RG_COND_BOUNDARY_EDGE) {  // :228-253, serial build
        if (fc.x >= m.n) applies = true;
        else if (fc.y >= m.n) applies = ax = true;
      } else if (cond == RG_COND_BULK_EDGE) {  // :255-271
        applies = (fc.x < m.n && fc.y < m.n) || orig_of(m, fc.x) != orig_of(m, fc.y);
      } else {  // :273-289 RegularSpecialEdge: exactly one side carries the sticker
        const bool sa = has_sticker(a, fc.x, a.rules[k][2]), sb = has_sticker(a, fc.y, a.rules[k][2]);
        applies = sa ? !sb : sb;
        ax = !sa && sb;
      }
      if (applies) {
        chosen = k;
        aux = ax;
      }
    }
  }
  if (a.tr_side) a.tr_side[e] = 0;  // no tracer flux unless an action sets one
  if (chosen < 0) {  // "Error in ConditionActionSequence"
    record_error(a.status, a.step, RG_ERR_INVALID_ARGUMENT, 3, e, 0.0);
    return;
  }
  if (a.lag_ws) {
    // LagrangianFlux::Reset: faces of other actions carry no ws / speed
    a.lag_ws[e] = 0.0;
    a.lag_ev[e] = 0.0;
  }
  const dbl4 v = m.face_vertices[e];
  const double2 p = normalize2(v.z - v.x, v.w - v.y);
  const double pa = root(p.x * p.x + p.y * p.y);
  const double g = a.gamma;
  const Cell c0 = load_cell(a.cells, orig_of(m, fc.x)), c1 = load_cell(a.cells, orig_of(m, fc.y));
  int action = a.rules[chosen][3];
  if (action == RG_ACT_RATCHET) {
    // condition_action_sequence_2.cpp:232-249
    const double2 x0 = m.points[fc.x], x1 = m.points[fc.y];
    const double nx = aux ? x1.x - x0.x : x0.x - x1.x, ny = aux ? x1.y - x0.y : x0.y - x1.y;
    const Cell& sc = aux ? c0 : c1;
    const double sign = 2.0 * (a.rules[chosen][4] != 0 ? 1.0 : 0.0) - 1.0;
    action = (nx * sc.vx + ny * sc.vy) * sign < 0 ? RG_ACT_FREE_FLOW : RG_ACT_RIGID_WALL2;
  }
  // LinearGaussImproved face states (order 2), as lgi_states forms them
  Cell s0 = c0, s1 = c1;
  if (action == RG_ACT_REGULAR2 || action == RG_ACT_RIGID_WALL2 || action == RG_ACT_LAGRANGIAN) {
    const int ids[2] = {fc.x, fc.y};
    const double2 dms[2] = {a.geom.dm0[e], a.geom.dm1[e]};
    Cell side[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int pid = ids[s];
      Cell c = point_state(a, pid);
      int sid = pid;
      bool zero = false;
      if (pid >= m.n) {
        if (a.ghost_kind == RG_GHOST_PERIODIC)
          sid = m.ghost_source[pid - m.n];
        else
          zero = true;
      }
      Cell gx{0, 0, 0, 0}, gy{0, 0, 0, 0};
      if (!zero) {
        const double2* sp = reinterpret_cast<const double2*>(a.slopes) + 4 * sid;
        const double2 q0 = sp[0], q1 = sp[1], q2 = sp[2], q3 = sp[3];
        gx = Cell{q0.x, q0.y, q1.x, q1.y};
        gy = Cell{q2.x, q2.y, q3.x, q3.y};
      }
      addmult(c, gx, dms[s].x);
      addmult(c, gy, dms[s].y);
      side[s] = c;
    }
    s0 = side[0];
    s1 = side[1];
  }
  if (action == RG_ACT_LAGRANGIAN) {
    // condition_action_sequence_2.cpp:270-294: ModularFluxCalculator's frame
    // and face speed, WallsMassFlux (:300-312) picking rs or rs2
    const double2 w = a.ev_zero ? make_double2(0.0, 0.0) : reinterpret_cast<const double2*>(a.ev)[e];
    const double2 nn = a.geom.nrm[e], pp = a.geom.par[e];
    const double na = a.geom.nabs[e], ppa = a.geom.area[e];
    const double speed = (w.x == 0.0 && w.y == 0.0) ? 0.0 : quot(nn.x * w.x + nn.y * w.y, na);
    const bool lag = orig_of(m, fc.x) != orig_of(m, fc.y);
    const bool mf = (((lag ? a.rules[chosen][5] : a.rules[chosen][5] >> 1)) & 1) != 0;
    Cons c;
    double energy = 0.0;
    if (!solve_face_lagrangian(to_prim(g, s0), to_prim(g, s1), speed, mf, nn, na, pp, ppa, c, energy, a, e)) return;
    if (a.lag_ws) {
      a.lag_ws[e] = lag ? energy : 0.0;
      a.lag_ev[e] = speed;
    }
    // convert_conserved_to_extensive (:29-40): Mass * the face value upwind
    if (a.tr_side) {
      a.mflux[e] = c.m;
      a.tr_side[e] = kTrSideFace | (c.m > 0 ? kTrSideFirst : kTrSideSecond);
    }
    write_flux<false>(a, e, fc.x < m.n ? fc.x : fc.y, c, kScaled, a.geom.xarea[e]);
    return;
  }
  Prim l, r;
  double2 n;
  double vel = 0;
  if (action == RG_ACT_REGULAR || action == RG_ACT_REGULAR2) {
    // condition_action_sequence.cpp:84-110, condition_action_sequence_2.cpp:129-157
    const double2 x0 = m.points[fc.x], x1 = m.points[fc.y];
    n = normalize2(x1.x - x0.x, x1.y - x0.y);
    const double2 w = a.ev_zero ? make_double2(0.0, 0.0) : reinterpret_cast<const double2*>(a.ev)[e];
    vel = n.x * w.x + n.y * w.y;
    l = to_prim(g, action == RG_ACT_REGULAR ? c0 : s0);
    r = to_prim(g, action == RG_ACT_REGULAR ? c1 : s1);
  } else {
    // RigidWallFlux / RigidWallFlux2 / FreeFlowFlux: the wall frame
    const double2 x0 = m.points[fc.x], x1 = m.points[fc.y];
    n = aux ? wall_normal(v.x - x0.x, v.y - x0.y, p) : wall_normal(x1.x - v.x, x1.y - v.y, p);
    if (action == RG_ACT_FREE_FLOW) {
      l = r = to_prim(g, aux ? c0 : c1);
    } else {
      const Prim q = to_prim(g, action == RG_ACT_RIGID_WALL ? (aux ? c0 : c1) : (aux ? s0 : s1));
      if (aux) {
        l = q;
        r = reflect(q, p, pa);
      } else {
        r = q;
        l = reflect(q, p, pa);
      }
    }
  }
  const double na = root(n.x * n.x + n.y * n.y);
  Cons c;
  if (!solve_face(l, r, vel, n, na, p, pa, c, a, e)) return;
  if (a.tr_side) {
    // the tracer flux is Mass times the tracers of: the upwind cell
    // (RegularFlux, condition_action_sequence.cpp:110-114) or face value
    // (RegularFlux2, condition_action_sequence_2.cpp:156), the cell on the
    // aux side (RigidWallFlux, FreeFlowFlux: :178, :221) or its face value
    // (RigidWallFlux2, condition_action_sequence_2.cpp:221)
    a.mflux[e] = c.m;
    const bool regular = action == RG_ACT_REGULAR || action == RG_ACT_REGULAR2;
    const bool face = action == RG_ACT_REGULAR2 || action == RG_ACT_RIGID_WALL2;
    const bool first = regular ? c.m > 0 : aux;
    a.tr_side[e] = (face ? kTrSideFace : 0) | (first ? kTrSideFirst : kTrSideSecond);
  }
  const int real_side = fc.x < m.n ? fc.x : fc.y;
  write_flux<false>(a, e, real_side, c, kScaled, a.geom.xarea[e]);
}

template <bool kScaled>
__global__ void __launch_bounds__(kMaxBlock) k_faces_cas(StepArgs a) {
  chain_wait();
  if (a.order == 1) take_next_dt(a);
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < a.mesh.e; e += gridDim.x * blockDim.x)
    k_faces_cas_item<kScaled>(a, e);
}

// ---------------------------------------------------------------- cells

// What one launch of the update kernel does
constexpr int kUpFused = 0;     // extensives from the scaled fluxes, then the cells
constexpr int kUpAverage = 1;   // the same, the extensives averaged with ext_avg (Heun)
constexpr int kUpUnscaled = 2;  // extensives only, from unscaled fluxes
constexpr int kUpScaled = 3;    // extensives only, from scaled fluxes
constexpr int kUpCells = 4;     // cells only

// SimpleExtensiveUpdater (simple_extensive_updater.cpp:11-35) as a gather:
// each cell applies its faces' contributions in ascending face order, which
// is the order the reference's edge loop applies them to that cell; then
// SimpleCellUpdater::regular_update (simple_cell_updater.cpp:22-59).  Returns
// whether c holds the cell's new state.  kMode is a compile-time constant: the
// FP64 instructions of a mode that is off would still take the FP64 unit where
// the compiler predicates them, and so would a choice between + and -.
template <bool kBatch, int kMode>
__device__ __forceinline__ bool update_cell(const StepArgs& a, int i, Cell& c) {
  const MeshDev& m = a.mesh;
  double2* ext2 = reinterpret_cast<double2*>(a.ext);
  double2 e01 = ext2[2 * i], e23 = ext2[2 * i + 1];
  double mass = e01.x, en = e01.y, px = e23.x, py = e23.y;
  if (kMode != kUpCells) {
    const double dt = kMode == kUpUnscaled ? step_dt(a) : 0.0;
    const int b = m.cell_off[i], e1 = m.cell_off[i + 1];
    for (int k = b; k < e1; ++k) {
      const int e = m.cell_faces[k];
      const double2* f = reinterpret_cast<const double2*>(a.fluxes) + 2 * e;
      const double2 f01 = f[0], f23 = f[1];
      double dm = f01.x, de = f01.y, dx = f23.x, dy = f23.y;
      if (kMode == kUpUnscaled) {
        const double s = dt * a.geom.xarea[e];
        dm *= s;
        de *= s;
        dx *= s;
        dy *= s;
      }
      const uint32_t flip = a.geom.nbr[k] & kNbrFirst;  // bit 31
      mass += flip_sign(dm, flip);
      en += flip_sign(de, flip);
      px += flip_sign(dx, flip);
      py += flip_sign(dy, flip);
    }
    if (a.lag_update) {
      const double f = lag_factor(a, i);
      mass *= f;
      en *= f;
      px *= f;
      py *= f;
    }
    if (kMode == kUpAverage) {
      // hdsim2d.cpp:311-320 average_extensive: 0.5*(mid + old)
      const double2* o = reinterpret_cast<const double2*>(a.ext_avg);
      const double2 o01 = o[2 * i], o23 = o[2 * i + 1];
      mass = 0.5 * (mass + o01.x);
      en = 0.5 * (en + o01.y);
      px = 0.5 * (px + o23.x);
      py = 0.5 * (py + o23.y);
    }
    double2* out2 = reinterpret_cast<double2*>(a.ext_out ? a.ext_out : a.ext);
    out2[2 * i] = make_double2(mass, en);
    out2[2 * i + 1] = make_double2(px, py);
    if (kMode == kUpUnscaled || kMode == kUpScaled) return false;
  }
  if (a.frozen_mask && (a.stickers[i] & a.frozen_mask)) {
    // simple_cell_updater.cpp:61-83 with (HasSticker, SkipUpdate): the old
    // cell stays (its extensives above still took the fluxes)
    c = load_cell(a.cells, i);
    if (a.cells_out) store4(a.cells_out, i, c.d, c.p, c.vx, c.vy);
    return true;
  }
  const double d = quot(mass, m.cd_volume[i]);
  if (lt(d, 0.0)) {
    record_error(a.status, a.step, RG_ERR_NEGATIVE_DENSITY, 5, i, d);
    return false;
  }
  // four quotients by the mass share its preparation
  const Divisor dm = divisor(mass, RcpSeedDevice{});
  double vx, vy, em;
  bool ok = div_by(px, dm, &vx);
  ok = div_by(py, dm, &vy) && ok;
  ok = div_by(en, dm, &em) && ok;
  if (!ok) {
    vx = quot(px, mass);
    vy = quot(py, mass);
    em = quot(en, mass);
  }
  const double energy = em - 0.5 * (vx * vx + vy * vy);
  if (lt(energy, 0.0)) {
    record_error(a.status, a.step, RG_ERR_NEGATIVE_ENERGY, 5, i, energy);
    return false;
  }
  c = Cell{d, (gamma_at<kBatch>(a, i) - 1) * energy * d, vx, vy};
  store4(a.cells_out ? a.cells_out : a.cells, i, c.d, c.p, c.vx, c.vy);
  return true;
}

// Bound by the FP64 unit and its gathers.  512^2 with face velocities, with the
// next dt: 76 -> 44 us (256^2: 15 -> 10 us).  The modes as template arguments,
// signs flipped instead of + / - chosen and the CFL bound estimated took a
// warp's FP64 instructions from 128 to about 40.
template <bool kBatch, int kMode>
__global__ void __launch_bounds__(kMaxBlock) k_update(StepArgs a) {
  chain_wait();
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  if (kBatch && kMode <= kUpAverage && !a.batch_keep_dt) {
    for (int p = t0; p < a.n_problems; p += stride) {
      // every face of this step has read its problem's minimum: record the dt,
      // advance the problem's time and reset the minimum for the next step
      const double dt = a.cfl * __longlong_as_double(static_cast<long long>(a.dtmin_p[p]));
      a.dt_p[p] = dt;
      a.time_p[p] += dt;
      a.dtmin_p[p] = kInfBits;
      if (p == 0) {  // what the step's call returns, and the run's record
        a.status->dt = dt;
        if (a.dt_trace) *a.dt_trace = dt;
      }
    }
  }
  unsigned long long bits = kInfBits;
  const int* order = a.geom.cell_order;
  // the next step's SimpleCFL minimum, from the states just stored
  const bool next = !kBatch && kMode <= kUpAverage && a.cfl_next;
  for (int base = blockIdx.x * blockDim.x; base < a.mesh.n; base += stride) {
    const int t = base + threadIdx.x;
    Cell c{1, 1, 0, 0};
    bool live = false;
    int i = 0;
    if (t < a.mesh.n) {
      i = order ? order[t] : t;
      live = update_cell<kBatch, kMode>(a, i, c);
      if (next && !live) {
        // a rejected cell keeps its record, which a CFL pass reads
        c = load_cell(a.cells, i);
        live = true;
      }
    }
    if (next) {
      const unsigned long long b = cfl_block_bits<kBatch>(a, live, i, c);
      bits = b < bits ? b : bits;
    }
  }
  if (next) grid_min_times(a.status, bits, a.cfl, &a.status->dt_next);
}

// hdsim2d.cpp:41-67 init_extensives
template <bool kBatch>
__global__ void __launch_bounds__(kBlock) k_init_ext(StepArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.mesh.n) return;
  const Cell c = load_cell(a.cells, i);
  const double mass = a.mesh.cd_volume[i] * c.d;
  store4(a.ext, i, mass, quot(quot(c.p, c.d), gamma_at<kBatch>(a, i) - 1) * mass + 0.5 * mass * (c.vx * c.vx + c.vy * c.vy),
         c.vx * mass, c.vy * mass);
}

// The error part of `count` status blocks, emptied: one launch (about 1 us
// in a chain of kernels), where the two memsets of a block took 5 us.
__global__ void k_reset_status(DevStatus* st, int count) {
  chain_wait();
  if (static_cast<int>(threadIdx.x) < count) {
    st[threadIdx.x].err_key = ~0ull;
    st[threadIdx.x].err_status = 0;
    st[threadIdx.x].lock = 0;
  }
}

// *flag = 1 if any of v[0..n) is not +-0 (NaN counts as nonzero)
__global__ void __launch_bounds__(kBlock) k_any_nonzero(const double* v, long long n, int* flag) {
  bool any = false;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    any = any || !(v[i] == 0.0);
  if (__any_sync(0xffffffffu, any) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

inline int blocks(int n) { return (n + kBlock - 1) / kBlock; }

}  // namespace

// Problem of every point of a batch (real cells by the offset table, ghosts by
// their source cell) and the check that no face joins two problems.
__global__ void __launch_bounds__(kBlock) k_problems(MeshDev m, const int* offsets, int P, int* cell_problem,
                                                     DevStatus* st) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < m.n) {
    int lo = 0, hi = P;  // largest p with offsets[p] <= t
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (offsets[mid] <= t) lo = mid; else hi = mid;
    }
    cell_problem[t] = lo;
  }
  __syncthreads();
  if (t < m.g) {
    const int src = m.ghost_source[t];
    int lo = 0, hi = P;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (offsets[mid] <= src) lo = mid; else hi = mid;
    }
    cell_problem[m.n + t] = lo;
  }
}

__global__ void __launch_bounds__(kBlock) k_check_problems(MeshDev m, const int* cell_problem, DevStatus* st) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < m.e) {
    const int2 fc = m.face_cells[t];
    if (cell_problem[fc.x] != cell_problem[fc.y]) record_error(st, 0, RG_ERR_INVALID_ARGUMENT, 0, t, fc.y);
  }
}

cudaError_t launch_problems(const MeshDev& m, const int* offsets, int P, int* cell_problem, DevStatus* st,
                            cudaStream_t s) {
  const int work = m.n > m.g ? m.n : m.g;
  k_problems<<<blocks(work > 0 ? work : 1), kBlock, 0, s>>>(m, offsets, P, cell_problem, st);
  if (m.e > 0) k_check_problems<<<blocks(m.e), kBlock, 0, s>>>(m, cell_problem, st);
  return cudaGetLastError();
}

cudaError_t launch_any_nonzero(const double* v, long long n, int* flag, cudaStream_t s) {
  if (n > 0) {
    const long long nb = (n + kBlock - 1) / kBlock;
    k_any_nonzero<<<static_cast<int>(nb < 4096 ? nb : 4096), kBlock, 0, s>>>(v, n, flag);
  }
  return cudaGetLastError();
}

cudaError_t launch_reset_status(DevStatus* st, int count, cudaStream_t s) {
  chain(s, 1, 32, k_reset_status, st, count);
  return cudaGetLastError();
}

cudaError_t launch_validate(const MeshDev& m, DevStatus* st, cudaStream_t s) {
  int work = m.e > m.n ? m.e : m.n;
  work = work > m.g ? work : m.g;
  chain(s, blocks(work > 0 ? work : 1), kBlock, k_validate, m, st);
  return cudaGetLastError();
}

cudaError_t launch_cell_order(const MeshDev& m, int* order, int* cflags, cudaStream_t s) {
  if (m.n > 0) chain(s, (m.n + kOrderTile - 1) / kOrderTile, kOrderTile, k_cell_order, m, order, cflags);
  return cudaGetLastError();
}

cudaError_t launch_geometry(const GeomArgs& a, cudaStream_t s) {
  if (a.mesh.e > 0) chain(s, blocks(a.mesh.e), kBlock, k_geom_faces, a);
  if (a.mesh.n > 0) chain(s, blocks(a.mesh.n), kBlock, k_geom_cells, a);
  if (a.mesh.g > 0) chain(s, blocks(a.mesh.g), kBlock, k_geom_ghosts, a);
  return cudaGetLastError();
}

cudaError_t launch_geom_ghosts(const GeomArgs& a, cudaStream_t s) {
  if (a.mesh.g > 0) chain(s, blocks(a.mesh.g), kBlock, k_geom_ghosts, a);
  return cudaGetLastError();
}

cudaError_t launch_cfl(const StepArgs& a, cudaStream_t s) {
  const LaunchShape sh = fit_shape(a.shapes.cfl, a.mesh.n);
  const int nb = grid_of(sh, a.mesh.n);
  a.cell_problem ? chain(s, nb, sh.block, k_cfl<true>, a) : chain(s, nb, sh.block, k_cfl<false>, a);
  return cudaGetLastError();
}

cudaError_t launch_slopes(const StepArgs& a, cudaStream_t s) {
  if (a.mesh.n > 0) {
    const LaunchShape sh = fit_shape(a.shapes.slopes, 4LL * a.mesh.n);
    const int nb = grid_of(sh, 4LL * a.mesh.n), bs = sh.block;
    const bool b = a.cell_problem != nullptr;
    // builds: 0 plain, 2 and 3 register-capped for 3 and 4 resident blocks of
    // up to 256 threads
    switch (sh.variant) {
      case 2: b ? chain(s, nb, bs, k_slopes<true, 3>, a, nullptr) : chain(s, nb, bs, k_slopes<false, 3>, a, nullptr); break;
      case 3: b ? chain(s, nb, bs, k_slopes<true, 4>, a, nullptr) : chain(s, nb, bs, k_slopes<false, 4>, a, nullptr); break;
      default: b ? chain(s, nb, bs, k_slopes<true>, a, nullptr) : chain(s, nb, bs, k_slopes<false>, a, nullptr);
    }
  }
  return cudaGetLastError();
}

cudaError_t launch_slopes_trace(const StepArgs& a, SlopeTrace* trace, cudaStream_t s) {
  // (held to 4 resident blocks of 256, as the plain build: 256^2 50.7 -> 42.9 us,
  // 43.5 for 3, 50.4 for 2, blocks of 128 in 8 47.6)
  if (a.mesh.n > 0)
    chain(s, grid_of(kDefaultShape, 4LL * a.mesh.n), kDefaultShape.block, k_slopes<false, 4, true>, a, trace);
  return cudaGetLastError();
}

cudaError_t launch_faces(const StepArgs& a, cudaStream_t s, bool scaled) {
  if (a.mesh.e == 0 && !a.take_next_dt) return cudaSuccess;
  const LaunchShape sh = fit_shape(a.shapes.faces, a.mesh.e);
  const int nb = grid_of(sh, a.mesh.e), bs = sh.block;
  const bool b = a.cell_problem != nullptr;
  if (a.n_rules > 0) {
    scaled ? chain(s, nb, bs, k_faces_cas<true>, a) : chain(s, nb, bs, k_faces_cas<false>, a);
    return cudaGetLastError();
  }
  if (a.order == 1) {
    if (scaled)
      b ? chain(s, nb, bs, k_faces<true, true, false>, a) : chain(s, nb, bs, k_faces<true, false, false>, a);
    else
      b ? chain(s, nb, bs, k_faces<false, true, false>, a) : chain(s, nb, bs, k_faces<false, false, false>, a);
  } else {
    if (scaled)
      b ? chain(s, nb, bs, k_faces<true, true, true>, a) : chain(s, nb, bs, k_faces<true, false, true>, a);
    else
      b ? chain(s, nb, bs, k_faces<false, true, true>, a) : chain(s, nb, bs, k_faces<false, false, true>, a);
  }
  return cudaGetLastError();
}

cudaError_t launch_update(const StepArgs& a, cudaStream_t s, bool from_unscaled, bool extensive, bool cells) {
  const int work = a.cell_problem && a.n_problems > a.mesh.n ? a.n_problems : a.mesh.n;
  if (work > 0) {
    const LaunchShape sh = fit_shape(a.shapes.update, work);
    const int nb = grid_of(sh, work), bs = sh.block;
    const bool b = a.cell_problem != nullptr;
    if (extensive && cells) {
      // (the fused update reads scaled fluxes)
      if (a.ext_avg)
        b ? chain(s, nb, bs, k_update<true, kUpAverage>, a) : chain(s, nb, bs, k_update<false, kUpAverage>, a);
      else
        b ? chain(s, nb, bs, k_update<true, kUpFused>, a) : chain(s, nb, bs, k_update<false, kUpFused>, a);
    } else if (extensive && from_unscaled) {
      b ? chain(s, nb, bs, k_update<true, kUpUnscaled>, a) : chain(s, nb, bs, k_update<false, kUpUnscaled>, a);
    } else if (extensive) {
      b ? chain(s, nb, bs, k_update<true, kUpScaled>, a) : chain(s, nb, bs, k_update<false, kUpScaled>, a);
    } else {
      b ? chain(s, nb, bs, k_update<true, kUpCells>, a) : chain(s, nb, bs, k_update<false, kUpCells>, a);
    }
  }
  return cudaGetLastError();
}

cudaError_t launch_init_extensives(const StepArgs& a, cudaStream_t s) {
  if (a.mesh.n > 0) {
    if (a.cell_problem)
      k_init_ext<true><<<blocks(a.mesh.n), kBlock, 0, s>>>(a);
    else
      k_init_ext<false><<<blocks(a.mesh.n), kBlock, 0, s>>>(a);
  }
  return cudaGetLastError();
}

}  // namespace rg
