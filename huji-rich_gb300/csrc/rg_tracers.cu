// rg_tracers.cu -- tracer passes of the FP64 path (ComputationalCell::tracers,
// Extensive::tracers), compiled with --fmad=false like rg_fp64.cu.
//
// Every ComputationalCell / Extensive operation of the reference applies to
// each tracer exactly as to a hydro field (computational_cell_2d.cpp:20-110,
// extensive.cpp), with the same geometric scalars, so each tracer pass runs
// after its hydro pass and reads what that pass decided:
//   k_tr_slopes   per cell: LinearGaussImproved slope of every tracer
//                 (:67-134 / :401-422), zero outside calc_tracers (:470-479),
//                 the limiter chosen by the hydro shock test (:481-492)
//   k_tr_faces_*  per face: mass flux (kept by the hydro face kernel) times
//                 the upwind side's tracer (modular_flux_calculator.cpp:24-35,
//                 simple_flux_calculator.cpp:193-213)
//   k_tr_update   per cell: ascending-face gather of the tracer fluxes
//                 (simple_extensive_updater.cpp:11-35), then tracer =
//                 extensive / mass and the "Entropy" tracer
//                 (simple_cell_updater.cpp:22-59), or the old tracers of a
//                 SkipUpdate cell
// Tracers are cell-major (cell i's tracer j at i*nt + j).  k_tr_update is
// instantiated for each tracer count NT (1..kMaxTracers) so its loops over
// tracers have exact compile-time bounds: the per-cell arrays stay in
// registers and no FP64 work is spent on absent tracers.
#include <math.h>

#include "rg_launch.cuh"
#include "rg_lgi.cuh"

namespace rg {
namespace {

constexpr int kTrBlock = 256;


// LinearGaussImproved.cpp:425-494 calc_slope, tracer part: one thread per
// tracer of a cell (the hydro slopes' lanes, rg_lgi.cuh), cells in the
// per-tile neighbour-count order.  Tracers share only the geometry and the
// shock decision, which the hydro pass kept.
__global__ void __launch_bounds__(kTrBlock) k_tr_slopes(StepArgs a, TracerArgs t) {
  chain_wait();
  const long long id = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  const MeshDev& m = a.mesh;
  const int nt = t.nt;
  const int at = static_cast<int>(id / nt), j = static_cast<int>(id % nt);
  if (at >= m.n) return;
  const int i = a.geom.cell_order ? a.geom.cell_order[at] : at;
  double* o = t.tr_slopes + static_cast<size_t>(i) * 2 * nt + j;
  if (!((t.limited >> j) & 1u)) {
    // :470-479 tracers outside calc_tracers get zero slopes
    o[0] = 0.0;
    o[nt] = 0.0;
    return;
  }
  const TracerComp load{a, t.tr, nt, j};
  const double c = load.at(i);
  const int b = m.cell_off[i], nn = m.cell_off[i + 1] - b;
  const bool boundary = a.geom.cflags[i] & kCellBoundarySlope;
  const bool fits = nn <= kFit;
  LaneNeighbours nb;
  double sx, sy;
  if (fits) {
    lane_load(a, b, nn, load, nb);
    lane_slope(a, i, b, nn, boundary, c, nb, sx, sy);
  } else {
    lane_slope_any(a, i, b, nn, boundary, c, load, sx, sy);
  }
  if (a.slf) {
    // both limiters take |1e-9*t| (:268-283, :367-385)
    const bool shock = a.shock[i] != 0;
    double psi, dphi_at;
    int code;
    if (fits)
      lane_limit<false>(a, b, nn, c, sx, sy, shock, true, true, nb, load, psi, dphi_at, code);
    else
      lane_limit_any<false>(a, b, nn, c, sx, sy, shock, true, true, load, psi, dphi_at, code);
    sx *= psi;
    sy *= psi;
  }
  o[0] = sx;
  o[nt] = sy;
}

// dt*area of face e (simple_extensive_updater.cpp:26-27); in a batch the dt
// of the problem of the face's real side, as the hydro face kernel scales it
__device__ __forceinline__ double tr_scale(const StepArgs& a, int e) {
  if (a.cell_problem) {
    const int2 fc = a.mesh.face_cells[e];
    return scaled_dt<true>(a, fc.x < a.mesh.n ? fc.x : fc.y) * a.geom.xarea[e];
  }
  return scaled_dt<false>(a, 0) * a.geom.xarea[e];
}

// ModularFluxCalculator tracer fluxes: Mass * (Mass > 0 ? first : second)
// side's LinearGaussImproved value (:570-590 real sides; :596-634 ghost sides:
// the copied cell's tracers plus the periodic source's gradient, or a zero
// gradient at rigid walls, RigidWallGenerator.cpp:39-54).
template <bool kScaled>
__global__ void __launch_bounds__(kTrBlock) k_tr_faces_lgi(StepArgs a, TracerArgs t) {
  chain_wait();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const MeshDev& m = a.mesh;
  if (e >= m.e) return;
  const int nt = t.nt;
  const int2 fc = m.face_cells[e];
  const double mass = a.mflux[e];
  const bool first = mass > 0;
  const int pid = first ? fc.x : fc.y;
  const double2 dm = first ? a.geom.dm0[e] : a.geom.dm1[e];
  const int src = copied_cell(a, pid);
  const bool zero_grad = pid >= m.n && a.ghost_kind != RG_GHOST_PERIODIC;
  const double* q = t.tr + static_cast<size_t>(src) * nt;
  const double* g = t.tr_slopes + static_cast<size_t>(src) * 2 * nt;
  const double s = kScaled ? tr_scale(a, e) : 1.0;
  double* o = t.tr_flux + static_cast<size_t>(e) * nt;
  for (int j = 0; j < nt; ++j) {
    double v = q[j];
    v += (zero_grad ? 0.0 : g[j]) * dm.x;
    v += (zero_grad ? 0.0 : g[nt + j]) * dm.y;
    const double f = mass * v;
    o[j] = kScaled ? f * s : f;
  }
}

// The condition/action fluxes' tracer part: Mass times the tracers of the
// side the face's action chose (a.tr_side): that neighbour's own cell (a
// ghost's cell, as the hydro state), or its LinearGaussImproved face value as
// k_tr_faces_lgi forms it.  Faces with no action carry none.
template <bool kScaled>
__global__ void __launch_bounds__(kTrBlock) k_tr_faces_cas(StepArgs a, TracerArgs t) {
  chain_wait();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const MeshDev& m = a.mesh;
  if (e >= m.e) return;
  const int nt = t.nt;
  const unsigned char side = a.tr_side[e];
  double* o = t.tr_flux + static_cast<size_t>(e) * nt;
  if (!(side & (kTrSideFirst | kTrSideSecond))) {
    for (int j = 0; j < nt; ++j) o[j] = 0.0;
    return;
  }
  const int2 fc = m.face_cells[e];
  const double mass = a.mflux[e];
  const bool first = (side & kTrSideFirst) != 0;
  const int pid = first ? fc.x : fc.y;
  const double s = kScaled ? tr_scale(a, e) : 1.0;
  if (side & kTrSideFace) {
    const double2 dm = (first ? a.geom.dm0 : a.geom.dm1)[e];
    const int src = copied_cell(a, pid);
    const bool zero_grad = pid >= m.n && a.ghost_kind != RG_GHOST_PERIODIC;
    const double* q = t.tr + static_cast<size_t>(src) * nt;
    const double* g = t.tr_slopes + static_cast<size_t>(src) * 2 * nt;
    for (int j = 0; j < nt; ++j) {
      double v = q[j];
      v += (zero_grad ? 0.0 : g[j]) * dm.x;
      v += (zero_grad ? 0.0 : g[nt + j]) * dm.y;
      const double f = mass * v;
      o[j] = kScaled ? f * s : f;
    }
  } else {
    const double* q = t.tr + static_cast<size_t>(orig_of(m, pid)) * nt;
    for (int j = 0; j < nt; ++j) {
      const double f = mass * q[j];
      o[j] = kScaled ? f * s : f;
    }
  }
}

// SimpleFluxCalculator calc_tracer_flux (simple_flux_calculator.cpp:193-213):
// Mass * the upwind point's tracer, 0 when that point is a self-mirror ghost
// or Mass is 0; a periodic ghost reads its source cell, as the hydro state does.
template <bool kScaled>
__global__ void __launch_bounds__(kTrBlock) k_tr_faces_pcm(StepArgs a, TracerArgs t) {
  chain_wait();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const MeshDev& m = a.mesh;
  if (e >= m.e) return;
  const int nt = t.nt;
  const int2 fc = m.face_cells[e];
  const double mass = a.mflux[e];
  const bool mirror = orig_of(m, fc.x) == orig_of(m, fc.y);
  int up = -1;
  if (mass > 0 && (fc.x < m.n || !mirror))
    up = fc.x;
  else if (mass < 0 && (fc.y < m.n || !mirror))
    up = fc.y;
  const double s = kScaled ? tr_scale(a, e) : 1.0;
  double* o = t.tr_flux + static_cast<size_t>(e) * nt;
  for (int j = 0; j < nt; ++j) {
    const double f = up >= 0 ? mass * t.tr[static_cast<size_t>(orig_of(m, up)) * nt + j] : 0.0;
    o[j] = kScaled ? f * s : f;
  }
}

// SimpleExtensiveUpdater for the extensive tracers (gather in ascending face
// order) and SimpleCellUpdater's tracer part; runs after the hydro update,
// whose new mass, density and pressure it reads.
// kUnscaled, kAverage: template arguments, since the FP64 products of a form
// that is off still take the FP64 unit where the compiler predicates them.
template <int NT, bool kUnscaled, bool kAverage>
__global__ void __launch_bounds__(kTrBlock) k_tr_update(StepArgs a, TracerArgs t, int do_ext, int do_cells) {
  chain_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const MeshDev& m = a.mesh;
  if (i >= m.n) return;
  constexpr int nt = NT;
  constexpr int kMaxTracers = NT;
  double te[kMaxTracers];
  double* ext_t = t.tr_ext + static_cast<size_t>(i) * nt;
#pragma unroll
  for (int j = 0; j < kMaxTracers; ++j) te[j] = j < nt ? ext_t[j] : 0.0;
  if (do_ext) {
    const double dt = kUnscaled ? step_dt(a) : 0.0;
    for (int k = m.cell_off[i]; k < m.cell_off[i + 1]; ++k) {
      const int e = m.cell_faces[k];
      const uint32_t flip = a.geom.nbr[k] & kNbrFirst;  // bit 31
      const double s = kUnscaled ? dt * a.geom.xarea[e] : 1.0;
      const double* f = t.tr_flux + static_cast<size_t>(e) * nt;
#pragma unroll
      for (int j = 0; j < kMaxTracers; ++j) {
        if (j < nt) {
          te[j] += flip_sign(kUnscaled ? f[j] * s : f[j], flip);
        }
      }
    }
    if (a.lag_update) {
      // LagrangianExtensiveUpdater scales every extensive of the cell
      const double f = lag_factor(a, i);
#pragma unroll
      for (int j = 0; j < kMaxTracers; ++j)
        if (j < nt) te[j] *= f;
    }
  }
  if (kAverage) {
    // hdsim2d.cpp:311-320 average_extensive: 0.5*(mid + old)
    const double* o = t.tr_ext_avg + static_cast<size_t>(i) * nt;
#pragma unroll
    for (int j = 0; j < kMaxTracers; ++j)
      if (j < nt) te[j] = 0.5 * (te[j] + o[j]);
  }
  const bool frozen = a.frozen_mask && (a.stickers[i] & a.frozen_mask);
  if (do_cells && frozen && t.tr_out) {
    // SkipUpdate keeps the step's old cell, its tracers included
#pragma unroll
    for (int j = 0; j < kMaxTracers; ++j)
      if (j < nt) t.tr_out[static_cast<size_t>(i) * nt + j] = t.tr[static_cast<size_t>(i) * nt + j];
  }
  if (do_cells && !frozen) {
    const double mass = (a.ext_out ? a.ext_out : a.ext)[4 * i];
    double* tr = (t.tr_out ? t.tr_out : t.tr) + static_cast<size_t>(i) * nt;
#pragma unroll
    for (int j = 0; j < kMaxTracers; ++j)
      if (j < nt) tr[j] = quot(te[j], mass);
    if (t.entropy >= 0) {
      // ideal_gas.cpp:52-55 dp2s of the updated cell
      const Cell c = load_cell(a.cells_out ? a.cells_out : a.cells, i);
      const double sv = c.p * pow(c.d, -(a.cell_problem ? a.gamma_p[a.cell_problem[i]] : a.gamma));
      tr[t.entropy] = sv;
#pragma unroll
      for (int j = 0; j < kMaxTracers; ++j)
        if (j == t.entropy) te[j] = sv * mass;
    }
  }
  if (do_ext || (do_cells && t.entropy >= 0) || t.tr_ext_out) {
    double* out = t.tr_ext_out ? t.tr_ext_out + static_cast<size_t>(i) * nt : ext_t;
#pragma unroll
    for (int j = 0; j < kMaxTracers; ++j)
      if (j < nt) out[j] = te[j];
  }
}

// hdsim2d.cpp:56-63 init_extensives: tracer * mass, mass = volume * density
__global__ void __launch_bounds__(kTrBlock) k_tr_init(StepArgs a, TracerArgs t) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.mesh.n) return;
  const double mass = a.mesh.cd_volume[i] * load_cell(a.cells, i).d;
  for (int j = 0; j < t.nt; ++j)
    t.tr_ext[static_cast<size_t>(i) * t.nt + j] = t.tr[static_cast<size_t>(i) * t.nt + j] * mass;
}

inline int tr_blocks(int n) { return (n + kTrBlock - 1) / kTrBlock; }

}  // namespace

// k_tr_update for NT = t.nt
#define RG_TR_CASE(NT, U, A, grid, s, ...) \
  case NT: chain(s, grid, kTrBlock, k_tr_update<NT, U, A>, __VA_ARGS__); break;
#define RG_TR_DISPATCH(U, A, grid, s, ...)  \
  switch (t.nt) {                           \
    RG_TR_CASE(1, U, A, grid, s, __VA_ARGS__) \
    RG_TR_CASE(2, U, A, grid, s, __VA_ARGS__) \
    RG_TR_CASE(3, U, A, grid, s, __VA_ARGS__) \
    RG_TR_CASE(4, U, A, grid, s, __VA_ARGS__) \
    RG_TR_CASE(5, U, A, grid, s, __VA_ARGS__) \
    RG_TR_CASE(6, U, A, grid, s, __VA_ARGS__) \
    RG_TR_CASE(7, U, A, grid, s, __VA_ARGS__) \
    RG_TR_CASE(8, U, A, grid, s, __VA_ARGS__) \
    default: break;                         \
  }

cudaError_t launch_tr_slopes(const StepArgs& a, const TracerArgs& t, cudaStream_t s) {
  if (a.mesh.n > 0 && t.nt > 0 && t.nt <= kMaxTracers) {
    const long long lanes = static_cast<long long>(a.mesh.n) * t.nt;
    chain(s, static_cast<unsigned>((lanes + kTrBlock - 1) / kTrBlock), kTrBlock, k_tr_slopes, a, t);
  }
  return cudaGetLastError();
}

cudaError_t launch_tr_faces(const StepArgs& a, const TracerArgs& t, cudaStream_t s, bool scaled) {
  if (a.mesh.e == 0 || t.nt == 0) return cudaSuccess;
  const int nb = tr_blocks(a.mesh.e);
  if (a.n_rules > 0)
    scaled ? chain(s, nb, kTrBlock, k_tr_faces_cas<true>, a, t) : chain(s, nb, kTrBlock, k_tr_faces_cas<false>, a, t);
  else if (a.order == 1)
    scaled ? chain(s, nb, kTrBlock, k_tr_faces_pcm<true>, a, t) : chain(s, nb, kTrBlock, k_tr_faces_pcm<false>, a, t);
  else
    scaled ? chain(s, nb, kTrBlock, k_tr_faces_lgi<true>, a, t) : chain(s, nb, kTrBlock, k_tr_faces_lgi<false>, a, t);
  return cudaGetLastError();
}

cudaError_t launch_tr_update(const StepArgs& a, const TracerArgs& t, cudaStream_t s, bool from_unscaled,
                             bool extensive, bool cells) {
  if (a.mesh.n > 0 && t.nt > 0 && t.nt <= kMaxTracers) {
    const int ex = extensive ? 1 : 0, ce = cells ? 1 : 0;
    // (only the fused Heun step, whose fluxes are scaled, averages)
    if (t.tr_ext_avg) {
      RG_TR_DISPATCH(false, true, tr_blocks(a.mesh.n), s, a, t, ex, ce)
    } else if (from_unscaled) {
      RG_TR_DISPATCH(true, false, tr_blocks(a.mesh.n), s, a, t, ex, ce)
    } else {
      RG_TR_DISPATCH(false, false, tr_blocks(a.mesh.n), s, a, t, ex, ce)
    }
  }
  return cudaGetLastError();
}

cudaError_t launch_tr_init(const StepArgs& a, const TracerArgs& t, cudaStream_t s) {
  if (a.mesh.n > 0 && t.nt > 0) k_tr_init<<<tr_blocks(a.mesh.n), kTrBlock, 0, s>>>(a, t);
  return cudaGetLastError();
}

}  // namespace rg
