// rg_3d.cu -- FP64 kernels of the 3D first-order path (HDSim3D on a fixed
// mesh), compiled without FMA contraction: every operation rounds as the
// reference's does, in its evaluation order.
//
//   k3_cfl     per cell width/(|v| + c), grid minimum, times cfl
//              (CourantFriedrichsLewy.cpp:23-46)
//   k3_faces   per face FirstOrderHydroFlux (FirstOrderHydroFlux.cpp:42-114):
//              rigid wall against the reflected state on boundary faces, Hllc
//              on (v.n, |v - (v.n)n|) in the bulk, momentum rebuilt along the
//              normal and the donor's tangential direction; optionally times
//              dt*area (hdsim_3d.cpp:63-76)
//   k3_update  per cell: the face deltas in ascending face order (the order
//              update_extensive applies them to the cell), then
//              extensive/volume and DefaultCellUpdater
//              (default_cell_updater.cpp:5-14, ideal_gas.cpp:18-23)
//   k3_init    ExtensiveGenerator (extensive_generator.cpp:3-28)
#include <math.h>

#include "rg_launch.cuh"
#include "rg_3d.cuh"
#include "rg_face.cuh"
#include "rg_hllc.cuh"
#include "rg_trunc.cuh"

namespace rg {
namespace {

constexpr int kBlock = 256;

struct V3 {
  double x, y, z;
};
// Vector3D.cpp: abs, ScalarProd, d*v (v.x*d), v/d, -, +
__device__ __forceinline__ double vabs(V3 v) { return root(v.x * v.x + v.y * v.y + v.z * v.z); }
__device__ __forceinline__ double vdot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 vscale(double d, V3 v) { return V3{v.x * d, v.y * d, v.z * d}; }
__device__ __forceinline__ V3 vdiv(V3 v, double d) { return V3{quot(v.x, d), quot(v.y, d), quot(v.z, d)}; }
__device__ __forceinline__ V3 vsub(V3 a, V3 b) { return V3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 vadd(V3 a, V3 b) { return V3{a.x + b.x, a.y + b.y, a.z + b.z}; }

struct Cell3 {
  double d, p;
  V3 v;
};
__device__ __forceinline__ Cell3 load_cell3(const double* c, int i) {
  const double2* r = reinterpret_cast<const double2*>(c) + 3 * i;
  const double2 a = r[0], b = r[1], cz = r[2];
  return Cell3{a.x, a.y, V3{b.x, b.y, cz.x}};
}
__device__ __forceinline__ void store6(double* out, int i, double a, double b, double c, double d, double e) {
  double2* r = reinterpret_cast<double2*>(out) + 3 * i;
  r[0] = make_double2(a, b);
  r[1] = make_double2(c, d);
  r[2] = make_double2(e, 0.0);
}

__device__ __forceinline__ double dp2e(double g, double d, double p) { return quot(quot(p, d), g - 1); }
__device__ __forceinline__ double dp2c(double g, double d, double p) { return root(quot(g * p, d)); }

// FirstOrderHydroFlux.cpp:32-40 calc_primitive: (d, p, (v.n, |v - (v.n)n|), e, c)
__device__ __forceinline__ Prim prim3(double g, const Cell3& c, V3 n) {
  const double sp = vdot(c.v, n);
  return Prim{c.d, c.p, sp, vabs(vsub(c.v, vscale(sp, n))), dp2e(g, c.d, c.p), dp2c(g, c.d, c.p)};
}

// FirstOrderHydroFlux.cpp:16-30 GetParallel
__device__ __forceinline__ V3 parallel3(V3 vel, V3 n) {
  V3 par = vsub(vel, vscale(vdot(vel, n), n));
  const double p = vabs(par);
  const double v = vabs(vel);
  if (1e-9 > fabs(v - 0)) return par;
  return p < 1e-8 * v ? vdiv(par, v) : vdiv(par, p);
}

// Vector3D.cpp:203-206 Reflect: v - 2*ScalarProd(v,n)*n/pow(abs(n),2)
__device__ __forceinline__ V3 reflect3(V3 v, V3 n) {
  const double s = 2 * vdot(v, n);
  const double a = vabs(n);
  return vsub(v, vdiv(vscale(s, n), a * a));
}

// ---------------------------------------------------------------- mesh checks

// Every index of a packed 3D mesh, before any other kernel uses it.
__global__ void __launch_bounds__(kBlock) k3_validate(Mesh3Dev m, DevStatus* st) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < m.e) {
    const int2 fc = m.face_cells[t];
    if (fc.x < -1 || fc.x >= m.n || fc.y < -1 || fc.y >= m.n || (fc.x < 0 && fc.y < 0))
      record_error(st, 0, RG_ERR_INVALID_ARGUMENT, 0, t, fc.x < -1 || fc.x >= m.n ? fc.x : fc.y);
  }
  if (t < m.n) {
    const int b = m.cell_off[t], e1 = m.cell_off[t + 1];
    if (b < 0 || e1 < b || e1 > m.m)
      record_error(st, 0, RG_ERR_INVALID_ARGUMENT, 2, t, e1);
    else
      for (int k = b; k < e1; ++k) {
        const int f = m.cell_faces[k];
        if (f < 0 || f >= m.e) {
          record_error(st, 0, RG_ERR_INVALID_ARGUMENT, 2, t, f);
          break;
        }
        const int2 fc = m.face_cells[f];
        if (fc.x != t && fc.y != t) {
          record_error(st, 0, RG_ERR_INVALID_ARGUMENT, 2, t, f);
          break;
        }
      }
  }
}

// Unit normals (FirstOrderHydroFlux.cpp:11-14 normalize) and the CSR signs.
// axis: the axis a unit normal lies along (0-2, +4 in its negative direction), 3: none.
__global__ void __launch_bounds__(kBlock) k3_geometry(Mesh3Dev m, dbl4* nhat, int* fsign, unsigned char* axis) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < m.e) {
    const V3 n{m.normal[3 * t], m.normal[3 * t + 1], m.normal[3 * t + 2]};
    const V3 u = vdiv(n, vabs(n));
    nhat[t] = make_dbl4(u.x, u.y, u.z, 0.0);
    int ax = 3;
    if (u.y == 0.0 && u.z == 0.0 && (u.x == 1.0 || u.x == -1.0)) ax = u.x < 0 ? 4 : 0;
    if (u.x == 0.0 && u.z == 0.0 && (u.y == 1.0 || u.y == -1.0)) ax = u.y < 0 ? 5 : 1;
    if (u.x == 0.0 && u.y == 0.0 && (u.z == 1.0 || u.z == -1.0)) ax = u.z < 0 ? 6 : 2;
    axis[t] = static_cast<unsigned char>(ax);
  }
  if (t < m.n)
    for (int k = m.cell_off[t]; k < m.cell_off[t + 1]; ++k) {
      const int f = m.cell_faces[k];
      fsign[k] = f | (m.face_cells[f].x == t ? static_cast<int>(0x80000000u) : 0);
    }
}

// ---------------------------------------------------------------- step

// Cell i's CFL bound width/(|v| + c) (CourantFriedrichsLewy.cpp:23-46), as its
// bit pattern (which orders as an integer)
static __device__ __noinline__ unsigned long long cfl3_bound_bits(const Step3Args& a, int i, Cell3 c) {
  const double b = quot(a.mesh.width[i], vabs(c.v) + dp2c(a.gamma, c.d, c.p));
  return static_cast<unsigned long long>(__double_as_longlong(b));
}
// The smallest bound of the block's cells, formed on the threads whose cell can
// hold it (the others return +inf): an FP32 estimate of the rate (|v| + c)/width,
// good to 1e-5, rules the rest out.  Operands outside the normal floats are
// formed, and rates below 1e-30 (widths above 2^126, by which the approximate
// quotient is 0, among them).  Every thread of the block calls this.
__device__ __forceinline__ unsigned long long cfl3_block_bits(const Step3Args& a, bool live, int i, const Cell3& c) {
  __shared__ unsigned best;
  if (threadIdx.x == 0) best = 0u;
  float lo = 0.0f, hi = -1.0f;
  if (live) {
    bool ok = true;
    const float x = trunc32_any(c.v.x, ok), y = trunc32_any(c.v.y, ok), z = trunc32_any(c.v.z, ok);
    const float cs = sqrtf(__fdividef(trunc32(a.gamma, ok) * trunc32(c.p, ok), trunc32(c.d, ok)));
    const float w = trunc32(a.mesh.width[i], ok);
    const float r = __fdividef(sqrtf(fmaf(x, x, fmaf(y, y, z * z))) + cs, w);
    lo = r * 0.9999f;
    hi = r * 1.0001f;
    if (!(ok && hi > 1e-30f && hi < 1e30f && cs > 1e-15f && w > 0.0f)) {
      lo = 0.0f;
      hi = 3e38f;
    }
  }
  __syncthreads();
  const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(lo));
  if ((threadIdx.x & 31) == 0) atomicMax(&best, top);
  __syncthreads();
  return live && hi >= __uint_as_float(best) ? cfl3_bound_bits(a, i, c) : kInfBits;
}

__global__ void __launch_bounds__(kBlock) k3_cfl(Step3Args a) {
  chain_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < a.mesh.n;
  const unsigned long long bits = cfl3_block_bits(a, live, i, live ? load_cell3(a.cells, i) : Cell3{1, 1, V3{0, 0, 0}});
  grid_min_times(a.status, bits, a.cfl, &a.status->dt, nullptr, a.dt_trace);
}

template <bool kScaled>
__device__ __forceinline__ void store_flux3(const Step3Args& a, int f, double m, double x, double y, double z,
                                            double en) {
  if (kScaled) {
    const double s = (a.take_next_dt ? a.status->dt_next : (a.dt_from_device ? a.status->dt : a.dt_host)) * a.mesh.area[f];
    store6(a.fluxes, f, s * m, s * x, s * y, s * z, s * en);
  } else {
    store6(a.fluxes, f, m, x, y, z, en);
  }
}

// Face f in the reference's own operations: walls, normals that no axis
// carries, and operands outside face3_axis's range or failures.
template <bool kScaled>
static __device__ __noinline__ void face3_exact(const Step3Args& a, int f) {
  const int2 fc = a.mesh.face_cells[f];
  const dbl4 nn = a.nhat[f];
  const V3 n{nn.x, nn.y, nn.z};
  Cons sol;
  V3 par;
  if (fc.x < 0 || fc.y < 0) {
    // CalcRigidWall: the real cell against its reflection
    const bool real_first = fc.x >= 0;
    const Cell3 real = load_cell3(a.cells, real_first ? fc.x : fc.y);
    const Prim preal = prim3(a.gamma, real, n);
    par = parallel3(real.v, n);
    Cell3 other = real;
    other.v = reflect3(real.v, n);
    const Prim pghost = prim3(a.gamma, other, n);
    const bool ok = real_first ? hllc(preal, pghost, 0.0, sol, a.status, a.step, f)
                               : hllc(pghost, preal, 0.0, sol, a.status, a.step, f);
    if (!ok) return;
  } else {
    // CalcSingleFluxInBulk
    double fv = 0.0;
    if (a.fvel) fv = vdot(V3{a.fvel[3 * f], a.fvel[3 * f + 1], a.fvel[3 * f + 2]}, n);
    const Cell3 ca = load_cell3(a.cells, fc.x), cb = load_cell3(a.cells, fc.y);
    if (!hllc(prim3(a.gamma, ca, n), prim3(a.gamma, cb, n), fv, sol, a.status, a.step, f)) return;
    par = parallel3(sol.m > 0 ? ca.v : cb.v, n);
  }
  // Conserved3D(sol.Mass, sol.Momentum.x*normal + sol.Momentum.y*parallel, sol.Energy)
  const V3 mom = vadd(vscale(sol.mx, n), vscale(sol.my, par));
  store_flux3<kScaled>(a, f, sol.m, mom.x, mom.y, mom.z, sol.en);
}

// A bulk face whose unit normal is an axis, +-1 times (CubeGrid's every face,
// axis: 0 x, 1 y, 2 z): v.n is that component, v - (v.n)n the other two, and the
// products with the normal's zeros drop out, which leaves 55 of the general
// form's 125 FP64 operations and the same bits (finite operands; up to the sign
// of zeros).  The tangential speed is formed for the upwind side only.
template <bool kScaled>
__device__ __forceinline__ bool face3_axis(const Step3Args& a, int f, int2 fc, int axis, uint32_t flip) {
  FaceOps o;
  const Cell3 ca = load_cell3(a.cells, fc.x), cb = load_cell3(a.cells, fc.y);
  // normal and tangential components (in x, y, z order)
  const bool ax = axis == 0, az = axis == 2;
  const double an = flip_sign(ax ? ca.v.x : (az ? ca.v.z : ca.v.y), flip), bn = flip_sign(ax ? cb.v.x : (az ? cb.v.z : cb.v.y), flip);
  const double a1 = ax ? ca.v.y : ca.v.x, a2 = az ? ca.v.y : ca.v.z;
  const double b1 = ax ? cb.v.y : cb.v.x, b2 = az ? cb.v.y : cb.v.z;
  double fv = 0.0;
  if (a.fvel) {
    const dbl4 nn = a.nhat[f];
    fv = vdot(V3{a.fvel[3 * f], a.fvel[3 * f + 1], a.fvel[3 * f + 2]}, V3{nn.x, nn.y, nn.z});
  }
  auto speed = [&](bool first) {
    const double x = first ? a1 : b1, y = first ? a2 : b2;
    return o.sqrt(o.mul(x, x) + o.mul(y, y));
  };
  Cons sol;
  bool left;
  double vt = 0.0;
  o.ok = a.gm1.ok;
  hllc_face(
      o, FaceSide{ca.d, ca.p, an}, FaceSide{cb.d, cb.p, bn}, a.gamma, a.gm1, !is_zero(fv), fv,
      [&](bool l) { return vt = speed(l); }, sol, left);
  uint32_t top = max(max(mag_hi(a1), mag_hi(a2)), max(mag_hi(b1), mag_hi(b2)));
  top = max(max(top, max(mag_hi(sol.mx), mag_hi(sol.my))), mag_hi(sol.m));
  if (!o.ok || top >= 0x7ff00000u) return false;
  // GetParallel (FirstOrderHydroFlux.cpp:16-30) of the donor
  const bool first = !sign_bit(sol.m) && !is_zero(sol.m);  // sol.m > 0
  if (first != left) {
    vt = speed(first);
    if (!o.ok) return false;
  }
  double p1 = first ? a1 : b1, p2 = first ? a2 : b2;
  if (is_zero(vt)) {
    if (!(is_zero(p1) && is_zero(p2))) return false;  // squares that underflow
  } else {
    bool ok = true;
    const float tf = trunc32(vt, ok), nf = trunc32_any(first ? an : bn, ok);
    const float v = sqrtf(fmaf(tf, tf, nf * nf));
    double den = vt;
    // |v| against 1e-9 and the tangential speed against 1e-8 |v|
    if (!(ok && tf > 1e-15f && v > 1.00001e-9f && v < 1e15f && tf > 1.00001e-8f * v)) {
      const V3 vel = first ? ca.v : cb.v;
      const double vv = vabs(vel);
      if (1e-9 > vv)
        den = 0.0;  // not divided
      else if (vt < 1e-8 * vv)
        den = vv;
    }
    if (!is_zero(den)) {
      const Divisor D = o.by(den);
      p1 = o.div(p1, D);
      p2 = o.div(p2, D);
      if (!o.ok) return false;
    }
  }
  const double mn = flip_sign(sol.mx, flip), m1 = o.mul(sol.my, p1), m2 = o.mul(sol.my, p2);
  store_flux3<kScaled>(a, f, sol.m, ax ? mn : m1, ax ? m1 : (az ? m2 : mn), az ? mn : m2, sol.en);
  return true;
}

// One thread per face, 64 registers.  96^3 (2.68 M faces), events around the
// launch: 871 -> 360 us with CubeGrid's normals, and 872 -> 836 us with the grid
// turned so that none lies on an axis and every face takes face3_exact.
template <bool kScaled>
__global__ void __launch_bounds__(kBlock, 4) k3_faces(Step3Args a) {
  chain_wait();
  if (a.take_next_dt && blockIdx.x == 0 && threadIdx.x == 0) {
    const double dt = a.status->dt_next;
    a.status->dt = dt;
    if (a.dt_trace) *a.dt_trace = dt;
  }
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= a.mesh.e) return;
  const int2 fc = a.mesh.face_cells[f];
  const int axis = a.axis[f];  // 0-2, +4: the negative direction; 3: none
  if ((axis & 3) != 3 && fc.x >= 0 && fc.y >= 0 &&
      face3_axis<kScaled>(a, f, fc, axis & 3, (axis & 4) ? 0x80000000u : 0u))
    return;
  face3_exact<kScaled>(a, f);
}

// kExt / kUnscaled / kCells: template arguments, since FP64 instructions of a
// form that is off still take the FP64 unit where the compiler predicates them
template <bool kUnscaled, bool kExt, bool kCells>
__device__ __forceinline__ bool update_cell3(const Step3Args& a, int i, Cell3& c) {
  const Mesh3Dev& m = a.mesh;
  const double2* e2 = reinterpret_cast<const double2*>(a.ext) + 3 * i;
  const double2 e01 = e2[0], e23 = e2[1], e45 = e2[2];
  double u[5] = {e01.x, e01.y, e23.x, e23.y, e45.x};
  if (kExt) {
    const double dt = kUnscaled ? (a.dt_from_device ? a.status->dt : a.dt_host) : 0.0;
    for (int k = m.cell_off[i]; k < m.cell_off[i + 1]; ++k) {
      const int fs = a.fsign[k];
      const int f = fs & 0x7fffffff;
      const double2* fl = reinterpret_cast<const double2*>(a.fluxes) + 3 * f;
      const double2 f01 = fl[0], f23 = fl[1], f45 = fl[2];
      double d[5] = {f01.x, f01.y, f23.x, f23.y, f45.x};
      if (kUnscaled) {
        const double s = dt * m.area[f];  // dt*GetArea()*flux (hdsim_3d.cpp:69)
#pragma unroll
        for (int q = 0; q < 5; ++q) d[q] = s * d[q];
      }
#pragma unroll
      for (int q = 0; q < 5; ++q) u[q] += flip_sign(d[q], static_cast<uint32_t>(fs) & 0x80000000u);
    }
    store6(a.ext, i, u[0], u[1], u[2], u[3], u[4]);
  }
  if (kCells) {
    // nine quotients by two divisors
    const Divisor dv = divisor(m.volume[i], RcpSeedDevice{});
    bool ok = true;
    auto by = [&ok](double x, const Divisor& D) {
      double q;
      ok = div_by(x, D, &q) && ok;
      return q;
    };
    double density = by(u[0], dv);
    const Divisor dd = divisor(density, RcpSeedDevice{});
    V3 vel{by(by(u[1], dv), dd), by(by(u[2], dv), dd), by(by(u[3], dv), dd)};
    double ev = by(u[4], dv);
    if (!ok) {
      const double V = m.volume[i];
      density = quot(u[0], V);
      vel = vdiv(V3{quot(u[1], V), quot(u[2], V), quot(u[3], V)}, density);
      ev = quot(u[4], V);
    }
    const double thermal = ev - 0.5 * density * vdot(vel, vel);
    double eint;
    if (!ok || !div_by(thermal, dd, &eint)) eint = quot(thermal, density);
    if (lt(eint, 0.0)) {
      record_error(a.status, a.step, RG_ERR_NEGATIVE_ENERGY, 5, i, eint);
      return false;
    }
    c = Cell3{density, (a.gamma - 1) * eint * density, vel};
    store6(a.cells, i, c.d, c.p, vel.x, vel.y, vel.z);
  }
  return kCells;
}
template <bool kUnscaled, bool kExt, bool kCells>
__global__ void __launch_bounds__(kBlock) k3_update(Step3Args a) {
  chain_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  Cell3 c{1, 1, V3{0, 0, 0}};
  const bool in = i < a.mesh.n, live = in && update_cell3<kUnscaled, kExt, kCells>(a, i, c);
  if (kExt && kCells && a.cfl_next) {
    if (in && !live) c = load_cell3(a.cells, i);  // a rejected cell keeps its record, which a CFL pass reads
    grid_min_times(a.status, cfl3_block_bits(a, in, i, c), a.cfl, &a.status->dt_next);
  }
}

// Records of 5 doubles (the host's) <-> 6 (the device's, the last one 0), one
// value per thread, coalesced on both sides.  The copies between host and
// device then move one contiguous block: a pitched copy of 40-byte rows runs
// at 3.8 GB/s host to device (35 MB, the 96^3 cells: 9.25 ms; 0.19 ms as one
// block at 190 GB/s plus 18 us here).
__global__ void __launch_bounds__(kBlock) k3_unpack(const double* packed, double* rec, int rows) {
  const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (t >= 6LL * rows) return;
  const long long r = t / 6;
  const int q = static_cast<int>(t - 6 * r);
  rec[t] = q < 5 ? packed[5 * r + q] : 0.0;
}
__global__ void __launch_bounds__(kBlock) k3_pack(const double* rec, double* packed, int rows) {
  const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (t >= 5LL * rows) return;
  const long long r = t / 5;
  packed[t] = rec[6 * r + (t - 5 * r)];
}

__global__ void __launch_bounds__(kBlock) k3_init(Step3Args a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.mesh.n) return;
  const Cell3 c = load_cell3(a.cells, i);
  const double V = a.mesh.volume[i];
  const V3 mom = vscale(c.d, c.v);
  const double en = c.d * (0.5 * vdot(c.v, c.v) + dp2e(a.gamma, c.d, c.p));
  store6(a.ext, i, V * c.d, mom.x * V, mom.y * V, mom.z * V, V * en);
}

inline int blocks(long long n) { return n > 0 ? static_cast<int>((n + kBlock - 1) / kBlock) : 1; }

}  // namespace

cudaError_t launch3_unpack(const double* packed, double* rec, int rows, cudaStream_t s) {
  k3_unpack<<<blocks(6LL * rows), kBlock, 0, s>>>(packed, rec, rows);
  return cudaGetLastError();
}
cudaError_t launch3_pack(const double* rec, double* packed, int rows, cudaStream_t s) {
  k3_pack<<<blocks(5LL * rows), kBlock, 0, s>>>(rec, packed, rows);
  return cudaGetLastError();
}

cudaError_t launch3_validate(const Mesh3Dev& m, DevStatus* st, cudaStream_t s) {
  k3_validate<<<blocks(m.e > m.n ? m.e : m.n), kBlock, 0, s>>>(m, st);
  return cudaGetLastError();
}

cudaError_t launch3_geometry(const Mesh3Dev& m, dbl4* nhat, int* fsign, unsigned char* axis, cudaStream_t s) {
  k3_geometry<<<blocks(m.e > m.n ? m.e : m.n), kBlock, 0, s>>>(m, nhat, fsign, axis);
  return cudaGetLastError();
}

cudaError_t launch3_init_extensives(const Step3Args& a, cudaStream_t s) {
  k3_init<<<blocks(a.mesh.n), kBlock, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch3_cfl(const Step3Args& a, cudaStream_t s) {
  chain(s, blocks(a.mesh.n), kBlock, k3_cfl, a);
  return cudaGetLastError();
}

cudaError_t launch3_faces(const Step3Args& a, bool scaled, cudaStream_t s) {
  if (a.mesh.e == 0) return cudaSuccess;
  const LaunchShape sh = fit_shape(LaunchShape{kBlock, 0, 0, a.sms}, a.mesh.e);
  const int nb = grid_of(sh, a.mesh.e);
  if (scaled)
    chain(s, nb, sh.block, k3_faces<true>, a);
  else
    chain(s, nb, sh.block, k3_faces<false>, a);
  return cudaGetLastError();
}

cudaError_t launch3_update(const Step3Args& a, bool from_unscaled, bool do_ext, bool do_cells, cudaStream_t s) {
  const int nb = blocks(a.mesh.n);
  if (do_ext && do_cells)
    chain(s, nb, kBlock, k3_update<false, true, true>, a);  // (the fused step's fluxes are scaled)
  else if (do_ext && from_unscaled)
    chain(s, nb, kBlock, k3_update<true, true, false>, a);
  else if (do_ext)
    chain(s, nb, kBlock, k3_update<false, true, false>, a);
  else
    chain(s, nb, kBlock, k3_update<false, false, true>, a);
  return cudaGetLastError();
}

}  // namespace rg
