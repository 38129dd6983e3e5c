// Patch-face (wall) fluxes of a stage: the flux functor's x/y/zWall{M,P}
// called for the outer faces of a non-periodic patch axis
// (iterators/cartesianiterator.h:190-308, gpu_cartesianiterator.h:117-186).
//
// Each face uses the first-order state of its own boundary cell (the
// reference's Upwind2 projection drops to first order at the patch edge,
// reconstruction/upwind2.h:39-42) and is added to that cell's residual after
// all interior faces, in the reference's order x-min, x-max, y-min, y-max,
// z-min, z-max, with + on min sides and - on max sides.  Axes of two cells or
// fewer get no wall flux (cartesianiterator.h:193,212,...).
//
// Kinds:
//   zero flux    a functor whose wall methods add nothing
//   far field    CompressibleFarfieldFlux (fluxes/compressiblefarfieldflux.h:26-181)
//   slip wall    CompressibleSlipFlux (fluxes/compressibleslipflux.h:34-98): pressure only
//   inflow       a prescribed face state (u, v, w, T and optionally p) per face, the
//                JetFlux::xWallM form of applications/drnumJetDemo/jetflux.h:158-192;
//                p from the boundary cell where the table's p is NaN
#pragma once

#include "fv_numerics.cuh"

namespace dn {

enum WallKind : int { kWallZero = 0, kWallFarfield = 1, kWallSlip = 2, kWallInflow = 3 };

struct WallBC {
  int any;                // 0: every side has zero flux
  int kind[6];            // per side: x-min, x-max, y-min, y-max, z-min, z-max
  double ff[6][6];        // far field per side: p0, T0, u0, v0, w0, a0 (primitive, from the
                          // conservative far-field state, perfectgas.h:84-93)
  const double* table[6]; // inflow per side: [faces][5] = p (NaN: boundary cell), T, u, v, w;
                          // x sides: face j*nk+k, y sides: i*nk+k, z sides: i*nj+j
};

constexpr double kGasCp = 1004.5;   // PerfectGas::cp (perfectgas.h:33)

// Primitive state of a conservative state (PerfectGas::conservativeToPrimitive,
// perfectgas.h:84-93; COMPR_VARS, compressibleflux.h:26-38).
template <typename T>
__device__ __forceinline__ void wall_prim(const T U[5], T& p, T& Tt, T& u, T& v, T& w)
{
  const T ir = T(1.0) / U[0];
  u = U[1] * ir;
  v = U[2] * ir;
  w = U[3] * ir;
  Tt = (U[4] * ir - T(0.5) * (u * u + v * v + w * w)) / T(Gas::cv);
  p = U[0] * T(Gas::R) * Tt;
}

// Wall flux of side `side` (2 * axis + 1 on the max side) for a boundary cell
// with state U; `face` indexes the side's inflow table.  Returns false for a
// zero-flux side (nothing to add).  The kinds choose a face state (p, T, u, v, w)
// and share the flux from it, the tail of CompressibleFarfieldFlux and
// JetFlux::xWallM (a slip wall has its pressure only).
template <typename T>
__device__ __forceinline__ bool wall_flux(const WallBC& bc, int axis, int side, int face, const T U[5], T A, T F[5])
{
  const int kind = bc.kind[side];
  if (kind == kWallZero) return false;
  T p1, T1, u1, v1, w1;
  wall_prim(U, p1, T1, u1, v1, w1);
  T p = p1;
  F[0] = T(0); F[1] = T(0); F[2] = T(0); F[3] = T(0); F[4] = T(0);
  if (kind != kWallSlip) {
    T Tt = T1, u = u1, v = v1, w = w1;
    if (kind == kWallInflow) {
      const double* e = bc.table[side] + (size_t)face * 5;
      if (e[0] == e[0]) p = (T)e[0];               // NaN: pressure of the boundary cell
      Tt = (T)e[1];
      u = (T)e[2];
      v = (T)e[3];
      w = (T)e[4];
    } else {
      // far field: face state from the sign and size of the mean inward Mach number
      const double* f = bc.ff[side];
      const T u0 = (T)f[2], v0 = (T)f[3], w0 = (T)f[4], a0 = (T)f[5];
      const T a1 = dn_sqrt(T(Gas::gamma) * T(Gas::R) * T1);
      T M0 = (axis == 0 ? u0 : (axis == 1 ? v0 : w0)) / a0;
      T M1 = (axis == 0 ? u1 : (axis == 1 ? v1 : w1)) / a1;
      if (side & 1) {
        M0 = -M0;
        M1 = -M1;
      }
      const T M = T(0.5) * (M0 + M1);
      // outflow: the reference's test `M <= 1` holds for every M < 0, so the
      // whole face state comes from the boundary cell
      if (M >= T(0)) {
        if (M >= T(1)) p = (T)f[0];                // supersonic, else subsonic inflow
        Tt = (T)f[1];
        u = u0;
        v = v0;
        w = w0;
      }
    }
    F[0] = A * p / (T(Gas::R) * Tt) * (axis == 0 ? u : (axis == 1 ? v : w));
    F[1] = F[0] * u;
    F[2] = F[0] * v;
    F[3] = F[0] * w;
    F[4] = F[0] * (T(kGasCp) * Tt + T(0.5) * (u * u + v * v + w * w));
  }
  const T Ap = A * p;
  F[1] = axis == 0 ? F[1] + Ap : F[1];
  F[2] = axis == 1 ? F[2] + Ap : F[2];
  F[3] = axis == 2 ? F[3] + Ap : F[3];
  return true;
}

// Adds the wall fluxes of a boundary cell (i, j, k) to its residual r in the
// reference's order; F_to_r converts a flux to the residual's type.
template <typename T, typename R, typename Conv>
__device__ __forceinline__ void add_wall_fluxes(const WallBC& bc, int ni, int nj, int nk, int per_x, int per_y,
                                                int per_z, int i, int j, int k, const T U[5], T Ax, T Ay, T Az,
                                                R r[5], Conv F_to_r)
{
  T F[5];
  if (!per_x && ni > 2) {
    if (i == 0 && wall_flux(bc, 0, 0, j * nk + k, U, Ax, F)) {
      #pragma unroll
      for (int v = 0; v < 5; ++v) r[v] += F_to_r(v, F[v]);
    }
    if (i == ni - 1 && wall_flux(bc, 0, 1, j * nk + k, U, Ax, F)) {
      #pragma unroll
      for (int v = 0; v < 5; ++v) r[v] -= F_to_r(v, F[v]);
    }
  }
  if (!per_y && nj > 2) {
    if (j == 0 && wall_flux(bc, 1, 2, i * nk + k, U, Ay, F)) {
      #pragma unroll
      for (int v = 0; v < 5; ++v) r[v] += F_to_r(v, F[v]);
    }
    if (j == nj - 1 && wall_flux(bc, 1, 3, i * nk + k, U, Ay, F)) {
      #pragma unroll
      for (int v = 0; v < 5; ++v) r[v] -= F_to_r(v, F[v]);
    }
  }
  if (!per_z && nk > 2) {
    if (k == 0 && wall_flux(bc, 2, 4, i * nj + j, U, Az, F)) {
      #pragma unroll
      for (int v = 0; v < 5; ++v) r[v] += F_to_r(v, F[v]);
    }
    if (k == nk - 1 && wall_flux(bc, 2, 5, i * nj + j, U, Az, F)) {
      #pragma unroll
      for (int v = 0; v < 5; ++v) r[v] -= F_to_r(v, F[v]);
    }
  }
}

} // namespace dn
