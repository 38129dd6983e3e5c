// Fused RK-stage kernel for one Cartesian patch: residual (all x, y and z
// face fluxes) and update f_out = f_n + factor/dV * Res(f_in) in one launch.
//
// Replaces the reference's per-stage sequence of a residual memset plus ten
// launches (six colour-split flux kernels, three boundary kernels, advance;
// iterators/gpu_cartesianiterator.h:54-304) that read-modify-write a residual
// field in HBM.  Here:
//   - a CTA owns a TJ x TK tile of (j, k) columns (k fastest, coalesced) and
//     marches along i through a chunk of planes;
//   - each plane of the stencil state is staged once in shared memory with a
//     two-cell halo in j and k, in a ring of three planes (i .. i+2; the own
//     column of plane i-1 is set aside beside it); plane i+2 is loaded while
//     the y and z faces of plane i are evaluated: by one TMA box load where
//     no periodic seam crosses the tile's halo, else cell by cell with
//     cp.async;
//   - every face flux is evaluated exactly once (fv_f64.cuh): x faces per
//     thread along its own column (the upper face of cell i is kept in
//     registers as the lower face of cell i+1), y and z faces of the current
//     plane into shared memory;
//   - the residual is summed per cell in registers in the reference's order
//     (+Fx_lo +Fy_lo +Fz_lo -Fz_hi -Fy_hi -Fx_hi, the order the single-thread
//     CPU iterator produces, cartesianiterator.h:115-188), no atomics;
//   - the update is written once; inactive cells copy their input
//     (cartesianiterator.h:315, gpu_cartesianiterator.h:199-201).
//
// The storage form is a policy (fv_policies.cuh): its 8-byte values are staged
// and computed with as they are, and Policy::update(un, r) makes the new value
// from f_n and the residual.
#pragma once

#include <cstdint>
#include "fv_numerics.cuh"
#include "fv_f64.cuh"
#include "fv_wall.cuh"
#include "fv_tma.cuh"

namespace dn {

struct StageGeom {
  int ni, nj, nk;
  int per_x, per_y, per_z;   // 1 = periodic wrap, 0 = closed
  int i_chunk;               // planes per CTA along i
};

template <class Policy>
struct StageArgs {
  const typename Policy::Store* in;   // stencil state f(k-1), [5][ni][nj][nk]
  const typename Policy::Store* un;   // step-start state f(n), own cell only
  typename Policy::Store* out;        // f(k)
  const uint8_t* active;              // per cell, NULL = all active
  int* err;                           // device error word (bit flags; here 32, a plane load that did not arrive)
  StageGeom g;
  typename Policy::Params p;
  WallBC wall;                        // patch-face fluxes of the non-periodic axes
};

// index along an axis with periodic wrap; returns -1 if outside a closed axis
__device__ __forceinline__ int axis_idx(int x, int n, int per)
{
  if ((unsigned)x < (unsigned)n) return x;
  if (!per) return -1;
  x = x < 0 ? x + n : x - n;                     // one wrap, but for tiles reaching far beyond a small patch
  if ((unsigned)x < (unsigned)n) return x;
  x %= n;
  return x < 0 ? x + n : x;
}

// does the face below cell index x (between x-1 and x) exist?
__device__ __forceinline__ bool face_exists(int x, int n, int per)
{
  if (n <= 2) return false;               // cartesianiterator.h:149,160,171
  return per ? true : (x >= 1 && x <= n - 1);
}

// is cell index x inside the axis (or wrapped)?
__device__ __forceinline__ bool cell_ok(int x, int n, int per)
{
  return per ? true : (x >= 0 && x < n);
}

template <class Policy, int TJ, int TK>
struct StageSmem {
  using Real = typename Policy::Real;
  static constexpr int PJ = TJ + 4;
  static constexpr int PK = TK + 4;
  alignas(128) Real plane[3][5][PJ][PK];   // planes i .. i+2
  Real xm[5][TJ * TK];                     // own column of plane i-1 (each thread its own cell)
  Real fy[5][TJ + 1][TK];
  Real fz[5][TJ][TK + 1];
  alignas(8) uint64_t bar;                 // mbarrier of the TMA plane loads
};

// Resident CTAs per SM the register allocation is sized for: 16 warps of 128
// registers (the unconstrained 138 cost a quarter of the warps).
template <int NT>
struct F64Occupancy {
  static constexpr int min_blocks = NT >= 512 ? 1 : 512 / NT;
};

// One tile of one patch: columns (j0 .. j0+TJ-1, k0 .. k0+TK-1), planes i0 .. i1-1.
// tm: tensor map of the stage input with box (TK+4, TJ+4, 1, 5), or null.
//
// A plane's faces run through one copy of the face code (per thread its y, z
// and x face, two warps one halo face more): four inlined copies, one per
// use, overflowed the instruction cache.
template <class Policy, class Scheme, int TJ, int TK>
__device__ __forceinline__ void fv_stage_tile(const StageArgs<Policy>& a, const CUtensorMap* tm, int j0, int k0,
                                              int i0, int i1)
{
  using Real = typename Policy::Real;
  using Smem = StageSmem<Policy, TJ, TK>;
  static_assert(sizeof(typename Policy::Store) == 8 && sizeof(Real) == 8, "cell copies move the stored 8-byte value");
  constexpr int PJ = TJ + 4, PK = TK + 4, NT = TJ * TK, NW = NT / 32;
  constexpr int VS = PJ * PK, SS = 5 * VS;          // variable and slot strides of the ring
  constexpr int PPT = (VS + NT - 1) / NT;           // positions of a plane per thread and variable
  extern __shared__ __align__(128) unsigned char dn_smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(dn_smem_raw);

  const StageGeom& g = a.g;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int j = j0 + ty, k = k0 + tx;
  const bool own = (j < g.nj) && (k < g.nk);
  const size_t nc = (size_t)g.ni * g.nj * g.nk;
  const size_t njk = (size_t)g.nj * g.nk;
  const int tid = ty * TK + tx;
  const int warp = tid >> 5, lane = tid & 31;
  Real* const ring = &sm.plane[0][0][0][0];
  const int me = (ty + 2) * PK + tx + 2;            // own cell in a plane of the ring
  // TMA plane loads where no periodic seam crosses the tile's halo (on a
  // closed axis the box cells outside the patch are zero-filled, as the
  // cell copies write them); the box starts at column k0-2, a multiple of 2
  // elements (16 bytes) since TK is even
  constexpr unsigned kPlaneBytes = 5u * VS * sizeof(Real);
  const bool tma = tm != nullptr && (!g.per_y || (j0 >= 2 && j0 + TJ + 2 <= g.nj)) &&
                   (!g.per_z || (k0 >= 2 && k0 + TK + 2 <= g.nk)) && (smem_u32(ring) & 127) == 0;
  if (tma && tid == 0) {
    mbar_init(&sm.bar, 1);
    mbar_init_fence();
  }
  unsigned phase = 0;
  bool tbad = false;

  // in-plane offsets of this thread's positions for cell copies (-1: outside a closed axis)
  int poff[PPT];
  #pragma unroll
  for (int m = 0; m < PPT; ++m) {
    const int e = tid + m * NT;
    const int jg = axis_idx(j0 - 2 + e / PK, g.nj, g.per_y), kg = axis_idx(k0 - 2 + e % PK, g.nk, g.per_z);
    poff[m] = (e < VS && jg >= 0 && kg >= 0) ? jg * g.nk + kg : -1;
  }
  // plane i (inside the patch) into ring slot `slot` cell by cell: cp.async
  // of the cells inside the patch, zero outside a closed axis (never read)
  auto copy_plane = [&](int slot, int i) {
    const Real* src = a.in + (size_t)i * njk;
    Real* dst = ring + slot * SS;
    #pragma unroll
    for (int m = 0; m < PPT; ++m) {
      const int e = tid + m * NT;
      if (e >= VS) continue;
      #pragma unroll
      for (int v = 0; v < 5; ++v) {
        if (poff[m] >= 0) {
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;"
                       :: "r"(smem_u32(dst + v * VS + e)), "l"(src + v * nc + poff[m]) : "memory");
        } else {
          dst[v * VS + e] = Real(0);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // a three-plane ring, rotated by hand: sa, sb, sc hold planes i-1, i, i+1
  // at the top of iteration i.  Prologue: planes i0-1 .. i0+1, and the own
  // column of plane i0-2 (plane i0-1 again where it does not exist)
  int sa = 0, sb = 1, sc = 2;
  for (int q = -1; q <= 1; ++q) {
    const int ip = axis_idx(i0 + q, g.ni, g.per_x);
    if (ip >= 0) copy_plane(q + 1, ip);   // planes outside a closed patch are never read
  }
  const bool face0 = face_exists(i0, g.ni, g.per_x);
  if (own && face0) {
    const Real* col = a.in + (size_t)axis_idx(cell_ok(i0 - 2, g.ni, g.per_x) ? i0 - 2 : i0 - 1, g.ni, g.per_x) * njk +
                      (size_t)j * g.nk + k;
    #pragma unroll
    for (int v = 0; v < 5; ++v) sm.xm[v][tid] = col[v * nc];
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  const bool ey = face_exists(j, g.nj, g.per_y) && k < g.nk && (g.per_y || j < g.nj);
  const bool ez = face_exists(k, g.nk, g.per_z) && j < g.nj && (g.per_z || k < g.nk);
  Real fx_lo[5];
  // iteration i0-1 evaluates the x face below cell i0 only
  for (int i = i0 - 1; i < i1; ++i) {
    const bool first = i < i0;
    int s0, sp1, sp2;                     // slots of planes i, i+1, i+2
    int ip2 = -1;
    if (first) {
      s0 = sa; sp1 = sb; sp2 = sc;
    } else {
      // plane i+2 replaces plane i-1 in the ring; the own column of plane
      // i-1 (the x face above cell i reads it) is set aside first (plane i
      // itself where plane i-1 lies outside a closed patch)
      const Real* src = ring + (cell_ok(i - 1, g.ni, g.per_x) ? sa : sb) * SS + me;
      #pragma unroll
      for (int v = 0; v < 5; ++v) sm.xm[v][tid] = src[v * VS];
      __syncthreads();
      // plane i+2 into the freed slot, arriving while the y and z faces of
      // plane i are evaluated (a plane outside a closed patch is never read)
      ip2 = axis_idx(i + 2, g.ni, g.per_x);
      if (ip2 >= 0) {
        if (tma) {
          if (tid == 0) {
            fence_proxy_async_smem();
            mbar_arrive_expect_tx(&sm.bar, kPlaneBytes);
            tma_load_4d(ring + sa * SS, tm, &sm.bar, k0 - 2, j0 - 2, ip2, 0);
          }
        } else {
          copy_plane(sa, ip2);
        }
      }
      s0 = sb; sp1 = sc; sp2 = sa;
    }

    Real F[5];
    #pragma unroll 1
    for (int t = first ? 3 : 0; t < 4; ++t) {
      // t = 0, 1: the y and z faces below the own cell; 2: the faces below
      // halo row TJ (last warp) and halo column TK (the warp before it); 3:
      // the x face above the own cell
      if (t == 2 && warp < NW - 2) continue;
      FaceCells c;
      int dir;
      bool ex;
      Real A;
      Real* o = nullptr;
      int os = 0;
      if (t == 3) {
        if (!first) {
          // plane i+2 has arrived (this thread's copies, or the TMA box);
          // the barrier publishes it and the y and z faces
          if (ip2 >= 0) {
            if (tma) {
              tbad |= !mbar_wait(&sm.bar, phase);
              phase ^= 1u;
            } else {
              asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
          }
          __syncthreads();
        }
        dir = 0;
        A = a.p.Ax;
        ex = own && face_exists(i + 1, g.ni, g.per_x);
        c.sl = cell_ok(i - 1, g.ni, g.per_x);
        c.sr = cell_ok(i + 2, g.ni, g.per_x);
        c.m2 = &sm.xm[0][tid];
        c.s2 = NT;
        c.m1 = ring + s0 * SS + me;
        c.p0 = ring + sp1 * SS + me;
        c.p1 = ring + (c.sr ? sp2 : sp1) * SS + me;
      } else {
        const bool halo = t == 2;
        dir = halo ? (warp == NW - 1 ? 1 : 2) : t + 1;
        const bool ydir = dir == 1;
        const int jj = halo ? (ydir ? TJ : lane) : ty, kk = halo ? (ydir ? lane : TK) : tx;
        const int jf = j0 + jj, kf = k0 + kk;
        if (ydir) {
          ex = halo ? (lane < TK && face_exists(jf, g.nj, g.per_y) && kf < g.nk && (g.per_y || jf < g.nj)) : ey;
          c.sl = cell_ok(jf - 2, g.nj, g.per_y);
          c.sr = cell_ok(jf + 1, g.nj, g.per_y);
          A = a.p.Ay;
          if (!halo || lane < TK) o = &sm.fy[0][jj][kk];
          os = (TJ + 1) * TK;
        } else {
          ex = halo ? (lane < TJ && face_exists(kf, g.nk, g.per_z) && jf < g.nj && (g.per_z || kf < g.nk)) : ez;
          c.sl = cell_ok(kf - 2, g.nk, g.per_z);
          c.sr = cell_ok(kf + 1, g.nk, g.per_z);
          A = a.p.Az;
          if (!halo || lane < TJ) o = &sm.fz[0][jj][kk];
          os = TJ * (TK + 1);
        }
        const int step = ydir ? PK : 1;
        c.p0 = ring + s0 * SS + (jj + 2) * PK + kk + 2;
        c.m1 = c.p0 - step;
        c.m2 = c.m1 - (c.sl ? step : 0);
        c.p1 = c.p0 + (c.sr ? step : 0);
        c.s2 = VS;
      }
      if (ex) {
        face_flux<Scheme, VS>(dir, c, A, F);
      } else {
        #pragma unroll
        for (int v = 0; v < 5; ++v) F[v] = Real(0);
      }
      if (o) {
        #pragma unroll
        for (int v = 0; v < 5; ++v) o[v * os] = F[v];
      }
    }

    if (!first && own) {
      const size_t c = (size_t)i * njk + (size_t)j * g.nk + k;
      const bool act = a.active ? (a.active[c] != 0) : true;
      Real res[5];
      #pragma unroll
      for (int v = 0; v < 5; ++v) {
        Real r = fx_lo[v];
        r += sm.fy[v][ty][tx];
        r += sm.fz[v][ty][tx];
        r -= sm.fz[v][ty][tx + 1];
        r -= sm.fy[v][ty + 1][tx];
        r -= F[v];
        res[v] = r;
      }
      if (a.wall.any && (i == 0 || i == g.ni - 1 || j == 0 || j == g.nj - 1 || k == 0 || k == g.nk - 1)) {
        Real U[5];
        #pragma unroll
        for (int v = 0; v < 5; ++v) U[v] = ring[s0 * SS + v * VS + me];
        add_wall_fluxes(a.wall, g.ni, g.nj, g.nk, g.per_x, g.per_y, g.per_z, i, j, k, U, a.p.Ax, a.p.Ay, a.p.Az, res,
                        [](int, Real x) { return x; });
      }
      #pragma unroll
      for (int v = 0; v < 5; ++v) {
        typename Policy::Store o;
        if (act) {
          o = Policy::update(a.p, a.un[v * nc + c], res[v]);
        } else {
          o = a.in[v * nc + c];
        }
        a.out[v * nc + c] = o;
      }
    }
    #pragma unroll
    for (int v = 0; v < 5; ++v) fx_lo[v] = F[v];
    if (!first) {
      sa = s0;
      sb = sp1;
      sc = sp2;
    }
  }
  if (tbad && a.err) atomicOr(a.err, 32);
}

// Parameters of the single-patch launch: the stage arguments and the tensor
// map of the stage input (valid when tma != 0).
template <class Policy>
struct StageLaunch {
  CUtensorMap tm;
  StageArgs<Policy> a;
  int tma;
};

// One patch per launch: grid (k tiles, j tiles, i chunks).
template <class Policy, class Scheme, int TJ, int TK>
__global__ void __launch_bounds__(TJ * TK, F64Occupancy<TJ * TK>::min_blocks)
fv_stage_kernel(const __grid_constant__ StageLaunch<Policy> L)
{
  const int i0 = blockIdx.z * L.a.g.i_chunk;
  fv_stage_tile<Policy, Scheme, TJ, TK>(L.a, L.tma ? &L.tm : nullptr, blockIdx.y * TJ, blockIdx.x * TK, i0,
                                min(L.a.g.ni, i0 + L.a.g.i_chunk));
}

} // namespace dn
