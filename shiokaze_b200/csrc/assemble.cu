// Assembly of the variational pressure system and the velocity update.
//
// This translation unit is compiled with -fmad=false: the face areas, liquid
// fractions, matrix weights and right-hand side are evaluated in FP64 with
// the same operation order as the reference CPU code, so masks are bit-exact
// and the FP64 system equals the reference's RCMatrix values.
//
//   face solid area   macutility3::compute_area_fraction (src/utility/macutility3.cpp:98-171)
//                     + utility::get_area (include/shiokaze/utility/utility.h:191-226)
//   face liquid rho   macutility3::compute_fluid_fraction (macutility3.cpp:172-200)
//                     + utility::fraction (utility.h:174-182)
//   unknowns          mark_body (src/projection/macpressuresolver3.cpp:134-158)
//   weights, rhs      macpressuresolver3.cpp:179-216
//   velocity update   macpressuresolver3.cpp:262-284
//   solid density     macpressuresolver3.cpp:75-80 (areas), 286-293 (velocity scale)
//   surface tension   macpressuresolver3.cpp:98-128
//   volume correction macpressuresolver3.cpp:219-234 (constant added to every rhs row)
#include "common.cuh"
#include "kernels.h"
#include <float.h>

#include <algorithm>

namespace shkz {

struct FaceParams {
  const float *solid;          // nodal effective values, or null (no solid level set)
  const uint8_t *solid_active;
  const float *fluid;          // cell effective values
  int nx, ny, nz;
  int solid_exists, fluid_exists;
  double eps_solid, eps_fluid;
  int second_order_fluid, second_order_solid;
  const float *density[3];     // per-face solid density (set_solid_density), or null
};

// Marching-squares area of the negative region on the unit square, corners
// in (0,0),(1,0),(1,1),(0,1) order, followed by the shoelace sum.
__device__ __forceinline__ double get_area4(const float c[4]) {
  const double qx[4] = {0.0, 1.0, 1.0, 0.0};
  const double qy[4] = {0.0, 0.0, 1.0, 1.0};
  bool all_neg = true, all_nonneg = true;
  #pragma unroll
  for (int n = 0; n < 4; ++n) {
    all_neg &= (c[n] < 0.0f);
    all_nonneg &= !(c[n] < 0.0f);
  }
  // Uniform corners give no crossing points: an empty list (area 0) or the
  // unit square (shoelace sum 2, area 1), exactly as the general path does.
  if (all_nonneg) return 0.0;
  if (all_neg) return 1.0;
  const double v[4] = {(double)c[0], (double)c[1], (double)c[2], (double)c[3]};
  double px[8], py[8];
  int pnum = 0;
  #pragma unroll
  for (int n = 0; n < 4; ++n) {
    if (v[n] < 0.0) {
      px[pnum] = qx[n];
      py[pnum] = qy[n];
      pnum++;
    }
    const int m = (n + 1) & 3;
    if (v[n] * v[m] < 0) {
      const double y0 = v[n], y1 = v[m];
      if (y0 - y1 != 0.0) {
        const double a = y0 / (y0 - y1);
        px[pnum] = (1.0 - a) * qx[n] + a * qx[m];
        py[pnum] = (1.0 - a) * qy[n] + a * qy[m];
        pnum++;
      }
    }
  }
  double sum = 0.0;
  for (int m = 0; m < pnum; m++) {
    const int m1 = (m + 1 == pnum) ? 0 : m + 1;
    sum += px[m] * py[m1] - py[m] * px[m1];
  }
  return 0.5 * sum;
}

__device__ __forceinline__ size_t nidx(const FaceParams &P, int i, int j, int k) {
  return (size_t)i + (size_t)(P.nx + 1) * ((size_t)j + (size_t)(P.ny + 1) * (size_t)k);
}
__device__ __forceinline__ size_t cidx(const FaceParams &P, int i, int j, int k) {
  return (size_t)i + (size_t)P.nx * ((size_t)j + (size_t)P.ny * (size_t)k);
}

// Solid area of face (d; i,j,k) as the reference stores it (float).
__device__ float face_area(const FaceParams &P, int d, int i, int j, int k) {
  const int pd = d == 0 ? i : (d == 1 ? j : k);
  const int nd = d == 0 ? P.nx : (d == 1 ? P.ny : P.nz);
  double a;
  bool act = false;  // face active in the reference's area grid
  if (!P.solid_exists) {
    // areas.clear(1.0) with the domain walls closed (macutility3.cpp:158-170)
    a = (pd == 0 || pd == nd) ? 0.0 : 1.0;
  } else {
    // the face's corners (0,0), (1,0), (1,1), (0,1) of its two axes
    const size_t sy = (size_t)(P.nx + 1), sz = sy * (size_t)(P.ny + 1);
    const size_t ua = d == 0 ? sy : 1, ub = d == 2 ? sy : sz;
    const size_t s0 = nidx(P, i, j, k), s1 = s0 + ua, s2 = s1 + ub, s3 = s0 + ub;
    // quadsolid[0][0], [1][0], [1][1], [0][1] -> corners (0,0),(1,0),(1,1),(0,1)
    const float c[4] = {P.solid[s0], P.solid[s1], P.solid[s2], P.solid[s3]};
    act = P.solid_active[s0] | P.solid_active[s1] | P.solid_active[s2] | P.solid_active[s3];
    if (act) {
      if (pd == 0 || pd == nd) a = 0.0;
      else a = 1.0 - get_area4(c);
      if (a != 0.0 && a < P.eps_solid) a = P.eps_solid;
    } else {
      // inactive face: the flood-filled value, 1 outside the solid and the
      // background 0 inside; all four corners lie on one side of the band
      a = 1.0 - get_area4(c);
    }
  }
  float af = (float)a;
  if (act && P.density[d]) {
    // solid density on the active faces of the area grid: density*area + (1 - density)
    const int fw = P.nx + (d == 0), fh = P.ny + (d == 1);
    const float dens = P.density[d][(size_t)i + (size_t)fw * ((size_t)j + (size_t)fh * (size_t)k)];
    const float da = dens * af;
    af = (float)((double)da + (1.0 - (double)dens));
  }
  if (!P.second_order_solid && af != 0.0f) af = 1.0f;
  return af;
}

__device__ __forceinline__ double fraction(double phi0, double phi1) {
  if (phi0 * phi1 >= 0.0) {
    if (phi0 < 0.0 || phi1 < 0.0) return 1.0;
    return 0.0;
  }
  return -fmin(phi0, phi1) / fmax(fabs(phi1 - phi0), DBL_MIN);
}

// Liquid fraction of face (d; i,j,k) as the reference stores it (float).
__device__ float face_rho(const FaceParams &P, int d, int i, int j, int k) {
  double r;
  if (!P.fluid_exists) {
    r = 1.0;
  } else {
    // the cells on both sides; at the domain's faces, both are the inner one
    const int pd = d == 0 ? i : (d == 1 ? j : k), nd = d == 0 ? P.nx : (d == 1 ? P.ny : P.nz);
    const size_t step = d == 0 ? 1 : d == 1 ? (size_t)P.nx : (size_t)P.nx * (size_t)P.ny;
    const size_t at = cidx(P, i, j, k);
    const float hi = P.fluid[pd == nd ? at - step : at], lo = P.fluid[pd == 0 ? at : at - step];
    r = fraction((double)hi, (double)lo);
    if (r != 0.0 && r < P.eps_fluid) r = P.eps_fluid;
  }
  float rf = (float)r;
  if (!P.second_order_fluid && rf != 0.0f) rf = 1.0f;
  return rf;
}

// ---------------------------------------------------------------------------
// levelset_exist (include/shiokaze/array/array_utility3.h:112-122) for the
// liquid (flag bit 0) and solid (bit 1) grids.
__global__ void k_levelset_exist(const float *fluid, const uint8_t *fluid_active, size_t ncell, const float *solid,
                                 const uint8_t *solid_active, size_t nnode, int *flags) {
  // four cells a trip, and a look at what others have found (512^3: 248 us
  // without, 11 with)
  const size_t step = (size_t)gridDim.x * blockDim.x, first = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  auto any_inside = [&](const float *phi, const uint8_t *active, size_t n, int bit) {
    bool in = false;
    for (size_t c = first; c < n && !in; c += 4 * step) {
      if (*(volatile const int *)flags & bit) break;
      uint8_t a[4];
      #pragma unroll
      for (int q = 0; q < 4; ++q) a[q] = c + q * step < n ? active[c + q * step] : 0;
      #pragma unroll
      for (int q = 0; q < 4; ++q) in |= a[q] && phi[c + q * step] < 0.0f;
    }
    if (__syncthreads_or(in) && threadIdx.x == 0) atomicOr(flags, bit);
  };
  any_inside(fluid, fluid_active, ncell, 1);
  if (solid) any_inside(solid, solid_active, nnode, 2);
}

// ---------------------------------------------------------------------------
// Strips: four 8^3 tiles along x, one CTA each. A warp takes rows of 32 cells,
// 8 of the strip's 64, so that every access is a row's. (A thread per cell of
// a tile, or of the grid with its coordinates from divisions, left HBM idle:
// 512^3, label 1351 -> 600 us, pressure scatter 628 -> 212; at 64^3, where a
// warp's eight rows follow one another, label 8 -> 12.)
constexpr int kStripTiles = 4;
static __host__ __device__ __forceinline__ long long strip_count(const Geometry &G) {
  return (long long)((G.bx + kStripTiles - 1) / kStripTiles) * G.by * G.bz;
}

// Unknown labelling. Writes the dense unknown mask and the number of unknowns
// per tile.
__global__ void __launch_bounds__(256) k_label(FaceParams P, Geometry G, const int *flags, uint8_t *unk, int *tile_count) {
  __shared__ int count[kStripTiles];
  P.fluid_exists = (*flags) & 1;
  P.solid_exists = P.solid ? (((*flags) >> 1) & 1) : 0;
  const int sx = (G.bx + kStripTiles - 1) / kStripTiles;
  const int b = blockIdx.x, s0 = b % sx * kStripTiles, tj = b / sx % G.by, tk = b / sx / G.by;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < kStripTiles) count[threadIdx.x] = 0;
  __syncthreads();
  const int i = s0 * SHKZ_T + lane, k = tk * SHKZ_T + warp;
  float phi[SHKZ_T];
  #pragma unroll
  for (int y = 0; y < SHKZ_T; ++y) {
    const int j = tj * SHKZ_T + y;
    phi[y] = i < G.nx && j < G.ny && k < G.nz ? P.fluid[cidx(P, i, j, k)] : 0.0f;
  }
  int mine = 0;
  for (int y = 0; y < SHKZ_T; ++y) {
    const int j = tj * SHKZ_T + y;
    bool inside = false;
    if (phi[y] < 0.0f) {
      // neighbours in the reference's order: +x, -x, +y, -y, +z, -z
      #pragma unroll 1
      for (int nq = 0; nq < 6 && !inside; ++nq) {
        const int d = nq >> 1, s = (nq & 1) ? -1 : 1;
        const int qi = i + (d == 0) * s, qj = j + (d == 1) * s, qk = k + (d == 2) * s;
        if (qi < 0 || qj < 0 || qk < 0 || qi >= G.nx || qj >= G.ny || qk >= G.nz) continue;
        if (!(P.fluid[cidx(P, qi, qj, qk)] < 0.0f)) continue;
        const int fi = s > 0 ? qi : i, fj = s > 0 ? qj : j, fk = s > 0 ? qk : k;
        if (face_area(P, d, fi, fj, fk) != 0.0f && face_rho(P, d, fi, fj, fk) != 0.0f) inside = true;
      }
    }
    if (i < G.nx && j < G.ny && k < G.nz) unk[cidx(P, i, j, k)] = inside ? 1 : 0;
    const unsigned in = __ballot_sync(0xffffffffu, inside);
    if (lane < kStripTiles) mine += __popc((in >> (8 * lane)) & 0xffu);
  }
  if (lane < kStripTiles && mine) atomicAdd(&count[lane], mine);
  __syncthreads();
  if (threadIdx.x < kStripTiles && s0 + (int)threadIdx.x < G.bx)
    tile_count[s0 + threadIdx.x + (long long)G.bx * (tj + (long long)G.by * tk)] = count[threadIdx.x];
}

// ---------------------------------------------------------------------------
// Weights and right-hand side per pool tile. For every unknown cell:
//   w_f   = dt*area/(dx*dx*rho) for in-domain faces with area, rho != 0
//   A_ii  = sum of w_f in the order +x,-x,+y,-y,+z,-z
//   A_i,i-e = -w_f when the neighbour is liquid (it is then an unknown);
//             stored as the positive lower weight off_e
//   b_i   = sum_f -sgn*area*u_f/dx (+ -sgn*(1-area)*u_solid/dx where area<1)
// Non-unknown cells get zeros everywhere, which keeps y = A x zero there.
__global__ void __launch_bounds__(256) k_coeff(FaceParams P, Geometry G, const int *flags, const int *pool_tile,
                                               const uint8_t *unk, const float *vel0, const float *vel1,
                                               const float *vel2, const float *svel0, const float *svel1,
                                               const float *svel2, double dx, double dt, float *diag, float *offx,
                                               float *offy, float *offz, double *diag64, double *offx64,
                                               double *offy64, double *offz64, double *rhs64, double rhs_add) {
  // Each face of the tile once, for the cells on both its sides: its weight
  // and its two terms of the right-hand side, before the sign. (Six faces a cell,
  // every one with its corners and divisions, took 678 us for a 256^3 tank's
  // tiles, 530 so.)
  __shared__ double wface[3][576], bface[3][576], sface[3][576];
  P.fluid_exists = (*flags) & 1;
  P.solid_exists = P.solid ? (((*flags) >> 1) & 1) : 0;
  const int pt = blockIdx.x;
  const long long t = pool_tile[pt];
  const int ti = (int)(t % G.bx), tj = (int)((t / G.bx) % G.by), tk = (int)(t / ((long long)G.bx * G.by));
  const float *vel[3] = {vel0, vel1, vel2};
  const float *svel[3] = {svel0, svel1, svel2};
  const double inner = dt / (dx * dx);  // of a face in the liquid, off the solid
  // face (d; place p): 9 along d, 8 along the others, x fastest
  #pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int wx = 8 + (d == 0), wy = 8 + (d == 1);
    const int fw = G.nx + (d == 0), fh = G.ny + (d == 1), fd = G.nz + (d == 2);
    for (int p = threadIdx.x; p < 576; p += blockDim.x) {
      const int i = ti * SHKZ_T + p % wx, j = tj * SHKZ_T + p / wx % wy, k = tk * SHKZ_T + p / (wx * wy);
      if (i >= fw || j >= fh || k >= fd) continue;
      const int pd = d == 0 ? i : d == 1 ? j : k, nd = d == 0 ? G.nx : d == 1 ? G.ny : G.nz;
      const double area = (double)face_area(P, d, i, j, k);
      double w = 0.0, us = 0.0;
      if (pd != 0 && pd != nd && area != 0.0) {
        const double rho = (double)face_rho(P, d, i, j, k);
        if (area == 1.0 && rho == 1.0) w = inner;
        else if (rho != 0.0) w = dt * area / (dx * dx * rho);
      }
      const size_t f = (size_t)i + (size_t)fw * ((size_t)j + (size_t)fh * (size_t)k);
      if (area < 1.0 && svel[d]) us = (1.0 - area) * (double)svel[d][f] / dx;
      wface[d][p] = w;
      bface[d][p] = area * (double)vel[d][f] / dx;
      sface[d][p] = us;
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < SHKZ_TC; c += blockDim.x) {
    const int x = c & 7, y = (c >> 3) & 7, z = c >> 6;
    const int i = ti * SHKZ_T + x, j = tj * SHKZ_T + y, k = tk * SHKZ_T + z;
    const size_t o = (size_t)pt * SHKZ_TC + c;
    double dg = 0.0, b = 0.0, lo[3] = {0.0, 0.0, 0.0};
    const bool in_grid = i < G.nx && j < G.ny && k < G.nz;
    if (in_grid && unk[cidx(P, i, j, k)]) {
      #pragma unroll
      for (int nq = 0; nq < 6; ++nq) {
        const int d = nq >> 1, up = 1 - (nq & 1);
        const int fx = x + (d == 0) * up, fy = y + (d == 1) * up, fz = z + (d == 2) * up;
        const int p = fx + (8 + (d == 0)) * (fy + (8 + (d == 1)) * fz);
        const double w = wface[d][p];
        dg += w;
        // (at the domain's faces the weight is zero)
        if (!up && w != 0.0 && P.fluid[cidx(P, i - (d == 0), j - (d == 1), k - (d == 2))] < 0.0f) lo[d] = w;
        b += up ? -bface[d][p] : bface[d][p];
        b += up ? -sface[d][p] : sface[d][p];
      }
      b += rhs_add;
    }
    diag[o] = (float)dg;
    offx[o] = (float)lo[0];
    offy[o] = (float)lo[1];
    offz[o] = (float)lo[2];
    if (diag64) {
      diag64[o] = dg;
      offx64[o] = lo[0];
      offy64[o] = lo[1];
      offz64[o] = lo[2];
    }
    rhs64[o] = b;
  }
}

// ---------------------------------------------------------------------------
// Velocity update over every face of dimension d (macpressuresolver3.cpp:269-284):
// active faces with area and rho != 0 get u -= dt*(p_i - p_{i-1})/(rho*dx)
// (u = u_solid on the domain walls); other active faces are switched off.
// The pressure is read as the FP32 grid the reference stores (m_pressure).
// A warp takes a row of faces, 128 at a time: four coalesced looks at the
// active bytes, then the active faces 32 at a time. Bound by the latency of a
// face's corner, cell and pressure loads, hence 32 registers and eight blocks a
// SM: 512^3 1310 us (1841 with four), 1985 with a thread per face, a launch per
// axis and coordinates from 64-bit divisions; 64^3 29 -> 12 us.
struct FaceFields {
  const float *svel[3];
  float *vel[3];
  uint8_t *vact[3];
};
template <int d>
__device__ __forceinline__ void update_row(const FaceParams &P, const Geometry &G, const int *tile_state,
                                           const float *pressure_pool, const float *svel, double dx, double dt,
                                           float *vel, uint8_t *vact, int j, int k) {
  const int fw = G.nx + (d == 0), fh = G.ny + (d == 1), lane = threadIdx.x & 31;
  const int nd = d == 0 ? G.nx : (d == 1 ? G.ny : G.nz);
  const size_t row = (size_t)fw * ((size_t)j + (size_t)fh * (size_t)k);
  for (int i0 = 0; i0 < fw; i0 += 128) {
    uint8_t on[4];
    #pragma unroll
    for (int q = 0; q < 4; ++q) on[q] = i0 + 32 * q + lane < fw ? vact[row + i0 + 32 * q + lane] : 0;
    #pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      const bool mine = q == 0 ? on[0] : q == 1 ? on[1] : q == 2 ? on[2] : on[3];
      if (!mine) continue;
      const int i = i0 + 32 * q + lane;
      const size_t f = row + i;
      const float area = face_area(P, d, i, j, k);
      const float rhof = face_rho(P, d, i, j, k);
      const int pd = d == 0 ? i : (d == 1 ? j : k);
      if (area != 0.0f && rhof != 0.0f) {
        if (pd == 0 || pd == nd) {
          vel[f] = svel ? svel[f] : 0.0f;
        } else {
          auto pread = [&](int ci, int cj, int ck) -> float {
            const long long t = (long long)(ci >> SHKZ_LOG_T) +
                                (long long)G.bx * ((long long)(cj >> SHKZ_LOG_T) + (long long)G.by * (ck >> SHKZ_LOG_T));
            const int pt = tile_state[t];
            if (pt < 0) return 0.0f;
            return pressure_pool[(size_t)pt * SHKZ_TC + (ci & 7) + 8 * (cj & 7) + 64 * (ck & 7)];
          };
          const float p1 = pread(i, j, k);
          const float p0 = pread(i - (d == 0), j - (d == 1), k - (d == 2));
          const float diff = p1 - p0;
          const float value = (float)(dt * (double)diff / ((double)rhof * dx));
          vel[f] = vel[f] - value;
        }
        if (P.density[d]) {
          const float scale = (float)(1.0 - (1.0 - (double)area) * (double)P.density[d][f]);
          vel[f] = scale * vel[f];
        }
      } else {
        vel[f] = 0.0f;
        vact[f] = 0;
      }
    }
  }
}

__global__ void __launch_bounds__(256, 8) k_velocity_update(FaceParams P, Geometry G, const int *flags,
                                                         const int *tile_state, const float *pressure_pool, double dx,
                                                         double dt, FaceFields F) {
  P.fluid_exists = (*flags) & 1;
  P.solid_exists = P.solid ? (((*flags) >> 1) & 1) : 0;
  const int d = blockIdx.y, fh = G.ny + (d == 1), fd = G.nz + (d == 2);
  const unsigned rows = (unsigned)((long long)fh * fd > 0 ? (long long)fh * fd : 0);
  const unsigned step = gridDim.x * (blockDim.x >> 5);
  for (unsigned r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += step) {
    const int j = (int)(r % (unsigned)fh), k = (int)(r / (unsigned)fh);
    if (d == 0) update_row<0>(P, G, tile_state, pressure_pool, F.svel[0], dx, dt, F.vel[0], F.vact[0], j, k);
    else if (d == 1) update_row<1>(P, G, tile_state, pressure_pool, F.svel[1], dx, dt, F.vel[1], F.vact[1], j, k);
    else update_row<2>(P, G, tile_state, pressure_pool, F.svel[2], dx, dt, F.vel[2], F.vact[2], j, k);
  }
}

// ---------------------------------------------------------------------------
// Surface tension (macpressuresolver3.cpp:98-128): curvature as the 7-point
// Laplacian of the liquid level set with clamped neighbours, then every active
// face with 0 < rho < 1 gets u += -sgn*dt/(dx*rho)*kappa*kappa_face, the face
// curvature interpolated by the liquid fraction.
__global__ void k_curvature(FaceParams P, double dx, float *curv) {
  const size_t n = (size_t)P.nx * P.ny * P.nz;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(c % P.nx), j = (int)((c / P.nx) % P.ny), k = (int)(c / ((size_t)P.nx * P.ny));
    auto f = [&](int a, int b, int e) -> float {
      a = min(max(a, 0), P.nx - 1);
      b = min(max(b, 0), P.ny - 1);
      e = min(max(e, 0), P.nz - 1);
      return P.fluid[cidx(P, a, b, e)];
    };
    // the six neighbours are summed in FP32, as the reference's float operands are
    const float s6 = f(i - 1, j, k) + f(i + 1, j, k) + f(i, j - 1, k) + f(i, j + 1, k) + f(i, j, k - 1) + f(i, j, k + 1);
    const double value = ((double)s6 - 6.0 * (double)P.fluid[c]) / (dx * dx);
    curv[c] = (float)value;
  }
}

__global__ void k_surface_tension(FaceParams P, Geometry G, const int *flags, int d, const float *curv, double kappa,
                                  double dx, double dt, float *vel, const uint8_t *vact) {
  P.fluid_exists = (*flags) & 1;
  P.solid_exists = P.solid ? (((*flags) >> 1) & 1) : 0;
  const int fw = G.nx + (d == 0), fh = G.ny + (d == 1), fd = G.nz + (d == 2);
  const size_t nf = (size_t)fw * fh * fd;
  for (size_t f = blockIdx.x * (size_t)blockDim.x + threadIdx.x; f < nf; f += (size_t)gridDim.x * blockDim.x) {
    if (!vact[f]) continue;
    const int i = (int)(f % fw), j = (int)((f / fw) % fh), k = (int)(f / ((size_t)fw * fh));
    const double rho = (double)face_rho(P, d, i, j, k);
    if (rho != 0.0 && rho < 1.0) {
      const int ci = min(i, G.nx - 1), cj = min(j, G.ny - 1), ck = min(k, G.nz - 1);
      const int bi = max(i - (d == 0), 0), bj = max(j - (d == 1), 0), bk = max(k - (d == 2), 0);
      const size_t c1 = cidx(P, ci, cj, ck), c0 = cidx(P, min(bi, G.nx - 1), min(bj, G.ny - 1), min(bk, G.nz - 1));
      const double sgn = P.fluid[c1] < 0.0f ? -1.0 : 1.0;
      const double theta = sgn < 0 ? 1.0 - rho : rho;
      const double face_c = theta * (double)curv[c1] + (1.0 - theta) * (double)curv[c0];
      const float inc = (float)(-sgn * dt / (dx * rho) * kappa * face_c);
      vel[f] = vel[f] + inc;
    }
  }
}

// Dense pressure grid (FP32, 0 outside unknowns) from the pool.
__global__ void __launch_bounds__(256) k_scatter_pressure(Geometry G, const int *tile_state,
                                                          const float *pressure_pool, const uint8_t *unk,
                                                          float *pressure, uint8_t *pressure_active) {
  const int sx = (G.bx + kStripTiles - 1) / kStripTiles;
  const int b = blockIdx.x, s0 = b % sx * kStripTiles, tj = b / sx % G.by, tk = b / sx / G.by;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = s0 * SHKZ_T + lane, k = tk * SHKZ_T + warp;
  if (i >= G.nx || k >= G.nz) return;
  const int pt = tile_state[s0 + (lane >> 3) + (long long)G.bx * (tj + (long long)G.by * tk)];
  size_t c = (size_t)i + (size_t)G.nx * ((size_t)(tj * SHKZ_T) + (size_t)G.ny * k);
  #pragma unroll
  for (int y = 0; y < SHKZ_T; ++y, c += G.nx) {
    if (tj * SHKZ_T + y >= G.ny) break;
    const uint8_t on = pt >= 0 ? unk[c] : 0;  // a tile outside the pool holds no unknown
    if (pressure) pressure[c] = on ? pressure_pool[(size_t)pt * SHKZ_TC + (lane & 7) + 8 * y + 64 * warp] : 0.0f;
    if (pressure_active) pressure_active[c] = on;
  }
}

// ---------------------------------------------------------------------------
// host launchers

static FaceParams make_params(const AssemblyInputs &in) {
  FaceParams P;
  P.solid = in.solid;
  P.solid_active = in.solid_active;
  P.fluid = in.fluid;
  P.nx = in.G.nx;
  P.ny = in.G.ny;
  P.nz = in.G.nz;
  P.solid_exists = 0;
  P.fluid_exists = 0;
  P.eps_solid = in.eps_solid;
  P.eps_fluid = in.eps_fluid;
  P.second_order_fluid = in.second_order_fluid;
  P.second_order_solid = in.second_order_solid;
  for (int d = 0; d < 3; ++d) P.density[d] = in.density[d];
  return P;
}

void launch_label(const AssemblyInputs &in, int *flags, uint8_t *unk, int *tile_count, cudaStream_t s) {
  const size_t ncell = (size_t)in.G.nx * in.G.ny * in.G.nz;
  const size_t nnode = (size_t)(in.G.nx + 1) * (in.G.ny + 1) * (in.G.nz + 1);
  cudaMemsetAsync(flags, 0, sizeof(int), s);
  count_launches(1);
  // four cells a thread, up to what fills the chip
  const unsigned blocks = (unsigned)std::min<size_t>(148 * 8, ncell / 1024 + 1);
  k_levelset_exist<<<blocks, 256, 0, s>>>(in.fluid, in.fluid_active, ncell, in.solid, in.solid_active, nnode, flags);
  count_launches(1);
  k_label<<<(unsigned)strip_count(in.G), 256, 0, s>>>(make_params(in), in.G, flags, unk, tile_count);
}

void launch_coeff(const AssemblyInputs &in, const int *flags, const int *pool_tile, int K, const uint8_t *unk,
                  const CoeffOutputs &out, cudaStream_t s) {
  if (K <= 0) return;
  count_launches(1);
  k_coeff<<<K, 256, 0, s>>>(make_params(in), in.G, flags, pool_tile, unk, in.vel[0], in.vel[1], in.vel[2],
                             in.svel[0], in.svel[1], in.svel[2], in.dx, in.dt, out.diag, out.offx, out.offy, out.offz,
                             out.diag64, out.offx64, out.offy64, out.offz64, out.rhs64, in.rhs_add);
}

void launch_surface_tension(const AssemblyInputs &in, const int *flags, float *curv, double kappa, float *const vel[3],
                            const uint8_t *const vact[3], cudaStream_t s) {
  count_launches(1);
  k_curvature<<<148 * 16, 256, 0, s>>>(make_params(in), in.dx, curv);
  for (int d = 0; d < 3; ++d) {
    count_launches(1);
    k_surface_tension<<<148 * 16, 256, 0, s>>>(make_params(in), in.G, flags, d, curv, kappa, in.dx, in.dt, vel[d],
                                               vact[d]);
  }
}

void launch_velocity_update(const AssemblyInputs &in, const int *flags, const int *tile_state,
                            const float *pressure_pool, float *const vel[3], uint8_t *const vact[3], cudaStream_t s) {
  FaceFields F;
  for (int d = 0; d < 3; ++d) {
    F.svel[d] = in.svel[d];
    F.vel[d] = vel[d];
    F.vact[d] = vact[d];
  }
  count_launches(1);
  const long long rows = std::max((long long)(in.G.ny + 1) * in.G.nz, (long long)in.G.ny * (in.G.nz + 1));
  k_velocity_update<<<dim3((unsigned)std::min((rows + 7) / 8, 1ll << 20), 3), 256, 0, s>>>(make_params(in), in.G, flags, tile_state, pressure_pool, in.dx, in.dt,
                                                     F);
}

void launch_scatter_pressure(const Geometry &G, const int *tile_state, const float *pressure_pool, const uint8_t *unk,
                             float *pressure, uint8_t *pressure_active, cudaStream_t s) {
  count_launches(1);
  k_scatter_pressure<<<(unsigned)strip_count(G), 256, 0, s>>>(G, tile_state, pressure_pool, unk, pressure, pressure_active);
}

}  // namespace shkz
