// MIC(0) sweeps over x-pencils of 16^3 macro tiles.
//
// The recurrences are those of solver.cu's 8^3-tile kernels,
//   t_j = d_j (r_j + sum_{lower} w t)     (forward, x, y, z ascending)
//   z_j = t_j + d_j sum_{upper} w z       (backward, descending)
// with the same order of operations per cell, so both layouts give the same
// bits. What bounds them is the chain of dependent cells, so the work is cut
// to make that chain short:
//
// * A CTA owns a pencil: a run of macro tiles that follow one another along x
//   (16 x 16 cells across). It streams through x without stopping at tile
//   borders, so a hand-off between CTAs happens only along y and z, and the
//   skewed start of the wavefront is paid once per pencil, not once per tile.
// * One warp, the solver, does the recurrence. Lane (by, bz) = (lane >> 2,
//   lane & 3) holds a column of 2 x 4 cells (y = 2 by, +1, z = 4 bz .. +3) and
//   advances one x a step, by + bz steps behind lane 0. The -x values are its
//   own registers, the -y / -z values come from lanes - 4 and - 1 by shuffle,
//   and no barrier is needed. A step is bound by that dependency chain
//   (shuffle, four z-cells, a y-cell) and by the warp's own issue rate; z is
//   the long side of a lane's block because the z term is the last of a
//   cell's sum and so the shortest way through it.
// * Everything else is done by other warps around it: coefficients arrive by
//   bulk copies from an array laid out in the solver's order (k_pencil_coefs),
//   the residual is updated and transposed into shared memory by eight loader
//   warps, two poller warps fetch the upstream faces, and the forward result
//   leaves by bulk copies. They meet in a ring of units (4 x-planes of the
//   pencil) through mbarriers.
// * A face value is its own flag: the words hold a bit pattern no arithmetic
//   produces until the solver lane stores the value, in the step that computes
//   it, and the consumer puts the pattern back. Face rows follow the solver's
//   steps, not the x-planes: row s of a pencil's +y face holds, for z-block bz,
//   plane s - bz, which the upstream lane computes 7 steps after it computed
//   row s - 7's first, and which the downstream lane needs in step s (and the
//   +z face with by in place of bz, 3 steps). So a downstream pencil trails by
//   7 (or 3) steps, one unit and one trip through L2, not by the whole skew.
//
// CTAs take pencils in level order (y + z of the macro tiles) from an atomic
// counter and wait only for pencils with an earlier number, which running CTAs
// hold, so every wait ends; all are bounded anyway.
//
// Measured on a B200 against a CTA per macro tile with a barrier per diagonal
// and whole-tile hand-offs (same values): sweep pair on a full 256 x 128 x 256
// grid, 8.4 M cells, 246 us against 341 us, 256^3 340 against 526 us; a hop
// between pencils takes 2.1 (z) and 2.7 us (y), of which the trip through L2 is
// 1.2, and a step 153 ns, set by the solver's instructions (10 shared loads, 6
// shuffles, 32 multiply-adds). Tried: 4 x 2 blocks with plane-wise faces (3.95 us
// a hop), tagged 64-bit face words, fences or branches in the solver's loop
// (each 60 - 200 ns a step).
#include "common.cuh"
#include "kernels.h"
#include "solver.h"
#include "wave.cuh"
#include <math_constants.h>
#include <type_traits>

namespace shkz {

namespace {

constexpr int NU = 10;              // units in the ring: the skewed lanes use 4, the others are on their way
constexpr int UX = 4;               // x-planes of a unit
constexpr int ROWS = NU * UX;       // x-planes of the ring
// One x-plane in the ring: coefficients [field 4][y 2][lane 32][z 4], then the
// right-hand side (and the result in its place) [y 2][lane 32][z 4], then 12
// floats that make the plane stride 3 (mod 8) 16-byte banks: lanes by + bz
// planes apart then read 16 bytes each without a conflict.
constexpr int CROW = 1024, RROW = kPencilRow;
constexpr int ROW = CROW + RROW + 12;
constexpr int CUNIT = UX * CROW, RUNIT = UX * RROW;
constexpr int NG = 8;               // units of upstream face rows in their ring
constexpr int GROW = 32;            // floats of a face row: [z 16] of the y face, [y 16] of the z face
constexpr int PREFETCH = 6;         // units ahead of a copy into the ring that L2 is told of
constexpr int SEGQ = 16;            // pencils known ahead (a pencil has >= 4 units, the roles are < 2 NU units apart)
constexpr int REDS = 8;             // macro tiles whose sums may be under way (the ring holds fewer)
constexpr int NWARPS = 12;           // three to a sub-partition, so that the solver may have 168 registers
constexpr int NTHREADS = NWARPS * 32;

// Warps share an SM sub-partition when their numbers agree mod 4: the solver's
// (0) holds only warps that wait most of the time.
constexpr int W_SOLVE = 0, W_COPY = 4, W_POLL0 = 8, W_POLL1 = 11;
// index 0..7 of a loader / storer warp, -1 for the others
__device__ __forceinline__ int mover_index(int warp) {
  return (warp >= 1 && warp <= 3) ? warp - 1 : (warp >= 5 && warp <= 7) ? warp - 2 : (warp == 9 || warp == 10) ? warp - 3 : -1;
}

struct __align__(128) Smem {
  float ring[ROWS * ROW];
  float ghost[NG * UX * GROW];
  double red[REDS][2][8];
  double fin[NWARPS];
  int4 seg[SEGQ];                      // first macro tile, macro tiles, slot
  // per unit: coefficients and right-hand side in, solved, slot free; face rows in, used
  unsigned long long full[NU], empty[NU], freed[NU], gfull[NG], gempty[NG], segfull[SEGQ];
  int arrived[REDS];
  int limit, skip, dead;
  long long patience;                  // clocks of a wait inside the CTA
};

static_assert(sizeof(Smem) <= 227 * 1024, "the ring fits one CTA's shared memory");

__device__ __forceinline__ uint32_t su32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mb_init(unsigned long long *b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mb_arrive(unsigned long long *b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(b)) : "memory");
}
__device__ __forceinline__ void mb_expect(unsigned long long *b, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(b)), "r"(bytes) : "memory");
}
// Bounded wait for the phase with this parity. The roles wait for one another
// inside the CTA and, in the end, for its pollers, whose rounds (0.24 us, 470
// clocks each) are bounded by the configured limit. This limit is several times
// theirs, and 4 s at least, so it is not met; if it were, the sweep reports its
// error, the CTA's remaining waits return at once, and it loads nothing more.
constexpr long long kWaitClocks = 1ll << 33;
constexpr int kWaitClocksPerRound = 1 << 12;
__device__ __forceinline__ bool mb_try(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(a), "r"(parity)
      : "memory");
  return ok;
}
__device__ __forceinline__ void mb_wait(Smem &sm, unsigned long long *b, uint32_t parity, WaveSync *ws) {
  const uint32_t a = su32(b);
  if (mb_try(a, parity)) return;
  const long long t0 = clock64();
  while (!mb_try(a, parity)) {
    if (*(volatile int *)&sm.dead) return;
    if (clock64() - t0 > *(volatile long long *)&sm.patience) {
      *(volatile int *)&sm.dead = 1;
      atomicCAS(&ws->error, 0, 1);
      return;
    }
  }
}
// Whether that phase is complete, asked ahead of the wait so that the answer
// arrives while the caller computes.
__device__ __forceinline__ bool mb_test(unsigned long long *b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(su32(b)), "r"(parity)
      : "memory");
  return ok;
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, int bytes, unsigned long long *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(su32(dst)),
               "l"(src), "r"(bytes), "r"(su32(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_prefetch(const void *src, int bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_store(void *dst, const void *src, int bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
               "r"(su32(src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_read_done() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_all_done() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// A face word not yet written: a NaN that no arithmetic result has (those are
// 0x7fffffff).
constexpr unsigned kUnset = 0xffffffffu;
__device__ __forceinline__ bool is_set(float v) { return __float_as_uint(v) != kUnset; }
__device__ __forceinline__ bool is_set(float4 v) { return is_set(v.x) && is_set(v.y) && is_set(v.z) && is_set(v.w); }
// OFF: bytes
template <int OFF>
__device__ __forceinline__ void put2(float *p, float a, float b) {
  asm volatile("st.relaxed.gpu.global.v2.f32 [%0+%1], {%2, %3};" ::"l"(p), "n"(OFF), "f"(a), "f"(b) : "memory");
}
template <int OFF>
__device__ __forceinline__ void put4(float *p, float4 v) {
  asm volatile("st.relaxed.gpu.global.v4.f32 [%0+%1], {%2, %3, %4, %5};" ::"l"(p), "n"(OFF), "f"(v.x), "f"(v.y), "f"(v.z),
               "f"(v.w)
               : "memory");
}
__device__ __forceinline__ float4 get4(const float *p) {
  float4 v;
  asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p)
               : "memory");
  return v;
}

__device__ __forceinline__ float2 get2(const float *p) {
  float2 v;
  asm volatile("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool is_set(float2 v) { return is_set(v.x) && is_set(v.y); }

// Position of a role in a ring of N units: the unit's slot and the parity of its use.
template <int N>
struct RingOf {
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next(int n = 1) {
    slot += n;
    if (slot >= N) { slot -= N; phase ^= 1u; }
  }
};
using Ring = RingOf<NU>;

// Prologue shared by the sweeps: barriers, wait limit.
// False: the solve has stopped, nothing to do.
__device__ __forceinline__ bool begin(Smem &sm, WaveSync *ws, const SolverState *st, int full_count, int freed_count) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < NU; ++i) {
      mb_init(&sm.full[i], full_count);
      mb_init(&sm.empty[i], 1);
      mb_init(&sm.freed[i], freed_count);
    }
    for (int i = 0; i < NG; ++i) {
      mb_init(&sm.gfull[i], 1);
      mb_init(&sm.gempty[i], 1);
    }
    for (int i = 0; i < REDS; ++i) sm.arrived[i] = 0;
    for (int i = 0; i < SEGQ; ++i) mb_init(&sm.segfull[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async();
  }
  wait_for_previous();
  if (st && *(volatile const int *)&st->done) return false;
  if (threadIdx.x == 0) {
    sm.dead = 0;
    sm.limit = spin_rounds(ws);
    sm.patience = max(kWaitClocks, (long long)sm.limit * kWaitClocksPerRound);
    sm.skip = *((volatile int *)&ws->skip_publish);
  }
  __syncthreads();
  return true;
}

// The next pencil of this CTA for one role; false after the last.
__device__ __forceinline__ bool next_pencil(Smem &sm, int i, WaveSync *ws, int4 &info) {
  mb_wait(sm, &sm.segfull[i & (SEGQ - 1)], (uint32_t)(i / SEGQ) & 1u, ws);
  info = sm.seg[i & (SEGQ - 1)];
  return info.y > 0 && !*(volatile int *)&sm.dead;
}

// Scheduler (one thread): takes the CTA's next pencil number and shows it to
// the roles. Also returns it.
template <bool BACK>
__device__ __forceinline__ int4 take_pencil(Smem &sm, const PoolSystem &S, int i, WaveSync *ws, int nseg) {
  const int slot = atomicAdd(&ws->slot, 1);
  int4 info = make_int4(0, 0, slot, 0);
  if (slot < nseg) {
    const int2 g = S.seg[BACK ? nseg - 1 - slot : slot];
    info.x = g.x;
    info.y = g.y;
  }
  sm.seg[i & (SEGQ - 1)] = info;
  mb_arrive(&sm.segfull[i & (SEGQ - 1)]);
  return info;
}

// Poller p of two: every second pair of units of face rows, eight rows at a
// time, the other poller on the next pair meanwhile, so that the L2 round trips
// overlap. A lane fetches 16 bytes of its row's y face and 2 x 8 of its z
// face. The words read are unset again for the next sweep. Rows run to the
// last lane's last plane, in whole pairs of units.
template <bool BACK>
__device__ __forceinline__ void poll_faces(Smem &sm, const PoolSystem &S, float *faces, int p, WaveSync *ws) {
  const int lane = threadIdx.x & 31, sl = lane >> 2, part = lane & 3;
  const int limit = sm.limit;
  const float unset = __uint_as_float(kUnset);
  const float4 unset4 = make_float4(unset, unset, unset, unset);
  const float2 unset2 = make_float2(unset, unset);
  RingOf<NG> ring;
  ring.next(2 * p);
  int k = 2 * p;  // units before this one
  int4 info;
  for (int i = 0; next_pencil(sm, i, ws, info); ++i) {
    const int planes = 16 * info.y;
    // word of the face row that holds plane q of this pencil in block blk of
    // the neighbour across face nb (row q + its block's trail), or null
    auto source = [&](int q, int nb, int trail, int at) -> float * {
      if ((unsigned)q >= (unsigned)planes) return nullptr;
      const int mt = BACK ? info.x + info.y - 1 - (q >> 4) : info.x + (q >> 4);
      const int n = S.mnbr[mt * 6 + nb];
      if (n < 0) return nullptr;
      const int2 g = S.mseg[n];
      const int qn = 16 * (BACK ? g.x + g.y - 1 - n : n - g.x) + (q & 15);
      return faces + ((size_t)kFaceRows * g.x + qn + trail) * GROW + at;
    };
    for (int j = 0; j < info.y + 1; ++j, k += 4, ring.next(4)) {
      const int s = 16 * j + 8 * p + sl;  // the row, the step that needs it
      const int bz = part, b0 = 2 * part, b1 = 2 * part + 1;
      const int tz = BACK ? 3 - bz : bz, t0 = BACK ? 7 - b0 : b0, t1 = BACK ? 7 - b1 : b1;
      float *ey = source(s - tz, BACK ? NB_YP : NB_YM, tz, 4 * bz);
      float *e0 = source(s - t0, BACK ? NB_ZP : NB_ZM, t0, 16 + 2 * b0);
      float *e1 = source(s - t1, BACK ? NB_ZP : NB_ZM, t1, 16 + 2 * b1);
      if (k >= NG) {
        mb_wait(sm, &sm.gempty[ring.slot], ring.phase ^ 1u, ws);
        mb_wait(sm, &sm.gempty[ring.slot + 1], ring.phase ^ 1u, ws);
      }
      float4 y = ey ? unset4 : make_float4(0.f, 0.f, 0.f, 0.f);
      float2 z0 = e0 ? unset2 : make_float2(0.f, 0.f), z1 = e1 ? unset2 : make_float2(0.f, 0.f);
      float *dst = sm.ghost + ring.slot * (UX * GROW) + sl * GROW;
      auto tell = [&](int unit) {
        if ((lane >> 4) == unit) {
          *reinterpret_cast<float4 *>(dst + 4 * part) = y;
          *reinterpret_cast<float4 *>(dst + 16 + 4 * part) = make_float4(z0.x, z0.y, z1.x, z1.y);
        }
        __syncwarp();
        if (lane == 0) mb_arrive(&sm.gfull[ring.slot + unit]);
      };
      bool told = false, dead = false;
      for (int it = 1;; ++it) {
        const unsigned have = __ballot_sync(0xffffffffu, (is_set(y) && is_set(z0) && is_set(z1)) || dead);
        if (!told && (have & 0xffffu) == 0xffffu) {
          told = true;
          tell(0);
        }
        if (have == 0xffffffffu) break;
        if (!is_set(y)) y = get4(ey);
        if (!is_set(z0)) z0 = get2(e0);
        if (!is_set(z1)) z1 = get2(e1);
        // gave up, or another wait of this sweep has
        if (it >= limit || ((it & 255) == 0 && *((volatile int *)&ws->error))) {
          atomicCAS(&ws->error, 0, info.z + 1);
          dead = true;
        }
        dead = __any_sync(0xffffffffu, dead);
        if (it > 64) __nanosleep(32);  // far from its turn (the start of a pencil)
      }
      tell(1);
      if (ey) *reinterpret_cast<float4 *>(ey) = unset4;
      if (e0) *reinterpret_cast<float2 *>(e0) = unset2;
      if (e1) *reinterpret_cast<float2 *>(e1) = unset2;
    }
  }
}

// A solver lane's coefficients and right-hand side at one x-plane: y even (0)
// and odd (1), z ascending.
struct Plane {
  float4 d0, d1, x0, x1, y0, y1, z0, z1, r0, r1;
};
template <int OFF>
__device__ __forceinline__ float4 lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4+%5];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF>
__device__ __forceinline__ float2 lds2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2+%3];" : "=f"(v.x), "=f"(v.y) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF>
__device__ __forceinline__ void sts4(uint32_t a, float4 v) {
  asm volatile("st.shared.v4.f32 [%0+%1], {%2, %3, %4, %5};" ::"r"(a), "n"(OFF), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
// a: the lane's place in the plane
__device__ __forceinline__ void load_plane(uint32_t a, Plane &P) {
  P.x0 = lds4<1024>(a);
  P.r0 = lds4<4096>(a);
  P.y0 = lds4<2048>(a);
  P.z0 = lds4<3072>(a);
  P.d0 = lds4<0>(a);
  P.x1 = lds4<1536>(a);
  P.r1 = lds4<4608>(a);
  P.y1 = lds4<2560>(a);
  P.z1 = lds4<3584>(a);
  P.d1 = lds4<512>(a);
}

// The roundings of solver.cu's 8^3-tile sweeps, which both layouts share.
__device__ __forceinline__ float fwd_cell(float d, float r, float wx, float tx, float wy, float ty, float wz, float tz) {
  return d * __fmaf_rn(wz, tz, __fmaf_rn(wy, ty, __fmaf_rn(wx, tx, r)));
}
__device__ __forceinline__ float bwd_cell(float d, float t, float wx, float zx, float wy, float zy, float wz, float zz) {
  return __fmaf_rn(d, __fmaf_rn(wz, zz, __fmaf_rn(wx, zx, __fmul_rn(wy, zy))), t);
}

// The solver's state: the lane's last results and its place in the pencil.
struct Solver {
  float4 a, b;              // y even and odd, z ascending
  int q;                    // x-planes done (negative: not started)
  uint32_t at;              // shared-memory address of the lane's place in plane q
  float *fy, *fz;           // this trip's words of the lane's y and z face
  bool ey, ez;              // the lane takes its y / z neighbours from the upstream faces
  bool py, pz;              // and publishes its own
};

// One step (the T-th of a trip) on the plane in P, the next one's into N.
// EDGE: some lanes are before the first or after the last plane.
template <bool BACK, bool EDGE, int T>
__device__ __forceinline__ void solve_step(Solver &L, const Plane &P, Plane &N, float4 gy, float2 gz, uint32_t end,
                                           int planes) {
  const bool on = !EDGE || (unsigned)L.q < (unsigned)planes;
  float4 ty;
  float tz0, tz1;
  if (!BACK) {
    tz0 = __shfl_up_sync(0xffffffffu, L.a.w, 1);
    tz1 = __shfl_up_sync(0xffffffffu, L.b.w, 1);
    ty.x = __shfl_up_sync(0xffffffffu, L.b.x, 4);
    ty.y = __shfl_up_sync(0xffffffffu, L.b.y, 4);
    ty.z = __shfl_up_sync(0xffffffffu, L.b.z, 4);
    ty.w = __shfl_up_sync(0xffffffffu, L.b.w, 4);
  } else {
    tz0 = __shfl_down_sync(0xffffffffu, L.a.x, 1);
    tz1 = __shfl_down_sync(0xffffffffu, L.b.x, 1);
    ty.w = __shfl_down_sync(0xffffffffu, L.a.w, 4);
    ty.z = __shfl_down_sync(0xffffffffu, L.a.z, 4);
    ty.y = __shfl_down_sync(0xffffffffu, L.a.y, 4);
    ty.x = __shfl_down_sync(0xffffffffu, L.a.x, 4);
  }
  uint32_t next = L.at + ROW * 4;
  if (next >= end) next -= ROWS * ROW * 4;
  load_plane(next, N);
  tz0 = L.ez ? gz.x : tz0;
  tz1 = L.ez ? gz.y : tz1;
  ty.x = L.ey ? gy.x : ty.x;
  ty.y = L.ey ? gy.y : ty.y;
  ty.z = L.ey ? gy.z : ty.z;
  ty.w = L.ey ? gy.w : ty.w;
  float4 a, b;
  if (!BACK) {
    a.x = fwd_cell(P.d0.x, P.r0.x, P.x0.x, L.a.x, P.y0.x, ty.x, P.z0.x, tz0);
    a.y = fwd_cell(P.d0.y, P.r0.y, P.x0.y, L.a.y, P.y0.y, ty.y, P.z0.y, a.x);
    a.z = fwd_cell(P.d0.z, P.r0.z, P.x0.z, L.a.z, P.y0.z, ty.z, P.z0.z, a.y);
    a.w = fwd_cell(P.d0.w, P.r0.w, P.x0.w, L.a.w, P.y0.w, ty.w, P.z0.w, a.z);
    b.x = fwd_cell(P.d1.x, P.r1.x, P.x1.x, L.b.x, P.y1.x, a.x, P.z1.x, tz1);
    b.y = fwd_cell(P.d1.y, P.r1.y, P.x1.y, L.b.y, P.y1.y, a.y, P.z1.y, b.x);
    b.z = fwd_cell(P.d1.z, P.r1.z, P.x1.z, L.b.z, P.y1.z, a.z, P.z1.z, b.y);
    b.w = fwd_cell(P.d1.w, P.r1.w, P.x1.w, L.b.w, P.y1.w, a.w, P.z1.w, b.z);
  } else {
    b.w = bwd_cell(P.d1.w, P.r1.w, P.x1.w, L.b.w, P.y1.w, ty.w, P.z1.w, tz1);
    b.z = bwd_cell(P.d1.z, P.r1.z, P.x1.z, L.b.z, P.y1.z, ty.z, P.z1.z, b.w);
    b.y = bwd_cell(P.d1.y, P.r1.y, P.x1.y, L.b.y, P.y1.y, ty.y, P.z1.y, b.z);
    b.x = bwd_cell(P.d1.x, P.r1.x, P.x1.x, L.b.x, P.y1.x, ty.x, P.z1.x, b.y);
    a.w = bwd_cell(P.d0.w, P.r0.w, P.x0.w, L.a.w, P.y0.w, b.w, P.z0.w, tz0);
    a.z = bwd_cell(P.d0.z, P.r0.z, P.x0.z, L.a.z, P.y0.z, b.z, P.z0.z, a.w);
    a.y = bwd_cell(P.d0.y, P.r0.y, P.x0.y, L.a.y, P.y0.y, b.y, P.z0.y, a.z);
    a.x = bwd_cell(P.d0.x, P.r0.x, P.x0.x, L.a.x, P.y0.x, b.x, P.z0.x, a.y);
  }
  if (on) {
    L.a = a;
    L.b = b;
    sts4<4096>(L.at, a);
    sts4<4608>(L.at, b);
  }
  if (L.py && on) put4<T * GROW * 4>(L.fy, BACK ? a : b);
  if (L.pz && on) put2<T * GROW * 4>(L.fz, BACK ? a.x : a.w, BACK ? b.x : b.w);
  ++L.q;
  L.at = next;
}

template <bool BACK>
__device__ __forceinline__ void solve_pencils(Smem &sm, float *faces, WaveSync *ws) {
  const int lane = threadIdx.x & 31, by = lane >> 2, bz = lane & 3;
  const int ty = BACK ? 7 - by : by, tz = BACK ? 3 - bz : bz, off = ty + tz;
  const int skip = BACK ? 0 : sm.skip;
  const uint32_t base = su32(sm.ring) + 16 * lane, end = base + ROWS * ROW * 4;
  const uint32_t gya = su32(sm.ghost) + 16 * bz, gza = su32(sm.ghost) + 64 + 8 * by;
  int slot0 = 0;           // slot of the pencil's first unit
  Ring fr, er;             // units awaited, units done
  RingOf<NG> gr;           // face rows awaited
  int4 info;
  for (int i = 0; next_pencil(sm, i, ws, info); ++i) {
    const int planes = 16 * info.y, groups = planes / 4;
    Solver L;
    L.a = L.b = make_float4(0.f, 0.f, 0.f, 0.f);
    L.q = -off;
    int row = slot0 * UX - off;
    if (row < 0) row += ROWS;
    L.at = base + row * (ROW * 4);
    L.fy = faces + ((long long)kFaceRows * info.x - off + tz) * GROW + 4 * bz;
    L.fz = faces + ((long long)kFaceRows * info.x - off + ty) * GROW + 16 + 2 * by;
    L.ey = by == (BACK ? 7 : 0);
    L.ez = bz == (BACK ? 3 : 0);
    L.py = skip != info.z + 1 && by == (BACK ? 0 : 7);
    L.pz = skip != info.z + 1 && bz == (BACK ? 0 : 3);
    mb_wait(sm, &sm.full[fr.slot], fr.phase, ws);
    fr.next();
    Plane P, N;
    load_plane(L.at, P);
    // one unit a trip; the skewed lanes end 10 (< 12) steps after lane 0. The
    // first and last three trips, where lanes start and stop, are loops of
    // their own, so that the main one is free of branches.
    bool ready = false;
    auto trip = [&](auto edge, int g) {
      constexpr bool EDGE = decltype(edge)::value;
      if (!ready) mb_wait(sm, &sm.gfull[gr.slot], gr.phase, ws);
      // the trip's last step loads the next unit's first plane
      if (!EDGE || g < 3 ? g + 1 < groups : false) {
        mb_wait(sm, &sm.full[fr.slot], fr.phase, ws);
        fr.next();
      }
      const uint32_t go = gr.slot * (UX * GROW * 4);
      const float4 y0 = lds4<0>(gya + go), y1 = lds4<128>(gya + go), y2 = lds4<256>(gya + go), y3 = lds4<384>(gya + go);
      const float2 z0 = lds2<0>(gza + go), z1 = lds2<128>(gza + go), z2 = lds2<256>(gza + go), z3 = lds2<384>(gza + go);
      const int used = gr.slot;
      gr.next();
      ready = mb_test(&sm.gfull[gr.slot], gr.phase);
      solve_step<BACK, EDGE, 0>(L, P, N, y0, z0, end, planes);
      solve_step<BACK, EDGE, 1>(L, N, P, y1, z1, end, planes);
      solve_step<BACK, EDGE, 2>(L, P, N, y2, z2, end, planes);
      solve_step<BACK, EDGE, 3>(L, N, P, y3, z3, end, planes);
      L.fy += UX * GROW;
      L.fz += UX * GROW;
      __syncwarp();
      if (lane == 0) {
        mb_arrive(&sm.gempty[used]);
        // after trip u + 3 every lane has left unit u (step 4 u + 3 + 10)
        if (!EDGE || g >= 3) mb_arrive(&sm.empty[er.slot]);
      }
      if (!EDGE || g >= 3) er.next();
    };
    int g = 0;
    for (; g < 3; ++g) trip(std::true_type{}, g);
    for (; g < groups; ++g) trip(std::false_type{}, g);
    for (; g < groups + 3; ++g) trip(std::true_type{}, g);
    // rows come in pairs of units: one more than the trips
    if (!ready) mb_wait(sm, &sm.gfull[gr.slot], gr.phase, ws);
    if (lane == 0) mb_arrive(&sm.gempty[gr.slot]);
    gr.next();
    slot0 = er.slot;
  }
}

// Mover thread v (0..127) of half a macro tile (a pair of units) holds four
// x-cells of one row in each of the half's four pool tiles (i = y half + 2 z
// half). Ring offset of its cell on plane 4 (v & 1) + e of the pair:
__device__ __forceinline__ int rt_offset(int v, int i, int e) {
  const int y = ((v >> 1) & 7) + 8 * (i & 1), z = (v >> 4) + 8 * (i >> 1);
  return e * ROW + CROW + (y & 1) * 128 + ((z >> 2) + 4 * (y >> 1)) * 4 + (z & 3);
}
// The four cells are written (read) in an order turned by the row's y / 2, so
// that the warp's accesses fall on four planes at a time: two cells a bank
// instead of four.
__device__ __forceinline__ void to_ring(float *pair, int v, int i, float4 w) {
  const int t = (v >> 2) & 3;
  if (t & 1) w = make_float4(w.y, w.z, w.w, w.x);
  if (t & 2) w = make_float4(w.z, w.w, w.x, w.y);
  float *p = pair + (v & 1) * (UX * ROW);
  p[rt_offset(v, i, t)] = w.x;
  p[rt_offset(v, i, (t + 1) & 3)] = w.y;
  p[rt_offset(v, i, (t + 2) & 3)] = w.z;
  p[rt_offset(v, i, (t + 3) & 3)] = w.w;
}
// unit: of the backward ring, where planes descend
__device__ __forceinline__ float4 from_ring(const float *unit, int v, int i) {
  const int t = (v >> 2) & 3;
  float4 w;
  w.x = unit[rt_offset(v, i, 3 - t)];
  w.y = unit[rt_offset(v, i, 3 - ((t + 1) & 3))];
  w.z = unit[rt_offset(v, i, 3 - ((t + 2) & 3))];
  w.w = unit[rt_offset(v, i, 3 - ((t + 3) & 3))];
  if (t & 2) w = make_float4(w.z, w.w, w.x, w.y);
  if (t & 1) w = make_float4(w.w, w.x, w.y, w.z);
  return w;
}

// True in the last of the eight mover warps to bring its part of macro tile
// number n (of this CTA), which then adds the parts up in warp order, as one
// 256-thread block's sum does.
__device__ __forceinline__ bool last_mover(Smem &sm, int n) {
  __threadfence_block();
  int *c = &sm.arrived[n & (REDS - 1)];
  if (atomicAdd(c, 1) != 7) return false;
  *c = 0;
  __threadfence_block();
  return true;
}

__device__ __forceinline__ double warp_sum(double v) {
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ void finish_sweep(Smem &sm, WaveSync *ws) {
  if (threadIdx.x == 0) {
    if (sm.dead) {  // copies already issued land before the CTA's shared memory goes
      const long long t0 = clock64();
      while (clock64() - t0 < (1ll << 21)) {}
    }
    const unsigned f = atomicAdd(&ws->finished, 1u);
    if (f == gridDim.x - 1) {
      ws->slot = 0;
      ws->finished = 0;
    }
  }
}

}  // namespace

// Forward sweep. With fu.st the residual is updated on the way in
// (r -= alpha q, k_update_xr's arithmetic; its x update rides in the next
// stencil) and the last CTA does the iteration's convergence bookkeeping.
__global__ void __launch_bounds__(NTHREADS, 1) k_pencil_forward(PoolSystem S, const float *r,
                                                                WaveSync *ws, const SolverState *st, SweepUpdate fu) {
  extern __shared__ __align__(128) unsigned char raw[];
  Smem &sm = *reinterpret_cast<Smem *>(raw);
  if (!begin(sm, ws, st, 1 + 4, 1)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nseg = *S.nseg;
  const int mover = mover_index(warp);
  if (warp == W_SOLVE) {
    solve_pencils<false>(sm, S.mfaces_f, ws);
  } else if (warp == W_POLL0 || warp == W_POLL1) {
    poll_faces<false>(sm, S, S.mfaces_f, warp == W_POLL1, ws);
  } else if (warp == W_COPY) {
    if (lane == 0) {
      // coefficients in, results out: as a unit is done its result is stored
      // and its slot's coefficients replaced by those of the unit NU later
      Ring ring;
      int4 in = make_int4(0, 0, 0, 0), out;
      int taken = 0, u = 0;  // pencils taken, next unit of the last one
      bool more = true;
      auto load = [&](int slot) {
        if (u == 4 * in.y && more) {
          in = take_pencil<false>(sm, S, taken++, ws, nseg);
          u = 0;
          more = in.y > 0;
        }
        if (!more || *(volatile int *)&sm.dead) return;
        mb_expect(&sm.full[slot], CUNIT * 4);
        const float *src = S.coef_f + ((size_t)in.x * 4 + u) * CUNIT;
        for (int x = 0; x < UX; ++x)
          bulk_load(sm.ring + (slot * UX + x) * ROW, src + x * CROW, CROW * 4, &sm.full[slot]);
        if (u + PREFETCH < 4 * in.y) bulk_prefetch(src + PREFETCH * CUNIT, CUNIT * 4);
        ++u;
      };
      for (int i = 0; i < NU; ++i) load(i);
      for (int i = 0; next_pencil(sm, i, ws, out); ++i) {
        for (int v = 0; v < 4 * out.y; ++v, ring.next()) {
          mb_wait(sm, &sm.empty[ring.slot], ring.phase, ws);
          load(ring.slot);
          fence_async();  // the solver's stores, seen through the barrier, before the copy's reads
          for (int x = 0; x < UX; ++x)
            bulk_store(S.tp + ((size_t)out.x * 4 + v) * RUNIT + x * RROW, sm.ring + (ring.slot * UX + x) * ROW + CROW, RROW * 4);
          bulk_commit();
          bulk_read_done();
          mb_arrive(&sm.freed[ring.slot]);
        }
      }
      bulk_all_done();
    }
  } else if (mover >= 0) {
    const int h = mover >> 2, v = (mover & 3) * 32 + lane;
    const float alpha = fu.st ? (float)fu.st->alpha : 0.0f;
    Ring ring;
    ring.next(2 * h);
    int k = 2 * h, m2 = 0;
    int4 info;
    for (int i = 0; next_pencil(sm, i, ws, info); ++i) {
      int pt[4], pn[4];
      float4 rv[4], qv[4], rn[4], qn[4];
      auto subs = [&](int j, int *p) {
        #pragma unroll
        for (int a = 0; a < 4; ++a) p[a] = j < info.y ? __ldg(S.msub + (info.x + j) * 8 + h + 2 * a) : -1;
      };
      auto fetch = [&](const int *p, float4 *rr, float4 *qq) {
        #pragma unroll
        for (int a = 0; a < 4; ++a) {
          rr[a] = qq[a] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (p[a] >= 0) {
            const size_t b = (size_t)p[a] * (SHKZ_TC / 4) + v;
            rr[a] = reinterpret_cast<const float4 *>(r)[b];
            if (fu.st) qq[a] = reinterpret_cast<const float4 *>(fu.q)[b];
          }
        }
      };
      subs(0, pt);
      fetch(pt, rv, qv);
      subs(1, pn);
      for (int j = 0; j < info.y; ++j, k += 4, ring.next(4)) {
        // the next macro tile's loads are in flight while this one waits for its slot
        fetch(pn, rn, qn);
        int pnn[4];
        subs(j + 2, pnn);
        double m = 0.0, s2 = 0.0;
        if (fu.st) {
          #pragma unroll
          for (int a = 0; a < 4; ++a) {
            if (pt[a] < 0) continue;
            float4 &w = rv[a];
            w.x = __fmaf_rn(-alpha, qv[a].x, w.x);
            w.y = __fmaf_rn(-alpha, qv[a].y, w.y);
            w.z = __fmaf_rn(-alpha, qv[a].z, w.z);
            w.w = __fmaf_rn(-alpha, qv[a].w, w.w);
            reinterpret_cast<float4 *>(fu.r)[(size_t)pt[a] * (SHKZ_TC / 4) + v] = w;
            m = fmax(m, fmax(fmax(fabs((double)w.x), fabs((double)w.y)), fmax(fabs((double)w.z), fabs((double)w.w))));
            s2 += (double)w.x * w.x + (double)w.y * w.y + (double)w.z * w.z + (double)w.w * w.w;
          }
        }
        if (k >= NU) {
          mb_wait(sm, &sm.freed[ring.slot], ring.phase ^ 1u, ws);
          mb_wait(sm, &sm.freed[ring.slot + 1], ring.phase ^ 1u, ws);
        }
        #pragma unroll
        for (int a = 0; a < 4; ++a) to_ring(sm.ring + ring.slot * (UX * ROW), v, a, rv[a]);
        __syncwarp();
        if (lane == 0) {
          mb_arrive(&sm.full[ring.slot]);
          mb_arrive(&sm.full[ring.slot + 1]);
        }
        if (fu.st) {
          // norms of the macro tile, summed as one 256-thread block would
          m = warp_max(m);
          s2 = warp_sum(s2);
          if (lane == 0) {
            volatile double *rm = sm.red[m2 & (REDS - 1)][0], *rs = sm.red[m2 & (REDS - 1)][1];
            rm[mover] = m;
            rs[mover] = s2;
            if (last_mover(sm, m2)) {
              double mm = 0.0, ss = 0.0;
              for (int w = 0; w < 8; ++w) {
                mm = fmax(mm, rm[w]);
                ss += rs[w];
              }
              fu.part[info.x + j] = mm;
              fu.part[S.KM + info.x + j] = ss;
            }
          }
          ++m2;
        }
        #pragma unroll
        for (int a = 0; a < 4; ++a) {
          pt[a] = pn[a];
          pn[a] = pnn[a];
          rv[a] = rn[a];
          qv[a] = qn[a];
        }
      }
    }
  }
  __syncthreads();
  if (fu.st && last_block(fu.counter)) {
    // the convergence bookkeeping of k_update_xr, on the new residual
    double mm = 0.0, ss = 0.0;
    if (threadIdx.x < 256)
      for (int i = threadIdx.x; i < S.KM; i += 256) {
        mm = fmax(mm, fu.part[i]);
        ss += fu.part[S.KM + i];
      }
    mm = block_max<NTHREADS>(mm, sm.fin);
    ss = block_sum<NTHREADS>(ss, sm.fin);
    const bool nan = !(ss == ss);
    if (threadIdx.x == 0) {
      SolverState *sw = fu.st;
      sw->rmax = nan ? CUDART_NAN : mm;
      sw->r2 = ss;
      sw->iter += 1;
      sw->x_pending = 1;
      if (nan) { sw->done = 3; sw->status = -5; }
      else if (mm <= sw->tol_abs) sw->done = 1;
      else if (sw->iter >= fu.max_iterations) sw->done = 2;
      else if (mm < sw->ru_threshold) sw->done = 4;
      if (sw->done) report_progress(sw);  // otherwise the backward sweep does
      *fu.counter = 0;
    }
  }
  finish_sweep(sm, ws);
}

// Backward sweep with the fused z.r (r: the residual the forward sweep used);
// with finish the last CTA also turns the partials into rho and beta.
__global__ void __launch_bounds__(NTHREADS, 1) k_pencil_backward(PoolSystem S, const float *r, float *z,
                                                                 double *partials, WaveSync *ws,
                                                                 SolverState *st, unsigned *finish) {
  extern __shared__ __align__(128) unsigned char raw[];
  Smem &sm = *reinterpret_cast<Smem *>(raw);
  if (!begin(sm, ws, st, 1, 4)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nseg = *S.nseg;
  const int mover = mover_index(warp);
  if (warp == W_SOLVE) {
    solve_pencils<true>(sm, S.mfaces_b, ws);
  } else if (warp == W_POLL0 || warp == W_POLL1) {
    poll_faces<true>(sm, S, S.mfaces_b, warp == W_POLL1, ws);
  } else if (warp == W_COPY) {
    if (lane == 0) {
      Ring ring;
      int k = 0;
      for (int i = 0;; ++i) {
        const int4 info = take_pencil<true>(sm, S, i, ws, nseg);
        if (!info.y) break;
        for (int u = 4 * info.y - 1; u >= 0; --u, ++k, ring.next()) {
          if (k >= NU) mb_wait(sm, &sm.empty[ring.slot], ring.phase ^ 1u, ws);
          if (*(volatile int *)&sm.dead) continue;
          mb_expect(&sm.full[ring.slot], (CUNIT + RUNIT) * 4);
          const float *src = S.coef_b + ((size_t)info.x * 4 + u) * CUNIT;
          float *dst = sm.ring + ring.slot * (UX * ROW);
          // the ring is in processing order, x descending
          for (int x = 0; x < UX; ++x)
            bulk_load(dst + (UX - 1 - x) * ROW, src + x * CROW, CROW * 4, &sm.full[ring.slot]);
          if (u >= PREFETCH) bulk_prefetch(src - PREFETCH * CUNIT, CUNIT * 4);
          // the slot's z has been read out
          if (k >= NU) mb_wait(sm, &sm.freed[ring.slot], ring.phase ^ 1u, ws);
          for (int x = 0; x < UX; ++x)
            bulk_load(dst + (UX - 1 - x) * ROW + CROW, S.tp + ((size_t)info.x * 4 + u) * RUNIT + x * RROW, RROW * 4,
                      &sm.full[ring.slot]);
        }
      }
    }
  } else if (mover >= 0) {
    // group g stores the units of the x-halves 1 - g, the order they come in
    const int g = mover >> 2, h = 1 - g, v = (mover & 3) * 32 + lane;
    Ring ring;
    ring.next(2 * g);
    int m2 = 0;
    int4 info;
    for (int i = 0; next_pencil(sm, i, ws, info); ++i) {
      for (int j = 0; j < info.y; ++j, ring.next(4)) {
        const int mt = info.x + info.y - 1 - j;
        int pt[4];
        float4 rv[4];
        #pragma unroll
        for (int a = 0; a < 4; ++a) pt[a] = __ldg(S.msub + mt * 8 + h + 2 * a);
        #pragma unroll
        for (int a = 0; a < 4; ++a)
          rv[a] = (partials && pt[a] >= 0) ? reinterpret_cast<const float4 *>(r)[(size_t)pt[a] * (SHKZ_TC / 4) + v]
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
        mb_wait(sm, &sm.empty[ring.slot], ring.phase, ws);
        mb_wait(sm, &sm.empty[ring.slot + 1], ring.phase, ws);
        // x descends with the units: the pair's first slot holds planes 4..7
        float4 zv[4];
        #pragma unroll
        for (int a = 0; a < 4; ++a) zv[a] = from_ring(sm.ring + (ring.slot + 1 - (v & 1)) * (UX * ROW), v, a);
        fence_async();
        __syncwarp();
        if (lane == 0) {
          mb_arrive(&sm.freed[ring.slot]);
          mb_arrive(&sm.freed[ring.slot + 1]);
        }
        double dot = 0.0;
        #pragma unroll
        for (int a = 0; a < 4; ++a) {
          if (pt[a] < 0) continue;
          reinterpret_cast<float4 *>(z)[(size_t)pt[a] * (SHKZ_TC / 4) + v] = zv[a];
          dot += (double)zv[a].x * rv[a].x + (double)zv[a].y * rv[a].y + (double)zv[a].z * rv[a].z +
                 (double)zv[a].w * rv[a].w;
        }
        if (partials) {
          // z.r of the macro tile, summed as one 256-thread block would
          dot = warp_sum(dot);
          if (lane == 0) {
            volatile double *rs = sm.red[m2 & (REDS - 1)][0];
            rs[4 * h + (mover & 3)] = dot;
            if (last_mover(sm, m2)) {
              double s = 0.0;
              for (int w = 0; w < 8; ++w) s += rs[w];
              partials[mt] = s;
            }
          }
          ++m2;
        }
      }
    }
  }
  __syncthreads();
  if (finish && last_block(finish)) {
    // k_finish_rho of the PCG iteration: rho_new = z.r from the macro-tile
    // partials in tile order, beta = rho_new / rho
    double s = 0.0;
    if (threadIdx.x < 256)
      for (int i = threadIdx.x; i < S.KM; i += 256) s += partials[i];
    const double rho_new = block_sum<NTHREADS>(s, sm.fin);
    if (threadIdx.x == 0) {
      st->beta = rho_new / st->rho;
      st->rho = rho_new;
      report_progress(st);
      *finish = 0;
    }
  }
  finish_sweep(sm, ws);
}

// ---------------------------------------------------------------------------
// Coefficients in the solver's order: [macro tile][x 16][field 4][y 2][lane 32]
// float4 over z, fields d and the three lower weights (forward) or upper
// weights (backward: the lower weight of the +x/+y/+z neighbour cell, zero
// where that tile is not in the pool). Cells of absent tiles are zero. Once
// per factorisation, so that the sweeps' staging is plain bulk copies.
__global__ void __launch_bounds__(256) k_pencil_coefs(PoolSystem S, const float *__restrict__ d32,
                                                      float *__restrict__ cf, float *__restrict__ cb) {
  const int mt = blockIdx.x, x0 = 4 * blockIdx.y, lane = threadIdx.x & 31, j = threadIdx.x >> 5;
  const int field = j >> 1, y = 2 * (lane >> 2) + (j & 1), bz = lane & 3;
  const float *src = field == 0 ? d32 : field == 1 ? S.offx : field == 2 ? S.offy : S.offz;
  __shared__ int sub[8];
  if (threadIdx.x < 8) sub[threadIdx.x] = S.msub[mt * 8 + threadIdx.x];
  __syncthreads();
  for (int x = x0; x < x0 + 4; ++x) {
    float lo[4], up[4];
    #pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int z = 4 * bz + e;
      const int pt = sub[(x >> 3) + 2 * (y >> 3) + 4 * (z >> 3)];
      const int c = (x & 7) + 8 * (y & 7) + 64 * (z & 7);
      lo[e] = up[e] = 0.0f;
      if (pt < 0) continue;
      lo[e] = src[(size_t)pt * SHKZ_TC + c];
      if (field == 0) { up[e] = lo[e]; continue; }
      const int step = field == 1 ? 1 : field == 2 ? 8 : 64;
      const int at = field == 1 ? (x & 7) : field == 2 ? (y & 7) : (z & 7);
      int nb = pt, cell = c + step;
      if (at == 7) { nb = S.nbr[pt * 6 + 2 * (field - 1) + 1]; cell = c - 7 * step; }
      if (nb >= 0) up[e] = src[(size_t)nb * SHKZ_TC + cell];
    }
    const size_t o = (((size_t)mt * 16 + x) * 8 + j) * 32 + lane;
    reinterpret_cast<float4 *>(cf)[o] = make_float4(lo[0], lo[1], lo[2], lo[3]);
    reinterpret_cast<float4 *>(cb)[o] = make_float4(up[0], up[1], up[2], up[3]);
  }
}

// ---------------------------------------------------------------------------
// Pencils: runs of macro tiles along x. Macro tiles are numbered x fastest, so
// a run is a range of numbers; it starts where the -x neighbour is absent.
__global__ void k_pencil_count(Geometry M, const int *mtile, const int *mnbr, int KM, int *level_count) {
  const int mt = blockIdx.x * blockDim.x + threadIdx.x;
  if (mt >= KM || mnbr[mt * 6 + NB_XM] >= 0) return;
  const long long t = mtile[mt];
  atomicAdd(&level_count[(int)((t / M.bx) % M.by) + (int)(t / ((long long)M.bx * M.by))], 1);
}
__global__ void k_pencil_scan(int *level_count, int nlev, int *nseg) {
  const int n = warp_scan_counts(level_count, nlev);
  if (threadIdx.x == 0) *nseg = n;
}
__global__ void k_pencil_scatter(Geometry M, const int *mtile, const int *mnbr, int KM, int *cursor, int2 *seg,
                                 int2 *mseg) {
  const int mt = blockIdx.x * blockDim.x + threadIdx.x;
  if (mt >= KM || mnbr[mt * 6 + NB_XM] >= 0) return;
  int n = 1;
  while (mt + n < KM && mnbr[(mt + n) * 6 + NB_XM] == mt + n - 1) ++n;
  const long long t = mtile[mt];
  const int pos = atomicAdd(&cursor[(int)((t / M.bx) % M.by) + (int)(t / ((long long)M.bx * M.by))], 1);
  seg[pos] = make_int2(mt, n);
  for (int i = 0; i < n; ++i) mseg[mt + i] = make_int2(mt, n);
}

void build_pencils(const Geometry &M, const int *mtile, const int *mnbr, int KM, int *level_count, int2 *seg,
                   int2 *mseg, int *nseg, cudaStream_t s) {
  const int nlev = M.by + M.bz;
  cudaMemsetAsync(level_count, 0, sizeof(int) * (nlev + 1), s);
  count_launches(3);
  k_pencil_count<<<(KM + 255) / 256, 256, 0, s>>>(M, mtile, mnbr, KM, level_count);
  k_pencil_scan<<<1, 32, 0, s>>>(level_count, nlev, nseg);
  k_pencil_scatter<<<(KM + 255) / 256, 256, 0, s>>>(M, mtile, mnbr, KM, level_count, seg, mseg);
}

void launch_pencil_coefs(const PoolSystem &S, const float *d32, cudaStream_t s) {
  count_launches(1);
  // four x-planes a block: 16 as one block's work took 17 us however small the grid
  k_pencil_coefs<<<dim3(S.KM, 4), 256, 0, s>>>(S, d32, S.coef_f, S.coef_b);
}

// one CTA per SM (its ring takes the shared memory), no more than there may be pencils
static int pencil_grid(const PoolSystem &S) {
  static int sms[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  int n = dev >= 0 && dev < 64 ? sms[dev] : 0;
  if (!n) {
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    cudaFuncSetAttribute(k_pencil_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
    cudaFuncSetAttribute(k_pencil_backward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
    if (dev >= 0 && dev < 64) sms[dev] = n;
  }
  return S.KM < n ? S.KM : n;
}

void launch_pencil_sweeps(const PoolSystem &S, const float *r, float *z, double *partials, void *ws_f, void *ws_b,
                          const SolverState *st, const SweepUpdate &fu, unsigned *finish, cudaStream_t s) {
  const int grid = pencil_grid(S);
  count_launches(2);
  launch_overlapped(k_pencil_forward, grid, NTHREADS, sizeof(Smem), s, S, r, (WaveSync *)ws_f, st, fu);
  launch_overlapped(k_pencil_backward, grid, NTHREADS, sizeof(Smem), s, S, r, z, partials, (WaveSync *)ws_b,
                    const_cast<SolverState *>(st), finish);
}

}  // namespace shkz
