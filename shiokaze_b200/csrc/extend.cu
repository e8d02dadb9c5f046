// Velocity extension after a projection, as macliquid3::extend_both runs it
// (src/liquid/macliquid3.cpp:330-340): macarray_extrapolator3::extrapolate
// followed by macutility3::constrain_velocity.
//
// Built with -fmad=false: the reference's double expressions (trilinear
// weights, products added into FP32 sums, the normal projection) round after
// every operation, and so do these, so the results are bit-identical.
//
// Grids are dense, x fastest; a face component d has
// (nx + (d == 0)) x (ny + (d == 1)) x (nz + (d == 2)) entries with a uint8
// active mask; the solid level set is nodal, (nx+1) x (ny+1) x (nz+1), holding
// the values the reference's array3 returns for every node (active value,
// flood-fill value or background), with its active mask.
//
// The active masks and the solid's "not outside" nodes are packed into bits
// (flat, 32 faces or nodes a word), so that finding the few faces there is
// anything to do for costs 1/8 byte a face and pass instead of the byte masks
// and per-face arithmetic; what is left is one read of the byte masks and one
// of the solid. At 256^3 (50.5 M faces, width 3 + constraint, B200) a call
// took 1.43 ms with byte masks read 16 at a time, two launches a pass and
// component and the FP64 set-up on every active face, and takes 0.19 ms so.
#include "common.cuh"
#include "kernels.h"

namespace shkz {

// nonzero bytes of four into bits 0..3
__device__ __forceinline__ unsigned byte_bits(unsigned x) {
  return (((__vcmpne4(x, 0u) & 0x01010101u) * 0x01020408u) >> 24) & 0xfu;
}
__device__ __forceinline__ unsigned byte_bits(uint4 q) {
  return byte_bits(q.x) | (byte_bits(q.y) << 4) | (byte_bits(q.z) << 8) | (byte_bits(q.w) << 12);
}

// Byte masks of the three components into bits. The masks start 16-byte
// aligned (checked at the entry), a word's 32 bytes with them.
__global__ void __launch_bounds__(256) k_ext_pack(ExtendFields f) {
  const int d = blockIdx.y;
  const unsigned n = f.n[d], nw = (n + 31) / 32;
  const uint8_t *__restrict__ a = f.act[d];
  for (unsigned w = blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += gridDim.x * blockDim.x) {
    unsigned m = 0;
    if (32 * w + 32 <= n) {
      const uint4 *q = reinterpret_cast<const uint4 *>(a) + 2 * (size_t)w;
      m = byte_bits(q[0]) | (byte_bits(q[1]) << 16);
    } else {
      for (unsigned b = 0; 32 * w + b < n; ++b) m |= (a[32 * (size_t)w + b] ? 1u : 0u) << b;
    }
    f.bits[d][w] = m;
  }
}

// 32 bits from bit position at (any sign); zero outside the nw words.
__device__ __forceinline__ unsigned bits_at(const unsigned *__restrict__ b, long long at, unsigned nw) {
  // a position before 0 becomes a word number past the end
  const unsigned w = (unsigned)(at >> 5);
  const unsigned lo = w < nw ? b[w] : 0u, hi = w + 1u < nw ? b[w + 1u] : 0u;
  return __funnelshift_r(lo, hi, (unsigned)at & 31u);
}
// bits [lo, hi) of a word
__device__ __forceinline__ unsigned bit_range(int lo, int hi) {
  lo = max(lo, 0);
  hi = min(hi, 32);
  if (lo >= hi) return 0u;
  return (0xffffffffu >> (32 - (hi - lo))) << lo;
}

// One pass of array_extrapolator3::extrapolate
// (include/shiokaze/array/array_extrapolator3.h) through array3::dilate
// (src/array/dilate3.h): every inactive face with an active 6-neighbour in the
// state before the pass becomes active with the FP32 mean of its active
// neighbours, summed in the reference's query order (i+1, i-1, j+1, j-1, k-1,
// k+1). The state before the pass is the bit mask read; the one after it goes
// to the other mask. Values are read only where the former is set and written
// only where it is not, so the pass works in place. A thread looks at 32 faces
// and queues the new ones; the block then fills them in with all its threads
// (a word at a time, the loads of one word waited for those of the last: 27 us
// a pass at 256^3).
constexpr int kExtrapolateThreads = 128;
__global__ void __launch_bounds__(kExtrapolateThreads) k_extrapolate(ExtendFields f) {
  __shared__ unsigned queue[32 * kExtrapolateThreads];
  __shared__ uint8_t sides[32 * kExtrapolateThreads];  // active neighbours, in query order
  __shared__ int queued;
  const int d = blockIdx.y;
  const unsigned n = f.n[d], nw = (n + 31) / 32;
  const int W = f.W[d], H = f.H[d];
  const unsigned WH = (unsigned)W * H;
  const unsigned *__restrict__ in = f.bits[d];
  float *v = f.vel[d];
  uint8_t *act = f.act[d];
  for (unsigned w0 = blockIdx.x * kExtrapolateThreads; w0 < nw; w0 += gridDim.x * kExtrapolateThreads) {
    if (threadIdx.x == 0) queued = 0;
    __syncthreads();
    const unsigned w = w0 + threadIdx.x;
    if (w < nw) {
      const unsigned c = in[w];
      unsigned fresh = 0;
      if (c != 0xffffffffu) {
        const long long o = 32ll * w;
        const unsigned row = 32u * w % (unsigned)W, plane = 32u * w % WH;
        // faces at the ends of rows and planes have no neighbour beyond
        unsigned x0 = 0, x1 = 0, y0 = 0, y1 = 0;
        for (int b = -(int)row; b < 32; b += W) {
          x0 |= bit_range(b, b + 1);
          x1 |= bit_range(b + W - 1, b + W);
        }
        if (plane < (unsigned)W || plane + 32 > WH - W) {
          for (long long b = -(long long)plane; b < 32; b += WH) {
            y0 |= bit_range((int)max(b, -64ll), (int)min(max(b + W, -64ll), 64ll));
            y1 |= bit_range((int)min(max(b + WH - W, -64ll), 64ll), (int)min(max(b + WH, -64ll), 64ll));
          }
        }
        const unsigned xp = bits_at(in, o + 1, nw) & ~x1, xm = bits_at(in, o - 1, nw) & ~x0;
        const unsigned yp = bits_at(in, o + W, nw) & ~y1, ym = bits_at(in, o - W, nw) & ~y0;
        const unsigned zm = bits_at(in, o - WH, nw), zp = bits_at(in, o + WH, nw);
        fresh = ~c & (xp | xm | yp | ym | zm | zp) & bit_range(0, (int)min((long long)n - o, 32ll));
        if (fresh) {
          int at = atomicAdd(&queued, __popc(fresh));
          for (unsigned m = fresh; m; m &= m - 1, ++at) {
            const int b = __ffs(m) - 1;
            queue[at] = (unsigned)o + b;
            sides[at] = (uint8_t)(((xp >> b) & 1u) | (((xm >> b) & 1u) << 1) | (((yp >> b) & 1u) << 2) |
                                  (((ym >> b) & 1u) << 3) | (((zm >> b) & 1u) << 4) | (((zp >> b) & 1u) << 5));
          }
        }
      }
      f.next[d][w] = c | fresh;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < queued; e += kExtrapolateThreads) {
      const size_t o = queue[e];
      const unsigned m = sides[e];
      // all loads first, the sum in order
      const float q[6] = {m & 1u ? v[o + 1] : 0.f,  m & 2u ? v[o - 1] : 0.f,  m & 4u ? v[o + W] : 0.f,
                          m & 8u ? v[o - W] : 0.f, m & 16u ? v[o - WH] : 0.f, m & 32u ? v[o + WH] : 0.f};
      float s = 0.0f;
      #pragma unroll
      for (int b = 0; b < 6; ++b)
        if ((m >> b) & 1u) s += q[b];
      v[o] = __fdiv_rn(s, (float)__popc(m));
      act[o] = 1;
    }
    __syncthreads();
  }
}

// Nodes that are not outside the solid (value not > 0) into bits, and
// levelset_exist (include/shiokaze/array/array_utility3.h:112-123): an active
// node with a negative value.
__global__ void __launch_bounds__(256) k_solid_bits(const float *__restrict__ solid, const uint8_t *__restrict__ act,
                                                    unsigned n, unsigned *__restrict__ bits, int *flag) {
  const unsigned nw = (n + 31) / 32;
  bool exists = false;
  for (unsigned w = blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += gridDim.x * blockDim.x) {
    unsigned near = 0, neg = 0, on = 0;
    if (32 * w + 32 <= n) {
      const float4 *s = reinterpret_cast<const float4 *>(solid) + 8 * (size_t)w;
      const uint4 *q = reinterpret_cast<const uint4 *>(act) + 2 * (size_t)w;
      on = byte_bits(q[0]) | (byte_bits(q[1]) << 16);
      #pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float4 x = s[e];
        near |= ((unsigned)!(x.x > 0.0f) | ((unsigned)!(x.y > 0.0f) << 1) | ((unsigned)!(x.z > 0.0f) << 2) |
                 ((unsigned)!(x.w > 0.0f) << 3)) << (4 * e);
        neg |= ((unsigned)(x.x < 0.0f) | ((unsigned)(x.y < 0.0f) << 1) | ((unsigned)(x.z < 0.0f) << 2) |
                ((unsigned)(x.w < 0.0f) << 3)) << (4 * e);
      }
    } else {
      for (unsigned b = 0; 32 * w + b < n; ++b) {
        const float x = solid[32 * (size_t)w + b];
        near |= (unsigned)!(x > 0.0f) << b;
        neg |= (unsigned)(x < 0.0f) << b;
        on |= (act[32 * (size_t)w + b] ? 1u : 0u) << b;
      }
    }
    bits[w] = near;
    exists = exists || (neg & on);
  }
  if (__any_sync(0xffffffffu, exists) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

// array_interpolator3::interpolate_coef's cell and fractions for one point
// (include/shiokaze/array/array_interpolator3.h): clamp into the grid, corner
// (i, j, k), and the weights' factors (i+1-x, x-i, ...).
struct Trilinear {
  int i, j, k;
  double ax, bx, ay, by, az, bz;
};
__device__ __forceinline__ Trilinear trilinear(int W, int H, int D, double px, double py, double pz) {
  Trilinear t;
  const double x = fmax(0.0, fmin(W - 1.0, px));
  const double y = fmax(0.0, fmin(H - 1.0, py));
  const double z = fmax(0.0, fmin(D - 1.0, pz));
  t.i = (int)fmin(x, W - 2.0);
  t.j = (int)fmin(y, H - 2.0);
  t.k = (int)fmin(z, D - 2.0);
  t.ax = (double)(t.i + 1) - x; t.bx = x - (double)t.i;
  t.ay = (double)(t.j + 1) - y; t.by = y - (double)t.j;
  t.az = (double)(t.k + 1) - z; t.bz = z - (double)t.k;
  return t;
}

// The 8 corner values of a grid (0 where the optional mask is off: the
// background of an inactive face is 0).
__device__ __forceinline__ void corners(const float *a, const uint8_t *m, int W, int H, const Trilinear &t,
                                        float v[8]) {
  #pragma unroll
  for (int n = 0; n < 8; ++n) {
    const size_t o = (size_t)(t.i + (n & 1)) + (size_t)W * ((size_t)(t.j + ((n >> 1) & 1)) +
                                                              (size_t)H * (size_t)(t.k + (n >> 2)));
    v[n] = (m && !m[o]) ? 0.0f : a[o];
  }
}

// array_interpolator3::interpolate (only_actives false): FP32 value, each
// corner with a non-zero weight added as value += corner * weight in FP64.
__device__ __forceinline__ float interpolate(const float v[8], const Trilinear &t) {
  const double c[8] = {t.az * t.ax * t.ay, t.az * t.bx * t.ay, t.az * t.ax * t.by, t.az * t.bx * t.by,
                       t.bz * t.ax * t.ay, t.bz * t.bx * t.ay, t.bz * t.ax * t.by, t.bz * t.bx * t.by};
  float r = 0.0f;
  #pragma unroll
  for (int n = 0; n < 8; ++n)
    if (c[n] != 0.0) r = (float)((double)r + (double)v[n] * c[n]);
  return r;
}

// array_derivative3::derivative (include/shiokaze/array/array_derivative3.h):
// FP32 gradient in index space, every term coef * corner in FP64.
__device__ __forceinline__ void derivative(const float v[8], const Trilinear &t, float g[3]) {
  const double cx[8] = {-t.az * t.ay, t.az * t.ay, -t.az * t.by, t.az * t.by,
                        -t.bz * t.ay, t.bz * t.ay, -t.bz * t.by, t.bz * t.by};
  const double cy[8] = {-t.az * t.ax, -t.az * t.bx, t.az * t.ax, t.az * t.bx,
                        -t.bz * t.ax, -t.bz * t.bx, t.bz * t.ax, t.bz * t.bx};
  const double cz[8] = {-t.ax * t.ay, -t.bx * t.ay, -t.ax * t.by, -t.bx * t.by,
                        t.ax * t.ay, t.bx * t.ay, t.ax * t.by, t.bx * t.by};
  float rx = 0.0f, ry = 0.0f, rz = 0.0f;
  #pragma unroll
  for (int n = 0; n < 8; ++n) rx = (float)((double)rx + cx[n] * (double)v[n]);
  #pragma unroll
  for (int n = 0; n < 8; ++n) ry = (float)((double)ry + cy[n] * (double)v[n]);
  #pragma unroll
  for (int n = 0; n < 8; ++n) rz = (float)((double)rz + cz[n] * (double)v[n]);
  g[0] = rx;
  g[1] = ry;
  g[2] = rz;
}

// macutility3::constrain_velocity (src/utility/macutility3.cpp:61-92) at one
// face of component d: where the solid level set interpolated at the face
// centre is negative, a velocity (interpolated from the field as it was before
// the constraint) that points into the solid loses its normal part; then no
// y-face lets flow out through the floor or the ceiling.
__device__ __forceinline__ float constrained(const ExtendFields &f, int d, int i, int j, int k, float v0,
                                             bool has_solid) {
  float v = v0;
  if (has_solid) {
    const double px = i + 0.5 * (d != 0), py = j + 0.5 * (d != 1), pz = k + 0.5 * (d != 2);
    const Trilinear ts = trilinear(f.nx + 1, f.ny + 1, f.nz + 1, px, py, pz);
    float sv[8];
    corners(f.solid, nullptr, f.nx + 1, f.ny + 1, ts, sv);
    bool near = false;  // all corners outside: so is the face
    #pragma unroll
    for (int c = 0; c < 8; ++c) near = near || !(sv[c] > 0.0f);
    if (near && interpolate(sv, ts) < 0.0f) {
      float g[3];
      derivative(sv, ts, g);
      const double nrm0 = (double)g[0] / f.dx, nrm1 = (double)g[1] / f.dx, nrm2 = (double)g[2] / f.dx;
      const double norm2 = ((0.0 + nrm0 * nrm0) + nrm1 * nrm1) + nrm2 * nrm2;
      if (norm2 != 0.0) {
        double u[3];
        #pragma unroll
        for (int c = 0; c < 3; ++c) {
          const Trilinear tc = trilinear(f.W[c], f.H[c], f.D[c], px - 0.5 * (c != 0), py - 0.5 * (c != 1),
                                         pz - 0.5 * (c != 2));
          float cv[8];
          corners(f.vel[c], f.act[c], f.W[c], f.H[c], tc, cv);
          u[c] = (double)interpolate(cv, tc);
        }
        const double un = ((0.0 + u[0] * nrm0) + u[1] * nrm1) + u[2] * nrm2;
        if (un < 0.0) {
          const double ud = d == 0 ? u[0] : (d == 1 ? u[1] : u[2]);
          const double nd = d == 0 ? nrm0 : (d == 1 ? nrm1 : nrm2);
          v = (float)(ud - nd * un);
        }
      }
    }
  }
  if (d == 1) {
    if (j == 0 && v < 0.0f) v = 0.0f;
    if (j == f.ny && v > 0.0f) v = 0.0f;
  }
  return v;
}

// Active faces the constraint may change, into a list: those with a node of
// theirs not outside the solid (the interpolated level set is a non-negative
// combination of the face's four nodes, the only ones with a non-zero weight,
// so it is negative only then), and the floor's and ceiling's. A thread looks
// at 32 faces of one row. They are few and lie together, so a list gives the
// FP64 kernel full warps (worked off by the block that found them: 90 us at
// 256^3, 140 with the rows dealt out over the blocks).
constexpr int kListThreads = 256;
__global__ void __launch_bounds__(kListThreads) k_constrain_list(ExtendFields f) {
  __shared__ int sums[kListThreads / 32];
  __shared__ unsigned base;
  const int d = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned n = f.n[d], nw = (n + 31) / 32;
  const int W = f.W[d], H = f.H[d], D = f.D[d], C = (W + 31) / 32;
  const int NX = f.nx + 1, NY = f.ny + 1;
  const unsigned nodes = (unsigned)NX * NY * (f.nz + 1), nnw = (nodes + 31) / 32;
  const bool has_solid = f.solid && *f.solid_flag;
  const unsigned words = (unsigned)C * H * D;
  for (unsigned t0 = blockIdx.x * kListThreads; t0 < words; t0 += gridDim.x * kListThreads) {
    const unsigned t = t0 + threadIdx.x;
    unsigned m = 0, o = 0;
    if (t < words) {
      const int c = (int)(t % (unsigned)C), j = (int)(t / (unsigned)C % (unsigned)H), k = (int)(t / ((unsigned)C * H));
      o = 32u * c + (unsigned)W * (j + (unsigned)H * k);
      const bool border = d == 1 && (j == 0 || j == f.ny);
      if (has_solid || border) {
        m = bits_at(f.bits[d], o, nw) & bit_range(0, W - 32 * c);
        if (m && !border) {
          const long long q = 32ll * c + (long long)NX * (j + (long long)NY * k);
          const long long dy = NX, dz = (long long)NX * NY;
          const long long u = d == 0 ? dy : 1, w = d == 2 ? dy : dz;
          m &= bits_at(f.solid_bits, q, nnw) | bits_at(f.solid_bits, q + u, nnw) | bits_at(f.solid_bits, q + w, nnw) |
               bits_at(f.solid_bits, q + u + w, nnw);
        }
      }
    }
    // one atomic a block
    int incl = __popc(m);
    #pragma unroll
    for (int e = 1; e < 32; e <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, e);
      if (lane >= e) incl += y;
    }
    if (lane == 31) sums[warp] = incl;
    __syncthreads();
    int before = 0, total = 0;
    #pragma unroll
    for (int w = 0; w < kListThreads / 32; ++w) {
      before += w < warp ? sums[w] : 0;
      total += sums[w];
    }
    if (threadIdx.x == 0 && total) base = atomicAdd(&f.listed[d], (unsigned)total);
    __syncthreads();
    unsigned at = base + before + incl - __popc(m);
    for (; m; m &= m - 1, ++at)
      if (at < f.room[d]) f.list[d][at] = o + (__ffs(m) - 1);
  }
}

// A list that did not fit: nothing is constrained, the host makes room and
// calls again.
__device__ __forceinline__ bool overfull(const ExtendFields &f) {
  return f.listed[0] > f.room[0] || f.listed[1] > f.room[1] || f.listed[2] > f.room[2];
}

// The listed faces' constrained values. The field is not modified here: a new
// value goes to side, an entry that keeps its value is struck out, so every
// interpolation reads the pre-constraint field, as the reference's
// velocity_save copy provides.
constexpr unsigned kStruck = 0xffffffffu;
__global__ void __launch_bounds__(128) k_constrain_find(ExtendFields f) {
  const int d = blockIdx.y, W = f.W[d], H = f.H[d];
  const unsigned listed = overfull(f) ? 0u : f.listed[d];
  const bool has_solid = f.solid && *f.solid_flag;
  for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < listed; e += gridDim.x * blockDim.x) {
    const unsigned o = f.list[d][e];
    const float v0 = f.vel[d][o];
    const float v = constrained(f, d, (int)(o % (unsigned)W), (int)(o / (unsigned)W % (unsigned)H),
                                (int)(o / ((unsigned)W * H)), v0, has_solid);
    f.side[d][e] = v;
    if (__float_as_uint(v) == __float_as_uint(v0)) f.list[d][e] = kStruck;
  }
}

// The new values, into the field.
__global__ void __launch_bounds__(256) k_constrain_apply(ExtendFields f) {
  const int d = blockIdx.y;
  const unsigned listed = overfull(f) ? 0u : f.listed[d];
  for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < listed; e += gridDim.x * blockDim.x)
    if (f.list[d][e] != kStruck) f.vel[d][f.list[d][e]] = f.side[d][e];
}

// blocks of `threads` for n items, at most 16 CTAs' worth per SM over the three components
static dim3 ext_grid(unsigned n, int threads) {
  const unsigned b = (n + threads - 1) / threads, cap = 148 * 16;
  return dim3(b < cap ? (b ? b : 1) : cap, 3);
}
static unsigned most_words(const ExtendFields &f) {
  unsigned m = 0;
  for (int d = 0; d < 3; ++d) m = f.n[d] > m ? f.n[d] : m;
  return (m + 31) / 32;
}

void launch_ext_pack(const ExtendFields &f, cudaStream_t s) {
  count_launches(1);
  k_ext_pack<<<ext_grid(most_words(f), 256), 256, 0, s>>>(f);
}

void launch_extrapolate(const ExtendFields &f, cudaStream_t s) {
  count_launches(1);
  k_extrapolate<<<ext_grid(most_words(f), kExtrapolateThreads), kExtrapolateThreads, 0, s>>>(f);
}

void launch_solid_bits(const ExtendFields &f, const uint8_t *solid_active, int *solid_flag, cudaStream_t s) {
  if (f.solid) {
    const unsigned nodes = (unsigned)(f.nx + 1) * (f.ny + 1) * (f.nz + 1);
    count_launches(1);
    k_solid_bits<<<ext_grid((nodes + 31) / 32, 256).x, 256, 0, s>>>(f.solid, solid_active, nodes, f.solid_bits, solid_flag);
  }
}

void launch_constrain(const ExtendFields &f, cudaStream_t s) {
  count_launches(3);
  // rows are cut into words of their own: a few more than the flat masks have
  const unsigned words = (unsigned)((f.nx + 32) / 32) * (f.ny + 1) * (f.nz + 1);
  k_constrain_list<<<ext_grid(words, kListThreads), kListThreads, 0, s>>>(f);
  // the list's length stays on the device: a fixed grid strides over it
  k_constrain_find<<<ext_grid(32 * words, 128), 128, 0, s>>>(f);
  k_constrain_apply<<<ext_grid(32 * words, 256), 256, 0, s>>>(f);
}

}  // namespace shkz
