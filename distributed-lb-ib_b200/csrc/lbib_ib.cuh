/*
 * Immersed-boundary device code shared by the one-grid kernels
 * (lbib_ib.cu) and the batched ones (lbib_batch.cu).
 *
 *   fiber_forces_node   compute_bendingforce + compute_stretchingforce +
 *                       compute_elasticforce (cube_pthread/lbm_ib.c:961-1318),
 *                       one node, both passes of each force in the
 *                       reference's order.
 *   node_prep_part      stencil start floor(X - 2) + 1 per axis, the twelve
 *                       delta-kernel factors 1 + cos(pi/2 r) (shared by the
 *                       spread and the interpolation of the step);
 *                       chunk_box_reduce: per 32-node chunk (and per 1024)
 *                       the bounding box of its stencils; touch_tiles: the
 *                       4^3 tiles the stencils touch, appended to the
 *                       step's tile list as they are met (or only marked,
 *                       for the compaction below).
 *   compaction kernels  x-slabs only: marked tiles -> dense list in tile
 *                       order and tile -> slot map (deterministic prefix
 *                       sums, three launches or one single-pass launch), so
 *                       that every slab numbers the slots alike.
 *   gather_tile         fiber_SpreadForce + fluid_get_SpreadForce
 *                       (lbm_ib.c:1323-1525) as a gather: one CTA per touched
 *                       tile finds the nodes that touch it, in index order,
 *                       from the boxes; then each of 64 threads (cells)
 *                       sums its contributions in that order -- the
 *                       reference's (sheet, row, col) order -- so the result
 *                       is deterministic and needs no atomics on forces.
 *   move_node /         moveFiberSheet (lbm_ib.c:2540-2723): u * w summed over
 *   move_warp           the 64 stencil cells in the reference's (x, y, z)
 *                       order, then X += dt U (move_warp: a warp's nodes
 *                       with their stencils' union staged in shared memory).
 * All arithmetic keeps the reference's operation order; translation units
 * that include this file are compiled with -fmad=false, except that the
 * gather (explicitly rounded operations) is also used by the low-precision
 * fluid kernels, which allow contraction.
 */
#ifndef LBIB_IB_CUH
#define LBIB_IB_CUH

#include <climits>

#include "lbib_cos.h"
#include "lbib_internal.h"
#include "lbib_lattice.cuh"

namespace lbib {


/* PI as truncated in the reference, cube_pthread/lbm_ib.c:33. */
constexpr double kPi = 3.14159265358979;

__device__ __forceinline__ void set_error(int* err, int code, int step) {
  if (atomicCAS(err, 0, code) == 0) err[1] = step;
}

/* compute_bendingforce + compute_stretchingforce + compute_elasticforce for
 * node i of one R x C sheet whose records start at `nodes`. */
__device__ __forceinline__ void fiber_forces_node(double* __restrict__ nodes, int R, int C, double bc, double sc,
                                                  double sc2, double ds1, double ds2, int bend_bug, int i) {
  const int r = i / C, c = i % C;
#define P(rr, cc) (nodes + ((long)(rr) * C + (cc)) * 12)
  const double* m = P(r, c);
  double b[3], s[3];
  /* bending along the fiber (row), lbm_ib.c:1002-1052 */
  for (int d = 0; d < 3; ++d) {
    if (c == 0) {
      b[d] = bc * (-P(r, 2)[d] + 2 * P(r, 1)[d] - P(r, 0)[d]);
    } else if (c == 1) {
      b[d] = bc * (-P(r, 3)[d] + 4 * P(r, 2)[d] - 5 * P(r, 1)[d] + 2 * P(r, 0)[d]);
    } else if (c == C - 1) {
      b[d] = bc * (-P(r, c)[d] + 2 * P(r, c - 1)[d] - P(r, c - 2)[d]);
    } else if (c == C - 2) {
      const double last = (d == 0 && bend_bug) ? P(r, c)[d] : P(r, c - 2)[d];
      b[d] = bc * (2 * P(r, c + 1)[d] - 5 * P(r, c)[d] + 4 * P(r, c - 1)[d] - last);
    } else {
      b[d] = bc * (-P(r, c + 2)[d] + 4.0 * P(r, c + 1)[d] - 6.0 * P(r, c)[d] + 4.0 * P(r, c - 1)[d] - P(r, c - 2)[d]);
    }
  }
  /* bending across fibers (column), lbm_ib.c:1062-1145 */
  for (int d = 0; d < 3; ++d) {
    double v;
    if (r == 0) {
      v = bc * (-P(2, c)[d] + 2 * (P(1, c)[d]) - (P(0, c)[d]));
    } else if (r == 1) {
      v = bc * (-P(3, c)[d] + 4 * (P(2, c)[d]) - 5 * (P(1, c)[d]) + 2 * (P(0, c)[d]));
    } else if (r == R - 1) {
      v = bc * (-(P(r, c)[d]) + 2 * (P(r - 1, c)[d]) - (P(r - 2, c)[d]));
    } else if (r == R - 2) {
      v = bc * (2 * P(r + 1, c)[d] - 5 * (P(r, c)[d]) + 4 * (P(r - 1, c)[d]) - (P(r - 2, c)[d]));
    } else {
      v = bc * (-P(r + 2, c)[d] + 4.0 * (P(r + 1, c)[d]) - 6.0 * (P(r, c)[d]) + 4.0 * (P(r - 1, c)[d]) - (P(r - 2, c)[d]));
    }
    b[d] = b[d] + v;
  }
  /* stretching along the fiber (row), lbm_ib.c:1179-1221 */
  if (c == 0) {
    const double* p = P(r, 1);
    const double t0 = p[0] - m[0], t1 = p[1] - m[1], t2 = p[2] - m[2];
    const double dr = sqrt(t0 * t0 + t1 * t1 + t2 * t2);
    s[0] = sc * ((dr - ds1) * (t0 / dr));
    s[1] = sc * ((dr - ds1) * (t1 / dr));
    s[2] = sc * ((dr - ds1) * (t2 / dr));
  } else if (c == C - 1) {
    const double* q = P(r, C - 2);
    const double t0 = m[0] - q[0], t1 = m[1] - q[1], t2 = m[2] - q[2];
    const double dl = sqrt(t0 * t0 + t1 * t1 + t2 * t2);
    s[0] = sc * ((dl - ds1) * (t0 / dl));
    s[1] = sc * ((dl - ds1) * (t1 / dl));
    s[2] = sc * ((dl - ds1) * (t2 / dl));
  } else {
    const double* p = P(r, c + 1);
    const double* q = P(r, c - 1);
    const double r0 = p[0] - m[0], r1 = p[1] - m[1], r2 = p[2] - m[2];
    const double l0 = q[0] - m[0], l1 = q[1] - m[1], l2 = q[2] - m[2];
    const double dr = sqrt(r0 * r0 + r1 * r1 + r2 * r2);
    const double dl = sqrt(l0 * l0 + l1 * l1 + l2 * l2);
    s[0] = sc * ((dr - ds1) * (r0 / dr) + (dl - ds1) * (l0 / dl));
    s[1] = sc * ((dr - ds1) * (r1 / dr) + (dl - ds1) * (l1 / dl));
    s[2] = sc * ((dr - ds1) * (r2 / dr) + (dl - ds1) * (l2 / dl));
  }
  /* stretching across fibers (column), lbm_ib.c:1233-1278 */
  if (r == 0) {
    const double* p = P(1, c);
    const double t0 = p[0] - m[0], t1 = p[1] - m[1], t2 = p[2] - m[2];
    const double dt = sqrt(t0 * t0 + t1 * t1 + t2 * t2);
    s[0] = s[0] + sc2 * ((dt - ds2) * (t0 / dt));
    s[1] = s[1] + sc2 * ((dt - ds2) * (t1 / dt));
    s[2] = s[2] + sc2 * ((dt - ds2) * (t2 / dt));
  } else if (r == R - 1) {
    const double* q = P(R - 2, c);
    const double t0 = m[0] - q[0], t1 = m[1] - q[1], t2 = m[2] - q[2];
    const double db = sqrt(t0 * t0 + t1 * t1 + t2 * t2);
    s[0] = s[0] + sc2 * ((db - ds2) * (t0 / db));
    s[1] = s[1] + sc2 * ((db - ds2) * (t1 / db));
    s[2] = s[2] + sc2 * ((db - ds2) * (t2 / db));
  } else {
    const double* p = P(r + 1, c);
    const double* q = P(r - 1, c);
    const double a0 = p[0] - m[0], a1 = p[1] - m[1], a2 = p[2] - m[2];
    const double e0 = q[0] - m[0], e1 = q[1] - m[1], e2 = q[2] - m[2];
    const double dt = sqrt(a0 * a0 + a1 * a1 + a2 * a2);
    const double db = sqrt(e0 * e0 + e1 * e1 + e2 * e2);
    s[0] = s[0] + sc2 * ((dt - ds2) * (a0 / dt) + (db - ds2) * (e0 / db));
    s[1] = s[1] + sc2 * ((dt - ds2) * (a1 / dt) + (db - ds2) * (e1 / db));
    s[2] = s[2] + sc2 * ((dt - ds2) * (a2 / dt) + (db - ds2) * (e2 / db));
  }
#undef P
  double* o = nodes + (long)i * 12;
  o[3] = b[0]; o[4] = b[1]; o[5] = b[2];
  o[6] = s[0]; o[7] = s[1]; o[8] = s[2];
  /* compute_elasticforce, lbm_ib.c:1303-1308: stretch + bend */
  o[9] = s[0] + b[0]; o[10] = s[1] + b[1]; o[11] = s[2] + b[2];
}

__device__ __forceinline__ int stencil_start(double p) { return (int)(floor(p / 1.0 - 2) + 1); }

/* The stencil of a node at coordinate p lies inside an axis of n cells:
 * start = floor(p - 2) + 1 in [0, n - 4], i.e. 1 <= p < n - 2, decided on
 * the double itself so that NaN and huge coordinates fail the test (the
 * reference stops with "out of bound" there; an int conversion first would
 * turn NaN into 0 and pass). */
__device__ __forceinline__ bool stencil_inside(double p, int n) { return p >= 1.0 && p < (double)n - 2.0; }

/* Node i, split over four threads: part p (0..3) evaluates the three delta
 * factors of stencil offset p (one per axis); part 0 also writes the stencil
 * start and checks the grid.  Returns whether the stencil lies inside, its
 * start in is, js, ks. */
__device__ __forceinline__ bool node_prep_part(const double* __restrict__ nodes, long i, int part, int nx, int ny,
                                               int nz, double* __restrict__ W, int* __restrict__ st, int* err,
                                               int step, int& is, int& js, int& ks) {
  const double* m = nodes + i * 12;
  const bool inside = stencil_inside(m[0], nx) && stencil_inside(m[1], ny) && stencil_inside(m[2], nz);
  is = inside ? stencil_start(m[0]) : 0;
  js = inside ? stencil_start(m[1]) : 0;
  ks = inside ? stencil_start(m[2]) : 0;
  const double cxk = kPi / (2.0 * 1.0);
  double* w = W + i * 12;
  w[part] = 1.0e0 + lbib_cos_2phase(cxk * (1.0 * (is + part) - m[0]));
  w[4 + part] = 1.0e0 + lbib_cos_2phase(cxk * (1.0 * (js + part) - m[1]));
  w[8 + part] = 1.0e0 + lbib_cos_2phase(cxk * (1.0 * (ks + part) - m[2]));
  if (part != 0) return inside;
  st[i * 3 + 0] = is; st[i * 3 + 1] = js; st[i * 3 + 2] = ks;
  if (!inside) set_error(err, -3, step);
  return inside;
}

/* The 4^3 tiles (ids offset by tile0) that a warp's stencils touch, ok: the
 * lane has one.  The lanes that touch a tile at the same stencil offset act
 * once, through the first of them.  With `list`: the warp that meets a tile
 * first (slot[tile] goes from -1 through -2) gives it the next slot --
 * which one depends on timing, no result does -- so that one launch does
 * what took a count, a prefix sum over all tiles and a scatter (22 us of a
 * 512x256x256 step's spread).  Without: mark[tile] = 1.  The eight offsets'
 * loads and atomics are each issued together. */
__device__ __forceinline__ void touch_tiles(int is, int js, int ks, bool ok, int ntx, int nty, long tile0,
                                            int* __restrict__ slot, int* __restrict__ list, int* __restrict__ count,
                                            int* __restrict__ mark) {
  const int lane = threadIdx.x & 31;
  long tile[8];
  int was[8];
#pragma unroll
  for (int o = 0; o < 8; ++o) {
    const int tx = (is >> 2) + (o & 1), ty = (js >> 2) + ((o >> 1) & 1), tz = (ks >> 2) + (o >> 2);
    const bool here = ok && tx <= (is + 3) >> 2 && ty <= (js + 3) >> 2 && tz <= (ks + 3) >> 2;
    const long id = here ? tile0 + ((long)tz * nty + ty) * ntx + tx : -1;
    const unsigned grp = __match_any_sync(0xffffffffu, id);
    tile[o] = here && lane == __ffs(grp) - 1 ? id : -1;
  }
  if (!list) {
#pragma unroll
    for (int o = 0; o < 8; ++o)
      if (tile[o] >= 0) mark[tile[o]] = 1;
    return;
  }
  volatile int* vs = slot;
#pragma unroll
  for (int o = 0; o < 8; ++o) was[o] = tile[o] >= 0 ? vs[tile[o]] : 0;
#pragma unroll
  for (int o = 0; o < 8; ++o)
    if (tile[o] >= 0 && was[o] == -1) was[o] = atomicCAS(&slot[tile[o]], -1, -2);
    else was[o] = 0;
#pragma unroll
  for (int o = 0; o < 8; ++o)
    if (was[o] == -1) was[o] = atomicAdd(count, 1);
    else was[o] = -1;
#pragma unroll
  for (int o = 0; o < 8; ++o)
    if (was[o] >= 0) {
      list[was[o]] = (int)tile[o];
      slot[tile[o]] = was[o];
    }
}

constexpr int kSuper = 32;   /* chunks per super-chunk */

/* The bounding box of a warp's stencils (ok: the lane has one), written by
 * lane 0 for chunk i >> 5, and merged into its super-chunk's (`super` may be
 * NULL: few chunks). */
__device__ __forceinline__ void chunk_box_reduce(long i, long S, int* __restrict__ chunk_box,
                                                 int* __restrict__ super, int is, int js, int ks, bool ok) {
  int b0 = ok ? is : INT_MAX, b1 = ok ? is + 3 : INT_MIN, b2 = ok ? js : INT_MAX, b3 = ok ? js + 3 : INT_MIN,
      b4 = ok ? ks : INT_MAX, b5 = ok ? ks + 3 : INT_MIN;
  b0 = __reduce_min_sync(0xffffffffu, b0); b1 = __reduce_max_sync(0xffffffffu, b1);
  b2 = __reduce_min_sync(0xffffffffu, b2); b3 = __reduce_max_sync(0xffffffffu, b3);
  b4 = __reduce_min_sync(0xffffffffu, b4); b5 = __reduce_max_sync(0xffffffffu, b5);
  const long chunk = i >> 5;
  if ((threadIdx.x & 31) != 0 || chunk * 32 >= S) return;
  int* bx = chunk_box + chunk * 6;
  bx[0] = b0; bx[1] = b1; bx[2] = b2; bx[3] = b3; bx[4] = b4; bx[5] = b5;
  if (!super) return;
  int* sx = super + chunk / kSuper * 6;
  atomicMin(&sx[0], b0); atomicMax(&sx[1], b1);
  atomicMin(&sx[2], b2); atomicMax(&sx[3], b3);
  atomicMin(&sx[4], b4); atomicMax(&sx[5], b5);
}

/* Deterministic compaction of the marked tiles, in tile-index order:
 * per-block sums, a one-block scan, then every marked tile gets its slot. */
constexpr int kScanBlock = 1024;

static __global__ void lbib_compact_count(const int* __restrict__ mark, long n, int* __restrict__ block_tiles) {
  __shared__ int s[32];
  const long i = (long)blockIdx.x * kScanBlock + threadIdx.x;
  int v = i < n && mark[i] != 0;
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int a = __reduce_add_sync(0xffffffffu, s[threadIdx.x]);
    if (threadIdx.x == 0) block_tiles[blockIdx.x] = a;
  }
}

static __global__ void lbib_compact_scan(int* __restrict__ a, int n, int* __restrict__ total) {
  __shared__ int s[kScanBlock];
  int carry = 0;
  for (int base = 0; base < n; base += kScanBlock) {
    const int i = base + threadIdx.x;
    const int v = (i < n) ? a[i] : 0;
    s[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < kScanBlock; o <<= 1) {
      const int t = (threadIdx.x >= (unsigned)o) ? s[threadIdx.x - o] : 0;
      __syncthreads();
      s[threadIdx.x] += t;
      __syncthreads();
    }
    if (i < n) a[i] = carry + s[threadIdx.x] - v;
    const int last = s[kScanBlock - 1];
    __syncthreads();
    carry += last;
  }
  if (threadIdx.x == 0) *total = carry;
}

static __global__ void lbib_compact_write(int* __restrict__ mark, long n, const int* __restrict__ block_tiles,
                                          int* __restrict__ list, int* __restrict__ slot) {
  __shared__ int sv[32];
  const long i = (long)blockIdx.x * kScanBlock + threadIdx.x;
  const int v = i < n && mark[i] != 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned m = __ballot_sync(0xffffffffu, v);
  if (lane == 0) sv[warp] = __popc(m);
  __syncthreads();
  if (threadIdx.x < 32) {
    const int a = sv[threadIdx.x];
    int ia = a;
    for (int o = 1; o < 32; o <<= 1) {
      const int ta = __shfl_up_sync(0xffffffffu, ia, o);
      if (lane >= o) ia += ta;
    }
    sv[threadIdx.x] = ia - a;
  }
  __syncthreads();
  if (v) {
    const int pos = block_tiles[blockIdx.x] + sv[warp] + __popc(m & ((1u << lane) - 1u));
    list[pos] = (int)i;
    slot[i] = pos;
    mark[i] = 0;      /* the next step starts unmarked */
  } else if (i < n) {
    slot[i] = -1;     /* the whole map is written: no clearing pass before the step */
  }
}

/* The same compaction in one launch: a single-pass scan with decoupled
 * look-back (Merrill & Garland, "Single-pass Parallel Prefix Scan with
 * Decoupled Look-back", 2016).  A block takes its place in tile order from
 * a ticket counter (so every block before it has started), publishes its
 * block total, walks back over its predecessors' published totals until
 * one carries an inclusive prefix, publishes its own inclusive prefix and
 * writes its tiles' slots.  Each published word is 64 bits: an 8-bit
 * launch tag (1..255, never 0, so a zeroed or stale word never matches),
 * a 2-bit flag (1 block total, 2 inclusive prefix) and 32 bits of tiles.
 * Every wait is bounded: a walk that runs out sets err (the step
 * then fails) instead of spinning on.  state[nblk] holds the ticket,
 * which the last block resets for the next launch. */
constexpr long kLookbackSpin = 1L << 22;
constexpr int kOnepassTiles = 4;   /* tiles per thread: a block covers 4096 tiles */
constexpr int kErrLookback = -2;   /* the error word's code: LBIB_E_CUDA of include/lbib.h */

__device__ __forceinline__ unsigned long long lookback_word(unsigned tag, unsigned flag, unsigned long long t) {
  return ((unsigned long long)tag << 56) | ((unsigned long long)flag << 54) | (t & 0xFFFFFFFFull);
}

static __global__ void __launch_bounds__(kScanBlock) lbib_compact_onepass(int* __restrict__ mark, long n, int nblk,
                                                                          unsigned long long* __restrict__ state,
                                                                          unsigned tag, int* __restrict__ list,
                                                                          int* __restrict__ slot,
                                                                          int* __restrict__ total, int* err) {
  __shared__ int sv[32];
  __shared__ int s_vb, s_tt, s_pt;
  unsigned* ticket = reinterpret_cast<unsigned*>(state + nblk);
  if (threadIdx.x == 0) s_vb = (int)atomicAdd(ticket, 1u);
  __syncthreads();
  const int vb = s_vb;
  /* kOnepassTiles consecutive tiles per thread: fewer, fuller blocks, so
     that every block is resident at once and the look-back walks short */
  const long i0 = ((long)vb * kScanBlock + threadIdx.x) * kOnepassTiles;
  int c[kOnepassTiles], tv = 0;
#pragma unroll
  for (int k = 0; k < kOnepassTiles; ++k) {
    c[k] = (i0 + k < n) ? mark[i0 + k] : 0;
    tv += c[k] > 0;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int iv = tv;  /* inclusive warp scan of the threads' totals */
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, iv, o);
    if (lane >= o) iv += u;
  }
  if (lane == 31) sv[warp] = iv;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int a = sv[threadIdx.x];
    int ia = a;
    for (int o = 1; o < 32; o <<= 1) {
      const int ta = __shfl_up_sync(0xffffffffu, ia, o);
      if (lane >= o) ia += ta;
    }
    sv[threadIdx.x] = ia - a;
    if (threadIdx.x == 31) s_tt = ia;
  }
  __syncthreads();
  if (warp == 0) {
    /* warp 0 walks back 32 predecessors at a time: lane k reads block
       j - k; the window is summed up to its nearest inclusive word once
       every word up to there has been published */
    volatile unsigned long long* vs = state;
    const unsigned long long at = (unsigned)s_tt;
    if (vb > 0 && lane == 0) vs[vb] = lookback_word(tag, 1u, at);
    __syncwarp();
    unsigned long long et = 0;
    long spins = 0;
    for (int j = vb - 1; j >= 0;) {
      const int jj = j - lane;
      const unsigned long long w = jj >= 0 ? vs[jj] : lookback_word(tag, 2u, 0ull);
      const unsigned f = (unsigned)(w >> 54) & 3u;
      const bool ready = (unsigned)(w >> 56) == tag && f != 0u;
      const unsigned incl = __ballot_sync(0xffffffffu, ready && f == 2u);
      const unsigned rdy = __ballot_sync(0xffffffffu, ready);
      const int lim = incl ? __ffs(incl) - 1 : 31;
      const unsigned need = lim == 31 ? 0xffffffffu : (1u << (lim + 1)) - 1u;
      if ((rdy & need) != need) {
        if (++spins > kLookbackSpin) {
          if (lane == 0) atomicCAS(err, 0, kErrLookback);
          break;
        }
        continue;
      }
      et += __reduce_add_sync(0xffffffffu, lane <= lim ? (unsigned)w : 0u);
      if (incl) break;
      j -= 32;
    }
    if (lane == 0) {
      vs[vb] = lookback_word(tag, 2u, et + at);
      s_pt = (int)et;
      if (vb == nblk - 1) {
        *total = (int)(et + at);
        *ticket = 0u;   /* every block has taken its ticket */
      }
    }
  }
  __syncthreads();
  int pos = s_pt + sv[warp] + iv - tv;
#pragma unroll
  for (int k = 0; k < kOnepassTiles; ++k) {
    const long i = i0 + k;
    if (c[k] > 0) {
      list[pos] = (int)i;
      slot[i] = pos++;
      mark[i] = 0;      /* the next step starts unmarked */
    } else if (i < n) {
      slot[i] = -1;   /* the whole map is written: no clearing pass before the step */
    }
  }
}

/* The columns [d, d + 3] of a stencil that starts d cells from a tile's
 * origin, as a 4-bit mask of the tile's columns 0..3 (0 when |d| > 3). */
__device__ __forceinline__ unsigned span4(int d) {
  if (d >= 4 || d <= -4) return 0u;
  return d >= 0 ? (0xFu << d) & 0xFu : 0xFu >> (-d);
}

/* The 64 cells of a tile (cell = 16 z + 4 y + x) that a stencil starting at
 * (dx, dy, dz) from the tile's origin covers, as a 64-bit mask. */
__device__ __forceinline__ unsigned long long stencil_tile_mask(int dx, int dy, int dz) {
  const unsigned mx = span4(dx), my = span4(dy), mz = span4(dz);
  unsigned row = 0u;
#pragma unroll
  for (int j = 0; j < 4; ++j) row |= ((my >> j) & 1u) ? mx << (4 * j) : 0u;
  unsigned long long m = 0ull;
#pragma unroll
  for (int k = 0; k < 4; ++k) m |= ((mz >> k) & 1u) ? (unsigned long long)row << (16 * k) : 0ull;
  return m;
}

/* A gather CTA: warps 0 and 1 hold the tile's 64 cells, warps 2 and 3 bring
 * the nodes. */
constexpr int kGatherTPB = 128;
constexpr int kGatherWarps = kGatherTPB / 32;
constexpr int kHitCap = 256;     /* chunks whose box meets the tile  */
constexpr int kOffHits = 64;     /* of those, with the starts kept   */
constexpr int kListCap = 1024;   /* nodes whose stencil meets it     */
constexpr int kBatch = 64;       /* nodes staged at once             */

/* A staged node: its x, y and z delta weights at the tile's four cell
 * positions per axis (unset where the stencil misses the position: no cell
 * it covers reads them), then its force.  An odd stride of 15 doubles puts 16 different nodes in 16
 * different bank pairs. */
constexpr int kNodeRec = 15;

struct GatherSmem {
  int hit[kHitCap];                     /* chunks in index order               */
  unsigned mask[kHitCap];               /* the nodes of each that touch        */
  unsigned short hoff[kOffHits][32];    /* their stencil starts, the first chunks' */
  int pos[kHitCap];                     /* their places in ids                 */
  int ids[kListCap];                    /* the tile's nodes in index order     */
  int off[kListCap];                    /* their stencil starts from the tile's origin */
  unsigned cover[2][2][kBatch];         /* per staged node: cells of warp 0, 1 */
  double rec[2][kBatch * kNodeRec];
  int warp_n[kGatherWarps];
  int n;
};

__device__ __forceinline__ bool box_meets(const int* __restrict__ b, int x0, int y0, int z0) {
  const int2 x = *reinterpret_cast<const int2*>(b), y = *reinterpret_cast<const int2*>(b + 2),
             z = *reinterpret_cast<const int2*>(b + 4);
  return !(x.y < x0 || x.x > x0 + 3 || y.y < y0 || y.x > y0 + 3 || z.y < z0 || z.x > z0 + 3);
}

/* Where the sheet's nodes are found: stencil starts and weights, the boxes
 * of chunks [c_lo, c_hi) and (NULL: few chunks) of the super-chunks; nodes
 * end at S. */
struct GatherNodes {
  const double* nodes;
  const double* W;
  const int* st;
  const int* chunk_box;
  const int* super;
  long S, c_lo, c_hi;
};

/* What the gather of grid d's current step reads. */
inline GatherNodes gather_nodes(const lbib_device* d) {
  return GatherNodes{d->nodes, d->W, d->st, d->chunk_box, d->super[d->cur], d->S, 0, d->nchunks};
}

/* The next step's super-chunk boxes start empty (its node preparation
 * merges into them); by the whole grid, in a launch after the last reader. */
__device__ __forceinline__ void clear_super(int* __restrict__ super, long n) {
  if (!super) return;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < 6 * n; i += (long)gridDim.x * blockDim.x)
    super[i] = (i % 6) & 1 ? INT_MIN : INT_MAX;
}

/* The CTA's threads with `flag` set append `value` in thread order to
 * out[*n ..) (up to cap); *n grows by their number.  Ends with a barrier. */
__device__ __forceinline__ void append_in_order(GatherSmem& sm, bool flag, int value, int* out, int cap, int& n) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned m = __ballot_sync(0xffffffffu, flag);
  if (lane == 0) sm.warp_n[warp] = __popc(m);
  __syncthreads();
  int at = n;
#pragma unroll
  for (int w = 0; w < kGatherWarps; ++w) {
    if (w == warp && flag) {
      const int k = at + __popc(m & ((1u << lane) - 1u));
      if (k < cap) out[k] = value;
    }
    at += sm.warp_n[w];
  }
  n = at;
  __syncthreads();
}

/* The nodes that touch the tile at (x0, y0, z0), in index order, into
 * sm.ids; returns their number, or -1 when a list overflows (a crumpled
 * sheet).  Boxes of 1024 nodes first (sheets of more than 128 chunks),
 * then of 32, then the nodes themselves: every level is a handful of
 * coalesced loads per CTA, nothing is sorted, and no list has to be built
 * beforehand. */
__device__ __forceinline__ int gather_list(GatherSmem& sm, const GatherNodes& g, int x0, int y0, int z0) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int nh = 0;
  if (!g.super || g.c_hi - g.c_lo <= kGatherTPB) {
    for (long c0 = g.c_lo; c0 < g.c_hi; c0 += kGatherTPB) {
      const long c = c0 + t;
      append_in_order(sm, c < g.c_hi && box_meets(g.chunk_box + c * 6, x0, y0, z0), (int)c, sm.hit, kHitCap, nh);
    }
  } else {
    int ns = 0;
    const long s1 = (g.c_hi + kSuper - 1) / kSuper;
    for (long s0 = g.c_lo / kSuper; s0 < s1; s0 += kGatherTPB) {
      const long s = s0 + t;
      append_in_order(sm, s < s1 && box_meets(g.super + s * 6, x0, y0, z0), (int)s, sm.pos, kHitCap, ns);
    }
    if (ns > kHitCap) return -1;
    for (int k = 0; k < ns; k += kGatherWarps) {
      const long c = k + warp < ns ? (long)sm.pos[k + warp] * kSuper + lane : -1;
      append_in_order(sm, c >= g.c_lo && c < g.c_hi && box_meets(g.chunk_box + c * 6, x0, y0, z0), (int)c, sm.hit,
                      kHitCap, nh);
    }
  }
  if (nh > kHitCap) return -1;
  for (int h = warp; h < nh; h += kGatherWarps) {
    const long i = (long)sm.hit[h] * 32 + lane;
    unsigned dx = 8u, dy = 8u, dz = 8u;   /* start - origin + 3: 0..6 where they meet */
    if (i < g.S) {
      const int* s = g.st + i * 3;
      dx = (unsigned)(s[0] - x0 + 3); dy = (unsigned)(s[1] - y0 + 3); dz = (unsigned)(s[2] - z0 + 3);
    }
    const bool in = dx < 7u && dy < 7u && dz < 7u;
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (lane == 0) sm.mask[h] = m;
    if (h < kOffHits) sm.hoff[h][lane] = (unsigned short)(dx | dy << 4 | dz << 8);
  }
  __syncthreads();
  if (warp == 0) {
    int run = 0;
    for (int h0 = 0; h0 < nh; h0 += 32) {
      const int v = h0 + lane < nh ? __popc(sm.mask[h0 + lane]) : 0;
      int iv = v;
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, iv, o);
        if (lane >= o) iv += u;
      }
      if (h0 + lane < nh) sm.pos[h0 + lane] = run + iv - v;
      run += __shfl_sync(0xffffffffu, iv, 31);
    }
    if (lane == 0) sm.n = run;
  }
  __syncthreads();
  const int L = sm.n;
  if (L > kListCap) return -1;
  for (int h = warp; h < nh; h += kGatherWarps) {
    const unsigned m = sm.mask[h];
    if ((m >> lane) & 1u) {
      const int k = sm.pos[h] + __popc(m & ((1u << lane) - 1u)), i = sm.hit[h] * 32 + lane;
      unsigned o;
      if (h < kOffHits) {
        o = sm.hoff[h][lane];
      } else {
        const int* s = g.st + (long)i * 3;
        o = (unsigned)(s[0] - x0 + 3) | (unsigned)(s[1] - y0 + 3) << 4 | (unsigned)(s[2] - z0 + 3) << 8;
      }
      sm.ids[k] = i;
      sm.off[k] = (int)o;
    }
  }
  __syncthreads();
  return L;
}

/* 8 bytes global -> shared, asynchronously. */
__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

/* Bring nodes b0 .. b0 + kBatch - 1 of the list to buffer `buf`, a thread of
 * warps 2 and 3 per node, asynchronously: a record goes to its place without
 * passing through registers (the cell's own state needs them). */
__device__ __forceinline__ void gather_stage(GatherSmem& sm, const GatherNodes& g, int L, int b0, int buf) {
  const int k = (int)threadIdx.x - 64;
  if (b0 + k >= L) return;
  const long nd = sm.ids[b0 + k];
  const int off = sm.off[b0 + k];
  double* r = sm.rec[buf] + k * kNodeRec;
  const double* w = g.W + nd * 12;
  const int d[3] = {(off & 15) - 3, ((off >> 4) & 15) - 3, (off >> 8) - 3};
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c)   /* cell position c of the tile is stencil position c - d */
      if ((unsigned)(c - d[a]) < 4u) cp_async8(r + 4 * a + c, w + 4 * a + c - d[a]);
#pragma unroll
  for (int a = 0; a < 3; ++a) cp_async8(r + 12 + a, g.nodes + nd * 12 + 9 + a);
  const unsigned long long cov = stencil_tile_mask(d[0], d[1], d[2]);
  sm.cover[buf][0][k] = (unsigned)cov;
  sm.cover[buf][1][k] = (unsigned)(cov >> 32);
}

/* Too many nodes for the lists: visit the chunks in order, skipping those
 * whose box misses the tile.  Same summation order. */
struct ScanSmem {
  int hit[kGatherTPB];
  int st[32][3];
  double w[32][12];
  double fe[32][3];
};

__device__ __forceinline__ void gather_scan(ScanSmem& sm, const GatherNodes& g, int x0, int y0, int z0, double& Fx,
                                            double& Fy, double& Fz) {
  const int t = threadIdx.x;
  const double cf = 1.0 / (64.0 * 1.0 * 1.0 * 1.0);
  const int gx = x0 + (t & 3), gy = y0 + ((t >> 2) & 3), gz = z0 + ((t & 63) >> 4);
  for (long c0 = g.c_lo; c0 < g.c_hi; c0 += kGatherTPB) {
    const long c = c0 + t;
    __syncthreads();
    sm.hit[t] = c < g.c_hi && box_meets(g.chunk_box + c * 6, x0, y0, z0);
    __syncthreads();
    for (int k = 0; k < kGatherTPB; ++k) {
      if (!sm.hit[k]) continue;
      if (t < 32) {
        const long nd = (c0 + k) * 32 + t;
        if (nd < g.S) {
          for (int a = 0; a < 3; ++a) sm.st[t][a] = g.st[nd * 3 + a];
          for (int a = 0; a < 12; ++a) sm.w[t][a] = g.W[nd * 12 + a];
          for (int a = 0; a < 3; ++a) sm.fe[t][a] = g.nodes[nd * 12 + 9 + a];
        } else {
          sm.st[t][0] = sm.st[t][1] = sm.st[t][2] = INT_MIN / 2;
        }
      }
      __syncthreads();
      for (int j = 0; j < 32 && t < 64; ++j) {
        const int a = gx - sm.st[j][0], b = gy - sm.st[j][1], e = gz - sm.st[j][2];
        if ((unsigned)a < 4u && (unsigned)b < 4u && (unsigned)e < 4u) {
          const double tmp = __dmul_rn(__dmul_rn(__dmul_rn(cf, sm.w[j][a]), sm.w[j][4 + b]), sm.w[j][8 + e]);
          Fx = __dadd_rn(Fx, __dmul_rn(sm.fe[j][0], tmp));
          Fy = __dadd_rn(Fy, __dmul_rn(sm.fe[j][1], tmp));
          Fz = __dadd_rn(Fz, __dmul_rn(sm.fe[j][2], tmp));
        }
      }
      __syncthreads();
    }
  }
}

union GatherShared {
  GatherSmem g;
  ScanSmem s;
};

/* The spread force of the tile at (x0, y0, z0): thread t < 64 gets its
 * cell's sum over the nodes in index order (cell = 16 z + 4 y + x).  Called
 * by all kGatherTPB threads.  Warps 2 and 3 stage the next 64 nodes while
 * warps 0 and 1 sum the last: each sum is a serial chain (its order is the
 * reference's), so latency is kept out of it. */
__device__ __forceinline__ void gather_tile(GatherShared& sh, const GatherNodes& g, int x0, int y0, int z0,
                                            double& Fx, double& Fy, double& Fz) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const double cf = 1.0 / (64.0 * 1.0 * 1.0 * 1.0);
  Fx = Fy = Fz = 0.0;
  __syncthreads();   /* the previous tile's data is no longer read */
  GatherSmem& sm = sh.g;
  const int L = gather_list(sm, g, x0, y0, z0);
  if (L < 0) {
    gather_scan(sh.s, g, x0, y0, z0, Fx, Fy, Fz);
    return;
  }
  /* the thread's cell in a record: its x, y and z weight positions */
  const int ox = t & 3, oy = 4 + ((t >> 2) & 3), oz = 8 + ((t & 63) >> 4);
  if (warp >= 2) {
    gather_stage(sm, g, L, 0, 0);
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  __syncthreads();
  for (int b0 = 0, buf = 0; b0 < L; b0 += kBatch, buf ^= 1) {
    if (warp >= 2) {
      gather_stage(sm, g, L, b0 + kBatch, buf ^ 1);
      asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
#pragma unroll 1
      for (int j0 = 0; j0 < kBatch && b0 + j0 < L; j0 += 32) {
        /* the warp's 32 x 32 cover bits (node j covers lane l's cell) are
           transposed with five shuffle stages, so that each lane walks only
           the nodes that cover its cell, in node order, two at a time */
        unsigned x = b0 + j0 + lane < L ? sm.cover[buf][warp][j0 + lane] : 0u;
#pragma unroll
        for (int k = 16; k >= 1; k >>= 1) {
          const unsigned M = k == 16 ? 0x0000FFFFu : k == 8 ? 0x00FF00FFu : k == 4 ? 0x0F0F0F0Fu
                           : k == 2 ? 0x33333333u : 0x55555555u;
          const unsigned y = __shfl_xor_sync(0xffffffffu, x, k);
          x = (lane & k) ? (x & ~M) | ((y & ~M) >> k) : (x & M) | ((y & M) << k);
        }
        const double* rec = sm.rec[buf] + j0 * kNodeRec;
        for (unsigned bits = x; bits;) {
          const double* r = rec + (__ffs(bits) - 1) * kNodeRec;
          bits &= bits - 1u;
          const bool two = bits != 0u;
          const double* q = two ? rec + (__ffs(bits) - 1) * kNodeRec : r;
          bits &= bits - 1u;   /* 0 stays 0 */
          const double tr = __dmul_rn(__dmul_rn(__dmul_rn(cf, r[ox]), r[oy]), r[oz]);
          const double tq = __dmul_rn(__dmul_rn(__dmul_rn(cf, q[ox]), q[oy]), q[oz]);
          Fx = __dadd_rn(Fx, __dmul_rn(r[12], tr));
          Fy = __dadd_rn(Fy, __dmul_rn(r[13], tr));
          Fz = __dadd_rn(Fz, __dmul_rn(r[14], tr));
          if (two) {
            Fx = __dadd_rn(Fx, __dmul_rn(q[12], tq));
            Fy = __dadd_rn(Fy, __dmul_rn(q[13], tq));
            Fz = __dadd_rn(Fz, __dmul_rn(q[14], tq));
          }
        }
      }
    }
    __syncthreads();
  }
}

/* moveFiberSheet for node i; slot maps local tiles to global slots. */
__device__ __forceinline__ void move_node(double* __restrict__ nodes, const double* __restrict__ W,
                                          const int* __restrict__ st, long i, int ntx, int nty,
                                          const int* __restrict__ slot, const double* __restrict__ Utile, double dt) {
  const double c_64 = 1.0 / (6.4e1);
  const int is = st[i * 3 + 0], js = st[i * 3 + 1], ks = st[i * 3 + 2];
  const double* w = W + i * 12;
  /* the stencil spans at most 2 tiles per axis: look their slots up first,
     so that the 64 cells' loads below do not wait on one another */
  const int tx0 = is >> 2, ty0 = js >> 2, tz0 = ks >> 2;
  int sp8[8];
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const int tx = tx0 + (a & 1), ty = ty0 + ((a >> 1) & 1), tz = tz0 + (a >> 2);
    const bool need = tx * 4 <= is + 3 && ty * 4 <= js + 3 && tz * 4 <= ks + 3;
    sp8[a] = need ? slot[(tz * nty + ty) * ntx + tx] : 0;
  }
  double s1 = 0, s2 = 0, s3 = 0;
#pragma unroll
  for (int i2 = 0; i2 <= 3; i2++) {
    const int gi = is + i2;
#pragma unroll
    for (int j2 = 0; j2 <= 3; j2++) {
      const int gj = js + j2;
#pragma unroll
      for (int k2 = 0; k2 <= 3; k2++) {
        const int gk = ks + k2;
        const int sp = sp8[((gi >> 2) - tx0) | (((gj >> 2) - ty0) << 1) | (((gk >> 2) - tz0) << 2)];
        const double* U = Utile + (long)sp * 256;
        const int cell = lbib::cell_in_tile(gi, gj, gk);
        const double vx = U[64 + cell], vy = U[128 + cell], vz = U[192 + cell];
        s1 += vx * w[i2] * w[4 + j2] * w[8 + k2] * c_64;
        s2 += vy * w[i2] * w[4 + j2] * w[8 + k2] * c_64;
        s3 += vz * w[i2] * w[4 + j2] * w[8 + k2] * c_64;
      }
    }
  }
  double* m = nodes + i * 12;
  m[0] += dt * s1;
  m[1] += dt * s2;
  m[2] += dt * s3;
}


/* A move CTA: the 32 nodes of a chunk, four warps. */
constexpr int kMoveTPB = 128;
/* Cells a CTA's staged move holds in shared memory: the union box of its 32
 * nodes' stencils (along a fiber row ~5 x 20 x 5 cells); a larger union (a
 * chunk straddling two rows, a crumpled sheet) takes move_node. */
constexpr int kMoveCap = 640;
constexpr int kMoveTiles = 64;   /* tiles of the union box whose slots are staged */

struct MoveSmem {
  double U[3][kMoveCap];
  int slot[kMoveTiles];
};

/* The move of the 32 nodes of a chunk (node i on lane l of every warp,
 * `live` if it moves), with the velocity of the union box of their stencils
 * staged once in shared memory: the four warps read each box cell's u from
 * its moment tile, then warp a < 3 sums component a of every node's 64
 * terms from shared memory -- the same values in the same order as
 * move_node, with ~5x fewer L2 requests (neighbouring nodes' stencils
 * overlap by 3 cells of 4).  A node's sum is a serial chain of 64 terms, so
 * a thread holds one component only; with one warp that staged and summed
 * all three for its nodes the launch took 10 us at 16 x 16 nodes, this 6.
 * Called by all kMoveTPB threads; ends with a barrier. */
__device__ __forceinline__ void move_chunk(MoveSmem& sm, double* __restrict__ nodes, const double* __restrict__ W,
                                           const int* __restrict__ st, long i, bool live, int ntx, int nty,
                                           const int* __restrict__ slot, const double* __restrict__ Utile, double dt) {
  const int t = threadIdx.x, warp = t >> 5;
  int is = 0, js = 0, ks = 0;
  if (live) { is = st[i * 3 + 0]; js = st[i * 3 + 1]; ks = st[i * 3 + 2]; }
  const int x0 = __reduce_min_sync(0xffffffffu, live ? is : INT_MAX), x1 = __reduce_max_sync(0xffffffffu, live ? is + 3 : INT_MIN);
  const int y0 = __reduce_min_sync(0xffffffffu, live ? js : INT_MAX), y1 = __reduce_max_sync(0xffffffffu, live ? js + 3 : INT_MIN);
  const int z0 = __reduce_min_sync(0xffffffffu, live ? ks : INT_MAX), z1 = __reduce_max_sync(0xffffffffu, live ? ks + 3 : INT_MIN);
  if (x0 > x1) {   /* no live node: uniform over the CTA */
    __syncthreads();
    return;
  }
  const int bx = x1 - x0 + 1, by = y1 - y0 + 1, bz = z1 - z0 + 1;
  const long vol = (long)bx * by * bz;
  const int tx0 = x0 >> 2, ty0 = y0 >> 2, tz0 = z0 >> 2;
  const int tbx = (x1 >> 2) - tx0 + 1, tby = (y1 >> 2) - ty0 + 1;
  const long ntb = (long)tbx * tby * ((z1 >> 2) - tz0 + 1);
  if (vol > kMoveCap || ntb > kMoveTiles) {   /* uniform over the CTA */
    if (live && warp == 0) move_node(nodes, W, st, i, ntx, nty, slot, Utile, dt);
    __syncthreads();
    return;
  }
  /* the weights this thread will need, on their way while the box is staged */
  double w[12];
  double at = 0.0;
  if (live && warp < 3) {
    const double2* p = reinterpret_cast<const double2*>(W + i * 12);
#pragma unroll
    for (int a = 0; a < 6; ++a) { w[2 * a] = p[a].x; w[2 * a + 1] = p[a].y; }
    at = nodes[i * 12 + warp];
  }
  /* the slots of the box's tiles first (at most 3 x 7 x 3 for a box that
     fits), so that the cell loads below depend on one shared-memory read */
  if (t < (int)ntb) {
    const int tx = tx0 + t % tbx, ty = ty0 + (t / tbx) % tby, tz = tz0 + t / (tbx * tby);
    sm.slot[t] = slot[(tz * nty + ty) * ntx + tx];
  }
  __syncthreads();
  /* the box's longest axis (the fiber direction: neighbouring lanes'
     stencils are offset along it) is stored fastest, so that the lanes'
     reads below fall on consecutive words, not on one bank */
  const int f = (bx >= by && bx >= bz) ? 0 : (by >= bz ? 1 : 2);
  const int ef = f == 0 ? bx : f == 1 ? by : bz, ea = f == 0 ? by : bx;
  const int sx = f == 0 ? 1 : ef, sy = f == 1 ? 1 : f == 0 ? ef : ef * ea, sz = f == 2 ? 1 : ef * ea;
  /* j / ef and j / ea by reciprocals: exact for j < 640, divisors < 100 */
  const unsigned rf = (65535u + ef) / ef, ra = (65535u + ea) / ea;
#pragma unroll 5
  for (int j = t; j < (int)vol; j += kMoveTPB) {   /* 640 / 128: the loads of all rounds in flight */
    const int q = ef < 100 ? (int)(j * rf >> 16) : j / ef, uf = j - q * ef;
    const int ub = ea < 100 ? (int)(q * ra >> 16) : q / ea, ua = q - ub * ea;
    const int cx = x0 + (f == 0 ? uf : ua), cy = y0 + (f == 1 ? uf : f == 0 ? ua : ub), cz = z0 + (f == 2 ? uf : ub);
    /* a box corner no stencil covers may lie in an untouched tile: never read */
    const int sp = sm.slot[((cz >> 2) - tz0) * tbx * tby + ((cy >> 2) - ty0) * tbx + ((cx >> 2) - tx0)];
    double vx = 0.0, vy = 0.0, vz = 0.0;
    if (sp >= 0) {
      const double* U = Utile + (long)sp * 256 + lbib::cell_in_tile(cx, cy, cz);
      vx = U[64]; vy = U[128]; vz = U[192];
    }
    sm.U[0][j] = vx; sm.U[1][j] = vy; sm.U[2][j] = vz;
  }
  __syncthreads();
  if (live && warp < 3) {
    const double c_64 = 1.0 / (6.4e1);
    const double* u = sm.U[warp] + (is - x0) * sx + (js - y0) * sy + (ks - z0) * sz;
    double s = 0;
#pragma unroll
    for (int i2 = 0; i2 <= 3; i2++)
#pragma unroll
      for (int j2 = 0; j2 <= 3; j2++)
#pragma unroll
        for (int k2 = 0; k2 <= 3; k2++)
          s += u[i2 * sx + j2 * sy + k2 * sz] * w[i2] * w[4 + j2] * w[8 + k2] * c_64;
    nodes[i * 12 + warp] = at + dt * s;
  }
  __syncthreads();
}

}  // namespace lbib

#endif
