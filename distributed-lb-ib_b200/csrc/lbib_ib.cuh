/*
 * Immersed-boundary device code shared by the one-grid kernels
 * (lbib_ib.cu) and the batched ones (lbib_batch.cu).
 *
 *   fiber_forces_node   compute_bendingforce + compute_stretchingforce +
 *                       compute_elasticforce (cube_pthread/lbm_ib.c:961-1318),
 *                       one node, both passes of each force in the
 *                       reference's order.
 *   node_prep_warp      stencil start floor(X - 2) + 1 per axis, the twelve
 *                       delta-kernel factors 1 + cos(pi/2 r) (shared by the
 *                       spread and the interpolation of the step);
 *                       chunk_box_reduce: per 32-node chunk (and per 1024)
 *                       the bounding box of its stencils; TouchTiles: the
 *                       4^3 tiles the stencils touch, appended to the
 *                       step's tile list as they are met (or only marked,
 *                       for the compaction below).
 *   lbib_compact_onepass  x-slabs only: marked tiles -> dense list in tile
 *                       order and tile -> slot map (deterministic prefix
 *                       sums), so that every slab numbers the slots alike.
 *   gather_tile         fiber_SpreadForce + fluid_get_SpreadForce
 *                       (lbm_ib.c:1323-1525) as a gather: one CTA per touched
 *                       tile finds the nodes that touch it, in index order,
 *                       from the boxes; then each of 64 threads (cells)
 *                       sums its contributions in that order -- the
 *                       reference's (sheet, row, col) order -- so the result
 *                       is deterministic and needs no atomics on forces.
 *   move_chunk          moveFiberSheet (lbm_ib.c:2540-2723): u * w summed over
 *                       the 64 stencil cells in the reference's (x, y, z)
 *                       order, then X += dt U, with the union of a chunk's
 *                       stencils staged in shared memory.
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

/* The error words {code, step} in one go, the first one to come; no reader
 * sees a code without its step. */
__device__ __forceinline__ void set_error(int* err, int code, int step) {
  atomicCAS(reinterpret_cast<unsigned long long*>(err), 0ull,
            (unsigned long long)(unsigned)step << 32 | (unsigned)code);
}

/* An error from before this step: one that another CTA of this launch sets
 * meanwhile does not count. */
__device__ __forceinline__ bool failed_before(const int* err, int step) {
  const unsigned long long w = *reinterpret_cast<const volatile unsigned long long*>(err);
  return (unsigned)w != 0u && (int)(w >> 32) != step;
}

/* One direction's share of a node's bending and stretching force: along the
 * fiber (k = c, n = C nodes, stride 1 node, rest length ds1) or across the
 * fibers (k = r, n = R, stride C, ds2).  `slip`: at the last node but one
 * the x component takes the node's own position for the one two nodes back
 * (lbm_ib.c:1032-1035, the row pass only).  The node and its neighbours
 * k - 2 .. k + 2 are loaded together before any is used.  Bending lbm_ib.c:1002-1052 and 1062-1145, stretching 1179-1221 and
 * 1233-1278. */
__device__ __forceinline__ void fiber_line_forces(const double* __restrict__ m, int k, int n, long stride, double bc,
                                                  double sc, double rest, bool slip, double b[3], double s[3]) {
  double p[5][3];
#pragma unroll
  for (int o = -2; o <= 2; ++o) {
    /* the neighbours its formula reads; its own place for the others */
    const bool used = o == 0 || (k == 0 ? o > 0 : k == 1 ? o != -2 : k == n - 1 ? o < 0 : k == n - 2 ? o != 2 : true);
    const double* q = m + (used ? (long)o * stride * 12 : 0);
#pragma unroll
    for (int d = 0; d < 3; ++d) p[o + 2][d] = q[d];
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double a2 = p[0][d], a1 = p[1][d], x = p[2][d], c1 = p[3][d], c2 = p[4][d];
    if (k == 0) b[d] = bc * (-c2 + 2 * c1 - x);
    else if (k == 1) b[d] = bc * (-c2 + 4 * c1 - 5 * x + 2 * a1);
    else if (k == n - 1) b[d] = bc * (-x + 2 * a1 - a2);
    else if (k == n - 2) b[d] = bc * (2 * c1 - 5 * x + 4 * a1 - (d == 0 && slip ? x : a2));
    else b[d] = bc * (-c2 + 4.0 * c1 - 6.0 * x + 4.0 * a1 - a2);
  }
  /* towards the next node (k = 0), from the previous one (the last: the
     reference's reversed tangent), or both */
  const bool first = k == 0, last = k == n - 1;
  double u[3], v[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    u[d] = last ? p[2][d] - p[1][d] : p[3][d] - p[2][d];
    v[d] = p[1][d] - p[2][d];
  }
  const double lu = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
  if (first || last) {
#pragma unroll
    for (int d = 0; d < 3; ++d) s[d] = sc * ((lu - rest) * (u[d] / lu));
  } else {
    const double lv = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
#pragma unroll
    for (int d = 0; d < 3; ++d) s[d] = sc * ((lu - rest) * (u[d] / lu) + (lv - rest) * (v[d] / lv));
  }
}

/* The node's record: the along-fiber shares plus the across-fiber ones, and
 * compute_elasticforce (lbm_ib.c:1303-1308): stretch + bend. */
__device__ __forceinline__ void fiber_store(double* __restrict__ o, const double b1[3], const double s1[3],
                                            const double b2[3], const double s2[3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double b = b1[d] + b2[d], s = s1[d] + s2[d];
    o[3 + d] = b;
    o[6 + d] = s;
    o[9 + d] = s + b;
  }
}

/* compute_bendingforce + compute_stretchingforce + compute_elasticforce for
 * node i of one R x C sheet whose records start at `nodes`. */
__device__ __forceinline__ void fiber_forces_node(double* __restrict__ nodes, int R, int C, double bc, double sc,
                                                  double sc2, double ds1, double ds2, int bend_bug, int i) {
  double* m = nodes + (long)i * 12;
  double b1[3], s1[3], b2[3], s2[3];
  fiber_line_forces(m, i % C, C, 1, bc, sc, ds1, bend_bug, b1, s1);
  fiber_line_forces(m, i / C, R, C, bc, sc2, ds2, false, b2, s2);
  fiber_store(m, b1, s1, b2, s2);
}

/* The same by two warps of a CTA, a lane of each for node i (`ok`: there is
 * one): warp `half` 0 the along-fiber share, 1 the across-fiber one, which it
 * hands over through shared memory x[6][32]; named barrier 1 is theirs. */
__device__ __forceinline__ void fiber_forces_pair(double* __restrict__ nodes, int R, int C, double bc, double sc,
                                                  double sc2, double ds1, double ds2, int bend_bug, int i, bool ok,
                                                  int half, double (*x)[32]) {
  const int lane = threadIdx.x & 31;
  double* m = nodes + (long)i * 12;
  double b[3], s[3];
  if (ok) {
    if (half) fiber_line_forces(m, i / C, R, C, bc, sc2, ds2, false, b, s);
    else fiber_line_forces(m, i % C, C, 1, bc, sc, ds1, bend_bug, b, s);
  }
  if (half && ok)
#pragma unroll
    for (int d = 0; d < 3; ++d) { x[d][lane] = b[d]; x[3 + d][lane] = s[d]; }
  asm volatile("bar.sync 1, 64;" ::: "memory");
  if (!half && ok) {
    const double b2[3] = {x[0][lane], x[1][lane], x[2][lane]}, s2[3] = {x[3][lane], x[4][lane], x[5][lane]};
    fiber_store(m, b, s, b2, s2);
  }
}

__device__ __forceinline__ int stencil_start(double p) { return (int)(floor(p / 1.0 - 2) + 1); }

/* The stencil of a node at coordinate p lies inside an axis of n cells:
 * start = floor(p - 2) + 1 in [0, n - 4], i.e. 1 <= p < n - 2, decided on
 * the double itself so that NaN and huge coordinates fail the test (the
 * reference stops with "out of bound" there; an int conversion first would
 * turn NaN into 0 and pass). */
__device__ __forceinline__ bool stencil_inside(double p, int n) { return p >= 1.0 && p < (double)n - 2.0; }

/* The 4^3 tiles (ids offset by tile0) that a warp's stencils touch at offsets
 * 2 part and 2 part + 1 of the eight (the four warps of a chunk share them;
 * ok: the lane has a stencil).  The lanes that touch a tile at the same
 * offset act once, through the first of them.  With `list`: the warp that
 * meets a tile first (slot[tile] goes from -1 through -2) gives it the next
 * slot -- which one depends on timing, no result does -- so that one launch
 * does what took a count, a prefix sum over all tiles and a scatter (22 us
 * of a 512x256x256 step's spread).  Without: mark[tile] = 1.  begin sends
 * the atomics off, finish uses their answers: the cosines come in between.
 * (All eight offsets by one warp after its cosines: 8,000 of the
 * launch's 16,000 cycles.) */
struct TouchTiles {
  int tile[2], was[2];
  __device__ __forceinline__ void begin(int part, int is, int js, int ks, bool ok, int ntx, int nty, int tile0,
                                        int* __restrict__ slot, bool listed, int* __restrict__ mark) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int tx = (is >> 2) + u, ty = (js >> 2) + (part & 1), tz = (ks >> 2) + (part >> 1);
      const bool here = ok && tx <= (is + 3) >> 2 && ty <= (js + 3) >> 2 && tz <= (ks + 3) >> 2;
      const int id = here ? tile0 + (tz * nty + ty) * ntx + tx : -1;
      const unsigned grp = __match_any_sync(0xffffffffu, id);
      tile[u] = here && lane == __ffs(grp) - 1 ? id : -1;
      was[u] = 0;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (tile[u] < 0) continue;
      if (listed) was[u] = atomicCAS(&slot[tile[u]], -1, -2);
      else mark[tile[u]] = 1;
    }
  }
  __device__ __forceinline__ void finish(int* __restrict__ slot, int* __restrict__ list, int* __restrict__ count) {
    const int lane = threadIdx.x & 31;
    const unsigned a = __ballot_sync(0xffffffffu, was[0] == -1), b = __ballot_sync(0xffffffffu, was[1] == -1);
    const int na = __popc(a), n = na + __popc(b);
    if (!n) return;
    int base = 0;
    if (lane == 0) base = atomicAdd(count, n);
    base = __shfl_sync(0xffffffffu, base, 0);
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (was[u] != -1) continue;
      const int k = base + (u ? na + __popc(b & below) : __popc(a & below));
      list[k] = tile[u];
      slot[tile[u]] = k;
    }
  }
};

/* A node's stencil start per axis; false when it leaves the grid. */
__device__ __forceinline__ bool node_stencil(const double m[3], int nx, int ny, int nz, int& is, int& js, int& ks) {
  const bool inside = stencil_inside(m[0], nx) && stencil_inside(m[1], ny) && stencil_inside(m[2], nz);
  is = inside ? stencil_start(m[0]) : 0;
  js = inside ? stencil_start(m[1]) : 0;
  ks = inside ? stencil_start(m[2]) : 0;
  return inside;
}

/* The three delta factors (one per axis) of stencil offset `part` of a node
 * at m whose stencil starts at is, js, ks. */
__device__ __forceinline__ void delta_factors(double* __restrict__ w, const double m[3], int part, int is, int js,
                                              int ks) {
  const double cxk = kPi / (2.0 * 1.0);
  w[part] = 1.0e0 + lbib_cos_2phase(cxk * (1.0 * (is + part) - m[0]));
  w[4 + part] = 1.0e0 + lbib_cos_2phase(cxk * (1.0 * (js + part) - m[1]));
  w[8 + part] = 1.0e0 + lbib_cos_2phase(cxk * (1.0 * (ks + part) - m[2]));
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

/* Node preparation of a chunk's 32 nodes (node i on lane l of each of the
 * four warps, `have`: there is one): warp `part` evaluates its delta factors
 * and enters its share of the touched tiles; the first also writes the
 * stencil starts, checks the grid and reduces the chunk's box. */
__device__ __forceinline__ void node_prep_warp(const double* __restrict__ nodes, long i, bool have, long S, int part,
                                               int nx, int ny, int nz, int ntx, int nty, long tile0,
                                               double* __restrict__ W, int* __restrict__ st,
                                               int* __restrict__ chunk_box, int* __restrict__ super,
                                               int* __restrict__ slot, int* __restrict__ list,
                                               int* __restrict__ count, int* __restrict__ mark, int* err, int step) {
  double m[3] = {-1.0, 0.0, 0.0};
  if (have) { m[0] = nodes[i * 12]; m[1] = nodes[i * 12 + 1]; m[2] = nodes[i * 12 + 2]; }
  int is, js, ks;
  const bool ok = node_stencil(m, nx, ny, nz, is, js, ks);
  TouchTiles t;
  t.begin(part, is, js, ks, ok, ntx, nty, (int)tile0, slot, list != nullptr, mark);
  if (part == 0) {
    if (have) {
      st[i * 3 + 0] = is; st[i * 3 + 1] = js; st[i * 3 + 2] = ks;
      if (!ok) set_error(err, -3, step);
    }
    chunk_box_reduce(i, S, chunk_box, super, is, js, ks, ok);
  }
  if (have) delta_factors(W + i * 12, m, part, is, js, ks);
  if (list) t.finish(slot, list, count);
}

constexpr int kScanBlock = 1024;

/* Deterministic compaction of the marked tiles, in tile-index order, in one
 * launch: a single-pass scan with decoupled look-back (Merrill & Garland,
 * "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016).  A block
 * takes its place in tile order from a ticket counter (so every block before
 * it has started), publishes its block total, walks back over its predecessors' published totals until
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

/* A gather CTA: warps 0 and 1 sum the tile's 64 cells, warps 2 and 3 bring
 * the nodes. */
constexpr int kGatherTPB = 128;
constexpr int kGatherWarps = kGatherTPB / 32;
constexpr int kHitCap = 256;     /* chunks whose box meets the tile, at once */
constexpr int kOffHits = 64;     /* of those, with the starts kept   */
constexpr int kHitsAhead = 8;
constexpr int kListCap = 1024;   /* nodes whose stencil meets it, at once */
constexpr int kBatch = 64;       /* nodes staged at once             */
static_assert(kHitCap >= kGatherTPB && kListCap >= 32, "a round of candidates, a chunk");

/* A staged node: its x, y and z delta weights at the tile's four cell
 * positions per axis (unset where the stencil misses the position: no cell
 * it covers reads them), then its force. */
constexpr int kNodeRec = 16;

struct GatherSmem {
  int hit[kHitCap];                     /* chunks in index order               */
  unsigned mask[kHitCap];               /* the nodes of each that touch        */
  unsigned short hoff[kOffHits][32];    /* their stencil starts, the first chunks' */
  int pos[kHitCap + 1];                 /* nodes before each                   */
  int ids[kListCap];                    /* the tile's nodes in index order     */
  int off[kListCap];                    /* their stencil starts from the tile's origin */
  unsigned cover[2][2][kBatch];         /* per staged node: cells 0..31, 32..63 */
  alignas(16) double rec[2][kBatch * kNodeRec];
  int warp_n[kGatherWarps];
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
 * out[n ..) (up to kHitCap); n grows by their number.  Ends with a barrier. */
__device__ __forceinline__ void append_in_order(GatherSmem& sm, bool flag, int value, int* out, int& n) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned m = __ballot_sync(0xffffffffu, flag);
  if (lane == 0) sm.warp_n[warp] = __popc(m);
  __syncthreads();
  int at = n;
#pragma unroll
  for (int w = 0; w < kGatherWarps; ++w) {
    if (w == warp && flag) {
      const int k = at + __popc(m & ((1u << lane) - 1u));
      if (k < kHitCap) out[k] = value;
    }
    at += sm.warp_n[w];
  }
  n = at;
  __syncthreads();
}

/* The chunks whose box meets the tile at (x0, y0, z0), in index order, into
 * sm.hit; returns their number, above kHitCap when they do not fit.  Boxes of
 * 1024 nodes first (sheets of more than 128 chunks), then of 32. */
__device__ __forceinline__ int gather_chunks(GatherSmem& sm, const GatherNodes& g, int x0, int y0, int z0) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int nh = 0;
  if (!g.super || g.c_hi - g.c_lo <= kGatherTPB) {
    for (long c0 = g.c_lo; c0 < g.c_hi; c0 += kGatherTPB) {
      const long c = c0 + t;
      append_in_order(sm, c < g.c_hi && box_meets(g.chunk_box + c * 6, x0, y0, z0), (int)c, sm.hit, nh);
    }
  } else {
    int ns = 0;
    const long s1 = (g.c_hi + kSuper - 1) / kSuper;
    for (long s0 = g.c_lo / kSuper; s0 < s1; s0 += kGatherTPB) {
      const long s = s0 + t;
      append_in_order(sm, s < s1 && box_meets(g.super + s * 6, x0, y0, z0), (int)s, sm.pos, ns);
    }
    if (ns > kHitCap) return kHitCap + 1;
    for (int k = 0; k < ns; k += kGatherWarps) {
      const long c = k + warp < ns ? (long)sm.pos[k + warp] * kSuper + lane : -1;
      append_in_order(sm, c >= g.c_lo && c < g.c_hi && box_meets(g.chunk_box + c * 6, x0, y0, z0), (int)c, sm.hit, nh);
    }
  }
  return nh;
}

/* The nodes of the nh chunks in sm.hit that touch the tile: a mask per chunk
 * and the number of nodes before it.  Returns their number.  Every level is a
 * handful of coalesced loads per CTA, nothing is sorted, and no list has to be
 * built beforehand. */
__device__ __forceinline__ int gather_masks(GatherSmem& sm, const GatherNodes& g, int nh, int x0, int y0, int z0) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  /* kHitsAhead chunks of a warp at a time: their loads in flight together */
  for (int h0 = warp; h0 < nh; h0 += kGatherWarps * kHitsAhead) {
    unsigned o[kHitsAhead][3];
#pragma unroll
    for (int u = 0; u < kHitsAhead; ++u) {
      const int h = h0 + u * kGatherWarps;
      const long i = h < nh ? (long)sm.hit[h] * 32 + lane : g.S;
      o[u][0] = o[u][1] = o[u][2] = 8u;   /* start - origin + 3: 0..6 where they meet */
      if (i < g.S) {
        const int* s = g.st + i * 3;
        o[u][0] = (unsigned)(s[0] - x0 + 3); o[u][1] = (unsigned)(s[1] - y0 + 3); o[u][2] = (unsigned)(s[2] - z0 + 3);
      }
    }
#pragma unroll
    for (int u = 0; u < kHitsAhead; ++u) {
      const int h = h0 + u * kGatherWarps;
      const unsigned m = __ballot_sync(0xffffffffu, o[u][0] < 7u && o[u][1] < 7u && o[u][2] < 7u);
      if (h >= nh) break;   /* uniform over the warp */
      if (lane == 0) sm.mask[h] = m;
      if (h < kOffHits) sm.hoff[h][lane] = (unsigned short)(o[u][0] | o[u][1] << 4 | o[u][2] << 8);
    }
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
    if (lane == 0) sm.pos[nh] = run;
  }
  __syncthreads();
  return sm.pos[nh];
}

/* The nodes of chunks [h0, h1) of sm.hit, in index order, into sm.ids. */
__device__ __forceinline__ void gather_ids(GatherSmem& sm, const GatherNodes& g, int h0, int h1, int x0, int y0,
                                           int z0) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, first = sm.pos[h0];
#pragma unroll 4
  for (int h = h0 + warp; h < h1; h += kGatherWarps) {
    const unsigned m = sm.mask[h];
    if ((m >> lane) & 1u) {
      const int k = sm.pos[h] - first + __popc(m & ((1u << lane) - 1u)), i = sm.hit[h] * 32 + lane;
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

/* Chunks [h0, h1) of sm.hit, L <= kListCap nodes, added to the threads' sums. */
__device__ __forceinline__ void gather_sum(GatherSmem& sm, const GatherNodes& g, int h0, int h1, int L, int x0, int y0,
                                           int z0, double& Fx, double& Fy, double& Fz) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const double cf = 1.0 / (64.0 * 1.0 * 1.0 * 1.0);
  gather_ids(sm, g, h0, h1, x0, y0, z0);
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
      const double* rec = sm.rec[buf];
      const unsigned* cov = sm.cover[buf][warp];
      const int n = min(kBatch, L - b0);
#pragma unroll 4
      for (int k = 0; k < n; ++k) {
        const double* r = rec + k * kNodeRec;
        const double2 fxy = *reinterpret_cast<const double2*>(r + 12);
        const double fz = r[14];
        const double tmp = __dmul_rn(__dmul_rn(__dmul_rn(cf, r[ox]), r[oy]), r[oz]);
        const double ax = __dmul_rn(fxy.x, tmp), ay = __dmul_rn(fxy.y, tmp), az = __dmul_rn(fz, tmp);
        if ((cov[k] >> lane) & 1u) {
          Fx = __dadd_rn(Fx, ax);
          Fy = __dadd_rn(Fy, ay);
          Fz = __dadd_rn(Fz, az);
        }
      }
    }
    __syncthreads();
  }
}

/* gather_tile of a tile with more chunks or nodes than the lists hold (a
 * crumpled sheet): a list at a time, from the start.  Apart from the common
 * form, because what it keeps over a sum would cost that one registers which
 * hold the cell's state (2% of a 128x64x64 step).  10,816 nodes strewn over a
 * 128x96x96 grid, us per step, with every chunk that meets the tile visited by
 * itself / a list at a time: 12,240 / 1,020; strewn over 30^3 690 / 193, over
 * 12^3 612 / 214, on a plane at 0.1 cells 558 / 268. */
__device__ __forceinline__ void gather_long(GatherSmem& sm, const GatherNodes& g, int x0, int y0, int z0, double& Fx,
                                            double& Fy, double& Fz) {
  for (long c0 = g.c_lo; c0 < g.c_hi;) {
    int nh = 0;
    __syncthreads();   /* the lists are no longer read */
    for (; c0 < g.c_hi && nh <= kHitCap - kGatherTPB; c0 += kGatherTPB) {
      const long c = c0 + threadIdx.x;
      append_in_order(sm, c < g.c_hi && box_meets(g.chunk_box + c * 6, x0, y0, z0), (int)c, sm.hit, nh);
    }
    const int n = gather_masks(sm, g, nh, x0, y0, z0);
    for (int h0 = 0, h1; h0 < nh; h0 = h1) {
      /* all of these chunks' nodes, or as many chunks as the list holds */
      h1 = nh;
      if (n - sm.pos[h0] > kListCap)
        for (h1 = h0 + 1; sm.pos[h1 + 1] - sm.pos[h0] <= kListCap;) ++h1;
      gather_sum(sm, g, h0, h1, sm.pos[h1] - sm.pos[h0], x0, y0, z0, Fx, Fy, Fz);
    }
  }
}

/* The spread force of the tile at (x0, y0, z0): thread t < 64 gets its
 * cell's sum over the nodes in index order (cell = 16 z + 4 y + x).  Called
 * by all kGatherTPB threads.  Warps 2 and 3 stage the next 64 nodes while
 * warps 0 and 1 sum the last: each sum is a serial chain (its order is the
 * reference's), so latency is kept out of it.  The 32 cells of a warp go
 * through the nodes together, a lane adding those that cover its cell: at
 * 128x64x64 (182 nodes on a tile, 64 of them on each cell) 11,500 cycles,
 * against 21,000 with each lane on its own list of covering nodes
 * (scattered shared-memory reads).  One warp with two cells per lane, which
 * halves those reads, took the launch at 128x64x64 from 17 to 20 us. */
__device__ __forceinline__ void gather_tile(GatherSmem& sm, const GatherNodes& g, int x0, int y0, int z0, double& Fx,
                                            double& Fy, double& Fz) {
  __syncthreads();   /* the previous tile's data is no longer read */
  const int nh = gather_chunks(sm, g, x0, y0, z0);
  const int n = nh <= kHitCap ? gather_masks(sm, g, nh, x0, y0, z0) : kListCap + 1;
  Fx = Fy = Fz = 0.0;
  if (n <= kListCap) gather_sum(sm, g, 0, nh, n, x0, y0, z0, Fx, Fy, Fz);
  else gather_long(sm, g, x0, y0, z0, Fx, Fy, Fz);
}

/* A move CTA: the 32 nodes of a chunk, four warps. */
constexpr int kMoveTPB = 128;
/* Cells a CTA's staged move holds in shared memory: the union box of its 32
 * nodes' stencils (along a fiber row ~5 x 20 x 5 cells).  Nodes whose starts
 * differ by 1 from one node's always fit. */
constexpr int kMoveCap = 640;
constexpr int kMoveTiles = 64;   /* tiles of the union box whose slots are staged */
static_assert(6 * 6 * 6 <= kMoveCap && 3 * 3 * 3 <= kMoveTiles, "a group of reach 1");

struct MoveSmem {
  double U[3][kMoveCap];
  int slot[kMoveTiles];
};

/* The move of the 32 nodes of a chunk (node i on lane l of every warp,
 * `live` if it moves), with the velocity of the union box of their stencils
 * staged once in shared memory: the four warps read each box cell's u from
 * its moment tile, then warp a < 3 sums component a of every node's 64
 * terms from shared memory, with ~5x fewer L2 requests than a node at a time
 * (neighbouring nodes' stencils overlap by 3 cells of 4).  A node's sum is a
 * serial chain of 64 terms, so a thread holds one component only; with one
 * warp that staged and summed all three for its nodes the launch took 10 us
 * at 16 x 16 nodes, this 6.
 * Nodes whose stencils lie too far apart for one box (a chunk that straddles
 * two rows of its sheet) are taken in groups near one another.  Called by
 * all kMoveTPB threads; ends with a barrier. */
__device__ __forceinline__ void move_chunk(MoveSmem& sm, double* __restrict__ nodes, const double* __restrict__ W,
                                           const int* __restrict__ st, long i, bool live, int ntx, int nty,
                                           const int* __restrict__ slot, const double* __restrict__ Utile, double dt) {
  const int t = threadIdx.x, warp = t >> 5;
  int is = 0, js = 0, ks = 0;
  double w[12], at = 0.0;
  if (live) {
    is = st[i * 3 + 0]; js = st[i * 3 + 1]; ks = st[i * 3 + 2];
    if (warp < 3) {   /* the weights this thread will need, on their way while the box is staged */
      const double2* p = reinterpret_cast<const double2*>(W + i * 12);
#pragma unroll
      for (int a = 0; a < 6; ++a) { w[2 * a] = p[a].x; w[2 * a + 1] = p[a].y; }
      at = nodes[i * 12 + warp];
    }
  }
  /* every warp holds the same 32 stencils, so what follows is uniform over
     the CTA */
  unsigned left = __ballot_sync(0xffffffffu, live);
  bool now = live;   /* the lane's node is in the group being moved */
  int reach = 16;
  while (left) {
    const int x0 = __reduce_min_sync(0xffffffffu, now ? is : INT_MAX), x1 = __reduce_max_sync(0xffffffffu, now ? is + 3 : INT_MIN);
    const int y0 = __reduce_min_sync(0xffffffffu, now ? js : INT_MAX), y1 = __reduce_max_sync(0xffffffffu, now ? js + 3 : INT_MIN);
    const int z0 = __reduce_min_sync(0xffffffffu, now ? ks : INT_MAX), z1 = __reduce_max_sync(0xffffffffu, now ? ks + 3 : INT_MIN);
    const int bx = x1 - x0 + 1, by = y1 - y0 + 1, bz = z1 - z0 + 1;
    const long vol = (long)bx * by * bz;
    const int tx0 = x0 >> 2, ty0 = y0 >> 2, tz0 = z0 >> 2;
    const int tbx = (x1 >> 2) - tx0 + 1, tby = (y1 >> 2) - ty0 + 1;
    const long ntb = (long)tbx * tby * ((z1 >> 2) - tz0 + 1);
    if (vol > kMoveCap || ntb > kMoveTiles) {
      /* too large: the nodes within `reach` of the first one, nearer and
         nearer until the box fits (at the latest at 1) */
      const int f = __ffs(left) - 1;
      const int fx = __shfl_sync(0xffffffffu, is, f), fy = __shfl_sync(0xffffffffu, js, f),
                fz = __shfl_sync(0xffffffffu, ks, f);
      now = ((left >> (t & 31)) & 1u) && abs(is - fx) <= reach && abs(js - fy) <= reach && abs(ks - fz) <= reach;
      reach >>= 1;
      continue;
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
    if (now && warp < 3) {
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
    left &= ~__ballot_sync(0xffffffffu, now);
    now = (left >> (t & 31)) & 1u;
    reach = 16;
    __syncthreads();
  }
}

}  // namespace lbib

#endif
