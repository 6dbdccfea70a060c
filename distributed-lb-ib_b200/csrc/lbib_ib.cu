/*
 * Immersed-boundary kernels of one grid: thin wrappers over the device code
 * of lbib_ib.cuh (fiber forces, node preparation, the deterministic spread
 * as a per-tile gather, interpolation and move) and their launchers.
 * Compiled with -fmad=false: every expression keeps the reference's
 * operation order.
 */
#include "lbib_ib.cuh"

using namespace lbib;

namespace {

__global__ void lbib_fiber_forces(double* __restrict__ nodes, int R, int C, double bc, double sc, double sc2,
                                  double ds1, double ds2, int bend_bug) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= R * C) return;
  fiber_forces_node(nodes, R, C, bc, sc, sc2, ds1, ds2, bend_bug, i);
}

/* The sheets whose fiber forces the node preparation computes as well
 * (n = 0: none; the forces then come from lbib_fiber_forces). */
constexpr int kFuseSheets = 4;
struct SheetForces {
  int n, bend_bug;
  lbib_sheet_dev s[kFuseSheets];
};

/* A CTA per 32-node chunk: node_prep_warp by warps 0 to 3; warps 4 and 5,
 * when it has them, compute the nodes' fiber forces for the sheets `sf`
 * names (they read neighbours' positions and write the node's own force
 * fields only, so they run alongside).  list NULL: mark the tiles only.
 * Bound by the latency of one chunk's chain, 16,000 cycles when one warp took
 * all of its tiles: 11.1 -> 6.1 us a launch at 64x32x32, 23 -> 17.4 at
 * 512x256x256. */
__global__ void __launch_bounds__(192, 4) lbib_node_prep(double* __restrict__ nodes, long S, int nx, int ny, int nz,
                                                      int ntx, int nty, double* __restrict__ W, int* __restrict__ st,
                                                      int* __restrict__ chunk_box, int* __restrict__ super,
                                                      int* __restrict__ slot, int* __restrict__ list,
                                                      int* __restrict__ count, int* __restrict__ mark, int* err,
                                                      int step, SheetForces sf) {
  __shared__ double x[6][32];
  const long i = (long)blockIdx.x * 32 + (threadIdx.x & 31);
  const int part = threadIdx.x >> 5;
  if (part >= 4) {
    int k = 0;
    while (k + 1 < sf.n && i >= sf.s[k + 1].offset) ++k;
    const lbib_sheet_dev& h = sf.s[k];
    fiber_forces_pair(nodes + h.offset * 12, h.rows, h.cols, h.bc, h.sc, h.sc2, h.ds1, h.ds2, sf.bend_bug,
                      (int)(i - h.offset), i < S, part - 4, x);
    return;
  }
  node_prep_warp(nodes, i, i < S, S, part, nx, ny, nz, ntx, nty, 0, W, st, chunk_box, super, slot, list, count, mark,
                 err, step);
}

/* Every listed tile of columns tx in [tlo, thi) (an x-slab gathers the
 * tiles its own fluid cells read; the whole grid all): its force into its
 * slot.  super_next: the super-chunk boxes of the next step, emptied. */
__global__ void __launch_bounds__(kGatherTPB) lbib_spread_gather(GatherNodes g, const int* __restrict__ list,
                                                                 const int* __restrict__ count, int ntx, int nty,
                                                                 int tlo, int thi, double* __restrict__ Ftile,
                                                                 int* __restrict__ super_next, long nsuper,
                                                                 const int* err) {
  __shared__ GatherSmem sm;
  clear_super(super_next, nsuper);
  if (*(volatile const int*)err) return;
  const int n = *count;
  for (int it = blockIdx.x; it < n; it += gridDim.x) {
    const int tile = list[it], tx = tile % ntx;
    if (tx < tlo || tx >= thi) continue;   /* uniform over the block */
    double Fx, Fy, Fz;
    gather_tile(sm, g, tx * 4, (tile / ntx) % nty * 4, tile / (ntx * nty) * 4, Fx, Fy, Fz);
    if (threadIdx.x < 64) {
      double* Ft = Ftile + (long)it * 192;
      Ft[threadIdx.x] = Fx; Ft[64 + threadIdx.x] = Fy; Ft[128 + threadIdx.x] = Fz;
    }
  }
}

/* Nodes [i0, i1) that stay where they are (the pinned-row option). */
struct PinnedRows {
  int n;
  long lo[kFuseSheets], hi[kFuseSheets];
};

/* Nodes [i0, i1) of the concatenated sheets.  With `box` (a box-mode step's
 * next box), the box in tiles of the nodes' stencils, pinned ones included,
 * and `ring` tiles around them, is reduced into it (a warp reduction, then
 * six atomics per block). */
__global__ void __launch_bounds__(kMoveTPB) lbib_move_nodes(double* __restrict__ nodes, const double* __restrict__ W,
                                                            const int* __restrict__ st, long i0, long i1, int ntx,
                                                            int nty, const int* __restrict__ slot,
                                                            const double* __restrict__ Utile, double dt,
                                                            const int* err, int* __restrict__ box, int ring, int nx,
                                                            int ny, int nz, int* __restrict__ old_count,
                                                            PinnedRows pin) {
  __shared__ MoveSmem sm;
  if (old_count && blockIdx.x == 0 && threadIdx.x == 0) *old_count = 0;   /* the next step's list starts empty */
  const long i = i0 + (long)blockIdx.x * 32 + (threadIdx.x & 31);
  if (*(volatile const int*)err) return;   /* set by earlier launches only: uniform */
  const bool have = i < i1;
  bool live = have;
  for (int k = 0; k < pin.n; ++k) live = live && !(i >= pin.lo[k] && i < pin.hi[k]);
  move_chunk(sm, nodes, W, st, i, live, ntx, nty, slot, Utile, dt);
  if (!box || threadIdx.x >= 32) return;
  bool in = false;
  int is = 0, js = 0, ks = 0;
  if (have) {
    const double* m = nodes + i * 12;
    in = stencil_inside(m[0], nx) && stencil_inside(m[1], ny) && stencil_inside(m[2], nz);
    if (in) { is = stencil_start(m[0]); js = stencil_start(m[1]); ks = stencil_start(m[2]); }
  }
  const int b[6] = {__reduce_min_sync(0xffffffffu, in ? is >> 2 : INT_MAX),
                    __reduce_max_sync(0xffffffffu, in ? (is + 3) >> 2 : INT_MIN),
                    __reduce_min_sync(0xffffffffu, in ? js >> 2 : INT_MAX),
                    __reduce_max_sync(0xffffffffu, in ? (js + 3) >> 2 : INT_MIN),
                    __reduce_min_sync(0xffffffffu, in ? ks >> 2 : INT_MAX),
                    __reduce_max_sync(0xffffffffu, in ? (ks + 3) >> 2 : INT_MIN)};
  if (threadIdx.x == 0 && b[0] <= b[1]) {
    const int t[6] = {b[0], b[1], b[2], b[3], b[4], b[5]};
    const int n[3] = {(nx + 3) / 4, (ny + 3) / 4, (nz + 3) / 4};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      atomicMin(&box[2 * a], max(t[2 * a] - ring, 0));
      atomicMax(&box[2 * a + 1], min(t[2 * a + 1] + ring, n[a] - 1));
    }
  }
}

/* A tile map and its list: every entry out of the map, the list empty (one
 * block: the count is reset after its last read). */
__global__ void __launch_bounds__(1024) lbib_clear_tiles(int* __restrict__ slot, const int* __restrict__ list,
                                                         int* __restrict__ count) {
  const int n = *count;
  for (int i = threadIdx.x; i < n; i += blockDim.x) slot[list[i]] = -1;
  __syncthreads();
  if (threadIdx.x == 0) *count = 0;
}

/* The box, in tiles, of all stencils of the current node positions (one
 * block): what an overlapped fluid step leaves to the cells kernel that
 * runs after the spread.  Nodes whose stencil leaves the grid are left out
 * (the spread reports them).  No valid node: an empty box. */
__global__ void __launch_bounds__(1024) lbib_stencil_box(const double* __restrict__ nodes, long S, int nx, int ny,
                                                         int nz, int ring, int* __restrict__ box) {
  __shared__ int red[6][32];
  int b0 = INT_MAX, b1 = INT_MIN, b2 = INT_MAX, b3 = INT_MIN, b4 = INT_MAX, b5 = INT_MIN;
  for (long i0 = threadIdx.x; i0 < S; i0 += 4L * blockDim.x) {
    double x[4][3];   /* four nodes' loads in flight before any is used */
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long i = i0 + (long)u * blockDim.x;
      const double* m = nodes + (i < S ? i : 0) * 12;
      x[u][0] = i < S ? m[0] : -1.0; x[u][1] = m[1]; x[u][2] = m[2];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (!(stencil_inside(x[u][0], nx) && stencil_inside(x[u][1], ny) && stencil_inside(x[u][2], nz))) continue;
      const int is = stencil_start(x[u][0]), js = stencil_start(x[u][1]), ks = stencil_start(x[u][2]);
      b0 = min(b0, is); b1 = max(b1, is + 3);
      b2 = min(b2, js); b3 = max(b3, js + 3);
      b4 = min(b4, ks); b5 = max(b5, ks + 3);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    b0 = min(b0, __shfl_xor_sync(0xffffffffu, b0, o)); b1 = max(b1, __shfl_xor_sync(0xffffffffu, b1, o));
    b2 = min(b2, __shfl_xor_sync(0xffffffffu, b2, o)); b3 = max(b3, __shfl_xor_sync(0xffffffffu, b3, o));
    b4 = min(b4, __shfl_xor_sync(0xffffffffu, b4, o)); b5 = max(b5, __shfl_xor_sync(0xffffffffu, b5, o));
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0) { red[0][w] = b0; red[1][w] = b1; red[2][w] = b2; red[3][w] = b3; red[4][w] = b4; red[5][w] = b5; }
  __syncthreads();
  if (w == 0) {
    b0 = lane < nw ? red[0][lane] : INT_MAX; b1 = lane < nw ? red[1][lane] : INT_MIN;
    b2 = lane < nw ? red[2][lane] : INT_MAX; b3 = lane < nw ? red[3][lane] : INT_MIN;
    b4 = lane < nw ? red[4][lane] : INT_MAX; b5 = lane < nw ? red[5][lane] : INT_MIN;
    for (int o = 16; o > 0; o >>= 1) {
      b0 = min(b0, __shfl_xor_sync(0xffffffffu, b0, o)); b1 = max(b1, __shfl_xor_sync(0xffffffffu, b1, o));
      b2 = min(b2, __shfl_xor_sync(0xffffffffu, b2, o)); b3 = max(b3, __shfl_xor_sync(0xffffffffu, b3, o));
      b4 = min(b4, __shfl_xor_sync(0xffffffffu, b4, o)); b5 = max(b5, __shfl_xor_sync(0xffffffffu, b5, o));
    }
    if (lane == 0) {
      if (b0 > b1) { box[0] = 1; box[1] = 0; box[2] = 1; box[3] = 0; box[4] = 1; box[5] = 0; }
      else {
        box[0] = max((b0 >> 2) - ring, 0); box[1] = min((b1 >> 2) + ring, (nx + 3) / 4 - 1);
        box[2] = max((b2 >> 2) - ring, 0); box[3] = min((b3 >> 2) + ring, (ny + 3) / 4 - 1);
        box[4] = max((b4 >> 2) - ring, 0); box[5] = min((b5 >> 2) + ring, (nz + 3) / 4 - 1);
      }
    }
  }
}

/* Dense copy of the spread force for getters: zero, then each touched tile
 * of columns tx in [tlo, thi) (the tiles this state gathered). */
__global__ void lbib_scatter_force(const int* __restrict__ list, const int* __restrict__ count,
                                   const double* __restrict__ Ftile, int nx, int ny, int nz, int ntx, int nty, int tlo,
                                   int thi, double* __restrict__ fx, double* __restrict__ fy, double* __restrict__ fz) {
  const int n = *count;
  const int cell = threadIdx.x;
  for (int it = blockIdx.x; it < n; it += gridDim.x) {
    const int tile = list[it];
    const int tx = tile % ntx, ty = (tile / ntx) % nty, tz = tile / (ntx * nty);
    if (tx < tlo || tx >= thi) continue;
    const int x = tx * 4 + (cell & 3), y = ty * 4 + ((cell >> 2) & 3), z = tz * 4 + (cell >> 4);
    if (x < nx && y < ny && z < nz) {
      const long idx = ((long)z * ny + y) * nx + x;
      const double* Ft = Ftile + (long)it * 192;
      fx[idx] = Ft[cell]; fy[idx] = Ft[64 + cell]; fz[idx] = Ft[128 + cell];
    }
  }
}

}  // namespace

extern "C" int lbdev_launch_fiber_forces(lbib_device* d, int k) {
  const lbib_sheet_dev* s = &d->sh[k];
  const int n = s->rows * s->cols;
  lbib_fiber_forces<<<(n + 127) / 128, 128, 0, d->stream>>>(d->nodes + s->offset * 12, s->rows, s->cols, s->bc,
                                                            s->sc, s->sc2, s->ds1, s->ds2,
                                                            (d->compat & 1) != 0);
  d->kernel_launches++;
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int lbdev_launch_stencil_box(lbib_device* d) {
  lbib_stencil_box<<<1, 1024, 0, d->stream>>>(d->nodes, d->S, d->nx, d->ny, d->nz, lbdev_late_join(d), d->box + 6 * d->box_cur);
  d->kernel_launches++;
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

/* Buffer b's map and list emptied on `st`, after the launches that read them;
 * nothing to do where the last spread's entries are gone already. */
extern "C" int lbdev_launch_clear_tiles(lbib_device* d, int b, cudaStream_t st) {
  if (!d->tiles_left[b]) return 0;
  lbib_clear_tiles<<<1, 1024, 0, st>>>(d->tile_slot[b], d->tile_list[b], d->tile_count[b]);
  d->kernel_launches++;
  d->tiles_left[b] = 0;
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

/* The fiber forces fold into the node preparation for up to kFuseSheets
 * sheets: lbdev_launch_spread computes them when d->fuse_forces is set. */
extern "C" int lbdev_can_fuse_forces(const lbib_device* d) { return d->nsheets <= kFuseSheets; }

/* Node preparation: weights, stencil starts, boxes, the touched tiles (and,
 * with d->fuse_forces, the fiber forces).  The whole grid lists the tiles as
 * it meets them, from an empty list and a map that is all -1: a box-mode step
 * empties the buffer its successor fills, whatever else ran before (the
 * stages one by one, with some of them left out or repeated) is cleared here.
 * Every tile enters the list once and a node touches at most eight, so the
 * list ends below its d->cap entries.  An x-slab marks the tiles and compacts
 * the marks, because the slabs of one grid number their slots alike. */
extern "C" int lbdev_launch_prep(lbib_device* d, int step) {
  const int c = d->cur;
  cudaStream_t st = d->stream;
  SheetForces sf;
  sf.n = 0;
  sf.bend_bug = (d->compat & 1) != 0;
  if (d->fuse_forces && d->nsheets <= kFuseSheets) {
    sf.n = d->nsheets;
    for (int k = 0; k < d->nsheets; ++k) sf.s[k] = d->sh[k];
  }
  const int slab = lbdev_is_slab(d);
  if (!slab) {
    if (lbdev_launch_clear_tiles(d, c, st)) return -2;
    d->tiles_left[c] = LBIB_TILES_ALL;
  }
  lbib_node_prep<<<(unsigned)d->nchunks, sf.n ? 192 : 128, 0, st>>>(
      d->nodes, d->S, d->nx, d->ny, d->nz, d->ntx, d->nty, d->W, d->st, d->chunk_box, d->super[c], d->tile_slot[c],
      slab ? nullptr : d->tile_list[c], d->tile_count[c], d->tile_mark, d->err, step, sf);
  d->kernel_launches++;
  if (slab) {
    d->scan_tag = d->scan_tag % 255u + 1u;
    const unsigned nb = (unsigned)((d->ntiles + kScanBlock * kOnepassTiles - 1) / (kScanBlock * kOnepassTiles));
    lbib_compact_onepass<<<nb, kScanBlock, 0, st>>>(d->tile_mark, d->ntiles, (int)nb, d->scan_state, d->scan_tag,
                                                     d->tile_list[c], d->tile_slot[c], d->tile_count[c], d->err);
    d->kernel_launches++;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

/* Node preparation and the gather over the listed tiles. */
extern "C" int lbdev_launch_spread(lbib_device* d, int step) {
  if (lbdev_launch_prep(d, step)) return -2;
  const int c = d->cur;
  lbib_spread_gather<<<148 * 8, kGatherTPB, 0, d->stream>>>(gather_nodes(d), d->tile_list[c], d->tile_count[c], d->ntx,
                                                             d->nty, d->x_lo / 4, (d->x_hi + 3) / 4, d->Ftile[c],
                                                             d->super[c ^ 1], d->nsuper, d->err);
  d->kernel_launches++;
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

/* moveFiberSheet over all nodes; with the pinned-row option (no reference
 * counterpart) row 0 of every sheet stays where it is: kFuseSheets sheets
 * to a launch. */
extern "C" int lbdev_launch_move(lbib_device* d) {
  const int c = d->cur, pinned = (d->compat & LBIB_OPT_PIN_ROW0) != 0;
  /* the old list is emptied only once its map has been (a box-mode step) */
  int* old_count = d->tiles_left[c ^ 1] == LBIB_TILES_LIST ? d->tile_count[c ^ 1] : nullptr;
  const int per = pinned ? kFuseSheets : d->nsheets;
  for (int k0 = 0; k0 < d->nsheets; k0 += per) {
    const int k1 = k0 + per < d->nsheets ? k0 + per : d->nsheets;
    const long i0 = d->sh[k0].offset, i1 = d->sh[k1 - 1].offset + (long)d->sh[k1 - 1].rows * d->sh[k1 - 1].cols;
    PinnedRows pin;
    pin.n = pinned ? k1 - k0 : 0;
    for (int k = 0; k < pin.n; ++k) {
      pin.lo[k] = d->sh[k0 + k].offset;
      pin.hi[k] = pin.lo[k] + d->sh[k0 + k].cols;
    }
    lbib_move_nodes<<<(unsigned)((i1 - i0 + 31) / 32), kMoveTPB, 0, d->stream>>>(
        d->nodes, d->W, d->st, i0, i1, d->ntx, d->nty, d->tile_slot[c], d->Utile[c], (double)d->dt, d->err, d->box_next,
        lbdev_late_join(d), d->nx, d->ny, d->nz, k0 == 0 ? old_count : nullptr, pin);
    d->kernel_launches++;
  }
  if (old_count) d->tiles_left[c ^ 1] = 0;
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int lbdev_launch_scatter_force(lbib_device* d, double* fx, double* fy, double* fz) {
  const int c = d->cur;
  lbib_scatter_force<<<148 * 8, 64, 0, d->stream>>>(d->tile_list[c], d->tile_count[c], d->Ftile[c], d->nx, d->ny,
                                                     d->nz, d->ntx, d->nty, d->x_lo / 4, (d->x_hi + 3) / 4, fx, fy,
                                                     fz);
  d->kernel_launches++;
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
