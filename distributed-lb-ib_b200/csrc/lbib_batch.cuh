/*
 * Batched fluid kernels: many independent problems of uneven size advanced
 * by one launch per stage.
 *
 * Every problem keeps its own populations, tables and parameters (a
 * FluidParamsT<T> per problem in device memory, whose pointers reach into
 * the batch's pools); its tiles are a slice [tile0, tile0 + ntiles) of one
 * global tile space, so one touched-tile list and one slot space serve the
 * whole batch.  Work is enumerated across problems:
 *   rows     blocks of 128 cells over the rows the generic kernel takes,
 *            each problem's rows laid end to end;
 *   pairs    (FP64) blocks of 128 cell pairs of the two-cell kernel;
 *   words    blocks of the word kernel, (problem, block within problem);
 *            (the word blocks also step the cells x in {2, 3, nx-4, nx-3}
 *            of the rows whose first word they hold);
 *   tiles    the global touched-tile list, tile -> problem by a table.
 * A problem whose error word is set (a fiber stencil left its grid) is
 * skipped by every kernel from then on; the others continue.
 *
 * The per-cell arithmetic is the one-grid code (step_cell, x2_pair,
 * words_item, tile_moments_cell), so a problem advanced in a batch gets the same
 * numbers as the same problem on its own.
 */
#ifndef LBIB_BATCH_CUH
#define LBIB_BATCH_CUH

#include "lbib_ib.cuh"
#include "lbib_words.cuh"

namespace lbib {

/* What the node- and tile-level kernels need of a problem. */
struct BatchDesc {
  int nx, ny, nz, ntx, nty;
  int rows, cols;          /* its one sheet */
  int bulk;                /* bulk rows run the word kernel */
  int pinned;              /* row 0 of the sheet stays put */
  long tile0, ntiles;      /* slice of the global tile space */
  long node0, S;           /* nodes [node0, node0 + S); node0 % 32 == 0 */
  double bc, sc, sc2, ds1, ds2, dt;
};

/* A CTA's share of the word kernel: a run of consecutive blocks of one
 * problem, {problem, first block, blocks, 0}.  Before its first load a CTA
 * waits for its item, the problem's error word and its parameters, one after
 * the other; runs took a 128-problem 16-bit step from 1130 to 1050 us.  Up to
 * kRun blocks, fewer where the batch would not fill the chip several times
 * over.  (The FP64 pair kernel lost by it, 415 -> 435 and 519 us in even and odd
 * steps at 24 problems; its items have one block.) */
constexpr int kRun = 8;
inline int run_length(long blocks) {
  const long r = blocks / (148 * 24);
  return r < 1 ? 1 : r > kRun ? kRun : (int)r;
}

/* Copy a parameter struct into shared memory with the whole block. */
template <typename S>
__device__ __forceinline__ void block_copy(S& dst, const S* __restrict__ src) {
  static_assert(sizeof(S) % 4 == 0, "word copy");
  const uint32_t* a = reinterpret_cast<const uint32_t*>(src);
  uint32_t* b = reinterpret_cast<uint32_t*>(&dst);
  for (int i = threadIdx.x; i < (int)(sizeof(S) / 4); i += blockDim.x) b[i] = a[i];
  __syncthreads();
}

/* Generic rows: a block per 128 cells of a problem's rows, the rows of
 * problem k laid end to end (cell c of the item: row c / (nx-4), x = 2 +
 * c % (nx-4)), so small grids fill their blocks.  Item m = (problem, first
 * row in rowyz, rows of the problem, chunk). */
template <typename T, int PAR>
__global__ void __launch_bounds__(128) lbib_b_rows(const FluidParamsT<T>* __restrict__ P, const int2* __restrict__ rowyz,
                                                   const int4* __restrict__ rblk, const int* __restrict__ err) {
  __shared__ __align__(16) FluidParamsT<T> sp;
  const int4 m = rblk[blockIdx.x];
  if (err[2 * m.x]) return;
  block_copy(sp, P + m.x);
  const int w = sp.nx - 4;
  const int c = m.w * 128 + threadIdx.x;
  const int r = c / w;
  if (r >= m.z) return;
  const int2 yz = rowyz[m.y + r];
  step_cell<T, PAR>(sp, 2 + c % w, yz.x, yz.y);
}

/* Word kernel over the blocks of all problems that run it.  A block also
 * steps the plane-adjacent cells x in {2, 3, nx-4, nx-3} of the rows whose
 * first word it holds (generic per-cell rules), right after their words
 * went through the caches: a launch of their own re-read each of their
 * 2-byte populations from DRAM as a whole sector.  The slots those cells
 * read and write are theirs alone (AA), so the order within the launch
 * does not matter. */
template <typename T, int V, int PAR, int MINB>
__global__ void __launch_bounds__(WTPB, MINB) lbib_b_words(const WordsParams<T>* __restrict__ WP,
                                                           const int4* __restrict__ blk, const int* __restrict__ err) {
  __shared__ __align__(16) WordsParams<T> sb;
  const int4 m = blk[blockIdx.x];
  if (err[2 * m.x]) return;
  block_copy(sb, WP + m.x);
  const long first = (long)m.y * WTPB, end = first + (long)m.z * WTPB;
#pragma unroll 1
  for (long t = first; t < end; t += WTPB) words_item<T, V, PAR>(sb, t + threadIdx.x);
  const long r0 = fdiv((unsigned)(first + sb.gpr - 1), sb.dgpr);
  long r1 = fdiv((unsigned)(end + sb.gpr - 1), sb.dgpr);
  if (r1 > sb.nrows) r1 = sb.nrows;
  for (long i = threadIdx.x; i < 4 * (r1 - r0); i += WTPB) edge_cell<T, PAR>(sb.p, sb.nry, (int)(r0 + i / 4), (int)(i & 3));
}

/* The batch's sheets as problem d's gather sees them: its own chunks. */
__device__ __forceinline__ GatherNodes batch_nodes(GatherNodes g, const BatchDesc& d) {
  g.S = d.node0 + d.S;
  g.c_lo = d.node0 >> 5;
  g.c_hi = (g.S + 31) >> 5;
  return g;
}

/* Every listed tile: its spread force into its slot, and the step of its
 * cells in the word or pair kernel's range (which leaves them out), by the
 * CTA that has just written the force.  Launched before the generic rows,
 * which read the forces of their own cells. */
template <typename T, int PAR>
__global__ void __launch_bounds__(kGatherTPB, sizeof(T) == 8 ? 4 : 5) lbib_b_gather_step(const FluidParamsT<T>* __restrict__ P,
                                                                    const BatchDesc* __restrict__ D, GatherNodes g,
                                                                    const int* __restrict__ list,
                                                                    const int* __restrict__ count,
                                                                    const int* __restrict__ tile_inst,
                                                                    double* __restrict__ Ftile,
                                                                    const int* __restrict__ err) {
  __shared__ GatherSmem sm;
  const int n = *count, t = threadIdx.x;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int k = tile_inst[list[i]];
    if (err[2 * k]) continue;
    const BatchDesc& d = D[k];
    const int tile = (int)(list[i] - d.tile0);
    double Fx, Fy, Fz;
    gather_tile(sm, batch_nodes(g, d), tile % d.ntx * 4, tile / d.ntx % d.nty * 4, tile / (d.ntx * d.nty) * 4, Fx, Fy,
                Fz);
    if (t >= 64) continue;
    double* Ft = Ftile + (long)i * 192;
    Ft[t] = Fx; Ft[64 + t] = Fy; Ft[128 + t] = Fz;
    const FluidParamsT<T>& p = P[k];
    /* the thread reads back the force it has just written */
    if (d.bulk) forced_cell<T, PAR>(p, tile, t, min(p.nz - 4, p.zin_hi));
  }
}

/* (rho, u) of the touched tiles, over the global list. */
template <typename T, int PAR>
__global__ void lbib_b_tile_moments(const FluidParamsT<T>* __restrict__ P, const BatchDesc* __restrict__ D,
                                    const int* __restrict__ list, const int* __restrict__ count,
                                    const int* __restrict__ tile_inst, const double* __restrict__ Ftile,
                                    double* __restrict__ Utile, const int* __restrict__ err,
                                    int* __restrict__ old_slot, const int* __restrict__ old_list,
                                    const int* __restrict__ old_count) {
  clear_slots(old_slot, old_list, old_count);
  const int n = *count;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int tile = list[i];
    const int k = tile_inst[tile];
    if (err[2 * k]) continue;
    tile_moments_cell<T, PAR>(P[k], (int)(tile - D[k].tile0), i, threadIdx.x, Ftile, Utile);
  }
}

}  // namespace lbib

#endif
