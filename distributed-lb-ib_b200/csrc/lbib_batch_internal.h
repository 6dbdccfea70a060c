/*
 * Interface between the batched step's host code (lbib_batch.cu, FP64 and
 * the immersed boundary, compiled with -fmad=false) and its low-precision
 * fluid kernels (lbib_batch_lp.cu, contraction allowed).
 */
#ifndef LBIB_BATCH_INTERNAL_H
#define LBIB_BATCH_INTERNAL_H

#include <cuda_runtime_api.h>

#include "lbib_ib.cuh"

namespace lbib {

struct BatchDesc;

/* One fluid launch set of a batch. */
struct BatchFluid {
  cudaStream_t stream;
  int prec;                /* LBIB_PREC_* storage type */
  int par;                 /* AA parity of this step */
  int B;
  const void* P;           /* FluidParamsT<T>[B] */
  const void* WP;          /* WordsParams<T>[B] */
  const BatchDesc* desc;
  const int2* rowyz;       /* generic rows (y, z), each problem's contiguous */
  const int4* rblk;        /* generic-row blocks: (problem, first row, rows, chunk) */
  long nrblk;
  const int4* xblk;        /* FP64 two-cell items: (problem, first block, blocks) */
  long nxblk;
  const int* list;         /* touched tiles (global ids) */
  const int* count;
  const int* tile_inst;
  GatherNodes nodes;       /* the batch's sheets (a problem's chunks: batch_nodes) */
  double* Ftile;
  double* Utile;
  int* old_slot;           /* the other buffer's tile map, list and count: cleared for the next step */
  const int* old_list;
  const int* old_count;
  const int* err;
  int grid_tiles;          /* persistent grid for tile-list kernels */
};

/* The spread's gather and the forced cells: before everything else that reads
 * the forces. */
int batch_gather_lp(const BatchFluid& f);
int batch_gather_f64(const BatchFluid& f);
/* Generic rows. */
int batch_rows_lp(const BatchFluid& f);
int batch_rows_f64(const BatchFluid& f);
/* FP64 two-cell blocks. */
int batch_pairs_f64(const BatchFluid& f);
/* Word-kernel items (problem, first block, blocks) of one variant; the
 * variant a problem starts with. */
int batch_words_lp(const BatchFluid& f, int variant, const int4* blk, long nblk);
int batch_default_variant_lp(int prec);
int batch_variants_lp(int prec);
int batch_variant_cells_lp(int prec, int variant);   /* V of a variant */
/* Tile moments after the step (parity = the next step's). */
int batch_tile_moments_f64(const BatchFluid& f);
int batch_tile_moments_lp(const BatchFluid& f);

}  // namespace lbib

#endif
