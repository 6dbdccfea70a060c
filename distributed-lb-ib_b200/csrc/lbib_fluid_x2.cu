/*
 * The one-grid launch of the FP64 two-cell step (lbib_x2.cuh) over the rows
 * away from the walls.  Twice the bytes per memory instruction of the
 * one-cell kernel: the AA pattern alone measures 87% of the HBM copy peak at
 * one cell per thread and 96% at two.
 */
#include "lbib_internal.h"
#include "lbib_x2.cuh"

using namespace lbib;

namespace {

constexpr int TPB = 128;

/* Resident blocks per SM each parity's kernel is compiled for (the register
 * budget): 3 x 128 threads at up to 168 registers. */
#ifndef LBIB_X2_MINB0
#define LBIB_X2_MINB0 3
#endif
#ifndef LBIB_X2_MINB1
#define LBIB_X2_MINB1 3
#endif

struct X2Params {
  FluidParams p;
  int nry;       /* interior rows in y: ny - 6 */
  int npairs;    /* pairs per row: (xhi - xlo + 1) / 2 */
  long pf;       /* L2 prefetch distance in blocks (0: none) */
  unsigned flat; /* pairs in all, rows end to end; 0: blocks per row */
  FastDiv dpairs, dnry;
};

/* Threads 0..18 ask L2 for plane q of the rows of the block pf blocks
 * later in launch order (blockIdx.x fastest): the loads it will issue. */
template <int PAR>
__device__ __forceinline__ void x2_prefetch(const X2Params& b, int q) {
  const long nrow = gridDim.x;
  const long L = (long)blockIdx.y * nrow + blockIdx.x + b.pf;
  if (L >= nrow * gridDim.y) return;
  const int row = (int)(L % nrow), pb = (int)(L / nrow);
  const int y = 3 + row % b.nry, z = 3 + row / b.nry;
  const int pr0 = pb * TPB;
  const int pr1 = pr0 + TPB < b.npairs ? pr0 + TPB : b.npairs;
  const FluidParams& p = b.p;
  const long idx = sidx(p, p.xlo + 2 * pr0, y, z);
  const double* src = PAR ? p.f + opp(q) * p.N + idx - link_offset(q, p.sx, (long)p.sx * p.ny) : p.f + q * p.N + idx;
  l2_prefetch(src, src + 2L * (pr1 - pr0), p.f, p.f + 19 * p.N);
}

template <int PAR>
__global__ void __launch_bounds__(TPB, PAR ? LBIB_X2_MINB1 : LBIB_X2_MINB0) lbib_fluid_step_x2(X2Params b) {
  if (b.flat) {
    const unsigned t = blockIdx.x * TPB + threadIdx.x;
    if (t >= b.flat) return;
    const unsigned row = fdiv(t, b.dpairs), z = fdiv(row, b.dnry);
    x2_pair<PAR>(b.p, b.p.xlo + 2 * (int)(t - row * b.npairs), 3 + (int)(row - z * b.nry), 3 + (int)z);
    return;
  }
  if (b.pf > 0 && threadIdx.x < 19) x2_prefetch<PAR>(b, threadIdx.x);
  const int pr = blockIdx.y * TPB + threadIdx.x;
  if (pr >= b.npairs) return;
  const int y = 3 + (int)(blockIdx.x % b.nry);
  const int z = 3 + (int)(blockIdx.x / b.nry);
  x2_pair<PAR>(b.p, b.p.xlo + 2 * pr, y, z);
}

}  // namespace

/* Interior-row ranges of this kernel: y in [3, ny-4], z in
 * [3, min(nz-4, zin_hi)].  Returns 0 when there are none. */
extern "C" int lbdev_bulk_rows(const lbib_device* d, int* nrows_y, int* nrows_z) {
  *nrows_y = d->ny - 6;
  int zb = d->nz - 4;
  if (d->zin_hi < zb) zb = d->zin_hi;
  *nrows_z = zb - 2;
  return (*nrows_y > 0 && *nrows_z > 0);
}

extern "C" int lbdev_launch_fluid_bulk(lbib_device* d, const void* fluid_params) {
  X2Params b;
  b.p = *(const FluidParams*)fluid_params;
  int nrz = 0;
  if (!lbdev_bulk_rows(d, &b.nry, &nrz)) return 0;
  b.npairs = (b.p.xhi - b.p.xlo + 1) / 2;
  b.pf = 0;
  if (d->l2_pf > 0) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d->device);
    b.pf = (long)d->l2_pf * sms * (d->parity ? LBIB_X2_MINB1 : LBIB_X2_MINB0);
  }
  dim3 grid((unsigned)((long)b.nry * nrz), (unsigned)((b.npairs + TPB - 1) / TPB));
  /* a block per TPB pairs of a row keeps every warp on one row; where that
     leaves more than 5% of the threads without a pair (62 pairs in rows of
     128 cells: half), the rows are laid end to end instead.  us of the
     kernel in even, odd steps, per row -> end to end: 9.3, 9.8 -> 7.2, 7.7
     at 64x32x32, 29, 32 -> 23, 25 at 128x64x64, 34, 39 -> 19, 24 at
     100x55x75 */
  const long pairs = (long)b.nry * nrz * b.npairs, slots = (long)grid.x * grid.y * TPB;
  b.flat = 0;
  if (pairs < 0.95 * slots && pairs + TPB < (1L << 31)) {
    b.flat = (unsigned)pairs;
    b.dpairs = fast_div((unsigned)b.npairs);
    b.dnry = fast_div((unsigned)b.nry);
    grid = dim3((unsigned)((pairs + TPB - 1) / TPB));
  }
  if (d->parity == 0) lbib_fluid_step_x2<0><<<grid, TPB, 0, d->fluid_stream>>>(b);
  else lbib_fluid_step_x2<1><<<grid, TPB, 0, d->fluid_stream>>>(b);
  d->kernel_launches++;
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
