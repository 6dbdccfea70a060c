/*
 * A small multilayer perceptron on the GPU -- the surrogate that screens
 * parameter sweeps -- with its training: BF16 weights and activations, FP32
 * accumulation on the tcgen05 tensor cores, FP32 master weights, GELU
 * hidden layers, a linear output layer, mean-squared error and Adam.  No
 * reference counterpart.
 *
 * Matrices: see lbib_mlp_tc.cuh for the chunk layout of the BF16 ones
 * (activations, dZ, weights); Z (FP32) has the same order, 8 consecutive
 * columns of a row together.  Row padding (to 128) is written as zeros by
 * every epilogue; columns are padded to 16 only.  Device memory of a net, per
 * batch row: 2 bytes for each width that is a layer's input, 4 more for each
 * hidden one, and twice 2 for the widest output.
 *
 * Shapes: widths w_0 .. w_L (input, hidden..., output); layer l maps w_l to
 * w_{l+1}.  Every width is padded to a multiple of 16 inside (the padded
 * weight rows and columns are zero and stay zero: their gradients vanish);
 * the ABI sees the unpadded shapes.  Parameters, in ABI order: for each
 * layer W_l [w_{l+1}][w_l] row-major, then b_l [w_{l+1}].
 *
 * One tile routine serves all products, C[M][N] = sum_k A(m,k) B(k,n), with
 * any operand transposed in place (so a transposed one needs no copy):
 * tcgen05.mma on 128 x 32 tiles with the accumulator in TMEM (gemm_tile
 * below), the weight gradients' long K split four ways with a fixed-order
 * reduction.  A training step is one
 * launch per layer forward, one per layer backward (that layer's dW, db and
 * the dZ of the layer below, which all need only its dZ) and Adam: 2L + 1
 * launches, chained by programmatic dependent launch, and one more for an
 * input of more than 16 columns.
 */
#include <math.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <type_traits>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/lbib.h"
#include "lbib_mlp_tc.cuh"

namespace {


/* Epilogues of a tile. */
enum Epi {
  EPI_STORE = 0,        /* C (fp32 out0) = acc, or a split-K partial            */
  EPI_GELU = 1,         /* A = gelu(acc + b) (bf16 out1)                        */
  EPI_GELU_KEEP = 2,    /* the same, and Z = acc + b (fp32 out0) for training   */
  EPI_OUT = 3,          /* Y = acc + b (fp32 out0, the first w columns)         */
  EPI_MSE = 4,          /* out1 = d(mean squared error)/dY (bf16), loss partial */
  EPI_GELU_BACK = 5,    /* out1 = acc * gelu'(Z) (bf16)                         */
};

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }

__device__ __forceinline__ float gelu_grad(float z) {
  const float cdf = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
  return cdf + z * pdf;
}

using lbib_tc::BK;
using lbib_tc::BM;
using lbib_tc::kStages;
using lbib_tc::NT;
using lbib_tc::Operand;

/* 128 x 32 tiles: at a batch of 1024 and a width of 256 (the sweep
 * surrogate) that is 64 tiles; 64-column tiles were 32 CTAs on 148 SMs. */
constexpr int BN = 32;
constexpr int kMaxSplit = 8;      /* split-K factors 1, 2, 4, 8             */
constexpr int kStageBytes = (BM + BN) * BK * 2;
constexpr int kSmem = kStages * kStageBytes + (2 * kStages + 1) * 8 + 16;
constexpr int kChunks = BN / 8;   /* column chunks of a tile: one per group of 4 warps */
constexpr int kEpiLd = BN + 1;    /* row stride of a split's partial tile */
static_assert(BM * kEpiLd * 4 <= kStages * kStageBytes, "the partial tile reuses the operand buffers");
static_assert(NT == 32 * 4 * kChunks, "an epilogue thread per chunk");

/* One product and what is done with it. */
struct Gemm {
  Operand A, B;           /* A(m, k), and B as X(n, k)                      */
  const float* X;         /* A instead: FP32 rows [M][xw] of few columns, rounded on the way in */
  int xw;
  __nv_bfloat16* copy;    /* with X: the rounded rows, in A's layout, or NULL */
  int M, N, K;
  int tn, tiles, split;   /* tiles along N, tiles, K splits                 */
  float* out0;            /* row-major, row stride ldc (EPI_STORE, EPI_OUT); Z (EPI_GELU_KEEP) */
  long ldc;
  __nv_bfloat16* out1;    /* BF16 result, in blocks of 128 rows of oC chunks */
  int oC;
  const float* aux;       /* bias                                           */
  const float* z;         /* EPI_GELU_BACK: pre-activations, in out1's order */
  const float* T;         /* EPI_MSE: targets [M][w]                        */
  int w;                  /* EPI_OUT, EPI_MSE: unpadded columns             */
  float* loss;            /* EPI_MSE: per-tile squared-error sums, or NULL  */
};

/* 8 floats of 32-byte aligned memory. */
__device__ __forceinline__ void load8(const float* p, float* v) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void store8(float* p, const float* v) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ uint4 pack8(const float* v) {
  __align__(16) __nv_bfloat16 e[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) e[i] = __float2bfloat16(v[i]);
  return *reinterpret_cast<const uint4*>(e);
}

/* The barriers and the TMEM address of a CTA, after its operand buffers. */
struct TileCtx {
  uint64_t *full, *done;   /* [kStages] slice arrived / its MMAs finished */
  uint32_t tmem;
};

/* Tile `tile` of product g, split z of g.split.
 *
 * Split K (EPI_STORE only): the g.split CTAs of a cluster share a tile;
 * CTA z sums the K elements [z Kc, (z+1) Kc), then each adds the partials of
 * its share of the tile's rows in z order, read from the others' shared
 * memory -- the same bits whatever the order in which the CTAs run.
 * `err` is set if an mbarrier wait ran out (the tile is then not written).
 *
 * An epilogue thread holds 8 columns of one row, as tcgen05.ld delivers
 * them; what it reads (Z, targets, bias) is loaded before it waits for the
 * products. */
template <int EPI>
__device__ __forceinline__ void gemm_tile(const Gemm& g, int tile, int z, uint8_t* smem, const TileCtx& c,
                                          int* __restrict__ err) {
  using namespace lbib_tc;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int m0 = (tile / g.tn) * BM, n0 = (tile % g.tn) * BN;
  /* this CTA's K range, all of it or its share of a split (shares in units
     of 64), and the slices of BK it lies in */
  const int units = (g.K + 63) / 64, per = (units + g.split - 1) / g.split;
  const int kbeg = min(z * per * 64, g.K), kend = min((z + 1) * per * 64, g.K);
  const int k00 = kbeg / BK * BK, nk = kend > kbeg ? (kend - k00 + BK - 1) / BK : 0;
  const uint32_t s0 = smem_u32(smem);
  const bool fp32_in = (EPI == EPI_GELU || EPI == EPI_GELU_KEEP || EPI == EPI_OUT || EPI == EPI_MSE) && g.X;
  auto extent = [&](int kk) { return min(BK, (kend - (k00 + kk * BK) + 15) / 16 * 16); };
  auto fetch = [&](int kk) {   /* one thread: the copies of slice kk */
    const int b = kk % kStages, kn = extent(kk), k0 = k00 + kk * BK;
    const uint32_t s = s0 + b * kStageBytes;
    mbar_expect(&c.full[b], (fp32_in ? 0 : slice_bytes<BM>(g.A, m0, kn)) + slice_bytes<BN>(g.B, n0, kn));
    if (!fp32_in) fetch_slice<BM>(s, g.A, m0, k0, kn, &c.full[b]);
    fetch_slice<BN>(s + BM * BK * 2, g.B, n0, k0, kn, &c.full[b]);
  };
  /* the FP32 input (kInlineInput columns at most: one slice), by all threads */
  auto convert = [&]() {
    for (int v = t; v < BM * (g.K / 8); v += NT) {
      const int r = v % BM, kb = v / BM, m = m0 + r, k = kb * 8;
      float x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = m < g.M && k + i < g.xw ? g.X[(long)m * g.xw + k + i] : 0.0f;
      const uint4 u = pack8(x);
      *reinterpret_cast<uint4*>(smem + (kb * BM + r) * 16) = u;
      if (g.copy && n0 == 0) *reinterpret_cast<uint4*>(g.copy + (((long)(m0 / BM) * g.A.C + kb) * BM + r) * 8) = u;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  };
  bool ok = true;
  const int lead = nk < kStages ? nk : kStages;
  if (t == 0)
    for (int kk = 0; kk < lead; ++kk) fetch(kk);
  if (fp32_in) {
    convert();
    __syncthreads();
  }
  const uint32_t idesc = instr_desc_bf16(BM, BN, g.A.mn, g.B.mn);
  auto multiply = [&](int kk) {   /* one thread: the MMAs of slice kk */
    const int b = kk % kStages, k0 = k00 + kk * BK;
    if (!mbar_wait(&c.full[b], (kk / kStages) & 1)) return false;
    tc_fence_after();
    const uint32_t a = s0 + b * kStageBytes;
    const int j0 = kk == 0 ? (kbeg - k0) / 16 : 0, j1 = extent(kk) / 16;
#pragma unroll 4
    for (int j = j0; j < j1; ++j)
      mma_bf16(c.tmem, operand_desc<BM>(a, g.A.mn, j), operand_desc<BN>(a + BM * BK * 2, g.B.mn, j), idesc,
               (kk > 0 || j > j0) ? 1u : 0u);
    mma_commit(&c.done[b]);
    return true;
  };
  if (t == 32)
    for (int kk = 0; kk < nk && ok; ++kk) ok = multiply(kk);
  /* refills, each once the MMAs that read the buffer are done */
  if (t == 0)
    for (int kk = kStages; kk < nk && ok; ++kk) {
      ok = mbar_wait(&c.done[kk % kStages], (kk / kStages - 1) & 1);
      if (ok) fetch(kk);
    }
  /* warp w holds TMEM lanes 32 (w % 4) .., columns 8 (w / 4) .. */
  const int row = (warp & 3) * 32 + lane, ch = warp >> 2;
  const int m = m0 + row, n = n0 + 8 * ch;
  const bool nin = n < g.N, live = nin && m < g.M;
  const long at = (((long)(m0 / BM) * g.oC + n / 8) * BM + row) * 8;   /* the thread's chunk */
  float pre[8], bias[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) { pre[i] = 0.0f; bias[i] = 0.0f; }
  if constexpr (EPI == EPI_GELU_BACK) {
    if (live) load8(g.z + at, pre);
  } else if constexpr (EPI != EPI_STORE) {
    if (nin) load8(g.aux + n, bias);
    if constexpr (EPI == EPI_MSE) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (live && n + i < g.w) pre[i] = g.T[(long)m * g.w + n + i];
    }
  }
  /* the last commit covers every MMA of the tile */
  if (nk > 0) ok = ok && mbar_wait(&c.done[(nk - 1) % kStages], ((nk - 1) / kStages) & 1);
  ok = __syncthreads_and(ok);
  tc_fence_after();
  const bool split = EPI == EPI_STORE && g.split > 1;
  if (!ok) {
    if (t == 0) atomicExch(err, 1);
    if (split) { cluster_sync(); cluster_sync(); }   /* the cluster's other CTAs meet here */
    return;
  }
  float v[8];
  if (nk > 0) tmem_ld8(c.tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(8 * ch), v);
  else
    for (int i = 0; i < 8; ++i) v[i] = 0.0f;   /* no K slice in this split */
  tc_fence_before();
  if constexpr (EPI == EPI_STORE) {
    if (!split) {
      if (live) store8(g.out0 + (long)m * g.ldc + n, v);
      return;
    }
    float* ep = reinterpret_cast<float*>(smem);
#pragma unroll
    for (int i = 0; i < 8; ++i) ep[row * kEpiLd + 8 * ch + i] = v[i];
    cluster_sync();
    const int rows = BM / g.split;   /* this CTA's share: rows z * rows .. */
    for (int r = z * rows + warp; r < (z + 1) * rows; r += NT / 32) {
      float p[kMaxSplit];
#pragma unroll
      for (int k = 0; k < kMaxSplit; ++k) p[k] = k < g.split ? ld_cluster(ep + r * kEpiLd + lane, k) : 0.0f;
      float acc = 0.0f;
#pragma unroll
      for (int k = 0; k < kMaxSplit; ++k)
        if (k < g.split) acc += p[k];
      if (m0 + r < g.M && n0 + lane < g.N) g.out0[(long)(m0 + r) * g.ldc + n0 + lane] = acc;
    }
    cluster_sync();   /* no CTA leaves while its partials are read */
    return;
  } else {
    float loss = 0.0f, y[8];
    const float mse_n = (float)g.M * (float)g.w;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float x = v[i];
      if constexpr (EPI == EPI_GELU_BACK) {
        y[i] = x * gelu_grad(pre[i]);
      } else {
        x += bias[i];
        v[i] = x;
        if constexpr (EPI == EPI_MSE) {
          float d = 0.0f;
          if (live && n + i < g.w) {
            const float e = x - pre[i];
            loss += e * e;
            d = 2.0f * e / mse_n;
          }
          y[i] = d;
        } else {
          y[i] = EPI == EPI_OUT ? x : gelu(x);
        }
      }
      if (!live) y[i] = 0.0f;   /* the padding rows */
    }
    if constexpr (EPI == EPI_OUT) {
      if (live) {
        float* o = g.out0 + (long)m * g.ldc + n;
        if (n + 8 <= g.w && ((reinterpret_cast<uintptr_t>(o) | (uintptr_t)(g.ldc * 4)) & 15) == 0) {
          store8(o, y);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (n + i < g.w) o[i] = y[i];
        }
      }
    } else if (nin) {
      *reinterpret_cast<uint4*>(g.out1 + at) = pack8(y);
      if (EPI == EPI_GELU_KEEP) store8(g.out0 + at, v);
    }
    if constexpr (EPI == EPI_MSE) {
      if (g.loss) {
        /* the tile's squared error, in a fixed order (the operand buffers
           are free: every MMA is done) */
        float* ep = reinterpret_cast<float*>(smem);
        for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
        if (lane == 0) ep[warp] = loss;
        __syncthreads();
        if (t == 0) {
          float s = 0.0f;
          for (int k = 0; k < NT / 32; ++k) s += ep[k];
          g.loss[tile] = s;
        }
      }
    }
  }
}

/* TMEM columns and the slice barriers, before the kernel's first global
 * access (so that they overlap the tail of the kernel before it). */
__device__ __forceinline__ TileCtx tile_begin(uint8_t* smem) {
  using namespace lbib_tc;
  TileCtx c;
  c.full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
  c.done = c.full + kStages;
  uint32_t* slot = reinterpret_cast<uint32_t*>(c.done + kStages);
  if (threadIdx.x < 32) tmem_alloc<BN>(slot);
  if (threadIdx.x == 32) {
    for (int k = 0; k < 2 * kStages; ++k) mbar_init(&c.full[k], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  c.tmem = *slot;
  return c;
}

__device__ __forceinline__ void tile_end(uint32_t tmem) {
  lbib_tc::tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) lbib_tc::tmem_free<BN>(tmem);
}

/* FP32 rows [M][w] rounded into the chunk layout of `out` (C chunks a row, the
 * rows up to a multiple of 128 and the columns past w zero): 32 rows of 8
 * chunks a CTA, 256 bytes read and 64 written at a time. */
constexpr int kInputRows = 32, kInputChunks = 8;
__global__ void __launch_bounds__(kInputRows * kInputChunks) mlp_input(const float* __restrict__ X, int M, int w, int C,
                                                                      __nv_bfloat16* __restrict__ out) {
  lbib_tc::pdl_trigger();
  const int nc = (C + kInputChunks - 1) / kInputChunks;
  const int c = blockIdx.x % nc * kInputChunks + threadIdx.x % kInputChunks;
  const long r = (long)(blockIdx.x / nc) * kInputRows + threadIdx.x / kInputChunks;
  lbib_tc::pdl_wait();
  if (c >= C) return;
  const float* p = X + r * w + 8 * c;
  float x[8];
  if (r < M && 8 * c + 8 <= w && ((reinterpret_cast<uintptr_t>(X) | (uintptr_t)w * 4) & 15) == 0) {
    load8(p, x);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = r < M && 8 * c + i < w ? p[i] : 0.0f;
  }
  *reinterpret_cast<uint4*>(out + ((r / BM * C + c) * BM + r % BM) * 8) = pack8(x);
}

/* A layer forward: C = A W^T + b and its epilogue, a CTA per tile.  At
 * 1024 x 256 x 256 with GELU 6.0 us (46 us with 128 x 64 tiles staged one K
 * slice at a time by dependent loads): 3.5 us in the CTA -- the copies'
 * latency, 16 MMAs, 2000 cycles of erf -- and the launch.  A training step
 * of the sweep surrogate (batch 1024, 5 -> 4 x 256 -> 192) went from 27
 * launches and 590 us to 11 and 76 us. */
template <int EPI>
__global__ void __launch_bounds__(NT) mlp_layer(const __grid_constant__ Gemm g, int* __restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  lbib_tc::pdl_trigger();
  const TileCtx c = tile_begin(smem);
  lbib_tc::pdl_wait();
  gemm_tile<EPI>(g, blockIdx.x, 0, smem, c, err);
  tile_end(c.tmem);
}

/* db[n] = sum over the batch of dZ[:, n] for the 16 columns of block j, in a
 * fixed order: 32 row groups r, r + 32, ... summed in turn, then the 32
 * partial sums of a column in order. */
constexpr int kBiasCols = 16;
__device__ __forceinline__ void bias_grad(const Operand& dZ, int B, int w, int j, float* __restrict__ db,
                                          float* __restrict__ part) {
  /* 8 consecutive threads on a chunk, consecutive rows next */
  const int r0 = (threadIdx.x >> 3) & 31, c = (threadIdx.x & 7) + 8 * (threadIdx.x >> 8);
  const int n = j * kBiasCols + c;
  float s = 0.0f;
  if (n < w) {
    const __nv_bfloat16* p = dZ.p + (long)(n / 8) * BM * 8 + n % 8;
#pragma unroll 16
    for (int r = r0; r < B; r += 32) s += __bfloat162float(p[((long)(r / BM) * dZ.C * BM + r % BM) * 8]);
  }
  part[r0 * kBiasCols + c] = s;
  __syncthreads();
  if (threadIdx.x < kBiasCols && j * kBiasCols + threadIdx.x < w) {
    float t = 0.0f;
    for (int k = 0; k < 32; ++k) t += part[k * kBiasCols + threadIdx.x];
    db[j * kBiasCols + threadIdx.x] = t;
  }
}
static_assert(NT / kBiasCols == 32, "32 row groups");

/* A layer backward, from its dZ: the CTAs of one launch share three
 * independent jobs -- the tiles of dW = dZ^T X (split along the batch), the
 * tiles of dZ_below = (dZ W) gelu'(Z_below), and the bias gradient's column
 * blocks -- so that a layer costs one launch and its jobs fill the chip
 * together (64 + 64 + 16 CTAs at the surrogate's hidden layers). */
struct LayerBack {
  Gemm dW, dA;
  int n_dW, n_dA;                /* CTAs of each (dA: 0 at the first layer), whole clusters */
  Operand dZ;
  int batch, w;
  float* db;
};

__global__ void __launch_bounds__(NT, 2) mlp_layer_back(const __grid_constant__ LayerBack a, int* __restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  lbib_tc::pdl_trigger();
  const int b = blockIdx.x;
  if (b >= a.n_dW + a.n_dA) {
    lbib_tc::pdl_wait();
    bias_grad(a.dZ, a.batch, a.w, b - a.n_dW - a.n_dA, a.db, reinterpret_cast<float*>(smem));
    return;
  }
  const TileCtx c = tile_begin(smem);
  lbib_tc::pdl_wait();
  if (b >= a.n_dA) {
    /* a cluster's CTAs are consecutive: rank z sums split z of the tile */
    gemm_tile<EPI_STORE>(a.dW, (b - a.n_dA) / a.dW.split, (b - a.n_dA) % a.dW.split, smem, c, err);
  } else if (b < a.dA.tiles) {
    gemm_tile<EPI_GELU_BACK>(a.dA, b, 0, smem, c, err);
  }
  tile_end(c.tmem);
}

/* The loss from the tiles' squared-error sums. */
__global__ void mlp_sum(const float* __restrict__ part, int n, float scale, float* __restrict__ out) {
  __shared__ float s[256];
  lbib_tc::pdl_trigger();
  lbib_tc::pdl_wait();
  float v = 0.0f;
  for (int i = threadIdx.x; i < n; i += 256) v += part[i];
  s[threadIdx.x] = v;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = s[0] * scale;
}

/* Adam on the fp32 master copy; refresh the bf16 weights. */
__global__ void mlp_adam(float* __restrict__ p, const float* __restrict__ gr, float* __restrict__ m,
                         float* __restrict__ v, long n, float lr, float b1, float b2, float eps, float c1, float c2,
                         __nv_bfloat16* __restrict__ wbf, const int2* __restrict__ is_w) {
  lbib_tc::pdl_trigger();
  lbib_tc::pdl_wait();
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float g = gr[i];
  const float mi = b1 * m[i] + (1.0f - b1) * g;
  const float vi = b2 * v[i] + (1.0f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  const float x = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  p[i] = x;
  const int2 at = is_w[i];
  if (at.x >= 0) {
    const __nv_bfloat16 w = __float2bfloat16(x);
    wbf[at.x] = w;   /* W_l, and its transpose */
    wbf[at.y] = w;
  }
}

long align_up(long v, long a) { return (v + a - 1) / a * a; }

}  // namespace

/* ------------------------------------------------------------ state */

struct lbib_mlp {
  int L;
  int* w;               /* [L+1] widths */
  int* wp;              /* [L+1] padded */
  int max_batch;
  char* mem;            /* the device allocation the buffers below are parts of */
  long np;              /* padded parameter count */
  float *p, *g, *m, *v; /* master params, grads, Adam moments (padded layout) */
  int2* wmap;           /* padded param index -> its places in wbf, or -1 */
  /* the chunk-layout matrices (lbib_mlp_tc.cuh) */
  long rows;            /* batch rows: max_batch to a multiple of 128     */
  __nv_bfloat16* wbf;   /* bf16 weights: per layer W [wp_{l+1}][wp_l] and its transpose, */
  long nw;              /*   rows padded to 32, in blocks of 32           */
  long* woff;           /* [L] offset of W_l in p (padded) */
  long* boff;           /* [L] offset of b_l in p */
  long* wbo;            /* [2 L] offsets of W_l and its transpose in wbf  */
  __nv_bfloat16** act;  /* [L] activations, rows x wp_l; act[0] = input   */
  __nv_bfloat16* dz[2]; /* layer l's dZ, rows x wp_{l+1}, in dz[l & 1]    */
  float** z;            /* [L-1] pre-activations fp32, rows x wp_{l+1}    */
  float* part;          /* squared-error sums of the output layer's tiles */
  float* d_loss;
  int* d_err;           /* a tensor-core GEMM's mbarrier wait ran out     */
  long steps;
  cudaStream_t stream;  /* where the work runs: own_stream or the caller's */
  cudaStream_t own_stream;
};

namespace {

int set_smem_limits() {
  const void* k[] = {(const void*)mlp_layer<EPI_GELU>, (const void*)mlp_layer<EPI_GELU_KEEP>,
                     (const void*)mlp_layer<EPI_OUT>, (const void*)mlp_layer<EPI_MSE>, (const void*)mlp_layer_back};
  for (const void* f : k)
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) return -2;
  return 0;
}

/* A launch whose kernel may start while the one before it on the stream
 * finishes (it waits, before its first global access, until that one is
 * done: pdl_wait). */
template <typename... P, typename... A>
int launch(void (*kernel)(P...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t st, unsigned cluster,
           A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(blocks);
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  c.attrs = at;
  c.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&c, kernel, (P)args...) == cudaSuccess ? 0 : -2;
}

/* Layer l's matrices as operands: rows as the tile's rows, or columns; W_l
 * [out][in] or its transpose. */
Operand act_op(const lbib_mlp* n, int l, int mn) { return Operand{n->act[l], n->wp[l] / 8, BM, mn}; }
Operand dz_op(const lbib_mlp* n, int l, int mn) { return Operand{n->dz[l & 1], n->wp[l + 1] / 8, BM, mn}; }
Operand w_op(const lbib_mlp* n, int l, int transposed) {
  return Operand{n->wbf + n->wbo[2 * l + transposed], n->wp[l + transposed] / 8, BN, 0};
}

Gemm product(Operand A, Operand B, int M, int N, int K) {
  Gemm g;
  memset(&g, 0, sizeof(g));
  g.A = A; g.B = B;
  g.M = M; g.N = N; g.K = K;
  g.tn = (N + BN - 1) / BN;
  g.tiles = g.tn * ((M + BM - 1) / BM);
  g.split = 1;
  return g;
}

/* Layer 0 rounds up to kInlineInput columns of the caller's FP32 rows itself,
 * in every column tile; wider ones are rounded once by a launch before it.  us
 * of a forward, itself / launch before, batch 1024: 16 -> 64 columns 30.6 /
 * 29.2 (batch 128: 27.2 / 28.3; training steps 22.0 / 23.1 and 16.4 / 16.6),
 * 32 -> 64 35.1 / 29.2, 256 -> 256 47 / 37, 4096 -> 4096 2400 / 148. */
constexpr int kInlineInput = 16;
static_assert(kInlineInput <= BK, "one slice");
bool inline_input(const lbib_mlp* n) { return n->wp[0] <= kInlineInput; }

/* `batch` wider FP32 rows into act[0]. */
int stage_input(lbib_mlp* n, const float* X, int batch) {
  if (inline_input(n)) return 0;
  const int C = n->wp[0] / 8;
  const long blocks = align_up(batch, BM) / kInputRows * ((C + kInputChunks - 1) / kInputChunks);
  return launch(mlp_input, (unsigned)blocks, kInputRows * kInputChunks, 0, n->stream, 1, X, batch, n->w[0], C, n->act[0]);
}

/* Layer l forward of `batch` rows; X: layer 0's input, if it reads it itself. */
Gemm layer_product(lbib_mlp* n, int l, const float* X, int batch) {
  Gemm g = product(act_op(n, l, 0), w_op(n, l, 0), batch, n->wp[l + 1], n->wp[l]);
  if (l == 0 && inline_input(n)) { g.X = X; g.xw = n->w[0]; }
  g.aux = n->p + n->boff[l];
  g.oC = n->wp[l + 1] / 8;
  if (l + 1 < n->L) g.out1 = n->act[l + 1];
  return g;
}

/* Y [batch][w_L] of `batch` rows. */
int forward(lbib_mlp* n, const float* X, int batch, float* Y) {
  if (stage_input(n, X, batch)) return -2;
  for (int l = 0; l < n->L; ++l) {
    Gemm g = layer_product(n, l, X, batch);
    int rc;
    if (l + 1 < n->L) {
      rc = launch(mlp_layer<EPI_GELU>, g.tiles, NT, kSmem, n->stream, 1, g, n->d_err);
    } else {
      g.out0 = Y; g.w = n->w[n->L]; g.ldc = n->w[n->L];
      rc = launch(mlp_layer<EPI_OUT>, g.tiles, NT, kSmem, n->stream, 1, g, n->d_err);
    }
    if (rc) return rc;
  }
  return 0;
}

/* Gradients of the mean-squared error on one batch into n->g (padded
 * layout), and the loss into n->d_loss when it is wanted. */
int gradients(lbib_mlp* n, const float* X, const float* T, int batch, bool want_loss) {
  const int L = n->L;
  if (stage_input(n, X, batch)) return -2;
  for (int l = 0; l < L; ++l) {
    Gemm g = layer_product(n, l, X, batch);
    if (l == 0 && g.X) g.copy = n->act[0];                     /* read again by dW of layer 0 */
    int rc;
    if (l + 1 < L) {
      g.out0 = n->z[l];
      rc = launch(mlp_layer<EPI_GELU_KEEP>, g.tiles, NT, kSmem, n->stream, 1, g, n->d_err);
    } else {
      g.out1 = n->dz[l & 1]; g.T = T; g.w = n->w[L];
      g.loss = want_loss ? n->part : NULL;
      rc = launch(mlp_layer<EPI_MSE>, g.tiles, NT, kSmem, n->stream, 1, g, n->d_err);
      if (!rc && want_loss)
        rc = launch(mlp_sum, 1, 256, 0, n->stream, 1, (const float*)n->part, g.tiles,
                    1.0f / ((float)batch * (float)n->w[L]), n->d_loss);
    }
    if (rc) return rc;
  }
  for (int l = L - 1; l >= 0; --l) {
    const int in = n->wp[l], out = n->wp[l + 1];
    LayerBack a;
    memset(&a, 0, sizeof(a));
    /* dW = dZ^T X: M = out, N = in, K = batch.  A long K over few output
       tiles is split so that enough CTAs share it; the factor depends on
       the shape only (counted in tiles of 64 columns and K slices of 64;
       4 ways at the surrogate's hidden layers) */
    a.dW = product(dz_op(n, l, 1), act_op(n, l, 1), out, in, batch);
    const int wide = ((in + 63) / 64) * ((out + BM - 1) / BM), nkt = (batch + 63) / 64;
    int sk = 1;
    while (sk * 2 <= kMaxSplit && wide * sk < 32 && nkt >= 4 * sk * 2) sk *= 2;
    a.dW.split = sk;
    a.dW.out0 = n->g + n->woff[l];
    a.dW.ldc = in;
    a.n_dW = a.dW.tiles * sk;
    a.dZ = dz_op(n, l, 0); a.batch = batch; a.w = out;
    a.db = n->g + n->boff[l];
    if (l > 0) {
      /* dZ_{l-1} = (dZ W) * gelu'(Z_{l-1}): M = batch, N = in, K = out */
      a.dA = product(dz_op(n, l, 0), w_op(n, l, 1), batch, in, out);
      a.dA.out1 = n->dz[(l - 1) & 1];
      a.dA.oC = in / 8;
      a.dA.z = n->z[l - 1];
      a.n_dA = (a.dA.tiles + sk - 1) / sk * sk;
    }
    const int n_db = ((out + kBiasCols - 1) / kBiasCols + sk - 1) / sk * sk;
    if (launch(mlp_layer_back, (unsigned)(a.n_dW + a.n_dA + n_db), NT, kSmem, n->stream, sk, a, n->d_err)) return -2;
  }
  return 0;
}

/* ABI parameter index <-> padded index. */
long abi_count(const lbib_mlp* n) {
  long c = 0;
  for (int l = 0; l < n->L; ++l) c += (long)n->w[l + 1] * n->w[l] + n->w[l + 1];
  return c;
}

template <typename F>
void for_each_param(const lbib_mlp* n, F f) {
  long a = 0;
  for (int l = 0; l < n->L; ++l) {
    for (int r = 0; r < n->w[l + 1]; ++r)
      for (int c = 0; c < n->w[l]; ++c) f(a++, n->woff[l] + (long)r * n->wp[l] + c);
    for (int r = 0; r < n->w[l + 1]; ++r) f(a++, n->boff[l] + r);
  }
}

int refresh_bf16(lbib_mlp* n) {
  /* wbf from the master copy (host round trip; set-up only) */
  float* hp = (float*)malloc(sizeof(float) * n->np);
  int2* map = (int2*)malloc(sizeof(int2) * n->np);
  const long nw = n->nw;
  __nv_bfloat16* hw = (__nv_bfloat16*)malloc(sizeof(__nv_bfloat16) * nw);
  int rc = (!hp || !map || !hw) ? -5 : 0;
  if (!rc && cudaMemcpy(hp, n->p, sizeof(float) * n->np, cudaMemcpyDeviceToHost) != cudaSuccess) rc = -2;
  if (!rc && cudaMemcpy(map, n->wmap, sizeof(int2) * n->np, cudaMemcpyDeviceToHost) != cudaSuccess) rc = -2;
  if (!rc) {
    for (long i = 0; i < nw; ++i) hw[i] = __float2bfloat16(0.0f);
    for (long i = 0; i < n->np; ++i)
      if (map[i].x >= 0) hw[map[i].x] = hw[map[i].y] = __float2bfloat16(hp[i]);
    if (cudaMemcpy(n->wbf, hw, sizeof(__nv_bfloat16) * nw, cudaMemcpyHostToDevice) != cudaSuccess) rc = -2;
  }
  free(hp);
  free(map);
  free(hw);
  return rc;
}

/* splitmix64 stream for the initial weights */
double uniform01(uint64_t* s) {
  uint64_t z = (*s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

}  // namespace

extern "C" {

lbib_mlp* lbib_mlp_create(int n_layers, const int* widths, int max_batch, unsigned long long seed) {
  if (n_layers < 1 || n_layers > 16 || !widths || max_batch < 1) return NULL;
  for (int l = 0; l <= n_layers; ++l)
    if (widths[l] < 1 || widths[l] > 4096) return NULL;
  lbib_mlp* n = (lbib_mlp*)calloc(1, sizeof(lbib_mlp));
  if (!n) return NULL;
  const int L = n_layers;
  n->L = L;
  n->max_batch = max_batch;
  n->w = (int*)calloc(L + 1, sizeof(int));
  n->wp = (int*)calloc(L + 1, sizeof(int));
  n->woff = (long*)calloc(L, sizeof(long));
  n->boff = (long*)calloc(L, sizeof(long));
  n->wbo = (long*)calloc(2 * L, sizeof(long));
  n->act = (__nv_bfloat16**)calloc(L + 1, sizeof(void*));
  n->z = (float**)calloc(L, sizeof(void*));
  int rc = (!n->w || !n->wp || !n->woff || !n->boff || !n->wbo || !n->act || !n->z) ? -5 : 0;
  n->rows = align_up(max_batch, BM);
  long np = 0, nw = 0;
  for (int l = 0; l <= L && !rc; ++l) {
    n->w[l] = widths[l];
    n->wp[l] = (int)align_up(widths[l], 16);
  }
  for (int l = 0; l < L && !rc; ++l) {
    n->woff[l] = np;
    np += (long)n->wp[l + 1] * n->wp[l];
    n->boff[l] = np;
    np += n->wp[l + 1];
    n->wbo[2 * l] = nw;
    nw += align_up(n->wp[l + 1], BN) * n->wp[l];
    n->wbo[2 * l + 1] = nw;
    nw += align_up(n->wp[l], BN) * n->wp[l + 1];
  }
  n->np = np;
  n->nw = nw;
  if (!rc && cudaStreamCreateWithFlags(&n->own_stream, cudaStreamNonBlocking) != cudaSuccess) rc = -2;
  n->stream = n->own_stream;
  /* every device buffer in one allocation (256-byte aligned parts), zeroed */
  const size_t fp = sizeof(float) * np;
  const long out_tiles = (n->rows / BM) * ((widths[L] + BN - 1) / BN + 1);
  for (int pass = 0; pass < 2 && !rc; ++pass) {
    size_t at = 0;
    auto part = [&](auto& ptr, size_t bytes) {
      if (pass) ptr = reinterpret_cast<std::decay_t<decltype(ptr)>>(n->mem + at);
      at += (bytes + 255) / 256 * 256;
    };
    part(n->p, fp); part(n->g, fp); part(n->m, fp); part(n->v, fp);
    part(n->wmap, sizeof(int2) * np);
    part(n->wbf, sizeof(__nv_bfloat16) * nw);
    long dzw[2] = {0, 0};
    for (int l = 0; l < L; ++l) {
      part(n->act[l], sizeof(__nv_bfloat16) * n->rows * n->wp[l]);
      if (l + 1 < L) part(n->z[l], sizeof(float) * n->rows * n->wp[l + 1]);
      if (n->wp[l + 1] > dzw[l & 1]) dzw[l & 1] = n->wp[l + 1];
    }
    for (int k = 0; k < 2; ++k) part(n->dz[k], sizeof(__nv_bfloat16) * n->rows * dzw[k]);
    part(n->part, sizeof(float) * out_tiles);
    part(n->d_loss, sizeof(float));
    part(n->d_err, sizeof(int));
    if (pass) break;
    if (cudaMalloc(&n->mem, at) != cudaSuccess) rc = -5;
    else if (cudaMemset(n->mem, 0, at) != cudaSuccess) rc = -2;
  }
  if (!rc) rc = set_smem_limits();
  if (!rc) {
    /* He-uniform weights for the GELU layers (bound sqrt(6 / fan_in)),
       zero biases, zero padding */
    float* hp = (float*)calloc(np, sizeof(float));
    int2* map = (int2*)malloc(sizeof(int2) * np);
    uint64_t s = seed;
    if (!hp || !map) rc = -5;
    for (long i = 0; i < np && !rc; ++i) map[i] = make_int2(-1, -1);
    for (int l = 0; l < L && !rc; ++l) {
      const double bound = sqrt(6.0 / n->w[l]);
      for (int r = 0; r < n->wp[l + 1]; ++r)
        for (int c = 0; c < n->wp[l]; ++c) {
          const long i = n->woff[l] + (long)r * n->wp[l] + c;
          auto at = [](int row, int col, int cols) { return ((long)(row / BN * (cols / 8) + col / 8) * BN + row % BN) * 8 + col % 8; };
          map[i] = make_int2((int)(n->wbo[2 * l] + at(r, c, n->wp[l])), (int)(n->wbo[2 * l + 1] + at(c, r, n->wp[l + 1])));
          if (r < n->w[l + 1] && c < n->w[l]) hp[i] = (float)((2.0 * uniform01(&s) - 1.0) * bound);
        }
    }
    if (!rc && cudaMemcpy(n->p, hp, fp, cudaMemcpyHostToDevice) != cudaSuccess) rc = -2;
    if (!rc && cudaMemcpy(n->wmap, map, sizeof(int2) * np, cudaMemcpyHostToDevice) != cudaSuccess) rc = -2;
    free(hp);
    free(map);
  }
  if (!rc) rc = refresh_bf16(n);
  if (rc) {
    lbib_mlp_free(n);
    return NULL;
  }
  return n;
}

void lbib_mlp_free(lbib_mlp* n) {
  if (!n) return;
  if (n->stream) cudaStreamSynchronize(n->stream);
  cudaFree(n->mem);
  if (n->own_stream) cudaStreamDestroy(n->own_stream);
  free(n->w); free(n->wp); free(n->woff); free(n->boff); free(n->wbo); free(n->act); free(n->z);
  free(n);
}

long lbib_mlp_param_count(lbib_mlp* n) { return n ? abi_count(n) : 0; }

void* lbib_mlp_stream(lbib_mlp* n) { return n ? (void*)n->stream : NULL; }

/* Run on the caller's stream (NULL is the CUDA default stream, as in every
 * CUDA call), so the caller's writes of X and T are ordered before the
 * kernels that read them and its allocator may recycle their memory as
 * soon as later work on that stream starts. */
int lbib_mlp_set_stream(lbib_mlp* n, void* stream) {
  if (!n) return LBIB_E_ARG;
  if (cudaStreamSynchronize(n->stream) != cudaSuccess) return LBIB_E_CUDA;
  n->stream = (cudaStream_t)stream;
  return LBIB_OK;
}

int lbib_mlp_get_params(lbib_mlp* n, float* out) {
  if (!n || !out) return LBIB_E_ARG;
  float* hp = (float*)malloc(sizeof(float) * n->np);
  if (!hp) return LBIB_E_NOMEM;
  int rc = cudaMemcpy(hp, n->p, sizeof(float) * n->np, cudaMemcpyDeviceToHost) == cudaSuccess ? 0 : LBIB_E_CUDA;
  if (!rc) for_each_param(n, [&](long a, long i) { out[a] = hp[i]; });
  free(hp);
  return rc;
}

int lbib_mlp_set_params(lbib_mlp* n, const float* in) {
  if (!n || !in) return LBIB_E_ARG;
  float* hp = (float*)calloc(n->np, sizeof(float));
  if (!hp) return LBIB_E_NOMEM;
  for_each_param(n, [&](long a, long i) { hp[i] = in[a]; });
  int rc = cudaMemcpy(n->p, hp, sizeof(float) * n->np, cudaMemcpyHostToDevice) == cudaSuccess ? 0 : LBIB_E_CUDA;
  free(hp);
  if (!rc && refresh_bf16(n)) rc = LBIB_E_CUDA;
  return rc;
}

/* X [batch][w_0] fp32 and Y [batch][w_L] fp32, device pointers. */
int lbib_mlp_forward(lbib_mlp* n, const float* X, int batch, float* Y) {
  if (!n || !X || !Y || batch < 1 || batch > n->max_batch) return LBIB_E_ARG;
  if (forward(n, X, batch, Y)) return LBIB_E_CUDA;
  return lbib_mlp_synchronize(n);
}

/* Loss and gradient (ABI order, host array of lbib_mlp_param_count floats)
 * of the mean-squared error on one batch, without updating anything. */
int lbib_mlp_gradient(lbib_mlp* n, const float* X, const float* T, int batch, float* grad, float* loss) {
  if (!n || !X || !T || batch < 1 || batch > n->max_batch) return LBIB_E_ARG;
  if (gradients(n, X, T, batch, loss != NULL)) return LBIB_E_CUDA;
  float* hg = (float*)malloc(sizeof(float) * n->np);
  if (!hg) return LBIB_E_NOMEM;
  int rc = 0;
  if (cudaMemcpyAsync(hg, n->g, sizeof(float) * n->np, cudaMemcpyDeviceToHost, n->stream) != cudaSuccess ||
      (loss && cudaMemcpyAsync(loss, n->d_loss, sizeof(float), cudaMemcpyDeviceToHost, n->stream) != cudaSuccess) ||
      cudaStreamSynchronize(n->stream) != cudaSuccess)
    rc = LBIB_E_CUDA;
  if (!rc) rc = lbib_mlp_synchronize(n);
  if (!rc && grad) for_each_param(n, [&](long a, long i) { grad[a] = hg[i]; });
  free(hg);
  return rc;
}

/* One Adam step (beta1 0.9, beta2 0.999, eps 1e-8) on one batch; X, T are
 * device pointers; loss (host, may be NULL) gets the batch's loss before
 * the step.  Asynchronous unless loss is asked for. */
int lbib_mlp_train_step(lbib_mlp* n, const float* X, const float* T, int batch, float lr, float* loss) {
  if (!n || !X || !T || batch < 1 || batch > n->max_batch || !(lr > 0)) return LBIB_E_ARG;
  if (gradients(n, X, T, batch, loss != NULL)) return LBIB_E_CUDA;
  n->steps++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = (float)(1.0 - pow(b1, (double)n->steps)), c2 = (float)(1.0 - pow(b2, (double)n->steps));
  if (launch(mlp_adam, (unsigned)((n->np + 255) / 256), 256, 0, n->stream, 1, n->p, (const float*)n->g, n->m, n->v, n->np,
             lr, b1, b2, 1e-8f, c1, c2, n->wbf, (const int2*)n->wmap))
    return LBIB_E_CUDA;
  if (loss) {
    if (cudaMemcpyAsync(loss, n->d_loss, sizeof(float), cudaMemcpyDeviceToHost, n->stream) != cudaSuccess ||
        cudaStreamSynchronize(n->stream) != cudaSuccess)
      return LBIB_E_CUDA;
  }
  return LBIB_OK;
}

/* Waits for the MLP's work; LBIB_E_CUDA also when a tensor-core GEMM
 * gave up waiting on its mbarrier (its output tile was not written). */
int lbib_mlp_synchronize(lbib_mlp* n) {
  if (!n) return LBIB_E_ARG;
  int e = 0;
  if (cudaMemcpyAsync(&e, n->d_err, sizeof(int), cudaMemcpyDeviceToHost, n->stream) != cudaSuccess ||
      cudaStreamSynchronize(n->stream) != cudaSuccess)
    return LBIB_E_CUDA;
  return e ? LBIB_E_CUDA : LBIB_OK;
}

}  /* extern "C" */
