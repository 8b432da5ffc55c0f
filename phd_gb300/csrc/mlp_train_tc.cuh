// Training GEMMs of the surrogate network on the 5th-generation tensor
// cores (sm_103a).
//
// Every GEMM of one training step -- the forward layers, the input
// gradients and the weight gradients -- is D (128 x NT) = A (128 x K) B^T
// with both operands K-major, issued as tcgen05.mma kind::f16 (BF16 x BF16
// -> FP32, M = 128, K = 16 per instruction) by one thread, with the
// accumulator in tensor memory.  The operands are kept in global memory in
// the "K-slab" layout below, so the block of 128 (or NT) rows by one K chunk
// that a pipeline stage needs is one contiguous run of bytes: it arrives in
// shared memory by one cp.async.bulk, counted on that stage's mbarrier.
// Four stages overlap the copies with the MMAs.  The epilogue (4 warps, one
// TMEM lane = one output row per thread) fuses bias and GELU (forward),
// GELU' (backward), the loss and its gradient (last layer) and writes each result in the layouts the next GEMMs read:
//   * activations and output gradients as A operands (rows = batch rows,
//     K = features) and, transposed, as operands of the weight gradient
//     (rows = features, K = batch rows);
//   * weight gradients as FP32 partial sums of a K split (the batch is split
//     over CTAs), added in a fixed order afterwards.
// Every mbarrier wait is bounded; on a timeout the kernel records it in
// *err, waits (bounded) once more, frees its TMEM and returns.
#pragma once
#include <cstdint>
#include <cuda_bf16.h>

namespace mlptt {

using mlptc::core_off;

constexpr int GT_THREADS = 128;   // 4 warps: warp w owns TMEM lanes (tile rows) 32 w .. 32 w + 31
constexpr int STAGES = 4;
constexpr int KCMAX = 64;          // K columns per pipeline stage

// K-slab layout of a BF16 matrix X with R rows and K columns (R a multiple
// of 8, K a multiple of 8, K <= 64 or a multiple of 64): K is cut into
// chunks of kc = min(K, 64) columns; chunk c holds all R rows in the
// core-matrix K-major layout of an R x kc block (core_off), chunks one after
// the other.  Rows r0 .. r0 + n - 1 of one chunk are n * kc * 2 contiguous
// bytes starting at byte kslab_off(r0, c * kc, R, K).
__host__ __device__ constexpr int kslab_kc(int K) { return K < KCMAX ? K : KCMAX; }
__host__ __device__ constexpr size_t kslab_off(int r, int k, int R, int K) {
  return (size_t)(k / kslab_kc(K)) * (size_t)R * kslab_kc(K) * 2 + core_off(r, k % kslab_kc(K), kslab_kc(K));
}

enum TgMode { TG_FWD_GELU = 0, TG_FWD_LOSS = 1, TG_BWD_GELU = 2, TG_WGRAD = 3 };

// Every launch of a training step is a programmatic dependent of the one
// before it: its CTAs take their places, set up barriers and tensor memory
// and then wait here for that launch's end, of which the next launch's CTAs
// are let in at once.  The wait comes before any access to global memory.
__device__ __forceinline__ void after_previous_launch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

struct TgArgs {
  const uint8_t* A;     // K-slab, RA rows x K
  const uint8_t* B;     // K-slab, RB rows x K
  int RA, RB, K;
  int chunks;           // K chunks per CTA (the grid's z dimension splits K)
  int N;                // columns of the FP32 outputs (their row stride)
  const float* bias;    // TG_FWD_*: per column
  float* outf;          // TG_FWD_GELU: pre-activation; TG_FWD_LOSS, TG_BWD_GELU: gradient;
                        // TG_WGRAD: partial sums [z][RA][N]
  const float* zin;     // TG_BWD_GELU: pre-activation of the layer below (stride N)
  const float* target;  // TG_FWD_LOSS: targets of the M_valid real rows (10 columns)
  int M_valid;
  double* loss;         // TG_FWD_LOSS: the loss sum is added here
  uint8_t* oa;          // all but TG_WGRAD: BF16 result as an A operand (K-slab, oaR rows x N)
  uint8_t* ot;          // ... and transposed (K-slab, N rows x otK)
  int oaR, otK;
  int* err;
};

__host__ __device__ constexpr uint32_t tg_stage_bytes(int NT) { return (uint32_t)(128 + NT) * KCMAX * 2; }
__host__ __device__ constexpr uint32_t tg_smem_bytes(int NT) { return STAGES * tg_stage_bytes(NT) + 128; }

// One output tile: rows m0 .. m0 + 127, columns n0 .. n0 + nt - 1 (nt <= NT),
// K chunks z * a.chunks onwards.
template <int NT, int MODE>
__device__ __forceinline__ void tg_tile(const TgArgs& a, int m0, int n0, int nt, int z) {
  using namespace mlptc;
  constexpr uint32_t TCOLS = NT < 32 ? 32 : NT;
  extern __shared__ __align__(1024) uint8_t sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = saddr(sm);
  const uint32_t bars = base + STAGES * tg_stage_bytes(NT);   // full[s], empty[s], done, TMEM address
  auto full = [&](int s) { return bars + 8 * s; };
  auto empty = [&](int s) { return bars + 8 * (STAGES + s); };
  const uint32_t done = bars + 16 * STAGES;
  const uint32_t tslot = done + 8;
  const int kc = kslab_kc(a.K);
  const uint32_t abytes = 128u * kc * 2, bbytes = (uint32_t)nt * kc * 2;
  const int nkc = a.K / kc;
  const int c0 = z * a.chunks;
  const int nk = min(a.chunks, nkc - c0);
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    mbar_init(done, 1);
    fence_async_smem();
  }
  if (warp == 0) tmem_alloc(tslot, TCOLS);
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  after_previous_launch();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sm + (tslot - base));
  int failed = 0;
  if (tid == 0 && nk > 0) {
    auto load = [&](int i) {
      const int s = i % STAGES, c = c0 + i;
      const uint32_t sa = base + s * tg_stage_bytes(NT), sb = sa + 128u * KCMAX * 2;
      mbar_expect_tx(full(s), abytes + bbytes);
      bulk_g2s(sa, a.A + kslab_off(m0, c * kc, a.RA, a.K), abytes, full(s));
      bulk_g2s(sb, a.B + kslab_off(n0, c * kc, a.RB, a.K), bbytes, full(s));
    };
    for (int i = 0; i < STAGES && i < nk; ++i) load(i);
    const uint32_t idesc = idesc_bf16(128, nt);
    for (int i = 0; i < nk && !failed; ++i) {
      const int s = i % STAGES;
      const uint32_t par = (uint32_t)(i / STAGES) & 1u;
      if (!mbar_wait(full(s), par)) { failed = 2; break; }
      tc_after_sync();
      const uint32_t sa = base + s * tg_stage_bytes(NT), sb = sa + 128u * KCMAX * 2;
      for (int k = 0; k < kc / 16; ++k)
        mma_bf16(tmem, sdesc(sa + k * 256, 128, kc * 16), sdesc(sb + k * 256, 128, kc * 16), idesc, (i > 0 || k > 0));
      mma_commit(empty(s));
      if (i + STAGES < nk) {   // this stage is refilled once its MMAs have read it
        if (!mbar_wait(empty(s), par)) { failed = 1; break; }
        load(i + STAGES);
      }
    }
    if (!failed) mma_commit(done);
  }
  // everyone waits for the accumulator
  bool ok = true;
  if (nk > 0) {
    const int f = __syncthreads_or(failed);
    ok = f == 0 && __syncthreads_and(mbar_wait(done, 0));
  }
  tc_after_sync();
  if (ok && nk > 0) {
    const int r = warp * 32 + lane;   // tile row = TMEM lane
    const int gr = m0 + r;
    const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
    constexpr int CW = NT < 32 || MODE == TG_WGRAD ? 16 : 32;
#pragma unroll 1
    for (int cb = 0; cb < nt; cb += CW) {
      uint32_t v[32];
      if constexpr (CW == 32) tmem_ld32(lane_addr + (uint32_t)cb, v);
      else tmem_ld16(lane_addr + (uint32_t)cb, v);
      tmem_wait_ld();
      const int gc0 = n0 + cb;
      if constexpr (MODE == TG_WGRAD) {
        float4* dst = reinterpret_cast<float4*>(a.outf + ((size_t)z * a.RA + gr) * a.N + gc0);
#pragma unroll
        for (int q = 0; q < CW / 4; ++q)
          dst[q] = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]), __uint_as_float(v[4 * q + 2]),
                               __uint_as_float(v[4 * q + 3]));
      } else {
        float f[CW];
        if constexpr (MODE == TG_FWD_GELU) {
#pragma unroll
          for (int q = 0; q < CW; ++q) f[q] = __uint_as_float(v[q]) + a.bias[gc0 + q];
          float4* zd = reinterpret_cast<float4*>(a.outf + (size_t)gr * a.N + gc0);
#pragma unroll
          for (int q = 0; q < CW / 4; ++q) zd[q] = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
#pragma unroll
          for (int q = 0; q < CW; ++q) f[q] = gelu(f[q]);
        } else if constexpr (MODE == TG_FWD_LOSS) {
          // MSE loss on the 10 real outputs of the real rows and its gradient
          // 2 (out - t) / (M_valid * 10); padded columns and rows get zero
          static_assert(NT == 16, "all outputs of a row in one thread");
          double l2 = 0.0;
#pragma unroll
          for (int q = 0; q < CW; ++q) f[q] = 0.0f;
          if (gr < a.M_valid) {
#pragma unroll
            for (int q = 0; q < 10; ++q) {
              const float out = __uint_as_float(v[q]) + a.bias[q];
              const float d = out - a.target[(size_t)gr * 10 + q];
              l2 += (double)d * (double)d;
              f[q] = 2.0f * d / (float)(a.M_valid * 10);
            }
          }
          for (int o = 16; o > 0; o >>= 1) l2 += __shfl_xor_sync(0xffffffffu, l2, o);
          if (lane == 0) atomicAdd(a.loss, l2);
          float4* gd = reinterpret_cast<float4*>(a.outf + (size_t)gr * a.N);
#pragma unroll
          for (int q = 0; q < CW / 4; ++q) gd[q] = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
        } else {   // TG_BWD_GELU
          const float4* zs = reinterpret_cast<const float4*>(a.zin + (size_t)gr * a.N + gc0);
#pragma unroll
          for (int q = 0; q < CW / 4; ++q) {
            const float4 z = zs[q];
            f[4 * q] = __uint_as_float(v[4 * q]) * gelu_grad(z.x);
            f[4 * q + 1] = __uint_as_float(v[4 * q + 1]) * gelu_grad(z.y);
            f[4 * q + 2] = __uint_as_float(v[4 * q + 2]) * gelu_grad(z.z);
            f[4 * q + 3] = __uint_as_float(v[4 * q + 3]) * gelu_grad(z.w);
          }
          float4* gd = reinterpret_cast<float4*>(a.outf + (size_t)gr * a.N + gc0);
#pragma unroll
          for (int q = 0; q < CW / 4; ++q) gd[q] = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
        }
        // BF16 copies: as an A operand (row gr, K = column), 16-byte stores
        // of 8 columns; transposed (row = column, K = gr), 2-byte stores
#pragma unroll
        for (int q = 0; q < CW / 8; ++q) {
          uint32_t pk[4];
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            __nv_bfloat162 b2 = __floats2bfloat162_rn(f[8 * q + 2 * h], f[8 * q + 2 * h + 1]);
            pk[h] = *reinterpret_cast<uint32_t*>(&b2);
          }
          *reinterpret_cast<uint4*>(a.oa + kslab_off(gr, gc0 + 8 * q, a.oaR, a.N)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
#pragma unroll
        for (int q = 0; q < CW; ++q)
          *reinterpret_cast<__nv_bfloat16*>(a.ot + kslab_off(gc0 + q, gr, a.N, a.otK)) = __float2bfloat16(f[q]);
      }
    }
  }
  if (!ok && nk > 0) {
    if (tid == 0) atomicExch(a.err, 1);
    mbar_wait(done, 0);   // a second bounded wait for the MMAs this CTA issued
  }
  tc_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_after_sync();
    tmem_dealloc(tmem, TCOLS);
  }
}

// The tile is a CTA's whole work, a few microseconds of which the epilogue is
// most (a row a thread, column after column), so narrow tiles pay: they spread
// the columns over more CTAs, and read A once more each, from L2.  A batch of
// 4096 rows and 256 columns: tiles of 128 columns, 64 CTAs, take 12.9 us
// forward and 14.9 backward; of 64, 10.6 and 11.8; of 32, half a microsecond
// a launch less again.
template <int NT, int MODE>
__global__ void __launch_bounds__(GT_THREADS) k_tgemm(TgArgs a) {
  tg_tile<NT, MODE>(a, blockIdx.x * 128, blockIdx.y * NT, NT, blockIdx.z);
}

// The weight gradients of all layers in one launch, up to 128 columns a tile:
// they depend on the activations and output gradients alone, and a layer by
// itself leaves most SMs idle (five launches of 64 CTAs took 44 us of a step
// of 4096 rows, this one takes 22).  first[l] is the first tile of layer l;
// blockIdx.y splits the batch.
constexpr int WG_NT = 128, WG_LAYERS = 5;
struct TgLayers {
  TgArgs l[WG_LAYERS];
  int first[WG_LAYERS + 1];
};
__global__ void __launch_bounds__(GT_THREADS) k_tg_wgrad(const __grid_constant__ TgLayers b) {
  int l = 0;
  while (l + 1 < WG_LAYERS && (int)blockIdx.x >= b.first[l + 1]) ++l;
  const TgArgs& a = b.l[l];
  const int q = blockIdx.x - b.first[l], nt = a.N < WG_NT ? a.N : WG_NT, mt = a.RA / 128;
  tg_tile<WG_NT, TG_WGRAD>(a, (q % mt) * 128, (q / mt) * nt, nt, blockIdx.y);
}

// Normalised inputs of one batch (rows r0 .. r0 + M - 1 of x, 12 FP32
// columns; the caller passes x + 12 r0) -> BF16 K-slab operands: xa
// (M x 16, columns 12..15 zero) for the first layer and xt (rows 0..15 of a
// 128 x M K-slab; rows 16..127 stay zero) for its weight gradient.  Rows at
// or beyond M_valid are zero.
struct PackArgs {
  const float* x;
  int M, M_valid;
  uint8_t *xa, *xt;
};
__global__ void k_tg_pack_input(PackArgs a) {
  after_previous_launch();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.M * 16) return;
  const int r = i >> 4, c = i & 15;
  const __nv_bfloat16 b = __float2bfloat16(c < 12 && r < a.M_valid ? a.x[(size_t)r * 12 + c] : 0.0f);
  *reinterpret_cast<__nv_bfloat16*>(a.xa + kslab_off(r, c, a.M, 16)) = b;
  *reinterpret_cast<__nv_bfloat16*>(a.xt + kslab_off(c, r, 128, a.M)) = b;
}

// The end of a training step, all layers in one launch: the weight gradients
// from their split-K partials (added in split order) and the bias gradients,
// the column sums of the FP32 output gradients (in a fixed order), and either
// one Adam update of every parameter with the BF16 copies that the GEMMs read
// (row-major, W^T and W K-slabs) or, with adam = 0, the gradients themselves.
// Bound by L2: 27 MB of partials and 17 MB of gradients at 4096 rows.  Column
// sums take eight columns a block, a whole 32-byte sector of each row; a
// block a column read eight times the bytes.  As twenty launches (a
// reduction, a column sum and two updates a layer) it took 136 us of a step
// of 4096 rows, as one 20.
struct UpdLayer {
  const float* part;    // [splits][rows][lout]
  const float* dz;      // M x lout
  float *w, *mw, *vw, *gw, *b, *mb, *vb, *gb;
  __nv_bfloat16* wb;
  uint8_t *wt, *wn;
  int rows, lin, lout;
  int first_b, first_w;   // first block of the biases and of the weights
};
struct UpdArgs {
  UpdLayer l[WG_LAYERS];
  int splits, M, nblk_b, adam;
  float lr, b1, b2, eps, c1, c2;
};
constexpr int UPD_THREADS = 256;

// The roundings of the two moments are spelled out, so that a training run
// gives the same weights wherever this is inlined.
__device__ __forceinline__ float adam_update(const UpdArgs& u, float gr, float* w, float* mw, float* vw) {
  const float m = __fmaf_rn(1.f - u.b1, gr, __fmul_rn(u.b1, *mw));
  const float v = __fmaf_rn(__fmul_rn(1.f - u.b2, gr), gr, __fmul_rn(u.b2, *vw));
  *mw = m;
  *vw = v;
  const float wv = *w - u.lr * (m / u.c1) / (sqrtf(v / u.c2) + u.eps);
  *w = wv;
  return wv;
}

__global__ void __launch_bounds__(UPD_THREADS) k_tg_update(const __grid_constant__ UpdArgs u) {
  after_previous_launch();
  int l = 0;
  if ((int)blockIdx.x < u.nblk_b) {   // biases: the longer blocks, first
    while (l + 1 < WG_LAYERS && (int)blockIdx.x >= u.l[l + 1].first_b) ++l;
    const UpdLayer& p = u.l[l];
    __shared__ float red[8][8];
    const int c0 = (blockIdx.x - p.first_b) * 8;
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int r = threadIdx.x; r < u.M; r += UPD_THREADS) {
      const float4* g = reinterpret_cast<const float4*>(p.dz + (size_t)r * p.lout + c0);
      const float4 x = g[0], y = g[1];
      s[0] += x.x; s[1] += x.y; s[2] += x.z; s[3] += x.w;
      s[4] += y.x; s[5] += y.y; s[6] += y.z; s[7] += y.w;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      for (int o = 16; o > 0; o >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
      if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = s[q];
    }
    __syncthreads();
    if (threadIdx.x < 8) {
      const int c = c0 + threadIdx.x;
      float t = 0.0f;
      for (int w = 0; w < UPD_THREADS / 32; ++w) t += red[threadIdx.x][w];
      if (u.adam) adam_update(u, t, p.b + c, p.mb + c, p.vb + c);
      else p.gb[c] = t;
    }
    return;
  }
  const int blk = blockIdx.x - u.nblk_b;
  while (l + 1 < WG_LAYERS && blk >= u.l[l + 1].first_w) ++l;
  const UpdLayer& p = u.l[l];
  const int i = (blk - p.first_w) * UPD_THREADS + threadIdx.x;
  if (i >= p.lin * p.lout) return;
  const size_t plane = (size_t)p.rows * p.lout;
  float s = 0.0f;
#pragma unroll 8
  for (int z = 0; z < u.splits; ++z) s += p.part[z * plane + i];
  if (!u.adam) {
    p.gw[i] = s;
    return;
  }
  const __nv_bfloat16 h = __float2bfloat16(adam_update(u, s, p.w + i, p.mw + i, p.vw + i));
  const int r = i / p.lout, c = i % p.lout;
  p.wb[i] = h;
  *reinterpret_cast<__nv_bfloat16*>(p.wt + kslab_off(c, r, p.lout, p.lin)) = h;
  *reinterpret_cast<__nv_bfloat16*>(p.wn + kslab_off(r, c, p.lin, p.lout)) = h;
}

// The BF16 operand copies of layer weights W (lin x lout, row-major FP32):
// wb (row-major), wt = W^T as a K-slab (lout rows, K = lin; forward) and
// wn = W as a K-slab (lin rows, K = lout; input gradient).
__global__ void k_tg_weights(const float* __restrict__ w, int lin, int lout, __nv_bfloat16* __restrict__ wb,
                             uint8_t* __restrict__ wt, uint8_t* __restrict__ wn) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= lin * lout) return;
  const int r = i / lout, c = i % lout;
  const __nv_bfloat16 b = __float2bfloat16(w[i]);
  wb[i] = b;
  *reinterpret_cast<__nv_bfloat16*>(wt + kslab_off(c, r, lout, lin)) = b;
  *reinterpret_cast<__nv_bfloat16*>(wn + kslab_off(r, c, lin, lout)) = b;
}

}  // namespace mlptt
