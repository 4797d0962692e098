// Tensor-core (tcgen05) kernels of the learned preconditioner.
//
// xf_tc_gemm_bf16: one 128 x N x K tile, D = A B^T with BF16 A (128 x K) and
// B (N x K), K contiguous, FP32 accumulation in tensor memory.  It is the
// building block the implicit-GEMM convolutions below use, exposed so that
// its operand layout and descriptors are checked on their own.
#include <cuda_bf16.h>

#include <stdlib.h>

#include <algorithm>

#include "xf_common.cuh"
#include "xf_tc.cuh"

constexpr int TC_M = 128;

// Copies a rows x K BF16 matrix (K contiguous, `ld` elements per row) into
// the canonical no-swizzle K-major layout: core matrix (row group g, K group
// q) at g * (K / 8) * 128 + q * 128 bytes.
__device__ __forceinline__ void stage_kmajor(uint8_t* dst, const uint16_t* src, int rows, int K, int ld) {
  const int kg = K / 8;
  for (int u = threadIdx.x; u < rows * kg; u += blockDim.x) {
    const int r = u / kg, q = u - r * kg;
    const uint4 v = *reinterpret_cast<const uint4*>(src + (int64_t)r * ld + q * 8);
    *reinterpret_cast<uint4*>(dst + (r >> 3) * kg * 128 + q * 128 + (r & 7) * 16) = v;
  }
}

__host__ __device__ inline uint32_t tmem_cols(int n) {
  uint32_t c = 32;
  while ((int)c < n) c <<= 1;
  return c;
}

// variant 0: LBO = distance between K-adjacent core matrices, SBO = between
// row-adjacent ones; variant 1: the two swapped (both stay inside the tiles).
__global__ void __launch_bounds__(128) k_tc_gemm(const uint16_t* __restrict__ A, const uint16_t* __restrict__ B,
                                                 float* __restrict__ D, int N, int K, int variant,
                                                 int* __restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t mbar;
  __shared__ uint32_t tmem_base;
  uint8_t* sA = smem;
  uint8_t* sB = smem + TC_M * K * 2;
  stage_kmajor(sA, A, TC_M, K, K);
  stage_kmajor(sB, B, N, K, K);
  tc::fence_async_smem();
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t ncols = tmem_cols(N);
  if (warp == 0) tc::tmem_alloc(&tmem_base, ncols);
  if (threadIdx.x == 0) tc::mbar_init(&mbar, 1);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = tmem_base;
  const uint32_t kstride = 128, rstride = (uint32_t)(K / 8) * 128;
  const uint32_t lbo = variant ? rstride : kstride, sbo = variant ? kstride : rstride;
  if (threadIdx.x == 0) {
    const uint32_t idesc = tc::idesc_bf16_f32(TC_M, N);
    for (int s = 0; s < K / 16; s++) {
      const uint64_t ad = tc::smem_desc(tc::smem_addr(sA + s * 256), lbo, sbo);
      const uint64_t bd = tc::smem_desc(tc::smem_addr(sB + s * 256), lbo, sbo);
      tc::mma_bf16(tbase, ad, bd, idesc, s > 0);
    }
    tc::mma_commit(&mbar);
  }
  bool ok = __syncthreads_and(tc::mbar_wait(&mbar, 0));
  if (!ok) {
    if (threadIdx.x == 0) atomicExch(err, 1);
    ok = __syncthreads_and(tc::mbar_wait(&mbar, 0));   // let the MMAs drain before the columns are freed
  }
  tc::fence_after_sync();
  if (ok) {
    const int row = warp * 32 + lane;
    for (int c = 0; c < N; c += 8) {
      float v[8];
      tc::tmem_ld8(tbase + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
#pragma unroll
      for (int q = 0; q < 8; q++) D[(int64_t)row * N + c + q] = v[q];
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tbase, ncols);
}

extern "C" int xf_tc_gemm_bf16(xf_ctx* ctx, int N, int K, const uint16_t* host_a, const uint16_t* host_b,
                               float* host_d, int variant) {
  if (!ctx || !host_a || !host_b || !host_d) return XF_ERR_ARG;
  if (N < 16 || N > 256 || N % 16 || K < 16 || K > 256 || K % 16 || (variant != 0 && variant != 1))
    return xf_fail(ctx, XF_ERR_ARG, "xf_tc_gemm_bf16: N in 16..256 and K in 16..256, multiples of 16");
  XF_CUDA(ctx, cudaSetDevice(ctx->device));
  uint16_t *a = nullptr, *b = nullptr;
  float* d = nullptr;
  int* err = nullptr;
  auto cleanup = [&]() {
    cudaFree(a); cudaFree(b); cudaFree(d); cudaFree(err);
  };
  if (cudaMalloc(&a, TC_M * K * 2) || cudaMalloc(&b, N * K * 2) || cudaMalloc(&d, TC_M * N * 4) ||
      cudaMalloc(&err, 4)) {
    cleanup();
    cudaGetLastError();
    return xf_fail(ctx, XF_ERR_NOMEM, "xf_tc_gemm_bf16: allocation");
  }
  cudaStream_t s = ctx->stream;
  cudaMemcpyAsync(a, host_a, TC_M * K * 2, cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(b, host_b, N * K * 2, cudaMemcpyHostToDevice, s);
  cudaMemsetAsync(d, 0, TC_M * N * 4, s);
  cudaMemsetAsync(err, 0, 4, s);
  const size_t smem = (size_t)(TC_M + N) * K * 2;
  if (cudaFuncSetAttribute(k_tc_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    cleanup();
    return xf_fail(ctx, XF_ERR_CUDA, "xf_tc_gemm_bf16: shared memory attribute");
  }
  k_tc_gemm<<<1, 128, smem, s>>>(a, b, d, N, K, variant, err);
  int herr = 0;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(host_d, d, TC_M * N * 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cleanup();
  if (e != cudaSuccess) return xf_fail(ctx, XF_ERR_CUDA, "xf_tc_gemm_bf16: %s", cudaGetErrorString(e));
  if (herr) return xf_fail(ctx, XF_ERR_CUDA, "xf_tc_gemm_bf16: the MMA completion wait ran out");
  return XF_OK;
}

// ---------------------------------------------------------------------------
// 3x3x3 convolution as an implicit GEMM on the tensor cores.
//
// Activations are BF16 boxes of the level's grid (the box with its ghost
// layer, cell c = (i n2 + j) n3 + k) in channel planes of 8 (xf_common.cuh),
// every plane allocated with a zero margin of XF_CONV_MARGIN(n2, n3) rows
// before cell 0 and after the last cell, so every tap of every tile reads
// inside the allocation.  Ghost and inactive cells hold 0 in every activation
// (the epilogue multiplies by the level's mask), which makes the ghost layer
// the zero padding of the convolution, also across the flattened row ends.
// Epilogue: + bias, ReLU (optional), x mask, then the first `out_ch`
// channels stored as BF16 planes or as FP32 cell rows (pitch out_ld).
struct ConvArgs {
  const uint16_t* in;   // plane 0, cell 0 of the input slice
  int64_t in_ps;        // plane stride (elements)
  int Ci;
  const uint16_t* Wt;   // weights tiled (conv_tiled_index)
  const float* bias;    // [Co] or null
  int Co;
  const uint8_t* mask;  // [ncell]
  int n2, n3;
  int64_t ncell;
  uint16_t* out16;      // plane 0, cell 0 of the output slice (BF16 planes), or null
  int64_t out_ps;
  float* out32;         // or FP32 rows of pitch out_ld
  int out_ld, out_ch, relu;
  const uint16_t* gate;   // optional BF16 planes: zero the outputs where the gate value <= 0 (ReLU backward)
  int64_t gate_ps;
  int* err;
};

// Epilogue of one cell and 8 output channels (co .. co+7).
__device__ __forceinline__ void conv_store8(const ConvArgs& a, int64_t c, int co, float m, float (&v)[8]) {
  uint16_t gt[8];
  if (a.gate) *reinterpret_cast<uint4*>(gt) = *reinterpret_cast<const uint4*>(a.gate + (co >> 3) * a.gate_ps + c * 8);
#pragma unroll
  for (int q = 0; q < 8; q++) {
    float x = v[q] + (a.bias ? a.bias[co + q] : 0.f);
    if (a.relu) x = fmaxf(x, 0.f);
    if (a.gate && ((gt[q] & 0x8000u) || !(gt[q] & 0x7FFFu))) x = 0.f;   // gate value <= 0
    v[q] = x * m;
  }
  if (a.out16) {
    uint32_t pk[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
      pk[q] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(a.out16 + (co >> 3) * a.out_ps + c * 8) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
  } else {
    const int nq = min(8, a.out_ch - co);
    float* dst = a.out32 + c * a.out_ld + co;
    if (nq == 8 && ((uintptr_t)dst & 15) == 0) {   // a cell's 32 bytes by two stores (scalar ones: 8 sectors a lane)
      reinterpret_cast<float4*>(dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
      reinterpret_cast<float4*>(dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else {
      for (int q = 0; q < nq; q++) dst[q] = v[q];
    }
  }
}

// ---------------------------------------------------------------------------
// The convolution with the three k-taps of each (di, dj) stacked along N, fed
// by bulk copies.
//
// A tcgen05.mma of M = 128, K = 16 costs about the same time for any N up to
// 32 (about 39 cycles on GB300; 44 at N = 64, 60 at 128), so one MMA of
// N = 3 Co replaces three of N = Co.  For slab (di, dj) the A operand is the
// 128 rows X[c0 - 1 + di P + dj n3 + r], the B operand the taps (di, dj, -1),
// (di, dj, 0), (di, dj, +1) stacked, 3 Co x 16 per input chunk; TMEM
// accumulates D_dk over the nine slabs and the input chunks, and the epilogue
// applies the k shift on the output side:
//     y[c0 + r - 1] = D_-1[r - 1] + D_0[r] + D_+1[r + 1],   r = 1 .. 126,
// neighbouring TMEM rows coming from the neighbouring lanes (warp shuffles;
// across warps, the edge rows through shared memory as 16-byte stores by
// lanes 31 and 0 and 16-byte loads by every lane: scalar single-lane
// exchanges cost about three times as long).  A tile therefore yields 126 cells;
// the last tile starts at ncell - 126 (its overlap rewrites identical values).
//
// A pipeline stage is one (tile, 16-channel input chunk): for each di and
// 8-channel plane the rows of its three slabs, which is already the canonical
// K-major operand layout; nine MMAs read it.  Where a row of the box is
// shorter than a tile, the slabs of dj = -1, 0, 1 overlap and come as one copy of
// 128 + 2 n3 rows (cp.async.bulk), the MMAs starting n3 rows apart: 25 KB a
// stage at n3 = 66 instead of 37, so that three CTAs fit an SM (64^3, 16 -> 16:
// 14.5 -> 13.1 us; 48 -> 16 27.3 -> 19.6; 96 -> 32 at 34^3 20.3 -> 14.1);
// otherwise nine copies of 128 rows a plane.  The tiled weights stay resident in shared
// memory when they fit beside two stages, else each stage also carries its
// chunk's nine B blocks.  Each control step therefore covers nine MMAs.
// The CTA is persistent and warp-specialised:
//   warp 4: issues each stage's copies into a ring, one copy per lane (one
//       thread issuing all of them was the pipeline's bottleneck), lane 0
//       keeping the barriers (full: the copies' transaction bytes; empty: the MMAs that
//       read the stage have completed);
//   warp 5: the MMAs into one of two TMEM accumulators (the epilogue of a
//       tile overlaps the next tile's MMAs), a commit per stage and one per
//       finished tile.  The whole warp walks the loop and one elected lane
//       issues, so that the descriptors are uniform;
//   warps 0-3: the epilogue, TMEM lanes 32 w .. 32 w + 31.
// Every wait is bounded by the SM clock; a wait that runs out sets the
// kernel's error flag and an abort flag in shared memory that ends every
// role's loop, after which the copies and MMAs in flight are waited for
// (bounded) before TMEM is freed.  Requires 3 Co <= 256 (Co <= 80), Ci and Co
// multiples of 16.
constexpr int BK_THREADS = 192;
constexpr int BK_MAX_STAGES = 6;
constexpr long long BK_WAIT_CYCLES = 1ll << 31;   // about a second at the SM clock

__device__ __forceinline__ void mbar_expect_tx(uint64_t* mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_addr(mbar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_addr(mbar)) : "memory");
}
// Bulk copy global -> shared (16-byte aligned, size a multiple of 16),
// completing on `mbar` (transaction bytes).
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   tc::smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(tc::smem_addr(mbar))
               : "memory");
}
// Waits for phase `parity` of `mbar`; false when the abort flag is raised or
// the wait runs past BK_WAIT_CYCLES (which raises it).
__device__ __forceinline__ bool bk_wait(uint64_t* mbar, uint32_t parity, volatile int* abort_flag,
                                        bool honour_abort = true) {
  const uint32_t a = tc::smem_addr(mbar);
  const long long t0 = clock64();
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if (honour_abort && *abort_flag) return false;
    if (clock64() - t0 > BK_WAIT_CYCLES) {
      *abort_flag = 1;
      return false;
    }
  }
}
// The same by a whole warp, with one answer.
__device__ __forceinline__ bool bk_wait_warp(uint64_t* mbar, uint32_t parity, volatile int* abort_flag,
                                             bool honour_abort = true) {
  return __all_sync(0xffffffffu, bk_wait(mbar, parity, abort_flag, honour_abort));
}
// Barrier 1 over the four epilogue warps with an AND of `pred`.
__device__ __forceinline__ bool epi_sync_and(bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, 1, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)pred)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void epi_sync() { asm volatile("barrier.cta.sync 1, 128;" ::: "memory"); }

// Shared-memory plan of one CTA.
struct BkPlan {
  int stages, per_sm, resident, acc_off, tmem_cols, smem_bytes;
  uint32_t w_bytes, b_bytes, stage_bytes, w_region;
  uint32_t a_bytes, plane_bytes;   // A of a stage; one plane's rows of one di
  int step, merged;                // rows between the slabs of dj = -1, 0, 1; they overlap and come as one copy
};
static BkPlan bk_plan(int ci, int co, int rows, int static_smem) {
  BkPlan p = {};
  p.merged = rows < 128;
  p.step = std::min(rows, 128);
  p.plane_bytes = (uint32_t)(128 + 2 * p.step) * 16;
  p.a_bytes = (6 * p.plane_bytes + 127) / 128 * 128;   // B behind it keeps its 128-byte rows
  const int n3 = 3 * co;
  p.acc_off = (n3 + 31) / 32 * 32;
  p.tmem_cols = (int)tmem_cols(p.acc_off + n3);
  const int per_sm_t = std::min(3, 512 / p.tmem_cols);
  p.w_bytes = (uint32_t)(27 * co * ci * 2);
  p.b_bytes = (uint32_t)(9 * n3 * 32);
  const uint32_t w_region = (p.w_bytes + 1023) / 1024 * 1024;
  const uint32_t st_res = (p.a_bytes + 1023) / 1024 * 1024, st_str = (p.a_bytes + p.b_bytes + 1023) / 1024 * 1024;
  // (CTAs per SM, weights resident): three CTAs with resident weights, then two, resident weights first, then one
  const int order[5][2] = {{3, 1}, {2, 1}, {2, 0}, {1, 1}, {1, 0}};
  for (const auto& way : order) {
    const int per_sm = way[0];
    const bool res = way[1];
    if (per_sm > per_sm_t) continue;
    // dynamic shared memory of one CTA: 228 KB per SM less 1 KB reserved per
    // CTA, at most 227 KB per CTA, less the static part and the alignment slack
    const int dyn = std::min(227 * 1024, (228 * 1024) / per_sm - 1024) - static_smem - 1024;
    const int avail = dyn - (res ? (int)w_region : 0);
    const int st = avail > 0 ? avail / (int)(res ? st_res : st_str) : 0;
    if (st >= 2) {
      p.per_sm = per_sm;
      p.resident = res;
      p.stages = std::min(st, BK_MAX_STAGES);
      p.stage_bytes = res ? st_res : st_str;
      p.w_region = res ? w_region : 0;
      p.smem_bytes = (int)(p.w_region + p.stages * p.stage_bytes + 1024);
      return p;
    }
  }
  return p;   // stages = 0: no plan (never for Co <= 80)
}

__global__ void __launch_bounds__(BK_THREADS) k_conv3_bulk(ConvArgs a, BkPlan plan) {
  extern __shared__ uint8_t dsm[];
  __shared__ uint64_t full[BK_MAX_STAGES], empty[BK_MAX_STAGES], tfull[2], tempty[2], wfull, mdone;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  __shared__ __align__(16) float xch[2][4][2][80];   // per tile parity and warp: lane 31's D_-1 row, lane 0's D_+1 row
  const int Ci = a.Ci, Co = a.Co, N3 = 3 * Co, nk = Ci / 16;
  const int S = plan.stages;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t raw = tc::smem_addr(dsm);
  uint8_t* smem = dsm + ((1024u - (raw & 1023u)) & 1023u);
  uint8_t* wsm = smem;                    // resident tiled weights
  uint8_t* stg = smem + plan.w_region;    // the stages
  if (warp == 0) tc::tmem_alloc(&tmem_base, (uint32_t)plan.tmem_cols);
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int q = 0; q < 2; q++) {
      tc::mbar_init(&tfull[q], 1);
      tc::mbar_init(&tempty[q], 4);
    }
    tc::mbar_init(&wfull, 1);
    tc::mbar_init(&mdone, 1);
    abort_flag = 0;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = tmem_base;
  volatile int* abort_p = &abort_flag;
  const int64_t P = (int64_t)a.n2 * a.n3;
  const int64_t ntiles = (a.ncell + 125) / 126;
  const int my_tiles = ntiles > blockIdx.x ? (int)((ntiles - 1 - blockIdx.x) / gridDim.x + 1) : 0;
  auto tile_start = [&](int k) {   // first output cell of this CTA's k-th tile
    const int64_t st = ((int64_t)blockIdx.x + (int64_t)k * gridDim.x) * 126;
    return st + 126 > a.ncell ? (a.ncell > 126 ? a.ncell - 126 : (int64_t)0) : st;
  };

  dep_trigger();
  if (warp == 4) {   // ---- producer: lane 0 takes the barriers, lanes 0..17 one A copy each
    if (plan.resident && my_tiles > 0 && lane == 0) {   // weights: not written by the kernels before
      mbar_expect_tx(&wfull, plan.w_bytes);
      bulk_load(wsm, a.Wt, plan.w_bytes, &wfull);
    }
    dep_wait();
    // this lane's copy: (di, plane q), and dj where the slabs do not overlap
    // (the lane after: the streamed weights)
    const int copies = plan.merged ? 6 : 18, sl = lane >> 1, q = lane & 1;
    const int di = plan.merged ? sl : sl / 3, dj = plan.merged ? 0 : sl % 3;
    const int64_t slab_off = (di - 1) * P + (dj - 1) * (int64_t)a.n3;
    const uint32_t slab_dst = (uint32_t)(2 * di + q) * plan.plane_bytes + (uint32_t)dj * 2048u;
    const uint32_t slab_bytes = plan.merged ? plan.plane_bytes : 2048u;
    int st = 0, pass = 0, issued = 0;
    bool ok = true;
    for (int k = 0; k < my_tiles && ok; k++) {
      const int64_t row_base = tile_start(k) - 1;
      for (int c = 0; c < nk; c++) {
        if (pass > 0) {
          bool w = true;
          if (lane == 0) w = bk_wait(&empty[st], (uint32_t)((pass - 1) & 1), abort_p);
          if (!__shfl_sync(0xffffffffu, w, 0)) {
            ok = false;
            break;
          }
        }
        uint8_t* sa = stg + st * plan.stage_bytes;
        if (lane == 0) mbar_expect_tx(&full[st], 6u * plan.plane_bytes + (plan.resident ? 0u : plan.b_bytes));
        if (lane < copies)
          bulk_load(sa + slab_dst, a.in + (2 * c + q) * a.in_ps + (row_base + slab_off) * 8, slab_bytes, &full[st]);
        else if (lane == copies && !plan.resident)
          bulk_load(sa + plan.a_bytes, a.Wt + (int64_t)c * 9 * N3 * 16, plan.b_bytes, &full[st]);
        issued++;
        if (++st == S) {
          st = 0;
          pass++;
        }
      }
    }
    // every copy issued has landed before the CTA may leave: the last phase
    // of each stage used, and the weights
    if (lane == 0) {
      for (int s = 0; s < S; s++) {
        const int n = issued / S + (s < issued % S ? 1 : 0);   // uses of stage s
        if (n > 0) bk_wait(&full[s], (uint32_t)((n - 1) & 1), abort_p, false);
      }
      if (plan.resident && my_tiles > 0) bk_wait(&wfull, 0, abort_p, false);
    }
    __syncwarp();
  } else if (warp == 5) {
    {   // ---- MMA issuer
      const bool leader = tc::elect_one();
      const uint32_t idesc = tc::idesc_bf16_f32(128, N3);
      const uint32_t b_lbo = (uint32_t)N3 * 16;
      bool ok = !plan.resident || my_tiles == 0 || bk_wait_warp(&wfull, 0, abort_p);
      int st = 0, pass = 0;
      for (int k = 0; k < my_tiles && ok; k++) {
        const int acc = k & 1;
        if (k >= 2 && !bk_wait_warp(&tempty[acc], (uint32_t)(((k >> 1) - 1) & 1), abort_p)) break;
        tc::fence_after_sync();
        const uint32_t dacc = tbase + (uint32_t)(acc * plan.acc_off);
        for (int c = 0; c < nk; c++) {
          if (!bk_wait_warp(&full[st], (uint32_t)(pass & 1), abort_p)) {
            ok = false;
            break;
          }
          tc::fence_after_sync();
          const uint8_t* sa = stg + st * plan.stage_bytes;
          const uint8_t* sb = plan.resident ? wsm + (size_t)c * 9 * N3 * 32 : sa + plan.a_bytes;
#pragma unroll
          for (int sl = 0; sl < 9; sl++) {
            const uint64_t ad = tc::smem_desc(tc::smem_addr(sa) + (uint32_t)(sl / 3) * 2u * plan.plane_bytes +
                                                  (uint32_t)((sl % 3) * plan.step) * 16u, plan.plane_bytes, 128);
            const uint64_t bd = tc::smem_desc(tc::smem_addr(sb + sl * N3 * 32), b_lbo, 128);
            if (leader) tc::mma_bf16(dacc, ad, bd, idesc, c > 0 || sl > 0);
          }
          if (leader) tc::mma_commit(&empty[st]);
          if (++st == S) {
            st = 0;
            pass++;
          }
        }
        if (ok && leader) tc::mma_commit(&tfull[acc]);
      }
      // every MMA issued has completed before TMEM is freed
      if (leader) tc::mma_commit(&mdone);
      bk_wait_warp(&mdone, 0, abort_p, false);
    }
    __syncwarp();
  } else {   // ---- epilogue, warps 0-3
    dep_wait();
    for (int k = 0; k < my_tiles; k++) {
      const int acc = k & 1;
      const bool got = bk_wait(&tfull[acc], (uint32_t)((k >> 1) & 1), abort_p);
      if (!epi_sync_and(got)) break;
      tc::fence_after_sync();
      const int64_t c0 = tile_start(k);
      const uint32_t trow = tbase + (uint32_t)(acc * plan.acc_off) + ((uint32_t)(warp * 32) << 16);
      float(*xc)[2][80] = xch[acc];
      const int r = warp * 32 + lane;
      const int64_t c = c0 + r - 1;
      const bool live = r >= 1 && r <= 126 && c < a.ncell;
      const float m = live ? (float)a.mask[c] : 0.f;
      // the neighbour row a lane needs from another warp: lane 0 warp-1's
      // D_-1 edge, lane 31 warp+1's D_+1 edge (others read one and discard it)
      const float* nbr = lane == 0 ? xc[warp > 0 ? warp - 1 : 0][0] : xc[warp < 3 ? warp + 1 : 3][1];
      const bool has_nbr = lane == 0 ? warp > 0 : warp < 3;
      // 16 output channels at a time: D_-1, D_0 and D_+1 columns in three
      // loads under one wait
      for (int co = 0; co < Co; co += 16) {
        uint32_t dm[16], d0[16], dp[16];
        tc::tmem_ld16_nowait(trow + (uint32_t)co, dm);
        tc::tmem_ld16_nowait(trow + (uint32_t)(Co + co), d0);
        tc::tmem_ld16_nowait(trow + (uint32_t)(2 * Co + co), dp);
        tc::tmem_wait_ld(dm, d0, dp);
        if (lane == 31 || lane == 0) {
          const uint32_t* e = lane == 31 ? dm : dp;
          float4* dst = reinterpret_cast<float4*>(&xc[warp][lane == 31 ? 0 : 1][co]);
#pragma unroll
          for (int j = 0; j < 4; j++)
            dst[j] = make_float4(__uint_as_float(e[4 * j]), __uint_as_float(e[4 * j + 1]),
                                 __uint_as_float(e[4 * j + 2]), __uint_as_float(e[4 * j + 3]));
        }
        epi_sync();
        float nb[16];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const float4 w4 = reinterpret_cast<const float4*>(nbr + co)[j];
          nb[4 * j] = w4.x; nb[4 * j + 1] = w4.y; nb[4 * j + 2] = w4.z; nb[4 * j + 3] = w4.w;
        }
        float v[2][8];
#pragma unroll
        for (int q = 0; q < 16; q++) {
          float prev = __shfl_up_sync(0xffffffffu, __uint_as_float(dm[q]), 1);
          float next = __shfl_down_sync(0xffffffffu, __uint_as_float(dp[q]), 1);
          const float e = has_nbr ? nb[q] : 0.f;
          if (lane == 0) prev = e;
          if (lane == 31) next = e;
          v[q >> 3][q & 7] = prev + __uint_as_float(d0[q]) + next;
        }
        if (live && co < a.out_ch) conv_store8(a, c, co, m, v[0]);
        if (live && co + 8 < a.out_ch) conv_store8(a, c, co + 8, m, v[1]);
      }
      // the accumulator is read: the MMA issuer may overwrite it two tiles on
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag) atomicExch(a.err, 1);
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tbase, (uint32_t)plan.tmem_cols);
}

// Wide outputs (3 Co > 256), tap by tap: a tile is 128 consecutive cells, the
// A operand of tap t the rows c0 + o_t .. c0 + o_t + 127, the B operand W[t]; the
// 27 taps x Ci / 16 MMAs of N = Co accumulate in order.  A stage is one tap: its
// planes' rows and its weights by bulk copies, already in operand layout, with
// the roles, waits and two accumulators of the kernel above.  The tensor core
// is idle most of the time here too (27 x 2 MMAs a tile at Ci = 32); what
// counts is how many taps are in flight.  32 -> 96 at 34^3: 29.5 us, with the
// operands staged by the threads and one barrier a tap 81.
constexpr int WD_MAX_STAGES = 8;
struct WdPlan { int stages, acc_off, tmem_cols, smem_bytes, per_sm; uint32_t a_bytes, b_bytes, stage_bytes; };
static WdPlan wd_plan(int ci, int co) {
  WdPlan p = {};
  p.acc_off = (co + 31) / 32 * 32;
  p.tmem_cols = (int)tmem_cols(p.acc_off + co);   // at most 256: two CTAs an SM
  p.a_bytes = (uint32_t)(ci / 8) * 2048;
  p.b_bytes = (uint32_t)(co * ci * 2);
  p.stage_bytes = (p.a_bytes + p.b_bytes + 1023) / 1024 * 1024;
  for (p.per_sm = 2; p.per_sm >= 1; p.per_sm--) {
    const int avail = 228 * 1024 / p.per_sm - 1024 - 2048;   // less the part reserved, the static and the slack
    p.stages = std::min(WD_MAX_STAGES, avail / (int)p.stage_bytes);
    if (p.stages >= 3 || p.per_sm == 1) break;
  }
  p.smem_bytes = p.stages * (int)p.stage_bytes + 1024;
  return p;
}
__global__ void __launch_bounds__(BK_THREADS) k_conv3_wide(ConvArgs a, WdPlan plan) {
  extern __shared__ uint8_t dsm[];
  __shared__ uint64_t full[WD_MAX_STAGES], empty[WD_MAX_STAGES], tfull[2], tempty[2], mdone;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  const int Ci = a.Ci, Co = a.Co, S = plan.stages;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t raw = tc::smem_addr(dsm);
  uint8_t* stg = dsm + ((1024u - (raw & 1023u)) & 1023u);
  if (warp == 0) tc::tmem_alloc(&tmem_base, (uint32_t)plan.tmem_cols);
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int q = 0; q < 2; q++) {
      tc::mbar_init(&tfull[q], 1);
      tc::mbar_init(&tempty[q], 4);
    }
    tc::mbar_init(&mdone, 1);
    abort_flag = 0;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = tmem_base;
  volatile int* abort_p = &abort_flag;
  const int64_t P = (int64_t)a.n2 * a.n3;
  const int64_t ntiles = (a.ncell + TC_M - 1) / TC_M;
  const int my_tiles = ntiles > blockIdx.x ? (int)((ntiles - 1 - blockIdx.x) / gridDim.x + 1) : 0;
  dep_trigger();
  if (warp == 4) {   // ---- producer: a plane of A per lane (at most 16), the weights by lane 16
    dep_wait();
    int st = 0, pass = 0, issued = 0;
    bool ok = true;
    for (int k = 0; k < my_tiles && ok; k++) {
      const int64_t c0 = ((int64_t)blockIdx.x + (int64_t)k * gridDim.x) * TC_M;
      for (int t = 0; t < 27; t++) {
        if (pass > 0) {
          bool w = true;
          if (lane == 0) w = bk_wait(&empty[st], (uint32_t)((pass - 1) & 1), abort_p);
          if (!__shfl_sync(0xffffffffu, w, 0)) {
            ok = false;
            break;
          }
        }
        uint8_t* sa = stg + (size_t)st * plan.stage_bytes;
        if (lane == 0) mbar_expect_tx(&full[st], plan.a_bytes + plan.b_bytes);
        __syncwarp();
        const int64_t off = (t / 9 - 1) * P + ((t / 3) % 3 - 1) * (int64_t)a.n3 + (t % 3 - 1);
        if (lane < Ci / 8) bulk_load(sa + lane * 2048, a.in + lane * a.in_ps + (c0 + off) * 8, 2048, &full[st]);
        else if (lane == 16) bulk_load(sa + plan.a_bytes, a.Wt + (int64_t)t * Co * Ci, plan.b_bytes, &full[st]);
        issued++;
        if (++st == S) {
          st = 0;
          pass++;
        }
      }
    }
    if (lane == 0)   // every copy issued has landed before the CTA may leave
      for (int s = 0; s < S; s++) {
        const int n = issued / S + (s < issued % S ? 1 : 0);
        if (n > 0) bk_wait(&full[s], (uint32_t)((n - 1) & 1), abort_p, false);
      }
    __syncwarp();
  } else if (warp == 5) {   // ---- MMA issuer
    const bool leader = tc::elect_one();
    const uint32_t idesc = tc::idesc_bf16_f32(TC_M, Co);
    int st = 0, pass = 0;
    bool ok = true;
    for (int k = 0; k < my_tiles && ok; k++) {
      const int acc = k & 1;
      if (k >= 2 && !bk_wait_warp(&tempty[acc], (uint32_t)(((k >> 1) - 1) & 1), abort_p)) break;
      tc::fence_after_sync();
      const uint32_t dacc = tbase + (uint32_t)(acc * plan.acc_off);
      for (int t = 0; t < 27; t++) {
        if (!bk_wait_warp(&full[st], (uint32_t)(pass & 1), abort_p)) {
          ok = false;
          break;
        }
        tc::fence_after_sync();
        const uint32_t sa = tc::smem_addr(stg + (size_t)st * plan.stage_bytes), sb = sa + plan.a_bytes;
        for (int q = 0; q < Ci / 16; q++) {
          const uint64_t ad = tc::smem_desc(sa + (uint32_t)q * 4096, 2048, 128);
          const uint64_t bd = tc::smem_desc(sb + (uint32_t)(q * Co * 32), (uint32_t)Co * 16, 128);
          if (leader) tc::mma_bf16(dacc, ad, bd, idesc, t > 0 || q > 0);
        }
        if (leader) tc::mma_commit(&empty[st]);
        if (++st == S) {
          st = 0;
          pass++;
        }
      }
      if (ok && leader) tc::mma_commit(&tfull[acc]);
    }
    // every MMA issued has completed before TMEM is freed
    if (leader) tc::mma_commit(&mdone);
    bk_wait_warp(&mdone, 0, abort_p, false);
    __syncwarp();
  } else {   // ---- epilogue, warps 0-3: TMEM lanes 32 w .. 32 w + 31
    dep_wait();
    for (int k = 0; k < my_tiles; k++) {
      const int acc = k & 1;
      const bool got = bk_wait(&tfull[acc], (uint32_t)((k >> 1) & 1), abort_p);
      if (!epi_sync_and(got)) break;
      tc::fence_after_sync();
      const int64_t c = ((int64_t)blockIdx.x + (int64_t)k * gridDim.x) * TC_M + warp * 32 + lane;
      const bool live = c < a.ncell;
      const float m = live ? (float)a.mask[c] : 0.f;
      const uint32_t trow = tbase + (uint32_t)(acc * plan.acc_off) + ((uint32_t)(warp * 32) << 16);
      for (int co = 0; co < Co; co += 8) {
        float v[8];
        tc::tmem_ld8(trow + (uint32_t)co, v);
        if (live && co < a.out_ch) conv_store8(a, c, co, m, v);
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag) atomicExch(a.err, 1);
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tbase, (uint32_t)plan.tmem_cols);
}

// Error flag of the convolutions: a slot of the context scratch, cleared by
// xf_conv_status.
constexpr int I_CONV_ERR = 60;
static int* conv_err_flag(xf_ctx* ctx) { return reinterpret_cast<int*>(&ctx->scratch->iscalars[I_CONV_ERR]); }

// The dynamic shared-memory attribute of a convolution kernel, raised once
// per kernel and device to the largest size asked for (so that the launches
// of a captured solve set no attribute).
static cudaError_t set_max_smem(const void* kern, int which, int device, size_t smem) {
  static size_t done[3][64] = {};
  size_t& d = done[which][device & 63];
  if (smem <= d) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) d = smem;
  return e;
}

// ---------------------------------------------------------------------------
// Weight gradient of the convolution on the tensor cores:
//     dW[t][co][ci] = sum over cells c of g[c][co] x[c + off_t][ci].
// With the activations in channel planes, 8 consecutive cells of one plane
// are also the canonical MN-major core matrix (8 channels along M or N, one
// cell per 16-byte row along K), so the sum over cells is the K dimension of
// an MMA: M = 128 rows of stacked (di, dj, input channel) groups of 8, N = co, A
// = the shifted x blocks, B = g.  The three dk of a (di, dj) read the same block
// of 130 cells a cell (16 bytes) apart, into accumulators of their own: a row
// tile of single taps copied every block three times, and the copies were what
// bound it (48 -> 16 at 66^3: 880 MB from L2 in 107 us, now 280 MB in 77; 96 -> 32
// at 34^3 58 -> 27).  Now shared memory does (58 to 62% of its throughput, the tensor
// pipe at 7 to 11%): an MMA of N = 16 takes about 60 cycles.  A stage is 128 cells:
// per group of the row tile and per plane of g one bulk copy (one per lane of
// the producer warp), eight K steps of 16 cells, three MMAs each.  Each CTA
// takes one row tile and one range of cells (a multiple of 128: the cells past
// the box read the zero margins), accumulates in TMEM, and writes its FP32
// partials where the sum looks for them: [tile of 128 / ci taps][range][row];
// k_grad_sum adds the ranges in a fixed order (deterministic).  Groups past
// the last compute on whatever the stage holds, in rows that nothing reads.
// Descriptors: no swizzle, MN-major (instruction descriptor bits 15 and 16),
// LBO = the K-direction core-matrix stride (128 bytes), SBO = the MN-direction
// stride (a block).
constexpr int WG_KC = 128;                         // cells per stage
constexpr int WG_STAGES = 3;
constexpr uint32_t WG_BLOCK = WG_KC * 16;          // one plane of g of a stage
constexpr uint32_t WG_GROUP = (WG_KC + 2) * 16;    // one (di, dj, plane) group
struct WgArgs {
  const uint16_t* g;   // plane 0, cell 0
  int64_t gps;
  int co;
  const uint16_t* x;
  int64_t xps;
  int ci;
  int n2, n3;
  int taps, splits, stages;      // of the partials: taps a tile, cell ranges; stages a range
  int tiles, per_tile;           // row tiles here, groups a tile
  uint32_t a_bytes;              // A's part of a stage
  int64_t chunks;                      // 128-cell stages in all
  uint32_t stage_bytes;
  float* partial;   // [mtile][split][128][co]
  int* err;
};

__global__ void __launch_bounds__(BK_THREADS) k_wgrad_tc(WgArgs a) {
  extern __shared__ uint8_t dsm[];
  __shared__ uint64_t full[WG_STAGES], empty[WG_STAGES], mdone;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int mt = blockIdx.x % a.tiles, sp = blockIdx.x / a.tiles;
  const int cp = a.ci / 8, g0 = mt * a.per_tile;
  const int ga = min(9 * cp - g0, a.per_tile), gb = a.co / 8;   // blocks of A and of B per stage
  const uint32_t raw = tc::smem_addr(dsm);
  uint8_t* smem = dsm + ((1024u - (raw & 1023u)) & 1023u);
  const uint32_t ncols = tmem_cols(3 * a.co);
  if (warp == 0) tc::tmem_alloc(&tmem_base, ncols);
  if (threadIdx.x == 0) {
    for (int st = 0; st < WG_STAGES; st++) {
      tc::mbar_init(&full[st], 1);
      tc::mbar_init(&empty[st], 1);
    }
    tc::mbar_init(&mdone, 1);
    abort_flag = 0;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = tmem_base;
  volatile int* abort_p = &abort_flag;
  const int64_t P = (int64_t)a.n2 * a.n3;
  const int64_t cell0 = (int64_t)sp * a.stages * WG_KC;
  // this range's stages: the last range stops at the box's last 128-cell chunk
  const int my_stages = (int)min((int64_t)a.stages, a.chunks - (int64_t)sp * a.stages);
  dep_trigger();
  if (warp == 4) {   // ---- producer: one copy per lane
    dep_wait();
    const bool is_a = lane < ga, is_b = lane >= ga && lane < ga + gb;
    const uint16_t* src = nullptr;
    uint32_t dst_off = 0;
    if (is_a) {   // from the cell before the range's first
      const int dij = (g0 + lane) / cp, q = (g0 + lane) % cp;
      src = a.x + q * a.xps + ((dij / 3 - 1) * P + (dij % 3 - 1) * (int64_t)a.n3 - 1) * 8;
      dst_off = (uint32_t)lane * WG_GROUP;
    } else if (is_b) {
      const int q = lane - ga;
      src = a.g + q * a.gps;
      dst_off = a.a_bytes + (uint32_t)q * WG_BLOCK;
    }
    const uint32_t bytes = is_a ? WG_GROUP : WG_BLOCK;
    int st = 0, pass = 0, issued = 0;
    for (int k = 0; k < my_stages; k++) {
      if (pass > 0) {
        bool w = true;
        if (lane == 0) w = bk_wait(&empty[st], (uint32_t)((pass - 1) & 1), abort_p);
        if (!__shfl_sync(0xffffffffu, w, 0)) break;
      }
      uint8_t* sa = smem + st * a.stage_bytes;
      if (lane == 0) mbar_expect_tx(&full[st], (uint32_t)ga * WG_GROUP + (uint32_t)gb * WG_BLOCK);
      if (is_a || is_b) bulk_load(sa + dst_off, src + (cell0 + (int64_t)k * WG_KC) * 8, bytes, &full[st]);
      issued++;
      if (++st == WG_STAGES) {
        st = 0;
        pass++;
      }
    }
    if (lane == 0)   // every copy issued has landed before the CTA may leave
      for (int s2 = 0; s2 < WG_STAGES; s2++) {
        const int n = issued / WG_STAGES + (s2 < issued % WG_STAGES ? 1 : 0);
        if (n > 0) bk_wait(&full[s2], (uint32_t)((n - 1) & 1), abort_p, false);
      }
    __syncwarp();
  } else if (warp == 5) {
    {   // ---- MMA issuer
      const bool leader = tc::elect_one();
      const uint32_t idesc = tc::idesc_bf16_f32(128, a.co) | (1u << 15) | (1u << 16);   // A and B MN-major
      int st = 0, pass = 0;
      for (int k = 0; k < my_stages; k++) {
        if (!bk_wait_warp(&full[st], (uint32_t)(pass & 1), abort_p)) break;
        tc::fence_after_sync();
        const uint8_t* sa = smem + st * a.stage_bytes;
#pragma unroll
        for (int kk = 0; kk < WG_KC / 16; kk++) {
          const uint64_t bd = tc::smem_desc(tc::smem_addr(sa) + a.a_bytes + (uint32_t)kk * 256u, 128, WG_BLOCK);
#pragma unroll
          for (int dk = 0; dk < 3; dk++) {
            const uint64_t ad = tc::smem_desc(tc::smem_addr(sa) + (uint32_t)kk * 256u + (uint32_t)dk * 16u, 128, WG_GROUP);
            if (leader) tc::mma_bf16(tbase + (uint32_t)(dk * a.co), ad, bd, idesc, k > 0 || kk > 0);
          }
        }
        if (leader) tc::mma_commit(&empty[st]);
        if (++st == WG_STAGES) {
          st = 0;
          pass++;
        }
      }
      if (leader) tc::mma_commit(&mdone);   // every MMA issued
    }
    __syncwarp();
  } else {   // ---- epilogue, warps 0-3: the partial of this tile and range
    dep_wait();
    const bool got = bk_wait(&mdone, 0, abort_p, false);
    if (__all_sync(0xffffffffu, got) && !*abort_p) {
      tc::fence_after_sync();
      const int row = warp * 32 + lane, grp = g0 + (row >> 3);
      const bool live = (row >> 3) < ga;
      for (int dk = 0; dk < 3; dk++) {
        const int t = grp / cp * 3 + dk, r = (t % a.taps) * a.ci + grp % cp * 8 + (row & 7);
        float* dst = a.partial + (((int64_t)(t / a.taps) * a.splits + sp) * 128 + r) * a.co;
        for (int co = 0; co < a.co; co += 8) {
          float v[8];
          tc::tmem_ld8(tbase + ((uint32_t)(warp * 32) << 16) + (uint32_t)(dk * a.co + co), v);
          if (!live) continue;
          *reinterpret_cast<float4*>(dst + co) = make_float4(v[0], v[1], v[2], v[3]);
          *reinterpret_cast<float4*>(dst + co + 4) = make_float4(v[4], v[5], v[6], v[7]);
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag) atomicExch(a.err, 1);
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tbase, ncols);
}

// Bias gradient: partial sums over chunks of cells, a block per chunk and
// 8-channel plane of g.  Bound by latency (142 blocks at 64^3): a thread's 16
// loads of a 4,096-cell chunk are in flight together, then a fixed tree over
// the threads.
__global__ void __launch_bounds__(256) k_bgrad(const uint16_t* __restrict__ g, int64_t gps, int64_t ncell, int chunk,
                                               int co, float* __restrict__ bpart) {
  __shared__ float part[8][256];
  dep_trigger();
  dep_wait();
  const int q = blockIdx.y, u = threadIdx.x;
  const int64_t beg = (int64_t)blockIdx.x * chunk, end = min(ncell, beg + chunk);
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int64_t c0 = beg + u; c0 < end; c0 += 16 * 256) {
    uint4 v[16];
#pragma unroll
    for (int k = 0; k < 16; k++) {
      v[k] = make_uint4(0, 0, 0, 0);
      if (c0 + k * 256 < end) v[k] = __ldg(reinterpret_cast<const uint4*>(g + q * gps + (c0 + k * 256) * 8));
    }
#pragma unroll
    for (int k = 0; k < 16; k++) {
      if (c0 + k * 256 >= end) break;
      const uint32_t w[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
      for (int e = 0; e < 4; e++) {
        s[2 * e] += __uint_as_float(w[e] << 16);
        s[2 * e + 1] += __uint_as_float(w[e] & 0xFFFF0000u);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 8; e++) part[e][u] = s[e];
  __syncthreads();
  // warp e takes channel e: 128, 64, 32 by shared memory, the rest by shuffles, t += t + h at every level
  const int e = u >> 5, l = u & 31;
  float a[8];
#pragma unroll
  for (int k = 0; k < 8; k++) a[k] = part[e][l + 32 * k];
#pragma unroll
  for (int h = 4; h > 0; h >>= 1)
#pragma unroll
    for (int k = 0; k < h; k++) a[k] += a[k + h];
#pragma unroll
  for (int h = 16; h > 0; h >>= 1) a[0] += __shfl_down_sync(0xffffffffu, a[0], h);
  if (l == 0) bpart[(int64_t)blockIdx.x * co + q * 8 + e] = a[0];
}

// The layers' partials summed in order: every layer's weights and biases in
// one launch (11 took 9.9 us each at 64^3, their loads strided by co).  Threads
// run along co, as the partials lie; a layer's last block sums its bias
// chunks.
__global__ void __launch_bounds__(256) k_grad_sum(const __grid_constant__ WgSegs segs) {
  dep_trigger();
  dep_wait();
  int k = 0;
  while (k + 1 < WG_LAYERS && (int)blockIdx.x >= segs.s[k + 1].block0) k++;
  const WgSeg& g = segs.s[k];
  const int nw = 27 * g.co * g.ci, u = ((int)blockIdx.x - g.block0) * 256 + threadIdx.x;
  if (u < nw) {   // nw is a multiple of 256
    const int o = u % g.co, ti = u / g.co, t = ti / g.ci, i = ti - t * g.ci;
    const int mt = t / g.taps, row = (t - mt * g.taps) * g.ci + i;
    const float* p = g.wpart + ((int64_t)mt * g.splits * 128 + row) * g.co + o;
    const int64_t step = (int64_t)128 * g.co;
    float s = 0.f;
#pragma unroll 16
    for (int sp = 0; sp < g.splits; sp++) s += __ldg(p + sp * step);
    g.gw[(t * g.co + o) * g.ci + i] = s;
    return;
  }
  const int o = threadIdx.x;   // the chunks in order
  if (o >= g.co) return;
  float s = 0.f;
#pragma unroll 16
  for (int c = 0; c < g.nchunk; c++) s += __ldg(g.bpart + (int64_t)c * g.co + o);
  g.gb[o] = s;
}
int xf_grad_sum_blocks(int ci, int co) { return 27 * co * ci / 256 + 1; }
void xf_grad_sum(xf_ctx* ctx, const WgSegs& segs, int blocks) { launch_dep(k_grad_sum, dim3(blocks), 256, 0, ctx->stream, segs); }

// Chunks of the bias gradient: 4,096 cells, or more in steps of 256 so that there are at most 128.
void xf_bgrad_plan(int64_t ncell, int* nchunk, int* chunk) {
  int64_t c = ((ncell + 127) / 128 + 255) / 256 * 256;
  if (c < 4096) c = 4096;
  *chunk = (int)c;
  *nchunk = (int)((ncell + c - 1) / c);
}
// The row tiles and cell ranges of a layer's weight-gradient partials, and the FP32 buffer they need (floats).
void xf_wgrad_tc_plan(const xf_ctx* ctx, int64_t ncell, int ci, int co, int* mtiles, int* splits, int* stages,
                      int64_t* partial_floats) {
  const int taps = 128 / ci;
  *mtiles = (27 + taps - 1) / taps;
  const int64_t chunks = (ncell + WG_KC - 1) / WG_KC;
  int64_t sp = ((int64_t)ctx->sm_count * 2 + *mtiles - 1) / *mtiles;
  if (sp > chunks) sp = chunks;
  if (sp < 1) sp = 1;
  *stages = (int)((chunks + sp - 1) / sp);
  *splits = (int)((chunks + *stages - 1) / *stages);
  *partial_floats = (int64_t)*mtiles * *splits * 128 * co;
}

// The partials of the weight gradient of g (co channels) against x (ci channels),
// both BF16 planes with their zero margins, into `partial` (xf_wgrad_tc_plan's
// floats), and of the bias gradient into bpart; xf_grad_sum adds them.  ci and co
// multiples of 16, ci <= 128, co <= 64.
int xf_wgrad_tc(xf_ctx* ctx, int n1, int n2, int n3, const void* g, int64_t gps, int co, const void* x, int64_t xps,
                int ci, float* partial, float* bpart) {
  if (ci % 16 || co % 16 || ci < 16 || ci > 128 || co < 16 || co > 64)
    return xf_fail(ctx, XF_ERR_ARG, "weight gradient: channel counts out of range");
  WgArgs a;
  a.g = (const uint16_t*)g; a.gps = gps; a.co = co;
  a.x = (const uint16_t*)x; a.xps = xps; a.ci = ci;
  a.n2 = n2; a.n3 = n3;
  int64_t pf = 0;
  int mtiles;
  xf_wgrad_tc_plan(ctx, (int64_t)n1 * n2 * n3, ci, co, &mtiles, &a.splits, &a.stages, &pf);
  a.taps = 128 / ci;
  const int groups = 9 * (ci / 8);
  a.tiles = (groups + 15) / 16;
  a.per_tile = (groups + a.tiles - 1) / a.tiles;
  a.a_bytes = ((uint32_t)a.per_tile * WG_GROUP + 127) / 128 * 128;
  a.chunks = ((int64_t)n1 * n2 * n3 + WG_KC - 1) / WG_KC;
  a.stage_bytes = (a.a_bytes + (uint32_t)co / 8 * WG_BLOCK + 1023) / 1024 * 1024;
  a.partial = partial;
  a.err = conv_err_flag(ctx);
  // the last stage's rows of absent groups lie past it, in memory of the block's own
  const size_t smem = (size_t)WG_STAGES * a.stage_bytes + 1024 + 16 * WG_GROUP;
  XF_CUDA(ctx, set_max_smem((const void*)k_wgrad_tc, 1, ctx->device, smem));
  launch_dep(k_wgrad_tc, dim3((unsigned)(a.tiles * a.splits)), BK_THREADS, smem, ctx->stream, a);
  int nchunk, chunk;
  xf_bgrad_plan((int64_t)n1 * n2 * n3, &nchunk, &chunk);
  launch_dep(k_bgrad, dim3((unsigned)nchunk, (unsigned)(co / 8)), 256, 0, ctx->stream, a.g, gps, (int64_t)n1 * n2 * n3,
             chunk, co, bpart);
  XF_CUDA(ctx, cudaGetLastError());
  return XF_OK;
}

// Launch on the context stream (arguments checked by the caller).  `tiled`: the
// weights in conv_tiled_index order.  dep: launched by launch_dep, the weights not
// written by the kernel before.
int xf_conv_launch(xf_ctx* ctx, int n1, int n2, int n3, const void* in, int64_t in_ps, int ci, const void* tiled,
                   const float* bias, int co, const uint8_t* mask, void* out, int64_t out_pitch, int out_ch,
                   int out_fp32, int relu, const void* gate, int64_t gate_ps, bool dep) {
  ConvArgs a;
  a.gate = (const uint16_t*)gate; a.gate_ps = gate_ps;
  a.in = (const uint16_t*)in; a.in_ps = in_ps; a.Ci = ci;
  a.Wt = (const uint16_t*)tiled; a.bias = bias; a.Co = co;
  a.mask = mask; a.n2 = n2; a.n3 = n3; a.ncell = (int64_t)n1 * n2 * n3;
  a.out16 = out_fp32 ? nullptr : (uint16_t*)out;
  a.out32 = out_fp32 ? (float*)out : nullptr;
  a.out_ps = out_fp32 ? 0 : out_pitch;
  a.out_ld = out_fp32 ? (int)out_pitch : 0;
  a.out_ch = out_ch; a.relu = relu; a.err = conv_err_flag(ctx);
  if (conv_wide(co)) {
    const WdPlan plan = wd_plan(ci, co);
    XF_CUDA(ctx, set_max_smem((const void*)k_conv3_wide, 2, ctx->device, (size_t)plan.smem_bytes));
    const int64_t tiles = (a.ncell + TC_M - 1) / TC_M;
    const int64_t blocks = std::min(tiles, (int64_t)ctx->sm_count * plan.per_sm);
    if (dep) launch_dep(k_conv3_wide, dim3((unsigned)blocks), BK_THREADS, plan.smem_bytes, ctx->stream, a, plan);
    else k_conv3_wide<<<(int)blocks, BK_THREADS, plan.smem_bytes, ctx->stream>>>(a, plan);
    XF_CUDA(ctx, cudaGetLastError());
    return XF_OK;
  }
  // k-taps stacked along N
  static int static_smem = -1;
  if (static_smem < 0) {
    cudaFuncAttributes fa;
    XF_CUDA(ctx, cudaFuncGetAttributes(&fa, k_conv3_bulk));
    static_smem = (int)fa.sharedSizeBytes;
  }
  const BkPlan plan = bk_plan(ci, co, n3, static_smem);
  if (plan.stages < 2) return xf_fail(ctx, XF_ERR_ARG, "convolution: no stacked-tap plan");
  XF_CUDA(ctx, set_max_smem((const void*)k_conv3_bulk, 0, ctx->device, (size_t)plan.smem_bytes));
  const int64_t tiles = (a.ncell + 125) / 126;
  int64_t blocks = (int64_t)ctx->sm_count * plan.per_sm;
  if (blocks > tiles) blocks = tiles;
  if (dep) launch_dep(k_conv3_bulk, dim3((unsigned)blocks), BK_THREADS, plan.smem_bytes, ctx->stream, a, plan);
  else k_conv3_bulk<<<(int)blocks, BK_THREADS, plan.smem_bytes, ctx->stream>>>(a, plan);
  XF_CUDA(ctx, cudaGetLastError());
  return XF_OK;
}

// Weights [27][co][ci] into the tiled order (conv_tiled_index).
__global__ void k_tile_weights(const uint16_t* __restrict__ w, int co, int ci, uint16_t* __restrict__ wt) {
  const int64_t n = (int64_t)27 * co * ci;
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < n; u += (int64_t)gridDim.x * blockDim.x) {
    const int t = (int)(u / ((int64_t)co * ci));
    const int o = (int)((u / ci) % co), i = (int)(u % ci);
    wt[conv_tiled_index(t, o, i, co, ci)] = w[u];
  }
}

extern "C" int xf_conv3d_bf16(xf_ctx* ctx, int n1, int n2, int n3, const void* in, int64_t in_ps, int ci,
                              const void* weights, const float* bias, int co, const uint8_t* mask, void* out,
                              int64_t out_pitch, int out_ch, int out_fp32, int relu) {
  if (!ctx || !in || !weights || !mask || !out) return XF_ERR_ARG;
  const int64_t ncell = (int64_t)n1 * n2 * n3;
  const int64_t rows_min = ncell + XF_CONV_MARGIN(n2, n3);   // a plane's rows from cell 0 on
  if (ci < 16 || ci > 128 || ci % 16 || co < 16 || co > 128 || co % 16 || out_ch < 1 || out_ch > co ||
      n1 < 3 || n2 < 3 || n3 < 3 || in_ps < (rows_min + XF_CONV_MARGIN(n2, n3)) * 8 || in_ps % 8 ||
      (out_fp32 ? out_pitch < out_ch : (out_pitch < ncell * 8 || out_pitch % 8 || out_ch % 8)))
    return xf_fail(ctx, XF_ERR_ARG, "xf_conv3d_bf16: channel counts / plane strides out of range");
  if (((uintptr_t)in | (uintptr_t)weights | (uintptr_t)out) & 15)
    return xf_fail(ctx, XF_ERR_ARG, "xf_conv3d_bf16: pointers must be 16-byte aligned");
  XF_CUDA(ctx, cudaSetDevice(ctx->device));
  void* tiled = nullptr;
  const int64_t nw = (int64_t)27 * co * ci;
  XF_CUDA(ctx, cudaMallocAsync(&tiled, nw * 2, ctx->stream));
  k_tile_weights<<<(unsigned)((nw + 255) / 256), 256, 0, ctx->stream>>>((const uint16_t*)weights, co, ci,
                                                                        (uint16_t*)tiled);
  const int st = xf_conv_launch(ctx, n1, n2, n3, in, in_ps, ci, tiled, bias, co, mask, out, out_pitch,
                                out_ch, out_fp32, relu, nullptr, 0, false);
  cudaFreeAsync(tiled, ctx->stream);
  return st;
}

// Reads and clears the error flag of the convolutions since the last call
// (synchronises the stream).
extern "C" int xf_conv_status(xf_ctx* ctx) {
  if (!ctx) return XF_ERR_ARG;
  int* err = conv_err_flag(ctx);
  int h = 0;
  XF_CUDA(ctx, cudaMemcpyAsync(&h, err, 4, cudaMemcpyDeviceToHost, ctx->stream));
  XF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  XF_CUDA(ctx, cudaMemsetAsync(err, 0, 4, ctx->stream));
  if (h) return xf_fail(ctx, XF_ERR_CUDA, "convolution: a tensor-core completion wait ran out");
  return XF_OK;
}
