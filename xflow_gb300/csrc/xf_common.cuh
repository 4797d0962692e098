// Internal definitions shared by the xflow_gb300 CUDA translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "../../include/xflow.h"

// ---------------------------------------------------------------------------
// Cell kind byte: bits 0..5 = neighbour in direction (-x,+x,-y,+y,-z,+z) is
// not Fictive (flux open, XOperator.cpp:1003-1008); bits 6..7 = row kind.
enum : uint8_t {
  K_MX = 1, K_PX = 2, K_MY = 4, K_PY = 8, K_MZ = 16, K_PZ = 32,
  K_ROW_SHIFT = 6,
  ROW_NONE = 0, ROW_ACTUAL = 1, ROW_PREDEF = 2, ROW_PRENORM = 3
};
__host__ __device__ inline int row_of(uint8_t k) { return k >> K_ROW_SHIFT; }

// Fixed reduction geometry: deterministic partial sums (one per block, then a
// fixed-order final pass by the last block to finish).
constexpr int RED_THREADS = 256;
constexpr int RED_MAX_BLOCKS = 8192;  // partials per slot (stencil grids can be 2-D)
constexpr int NUM_SLOTS = 16;         // independent reductions in flight

// Device-resident scratch of a context.
struct DevScratch {
  double partials[NUM_SLOTS][RED_MAX_BLOCKS];
  unsigned int tickets[NUM_SLOTS];
  double scalars[256];
  long long iscalars[64];
  volatile long long* progress;   // pinned host word: ends of iterations seen, bit 62 once the solve is done
};

struct xf_ctx {
  int device;
  int sm_count;
  cudaStream_t stream;
  DevScratch* scratch;       // device
  double* host_scalars;      // pinned, 256 doubles
  cudaEvent_t ev0, ev1;
  void* work = nullptr;       // device workspace of line solvers (grows, freed by xf_destroy)
  size_t work_bytes = 0;
  char err[512];
};

// Device workspace of at least `bytes` (nullptr when it cannot grow).
void* xf_ctx_work(xf_ctx* ctx, size_t bytes);

// Split of a grid's interior into the bricks of the resident CG (xf_cgc.cu):
// state 0 not looked at, 1 valid, -1 the grid does not fit.
struct xf_coop_plan {
  int state, bi, bj, bk, mi, mj, mk, threads;
  size_t smem;
};

struct xf_grid {
  xf_ctx* ctx;
  int n1, n2, n3;
  int64_t ncell, s1, s2;
  int64_t end_index;
  uint8_t* code;             // device, per cell: the reference point code (0..8)
  uint8_t* nflag;            // device, per Normal (code 5) cell: bit 0/1/2 = normal x/y/z nonzero
  uint8_t* kind;             // device, per cell, then 64 zero bytes
  uint8_t* smask;            // device, per cell (0/1)
  int32_t* inv;              // device, Rn index per cell (0 inactive)
  int32_t* brow_of;          // device, per cell: index into brow arrays or -1
  int64_t nbrow;             // PreDefined + PreNormal rows
  double* brow_nrm;          // device, 3 per boundary row
  double *hx, *hy, *hz;      // device separations (n-1 each)
  float *fhx, *fhy, *fhz;
  // fast-path coefficients per index: c?m[i] = 1/(h[i-1]*hh[i]), c?p[i] = 1/(h[i]*hh[i]),
  // hh[i] = (h[i-1]+h[i])/2; rh = 1/h; rhh = 1/hh
  double *cxm, *cxp, *cym, *cyp, *czm, *czp;
  float *fxm, *fxp, *fym, *fyp, *fzm, *fzp;
  double *rhx, *rhy, *rhz, *rhhx, *rhhy, *rhhz;
  float *frhx, *frhy, *frhz, *frhhx, *frhhy, *frhhz;
  double* diag;              // device, per cell: diagonal of the Laplace Actual row (fast FP64)
  int uniform;               // every separation of each axis is equal: coefficients are per-axis constants
  double ucx, ucy, ucz;      // then 1/h^2 per axis (== c?m[i] == c?p[i] for every interior index)
  xf_coop_plan coop[2];      // FP64, mixed
  int lap_status, vardiv_status;
  int64_t lap_bad, vardiv_bad;
};

struct xf_vec {
  xf_grid* g;
  int dtype;
  void* data;
};

struct PackData;   // packed operator storage (xf_pack.cu)
struct xf_op {
  xf_grid* g;
  int kind;
  double* rho;     // device density box (VARDIV)
  float* rho32;
  int rho_set;
  PackData* pack = nullptr;   // XF_OP_PACK
  int transposed = 0;         // XF_OP_PACK: applies A^T (T1dPackOperator::operator~)
  // XF_OP_ADVDIFF: advecting velocity boxes (FP64 and FP32 copies) and coefficients
  double* adv64[3] = {nullptr, nullptr, nullptr};
  float* adv32[3] = {nullptr, nullptr, nullptr};
  double* adD64 = nullptr;   // per-cell diffusion coefficient (null: the constant ad_D)
  float* adD32 = nullptr;
  int adD_set = 0;
  double ad_tau = 1, ad_D = 0;
  int ad_flags = 0, adv_set = 0;
  // the FP64 fast Actual rows' coefficients (7 per cell, SoA), refreshed by
  // xf_op_ready after either setter; invalid until then (the rows then take
  // the exact form)
  mutable double* adc64 = nullptr;
  mutable int adc_valid = 0;
  // per cell, with the table: the neighbours its row reads (bits 0..5, x- to
  // z+), AD_ROW for a row, AD_OBLIQUE for one that is not of seven points
  mutable uint8_t* adk = nullptr;
  mutable int adv32_valid = 0;   // the FP32 copies are made on first use
  // and the inverse row diagonals (0 off the active set), for the Jacobi
  // preconditioner of BiCGStab, refreshed with the table
  mutable double* adj64 = nullptr;
  // the six neighbour coefficients times the neighbours' inverse diagonals
  // (A D^-1 has a unit diagonal) and their use bytes, made by xf_op_scaled
  // for the solves that want them; invalid whenever the table is
  mutable double* ads64 = nullptr;
  mutable uint8_t* adks = nullptr;
  mutable int ads_valid = 0;
  mutable int lap_jac_valid = 0;   // XF_OP_LAPLACE: adj64 holds its inverse diagonals (built on first use)
  // device staging boxes of xf_solve_host, kept between calls
  xf_vec* host_x = nullptr;
  xf_vec* host_b = nullptr;
  // unique per operator ever created (a graph built for one operator is never
  // replayed on another that reuses its address)
  unsigned long long serial = 0;
};

// ---------------------------------------------------------------------------
int xf_fail(xf_ctx* ctx, int status, const char* fmt, ...);
#define XF_CUDA(ctx, call)                                                              \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess) return xf_fail((ctx), XF_ERR_CUDA, "%s: %s (%s:%d)", #call,  \
                                          cudaGetErrorString(e_), __FILE__, __LINE__);   \
  } while (0)

// Programmatic dependent launch: a kernel launched by launch_dep may start while
// the kernel before it on the stream drains (once all its blocks have left or
// called dep_trigger); dep_wait returns when that kernel has completed and its
// writes are visible, and before it only data that no kernel of the chain
// writes may be touched.  A plain launch makes both calls empty.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... P, typename... A>
inline void launch_dep(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3((unsigned)threads); cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cfg.attrs = at; cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, P(args)...);   // an error shows in cudaGetLastError
}

inline int grid_blocks(const xf_ctx* ctx, int64_t n, int threads, int per_sm = 8) {
  int64_t b = (n + threads - 1) / threads;
  int64_t cap = (int64_t)ctx->sm_count * per_sm;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}
inline int red_blocks(const xf_ctx* ctx, int64_t n) {
  int b = grid_blocks(ctx, n, RED_THREADS, 8);
  return b > RED_MAX_BLOCKS ? RED_MAX_BLOCKS : b;
}
__device__ __forceinline__ int lin_block() { return blockIdx.y * gridDim.x + blockIdx.x; }
__device__ __forceinline__ int num_blocks() { return gridDim.x * gridDim.y; }

// ---------------------------------------------------------------------------
// Per-thread dot accumulators.  FP64 data: plain FP64 FMA.  FP32 data: the
// product a*b is split exactly into hi + lo with one FMA (TwoProduct) and
// summed in float-float (TwoSum), so the per-thread partial carries ~44 bits
// without touching the FP64 pipe (1/58 of the FP32 rate on GB300); partials
// are combined in FP64 across threads and blocks.
template <typename T>
struct DotAcc;
template <>
struct DotAcc<double> {
  double s = 0.0;
  __device__ __forceinline__ void add(double a, double b) { s = fma(a, b, s); }
  __device__ __forceinline__ double value() const { return s; }
};
template <>
struct DotAcc<float> {
  float hi = 0.f, lo = 0.f;
  __device__ __forceinline__ void add(float a, float b) {
    const float p = a * b;
    const float e = fmaf(a, b, -p);
    const float s = hi + p;
    const float bp = s - hi;
    const float err = (hi - (s - bp)) + (p - bp);
    hi = s;
    lo = lo + (err + e);
  }
  __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// Sum of the block's accumulators, valid in thread 0.  FP32 accumulators are
// reduced across each warp in float-float (FP32 pipe) and reach FP64 once per
// warp, so the epilogue issues ~1/32 of the FP64 instructions of a per-thread
// conversion.
__device__ inline double warp_sum(double v);
template <typename T>
__device__ inline double block_sum_acc(const DotAcc<T>& acc, double* sh);
template <>
__device__ inline double block_sum_acc<double>(const DotAcc<double>& acc, double* sh);
template <>
__device__ inline double block_sum_acc<float>(const DotAcc<float>& acc, double* sh) {
  float hi = acc.hi, lo = acc.lo;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float bh = __shfl_xor_sync(0xffffffffu, hi, o), bl = __shfl_xor_sync(0xffffffffu, lo, o);
    const float s = hi + bh;
    const float bp = s - hi;
    const float err = (hi - (s - bp)) + (bh - bp);
    hi = s;
    lo = lo + (bl + err);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[w] = (double)hi + (double)lo;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  double v = (threadIdx.x < nw) ? sh[threadIdx.x] : 0.0;
  if (w == 0) v = warp_sum(v);
  return v;
}

// First strict maximum of |a| in flat order: (value, cell) pairs combine by
// larger value, then smaller cell.
struct AbsMax { double v; long long c; };
__device__ __forceinline__ AbsMax am_combine(AbsMax x, AbsMax y) {
  if (y.c < 0) return x;
  if (x.c < 0) return y;
  if (y.v > x.v || (y.v == x.v && y.c < x.c)) return y;
  return x;
}
__device__ __forceinline__ AbsMax am_warp(AbsMax a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    AbsMax b;
    b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
    b.c = __shfl_xor_sync(0xffffffffu, a.c, o);
    a = am_combine(a, b);
  }
  return a;
}
__device__ inline AbsMax am_block(AbsMax a, AbsMax* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  a = am_warp(a);
  __syncthreads();
  if (lane == 0) sh[w] = a;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  AbsMax r;
  r.v = 0; r.c = -1;
  if (threadIdx.x < nw) r = sh[threadIdx.x];
  if (w == 0) r = am_warp(r);
  return r;
}

// Block reduction helpers (FP64).
__device__ inline double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum over the block; result valid in thread 0.  sh must hold 32 doubles.
__device__ inline double block_sum(double v, double* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  v = (threadIdx.x < nw) ? sh[threadIdx.x] : 0.0;
  if (w == 0) v = warp_sum(v);
  return v;
}

// Sums of NV values a thread over a block of at most RED_THREADS threads,
// valid in thread 0: the threads' values go through shared memory and a warp a
// value adds them.  With every warp adding its own lanes by shuffles, the FP64
// pipe (16 cycles an instruction here) spent as much on a block's sums as on
// half a row a thread: 45 additions a value and block instead of 12.
template <int NV>
__device__ inline void block_sums(const double (&v)[NV], double (&out)[NV]) {
  __shared__ double buf[NV * RED_THREADS];
  const int n = blockDim.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = n >> 5;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; q++) buf[q * RED_THREADS + threadIdx.x] = v[q];
  __syncthreads();
  for (int q = w; q < NV; q += nw) {
    double a = 0.0, b = 0.0;
    for (int t = lane; t < n; t += 64) {
      a += buf[q * RED_THREADS + t];
      if (t + 32 < n) b += buf[q * RED_THREADS + t + 32];
    }
    a = warp_sum(a + b);
    __syncwarp();
    if (lane == 0) buf[q * RED_THREADS] = a;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; q++) out[q] = buf[q * RED_THREADS];
}

template <>
__device__ inline double block_sum_acc<double>(const DotAcc<double>& acc, double*) {
  const double v[1] = {acc.value()};
  double s[1];
  block_sums<1>(v, s);
  return s[0];
}

// Publishes one accumulator into partials[slot] under tickets[ticket]; true in
// the last block to arrive.
template <typename T>
__device__ inline bool publish_acc(DevScratch* S, int slot, int ticket, const DotAcc<T>& acc, double* sh, bool* flag) {
  const double s = block_sum_acc<T>(acc, sh);
  if (threadIdx.x == 0) {
    S->partials[slot][lin_block()] = s;
    __threadfence();
    unsigned int t = atomicAdd(&S->tickets[ticket], 1u);
    *flag = (t == (unsigned)num_blocks() - 1);
  }
  __syncthreads();
  return *flag;
}

// Publishes this block's partial of `nval` sums into slot partials and returns
// true in the last block to arrive (all partials visible).  `flag` is shared.
template <int NV>
__device__ inline bool publish_partials(DevScratch* S, int slot0, const double (&v)[NV], double*, bool* flag) {
  double s[NV];
  block_sums<NV>(v, s);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < NV; q++) S->partials[slot0 + q][lin_block()] = s[q];
    __threadfence();
    unsigned int t = atomicAdd(&S->tickets[slot0], 1u);
    *flag = (t == (unsigned)num_blocks() - 1);
  }
  __syncthreads();
  return *flag;
}

// In the last block: fixed-order sum of the published partials of slot.
__device__ inline double finish_partials(DevScratch* S, int slot, double* sh) {
  __threadfence();
  double v = 0.0;
  const int nb = num_blocks();
  for (int b = threadIdx.x; b < nb; b += blockDim.x) v += __ldcg(&S->partials[slot][b]);
  return block_sum(v, sh);
}

// ---------------------------------------------------------------------------
// -v by the sign bit: compiled from a minus sign, the negated operand of an
// FP64 FMA was an instruction of the FP64 pipe of its own (7 of the 18 that a
// Laplace row took), where this is one integer operation.
__device__ __forceinline__ double xneg(double v) {
  return __hiloint2double(__double2hiint(v) ^ (int)0x80000000, __double2loint(v));
}
__device__ __forceinline__ float xneg(float v) { return -v; }

// a / b correctly rounded, from y = RN(1/b), itself a normal number (the grid's
// reciprocal tables, 1/tau from the host, or __drcp_rn).  q = RN(a y) lies within an ulp of a / b, the
// residual r = a - b q is exact (one FMA), and RN(q + r y) = RN(a / b):
// Markstein's theorem for FMA-based division (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34(1), 1990; also Muller et al., Handbook of Floating-Point
// Arithmetic, ch. 5).  Three FP64 operations instead of the IEEE division's
// reciprocal iteration, which matters at GB300's FP64 rate (1/58 of FP32).
// The theorem needs a normal, unclamped residual: a numerator or quotient
// outside [2^-950, 2^1000) in magnitude (zero, tiny, huge, not finite, or a
// divisor of 0 or infinity) takes the IEEE division itself.  Checked bit for
// bit against the IEEE division by xf_selftest_division.
__device__ __forceinline__ double div_rcp(double a, double b, double y) {
  const double q = a * y;
  const unsigned ea = ((unsigned)__double2hiint(a) >> 20) & 0x7ffu, eq = ((unsigned)__double2hiint(q) >> 20) & 0x7ffu;
  if (ea - (1023u - 950u) >= 1950u || eq - (1023u - 950u) >= 1950u) return a / b;
  const double r = fma(xneg(b), q, a);
  return fma(r, y, q);
}

// ---------------------------------------------------------------------------
// BF16 activations of the learned preconditioner are stored in channel planes
// of 8: plane q holds channels 8q .. 8q+7 of every cell, 16 bytes per cell,
// so element (cell c, channel ch) sits at (ch / 8) * plane_stride + c * 8 +
// ch % 8.  A block of consecutive cells of one plane is then the canonical
// K-major operand layout of the tensor cores (core matrices of 8 rows x 16
// bytes), copied by one bulk copy whatever its first cell.
//
// Convolution weights for the tensor cores, tiled per (16-channel input
// chunk c, slab s = 3 (di+1) + (dj+1), 8-channel half q, stacked output row
// n = dk_index * Co + o, 8 channels): the 9 slabs of one chunk are contiguous,
// and each (c, s) block is the canonical K-major B operand of one MMA.
// Outputs wider than 80 channels (3 Co columns of an MMA are at most 256) go
// tap by tap: per (tap, 8-channel plane, output row, 8 channels).
__host__ __device__ inline bool conv_wide(int co) { return 3 * co > 256; }
__host__ __device__ inline int64_t conv_tiled_index(int t, int o, int i, int co, int ci) {
  if (conv_wide(co)) return (((int64_t)t * (ci / 8) + (i >> 3)) * co + o) * 8 + (i & 7);
  const int s = t / 3, n = (t % 3) * co + o, c = i >> 4, q = (i >> 3) & 1, e = i & 7;
  return ((((int64_t)c * 9 + s) * 2 + q) * (3 * co) + n) * 8 + e;
}

// The partial sums of one layer's gradients and where their totals go.
constexpr int WG_LAYERS = 11;
struct WgSeg {
  const float *wpart, *bpart;   // [row tile][cell range][128][co]; [chunk][co]
  float *gw, *gb;               // [27][co][ci]; [co]
  int mtiles, splits, taps, ci, co, nchunk, block0;
};
struct WgSegs { WgSeg s[WG_LAYERS]; };
