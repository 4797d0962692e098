// Batched tridiagonal lines: TSLAE::SolveByScalarRunning (XSLAE.cpp:416-445)
// for every grid line of an ADI sweep at once.
//
// Line (l1, l2), element m of every array sits at l1*ls1 + l2*ls2 + m*ms, so
// the lines of a box along any axis are one call (e.g. along i: ms = s1,
// ls1 = s2 over j, ls2 = 1 over k).  One thread per line runs the reference's
// recurrences in its operation order:
//     A[0] = 0, B[0] = u[0];
//     A[m] = -c[m] / (a[m] A[m-1] + b[m]),  B[m] = (f[m] - a[m] B[m-1]) / (a[m] A[m-1] + b[m]);
//     u[m] = A[m] u[m+1] + B[m],  m = M-1 .. 1  (u[0], u[M] are boundary values).
// FP64 without contraction and with correctly rounded division: bit-identical
// to the serial reference.
//
// What bounds it: the FP64 pipe, once the loads no longer stall the chain.  A
// step's two quotients share their divisor, so one correctly rounded
// reciprocal and two Markstein corrections (div_rcp, 3 operations each) give
// both; and a thread loads the LN_STEPS steps after the ones it computes.  A
// 130^3 box took 239 us a sweep with the loads of each step behind the last
// one's divisions.  A[m] goes to the context's workspace laid out [m][line]
// (coalesced across the threads of a warp).  Lines whose elements are
// neighbours in memory (ms = 1, the sweep along k) are staged through shared
// memory in tiles of LN_TILE steps by asynchronous copies, two tiles in
// flight: the threads of a warp would otherwise touch a sector each for 8
// bytes of it.  Their B goes back to u by the same tiles, so that the workspace
// is A's alone on every axis (a box of its own for B was freed for and allocated
// again between two axes: the first pass over a 66^3 box took 402 us, 283 now).
#include "xf_common.cuh"

constexpr int LN_THREADS = 64, LN_STEPS = 4, LN_TILE = 16;

// One step of the forward recurrence.
__device__ __forceinline__ void ln_step(double a, double b, double c, double f, double& A, double& B) {
  const double den = a * A + b, num = f - a * B;
  const unsigned e = ((unsigned)__double2hiint(den) >> 20) & 0x7ffu;
  if (e - 64u < 1900u) {   // the reciprocal is a normal number
    const double y = __drcp_rn(den);
    A = div_rcp(xneg(c), den, y);
    B = div_rcp(num, den, y);
  } else {
    A = xneg(c) / den;
    B = num / den;
  }
}

struct LnArgs {
  int M, nl2;
  int64_t nl, ls1, ls2, ms;
  double* __restrict__ u;
  const double* __restrict__ a;
  const double* __restrict__ b;
  const double* __restrict__ c;
  const double* __restrict__ f;
  double* __restrict__ Aw;   // [m][line]
};

// Lines side by side in memory.  B[m] waits in u[m] until the back-substitution.
__global__ void __launch_bounds__(LN_THREADS) k_thomas(LnArgs g) {
  const int64_t l = blockIdx.x * (int64_t)LN_THREADS + threadIdx.x;
  if (l >= g.nl) return;
  const int l1 = (int)(l / g.nl2), l2 = (int)(l - (int64_t)l1 * g.nl2);
  const int64_t base = l1 * g.ls1 + l2 * g.ls2;
  const int last = g.M - 1;
  double A = 0, B = g.u[base];
  double na[LN_STEPS], nb[LN_STEPS], nc[LN_STEPS], nf[LN_STEPS];
  auto load = [&](int m0) {
#pragma unroll
    for (int q = 0; q < LN_STEPS; q++) {
      const int64_t e = base + min(m0 + q, last) * g.ms;   // past the end: the last step's, unused
      na[q] = g.a[e]; nb[q] = g.b[e]; nc[q] = g.c[e]; nf[q] = g.f[e];
    }
  };
  load(1);
  for (int m0 = 1; m0 <= last; m0 += LN_STEPS) {
    double a[LN_STEPS], b[LN_STEPS], c[LN_STEPS], f[LN_STEPS];
#pragma unroll
    for (int q = 0; q < LN_STEPS; q++) { a[q] = na[q]; b[q] = nb[q]; c[q] = nc[q]; f[q] = nf[q]; }
    if (m0 + LN_STEPS <= last) load(m0 + LN_STEPS);
#pragma unroll
    for (int q = 0; q < LN_STEPS; q++) {
      const int m = m0 + q;
      if (m <= last) {
        ln_step(a[q], b[q], c[q], f[q], A, B);
        g.Aw[(int64_t)m * g.nl + l] = A;
        g.u[base + m * g.ms] = B;
      }
    }
  }
  double un = g.u[base + (int64_t)g.M * g.ms];
  constexpr int BS = 2 * LN_STEPS;
  double pa[BS], pb[BS];
  auto back = [&](int m0) {   // steps m0, m0 - 1, ...
#pragma unroll
    for (int q = 0; q < BS; q++) {
      const int m = max(m0 - q, 1);
      pa[q] = g.Aw[(int64_t)m * g.nl + l];
      pb[q] = g.u[base + m * g.ms];
    }
  };
  back(last);
  for (int m0 = last; m0 >= 1; m0 -= BS) {
    double a[BS], b[BS];
#pragma unroll
    for (int q = 0; q < BS; q++) { a[q] = pa[q]; b[q] = pb[q]; }
    if (m0 - BS >= 1) back(m0 - BS);
#pragma unroll
    for (int q = 0; q < BS; q++)
      if (m0 - q >= 1) {
        un = a[q] * un + b[q];
        g.u[base + (m0 - q) * g.ms] = un;
      }
  }
}

__device__ __forceinline__ void ln_copy8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// Lines along the memory (ms = 1).
constexpr int LN_PITCH = LN_TILE + 1;                 // doubles of a line in a tile: 16 lanes hit 32 banks
constexpr int LN_BOX = LN_THREADS * LN_PITCH;         // a tile of one array
__global__ void __launch_bounds__(LN_THREADS) k_thomas_k(LnArgs g) {
  extern __shared__ double ln_sm[];   // two stages of a, b, c, f
  __shared__ int64_t bases[LN_THREADS];
  const int t = threadIdx.x;
  const int64_t l0 = blockIdx.x * (int64_t)LN_THREADS, l = l0 + t;
  const bool mine = l < g.nl;
  const int64_t lc = mine ? l : g.nl - 1;
  const int l1 = (int)(lc / g.nl2), l2 = (int)(lc - (int64_t)l1 * g.nl2);
  const int64_t base = l1 * g.ls1 + l2 * g.ls2;
  bases[t] = base;
  __syncthreads();
  const int last = g.M - 1;
  // a half warp a line: LN_TILE consecutive elements of each array
  const int e = t % LN_TILE, q0 = t / LN_TILE;
  constexpr int LINES = LN_THREADS / LN_TILE;
  auto stage = [&](int tile) {
    double* s = ln_sm + (tile & 1) * 4 * LN_BOX + e;
    const int m = 1 + tile * LN_TILE + e;
    if (m <= last)
      for (int q = q0; q < LN_THREADS; q += LINES) {
        const int64_t src = bases[q] + m;
        double* dst = s + q * LN_PITCH;
        ln_copy8(dst, g.a + src);
        ln_copy8(dst + LN_BOX, g.b + src);
        ln_copy8(dst + 2 * LN_BOX, g.c + src);
        ln_copy8(dst + 3 * LN_BOX, g.f + src);
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto stage_u = [&](int tile) {
    const int m = 1 + tile * LN_TILE + e;
    if (tile >= 0 && m <= last)
      for (int q = q0; q < LN_THREADS; q += LINES) ln_copy8(ln_sm + (tile & 1) * LN_BOX + q * LN_PITCH + e, g.u + bases[q] + m);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto put_u = [&](int tile, const double* box) {   // between two block barriers
    const int m = 1 + tile * LN_TILE + e;
    if (m <= last)
      for (int q = q0; q < LN_THREADS && l0 + q < g.nl; q += LINES) g.u[bases[q] + m] = box[q * LN_PITCH + e];
  };
  const int tiles = (last + LN_TILE - 1) / LN_TILE;
  double A = 0, B = g.u[base];
  stage(0);
  for (int tile = 0; tile < tiles; tile++) {
    stage(tile + 1);   // past the end: an empty group
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    double* s = ln_sm + (tile & 1) * 4 * LN_BOX + t * LN_PITCH;
    const int m0 = 1 + tile * LN_TILE;
#pragma unroll 4
    for (int q = 0; q < LN_TILE; q++) {
      const int m = m0 + q;
      if (m > last) break;
      ln_step(s[q], s[LN_BOX + q], s[2 * LN_BOX + q], s[3 * LN_BOX + q], A, B);
      if (mine) g.Aw[(int64_t)m * g.nl + l] = A;
      s[3 * LN_BOX + q] = B;
    }
    __syncthreads();
    put_u(tile, s + 3 * LN_BOX - t * LN_PITCH);
    __syncthreads();   // the tile's place is filled again two stages on
  }
  double un = g.u[base + g.M];
  stage_u(tiles - 1);
  for (int tile = tiles - 1; tile >= 0; tile--) {
    const int m0 = 1 + tile * LN_TILE;
    double a[LN_TILE];
#pragma unroll
    for (int q = 0; q < LN_TILE; q++) a[q] = g.Aw[(int64_t)min(m0 + q, last) * g.nl + lc];
    stage_u(tile - 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    double* box = ln_sm + (tile & 1) * LN_BOX;
    double* row = box + t * LN_PITCH;
#pragma unroll
    for (int q = LN_TILE - 1; q >= 0; q--)
      if (m0 + q <= last) {
        un = a[q] * un + row[q];
        row[q] = un;
      }
    __syncthreads();
    put_u(tile, box);
    __syncthreads();
  }
}

extern "C" int xf_thomas_lines(xf_ctx* ctx, int M, int nl1, int nl2, int64_t ls1, int64_t ls2, int64_t ms, double* u,
                               const double* a, const double* b, const double* c, const double* f) {
  if (!ctx || !u || !a || !b || !c || !f) return XF_ERR_ARG;
  if (M < 1 || nl1 < 0 || nl2 < 0) return xf_fail(ctx, XF_ERR_ARG, "xf_thomas_lines: M >= 1 and line counts >= 0");
  const int64_t nl = (int64_t)nl1 * nl2;
  if (nl == 0 || M == 1) return XF_OK;   // nothing between the two boundary values
  XF_CUDA(ctx, cudaSetDevice(ctx->device));
  double* Aw = (double*)xf_ctx_work(ctx, (size_t)M * nl * sizeof(double));
  if (!Aw) return xf_fail(ctx, XF_ERR_NOMEM, "xf_thomas_lines: workspace of %lld doubles", (long long)(M * nl));
  LnArgs g = {M, nl2, nl, ls1, ls2, ms, u, a, b, c, f, Aw};
  const unsigned blocks = (unsigned)((nl + LN_THREADS - 1) / LN_THREADS);
  if (ms == 1 && !(nl2 > 1 ? ls2 == 1 : ls1 == 1)) {   // along the memory, and neighbouring lines not one element apart
    const int smem = 2 * 4 * LN_BOX * (int)sizeof(double);
    XF_CUDA(ctx, cudaFuncSetAttribute(k_thomas_k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k_thomas_k<<<blocks, LN_THREADS, smem, ctx->stream>>>(g);
  } else {
    k_thomas<<<blocks, LN_THREADS, 0, ctx->stream>>>(g);
  }
  XF_CUDA(ctx, cudaGetLastError());
  return XF_OK;
}
