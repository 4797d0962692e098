// The learned two-level preconditioner between its grids, F = 4 (blocks of
// 4 x 4 x 4 fine cells under a coarse cell): omega of the coarse correction,
// and the smoother's input.
//
// With y = P zc (a block's value in its active cells) the rows A y differ from
// zero only at the faces between blocks, so nothing of y or A y is stored:
//   (y, A y) is a sum over the coarse cells, with the open fine faces of each
//   block side counted once a solve (k_tl_faces),
//   (y, r) = (zc, P^T r) is one too,
//   r - omega A y takes A y from the coarse values as it passes over r.
// Before, a pass wrote y and A y (134 MB at 256^3, 66 us), two dots followed
// and the smoother's first pass read both (92 us).
#include <stdint.h>

#include "xf_control.cuh"
#include "xf_stencil.cuh"

namespace {

// Open faces of each side of the block under a coarse cell (0 to 16: five bits
// a side, MX, PX, MY, PY, MZ, PZ), of rows with an equation.
__global__ void k_tl_faces(const uint8_t* __restrict__ kind, int f2, int f3, uint32_t* __restrict__ cnt, int c1, int c2,
                           int c3) {
  const int K = blockIdx.x * blockDim.x + threadIdx.x, J = blockIdx.y, I = blockIdx.z;
  if (K >= c3) return;
  uint32_t v = 0;
  if (I > 0 && I < c1 - 1 && J > 0 && J < c2 - 1 && K > 0 && K < c3 - 1) {
    const uint8_t* b = kind + ((int64_t)(1 + 4 * (I - 1)) * f2 + (1 + 4 * (J - 1))) * f3 + (1 + 4 * (K - 1));
    const int64_t s1 = (int64_t)f2 * f3, s2 = f3;
    auto side = [&](int64_t at, int64_t u, int64_t w, uint8_t bit, int shift) {
      uint32_t n = 0;
      for (int p = 0; p < 4; p++)
        for (int q = 0; q < 4; q++) {
          const uint8_t kb = b[at + p * u + q * w];
          n += (kb >> K_ROW_SHIFT) != ROW_NONE && (kb & bit) ? 1u : 0u;
        }
      v |= n << shift;
    };
    side(0, s2, 1, K_MX, 0);
    side(3 * s1, s2, 1, K_PX, 5);
    side(0, s1, 1, K_MY, 10);
    side(3 * s2, s1, 1, K_PY, 15);
    side(0, s1, s2, K_MZ, 20);
    side(3, s1, s2, K_PZ, 25);
  }
  cnt[((int64_t)I * c2 + J) * c3 + K] = v;
}

// omega = (y, r) / (y, A y) -> scalars[s_om], 0 when (y, A y) is not positive
// or either sum is not finite.  Row differences in FP32 (as the rows of A y),
// sums in FP64.  Bound by latency: 287,496 coarse cells under 256^3.
__global__ void __launch_bounds__(RED_THREADS) k_tl_omega(const float* __restrict__ zc, const uint32_t* __restrict__ cnt,
                                                          const double* __restrict__ rc, int64_t nc, int sI, int sJ,
                                                          float cx, float cy, float cz, DevScratch* S, int slot,
                                                          int s_om) {
  __shared__ double sh[32];
  __shared__ bool last;
  dep_trigger();
  dep_wait();
  double v[2] = {0.0, 0.0};
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < nc; c += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t m = cnt[c];
    const float z = zc[c];
    auto face = [&](int shift, int64_t off) -> float {   // a closed side's neighbour is not read
      const uint32_t n = (m >> shift) & 31u;
      return n ? (float)n * (z - __ldg(zc + c + off)) : 0.f;
    };
    const float d = fmaf(cx, face(0, -sI) + face(5, sI), fmaf(cy, face(10, -sJ) + face(15, sJ),
                                                              cz * (face(20, -1) + face(25, 1))));
    v[0] = fma((double)z, (double)d, v[0]);
    v[1] = fma((double)z, rc[c], v[1]);
  }
  if (!publish_partials<2>(S, slot, v, sh, &last)) return;
  const double yay = finish_partials(S, slot, sh), yr = finish_partials(S, slot + 1, sh);
  if (threadIdx.x == 0) {
    S->scalars[slot] = yay;
    S->scalars[slot + 1] = yr;
    S->scalars[s_om] = tl_omega(yay, yr);
    S->tickets[slot] = 0;
  }
}

// out = r - omega A P zc.  Bound by memory: r, a byte of row kind and out, 9
// bytes a cell.  A thread takes four consecutive cells of a plane (two pairs;
// rows and blocks start at odd k, so a pair lies in one row, and a difference
// between its two blocks is the pair's only one along k) and marches over the
// planes: of the six neighbours only the one across the block's j side and
// the next block along i are loaded, once per four planes.  256^3: 151 MB, 22 us
// of memory time, 37 us measured (41 with two blocks an SM at 90 registers).
__global__ void __launch_bounds__(256, 3) k_tl_sub(const uint8_t* __restrict__ kind, const float* __restrict__ r,
                                                const float* __restrict__ zc, int n1, int n3, int P, int c2, int c3,
                                                int chunk, float cx, float cy, float cz, const DevScratch* S, int s_om,
                                                float* __restrict__ out) {
  dep_trigger();
  dep_wait();
  const int p0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (p0 >= P) return;
  const float om = (float)S->scalars[s_om];
  const int i0 = blockIdx.y * chunk, i1 = min(n1, i0 + chunk);
  const int sI = c2 * c3;
  int o[4], jo[2];        // the cells' coarse offsets in a plane; the pairs' neighbour rows
  uint8_t jbit[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int p = p0 + 2 * h, j = p / n3, k = p - j * n3;
    const int row = (1 + ((j - 1) >> 2)) * c3;
    o[2 * h] = row + 1 + ((k - 1) >> 2);
    o[2 * h + 1] = row + 1 + (k >> 2);
    const int jm = (j - 1) & 3;
    jo[h] = jm == 0 ? -c3 : jm == 3 ? c3 : 0;
    jbit[h] = jm == 0 ? K_MY : jm == 3 ? K_PY : 0;
  }
  float zm[4], z[4], zp[4], dy[4], dz[2];   // the cells' blocks before, at and after; differences along j and k
  auto load = [&](int I, float (&v)[4]) {
    const float* b = zc + (int64_t)min(max(I, 0), (n1 - 2) / 4 + 1) * sI;
#pragma unroll
    for (int q = 0; q < 4; q++) v[q] = __ldg(b + o[q]);
  };
  auto turn = [&](int I) {   // zm, z, zp stand around block I
    const float* b = zc + (int64_t)I * sI;
#pragma unroll
    for (int q = 0; q < 4; q++) dy[q] = cy * (z[q] - __ldg(b + o[q] + jo[q >> 1]));
    dz[0] = cz * (z[0] - z[1]);
    dz[1] = cz * (z[2] - z[3]);
  };
  int I = 1 + ((i0 - 1) >> 2);
  load(I - 1, zm);
  load(I, z);
  load(I + 1, zp);
  turn(I);
  int64_t c = (int64_t)i0 * P + p0;
  for (int i = i0; i < i1;) {
    const int im0 = (i - 1) & 3, cnt = min(4 - im0, i1 - i);   // planes left in this block
    float4 rv[4];
    uchar4 kk[4];
#pragma unroll
    for (int t = 0; t < 4; t++)
      if (t < cnt) {
        rv[t] = *reinterpret_cast<const float4*>(r + c + (int64_t)t * P);
        kk[t] = *reinterpret_cast<const uchar4*>(kind + c + (int64_t)t * P);
      }
#pragma unroll
    for (int t = 0; t < 4; t++)
      if (t < cnt) {
        const bool lo = im0 + t == 0, hi = im0 + t == 3;
        const uint8_t kb[4] = {kk[t].x, kk[t].y, kk[t].z, kk[t].w};
        float v[4] = {rv[t].x, rv[t].y, rv[t].z, rv[t].w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
          float d = kb[q] & jbit[q >> 1] ? dy[q] : 0.f;
          if (kb[q] & (q & 1 ? K_MZ : K_PZ)) d += q & 1 ? -dz[q >> 1] : dz[q >> 1];
          if (lo && (kb[q] & K_MX)) d = fmaf(cx, z[q] - zm[q], d);
          if (hi && (kb[q] & K_PX)) d = fmaf(cx, z[q] - zp[q], d);
          if ((kb[q] >> K_ROW_SHIFT) != ROW_NONE) v[q] = fmaf(-om, d, v[q]);
        }
        *reinterpret_cast<float4*>(out + c + (int64_t)t * P) = make_float4(v[0], v[1], v[2], v[3]);
      }
    i += cnt;
    c += (int64_t)cnt * P;
    if (i < i1) {
      I++;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        zm[q] = z[q];
        z[q] = zp[q];
      }
      load(I + 1, zp);
      turn(I);
    }
  }
}

// The same from a stored A y, any F: omega from its two sums first.
__global__ void k_tl_sub_ay(const float* __restrict__ r, const float* __restrict__ ay, int64_t n, DevScratch* S,
                            int s_yay, int s_yr, int s_om, float* __restrict__ out) {
  __shared__ float som;
  if (threadIdx.x == 0) {
    const double w = tl_omega(S->scalars[s_yay], S->scalars[s_yr]);
    if (blockIdx.x == 0) S->scalars[s_om] = w;
    som = (float)w;
  }
  __syncthreads();
  const float om = som;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x)
    out[c] = fmaf(-om, ay[c], r[c]);
}

}  // namespace

void xf_tl_faces(const xf_grid* g, const xf_grid* cg, uint32_t* cnt) {
  k_tl_faces<<<dim3((cg->n3 + 63) / 64, cg->n2, cg->n1), 64, 0, g->ctx->stream>>>(g->kind, g->n2, g->n3, cnt, cg->n1,
                                                                                 cg->n2, cg->n3);
}

// (y, A y), (y, r) -> scalars[slot], scalars[slot + 1]; omega -> scalars[s_om].
void xf_tl_omega(const xf_grid* g, const xf_grid* cg, const float* zc, const uint32_t* cnt, const double* rc, int slot,
                 int s_om) {
  const int blocks = red_blocks(g->ctx, cg->ncell);
  launch_dep(k_tl_omega, dim3(blocks), RED_THREADS, 0, g->ctx->stream, zc, cnt, rc, cg->ncell, cg->n2 * cg->n3, cg->n3,
             (float)g->ucx, (float)g->ucy, (float)g->ucz, g->ctx->scratch, slot, s_om);
}

// Plane sizes and row lengths of the grid fit four-cell groups of whole pairs:
// n2 n3 a multiple of 4 and n3 even, as F = 4 gives them (4 a + 2 each).
void xf_tl_sub(const xf_grid* g, const float* r, const float* zc, int c2, int c3, int s_om, float* out) {
  const int P = g->n2 * g->n3;
  const int bx = (P / 4 + 255) / 256;
  int chunk = 16;   // blocks of 4 planes: z and its neighbours are reloaded at a chunk's start
  while (chunk > 4 && (int64_t)bx * ((g->n1 + chunk - 1) / chunk) < 4 * g->ctx->sm_count) chunk >>= 1;
  launch_dep(k_tl_sub, dim3(bx, (g->n1 + chunk - 1) / chunk), 256, 0, g->ctx->stream, g->kind, r, zc, g->n1, g->n3, P, c2,
             c3, chunk, (float)g->ucx, (float)g->ucy, (float)g->ucz, g->ctx->scratch, s_om, out);
}

void xf_tl_sub_ay(const xf_grid* g, const float* r, const float* ay, int s_yay, int s_yr, int s_om, float* out) {
  k_tl_sub_ay<<<grid_blocks(g->ctx, g->ncell, 256), 256, 0, g->ctx->stream>>>(r, ay, g->ncell, g->ctx->scratch, s_yay,
                                                                              s_yr, s_om, out);
}
