// State and control of the device-driven flexible CG of the learned two-level
// preconditioner (xf_unet.cu).  Its scalar decisions run in the last block of
// the reduction that feeds them: as one-thread launches of their own (six an
// iteration, 16 us at 256^3 with the gaps around them) they stood in the
// chain of every iteration.
#pragma once
#include "xf_control.cuh"

constexpr int FCG_STRIKES = 3;   // (z, r) <= 0 this often: the network is off for the rest of the solve

// scalar slots: 0..7 (z, A p_j); 8 (y, A y), 9 (y, r) of the two-level preconditioner; 10 (z, r); 11 (r, r);
// 12 (p, r); 13 omega; 14/15 matvec dots
enum { FS_YAY = 8, FS_YR = 9, FS_ZR = 10, FS_RR = 11, FS_PR = 12, FS_OM = 13, FS_PQ = 14 };

struct TlCtl {
  double bb, thr, rr_true, rr_prev_true, rr, rr_start, alpha;
  double pq_win[9];
  float coef[8];
  int use_coef[8];
  int win_off[8];   // window dot j skipped (j >= nwin)
  int it, it_start, maxit, every, repl, prev_cycle, fallbacks, precond_on, head, nwin, done, status, brk, cycle_ran;
  int passes, steps, steps_seen;   // the loop guard
  long long launches;
};
struct TlParams {
  double rtol2;
  int maxit, every;
  // kernels per segment, for the launch count
  int n_init, n_ref, n_iter, n_on, n_off, n_fb;
};
enum { TL_ON = 0, TL_OFF = 1, TL_SKIP = 2 };   // a block's switch: with the network, without, not this pass
struct TlHandles {
  cudaGraphConditionalHandle main, ref, blk[9], fb[9];
};
// What a control step of the block with direction slot hd needs (ctl null: no step).
struct TlStep {
  TlCtl* ctl;
  const TlParams* prm;
  TlHandles h;
  int hd, m;
};

// The iteration of block hd is next.
__device__ __forceinline__ void tl_next(TlCtl* c, const TlParams* p, const TlHandles& h, int hd, int m) {
  c->it++;
  for (int j = 0; j < m; j++) c->win_off[j] = j >= c->nwin;
  c->launches += p->n_iter + (c->precond_on ? p->n_on : p->n_off);
  cudaGraphSetConditional(h.blk[hd], c->precond_on ? TL_ON : TL_OFF);
}

// The window coefficients -(z, q_j) / (p_j, q_j); the last one is the fused
// direction pass's beta (0: no term).
__device__ __forceinline__ void tl_coef(DevScratch* S, TlCtl* c, int hd, int m) {
  for (int j = 0; j < m; j++) {
    const int sl = (hd + m - j) % (m + 1);
    const bool use = j < c->nwin && c->pq_win[sl] > 0;
    c->use_coef[j] = use;
    c->coef[j] = use ? (float)(-S->scalars[j] / c->pq_win[sl]) : 0.f;
  }
  S->scalars[D_BETA] = (double)c->coef[m - 1];
}

// (z, r) is known: no descent direction, use r this time (the fallback block
// follows), and from the third time on for good.
__device__ __forceinline__ void tl_z(DevScratch* S, const TlStep& t) {
  TlCtl* c = t.ctl;
  const bool bad = !(S->scalars[FS_ZR] > 0);
  if (bad) {
    if (++c->fallbacks >= FCG_STRIKES) c->precond_on = 0;
    c->launches += t.prm->n_fb;
  }
  cudaGraphSetConditional(t.h.fb[t.hd], bad ? 1u : 0u);
  if (t.m == 1) tl_coef(S, c, t.hd, 1);   // its one dot came with (z, r)
}

// (p, q) is known.  (p, r) = (z, r): r is orthogonal to every direction of the
// window after its line search, up to FP32's rounding and what a refresh of r
// changes.  That makes alpha's error up to 3e-5 late in a cycle (1e-6 with (p, r)
// measured, which costs the direction pass a stream more); a step's part of the
// decrease loses its square, and the iterations are as many.
__device__ __forceinline__ void tl_alpha(DevScratch* S, const TlStep& t) {
  TlCtl* c = t.ctl;
  const double pr = S->scalars[FS_ZR], pq = S->scalars[FS_PQ];
  if (!(pq > 0)) {
    c->status = isnan(pq) ? XF_NAN : XF_BREAKDOWN;
    c->brk = 1;
    c->alpha = 0;   // e has taken the step before
    return;
  }
  c->alpha = pr / pq;
  c->pq_win[t.hd] = pq;
  c->head = (t.hd + 1) % (t.m + 1);
  if (c->nwin < t.m) c->nwin++;
}

// (r, r) is known (or the iteration broke down): the cycle-end test, and the
// next block or the refresh.
__device__ __forceinline__ void tl_rr(DevScratch* S, const TlStep& t) {
  TlCtl* c = t.ctl;
  c->steps++;
  bool end = c->brk != 0;
  if (!end) {
    const double rr = S->scalars[FS_RR];
    c->rr = rr;
    end = isnan(rr) || rr <= c->thr || rr <= 1e-6 * c->rr_start || c->it - c->it_start >= c->every ||
          c->it >= c->maxit;
  }
  if (end) {
    c->cycle_ran = 1;
    c->repl++;
    c->prev_cycle = c->it - c->it_start;
    cudaGraphSetConditional(t.h.ref, 1u);
    for (int k = t.hd + 1; k <= t.m; k++) cudaGraphSetConditional(t.h.blk[k], TL_SKIP);
  } else {
    tl_next(c, t.prm, t.h, t.hd < t.m ? t.hd + 1 : 0, t.m);
  }
}
