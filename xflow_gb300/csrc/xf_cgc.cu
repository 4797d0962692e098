// Conjugate gradients of a small or middle grid as one resident kernel.
//
// What bounds such a solve is not memory but the chain of launches: at 64^3
// an iteration of three kernels took 37 us where its arithmetic takes about 6
// (FP64) or 1 (FP32).  Here the whole solve is one cooperative launch, one
// block an SM.  A block owns a brick of the interior and keeps it on the chip
// for the whole solve; a thread owns a column of the brick along i: the
// residual r and the image q = A p of its cells in registers, the direction p
// with its one-cell halo and the iterate (FP64) or the correction e (mixed) in
// shared memory.  The loops over a column run
// over all K cells of the kernel's form, with no branch between them (a
// column that is shorter only leaves out stores), so that their loads from
// shared memory overlap: with a branch a cell they cost 5 us of an iteration.
//
//   p = r + beta p           on the brick and its halo
//   q = A p; q of the brick's faces to memory
//   (p, q), (r, q), (q, q), (r, r)  -> one grid sum -> alpha, beta
//   x += alpha p, r -= alpha q      r on the halo too
//
// One sum an iteration: with alpha = (r, r) / (p, q), the next (r, r) is
// (r, r) - 2 alpha (r, q) + alpha^2 (q, q), so beta and the stop test need no
// second one; (r, r) is measured again each time, so nothing drifts.  Where it
// falls a thousandfold in one step, as it does when CG has come to the end of
// its space, too few bits of that difference are left: the true residual is
// taken there and the direction goes on from it (without it, right-hand sides of
// 1 to 5 eigenvectors took an iteration more in FP64 than with a measured (r, r)).
// Only q
// travels: a block keeps r and p of its halo and forms them as their owner
// does, from the same bits.
//
// The grid sum is the only wait, and its barrier the same step: a block
// stores its partials (a warp a value), adds to a counter and polls it; once
// every block has arrived it adds the partials in block order, so all blocks
// hold the same bits.  2.3 us a step for 152 blocks; polling the partials
// themselves, with no counter, took 5.6 (one level) or 3.3 us (groups of 16),
// because the polls of 152 SMs queue at the few L2 lines that hold them.
// Polls are counted: past the limit a block raises the error flag and leaves,
// and so do the others.
//
// All scalar work (the divisions behind alpha and beta, the tests) is one
// thread's, and the mixed solve's sums travel as float-float: an FP64
// instruction takes 16 cycles of the SM's FP64 pipe, and 16 warps repeating
// the scalars were a third of an iteration.  Float-float across warps and
// blocks too leaves a sum of a million products off by 2e-15 on average and
// 5e-15 at most (2e-15 at most with FP64 from the warps on, for 0.5 us an
// iteration more); alpha and beta are rounded to FP32 right after.
//
// The mixed solve folds e into the FP64 iterate and takes r = b - A x in FP64
// every `every` iterations and whenever the FP32 recursion meets the
// tolerance; the FP64 solve takes its true residual at the end too and starts
// again from it while that misses the tolerance (three times at most).  The
// mixed solve's direction goes on from a replaced residual, but where the true
// (r, r) is twice the recursion's, or misses a tolerance that the recursion
// meets, the recursion was rounding and its direction is worth nothing: it starts
// again too.  (Kept, the direction took smooth right-hand sides at 1e-12 away
// from the solution: 18 of 40 solves between 40 x 36 x 44 and 128 x 64 x 64 ran
// to a cap of 4,000 iterations, now none, 830 on average; right-hand sides of
// 1 to 7 eigenvectors met 1e-9 in none of 15, now in 76 iterations on average.
// Right-hand sides of noise take as many iterations as before.)
//
// r, p, q and the iterate (mixed: e) are kept times a power of two, exact
// wherever nothing under- or overflows, that puts the norms of r between the
// first and the last, rtol |b|, around 1: the sums of squares stay in range, in
// FP32 for any |b| (without it, a mixed solve of |b| = 1e-14 or below ended in
// NaN, and an FP64 one of 1e150).  A mixed solve that started further out than
// that takes a new power, and a new direction, once r is small.
#include <math.h>

#include "xf_control.cuh"
#include "xf_stencil.cuh"

namespace {

constexpr int CC_THREADS = 512;           // columns of a brick at most
constexpr int CC_KMAX = 16;               // cells of a column at most: 128 registers hold r and q of 16 FP64 cells
constexpr int CC_HALO = 4;                // halo loads a thread keeps in flight
constexpr int CC_MAX_BLOCKS = 256;
constexpr uint32_t CC_SPIN_LIMIT = 1u << 22;
constexpr double CC_CANCEL = 1.0 / 1024;   // the recurrence of (r, r) is taken down to this part of it
constexpr double CC_LOW = 0x1p-60;         // mixed: a (r, r) in its scale below which the scale is taken anew
constexpr double CC_DRIFT = 2.0;           // mixed: a true (r, r) beyond this many of the recursion's starts the direction again

struct CoopArgs {
  int n1, n2, n3;
  int bi, bj, bk;          // brick extents (the last brick of an axis may be shorter)
  int mj, mk;              // bricks along j and k
  const uint8_t* kind;
  const double* b;
  double* x;
  void *ex0, *ex1;         // what the bricks exchange, two boxes of T used in turn
  unsigned long long* slots;   // the blocks' partials, two sets of CC_VALUES x CC_MAX_BLOCKS, then the arrival counter (zeros)
  DevScratch* S;
  double cx, cy, cz, rtol;
  int maxit, every;
};

__device__ __forceinline__ void cc_arrive(unsigned long long* counter) {
  asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(counter) : "memory");
}
__device__ __forceinline__ unsigned long long cc_arrived(const unsigned long long* counter) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(counter) : "memory");
  return v;
}

__device__ __forceinline__ void cc_merge(float& hi, float& lo, float bh, float bl) {
  const float s = hi + bh;
  const float bp = s - hi;
  const float err = (hi - (s - bp)) + (bh - bp);
  hi = s;
  lo = lo + (bl + err);
}
__device__ __forceinline__ void cc_merge(double& v, double, double o, double) { v += o; }
// The warps' sums of N accumulators a thread, value v of warp w to
// out[v * 16 + w].  With four values a lane hands half of them over at each of
// the first two steps and ends with one: 6 additions a lane instead of 20.
template <typename T, int N> struct CcBlockSum {
  template <class P>
  static __device__ __forceinline__ void run(const DotAcc<T> (&acc)[N], P* out) {
    static_assert(N == 1 || N == 4, "one value or four");
    constexpr bool F = sizeof(T) == 4;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T hi, lo = T(0);
    auto high = [&](int v) { if constexpr (F) return acc[v].hi; else return acc[v].s; };
    auto low = [&](int v) { if constexpr (F) return acc[v].lo; else return T(0); };
    auto take = [&](T& h, T& l, T gh, T gl, int o) {
      const T bh = __shfl_xor_sync(0xffffffffu, gh, o);
      T bl = T(0);
      if constexpr (F) bl = __shfl_xor_sync(0xffffffffu, gl, o);
      cc_merge(h, l, bh, bl);
    };
    if constexpr (N == 4) {
      const bool up = lane & 16, up2 = lane & 8;   // lanes 16..31 take values 2 and 3, then 8..15 of either the odd one
      T h0 = up ? high(2) : high(0), l0 = up ? low(2) : low(0), h1 = up ? high(3) : high(1), l1 = up ? low(3) : low(1);
      take(h0, l0, up ? high(0) : high(2), up ? low(0) : low(2), 16);
      take(h1, l1, up ? high(1) : high(3), up ? low(1) : low(3), 16);
      hi = up2 ? h1 : h0;
      lo = up2 ? l1 : l0;
      take(hi, lo, up2 ? h0 : h1, up2 ? l0 : l1, 8);
    } else {
      hi = high(0);
      lo = low(0);
      take(hi, lo, hi, lo, 16);
      take(hi, lo, hi, lo, 8);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) take(hi, lo, hi, lo, o);
    if (N == 4 ? (lane & 7) == 0 : lane == 0) {
      P* dst = out + (N == 4 ? lane >> 3 : 0) * 16 + w;
      if constexpr (F) dst->v = make_float2(hi, lo);
      else dst->v = hi;
    }
  }
};

// Sum over the grid of the blocks' sums and a barrier: what the block's
// threads stored before it is visible to every thread after it.  Thread 0
// runs `control(total)` between the two (in every block, on the same bits);
// `fail` is set when a wait ran out.
constexpr int CC_VALUES = 4;   // values of a sum at most
// A partial as it travels: float-float for FP32 accumulators, a double for FP64 ones.
template <typename T> struct CcPart;
template <> struct CcPart<float> {
  float2 v;
  __device__ __forceinline__ void zero() { v = make_float2(0.f, 0.f); }
  __device__ __forceinline__ void merge(const CcPart& o) { cc_merge(v.x, v.y, o.v.x, o.v.y); }
  __device__ __forceinline__ CcPart shuffle(int o) const {
    CcPart s;
    s.v.x = __shfl_xor_sync(0xffffffffu, v.x, o);
    s.v.y = __shfl_xor_sync(0xffffffffu, v.y, o);
    return s;
  }
  __device__ __forceinline__ double value() const { return (double)v.x + (double)v.y; }
};
template <> struct CcPart<double> {
  double v;
  __device__ __forceinline__ void zero() { v = 0.0; }
  __device__ __forceinline__ void merge(const CcPart& o) { v += o.v; }
  __device__ __forceinline__ CcPart shuffle(int o) const {
    CcPart s;
    s.v = __shfl_xor_sync(0xffffffffu, v, o);
    return s;
  }
  __device__ __forceinline__ double value() const { return v; }
};

struct GridSum {
  unsigned long long* slots;
  int nb;
  unsigned step = 0;
  unsigned long long want = 0;
  int* fail;       // shared
  double* total;   // shared, CC_VALUES
  template <typename T, int N, class Control>
  __device__ __forceinline__ void run(const DotAcc<T> (&acc)[N], void* sh, const Control& control) {
    // part v of this block, in lane 0 of warp v (N <= 2: of warp 0, when the block has no more warps)
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    CcPart<T>* shp = reinterpret_cast<CcPart<T>*>(sh);
    CcBlockSum<T, N>::run(acc, shp);   // shp[v * 16 + warp]: the warps' sums
    __syncthreads();
    // two sets: a block is at most one step ahead of another's reads
    unsigned long long* set = slots + (step & 1) * (CC_VALUES * CC_MAX_BLOCKS);
    unsigned long long* counter = slots + 2 * CC_VALUES * CC_MAX_BLOCKS;
    want += (unsigned long long)nb * N;   // one arrival a block and value, over all sums so far
    // a warp a value: its FP64 or float-float chain runs beside the others'
    for (int v = w; v < N; v += nw) {
      CcPart<T> s;
      s.zero();
      if (lane < nw) s = shp[v * 16 + lane];
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) s.merge(s.shuffle(o));   // at most 16 warps
      if (lane == 0) {
        __stcg(set + v * CC_MAX_BLOCKS + blockIdx.x, *reinterpret_cast<unsigned long long*>(&s.v));
        cc_arrive(counter);
      }
    }
    for (int v = w; v < N; v += nw) {
      uint32_t spin = 0;
      bool wait;
      while ((wait = cc_arrived(counter) < want) && ++spin < CC_SPIN_LIMIT) {}
      wait = __any_sync(0xffffffffu, wait);
      CcPart<T> s;
      s.zero();
      for (int b0 = 0; b0 < nb; b0 += 160) {
        unsigned long long x[5];
#pragma unroll
        for (int u = 0; u < 5; u++)
          x[u] = b0 + lane + 32 * u < nb ? __ldcg(set + v * CC_MAX_BLOCKS + b0 + lane + 32 * u) : 0ull;
#pragma unroll
        for (int u = 0; u < 5; u++) s.merge(*reinterpret_cast<CcPart<T>*>(&x[u]));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s.merge(s.shuffle(o));
      if (lane == 0) {
        if (wait) *fail = 1;
        total[v] = s.value();
      }
    }
    step++;
    __syncthreads();
    if (threadIdx.x == 0) {
      double s[N];
#pragma unroll
      for (int v = 0; v < N; v++) s[v] = total[v];
      control(s);
    }
    __syncthreads();
  }
};

// r = b - A x of one cell in FP64, x through L2 (other blocks write it)
__device__ __forceinline__ double cc_residual(const CoopArgs& a, const double* dtab, int c, int kb) {
  const int s1 = a.n2 * a.n3, s2 = a.n3;
  const double* x = a.x;
  double s = ((kb & K_PX) ? a.cx : 0.0) * __ldcg(x + c + s1);
  s = fma((kb & K_MX) ? a.cx : 0.0, __ldcg(x + c - s1), s);
  s = fma((kb & K_PY) ? a.cy : 0.0, __ldcg(x + c + s2), s);
  s = fma((kb & K_MY) ? a.cy : 0.0, __ldcg(x + c - s2), s);
  s = fma((kb & K_PZ) ? a.cz : 0.0, __ldcg(x + c + 1), s);
  s = fma((kb & K_MZ) ? a.cz : 0.0, __ldcg(x + c - 1), s);
  return a.b[c] - fma(dtab[kb & 63], __ldcg(x + c), xneg(s));
}

// The power of two for a solve from (r, r) = v down to `end`: the first norm of r a half of the way above 1, but no more
// than 2^20, for the sake of (q, q).
__device__ __forceinline__ double cc_scale(double v, double end) {
  auto log2 = [](double s) { return (__double2hiint(s) >> 20 & 0x7ff) - 1023; };
  const int up = end > 0.0 ? max(0, min(20, (log2(v) - log2(end)) >> 2)) : 0;
  return __hiloint2double((1023 + max(-500, min(500, up - (log2(v) >> 1)))) << 20, 0);
}

// The solve's scalars, thread 0's (shared memory; every block holds the same).
enum { CC_GO, CC_REPLACE, CC_AGAIN, CC_STOP };
template <typename T>
struct CoopState {
  double rr_prev, rr_next, rr_true, bb, thr, scale;   // rr_prev, rr_next and thr in the scale of r
  T alpha, beta;
  int it, repl, since, starts, fail, next, floor32, cancel;
  long long status;
};

// T: float the mixed solve, double the FP64 one.  K: cells a column.
template <typename T, int K>
__global__ void __launch_bounds__(CC_THREADS, 1) k_cg_coop(const __grid_constant__ CoopArgs a) {
  constexpr bool MIXED = sizeof(T) == 4;
  extern __shared__ double smem[];
  __shared__ double sh[16 * CC_VALUES];
  __shared__ double total[CC_VALUES];
  __shared__ double dtab64[64];
  __shared__ T dtab[64];
  __shared__ CoopState<T> st;
  const int t = threadIdx.x, nt = blockDim.x;
  // this block's brick
  const int q1 = blockIdx.x / (a.mj * a.mk), q2 = (blockIdx.x / a.mk) % a.mj, q3 = blockIdx.x % a.mk;
  const int gi = 1 + q1 * a.bi, gj = 1 + q2 * a.bj, gk = 1 + q3 * a.bk;
  const int ei = min(a.bi, a.n1 - 1 - gi), ej = min(a.bj, a.n2 - 1 - gj), ek = min(a.bk, a.n3 - 1 - gk);
  const int t2 = ek + 2, t1 = (ej + 2) * t2;   // strides of p with its halo: planes -1 .. K of rows -1 .. ej
  const int cols = ej * ek, nh = 2 * ei * (ej + ek), s1 = a.n2 * a.n3;
  // shared memory: [iterate or correction, a row of nt a plane] [p]
  //   [the halo along j and k: (cell of the box, place in p), r]
  const int fbox = (K + 2) * (a.bj + 2) * (a.bk + 2), fhalo = 2 * a.bi * (a.bj + a.bk);
  T* xs = reinterpret_cast<T*>(smem);
  T* p = xs + K * nt;   // nt even
  int2* halo = reinterpret_cast<int2*>(p + ((fbox + 1) & ~1));
  T* rh = reinterpret_cast<T*>(halo + fhalo);
  T* const ex0 = reinterpret_cast<T*>(a.ex0);
  T* const ex1 = reinterpret_cast<T*>(a.ex1);
  DevScratch* S = a.S;

  if (t == 0) {
    st.fail = 0;
    st.it = st.repl = st.since = st.starts = st.floor32 = st.cancel = 0;
    st.status = XF_OK;
    st.alpha = st.beta = T(0);
    st.scale = 0.0;
  }
  for (int q = t; q < 64; q += nt) {
    const T cx = (T)a.cx, cy = (T)a.cy, cz = (T)a.cz;
    dtab[q] = cx * (T)((q & 1) + ((q >> 1) & 1)) + cy * (T)(((q >> 2) & 1) + ((q >> 3) & 1)) +
              cz * (T)(((q >> 4) & 1) + ((q >> 5) & 1));
    dtab64[q] = a.cx * (double)((q & 1) + ((q >> 1) & 1)) + a.cy * (double)(((q >> 2) & 1) + ((q >> 3) & 1)) +
                a.cz * (double)(((q >> 4) & 1) + ((q >> 5) & 1));
  }
  for (int q = t; q < fbox; q += nt) p[q] = T(0);
  for (int q = t; q < K * nt; q += nt) xs[q] = T(0);
  // the halo along j and k; a cell of the ghost layer (place -1) keeps p = 0
  for (int h = t; h < nh; h += nt) {
    int u = h, lj, lk;
    const int per = 2 * (ej + ek), li = u / per;
    u -= li * per;
    if (u < 2 * ek) {
      lj = u < ek ? -1 : ej;
      lk = u < ek ? u : u - ek;
    } else {
      u -= 2 * ek;
      lk = u < ej ? -1 : ek;
      lj = u < ej ? u : u - ej;
    }
    const int j = gj + lj, k = gk + lk;
    const bool in = j >= 1 && j <= a.n2 - 2 && k >= 1 && k <= a.n3 - 2;
    halo[h] = make_int2(((gi + li) * a.n2 + j) * a.n3 + k, in ? (li + 1) * t1 + (lj + 1) * t2 + lk + 1 : -1);
  }
  // this thread's column
  const bool mine = t < cols;
  const int lj = mine ? t / ek : 0, lk = mine ? t - lj * ek : 0;
  const bool edge = lj == 0 || lj == ej - 1 || lk == 0 || lk == ek - 1;
  const int c0 = (gi * a.n2 + gj + lj) * a.n3 + gk + lk;
  T* pc = p + t1 + (lj + 1) * t2 + lk + 1;
  const int eim = mine ? ei : 0;   // cells of this column
  const bool lo_in = mine && gi > 1, hi_in = mine && gi + ei <= a.n1 - 2;
  T rlo = T(0), rhi = T(0);   // r of the halo along i
  uint32_t kinds[(K + 3) / 4];
#pragma unroll
  for (int m = 0; m < K; m += 4) {
    uint32_t w = 0;
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (mine && m + u < ei) w |= (uint32_t)a.kind[c0 + (m + u) * s1] << (8 * u);
    kinds[m / 4] = w;
  }
  auto kind = [&](int m) { return (int)(kinds[m / 4] >> (8 * (m & 3))) & 0xff; };
  __syncthreads();

  GridSum G;
  G.slots = a.slots; G.nb = gridDim.x; G.fail = &st.fail; G.total = total;
  T r[K], q[K];
  const T cx = (T)a.cx, cy = (T)a.cy, cz = (T)a.cz;
  auto met = [&](double v) { return (st.bb > 0 ? sqrt(v / st.bb) : sqrt(v)) <= a.rtol; };
  // whether the scale changes for a residual with (r, r) = v, which is then taken again (thread 0)
  auto rescale = [&](double v) {
    const double end = a.rtol * a.rtol * st.bb, now = cc_scale(v, end);
    if (now == st.scale) return false;
    st.scale = now;
    st.thr = a.rtol * a.rtol * (st.bb * now * now);
    st.next = CC_AGAIN;
    return true;
  };
  // r = b - A x from the box, (r, r) in FP64; by way of a box, so that this
  // rare step is a rolled loop that leaves the iteration its registers
  auto take_residual = [&](auto control) {
    do {
      DotAcc<double> acc[1];
      if (mine) {
        const double scale = st.scale;
#pragma unroll 1
        for (int m = 0; m < ei; m++) {
          const int c = c0 + m * s1, kb = a.kind[c];
          double v = 0.0;
          if (kb >> K_ROW_SHIFT == ROW_ACTUAL) v = cc_residual(a, dtab64, c, kb);
          acc[0].add(v, v);
          ex0[c] = (T)(scale * v);
        }
      }
      G.run(acc, sh, [&](const double (&v)[1]) { control(v[0]); });
    } while (!st.fail && st.next == CC_AGAIN);
#pragma unroll
    for (int m = 0; m < K; m++) r[m] = m < eim ? __ldcg(ex0 + c0 + m * s1) : T(0);
    rlo = lo_in ? __ldcg(ex0 + c0 - s1) : T(0);
    rhi = hi_in ? __ldcg(ex0 + c0 + ei * s1) : T(0);
    for (int h = t; h < nh; h += nt) rh[h] = halo[h].y >= 0 ? __ldcg(ex0 + halo[h].x) : T(0);
  };
  // the iterate of the active cells to the box (mixed: x += e)
  auto put_iterate = [&]() {
    if (!mine) return;
    const double back = 1.0 / st.scale;
#pragma unroll 1
    for (int m = 0; m < ei; m++) {
      const int c = c0 + m * s1;
      if (a.kind[c] >> K_ROW_SHIFT == ROW_ACTUAL) {
        const double v = back * (double)xs[m * nt + t];
        a.x[c] = MIXED ? __ldcg(a.x + c) + v : v;
      }
      if (MIXED) xs[m * nt + t] = T(0);
    }
  };
  {
    DotAcc<double> acc[1];
    if (mine) {
#pragma unroll 1
      for (int m = 0; m < ei; m++) {
        const int c = c0 + m * s1;
        const double bv = a.kind[c] >> K_ROW_SHIFT == ROW_ACTUAL ? a.b[c] : 0.0;
        acc[0].add(bv, bv);
      }
    }
    G.run(acc, sh, [&](const double (&v)[1]) {
      st.bb = v[0];
      rescale(v[0]);
    });
    take_residual([&](double v) {
      st.rr_true = v;
      st.next = CC_GO;
      if (rescale(v)) return;   // another first residual than b
      if (isnan(v)) { st.status = XF_NAN; st.next = CC_STOP; }
      else if (v <= a.rtol * a.rtol * st.bb) st.next = CC_STOP;
    });
    if (!MIXED && mine) {
      const double scale = st.scale;
#pragma unroll 1
      for (int m = 0; m < ei; m++) xs[m * nt + t] = (T)(scale * a.x[c0 + m * s1]);
    }
  }
  // p = r + beta p of the column and of the halo (r of both in place)
  auto direct = [&](T bt, int t1v) {
    T v[K];
#pragma unroll
    for (int m = 0; m < K; m++) v[m] = fma(bt, pc[m * t1v], r[m]);
#pragma unroll
    for (int m = 0; m < K; m++)
      if (m < eim) pc[m * t1v] = v[m];
    if (lo_in) pc[-t1v] = fma(bt, pc[-t1v], rlo);
    if (hi_in) pc[ei * t1v] = fma(bt, pc[ei * t1v], rhi);
  };
  bool fresh = true;   // r is a true residual: p is still to be formed from it
  int side = 1;        // the exchange box of this iteration (0 holds the residual)
  // opaque strides (and the column's length, mixed): what the loop derives from them is not kept in registers across it
  int s1v = s1, t1v = t1, eiv = ei;
  while (!st.fail && st.next != CC_STOP) {
    asm volatile("" : "+r"(s1v), "+r"(t1v));
    if (MIXED) asm volatile("" : "+r"(eiv));   // the tests for a column's last cell: 10.0 -> 9.2 us at 256 x 64 x 64, none in FP64
#pragma unroll
    for (int m = 0; m < (K + 3) / 4; m++) asm volatile("" : "+r"(kinds[m]));
    const T alpha = st.alpha, bt = st.beta;
    if (fresh) {
      direct(bt, t1v);
      for (int h = t; h < nh; h += nt)
        if (halo[h].y >= 0) p[halo[h].y] = fma(bt, p[halo[h].y], rh[h]);
      fresh = false;
    } else {
      // x += alpha p, r -= alpha q, p = r + beta p; the halo's q in flight first
      const T* qx = side ? ex0 : ex1;
      const T qlo = lo_in ? __ldcg(qx + c0 - s1v) : T(0), qhi = hi_in ? __ldcg(qx + c0 + ei * s1v) : T(0);
      int h0 = t;
      do {   // at least once: the first round's loads fly over the update of the column
        int place[CC_HALO];
        T v[CC_HALO];
#pragma unroll
        for (int u = 0; u < CC_HALO; u++) {
          const int2 hc = h0 + u * nt < nh ? halo[h0 + u * nt] : make_int2(0, -1);
          place[u] = hc.y;
          v[u] = hc.y >= 0 ? __ldcg(qx + hc.x) : T(0);
        }
        if (h0 == t) {
#pragma unroll
          for (int m = 0; m < K; m++) {
            const T pm = pc[m * t1v];
            xs[m * nt + t] = fma(alpha, pm, xs[m * nt + t]);
            r[m] = fma(xneg(alpha), q[m], r[m]);
          }
          rlo = fma(xneg(alpha), qlo, rlo);
          rhi = fma(xneg(alpha), qhi, rhi);
          direct(bt, t1v);
        }
#pragma unroll
        for (int u = 0; u < CC_HALO; u++)
          if (place[u] >= 0) {
            const T rn = fma(xneg(alpha), v[u], rh[h0 + u * nt]);
            rh[h0 + u * nt] = rn;
            p[place[u]] = fma(bt, p[place[u]], rn);
          }
        h0 += CC_HALO * nt;
      } while (h0 < nh);
    }
    __syncthreads();
    // q = A p.  p is 0 behind every closed face, so the neighbours need no mask
    DotAcc<T> acc[4];   // (p, q), (r, q), (q, q), (r, r)
    {
      T* qx = side ? ex1 : ex0;
      T below = pc[-t1v], c = pc[0];
#pragma unroll
      for (int m = 0; m < K; m++) {
        const T* pm = pc + m * t1v;
        const T above = pm[t1v];
        const T s = fma(cx, above + below, fma(cy, pm[t2] + pm[-t2], cz * (pm[1] + pm[-1])));
        const int kb = kind(m);
        q[m] = kb >> K_ROW_SHIFT == ROW_ACTUAL ? fma(dtab[kb & 63], c, xneg(s)) : T(0);
        if (m < eim && (edge || m == 0 || m == eiv - 1)) qx[c0 + m * s1v] = q[m];
        acc[0].add(c, q[m]);
        acc[1].add(r[m], q[m]);
        acc[2].add(q[m], q[m]);
        acc[3].add(r[m], r[m]);
        below = c;
        c = above;
      }
    }
    side ^= 1;
    G.run(acc, sh, [&](const double (&v)[4]) {
      const double pq = v[0], rr = v[3];
      st.next = CC_GO;
      st.floor32 = 0;
      if (isnan(pq)) {
        st.status = XF_NAN;
        st.next = CC_STOP;
        return;
      }
      if (!(pq > 0.0)) {
        if (!MIXED || st.since == 0) {
          st.status = XF_BREAKDOWN;
          st.next = CC_STOP;
          return;
        }
        // a small system can run the FP32 recursion to its floor, where (p, q) is
        // rounding: the mixed solve then replaces the residual and starts again
        st.alpha = T(0);
        st.floor32 = 1;
        st.next = CC_REPLACE;
        return;
      }
      st.alpha = (T)(rr / pq);
      const double al = (double)st.alpha;   // the step as it is taken
      const double rn = fma(al, fma(al, v[2], -2.0 * v[1]), rr);
      st.it++;
      st.since++;
      if (isnan(rn)) {
        st.status = XF_NAN;
        st.next = CC_STOP;
        return;
      }
      st.rr_prev = rr;
      st.beta = rn > 0.0 ? (T)(rn / rr) : T(0);
      st.rr_next = rn;
      st.cancel = rn < CC_CANCEL * rr;
      if (rn <= st.thr || st.cancel || st.it >= a.maxit || (MIXED && st.since >= a.every)) st.next = CC_REPLACE;
    });
    if (!st.fail && st.next == CC_REPLACE) {   // take the step; the true residual of the iterate
      const T al = st.alpha;
#pragma unroll
      for (int m = 0; m < K; m++) xs[m * nt + t] = fma(al, pc[m * t1v], xs[m * nt + t]);
      put_iterate();
      const DotAcc<T> none[1];
      G.run(none, sh, [](const double (&)[1]) {});   // every block's part of x is in the box
      take_residual([&](double v) {
        const double w = v * st.scale * st.scale;
        if (MIXED && w < CC_LOW && rescale(v)) {
          st.floor32 = 1;   // no direction is kept
          st.cancel = 0;
          return;
        }
        st.rr_true = v;
        st.since = 0;
        if (MIXED) st.repl++;
        st.next = CC_STOP;
        if (isnan(v)) st.status = XF_NAN;
        else if (met(v)) return;
        else if (st.it >= a.maxit) st.status = XF_MAXIT;
        else if (!MIXED && !st.cancel && ++st.starts >= 3) return;
        else {
          // mixed, and after a cancelled recurrence: the direction goes on from the replaced residual, unless the
          // recursive one has drifted from it: then the solve starts again from the iterate
          const bool on = st.cancel || (MIXED && !st.floor32 && st.rr_next > st.thr && w <= CC_DRIFT * st.rr_next);
          st.beta = on ? (T)(w / st.rr_prev) : T(0);
          st.next = CC_GO;
        }
      });
      fresh = true;
      side = 1;
    }
  }
  // a solve that ended between two replacements still owes the iterate its last steps
  if (st.it > 0) put_iterate();
  if (st.fail) S->iscalars[I_ERR] = 1;
  if (blockIdx.x == 0 && t == 0) {
    S->iscalars[I_STATUS] = st.status;
    S->iscalars[I_IT] = st.it;
    S->iscalars[I_REPL] = st.repl;
    S->scalars[D_RR64] = st.rr_true;
    S->scalars[D_BB] = st.bb;
    S->iscalars[I_DONE] = 1;
  }
}

typedef xf_coop_plan Plan;

// The kernel's form (cells a column, even) for bricks of bi planes.
int column_form(int bi) { return (bi + 1) / 2 * 2; }

// The split of an interior of ni x nj x nk cells into at most `blocks`
// bricks of at most CC_THREADS columns of CC_KMAX cells: the least cells a
// brick (few cells cost as much as half a block's threads), a cell of a
// column's length counted by CC_LENGTH more (the latency of a column's steps;
// long columns leave few warps to hide it), a halo cell by a third (a copy and
// an FMA against the row's work), a block by half a cell (the polls).
constexpr int CC_LENGTH = 48;
constexpr size_t CC_SMEM[2] = {205 * 1024, 215 * 1024};   // dynamic shared memory at most, beside the static part: FP64, mixed
bool make_plan(int ni, int nj, int nk, int blocks, bool mixed, Plan* out) {
  double best = 1e300;
  const int top = blocks < CC_MAX_BLOCKS ? blocks : CC_MAX_BLOCKS;
  for (int a = 1; a <= ni && a <= top; a++)
    for (int b = 1; b <= nj && a * b <= top; b++)
      for (int c = 1; c <= nk && a * b * c <= top; c++) {
        const int bi = (ni + a - 1) / a, bj = (nj + b - 1) / b, bk = (nk + c - 1) / c;
        const int64_t cols = (int64_t)bj * bk;
        if (bi > CC_KMAX || cols > CC_THREADS) continue;
        const int mi = (ni + bi - 1) / bi, mj = (nj + bj - 1) / bj, mk = (nk + bk - 1) / bk;   // no empty brick
        const int threads = cols < 64 ? 64 : (int)((cols + 31) / 32 * 32);
        const int K = column_form(bi);
        const int64_t cells = K * cols, halo = 2 * cols + 2ll * bi * (bj + bk);
        const int64_t box = (int64_t)(K + 2) * (bj + 2) * (bk + 2);
        const size_t smem = (size_t)K * threads * (mixed ? 4 : 8) + ((box + 1) & ~1ll) * (mixed ? 4 : 8) +
                            2ll * bi * (bj + bk) * (8 + (mixed ? 4 : 8));
        if (smem > CC_SMEM[mixed]) continue;
        const double cost = (double)(cells > CC_THREADS / 2 ? cells : CC_THREADS / 2) + CC_LENGTH * K + 0.3 * halo +
                            0.5 * mi * mj * mk;
        if (cost < best) {
          best = cost;
          *out = {1, bi, bj, bk, mi, mj, mk, threads, smem};
        }
      }
  return best < 1e300;
}

template <typename T>
const void* kernel_for(int bi) {
  switch (column_form(bi)) {
    case 2: return (const void*)k_cg_coop<T, 2>;
    case 4: return (const void*)k_cg_coop<T, 4>;
    case 6: return (const void*)k_cg_coop<T, 6>;
    case 8: return (const void*)k_cg_coop<T, 8>;
    case 10: return (const void*)k_cg_coop<T, 10>;
    case 12: return (const void*)k_cg_coop<T, 12>;
    case 14: return (const void*)k_cg_coop<T, 14>;
    default: return (const void*)k_cg_coop<T, CC_KMAX>;
  }
}

}  // namespace

// Uniform Laplace grids without border rows whose interior fits the chip (16
// cells a column, 512 columns a brick, a brick an SM: on 152 SMs 102^3 and
// 128 x 152 x 64 do, 104 x 108 x 104 does not): there it is the faster form
// throughout, and past that the vectors no longer fit, so the kernel chain takes
// over.  Measured on GB300 (us an iteration), chain and resident: 64^3 FP64 39.0
// and 14.6; 75 x 61 x 83 mixed 23.3 and 6.6; 256 x 64 x 64 mixed 24.3 and 9.25;
// 128 x 152 x 64 FP64 60.4 and 40.2, mixed 25.1 and 10.7.  What bounds it now:
// FP64 issue (14 operations a cell) in the first, rows 6.1, update 3.3, grid sum
// with its reductions and scalars 5.0; the grid sum (3.8 to 4.1) in the mixed ones.
// The split depends on the grid's extents alone and stays with the grid.
bool xf_cg_coop_supported(const xf_op* op, bool mixed) {
  xf_grid* g = op->g;
  if (op->kind != XF_OP_LAPLACE || !g->uniform || g->nbrow != 0 || g->n1 < 3 || g->n2 < 3 || g->n3 < 3) return false;
  Plan& p = g->coop[mixed];
  if (p.state == 0 && !make_plan(g->n1 - 2, g->n2 - 2, g->n3 - 2, g->ctx->sm_count, mixed, &p)) p.state = -1;
  return p.state == 1;
}

// The whole solve, for a supported operator.  ex: two boxes of float (mixed)
// or double; slots: xf_cg_coop_slots() doubles.  The state (status,
// iterations, replacements, the true residual and (b, b)) is left in the
// context's scratch.  False where the driver refuses the cooperative launch
// (nothing of the solve has run then): the grid keeps to the kernel chain from
// there on.
size_t xf_cg_coop_slots() { return 2 * CC_VALUES * CC_MAX_BLOCKS + 1; }

bool xf_cg_coop_launch(const xf_op* op, double* x, const double* b, void* const ex[2], double* slots, bool mixed, double rtol,
                       int maxit, int every) {
  xf_grid* g = op->g;
  xf_ctx* ctx = g->ctx;
  Plan& p = g->coop[mixed];
  CoopArgs a;
  a.n1 = g->n1; a.n2 = g->n2; a.n3 = g->n3;
  a.bi = p.bi; a.bj = p.bj; a.bk = p.bk; a.mj = p.mj; a.mk = p.mk;
  a.kind = g->kind; a.b = b; a.x = x; a.ex0 = ex[0]; a.ex1 = ex[1]; a.slots = reinterpret_cast<unsigned long long*>(slots); a.S = ctx->scratch;
  a.cx = g->ucx; a.cy = g->ucy; a.cz = g->ucz; a.rtol = rtol; a.maxit = maxit; a.every = every;
  const void* f = mixed ? kernel_for<float>(p.bi) : kernel_for<double>(p.bi);
  void* args[] = {&a};
  // The attribute is the kernel's, whatever context sets it, and plans of different sizes share a kernel: always
  // the same value, so that no thread lowers it under another's launch.
  cudaError_t e = cudaMemsetAsync(slots, 0, xf_cg_coop_slots() * sizeof(double), ctx->stream);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CC_SMEM[mixed]);
  if (e == cudaSuccess)
    e = cudaLaunchCooperativeKernel(f, dim3(p.mi * p.mj * p.mk), dim3(p.threads), args, p.smem, ctx->stream);
  if (e == cudaSuccess) return true;
  cudaGetLastError();
  p.state = -1;
  return false;
}
