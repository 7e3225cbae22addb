// tl_persist.cu -- the persistent CG kernel of meshes that fit on chip: one cooperative launch
// runs many iterations of the CG loop (tea_solve.f90:341-369) with the whole problem held in
// shared memory and registers.
//
// Each CTA (one per SM) owns a tile of the mesh.  p with its one-cell halo, the scaled face
// coefficients and Di live in shared memory, r, w (and u, when the registers allow) in the
// registers of the thread that owns the cell: a thread owns one column and every ry-th row of its
// tile.  Per iteration:
//   phase A  p_n = src + beta p_{n-1} on the tile and its halo (from the neighbours' src at the
//            tile's rim), w = A p_n, p.w; grid sum -> alpha;
//   phase B  u += alpha p_n, r -= alpha w (z = Mi r with jac_diag), r.z, the rim's src sent to the
//            neighbour tiles; grid sum -> beta, error, the EXIT / switch tests.
// HBM and L2 see the rims and the partial sums only; the fields are read when a launch starts and
// written when it ends.
//
// What bounds it: below about 300^2 cells the latency of the two grid sums and of the FP64
// operations in a row (61 cycles each for one warp), above that the FP64 pipe.  So
// - a grid sum is one hop: the first warp stores the CTA's partial, tagged with the sum's number,
//   into every CTA's inbox, and five warps poll the CTA's own inbox, a word a lane, until all
//   partials have come (3300 cycles on 152 CTAs; 4400 when one warp polls five words a lane).  One
//   table of partials that all CTAs poll takes 7000 cycles, since every store then waits behind the
//   polls of its line; an arrival counter with a generation word is two dependent atomics and a
//   second read.  A mesh of up to about a thousand cells takes a single CTA, which has nobody to wait
//   for (4.4 us an iteration at 22^2, against 5.9 on the grid at 32^2);
// - the rim goes the same way: its owner stores each value with the sum's number into the
//   neighbour tile's box, and the neighbour's threads poll for it while the first warp waits for
//   the sum.  Publishing it through the field needs a fence (1900 cycles) before the sum;
// - sums across threads are integers relative to the largest exponent, not FP64 additions: an FP64
//   instruction holds a sub-partition's pipe for 64 cycles however few lanes need it.
//
// Time per CG iteration, the solve's set-up included, against the form before it (up to 640K cells
// one persistent kernel with the fields in memory and two barriers an iteration, above the batched
// sweeps of tl_fused.cu in CUDA graphs): 64^2 5.6 against 12 us, 128^2 5.5 / 13.8, 256^2 6.5 / 14.5,
// 512^2 9.3 / 27.6, 700^2 13.3 / 34.8; meshes from about 800K cells, to about 1400^2, take
// k_persistent_cg_wide.  The FP64 pipe's share is 1.1 us at 256^2 and 8 us at 700^2.
#include "tl_mixed.cuh"

namespace tl {

namespace {

constexpr int PTHREADS = 512;  // threads per CTA
constexpr int PT = PTHREADS - 32;  // those that own cells: all but the first warp, which exchanges the sums
constexpr int PW = PT / 32;    // their warps
constexpr int PH = 2;          // halo cells per thread at most
constexpr int POLLW = 5;       // warps that poll the inbox at most
constexpr int SLOTS = 32 * POLLW;            // words of an inbox
constexpr int PERSIST_MAX_CTAS = SLOTS - 1;  // one is left for the test of the bounded wait
constexpr size_t PERSIST_SMEM_MAX = 225 * 1024;
// polls before a wait gives up (some tenths of a second: a poll takes an L2 round trip)
constexpr unsigned PERSIST_POLL_LIMIT = 1u << 21;

struct PersistArgs {
  LoopArgs a;
  PersistPlan pl;
  int max_run;
  unsigned epoch;   // number of the launch's first grid sum
  ulonglong2* box;  // by parity of the sum's number, an inbox per CTA; then the tiles' halo boxes
  LoopState* st_host;
  unsigned* err;    // set when a wait ran out in any CTA: the results are void
  int extra;        // partials waited for beyond the grid's (test of the bounded wait)
  int lame;         // this CTA gives its rims up at once (test of the report; -1: none)
};

// Sums across lanes: a value as an integer multiple of 2^(e - 1075 - FSH), e the largest biased
// exponent among the values, rounded to nearest; the integers are added exactly, so the result does
// not depend on an order.  A value's rounding error is at most 2^-54 of the warp's largest, and those of
// its 32 values add up; an FP64 tree rounds by 2^-53 of the partial sum at each of its levels.  Against
// sums in 64 bits a 256^2 run's error is 2.3e-15 (2.2e-15 with the tree), 777 x 1013's 1.4e-14 (1.3e-14).
constexpr int FSH = 1;  // 53 + FSH bits for the largest value: a CTA's 480 fit 63 bits
struct Fix {
  long long q;
  unsigned e;  // 0x7ff: an infinity or NaN among the values; q is then the infinity's sign, 0 for NaN
};
using emu::expo;
// the sum over the warp of q, as limbs of 21 bits through redux.sync: of single values (|q| <= 2^54), or of
// at most 16 lanes' sums of a warp (|q| <= 2^59, together below 2^63)
__device__ __forceinline__ long long warp_add(long long q) {
  const int l0 = __reduce_add_sync(0xffffffffu, (int)(q & 0x1fffff));
  const int l1 = __reduce_add_sync(0xffffffffu, (int)((q >> 21) & 0x1fffff));
  const int l2 = __reduce_add_sync(0xffffffffu, (int)(q >> 42));
  return (long long)l0 + ((long long)l1 << 21) + ((long long)l2 << 42);
}
// the sum when a lane holds an infinity or NaN, as IEEE addition gives it
__device__ __noinline__ Fix warp_nonfinite(int sign, bool nan) {
  const bool p = __any_sync(0xffffffffu, sign > 0), m = __any_sync(0xffffffffu, sign < 0);
  return Fix{__any_sync(0xffffffffu, nan) || p == m ? 0ll : (p ? 1ll : -1ll), 0x7ffu};
}
__device__ __forceinline__ Fix warp_fix(double v) {
  const uint64_t b = emu::bits(v);
  const unsigned ev = max((unsigned)(b >> 52) & 0x7ffu, 1u);
  const unsigned e = __reduce_max_sync(0xffffffffu, ev);
  if (e == 0x7ffu) {
    const bool nan = (b & ~emu::SIGN) > emu::INF, inf = (b & ~emu::SIGN) == emu::INF;
    return warp_nonfinite(inf ? ((b & emu::SIGN) ? -1 : 1) : 0, nan);
  }
  const uint64_t m = (b & emu::FRAC) | ((b << 1 >> 53) ? emu::HIDDEN : 0ull);
  const long long i = (long long)((((m << (FSH + 1)) >> min(e - ev, 63u)) + 1ull) >> 1);
  return Fix{warp_add((b & emu::SIGN) ? -i : i), e};
}
// the sum over the warp of sums, one a lane, of at most 16 lanes or of single values
__device__ __forceinline__ Fix warp_fix(const Fix& f) {
  const unsigned e = __reduce_max_sync(0xffffffffu, f.e);
  if (e == 0x7ffu) {
    const bool odd = f.e == 0x7ffu;
    return warp_nonfinite(odd ? (f.q > 0) - (f.q < 0) : 0, odd && f.q == 0);
  }
  const unsigned d = min(e - f.e, 63u);
  return Fix{warp_add((f.q + (d ? 1ll << (d - 1) : 0ll)) >> d), e};
}
__device__ __noinline__ double scale_slowly(double t, int k) { return ldexp(t, k); }
__device__ __forceinline__ double fix_value(const Fix& f) {
  if (f.e == 0x7ffu) return emu::from_bits(f.q ? (f.q < 0 ? emu::SIGN : 0ull) | emu::INF : emu::QNAN);
  const double t = (double)f.q;
  const int k = (int)f.e - 1075 - FSH, et = (int)expo(t);
  if (et == 0) return t;  // zero
  if (et + k >= 1 && et + k < 0x7ff) return emu::from_bits(emu::bits(t) + ((uint64_t)(long long)k << 52));
  return scale_slowly(t, k);
}

// A value in a box: its halves, each beside the sum's number, so that either word shows by itself
// that it belongs to this sum.
__device__ __forceinline__ void box_put(ulonglong2* s, double v, unsigned epoch) {
  const unsigned long long b = emu::bits(v);
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(s), "l"((b & 0xffffffff00000000ull) | epoch),
               "l"((b << 32) | epoch)
               : "memory");
}
__device__ __forceinline__ ulonglong2 box_get(const ulonglong2* s) {
  ulonglong2 w;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w.x), "=l"(w.y) : "l"(s) : "memory");
  return w;
}
__device__ __forceinline__ bool box_is(const ulonglong2& w, unsigned epoch) {
  return (unsigned)w.x == epoch && (unsigned)w.y == epoch;
}
__device__ __forceinline__ double box_value(const ulonglong2& w) {
  return emu::from_bits((w.x & 0xffffffff00000000ull) | (w.y >> 32));
}
__device__ __forceinline__ bool finite_bits(double v) { return expo(v) != 0x7ffu; }
template <int ID, int N>
__device__ __forceinline__ void bar_sync() {
  asm volatile("barrier.sync %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
template <int ID, int N>
__device__ __forceinline__ void bar_arrive() {
  asm volatile("barrier.arrive %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("barrier.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
  asm volatile("barrier.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// x, in a way that keeps the compiler from computing what follows from it once for all iterations:
// the addresses of a thread's cells would take as many registers as the cells themselves
__device__ __forceinline__ int fresh(int x) {
  asm volatile("" : "+r"(x));
  return x;
}

// What the exchange of a sum needs, in shared memory.
struct Exchange {
  Fix part[PW];        // the owning warps' sums
  Fix inbox[POLLW];    // the polling warps' sums
  int fail;            // a wait ran out
};

// First warp: the owning warps' sums added up over the grid; meanwhile() runs while the partials
// are on their way.  in: the inboxes of this parity.  Not inlined, so that both sums of an
// iteration run the same instructions.
__device__ __noinline__ double exchange_sum(Exchange* x, ulonglong2* in, unsigned epoch, int ctas, int extra, double rro,
                                            double* inv_rro) {
  const int lane = threadIdx.x & 31;
  bar_sync<1, PTHREADS>();
  Fix p{0, 1u};
  if (lane < PW) p = x->part[lane];
  double total = fix_value(warp_fix(p));
  if (ctas > 1) {
#pragma unroll
    for (int q = 0; q < POLLW; ++q)
      if (lane + 32 * q < ctas) box_put(in + (size_t)(lane + 32 * q) * SLOTS + blockIdx.x, total, epoch);
    if (inv_rro) *inv_rro = 1.0 / rro;  // while the partials are on their way
    const int nq = (ctas + extra + 31) / 32;
    bar_sync(3, 32 * (nq + 1));
    p = Fix{0, 1u};
    if (lane < nq) p = x->inbox[lane];
    total = fix_value(warp_fix(p));
  } else if (inv_rro) {
    *inv_rro = 1.0 / rro;
  }
  return total;
}

// The threads but the first warp's own the cells.  The first warp exchanges the sums and runs the
// loop's scalar steps, so that in the wait for beta the owners update u and fetch the halo.  The
// warps meet at
//   1  the owning warps' sums are in shared memory (owners arrive, the first warp waits);
//   2  owners only: p is complete in shared memory;
//   3  the words of the inbox are added up (the polling warps arrive, the first warp waits);
//   0  the sum's outcome is in shared memory (all).
// The loop's scalars in the first warp (tea_solve.f90:341-369), and their epilogues.
struct CgScalars {
  double rro, inv_rro = 0.0, pw, alpha, beta, rrn;
  uint64_t goal2;
  bool check_switch, error_due = false;
  int max_iters;

  __device__ __forceinline__ explicit CgScalars(const LoopState& S)
      : rro(S.rro), pw(S.pw), alpha(S.alpha), beta(S.beta), rrn(S.rrn), check_switch(S.check_switch != 0),
        max_iters(S.max_iters) {
    const double goal = S.eps * S.initial_residual;
    goal2 = emu::bits(goal > 1e-140 ? goal * goal * (1.0 + 1e-12) : INFINITY);
  }
  // pw is known: alpha
  __device__ __forceinline__ void after_pw(LoopState* S, int n, double* sh_alpha, int* sh_status, double* hist) {
    alpha = rro / pw;
    if ((threadIdx.x & 31) == 0) {
      *sh_alpha = alpha;
      if (!finite_bits(alpha)) {
        S->status = EXIT_BREAKDOWN;
        S->n_exit = n;
        *sh_status = EXIT_BREAKDOWN;
      }
      if (blockIdx.x == 0) hist[n] = alpha;
    }
  }
  // rrn is known: beta, the error, the loop's tests
  __device__ __forceinline__ void after_rrn(LoopState* S, int n, double* sh_beta, int* sh_status, double* hist) {
    const double b = beta = emu::quotient(rrn, rro, inv_rro);
    // without the square root when the outcome is plain: the error is far enough above the goal
    // (goal2: its square with a margin; non-negative doubles order as their bits) and nothing
    // else can stop the loop.  The error itself is then left to the launch's end.
    error_due = !check_switch && n < max_iters && (emu::bits(rrn) & ~emu::SIGN) > goal2 && expo(rrn) < 2000u;
    if ((threadIdx.x & 31) == 0) {
      *sh_beta = b;
      if (!error_due) {
        S->n = n;
        loop_finish_iteration(S, rrn);
        *sh_status = S->status;
      }
      if (blockIdx.x == 0) hist[n] = b;
    }
    rro = rrn;
  }
  // one thread: the state after `done` iterations, the next being n
  __device__ __forceinline__ void store(LoopState& S, int n, int done) const {
    S.u_pending = 0;
    S.pw = pw;
    S.alpha = alpha;
    S.cg_calc_steps += done;
    if (done > 0) {
      S.rrn = rrn;
      S.beta = beta;
      S.rro = rro;
      S.p_pending = 1;
      if (error_due) {
        S.n = n;
        S.error = S.old_error = sqrt(fabs(rrn));
      }
    }
  }
};

// M: cells a thread may own.  p of the owned cells stays in registers too up to 4, u and Mi up to 6 (they
// are in the fields otherwise, u updated in the wait for beta).
template <int M, bool DIAG>
__global__ void __launch_bounds__(PTHREADS, 1) k_persistent_cg(PersistArgs g) {
  constexpr bool PREG = M <= 4, UREG = M <= 6;
  constexpr int MG = M < 6 ? M : 6;  // rows whose loads from the fields are in flight together
  // Where the FP64 pipe bounds the iteration the products Di p and Mi r run on the integer pipes
  // (dmul_int, the same bits): 14.8 -> 14.2 us at 700^2; 7.2 -> 7.3 at 256^2, one cell a thread.
  constexpr bool EMU = M > 2;
  __shared__ LoopState S;
  __shared__ Exchange X;
  __shared__ double sh_alpha, sh_beta;
  __shared__ int sh_status;
  extern __shared__ __align__(16) double psm[];
  const Layout L = g.a.L;
  const Fields& f = g.a.f;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const bool owner = wid != 0;
  const int to = t - 32;  // number of the owner
  const int ctas = gridDim.x;
  if (t == 0) {
    S = *g.a.rd.st;
    sh_status = S.status;
    sh_beta = S.beta;
    X.fail = 0;
  }
  __syncthreads();
  if (sh_status != RUN) {  // in every CTA
    if (blockIdx.x == 0 && t == 0) *g.st_host = S;
    return;
  }

  const int bx = blockIdx.x % g.pl.gx, by = blockIdx.x / g.pl.gx;
  const int j0 = bx * g.pl.tw, k0 = by * g.pl.th;  // first cell of the tile, from 0
  const int tw = min(g.pl.tw, L.nx - j0), th = min(g.pl.th, L.ny - k0);
  const int P = g.pl.tw + 2, ry = g.pl.ry;
  const int asz = (g.pl.th + 2) * P;
  double* const sp = psm;
  double* const scx = psm + asz;
  double* const scy = psm + 2 * asz;
  double* const sdi = psm + 3 * asz;

  // the thread's column and first row; cells i = 0 .. mine-1 at rows ty + i ry
  const int tx = owner ? to % g.pl.tw : 0, ty = owner ? to / g.pl.tw : 0;
  const int mine = (owner && tx < tw && ty < ry && ty < th) ? (th - 1 - ty) / ry + 1 : 0;
  const int o0 = (ty + 1) * P + tx + 1;
  const int c0 = (int)L.at(j0 + tx + 1, k0 + ty + 1);
  const int ostep = ry * P, cstep = ry * L.ld;
  const int i_first = ty == 0 ? 0 : -1, i_last = (mine > 0 && (th - 1 - ty) % ry == 0) ? mine - 1 : -1;
  const bool at_l = tx == 0 && j0 == 0, at_r = tx == tw - 1 && j0 + tw == L.nx;  // at the domain's side
  const int i_b = k0 == 0 ? i_first : -1, i_t = k0 + th == L.ny ? i_last : -1;

  // A tile's halo box: its left column, right column (th each), bottom row, top row (tw each).
  const int hbox = 2 * (g.pl.th + g.pl.tw);
  ulonglong2* const halo = g.box + (size_t)2 * gridDim.x * SLOTS;
  // halo cells this thread fetches (those beside other tiles): p there, and the next source
  int ho[PH], hh[PH];
  double hp[PH], hs[PH];
  double* const src = DIAG ? f.z : f.r;
  int n = S.n;
  const double* const pold = (n & 1) ? f.p : f.p2;
  bool upd = S.p_pending != 0;
#pragma unroll
  for (int q = 0; q < PH; ++q) {
    const int h = to + q * PT;
    ho[q] = -1;
    hh[q] = 0;
    hp[q] = hs[q] = 0.0;
    int x = -1, y = h;
    bool is = j0 > 0 && y < th;
    if (h >= g.pl.th) x = tw, y = h - g.pl.th, is = j0 + tw < L.nx && y < th;
    if (h >= 2 * g.pl.th) x = h - 2 * g.pl.th, y = -1, is = k0 > 0 && x < tw;
    if (h >= 2 * g.pl.th + g.pl.tw) x = h - 2 * g.pl.th - g.pl.tw, y = th, is = k0 + th < L.ny && x < tw;
    if (is && owner && h < hbox) {
      ho[q] = (y + 1) * P + x + 1;
      hh[q] = (int)blockIdx.x * hbox + h;
      const int c = (int)L.at(j0 + x + 1, k0 + y + 1);
      hp[q] = pold[c];
      if (upd) hs[q] = src[c];
    }
  }
  // where the thread's rim cells go: the neighbour tiles' boxes (-1: no such neighbour)
  const int to_l = (tx == 0 && j0 > 0) ? ((int)blockIdx.x - 1) * hbox + g.pl.th + ty : -1;
  const int to_r = (tx == tw - 1 && j0 + tw < L.nx) ? ((int)blockIdx.x + 1) * hbox + ty : -1;
  const int rim_b = k0 > 0 ? i_first : -1, rim_t = k0 + th < L.ny ? i_last : -1;
  const int to_b = ((int)blockIdx.x - g.pl.gx) * hbox + 2 * g.pl.th + g.pl.tw + tx;
  const int to_t = ((int)blockIdx.x + g.pl.gx) * hbox + 2 * g.pl.th + tx;

  double r[M], w[M], u[UREG ? M : 1], mi[UREG && DIAG ? M : 1], pr[PREG ? M : 1];
  // (w holds the source z of the next p between phases B and A with DIAG)
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const int o = o0 + i * ostep, c = c0 + i * cstep;
    r[i] = w[i] = 0.0;
    if (UREG) u[i] = 0.0;
    if (UREG && DIAG) mi[i] = 0.0;
    if (PREG) pr[i] = 0.0;
    if (i < mine) {
      r[i] = f.r[c];
      if (DIAG) w[i] = f.z[c];
      if (UREG) u[i] = f.u[c];
      if (UREG && DIAG) mi[i] = f.mi[c];
      if (PREG)
        pr[i] = pold[c];
      else
        sp[o] = pold[c];
      sdi[o] = f.di[c];
      scx[o] = f.cx[c];
      scy[o] = f.cy[c];
      if (tx == tw - 1) scx[o + 1] = f.cx[c + 1];
      if (i == i_last) scy[o + P] = f.cy[c + L.ld];
    }
  }

  CgScalars C(S);  // in the first warp
  unsigned epoch = g.epoch;
  __syncthreads();

  // owners: the warp's sum of v; then the polling warps' share of the grid's
  auto give = [&](double v) {
    const Fix s = warp_fix(v);
    if (lane == 0) X.part[wid - 1] = s;
    bar_arrive<1, PTHREADS>();
  };
  const int nwait = ctas > 1 ? ctas + g.extra : 0, nq = (nwait + 31) / 32;
  auto poll = [&] {
    if (wid > nq) return;
    const int slot = (wid - 1) * 32 + lane;
    const ulonglong2* in = g.box + ((size_t)(epoch & 1u) * ctas + blockIdx.x) * SLOTS + slot;
    ulonglong2 x = make_ulonglong2(0ull, 0ull);
    bool here = slot >= nwait;
    for (unsigned tries = 0; !here && tries < PERSIST_POLL_LIMIT; ++tries) {
      x = box_get(in);
      here = box_is(x, epoch);
    }
    if (!here) X.fail = 1;
    __syncwarp();
    const Fix q = warp_fix(slot < nwait ? box_value(x) : 0.0);
    if (lane == 0) X.inbox[wid - 1] = q;
    bar_arrive(3, 32 * (nq + 1));
  };
  auto inboxes = [&] { return g.box + (size_t)(epoch & 1u) * ctas * SLOTS; };

  int done = 0;
  bool updated = false;  // phase B of the last iteration ran
  for (; done < g.max_run; ++done) {
    // ---- phase A: p_n on the tile and its halo (off the domain the mirror value), w = A p_n, p.w ----
    updated = false;
    if (owner) {
      const double beta = sh_beta;
      // the even iterations' p is what the loop leaves in the field p
      double* const pf = (n & 1) ? nullptr : f.p;
      int o = fresh(o0), c = fresh(c0);
#pragma unroll
      for (int i = 0; i < M; ++i, o += ostep, c += cstep) {
        if (i < mine) {
          double p = PREG ? pr[i] : sp[o];
          if (upd) p = fma(beta, p, DIAG ? w[i] : r[i]);
          if (PREG) pr[i] = p;
          sp[o] = p;
          if (pf) pf[c] = p;
          if (at_l) sp[o - 1] = p;
          if (at_r) sp[o + 1] = p;
          if (i == i_b) sp[o - P] = p;
          if (i == i_t) sp[o + P] = p;
        }
      }
#pragma unroll
      for (int q = 0; q < PH; ++q)
        if (ho[q] >= 0) {
          if (upd) hp[q] = fma(beta, hp[q], hs[q]);
          sp[ho[q]] = hp[q];
        }
      bar_sync<2, PT>();
      double acc = 0.0;
      o = fresh(o0);
#pragma unroll
      for (int i0 = 0; i0 < M; i0 += MG) {
        if (i0 >= mine) break;
#pragma unroll
        for (int j = 0; j < MG; ++j, o += ostep) {
          const int i = i0 + j;
          if (i < M && i < mine) {
            const double pc = PREG ? pr[i] : sp[o];
            double wv = EMU ? dmul_int(sdi[o], pc) : sdi[o] * pc;
            wv = fma(-scy[o + P], sp[o + P], wv);
            wv = fma(-scy[o], sp[o - P], wv);
            wv = fma(-scx[o + 1], sp[o + 1], wv);
            wv = fma(-scx[o], sp[o - 1], wv);
            w[i] = wv;
            acc = fma(wv, pc, acc);
          }
        }
      }
      give(acc);
      poll();
    } else {
      C.pw = exchange_sum(&X, inboxes(), epoch, ctas, g.extra, C.rro, &C.inv_rro);
      C.after_pw(&S, n, &sh_alpha, &sh_status, g.a.rd.hist_a);
    }
    ++epoch;
    __syncthreads();
    if (X.fail || sh_status != RUN) break;
    // ---- phase B: r -= alpha w, z = Mi r, r.z; the rim to the neighbours; u += alpha p_n ----
    if (owner) {
      const double alpha = sh_alpha;
      double acc = 0.0;
      int c = fresh(c0), l = fresh(to_l), e = fresh(to_r);
#pragma unroll
      for (int i0 = 0; i0 < M; i0 += MG) {
        if (i0 >= mine) break;
        double mg[DIAG && !UREG ? MG : 1];
        if (DIAG && !UREG) {
#pragma unroll
          for (int j = 0; j < MG; ++j)
            if (i0 + j < mine) mg[j] = __ldg(f.mi + c + j * cstep);
          c += MG * cstep;
        }
#pragma unroll
        for (int j = 0; j < MG; ++j, l += ry, e += ry) {
          const int i = i0 + j;
          if (i < M && i < mine) {
            const double rv = fma(-alpha, w[i], r[i]);
            r[i] = rv;
            double zv = rv;
            if (DIAG) {
              const double mm = UREG ? mi[UREG ? i : 0] : mg[UREG ? 0 : j];
              zv = EMU ? dmul_int(mm, rv) : mm * rv;
              w[i] = zv;
            }
            if (to_l >= 0) box_put(halo + l, zv, epoch);
            if (to_r >= 0) box_put(halo + e, zv, epoch);
            if (i == rim_b) box_put(halo + to_b, zv, epoch);
            if (i == rim_t) box_put(halo + to_t, zv, epoch);
            acc = fma(rv, zv, acc);
          }
        }
      }
      give(acc);
      poll();
      int o = fresh(o0);
      c = fresh(c0);
#pragma unroll
      for (int i0 = 0; i0 < M; i0 += MG) {
        if (i0 >= mine) break;
        double ug[UREG ? 1 : MG];
        if (!UREG) {
#pragma unroll
          for (int j = 0; j < MG; ++j)
            if (i0 + j < mine) ug[j] = f.u[c + j * cstep];
        }
#pragma unroll
        for (int j = 0; j < MG; ++j, o += ostep) {
          const int i = i0 + j;
          if (i < M && i < mine) {
            const double pc = PREG ? pr[i] : sp[o];
            if (UREG)
              u[UREG ? i : 0] = fma(alpha, pc, u[UREG ? i : 0]);
            else
              f.u[c + j * cstep] = fma(alpha, pc, ug[UREG ? 0 : j]);
          }
        }
        c += MG * cstep;
      }
      bool got = false;
      const unsigned limit = g.lame == (int)blockIdx.x ? 0u : PERSIST_POLL_LIMIT;
      for (unsigned tries = 0; !got && tries < limit; ++tries) {
        got = true;
#pragma unroll
        for (int q = 0; q < PH; ++q)
          if (ho[q] >= 0) {
            const ulonglong2 x = box_get(halo + hh[q]);
            got = got && box_is(x, epoch);
            hs[q] = box_value(x);
          }
      }
      if (!got) X.fail = 1;
    } else {
      C.rrn = exchange_sum(&X, inboxes(), epoch, ctas, g.extra, C.rro, nullptr);
      C.after_rrn(&S, n, &sh_beta, &sh_status, g.a.rd.hist_b);
    }
    ++epoch;
    updated = true;
    upd = true;
    ++n;
    __syncthreads();
    if (X.fail || sh_status != RUN) {
      ++done;
      break;
    }
  }
  if (X.fail) {  // in a word of its own: CTA 0 may have ended its loop and store its state after this
    if (t == 0) *g.err = 1u;
    return;
  }
  // ---- the fields and the state as the loop's kernels leave them (w = A p_n formed again) ----
  const int last = updated ? n - 1 : n;  // the iteration whose p is in shared memory
  double* const pout = (last & 1) ? f.p2 : f.p;
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const int o = o0 + i * ostep, c = c0 + i * cstep;
    if (i < mine) {
      const double pc = sp[o];
      double wv = sdi[o] * pc;
      wv = fma(-scy[o + P], sp[o + P], wv);
      wv = fma(-scy[o], sp[o - P], wv);
      wv = fma(-scx[o + 1], sp[o + 1], wv);
      wv = fma(-scx[o], sp[o - 1], wv);
      f.w[c] = wv;
      pout[c] = pc;
      f.r[c] = r[i];
      if (UREG) f.u[c] = u[i];
      if (DIAG && updated) f.z[c] = w[i];
    }
  }
  if (blockIdx.x == 0 && t == 0) {
    C.store(S, n, done);
    *g.a.rd.st = S;
    *g.st_host = S;
  }
}

// ---- the FP32 process of the precision form (tl_mixed.cu) -------------------------------------
// The same loop on FP32 vectors: k_mix_w and k_mix_ur with d += alpha p in the wait for beta.  p
// with its halo and r live in shared memory, w and d in tensor memory (which no tensor core uses
// here: 128 words a thread); the operator's coefficients stay in the fields, which the L2 cache
// (and, for small tiles, the SM's own) holds.  8 bytes a cell in shared memory take meshes of up to
// 4.3 million cells, 2048^2 among them.  A thread owns consecutive rows of a column, so a row's
// upper face is the next row's lower one; rows go in groups of MC, whose loads precede its stores (the
// compiler cannot tell the arrays of shared memory apart, and a load behind a store waits for it), and the
// coefficients of the next group are in flight while one is used.  d is updated before the wait for beta's
// partials, in the time they take; the rim's columns are sent by whole warps.  Time per iteration, the
// replacements included, against the sweeps' two launches: 512^2 9.7 against 25.0 us, 1000^2 11.5 / 34.0,
// 1500 x 1999 17.1 / 48.0, 2048^2 20.4 / 50.4, with jac_diag 24.2 / 55.5.  Row by row, with a test of
// the row, a test of the mesh's walls and a store to the neighbour's box in each, 2048^2 took 32.4 us and
// 1000^2 13.2: the walls are mirrored by the neighbours' offsets, and what has no row works on a cell of
// zeros.  The sums' exchange, 6 us, bounds it up to about 1000^2, the coefficients' way from L2 (13 bytes
// a cell) above; taking the right face from the next lane instead of loading it gave nothing.
// The dot products are the sweeps': Dot2 per thread, then exact integers.
struct MixPersistArgs {
  MixFields m;
  Layout L;
  MixState* ms;
  PersistPlan pl;
  int max_run;
  unsigned epoch;
  ulonglong2* box;
  unsigned* err;  // set when a wait ran out in any CTA: the results are void
  int extra;      // as in PersistArgs
  int lame;
};

// a float beside the sum's number
__device__ __forceinline__ void fbox_put(unsigned long long* s, float v, unsigned epoch) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(s), "l"(((unsigned long long)__float_as_uint(v) << 32) | epoch)
               : "memory");
}
__device__ __forceinline__ unsigned long long fbox_get(const unsigned long long* s) {
  unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(s) : "memory");
  return w;
}

// s + c of every lane, summed over the warp
__device__ __forceinline__ Fix warp_fix(const Dot2& d) {
  const unsigned bs = __float_as_uint(d.s), bc = __float_as_uint(d.c);
  auto ex = [](unsigned b) {
    const unsigned e = (b >> 23) & 0xffu;
    return e == 0xffu ? 0x7ffu : max(e, 1u) + 896u;  // biased as a double's
  };
  auto fix = [](unsigned b, unsigned ev, unsigned e) {
    const uint64_t m = (uint64_t)((b & 0x7fffffu) | ((b & 0x7f800000u) ? 0x800000u : 0u)) << 29;
    const long long i = (long long)((((m << (FSH + 1)) >> min(e - ev, 63u)) + 1ull) >> 1);
    return (b >> 31) ? -i : i;
  };
  const unsigned es = ex(bs), ec = ex(bc);
  const unsigned e = __reduce_max_sync(0xffffffffu, max(es, ec));
  if (e == 0x7ffu) return Fix{0, e};  // beside an infinite sum the error terms are NaN
  return Fix{warp_add((fix(bs, es, e) >> 1) + (fix(bc, ec, e) >> 1)), e + 1u};
}

// Tensor memory as the threads' own storage: 512 columns of 128 lanes, of which a warp reaches the
// 32 lanes of its number modulo 4; the four warps of a quarter take 128 columns each, 2 MROWS words a
// thread.
constexpr int MROWS = 64;  // rows a thread may own
__device__ __forceinline__ void tmem_alloc(unsigned* at) {  // a whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(at))
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(unsigned a) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(a) : "memory");
}
__device__ __forceinline__ void tmem_put(unsigned a, const float (&v)[8]) {
  __syncwarp();
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(a), "f"(v[0]), "f"(v[1]),
               "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}
__device__ __forceinline__ void tmem_put(unsigned a, const float (&v)[4]) {
  __syncwarp();
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
               : "memory");
}
__device__ __forceinline__ void tmem_put(unsigned a, const float (&v)[2]) {
  __syncwarp();
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(a), "f"(v[0]), "f"(v[1]) : "memory");
}
// before the words are read again
__device__ __forceinline__ void tmem_put_done() {
  __syncwarp();
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_get(unsigned a, float (&v)[8]) {
  __syncwarp();
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n tcgen05.wait::ld.sync.aligned;"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "r"(a)
               : "memory");
}

__device__ __forceinline__ void tmem_get(unsigned a, float (&v)[4]) {
  __syncwarp();
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n tcgen05.wait::ld.sync.aligned;"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void tmem_get(unsigned a, float (&v)[2]) {
  __syncwarp();
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];\n tcgen05.wait::ld.sync.aligned;"
               : "=f"(v[0]), "=f"(v[1])
               : "r"(a)
               : "memory");
}

// MC: rows handled together.
template <bool DIAG, int MC>
__global__ void __launch_bounds__(PTHREADS, 1) k_persistent_mix(MixPersistArgs g) {
  __shared__ MixState S;
  __shared__ Exchange X;
  __shared__ float sh_alpha, sh_beta;
  __shared__ int sh_status;
  __shared__ unsigned sh_tmem;
  extern __shared__ __align__(16) float fsm[];
  const Layout L = g.L;
  const MixFields& f = g.m;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const bool owner = wid != 0;
  const int to = t - 32;
  const int ctas = gridDim.x;
  if (t == 0) {
    S = *g.ms;
    sh_status = S.status;
    sh_beta = (float)S.beta;
    X.fail = 0;
  }
  __syncthreads();
  if (sh_status != RUN) return;
  if (wid == 0) tmem_alloc(&sh_tmem);

  const int bx = blockIdx.x % g.pl.gx, by = blockIdx.x / g.pl.gx;
  const int j0 = bx * g.pl.tw, k0 = by * g.pl.th;
  const int tw = min(g.pl.tw, L.nx - j0), th = min(g.pl.th, L.ny - k0);
  const int P = g.pl.tw + 2;
  float* const sp = fsm;
  float* const sr = fsm + (g.pl.th + 2) * P;

  // the thread's column and rows y0 .. y0+mine-1: the rows split evenly, so that two threads' differ by
  // one at most.  The lanes left over of a warp that owns cells, and the rows left over of the last group of
  // rows, work on a cell of zeros past the tile: no row is a branch
  const int tx = owner ? to % g.pl.tw : 0, seg = owner ? to / g.pl.tw : 0;
  const int q_ = th / g.pl.ry, rem = th - q_ * g.pl.ry;
  const int mine = (owner && tx < tw && seg < g.pl.ry) ? q_ + (seg < rem) : 0, y0 = seg * q_ + min(seg, rem);
  const int own = mine ? mine : q_ + (rem > 0);
  const bool warp_owns = __any_sync(0xffffffffu, mine > 0);
  const int nfull = warp_owns ? (int)__reduce_min_sync(0xffffffffu, (unsigned)own) / MC : 0;  // groups of MC rows
  const int nch = warp_owns ? ((int)__reduce_max_sync(0xffffffffu, (unsigned)own) + MC - 1) / MC : 0;
  const int rz = g.pl.th * g.pl.tw, oz = (g.pl.th + 2) * P + rz;  // the cell of zeros, from sr and from sp
  const int r0 = mine ? y0 * g.pl.tw + tx : rz, o0 = mine ? (y0 + 1) * P + tx + 1 : oz;
  const int c0 = mine ? (int)L.at(j0 + tx + 1, k0 + y0 + 1) : (int)L.at(j0 + 1, k0 + 1);
  const int ld = L.ld, os = mine ? P : 0, rs = mine ? g.pl.tw : 0, cs = mine ? ld : 0;
  const bool at_l = tx == 0 && j0 == 0, at_r = tx == tw - 1 && j0 + tw == L.nx;
  // the neighbours' offsets: a reflecting wall mirrors the cell
  const int lo = (at_l || !mine) ? 0 : -1, ro = (at_r || !mine) ? 0 : 1;
  const int i_first = (mine > 0 && y0 == 0) ? 0 : -1, i_last = (mine > 0 && y0 + mine == th) ? mine - 1 : -1;
  const int i_b = k0 == 0 ? i_first : -1, i_t = k0 + th == L.ny ? i_last : -1;

  const int hbox = 2 * (g.pl.th + g.pl.tw);
  unsigned long long* const halo = reinterpret_cast<unsigned long long*>(g.box + (size_t)2 * ctas * SLOTS);
  int ho[PH], hh[PH];
  float hp[PH], hs[PH];
  float* const src = DIAG ? f.z : f.r;
  int n = S.n;
  const float* const pold = (n & 1) ? f.p : f.p2;
  bool upd = S.p_pending != 0;
#pragma unroll
  for (int q = 0; q < PH; ++q) {
    const int h = to + q * PT;
    ho[q] = -1;
    hh[q] = 0;
    hp[q] = hs[q] = 0.f;
    int x = -1, y = h;
    bool is = j0 > 0 && y < th;
    if (h >= g.pl.th) x = tw, y = h - g.pl.th, is = j0 + tw < L.nx && y < th;
    if (h >= 2 * g.pl.th) x = h - 2 * g.pl.th, y = -1, is = k0 > 0 && x < tw;
    if (h >= 2 * g.pl.th + g.pl.tw) x = h - 2 * g.pl.th - g.pl.tw, y = th, is = k0 + th < L.ny && x < tw;
    if (is && owner && h < hbox) {
      ho[q] = (y + 1) * P + x + 1;
      hh[q] = (int)blockIdx.x * hbox + h;
      const int c = (int)L.at(j0 + x + 1, k0 + y + 1);
      hp[q] = pold[c];
      if (upd) hs[q] = src[c];
    }
  }
  const int to_l = (mine && tx == 0 && j0 > 0) ? ((int)blockIdx.x - 1) * hbox + g.pl.th + y0 : -1;
  const int to_r = (mine && tx == tw - 1 && j0 + tw < L.nx) ? ((int)blockIdx.x + 1) * hbox + y0 : -1;
  const int rim_b = k0 > 0 ? i_first : -1, rim_t = k0 + th < L.ny ? i_last : -1;
  const int to_b = ((int)blockIdx.x - g.pl.gx) * hbox + 2 * g.pl.th + g.pl.tw + tx;
  const int to_t = ((int)blockIdx.x + g.pl.gx) * hbox + 2 * g.pl.th + tx;

  __syncthreads();
  // this thread's words of tensor memory: w (z between phases B and A with DIAG), then d
  const unsigned tw_ = sh_tmem + ((unsigned)(wid & 3) << 21) + (unsigned)(wid >> 2) * (2 * MROWS), td_ = tw_ + MROWS;
  if (t == 0) sp[oz] = 0.f;
  {
    int o = o0, rr = r0, c = c0;
    // the deferred d += alpha p of an earlier step (its p is the one read here)
    const bool upd_d = S.d_pending != 0;
    const float da = (float)S.d_alpha;
    for (int ch = 0; ch < nch; ++ch) {
      float z[MC], d[MC];
#pragma unroll
      for (int j = 0; j < MC; ++j, o += os, rr += rs, c += cs) {
        z[j] = d[j] = 0.f;
        if (ch * MC + j < mine) {
          const float p = pold[c];
          sp[o] = p;
          sr[rr] = f.r[c];
          if (DIAG) z[j] = f.z[c];
          d[j] = f.d[c];
          if (upd_d) d[j] = fmaf(da, p, d[j]);
        }
      }
      tmem_put(tw_ + ch * MC, z);
      tmem_put(td_ + ch * MC, d);
    }
    tmem_put_done();
  }

  double rro = S.rro, rro_prev = S.rro_prev, pw = S.pw, alpha_ = S.alpha, beta_ = S.beta, rr_ = S.rr;
  unsigned epoch = g.epoch;
  __syncthreads();

  auto give = [&](const Dot2& v) {
    const Fix s = warp_fix(v);
    if (lane == 0) X.part[wid - 1] = s;
    bar_arrive<1, PTHREADS>();
  };
  const int nwait = ctas > 1 ? ctas + g.extra : 0, nq = (nwait + 31) / 32;
  auto poll = [&] {
    if (wid > nq) return;
    const int slot = (wid - 1) * 32 + lane;
    const ulonglong2* in = g.box + ((size_t)(epoch & 1u) * ctas + blockIdx.x) * SLOTS + slot;
    ulonglong2 x = make_ulonglong2(0ull, 0ull);
    bool here = slot >= nwait;
    for (unsigned tries = 0; !here && tries < PERSIST_POLL_LIMIT; ++tries) {
      x = box_get(in);
      here = box_is(x, epoch);
    }
    if (!here) X.fail = 1;
    __syncwarp();
    const Fix q = warp_fix(slot < nwait ? box_value(x) : 0.0);
    if (lane == 0) X.inbox[wid - 1] = q;
    bar_arrive(3, 32 * (nq + 1));
  };
  auto inboxes = [&] { return g.box + (size_t)(epoch & 1u) * ctas * SLOTS; };
  struct Coefs {
    float di[MC], cl[MC], cr[MC], ct[MC];  // Di, the left, right and upper face of a group of rows
  } ka, kb;
  const std::true_type full;
  const std::false_type part;
  auto load_group = [&](int ch, Coefs& k, auto f_) {
    const int left = own - ch * MC, c1 = decltype(f_)::value || left > 0 ? c0 + ch * MC * cs : c0;
    const float *pd = f.di + c1, *px = f.cx + c1, *py = f.cy + c1 + ld;
#pragma unroll
    for (int j = 0; j < MC; ++j) {
      k.di[j] = __ldg(pd);
      k.cl[j] = __ldg(px);
      k.cr[j] = __ldg(px + 1);
      k.ct[j] = __ldg(py);
      if (decltype(f_)::value || j + 1 < left) pd += cs, px += cs, py += cs;
    }
  };
  auto load_coefs = [&](int ch, Coefs& k) {
    if (ch < nfull) load_group(ch, k, full);
    else if (ch < nch) load_group(ch, k, part);
  };
  // a sweep over the thread's groups of rows
  auto sweep = [&](auto&& group) {
    for (int ch = 0; ch < nfull; ++ch) group(ch, full);
    if (nfull < nch) group(nfull, part);
  };

  load_coefs(0, ka);

  bool any = false;
  for (int done = 0; done < g.max_run; ++done) {
    // ---- phase A: p_n, w = A p_n, p.w ----
    if (owner) {
      const float beta = sh_beta;
      if (upd) {
        sweep([&](int ch, auto f_) {
          // a group's loads before its stores, which the compiler cannot tell apart
          const int o = o0 + ch * MC * os, rr = r0 + ch * MC * rs, left = own - ch * MC;
          float p[MC], z[MC];
#pragma unroll
          for (int j = 0; j < MC; ++j) {
            const bool in = decltype(f_)::value || j < left;
            p[j] = sp[in ? o + j * os : oz];
            if (!DIAG) z[j] = sr[in ? rr + j * rs : rz];
          }
          if (DIAG) tmem_get(tw_ + ch * MC, z);
#pragma unroll
          for (int j = 0; j < MC; ++j) {
            const bool in = decltype(f_)::value || j < left;
            sp[in ? o + j * os : oz] = fmaf(beta, p[j], z[j]);
          }
        });
      }
      if (i_b >= 0) sp[o0 - P] = sp[o0];
      if (i_t >= 0) sp[o0 + mine * P] = sp[o0 + (mine - 1) * P];
#pragma unroll
      for (int q = 0; q < PH; ++q)
        if (ho[q] >= 0) {
          if (upd) hp[q] = fmaf(beta, hp[q], hs[q]);
          sp[ho[q]] = hp[q];
        }
      bar_sync<2, PT>();
      Dot2 dot;
      {
        int o = o0;
        float pb = 0.f, pc = 0.f, cyb = 0.f;
        if (nch > 0) pb = sp[o - os], pc = sp[o], cyb = __ldg(f.cy + c0);
        auto rows_of = [&](int ch, const Coefs& k, auto f_) {
          const int left = own - ch * MC;
          float w[MC];
#pragma unroll
          for (int j = 0; j < MC; ++j) {
            const bool in = decltype(f_)::value || j < left;
            if (!in) pb = pc = 0.f;
            const float pt = sp[in ? o + os : oz];
            float a = k.di[j] * pc;
            a = fmaf(-k.ct[j], pt, a);
            a = fmaf(-cyb, pb, a);
            a = fmaf(-k.cr[j], sp[in ? o + ro : oz], a);
            a = fmaf(-k.cl[j], sp[in ? o + lo : oz], a);
            w[j] = a;
            dot.add(a, pc);
            pb = pc;
            pc = pt;
            cyb = k.ct[j];
            o += os;
          }
          tmem_put(tw_ + ch * MC, w);
        };
        auto rows = [&](int ch, const Coefs& k) {
          if (ch < nfull) rows_of(ch, k, full);
          else if (ch < nch) rows_of(ch, k, part);
        };
        // two groups of coefficients: the next one's loads are in flight while one is used
        for (int ch = 0; ch < nch; ch += 2) {
          load_coefs(ch + 1, kb);
          rows(ch, ka);
          load_coefs(ch + 2, ka);
          rows(ch + 1, kb);
        }
        tmem_put_done();
      }
      give(dot);
      poll();
    } else {
      pw = exchange_sum(&X, inboxes(), epoch, ctas, g.extra, rro, nullptr);
      alpha_ = rro / pw;
      if (lane == 0) {
        sh_alpha = (float)alpha_;
        if (!finite_bits(alpha_)) sh_status = EXIT_BREAKDOWN;
        if (blockIdx.x == 0 && S.hist_a) S.hist_a[n] = alpha_;
      }
    }
    ++epoch;
    __syncthreads();
    if (X.fail || sh_status != RUN) break;
    // ---- phase B: r -= alpha w, z = Mi r, r.z; the rim to the neighbours; d += alpha p_n ----
    if (owner) {
      const float alpha = sh_alpha;
      Dot2 dot;
      sweep([&](int ch, auto f_) {
        const int rr = r0 + ch * MC * rs, left = own - ch * MC;
        float w[MC], r[MC], mi[MC];
#pragma unroll
        for (int j = 0; j < MC; ++j) {
          const bool in = decltype(f_)::value || j < left;
          r[j] = sr[in ? rr + j * rs : rz];
          if (DIAG) mi[j] = __ldg(f.mi + (in ? c0 + (ch * MC + j) * cs : c0));
        }
        tmem_get(tw_ + ch * MC, w);
#pragma unroll
        for (int j = 0; j < MC; ++j) {
          r[j] = fmaf(-alpha, w[j], r[j]);
          sr[decltype(f_)::value || j < left ? rr + j * rs : rz] = r[j];
          w[j] = DIAG ? mi[j] * r[j] : r[j];
          dot.add(r[j], w[j]);
        }
        if (DIAG) tmem_put(tw_ + ch * MC, w);
      });
      // the rim: a column's rows are its owner's, and the whole warp sends them
      auto rim = [&](int rr, int c) {
        const float r = sr[rr];
        return DIAG ? __ldg(f.mi + c) * r : r;
      };
      if (rim_b >= 0) fbox_put(halo + to_b, rim(r0 + rim_b * rs, c0 + rim_b * cs), epoch);
      if (rim_t >= 0) fbox_put(halo + to_t, rim(r0 + rim_t * rs, c0 + rim_t * cs), epoch);
      __syncwarp();
      auto columns = [&](int to_) {
        for (unsigned m = __ballot_sync(0xffffffffu, to_ >= 0); m; m &= m - 1) {
          const int l = __ffs(m) - 1;
          const int h = __shfl_sync(0xffffffffu, to_, l), r1 = __shfl_sync(0xffffffffu, r0, l),
                    c1 = __shfl_sync(0xffffffffu, c0, l), have = __shfl_sync(0xffffffffu, mine, l);
          for (int i = lane; i < have; i += 32) fbox_put(halo + h + i, rim(r1 + i * g.pl.tw, c1 + i * ld), epoch);
        }
      };
      columns(to_l);
      columns(to_r);
      give(dot);
      // d += alpha p_n while the sum is under way
      sweep([&](int ch, auto f_) {
        const int o = o0 + ch * MC * os, left = own - ch * MC;
        float d[MC], p[MC];
#pragma unroll
        for (int j = 0; j < MC; ++j) p[j] = sp[decltype(f_)::value || j < left ? o + j * os : oz];
        tmem_get(td_ + ch * MC, d);
#pragma unroll
        for (int j = 0; j < MC; ++j) d[j] = fmaf(alpha, p[j], d[j]);
        tmem_put(td_ + ch * MC, d);
      });
      tmem_put_done();
      load_coefs(0, ka);  // of the next phase A
      poll();
      bool got = false;
      const unsigned limit = g.lame == (int)blockIdx.x ? 0u : PERSIST_POLL_LIMIT;
      for (unsigned tries = 0; !got && tries < limit; ++tries) {
        got = true;
#pragma unroll
        for (int q = 0; q < PH; ++q)
          if (ho[q] >= 0) {
            const unsigned long long x = fbox_get(halo + hh[q]);
            got = got && (unsigned)x == epoch;
            hs[q] = __uint_as_float((unsigned)(x >> 32));
          }
      }
      if (!got) X.fail = 1;
    } else {
      rr_ = exchange_sum(&X, inboxes(), epoch, ctas, g.extra, rro, nullptr);
      beta_ = rr_ / rro;
      if (lane == 0) {
        sh_beta = (float)beta_;
        if (blockIdx.x == 0 && S.hist_b) S.hist_b[n] = beta_;
        if (!finite_bits(beta_)) {
          sh_status = EXIT_BREAKDOWN;
          S.n = n;
        } else {
          S.n = n;
          S.rr = rr_;
          mix_finish(&S);
          sh_status = S.status;
        }
      }
      rro_prev = rro;
      rro = rr_;
    }
    ++epoch;
    ++n;
    upd = true;
    any = true;
    __syncthreads();
    if (X.fail || sh_status != RUN) break;
  }
  const bool failed = X.fail != 0;
  // p in the buffer the next step reads, r (and z), d
  float* const pout = ((n - 1) & 1) ? f.p2 : f.p;
  {
    int o = o0, rr = r0, c = c0;
    for (int ch = 0; ch < (failed ? 0 : nch); ++ch) {
      float z[MC], d[MC];
      if (DIAG) tmem_get(tw_ + ch * MC, z);
      tmem_get(td_ + ch * MC, d);
#pragma unroll
      for (int j = 0; j < MC; ++j, o += os, rr += rs, c += cs) {
        if (ch * MC + j < mine) {
          pout[c] = sp[o];
          f.r[c] = sr[rr];
          if (DIAG && any) f.z[c] = z[j];
          f.d[c] = d[j];
        }
      }
    }
  }
  __syncthreads();  // every warp is done with tensor memory
  if (wid == 0) tmem_free(sh_tmem);
  if (failed) {
    if (t == 0) *g.err = 1u;
    return;
  }
  if (blockIdx.x == 0 && t == 0) {
    S.status = sh_status;
    S.pw = pw;
    S.alpha = alpha_;
    S.d_pending = 0;
    if (any) {
      S.rr = rr_;
      S.beta = beta_;
      S.rro = rro;
      S.rro_prev = rro_prev;
      S.p_pending = 1;
    }
    *g.ms = S;
  }
}

// ---- the FP64 CG loop on larger tiles ----------------------------------------------------------
// k_persistent_cg's loop laid out as k_persistent_mix: p with its halo and r in shared memory, w and u in
// tensor memory, the coefficients (and Mi) streamed from the fields through L2, a group of rows ahead.
// 16 bytes a cell in shared memory take meshes of up to 2.1 million cells.  It runs where k_persistent_cg's
// tiles do not fit (11 cells a thread, about 800K cells; 777 x 1013 runs here): at 700^2 it takes 14.5 us
// an iteration against 14.2; larger tiles there spilled from 14 cells a thread on (26.2 us at 1024^2 against
// 24.1).  Its two groups of four rows' coefficients fill the registers (68 to 72 bytes spilled).  Against
// the batched sweeps: 1000^2 22.3 us an iteration against 42.1, 1024^2 24.1 / 42.4, 1100^2 with jac_diag
// 31.2 / 50.4, 1200^2 28.4 / 48.1, 1300 x 1400 36.7 / 61.7.  The FP64 pipe's share is 17 us at 1000^2, 31 at
// 1300 x 1400.
constexpr int WROWS = 32;  // rows a thread may own
constexpr int WC = 4;      // rows handled together
__device__ __forceinline__ void tmem_put(unsigned a, const double (&v)[4]) {
  float w[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    w[2 * i] = __int_as_float(__double2loint(v[i]));
    w[2 * i + 1] = __int_as_float(__double2hiint(v[i]));
  }
  tmem_put(a, w);
}
__device__ __forceinline__ void tmem_get(unsigned a, double (&v)[4]) {
  float w[8];
  tmem_get(a, w);
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __hiloint2double(__float_as_int(w[2 * i + 1]), __float_as_int(w[2 * i]));
}

template <bool DIAG>
__global__ void __launch_bounds__(PTHREADS, 1) k_persistent_cg_wide(PersistArgs g) {
  __shared__ LoopState S;
  __shared__ Exchange X;
  __shared__ double sh_alpha, sh_beta;
  __shared__ int sh_status;
  __shared__ unsigned sh_tmem;
  extern __shared__ __align__(16) double wsm[];
  const Layout L = g.a.L;
  const Fields& f = g.a.f;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const bool owner = wid != 0;
  const int to = t - 32;
  const int ctas = gridDim.x;
  if (t == 0) {
    S = *g.a.rd.st;
    sh_status = S.status;
    sh_beta = S.beta;
    X.fail = 0;
  }
  __syncthreads();
  if (sh_status != RUN) {
    if (blockIdx.x == 0 && t == 0) *g.st_host = S;
    return;
  }
  if (wid == 0) tmem_alloc(&sh_tmem);

  const int bx = blockIdx.x % g.pl.gx, by = blockIdx.x / g.pl.gx;
  const int j0 = bx * g.pl.tw, k0 = by * g.pl.th;
  const int tw = min(g.pl.tw, L.nx - j0), th = min(g.pl.th, L.ny - k0);
  const int P = g.pl.tw + 2, rows = g.pl.rows;
  double* const sp = wsm;
  double* const sr = wsm + (g.pl.th + 2) * P;

  // the thread's column and rows y0 .. y0+mine-1
  const int tx = owner ? to % g.pl.tw : 0, seg = owner ? to / g.pl.tw : 0, y0 = seg * rows;
  const int mine = (owner && tx < tw && seg < g.pl.ry) ? max(0, min(rows, th - y0)) : 0;
  const int o0 = (y0 + 1) * P + tx + 1, r0 = y0 * g.pl.tw + tx;
  const int c0 = (int)L.at(j0 + tx + 1, k0 + y0 + 1);
  const int ld = L.ld, rst = g.pl.tw;
  const bool at_l = tx == 0 && j0 == 0, at_r = tx == tw - 1 && j0 + tw == L.nx;
  const int i_first = y0 == 0 ? 0 : -1, i_last = (mine > 0 && y0 + mine == th) ? mine - 1 : -1;
  const int i_b = k0 == 0 ? i_first : -1, i_t = k0 + th == L.ny ? i_last : -1;

  const int hbox = 2 * (g.pl.th + g.pl.tw);
  ulonglong2* const halo = g.box + (size_t)2 * ctas * SLOTS;
  int ho[PH], hh[PH];
  double hp[PH], hs[PH];
  double* const src = DIAG ? f.z : f.r;
  int n = S.n;
  const double* const pold = (n & 1) ? f.p : f.p2;
  bool upd = S.p_pending != 0;
#pragma unroll
  for (int q = 0; q < PH; ++q) {
    const int h = to + q * PT;
    ho[q] = -1;
    hh[q] = 0;
    hp[q] = hs[q] = 0.0;
    int x = -1, y = h;
    bool is = j0 > 0 && y < th;
    if (h >= g.pl.th) x = tw, y = h - g.pl.th, is = j0 + tw < L.nx && y < th;
    if (h >= 2 * g.pl.th) x = h - 2 * g.pl.th, y = -1, is = k0 > 0 && x < tw;
    if (h >= 2 * g.pl.th + g.pl.tw) x = h - 2 * g.pl.th - g.pl.tw, y = th, is = k0 + th < L.ny && x < tw;
    if (is && owner && h < hbox) {
      ho[q] = (y + 1) * P + x + 1;
      hh[q] = (int)blockIdx.x * hbox + h;
      const int c = (int)L.at(j0 + x + 1, k0 + y + 1);
      hp[q] = pold[c];
      if (upd) hs[q] = src[c];
    }
  }
  const int to_l = (mine && tx == 0 && j0 > 0) ? ((int)blockIdx.x - 1) * hbox + g.pl.th + y0 : -1;
  const int to_r = (mine && tx == tw - 1 && j0 + tw < L.nx) ? ((int)blockIdx.x + 1) * hbox + y0 : -1;
  const int rim_b = k0 > 0 ? i_first : -1, rim_t = k0 + th < L.ny ? i_last : -1;
  const int to_b = ((int)blockIdx.x - g.pl.gx) * hbox + 2 * g.pl.th + g.pl.tw + tx;
  const int to_t = ((int)blockIdx.x + g.pl.gx) * hbox + 2 * g.pl.th + tx;

  __syncthreads();
  // this thread's words of tensor memory: w (z between phases B and A with DIAG), then u
  const unsigned tw_ = sh_tmem + ((unsigned)(wid & 3) << 21) + (unsigned)(wid >> 2) * 128u, td_ = tw_ + 2 * WROWS;
  const int nch = owner ? (rows + WC - 1) / WC : 0;
  {
    int o = o0, rr = r0, c = c0;
    for (int ch = 0; ch < nch; ++ch) {
      double z[WC], d[WC];
#pragma unroll
      for (int j = 0; j < WC; ++j, o += P, rr += rst, c += ld) {
        z[j] = d[j] = 0.0;
        if (ch * WC + j < mine) {
          const double p = pold[c];
          sp[o] = p;
          sr[rr] = f.r[c];
          if (DIAG) z[j] = f.z[c];
          d[j] = f.u[c];
        }
      }
      tmem_put(tw_ + ch * 2 * WC, z);
      tmem_put(td_ + ch * 2 * WC, d);
    }
    tmem_put_done();
  }

  CgScalars C(S);  // in the first warp
  unsigned epoch = g.epoch;
  __syncthreads();

  auto give = [&](double v) {
    const Fix s = warp_fix(v);
    if (lane == 0) X.part[wid - 1] = s;
    bar_arrive<1, PTHREADS>();
  };
  const int nwait = ctas > 1 ? ctas + g.extra : 0, nq = (nwait + 31) / 32;
  auto poll = [&] {
    if (wid > nq) return;
    const int slot = (wid - 1) * 32 + lane;
    const ulonglong2* in = g.box + ((size_t)(epoch & 1u) * ctas + blockIdx.x) * SLOTS + slot;
    ulonglong2 x = make_ulonglong2(0ull, 0ull);
    bool here = slot >= nwait;
    for (unsigned tries = 0; !here && tries < PERSIST_POLL_LIMIT; ++tries) {
      x = box_get(in);
      here = box_is(x, epoch);
    }
    if (!here) X.fail = 1;
    __syncwarp();
    const Fix q = warp_fix(slot < nwait ? box_value(x) : 0.0);
    if (lane == 0) X.inbox[wid - 1] = q;
    bar_arrive(3, 32 * (nq + 1));
  };
  auto inboxes = [&] { return g.box + (size_t)(epoch & 1u) * ctas * SLOTS; };
  struct Coefs {
    double di[WC], cl[WC], cr[WC], ct[WC];  // Di, the left, right and upper face of a group of rows
  } ka, kb;
  auto load_coefs = [&](int ch, Coefs& k) {
    int c = c0 + ch * WC * ld;
#pragma unroll
    for (int j = 0; j < WC; ++j, c += ld) {
      k.di[j] = k.cl[j] = k.cr[j] = k.ct[j] = 0.0;
      if (ch * WC + j < mine) {
        k.di[j] = __ldg(f.di + c);
        k.cl[j] = __ldg(f.cx + c);
        k.cr[j] = __ldg(f.cx + c + 1);
        k.ct[j] = __ldg(f.cy + c + ld);
      }
    }
  };
  load_coefs(0, ka);

  int done = 0;
  bool any = false;  // phase B of the last iteration ran
  for (; done < g.max_run; ++done) {
    // ---- phase A: p_n, w = A p_n, p.w ----
    any = false;
    if (owner) {
      const double beta = sh_beta;
      {
        // the even iterations' p is what the loop leaves in the field p
        double* const pf = (n & 1) ? nullptr : f.p;
        int o = o0, rr = r0, c = c0;
        for (int ch = 0; ch < nch; ++ch) {
          double z[WC];
          if (DIAG) tmem_get(tw_ + ch * 2 * WC, z);
#pragma unroll
          for (int j = 0; j < WC; ++j, o += P, rr += rst, c += ld) {
            const int i = ch * WC + j;
            if (i < mine) {
              double p = sp[o];
              if (upd) p = fma(beta, p, DIAG ? z[j] : sr[rr]);
              sp[o] = p;
              if (pf) pf[c] = p;
              if (at_l) sp[o - 1] = p;
              if (at_r) sp[o + 1] = p;
              if (i == i_b) sp[o - P] = p;
              if (i == i_t) sp[o + P] = p;
            }
          }
        }
      }
#pragma unroll
      for (int q = 0; q < PH; ++q)
        if (ho[q] >= 0) {
          if (upd) hp[q] = fma(beta, hp[q], hs[q]);
          sp[ho[q]] = hp[q];
        }
      bar_sync<2, PT>();
      double dot = 0.0;
      {
        int o = o0;
        double pb = 0.0, pc = 0.0, cyb = 0.0;
        if (mine > 0) pb = sp[o - P], pc = sp[o], cyb = __ldg(f.cy + c0);
        auto rows_of = [&](int ch, const Coefs& k) {
          double w[WC];
#pragma unroll
          for (int j = 0; j < WC; ++j, o += P) {
            w[j] = 0.0;
            if (ch * WC + j < mine) {
              const double pt = sp[o + P];
              double a = dmul_int(k.di[j], pc);
              a = fma(-k.ct[j], pt, a);
              a = fma(-cyb, pb, a);
              a = fma(-k.cr[j], sp[o + 1], a);
              a = fma(-k.cl[j], sp[o - 1], a);
              w[j] = a;
              dot = fma(a, pc, dot);
              pb = pc;
              pc = pt;
              cyb = k.ct[j];
            }
          }
          tmem_put(tw_ + ch * 2 * WC, w);
        };
        // two groups of coefficients: the next one's loads are in flight while one is used
        for (int ch = 0; ch < nch; ch += 2) {
          if (ch + 1 < nch) load_coefs(ch + 1, kb);
          rows_of(ch, ka);
          if (ch + 1 < nch) {
            if (ch + 2 < nch) load_coefs(ch + 2, ka);
            rows_of(ch + 1, kb);
          }
        }
        tmem_put_done();
      }
      give(dot);
      poll();
    } else {
      C.pw = exchange_sum(&X, inboxes(), epoch, ctas, g.extra, C.rro, &C.inv_rro);
      C.after_pw(&S, n, &sh_alpha, &sh_status, g.a.rd.hist_a);
    }
    ++epoch;
    __syncthreads();
    if (X.fail || sh_status != RUN) break;
    // ---- phase B: r -= alpha w, z = Mi r, r.z; the rim to the neighbours; d += alpha p_n ----
    if (owner) {
      const double alpha = sh_alpha;
      double dot = 0.0;
      {
        int rr = r0, c = c0;
        for (int ch = 0; ch < nch; ++ch) {
          double w[WC], mi[WC];
          if (DIAG) {
#pragma unroll
            for (int j = 0; j < WC; ++j, c += ld)
              mi[j] = ch * WC + j < mine ? __ldg(f.mi + c) : 0.0;
          }
          tmem_get(tw_ + ch * 2 * WC, w);
#pragma unroll
          for (int j = 0; j < WC; ++j, rr += rst) {
            const int i = ch * WC + j;
            if (i < mine) {
              const double rv = fma(-alpha, w[j], sr[rr]);
              sr[rr] = rv;
              double zv = rv;
              if (DIAG) {
                zv = dmul_int(mi[j], rv);
                w[j] = zv;
              }
              dot = fma(rv, zv, dot);
              if (to_l >= 0) box_put(halo + to_l + i, zv, epoch);
              if (to_r >= 0) box_put(halo + to_r + i, zv, epoch);
              if (i == rim_b) box_put(halo + to_b, zv, epoch);
              if (i == rim_t) box_put(halo + to_t, zv, epoch);
            }
          }
          if (DIAG) tmem_put(tw_ + ch * 2 * WC, w);
        }
      }
      give(dot);
      load_coefs(0, ka);  // of the next phase A
      poll();
      {
        int o = o0;
        for (int ch = 0; ch < nch; ++ch) {
          double d[WC];
          tmem_get(td_ + ch * 2 * WC, d);
#pragma unroll
          for (int j = 0; j < WC; ++j, o += P)
            if (ch * WC + j < mine) d[j] = fma(alpha, sp[o], d[j]);
          tmem_put(td_ + ch * 2 * WC, d);
        }
        tmem_put_done();
      }
      bool got = false;
      const unsigned limit = g.lame == (int)blockIdx.x ? 0u : PERSIST_POLL_LIMIT;
      for (unsigned tries = 0; !got && tries < limit; ++tries) {
        got = true;
#pragma unroll
        for (int q = 0; q < PH; ++q)
          if (ho[q] >= 0) {
            const ulonglong2 x = box_get(halo + hh[q]);
            got = got && box_is(x, epoch);
            hs[q] = box_value(x);
          }
      }
      if (!got) X.fail = 1;
    } else {
      C.rrn = exchange_sum(&X, inboxes(), epoch, ctas, g.extra, C.rro, nullptr);
      C.after_rrn(&S, n, &sh_beta, &sh_status, g.a.rd.hist_b);
    }
    ++epoch;
    ++n;
    upd = true;
    any = true;
    __syncthreads();
    if (X.fail || sh_status != RUN) {
      ++done;
      break;
    }
  }
  const bool failed = X.fail != 0;
  // the fields and the state as the loop's kernels leave them
  double* const pout = ((any ? n - 1 : n) & 1) ? f.p2 : f.p;
  {
    int o = o0, rr = r0, c = c0;
    for (int ch = 0; ch < (failed ? 0 : nch); ++ch) {
      double z[WC], d[WC];
      tmem_get(tw_ + ch * 2 * WC, z);
      tmem_get(td_ + ch * 2 * WC, d);
#pragma unroll
      for (int j = 0; j < WC; ++j, o += P, rr += rst, c += ld) {
        if (ch * WC + j < mine) {
          pout[c] = sp[o];
          f.r[c] = sr[rr];
          f.u[c] = d[j];
          if (!DIAG || !any) {
            f.w[c] = z[j];
          } else {  // z took w's place: w = A p_n formed again
            f.z[c] = z[j];
            double a = dmul_int(f.di[c], sp[o]);
            a = fma(-f.cy[c + ld], sp[o + P], a);
            a = fma(-f.cy[c], sp[o - P], a);
            a = fma(-f.cx[c + 1], sp[o + 1], a);
            a = fma(-f.cx[c], sp[o - 1], a);
            f.w[c] = a;
          }
        }
      }
    }
  }
  __syncthreads();  // every warp is done with tensor memory
  if (wid == 0) tmem_free(sh_tmem);
  if (failed) {
    if (t == 0) *g.err = 1u;
    return;
  }
  if (blockIdx.x == 0 && t == 0) {
    C.store(S, n, done);
    *g.a.rd.st = S;
    *g.st_host = S;
  }
}

using PersistKernel = void (*)(PersistArgs);
struct PersistVariant {
  int m;
  PersistKernel k[2];  // without / with jac_diag
};
#define PERSIST_VARIANT(M) {M, {k_persistent_cg<M, false>, k_persistent_cg<M, true>}}
// A tile's rows are rounded up to the next of these: up to 4 p stays in registers, up to 6 u and Mi; at 11
// the registers are full (56 bytes spilled), and more cells go to k_persistent_cg_wide.
const PersistVariant kVariants[] = {PERSIST_VARIANT(1), PERSIST_VARIANT(2), PERSIST_VARIANT(4),
                                    PERSIST_VARIANT(6), PERSIST_VARIANT(8), PERSIST_VARIANT(11)};

// p, cx, cy and Di
size_t plan_smem(const PersistPlan& p) { return (size_t)4 * (p.th + 2) * (p.tw + 2) * sizeof(double); }

// CTAs of `threads` threads of kernel k that are co-resident (0: none).  Sets the attribute a launch needs,
// the same for every plan: contexts share it.
int coresident_ctas(const void* k, int threads, size_t smem) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PERSIST_SMEM_MAX) != cudaSuccess ||
      cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return sms * per_sm;
}

}  // namespace

int persist_ctas(const PersistPlan& p) { return p.gx * p.gy; }

// the inboxes of two sums and the halo boxes of two steps
size_t persist_box_bytes(const PersistPlan& p) {
  return (size_t)persist_ctas(p) * (2 * SLOTS + 4 * (p.th + p.tw)) * sizeof(ulonglong2);
}

// The tiling of an nx x ny mesh with the least cycles an iteration: FP64 instructions of a warp on
// the busiest SM (10 an iteration and cell, 17 cycles of the SM's four pipes each), the halo, and
// the two grid sums' exchange (3200 more cycles each across the grid).  all: co-resident CTAs.
bool persist_plan(int nx, int ny, int all, PersistPlan* out) {
  double best = 0.0;
  bool found = false;
  for (const int most : {1, PERSIST_MAX_CTAS}) {  // one CTA, all SMs
    const int ctas = all < most ? all : most;
    for (int g0 = 1; g0 <= ctas && g0 <= nx; ++g0) {
      const int tw = (nx + g0 - 1) / g0;
      if (tw > PT) continue;
      PersistPlan p{};
      p.tw = tw;
      p.gx = (nx + tw - 1) / tw;
      int gy = ctas / p.gx;
      if (gy > ny) gy = ny;
      if (gy < 1) continue;
      p.th = (ny + gy - 1) / gy;
      p.gy = (ny + p.th - 1) / p.th;
      p.ry = PT / tw < p.th ? PT / tw : p.th;
      const int m = (p.th + p.ry - 1) / p.ry;
      p.variant = -1;
      for (int v = (int)(sizeof(kVariants) / sizeof(kVariants[0])) - 1; v >= 0; --v)
        if (kVariants[v].m >= m) p.variant = v;
      const int halo = 2 * (p.tw + p.th);
      if (p.variant < 0 || halo > PH * PT || plan_smem(p) > PERSIST_SMEM_MAX) continue;
      const double slabs = (double)((p.ry * tw + 31) / 32) * m;
      const double sums = most > 1 ? 3200.0 : 0.0;
      const double cost = slabs * 170.0 + 0.5 * halo + 8.0 * p.th + 2.0 * sums;
      if (!found || cost < best) {
        best = cost;
        *out = p;
        found = true;
      }
    }
  }
  return found;
}

constexpr int WIDE = 100;  // PersistPlan::variant of k_persistent_cg_wide

// Kernels that keep fields in tensor memory ask for more than half of an SM's shared memory, so that no two
// of them share an SM: each waits in its allocation for all of tensor memory, and two grids that each hold
// the other's SM would wait for ever.
size_t tmem_smem(size_t cells, size_t cell_bytes) {
  const size_t n = cells * cell_bytes;
  return n > 118 * 1024 ? n : 118 * 1024;
}

namespace {
// The tiling with the fewest cycles an iteration (16 a row of a warp, 3200 for each of the two sums'
// exchange when there is more than one tile); tiles at least 32 columns wide, where the mesh is, for the
// sake of the coefficients' loads.
// FP32, from 7 rows a thread on: the warps of the busiest of the SM's four schedulers count, so 12 or 16
// warps rather than 13.  By their sum the FP32 CG step at 1400^2 with jac_diag took 18.8 us, so it takes 16.9;
// Chebyshev solves there 35.3 and 31.9 ms, at 1999 x 1500 59.6 and 57.2.  Below, at 512^2, 10.0 and 10.1 us.
// FP64: their sum, as a CTA's FP64 work sets the time: k_persistent_cg_wide at 1000^2 22.8 us, by the busiest
// scheduler 24.3; k_persistent_poly_wide at 1200^2 with jac_diag 23.0 and 25.6 ms.
template <typename F>
bool rows_plan(int nx, int ny, int ctas, int threads, int max_rows, bool fp32, F&& smem, PersistPlan* out) {
  double best = 0.0;
  bool found = false;
  if (ctas > PERSIST_MAX_CTAS) ctas = PERSIST_MAX_CTAS;
  for (int g0 = 1; g0 <= ctas && g0 <= nx; ++g0) {
    const int tw = (nx + g0 - 1) / g0;
    if (tw > threads || (tw < 32 && g0 > 1)) continue;
    PersistPlan p{};
    p.tw = tw;
    p.gx = (nx + tw - 1) / tw;
    for (int many = 0; many < 2; ++many) {
      int gy = many ? ctas / p.gx : 1;
      if (gy > ny) gy = ny;
      if (gy < 1) continue;
      p.th = (ny + gy - 1) / gy;
      p.gy = (ny + p.th - 1) / p.th;
      p.ry = threads / tw < p.th ? threads / tw : p.th;
      p.rows = (p.th + p.ry - 1) / p.ry;
      p.variant = 0;
      const int halo = 2 * (p.tw + p.th);
      if (p.rows > max_rows || halo > PH * threads || smem(p) > PERSIST_SMEM_MAX) continue;
      int warps = (p.ry * tw + 31) / 32;
      if (fp32 && p.rows > 6) warps = (warps + 3) / 4 * 4;
      const double cost = (double)warps * p.rows * 16.0 + 0.5 * halo + (p.gx * p.gy > 1 ? 6400.0 : 0.0);
      if (!found || cost < best) {
        best = cost;
        *out = p;
        found = true;
      }
    }
  }
  return found;
}
}  // namespace

const PersistKernel kWideKernels[2] = {k_persistent_cg_wide<false>, k_persistent_cg_wide<true>};
size_t wide_plan_smem(const PersistPlan& p) {
  return tmem_smem((size_t)(p.th + 2) * (p.tw + 2) + (size_t)p.th * p.tw, sizeof(double));
}
const void* cg_kernel(const PersistPlan& p, int precond) {
  const int diag = precond == 2 ? 1 : 0;
  return p.variant == WIDE ? (const void*)kWideKernels[diag] : (const void*)kVariants[p.variant].k[diag];
}
size_t cg_smem(const PersistPlan& p) { return p.variant == WIDE ? wide_plan_smem(p) : plan_smem(p); }

// Plans the mesh for the current device; false if it does not fit on chip.
bool persist_prepare(int nx, int ny, int precond, PersistPlan* out) {
  const int ctas = coresident_ctas((const void*)kVariants[0].k[precond == 2 ? 1 : 0], PTHREADS, PERSIST_SMEM_MAX);
  if (!persist_plan(nx, ny, ctas, out)) {
    if (!rows_plan(nx, ny, ctas, PT, WROWS, false, wide_plan_smem, out)) return false;
    out->variant = WIDE;
  }
  return coresident_ctas(cg_kernel(*out, precond), PTHREADS, cg_smem(*out)) >= persist_ctas(*out);
}

cudaError_t launch_persistent_cg(const LoopArgs& a, const PersistPlan& p, int max_run, unsigned epoch, void* box,
                                 LoopState* st_host, unsigned* err, int fault, cudaStream_t s) {
  PersistArgs g{a, p, max_run, epoch, static_cast<ulonglong2*>(box), st_host, err, fault == 1 ? 1 : 0, fault == 3 ? 1 : -1};
  void* args[] = {&g};
  ++launch_counter();
  return cudaLaunchCooperativeKernel(cg_kernel(p, a.precond), dim3(persist_ctas(p)), dim3(PTHREADS), args, cg_smem(p), s);
}

namespace {

using MixPersistKernel = void (*)(MixPersistArgs);
const MixPersistKernel kMixKernels[2][2] = {{k_persistent_mix<false, 2>, k_persistent_mix<true, 2>},   // without / with
                                            {k_persistent_mix<false, 4>, k_persistent_mix<true, 4>}};  // jac_diag
// Groups of 4 rows, of 2 where a thread owns 6 at most (to about 700^2): 200 x 300 11.2 us against 11.5, 300
// x 400 10.6 / 10.7, 700^2 10.8 / 10.8; 900 x 950 11.9 / 11.6, 1300^2 15.3 / 14.5, 2048^2 22.6 / 21.3.
// Groups of 8 spill: 13.0 us at 200 x 300, 22.5 at 2048^2.
const void* mix_kernel(const PersistPlan& p, bool diag) { return (const void*)kMixKernels[p.rows > 6][diag]; }
size_t mix_plan_smem(const PersistPlan& p) {
  return tmem_smem((size_t)(p.th + 2) * (p.tw + 2) + (size_t)p.th * p.tw + 1, sizeof(float));
}

}  // namespace

bool mix_persist_prepare(int nx, int ny, int precond, PersistPlan* out) {
  const bool diag = precond == 2;
  const int ctas = coresident_ctas((const void*)kMixKernels[1][diag], PTHREADS, PERSIST_SMEM_MAX);
  if (!rows_plan(nx, ny, ctas, PT, MROWS, true, mix_plan_smem, out)) return false;
  return coresident_ctas(mix_kernel(*out, diag), PTHREADS, mix_plan_smem(*out)) >= persist_ctas(*out);
}

cudaError_t launch_persistent_mix(const MixFields& m, const Layout& L, MixState* ms, const PersistPlan& p, int max_run,
                                  unsigned epoch, void* box, unsigned* err, int fault, cudaStream_t s) {
  MixPersistArgs g{m, L, ms, p, max_run, epoch, static_cast<ulonglong2*>(box), err, fault == 1 ? 1 : 0, fault == 3 ? 1 : -1};
  void* args[] = {&g};
  ++launch_counter();
  return cudaLaunchCooperativeKernel(mix_kernel(p, m.mi != nullptr), dim3(persist_ctas(p)), dim3(PTHREADS), args,
                                     mix_plan_smem(p), s);
}


// ---- the FP64 polynomial steps on chip ----------------------------------------------------------
// The PPCG inner steps (tea_leaf_kernel_ppcg_inner, ppcg_kernel.f90:204-310) and the Chebyshev
// iterations (tea_leaf_kernel_cheby_iterate, cheby_kernel.f90:111-200) of a mesh that fits, many steps a
// launch.  Tiles, rims and the waits are those of the CG kernel above; the steps need no sum, so a step
// costs its FP64 work and one hop for the rim.  The stencil variable x (sd; u) with its halo, the face
// coefficients and Di are in shared memory, the cell's other two values (rtemp, utemp; u0, p) in
// registers.  Every product and sum is that of the one-step kernels, in their order; Di x and b times
// the residual run on the integer pipes, as in the staged sweeps of tl_fused.cu.  Same bits.
//
// A PPCG solve of 124 inner steps an outer iteration took, per inner step, 2.2 us at 60^2 against 13.6
// with a launch a step, 2.7 / 14.9 at 256^2, 5.8 / 15.0 at 512^2, 11.5 / 19.3 at 777 x 813 and 16.9 /
// 21.7 at 1000^2, where the FP64 pipe's share is 11; 332 Chebyshev iterations with their presteps 3.8
// against 14.4 us each at 128^2 and 21.9 against 24.7 at 1000^2.
namespace {

constexpr int QT = 512;  // threads per CTA, all of which own cells
enum { ON_PPCG = 0, ON_CHEBY = 1 };
struct PolyPersistArgs {
  Fields f;
  Layout L;
  PersistPlan pl;
  const double* x_in;             // u where it lies now (Chebyshev); the steps leave it in f.u
  const double *ch_a, *ch_b;      // coefficients of the first step ..
  int steps;
  unsigned epoch;                 // number of the first step's rims
  ulonglong2* box;                // halo boxes, by parity of the number
  unsigned* err;                  // set when a wait ran out: the results are void
  int hold;                       // test of the bounded wait: the first tile sends no rims
};

template <int M, int MODE, bool DIAG>
__global__ void __launch_bounds__(QT, 1) k_persistent_poly(PolyPersistArgs g) {
  constexpr bool PPCG = MODE == ON_PPCG;
  __shared__ int sh_fail;
  extern __shared__ __align__(16) double qsm[];
  const Layout L = g.L;
  const Fields& f = g.f;
  const int t = threadIdx.x;
  if (t == 0) sh_fail = *reinterpret_cast<volatile unsigned*>(g.err) != 0u;

  const int bx = blockIdx.x % g.pl.gx, by = blockIdx.x / g.pl.gx;
  const int j0 = bx * g.pl.tw, k0 = by * g.pl.th;
  const int tw = min(g.pl.tw, L.nx - j0), th = min(g.pl.th, L.ny - k0);
  const int P = g.pl.tw + 2, ry = g.pl.ry;
  const int asz = (g.pl.th + 2) * P;
  double* const sx = qsm;
  double* const scx = qsm + asz;
  double* const scy = qsm + 2 * asz;
  double* const sdi = qsm + 3 * asz;
  const double* const xin = PPCG ? f.sd : g.x_in;

  const int tx = t % g.pl.tw, ty = t / g.pl.tw;
  const int mine = (tx < tw && ty < ry && ty < th) ? (th - 1 - ty) / ry + 1 : 0;
  const int o0 = (ty + 1) * P + tx + 1;
  const int c0 = (int)L.at(j0 + tx + 1, k0 + ty + 1);
  const int ostep = ry * P, cstep = ry * L.ld;
  const int i_first = ty == 0 ? 0 : -1, i_last = (mine > 0 && (th - 1 - ty) % ry == 0) ? mine - 1 : -1;

  const int hbox = 2 * (g.pl.th + g.pl.tw), hall = (int)gridDim.x * hbox;
  int ho[PH], hh[PH];
#pragma unroll
  for (int q = 0; q < PH; ++q) {
    const int h = t + q * QT;
    ho[q] = -1;
    hh[q] = 0;
    int x = -1, y = h;
    bool in = y < th, is = in && j0 > 0;
    if (h >= g.pl.th) x = tw, y = h - g.pl.th, in = y < th, is = in && j0 + tw < L.nx;
    if (h >= 2 * g.pl.th) x = h - 2 * g.pl.th, y = -1, in = x < tw, is = in && k0 > 0;
    if (h >= 2 * g.pl.th + g.pl.tw) x = h - 2 * g.pl.th - g.pl.tw, y = th, in = x < tw, is = in && k0 + th < L.ny;
    if (in && h < hbox) {
      const int o = (y + 1) * P + x + 1;
      sx[o] = xin[L.at(j0 + x + 1, k0 + y + 1)];  // off the domain: the field's halo, which stays
      if (is) {
        ho[q] = o;
        hh[q] = (int)blockIdx.x * hbox + h;
      }
    }
  }
  const bool sends = !(g.hold && blockIdx.x == 0);
  const int to_l = (sends && tx == 0 && j0 > 0) ? ((int)blockIdx.x - 1) * hbox + g.pl.th + ty : -1;
  const int to_r = (sends && tx == tw - 1 && j0 + tw < L.nx) ? ((int)blockIdx.x + 1) * hbox + ty : -1;
  const int rim_b = sends && k0 > 0 ? i_first : -1, rim_t = sends && k0 + th < L.ny ? i_last : -1;
  const int to_b = ((int)blockIdx.x - g.pl.gx) * hbox + 2 * g.pl.th + g.pl.tw + tx;
  const int to_t = ((int)blockIdx.x + g.pl.gx) * hbox + 2 * g.pl.th + tx;

  double r[M], s[M];  // PPCG: rtemp, utemp; Chebyshev: u0 and then the residual of the step, p
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const int o = o0 + i * ostep, c = c0 + i * cstep;
    r[i] = s[i] = 0.0;
    if (i < mine) {
      sx[o] = xin[c];
      r[i] = PPCG ? f.rtemp[c] : f.u0[c];
      s[i] = PPCG ? f.utemp[c] : f.p[c];
      sdi[o] = f.di[c];
      scx[o] = f.cx[c];
      scy[o] = f.cy[c];
      if (tx == tw - 1) scx[o + 1] = f.cx[c + 1];
      if (i == i_last) scy[o + P] = f.cy[c + L.ld];
    }
  }
  __syncthreads();
  if (sh_fail) return;

  unsigned epoch = g.epoch;
  bool failed = false;
  for (int step = 0; step < g.steps; ++step, ++epoch) {
    const bool last = step + 1 == g.steps;
    const double ca = __ldg(g.ch_a + step), cb = __ldg(g.ch_b + step);
    ulonglong2* const halo = g.box + (size_t)(epoch & 1u) * hall;
    int o = fresh(o0), c = fresh(c0);
    // the residual of the owned cells (x is complete in shared memory)
#pragma unroll
    for (int i = 0; i < M; ++i, o += ostep, c += cstep) {
      if (i < mine) {
        double a = dmul_int(sdi[o], sx[o]);
        a = fma(-scy[o + P], sx[o + P], a);
        a = fma(-scy[o], sx[o - P], a);
        a = fma(-scx[o + 1], sx[o + 1], a);
        a = fma(-scx[o], sx[o - 1], a);
        const double res = r[i] - a;
        r[i] = res;
        if (!PPCG && last) {
          f.w[c] = a;
          f.r[c] = res;
        }
      }
    }
    __syncthreads();  // every read of x is done
    o = fresh(o0), c = fresh(c0);
    int l = fresh(to_l), e = fresh(to_r);
#pragma unroll
    for (int i = 0; i < M; ++i, o += ostep, c += cstep, l += ry, e += ry) {
      if (i < mine) {
        double z = r[i];
        if (DIAG) {
          z = __ldg(f.mi + c) * z;
          if (!PPCG && last) f.z[c] = z;
        }
        const double bz = dmul_int(cb, z);
        double x = sx[o];
        if (PPCG) {
          x = fma(ca, x, bz);
          s[i] = s[i] + x;
        } else {
          s[i] = fma(ca, s[i], bz);
          x = x + s[i];
          r[i] = __ldg(f.u0 + c);
        }
        sx[o] = x;
        if (to_l >= 0) box_put(halo + l, x, epoch);
        if (to_r >= 0) box_put(halo + e, x, epoch);
        if (i == rim_b) box_put(halo + to_b, x, epoch);
        if (i == rim_t) box_put(halo + to_t, x, epoch);
      }
    }
    if (!last) {
      bool got = false;
      double hv[PH];
      for (unsigned tries = 0; !got && tries < PERSIST_POLL_LIMIT; ++tries) {
        got = true;
#pragma unroll
        for (int q = 0; q < PH; ++q)
          if (ho[q] >= 0) {
            const ulonglong2 v = box_get(halo + hh[q]);
            got = got && box_is(v, epoch);
            hv[q] = box_value(v);
          }
      }
#pragma unroll
      for (int q = 0; q < PH; ++q)
        if (ho[q] >= 0) sx[ho[q]] = hv[q];
      if (!got) sh_fail = 1;
      __syncthreads();
      if (sh_fail) {
        failed = true;
        break;
      }
    }
  }
  if (failed) {
    if (t == 0) atomicExch(g.err, 1u);
    return;
  }
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const int o = o0 + i * ostep, c = c0 + i * cstep;
    if (i < mine) {
      if (PPCG) {
        f.sd[c] = sx[o];
        f.rtemp[c] = r[i];
        f.utemp[c] = s[i];
      } else {
        f.u[c] = sx[o];
        f.p[c] = s[i];
      }
    }
  }
}

using PolyPersistKernel = void (*)(PolyPersistArgs);
struct PolyPersistVariant {
  int m;
  PolyPersistKernel k[2][2];  // PPCG / Chebyshev, without / with jac_diag
};
#define POLY_VARIANT(M)                                                                      \
  {M,                                                                                        \
   {{k_persistent_poly<M, ON_PPCG, false>, k_persistent_poly<M, ON_PPCG, true>},             \
    {k_persistent_poly<M, ON_CHEBY, false>, k_persistent_poly<M, ON_CHEBY, true>}}}
// 14 cells of 512 threads are what the four arrays of shared memory hold (36 to 48 bytes spilled); the steps
// between keep the rows a tile is rounded up by below half of its own.
const PolyPersistVariant kPolyVariants[] = {POLY_VARIANT(1), POLY_VARIANT(2), POLY_VARIANT(4),
                                            POLY_VARIANT(7), POLY_VARIANT(10), POLY_VARIANT(14)};
size_t poly_plan_smem(const PersistPlan& p) { return (size_t)4 * (p.th + 2) * (p.tw + 2) * sizeof(double); }

// The tiling with the fewest cycles a step: 7 FP64 instructions of a warp a row (17 cycles of the SM's
// four pipes each), the halo, and the rim's hop (1500 cycles) when there is more than one tile.
bool poly_plan(int nx, int ny, int ctas, PersistPlan* out) {
  double best = 0.0;
  bool found = false;
  for (int g0 = 1; g0 <= ctas && g0 <= nx; ++g0) {
    const int tw = (nx + g0 - 1) / g0;
    if (tw > QT) continue;
    PersistPlan p{};
    p.tw = tw;
    p.gx = (nx + tw - 1) / tw;
    for (int many = 0; many < 2; ++many) {
      int gy = many ? ctas / p.gx : 1;
      if (gy > ny) gy = ny;
      if (gy < 1) continue;
      p.th = (ny + gy - 1) / gy;
      p.gy = (ny + p.th - 1) / p.th;
      p.ry = QT / tw < p.th ? QT / tw : p.th;
      const int m = (p.th + p.ry - 1) / p.ry;
      p.variant = -1;
      for (int v = (int)(sizeof(kPolyVariants) / sizeof(kPolyVariants[0])) - 1; v >= 0; --v)
        if (kPolyVariants[v].m >= m) p.variant = v;
      const int halo = 2 * (p.tw + p.th);
      if (p.variant < 0 || halo > PH * QT || poly_plan_smem(p) > PERSIST_SMEM_MAX) continue;
      const double cost =
          (double)((p.ry * tw + 31) / 32) * m * 119.0 + 0.5 * halo + 4.0 * p.th + (p.gx * p.gy > 1 ? 1500.0 : 0.0);
      if (!found || cost < best) {
        best = cost;
        *out = p;
        found = true;
      }
    }
  }
  return found;
}

}  // namespace

// ---- the FP32 polynomial steps of the precision form on chip ------------------------------------
// The PPCG inner steps and the Chebyshev iterations on a correction (tl_mixed_poly.cu) of a mesh that
// fits, all of an outer iteration's or a cycle's steps in one launch.  Tiles, groups of rows and the
// coefficients' way from L2 are k_persistent_mix's, the rims' way k_persistent_poly's.  The stencil
// variable x (sd; d) has two buffers with halo in shared memory, so that a step reads one and writes the
// other and needs one barrier; the cell's other two values (rtemp, utemp; p, the right-hand side) are in
// tensor memory.  8 bytes a cell in shared memory take meshes of up to about 2040^2.  Every product and
// sum is that of the one-step kernels, in their order: same bits.
//
// A Chebyshev cycle's step took about 7 us at 1999 x 1500 against 15 in the blocked sweeps (four steps a
// pass over the fields), bound by the coefficients' way from L2.  Whole solves, CG presteps included,
// against the blocked sweeps: Chebyshev 200 x 300 3.8 ms against 10.4, 512^2 7.2 / 20.6, 1000^2 19.0 /
// 42.6, 1999 x 1500 56.6 / 94.8, 2040^2 82 / 118; PPCG with 10 inner steps 512^2 11.1 / 21.3, 1000^2 28.0 /
// 43.6, 1999 x 1500 77.4 / 94.7 (5 inner steps 103 / 120), 2040^2 with 20 inner steps 91 / 105.  Every mesh
// that fits runs here.
namespace {

constexpr int YC = 4;  // rows handled together
struct MixPolyArgs {
  MixFields m;
  Layout L;
  PersistPlan pl;
  const double* r64;          // PPCG: the FP64 residual the steps start from (Chebyshev: m.r)
  double* z;                  // PPCG: utemp after the last step
  float inv_theta;
  const double *ch_a, *ch_b;  // coefficients of the first step ..
  int steps;
  unsigned epoch;             // number of the first step's rims
  unsigned long long* box;    // halo boxes, by parity of the number
  unsigned* err;              // set when a wait ran out: the results are void
  int hold;                   // test of the bounded wait: the first tile sends no rims
};

__device__ __forceinline__ void tmem_get2(unsigned a, float (&v)[4], unsigned b, float (&w)[4]) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%8];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4, %5, %6, %7}, [%9];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3])
      : "r"(a), "r"(b)
      : "memory");
}

template <int MODE, bool DIAG>
__global__ void __launch_bounds__(QT, 1) k_persistent_mix_poly(MixPolyArgs g) {
  constexpr bool PPCG = MODE == ON_PPCG;
  __shared__ int sh_fail;
  __shared__ unsigned sh_tmem;
  extern __shared__ __align__(16) float ysm[];
  const Layout L = g.L;
  const MixFields& f = g.m;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  if (t == 0) sh_fail = *reinterpret_cast<volatile unsigned*>(g.err) != 0u;
  __syncthreads();
  if (sh_fail) return;
  if (wid == 0) tmem_alloc(&sh_tmem);

  const int bx = blockIdx.x % g.pl.gx, by = blockIdx.x / g.pl.gx;
  const int j0 = bx * g.pl.tw, k0 = by * g.pl.th;
  const int tw = min(g.pl.tw, L.nx - j0), th = min(g.pl.th, L.ny - k0);
  const int P = g.pl.tw + 2, asz = (g.pl.th + 2) * P;
  const int oz = 2 * asz;  // a cell of zeros, for the lanes and rows without a cell

  // the thread's column and rows y0 .. y0+mine-1, split evenly
  const int tx = t % g.pl.tw, seg = t / g.pl.tw;
  const int q_ = th / g.pl.ry, rem = th - q_ * g.pl.ry;
  const int mine = (tx < tw && seg < g.pl.ry) ? q_ + (seg < rem) : 0, y0 = seg * q_ + min(seg, rem);
  const int own = mine ? mine : q_ + (rem > 0);
  const bool warp_owns = __any_sync(0xffffffffu, mine > 0);
  const int nfull = warp_owns ? (int)__reduce_min_sync(0xffffffffu, (unsigned)own) / YC : 0;  // groups of YC rows
  const int nch = warp_owns ? ((int)__reduce_max_sync(0xffffffffu, (unsigned)own) + YC - 1) / YC : 0;
  const int o0 = mine ? (y0 + 1) * P + tx + 1 : oz, o_next = mine ? asz : 0;  // in the first buffer; to the second
  const int c0 = mine ? (int)L.at(j0 + tx + 1, k0 + y0 + 1) : (int)L.at(j0 + 1, k0 + 1);
  const int ld = L.ld, os = mine ? P : 0, cs = mine ? ld : 0;
  const bool at_l = tx == 0 && j0 == 0, at_r = tx == tw - 1 && j0 + tw == L.nx;
  // the neighbours' offsets: PPCG's sd is mirrored at a wall, the correction is zero outside
  const int lo = ((PPCG && at_l) || !mine) ? 0 : -1, ro = ((PPCG && at_r) || !mine) ? 0 : 1;
  const int i_first = (mine > 0 && y0 == 0) ? 0 : -1, i_last = (mine > 0 && y0 + mine == th) ? mine - 1 : -1;
  const int i_b = PPCG && k0 == 0 ? i_first : -1, i_t = PPCG && k0 + th == L.ny ? i_last : -1;

  // the start's value of a cell: z / theta
  auto start = [&](int c) {
    const float rv = PPCG ? (float)g.r64[c] : f.r[c];
    return (DIAG ? f.mi[c] * rv : rv) * g.inv_theta;
  };
  const int hbox = 2 * (g.pl.th + g.pl.tw), hall = (int)gridDim.x * hbox;
  int ho[PH], hh[PH];
#pragma unroll
  for (int q = 0; q < PH; ++q) {
    const int h = t + q * QT;
    ho[q] = -1;
    hh[q] = 0;
    int x = -1, y = h;
    bool in = y < th, is = in && j0 > 0;
    if (h >= g.pl.th) x = tw, y = h - g.pl.th, in = y < th, is = in && j0 + tw < L.nx;
    if (h >= 2 * g.pl.th) x = h - 2 * g.pl.th, y = -1, in = x < tw, is = in && k0 > 0;
    if (h >= 2 * g.pl.th + g.pl.tw) x = h - 2 * g.pl.th - g.pl.tw, y = th, in = x < tw, is = in && k0 + th < L.ny;
    if (in && h < hbox) {
      const int o = (y + 1) * P + x + 1;
      // off the domain: zero (a mirrored row is written with its cells)
      const bool mirror = PPCG && !is;
      if (!mirror) ysm[o] = is ? start((int)L.at(j0 + x + 1, k0 + y + 1)) : 0.f;
      if (!mirror && !is) ysm[asz + o] = 0.f;
      if (is) {
        ho[q] = o;
        hh[q] = (int)blockIdx.x * hbox + h;
      }
    }
  }
  const bool sends = !(g.hold && blockIdx.x == 0);
  const int to_l = (sends && mine && tx == 0 && j0 > 0) ? ((int)blockIdx.x - 1) * hbox + g.pl.th + y0 : -1;
  const int to_r = (sends && mine && tx == tw - 1 && j0 + tw < L.nx) ? ((int)blockIdx.x + 1) * hbox + y0 : -1;
  const int rim_b = sends && k0 > 0 ? i_first : -1, rim_t = sends && k0 + th < L.ny ? i_last : -1;
  const int to_b = ((int)blockIdx.x - g.pl.gx) * hbox + 2 * g.pl.th + g.pl.tw + tx;
  const int to_t = ((int)blockIdx.x + g.pl.gx) * hbox + 2 * g.pl.th + tx;

  __syncthreads();
  // this thread's words of tensor memory: rtemp / p, then utemp / the right-hand side
  const unsigned ta = sh_tmem + ((unsigned)(wid & 3) << 21) + (unsigned)(wid >> 2) * (2 * MROWS), tb = ta + MROWS;
  if (t == 0) ysm[oz] = 0.f;
  for (int ch = 0; ch < nch; ++ch) {
    float a[YC], b[YC];
#pragma unroll
    for (int j = 0; j < YC; ++j) {
      const int i = ch * YC + j, c = c0 + i * cs;
      a[j] = b[j] = 0.f;
      if (i < mine) {
        const float x = start(c);
        ysm[o0 + i * os] = x;
        a[j] = PPCG ? (float)g.r64[c] : x;
        b[j] = PPCG ? x : f.r[c];
        if (i == i_b) ysm[o0 + i * os - P] = x;
        if (i == i_t) ysm[o0 + i * os + P] = x;
      }
    }
    tmem_put(ta + ch * YC, a);
    tmem_put(tb + ch * YC, b);
  }
  tmem_put_done();

  struct Coefs {
    float di[YC], cl[YC], cr[YC], ct[YC], mi[YC];  // Di, the left, right and upper face, Mi of a group of rows
  } ka, kb;
  const std::true_type full;
  const std::false_type part;
  auto load_group = [&](int ch, Coefs& k, auto f_) {
    const int left = own - ch * YC, c1 = decltype(f_)::value || left > 0 ? c0 + ch * YC * cs : c0;
    const float *pd = f.di + c1, *px = f.cx + c1, *py = f.cy + c1 + ld, *pm = DIAG ? f.mi + c1 : nullptr;
#pragma unroll
    for (int j = 0; j < YC; ++j) {
      k.di[j] = __ldg(pd);
      k.cl[j] = __ldg(px);
      k.cr[j] = __ldg(px + 1);
      k.ct[j] = __ldg(py);
      if (DIAG) k.mi[j] = __ldg(pm);
      if (decltype(f_)::value || j + 1 < left) {
        pd += cs, px += cs, py += cs;
        if (DIAG) pm += cs;
      }
    }
  };
  auto load_coefs = [&](int ch, Coefs& k) {
    if (ch < nfull) load_group(ch, k, full);
    else if (ch < nch) load_group(ch, k, part);
  };
  load_coefs(0, ka);
  __syncthreads();

  unsigned epoch = g.epoch;
  bool failed = false;
  int cur = 0, nxt = o_next;  // the buffers' offsets, of this thread's cells
  int bufn = asz;             // the written buffer's, of the tile's
  for (int step = 0; step < g.steps; ++step, ++epoch) {
    const bool last = step + 1 == g.steps;
    const float ca = (float)__ldg(g.ch_a + step), cb = (float)__ldg(g.ch_b + step);
    unsigned long long* const halo = g.box + (size_t)(epoch & 1u) * hall;
    {
      float pb = 0.f, pc = 0.f, cyb = 0.f;
      if (nch > 0) pb = ysm[cur + o0 - os], pc = ysm[cur + o0], cyb = __ldg(f.cy + c0);
      auto rows_of = [&](int ch, const Coefs& k, auto f_) {
        const int o = o0 + ch * YC * os, left = own - ch * YC;
        float xl[YC], xr[YC], xt[YC], a[YC], b[YC];
        // a group's loads before its stores
#pragma unroll
        for (int j = 0; j < YC; ++j) {
          const bool in = decltype(f_)::value || j < left;
          xt[j] = ysm[in ? cur + o + (j + 1) * os : oz];
          xr[j] = ysm[in ? cur + o + j * os + ro : oz];
          xl[j] = ysm[in ? cur + o + j * os + lo : oz];
        }
        tmem_get2(ta + ch * YC, a, tb + ch * YC, b);
#pragma unroll
        for (int j = 0; j < YC; ++j) {
          const bool in = decltype(f_)::value || j < left;
          if (!in) pb = pc = 0.f;
          float v = k.di[j] * pc;
          v = fmaf(-k.ct[j], xt[j], v);
          v = fmaf(-cyb, pb, v);
          v = fmaf(-k.cr[j], xr[j], v);
          v = fmaf(-k.cl[j], xl[j], v);
          const float res = (PPCG ? a[j] : b[j]) - v;
          const float bz = cb * (DIAG ? k.mi[j] * res : res);
          float x;
          if (PPCG) {
            a[j] = res;
            x = fmaf(ca, pc, bz);
            b[j] = b[j] + x;
          } else {
            a[j] = fmaf(ca, a[j], bz);
            x = pc + a[j];
          }
          ysm[in ? nxt + o + j * os : oz] = in ? x : 0.f;
          pb = pc;
          pc = xt[j];
          cyb = k.ct[j];
        }
        tmem_put(ta + ch * YC, a);
        if (PPCG) tmem_put(tb + ch * YC, b);
      };
      auto rows = [&](int ch, const Coefs& k) {
        if (ch < nfull) rows_of(ch, k, full);
        else if (ch < nch) rows_of(ch, k, part);
      };
      // two groups of coefficients: the next one's loads are in flight while one is used
      for (int ch = 0; ch < nch; ch += 2) {
        load_coefs(ch + 1, kb);
        rows(ch, ka);
        load_coefs(ch + 2, ka);
        rows(ch + 1, kb);
      }
      tmem_put_done();
    }
    if (!last) {
      // the rim: a column's rows are its owner's, and the whole warp sends them
      if (i_b >= 0) ysm[nxt + o0 - P] = ysm[nxt + o0];
      if (i_t >= 0) ysm[nxt + o0 + mine * P] = ysm[nxt + o0 + (mine - 1) * P];
      if (rim_b >= 0) fbox_put(halo + to_b, ysm[nxt + o0 + rim_b * P], epoch);
      if (rim_t >= 0) fbox_put(halo + to_t, ysm[nxt + o0 + rim_t * P], epoch);
      __syncwarp();
      auto columns = [&](int to_) {
        for (unsigned m = __ballot_sync(0xffffffffu, to_ >= 0); m; m &= m - 1) {
          const int l = __ffs(m) - 1;
          const int h = __shfl_sync(0xffffffffu, to_, l), o1 = __shfl_sync(0xffffffffu, nxt + o0, l),
                    have = __shfl_sync(0xffffffffu, mine, l);
          for (int i = lane; i < have; i += 32) fbox_put(halo + h + i, ysm[o1 + i * P], epoch);
        }
      };
      columns(to_l);
      columns(to_r);
      load_coefs(0, ka);
      bool got = false;
      float hv[PH];
      for (unsigned tries = 0; !got && tries < PERSIST_POLL_LIMIT; ++tries) {
        got = true;
#pragma unroll
        for (int q = 0; q < PH; ++q)
          if (ho[q] >= 0) {
            const unsigned long long v = fbox_get(halo + hh[q]);
            got = got && (unsigned)v == epoch;
            hv[q] = __uint_as_float((unsigned)(v >> 32));
          }
      }
#pragma unroll
      for (int q = 0; q < PH; ++q)
        if (ho[q] >= 0) ysm[bufn + ho[q]] = hv[q];
      if (!got) sh_fail = 1;
      __syncthreads();
      if (sh_fail) {
        failed = true;
        break;
      }
    }
    const int swap = cur;
    cur = nxt;
    nxt = swap;
    bufn = asz - bufn;
  }
  for (int ch = 0; ch < (failed ? 0 : nch); ++ch) {
    float b[YC];
    if (PPCG) tmem_get(tb + ch * YC, b);
#pragma unroll
    for (int j = 0; j < YC; ++j) {
      const int i = ch * YC + j, c = c0 + i * cs;
      if (i < mine) {
        if (PPCG) g.z[c] = (double)b[j];
        else f.d[c] = ysm[cur + o0 + i * os];
      }
    }
  }
  __syncthreads();  // every warp is done with tensor memory
  if (wid == 0) tmem_free(sh_tmem);
  if (failed && t == 0) atomicExch(g.err, 1u);
}

// ---- the FP64 polynomial steps of larger tiles ---------------------------------------------------
// k_persistent_poly's steps laid out as k_persistent_mix_poly: two buffers of the stencil variable in shared
// memory, rtemp and utemp (p and u0) in tensor memory, the coefficients from L2.  Same bits.
// It runs where k_persistent_poly's tiles do not fit (about a million cells), to about 1400^2: 900 inner steps
// of 18 PPCG outer iterations took 22.0 ms at 1100^2 against 24.3 as sweeps in memory, 30.4 / 33.0 at 1400^2,
// 23.0 / 34.0 at 1200^2 with jac_diag, 402 Chebyshev iterations 11.5 / 12.4, 15.9 / 16.6 and 12.2 / 20.1.  At
// 1000^2 the two are even (17.0 and 16.9 ms), at 700^2 k_persistent_poly leads (10.4 and 9.3).  The FP64 pipe
// bounds it: 7 instructions a cell and step.
constexpr int VC = 2;  // rows handled together
__device__ __forceinline__ void tmem_put(unsigned a, const double (&v)[2]) {
  float w[4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    w[2 * i] = __int_as_float(__double2loint(v[i]));
    w[2 * i + 1] = __int_as_float(__double2hiint(v[i]));
  }
  tmem_put(a, w);
}
__device__ __forceinline__ void tmem_get2(unsigned a, double (&v)[2], unsigned b, double (&w)[2]) {
  float x[4], y[4];
  tmem_get2(a, x, b, y);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    v[i] = __hiloint2double(__float_as_int(x[2 * i + 1]), __float_as_int(x[2 * i]));
    w[i] = __hiloint2double(__float_as_int(y[2 * i + 1]), __float_as_int(y[2 * i]));
  }
}

template <int MODE, bool DIAG>
__global__ void __launch_bounds__(QT, 1) k_persistent_poly_wide(PolyPersistArgs g) {
  constexpr bool PPCG = MODE == ON_PPCG;
  __shared__ int sh_fail;
  __shared__ unsigned sh_tmem;
  extern __shared__ __align__(16) double vsm[];
  const Layout L = g.L;
  const Fields& f = g.f;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  if (t == 0) sh_fail = *reinterpret_cast<volatile unsigned*>(g.err) != 0u;
  __syncthreads();
  if (sh_fail) return;
  if (wid == 0) tmem_alloc(&sh_tmem);

  const int bx = blockIdx.x % g.pl.gx, by = blockIdx.x / g.pl.gx;
  const int j0 = bx * g.pl.tw, k0 = by * g.pl.th;
  const int tw = min(g.pl.tw, L.nx - j0), th = min(g.pl.th, L.ny - k0);
  const int P = g.pl.tw + 2, asz = (g.pl.th + 2) * P;
  const int oz = 2 * asz;  // a cell of zeros, for the lanes and rows without a cell

  // the thread's column and rows y0 .. y0+mine-1, split evenly
  const int tx = t % g.pl.tw, seg = t / g.pl.tw;
  const int q_ = th / g.pl.ry, rem = th - q_ * g.pl.ry;
  const int mine = (tx < tw && seg < g.pl.ry) ? q_ + (seg < rem) : 0, y0 = seg * q_ + min(seg, rem);
  const int own = mine ? mine : q_ + (rem > 0);
  const bool warp_owns = __any_sync(0xffffffffu, mine > 0);
  const int nfull = warp_owns ? (int)__reduce_min_sync(0xffffffffu, (unsigned)own) / VC : 0;  // groups of VC rows
  const int nch = warp_owns ? ((int)__reduce_max_sync(0xffffffffu, (unsigned)own) + VC - 1) / VC : 0;
  const int o0 = mine ? (y0 + 1) * P + tx + 1 : oz, o_next = mine ? asz : 0;  // in the first buffer; to the second
  const int c0 = mine ? (int)L.at(j0 + tx + 1, k0 + y0 + 1) : (int)L.at(j0 + 1, k0 + 1);
  const int ld = L.ld, os = mine ? P : 0, cs = mine ? ld : 0;
  const int lo = mine ? -1 : 0, ro = mine ? 1 : 0;  // the neighbours' offsets
  const int i_first = (mine > 0 && y0 == 0) ? 0 : -1, i_last = (mine > 0 && y0 + mine == th) ? mine - 1 : -1;

  const double* const xin = PPCG ? f.sd : g.x_in;
  const int hbox = 2 * (g.pl.th + g.pl.tw), hall = (int)gridDim.x * hbox;
  int ho[PH], hh[PH];
#pragma unroll
  for (int q = 0; q < PH; ++q) {
    const int h = t + q * QT;
    ho[q] = -1;
    hh[q] = 0;
    int x = -1, y = h;
    bool in = y < th, is = in && j0 > 0;
    if (h >= g.pl.th) x = tw, y = h - g.pl.th, in = y < th, is = in && j0 + tw < L.nx;
    if (h >= 2 * g.pl.th) x = h - 2 * g.pl.th, y = -1, in = x < tw, is = in && k0 > 0;
    if (h >= 2 * g.pl.th + g.pl.tw) x = h - 2 * g.pl.th - g.pl.tw, y = th, in = x < tw, is = in && k0 + th < L.ny;
    if (in && h < hbox) {
      const int o = (y + 1) * P + x + 1;
      vsm[o] = vsm[asz + o] = xin[L.at(j0 + x + 1, k0 + y + 1)];  // off the domain: the field's halo, which stays
      if (is) {
        ho[q] = o;
        hh[q] = (int)blockIdx.x * hbox + h;
      }
    }
  }
  const bool sends = !(g.hold && blockIdx.x == 0);
  const int to_l = (sends && mine && tx == 0 && j0 > 0) ? ((int)blockIdx.x - 1) * hbox + g.pl.th + y0 : -1;
  const int to_r = (sends && mine && tx == tw - 1 && j0 + tw < L.nx) ? ((int)blockIdx.x + 1) * hbox + y0 : -1;
  const int rim_b = sends && k0 > 0 ? i_first : -1, rim_t = sends && k0 + th < L.ny ? i_last : -1;
  const int to_b = ((int)blockIdx.x - g.pl.gx) * hbox + 2 * g.pl.th + g.pl.tw + tx;
  const int to_t = ((int)blockIdx.x + g.pl.gx) * hbox + 2 * g.pl.th + tx;

  __syncthreads();
  // this thread's words of tensor memory: rtemp / p, then utemp / u0
  const unsigned ta = sh_tmem + ((unsigned)(wid & 3) << 21) + (unsigned)(wid >> 2) * 128u, tb = ta + 2 * WROWS;
  if (t == 0) vsm[oz] = 0.0;
  for (int ch = 0; ch < nch; ++ch) {
    double a[VC], b[VC];
#pragma unroll
    for (int j = 0; j < VC; ++j) {
      const int i = ch * VC + j, c = c0 + i * cs;
      a[j] = b[j] = 0.0;
      if (i < mine) {
        vsm[o0 + i * os] = xin[c];
        a[j] = PPCG ? f.rtemp[c] : f.p[c];
        b[j] = PPCG ? f.utemp[c] : f.u0[c];
      }
    }
    tmem_put(ta + ch * 2 * VC, a);
    tmem_put(tb + ch * 2 * VC, b);
  }
  tmem_put_done();

  struct Coefs {
    double di[VC], cl[VC], cr[VC], ct[VC], mi[VC];  // Di, the left, right and upper face, Mi of a group of rows
  } ka, kb;
  const std::true_type full;
  const std::false_type part;
  auto load_group = [&](int ch, Coefs& k, auto f_) {
    const int left = own - ch * VC, c1 = decltype(f_)::value || left > 0 ? c0 + ch * VC * cs : c0;
    const double *pd = f.di + c1, *px = f.cx + c1, *py = f.cy + c1 + ld, *pm = DIAG ? f.mi + c1 : nullptr;
#pragma unroll
    for (int j = 0; j < VC; ++j) {
      k.di[j] = __ldg(pd);
      k.cl[j] = __ldg(px);
      k.cr[j] = __ldg(px + 1);
      k.ct[j] = __ldg(py);
      if (DIAG) k.mi[j] = __ldg(pm);
      if (decltype(f_)::value || j + 1 < left) {
        pd += cs, px += cs, py += cs;
        if (DIAG) pm += cs;
      }
    }
  };
  auto load_coefs = [&](int ch, Coefs& k) {
    if (ch < nfull) load_group(ch, k, full);
    else if (ch < nch) load_group(ch, k, part);
  };
  load_coefs(0, ka);
  __syncthreads();

  unsigned epoch = g.epoch;
  bool failed = false;
  int cur = 0, nxt = o_next;  // the buffers' offsets, of this thread's cells
  int bufn = asz;             // the written buffer's, of the tile's
  for (int step = 0; step < g.steps; ++step, ++epoch) {
    const bool last = step + 1 == g.steps;
    const double ca = __ldg(g.ch_a + step), cb = __ldg(g.ch_b + step);
    ulonglong2* const halo = g.box + (size_t)(epoch & 1u) * hall;
    {
      double pb = 0.0, pc = 0.0, cyb = 0.0;
      if (nch > 0) pb = vsm[cur + o0 - os], pc = vsm[cur + o0], cyb = __ldg(f.cy + c0);
      auto rows_of = [&](int ch, const Coefs& k, auto f_) {
        const int o = o0 + ch * VC * os, left = own - ch * VC;
        double xl[VC], xr[VC], xt[VC], a[VC], b[VC];
        // a group's loads before its stores
#pragma unroll
        for (int j = 0; j < VC; ++j) {
          const bool in = decltype(f_)::value || j < left;
          xt[j] = vsm[in ? cur + o + (j + 1) * os : oz];
          xr[j] = vsm[in ? cur + o + j * os + ro : oz];
          xl[j] = vsm[in ? cur + o + j * os + lo : oz];
        }
        tmem_get2(ta + ch * 2 * VC, a, tb + ch * 2 * VC, b);
#pragma unroll
        for (int j = 0; j < VC; ++j) {
          const bool in = decltype(f_)::value || j < left;
          if (!in) pb = pc = 0.0;
          double v = dmul_int(k.di[j], pc);
          v = fma(-k.ct[j], xt[j], v);
          v = fma(-cyb, pb, v);
          v = fma(-k.cr[j], xr[j], v);
          v = fma(-k.cl[j], xl[j], v);
          const double res = (PPCG ? a[j] : b[j]) - v;
          const double z = DIAG ? k.mi[j] * res : res;
          if (!PPCG && last && in && mine) {
            const int c = c0 + (ch * VC + j) * cs;
            f.w[c] = v;
            f.r[c] = res;
            if (DIAG) f.z[c] = z;
          }
          const double bz = dmul_int(cb, z);
          double x;
          if (PPCG) {
            a[j] = res;
            x = fma(ca, pc, bz);
            b[j] = b[j] + x;
          } else {
            a[j] = fma(ca, a[j], bz);
            x = pc + a[j];
          }
          vsm[in ? nxt + o + j * os : oz] = in ? x : 0.0;
          pb = pc;
          pc = xt[j];
          cyb = k.ct[j];
        }
        tmem_put(ta + ch * 2 * VC, a);
        if (PPCG) tmem_put(tb + ch * 2 * VC, b);
      };
      auto rows = [&](int ch, const Coefs& k) {
        if (ch < nfull) rows_of(ch, k, full);
        else if (ch < nch) rows_of(ch, k, part);
      };
      // two groups of coefficients: the next one's loads are in flight while one is used
      for (int ch = 0; ch < nch; ch += 2) {
        load_coefs(ch + 1, kb);
        rows(ch, ka);
        load_coefs(ch + 2, ka);
        rows(ch + 1, kb);
      }
      tmem_put_done();
    }
    if (!last) {
      // the rim: a column's rows are its owner's, and the whole warp sends them
      if (rim_b >= 0) box_put(halo + to_b, vsm[nxt + o0 + rim_b * P], epoch);
      if (rim_t >= 0) box_put(halo + to_t, vsm[nxt + o0 + rim_t * P], epoch);
      __syncwarp();
      auto columns = [&](int to_) {
        for (unsigned m = __ballot_sync(0xffffffffu, to_ >= 0); m; m &= m - 1) {
          const int l = __ffs(m) - 1;
          const int h = __shfl_sync(0xffffffffu, to_, l), o1 = __shfl_sync(0xffffffffu, nxt + o0, l),
                    have = __shfl_sync(0xffffffffu, mine, l);
          for (int i = lane; i < have; i += 32) box_put(halo + h + i, vsm[o1 + i * P], epoch);
        }
      };
      columns(to_l);
      columns(to_r);
      load_coefs(0, ka);
      bool got = false;
      double hv[PH];
      for (unsigned tries = 0; !got && tries < PERSIST_POLL_LIMIT; ++tries) {
        got = true;
#pragma unroll
        for (int q = 0; q < PH; ++q)
          if (ho[q] >= 0) {
            const ulonglong2 v = box_get(halo + hh[q]);
            got = got && box_is(v, epoch);
            hv[q] = box_value(v);
          }
      }
#pragma unroll
      for (int q = 0; q < PH; ++q)
        if (ho[q] >= 0) vsm[bufn + ho[q]] = hv[q];
      if (!got) sh_fail = 1;
      __syncthreads();
      if (sh_fail) {
        failed = true;
        break;
      }
    }
    const int swap = cur;
    cur = nxt;
    nxt = swap;
    bufn = asz - bufn;
  }
  for (int ch = 0; ch < (failed ? 0 : nch); ++ch) {
    double a[VC], b[VC];
    tmem_get2(ta + ch * 2 * VC, a, tb + ch * 2 * VC, b);
#pragma unroll
    for (int j = 0; j < VC; ++j) {
      const int i = ch * VC + j, c = c0 + i * cs;
      if (i < mine) {
        const double x = vsm[cur + o0 + i * os];
        if (PPCG) {
          f.sd[c] = x;
          f.rtemp[c] = a[j];
          f.utemp[c] = b[j];
        } else {
          f.u[c] = x;
          f.p[c] = a[j];
        }
      }
    }
  }
  __syncthreads();  // every warp is done with tensor memory
  if (wid == 0) tmem_free(sh_tmem);
  if (failed && t == 0) atomicExch(g.err, 1u);
}

using MixPolyKernel = void (*)(MixPolyArgs);
const MixPolyKernel kMixPolyKernels[2][2] = {  // PPCG / Chebyshev, without / with jac_diag
    {k_persistent_mix_poly<ON_PPCG, false>, k_persistent_mix_poly<ON_PPCG, true>},
    {k_persistent_mix_poly<ON_CHEBY, false>, k_persistent_mix_poly<ON_CHEBY, true>}};
const PolyPersistKernel kPolyWideKernels[2][2] = {  // PPCG / Chebyshev, without / with jac_diag
    {k_persistent_poly_wide<ON_PPCG, false>, k_persistent_poly_wide<ON_PPCG, true>},
    {k_persistent_poly_wide<ON_CHEBY, false>, k_persistent_poly_wide<ON_CHEBY, true>}};
size_t poly_wide_plan_smem(const PersistPlan& p) {
  return tmem_smem((size_t)2 * (p.th + 2) * (p.tw + 2) + 1, sizeof(double));
}
size_t mix_poly_plan_smem(const PersistPlan& p) {
  return tmem_smem((size_t)2 * (p.th + 2) * (p.tw + 2) + 1, sizeof(float));
}

}  // namespace

bool poly_persist_prepare(int nx, int ny, int precond, PersistPlan* out) {
  const int diag = precond == 2 ? 1 : 0;
  const int ctas = coresident_ctas((const void*)kPolyVariants[0].k[0][diag], QT, PERSIST_SMEM_MAX);
  bool fits = poly_plan(nx, ny, ctas, out);
  for (int mode = 0; mode < 2 && fits; ++mode)
    fits = coresident_ctas((const void*)kPolyVariants[out->variant].k[mode][diag], QT, poly_plan_smem(*out)) >= persist_ctas(*out);
  if (fits) return true;
  const int wide = coresident_ctas((const void*)kPolyWideKernels[0][diag], QT, PERSIST_SMEM_MAX);
  if (!rows_plan(nx, ny, wide, QT, WROWS, false, poly_wide_plan_smem, out)) return false;
  out->variant = WIDE;
  for (int mode = 0; mode < 2; ++mode)
    if (coresident_ctas((const void*)kPolyWideKernels[mode][diag], QT, poly_wide_plan_smem(*out)) < persist_ctas(*out))
      return false;
  return true;
}

cudaError_t launch_persistent_poly(const Fields& f, const Layout& L, const PersistPlan& p, bool ppcg, bool diag,
                                   const double* u_in, const double* ch_a, const double* ch_b, int steps,
                                   unsigned epoch, void* box, unsigned* err, bool hold, cudaStream_t s) {
  PolyPersistArgs g{f, L, p, u_in, ch_a, ch_b, steps, epoch, static_cast<ulonglong2*>(box), err, hold ? 1 : 0};
  void* args[] = {&g};
  ++launch_counter();
  const int mode = ppcg ? 0 : 1, d = diag ? 1 : 0;
  if (p.variant == WIDE)
    return cudaLaunchCooperativeKernel((const void*)kPolyWideKernels[mode][d], dim3(persist_ctas(p)), dim3(QT), args,
                                       poly_wide_plan_smem(p), s);
  return cudaLaunchCooperativeKernel((const void*)kPolyVariants[p.variant].k[mode][d], dim3(persist_ctas(p)), dim3(QT),
                                     args, poly_plan_smem(p), s);
}

bool mix_poly_persist_prepare(int nx, int ny, int precond, PersistPlan* out) {
  const int diag = precond == 2 ? 1 : 0;
  const int ctas = coresident_ctas((const void*)kMixPolyKernels[0][diag], QT, PERSIST_SMEM_MAX);
  if (!rows_plan(nx, ny, ctas, QT, MROWS, true, mix_poly_plan_smem, out)) return false;
  for (int mode = 0; mode < 2; ++mode)
    if (coresident_ctas((const void*)kMixPolyKernels[mode][diag], QT, mix_poly_plan_smem(*out)) < persist_ctas(*out))
      return false;
  return true;
}

cudaError_t launch_persistent_mix_poly(const MixFields& m, const Layout& L, const PersistPlan& p, bool ppcg,
                                       const double* r64, double* z, double theta, const double* ch_a,
                                       const double* ch_b, int steps, unsigned epoch, void* box, unsigned* err,
                                       bool hold, cudaStream_t s) {
  MixPolyArgs g{m, L, p, r64, z, (float)(1.0 / theta), ch_a, ch_b, steps, epoch,
                static_cast<unsigned long long*>(box), err, hold ? 1 : 0};
  void* args[] = {&g};
  ++launch_counter();
  return cudaLaunchCooperativeKernel((const void*)kMixPolyKernels[ppcg ? 0 : 1][m.mi ? 1 : 0], dim3(persist_ctas(p)),
                                     dim3(QT), args, mix_poly_plan_smem(p), s);
}

}  // namespace tl
