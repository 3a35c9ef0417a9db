// krylov.cuh -- device-resident Krylov state and the fused site functors used
// by the solvers (solvers.cu).  All scalars of a right-hand side live in
// device memory; the finalize step of each reduction (run by the last block,
// one thread per right-hand side) updates them, so an iteration needs no
// host round trip (the reference reads every dot product back with a blocking
// copy: Core/CudaHelper.cu:697-710).
#pragma once
#include "blas.cuh"
#include "dslash.cuh"

namespace clg {

constexpr int GM_MAXK = 16;  // longest GMRES cycle kept on the device

enum : int { ST_RUNNING = 0, ST_CONVERGED = 1, ST_BREAKDOWN = 2 };

struct KState {
  // BiCGStab / CG scalars
  double2 rho, alpha, omega, beta;
  double rr, rr0, tol2;
  double rr1;    // CG on one right-hand side: |r|^2 alternates between rr and rr1 (Cg1P)
  int done;      // this rhs needs no more work in the current inner solve
  int skip;      // kernels skip this rhs (done, or converged mid-iteration)
  int conv_s;    // BiCGStab: |s| small, finish with x += alpha p
  int status;
  int iters;     // operator applications
  int j;         // GMRES: columns built in this cycle
  int since;     // device-side inner loop: chunks without improving `best`
  int pad;
  // GMRES cycle
  double2 H[(GM_MAXK + 1) * GM_MAXK];  // H[i*GM_MAXK + j]
  double2 cs[GM_MAXK], sn[GM_MAXK];
  double2 g[GM_MAXK + 1];
  double2 y[GM_MAXK];
  double s[GM_MAXK + 1];   // lazy normalisation: v_i = s_i * V'_i
  double beta0;            // |r| at the start of the cycle
  double resid_est;        // |g_(j+1)| estimate
  double best;             // device-side inner loop: smallest residual seen (stagnation guard)
};

__device__ __forceinline__ bool bad(double v) { return !(v == v) || isinf(v); }

// ------------------------------------------------------------------ BiCGStab
// F_rv: (r^, v) -> alpha = rho / (r^, v)
template <int P, int NC>
struct BiAlpha {
  DField rh, v;
  KState* st;
  __device__ bool active(int r) const { return !st[r].skip; }
  __device__ void operator()(int rhs, int p, int64_t h, double* acc) const {
    using AT = typename AccT<P>::T;
    cpx<AT> a[NC], b[NC];
    ldv<P, NC, AT>(rh, rhs, p, h, a);
    ldv<P, NC, AT>(v, rhs, p, h, b);
    acc_dot<NC, AT>(a, b, acc);
  }
  __device__ void finalize(int r, const double* s) const {
    KState& k = st[r];
    if (k.skip) return;
    const double2 d = make_double2(s[0], s[1]);
    if ((d.x == 0.0 && d.y == 0.0) || bad(d.x) || bad(d.y)) {
      k.status = ST_BREAKDOWN;
      k.done = k.skip = 1;
      return;
    }
    k.alpha = cdiv(k.rho, d);
    k.iters += 1;
  }
};

// r <- r - alpha v ; |r|^2 -> conv_s
template <int P, int NC>
struct BiS {
  DField r, v;
  KState* st;
  __device__ bool active(int q) const { return !st[q].skip; }
  __device__ void operator()(int rhs, int p, int64_t h, double* acc) const {
    using AT = typename AccT<P>::T;
    cpx<AT> a[NC], b[NC];
    ldv<P, NC, AT>(r, rhs, p, h, a);
    ldv<P, NC, AT>(v, rhs, p, h, b);
    const double2 al = st[rhs].alpha;
    const cpx<AT> ca = mk<AT>((AT)al.x, (AT)al.y);
#pragma unroll
    for (int k = 0; k < NC; ++k) a[k] = a[k] - ca * b[k];
    stv<P, NC, AT>(r, rhs, p, h, a);
    acc[0] += site_norm2<NC, AT>(a);
  }
  __device__ void finalize(int q, const double* s) const {
    KState& k = st[q];
    if (k.skip) return;
    if (bad(s[0])) {
      k.status = ST_BREAKDOWN;
      k.done = k.skip = 1;
      return;
    }
    if (s[0] <= k.tol2 * k.rr0) {
      k.conv_s = 1;
      k.skip = 1;
    }
  }
};

// (t, s), (t, t) -> omega = (t, s) / (t, t)   [s stored in r]
template <int P, int NC>
struct BiOmega {
  DField t, r;
  KState* st;
  __device__ bool active(int q) const { return !st[q].skip; }
  __device__ void operator()(int rhs, int p, int64_t h, double* acc) const {
    using AT = typename AccT<P>::T;
    cpx<AT> a[NC], b[NC];
    ldv<P, NC, AT>(t, rhs, p, h, a);
    ldv<P, NC, AT>(r, rhs, p, h, b);
    acc_dot<NC, AT>(a, b, acc);
    acc[2] += site_norm2<NC, AT>(a);
  }
  __device__ void finalize(int q, const double* s) const {
    KState& k = st[q];
    if (k.skip) return;
    k.iters += 1;
    if (!(s[2] > 0.0) || bad(s[2])) {
      k.status = ST_BREAKDOWN;
      k.done = k.skip = 1;
      return;
    }
    k.omega = make_double2(s[0] / s[2], s[1] / s[2]);
  }
};

// x += alpha p + omega s ; r = s - omega t ; (r^, r), |r|^2 -> beta, rho
// (or, when |s| was already small: x += alpha p and stop)
template <int P, int NC>
struct BiUpdate {
  DField x, p, r, t, rh;
  KState* st;
  __device__ bool active(int q) const { return !st[q].done; }
  __device__ void operator()(int rhs, int par, int64_t h, double* acc) const {
    using AT = typename AccT<P>::T;
    const KState& k = st[rhs];
    cpx<AT> vx[NC], vp[NC];
    ldv<P, NC, AT>(x, rhs, par, h, vx);
    ldv<P, NC, AT>(p, rhs, par, h, vp);
    const cpx<AT> ca = mk<AT>((AT)k.alpha.x, (AT)k.alpha.y);
    if (k.conv_s) {
#pragma unroll
      for (int i = 0; i < NC; ++i) vx[i] = vx[i] + ca * vp[i];
      stv<P, NC, AT>(x, rhs, par, h, vx);
      return;
    }
    cpx<AT> vr[NC], vt[NC], vh[NC];
    ldv<P, NC, AT>(r, rhs, par, h, vr);
    ldv<P, NC, AT>(t, rhs, par, h, vt);
    ldv<P, NC, AT>(rh, rhs, par, h, vh);
    const cpx<AT> co = mk<AT>((AT)k.omega.x, (AT)k.omega.y);
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      vx[i] = vx[i] + ca * vp[i] + co * vr[i];
      vr[i] = vr[i] - co * vt[i];
    }
    stv<P, NC, AT>(x, rhs, par, h, vx);
    stv<P, NC, AT>(r, rhs, par, h, vr);
    acc_dot<NC, AT>(vh, vr, acc);
    acc[2] += site_norm2<NC, AT>(vr);
  }
  __device__ void finalize(int q, const double* s) const {
    KState& k = st[q];
    if (k.done) return;
    if (k.conv_s) {
      k.status = ST_CONVERGED;
      k.done = k.skip = 1;
      return;
    }
    const double2 rho_new = make_double2(s[0], s[1]);
    k.rr = s[2];
    if (bad(s[2]) || bad(rho_new.x)) {
      k.status = ST_BREAKDOWN;
      k.done = k.skip = 1;
      return;
    }
    if (s[2] <= k.tol2 * k.rr0) {
      k.status = ST_CONVERGED;
      k.done = k.skip = 1;
      return;
    }
    if ((rho_new.x == 0.0 && rho_new.y == 0.0) || (k.omega.x == 0.0 && k.omega.y == 0.0)) {
      k.status = ST_BREAKDOWN;
      k.done = k.skip = 1;
      return;
    }
    k.beta = cmul(cdiv(rho_new, k.rho), cdiv(k.alpha, k.omega));
    k.rho = rho_new;
  }
};

// p = r + beta (p - omega v)
template <int P, int NC>
struct BiP {
  DField p, r, v;
  KState* st;
  __device__ bool active(int q) const { return !st[q].skip; }
  __device__ void operator()(int rhs, int par, int64_t h, double*) const {
    using AT = typename AccT<P>::T;
    const KState& k = st[rhs];
    cpx<AT> vp[NC], vr[NC], vv[NC];
    ldv<P, NC, AT>(p, rhs, par, h, vp);
    ldv<P, NC, AT>(r, rhs, par, h, vr);
    ldv<P, NC, AT>(v, rhs, par, h, vv);
    const cpx<AT> cb = mk<AT>((AT)k.beta.x, (AT)k.beta.y), co = mk<AT>((AT)k.omega.x, (AT)k.omega.y);
#pragma unroll
    for (int i = 0; i < NC; ++i) vp[i] = vr[i] + cb * (vp[i] - co * vv[i]);
    stv<P, NC, AT>(p, rhs, par, h, vp);
  }
  __device__ void finalize(int, const double*) const {}
};

// start: r = b (x = 0), r^ = r, p = r, rho = |r|^2
template <int P, int NC>
struct BiInit {
  DField b, x, r, rh, p;
  KState* st;
  const double* tolv;  // relative tolerance per right-hand side
  __device__ bool active(int q) const { return !st[q].done; }
  __device__ void operator()(int rhs, int par, int64_t h, double* acc) const {
    using AT = typename AccT<P>::T;
    cpx<AT> vb[NC], z[NC];
    ldv<P, NC, AT>(b, rhs, par, h, vb);
#pragma unroll
    for (int i = 0; i < NC; ++i) z[i] = mk<AT>(0, 0);
    stv<P, NC, AT>(x, rhs, par, h, z);
    stv<P, NC, AT>(r, rhs, par, h, vb);
    stv<P, NC, AT>(rh, rhs, par, h, vb);
    stv<P, NC, AT>(p, rhs, par, h, vb);
    acc[0] += site_norm2<NC, AT>(vb);
  }
  __device__ void finalize(int q, const double* s) const {
    KState& k = st[q];
    if (k.done) return;
    k.rr0 = k.rr = s[0];
    k.rho = make_double2(s[0], 0.0);
    k.tol2 = tolv[q] * tolv[q];
    k.conv_s = 0;
    k.status = ST_RUNNING;
    if (!(s[0] > 0.0)) {  // zero right-hand side: x = 0 is exact
      k.status = ST_CONVERGED;
      k.done = k.skip = 1;
    }
  }
};

// ------------------------------------------------------------------ CG (Hermitian positive definite)
// start: r = b, p = b, x = 0, rr = |b|^2
template <int P, int NC>
struct CgInit {
  DField b, x, r, p;
  KState* st;
  const double* tolv;  // relative tolerance per right-hand side
  __device__ bool active(int q) const { return !st[q].done; }
  __device__ void operator()(int rhs, int par, int64_t h, double* acc) const {
    using AT = typename AccT<P>::T;
    cpx<AT> vb[NC], z[NC];
    ldv<P, NC, AT>(b, rhs, par, h, vb);
#pragma unroll
    for (int i = 0; i < NC; ++i) z[i] = mk<AT>(0, 0);
    stv<P, NC, AT>(x, rhs, par, h, z);
    stv<P, NC, AT>(r, rhs, par, h, vb);
    stv<P, NC, AT>(p, rhs, par, h, vb);
    acc[0] += site_norm2<NC, AT>(vb);
  }
  __device__ void finalize(int q, const double* s) const {
    KState& k = st[q];
    if (k.done) return;
    k.rr0 = k.rr = s[0];
    k.tol2 = tolv[q] * tolv[q];
    k.status = ST_RUNNING;
    if (!(s[0] > 0.0)) {
      k.status = ST_CONVERGED;
      k.done = k.skip = 1;
    }
  }
};
// pAp = (p, A p) -> alpha = rr / pAp; counts `weight` operator applications
__device__ __forceinline__ void cg_alpha_finalize(KState& k, double pAp, int weight) {
  if (k.skip) return;
  k.iters += weight;
  if (!(pAp > 0.0) || bad(pAp)) {
    k.status = ST_BREAKDOWN;
    k.done = k.skip = 1;
    return;
  }
  k.alpha = make_double2(k.rr / pAp, 0.0);
}
// rr_new = |r|^2 after the update -> beta, convergence
__device__ __forceinline__ void cg_update_finalize(KState& k, double rr_new) {
  if (k.skip) return;
  if (bad(rr_new)) {
    k.status = ST_BREAKDOWN;
    k.done = k.skip = 1;
    return;
  }
  k.beta = make_double2(rr_new / k.rr, 0.0);
  k.rr = rr_new;
  if (rr_new <= k.tol2 * k.rr0) {
    k.status = ST_CONVERGED;
    k.done = k.skip = 1;
  }
}

// (p, q) -> alpha = rr / (p, q)
template <int P, int NC>
struct CgAlpha {
  DField p, q;
  KState* st;
  int weight;  // operator applications per Krylov-operator application (2 for M M^+)
  __device__ bool active(int r) const { return !st[r].skip; }
  __device__ void operator()(int rhs, int par, int64_t h, double* acc) const {
    using AT = typename AccT<P>::T;
    cpx<AT> a[NC], b[NC];
    ldv<P, NC, AT>(p, rhs, par, h, a);
    ldv<P, NC, AT>(q, rhs, par, h, b);
    acc_dot<NC, AT>(a, b, acc);
  }
  __device__ void finalize(int r, const double* s) const { cg_alpha_finalize(st[r], s[0], weight); }
};
// x += alpha p ; r -= alpha q ; rr_new -> beta
template <int P, int NC>
struct CgUpdate {
  DField x, r, p, q;
  KState* st;
  __device__ bool active(int w) const { return !st[w].skip; }
  __device__ void operator()(int rhs, int par, int64_t h, double* acc) const {
    using AT = typename AccT<P>::T;
    const AT al = (AT)st[rhs].alpha.x;
    cpx<AT> vx[NC], vr[NC], vp[NC], vq[NC];
    ldv<P, NC, AT>(x, rhs, par, h, vx);
    ldv<P, NC, AT>(r, rhs, par, h, vr);
    ldv<P, NC, AT>(p, rhs, par, h, vp);
    ldv<P, NC, AT>(q, rhs, par, h, vq);
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      vx[i] = vx[i] + al * vp[i];
      vr[i] = vr[i] - al * vq[i];
    }
    stv<P, NC, AT>(x, rhs, par, h, vx);
    stv<P, NC, AT>(r, rhs, par, h, vr);
    acc[0] += site_norm2<NC, AT>(vr);
  }
  __device__ void finalize(int w, const double* s) const { cg_update_finalize(st[w], s[0]); }
};

// CG on A = M M^+ (or M^+ M) with the vector work fused into the Schur hops
// (wilson_hop_epi_kernel).  The second hop of the first factor produces
// q = M^+ p (or M p), stores it and reduces |q|^2 = (p, A p) -> alpha; the
// second hop of the second factor produces A p in registers only and applies
//   x += alpha p,  r -= alpha A p,  |r|^2 -> beta
// at its own site, so A p is never written and the separate (p, A p) and
// update passes disappear.  Both act on the even checkerboard (parity 0); their
// sums are left as partials for epi_final_kernel, or for the next kernel (one
// right-hand side, Cg1P).
template <int P>
struct CgHopAlpha {
  static constexpr bool PARTIALS = true;
  static constexpr int NRED = 1;
  static constexpr bool STORE = true;
  KState* st;
  int weight;
  template <typename AT>
  __device__ void site(int, int64_t, const cpx<AT> q[12], double* red) const {
    red[0] += site_norm2<12, AT>(q);
  }
  __device__ void finalize(int r, const double* s) const { cg_alpha_finalize(st[r], s[0], weight); }
};
template <int P>
struct CgHopUpdate {
  static constexpr bool PARTIALS = true;
  static constexpr int NRED = 1;
  static constexpr bool STORE = false;
  DField x, r, p;
  KState* st;
  template <typename AT>
  __device__ void site(int rhs, int64_t h, const cpx<AT> ap[12], double* red) const {
    const AT al = (AT)st[rhs].alpha.x;
    cpx<AT> vx[12], vr[12], vp[12];
    ldv<P, 12, AT>(x, rhs, 0, h, vx);
    ldv<P, 12, AT>(r, rhs, 0, h, vr);
    ldv<P, 12, AT>(p, rhs, 0, h, vp);
#pragma unroll
    for (int i = 0; i < 12; ++i) {
      vx[i] = vx[i] + al * vp[i];
      vr[i] = vr[i] - al * ap[i];
    }
    stv<P, 12, AT>(x, rhs, 0, h, vx);
    stv<P, 12, AT>(r, rhs, 0, h, vr);
    red[0] += site_norm2<12, AT>(vr);
  }
  __device__ void finalize(int w, const double* s) const { cg_update_finalize(st[w], s[0]); }
};
// E::finalize of right-hand side blockIdx.x from the partials [rhs][nslots] its
// hop left: all slots, or in a batch of lattices those of its lattice's tiles.
// The 28-right-hand-side update hop of 32^3x32 used to fence each partial and
// take a ticket per block, and a batch of lattices wrote zero partials for the
// other lattices' right-hand sides; without: the 28-right-hand-side solve 664 ->
// 639 ms, the uneven lattices 51.8 -> 44.0 ms.
template <class E>
__global__ void __launch_bounds__(512) epi_final_kernel(E e, const double* partials, int64_t nslots,
                                                        const int* skip, int skip_stride, const BatchTile* bt, int nbt,
                                                        int64_t btiles) {
  const int rhs = blockIdx.x;
  pdl_launch_dependents();
  int64_t lo = 0, hi = nslots;
  for (int l = 0; l < nbt; ++l)
    if (rhs >= bt[l].rhs0 && rhs < bt[l].rhs0 + bt[l].nrhs) {
      lo = bt[l].tile0;
      hi = l + 1 < nbt ? bt[l + 1].tile0 : btiles;
    }
  pdl_wait();
  if (skip[(int64_t)rhs * skip_stride]) return;  // finished before this hop: stale partials
  constexpr int U = 8;
  const double* p = partials + rhs * nslots;
  double s = 0.0;
  for (int64_t i0 = lo + threadIdx.x; i0 < hi; i0 += U * 512) {
    double v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = i0 + u * 512 < hi ? __ldcg(p + i0 + u * 512) : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) s += v[u];
  }
  __shared__ double sm[16];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t[1] = {0.0};
    for (int k = 0; k < 16; ++k) t[0] += sm[k];
    e.finalize(rhs, t);
  }
}

// CG on one right-hand side: the same iteration with the scalars made by the
// kernels that need them (block_total) instead of at the end of the reducing
// launch.  (p, A p) is left as partials by the alpha hop; the next hop, which
// does not need alpha, adds them up in a block of its own (AlphaFin); |r|^2 is
// left by the update hop and added up by every block of Cg1P, whose first block
// writes the state.
template <int P>
struct Cg1HopUpdate : CgHopUpdate<P> {};
// FP16: x, r and p, in DRAM where the vectors and links exceed L2, are requested
// before the stencil, 9 words of 16 bytes a thread (the update hop of 32^3x16 34.5
// -> 30.7 us).  The 18 and 36 words of FP32 and FP64 wait in front of the
// stencil's own loads instead: FP32 on 48^3x24 228 us without them, 280 with.
template <>
struct Cg1HopUpdate<P16> : CgHopUpdate<P16> {
  __device__ void prefetch(int rhs, int64_t h) const {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int64_t off = (k * x.Vh + h) * 16;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(x.base(rhs, 0) + off));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(r.base(rhs, 0) + off));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p.base(rhs, 0) + off));
    }
  }
};
// beta = |r_new|^2 / |r|^2; p = r + beta p.  `odd`: the iteration's parity, even
// ones hold the old |r|^2 in rr and leave the new one in rr1, so that no block
// reads what the first one writes (a finished solve leaves both in rr).
template <int P, int NC>
struct Cg1P {
  static constexpr bool ONE_LATTICE = true;
  DField p, r;
  KState* st;
  const double* rrp;  // nrr partials of |r_new|^2
  int nrr, odd, weight;
  __device__ static double* beta_of() {
    __shared__ double b;
    return &b;
  }
  __device__ bool active(int) const { return true; }
  __device__ bool prologue(int, bool first) const {
    KState& k = *st;
    const int skip = k.skip;
    const double old = odd ? k.rr1 : k.rr, lim = k.tol2 * k.rr0;
    const double rr_new = block_total(rrp, nrr);
    if (skip) return false;
    const bool wrong = bad(rr_new), conv = !wrong && rr_new <= lim;
    if (threadIdx.x == 0) *beta_of() = rr_new / old;
    if (first && threadIdx.x == 0) {
      k.iters += weight;
      if (wrong) {
        k.status = ST_BREAKDOWN;
        k.done = k.skip = 1;
      } else {
        k.beta = make_double2(rr_new / old, 0.0);
        if (odd || conv) k.rr = rr_new;
        if (!odd || conv) k.rr1 = rr_new;
        if (conv) {
          k.status = ST_CONVERGED;
          k.done = k.skip = 1;
        }
      }
    }
    __syncthreads();
    return !wrong && !conv;
  }
  __device__ void operator()(int rhs, int par, int64_t h, double*) const {
    using AT = typename AccT<P>::T;
    const AT be = (AT)*beta_of();
    cpx<AT> vp[NC], vr[NC];
    ldv<P, NC, AT>(p, rhs, par, h, vp);
    ldv<P, NC, AT>(r, rhs, par, h, vr);
#pragma unroll
    for (int i = 0; i < NC; ++i) vp[i] = vr[i] + be * vp[i];
    stv<P, NC, AT>(p, rhs, par, h, vp);
  }
  __device__ void finalize(int, const double*) const {}
};
// p = r + beta p
template <int P, int NC>
struct CgP {
  DField p, r;
  KState* st;
  __device__ bool active(int w) const { return !st[w].skip; }
  __device__ void operator()(int rhs, int par, int64_t h, double*) const {
    using AT = typename AccT<P>::T;
    const AT be = (AT)st[rhs].beta.x;
    cpx<AT> vp[NC], vr[NC];
    ldv<P, NC, AT>(p, rhs, par, h, vp);
    ldv<P, NC, AT>(r, rhs, par, h, vr);
#pragma unroll
    for (int i = 0; i < NC; ++i) vp[i] = vr[i] + be * vp[i];
    stv<P, NC, AT>(p, rhs, par, h, vp);
  }
  __device__ void finalize(int, const double*) const {}
};

// ------------------------------------------------------------------ GMRES(k)
// V' vectors are stored un-normalised; v_i = s_i V'_i (s_i in KState).
struct VList {
  DField v[GM_MAXK + 1];
};

// cycle start: V'_0 = b - (K x) [w holds K x, or nothing for x = 0]; beta = |V'_0|
template <int P, int NC>
struct GmStart {
  DField b, w, v0;
  KState* st;
  int have_x;
  const double* tolv;  // relative to |b| of the inner solve (stored in rr0 at first cycle)
  int first;
  __device__ bool active(int q) const { return !st[q].done; }
  __device__ void operator()(int rhs, int par, int64_t h, double* acc) const {
    using AT = typename AccT<P>::T;
    cpx<AT> vb[NC];
    ldv<P, NC, AT>(b, rhs, par, h, vb);
    if (have_x) {
      cpx<AT> vw[NC];
      ldv<P, NC, AT>(w, rhs, par, h, vw);
#pragma unroll
      for (int i = 0; i < NC; ++i) vb[i] = vb[i] - vw[i];
    }
    stv<P, NC, AT>(v0, rhs, par, h, vb);
    acc[0] += site_norm2<NC, AT>(vb);
  }
  __device__ void finalize(int q, const double* s) const {
    KState& k = st[q];
    if (k.done) return;
    if (first) {
      k.rr0 = s[0];
      k.tol2 = tolv[q] * tolv[q];
      k.status = ST_RUNNING;
    }
    k.skip = 0;
    k.j = 0;
    const double beta = sqrt(s[0]);
    k.beta0 = beta;
    k.resid_est = beta;
    if (bad(beta)) {
      k.status = ST_BREAKDOWN;
      k.done = k.skip = 1;
      return;
    }
    if (s[0] <= k.tol2 * k.rr0) {
      k.status = ST_CONVERGED;
      k.done = k.skip = 1;
      return;
    }
    k.g[0] = make_double2(beta, 0.0);
    k.s[0] = 1.0 / beta;
  }
};

// <V'_i, w>, i <= j: the column's j + 1 dot products, GM_DG of them per block
// (launch index y = rhs * groups + group), so that the groups run side by side
// and a block reduces 2 GM_DG numbers (one block over all columns took 8-21 us
// a launch on 8^4, growing with j).  Left as block partials: GmOrtho's blocks
// make the Hessenberg column of them.
constexpr int GM_DG = 4;
template <int P, int NC>
struct GmDots {
  static constexpr bool PARTIALS = true;
  VList V;
  DField w;
  KState* st;
  int j, groups;
  __device__ bool active(int y) const { return !st[y / groups].skip; }
  __device__ void operator()(int y, int par, int64_t h, double* acc) const {
    using AT = typename AccT<P>::T;
    const int rhs = y / groups, i0 = GM_DG * (y - rhs * groups);
    cpx<AT> vw[NC];
    ldv<P, NC, AT>(w, rhs, par, h, vw);
#pragma unroll
    for (int i = 0; i < GM_DG; ++i) {
      if (i0 + i > j) break;
      cpx<AT> vi[NC];
      ldv<P, NC, AT>(V.v[i0 + i], rhs, par, h, vi);
      acc_dot<NC, AT>(vi, vw, acc + 2 * i);
    }
  }
};

// The same for lattices that fill the chip (gm_wide): one block over all J + 1
// columns, so w is read once and every column's loads are in flight together; the
// last block stores the Hessenberg column.  FP32-inner GMRES(12) on 32^3x16:
// 12.9 ms, with the groups of GmDots and sums in GmOrtho's blocks 13.7.
template <int P, int NC, int J>
struct GmDotsJ {
  VList V;
  DField w;
  KState* st;
  __device__ bool active(int q) const { return !st[q].skip; }
  __device__ void operator()(int rhs, int par, int64_t h, double* acc) const {
    using AT = typename AccT<P>::T;
    cpx<AT> vw[NC];
    ldv<P, NC, AT>(w, rhs, par, h, vw);
#pragma unroll
    for (int i = 0; i <= J; ++i) {
      cpx<AT> vi[NC];
      ldv<P, NC, AT>(V.v[i], rhs, par, h, vi);
      acc_dot<NC, AT>(vi, vw, acc + 2 * i);
    }
  }
  __device__ void finalize(int q, const double* s) const {
    KState& k = st[q];
    if (k.skip) return;
    k.iters += 1;
    for (int i = 0; i <= J; ++i) k.H[i * GM_MAXK + J] = make_double2(k.s[i] * s[2 * i], k.s[i] * s[2 * i + 1]);
  }
};

// V'_{j+1} = w - sum_i h_ij v_i ; h_{j+1,j} = |V'_{j+1}| ; Givens rotation of column j
// (h_ij = s_i <V'_i, w> from GmDots's partials, summed by every block; block 0
// of the right-hand side stores the column for the last block's rotation; WIDE:
// GmDotsJ stored it)
template <int P, int NC, bool WIDE>
struct GmOrtho {
  VList V;
  DField w;
  KState* st;
  int j;
  const double* dots;  // [rhs * groups + group][nslots][2 GM_DG]
  int nslots;
  __device__ static double2* coef() {  // h_ij s_i
    __shared__ double2 c[GM_MAXK];
    return c;
  }
  __device__ bool active(int) const { return true; }
  __device__ bool prologue(int q, bool first) const {
    KState& k = st[q];
    const bool run = !k.skip;
    if constexpr (WIDE) {
      if (threadIdx.x <= j) {
        const double2 hv = k.H[threadIdx.x * GM_MAXK + j];
        const double si = k.s[threadIdx.x];
        coef()[threadIdx.x] = make_double2(hv.x * si, hv.y * si);
      }
    } else {
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
      const int groups = j / GM_DG + 1;
      double* c = reinterpret_cast<double*>(coef());
      for (int v = warp; v < 2 * (j + 1); v += nw) {
        const int i = v >> 1;
        const double* p = dots + (int64_t)(q * groups + i / GM_DG) * nslots * (2 * GM_DG) + 2 * (i % GM_DG) + (v & 1);
        const double si = k.s[i];
        double s = 0.0;
        for (int b = lane; b < nslots; b += 32) s += __ldcg(p + (int64_t)b * (2 * GM_DG));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const double h = si * s;
        if (lane == 0) {
          c[v] = h * si;
          if (first && run) reinterpret_cast<double*>(&k.H[i * GM_MAXK + j])[v & 1] = h;
        }
      }
      if (first && run && threadIdx.x == 0) k.iters += 1;
    }
    __syncthreads();
    return run;
  }
  __device__ void operator()(int rhs, int par, int64_t h, double* acc) const {
    using AT = typename AccT<P>::T;
    const double2* c = coef();
    cpx<AT> vw[NC];
    ldv<P, NC, AT>(w, rhs, par, h, vw);
    constexpr int U = WIDE ? GM_MAXK : 4;
#pragma unroll U
    for (int i = 0; i < GM_MAXK; ++i) {
      if (i > j) break;
      cpx<AT> vi[NC];
      ldv<P, NC, AT>(V.v[i], rhs, par, h, vi);
      const cpx<AT> cc = mk<AT>((AT)c[i].x, (AT)c[i].y);
#pragma unroll
      for (int m = 0; m < NC; ++m) vw[m] = vw[m] - cc * vi[m];
    }
    stv<P, NC, AT>(V.v[j + 1], rhs, par, h, vw);
    acc[0] += site_norm2<NC, AT>(vw);
  }
  // Lane i holds row i of column j and rotation i.  The previous rotations
  // (RotateH, CSolverGMRES.cpp:262-327, incrementally) run down the column as one
  // chain that every lane follows through shuffles: one round trip to memory,
  // and registers for one row.  One thread with the column and its rotations in
  // registers (49 complex numbers) held the whole site kernel at 248 registers, one
  // block per SM.
  __device__ void finalize_warp(int q, const double* s, int lane) const {
    static_assert(GM_MAXK <= 32, "one lane per row");
    KState& k = st[q];
    if (k.skip) return;  // uniform
    const double hn = sqrt(s[0]);
    const double2 zero = make_double2(0.0, 0.0);
    double2* H = k.H;
    double2 row = lane <= j ? H[lane * GM_MAXK + j] : zero;
    const double2 ci = lane < j ? k.cs[lane] : zero, si = lane < j ? k.sn[lane] : zero;
    const double2 gj = k.g[j];
    const double tol2 = k.tol2, rr0 = k.rr0;
    auto from = [](double2 v, int i) {
      return make_double2(__shfl_sync(0xffffffffu, v.x, i), __shfl_sync(0xffffffffu, v.y, i));
    };
    double2 hjj = from(row, 0);  // the chain: row i after the rotations above it
#pragma unroll 4
    for (int i = 0; i < j; ++i) {
      const double2 next = from(row, i + 1), cs = from(ci, i), sn = from(si, i);
      const double2 a = cmul(cconj(cs), hjj), b = cmul(cconj(sn), next);
      const double2 c = cmul(cs, next), d = cmul(sn, hjj);
      if (lane == i) row = make_double2(a.x + b.x, a.y + b.y);
      hjj = make_double2(c.x - d.x, c.y - d.y);
    }
    if (lane < j) H[lane * GM_MAXK + j] = row;
    if (lane != 0) return;
    k.s[j + 1] = hn > 0.0 ? 1.0 / hn : 0.0;
    const double den = sqrt(hjj.x * hjj.x + hjj.y * hjj.y + hn * hn);
    if (!(den > 0.0) || bad(den)) {
      k.status = ST_BREAKDOWN;
      k.skip = 1;
      return;
    }
    const double2 cs = make_double2(hjj.x / den, hjj.y / den), sn = make_double2(hn / den, 0.0);
    k.cs[j] = cs;
    k.sn[j] = sn;
    H[j * GM_MAXK + j] = make_double2(den, 0.0);
    H[(j + 1) * GM_MAXK + j] = zero;
    const double2 m = cmul(sn, gj);
    k.g[j + 1] = make_double2(-m.x, -m.y);
    k.g[j] = cmul(cconj(cs), gj);
    k.j = j + 1;
    const double est = sqrt(m.x * m.x + m.y * m.y);
    k.resid_est = est;
    // happy breakdown or converged: stop extending this cycle
    if (est * est <= tol2 * rr0 || hn == 0.0) k.skip = 1;
  }
};

// back substitution of the j x j triangle (SolveY, CSolverGMRES.cpp:329-358); coefficients y_i s_i
__global__ void gm_solve_y(KState* st, int nrhs);

// x += sum_i (y_i s_i) V'_i over the columns built in this cycle
template <int P, int NC>
struct GmUpdate {
  VList V;
  DField x;
  KState* st;
  int kmax;
  __device__ bool active(int q) const { return !st[q].done && st[q].j > 0; }
  __device__ void operator()(int rhs, int par, int64_t h, double*) const {
    using AT = typename AccT<P>::T;
    const KState& k = st[rhs];
    cpx<AT> vx[NC];
    ldv<P, NC, AT>(x, rhs, par, h, vx);
    const int kj = k.j;
    constexpr int U = NC == 12 ? 1 : 4;  // whole sites: 80 registers, 3 blocks per SM
#pragma unroll U
    for (int i = 0; i < kj; ++i) {
      cpx<AT> vi[NC];
      ldv<P, NC, AT>(V.v[i], rhs, par, h, vi);
      const double2 c = k.y[i];
      const cpx<AT> cc = mk<AT>((AT)c.x, (AT)c.y);
#pragma unroll
      for (int m = 0; m < NC; ++m) vx[m] = vx[m] + cc * vi[m];
    }
    stv<P, NC, AT>(x, rhs, par, h, vx);
  }
  __device__ void finalize(int, const double*) const {}
};

}  // namespace clg
