// hostkrylov.cuh -- FP64 Krylov building blocks driven from the host: one
// right-hand side, the small dense algebra on the host (dense.h), every
// orthogonalisation one multi-dot launch and one linear-combination launch per
// pass, with the coefficients read back (HostKrylov::orthogonalise) or kept on
// the device for a whole Arnoldi cycle (arnoldi_step).  Used by the recycled solver (GCRO-DR)
// and by the multi-shift solvers that share one Krylov space over all shifts
// (multi-shift FOM and BiCGStab-M), whose per-cycle work is dominated by the
// operator applications, not by these launches.
#pragma once
#include <algorithm>
#include <cmath>
#include <vector>

#include "blas.cuh"
#include "dense.h"

namespace clg {
namespace hk {

using dense::Z;

constexpr int MAXV = 34;  // vectors of one multi-dot or linear combination (m + 1 <= 33, + 1)
// Inner products per block of a multi-dot: w is read once per group.  MDH for the
// products read back to the host, whose launch ends with a last block: GCRO-DR on
// 16^3x32 takes 210 ms with 4 and 186 with 8, on 32^3x16 725 and 613.  In the
// device's Arnoldi cycle, where nothing waits for the products' last block, 8 are
// slower: FOM(30) on 16^3x32 24.4 ms with 4, 26.8 with 8.
constexpr int MDG = 4, MDH = 8;

// The vectors of one launch by their data pointers; all have the shape of the
// launch (HostVecs::proto), seen as NC / 3 times as many blocks of 3 components
// (the storage is [parity][component][h], so a block is a run of 3 Vh complex
// numbers): four times the threads of one per Wilson site, and a third of the
// registers.
struct VecTab {
  const char* v[MAXV];
};
__device__ __forceinline__ void ld3(const char* v, int64_t off, int64_t kstride, cpx<double> o[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double2 d = *reinterpret_cast<const double2*>(v + off + k * kstride);
    o[k] = mk<double>(d.x, d.y);
  }
}

// out[i] = v_i^+ w for n vectors, G of them per block (right-hand side g of the
// launch = vectors G g ..), so that the blocks of all vectors run side by side.
// One block over all vectors reduced 32 numbers per block on 32 blocks of 8^3x16
// (19 us a launch whatever n).  PART: left as block partials [group][slot][2 G]
// for the linear combination that follows (LinCombF::dots).
template <bool PART, int G>
struct MultiDotF {
  static constexpr bool PARTIALS = PART, ONE_LATTICE = true;
  const char* w;
  VecTab v;
  int64_t blk, kstride;
  int n;
  double2* out;
  __device__ bool active(int) const { return true; }
  __device__ void operator()(int g, int p, int64_t h, double* acc) const {
    const int64_t off = p * blk + h * 16;
    cpx<double> wv[3];
    ld3(w, off, kstride, wv);
#pragma unroll
    for (int i = 0; i < G; ++i) {
      if (G * g + i >= n) break;
      cpx<double> a[3];
      ld3(v.v[G * g + i], off, kstride, a);
      double re = 0.0, im = 0.0;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        re = fma(a[c].x, wv[c].x, fma(a[c].y, wv[c].y, re));
        im = fma(a[c].x, wv[c].y, fma(-a[c].y, wv[c].x, im));
      }
      acc[2 * i] += re;
      acc[2 * i + 1] += im;
    }
  }
  __device__ void finalize(int g, const double* s) const {
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int k = G * g + i;
      if (k >= n) break;
      out[k] = make_double2(s[2 * i], s[2 * i + 1]);
    }
  }
};

// out_r = beta in_r + sum_i c_(r,i) s_i v_i for the `rhs` outputs r of the
// launch (ostride bytes apart); the coefficients are kernel arguments (HOST),
// device-resident (DEV: dc), or minus s_i times the inner products whose
// partials precede the launch (DOTS: every block adds them up, the first one
// also adds them to the Hessenberg column hcol, or stores them: first).  NRED = 1
// also reduces |out|^2: its root goes to hn and its reciprocal (0 for a zero
// vector) to inv.
enum : int { LC_HOST = 0, LC_DEV = 1, LC_DOTS = 2 };
template <int NRED, int SRC>
struct LinCombF {
  static constexpr bool ONE_LATTICE = true;
  char* out;
  const char* in;
  int64_t ostride;
  VecTab v;
  double2 c[MAXV];
  const double2* dc;
  const double* scale;
  const double* dots;
  int nslots;
  double2* hcol;
  int first;
  double2 beta;
  int64_t blk, kstride;
  int n;
  double2* hn;
  double* inv;
  __device__ static double2* coef() {
    __shared__ double2 s_c[MAXV];
    return s_c;
  }
  __device__ bool active(int) const { return true; }
  // the coefficients to shared memory (all blocks the same)
  __device__ bool prologue(int r, bool first_block) const {
    double2* sc = coef();
    if constexpr (SRC == LC_DOTS) {
      // warp w adds up the products w, w + 8, ...: all their partials' loads in flight together
      constexpr int U = (MAXV + 7) / 8;
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      double2 t[U];
#pragma unroll
      for (int u = 0; u < U; ++u) t[u] = make_double2(0.0, 0.0);
      for (int b = lane; b < nslots; b += 32) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = warp + 8 * u;
          if (i < n) {
            const double2 d = __ldcg(reinterpret_cast<const double2*>(
                                         dots + ((int64_t)(i / MDG) * nslots + b) * (2 * MDG)) + i % MDG);
            t[u].x += d.x;
            t[u].y += d.y;
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = warp + 8 * u;
        if (i >= n) break;  // uniform over the warp
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          t[u].x += __shfl_xor_sync(0xffffffffu, t[u].x, o);
          t[u].y += __shfl_xor_sync(0xffffffffu, t[u].y, o);
        }
        if (lane == 0) {
          const double si = scale[i];
          const double2 d = make_double2(si * t[u].x, si * t[u].y);
          sc[i] = make_double2(-si * d.x, -si * d.y);
          if (first_block) hcol[i] = first ? d : make_double2(hcol[i].x + d.x, hcol[i].y + d.y);
        }
      }
    } else if (threadIdx.x < n) {
      const int i = threadIdx.x;
      const double2 ci = SRC == LC_DEV ? dc[r * n + i] : c[i];
      const double si = SRC == LC_DEV ? scale[i] : 1.0;
      sc[i] = make_double2(si * ci.x, si * ci.y);
    }
    __syncthreads();
    return true;
  }
  __device__ void operator()(int r, int p, int64_t h, double* acc) const {
    const int64_t off = p * blk + h * 16;
    const double2* sc = coef();
    cpx<double> o[3];
    if (beta.x != 0.0 || beta.y != 0.0) {
      ld3(in + r * ostride, off, kstride, o);
      const cpx<double> b = mk<double>(beta.x, beta.y);
#pragma unroll
      for (int k = 0; k < 3; ++k) o[k] = b * o[k];
    } else {
#pragma unroll
      for (int k = 0; k < 3; ++k) o[k] = mk<double>(0, 0);
    }
#pragma unroll 8
    for (int i = 0; i < n; ++i) {
      cpx<double> a[3];
      ld3(v.v[i], off, kstride, a);
      const cpx<double> cc = mk<double>(sc[i].x, sc[i].y);
#pragma unroll
      for (int k = 0; k < 3; ++k) o[k] = o[k] + cc * a[k];
    }
    char* q = out + r * ostride + off;
#pragma unroll
    for (int k = 0; k < 3; ++k) *reinterpret_cast<double2*>(q + k * kstride) = make_double2(o[k].x, o[k].y);
    if constexpr (NRED > 0) {
#pragma unroll
      for (int k = 0; k < 3; ++k) acc[0] = fma(o[k].x, o[k].x, fma(o[k].y, o[k].y, acc[0]));
    }
  }
  __device__ void finalize(int, const double* s) const {
    if constexpr (NRED > 0) {
      const double d = sqrt(s[0]);
      if (hn) *hn = make_double2(d, 0.0);
      if (inv) *inv = d > 0.0 ? 1.0 / d : 0.0;
    }
  }
};

// device vectors of one shape owned by a solver cache
struct HostVecs : SolveCacheBase {
  clg_context_s* ctx = nullptr;
  std::vector<void*> allocs;
  FieldRef proto;
  FieldRef tmp;  // the operators' temporary (a full field)
  double* dev_out = nullptr;
  ~HostVecs() override {
    for (void* p : allocs) dfree(p);
  }
  clg_status vec(FieldRef& f) {
    void* p = nullptr;
    const size_t bytes = (size_t)proto.blk * proto.nparity;
    if (clg_status st = dalloc(ctx, &p, bytes)) return st;
    allocs.push_back(p);
    f = proto;
    f.data = static_cast<char*>(p);
    return CLG_SUCCESS;
  }
  // a full (both parities) field of the proto's shape: the operators' temporary
  clg_status full_vec(FieldRef& f) {
    const FieldRef keep = proto;
    proto.nparity = 2;
    proto.first_parity = 0;
    proto.rstride = proto.blk * 2;
    const clg_status st = vec(f);
    proto = keep;
    return st;
  }
  clg_status out_buffer() {
    void* p = nullptr;
    if (clg_status st = dalloc(ctx, &p, sizeof(double) * 2 * MAXV)) return st;
    allocs.push_back(p);
    dev_out = static_cast<double*>(p);
    return CLG_SUCCESS;
  }
};

struct HostKrylov {
  clg_context_s* ctx;
  HostVecs& W;
  const clg_gauge_s* Ug;
  int kind, op, nc;
  double param;
  int64_t Vh;
  int apps = 0;

  clg_status apply(const FieldRef& out, const FieldRef& in, const double* scale = nullptr) {
    ++apps;
    return apply_op(ctx, op, Ug, kind, param, out, in, &W.tmp, make_double2(1.0, 0.0), 1, scale);
  }
  // blocks of 3 components of a vector (VecTab)
  int blocks() const { return W.proto.nparity * (nc / 3); }
  int64_t block_bytes() const { return 3 * Vh * 16; }
  template <bool PART, int G>
  MultiDotF<PART, G> multidot(const FieldRef& w, const FieldRef* const* vs, int n) const {
    MultiDotF<PART, G> f;
    f.w = w.data;
    for (int i = 0; i < MAXV; ++i) f.v.v[i] = i < n ? vs[i]->data : nullptr;
    f.blk = block_bytes();
    f.kstride = Vh * 16;
    f.n = n;
    f.out = reinterpret_cast<double2*>(W.dev_out);
    return f;
  }
  // out[i] = v_i^+ w for the n vectors vs (n arbitrary), read to the host
  clg_status dots(const FieldRef& w, const std::vector<const FieldRef*>& vs, std::vector<Z>& out) {
    out.assign(vs.size(), Z(0.0, 0.0));
    for (size_t i0 = 0; i0 < vs.size(); i0 += MAXV) {
      const int n = (int)std::min<size_t>(MAXV, vs.size() - i0);
      const FieldRef* const* v = vs.data() + i0;
      const clg_status st =
          n <= MDG ? launch_sites<2 * MDG>(ctx, multidot<false, MDG>(w, v, n), 0, blocks(), Vh, 1)
                   : launch_sites<2 * MDH>(ctx, multidot<false, MDH>(w, v, n), 0, blocks(), Vh, (n + MDH - 1) / MDH);
      if (st) return st;
      double h[2 * MAXV];
      cudaError_t e = cudaMemcpyAsync(h, W.dev_out, sizeof(double) * 2 * n, cudaMemcpyDeviceToHost, ctx->stream);
      if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
      if (e != cudaSuccess) return ctx->fail(cuda_status(e), cudaGetErrorString(e));
      for (int i = 0; i < n; ++i) out[i0 + i] = Z(h[2 * i], h[2 * i + 1]);
    }
    return CLG_SUCCESS;
  }
  double norm(const FieldRef& a) {
    std::vector<Z> d;
    if (dots(a, {&a}, d)) return -1.0;
    return std::sqrt(std::max(d[0].real(), 0.0));
  }
  template <int NRED, int SRC>
  LinCombF<NRED, SRC> combination(const FieldRef& out, const FieldRef& in, Z beta, const FieldRef* const* vs,
                                  int n) const {
    LinCombF<NRED, SRC> f;
    f.out = out.data;
    f.in = in.data;
    f.ostride = out.rstride;
    for (int i = 0; i < MAXV; ++i) {
      f.v.v[i] = i < n ? vs[i]->data : nullptr;
      f.c[i] = make_double2(0.0, 0.0);
    }
    f.dc = nullptr;
    f.scale = nullptr;
    f.dots = nullptr;
    f.nslots = 0;
    f.hcol = nullptr;
    f.first = 0;
    f.beta = make_double2(beta.real(), beta.imag());
    f.blk = block_bytes();
    f.kstride = Vh * 16;
    f.n = n;
    f.hn = nullptr;
    f.inv = nullptr;
    return f;
  }
  // out = beta out + sum_i c_i v_i
  clg_status lincomb(const FieldRef& out, Z beta, const std::vector<const FieldRef*>& vs, const std::vector<Z>& c) {
    if (vs.size() > (size_t)MAXV) return ctx->fail(CLG_ERR_UNSUPPORTED, "too many vectors in one linear combination");
    auto f = combination<0, LC_HOST>(out, out, beta, vs.data(), (int)vs.size());
    for (size_t i = 0; i < vs.size(); ++i) f.c[i] = make_double2(c[i].real(), c[i].imag());
    return launch_sites<0>(ctx, f, 0, blocks(), Vh, 1);
  }
  clg_status copy(const FieldRef& dst, const FieldRef& src) { return lincomb(dst, Z(0.0, 0.0), {&src}, {Z(1.0, 0.0)}); }
  clg_status scale(const FieldRef& a, Z s) { return lincomb(a, s, {}, {}); }
  // w <- w - sum_i (v_i^+ w) v_i, twice; the coefficients of both passes summed into h
  clg_status orthogonalise(const FieldRef& w, const std::vector<const FieldRef*>& vs, std::vector<Z>& h) {
    h.assign(vs.size(), Z(0.0, 0.0));
    for (int pass = 0; pass < 2; ++pass) {
      std::vector<Z> d;
      if (clg_status st = dots(w, vs, d)) return st;
      std::vector<Z> neg(d.size());
      for (size_t i = 0; i < d.size(); ++i) {
        h[i] += d[i];
        neg[i] = -d[i];
      }
      if (clg_status st = lincomb(w, Z(1.0, 0.0), vs, neg)) return st;
    }
    return CLG_SUCCESS;
  }
};

// Device state of an Arnoldi cycle (arnoldi_step): the basis vectors are
// V'_i = v_i / s_i, not normalised, so that no pass over a vector only scales it.
struct ArnoldiState {
  double2 H[(MAXV - 1) * MAXV];  // column j at H + j MAXV, h_(j+1,j) included
  double2 norm;                  // of the vector arnoldi_start normalised
  double s[MAXV];
};

// V'_0 = scale-free copy of src, s_0 = 1 / |src|, norm = |src|
inline clg_status arnoldi_start(HostKrylov& K, ArnoldiState* st, const FieldRef& v0, const FieldRef& src) {
  auto f = K.combination<1, LC_HOST>(v0, src, Z(1.0, 0.0), nullptr, 0);
  f.hn = &st->norm;
  f.inv = &st->s[0];
  return launch_sites<1>(K.ctx, f, 0, K.blocks(), K.Vh, 1);
}
// Column j of the Arnoldi relation: w = A v_j orthogonalised against
// v_0 .. v_j by classical Gram-Schmidt twice, left in next = V'_(j+1), all of
// it on the device: 4 launches after the operator, no host read.  The host
// reads the whole H at the end of a cycle.  part: the inner products' partials
// (arnoldi_partials doubles); the combination adds them up itself, since a last
// block that waits for all others costs 4 us a pass and a sum that every block
// repeats 1 us (one cycle of 30 with 6 shifts on 8^3x16: 3.35 -> 2.64 ms).
inline int64_t arnoldi_partials(const HostKrylov& K) {
  int64_t most = 0;
  for (int g = 1; g <= (MAXV + MDG - 1) / MDG; ++g)
    most = std::max(most, site_blocks<2 * MDG>(K.ctx, K.blocks(), K.Vh, g) * g * 2 * MDG);
  return most;
}
inline clg_status arnoldi_step(HostKrylov& K, ArnoldiState* st, double* part, const FieldRef* const* V, int j,
                               const FieldRef& w, const FieldRef& next) {
  if (clg_status e = K.apply(w, *V[j], &st->s[j])) return e;
  const int n = j + 1, groups = (n + MDG - 1) / MDG;
  auto fill = [&](auto& f, int first) {
    f.scale = st->s;
    f.dots = part;
    f.nslots = (int)site_blocks<2 * MDG>(K.ctx, K.blocks(), K.Vh, groups);
    f.hcol = st->H + (size_t)j * MAXV;
    f.first = first;
  };
  for (int pass = 0; pass < 2; ++pass) {
    if (clg_status e = launch_sites<2 * MDG>(K.ctx, K.multidot<true, MDG>(w, V, n), 0, K.blocks(), K.Vh, groups, part)) return e;
    if (pass == 0) {
      auto f = K.combination<0, LC_DOTS>(w, w, Z(1.0, 0.0), V, n);
      fill(f, 1);
      if (clg_status e = launch_sites<0>(K.ctx, f, 0, K.blocks(), K.Vh, 1)) return e;
    } else {
      auto f = K.combination<1, LC_DOTS>(next, w, Z(1.0, 0.0), V, n);
      fill(f, 0);
      f.hn = f.hcol + n;
      f.inv = &st->s[n];
      if (clg_status e = launch_sites<1>(K.ctx, f, 0, K.blocks(), K.Vh, 1)) return e;
    }
  }
  return CLG_SUCCESS;
}

}  // namespace hk
}  // namespace clg
