// gen.cu -- seeded field generation on the device, CLGBin / Bridge++ import and
// export (reordering into the even-odd structure-of-arrays layout), the
// plaquette and the unitarity check of the gauge field.
//
// Generator (published methods):
//   Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11), key = {seed_lo, seed_hi ^ field_id},
//   counter = {index_lo, index_hi, sub, tag}; Box-Muller Gaussians from two 53-bit
//   uniforms; Haar SU(3) by Gram-Schmidt QR of a complex Gaussian matrix (Mezzadri,
//   Notices AMS 54, 2007) with det fixed to 1; exp(i eps H) by a scaled Taylor series
//   and squaring, re-unitarised.  Field indices follow the reference's site order so a
//   field generated here equals the same field generated on the host.
#include <cstring>

#include "blas.cuh"

namespace clg {

namespace {

constexpr uint32_t TAG_GAUGE = 0x47415547u, TAG_SPINOR = 0x5350494eu, TAG_Z2 = 0x5a324e53u, TAG_Z4 = 0x5a344e53u;

__device__ __forceinline__ void philox(uint32_t c[4], uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
    const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
    c[0] = n0;
    c[1] = lo1;
    c[2] = n2;
    c[3] = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

__device__ __forceinline__ double u53(uint32_t a, uint32_t b) {
  const uint64_t x = ((uint64_t)a << 21) ^ (uint64_t)(b >> 11);
  return ((double)x + 0.5) * (1.0 / 9007199254740992.0);
}

__device__ __forceinline__ void gauss2(uint64_t seed, uint32_t fid, uint64_t index, uint32_t sub, uint32_t tag,
                                       double& g1, double& g2) {
  uint32_t c[4] = {(uint32_t)index, (uint32_t)(index >> 32), sub, tag};
  philox(c, (uint32_t)seed, (uint32_t)(seed >> 32) ^ fid);
  const double v1 = u53(c[0], c[1]), v2 = u53(c[2], c[3]);
  const double r = sqrt(-2.0 * log(v1));
  double sn, cs;
  sincospi(2.0 * v2, &sn, &cs);
  g1 = r * cs;
  g2 = r * sn;
}

using C = cpx<double>;

__device__ void haar(uint64_t seed, uint32_t fid, uint64_t link, C z[9]) {
  const double isq2 = 0.70710678118654752440084436210485;
  for (int k = 0; k < 9; ++k) {
    double a, b;
    gauss2(seed, fid, link, (uint32_t)k, TAG_GAUGE, a, b);
    z[k] = mk<double>(a * isq2, b * isq2);
  }
  for (int c = 0; c < 3; ++c) {
    for (int p = 0; p < c; ++p) {
      C d = mk<double>(0, 0);
      for (int r = 0; r < 3; ++r) d = d + cjmul(z[3 * r + p], z[3 * r + c]);
      for (int r = 0; r < 3; ++r) z[3 * r + c] = z[3 * r + c] - d * z[3 * r + p];
    }
    double nn = 0;
    for (int r = 0; r < 3; ++r) nn += z[3 * r + c].x * z[3 * r + c].x + z[3 * r + c].y * z[3 * r + c].y;
    const double inv = 1.0 / sqrt(nn);
    for (int r = 0; r < 3; ++r) z[3 * r + c] = inv * z[3 * r + c];
  }
  const C det = z[0] * (z[4] * z[8] - z[5] * z[7]) - z[1] * (z[3] * z[8] - z[5] * z[6]) + z[2] * (z[3] * z[7] - z[4] * z[6]);
  const C f = cj(det);
  for (int r = 0; r < 3; ++r) z[3 * r + 2] = z[3 * r + 2] * f;
}

__device__ void reunitarise(C m[9]) {
  double n0 = 0;
  for (int k = 0; k < 3; ++k) n0 += m[k].x * m[k].x + m[k].y * m[k].y;
  n0 = 1.0 / sqrt(n0);
  for (int k = 0; k < 3; ++k) m[k] = n0 * m[k];
  C d = mk<double>(0, 0);
  for (int k = 0; k < 3; ++k) d = d + cjmul(m[k], m[3 + k]);
  for (int k = 0; k < 3; ++k) m[3 + k] = m[3 + k] - d * m[k];
  double n1 = 0;
  for (int k = 0; k < 3; ++k) n1 += m[3 + k].x * m[3 + k].x + m[3 + k].y * m[3 + k].y;
  n1 = 1.0 / sqrt(n1);
  for (int k = 0; k < 3; ++k) m[3 + k] = n1 * m[3 + k];
  reconstruct_row2(m);
}

__device__ void expH(uint64_t seed, uint32_t fid, uint64_t link, double eps, C E[9]) {
  double h[8];
  for (int k = 0; k < 4; ++k) gauss2(seed, fid, link, (uint32_t)k, TAG_GAUGE, h[2 * k], h[2 * k + 1]);
  const double is3 = 0.57735026918962576450914878050196;
  C H[9];
  H[0] = mk<double>(0.5 * (h[2] + h[7] * is3), 0);
  H[4] = mk<double>(0.5 * (-h[2] + h[7] * is3), 0);
  H[8] = mk<double>(0.5 * (-2.0 * h[7] * is3), 0);
  H[1] = mk<double>(0.5 * h[0], -0.5 * h[1]);
  H[3] = cj(H[1]);
  H[2] = mk<double>(0.5 * h[3], -0.5 * h[4]);
  H[6] = cj(H[2]);
  H[5] = mk<double>(0.5 * h[5], -0.5 * h[6]);
  H[7] = cj(H[5]);
  C A[9];
  double fn = 0;
  for (int k = 0; k < 9; ++k) {
    A[k] = mk<double>(-eps * H[k].y, eps * H[k].x);  // i eps H
    fn += A[k].x * A[k].x + A[k].y * A[k].y;
  }
  fn = sqrt(fn);
  int s = 0;
  while (fn > 0.25) {
    fn *= 0.5;
    ++s;
  }
  const double scale = ldexp(1.0, -s);
  for (int k = 0; k < 9; ++k) A[k] = scale * A[k];
  for (int k = 0; k < 9; ++k) E[k] = mk<double>((k % 4 == 0) ? 1.0 : 0.0, 0);
  for (int n = 18; n >= 1; --n) {
    C P[9];
    for (int r = 0; r < 3; ++r)
      for (int c = 0; c < 3; ++c) P[3 * r + c] = A[3 * r] * E[c] + A[3 * r + 1] * E[3 + c] + A[3 * r + 2] * E[6 + c];
    const double inv = 1.0 / (double)n;
    for (int k = 0; k < 9; ++k) E[k] = mk<double>(((k % 4 == 0) ? 1.0 : 0.0) + P[k].x * inv, P[k].y * inv);
  }
  for (int q = 0; q < s; ++q) {
    C T[9];
    for (int r = 0; r < 3; ++r)
      for (int c = 0; c < 3; ++c) T[3 * r + c] = E[3 * r] * E[c] + E[3 * r + 1] * E[3 + c] + E[3 * r + 2] * E[6 + c];
    for (int k = 0; k < 9; ++k) E[k] = T[k];
  }
  reunitarise(E);
}

struct SiteIdx {
  int c[4];
  int64_t s;
  int p;
  int64_t h;
};
__device__ __forceinline__ SiteIdx site_from_linear(const Geom& g, int64_t s) {
  // V < 2^31: 32-bit multiply-high divisions by the extents
  SiteIdx r;
  unsigned t = (unsigned)s;
  unsigned q = g.dL[3].div(t);
  r.c[3] = (int)(t - q * (unsigned)g.L[3]);
  t = q;
  q = g.dL[2].div(t);
  r.c[2] = (int)(t - q * (unsigned)g.L[2]);
  t = q;
  q = g.dL[1].div(t);
  r.c[1] = (int)(t - q * (unsigned)g.L[1]);
  r.c[0] = (int)q;
  r.s = s;
  r.p = (r.c[0] + r.c[1] + r.c[2] + r.c[3]) & 1;
  r.h = s >> 1;
  return r;
}

__device__ __forceinline__ void store_link64(double2* const* u, int p, int mu, int64_t Vh, int64_t h, const C m[9]) {
  double2* b = u[p] + (int64_t)mu * 9 * Vh + h;
  for (int k = 0; k < 9; ++k) b[k * Vh] = make_double2(m[k].x, m[k].y);
}
__device__ __forceinline__ void load_link64(double2* const* u, int p, int mu, int64_t Vh, int64_t h, C m[9]) {
  const double2* b = u[p] + (int64_t)mu * 9 * Vh + h;
  for (int k = 0; k < 9; ++k) {
    const double2 d = b[k * Vh];
    m[k] = mk<double>(d.x, d.y);
  }
}

struct LinkPtrs {
  double2* u[2];
};

__global__ void gauge_gen_kernel(Geom g, LinkPtrs L, int init, uint64_t seed, uint32_t fid, double eps) {
  const int64_t l = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= 4 * g.V) return;
  const int64_t s = l >> 2;
  const int mu = (int)(l & 3);
  const SiteIdx si = site_from_linear(g, s);
  C m[9];
  if (init == CLG_GAUGE_HAAR)
    haar(seed, fid, (uint64_t)l, m);
  else if (init == CLG_GAUGE_EXPH)
    expH(seed, fid, (uint64_t)l, eps, m);
  else
    for (int k = 0; k < 9; ++k) m[k] = mk<double>((k % 4 == 0) ? 1.0 : 0.0, 0);
  store_link64(L.u, si.p, mu, g.Vh, si.h, m);
}

// max |U U^+ - 1| and |det U - 1| of one link; NaN counts as not unitary
__device__ __forceinline__ double link_deviation(const C m[9]) {
  double w2 = 0.0;
  auto each = [&](auto&& take) {
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = r; c < 3; ++c) {  // U U^+ is Hermitian
        const C d = m[3 * r] * cj(m[3 * c]) + m[3 * r + 1] * cj(m[3 * c + 1]) + m[3 * r + 2] * cj(m[3 * c + 2]);
        take(d.x - (r == c ? 1.0 : 0.0), d.y);
      }
    const C det =
        m[0] * (m[4] * m[8] - m[5] * m[7]) - m[1] * (m[3] * m[8] - m[5] * m[6]) + m[2] * (m[3] * m[7] - m[4] * m[6]);
    take(det.x - 1.0, det.y);
  };
  // one square root per link; a square out of range takes the careful form
  bool in_range = true;
  each([&](double x, double y) {
    const double e = fma(x, x, y * y);
    in_range = in_range && e < 1e300;
    w2 = fmax(w2, e);
  });
  if (in_range) return sqrt(w2);
  double w = 0.0;
  bool nan = false;
  each([&](double x, double y) {
    const double e = hypot(x, y);
    nan = nan || !(e == e);
    w = fmax(w, e);
  });
  return nan ? 1e300 : w;
}

// *worst <- max(*worst, w) over the block (w >= 0, so its bits order as
// integers): one atomic per block, all on one address
__device__ __forceinline__ void block_max(double w, unsigned long long* worst) {
  __shared__ double sm[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) w = fmax(w, __shfl_down_sync(0xffffffffu, w, o));
  if (lane == 0) sm[warp] = w;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < nw; ++k) w = fmax(w, sm[k]);
    atomicMax(worst, (unsigned long long)__double_as_longlong(w));
  }
}

// the low bit of lexicographic site 2h + b of checkerboard (p, h): the pair
// 2h, 2h + 1 shares x, y, z and an even t, so b = (p + x + y + z) & 1
__device__ __forceinline__ int site_low_bit(const Geom& g, int p, int64_t h) {
  int c[4];
  eo_coords(g, 0, h, c);
  return (p + c[0] + c[1] + c[2]) & 1;
}

// 16 bytes of lexicographic data: one access where the caller's array is
// 16-byte aligned, two where it is only 8-byte aligned
__device__ __forceinline__ double2 ld_pair(const double* p, bool al) {
  return al ? __ldcs(reinterpret_cast<const double2*>(p)) : make_double2(__ldcs(p), __ldcs(p + 1));
}
__device__ __forceinline__ void st_pair(double* p, double2 v, bool al) {
  if (al) {
    __stcs(reinterpret_cast<double2*>(p), v);
  } else {
    __stcs(p, v.x);
    __stcs(p + 1, v.y);
  }
}

// CLGBin (link = s*4+mu) or Bridge++ (site x-fastest) <-> even-odd SoA.
// Bound by DRAM: 576 B read and 576 B written per site.  A block moves the 64
// sites of 32 checkerboard indices: the SoA side with lanes over h (512-byte
// rows), the lexicographic side as consecutive 16-byte words, through a shared
// tile with one site per row of 37 words and the two sites of an h half a tile
// apart, so that neither side has bank conflicts.  On the way in it also takes
// every link's deviation from SU(3) (worst, nullable).  32^3x16, each way:
// 98 us, 6.2 TB/s (one thread per link, 288 bytes apart: 183 us, and the
// deviation a second pass over the links of 108 us).
constexpr int GR_H = 32, GR_ROW = 37;
__global__ void __launch_bounds__(256) gauge_reorder_kernel(Geom g, LinkPtrs L, double* buf, int layout, int to_device,
                                                           unsigned long long* worst) {
  __shared__ double2 tile[2 * GR_H * GR_ROW];
  __shared__ int64_t first[2 * GR_H];  // lexicographic word of the tile's sites
  __shared__ int bit[GR_H];            // low bit of the even site of each h
  const int64_t h0 = (int64_t)blockIdx.x * GR_H;
  const int nh = (int)min((int64_t)GR_H, g.Vh - h0);
  const bool al = (reinterpret_cast<uintptr_t>(buf) & 15) == 0;
  if (threadIdx.x < 2 * GR_H) {
    const int j = threadIdx.x >> 1, b = threadIdx.x & 1;
    if (j < nh) {
      const SiteIdx si = site_from_linear(g, 2 * (h0 + j) + b);
      int64_t at = si.s;
      if (layout == CLG_LAYOUT_BRIDGEPP)
        at = si.c[0] + (int64_t)si.c[1] * g.L[0] + (int64_t)si.c[2] * g.L[0] * g.L[1] +
             (int64_t)si.c[3] * g.L[0] * g.L[1] * g.L[2];
      first[threadIdx.x] = at * 36;
      if (b == 0) bit[j] = si.p;  // site 2h even <=> low bit 0 for parity 0
    }
  }
  __syncthreads();
  // this thread's link on the SoA side: warp = (parity, mu), lane = h
  const int j = threadIdx.x & 31, mu = (threadIdx.x >> 5) & 3, p = threadIdx.x >> 7;
  const bool live = j < nh;
  double2* row = tile;
  if (live) row += ((bit[j] ^ p) * GR_H + j) * GR_ROW + mu * 9;
  const int words = 2 * nh * 36;
  double w = 0.0;
  if (to_device) {
    double2 v[9];  // all of a thread's loads are issued before the first is used
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const int i = threadIdx.x + 256 * q, s = i / 36;
      if (i < words) v[q] = ld_pair(buf + 2 * (first[s] + i - 36 * s), al);
    }
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const int i = threadIdx.x + 256 * q, s = i / 36;
      if (i < words) tile[((s & 1) * GR_H + (s >> 1)) * GR_ROW + i - 36 * s] = v[q];
    }
    __syncthreads();
    if (live) {
      C m[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) m[k] = mk<double>(row[k].x, row[k].y);
      store_link64(L.u, p, mu, g.Vh, h0 + j, m);
      if (worst) w = link_deviation(m);
    }
    if (worst) block_max(w, worst);
  } else {
    if (live) {
      C m[9];
      load_link64(L.u, p, mu, g.Vh, h0 + j, m);
#pragma unroll
      for (int k = 0; k < 9; ++k) row[k] = make_double2(m[k].x, m[k].y);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const int i = threadIdx.x + 256 * q, s = i / 36, r = i - 36 * s;
      if (i < words) st_pair(buf + 2 * (first[s] + r), tile[((s & 1) * GR_H + (s >> 1)) * GR_ROW + r], al);
    }
  }
}

// full-lattice CLGBin field data (nc complex per site) <-> one rhs of a field.
// Bound by DRAM (FP64 Wilson: 192 B read and written per site).  A block of 128
// threads moves the 128 sites of 64 checkerboard indices: the field side one
// site per thread with lanes over h, the lexicographic side as consecutive
// 16-byte words, through a shared tile with one site per row of NC + 1 words
// (conflict-free both ways: the two sites of an h lie half a tile apart).
// One Wilson rhs: FP64 on 32^3x16 37 us, 5.5 TB/s, FP32 on 48^3x24 113 us,
// 6.8 TB/s (one thread per site, 192 bytes apart: 86 and 341 us).
template <int P, int NC>
__global__ void __launch_bounds__(128) field_reorder_kernel(Geom g, DField f, int nparity, int rhs, double* buf,
                                                            int to_device) {
  constexpr int XH = 64, ROW = NC + 1;
  __shared__ double2 tile[2 * XH * ROW];
  const int64_t h0 = (int64_t)blockIdx.x * XH;
  const int nh = (int)min((int64_t)XH, g.Vh - h0);
  const bool al = (reinterpret_cast<uintptr_t>(buf) & 15) == 0;
  double* lex = buf + 2 * NC * (2 * h0);
  const int words = 2 * nh * NC;
  const int j = threadIdx.x & (XH - 1), p = threadIdx.x / XH;
  const int64_t h = h0 + j;
  const bool live = j < nh;
  const bool held = nparity == 2 || p == f.first_parity;
  const double2* tr = tile + ((live ? site_low_bit(g, p, h) : 0) * XH + j) * ROW;
  // word i of the tile's lexicographic data: site 2 j + b, component k
  auto slot = [&](int i) {
    const int s = i / NC;
    return ((s & 1) * XH + (s >> 1)) * ROW + i - s * NC;
  };
  if (to_device) {
    double2 w[NC];  // all of a thread's loads are issued before the first is used
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const int i = threadIdx.x + 128 * q;
      if (i < words) w[q] = ld_pair(lex + 2 * i, al);
    }
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const int i = threadIdx.x + 128 * q;
      if (i < words) tile[slot(i)] = w[q];
    }
    __syncthreads();
    if (!live || !held) return;
    C v[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) v[k] = mk<double>(tr[k].x, tr[k].y);
    store_site<P, NC, double>(f.base(rhs, p), f.nbase(rhs, p), f.Vh, h, v);
  } else {
    if (live) {
      C v[NC];
      if (held)
        load_site<P, NC, double>(f.base(rhs, p), f.nbase(rhs, p), f.Vh, h, v);
      else
#pragma unroll
        for (int k = 0; k < NC; ++k) v[k] = mk<double>(0, 0);
      double2* tw = const_cast<double2*>(tr);
#pragma unroll
      for (int k = 0; k < NC; ++k) tw[k] = make_double2(v[k].x, v[k].y);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const int i = threadIdx.x + 128 * q;
      if (i < words) st_pair(lex + 2 * i, tile[slot(i)], al);
    }
  }
}

// The same reorder with the FP64 lexicographic data in mapped pinned host
// memory, read or written by the SMs over the host link (zero copy).  It runs
// on the copy stream beside a solve, so it is built not to disturb one:
//   - a block moves tiles of XS sites; the host side as consecutive 16-byte
//     chunks (whole, contiguous link requests, all a thread's loads issued
//     before the first is used), the device side one site per thread through
//     a shared tile padded to NC + 1 chunks per site (conflict-free);
//   - every access is a streaming one (ld/st .cs, evict-first in L2), so the
//     transfer's bytes do not displace the solve's L2 working set;
//   - a small grid-stride grid: a few blocks keep the link busy, and the SMs
//     stay with the solve.
// Used for FP64 fields only (the transfer format); others take the staging path.
template <int NC>
__global__ void __launch_bounds__(256) field_stream_kernel(Geom g, DField f, int nparity, int rhs, double2* host,
                                                           int to_device) {
  constexpr int XS = 128, ROW = NC + 1, CH = XS * NC, PER = (CH + 255) / 256;
  __shared__ double2 tile[XS * ROW];
  const int64_t ntiles = (g.V + XS - 1) / XS;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t s0 = t * XS;
    const int ns = (int)min((int64_t)XS, g.V - s0);
    double2* hb = host + s0 * NC;
    const int j = threadIdx.x;
    SiteIdx si;
    bool held = false;
    if (j < ns) {
      si = site_from_linear(g, s0 + j);
      held = nparity == 2 || si.p == f.first_parity;
    }
    if (to_device) {
      double2 r[PER];
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        const int i = j + q * 256;
        if (i < ns * NC) r[q] = __ldcs(hb + i);
      }
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        const int i = j + q * 256;
        if (i < ns * NC) tile[i + i / NC] = r[q];
      }
      __syncthreads();
      if (held) {
        double2* b = reinterpret_cast<double2*>(f.base(rhs, si.p));
#pragma unroll
        for (int k = 0; k < NC; ++k) __stcs(b + k * f.Vh + si.h, tile[j * ROW + k]);
      }
    } else {
      if (j < ns) {
        const double2* b = reinterpret_cast<const double2*>(f.base(rhs, held ? si.p : f.first_parity));
#pragma unroll
        for (int k = 0; k < NC; ++k) tile[j * ROW + k] = held ? __ldcs(b + k * f.Vh + si.h) : make_double2(0.0, 0.0);
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        const int i = j + q * 256;
        if (i < ns * NC) __stcs(hb + i, tile[i + i / NC]);
      }
    }
    __syncthreads();  // the tile is refilled by the next iteration
  }
}

template <int P, int NC>
struct SourceF {
  DField f;
  Geom g;
  int rhs0;
  int kind;
  uint64_t seed;
  uint32_t fid;
  int64_t site;
  int comp;
  __device__ bool active(int) const { return true; }
  __device__ void operator()(int r, int p, int64_t h, double*) const {
    // full-lattice index of checkerboard site (p, h)
    int c[4];
    eo_coords(g, p, h, c);
    const int64_t s = site_index(g, c);
    C v[NC];
    const double isq2 = 0.70710678118654752440084436210485;
    if (kind == CLG_SOURCE_GAUSS) {
      for (int k = 0; k < NC; ++k) {
        double a, b;
        gauss2(seed, fid, (uint64_t)s, (uint32_t)k, TAG_SPINOR, a, b);
        v[k] = mk<double>(a * isq2, b * isq2);
      }
    } else if (kind == CLG_SOURCE_Z2) {
      uint32_t w[4] = {(uint32_t)s, (uint32_t)((uint64_t)s >> 32), 0u, TAG_Z2};
      philox(w, (uint32_t)seed, (uint32_t)(seed >> 32) ^ fid);
      for (int k = 0; k < NC; ++k) {
        const int b0 = 2 * k, b1 = 2 * k + 1;
        const uint32_t x0 = w[b0 >> 5] >> (b0 & 31), x1 = w[b1 >> 5] >> (b1 & 31);
        v[k] = mk<double>((x0 & 1u) ? -isq2 : isq2, (x1 & 1u) ? -isq2 : isq2);
      }
    } else if (kind == CLG_SOURCE_Z4) {
      // i^b, b = bits 2k, 2k+1 of one Philox output
      uint32_t w[4] = {(uint32_t)s, (uint32_t)((uint64_t)s >> 32), 0u, TAG_Z4};
      philox(w, (uint32_t)seed, (uint32_t)(seed >> 32) ^ fid);
      for (int k = 0; k < NC; ++k) {
        const uint32_t b = (w[(2 * k) >> 5] >> ((2 * k) & 31)) & 3u;
        v[k] = mk<double>(b == 0 ? 1.0 : (b == 2 ? -1.0 : 0.0), b == 1 ? 1.0 : (b == 3 ? -1.0 : 0.0));
      }
    } else {
      for (int k = 0; k < NC; ++k) v[k] = mk<double>((kind == CLG_SOURCE_POINT && s == site && k == comp) ? 1.0 : 0.0, 0);
    }
    store_site<P, NC, double>(f.base(rhs0 + r, p), f.nbase(rhs0 + r, p), f.Vh, h, v);
  }
  __device__ void finalize(int, const double*) const {}
};

struct PlaqF {
  Geom g;
  LinkPtrs L;
  __device__ bool active(int) const { return true; }
  __device__ void operator()(int, int p, int64_t h, double* acc) const {
    int c[4];
    eo_coords(g, p, h, c);
    double tot = 0;
    for (int mu = 0; mu < 4; ++mu)
      for (int nu = mu + 1; nu < 4; ++nu) {
        int a[4] = {c[0], c[1], c[2], c[3]}, b[4] = {c[0], c[1], c[2], c[3]};
        a[mu] = (a[mu] + 1) % g.L[mu];
        b[nu] = (b[nu] + 1) % g.L[nu];
        const int pa = (a[0] + a[1] + a[2] + a[3]) & 1, pb = (b[0] + b[1] + b[2] + b[3]) & 1;
        C u1[9], u2[9], u3[9], u4[9], P[9], Q[9];
        load_link64(L.u, p, mu, g.Vh, h, u1);
        load_link64(L.u, pa, nu, g.Vh, site_index(g, a) >> 1, u2);
        load_link64(L.u, pb, mu, g.Vh, site_index(g, b) >> 1, u3);
        load_link64(L.u, p, nu, g.Vh, h, u4);
        for (int r = 0; r < 3; ++r)
          for (int cc = 0; cc < 3; ++cc) {
            P[3 * r + cc] = u1[3 * r] * u2[cc] + u1[3 * r + 1] * u2[3 + cc] + u1[3 * r + 2] * u2[6 + cc];
            Q[3 * r + cc] = u4[3 * r] * u3[cc] + u4[3 * r + 1] * u3[3 + cc] + u4[3 * r + 2] * u3[6 + cc];
          }
        for (int k = 0; k < 9; ++k) tot += P[k].x * Q[k].x + P[k].y * Q[k].y;
      }
    acc[0] += tot / 3.0;
  }
  __device__ void finalize(int, const double* s) const {}
};

struct PlaqOut {
  PlaqF f;
  double* out;
  __device__ bool active(int r) const { return f.active(r); }
  __device__ void operator()(int r, int p, int64_t h, double* acc) const { f(r, p, h, acc); }
  __device__ void finalize(int, const double* s) const { out[0] = s[0]; }
};

// warp = 32 consecutive h of one (parity, direction): whole 512-byte rows
__global__ void __launch_bounds__(256) unitarity_kernel(Geom g, LinkPtrs L, unsigned long long* worst) {
  const int64_t h = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int mu = blockIdx.y & 3, p = blockIdx.y >> 2;
  double w = 0.0;
  if (h < g.Vh) {
    C m[9];
    load_link64(L.u, p, mu, g.Vh, h, m);
    w = link_deviation(m);
  }
  block_max(w, worst);
}

}  // namespace

// ---------------------------------------------------------------- host entry points
clg_status gauge_generate(clg_gauge_s* U, int init, uint64_t seed, uint32_t fid, double eps) {
  clg_context_s* ctx = U->lat->ctx;
  const Geom& g = U->lat->g;
  LinkPtrs L{{(double2*)U->u64[0], (double2*)U->u64[1]}};
  if (init == CLG_GAUGE_ZERO) {
    for (int p = 0; p < 2; ++p)
      CLG_CUDA_OK(cudaMemsetAsync(U->u64[p], 0, (size_t)g.Vh * 4 * 9 * sizeof(double2), ctx->stream));
    U->dirty_lowp = true;
    return CLG_SUCCESS;
  }
  const int64_t n = 4 * g.V;
  gauge_gen_kernel<<<(unsigned)((n + 127) / 128), 128, 0, ctx->stream>>>(g, L, init, seed, fid, eps);
  ctx->kernels++;
  CLG_CUDA_OK(cudaGetLastError());
  U->dirty_lowp = true;
  return CLG_SUCCESS;
}

// worst (device, nullable): max over the links of their deviation from SU(3),
// taken on the way in
clg_status gauge_reorder(clg_gauge_s* U, double* dev_buf, int layout, int to_device, unsigned long long* worst) {
  clg_context_s* ctx = U->lat->ctx;
  const Geom& g = U->lat->g;
  LinkPtrs L{{(double2*)U->u64[0], (double2*)U->u64[1]}};
  gauge_reorder_kernel<<<(unsigned)((g.Vh + GR_H - 1) / GR_H), 256, 0, ctx->stream>>>(g, L, dev_buf, layout, to_device,
                                                                                    worst);
  ctx->kernels++;
  CLG_CUDA_OK(cudaGetLastError());
  if (to_device) U->dirty_lowp = true;
  return CLG_SUCCESS;
}

clg_status field_reorder(clg_field_s* f, int rhs, double* dev_buf, int to_device) {
  clg_context_s* ctx = f->lat->ctx;
  const Geom& g = f->lat->g;
  const FieldRef r = f->ref();
  return with_pn(f->prec, f->nc(), [&](auto P, auto NC) -> clg_status {
    field_reorder_kernel<P.value, NC.value>
        <<<(unsigned)((g.Vh + 63) / 64), 128, 0, ctx->stream>>>(g, dfield(r), r.nparity, rhs, dev_buf, to_device);
    ctx->kernels++;
    CLG_CUDA_OK(cudaGetLastError());
    return CLG_SUCCESS;
  });
}

clg_status field_stream(clg_field_s* f, int rhs, double* host_dev, int to_device, cudaStream_t s) {
  clg_context_s* ctx = f->lat->ctx;
  const Geom& g = f->lat->g;
  if (f->prec != CLG_PREC_DOUBLE) return CLG_ERR_BAD_ARG;
  const FieldRef r = f->ref();
  const int64_t tiles = (g.V + 127) / 128;
  const unsigned grid = (unsigned)std::min<int64_t>(tiles, ctx->xfer_blocks);
  double2* h = reinterpret_cast<double2*>(host_dev);
  if (f->nc() == 12)
    field_stream_kernel<12><<<grid, 256, 0, s>>>(g, dfield(r), r.nparity, rhs, h, to_device);
  else
    field_stream_kernel<3><<<grid, 256, 0, s>>>(g, dfield(r), r.nparity, rhs, h, to_device);
  ctx->kernels++;
  CLG_CUDA_OK(cudaGetLastError());
  return CLG_SUCCESS;
}

clg_status field_source(clg_field_s* f, int rhs, int kind, uint64_t seed, uint32_t fid, int64_t site, int comp) {
  clg_context_s* ctx = f->lat->ctx;
  const FieldRef r = f->ref();
  return with_pn(f->prec, f->nc(), [&](auto P, auto NC) {
    SourceF<P.value, NC.value> fn{dfield(r), f->lat->g, rhs, kind, seed, fid, site, comp};
    return launch_sites<0>(ctx, fn, r.first_parity, r.nparity, r.Vh, 1);
  });
}

clg_status gauge_plaquette(clg_gauge_s* U, double* host_out) {
  clg_context_s* ctx = U->lat->ctx;
  const Geom& g = U->lat->g;
  Scratch sd;
  clg_status st = sd.get(ctx, sizeof(double));
  if (st) return st;
  double* d = sd.as<double>();
  PlaqOut fn{PlaqF{g, LinkPtrs{{(double2*)U->u64[0], (double2*)U->u64[1]}}}, d};
  st = launch_sites<1>(ctx, fn, 0, 2, g.Vh, 1);
  if (!st) {
    cudaError_t e = cudaMemcpyAsync(host_out, d, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) st = ctx->fail(cuda_status(e), cudaGetErrorString(e));
    *host_out /= (6.0 * (double)g.V);
  }
  return st;
}

clg_status gauge_unitarity(clg_gauge_s* U, double* host_out) {
  clg_context_s* ctx = U->lat->ctx;
  const Geom& g = U->lat->g;
  Scratch sd;
  clg_status st = sd.get(ctx, sizeof(unsigned long long));
  if (st) return st;
  unsigned long long* d = sd.as<unsigned long long>();
  cudaError_t e = cudaMemsetAsync(d, 0, sizeof(unsigned long long), ctx->stream);
  if (e == cudaSuccess) {
    unitarity_kernel<<<dim3((unsigned)((g.Vh + 255) / 256), 8), 256, 0, ctx->stream>>>(
        g, LinkPtrs{{(double2*)U->u64[0], (double2*)U->u64[1]}}, d);
    ctx->kernels++;
    e = cudaGetLastError();
  }
  double w = 0.0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&w, d, sizeof(w), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return ctx->fail(cuda_status(e), cudaGetErrorString(e));
  *host_out = w;
  return CLG_SUCCESS;
}

}  // namespace clg
