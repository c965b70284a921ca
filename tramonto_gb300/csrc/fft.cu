// Three-dimensional real-to-complex FFTs for the stencil sums (FP64 in the accurate fills and FP64-accurate
// products, FP32 in the FP32 products and fills).
//
// A stencil sum out(i) = sum_o c(o) f(i + o) over the mesh, with the reference's boundary rules, is a
// correlation.  Along a periodic dimension of n nodes it is exactly the circular correlation of period n; along
// any other dimension the padded channel (the field extended by the boundary rules over the stencil's reach h)
// is transformed on a length F >= P = n + 2h, where the circular correlation equals the sum for every interior
// output.  Where the field has one boundary value beyond both ends (walls, bulk), F >= n + h is enough: the positions
// from n on hold that value and serve the reads beyond either end.  Along x the two ends may differ (a wall and a bulk):
// the box holds the high end's value and the outputs next to the low end take the difference times the stencil's weight
// beyond it, a profile in x.  So the transform box is [F2][F1][F0] with F_d = n_d on periodic dimensions (when n_d is a
// product of 2, 3, 5 and 7) and the smallest such F_d >= P_d elsewhere; with the correlation kernel g[(-o) mod F] = c(o)
// (points that wrap onto the same position add up, as the reference folds a stencil wider than a periodic box),
// one forward transform of the field, a product with the kernel's spectrum and one inverse transform give the
// sum at a cost that does not depend on the stencil's length.  At 128^3 with the attraction reach of 25 nodes
// that is a 160 x 128 x 128 box: 2.6e6 points (180 with both ends padded) against 5.8e6 for a box padded in every
// dimension.
//
// The field is real, so only the half spectrum k0 < F0/2 + 1 is kept ([F2][F1][F0/2 + 1] complex): along x two
// real lines are packed as the real and imaginary parts of one complex line, transformed together and split
// by Hermitian symmetry (2A[k] = Z[k] + conj Z[-k], 2B[k] = (Z[k] - conj Z[-k]) / i); the inverse packs
// two half-spectrum lines as Z = A + iB (extended by conjugate symmetry) and returns them as the real and
// imaginary parts of one inverse transform.  The x passes read the padded channel directly and write the
// interior outputs directly (no load or extraction pass); the y and z passes are batches of complex transforms
// over the half-spectrum box.
//
// Each 1-D transform of n = R1 R2 points (R1 >= R2, both <= 27) is two steps held in registers with one exchange
// through shared memory between them (the four-step decomposition, Bailey 1990): R2 threads per line take the R1
// points j2 + R2 r, transform them, multiply by W_n^{j2 k1} and store them; R1 threads read the R2 values of their
// k1, transform them and hold the outputs k1 + R1 k2.  Both steps address global memory themselves, so a y or z pass
// moves its data through shared memory once.  The y and z passes take 16 lines adjacent in x per CTA (16 lanes read
// 128 or 256 contiguous bytes; with the line as the fastest index of the exchange no access conflicts).
// Twiddles are tabulated on the host in extended precision.  The inverse uses conjugate twiddles; its 1/(F0 F1 F2) and
// the 1/2 of the split into two real lines are factors of the kernels' coefficients (1.6% of an FP64 fill).  The
// spectral products (one kernel spectrum per output, or the sum of channel-times-kernel products of a transposed sum)
// are formed while the first inverse pass loads its lines; FP32 sums of several products by a pass of their own.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "fft_dft.h"
#include "tgpu_internal.h"

namespace tgpu {

using dft::cfma;
using dft::cmul;

namespace {

constexpr int kFftMaxN = 432;      // longest transform
// adjacent lines per CTA of a y or z pass: 128 contiguous bytes, and CTAs small enough that several share an SM (one
// loads while another computes)
template <class C>
constexpr int lines_per_cta() { return 128 / (int)sizeof(C); }
constexpr int kMaxRadix = 27;

// f(integral_constant<int, R>) for the register DFT lengths LO < R <= HI
template <int LO, int HI, class F>
__device__ __forceinline__ void with_radix(int R, F &&f)
{
#define TGPU_RADIX(r)                                                              \
  case r:                                                                          \
    if constexpr (r > LO && r <= HI) f(std::integral_constant<int, r>{});          \
    break;
  switch (R) {
    TGPU_RADIX(1) TGPU_RADIX(2) TGPU_RADIX(3) TGPU_RADIX(4) TGPU_RADIX(5) TGPU_RADIX(6) TGPU_RADIX(7) TGPU_RADIX(8)
    TGPU_RADIX(9) TGPU_RADIX(10) TGPU_RADIX(12) TGPU_RADIX(14) TGPU_RADIX(15) TGPU_RADIX(16) TGPU_RADIX(18)
    TGPU_RADIX(20) TGPU_RADIX(21) TGPU_RADIX(24) TGPU_RADIX(25) TGPU_RADIX(27)
  }
#undef TGPU_RADIX
}

// a line's two radices and twiddle table exp(-2 pi i k / n), k < n
template <class C>
struct Line1d {
  int R1, R2;
  const C *tw;
};

// v[k] *= W^{j k} (INV: conjugate)
template <int R, bool INV, class C>
__device__ __forceinline__ void twiddle(C *v, const C *__restrict__ tw, int j)
{
#pragma unroll
  for (int k = 1; k < R; k++) {
    C w = __ldg(tw + j * k);
    if (INV) w.y = -w.y;
    v[k] = cmul(v[k], w);
  }
}

// Geometry of the real box as the x passes see it: where a line's values come from (forward) or go to (inverse)
struct XGeom {
  int F0, F1, Fh, Fp;        // transform lengths along x and y, half-spectrum length along x and its pitch
  long nlines;               // real lines F1 * F2
  // forward source: element (x, y, z) of the box is the source at padded position (x + off0, y + off1, z + off2)
  // when x < ext0, y < ext1, z < ext2, else 0
  int off[3], ext[3];
  // inverse destination: box position p holds output node p - e (interior nodes only)
  int e[3], nx[3];
  int last[3];               // last padded position (box positions past it read the same boundary value)
  int flat0;                 // x holds the nodes, then one boundary value to the end
};

// Sources of the forward x pass: element (x, y, z) of the real box (x < ext0, y < ext1, z < ext2; 0 beyond)
// at padded position (x + off0, y + off1, z + off2).  A line's y and z are resolved once (line); load then takes its
// elements first + x0, + 32, ..., all loads issued before their values are used, and at() any position around them.
template <class T>
struct BoxSrc {   // a real box [F2][F1][F0] (off 0)
  const T *p;
  long sy, sz;
  using Line = const T *;
  __device__ __forceinline__ Line line(const XGeom &g, int y, int z) const
  {
    return p + (long)(z + g.off[2]) * sz + (long)(y + g.off[1]) * sy + g.off[0];
  }
  // positions first .. first + count - 1 are the ones load reads: here all within the source's extent
  __device__ __forceinline__ int first(const XGeom &) const { return 0; }
  __device__ __forceinline__ int count(const XGeom &g) const { return g.ext[0]; }
  template <int NB>
  __device__ __forceinline__ void load(const Line &L, bool use, int x0, int n, T *v) const
  {
#pragma unroll
    for (int u = 0; u < NB; u++) v[u] = use && x0 + 32 * u < n ? L[x0 + 32 * u] : (T)0;
  }
  __device__ __forceinline__ T at(const XGeom &, const Line &L, int x) const { return L[x]; }
  __device__ __forceinline__ T flat(const XGeom &) const { return (T)0; }
};
template <class T>
struct MappedSrc {   // the unpadded channel through the boundary maps (the padded box's values, computed)
  MapSrc m;
  T lo, hi;          // the bulk values in arithmetic T (converted once)
  MappedSrc() : lo(0), hi(0) {}
  explicit MappedSrc(const MapSrc &s) : m(s), lo((T)s.bulk_lo), hi((T)s.bulk_hi) {}
  // the node offset and reflections of the line, or the sentinel of its first out-of-range dimension after x
  // (x still decides first)
  struct Line {
    long base;
    int refl, sent;   // sent 0: the line is inside
  };
  __device__ __forceinline__ Line line(const XGeom &g, int y, int z) const
  {
    Line L{0, 0, 0};
    const int q[3] = {0, min(y + g.off[1], g.last[1]), min(z + g.off[2], g.last[2])};
    long idx[3] = {0, 0, 0};
    for (int d = 1; d < m.ndim; d++) {
      const int v = m.map[d][q[d]];
      if (v < 0) {
        L.sent = v;
        return L;
      }
      if (v & kReflBit) L.refl |= 1 << d;
      idx[d] = v & ~kReflBit;
    }
    L.base = (long)m.nx[0] * (idx[1] + (long)m.nx[1] * idx[2]);
    return L;
  }
  __device__ __forceinline__ T sentinel(int v) const
  {
    if (v == kSentBulk) return lo;
    if (v == kSentBulkHi) return hi;
    if (v == kSentWall) return (T)0;
    return (T)__longlong_as_double(0x7ff8000000000000ULL);   // no node to read (as the padded box holds)
  }
  __device__ __forceinline__ T at(const XGeom &g, const Line &L, int x) const
  {
    const int v = m.map[0][min(x + g.off[0], g.last[0])], out = v < 0 ? v : L.sent;
    if (out) return sentinel(out);
    const int refl = L.refl | ((v & kReflBit) ? 1 : 0);
    const long node = L.base + (v & ~kReflBit);
    const T val = m.src32 ? (T)m.src32[node] : to_arith<T>(m.src[node]);
    if (m.zc >= 0 && m.zero[(long)m.zc * m.N + node]) return (T)0;
    return (__popc(refl & m.signmask) & 1) ? -val : val;
  }
  // the boundary value that follows the nodes of a flat x (x decides first: also on lines outside the mesh)
  __device__ __forceinline__ T flat(const XGeom &g) const { return sentinel(m.map[0][g.last[0]]); }
  // the mesh's nodes: the box holds node i at x = e[0] + i, with no map to read
  __device__ __forceinline__ int first(const XGeom &g) const { return g.e[0]; }
  __device__ __forceinline__ int count(const XGeom &) const { return m.nx[0]; }
  // nodes x0, x0 + 32, ... of a line; a line outside the mesh reads its sentinel's value
  template <int NB>
  __device__ __forceinline__ void load(const Line &L, bool use, int x0, int n, T *v) const
  {
    if (!use || L.sent) {
      const T c = use ? sentinel(L.sent) : (T)0;
#pragma unroll
      for (int u = 0; u < NB; u++) v[u] = c;
      return;
    }
    if (m.src32) {
      const float *s = m.src32 + L.base;
#pragma unroll
      for (int u = 0; u < NB; u++) v[u] = x0 + 32 * u < n ? (T)s[x0 + 32 * u] : (T)0;
    } else {
      const double *s = m.src + L.base;
      double t[NB];
#pragma unroll
      for (int u = 0; u < NB; u++) t[u] = x0 + 32 * u < n ? s[x0 + 32 * u] : 0.0;
#pragma unroll
      for (int u = 0; u < NB; u++) v[u] = to_arith<T>(t[u]);
    }
    if (m.zc >= 0) {
      const signed char *z = m.zero + (long)m.zc * m.N + L.base;
      signed char f[NB];
#pragma unroll
      for (int u = 0; u < NB; u++) f[u] = x0 + 32 * u < n ? z[x0 + 32 * u] : (signed char)0;
#pragma unroll
      for (int u = 0; u < NB; u++)
        if (f[u]) v[u] = 0;
    }
    if (__popc(L.refl & m.signmask) & 1) {
#pragma unroll
      for (int u = 0; u < NB; u++) v[u] = -v[u];
    }
  }
};

// spectral products formed by a pass as it loads its lines: value = sum_t a_t * k_t (n = 0: the input itself)
constexpr int kMaxTerms = 9;   // the adjoint's channels of one density: 5 and up to 4 mean fields
template <class C>
struct Terms {
  const C *a[kMaxTerms];
  const C *k[kMaxTerms];
  int n;
};

// up to kMaxBatch transforms of one plan in one launch (blockIdx.y selects the transform)
constexpr int kMaxBatch = 8;
template <class C>
struct PassBatch {
  const C *in[kMaxBatch];
  C *out[kMaxBatch];
  Terms<C> terms[kMaxBatch];
};

template <class Src, class C>
struct SrcBatch {
  Src src[kMaxBatch];
  C *spec[kMaxBatch];
};

template <class C>
struct OutBatch {
  const C *spec[kMaxBatch];
  double *out[kMaxBatch];
  float *out32[kMaxBatch];   // FP32 outputs (the FP32 transforms; used instead of out when set)
  FftProfile prof[kMaxBatch];
  FftCopies copies[kMaxBatch];
};

// ---- y and z passes ---------------------------------------------------------------------------------------------
// Bound: FP32 by latency (issue 50%, L2 27%: load, exchange, store with four CTAs per SM), FP64 by the FP64 pipe
// (~80% of its 304 operations per clock).  Measured on the 160 x 128 x 128 box of 128^3 nodes (81 x 128 x 128 half
// spectrum), five FP32 forward transforms per launch 21.7 us = 4.9 TB/s of spectrum read and written; six FP64 inverse
// transforms with their products 365 us.  Against radix-4 stages that each went through shared memory, both on a 180 x
// 128 x 128 box: 39 -> 26 us and 430 -> 400.
// lines_per_cta adjacent lines (element stride es) at one outer index; reads `in` (or, inverse, the products of `terms`) and
// writes `out` (in place when out == in: a CTA has read its lines before it writes them).  R1 in (LO, HI]: one kernel
// per range of radices, so that short ones do not carry the registers of long ones.
template <class C, int LO, int HI, bool INV>
__global__ void __launch_bounds__(lines_per_cta<C>() * HI) k_fft_lines(PassBatch<C> pb, int X, unsigned nlines,
                                                                           Line1d<C> ln, long es, long outer_stride)
{
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int kLines = lines_per_cta<C>();
  C *sm = reinterpret_cast<C *>(smraw);
  const C *in = pb.in[blockIdx.y];
  C *out = pb.out[blockIdx.y];
  const int l = threadIdx.x & (kLines - 1), q = threadIdx.x / kLines;
  const int R1 = ln.R1, R2 = ln.R2;
  // FP64 (bound by its arithmetic): lines numbered through the outer indices, so that only the last CTA has idle ones.
  // FP32 (bound by its accesses): CTAs start at multiples of 16 in x, on 128-byte boundaries (81 x 128 x 128 points, a
  // forward pass of one and five transforms: 12.6 us; numbered through 14.0; FP64 172 and 161 us).
  unsigned o, x;
  bool live;
  if constexpr (std::is_same<C, double2>::value) {
    const unsigned line = blockIdx.x * kLines + l;
    o = line / (unsigned)X;
    x = line - o * X;
    live = line < nlines;
  } else {
    const unsigned xblocks = (X + kLines - 1) / kLines;
    o = blockIdx.x / xblocks;
    x = (blockIdx.x - o * xblocks) * kLines + l;
    live = x < (unsigned)X;
  }
  const long base = (long)o * outer_stride + x;
  if (q < R2 && live)
    with_radix<LO, HI>(R1, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      C v[R];
      const long i0 = base + q * es, step = R2 * es;
      bool plain = true;
      if constexpr (INV) {
        const Terms<C> &terms = pb.terms[blockIdx.y];
        plain = terms.n == 0;
        if (!plain) {
          const C *a = terms.a[0] + i0, *k = terms.k[0] + i0;
#pragma unroll
          for (int r = 0; r < R; r++) v[r] = cmul(a[r * step], __ldg(k + r * step));
          if (std::is_same<C, double2>::value) {   // (FP32 sums of several products: launch_spec_terms)
            for (int t = 1; t < terms.n; t++) {
              a = terms.a[t] + i0;
              k = terms.k[t] + i0;
#pragma unroll
              for (int r = 0; r < R; r++) v[r] = cfma(a[r * step], __ldg(k + r * step), v[r]);
            }
          }
        }
      }
      if (plain) {
        const C *p = in + i0;
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = p[r * step];
      }
      dft::run<R, INV, C>(v);
      twiddle<R, INV, C>(v, ln.tw, q);
#pragma unroll
      for (int r = 0; r < R; r++) sm[(r * R2 + q) * kLines + l] = v[r];
    });
  __syncthreads();
  if (live)
    with_radix<0, HI>(R2, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      const long step = R1 * es;
      for (int k = q; k < R1; k += blockDim.x / kLines) {
        C v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = sm[(k * R + r) * kLines + l];
        dft::run<R, INV, C>(v);
        C *p = out + base + k * es;
#pragma unroll
        for (int r = 0; r < R; r++) p[r * step] = v[r];
      }
    });
}

// ---- x passes ---------------------------------------------------------------------------------------------------
// A CTA takes up to kXPairs complex lines (pairs of real ones).  A line's values lie along x, so they are staged through
// shared memory: one warp reads or writes a line with consecutive lanes, and the two register steps work on the tile.
// (Register steps that read and wrote global memory themselves, in runs of R1 or R2 elements, took 87 instead of 36 us
// per FP32 inverse launch.)  Bound as the y and z passes; 128^3 workload (160 x 128 x 128 box), per launch of 1 and 5 or 6
// lines' transforms: forward 35 us in FP32, inverse 28; FP64 232 and 278.  Against radix-4 stages, both on a 180 x 128 x 128
// box: 47 -> 42, 33 -> 35, 318 -> 271 and 338 -> 274.
// Eight pairs per CTA: more and smaller CTAs than sixteen overlap one's loads with another's steps in FP32 (forward 37.3
// -> 35.0 us, inverse 29.1 -> 27.7 on the 160 x 128 x 128 box; four: the same).
constexpr int kXPairs = 8;
constexpr int kXBatch = 4;   // positions a lane loads before it stores them

// shared pitch of the R2 values of one k1: odd, so that the R1 threads of a line read distinct banks
__host__ __device__ __forceinline__ int pitch2(int R2) { return R2 | 1; }

// the tile's transforms in place: sm[p * lp + x] -> sm[p * lp + k] (lp >= n and >= R1 pitch2(R2))
template <int LO, int HI, bool INV, class C>
__device__ __forceinline__ void tile_fft(C *sm, int NP, int lp, const Line1d<C> &ln)
{
  const int R1 = ln.R1, R2 = ln.R2, pr = pitch2(R2);
  __syncthreads();
  with_radix<LO, HI>(R1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int l = threadIdx.x / R2, j = threadIdx.x - l * R2;
    C v[R];
    if (l < NP) {
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = sm[l * lp + r * R2 + j];
      dft::run<R, INV, C>(v);
      twiddle<R, INV, C>(v, ln.tw, j);
    }
    __syncthreads();   // (uniform: every thread takes the same radix)
    if (l < NP) {
#pragma unroll
      for (int r = 0; r < R; r++) sm[l * lp + r * pr + j] = v[r];
    }
  });
  __syncthreads();
  with_radix<0, HI>(R2, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int l = threadIdx.x / R1, k1 = threadIdx.x - l * R1;
    C v[R];
    if (l < NP) {
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = sm[l * lp + k1 * pr + r];
      dft::run<R, INV, C>(v);
    }
    __syncthreads();
    if (l < NP) {
#pragma unroll
      for (int r = 0; r < R; r++) sm[l * lp + k1 + r * R1] = v[r];
    }
  });
  __syncthreads();
}

// forward: two real lines per complex line, split into two half-spectrum lines by Hermitian symmetry
template <class T, class C, class Src, int LO, int HI>
__global__ void __launch_bounds__((kXPairs * HI + 31) / 32 * 32) k_rfft_lines(SrcBatch<Src, C> sb, XGeom g,
                                                                               Line1d<C> ln, int NP, int lp)
{
  const Src src = sb.src[blockIdx.y];
  C *__restrict__ spec = sb.spec[blockIdx.y];
  extern __shared__ __align__(16) unsigned char smraw[];
  C *sm = reinterpret_cast<C *>(smraw);
  const int n = g.F0, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int npairs = (int)((g.nlines + 1) / 2), pair0 = blockIdx.x * NP, np = min(NP, npairs - pair0);
  const T beyond = g.flat0 ? src.flat(g) : (T)0;
  for (int p = warp; p < np; p += nw) {
    const int L = 2 * (pair0 + p);
    const int z0 = L / g.F1, y0 = L - z0 * g.F1, y1 = y0 + 1 < g.F1 ? y0 + 1 : 0, z1 = y0 + 1 < g.F1 ? z0 : z0 + 1;
    // (lines beyond the source's extent are zeros and read no map)
    const bool r0 = y0 < g.ext[1] && z0 < g.ext[2];
    const bool r1 = L + 1 < g.nlines && y1 < g.ext[1] && z1 < g.ext[2];
    const typename Src::Line l0 = r0 ? src.line(g, y0, z0) : typename Src::Line{};
    const typename Src::Line l1 = r1 ? src.line(g, y1, z1) : typename Src::Line{};
    // the mesh's nodes of both lines, with no test per node but the zero-density flag, then the positions around them
    const int e0 = src.first(g), nn = src.count(g);
    C *row = sm + p * lp;
    for (int x0 = lane; x0 < nn; x0 += 32 * kXBatch) {
      T a[kXBatch], b[kXBatch];
      src.template load<kXBatch>(l0, r0, x0, nn, a);
      src.template load<kXBatch>(l1, r1, x0, nn, b);
#pragma unroll
      for (int u = 0; u < kXBatch; u++)
        if (x0 + 32 * u < nn) row[e0 + x0 + 32 * u] = C{a[u], b[u]};
    }
    if (g.flat0) {
      const C v = C{r0 ? beyond : (T)0, r1 ? beyond : (T)0};
      for (int x = nn + lane; x < n; x += 32) row[x] = v;
      continue;
    }
    for (int t = lane; t < n - nn; t += 32) {
      const int x = t < e0 ? t : t + nn;
      C v = C{0, 0};
      if (x < g.ext[0]) {
        if (r0) v.x = src.at(g, l0, x);
        if (r1) v.y = src.at(g, l1, x);
      }
      row[x] = v;
    }
  }
  tile_fft<LO, HI, false, C>(sm, NP, lp, ln);
  for (int p = warp; p < np; p += nw) {
    const long L = 2 * (long)(pair0 + p);
    const bool two = L + 1 < g.nlines;
    C *o = spec + L * g.Fp;
    for (int k = lane; k < g.Fh; k += 32) {
      const C Z = sm[p * lp + k], Zm = sm[p * lp + (k == 0 ? 0 : n - k)];
      o[k] = C{Z.x + Zm.x, Z.y - Zm.y};   // twice the spectrum: the kernels carry the factor
      if (two) o[g.Fp + k] = C{Z.y + Zm.y, Zm.x - Z.x};
    }
  }
}

// one output line: out = value (+ out when accumulate), every load before the stores; times is a further factor of
// an output that is a multiple of the transform's (TIMES)
template <bool TIMES, class O, class C>
__device__ __forceinline__ void write_line(const C *z, bool imag, O *o, double times, int nx0, bool accumulate,
                                           const FftProfile &prof, int lane)
{
  for (int x0 = lane; x0 < nx0; x0 += 32 * kXBatch) {
    O old[kXBatch];
#pragma unroll
    for (int u = 0; u < kXBatch; u++) old[u] = accumulate && x0 + 32 * u < nx0 ? o[x0 + 32 * u] : (O)0;
#pragma unroll
    for (int u = 0; u < kXBatch; u++)
      if (x0 + 32 * u < nx0) {
        const C r = z[x0 + 32 * u];
        O v = (O)(imag ? r.y : r.x);
        if (prof.n > 0) v += (O)(prof.c[0] * prof.s[0][x0 + 32 * u]);
        if (prof.n > 1) v += (O)(prof.c[1] * prof.s[1][x0 + 32 * u]);
        if (TIMES) v *= (O)times;
        o[x0 + 32 * u] = accumulate ? old[u] + v : v;
      }
  }
}

// inverse: two half-spectrum lines as one complex line Z = A + iB, whose inverse's real and imaginary parts are the
// outputs of the interior nodes (out[node] = value, or += when accumulate)
template <class C, int LO, int HI>
__global__ void __launch_bounds__((kXPairs * HI + 31) / 32 * 32) k_irfft_lines(OutBatch<C> ob, XGeom g,
                                                                                Line1d<C> ln, int NP, int lp,
                                                                                int accumulate)
{
  const C *__restrict__ spec = ob.spec[blockIdx.y];
  extern __shared__ __align__(16) unsigned char smraw[];
  C *sm = reinterpret_cast<C *>(smraw);
  const int n = g.F0, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int npairs = (int)((g.nlines + 1) / 2), pair0 = blockIdx.x * NP, np = min(NP, npairs - pair0);
  for (int p = warp; p < np; p += nw) {
    const long L = 2 * (long)(pair0 + p);
    const bool two = L + 1 < g.nlines;
    const C *a = spec + L * g.Fp;
    for (int k = lane; k < g.Fh; k += 32) {
      const C A = a[k], B = two ? a[g.Fp + k] : C{0, 0};
      // A + iB on the stored half, conj(A) + i conj(B) on the mirrored half
      sm[p * lp + k] = C{A.x - B.y, A.y + B.x};
      if (k > 0 && 2 * k < n) sm[p * lp + n - k] = C{A.x + B.y, B.x - A.y};
    }
  }
  tile_fft<LO, HI, true, C>(sm, NP, lp, ln);
  const int nx0 = g.nx[0];
  const FftProfile prof = ob.prof[blockIdx.y];
  const int copies = ob.copies[blockIdx.y].n;
  for (int p = warp; p < np; p += nw) {
    const int L = 2 * (pair0 + p);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (L + h >= g.nlines) break;
      const int zz = (L + h) / g.F1, y = (L + h) - zz * g.F1 - g.e[1], z = zz - g.e[2];
      if (y < 0 || y >= g.nx[1] || z < 0 || z >= g.nx[2]) continue;
      const long row = ((long)z * g.nx[1] + y) * nx0;
      const C *zl = sm + p * lp + g.e[0];
      const bool acc = accumulate != 0;
      if (std::is_same<C, float2>::value && ob.out32[blockIdx.y]) {
        write_line<false, float>(zl, h != 0, ob.out32[blockIdx.y] + row, 1.0, nx0, acc, prof, lane);
        for (int q = 0; q < copies; q++)
          write_line<true, float>(zl, h != 0, ob.copies[blockIdx.y].out32[q] + row, ob.copies[blockIdx.y].f[q], nx0,
                                     acc, prof, lane);
      } else {
        write_line<false, double>(zl, h != 0, ob.out[blockIdx.y] + row, 1.0, nx0, acc, prof, lane);
        for (int q = 0; q < copies; q++)
          write_line<true, double>(zl, h != 0, ob.copies[blockIdx.y].out[q] + row, ob.copies[blockIdx.y].f[q], nx0,
                                      acc, prof, lane);
      }
    }
  }
}

// correlation kernel of coefficient q of a stencil in the real box: coef[k * ncoef + q] added at (-dir offset_k) mod F
// (offsets that wrap onto the same position add up); dir 1: sums over f(i + offset), -1: over f(i - offset)
__global__ void k_fft_kernel_box(const short *__restrict__ off3, const double *__restrict__ coef, int L, int ncoef,
                                 int q, int dir, double scale, double *__restrict__ box, int F0, int F1, int F2)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= L) return;
  const int x = ((-dir * (int)off3[3 * k]) % F0 + F0) % F0;
  const int y = ((-dir * (int)off3[3 * k + 1]) % F1 + F1) % F1;
  const int z = ((-dir * (int)off3[3 * k + 2]) % F2 + F2) % F2;
  atomicAdd(box + ((long)z * F1 + y) * F0 + x, scale * coef[(long)k * ncoef + q]);
}

// the products of `t` as a spectrum, two points per thread and iteration, every term's loads issued before the sums
template <int N, class C>
__global__ void __launch_bounds__(256) k_spec_terms(Terms<C> t, C *__restrict__ out, long n)
{
  for (long i = 2 * (blockIdx.x * (long)blockDim.x + threadIdx.x); i < n; i += 2L * gridDim.x * blockDim.x) {
    C a[N][2], k[N][2];
#pragma unroll
    for (int j = 0; j < N; j++) {
      if constexpr (std::is_same<C, float2>::value) {   // (spectra are 256-byte aligned and n is even)
        const float4 va = *reinterpret_cast<const float4 *>(t.a[j] + i), vk = *reinterpret_cast<const float4 *>(t.k[j] + i);
        a[j][0] = C{va.x, va.y};
        a[j][1] = C{va.z, va.w};
        k[j][0] = C{vk.x, vk.y};
        k[j][1] = C{vk.z, vk.w};
      } else {
        for (int h = 0; h < 2; h++) {
          a[j][h] = t.a[j][i + h];
          k[j][h] = t.k[j][i + h];
        }
      }
    }
    C v[2] = {cmul(a[0][0], k[0][0]), cmul(a[0][1], k[0][1])};
#pragma unroll
    for (int j = 1; j < N; j++)
      for (int h = 0; h < 2; h++) v[h] = cfma(a[j][h], k[j][h], v[h]);
    out[i] = v[0];
    out[i + 1] = v[1];
  }
}

template <class C>
void launch_spec_terms(const Terms<C> &t, C *out, long n, cudaStream_t s)
{
  const int grid = (int)std::min<long>((n / 2 + 255) / 256, 152L * 8);
  switch (t.n) {
#define TGPU_TERMS(N) case N: k_spec_terms<N, C><<<grid, 256, 0, s>>>(t, out, n); break;
    TGPU_TERMS(1) TGPU_TERMS(2) TGPU_TERMS(3) TGPU_TERMS(4) TGPU_TERMS(5) TGPU_TERMS(6) TGPU_TERMS(7) TGPU_TERMS(8)
    TGPU_TERMS(9)
#undef TGPU_TERMS
  }
  static_assert(kMaxTerms == 9, "a case per number of terms");
}

__global__ void k_to_float2(const double2 *__restrict__ in, float2 *__restrict__ out, long n)
{
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    out[i] = make_float2((float)in[i].x, (float)in[i].y);
}

int grid_for(long n) { return (int)std::min<long>((n + 255) / 256, 152L * 16); }

// the two radices of a length: the factors nearest each other among the register DFT lengths (every product of 2, 3,
// 5 and 7 up to 432 but 245, 343 and 392 has them)
bool radices_of(int F, int &R1, int &R2)
{
  static const int kRadix[] = {1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16, 18, 20, 21, 24, 25, 27};
  if (F < 1 || F > kFftMaxN) return false;
  for (int a : kRadix)
    for (int b : kRadix)
      if (b <= a && a * b == F) {
        R1 = a;
        R2 = b;
        return true;
      }
  return false;
}

// the range (LO, HI] of a kernel's first radix: f(integral_constant LO, integral_constant HI)
template <class F>
void with_range(int R1, F &&f)
{
  if (R1 <= 10) f(std::integral_constant<int, 0>{}, std::integral_constant<int, 10>{});
  else if (R1 <= 16) f(std::integral_constant<int, 10>{}, std::integral_constant<int, 16>{});
  else f(std::integral_constant<int, 16>{}, std::integral_constant<int, kMaxRadix>{});
}

template <class C>
Line1d<C> line_of(const FftAxis &a)
{
  if constexpr (std::is_same<C, float2>::value) return Line1d<C>{a.R1, a.R2, a.d_tw32};
  else return Line1d<C>{a.R1, a.R2, a.d_tw};
}

// Threads per line of a y or z pass: R2 (every thread has a first step, a few take two second steps) unless that leaves
// over a quarter of the second step's rounds idle, else R1.  128 = 16 x 8 with eight: twice the CTAs per SM, all of their
// warps loading (five FP32 forward transforms 26 -> 22 us).
int line_threads(const FftAxis &a)
{
  const int rounds = (a.R1 + a.R2 - 1) / a.R2, slots = rounds * a.R2;
  return 4 * (slots - a.R1) <= slots ? a.R2 : a.R1;
}
template <class C>
size_t lines_smem(const FftAxis &a) { return sizeof(C) * (size_t)lines_per_cta<C>() * a.n; }
int x_pairs(long npairs, int nb)   // fewer pairs per CTA where whole tiles would leave SMs idle (2-D boxes)
{
  int np = kXPairs;
  while (np > 2 && (npairs + np - 1) / np * nb < 2 * 152) np /= 2;
  return np;
}
int x_threads(const FftAxis &a, int np) { return (np * a.R1 + 31) / 32 * 32; }
int x_pitch(const FftAxis &a) { return std::max(a.R1 * pitch2(a.R2), a.n) | 1; }   // of a line in the tile
template <class C>
size_t x_smem(const FftAxis &a, int np) { return sizeof(C) * (size_t)np * x_pitch(a); }

template <class T, class C>
void set_smem_limits(const FftPlan &p)
{
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  const int most_x = (int)(sizeof(C) * kXPairs * (kMaxRadix * (kMaxRadix | 1) + 1)), most = 128 * kFftMaxN;
  with_range(p.ax[0].R1, [&](auto lo, auto hi) {
    constexpr int LO = decltype(lo)::value, HI = decltype(hi)::value;
    cudaFuncSetAttribute(k_rfft_lines<T, C, BoxSrc<T>, LO, HI>, attr, most_x);
    cudaFuncSetAttribute(k_rfft_lines<T, C, MappedSrc<T>, LO, HI>, attr, most_x);
    cudaFuncSetAttribute(k_irfft_lines<C, LO, HI>, attr, most_x);
  });
  for (int d = 1; d <= 2; d++)
    with_range(p.ax[d].R1, [&](auto lo, auto hi) {
      constexpr int LO = decltype(lo)::value, HI = decltype(hi)::value;
      cudaFuncSetAttribute(k_fft_lines<C, LO, HI, false>, attr, most);
      cudaFuncSetAttribute(k_fft_lines<C, LO, HI, true>, attr, most);
    });
}

XGeom xgeom(const FftPlan &p)
{
  XGeom g{};
  g.F0 = p.F[0];
  g.F1 = p.F[1];
  g.Fh = p.Fh;
  g.Fp = p.Fp;
  g.nlines = (long)p.F[1] * p.F[2];
  for (int d = 0; d < 3; d++) {
    g.off[d] = p.off[d];
    g.ext[d] = p.ext[d];
    g.e[d] = p.h[d] - p.off[d];
    g.nx[d] = p.nx[d];
    g.last[d] = p.P[d] - 1;
  }
  g.flat0 = p.shared[0];
  return g;
}

// Optional timing of every FP32 y/z pass launch (the solves' leading kernel): a CUDA event pair around each launch
// on its own stream and the launch's algorithmic bytes (per transform the half spectrum written once and read once,
// or the two operands of each spectral product read); collected and reset by pass_timer_collect.
struct PassTimer {
  bool on = false;
  std::vector<cudaEvent_t> ev;   // begin, end of each launch
  std::vector<double> bytes;
  std::vector<int> fields;
};
PassTimer g_pass_timer;

// one y (d = 1) or z (d = 2) pass of nb transforms of the plan in one launch
template <class C>
void strided_pass_batch(const PassBatch<C> &pb, int nb, const FftPlan &p, int d, bool inverse, cudaStream_t s)
{
  const int X = p.Fh;
  const long es = d == 1 ? (long)p.Fp : (long)p.Fp * p.F[1];
  const long outer = d == 1 ? (long)p.Fp * p.F[1] : (long)p.Fp;   // axis 1: outer index z; axis 2: outer index y
  const long nouter = d == 1 ? p.F[2] : p.F[1];
  const FftAxis &ax = p.ax[d];
  constexpr int kLines = lines_per_cta<C>();
  const long nlines = X * nouter;
  const long blocks = std::is_same<C, double2>::value ? (nlines + kLines - 1) / kLines : (X + kLines - 1) / kLines * nouter;
  const dim3 grid((unsigned)blocks, (unsigned)nb);
  const bool timed = std::is_same<C, float2>::value && g_pass_timer.on;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (timed) {
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
  }
  with_range(ax.R1, [&](auto lo, auto hi) {
    constexpr int LO = decltype(lo)::value, HI = decltype(hi)::value;
    if (inverse)
      k_fft_lines<C, LO, HI, true><<<grid, kLines * line_threads(ax), lines_smem<C>(ax), s>>>(pb, X, (unsigned)nlines, line_of<C>(ax), es, outer);
    else
      k_fft_lines<C, LO, HI, false><<<grid, kLines * line_threads(ax), lines_smem<C>(ax), s>>>(pb, X, (unsigned)nlines, line_of<C>(ax), es, outer);
  });
  if (timed) {
    cudaEventRecord(e1, s);
    double units = 0.0;   // half spectra moved
    for (int b = 0; b < nb; b++) units += 1.0 + (pb.terms[b].n > 0 ? 2.0 * pb.terms[b].n : 1.0);
    g_pass_timer.ev.push_back(e0);
    g_pass_timer.ev.push_back(e1);
    g_pass_timer.bytes.push_back(units * (double)p.NH * sizeof(float2));
    g_pass_timer.fields.push_back(nb);
  }
}

template <class T, class C, class Src>
void forward_x(const SrcBatch<Src, C> &sb, int nb, const XGeom &g, const FftPlan &p, cudaStream_t s)
{
  const FftAxis &ax = p.ax[0];
  const long npairs = (g.nlines + 1) / 2;
  const int np = x_pairs(npairs, nb);
  const dim3 grid((unsigned)((npairs + np - 1) / np), (unsigned)nb);
  with_range(ax.R1, [&](auto lo, auto hi) {
    constexpr int LO = decltype(lo)::value, HI = decltype(hi)::value;
    k_rfft_lines<T, C, Src, LO, HI><<<grid, x_threads(ax, np), x_smem<C>(ax, np), s>>>(sb, g, line_of<C>(ax), np, x_pitch(ax));
  });
}

template <class C>
void inverse_x(const OutBatch<C> &ob, int nb, const FftPlan &p, bool accumulate, cudaStream_t s)
{
  const XGeom g = xgeom(p);
  const FftAxis &ax = p.ax[0];
  const long npairs = (g.nlines + 1) / 2;
  const int np = x_pairs(npairs, nb);
  const dim3 grid((unsigned)((npairs + np - 1) / np), (unsigned)nb);
  with_range(ax.R1, [&](auto lo, auto hi) {
    constexpr int LO = decltype(lo)::value, HI = decltype(hi)::value;
    k_irfft_lines<C, LO, HI><<<grid, x_threads(ax, np), x_smem<C>(ax, np), s>>>(ob, g, line_of<C>(ax), np, x_pitch(ax),
                                                                        accumulate ? 1 : 0);
  });
}

// one y (d = 1) or z (d = 2) pass over the half-spectrum box
template <class C>
void strided_pass(const C *in, C *out, const Terms<C> &terms, const FftPlan &p, int d, bool inverse, cudaStream_t s)
{
  PassBatch<C> pb{};
  pb.in[0] = in;
  pb.out[0] = out;
  pb.terms[0] = terms;
  strided_pass_batch<C>(pb, 1, p, d, inverse, s);
}

template <class T, class C, class Src>
void rfft_forward_impl(const Src &src, bool mapped, C *spec, const FftPlan &p, cudaStream_t s)
{
  XGeom g = xgeom(p);
  if (!mapped)   // a real box [F2][F1][F0]
    for (int d = 0; d < 3; d++) {
      g.off[d] = 0;
      g.ext[d] = p.F[d];
      g.last[d] = p.F[d] - 1;
      g.flat0 = 0;
    }
  SrcBatch<Src, C> sb{};
  sb.src[0] = src;
  sb.spec[0] = spec;
  forward_x<T, C, Src>(sb, 1, g, p, s);
  const Terms<C> none{};
  for (int d = 1; d <= 2; d++)
    if (p.F[d] > 1) strided_pass<C>(spec, spec, none, p, d, false, s);
}

// inverse of the products in `terms`, formed by the first inverse pass into `spec` (the work box)
template <class C>
void rfft_inverse_impl(const Terms<C> &terms, C *spec, const FftPlan &p, double *out, float *out32,
                       bool accumulate, const FftProfile &prof, cudaStream_t s)
{
  const Terms<C> none{};
  // A sum of several FP32 products is formed by a pass of its own (five terms at 128^3: 20 + 9 us; 70 us inside the
  // z pass, whose threads wait for each term in turn).  FP64 sums stay in the z pass, bound by their arithmetic there.
  bool pending = !(std::is_same<C, float2>::value && terms.n > 1) && p.F[2] * p.F[1] > 1;   // products not formed yet
  if (!pending) launch_spec_terms<C>(terms, spec, p.NS, s);
  for (int d = 2; d >= 1; d--) {
    if (p.F[d] == 1) continue;
    strided_pass<C>(spec, spec, pending ? terms : none, p, d, true, s);
    pending = false;
  }
  OutBatch<C> ob{};
  ob.spec[0] = spec;
  ob.out[0] = out;
  ob.out32[0] = out32;
  ob.prof[0] = prof;
  inverse_x<C>(ob, 1, p, accumulate, s);
}

// nb forward transforms of mapped channels in one launch per pass
template <class T, class C>
void rfft_forward_mapped_batch_impl(const MapSrc *m, int nb, C *const *spec, const FftPlan &p, cudaStream_t s)
{
  SrcBatch<MappedSrc<T>, C> sb{};
  PassBatch<C> pb{};
  for (int b = 0; b < nb; b++) {
    sb.src[b] = MappedSrc<T>(m[b]);
    sb.spec[b] = spec[b];
    pb.in[b] = spec[b];
    pb.out[b] = spec[b];
  }
  forward_x<T, C, MappedSrc<T>>(sb, nb, xgeom(p), p, s);
  for (int d = 1; d <= 2; d++)
    if (p.F[d] > 1) strided_pass_batch<C>(pb, nb, p, d, false, s);
}

// nb inverse transforms, output b the inverse of a * k[b] (formed by the first inverse pass in work[b])
template <class C>
void rfft_inverse_batch_impl(const C *a, const C *const *k, int nb, C *const *work, const FftPlan &p,
                             double *const *out, float *const *out32, bool accumulate, const FftProfile *prof,
                             const FftCopies *copies, cudaStream_t s)
{
  PassBatch<C> pb{}, plain{};
  OutBatch<C> ob{};
  for (int b = 0; b < nb; b++) {
    pb.in[b] = plain.in[b] = work[b];
    pb.out[b] = plain.out[b] = work[b];
    pb.terms[b].a[0] = a;
    pb.terms[b].k[0] = k[b];
    pb.terms[b].n = 1;
    ob.spec[b] = work[b];
    ob.out[b] = out ? out[b] : nullptr;
    ob.out32[b] = out32 ? out32[b] : nullptr;
    if (prof) ob.prof[b] = prof[b];
    if (copies) ob.copies[b] = copies[b];
  }
  bool pending = true;
  for (int d = 2; d >= 1; d--) {
    if (p.F[d] == 1) continue;
    strided_pass_batch<C>(pending ? pb : plain, nb, p, d, true, s);
    pending = false;
  }
  if (pending)
    for (int b = 0; b < nb; b++) launch_spec_terms<C>(pb.terms[b], work[b], p.NS, s);
  inverse_x<C>(ob, nb, p, accumulate, s);
}

}  // namespace

bool fft_make_plan(FftPlan &p, const int P[3], const int nx[3], const int h[3], const int periodic[3],
                   const int share[3], int ndim, cudaStream_t s)
{
  p.NR = 1;
  for (int d = 0; d < 3; d++) {
    FftAxis &a = p.ax[d];
    p.shared[d] = 0;
    p.P[d] = d < ndim ? P[d] : 1;
    p.nx[d] = d < ndim ? nx[d] : 1;
    p.h[d] = d < ndim ? h[d] : 0;
    if (d >= ndim) {
      p.F[d] = 1;
      p.off[d] = 0;
      p.ext[d] = 1;
      a.n = a.R1 = a.R2 = 1;
      continue;
    }
    if (periodic[d] && radices_of(nx[d], a.R1, a.R2)) {   // the period itself: no padding
      p.F[d] = nx[d];
      p.off[d] = h[d];
      p.ext[d] = nx[d];
    } else {
      int F = P[d];
      while (F <= kFftMaxN && !radices_of(F, a.R1, a.R2)) F++;
      if (F > kFftMaxN) return false;
      p.F[d] = F;
      p.off[d] = 0;
      p.ext[d] = P[d];
      if (share[d]) {   // node i at box position i, the shared boundary value from nx on
        F = p.nx[d] + p.h[d];
        while (!radices_of(F, a.R1, a.R2)) F++;
        p.F[d] = p.ext[d] = F;
        p.off[d] = p.h[d];
        p.shared[d] = 1;
      }
    }
    a.n = p.F[d];
    std::vector<double2> tw(a.n);
    std::vector<float2> tw32(a.n);
    for (int k = 0; k < a.n; k++) {
      // exp(-2 pi i k / n) from the host library in extended precision, rounded once
      const long double ang = -2.0L * 3.141592653589793238462643383279502884L * (long double)k / (long double)a.n;
      tw[k] = make_double2((double)std::cos(ang), (double)std::sin(ang));
      tw32[k] = make_float2((float)std::cos(ang), (float)std::sin(ang));
    }
    if (cudaMalloc(&a.d_tw, sizeof(double2) * a.n) != cudaSuccess) return false;
    if (cudaMalloc(&a.d_tw32, sizeof(float2) * a.n) != cudaSuccess) return false;
    cudaMemcpyAsync(a.d_tw, tw.data(), sizeof(double2) * a.n, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(a.d_tw32, tw32.data(), sizeof(float2) * a.n, cudaMemcpyHostToDevice, s);
    cudaStreamSynchronize(s);   // the host tables go out of scope
    p.NR *= p.F[d];
  }
  p.Fh = p.F[0] / 2 + 1;
  p.Fp = (p.Fh + 15) / 16 * 16;   // lines start on 128-byte boundaries
  p.NH = (long)p.Fh * p.F[1] * p.F[2];
  p.NS = (long)p.Fp * p.F[1] * p.F[2];
  set_smem_limits<double, double2>(p);
  set_smem_limits<float, float2>(p);
  return true;
}

void fft_free_plan(FftPlan &p)
{
  for (auto &a : p.ax) {
    if (a.d_tw) cudaFree(a.d_tw);
    if (a.d_tw32) cudaFree(a.d_tw32);
    a.d_tw = nullptr;
    a.d_tw32 = nullptr;
  }
}

void rfft_forward_mapped(const MapSrc &m, double2 *spec, const FftPlan &p, cudaStream_t s)
{
  rfft_forward_impl<double, double2>(MappedSrc<double>(m), true, spec, p, s);
}

void rfft_forward_mapped(const MapSrc &m, float2 *spec, const FftPlan &p, cudaStream_t s)
{
  rfft_forward_impl<float, float2>(MappedSrc<float>(m), true, spec, p, s);
}

void rfft_forward_box(const double *box, double2 *spec, const FftPlan &p, cudaStream_t s)
{
  rfft_forward_impl<double, double2>(BoxSrc<double>{box, p.F[0], (long)p.F[0] * p.F[1]}, false, spec, p, s);
}

template <class C>
Terms<C> make_terms(const C *const *a, const C *const *k, int n)
{
  Terms<C> t{};
  t.n = n;
  for (int j = 0; j < n; j++) {
    t.a[j] = a[j];
    t.k[j] = k[j];
  }
  return t;
}

void rfft_inverse_products(const double2 *const *a, const double2 *const *k, int nterms, double2 *work,
                           const FftPlan &p, double *out, bool accumulate, cudaStream_t s,
                           const FftProfile &prof)
{
  rfft_inverse_impl<double2>(make_terms(a, k, nterms), work, p, out, nullptr, accumulate, prof, s);
}

void rfft_inverse_products(const float2 *const *a, const float2 *const *k, int nterms, float2 *work,
                           const FftPlan &p, double *out, bool accumulate, cudaStream_t s,
                           const FftProfile &prof)
{
  rfft_inverse_impl<float2>(make_terms(a, k, nterms), work, p, out, nullptr, accumulate, prof, s);
}

void rfft_inverse_products(const float2 *const *a, const float2 *const *k, int nterms, float2 *work,
                           const FftPlan &p, float *out, bool accumulate, cudaStream_t s)
{
  rfft_inverse_impl<float2>(make_terms(a, k, nterms), work, p, nullptr, out, accumulate, FftProfile{}, s);
}

int fft_max_terms() { return kMaxTerms; }
int fft_max_batch() { return kMaxBatch; }

void rfft_forward_mapped_batch(const MapSrc *m, int nb, float2 *const *spec, const FftPlan &p, cudaStream_t s)
{
  for (int b0 = 0; b0 < nb; b0 += kMaxBatch)
    rfft_forward_mapped_batch_impl<float, float2>(m + b0, std::min(kMaxBatch, nb - b0), spec + b0, p, s);
}

void rfft_forward_mapped_batch(const MapSrc *m, int nb, double2 *const *spec, const FftPlan &p, cudaStream_t s)
{
  for (int b0 = 0; b0 < nb; b0 += kMaxBatch)
    rfft_forward_mapped_batch_impl<double, double2>(m + b0, std::min(kMaxBatch, nb - b0), spec + b0, p, s);
}

void rfft_inverse_batch(const float2 *a, const float2 *const *k, int nb, float2 *const *work, const FftPlan &p,
                        double *const *out, bool accumulate, cudaStream_t s, const FftProfile *prof,
                        const FftCopies *copies)
{
  for (int b0 = 0; b0 < nb; b0 += kMaxBatch)
    rfft_inverse_batch_impl<float2>(a, k + b0, std::min(kMaxBatch, nb - b0), work + b0, p, out + b0, nullptr,
                                    accumulate, prof ? prof + b0 : nullptr, copies ? copies + b0 : nullptr, s);
}

void rfft_inverse_batch(const float2 *a, const float2 *const *k, int nb, float2 *const *work, const FftPlan &p,
                        float *const *out, bool accumulate, cudaStream_t s, const FftCopies *copies)
{
  for (int b0 = 0; b0 < nb; b0 += kMaxBatch)
    rfft_inverse_batch_impl<float2>(a, k + b0, std::min(kMaxBatch, nb - b0), work + b0, p, nullptr, out + b0,
                                    accumulate, nullptr, copies ? copies + b0 : nullptr, s);
}

void rfft_inverse_batch(const double2 *a, const double2 *const *k, int nb, double2 *const *work, const FftPlan &p,
                        double *const *out, bool accumulate, cudaStream_t s, const FftProfile *prof,
                        const FftCopies *copies)
{
  for (int b0 = 0; b0 < nb; b0 += kMaxBatch)
    rfft_inverse_batch_impl<double2>(a, k + b0, std::min(kMaxBatch, nb - b0), work + b0, p, out + b0, nullptr,
                                     accumulate, prof ? prof + b0 : nullptr, copies ? copies + b0 : nullptr, s);
}

void fft_pass(double2 *spec, const FftPlan &p, int d, bool inverse, cudaStream_t s)
{
  const Terms<double2> none{};
  strided_pass<double2>(spec, spec, none, p, d, inverse, s);
}

void fft_pass(float2 *spec, const FftPlan &p, int d, bool inverse, cudaStream_t s)
{
  const Terms<float2> none{};
  strided_pass<float2>(spec, spec, none, p, d, inverse, s);
}

void launch_fft_kernel_box(const short *off3, const double *coef, int L, int ncoef, int q, int dir, double *box,
                           const FftPlan &p, cudaStream_t s)
{
  cudaMemsetAsync(box, 0, sizeof(double) * p.NR, s);
  if (L > 0) k_fft_kernel_box<<<(L + 255) / 256, 256, 0, s>>>(off3, coef, L, ncoef, q, dir, 0.25 / (double)p.NR, box, p.F[0], p.F[1], p.F[2]);
}

void launch_to_float2(const double2 *in, float2 *out, long n, cudaStream_t s)
{
  k_to_float2<<<grid_for(n), 256, 0, s>>>(in, out, n);
}

void pass_timer_enable(bool on)
{
  g_pass_timer.on = on;
}

void pass_timer_collect(long *launches, double *ms_total, double *bytes_total, long *fields_total)
{
  double ms = 0.0, bytes = 0.0;
  long fields = 0;
  const size_t nl = g_pass_timer.bytes.size();
  for (size_t i = 0; i < nl; i++) {
    float t = 0.f;
    cudaEventSynchronize(g_pass_timer.ev[2 * i + 1]);
    cudaEventElapsedTime(&t, g_pass_timer.ev[2 * i], g_pass_timer.ev[2 * i + 1]);
    ms += t;
    bytes += g_pass_timer.bytes[i];
    fields += g_pass_timer.fields[i];
  }
  for (cudaEvent_t e : g_pass_timer.ev) cudaEventDestroy(e);
  g_pass_timer.ev.clear();
  g_pass_timer.bytes.clear();
  g_pass_timer.fields.clear();
  if (launches) *launches = (long)nl;
  if (ms_total) *ms_total = ms;
  if (bytes_total) *bytes_total = bytes;
  if (fields_total) *fields_total = fields;
}

}  // namespace tgpu
