// GMRES of a 1-D problem in one launch (included by kernels.cu).
//
// At 300 to 4000 nodes one GMRES iteration was about 25 launches of 2 to 20 us and a wait for the host, 190 to 210 us
// in all: every kernel was far below a wave, the FP64 stencil sums a serial chain of a few hundred FMAs on a handful
// of SMs.  Here one cooperative launch runs a whole GMRES cycle (the operator, diagonal preconditioner, classical
// Gram-Schmidt twice, rotations and the update x = V y), each CTA owning a few nodes and the phases separated by a
// barrier over the grid:
//   1  V_k = w / |w|; sums of the density-shaped vector over the CTA's window, local step, channels out   -> barrier
//   2  sums of the channels, row combination, preconditioner; V_j . w of the CTA's nodes                  -> barrier
//   3  h1 = V^T w; w -= V h1; V_j . w again                                                               -> barrier
//   4  h2; w -= V h2; w and its part of |w|^2 out                                                         -> barrier
// One more CTA owns no nodes and turns the new column by the rotations during the next phase 1, so that the chain of
// dependent FP64 operations costs nothing; the stopping test is read one barrier later.
//
// Work split: tiles of 8 nodes x 32 groups of taps (a warp holds 8 nodes x 4 groups), so that the FP64 pipe of as many
// SMs as there are tiles works on the sums; NT tiles at a time share the taps' loads, the shuffles (two values to a
// shuffle, each lane keeping one) and the barriers of the block.  Sums over groups, nodes and CTAs are taken in a fixed
// order.  Everything about the CTA's nodes that outlives an iteration stays in shared memory: window positions, the
// Hessian's coefficients, densities.
// Bound: latency (a warp's FP64 operation holds its scheduler's pipe for 64 cycles, so short serial steps count) and
// four barriers; 2001 nodes of hard spheres in FP64: 27 us per iteration against 210, 1487 nodes of the slit pore with
// FP32 products 25 against 185, adjoint of 801 nodes 25 (with a barrier after phase 4's norm, a tile at a time and global
// memory for the nodes' tables 43, 38 and 36).  The channels of the local step formed by a warp each: 2 % less, not kept.
//
// TR: the transposed Schur complement (adjoint solves), from the stencils with negated offsets.

constexpr int kLineThreads = 256, kLineTile = 8, kLineGroups = 32, kLineWarps = kLineThreads / 32;

template <class T>
struct LineSten {
  const int *off;   // tap offsets in nodes
  const T *coef;    // [L][columns]
  int L;
};

template <class T>
struct LineArgs {
  LineSten<T> th[kMaxC], de[kMaxC], ua[kMaxC * kMaxC];   // sums of densities (TR: of the adjoint, both phases)
  LineSten<T> tth[kMaxC], tde[kMaxC];                    // sums of channels
  const double *x, *vext, *hcoef, *rhs;
  const signed char *zero;
  double *V, *part, *R, *y, *xout;
  T *chan;
  signed char *kind;
  unsigned *bar;        // arrivals, error, stop (set by the block without nodes, nothing clears it within the launch)
  LineResult *res;
  long ldv;             // ncomp * N
  int per, kdim, m;     // nodes per CTA, vectors that R holds, steps of this cycle
  int spin;             // polls before a barrier gives up
  double tol;
};

// Barrier over the grid; false when it gave up (then every block returns)
__device__ __forceinline__ bool line_barrier(unsigned *bar, unsigned &gen, int limit)
{
  __shared__ int s_ok;
  __syncthreads();
  gen++;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" :: "l"(bar) : "memory");
    const unsigned target = gen * gridDim.x;
    int ok = 1, spins = 0;
    unsigned seen;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
      if (++spins > limit) {
        atomicExch(bar + 1, 1u);
        ok = 0;
        break;
      }
    } while (seen < target);
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// two values to a shuffle: a lane keeps v0 (bit clear) or v1 (bit set), summed with its partner's
template <class A>
__device__ __forceinline__ A line_pack(A v0, A v1, int bit)
{
  const bool up = (threadIdx.x & bit) != 0;
  return (up ? v1 : v0) + __shfl_xor_sync(0xffffffffu, up ? v0 : v1, bit);
}

// sums over the warp's 4 groups of M values, left in red[value][warp][node]
template <int M, class A>
__device__ __forceinline__ void line_warp_sums(const A (&v)[M], A *red)
{
  constexpr int P = (M + 1) / 2, Q = (P + 1) / 2;
  const int lane = threadIdx.x & 31, nl = lane & 7, warp = threadIdx.x >> 5;
  const int b8 = (lane >> 3) & 1, b16 = lane >> 4;
  A p[P];
#pragma unroll
  for (int i = 0; i < P; i++) {
    if (2 * i + 1 < M) p[i] = line_pack(v[2 * i], v[2 * i + 1], 8);
    else p[i] = v[2 * i] + __shfl_xor_sync(0xffffffffu, v[2 * i], 8);
  }
#pragma unroll
  for (int q = 0; q < Q; q++) {
    A s;
    if (2 * q + 1 < P) s = line_pack(p[2 * q], p[2 * q + 1], 16);
    else s = p[2 * q] + __shfl_xor_sync(0xffffffffu, p[2 * q], 16);
    const int pi = 2 * q + b16, id = 2 * pi + b8;
    if (pi < P && id < M) red[id * (kLineWarps * kLineTile) + warp * kLineTile + nl] = s;
  }
}

// the warps' parts of value id of a node
template <class A>
__device__ __forceinline__ A line_final(const A *red, int id, int nl)
{
  const A *r = red + id * (kLineWarps * kLineTile) + nl;
  A s = r[0];
#pragma unroll
  for (int w = 1; w < kLineWarps; w++) s += r[w * kLineTile];
  return s;
}

// a lane's part of row j: the blocks' values lane, lane + 32, ...
__device__ __forceinline__ double line_part(const double *part, int j, int nblk, int lane)
{
  double v[5], s = 0.0;
  const double *p = part + (long)j * nblk;
#pragma unroll
  for (int u = 0; u < 5; u++) v[u] = lane + 32 * u < nblk ? __ldcg(p + lane + 32 * u) : 0.0;
#pragma unroll
  for (int u = 0; u < 5; u++)
    if (32 * u < nblk) s += v[u];
  for (int b = lane + 160; b < nblk; b += 32) s += __ldcg(p + b);
  return s;
}

__device__ __forceinline__ double line_butterfly(double s, int from)
{
  for (int o = from; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// out[j] = sum over the blocks of part[j * nblk + b], j < cnt; a warp takes up to four rows at a time
__device__ __forceinline__ void line_reduce(const double *part, int cnt, int nblk, double *out)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j = warp; j < cnt; j += 4 * kLineWarps) {
    const int j1 = j + kLineWarps, j2 = j + 2 * kLineWarps, j3 = j + 3 * kLineWarps;
    double s = line_part(part, j, nblk, lane);
    if (j1 >= cnt) {
      s = line_butterfly(s, 16);
      if (lane == 0) out[j] = s;
    } else if (j2 >= cnt) {
      s = line_butterfly(line_pack(s, line_part(part, j1, nblk, lane), 16), 8);
      if (lane == 0) out[j] = s;
      if (lane == 16) out[j1] = s;
    } else {
      const double s1 = line_part(part, j1, nblk, lane), s2 = line_part(part, j2, nblk, lane);
      const double s3 = j3 < cnt ? line_part(part, j3, nblk, lane) : 0.0;
      s = line_butterfly(line_pack(line_pack(s, s1, 16), line_pack(s2, s3, 16), 8), 4);
      if (lane == 0) out[j] = s;
      if (lane == 16) out[j1] = s;
      if (lane == 8) out[j2] = s;
      if (lane == 24 && j3 < cnt) out[j3] = s;
    }
  }
  __syncthreads();
}

// sqrt of the sum over the blocks of part[b], the same in every thread
__device__ __forceinline__ double line_norm(const double *part, int nblk)
{
  __shared__ double s_norm;
  if (threadIdx.x < 32) {
    const double s = line_butterfly(line_part(part, 0, nblk, threadIdx.x), 16);
    if (threadIdx.x == 0) s_norm = sqrt(s);
  }
  __syncthreads();
  return s_norm;
}

// acc[o][u] += sum of the group's taps of one stencil, NI inputs (windows ld apart), NO outputs, NT tiles
template <int NI, int NO, int NT, class T>
__device__ __forceinline__ void line_taps(const LineSten<T> &st, const T *win, int ld, int grp, T (*acc)[NT])
{
#pragma unroll 4
  for (int k = grp; k < st.L; k += kLineGroups) {
    const T *w = win + __ldg(st.off + k);
#pragma unroll
    for (int o = 0; o < NO; o++)
#pragma unroll
      for (int c = 0; c < NI; c++) {
        const T cf = __ldg(st.coef + (k * NO + o) * NI + c);
#pragma unroll
        for (int u = 0; u < NT; u++) acc[o][u] = fma(cf, w[c * ld + u * kLineTile], acc[o][u]);
      }
  }
}

// the same for one input into sums over components; FP32 sums are added to them in FP64
template <int NO, int NT, class T, class A>
__device__ __forceinline__ void line_add(const LineSten<T> &st, const T *win, int ld, int grp, A (*acc)[NT])
{
  if constexpr (std::is_same<A, T>::value) {
    line_taps<1, NO, NT, T>(st, win, ld, grp, acc);
  } else {
    T d[NO][NT] = {};
    line_taps<1, NO, NT, T>(st, win, ld, grp, d);
#pragma unroll
    for (int o = 0; o < NO; o++)
#pragma unroll
      for (int u = 0; u < NT; u++) acc[o][u] += (A)d[o][u];
  }
}

// shared memory of a CTA; `per` nodes, a window of nw = per + 2 h positions, NT tiles at a time
constexpr int kLineRb = 6, kLineTable = kHessCoef + kLineRb;   // 1-D weighted densities; a node's table: n, coefficients
struct LineSmem {
  size_t win, red, tab, dbl, idx, bytes;   // offsets
};
__host__ __device__ inline LineSmem line_layout(int nc, int ncols, bool tr, int kdim, int per, int nw, int nt, size_t t)
{
  const size_t nch = (size_t)(tr ? 4 * nc : 3 * nc), rows = kLineRb + ncols, ts = ncols > 1 ? sizeof(double) : t;
  LineSmem m;
  m.win = 0;
  m.red = (t * nch * nw + 15) & ~(size_t)15;
  m.tab = m.red + sizeof(double) * rows * nt * kLineWarps * kLineTile;
  m.dbl = (m.tab + t * (size_t)kLineTable * per + ts * rows * nt * kLineTile + 15) & ~(size_t)15;
  // w, -u_MF, V_k, rho, V_k / rho; h1, h2; rotations and right-hand side
  m.idx = m.dbl + sizeof(double) * (5 * (size_t)nc * per + 2 * (kdim + 2) + 3 * (size_t)kdim + 1);
  m.bytes = m.idx + sizeof(int) * (size_t)(nc + 1) * nw + (size_t)nc * per;
  return m;
}

template <class T, bool TR, int NC, int NT>
__global__ void __launch_bounds__(kLineThreads) k_gmres_line(LineArgs<T> a)
{
  constexpr int NRB = kLineRb, CPC = 3, STEP = NT * kLineTile, ROWS = NRB + NC;
  using A = typename std::conditional<NC == 1, T, double>::type;   // sums over components: of FP32 sums in FP64
  extern __shared__ __align__(16) unsigned char smraw[];
  const int nc = NC == 1 ? 1 : c_g.ncomp, per = a.per, h = c_g.h[0], nw = per + 2 * h;
  const long N = c_g.N;
  const int nblk = gridDim.x - 1;                    // blocks that own nodes
  const bool owner = (int)blockIdx.x < nblk;
  const int i0 = blockIdx.x * per, own = owner ? (int)min((long)per, N - i0) : 0;
  const LineSmem lay = line_layout(nc, NC, TR, a.kdim, per, nw, NT, sizeof(T));
  T *win = reinterpret_cast<T *>(smraw);
  double *red = reinterpret_cast<double *>(smraw + lay.red);
  A *redA = reinterpret_cast<A *>(red);
  T *tab = reinterpret_cast<T *>(smraw + lay.tab);           // [kLineTable][per]
  A *sums = reinterpret_cast<A *>(tab + kLineTable * per);   // [ROWS][STEP]
  double *w = reinterpret_cast<double *>(smraw + lay.dbl), *ymf = w + nc * per, *vown = ymf + nc * per;
  double *rho = vown + nc * per, *vr = rho + nc * per;
  double *h1 = vr + nc * per, *h2 = h1 + a.kdim + 2, *cs = h2 + a.kdim + 2, *sn = cs + a.kdim, *gv = sn + a.kdim;
  int *ix2 = reinterpret_cast<int *>(smraw + lay.idx), *ix1 = ix2 + nw;
  signed char *kd = reinterpret_cast<signed char *>(ix1 + nc * nw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nl = lane & 7, grp = warp * 4 + (lane >> 3);
  double *partA = a.part, *partB = a.part + (long)(a.kdim + 2) * nblk;
  double *wbuf = a.V + (long)a.m * a.ldv;   // w for the neighbours (V_m is not needed)
  const bool att = c_g.attraction != 0, one = c_g.single_size != 0;
  unsigned gen = 0;

  // r0 = M^-1 b, beta = |r0|
  double s = 0.0;
  for (int t = tid; t < nc * own; t += kLineThreads) {
    const int ic = t / own, il = t - ic * own, i = i0 + il;
    const long k = (long)ic * N + i;
    const bool zr = zero_row(a.vext, a.zero, ic, i), lr = zr && log_row(a.vext, a.zero, ic, i);
    const double x = a.x[(long)(c_g.first_rho + ic) * N + i];
    const signed char kind = !zr ? 0 : lr ? 1 : 2;
    a.kind[k] = kind;
    kd[ic * per + il] = TR && a.zero[k] ? (signed char)3 : kind;
    rho[ic * per + il] = x;
    const double r = (zr && !lr) ? a.rhs[k] : a.rhs[k] * x;
    w[ic * per + il] = r;
    wbuf[k] = r;
    s = fma(r, r, s);
  }
  s = block_sum(s, red);
  if (owner && tid == 0) partA[blockIdx.x] = s;
  if (owner) {   // the table of the nodes
    for (int t = tid; t < kLineTable * own; t += kLineThreads) {
      const int r = t / own, il = t - r * own;
      const double *rb = a.x + (long)c_g.first_rb * N;
      double v;
      if (r >= NRB) v = a.hcoef[(long)(r - NRB) * N + i0 + il];
      else v = rb[(long)(r < 4 ? 3 - r : r == 4 ? 5 : 4) * N + i0 + il];   // n0 n1 n2 n3 V1 V2
      tab[r * per + il] = (T)v;
    }
  }
  if (!line_barrier(a.bar, gen, a.spin)) return;
  const double r0 = line_norm(partA, nblk);
  if (!(r0 > 0.0)) {   // a zero or non-finite right-hand side: the host decides
    for (int t = tid; t < nc * own; t += kLineThreads) {
      const int ic = t / own;
      a.xout[(long)ic * N + i0 + t - ic * own] = 0.0;
    }
    if (!owner && tid == 0) *a.res = LineResult{0, 0, r0, 0.0};
    return;
  }
  if (owner) {   // window positions: node, -1 reads 0, -2 outside the problem; ix1 with the nodes that read 0
    const signed char *flag = TR ? a.kind : a.zero;
    for (int t = tid; t < nw; t += kLineThreads) {
      const int q = i0 + t;
      const int m = q < c_g.P[0] ? c_g.map[0][q] : kSentBulk;
      const int at = m >= 0 ? m : m == kSentBad ? -2 : -1;
      ix2[t] = at;
      for (int ic = 0; ic < nc; ic++) {
        const int i = at & ~kReflBit;
        ix1[ic * nw + t] = at < 0 ? at : __ldcg(flag + (long)ic * N + i) ? -1 : i;
      }
    }
  }
  if (tid == 0) gv[0] = r0;
  __syncthreads();

  // the pending column (in h1, h2, norm hn) of the block without nodes: rotations; true when the residual meets tol
  double hn = r0, rel = 1.0;
  int k = 0, cols = 0, status = 0;
  auto rotate = [&](int c) {   // thread 0 of the last block
    double *col = a.R + (long)c * (a.kdim + 1);
    double av = h1[0] + h2[0];
    for (int j = 0; j < c; j++) {
      const double b = h1[j + 1] + h2[j + 1];
      col[j] = cs[j] * av + sn[j] * b;
      av = -sn[j] * av + cs[j] * b;
    }
    const double den = sqrt(av * av + hn * hn);
    cs[c] = den == 0.0 ? 1.0 : av / den;
    sn[c] = den == 0.0 ? 0.0 : hn / den;
    col[c] = den;
    gv[c + 1] = -sn[c] * gv[c];
    gv[c] = cs[c] * gv[c];
    rel = fabs(gv[c + 1]) / r0;
  };
  // per node and component: the sum over j < cnt of hv[j] V_j, through put(ic, il, sum)
  auto combine = [&](const double *hv, int cnt, auto put) {
    for (int t0 = 0; t0 < own; t0 += STEP) {
      double d[NC * NT];
#pragma unroll
      for (int e = 0; e < NC * NT; e++) {
        const int ic = e / NT, il = t0 + (e % NT) * kLineTile + nl;
        d[e] = 0.0;
        if (ic < nc && il < own)
          for (int j = grp; j < cnt; j += kLineGroups)
            d[e] = fma(hv[j], a.V[(long)j * a.ldv + (long)ic * N + i0 + il], d[e]);
      }
      line_warp_sums(d, red);
      __syncthreads();
      if (tid < nc * STEP) {
        const int ic = tid / STEP, il = t0 + tid % STEP;
        if (il < own) put(ic, il, line_final<double>(red, tid / kLineTile, nl));
      }
      __syncthreads();
    }
  };
  auto dots = [&](double *part) {   // V_j . w of the block's nodes
    for (int j = tid; j <= k; j += kLineThreads) {
      double d = 0.0;
      for (int ic = 0; ic < nc; ic++) {
        const double *v = a.V + (long)j * a.ldv + (long)ic * N + i0;
#pragma unroll 8
        for (int i = 0; i < own; i++) d = fma(v[i], w[ic * per + i], d);
      }
      part[(long)j * nblk + blockIdx.x] = d;
    }
  };
  for (; k < a.m; k++) {
    // ---- phase 1
    if (owner) {
      const double rhn = 1.0 / hn;
      const bool quick = sizeof(T) == sizeof(float) && hn > 1e-300 && hn < 1e300;   // (rhn neither infinite nor subnormal)
      for (int t = kLineThreads - 1 - tid; t < nc * own; t += kLineThreads) {
        const int ic = t / own, il = t - ic * own;
        const double v = w[ic * per + il] / hn;
        vown[ic * per + il] = v;
        a.V[(long)k * a.ldv + (long)ic * N + i0 + il] = v;
      }
      for (int ic = 0; ic < nc; ic++)
#pragma unroll 4
        for (int t = tid; t < nw; t += kLineThreads) {
          const int m = ix1[ic * nw + t];
          T v = m == -1 ? (T)0 : (T)__longlong_as_double(0x7ff8000000000000ULL);
          if (m >= 0) {
            const double u = __ldcg(wbuf + (long)ic * N + m);
            v = (T)(quick ? u * rhn : u / hn);
          }
          win[ic * nw + t] = v;
        }
      __syncthreads();
      for (int t0 = 0; t0 < own; t0 += STEP) {
        const int at = t0 + nl + h;
        if constexpr (NC == 1 && !TR) {
          if (one) {   // rows n3, n2, V2 and the mean field
            A acc[4][NT] = {};
            line_taps<1, 1, NT, T>(a.th[0], win + at, nw, grp, acc);
            line_taps<1, 2, NT, T>(a.de[0], win + at, nw, grp, acc + 1);
            if (att) {
              line_taps<1, 1, NT, T>(a.ua[0], win + at, nw, grp, acc + 3);
              line_warp_sums(reinterpret_cast<const A (&)[4 * NT]>(acc), redA);
            } else {
              line_warp_sums(reinterpret_cast<const A (&)[3 * NT]>(acc), redA);
            }
            __syncthreads();
            if (tid < (att ? 4 : 3) * STEP) {
              const int r = tid / STEP;
              const int row = r == 0 ? 0 : r == 1 ? 1 : r == 2 ? 4 : NRB;
              sums[row * STEP + tid % STEP] = line_final<A>(redA, tid / kLineTile, nl);
            }
          }
        }
        if (NC != 1 || TR || !one) {
          A acc[ROWS][NT] = {};
          if constexpr (TR) {
            // per component (scalar, vector) of the delta shell and the ball: combined at once into the rows of g
            // (n ordering: acc 0..5 = g0 g1 g2 g3 gV1 gV2)
#pragma unroll
            for (int ic = 0; ic < NC; ic++)
              if (ic < nc) {
                T d[2][NT] = {};
                line_taps<1, 2, NT, T>(a.de[ic], win + ic * nw + at, nw, grp, d);
                line_taps<1, 1, NT, T>(a.th[ic], win + ic * nw + at, nw, grp, acc + 3);
#pragma unroll
                for (int u = 0; u < NT; u++) {
                  acc[2][u] += d[0][u];
                  acc[1][u] += (T)c_g.inv_4pir[ic] * d[0][u];
                  acc[0][u] += (T)c_g.inv_4pirsq[ic] * d[0][u];
                  acc[5][u] -= d[1][u];
                  acc[4][u] -= (T)c_g.inv_4pir[ic] * d[1][u];
                }
              }
          } else {
#pragma unroll
            for (int jc = 0; jc < NC; jc++)
              if (jc < nc) {
                const T *wj = win + jc * nw + at;
                line_add<1, NT>(a.th[jc], wj, nw, grp, acc);             // n3
                if (one) {
                  T d[2][NT] = {};
                  line_taps<1, 2, NT, T>(a.de[jc], wj, nw, grp, d);      // n2, V2
#pragma unroll
                  for (int u = 0; u < NT; u++) {
                    acc[1][u] += (A)d[0][u];
                    acc[4][u] += (A)d[1][u];
                  }
                } else {
                  line_add<5, NT>(a.de[jc], wj, nw, grp, acc + 1);       // n2, n1, n0, V2, V1
                }
                if (att)
#pragma unroll
                  for (int ic = 0; ic < NC; ic++)
                    if (ic < nc) line_add<1, NT>(a.ua[ic + nc * jc], wj, nw, grp, acc + NRB + ic);
              }
          }
          line_warp_sums(reinterpret_cast<const A (&)[ROWS * NT]>(acc), redA);
          __syncthreads();
          if (tid < ROWS * STEP) sums[tid] = line_final<A>(redA, tid / kLineTile, nl);
        }
        __syncthreads();
        // local step; another warp forms what depends on the vector alone
        const int tl = lane, il = t0 + tl;
        if (tl < STEP && il < own && warp < 2) {
          const long i = i0 + il;
          if (warp == 1) {
            for (int ic = 0; ic < nc; ic++) {
              vr[ic * per + il] = vown[ic * per + il] / rho[ic * per + il];
              if (!TR && att) ymf[ic * per + il] = -(double)sums[(NRB + ic) * STEP + tl];
              // mean-field row: t = w_EL (full rows), y = -t
              if (TR && att) a.chan[(long)(nc * CPC + ic) * N + i] = (T)(-win[ic * nw + il + h]);
            }
          } else {
            const auto table = [&](T *n, HessCoefT<T> &c) {
              const T *tb = tab + il;
#pragma unroll
              for (int r = 0; r < NRB; r++) n[r] = tb[r * per];
              tb += NRB * per;
              c = HessCoefT<T>{tb[0], tb[per], tb[2 * per], tb[3 * per], tb[4 * per], tb[5 * per], tb[6 * per],
                               tb[7 * per], tb[8 * per], tb[9 * per], tb[10 * per], tb[11 * per]};
            };
            T n[NRB], y[NRB], z[NRB];
            HessCoefT<T> c;
            if constexpr (TR) {
              for (int r = 0; r < NRB; r++) y[r] = (T)sums[r * STEP + tl];
            } else {
              T ysv[NRB];
              for (int r = 0; r < NRB; r++) {
                int src;
                double cd;
                if (dep_rb(r, &src, &cd)) ysv[r] = -to_arith<T>(cd) * (T)sums[src * STEP + tl];   // -u_dep - B u_ind
                else ysv[r] = -(T)sums[r * STEP + tl];
              }
              y[0] = ysv[3]; y[1] = ysv[2]; y[2] = ysv[1]; y[3] = ysv[0]; y[4] = ysv[5]; y[5] = ysv[4];
            }
            table(n, c);
            fmt_hess_apply_coef(c, n, y, z, c_g.ndim, TR);
            for (int ic = 0; ic < nc; ic++) {
              T *ch = a.chan + (long)ic * CPC * N + i;
              if constexpr (TR) {
                // t = J^T [0; v] on the block-1 rows, y = A11^-T t, and y's channels
                double v[NRB] = {-z[3], -z[2], -z[1], -z[0], -z[5], -z[4]};   // -t, rows n3 n2 n1 n0 V2 V1
                if (one) {
                  v[1] -= c_g.inv_4pir[0] * z[1] + c_g.inv_4pirsq[0] * z[0];
                  v[4] -= c_g.inv_4pir[0] * z[4];
                }
                const double wn1 = one ? 0.0 : v[2], wn0 = one ? 0.0 : v[3], wv1 = one ? 0.0 : v[5];
                ch[0] = (T)(v[1] + c_g.inv_4pir[ic] * wn1 + c_g.inv_4pirsq[ic] * wn0);
                ch[N] = (T)(v[4] + c_g.inv_4pir[ic] * wv1);
                ch[2 * N] = (T)v[0];
              } else {
                const T f = to_arith<T>(c_g.fac[ic]), r1 = to_arith<T>(c_g.inv_4pir[ic]), r2 = to_arith<T>(c_g.inv_4pirsq[ic]);
                ch[0] = f * (z[0] * r2 + z[1] * r1 + z[2]);
                ch[N] = f * (z[4] * r1 + z[5]);
                ch[2 * N] = f * z[3];
              }
            }
          }
        }
        __syncthreads();
      }
    } else if (k > 0 && tid == 0) {
      rotate(k - 1);
      if (rel < a.tol) __stcg(a.bar + 2, 1u);   // converged after k steps
    }
    if (!line_barrier(a.bar, gen, a.spin)) return;
    if (k > 0 && __ldcg(a.bar + 2) != 0u) {   // (a word of its own: late readers must not meet the result's)
      cols = k;
      break;
    }
    // ---- phase 2
    if (owner) {
      for (int t = tid; t < nw; t += kLineThreads) {
        const int m = ix2[t], i = m & ~kReflBit;
        const T out = m == -1 ? (T)0 : (T)__longlong_as_double(0x7ff8000000000000ULL);
        const bool flip = !TR && m >= 0 && (m & kReflBit);
        for (int ic = 0; ic < nc; ic++) {
          T v[CPC];
#pragma unroll
          for (int r = 0; r < CPC; r++) v[r] = m >= 0 ? __ldcg(a.chan + (long)(ic * CPC + r) * N + i) : out;
          if (flip) v[1] = -v[1];
#pragma unroll
          for (int r = 0; r < CPC; r++) win[(ic * CPC + r) * nw + t] = v[r];
          if (TR && att)
            win[(nc * CPC + ic) * nw + t] = m >= 0 ? __ldcg(a.chan + (long)(nc * CPC + ic) * N + i) : out;
        }
      }
      __syncthreads();
      for (int t0 = 0; t0 < own; t0 += STEP) {
        const int at = t0 + nl + h;
        double v[NC * NT];
#pragma unroll
        for (int ic = 0; ic < NC; ic++) {
          T d[1][NT] = {}, b[1][NT] = {};
          if (ic < nc) {
            const T *wi = win + ic * CPC * nw + at;
            line_taps<2, 1, NT, T>(TR ? a.de[ic] : a.tde[ic], wi, nw, grp, d);
            line_taps<1, 1, NT, T>(TR ? a.th[ic] : a.tth[ic], wi + 2 * nw, nw, grp, b);
            if (TR && att)
              for (int jc = 0; jc < nc; jc++)
                line_taps<1, 1, NT, T>(a.ua[jc + nc * ic], win + (nc * CPC + jc) * nw + at, nw, grp, b);
          }
#pragma unroll
          for (int u = 0; u < NT; u++) v[ic * NT + u] = (double)d[0][u] + (double)b[0][u];
        }
        line_warp_sums(v, red);
        __syncthreads();
        if (tid < nc * STEP) {
          const int ic = tid / STEP, il = t0 + tid % STEP, e = ic * per + il;
          if (il < own) {
            const double tr = line_final<double>(red, tid / kLineTile, nl);
            const int kind = kd[e];   // 3: a node whose density is held at zero
            double r;   // M^-1 S v
            if (TR) r = vown[e] - (kind == 3 ? 0.0 : kind == 2 ? tr : tr * rho[e]);
            else r = kind == 0 ? (vr[e] - (att ? tr + ymf[e] : tr)) * rho[e] : vown[e];
            w[e] = r;
          }
        }
        __syncthreads();
      }
      dots(partA);
    }
    if (!line_barrier(a.bar, gen, a.spin)) return;
    // ---- phase 3
    line_reduce(partA, k + 1, nblk, h1);
    if (owner) {
      combine(h1, k + 1, [&](int ic, int il, double d) { w[ic * per + il] -= d; });
      dots(partB);
    }
    if (!line_barrier(a.bar, gen, a.spin)) return;
    // ---- phase 4
    line_reduce(partB, k + 1, nblk, h2);
    if (owner) {
      combine(h2, k + 1, [&](int ic, int il, double d) {
        const double v = w[ic * per + il] - d;
        w[ic * per + il] = v;
        wbuf[(long)ic * N + i0 + il] = v;
      });
      double d = 0.0;
      if (nc * own <= 32) {   // one warp holds them all
        if (warp == 0) {
          if (lane < nc * own) {
            const int ic = lane / own;
            const double q = w[ic * per + lane - ic * own];
            d = fma(q, q, d);
          }
          for (int o = 16; o > 0; o >>= 1) d += __shfl_down_sync(0xffffffffu, d, o);
        }
      } else {
        for (int t = tid; t < nc * own; t += kLineThreads) {
          const int ic = t / own;
          const double q = w[ic * per + t - ic * own];
          d = fma(q, q, d);
        }
        d = block_sum(d, red);
      }
      if (tid == 0) partA[blockIdx.x] = d;   // (every block has read h1's partials)
    }
    if (!line_barrier(a.bar, gen, a.spin)) return;
    hn = line_norm(partA, nblk);
    if (!isfinite(hn) || hn == 0.0) {   // (the same in every block)
      status = isfinite(hn) ? 0 : 1;
      cols = k + 1;
      break;
    }
  }
  if (cols == 0) cols = k;   // m steps, or the loop ended at a converged column
  // the last block turns a column still pending and solves for y
  const bool pending = k >= a.m || hn == 0.0 || status != 0;
  if (!owner) {
    if (tid == 0) {
      if (pending && status == 0) rotate(cols - 1);
      cs[0] = rel;
    }
    __syncthreads();
    rel = cs[0];
    if (tid < 32 && status == 0) {
      __threadfence_block();
      for (int i = cols - 1; i >= 0; i--) {
        const double yi = gv[i] / a.R[(long)i * (a.kdim + 1) + i];
        __syncwarp();
        for (int j = lane; j < i; j += 32) gv[j] -= a.R[(long)i * (a.kdim + 1) + j] * yi;
        if (lane == 0) gv[i] = yi;
        __syncwarp();
      }
      for (int j = lane; j < cols; j += 32) a.y[j] = gv[j];
    }
    if (tid == 0) *a.res = LineResult{status, cols, r0, rel};
  }
  if (!line_barrier(a.bar, gen, a.spin)) return;
  if (status != 0 || !owner) return;
  for (int j = tid; j < cols; j += kLineThreads) h1[j] = __ldcg(a.y + j);
  __syncthreads();
  combine(h1, cols, [&](int ic, int il, double d) { a.xout[(long)ic * N + i0 + il] = d; });
}

// Nodes per CTA: one tile or pairs of tiles, the fewest that leave one SM for the block without nodes; at most 64, so that
// the tiles' sums stay short against the barriers (9600 nodes on 152 SMs; larger meshes fill the SMs with separate kernels)
int gmres_line_per(long N, int nsm)
{
  if (nsm < 2) return 0;
  const long need = (N + nsm - 2) / (nsm - 1), pair = 2 * kLineTile;
  const long per = need <= kLineTile ? kLineTile : (need + pair - 1) / pair * pair;
  return per <= 64 ? (int)per : 0;
}

// tiles at a time: pairs of one component (more components fill the registers)
static int line_tiles(int nc, int per) { return nc == 1 && per > kLineTile ? 2 : 1; }

size_t gmres_line_smem(int nc, bool tr, bool f32, int kdim, int per, int h)
{
  return line_layout(nc, nc == 1 ? 1 : kMaxC, tr, kdim, per, per + 2 * h, line_tiles(nc, per),
                     f32 ? sizeof(float) : sizeof(double)).bytes;
}

template <class T, bool TR, int NC, int NT>
static cudaError_t line_launch(const LineArgs<T> &a, int grid, size_t smem, cudaStream_t s)
{
  cudaError_t e = cudaFuncSetAttribute(k_gmres_line<T, TR, NC, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  void *args[] = {const_cast<LineArgs<T> *>(&a)};
  return cudaLaunchCooperativeKernel((const void *)k_gmres_line<T, TR, NC, NT>, dim3(grid), dim3(kLineThreads), args, smem, s);
}

template <class T, bool TR>
static cudaError_t line_launch_nt(const LineArgs<T> &a, int nc, int grid, size_t smem, cudaStream_t s)
{
  if (nc > 1) return line_launch<T, TR, kMaxC, 1>(a, grid, smem, s);
  return line_tiles(nc, a.per) == 2 ? line_launch<T, TR, 1, 2>(a, grid, smem, s) : line_launch<T, TR, 1, 1>(a, grid, smem, s);
}

template <class T>
static LineSten<T> line_sten(const DevStencil &st, const double *c64, const float *c32, bool negated)
{
  LineSten<T> o;
  o.off = negated ? st.d_loff_neg : st.d_loff;
  if constexpr (sizeof(T) == sizeof(float)) o.coef = c32;
  else o.coef = c64;
  o.L = st.L;
  return o;
}

template <class T>
static cudaError_t gmres_line_t(const LineCall &q, cudaStream_t s)
{
  LineArgs<T> a{};
  const int nc = q.ncomp;
  for (int ic = 0; ic < nc; ic++) {
    const DevStencil &th = q.sten[TGPU_STEN_THETA][ic], &de = q.sten[TGPU_STEN_DELTA][ic];
    a.th[ic] = line_sten<T>(th, th.d_coef_fwd, th.d_coef_fwd32, q.transpose);
    a.de[ic] = q.transpose ? line_sten<T>(de, de.d_coef_adj, nullptr, true)
                           : line_sten<T>(de, de.d_coef_fwd, de.d_coef_fwd32, false);
    a.tth[ic] = line_sten<T>(th, th.d_coef_tr, th.d_coef_tr32, false);
    a.tde[ic] = line_sten<T>(de, de.d_coef_tr, de.d_coef_tr32, false);
  }
  if (q.attraction)
    for (int k = 0; k < nc * nc; k++) {
      const DevStencil &ua = q.sten[TGPU_STEN_UATT][k];
      a.ua[k] = line_sten<T>(ua, ua.d_coef_fwd, ua.d_coef_fwd32, q.transpose);
    }
  a.x = q.x;
  a.vext = q.vext;
  a.hcoef = q.hcoef;
  a.rhs = q.rhs;
  a.zero = q.zero;
  a.V = q.V;
  a.part = q.part;
  a.R = q.R;
  a.y = q.y;
  a.xout = q.xout;
  a.chan = static_cast<T *>(q.chan);
  a.kind = q.kind;
  a.bar = q.bar;
  a.res = q.res;
  a.ldv = (long)nc * q.N;
  a.per = q.per;
  a.kdim = q.kdim;
  a.m = q.m;
  a.spin = q.spin;
  a.tol = q.tol;
  const int grid = (int)((q.N + q.per - 1) / q.per) + 1;
  const size_t smem = gmres_line_smem(nc, q.transpose, sizeof(T) == sizeof(float), q.kdim, q.per, q.h);
  if constexpr (sizeof(T) == sizeof(double))
    if (q.transpose) return line_launch_nt<T, true>(a, nc, grid, smem, s);
  return line_launch_nt<T, false>(a, nc, grid, smem, s);
}

// One GMRES cycle of a 1-D problem (the caller has zeroed q.bar's kLineBarWords words)
cudaError_t launch_gmres_line(const LineCall &q, cudaStream_t s)
{
  return q.f32 ? gmres_line_t<float>(q, s) : gmres_line_t<double>(q, s);
}
