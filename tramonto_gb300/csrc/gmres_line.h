// GMRES of a 1-D problem in one launch (included by kernels.cu).
//
// At 300 to 4000 nodes one GMRES iteration was about 25 launches of 2 to 20 us and a wait for the host, 190 to 210 us
// in all: every kernel was far below a wave, the FP64 stencil sums a serial chain of a few hundred FMAs on a handful
// of SMs.  Here one cooperative launch runs a whole GMRES cycle (the operator, diagonal preconditioner, classical
// Gram-Schmidt twice, rotations and the update x = V y), each CTA owning a few nodes and the phases separated by a
// barrier over the grid:
//   1  sums of the density-shaped vector over the CTA's window, local step, channels out        -> barrier
//   2  sums of the channels, row combination, preconditioner; V_j . w of the CTA's nodes        -> barrier
//   3  h1 = V^T w; w -= V h1; V_j . w again                                                     -> barrier
//   4  h2; w -= V h2; |w|^2                                                                     -> barrier
//   5  V_k+1 = w / |w|                                                                          -> barrier
// One more CTA owns no nodes and turns the new column by the rotations during the next phase 1, so that the chain of
// dependent FP64 operations costs nothing; the stopping test is read one barrier later.
//
// Work split: 8 nodes x 32 groups of taps per CTA (a warp holds 8 nodes x 4 groups), so that the FP64 pipe of as many
// SMs as there are 8-node tiles works on the sums; sums over groups, nodes and CTAs are taken in a fixed order.
// Bound: latency (a warp's FP64 operation holds its scheduler's pipe for 64 cycles, so short serial steps count) and
// five barriers; 2001 nodes of hard spheres in FP64: 43 us per iteration against 210, 1487 nodes of the slit pore with
// FP32 products 38 against 185.
//
// TR: the transposed Schur complement (adjoint solves), from the stencils with negated offsets.

constexpr int kLineThreads = 256, kLineTile = 8, kLineGroups = 32, kLineWarps = kLineThreads / 32;
constexpr int kLineSpin = 1 << 24;   // polls before a barrier gives up

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
  unsigned *bar;        // arrivals, error
  LineResult *res;
  long ldv;             // ncomp * N
  int per, kdim, m;     // nodes per CTA, vectors that R holds, steps of this cycle
  double tol;
};

// Barrier over the grid; false when it gave up (then every block returns)
__device__ __forceinline__ bool line_barrier(unsigned *bar, unsigned &gen)
{
  __shared__ int s_ok;
  __syncthreads();
  gen++;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    const unsigned target = gen * gridDim.x;
    int ok = 1, spins = 0;
    unsigned seen;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
      if (++spins > kLineSpin) {
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

// sum over the 32 groups of a tile's value; threads 0..7 return the nodes' sums (red: kLineWarps * 8 values)
template <class A>
__device__ __forceinline__ A line_group_sum(A v, A *red)
{
  v += __shfl_xor_sync(0xffffffffu, v, 8);
  v += __shfl_xor_sync(0xffffffffu, v, 16);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane < kLineTile) red[warp * kLineTile + lane] = v;
  __syncthreads();
  A s = 0;
  if (threadIdx.x < kLineTile)
#pragma unroll
    for (int w = 0; w < kLineWarps; w++) s += red[w * kLineTile + threadIdx.x];
  __syncthreads();
  return s;
}

// out[j] = sum over the blocks of part[j * nblk + b], j < cnt
__device__ __forceinline__ void line_reduce(const double *part, int cnt, int nblk, double *out)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j = warp; j < cnt; j += kLineWarps) {
    double s = 0.0;
#pragma unroll 5
    for (int b = lane; b < nblk; b += 32) s += __ldcg(part + (long)j * nblk + b);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[j] = s;
  }
  __syncthreads();
}

// acc[o] += sum of the group's taps of one stencil, NI inputs (windows ld apart) and NO outputs
template <int NI, int NO, class T>
__device__ __forceinline__ void line_taps(const LineSten<T> &st, const T *win, int ld, int at, int grp, T *acc)
{
#pragma unroll 2
  for (int k = grp; k < st.L; k += kLineGroups) {
    const int p = at + __ldg(st.off + k);
#pragma unroll
    for (int o = 0; o < NO; o++)
#pragma unroll
      for (int c = 0; c < NI; c++) acc[o] = fma(__ldg(st.coef + (k * NO + o) * NI + c), win[c * ld + p], acc[o]);
  }
}

// One row of a window: `src` at the padded positions q0 .. q0 + n - 1 (0 outside the mesh: the linear products' boundary
// values); flag: nodes that read 0; flip: reflected positions change sign
template <class T, class S>
__device__ __forceinline__ void line_window(T *win, const S *src, const signed char *flag, bool flip, int q0, int n)
{
  for (int t = threadIdx.x; t < n; t += kLineThreads) {
    const int q = q0 + t;
    T v = 0;
    if (q < c_g.P[0]) {
      const int m = c_g.map[0][q];
      if (m >= 0) {
        const int i = m & ~kReflBit;
        const S s = __ldcg(src + i);
        if (!(flag && __ldcg(flag + i))) v = (T)s;
        if (flip && (m & kReflBit)) v = -v;
      } else if (m == kSentBad) {
        v = (T)__longlong_as_double(0x7ff8000000000000ULL);
      }
    }
    win[t] = v;
  }
}

template <class T, bool TR, int NC>
__global__ void __launch_bounds__(kLineThreads) k_gmres_line(LineArgs<T> a)
{
  constexpr int ND = 1, NRB = 6, CPC = ND + 2;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int nc = NC == 1 ? 1 : c_g.ncomp, per = a.per, h = c_g.h[0], nw = per + 2 * h;
  const long N = c_g.N;
  const int nblk = gridDim.x - 1;                    // blocks that own nodes
  const bool owner = (int)blockIdx.x < nblk;
  const int i0 = blockIdx.x * per, own = owner ? (int)min((long)per, N - i0) : 0;
  // shared memory: window rows, then doubles: reductions, w, -u_MF, columns h1 h2, rotations and right-hand side
  const int nch = max(nc, nc * CPC + (TR ? nc : 0));
  T *win = reinterpret_cast<T *>(smraw);
  double *red = reinterpret_cast<double *>(smraw + ((sizeof(T) * (size_t)nch * nw + 15) & ~(size_t)15));
  double *w = red + kLineWarps * kLineTile, *ymf = w + nc * per, *hc = ymf + nc * per;
  double *h1 = hc, *h2 = hc + a.kdim + 2, *cs = h2 + a.kdim + 2, *sn = cs + a.kdim, *gv = sn + a.kdim;
  T *sums = reinterpret_cast<T *>(gv + a.kdim + 1);   // [NRB + NC][8]
  T *redT = reinterpret_cast<T *>(red);
  const int lane = threadIdx.x & 31, nl = lane & 7, grp = (threadIdx.x >> 5) * 4 + (lane >> 3);
  double *partA = a.part, *partB = a.part + (long)(a.kdim + 2) * nblk;
  const bool att = c_g.attraction != 0;
  unsigned gen = 0;

  // r0 = M^-1 b, beta = |r0|
  double s = 0.0;
  for (int t = threadIdx.x; t < nc * own; t += kLineThreads) {
    const int ic = t / own, i = i0 + t - ic * own;
    const long k = (long)ic * N + i;
    const bool zr = zero_row(a.vext, a.zero, ic, i), lr = zr && log_row(a.vext, a.zero, ic, i);
    a.kind[k] = !zr ? 0 : lr ? 1 : 2;
    const double r = (zr && !lr) ? a.rhs[k] : a.rhs[k] * a.x[(long)(c_g.first_rho + ic) * N + i];
    w[ic * per + i - i0] = r;
    s = fma(r, r, s);
  }
  s = block_sum(s, red);
  if (owner && threadIdx.x == 0) partA[blockIdx.x] = s;
  if (!line_barrier(a.bar, gen)) return;
  line_reduce(partA, 1, nblk, h1);
  const double r0 = sqrt(h1[0]);
  __syncthreads();
  if (!(r0 > 0.0)) {   // a zero or non-finite right-hand side: the host decides
    for (int t = threadIdx.x; t < nc * own; t += kLineThreads) {
      const int ic = t / own;
      a.xout[(long)ic * N + i0 + t - ic * own] = 0.0;
    }
    if (!owner && threadIdx.x == 0) *a.res = LineResult{0, 0, r0, 0.0};
    return;
  }
  for (int t = threadIdx.x; t < nc * own; t += kLineThreads) {
    const int ic = t / own, i = t - ic * own;
    a.V[(long)ic * N + i0 + i] = w[ic * per + i] / r0;
  }
  if (threadIdx.x == 0) gv[0] = r0;
  if (!line_barrier(a.bar, gen)) return;

  // the pending column (in h1, h2, norm hn) of the block without nodes: rotations; true when the residual meets tol
  double hn = 0.0, rel = 1.0;
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

  auto subtract = [&](const double *hv) {   // w -= V h
    for (int ic = 0; ic < nc; ic++)
      for (int t0 = 0; t0 < own; t0 += kLineTile) {
        const int il = t0 + nl;
        double d = 0.0;
        if (il < own)
          for (int j = grp; j <= k; j += kLineGroups)
            d = fma(hv[j], a.V[(long)j * a.ldv + (long)ic * N + i0 + il], d);
        d = line_group_sum<double>(d, red);
        const int io = t0 + (int)threadIdx.x;
        if (threadIdx.x < kLineTile && io < own) w[ic * per + io] -= d;
      }
    __syncthreads();
  };
  auto dots = [&](double *part) {   // V_j . w of the block's nodes
    for (int j = threadIdx.x; j <= k; j += kLineThreads) {
      double d = 0.0;
      for (int ic = 0; ic < nc; ic++) {
        const double *v = a.V + (long)j * a.ldv + (long)ic * N + i0;
        for (int i = 0; i < own; i++) d = fma(v[i], w[ic * per + i], d);
      }
      part[(long)j * nblk + blockIdx.x] = d;
    }
  };
  for (; k < a.m; k++) {
    const double *vk = a.V + (long)k * a.ldv;
    // ---- phase 1
    if (owner) {
      for (int ic = 0; ic < nc; ic++)
        line_window<T, double>(win + ic * nw, vk + (long)ic * N, (TR ? a.kind : a.zero) + (long)ic * N, false, i0, nw);
      __syncthreads();
      for (int t0 = 0; t0 < own; t0 += kLineTile) {
        const int at = t0 + nl + h;
        T acc[NRB + NC];
#pragma unroll
        for (int r = 0; r < NRB + NC; r++) acc[r] = 0;
        if constexpr (TR) {
          // per component (scalar, vector) of the delta shell and the ball: combined at once into the rows of g
          // (n ordering: acc 0..5 = g0 g1 g2 g3 gV1 gV2)
#pragma unroll
          for (int ic = 0; ic < NC; ic++)
            if (ic < nc) {
              T d[2] = {0, 0}, b[1] = {0};
              line_taps<1, 2, T>(a.de[ic], win + ic * nw, nw, at, grp, d);
              line_taps<1, 1, T>(a.th[ic], win + ic * nw, nw, at, grp, b);
              acc[2] += d[0];
              acc[1] += (T)c_g.inv_4pir[ic] * d[0];
              acc[0] += (T)c_g.inv_4pirsq[ic] * d[0];
              acc[3] += b[0];
              acc[5] -= d[1];
              acc[4] -= (T)c_g.inv_4pir[ic] * d[1];
            }
        } else {
#pragma unroll
          for (int jc = 0; jc < NC; jc++)
            if (jc < nc) {
              const T *wj = win + jc * nw;
              line_taps<1, 1, T>(a.th[jc], wj, nw, at, grp, acc);          // n3
              if (NC == 1 && c_g.single_size) {
                T d[2] = {0, 0};
                line_taps<1, 2, T>(a.de[jc], wj, nw, at, grp, d);          // n2, V2
                acc[1] += d[0];
                acc[4] += d[1];
              } else if (c_g.single_size) {
                T d[2] = {0, 0};
                line_taps<1, 2, T>(a.de[jc], wj, nw, at, grp, d);
                acc[1] += d[0];
                acc[4] += d[1];
              } else {
                line_taps<1, 5, T>(a.de[jc], wj, nw, at, grp, acc + 1);    // n2, n1, n0, V2, V1
              }
              if (att)
#pragma unroll
                for (int ic = 0; ic < NC; ic++)
                  if (ic < nc) line_taps<1, 1, T>(a.ua[ic + nc * jc], wj, nw, at, grp, acc + NRB + ic);
            }
        }
#pragma unroll
        for (int r = 0; r < NRB + NC; r++) {
          if (!TR && c_g.single_size && (r == 2 || r == 3 || r == 5)) continue;
          if (r >= NRB && (TR || !att || r - NRB >= nc)) continue;
          const T v = line_group_sum<T>(acc[r], redT);
          if (threadIdx.x < kLineTile) sums[r * kLineTile + threadIdx.x] = v;
        }
        // local step of a node
        if (threadIdx.x < kLineTile && t0 + (int)threadIdx.x < own) {
          const int tl = threadIdx.x, il = t0 + tl;
          const long i = i0 + il;
          if constexpr (TR) {
            double g[NRB], z[NRB];
            for (int r = 0; r < NRB; r++) g[r] = (double)sums[r * kLineTile + tl];
            hess_apply_node(a.x, a.hcoef, i, g, z, true);
            // t = J^T [0; v] on the block-1 rows, y = A11^-T t, and y's channels
            double v[NRB] = {-z[3], -z[2], -z[1], -z[0], -z[5], -z[4]};   // -t, rows n3 n2 n1 n0 V2 V1
            if (c_g.single_size) {
              v[1] -= c_g.inv_4pir[0] * z[1] + c_g.inv_4pirsq[0] * z[0];
              v[4] -= c_g.inv_4pir[0] * z[4];
            }
            const double wn1 = c_g.single_size ? 0.0 : v[2], wn0 = c_g.single_size ? 0.0 : v[3];
            const double wv1 = c_g.single_size ? 0.0 : v[5];
            for (int jc = 0; jc < nc; jc++) {
              T *ch = a.chan + (long)jc * CPC * N + i;
              ch[0] = (T)(v[1] + c_g.inv_4pir[jc] * wn1 + c_g.inv_4pirsq[jc] * wn0);
              ch[N] = (T)(v[4] + c_g.inv_4pir[jc] * wv1);
              ch[2 * N] = (T)v[0];
              // mean-field row: t = w_EL (full rows), y = -t
              if (att) a.chan[(long)(nc * CPC + jc) * N + i] = (T)(-win[jc * nw + il + h]);
            }
          } else {
            T ysv[NRB], y[NRB], z[NRB];
            for (int r = 0; r < NRB; r++) {
              int src;
              double cd;
              if (dep_rb(r, &src, &cd)) ysv[r] = -to_arith<T>(cd) * sums[src * kLineTile + tl];   // -u_dep - B u_ind
              else ysv[r] = -sums[r * kLineTile + tl];
            }
            y[0] = ysv[3]; y[1] = ysv[2]; y[2] = ysv[1]; y[3] = ysv[0]; y[4] = ysv[5]; y[5] = ysv[4];
            if constexpr (sizeof(T) == sizeof(double)) hess_apply_node(a.x, a.hcoef, i, y, z);
            else hess_apply_node_t<T>(a.x, a.hcoef, i, y, z);
            for (int ic = 0; ic < nc; ic++) {
              const T f = to_arith<T>(c_g.fac[ic]), r1 = to_arith<T>(c_g.inv_4pir[ic]), r2 = to_arith<T>(c_g.inv_4pirsq[ic]);
              T *ch = a.chan + (long)ic * CPC * N + i;
              ch[0] = f * (z[0] * r2 + z[1] * r1 + z[2]);
              ch[N] = f * (z[4] * r1 + z[5]);
              ch[2 * N] = f * z[3];
              if (att) ymf[ic * per + il] = -(double)sums[(NRB + ic) * kLineTile + tl];
            }
          }
        }
        __syncthreads();
      }
    } else if (k > 0 && threadIdx.x == 0) {
      rotate(k - 1);
      a.res->its = rel < a.tol ? -k : 0;   // its < 0: converged after -its steps
    }
    if (!line_barrier(a.bar, gen)) return;
    if (k > 0 && __ldcg(&a.res->its) < 0) {
      cols = k;
      break;
    }
    // ---- phase 2
    if (owner) {
      const int rows = nc * CPC + (TR && att ? nc : 0);
      for (int r = 0; r < rows; r++)
        line_window<T, T>(win + r * nw, a.chan + (long)r * N, nullptr, !TR && r % CPC == 1, i0, nw);
      __syncthreads();
      for (int t0 = 0; t0 < own; t0 += kLineTile) {
        const int at = t0 + nl + h;
        for (int ic = 0; ic < nc; ic++) {
          T d[1] = {0}, b[1] = {0};
          const T *wi = win + ic * CPC * nw;
          line_taps<2, 1, T>(TR ? a.de[ic] : a.tde[ic], wi, nw, at, grp, d);
          line_taps<1, 1, T>(TR ? a.th[ic] : a.tth[ic], wi + 2 * nw, nw, at, grp, b);
          if (TR && att)
            for (int jc = 0; jc < nc; jc++)
              line_taps<1, 1, T>(a.ua[jc + nc * ic], win + (nc * CPC + jc) * nw, nw, at, grp, b);
          const double tr = line_group_sum<double>((double)d[0] + (double)b[0], red);
          const int il = t0 + (int)threadIdx.x;
          if (threadIdx.x < kLineTile && il < own) {
            const long kk = (long)ic * N + i0 + il;
            const int kd = a.kind[kk];
            const double v2 = vk[kk], rho = a.x[(long)(c_g.first_rho + ic) * N + i0 + il];
            double r;   // M^-1 S v
            if (TR) r = v2 - (a.zero[kk] ? 0.0 : kd == 2 ? tr : tr * rho);
            else r = kd == 0 ? (v2 / rho - (att ? tr + ymf[ic * per + il] : tr)) * rho : v2;
            w[ic * per + il] = r;
          }
        }
      }
      __syncthreads();
      dots(partA);
    }
    if (!line_barrier(a.bar, gen)) return;
    // ---- phase 3
    line_reduce(partA, k + 1, nblk, h1);
    if (owner) {
      subtract(h1);
      dots(partB);
    }
    if (!line_barrier(a.bar, gen)) return;
    // ---- phase 4
    line_reduce(partB, k + 1, nblk, h2);
    if (owner) {
      subtract(h2);
      double d = 0.0;
      for (int t = threadIdx.x; t < nc * own; t += kLineThreads) {
        const int ic = t / own;
        const double q = w[ic * per + t - ic * own];
        d = fma(q, q, d);
      }
      d = block_sum(d, red);
      if (threadIdx.x == 0) partA[blockIdx.x] = d;   // (every block has read h1's partials)
    }
    if (!line_barrier(a.bar, gen)) return;
    // ---- phase 5
    line_reduce(partA, 1, nblk, red);
    hn = sqrt(red[0]);
    __syncthreads();
    if (!isfinite(hn) || hn == 0.0) {   // (the same in every block)
      status = isfinite(hn) ? 0 : 1;
      cols = k + 1;
      break;
    }
    for (int t = threadIdx.x; t < nc * own; t += kLineThreads) {
      const int ic = t / own, i = t - ic * own;
      a.V[(long)(k + 1) * a.ldv + (long)ic * N + i0 + i] = w[ic * per + i] / hn;
    }
    if (!line_barrier(a.bar, gen)) return;
  }
  if (cols == 0) cols = k;   // m steps, or the loop ended at a converged column
  // the last block turns a column still pending and solves for y
  const bool pending = k >= a.m || hn == 0.0 || status != 0;
  if (!owner) {
    if (threadIdx.x == 0) {
      if (pending && status == 0) rotate(cols - 1);
      cs[0] = rel;
    }
    __syncthreads();
    rel = cs[0];
    if (threadIdx.x < 32 && status == 0) {
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
    if (threadIdx.x == 0) *a.res = LineResult{status, cols, r0, rel};
  }
  if (!line_barrier(a.bar, gen)) return;
  if (status != 0) return;
  for (int ic = 0; ic < nc; ic++)
    for (int t0 = 0; t0 < own; t0 += kLineTile) {
      const int il = t0 + nl;
      double d = 0.0;
      if (il < own)
        for (int j = grp; j < cols; j += kLineGroups)
          d = fma(__ldcg(a.y + j), a.V[(long)j * a.ldv + (long)ic * N + i0 + il], d);
      d = line_group_sum<double>(d, red);
      const int io = t0 + (int)threadIdx.x;
      if (threadIdx.x < kLineTile && io < own) a.xout[(long)ic * N + i0 + io] = d;
    }
}

static size_t line_smem(int nc, bool tr, int kdim, int per, int h, size_t t)
{
  const size_t nch = (size_t)std::max(nc, nc * 3 + (tr ? nc : 0));
  const size_t win = (t * nch * (per + 2 * h) + 15) & ~(size_t)15;
  return win + sizeof(double) * (kLineWarps * kLineTile + 2 * (size_t)nc * per + 2 * (kdim + 2) + 3 * (size_t)kdim + 1) +
         t * (6 + (nc == 1 ? 1 : kMaxC)) * kLineTile;
}

// Nodes per CTA: whole tiles, the fewest that leave one SM for the block without nodes; at most 64, so that the tiles'
// sums stay short against the barriers (9600 nodes on 152 SMs; larger meshes fill the SMs with separate kernels)
int gmres_line_per(long N, int nsm)
{
  if (nsm < 2) return 0;
  const long per = ((N + nsm - 2) / (nsm - 1) + kLineTile - 1) / kLineTile * kLineTile;
  return per <= 64 ? (int)per : 0;
}

size_t gmres_line_smem(int nc, bool tr, bool f32, int kdim, int per, int h)
{
  return line_smem(nc, tr, kdim, per, h, f32 ? sizeof(float) : sizeof(double));
}

template <class T, bool TR, int NC>
static cudaError_t line_launch(const LineArgs<T> &a, int grid, size_t smem, cudaStream_t s)
{
  cudaError_t e = cudaFuncSetAttribute(k_gmres_line<T, TR, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  void *args[] = {const_cast<LineArgs<T> *>(&a)};
  return cudaLaunchCooperativeKernel((const void *)k_gmres_line<T, TR, NC>, dim3(grid), dim3(kLineThreads), args, smem, s);
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
  a.tol = q.tol;
  const int grid = (int)((q.N + q.per - 1) / q.per) + 1;
  const size_t smem = line_smem(nc, q.transpose, q.kdim, q.per, q.h, sizeof(T));
  if constexpr (sizeof(T) == sizeof(double))
    if (q.transpose) return nc == 1 ? line_launch<T, true, 1>(a, grid, smem, s) : line_launch<T, true, kMaxC>(a, grid, smem, s);
  return nc == 1 ? line_launch<T, false, 1>(a, grid, smem, s) : line_launch<T, false, kMaxC>(a, grid, smem, s);
}

// One GMRES cycle of a 1-D problem (the caller has zeroed q.bar's two words)
cudaError_t launch_gmres_line(const LineCall &q, cudaStream_t s)
{
  return q.f32 ? gmres_line_t<float>(q, s) : gmres_line_t<double>(q, s);
}
