// Point sums of 1-D problems, a whole pass in one launch (included by kernels.cu).
//
// A pass of k_pad and one k_conv per stencil was five launches, each far below a wave: 256 nodes to a block, a serial
// chain of a few hundred FMAs per node, each waiting for its loads.  Here a block owns 32 nodes and one stencil (for all
// densities), its window is read through the boundary map by all threads, and an output's chain runs in one warp from
// shared memory; blocks of different stencils run side by side.  A node's taps are still added in table order, output
// by output, as k_conv adds them: the sums are the same numbers.  Bound: that chain, 64 clocks of a scheduler's FP64
// pipe per tap.  Hard wall, 2001 nodes, FP64: a forward pass 30 -> 8 us, a transposed one 31 -> 13; slit pore, 1487
// nodes with the mean field's 501 taps: 49 -> 28 and 34 -> 16, in FP32 40 -> 10 and 26 -> 9.

constexpr int kLineSumThreads = 128, kLineSumWarps = kLineSumThreads / 32;

// window of a channel as k_pad fills the padded box; all threads
template <class T>
__device__ __forceinline__ void line_field(T *win, const double *src, const signed char *zero, double lo, double hi,
                                           bool flip, int q0, int n)
{
#pragma unroll 4
  for (int t = threadIdx.x; t < n; t += kLineSumThreads) {
    const int q = q0 + t;
    double v = 0.0;
    if (q < c_g.P[0]) {
      const int m = c_g.map[0][q];
      if (m >= 0) {
        const int i = m & ~kReflBit;
        v = src[i];
        if (zero && zero[i]) v = 0.0;
        if (flip && (m & kReflBit)) v = -v;
      } else {
        v = m == kSentBulk ? lo : m == kSentBulkHi ? hi : m == kSentWall ? 0.0 : __longlong_as_double(0x7ff8000000000000ULL);
      }
    }
    win[t] = (T)v;
  }
}

// output o of a node's sum over one stencil (no outputs, NI windows ld apart), taps in order; the warp's lanes fetch the
// next 32 taps while it adds the present ones from its part of shared memory
template <class T>
struct LineChunk {
  T coef[64];
  int off[32];
};
template <int NI, class T>
__device__ __forceinline__ T line_chain(const LineSten<T> &st, int no, int o, const T *win, int ld, LineChunk<T> *chunk)
{
  const int lane = threadIdx.x & 31;
  const auto fetch = [&](int k, int &p, T *cf) {
    if (k < st.L) {
      p = __ldg(st.off + k);
#pragma unroll
      for (int c = 0; c < NI; c++) cf[c] = __ldg(st.coef + (k * no + o) * NI + c);
    }
  };
  int p = 0;
  T cf[NI] = {}, acc = 0;
  fetch(lane, p, cf);
  for (int k0 = 0; k0 < st.L; k0 += 32) {
    __syncwarp();
    chunk->off[lane] = p;
#pragma unroll
    for (int c = 0; c < NI; c++) chunk->coef[lane * NI + c] = cf[c];
    __syncwarp();
    fetch(k0 + 32 + lane, p, cf);
    const int n = min(32, st.L - k0);
#pragma unroll 8
    for (int j = 0; j < n; j++) {
      const T *w = win + chunk->off[j];
#pragma unroll
      for (int c = 0; c < NI; c++) acc = fma(chunk->coef[j * NI + c], w[c * ld], acc);
    }
  }
  return acc;
}

template <class T>
struct LineSums {
  LineSten<T> th[kMaxC], de[kMaxC], ua[kMaxC * kMaxC];   // forward tables, or the transposed th and de
  const double *src, *bulk;    // channels; boundary values [low side channels][high side channels]
  const int *sign;
  const signed char *zero;
  double *out;                 // [nrb + ncomp][N], or [ncomp][N] transposed
  int nch;
};

// forward sums (every row of out): blockIdx.y 0 theta, 1 delta (a warp per output), 2 + ic the mean field of component ic
template <class T>
__global__ void __launch_bounds__(kLineSumThreads) k_line_forward(LineSums<T> a)
{
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ LineChunk<T> chunks[kLineSumWarps];
  T *win = reinterpret_cast<T *>(smraw);
  const long N = c_g.N;
  const int nc = c_g.ncomp, h = c_g.h[0], nw = 32 + 2 * h, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int job = blockIdx.y;
  const bool one = c_g.single_size != 0;
  const int no = job != 1 ? 1 : one ? 2 : 5;
  const long i = blockIdx.x * 32L + lane;
  double r[2] = {0, 0};   // outputs warp and warp + 4
  for (int jc = 0; jc < nc; jc++) {
    __syncthreads();
    line_field<T>(win, a.src + (long)jc * N, a.zero + (long)jc * N, a.bulk[jc], a.bulk[a.nch + jc], false,
                  blockIdx.x * 32, nw);
    __syncthreads();
    const LineSten<T> &st = job == 0 ? a.th[jc] : job == 1 ? a.de[jc] : a.ua[job - 2 + nc * jc];
#pragma unroll
    for (int u = 0; u < 2; u++)
      if (warp + 4 * u < no) r[u] += (double)line_chain<1, T>(st, no, warp + 4 * u, win + lane + h, nw, chunks + warp);
  }
  if (i >= N) return;
  if (job == 0) {
    if (warp == 0) a.out[i] = r[0];
    if (!c_g.attraction)
      for (int ic = warp; ic < nc; ic += kLineSumWarps) a.out[(long)(c_g.nrb + ic) * N + i] = 0.0;
  } else if (job >= 2) {
    if (warp == 0) a.out[(long)(c_g.nrb + job - 2) * N + i] = r[0];
  } else if (one) {   // rows n2 n1 n0 V2 V1: n1, n0 and V1 are multiples
    if (warp == 0) a.out[N + i] = r[0];
    else if (warp == 1) a.out[4 * N + i] = r[0];
    else for (int row : {2, 3, 5})
      if ((row == 2) == (warp == 2)) a.out[row * N + i] = 0.0;
  } else {
    a.out[(1 + warp) * N + i] = r[0];
    if (warp == 0) a.out[5 * N + i] = r[1];
  }
}

// transposed sums of component blockIdx.y: warp 0 the delta shell's two channels, warp 1 the ball's
template <class T>
__global__ void __launch_bounds__(kLineSumThreads) k_line_transposed(LineSums<T> a)
{
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ LineChunk<T> chunks[2];
  __shared__ double s_de[32];
  const long N = c_g.N;
  const int h = c_g.h[0], nw = 32 + 2 * h, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ic = blockIdx.y;
  T *win = reinterpret_cast<T *>(smraw);
  const long i = blockIdx.x * 32L + lane;
  for (int c = 0; c < 3; c++) {
    const int ch = 3 * ic + c;
    line_field<T>(win + c * nw, a.src + (long)ch * N, nullptr, a.bulk[ch], a.bulk[a.nch + ch], a.sign[ch] != 0,
                  blockIdx.x * 32, nw);
  }
  __syncthreads();
  double v = 0.0;
  if (warp == 0) s_de[lane] = (double)line_chain<2, T>(a.de[ic], 1, 0, win + lane + h, nw, chunks);
  else if (warp == 1) v = (double)line_chain<1, T>(a.th[ic], 1, 0, win + 2 * nw + lane + h, nw, chunks + 1);
  __syncthreads();
  if (warp == 1 && i < N) a.out[(long)ic * N + i] = s_de[lane] + v;
}

template <class T>
static void line_sums_t(const LineSumsCall &q, cudaStream_t s)
{
  LineSums<T> a{};
  for (int ic = 0; ic < q.ncomp; ic++) {
    const DevStencil &th = q.sten[TGPU_STEN_THETA][ic], &de = q.sten[TGPU_STEN_DELTA][ic];
    a.th[ic] = q.transposed ? line_sten<T>(th, th.d_coef_tr, th.d_coef_tr32, false)
                            : line_sten<T>(th, th.d_coef_fwd, th.d_coef_fwd32, false);
    a.de[ic] = q.transposed ? line_sten<T>(de, de.d_coef_tr, de.d_coef_tr32, false)
                            : line_sten<T>(de, de.d_coef_fwd, de.d_coef_fwd32, false);
  }
  if (!q.transposed && q.attraction)
    for (int k = 0; k < q.ncomp * q.ncomp; k++) {
      const DevStencil &ua = q.sten[TGPU_STEN_UATT][k];
      a.ua[k] = line_sten<T>(ua, ua.d_coef_fwd, ua.d_coef_fwd32, false);
    }
  a.src = q.src;
  a.bulk = q.bulk;
  a.sign = q.sign;
  a.zero = q.zero;
  a.out = q.out;
  a.nch = q.nch;
  const unsigned blocks = (unsigned)((q.N + 31) / 32);
  const size_t row = sizeof(T) * (size_t)(32 + 2 * q.h);
  if (q.transposed) k_line_transposed<T><<<dim3(blocks, q.ncomp), kLineSumThreads, 3 * row, s>>>(a);
  else k_line_forward<T><<<dim3(blocks, 2 + (q.attraction ? q.ncomp : 0)), kLineSumThreads, row, s>>>(a);
}

// The windows fit in the 48 KB of shared memory that need no attribute.  A whole FP64 fill against one launch per
// stencil: hard wall 4001 nodes 121 -> 67 us, 16001 124 -> 74, 32001 138 -> 103; slit pore 4001 160 -> 93, 32001
// 177 -> 156 (501 taps), 118 -> 82 (101 taps).  Past that the SMs are full either way.
bool line_sums_ok(int ndim, long N, int h)
{
  return ndim == 1 && N <= 32768 && 3 * sizeof(double) * (32 + 2L * h) <= 42 * 1024;
}

void launch_line_sums(const LineSumsCall &q, cudaStream_t s)
{
  if (q.f32) line_sums_t<float>(q, s);
  else line_sums_t<double>(q, s);
}
