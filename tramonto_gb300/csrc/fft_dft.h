// DFTs of a compile-time length R <= 27 held in a thread's registers (fft.cu).
//
// Lengths 2, 3, 4, 5, 7 are written out in the symmetric forms that share the sums and differences of mirrored
// inputs; 8 rotates the odd half by eighths of a turn (an addition and a subtraction scaled once); lengths with
// coprime factors use the prime-factor map (Good 1958, Thomas 1963: input (B a + A b) mod AB, output by the Chinese
// remainder theorem, no twiddles); 9, 16, 25 and 27 are two-factor Cooley-Tukey with constant twiddles.  Every index
// is a constant after unrolling, so the values never leave registers; the compiler contracts the products into FMAs.
#pragma once

#include <type_traits>
#include <utility>

namespace tgpu {
namespace dft {

template <class C>
struct Real;
template <>
struct Real<double2> {
  using T = double;
};
template <>
struct Real<float2> {
  using T = float;
};

template <class C>
__device__ __forceinline__ C cmul(C a, C b)
{
  return C{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
// c + a b, in four operations (a product and a sum: six)
template <class C>
__device__ __forceinline__ C cfma(C a, C b, C c)
{
  return C{fma(-a.y, b.y, fma(a.x, b.x, c.x)), fma(a.y, b.x, fma(a.x, b.y, c.y))};
}
template <class C>
__device__ __forceinline__ C cadd(C a, C b)
{
  return C{a.x + b.x, a.y + b.y};
}
template <class C>
__device__ __forceinline__ C csub(C a, C b)
{
  return C{a.x - b.x, a.y - b.y};
}
// a -/+ i b: the forward transform's next output and its mirror image (inverse: exchanged)
template <bool INV, class C>
__device__ __forceinline__ C add_mi(C a, C b)
{
  return INV ? C{a.x - b.y, a.y + b.x} : C{a.x + b.y, a.y - b.x};
}
template <bool INV, class C>
__device__ __forceinline__ C sub_mi(C a, C b)
{
  return add_mi<!INV, C>(a, b);
}

template <class F, int... I>
__device__ __forceinline__ void static_for_impl(F &&f, std::integer_sequence<int, I...>)
{
  (f(std::integral_constant<int, I>{}), ...);
}
// f(integral_constant<int, 0>) ... f(integral_constant<int, N - 1>)
template <int N, class F>
__device__ __forceinline__ void static_for(F &&f)
{
  static_for_impl(f, std::make_integer_sequence<int, N>{});
}

// cos and sin of 2 pi m / N
template <int N>
struct Circle;
template <>
struct Circle<9> {
  static constexpr double c[9] = {1.0000000000000000000, 0.76604444311897803520, 0.17364817766693034885, -0.50000000000000000000, -0.93969262078590838405, -0.93969262078590838405, -0.50000000000000000000, 0.17364817766693034885, 0.76604444311897803520};
  static constexpr double s[9] = {0.0, 0.64278760968653932632, 0.98480775301220805937, 0.86602540378443864676, 0.34202014332566873304, -0.34202014332566873304, -0.86602540378443864676, -0.98480775301220805937, -0.64278760968653932632};
};
template <>
struct Circle<16> {
  static constexpr double c[16] = {1.0000000000000000000, 0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173, 0.0, -0.38268343236508977173, -0.70710678118654752440, -0.92387953251128675613, -1.0000000000000000000, -0.92387953251128675613, -0.70710678118654752440, -0.38268343236508977173, 0.0, 0.38268343236508977173, 0.70710678118654752440, 0.92387953251128675613};
  static constexpr double s[16] = {0.0, 0.38268343236508977173, 0.70710678118654752440, 0.92387953251128675613, 1.0000000000000000000, 0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173, 0.0, -0.38268343236508977173, -0.70710678118654752440, -0.92387953251128675613, -1.0000000000000000000, -0.92387953251128675613, -0.70710678118654752440, -0.38268343236508977173};
};
template <>
struct Circle<25> {
  static constexpr double c[25] = {1.0000000000000000000, 0.96858316112863111949, 0.87630668004386358731, 0.72896862742141152315, 0.53582679497899661827, 0.30901699437494742410, 0.062790519529313376076, -0.18738131458572463054, -0.42577929156507264886, -0.63742398974868971018, -0.80901699437494742410, -0.92977648588825140366, -0.99211470131447783105, -0.99211470131447783105, -0.92977648588825140366, -0.80901699437494742410, -0.63742398974868971018, -0.42577929156507264886, -0.18738131458572463054, 0.062790519529313376076, 0.30901699437494742410, 0.53582679497899661827, 0.72896862742141152315, 0.87630668004386358731, 0.96858316112863111949};
  static constexpr double s[25] = {0.0, 0.24868988716485478824, 0.48175367410171527499, 0.68454710592868867373, 0.84432792550201507855, 0.95105651629515357212, 0.99802672842827156195, 0.98228725072868868109, 0.90482705246601952771, 0.77051324277578923080, 0.58778525229247312917, 0.36812455268467795916, 0.12533323356430424537, -0.12533323356430424537, -0.36812455268467795916, -0.58778525229247312917, -0.77051324277578923080, -0.90482705246601952771, -0.98228725072868868109, -0.99802672842827156195, -0.95105651629515357212, -0.84432792550201507855, -0.68454710592868867373, -0.48175367410171527499, -0.24868988716485478824};
};
template <>
struct Circle<27> {
  static constexpr double c[27] = {1.0000000000000000000, 0.97304487057982383883, 0.89363264032341224819, 0.76604444311897803520, 0.59715859170278616485, 0.39607976603915682370, 0.17364817766693034885, -0.058144828910475828539, -0.28680323271109025310, -0.50000000000000000000, -0.68624163786873358573, -0.83548781141293641965, -0.93969262078590838405, -0.99323835774194298855, -0.99323835774194298855, -0.93969262078590838405, -0.83548781141293641965, -0.68624163786873358573, -0.50000000000000000000, -0.28680323271109025310, -0.058144828910475828539, 0.17364817766693034885, 0.39607976603915682370, 0.59715859170278616485, 0.76604444311897803520, 0.89363264032341224819, 0.97304487057982383883};
  static constexpr double s[27] = {0.0, 0.23061587074244017845, 0.44879918020046217278, 0.64278760968653932632, 0.80212319275504378508, 0.91821610688027401476, 0.98480775301220805937, 0.99830815827126820805, 0.95798951231548887444, 0.86602540378443864676, 0.72737364157304869599, 0.54950897807080603526, 0.34202014332566873304, 0.11609291412523022968, -0.11609291412523022968, -0.34202014332566873304, -0.54950897807080603526, -0.72737364157304869599, -0.86602540378443864676, -0.95798951231548887444, -0.99830815827126820805, -0.98480775301220805937, -0.91821610688027401476, -0.80212319275504378508, -0.64278760968653932632, -0.44879918020046217278, -0.23061587074244017845};
};

// v exp(-2 pi i M / N) (INV: conjugate), M a constant
template <int N, int M, bool INV, class C>
__device__ __forceinline__ C rotate(C v)
{
  using T = typename Real<C>::T;
  constexpr int m = M % N;
  if constexpr (m == 0) {
    return v;
  } else if constexpr (4 * m == N) {
    return INV ? C{-v.y, v.x} : C{v.y, -v.x};
  } else {
    constexpr double cd = Circle<N>::c[m], sd = Circle<N>::s[m];
    constexpr T c = (T)cd, s = (T)(INV ? sd : -sd);
    return C{v.x * c - v.y * s, v.x * s + v.y * c};
  }
}

constexpr int inv_mod(int a, int m)
{
  for (int x = 1; x < m; x++)
    if (a * x % m == 1) return x;
  return 1;
}

template <int R, bool INV, class C>
__device__ __forceinline__ void run(C *v);

// coprime factors A and B
template <int A, int B, bool INV, class C>
__device__ __forceinline__ void prime_factor(C *v)
{
  constexpr int N = A * B;
  C t[N];
  static_for<B>([&](auto b) {
    C u[A];
    static_for<A>([&](auto a) { u[a] = v[(B * a + A * b) % N]; });
    run<A, INV, C>(u);
    static_for<A>([&](auto a) { t[a * B + b] = u[a]; });
  });
  static_for<A>([&](auto k1) {
    run<B, INV, C>(t + k1 * B);
    static_for<B>([&](auto k2) {
      constexpr int k = (k1 * B * inv_mod(B % A, A) + k2 * A * inv_mod(A % B, B)) % N;
      v[k] = t[k1 * B + k2];
    });
  });
}

// A-point transforms over a of inputs a B + b, twiddles, B-point transforms over b
template <int A, int B, bool INV, class C>
__device__ __forceinline__ void cooley_tukey(C *v)
{
  constexpr int N = A * B;
  C t[N];
  static_for<B>([&](auto b) {
    C u[A];
    static_for<A>([&](auto a) { u[a] = v[a * B + b]; });
    run<A, INV, C>(u);
    static_for<A>([&](auto k1) {
      constexpr int m = k1 * b;
      t[k1 * B + b] = rotate<N, m, INV, C>(u[k1]);
    });
  });
  static_for<A>([&](auto k1) {
    run<B, INV, C>(t + k1 * B);
    static_for<B>([&](auto k2) { v[k1 + A * k2] = t[k1 * B + k2]; });
  });
}

// R-point DFT of v in place, natural order (forward: exp(-2 pi i r k / R); INV: conjugate)
template <int R, bool INV, class C>
__device__ __forceinline__ void run(C *v)
{
  using T = typename Real<C>::T;
  if constexpr (R == 2) {
    const C a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (R == 3) {
    // y1,2 = v0 - (v1 + v2)/2 -/+ i (sqrt 3 / 2)(v1 - v2)
    const T s3 = (T)0.86602540378443864676;
    const C a = cadd(v[1], v[2]), b = csub(v[1], v[2]);
    const C m = C{v[0].x - (T)0.5 * a.x, v[0].y - (T)0.5 * a.y};
    const C s = C{s3 * b.x, s3 * b.y};
    v[0] = cadd(v[0], a);
    v[1] = add_mi<INV, C>(m, s);
    v[2] = sub_mi<INV, C>(m, s);
  } else if constexpr (R == 4) {
    const C y0 = cadd(v[0], v[2]), y1 = csub(v[0], v[2]), y2 = cadd(v[1], v[3]), y3 = csub(v[1], v[3]);
    v[0] = cadd(y0, y2);
    v[2] = csub(y0, y2);
    v[1] = add_mi<INV, C>(y1, y3);
    v[3] = sub_mi<INV, C>(y1, y3);
  } else if constexpr (R == 5) {
    // with a1 = v1 + v4, b1 = v1 - v4, a2 = v2 + v3, b2 = v2 - v3,
    // y1,4 = v0 + c1 a1 + c2 a2 -/+ i (s1 b1 + s2 b2),  y2,3 = v0 + c2 a1 + c1 a2 -/+ i (s2 b1 - s1 b2)
    const T c1 = (T)0.30901699437494742410, c2 = (T)-0.80901699437494742410;
    const T s1 = (T)0.95105651629515357212, s2 = (T)0.58778525229247312917;
    const C a1 = cadd(v[1], v[4]), b1 = csub(v[1], v[4]), a2 = cadd(v[2], v[3]), b2 = csub(v[2], v[3]);
    const C m1 = C{v[0].x + c1 * a1.x + c2 * a2.x, v[0].y + c1 * a1.y + c2 * a2.y};
    const C m2 = C{v[0].x + c2 * a1.x + c1 * a2.x, v[0].y + c2 * a1.y + c1 * a2.y};
    const C n1 = C{s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y};
    const C n2 = C{s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y};
    v[0] = C{v[0].x + a1.x + a2.x, v[0].y + a1.y + a2.y};
    v[1] = add_mi<INV, C>(m1, n1);
    v[4] = sub_mi<INV, C>(m1, n1);
    v[2] = add_mi<INV, C>(m2, n2);
    v[3] = sub_mi<INV, C>(m2, n2);
  } else if constexpr (R == 7) {
    // with a_k = v_k + v_7-k, b_k = v_k - v_7-k: y_k, y_7-k = v0 + sum_j cos(2 pi jk / 7) a_j -/+ i sum_j sin(2 pi jk / 7) b_j
    const T c1 = (T)0.62348980185873353053, c2 = (T)-0.22252093395631440429, c3 = (T)-0.90096886790241912624;
    const T s1 = (T)0.78183148246802980871, s2 = (T)0.97492791218182360702, s3 = (T)0.43388373911755812048;
    const C a1 = cadd(v[1], v[6]), a2 = cadd(v[2], v[5]), a3 = cadd(v[3], v[4]);
    const C b1 = csub(v[1], v[6]), b2 = csub(v[2], v[5]), b3 = csub(v[3], v[4]);
    const C m1 = C{v[0].x + c1 * a1.x + c2 * a2.x + c3 * a3.x, v[0].y + c1 * a1.y + c2 * a2.y + c3 * a3.y};
    const C m2 = C{v[0].x + c2 * a1.x + c3 * a2.x + c1 * a3.x, v[0].y + c2 * a1.y + c3 * a2.y + c1 * a3.y};
    const C m3 = C{v[0].x + c3 * a1.x + c1 * a2.x + c2 * a3.x, v[0].y + c3 * a1.y + c1 * a2.y + c2 * a3.y};
    const C n1 = C{s1 * b1.x + s2 * b2.x + s3 * b3.x, s1 * b1.y + s2 * b2.y + s3 * b3.y};
    const C n2 = C{s2 * b1.x - s3 * b2.x - s1 * b3.x, s2 * b1.y - s3 * b2.y - s1 * b3.y};
    const C n3 = C{s3 * b1.x - s1 * b2.x + s2 * b3.x, s3 * b1.y - s1 * b2.y + s2 * b3.y};
    v[0] = C{v[0].x + a1.x + a2.x + a3.x, v[0].y + a1.y + a2.y + a3.y};
    v[1] = add_mi<INV, C>(m1, n1);
    v[6] = sub_mi<INV, C>(m1, n1);
    v[2] = add_mi<INV, C>(m2, n2);
    v[5] = sub_mi<INV, C>(m2, n2);
    v[3] = add_mi<INV, C>(m3, n3);
    v[4] = sub_mi<INV, C>(m3, n3);
  } else if constexpr (R == 8) {
    C e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    run<4, INV, C>(e);
    run<4, INV, C>(o);
    const T h = (T)0.70710678118654752440;
    // o1 turned by an eighth: h (x + y, y - x); o3 by three: h (y - x, -(x + y)) (INV: conjugate)
    const C p = INV ? C{o[1].x - o[1].y, o[1].y + o[1].x} : C{o[1].x + o[1].y, o[1].y - o[1].x};
    const C q = INV ? C{-o[3].x - o[3].y, o[3].x - o[3].y} : C{o[3].y - o[3].x, -o[3].x - o[3].y};
    v[0] = cadd(e[0], o[0]);
    v[4] = csub(e[0], o[0]);
    v[1] = C{e[1].x + h * p.x, e[1].y + h * p.y};
    v[5] = C{e[1].x - h * p.x, e[1].y - h * p.y};
    v[2] = add_mi<INV, C>(e[2], o[2]);
    v[6] = sub_mi<INV, C>(e[2], o[2]);
    v[3] = C{e[3].x + h * q.x, e[3].y + h * q.y};
    v[7] = C{e[3].x - h * q.x, e[3].y - h * q.y};
  } else if constexpr (R == 6) {
    prime_factor<3, 2, INV, C>(v);
  } else if constexpr (R == 10) {
    prime_factor<5, 2, INV, C>(v);
  } else if constexpr (R == 12) {
    prime_factor<4, 3, INV, C>(v);
  } else if constexpr (R == 14) {
    prime_factor<7, 2, INV, C>(v);
  } else if constexpr (R == 21) {
    prime_factor<7, 3, INV, C>(v);
  } else if constexpr (R == 15) {
    prime_factor<5, 3, INV, C>(v);
  } else if constexpr (R == 18) {
    prime_factor<9, 2, INV, C>(v);
  } else if constexpr (R == 20) {
    prime_factor<5, 4, INV, C>(v);
  } else if constexpr (R == 24) {
    prime_factor<8, 3, INV, C>(v);
  } else if constexpr (R == 9) {
    cooley_tukey<3, 3, INV, C>(v);
  } else if constexpr (R == 16) {
    cooley_tukey<4, 4, INV, C>(v);
  } else if constexpr (R == 25) {
    cooley_tukey<5, 5, INV, C>(v);
  } else if constexpr (R == 27) {
    cooley_tukey<3, 9, INV, C>(v);
  } else {
    static_assert(R == 1, "no DFT of this length");
  }
}

}  // namespace dft
}  // namespace tgpu
