// Forward DFTs of a few points in registers, FP32 (float2) and FP64 (double2): v[k'] = sum_k v[k]
// exp(-2 pi i k k' / R).  Composite sizes of coprime factors take the Good-Thomas map (no twiddles),
// the others Cooley-Tukey with constant ones.
#pragma once

#include <cuda_runtime.h>

namespace mpsq {

__device__ __forceinline__ float2 operator+(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 operator-(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 operator-(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cpx(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ double2 cpx(double x, double y) { return make_double2(x, y); }
template <class V>
using Real = decltype(V::x);
template <class V>
__device__ __forceinline__ V rot(V a, Real<V> c, Real<V> s) {   // a (c - i s)
  return cpx(fma(a.x, c, a.y * s), fma(a.y, c, -a.x * s));
}

// Forward DFT of R points in place.
template <class V, int R>
struct Dft;
template <class V>
struct Dft<V, 2> {
  static __device__ __forceinline__ void run(V* v) {
    const V a = v[0];
    v[0] = a + v[1];
    v[1] = a - v[1];
  }
};
template <class V>
struct Dft<V, 3> {
  static __device__ __forceinline__ void run(V* v) {
    constexpr Real<V> s = 0.86602540378443864676;      // sin(2 pi / 3)
    const V t = v[1] + v[2], d = v[1] - v[2];
    const V m = cpx(fma((Real<V>)-0.5, t.x, v[0].x), fma((Real<V>)-0.5, t.y, v[0].y));
    v[0] = v[0] + t;
    v[1] = cpx(fma(s, d.y, m.x), fma(-s, d.x, m.y));
    v[2] = cpx(fma(-s, d.y, m.x), fma(s, d.x, m.y));
  }
};
template <class V>
struct Dft<V, 4> {
  static __device__ __forceinline__ void run(V* v) {
    const V a = v[0] + v[2], b = v[0] - v[2], c = v[1] + v[3], d = v[1] - v[3];
    v[0] = a + c;
    v[2] = a - c;
    v[1] = cpx(b.x + d.y, b.y - d.x);        // b - i d
    v[3] = cpx(b.x - d.y, b.y + d.x);
  }
};
template <class V>
struct Dft<V, 5> {
  static __device__ __forceinline__ void run(V* v) {
    constexpr Real<V> c1 = 0.30901699437494742410, s1 = 0.95105651629515357212;    // 2 pi / 5
    constexpr Real<V> c2 = -0.80901699437494742410, s2 = 0.58778525229247312917;   // 4 pi / 5
    const V t1 = v[1] + v[4], t2 = v[2] + v[3], d1 = v[1] - v[4], d2 = v[2] - v[3], v0 = v[0];
    v[0] = v0 + (t1 + t2);
    const V a = cpx(fma(c2, t2.x, fma(c1, t1.x, v0.x)), fma(c2, t2.y, fma(c1, t1.y, v0.y)));
    const V b = cpx(fma(c1, t2.x, fma(c2, t1.x, v0.x)), fma(c1, t2.y, fma(c2, t1.y, v0.y)));
    const V p = cpx(fma(s2, d2.x, s1 * d1.x), fma(s2, d2.y, s1 * d1.y));
    const V q = cpx(fma(-s1, d2.x, s2 * d1.x), fma(-s1, d2.y, s2 * d1.y));
    v[1] = cpx(a.x + p.y, a.y - p.x);        // a - i p
    v[4] = cpx(a.x - p.y, a.y + p.x);
    v[2] = cpx(b.x + q.y, b.y - q.x);
    v[3] = cpx(b.x - q.y, b.y + q.x);
  }
};
template <class V>
struct Dft<V, 8> {
  static __device__ __forceinline__ void run(V* v) {
    constexpr Real<V> r = 0.70710678118654752440;
    V e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    Dft<V, 4>::run(e);
    Dft<V, 4>::run(o);
    v[0] = e[0] + o[0];
    v[4] = e[0] - o[0];
    const V t1 = cpx(o[1].x + o[1].y, o[1].y - o[1].x);        // w8 o1 / r
    v[1] = cpx(fma(r, t1.x, e[1].x), fma(r, t1.y, e[1].y));
    v[5] = cpx(fma(-r, t1.x, e[1].x), fma(-r, t1.y, e[1].y));
    v[2] = cpx(e[2].x + o[2].y, e[2].y - o[2].x);
    v[6] = cpx(e[2].x - o[2].y, e[2].y + o[2].x);
    const V t3 = cpx(o[3].y - o[3].x, -(o[3].x + o[3].y));     // w8^3 o3 / r
    v[3] = cpx(fma(r, t3.x, e[3].x), fma(r, t3.y, e[3].y));
    v[7] = cpx(fma(-r, t3.x, e[3].x), fma(-r, t3.y, e[3].y));
  }
};
// Cooley-Tukey A x B: n = B n1 + n2, k = k1 + A k2, twiddles W_R^(n2 k1).
template <class V>
struct Dft<V, 9> {
  static __device__ __forceinline__ void run(V* v) {
    constexpr Real<V> c[5] = {1.0, 0.76604444311897803520, 0.17364817766693034885, -0.5, -0.93969262078590838405};
    constexpr Real<V> s[5] = {0.0, 0.64278760968653932632, 0.98480775301220805937, 0.86602540378443864676, 0.34202014332566873304};
    V y[3][3];
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) {
      V a[3] = {v[n2], v[3 + n2], v[6 + n2]};
      Dft<V, 3>::run(a);
#pragma unroll
      for (int k1 = 0; k1 < 3; ++k1) y[n2][k1] = n2 * k1 ? rot(a[k1], c[n2 * k1], s[n2 * k1]) : a[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
      V b[3] = {y[0][k1], y[1][k1], y[2][k1]};
      Dft<V, 3>::run(b);
#pragma unroll
      for (int k2 = 0; k2 < 3; ++k2) v[k1 + 3 * k2] = b[k2];
    }
  }
};
template <class V>
struct Dft<V, 16> {
  static __device__ __forceinline__ void run(V* v) {
    constexpr Real<V> r = 0.70710678118654752440, c1 = 0.92387953251128675613, s1 = 0.38268343236508977173;
    constexpr Real<V> c[10] = {1.0, c1, r, s1, 0.0, -s1, -r, -c1, -1.0, -c1};   // cos, sin of 2 pi m / 16
    constexpr Real<V> s[10] = {0.0, s1, r, c1, 1.0, c1, r, s1, 0.0, -s1};
    V y[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
      V a[4] = {v[n2], v[4 + n2], v[8 + n2], v[12 + n2]};
      Dft<V, 4>::run(a);
#pragma unroll
      for (int k1 = 0; k1 < 4; ++k1) {
        const int m = n2 * k1;
        y[n2][k1] = m == 0 ? a[k1] : m == 4 ? cpx(a[k1].y, -a[k1].x) : rot(a[k1], c[m], s[m]);
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      V b[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
      Dft<V, 4>::run(b);
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) v[k1 + 4 * k2] = b[k2];
    }
  }
};
// Good-Thomas A x B, coprime: n = B n1 + A n2 (mod R) and k = k1 B (B^-1 mod A) + k2 A (A^-1 mod B)
// (mod R) separate exactly, without twiddles.
__host__ __device__ constexpr int inverse_mod(int a, int m) {
  for (int x = 1; x < m; ++x)
    if (a * x % m == 1) return x;
  return 0;
}
template <class V, int A, int B>
struct DftCoprime {
  static __device__ __forceinline__ void run(V* v) {
    constexpr int R = A * B, ia = B * inverse_mod(B % A, A), ib = A * inverse_mod(A % B, B);
    V y[B][A];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) y[n2][n1] = v[(B * n1 + A * n2) % R];
      Dft<V, A>::run(y[n2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      V b[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) b[n2] = y[n2][k1];
      Dft<V, B>::run(b);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[(k1 * ia + k2 * ib) % R] = b[k2];
    }
  }
};
template <class V> struct Dft<V, 6> : DftCoprime<V, 2, 3> {};
template <class V> struct Dft<V, 10> : DftCoprime<V, 2, 5> {};
template <class V> struct Dft<V, 12> : DftCoprime<V, 4, 3> {};
template <class V> struct Dft<V, 15> : DftCoprime<V, 3, 5> {};
template <class V> struct Dft<V, 18> : DftCoprime<V, 2, 9> {};
template <class V> struct Dft<V, 20> : DftCoprime<V, 4, 5> {};
template <class V> struct Dft<V, 24> : DftCoprime<V, 8, 3> {};

// 32 = 4 x 8: n = 4 n1 + n2, k = k1 + 8 k2, twiddles W_32^(n2 k1).
template <class V>
struct Dft<V, 32> {
  static __device__ __forceinline__ void run(V* v) {
    constexpr Real<V> c[22] = {1.0, 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708,
                               0.70710678118654752440, 0.55557023301960222474, 0.38268343236508977173,
                               0.19509032201612826785, 0.0, -0.19509032201612826785, -0.38268343236508977173,
                               -0.55557023301960222474, -0.70710678118654752440, -0.83146961230254523708,
                               -0.92387953251128675613, -0.98078528040323044913, -1.0, -0.98078528040323044913,
                               -0.92387953251128675613, -0.83146961230254523708, -0.70710678118654752440,
                               -0.55557023301960222474};
    constexpr Real<V> s[22] = {0.0, 0.19509032201612826785, 0.38268343236508977173, 0.55557023301960222474,
                               0.70710678118654752440, 0.83146961230254523708, 0.92387953251128675613,
                               0.98078528040323044913, 1.0, 0.98078528040323044913, 0.92387953251128675613,
                               0.83146961230254523708, 0.70710678118654752440, 0.55557023301960222474,
                               0.38268343236508977173, 0.19509032201612826785, 0.0, -0.19509032201612826785,
                               -0.38268343236508977173, -0.55557023301960222474, -0.70710678118654752440,
                               -0.83146961230254523708};
    V y[4][8];
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < 8; ++n1) y[n2][n1] = v[4 * n1 + n2];
      Dft<V, 8>::run(y[n2]);
#pragma unroll
      for (int k1 = 1; k1 < 8; ++k1) {
        const int m = n2 * k1;
        if (m == 8) y[n2][k1] = cpx(y[n2][k1].y, -y[n2][k1].x);
        else if (m) y[n2][k1] = rot(y[n2][k1], c[m], s[m]);
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < 8; ++k1) {
      V b[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
      Dft<V, 4>::run(b);
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) v[k1 + 8 * k2] = b[k2];
    }
  }
};

}  // namespace mpsq
