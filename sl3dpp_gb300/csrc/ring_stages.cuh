// The butterflies of the ring transforms in a generic real type: FP32 (the
// mixed form's rings) and FP64 (small batches, both in sht.cu), double-float
// (ring_df.cu).
#pragma once

#include <cuda_runtime.h>

namespace sl3dgpu {

template <class T2>
struct Real;
template <>
struct Real<double2> {
  using type = double;
};
template <>
struct Real<float2> {
  using type = float;
};

template <class T2>
__device__ inline T2 Make(typename Real<T2>::type x, typename Real<T2>::type y) {
  T2 v;
  v.x = x;
  v.y = y;
  return v;
}
template <class T2>
__device__ inline T2 Mul(T2 a, T2 b) {
  return Make<T2>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <class T2>
__device__ inline T2 Add(T2 a, T2 b) {
  return Make<T2>(a.x + b.x, a.y + b.y);
}
template <class T2>
__device__ inline T2 Sub(T2 a, T2 b) {
  return Make<T2>(a.x - b.x, a.y - b.y);
}

// The DFT of R values in registers, y_u = sum_q v_q e^{sign 2 pi i q u / R},
// for the radices of the plans (2, 3, 4, 5), with the roots as constants.
template <class T2, int R>
__device__ inline void Butterfly(T2 (&v)[R], int sign) {
  using T = typename Real<T2>::type;
  auto I = [](T2 a) { return Make<T2>(-a.y, a.x); };  // i a
  auto S = [](T k, T2 a) { return Make<T2>(k * a.x, k * a.y); };
  const T sg = sign > 0 ? T(1) : T(-1);
  if constexpr (R == 2) {
    const T2 a = v[0], b = v[1];
    v[0] = Add(a, b);
    v[1] = Sub(a, b);
  } else if constexpr (R == 3) {
    const T2 t = Add(v[1], v[2]);
    const T2 d = S(sg * T(0.86602540378443864676), Sub(v[1], v[2]));
    const T2 a = Sub(v[0], S(T(0.5), t));
    v[0] = Add(v[0], t);
    v[1] = Add(a, I(d));
    v[2] = Sub(a, I(d));
  } else if constexpr (R == 4) {
    const T2 a0 = Add(v[0], v[2]), a1 = Sub(v[0], v[2]);
    const T2 b0 = Add(v[1], v[3]), b1 = S(sg, Sub(v[1], v[3]));
    v[0] = Add(a0, b0);
    v[1] = Add(a1, I(b1));
    v[2] = Sub(a0, b0);
    v[3] = Sub(a1, I(b1));
  } else {
    static_assert(R == 5, "radix");
    const T c1 = T(0.30901699437494742410), c2 = T(-0.80901699437494742410);
    const T s1 = T(0.95105651629515357212), s2 = T(0.58778525229247312917);
    const T2 t1 = Add(v[1], v[4]), t2 = Add(v[2], v[3]);
    const T2 d1 = Sub(v[1], v[4]), d2 = Sub(v[2], v[3]);
    const T2 a1 = Add(v[0], Add(S(c1, t1), S(c2, t2)));
    const T2 a2 = Add(v[0], Add(S(c2, t1), S(c1, t2)));
    const T2 b1 = S(sg, Add(S(s1, d1), S(s2, d2)));
    const T2 b2 = S(sg, Sub(S(s2, d1), S(s1, d2)));
    v[0] = Add(v[0], Add(t1, t2));
    v[1] = Add(a1, I(b1));
    v[4] = Sub(a1, I(b1));
    v[2] = Add(a2, I(b2));
    v[3] = Sub(a2, I(b2));
  }
}

}  // namespace sl3dgpu
