// Compile-time cosine tables in constant memory: with the indices of an unrolled transform known to
// the compiler its multiply-adds take their factors as constant operands.
#pragma once

namespace ves3d {

// cos(2 pi k / N), k = 0..N-1, to rounding: the angle is brought into [0, pi/4] by integer
// arithmetic on k and the Taylor series summed from its smallest term.
template <int N>
struct CosTab {
  double v[N];
  static constexpr double series(double x, bool sine) {
    const double x2 = x * x;
    double s = 0.0;
    for (int i = 12; i >= 1; i--) {
      const double a = sine ? (2.0 * i) * (2.0 * i + 1.0) : (2.0 * i - 1.0) * (2.0 * i);
      s = -(x2 / a) * (1.0 + s);
    }
    return sine ? x + x * s : 1.0 + s;
  }
  constexpr CosTab() : v{} {
    for (int k = 0; k < N; k++) {
      int h = k <= N - k ? k : N - k;            // cos is even: h / N <= 1/2
      const bool neg = 4 * h > N;                // cos(pi - x) = -cos x
      const double two_pi = 6.283185307179586476925286766559;
      double num = neg ? N - 2.0 * h : 2.0 * h;  // angle = pi num / N, num / N <= 1/2
      double c = 0.0;
      if (4.0 * num <= N)
        c = series(0.5 * two_pi * num / N, false);
      else
        c = series(0.5 * two_pi * (0.5 * N - num) / N, true);
      v[k] = neg ? -c : c;
    }
  }
};

template <int N>
__constant__ const CosTab<N> c_cos = CosTab<N>();

}  // namespace ves3d
