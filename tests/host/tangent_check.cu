// Host check of the binary64 engine's twiddled butterflies: for radix R behind
// a span p and every k < p, the butterfly on the tangent-form table entries
// against the same sums in long double.  Prints, per radix, the largest error
// of an output over the norm of the inputs.
#include <cmath>
#include <cstdio>
#include <random>

#include "fft_core.cuh"

using namespace fftoc;

template <int R>
static double check(std::mt19937_64& g) {
  std::normal_distribution<double> nd(0.0, 1.0);
  constexpr long double PI2 = 2.0L * 3.141592653589793238462643383279502884L;
  double worst = 0;
  for (int p = 2; p * R <= 4096; p *= 2)
    for (int k = 0; k < p; ++k) {
      double re[R], im[R];
      long double xr[R], xi[R], norm = 0;
      for (int m = 0; m < R; ++m) {
        re[m] = nd(g);
        im[m] = nd(g);
        norm += (long double)re[m] * re[m] + (long double)im[m] * im[m];
        const long double c = cosl(PI2 * (k * m) / (R * p)), s = -sinl(PI2 * (k * m) / (R * p));
        xr[m] = re[m] * c - im[m] * s;
        xi[m] = re[m] * s + im[m] * c;
      }
      auto entry = [&](int m) {
        const long double c = cosl(PI2 * (k * m) / (R * p)), s = -sinl(PI2 * (k * m) / (R * p));
        if (m < R / 2) return make_double2((double)c, (double)s);
        return EngF64::tangent_turned(k * m, R * p) ? make_double2((double)s, (double)(-c / s))
                                                    : make_double2((double)c, (double)(s / c));
      };
      for (int m = 1; m < R / 2; ++m) EngF64::cmul(re[m], im[m], entry(m));
      for (int m = 0; m < R / 2; ++m)
        EngF64::twiddled_sum(re[m], im[m], re[m + R / 2], im[m + R / 2], entry(m + R / 2),
                             EngF64::tangent_turned(k * (m + R / 2), R * p));
      f64_finish<R, 0, 1, R>(re, im);
      for (int q = 0; q < R; ++q) {
        long double sr = 0, si = 0;
        for (int m = 0; m < R; ++m) {
          const long double c = cosl(PI2 * (m * q % R) / R), s = -sinl(PI2 * (m * q % R) / R);
          sr += xr[m] * c - xi[m] * s;
          si += xr[m] * s + xi[m] * c;
        }
        const double e = (double)(hypotl(sr - re[q], si - im[q]) / sqrtl(norm));
        if (e > worst) worst = e;
      }
    }
  return worst;
}

int main() {
  std::mt19937_64 g(1);
  printf("radix2 %.3e\n", check<2>(g));
  printf("radix4 %.3e\n", check<4>(g));
  printf("radix8 %.3e\n", check<8>(g));
  printf("radix16 %.3e\n", check<16>(g));
  return 0;
}
