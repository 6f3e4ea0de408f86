// Host check, built with the signed-overflow sanitizer, of the natural-word
// engine and of what the exact slices make of its twiddles:
//   exact_tw_sum      on every entry of every span, against the sum in 128 bits
//   every fixed-point plan of N >= 64 that the library compiles, at the largest
//   input scale (natural_check.cu's check_plan)
// and natural_check.cu's own cases.  Prints "name value" lines; an overflow ends
// the program.
#define main natural_check_main
#include "natural_check.cu"
#undef main

#include <array>
#include <set>

#include "fft_exact.cuh"
#include "internal.h"
#include "plans.inc"

namespace {
std::set<std::array<int, 4>> g_plans;
struct Collect {
  template <class E, class PL>
  static void plain(SizeVariants&) {
    if (PL::N >= kNaturalMinN) g_plans.insert({PL::R[0], PL::R[1], PL::R[2], PL::R[3]});
  }
  template <class E, class PL, int NSTAGE>
  static void persistent(SizeVariants& sv) { plain<E, PL>(sv); }
};

// entries for which the sum's limbs are not -(wr + wi)
long long check_tw_sum() {
  constexpr ld PI2 = 2.0L * 3.141592653589793238462643383279502884L, ONE = 4611686018427387904.0L;  // 2^62
  long long bad = 0;
  for (int n = 16; n <= 4096; n *= 2)
    for (int k = 0; k < n; ++k) {
      const long long r = llroundl(cosl(PI2 * k / n) * ONE), d = llroundl((-sinl(PI2 * k / n) - cosl(PI2 * k / n)) * ONE);
      int4 w;
      w.y = (int)(unsigned)r;
      w.x = (int)((r - w.y) >> 32);
      w.w = (int)(unsigned)d;
      w.z = (int)((d - w.w) >> 32);
      const int2 c = exact_tw_sum(w);
      if ((__int128)c.x * ((__int128)1 << 32) + c.y != -((__int128)2 * r + d)) ++bad;
    }
  return bad;
}
}  // namespace

int main() {
  printf("tw_sum_bad %lld\n", check_tw_sum());
  static SizeVariants sv[kNumSizes];
  describe_all<EngFx, Collect>(sv);
  std::mt19937_64 g(7);
  double worst = 0;
  for (const auto& r : g_plans) {
    int s = 0;
    while (s < 4 && r[s] > 1) ++s;
    const double e = check_plan(g, r.data(), s);
    if (!(e <= worst)) worst = e;
  }
  printf("plans %zu\n", g_plans.size());
  printf("compiled_plans_rel %.3e\n", worst);
  return natural_check_main();
}
