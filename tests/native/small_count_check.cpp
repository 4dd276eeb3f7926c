// Checks div_by_small_count against the plain IEEE division on the host, for
// every count it takes: random operands over its range, sums of few-bit
// values (exact quotients and ties), mantissas next to a binade's ends, zero;
// and small_count_operand at the edges of the range it admits.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <limits>
#include <random>

#include "count_div.cuh"

using dense_b200::CountDivTraits;
using dense_b200::div_by_small_count;
using dense_b200::kSmallCount;
using dense_b200::small_count_operand;

template <typename T>
long check(T x, long& bad) {
  if (!small_count_operand(x)) return 0;
  for (int c = 1; c <= kSmallCount; ++c) {
    const T got = div_by_small_count(x, T(c), T(1) / T(c)), want = x / T(c);
    if (CountDivTraits<T>::bits(got) != CountDivTraits<T>::bits(want)) {
      if (bad++ < 5) std::printf("x=%a c=%d got %a want %a\n", double(x), c, double(got), double(want));
    }
  }
  return 1;
}

template <typename T>
int run(const char* name, int seed) {
  using Tr = CountDivTraits<T>;
  using Bits = typename Tr::Bits;
  std::mt19937_64 g(seed);
  long n = 0, bad = 0;
  for (int i = 0; i < 3000000; ++i) {
    n += check(Tr::from(static_cast<Bits>(g())), bad);             // any bit pattern
    n += check(T(std::ldexp(double(g() % 4096), int(g() % 40) - 20)), bad);  // few bits
    const Bits mant = g() % 64, one = Bits(1) << Tr::kMant;        // next to a binade's ends
    const Bits expo = Tr::bits(T(1)) + (Bits(g() % 60) << Tr::kMant) - (Bits(30) << Tr::kMant);
    n += check(Tr::from(expo + mant), bad);
    n += check(Tr::from(expo + one - 1 - mant), bad);
  }
  n += check(T(0), bad);
  const T inf = std::numeric_limits<T>::infinity();
  bad += !small_count_operand(T(0)) + !small_count_operand(Tr::kLo) + !small_count_operand(-Tr::kLo);
  bad += small_count_operand(std::nextafter(Tr::kHi, inf)) + small_count_operand(inf) +
         small_count_operand(std::numeric_limits<T>::quiet_NaN()) + small_count_operand(std::nextafter(Tr::kLo, T(0))) +
         small_count_operand(std::numeric_limits<T>::denorm_min());
  std::printf("%s: %ld operands, %ld wrong\n", name, n, bad);
  return bad != 0 || n < 1000000;
}

int main() { return run<double>("double", 1) | run<float>("float", 2); }
