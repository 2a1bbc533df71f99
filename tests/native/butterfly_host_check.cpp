// Rounding of the register butterflies of fft_core.cuh that are built from
// smaller ones, beside the symmetric DFT of the same size: prints per radix the
// relative error of forward + inverse on random data and the mean gain minus 1,
// for both.  Test infrastructure only.
#include <cmath>
#include <cstdio>
#include <random>

#include "fft_core.cuh"

using namespace odt;

template <template <int, bool> class F, int R>
void round_trip(double* err, double* gain) {
  std::mt19937 rg(R);
  std::normal_distribution<float> nd;
  double num = 0, den = 0, e = 0;
  for (int rep = 0; rep < 4000; ++rep) {
    float2 x[R], v[R];
    for (int i = 0; i < R; ++i) x[i] = v[i] = make_float2(nd(rg), nd(rg));
    F<R, false>::run(v, nullptr, R);
    F<R, true>::run(v, nullptr, R);
    for (int i = 0; i < R; ++i) {
      const double ux = (double)v[i].x / R, uy = (double)v[i].y / R;
      num += ux * x[i].x + uy * x[i].y;
      den += (double)x[i].x * x[i].x + (double)x[i].y * x[i].y;
      e += (ux - x[i].x) * (ux - x[i].x) + (uy - x[i].y) * (uy - x[i].y);
    }
  }
  *err = std::sqrt(e / den);
  *gain = num / den - 1;
}

template <int R>
void check() {
  double e0, g0, e1, g1;
  round_trip<Butterfly, R>(&e0, &g0);
  round_trip<OddButterfly, R>(&e1, &g1);
  std::printf("%d %.6e %.6e %.6e %.6e\n", R, e0, g0, e1, g1);
}

int main() {
  check<9>();
  check<15>();
  check<21>();
  check<25>();
  check<27>();
  return 0;
}
