// Host check of the constant twiddles' factored forms (tw_form in lf_fft.cuh): every W_32^k, float and double, both
// signs.  Prints the largest error of (f, f t) per type in units of the type's 2^-24 or 2^-53; exit status 1 if the
// float one exceeds the bound on the command line.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "../../cmblensing_b200/csrc/lf_fft.cuh"

using namespace lf;

template <typename T> double worst() {
  double w = 0.0;
  for (int k = 1; k < 16; ++k)
    for (int s = -1; s <= 1; s += 2) {
      const long double wr = cosl(M_PIl * k / 16), wi = s * sinl(M_PIl * k / 16);
      if (k == 8) continue;  // a rotation
      const TwForm<T> t = tw_form<T>((double)wr, (double)wi);
      const long double f = t.f, g = f * (long double)t.t;
      const long double er = (t.re ? f : g) - wr, ei = (t.re ? g : f) - wi;
      w = fmax(w, (double)sqrtl(er * er + ei * ei));
    }
  return w * (sizeof(T) == 4 ? 16777216.0 : 9007199254740992.0);
}

int main(int argc, char** argv) {
  const double bound = argc > 1 ? std::atof(argv[1]) : 0.4;
  const double w32 = worst<float>();
  std::printf("float %.3f\ndouble %.3f\n", w32, worst<double>());
  return w32 > bound;
}
