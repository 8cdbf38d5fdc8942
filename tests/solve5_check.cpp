// Host check of the refined 5x5 solve (csrc/local_solve.cuh): random systems
// K + sum w m m^T as the local solve assembles them, over the declared range
// of condition numbers, against the same FP32 system solved in long double.
// Prints per decade of the condition number's driver: systems, accepted, the
// largest and mean error of the refined solve and of an FP64 solve rounded
// to FP32, each in units of 2^-24 |x|.
#include <cstdio>
#include <cstdlib>
#include <random>
#include "mth_common.cuh"
#include "local_solve.cuh"

template <typename T>
static void dense_solve(const float* H, const float* b, T* x) {
  T a[5][6];
  for (int i = 0; i < 5; i++) {
    for (int j = 0; j < 5; j++) a[i][j] = (T)H[mth::pk5s(i, j)];
    a[i][5] = (T)b[i];
  }
  for (int c = 0; c < 5; c++)
    for (int r = c + 1; r < 5; r++) {
      const T f = a[r][c] / a[c][c];
      for (int j = c; j < 6; j++) a[r][j] -= f * a[c][j];
    }
  for (int i = 4; i >= 0; i--) {
    T s = a[i][5];
    for (int j = i + 1; j < 5; j++) s -= a[i][j] * x[j];
    x[i] = s / a[i][i];
  }
}

static double error_of(const float* x, const long double* e) {
  long double d = 0, n = 0;
  for (int i = 0; i < 5; i++) {
    d += (x[i] - e[i]) * (x[i] - e[i]);
    n += e[i] * e[i];
  }
  return (double)(sqrtl(d) / sqrtl(n) * 16777216.0L);
}

int main(int argc, char** argv) {
  const int n = argc > 1 ? atoi(argv[1]) : 20000;
  std::mt19937_64 g(7);
  std::normal_distribution<double> nd;
  std::uniform_real_distribution<double> ud(0.0, 1.0);
  for (int dec = -6; dec <= 3; dec++) {
    int taken = 0;
    double worst = 0, sum = 0, worst64 = 0, sum64 = 0;
    for (int k = 0; k < n; k++) {
      // elastic base: eigenvalues between 1/150000 and 1/40000 in random axes
      float H[15] = {0}, b[5];
      double M[5][5] = {{0}};
      for (int e = 0; e < 5; e++) {
        double v[5], s = 0;
        for (double& t : v) { t = nd(g); s += t * t; }
        const double lam = 7e-6 + 1.8e-5 * ud(g);
        for (int i = 0; i < 5; i++)
          for (int j = 0; j < 5; j++) M[i][j] += lam * v[i] * v[j] / s + (i == j ? 2e-6 : 0.0);
      }
      // slip systems, slopes spread over three decades below dt w = 10^dec
      for (int s = 0; s < 12; s++) {
        double v[5], q = 0;
        for (double& t : v) { t = nd(g); q += t * t; }
        const double w = pow(10.0, dec - 3.0 * ud(g)) * 0.5 / q;
        for (int i = 0; i < 5; i++)
          for (int j = 0; j < 5; j++) M[i][j] += w * v[i] * v[j];
      }
      for (int i = 0; i < 5; i++) {
        for (int j = i; j < 5; j++) H[mth::pk5u(i, j)] = (float)M[i][j];
        b[i] = (float)(1e-4 * nd(g));
      }
      long double e[5];
      double d[5];
      dense_solve<long double>(H, b, e);
      dense_solve<double>(H, b, d);
      mth::Ldl5 f;
      float x[5], x64[5];
      if (!mth::ldl5_factor(H, f) || !mth::solve5_refined(f, H, b, x)) continue;
      for (int i = 0; i < 5; i++) x64[i] = (float)d[i];
      taken++;
      const double er = error_of(x, e), e64 = error_of(x64, e);
      worst = er > worst ? er : worst;
      worst64 = e64 > worst64 ? e64 : worst64;
      sum += er;
      sum64 += e64;
    }
    printf("%d %d %d %.6f %.6f %.6f %.6f\n", dec, n, taken, worst, sum / (taken ? taken : 1), worst64,
           sum64 / (taken ? taken : 1));
  }
  return 0;
}
