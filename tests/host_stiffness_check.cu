// Host entry points of the element stiffness (elem_math.cuh) for test_host_stiffness.py: K[144] row-major.
#include "../ssim_gb300/csrc/elem_math.cuh"

template <typename S>
static void run(const double* F, const double* D, double lam, double mu, int spsd, double scale, double* K) {
  S f[9], d[4][3], k[78];
  for (int i = 0; i < 9; ++i) f[i] = (S)F[i];
  for (int v = 0; v < 4; ++v)
    for (int j = 0; j < 3; ++j) d[v][j] = (S)D[3 * v + j];
  ssim_gb::element_stiffness<S>(f, d, (S)lam, (S)mu, spsd != 0, (S)scale, k);
  for (int i = 0; i < 12; ++i)
    for (int j = 0; j < 12; ++j) K[12 * i + j] = (double)(i <= j ? k[ssim_gb::kup(i, j)] : k[ssim_gb::kup(j, i)]);
}

extern "C" void stiffness64(const double* F, const double* D, double lam, double mu, int spsd, double scale, double* K) {
  run<double>(F, D, lam, mu, spsd, scale, K);
}
extern "C" void stiffness32(const double* F, const double* D, double lam, double mu, int spsd, double scale, double* K) {
  run<float>(F, D, lam, mu, spsd, scale, K);
}
