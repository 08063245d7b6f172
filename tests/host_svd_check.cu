// Host entry point of the FP64 SVD (elem_math.cuh) for test_host_svd.py: out = U[9], s[3], V[9], row-major.
#include "../ssim_gb300/csrc/elem_math.cuh"

extern "C" void svd64(const double* F, double* out) { ssim_gb::svd3<double>(F, out, out + 9, out + 12); }
