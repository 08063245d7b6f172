// log_rcp.cuh -- log(x) and 1/x of a positive double in 16 FP64 operations, for the stable Neo-Hookean energy.
//
// GB300's FP64 units take a warp's operation every 64 cycles, so the energy pass counts them; log() and a division took
// about 35.  The logarithm is table-driven (P. T. P. Tang, "Table-driven implementation of the logarithm function in IEEE
// floating-point arithmetic", ACM TOMS 16(4), 1990): x = 2^k m with m in [1, 2), r = m / c - 1 for the table's c nearest
// to m (|r| <= 2^-7; one rounding, by fma), log x = k ln 2 + log c + log1p(r) with the Taylor polynomial of degree 8
// (the next term is below 2^-66).  The reciprocal shares r: 1 / x = 2^-k (1 / c) (1 - r)(1 + r^2)(1 + r^4), off by r^8
// (2^-56).  Tested against the host's long double on the range the energy uses.
#pragma once
#include <cuda_runtime.h>
#include <string.h>

namespace ssim_gb {

struct LogEntry {
  double rc, lc;  // 1 / c rounded, and -log of that double
};

#define SSIM_LOG_ENTRIES \
    {0x1.fc07f01fc07f0p-1, 0x1.fe02a6b106799p-8}, {0x1.f44659e4a4271p-1, 0x1.7b91b07d5b126p-6}, \
    {0x1.ecc07b301ecc0p-1, 0x1.39e87b9febd68p-5}, {0x1.e573ac901e574p-1, 0x1.b42dd711971b9p-5}, \
    {0x1.de5d6e3f8868ap-1, 0x1.16536eea37ae3p-4}, {0x1.d77b654b82c34p-1, 0x1.51b073f06183cp-4}, \
    {0x1.d0cb58f6ec074p-1, 0x1.8c345d6319b23p-4}, {0x1.ca4b3055ee191p-1, 0x1.c5e548f5bc743p-4}, \
    {0x1.c3f8f01c3f8f0p-1, 0x1.fec9131dbeabcp-4}, {0x1.bdd2b899406f7p-1, 0x1.1b72ad52f67a2p-3}, \
    {0x1.b7d6c3dda338bp-1, 0x1.371fc201e8f75p-3}, {0x1.b2036406c80d9p-1, 0x1.526e5e3a1b438p-3}, \
    {0x1.ac5701ac5701bp-1, 0x1.6d60fe719d21bp-3}, {0x1.a6d01a6d01a6dp-1, 0x1.87fa06520c911p-3}, \
    {0x1.a16d3f97a4b02p-1, 0x1.a23bc1fe2b561p-3}, {0x1.9c2d14ee4a102p-1, 0x1.bc286742d8cd4p-3}, \
    {0x1.970e4f80cb872p-1, 0x1.d5c216b4fbb94p-3}, {0x1.920fb49d0e229p-1, 0x1.ef0adcbdc5935p-3}, \
    {0x1.8d3018d3018d3p-1, 0x1.0402594b4d041p-2}, {0x1.886e5f0abb04ap-1, 0x1.1058bf9ae4ad4p-2}, \
    {0x1.83c977ab2beddp-1, 0x1.1c898c16999fbp-2}, {0x1.7f405fd017f40p-1, 0x1.2895a13de86a4p-2}, \
    {0x1.7ad2208e0ecc3p-1, 0x1.347dd9a987d56p-2}, {0x1.767dce434a9b1p-1, 0x1.404308686a7e4p-2}, \
    {0x1.724287f46debcp-1, 0x1.4be5f957778a1p-2}, {0x1.6e1f76b4337c7p-1, 0x1.5767717455a6cp-2}, \
    {0x1.6a13cd1537290p-1, 0x1.62c82f2b9c796p-2}, {0x1.661ec6a5122f9p-1, 0x1.6e08eaa2ba1e4p-2}, \
    {0x1.623fa77016240p-1, 0x1.792a55fdd47a1p-2}, {0x1.5e75bb8d015e7p-1, 0x1.842d1da1e8b18p-2}, \
    {0x1.5ac056b015ac0p-1, 0x1.8f11e873662c8p-2}, {0x1.571ed3c506b3ap-1, 0x1.99d958117e08ap-2}, \
    {0x1.5390948f40febp-1, 0x1.a484090e5bb09p-2}, {0x1.5015015015015p-1, 0x1.af1293247786bp-2}, \
    {0x1.4cab88725af6ep-1, 0x1.b9858969310fdp-2}, {0x1.49539e3b2d067p-1, 0x1.c3dd7a7cdad4dp-2}, \
    {0x1.460cbc7f5cf9ap-1, 0x1.ce1af0b85f3ecp-2}, {0x1.42d6625d51f87p-1, 0x1.d83e7258a2f3ep-2}, \
    {0x1.3fb013fb013fbp-1, 0x1.e24881a7c6c26p-2}, {0x1.3c995a47babe7p-1, 0x1.ec399d2468cc1p-2}, \
    {0x1.3991c2c187f63p-1, 0x1.f6123fa7028adp-2}, {0x1.3698df3de0748p-1, 0x1.ffd2e0857f497p-2}, \
    {0x1.33ae45b57bcb2p-1, 0x1.04bdf9da926d2p-1}, {0x1.30d190130d190p-1, 0x1.0986f4f573521p-1}, \
    {0x1.2e025c04b8097p-1, 0x1.0e44985d1cc8cp-1}, {0x1.2b404ad012b40p-1, 0x1.12f719593efbdp-1}, \
    {0x1.288b01288b013p-1, 0x1.179eabbd899a0p-1}, {0x1.25e22708092f1p-1, 0x1.1c3b81f713c25p-1}, \
    {0x1.23456789abcdfp-1, 0x1.20cdcd192ab6ep-1}, {0x1.20b470c67c0d9p-1, 0x1.2555bce98f7cap-1}, \
    {0x1.1e2ef3b3fb874p-1, 0x1.29d37fec2b08bp-1}, {0x1.1bb4a4046ed29p-1, 0x1.2e47436e40268p-1}, \
    {0x1.19453808ca29cp-1, 0x1.32b1339121d71p-1}, {0x1.16e0689427379p-1, 0x1.37117b54747b6p-1}, \
    {0x1.1485f0e0acd3bp-1, 0x1.3b68449fffc23p-1}, {0x1.12358e75d3033p-1, 0x1.3fb5b84d16f43p-1}, \
    {0x1.0fef010fef011p-1, 0x1.43f9fe2f9ce67p-1}, {0x1.0db20a88f4696p-1, 0x1.48353d1ea88dfp-1}, \
    {0x1.0b7e6ec259dc8p-1, 0x1.4c679afccee39p-1}, {0x1.0953f39010954p-1, 0x1.50913cc01686bp-1}, \
    {0x1.073260a47f7c6p-1, 0x1.54b2467999498p-1}, {0x1.05197f7d73404p-1, 0x1.58cadb5cd7989p-1}, \
    {0x1.03091b51f5e1ap-1, 0x1.5cdb1dc6c1765p-1}, {0x1.0101010101010p-1, 0x1.60e32f44788d9p-1}
static __device__ const LogEntry kLogTable[64] = {SSIM_LOG_ENTRIES};
[[maybe_unused]] static const LogEntry kLogTableHost[64] = {SSIM_LOG_ENTRIES};
#undef SSIM_LOG_ENTRIES

__host__ __device__ __forceinline__ long long double_bits(double x) {
#ifdef __CUDA_ARCH__
  return __double_as_longlong(x);
#else
  long long b;
  memcpy(&b, &x, sizeof b);
  return b;
#endif
}
__host__ __device__ __forceinline__ double bits_double(long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(b);
#else
  double x;
  memcpy(&x, &b, sizeof x);
  return x;
#endif
}

// rcp = 1 / x, returns log(x); x at least 1.  Not finite: the results are finite and meaningless (the energy's other terms
// are not finite then).
__host__ __device__ __forceinline__ double log_rcp(double x, double& rcp) {
  const long long xb = double_bits(x);
  const int k = (int)(xb >> 52) - 1023;
  const double m = bits_double((xb & 0x000fffffffffffffLL) | 0x3ff0000000000000LL);
#ifdef __CUDA_ARCH__
  const LogEntry t = kLogTable[(int)(xb >> 46) & 63];
#else
  const LogEntry t = kLogTableHost[(int)(xb >> 46) & 63];
#endif
  const double r = fma(m, t.rc, -1.0), r2 = r * r;
  double p = fma(r, -1.0 / 8, 1.0 / 7);
  p = fma(r, p, -1.0 / 6);
  p = fma(r, p, 1.0 / 5);
  p = fma(r, p, -1.0 / 4);
  p = fma(r, p, 1.0 / 3);
  p = fma(r, p, -0.5);
  const double l = fma(r2, p, r);
  // k as a double: 2^52 + 2^31 + k less 2^52 + 2^31
  const double kd = bits_double(0x4330000000000000LL | (long long)((unsigned int)k ^ 0x80000000u)) - 4503601774854144.0;
  const double q = (1.0 - r) * t.rc, r4 = r2 * r2, q2 = fma(q, r2, q);
  // (beyond 2^1000 a reciprocal of 2^-1000 stands for any smaller one: it is subtracted from 1)
  rcp = bits_double(double_bits(fma(q2, r4, q2)) - ((long long)(k < 1000 ? k : 1000) << 52));
  return fma(kd, 0.69314718055994530942, t.lc) + l;
}

}  // namespace ssim_gb
