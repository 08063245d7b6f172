// Host entry point of log_rcp (log_rcp.cuh) for test_host_log.py.
#include "../ssim_gb300/csrc/log_rcp.cuh"
extern "C" void log_rcp_n(int n, const double* x, double* l, double* r) {
  for (int i = 0; i < n; ++i) l[i] = ssim_gb::log_rcp(x[i], r[i]);
}
