// Solves on several handles at once, a host thread each, without Python's interpreter lock between the calls: every
// result has to be the bits of the handle's first solve, made alone.  Returns how many were not; why: the first reason.
#include <cstdio>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "ssim_gb.h"

extern "C" int solve_threads(int count, ssim_gb_timestep** handles, const double** rhs, const int* sizes, int solves,
                             char* why, int why_size) {
  std::vector<std::vector<double>> first(count);
  std::mutex m;
  int bad = 0;
  auto note = [&](const char* text) {
    std::lock_guard<std::mutex> lock(m);
    if (bad++ == 0) std::snprintf(why, (size_t)why_size, "%s", text);
  };
  for (int k = 0; k < count; ++k) {
    first[k].resize(sizes[k]);
    int it = 0;
    double rr = 0;
    if (ssim_gb_pcg(handles[k], rhs[k], first[k].data(), 5e-2, 5000, &it, &rr) != SSIM_GB_OK)
      note(ssim_gb_last_error(handles[k]));
  }
  if (bad) return bad;
  std::vector<std::thread> threads;
  for (int k = 0; k < count; ++k)
    threads.emplace_back([&, k] {
      std::vector<double> x(sizes[k]);
      for (int i = 0; i < solves; ++i) {
        int it = 0;
        double rr = 0;
        if (ssim_gb_pcg(handles[k], rhs[k], x.data(), 5e-2, 5000, &it, &rr) != SSIM_GB_OK)
          note(ssim_gb_last_error(handles[k]));
        else if (std::memcmp(x.data(), first[k].data(), sizeof(double) * x.size()) != 0)
          note("another solution");
      }
    });
  for (auto& t : threads) t.join();
  return bad;
}
