// Several host threads call the sweep and pre-run operators of libwlg.so at once,
// each on buffers and a stream of its own and with a lattice that takes another
// amount of shared memory.  Every call must succeed, and the buffers must end as
// after the same calls made alone.  Prints "ok" and exits 0 on success.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>

#include "wlg.h"

namespace {

struct Buffer {
  void* p = nullptr;
  size_t bytes = 0;
};

// One sample of X x X, `walkers` walkers in one window of the whole energy range.
struct Run {
  int X, N, walkers, L;
  cudaStream_t stream = nullptr;
  std::vector<Buffer> all;
  int8_t *lat, *J, *cond, *spectrum, *found_lat;
  int *E, *newE, *found, *start, *end, *off_hist, *off_lat, *off_spec, *cond_sample, *flag;
  unsigned long long *H, *pre_H;
  double *G, *factor;
  uint64_t* off;

  template <typename T>
  T* make(size_t n, const std::vector<T>& v = {})
  {
    Buffer b;
    b.bytes = n * sizeof(T);
    cudaMalloc(&b.p, b.bytes);
    cudaMemset(b.p, 0, b.bytes);
    if (!v.empty()) cudaMemcpy(b.p, v.data(), b.bytes, cudaMemcpyHostToDevice);
    all.push_back(b);
    return static_cast<T*>(b.p);
  }

  Run(int x, int w) : X(x), N(x * x), walkers(w), L(4 * x * x + 1)
  {
    cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
    const size_t T = static_cast<size_t>(w);
    std::vector<int> at(T), hist(T);
    for (int q = 0; q < w; ++q) {
      at[q] = q * N;
      hist[q] = q * L;
    }
    lat = make<int8_t>(T * N);
    J = make<int8_t>(2 * N);
    E = make<int>(T);
    newE = make<int>(T);
    found = make<int>(T);
    start = make<int>(1, {-2 * N});
    end = make<int>(1, {2 * N});
    off_hist = make<int>(T, hist);
    off_lat = make<int>(T, at);
    cond = make<int8_t>(1);
    spectrum = make<int8_t>(L, std::vector<int8_t>(L, 1));
    off_spec = make<int>(1);
    cond_sample = make<int>(1);
    H = make<unsigned long long>(T * L);
    G = make<double>(T * L);
    factor = make<double>(T, std::vector<double>(T, std::exp(1.0)));
    off = make<uint64_t>(T);
    pre_H = make<unsigned long long>(L);
    flag = make<int>(32);
    found_lat = make<int8_t>(32 * N);
    wlg_init_interactions(J, N, 1, 5, 0.1f, stream);
    wlg_init_lattice(lat, X, X, T, 5, w, stream);
    wlg_calc_energy(0, E, lat, J, off_lat, X, X, T, w, stream);
    cudaStreamSynchronize(stream);
  }

  wlg_status calls(int n)
  {
    for (int q = 0; q < n; ++q) {
      wlg_status st = wlg_wang_landau_pre_run(E, flag, lat, found_lat, pre_H, off, J, off_lat, -2 * N, 2 * N, 64, X, X, 5,
                                              32, L / 32, walkers, walkers, 0, stream);
      for (int k = 0; k < 4 && st == WLG_OK; ++k)
        st = wlg_wang_landau(lat, J, H, G, factor, E, newE, off, found, start, end, off_hist, off_lat, cond, spectrum,
                             off_spec, cond_sample, X, X, 64, walkers, 1, walkers, 5, 0, stream);
      if (st != WLG_OK) return st;
    }
    return cudaStreamSynchronize(stream) == cudaSuccess ? WLG_OK : WLG_ERR_CUDA;
  }

  std::vector<char> contents() const
  {
    std::vector<char> v;
    for (const Buffer& b : all) {
      v.resize(v.size() + b.bytes);
      cudaMemcpy(v.data() + v.size() - b.bytes, b.p, b.bytes, cudaMemcpyDeviceToHost);
    }
    return v;
  }
};

}  // namespace

int main()
{
  const int sizes[] = {14, 16, 20, 24};  // 54, 70, 107 and 154 KB for the sweep
  const int n = 300;
  std::vector<Run> alone, together;
  for (int x : sizes) {
    alone.emplace_back(x, 8);
    together.emplace_back(x, 8);
    if (alone.back().calls(n) != WLG_OK) {
      std::printf("%d x %d failed alone\n", x, x);
      return 1;
    }
  }
  std::atomic<int> waiting{4};
  std::vector<wlg_status> st(4, WLG_OK);
  std::vector<std::thread> threads;
  for (int i = 0; i < 4; ++i)
    threads.emplace_back([&, i] {
      --waiting;
      while (waiting.load() > 0) std::this_thread::yield();
      st[i] = together[i].calls(n);
    });
  for (auto& t : threads) t.join();
  for (int i = 0; i < 4; ++i) {
    if (st[i] != WLG_OK) {
      std::printf("%d x %d: status %d beside other threads\n", sizes[i], sizes[i], static_cast<int>(st[i]));
      return 1;
    }
    if (alone[i].contents() != together[i].contents()) {
      std::printf("%d x %d: other results beside other threads\n", sizes[i], sizes[i]);
      return 1;
    }
  }
  std::printf("ok\n");
  return 0;
}
