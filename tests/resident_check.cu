// k_resident on the identity LP of two variables, its error word set before
// the launch (as a block that gave up earlier leaves it) or not; prints the
// outcome that the host reads.  Usage: resident_check <blocks> <error word>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <vector>

#include "pdhg_resident.cuh"

#define CHECK(call)                                                               \
  do {                                                                            \
    const cudaError_t e = (call);                                                 \
    if (e != cudaSuccess) {                                                       \
      std::printf("%s: %s\n", #call, cudaGetErrorString(e));                      \
      return 1;                                                                   \
    }                                                                             \
  } while (0)

template <class T>
T* device(const std::vector<T>& h) {
  T* d = nullptr;
  if (cudaMalloc(&d, sizeof(T) * h.size()) != cudaSuccess) std::exit(1);
  if (cudaMemcpy(d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice) != cudaSuccess) std::exit(1);
  return d;
}

int main(int argc, char** argv) {
  using namespace b2p;
  const int blocks = argc > 1 ? std::atoi(argv[1]) : 1, preset = argc > 2 ? std::atoi(argv[2]) : 0;
  if (blocks != 1 && blocks != 2) return 1;
  const std::vector<int32_t> split = blocks == 1 ? std::vector<int32_t>{0, 2} : std::vector<int32_t>{0, 1, 2};
  const std::vector<double> ones{1.0, 1.0}, zeros{0.0, 0.0};
  ResidentArgs<double> a{};
  a.cb = a.rb = device(split);
  a.a_ptr = a.t_ptr = device(std::vector<int32_t>{0, 1, 2});
  a.a_idx = a.t_idx = device(std::vector<int32_t>{0, 1});
  a.a_val = a.t_val = device(ones);
  for (double** p : {&a.x, &a.x0, &a.xp, &a.y, &a.y0, &a.yp, &a.ax, &a.ax0, &a.axp}) *p = device(zeros);
  a.c = a.c64 = device(ones);
  a.lo = a.lo64 = device(zeros);
  a.up = a.up64 = device(std::vector<double>{2.0, 2.0});
  a.rl = a.rl64 = device(ones);
  a.ru = a.ru64 = device(ones);
  a.rfac = a.cfac = device(ones);
  a.tau = device(std::vector<double>{0.5});
  a.sigma = device(std::vector<double>{0.5});
  int64_t* it = device(std::vector<int64_t>{0});
  a.it_base = it;
  a.ck = IterClock{it, device(std::vector<int64_t>{0}), 0};
  a.rho = 1.0;
  a.L = 3;
  a.lt_cols = a.lt_rows = 2 * kResUnroll;
  a.arrive = device(std::vector<unsigned>{0});
  a.error = device(std::vector<int32_t>{preset});
  a.partial = device(std::vector<double>(static_cast<size_t>(blocks) * kNumSums, 0.0));
  CHECK(cudaMallocHost(&a.sums, sizeof(double) * kNumSums));
  CHECK(cudaMallocHost(&a.failed, sizeof(int32_t)));
  *a.failed = -1;
  a.m = a.n = 2;
  const size_t smem = resident_smem_bytes<double>(2, 2, 2, 2);
  const auto fn = k_resident<1, 1, double, false>;
  CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  void* args[] = {&a};
  CHECK(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(fn), dim3(blocks), dim3(kResidentThreads), args, smem,
                                    nullptr));
  CHECK(cudaDeviceSynchronize());
  std::printf("failed %d\n", *a.failed);
  return 0;
}
