// A training step after a wait inside the network's kernels ran out: the timeout flag is set from the host (no wait
// is made to run out), then dndsg_mlp_train_step has to report it and to leave the network as it was.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <vector>

#include "dndsg.h"
#include "dndsg_mlp.cuh"

#define REQUIRE(x) do { if (!(x)) { std::printf("failed: %s (line %d)\n", #x, __LINE__); return 1; } } while (0)

int main() {
  dndsg_mlp* m = nullptr;
  REQUIRE(dndsg_mlp_create(0, 7, &m) == 0);
  const int n = 300;
  std::vector<float> X(n * dg::kIn), T(n * dg::kOut);
  for (size_t e = 0; e < X.size(); e++) X[e] = 0.01f * (float)((int)(e % 37) - 18);
  for (size_t e = 0; e < T.size(); e++) T[e] = 0.1f * (float)(e % 5);
  float *dX = nullptr, *dT = nullptr;
  REQUIRE(cudaMalloc(&dX, X.size() * 4) == cudaSuccess && cudaMalloc(&dT, T.size() * 4) == cudaSuccess);
  REQUIRE(cudaMemcpy(dX, X.data(), X.size() * 4, cudaMemcpyHostToDevice) == cudaSuccess);
  REQUIRE(cudaMemcpy(dT, T.data(), T.size() * 4, cudaMemcpyHostToDevice) == cudaSuccess);
  // parameters, both moments and the BF16 copy
  auto state = [&] {
    std::vector<unsigned char> v(3 * dg::kNParam * 4 + dg::kNW * 2);
    unsigned char* p = v.data();
    cudaDeviceSynchronize();
    for (const float* q : {m->P, m->M, m->V}) cudaMemcpy(p, q, dg::kNParam * 4, cudaMemcpyDeviceToHost), p += dg::kNParam * 4;
    cudaMemcpy(p, m->W, dg::kNW * 2, cudaMemcpyDeviceToHost);
    return v;
  };
  const auto s0 = state();
  double loss = -1;
  REQUIRE(dndsg_mlp_train_step(m, dX, dT, n, 1e-3f, &loss, nullptr) == 0 && loss > 0);
  const auto s1 = state();
  REQUIRE(s1 != s0);
  const unsigned timeout = 4;  // kFlagTimeout
  REQUIRE(cudaMemcpy(m->flags, &timeout, sizeof(timeout), cudaMemcpyHostToDevice) == cudaSuccess);
  REQUIRE(dndsg_mlp_train_step(m, dX, dT, n, 1e-3f, &loss, nullptr) == DNDSG_TIMEOUT);
  REQUIRE(state() == s1);
  REQUIRE(dndsg_mlp_train_step(m, dX, dT, n, 1e-3f, nullptr, nullptr) == 0);  // not waited for: a later call reports it
  REQUIRE(state() == s1);
  REQUIRE(dndsg_mlp_gradient(m, dX, dT, n, &loss, nullptr, nullptr) == DNDSG_TIMEOUT);
  cudaFree(dX);
  cudaFree(dT);
  dndsg_mlp_destroy(m);
  std::printf("ok\n");
  return 0;
}
