// Self-test of the bounded waits in grid_sync.cuh: a small cooperative launch in which one block fails on purpose,
// by leaving early or by reporting a failure, never by a fault.
#include "engine.cuh"
#include "grid_sync.cuh"

namespace phastb {

namespace {

constexpr int kT = 256;
enum Failure { kNone = 0, kNoWord = 1, kNoSum = 2, kReports = 3 };

struct ExchangeTest {
  Tagged slots[4 * kGridValues * kGridBlocks];
  Tagged words[2 * kGridBlocks];
  PcgState st;
  unsigned err;
  int passed;
};

__global__ void __launch_bounds__(kT, 1)
    grid_exchange_test_kernel(ExchangeTest* t, int who, int failure, unsigned long long limit_ns) {
  const int tid = threadIdx.x, b = blockIdx.x, G = gridDim.x, next = (b + 1) % G;
  GridSync gs{t->slots, &t->err, 0ull, limit_ns};
  PcgState S = t->st;
  __shared__ int s_lost, s_wrong;
  if (tid == 0) s_lost = s_wrong = 0;
  auto fail = [&] {  // as the solves do
    if (tid == 0) atomicExch(&t->st.grid_error, 1);
  };
  __syncthreads();
  for (int it = 0; it < 3; ++it) {
    const bool here = it == 1 && b == who;
    if (here && failure == kNoWord) return;
    Tagged* words = t->words + (it & 1) * kGridBlocks;
    if (tid == 0) {
      st_node(words + b, float(b), float(it), -float(b), (unsigned)it + 1u);
      float v[3];
      if (!wait_node(words + next, (unsigned)it + 1u, v, &t->err, limit_ns))
        s_lost = 1;
      else if (v[0] != float(next) || v[1] != float(it) || v[2] != -float(next))
        s_wrong = 1;
    }
    if (here && failure == kNoSum) return;
    if (here && failure == kReports) fail();
    double v[3] = {1.0, double(b), double(b) + it};
    if (!grid_reduce<2, 1, kT>(v, gs) || s_lost) return fail();
    if (v[0] != double(kT) * G || v[1] != double(kT) * (G * (G - 1) / 2) || v[2] != double(it)) s_wrong = 1;
    S.iter += 1;
  }
  __syncthreads();
  if (tid == 0 && !s_wrong) atomicAdd(&t->passed, 1);
  if (b == 0 && tid == 0) store_pcg_state(&t->st, S);
}

}  // namespace

}  // namespace phastb

extern "C" int phastb_test_grid_exchange(int blocks, int who, int failure, double limit_s, int* grid_error_host,
                                         int* passed_host) {
  using namespace phastb;
  if (blocks < 1 || blocks > kGridBlocks || who < 0 || who >= blocks || failure < kNone || failure > kReports ||
      !(limit_s > 0) || limit_s > 10.0 || !grid_error_host || !passed_host)
    return PHASTB_ERR_ARG;
  int dev = 0, sms = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop || blocks > sms)
    return PHASTB_UNSUPPORTED;
  ExchangeTest* t = nullptr;
  if (cudaMalloc(&t, sizeof(ExchangeTest)) != cudaSuccess) return PHASTB_ERR_CUDA;
  int status = cuda_status(cudaMemset(t, 0, sizeof(ExchangeTest)));
  unsigned long long limit_ns = (unsigned long long)(limit_s * 1e9);
  void* args[] = {&t, &who, &failure, &limit_ns};
  if (!status) {
    note_launch();
    status = cuda_status(
        cudaLaunchCooperativeKernel((const void*)grid_exchange_test_kernel, dim3(blocks), dim3(kT), args, 0, nullptr));
  }
  if (!status) status = cuda_status(cudaDeviceSynchronize());
  PcgState hs{};
  if (!status) status = cuda_status(cudaMemcpy(&hs, &t->st, sizeof(hs), cudaMemcpyDeviceToHost));
  if (!status) status = cuda_status(cudaMemcpy(passed_host, &t->passed, sizeof(int), cudaMemcpyDeviceToHost));
  cudaFree(t);
  if (status) return status;
  *grid_error_host = hs.grid_error;
  return hs.grid_error ? PHASTB_ERR_CUDA : PHASTB_OK;
}
