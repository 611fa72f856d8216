// The digit contraction with a status word that is set already, as after a wait
// of the same launch has given up: its waits end at once, and it returns with
// none of its copies and MMAs in flight, the context usable.  Prints its flag
// without a status, with one, and without one again.
#include <cstdio>

#include "exact_gemm.cuh"

using namespace sigma;

static int run(const ExactPrep& ex, int sms, int* words, int status) {
  int h[2] = {0, status};
  cudaMemcpy(words, h, sizeof h, cudaMemcpyHostToDevice);
  cudaError_t e = launch_exact_gemm(ex, sms, words + 1, nullptr);
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return -1;
  cudaMemcpy(h, words, sizeof h, cudaMemcpyDeviceToHost);
  return h[1] == status ? h[0] : -2;
}

int main() {
  int sms = 0, bad = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0);
  for (int slices = 6; slices <= 7; ++slices) {
    ExactPrep ex{};
    ExactTables t;
    exact_size(ex, slices, 45, 20000, 670, 3, true, sms, nullptr, &t);  // several items and ring turns per CTA
    const size_t work = exact_work_bytes(ex), own = exact_own_bytes(ex);
    char* block = nullptr;
    int* words = nullptr;
    if (cudaMalloc(&block, work + own + 256) != cudaSuccess || cudaMalloc(&words, 256) != cudaSuccess) return 2;
    cudaMemset(block, 0, work + own + 256);
    exact_bind(ex, block, block + work);
    if (exact_upload_tables(ex, t) != cudaSuccess) return 2;
    ex.flag = words;
    const int plain = run(ex, sms, words, 0), gave_up = run(ex, sms, words, -5), again = run(ex, sms, words, 0);
    printf("slices %d: flag %d, %d with a set status, %d\n", slices, plain, gave_up, again);
      bad += plain < 0 || gave_up < 0 || again < 0;
    cudaFree(block);
    cudaFree(words);
  }
  printf("%d bad\n", bad);
  return bad != 0;
}
