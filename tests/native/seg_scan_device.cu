// The scan of the row-segment counts (dmsc_b200/csrc/scan.cuh) on its own, with
// a given status word and number of looks, for the GPU test: the five words of
// its readback area in `words`. Every segment counts 1, 2 and 3.
#include <vector>

#include "../../dmsc_b200/csrc/scan.cuh"

using namespace dmsc;

extern "C" int seg_scan_device(long long n, unsigned status, int looks, long long* words) {
  const long long tiles = (n + kScanTile - 1) / kScanTile;
  const size_t nw = 1 + 3 * (size_t)tiles;
  int* buf = nullptr;
  unsigned long long* w = nullptr;
  long long* rb = nullptr;
  unsigned* st = nullptr;
  const long long pitch = (n + 3) / 4 * 4;  // 16-byte aligned arrays
  std::vector<int> h(3 * (size_t)pitch);
  for (int k = 0; k < 3; ++k)
    for (long long i = 0; i < n; ++i) h[k * (size_t)pitch + i] = k + 1;
  bool ok = cudaMalloc(&buf, 6 * (size_t)pitch * sizeof(int)) == cudaSuccess &&
            cudaMalloc(&w, nw * sizeof *w) == cudaSuccess && cudaMalloc(&rb, 5 * sizeof *rb) == cudaSuccess &&
            cudaMalloc(&st, sizeof *st) == cudaSuccess &&
            cudaMemcpy(buf, h.data(), h.size() * sizeof(int), cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemset(w, 0, nw * sizeof *w) == cudaSuccess && cudaMemset(rb, 0, 5 * sizeof *rb) == cudaSuccess &&
            cudaMemcpy(st, &status, sizeof status, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) {
    SegScan S;
    for (int k = 0; k < 3; ++k) {
      S.in[k] = buf + k * pitch;
      S.out[k] = buf + (3 + k) * pitch;
    }
    S.rb = rb;
    S.status = st;
    scan_kernel<3, SegScan><<<(unsigned)tiles, kScanNT>>>(S, n, ScanState{(unsigned*)w, w + 1, 1u, looks, st});
    ok = cudaGetLastError() == cudaSuccess &&
         cudaMemcpy(words, rb, 5 * sizeof *rb, cudaMemcpyDeviceToHost) == cudaSuccess;
  }
  cudaFree(buf);
  cudaFree(w);
  cudaFree(rb);
  cudaFree(st);
  return ok ? 0 : 1;
}
