// A look-back wait that runs out (csrc/transpose.cu, compiled with a short bound): the first
// tile of a pass never runs, so its words stay unset.  The pass must report it, and the next pass
// and the offsets must leave their outputs alone.  Prints the three findings.
#include <cstdio>
#include <vector>

#include "transpose.cu"

using namespace psc;

int main() {
  const uint64_t n = 60000, m = 6 * kRsTile + 7, ntiles = (m + kRsTile - 1) / kRsTile;
  std::vector<uint32_t> keys(m);
  for (uint64_t i = 0; i < m; i++) keys[i] = (uint32_t)((i * 2654435761u) % n);
  uint32_t *k, *a, *b;
  unsigned long long *hist, *status, *failed, *ngaps;
  uint64_t* off;
  GapEnt* gaps;
  uint32_t* ticket;
  if (cudaMalloc(&k, m * 4) || cudaMalloc(&a, 2 * m * 4) || cudaMalloc(&b, 2 * m * 4) ||
      cudaMalloc(&hist, 2 * kRsBins * 8) || cudaMalloc(&status, ntiles * kRsBins * 8) ||
      cudaMalloc(&failed, 16) || cudaMalloc(&ticket, 4) || cudaMalloc(&off, (n + 1) * 8) ||
      cudaMalloc(&gaps, (n / kGapLong + 2) * sizeof(GapEnt)))
    return 2;
  ngaps = failed + 1;
  cudaMemcpy(k, keys.data(), m * 4, cudaMemcpyHostToDevice);
  cudaMemset(a, 0xFF, 2 * m * 4);
  cudaMemset(b, 0xEE, 2 * m * 4);
  cudaMemset(off, 0xDD, (n + 1) * 8);
  cudaMemset(failed, 0, 16);
  cudaMemset(hist, 0, 2 * kRsBins * 8);
  k_rs_count<2><<<4, kRsBlock>>>(k, m, hist);
  k_rs_starts<<<2, kRsBins>>>(hist);
  const uint32_t one = 1;  // tile 0's ticket is never drawn
  cudaMemset(status, 0, ntiles * kRsBins * 8);
  cudaMemcpy(ticket, &one, 4, cudaMemcpyHostToDevice);
  k_rs_pass<<<(unsigned)ntiles - 1, kRpBlock>>>(k, k, m, 0, hist, ticket, status, a, a + m, failed);
  unsigned long long first = 0;
  cudaMemcpy(&first, failed, 8, cudaMemcpyDeviceToHost);
  cudaMemset(status, 0, ntiles * kRsBins * 8);
  cudaMemset(ticket, 0, 4);
  k_rs_pass<<<(unsigned)ntiles, kRpBlock>>>(a, a + m, m, kRsBits, hist + kRsBins, ticket, status, b,
                                            b + m, failed);
  k_bounds<<<8, 256>>>(b, m, n, off, gaps, ngaps, failed);
  k_fill_gaps<<<8, 256>>>(gaps, ngaps, off);
  std::vector<uint32_t> hb(2 * m);
  std::vector<uint64_t> ho(n + 1);
  cudaMemcpy(hb.data(), b, 2 * m * 4, cudaMemcpyDeviceToHost);
  cudaMemcpy(ho.data(), off, (n + 1) * 8, cudaMemcpyDeviceToHost);
  uint64_t touched = 0, offs = 0;
  for (uint32_t x : hb) touched += x != 0xEEEEEEEEu;
  for (uint64_t x : ho) offs += x != 0xDDDDDDDDDDDDDDDDull;
  std::printf("failed %llu written %llu offsets %llu error %d\n", first, (unsigned long long)touched,
              (unsigned long long)offs, (int)cudaDeviceSynchronize());
  return 0;
}
