// One sort pass whose first tiles never run (the ticket starts past them), so
// every look-back of the others waits in vain and takes the missing counts
// from the keys.  Built and called by test_gpu_radix_recount.py.
#include "radix.cu"

// Tiles [first, tiles) of a pass over the digit (key >> shift) & mask;
// scratch: radix_hist_entries(count) words.  0: done.
extern "C" int
radix_recount(uint32_t const* kin, uint32_t const* vin, uint32_t* kout, uint32_t* vout, uint64_t count, int shift, uint32_t mask, uint32_t first, uint32_t polls, uint32_t* scratch)
{
  using namespace kspn;
  unsigned const tiles = div_up(count, RX_TILE);
  if (first >= tiles) return 1;
  rx_digits d{};
  d.passes   = 1;
  d.shift[0] = shift;
  d.mask[0]  = mask;
  cudaMemset(scratch, 0, radix_hist_entries(count) * sizeof(uint32_t));
  k_radix_hist<<<148, RX_THREADS>>>(kin, count, d, scratch);
  cudaMemcpy(scratch + RX_PASSES * RX_BINS, &first, sizeof(first), cudaMemcpyHostToDevice);
  k_radix_pass<<<tiles - first, RX_THREADS>>>(rx_args{ kin, vin, kout, vout, count, shift, mask, 0, scratch, scratch + RX_PASSES * RX_BINS, reinterpret_cast<unsigned long long*>(scratch + RX_HEAD),
                                                       polls ? polls : RX_POLLS });
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 2;
}

extern "C" uint64_t
radix_recount_scratch(uint64_t count)
{
  return kspn::radix_hist_entries(count);
}
