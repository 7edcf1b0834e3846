// sht_fft_mixed.cuh -- entry of the longitude transforms with radices 3 and 5
// (sht_fft_mixed.cu), called by the dispatch of sht_fft.cu.
#pragma once

#include "sht_fft_tile.cuh"

namespace sht {

// whether im = I is a product of two radices of the mixed-radix kernels
bool fft_mixed_supported(int I, int N);
int run_fft_mixed(bool inverse, const sht_plan *p, const FftArgs &args, cudaStream_t s);

}  // namespace sht
