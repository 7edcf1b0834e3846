// sht_fft_row.cuh -- entry of the longitude transforms of sht_fft_row.cu
// (im = 64 to 1024), called by the dispatch of sht_fft.cu.
#pragma once

#include "sht_fft_tile.cuh"

namespace sht {

bool fft_row_supported(int NC, bool inverse);
int run_fft_row(bool inverse, const sht_plan *p, const FftArgs &args, cudaStream_t s);

}  // namespace sht
