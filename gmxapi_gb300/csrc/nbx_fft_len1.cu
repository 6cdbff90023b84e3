// Transforms of the lengths 24, 64, 100, 144, 224 (nbx_fft_len.cuh).
#include "nbx_fft_len.cuh"

namespace nbx
{
extern const FftLen kFftLen1[] = {
    fftr::make_len<4, 6>(),
    fftr::make_len<8, 8>(),
    fftr::make_len<10, 10>(),
    fftr::make_len<12, 12>(),
    fftr::make_len<14, 16>(),
    { 0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr },
};
} // namespace nbx
