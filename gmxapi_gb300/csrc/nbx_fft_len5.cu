// Transforms of the lengths 56, 90, 120, 128 (nbx_fft_len.cuh).
#include "nbx_fft_len.cuh"

namespace nbx
{
extern const FftLen kFftLen5[] = {
    fftr::make_len<7, 8>(),
    fftr::make_len<9, 10>(),
    fftr::make_len<10, 12>(),
    fftr::make_len<8, 16>(),
    { 0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr },
};
} // namespace nbx
