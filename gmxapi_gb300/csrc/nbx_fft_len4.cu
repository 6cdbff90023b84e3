// Transforms of the lengths 48, 84, 112, 256, 52 (nbx_fft_len.cuh).
#include "nbx_fft_len.cuh"

namespace nbx
{
extern const FftLen kFftLen4[] = {
    fftr::make_len<6, 8>(),
    fftr::make_len<7, 12>(),
    fftr::make_len<8, 14>(),
    fftr::make_len<16, 16>(),
    fftr::make_len<4, 13>(),
    { 0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr },
};
} // namespace nbx
