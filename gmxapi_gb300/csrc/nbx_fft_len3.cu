// Transforms of the lengths 32, 80, 108, 240, 40, 42 (nbx_fft_len.cuh).
#include "nbx_fft_len.cuh"

namespace nbx
{
extern const FftLen kFftLen3[] = {
    fftr::make_len<4, 8>(),
    fftr::make_len<8, 10>(),
    fftr::make_len<9, 12>(),
    fftr::make_len<15, 16>(),
    fftr::make_len<5, 8>(),
    fftr::make_len<6, 7>(),
    { 0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr },
};
} // namespace nbx
