// Transforms of the lengths 20, 60, 96, 160, 168, 25 (nbx_fft_len.cuh).
#include "nbx_fft_len.cuh"

namespace nbx
{
extern const FftLen kFftLen0[] = {
    fftr::make_len<4, 5>(),
    fftr::make_len<6, 10>(),
    fftr::make_len<8, 12>(),
    fftr::make_len<10, 16>(),
    fftr::make_len<12, 14>(),
    fftr::make_len<5, 5>(),
    { 0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr },
};
} // namespace nbx
