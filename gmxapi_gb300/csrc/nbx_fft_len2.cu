// Transforms of the lengths 28, 72, 104, 192, 36, 44 (nbx_fft_len.cuh).
#include "nbx_fft_len.cuh"

namespace nbx
{
extern const FftLen kFftLen2[] = {
    fftr::make_len<4, 7>(),
    fftr::make_len<8, 9>(),
    fftr::make_len<8, 13>(),
    fftr::make_len<12, 16>(),
    fftr::make_len<6, 6>(),
    fftr::make_len<4, 11>(),
    { 0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr },
};
} // namespace nbx
