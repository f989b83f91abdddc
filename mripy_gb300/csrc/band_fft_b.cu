// Fused image <-> grid transforms (band_fft.cuh): the lengths 112, 120, 128, 144, 150, 160, 162.
#include "band_fft.cuh"

namespace gbn {

extern const FftEntry fft_b[];
const FftEntry fft_b[] = {
    FftLaunch<8, 14>::entry(),
    FftLaunch<10, 12>::entry(),
    FftLaunch<8, 16>::entry(),
    FftLaunch<12, 12>::entry(),
    FftLaunch<10, 15>::entry(),
    FftLaunch<10, 16>::entry(),
    FftLaunch<9, 18>::entry(),
    FftEntry{0, 0, nullptr, nullptr, nullptr}};

}  // namespace gbn
