// Fused image <-> grid transforms (band_fft.cuh): the lengths 64, 72, 80, 96, 100, 108.
#include "band_fft.cuh"

namespace gbn {

extern const FftEntry fft_a[];
const FftEntry fft_a[] = {
    FftLaunch<8, 8>::entry(),
    FftLaunch<8, 9>::entry(),
    FftLaunch<8, 10>::entry(),
    FftLaunch<8, 12>::entry(),
    FftLaunch<10, 10>::entry(),
    FftLaunch<9, 12>::entry(),
    FftEntry{0, 0, nullptr, nullptr, nullptr}};

}  // namespace gbn
