// Fused image <-> grid transforms (band_fft.cuh): the lengths 400, 432, 480, 512.
#include "band_fft.cuh"

namespace gbn {

extern const FftEntry fft_f[];
const FftEntry fft_f[] = {
    FftLaunch<20, 20>::entry(),
    FftLaunch<18, 24>::entry(),
    FftLaunch<20, 24>::entry(),
    FftLaunch<16, 32>::entry(),
    FftEntry{0, 0, nullptr, nullptr, nullptr}};

}  // namespace gbn
