// Fused image <-> grid transforms (band_fft.cuh): the lengths 240, 256, 270, 288, 300, 576.
#include "band_fft.cuh"

namespace gbn {

extern const FftEntry fft_d[];
const FftEntry fft_d[] = {
    FftLaunch<15, 16>::entry(),
    FftLaunch<16, 16>::entry(),
    FftLaunch<15, 18>::entry(),
    FftLaunch<16, 18>::entry(),
    FftLaunch<15, 20>::entry(),
    FftLaunch<24, 24>::entry(),
    FftEntry{0, 0, nullptr, nullptr, nullptr}};

}  // namespace gbn
