// Fused image <-> grid transforms (band_fft.cuh): the lengths 320, 324, 336, 360, 384, 768.
#include "band_fft.cuh"

namespace gbn {

extern const FftEntry fft_e[];
const FftEntry fft_e[] = {
    FftLaunch<16, 20>::entry(),
    FftLaunch<18, 18>::entry(),
    FftLaunch<14, 24>::entry(),
    FftLaunch<18, 20>::entry(),
    FftLaunch<16, 24>::entry(),
    FftLaunch<24, 32>::entry(),
    FftEntry{0, 0, nullptr, nullptr, nullptr}};

}  // namespace gbn
