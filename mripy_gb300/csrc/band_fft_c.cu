// Fused image <-> grid transforms (band_fft.cuh): the lengths 168, 180, 192, 200, 216, 224, 640.
#include "band_fft.cuh"

namespace gbn {

extern const FftEntry fft_c[];
const FftEntry fft_c[] = {
    FftLaunch<12, 14>::entry(),
    FftLaunch<12, 15>::entry(),
    FftLaunch<12, 16>::entry(),
    FftLaunch<10, 20>::entry(),
    FftLaunch<12, 18>::entry(),
    FftLaunch<14, 16>::entry(),
    FftLaunch<20, 32>::entry(),
    FftEntry{0, 0, nullptr, nullptr, nullptr}};

}  // namespace gbn
