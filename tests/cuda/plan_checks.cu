// Compile-time checks of the host rules over FFT plans: an access outside a
// plan's arrays is not a constant expression, so it does not compile.
#include "fft.cuh"

using phgpu::ends_in_prime_stage;
using phgpu::FftPlan;

constexpr FftPlan kOne{1, 0, {}, {}, {}, {}, nullptr};  // length 1: no stage
constexpr FftPlan k26{26, 2, {2, 13}, {26, 13}, {}, {}, nullptr};
constexpr FftPlan k201{201, 2, {3, 67}, {201, 67}, {}, {}, nullptr};

static_assert(!ends_in_prime_stage(kOne), "no stage, no prime stage");
static_assert(!ends_in_prime_stage(k26), "13 is a small radix");
static_assert(ends_in_prime_stage(k201), "67 is a prime stage");
