// CPU build of the zero products of the two-launch step's integer path
// (phonomena_gb300/csrc/soft_f64.cuh): the sign a zero takes from a factor.
#include "../phonomena_gb300/csrc/soft_f64.cuh"

// 0 * c as the kernels form it from c's record
extern "C" double zero_times(double zero, double c) {
  using namespace phono;
  const uint64_t u = soft_bits(zero);
  return soft_double(((uint32_t)(u >> 32) ^ soft_sign(soft_record(c, false, 0))) & 0x80000000u, 0u);
}
