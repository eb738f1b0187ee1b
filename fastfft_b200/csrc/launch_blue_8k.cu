// Chirp-z launchers on the power-of-two length 8192 (see launch_blue.cuh).
#include "launch_blue.cuh"

namespace ffb {
namespace blue {
FFB_BLUE_LAUNCHERS(, 8192)
}  // namespace blue
}  // namespace ffb
