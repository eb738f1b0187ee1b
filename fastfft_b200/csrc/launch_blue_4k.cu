// Chirp-z launchers on the power-of-two length 4096 (see launch_blue.cuh).
#include "launch_blue.cuh"

namespace ffb {
namespace blue {
FFB_BLUE_LAUNCHERS(, 4096)
}  // namespace blue
}  // namespace ffb
