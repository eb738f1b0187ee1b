// Chirp-z launchers on the power-of-two lengths 1024 and 2048 (see launch_blue.cuh).
#include "launch_blue.cuh"

namespace ffb {
namespace blue {
FFB_BLUE_LAUNCHERS(, 1024)
FFB_BLUE_LAUNCHERS(, 2048)
}  // namespace blue
}  // namespace ffb
