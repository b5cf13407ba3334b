// faults.h - host-side fault injection of the test builds.
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>

namespace pflbm {

// The grid of a launch. In the test build -DPFLBM_TEST_FAIL_LAUNCH (never the
// shipped library) it is empty while the environment variable
// PFLBM_FAIL_LAUNCH is 1: the runtime refuses the launch with an error code
// and nothing reaches the device.
inline dim3 launch_grid(dim3 g) {
#ifdef PFLBM_TEST_FAIL_LAUNCH
    const char *e = std::getenv("PFLBM_FAIL_LAUNCH");
    if (e && e[0] == '1') return dim3(0, 1, 1);
#endif
    return g;
}

}  // namespace pflbm
