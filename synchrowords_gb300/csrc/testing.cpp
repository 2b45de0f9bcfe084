// Hooks for the tests, outside the public header.
#include "common.cuh"

// The growth of a device buffer after `successes` more of them fails as it does
// when the device is full (negative: none).
extern "C" void sw_testing_fail_growth(int successes) { sw::g_growths_until_failure = successes; }
