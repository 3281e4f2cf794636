// How long a wait inside a kernel has lasted while the kernel ran. The clock goes on while the GPU serves another process or a debugger
// holds the kernel, and whoever is waited for stands still then too: a step between two looks counts for no more than WAIT_STEP.
#pragma once
#include <stdint.h>
#ifdef __CUDACC__
#define WAIT_CLOCK_FN __host__ __device__ __forceinline__
#else
#define WAIT_CLOCK_FN inline
#endif

constexpr uint32_t WAIT_LIMIT = 2048, WAIT_STEP = 256;       // in units of 2^20 ns: a wait gives up after about two seconds, at the ninth look or later

struct WaitClock {
    uint32_t last = 0;
    int waited = -1;                                         // -1: not looked at yet
    // takes a reading of the nanosecond clock; true: the wait has lasted too long
    WAIT_CLOCK_FN bool spent(unsigned long long now_ns) {
        const uint32_t now = (uint32_t)(now_ns >> 20), step = now - last;
        waited = waited < 0 ? 0 : waited + (int)(step < WAIT_STEP ? step : WAIT_STEP);
        last = now;
        return waited > (int)WAIT_LIMIT;
    }
};
