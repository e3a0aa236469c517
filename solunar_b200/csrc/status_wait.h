// status_wait.h -- whether a world's wait for its status polls pinned memory (host rule only).
#pragma once

#include <driver_types.h>

namespace slf {

// The device's scheduling flag says how its waits treat the host's cores.  Polling is how the runtime
// itself waits under `spin` and `auto` (which spins while the process has no more contexts than cores):
// 44 -> 38 us a substep of 720 particles against the runtime's wait.  A process that asked its waits to
// yield or to block leaves them to the runtime.
inline bool polls_under(unsigned int flags) {
    const unsigned int how = flags & cudaDeviceScheduleMask;
    return how == cudaDeviceScheduleAuto || how == cudaDeviceScheduleSpin;
}

}  // namespace slf
