// link_choice.h -- the way of a call's ion records where the in-place kernel alone could move them.
#pragma once
#include <algorithm>
#include <cstddef>

namespace ether {

// One direction of one context.  The kernel alone is the faster on a good link (16^3 x 190, 56 MB:
// 0.24 ms up and 0.32 down, shared with the host's cores 1.36 and 1.53), but the link of some hosts
// has been several times slower (27 GB/s of records), and then the cores are: 128 MB take about
// 4.8 ms by the kernel and 2.5 shared (the estimate below).  A call whose wall time is above the
// estimate -- its link may be slow, or it waited for sweeps -- has the next ones timed on the device
// (not done without that sign, and not again for 32 calls after a good time).  Where by the better
// of the last two such rates the kernel would take longer than the shared form, the call is shared,
// and every 32nd such call tries the kernel again.  Two rates, because a process's first call can be
// slow.
struct LinkChoice {
    double rate[2] = {0.0, 0.0};  // record bytes per ms of the last timed calls
    int shared = 0;               // calls shared since the last timed one
    int skip = 0;                 // calls that are not timed, whatever they take
    bool suspect = false;         // the last call took longer than the shared form would have
    // ms of the shared form: threads and staging, and the cores' conversion at 100 GB/s of records
    // (measured 132 down, 232 up)
    static double shared_ms(size_t bytes) { return 1.2 + (double)bytes / 1e8; }
    // Calls this looks at: below 16 MB the kernel is the faster on any link above 12 GB/s.
    static bool counts(size_t bytes) { return bytes >= (size_t(16) << 20); }
    bool kernel_alone(size_t bytes) {
        if (!counts(bytes) || rate[1] <= 0.0 || (double)bytes / std::max(rate[0], rate[1]) <= shared_ms(bytes)) return true;
        if (++shared < 32) return false;
        shared = 0;
        return true;
    }
    bool time_it(size_t bytes) {
        if (!counts(bytes) || !suspect) return false;
        if (skip > 0) --skip;
        return skip == 0;
    }
    // What a call by the kernel alone took: host time, and the device's where it was timed (else 0).
    void took(size_t bytes, double wall_ms, double device_ms) {
        if (!counts(bytes)) return;
        suspect = wall_ms > shared_ms(bytes);
        const double ms = device_ms > 0.0 ? device_ms : suspect ? 0.0 : wall_ms;
        if (ms <= 0.0) return;
        rate[1] = rate[0];
        rate[0] = (double)bytes / ms;
        if (ms <= shared_ms(bytes)) skip = 32;
    }
};

}  // namespace ether
