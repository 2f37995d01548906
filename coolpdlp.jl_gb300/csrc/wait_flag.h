// wait_flag.h -- the flag, in page-locked host memory, that kernels set when they
// give up a wait (plain C++: also built by the tests).
#pragma once

namespace cpdlp {

// It is cleared before the first of the kernels that are queued between two
// looks at it: clearing it for each would lose what an earlier one, still
// running, is about to report.
class WaitFlag {
    double* at_ = nullptr;
    bool queued_ = false;

  public:
    // the flag's place, for a kernel about to be queued
    double* arm(double* at) {
        if (!queued_ || at != at_) *at = 0.0;
        at_ = at;
        queued_ = true;
        return at;
    }
    // after a wait for the stream: whether one of the kernels gave up
    bool take() {
        const bool set = queued_ && *static_cast<volatile double*>(at_) != 0.0;
        queued_ = false;
        return set;
    }
};

}  // namespace cpdlp
