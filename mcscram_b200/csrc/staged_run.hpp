// staged_run.hpp -- how a staged run ends on the host, also where it fails part
// way (no CUDA calls).
#pragma once
#include <string>
#include <utility>

#include "error.hpp"

namespace mcg {

// A run on the side streams: fork, the chunks that body queues, join.  The join
// follows in every case: chunks queued before an error still read and write the
// engine's buffers, and whatever the engine stream gets next (the next run
// starts again at the first buffer) has to wait for them.  The first error is
// the run's.
template <class Fork, class Body, class Join>
mcg_status forked_run(Fork fork, Body body, Join join) {
    mcg_status st = fork();
    if (st == MCG_OK) st = body();
    const std::string first = last_error();
    const mcg_status joined = join();
    if (st == MCG_OK) return joined;
    last_error() = first;
    return st;
}

// Calls f at the end of the scope, whichever way it is left.
template <class F>
class AtExit {
public:
    explicit AtExit(F f) : f_(std::move(f)) {}
    ~AtExit() { f_(); }
    AtExit(const AtExit &) = delete;
    AtExit &operator=(const AtExit &) = delete;

private:
    F f_;
};

}  // namespace mcg
