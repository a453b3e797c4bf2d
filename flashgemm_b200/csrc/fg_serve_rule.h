// How a batch of the server is put on the device, so that grids whose CTAs wait on one
// another always have room to start. No CUDA here: the rule is tested on the host.
#pragma once

namespace fg {

// A "waiting" grid (pair kernel, static lists) spins on results of CTAs of its own that may
// not have started yet, so it has to become resident whole: two that are partly placed
// could hold the SMs that the other needs until their wait limits end them. With one grid
// at a time per slot, each at most SMs / slots CTAs, all in flight fit together. A grid that
// takes its tiles in turn waits only for tiles that running CTAs have taken and so ends
// wherever it is placed; any number of such grids may share the device.
struct BatchMode {
    bool spread;        // the dtypes' grids side by side, else in turn on the slot's stream
    bool all_sms;       // grids of up to all SMs, else of the batch's share
    bool after_spread;  // starts after the spread batches in flight
};

// waits: one of the batch's grids is a waiting one; beside_waiting: so is one of a batch in
// flight; alone: no batch is in flight; cap_given: the caller chose the grids' size.
constexpr BatchMode batch_mode(bool waits, bool beside_waiting, bool alone, bool cap_given)
{
    const bool spread = !waits && !beside_waiting;
    return BatchMode{spread, spread && alone && !cap_given, waits};
}

}  // namespace fg
