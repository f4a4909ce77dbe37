// cfd_share.cuh -- what else of the library is in flight on a device.
//
// The team kernel and the seams' kernels are launched as a whole (a cooperative grid, or
// clusters): they wait until all of their CTAs fit beside what is running. Two of them that fill
// the chip therefore take turns, where the launch-per-phase steps of two batches overlap; and a
// chained launch of such a step holds slots on the SMs while it waits for the one before it, which is
// free only where nothing else wants them. Each step and seam call enters itself here while it
// runs, with the SMs its whole launch asks for (0: it has none), so that a step can choose its route by
// its company (cfd_batch_step).
#pragma once
#include <atomic>

namespace cfd {
constexpr int kShareDevices = 64;
struct ChipUse {
    std::atomic<int> calls, sms;
};
inline ChipUse g_chip_use[kShareDevices];

class ChipShare {
    ChipUse& use_;
    int sms_;

public:
    ChipShare(int dev, int sms) : use_(g_chip_use[dev >= 0 && dev < kShareDevices ? dev : 0]), sms_(sms) {
        use_.calls += 1;
        use_.sms += sms_;
    }
    ~ChipShare() {
        use_.sms -= sms_;
        use_.calls -= 1;
    }
    ChipShare(const ChipShare&) = delete;
    ChipShare& operator=(const ChipShare&) = delete;
    int sms() const { return sms_; }
    bool company() const { return all_calls() > 1; }
    int all_calls() const { return use_.calls.load(); }
    int all_sms() const { return use_.sms.load(); }
};
}  // namespace cfd
