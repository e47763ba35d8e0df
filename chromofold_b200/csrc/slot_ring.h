// slot_ring.h — scratch slots that concurrent calls hand round (compat_kv.cu).
#ifndef CHROMOFOLD_B200_SLOT_RING_H
#define CHROMOFOLD_B200_SLOT_RING_H

#include <stdint.h>

#include <mutex>

namespace cfb {

// kSlots slots, used in turn. A call waits (on its stream) for the event of its slot's last user, launches, and records the event
// anew; use(slot) does all three and runs alone. Were the lock let go in between, other threads could go round the slots and
// wait for the event of the use before, while this call's launch is still to come: two launches would share the slot.
// Everything inside is asynchronous, so the lock is held for a launch, not for its execution.
template <uint32_t kSlots>
class SlotRing {
    std::mutex lock_;
    uint32_t next_ = 0;

public:
    template <class Use>
    auto take(Use use) {
        std::lock_guard<std::mutex> guard(lock_);
        return use(next_++ % kSlots);
    }
    template <class SetUp>
    auto locked(SetUp set_up) {
        std::lock_guard<std::mutex> guard(lock_);
        return set_up();
    }
};

}  // namespace cfb

#endif
