// spare_slots.h -- what destroyed batches leave behind for their contexts' next ones: at most one per owner.
#pragma once

#include <cstddef>
#include <cstdint>
#include <mutex>
#include <utility>
#include <vector>

namespace ghmm {

template <typename T>
class SpareSlots {
public:
    struct Slot {
        uint64_t owner;
        int device;
        T *kept;
    };

    // The owner's, which the caller then has; null when there is none.
    T *take(uint64_t owner) { return exchange(owner, 0, nullptr); }
    // Keeps `kept` for the owner; the one kept before, if any, is the caller's.
    T *put(uint64_t owner, int device, T *kept) { return exchange(owner, device, kept); }
    // Everybody's.
    std::vector<Slot> take_all() {
        std::vector<Slot> all;
        std::lock_guard<std::mutex> lk(mu_);
        all.swap(slots_);
        return all;
    }

private:
    // One step under the lock, so that an owner never has two.
    T *exchange(uint64_t owner, int device, T *kept) {
        std::lock_guard<std::mutex> lk(mu_);
        for (size_t i = 0; i < slots_.size(); i++)
            if (slots_[i].owner == owner) {
                T *old = slots_[i].kept;
                if (kept)
                    slots_[i] = Slot{owner, device, kept};
                else
                    slots_.erase(slots_.begin() + (ptrdiff_t)i);
                return old;
            }
        if (kept) slots_.push_back(Slot{owner, device, kept});
        return nullptr;
    }

    std::mutex mu_;
    std::vector<Slot> slots_;
};

}  // namespace ghmm
