// State of the library that exists once per device (scratch buffers of a call), each with a lock
// of its own: calls on different devices do not wait for one another.
#pragma once

#include <map>
#include <mutex>

template <typename T>
class PerDevice {
public:
    struct Slot {
        std::mutex mu;   // held while value is used
        T value{};
    };
    // the device's slot, made on first use; it stays where it is for the life of the process
    Slot &at(int device)
    {
        std::lock_guard<std::mutex> lk(mu_);
        return slots_[device];
    }

private:
    std::mutex mu_;   // the map only
    std::map<int, Slot> slots_;
};
