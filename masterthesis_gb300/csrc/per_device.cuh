// A value found once per device of the process, for properties that belong to
// a device (occupancy, function attributes that have to be set before a
// launch).  Safe with several threads: the first of a device finds the value,
// the others wait for it.
#pragma once

#include <mutex>

namespace scafes {

class PerDevice {
public:
    template <class Find>
    int get(int device, const Find& find) {
        if (device < 0 || device >= MAX) return find();
        std::call_once(once_[device], [&] { value_[device] = find(); });
        return value_[device];
    }

private:
    static constexpr int MAX = 64;
    std::once_flag once_[MAX];
    int value_[MAX] = {};
};

}  // namespace scafes
