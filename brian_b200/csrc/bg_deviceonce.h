// bg_deviceonce.h -- something done once per device and key, by whichever
// thread comes first (host only, no CUDA).
#pragma once
#include <mutex>
#include <set>
#include <utility>

class DeviceOnce {
    std::mutex mutex;
    std::set<std::pair<int, const void *>> done;

public:
    // set() unless it has succeeded for (device, key) before; false when it fails.
    template <typename F> bool operator()(int device, const void *key, F set) {
        std::lock_guard<std::mutex> lock(mutex);
        if (done.count({device, key})) return true;
        if (!set()) return false;
        done.insert({device, key});
        return true;
    }
};
