// pado_once.h -- answers of the CUDA runtime kept per device.
#pragma once

#include <map>
#include <mutex>
#include <utility>

namespace pado {

// A kernel's attributes and occupancy belong to one device's context: what was
// granted or answered on one device says nothing of the next.
template <class Key, class Value>
class OncePerDevice {
public:
    // The answer kept for key on dev, else ask()'s, kept unless it is Value()
    // (a call that failed is made again).
    template <class Ask>
    Value get(const Key &key, int dev, const Ask &ask)
    {
        const std::pair<Key, int> at(key, dev);
        std::lock_guard<std::mutex> g(mu_);
        const auto it = known_.find(at);
        if (it != known_.end()) return it->second;
        const Value v = ask();
        if (v != Value()) known_.emplace(at, v);
        return v;
    }

private:
    std::mutex mu_;
    std::map<std::pair<Key, int>, Value> known_;
};

}  // namespace pado
