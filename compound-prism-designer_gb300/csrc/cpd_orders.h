// cpd_orders.h -- the orders of the point sequence that a context keeps on its device.
//
// The points of a seed are fract(seed + j/phi): sorted, they are the seedless points' order turned
// by the seed. So one table per number of points R serves every seed (TableJob::order, rot).
// Host code; the device's calls are a parameter, so that tests/orders_check.cpp runs it without one.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <map>
#include <utility>
#include <vector>

#include "cpd_model.h"

namespace cpd {

// Sizes whose order a context keeps on the device (at most 64 KiB each).
constexpr size_t kMaxOrders = 64;

// An order is made when its size comes a second time and kept until release: passes in flight on
// any stream may read it. Sizes seen once give way to new ones. The caller serialises the calls.
// Device: uint32_t *alloc(n); bool upload(dst, src, n), which may return before the device has the
// data, and bool wait(), which does not; void free(p).
class PointOrders {
    struct Order {
        uint64_t since = 0;  // when the size came first
        uint32_t *dev = nullptr;
        std::vector<uint64_t> keys;  // the sorted points, in 2^-64
    };
    std::map<uint32_t, Order> orders;
    uint64_t clock = 0;

public:
    // The device's order of the sequence's first R points and, for a seed (in 2^-64), how far the
    // seed turns it; nullptr when this size is not kept (yet).
    template <class Device>
    const uint32_t *get(Device &device, uint32_t R, uint64_t seed_fixed, uint32_t &rot)
    {
        auto it = orders.find(R);
        if (it == orders.end()) {
            if (orders.size() >= kMaxOrders) {
                auto old = orders.end();
                for (auto i = orders.begin(); i != orders.end(); ++i)
                    if (!i->second.dev && (old == orders.end() || i->second.since < old->second.since)) old = i;
                if (old == orders.end()) return nullptr;
                orders.erase(old);
            }
            orders[R].since = ++clock;
            return nullptr;
        }
        Order &o = it->second;
        if (!o.dev) {
            const uint64_t alpha = (uint64_t)(kAlpha * 18446744073709551616.0);
            std::vector<std::pair<uint64_t, uint32_t>> kj(R);
            for (uint32_t j = 0; j < R; j++) kj[j] = {alpha * (j + 1u), j};
            std::sort(kj.begin(), kj.end());
            std::vector<uint32_t> order(R);
            std::vector<uint64_t> keys(R);
            for (uint32_t i = 0; i < R; i++) {
                keys[i] = kj[i].first;
                order[i] = kj[i].second;
            }
            uint32_t *dev = device.alloc(R);
            if (!dev) return nullptr;
            // complete before any pass can be given the address: the passes' streams wait for
            // nothing but their own work
            if (!device.upload(dev, order.data(), R) || !device.wait()) {
                device.free(dev);
                return nullptr;
            }
            o.keys.swap(keys);
            o.dev = dev;
        }
        // the points that the seed carries past 1 come first
        rot = seed_fixed ? (uint32_t)(std::lower_bound(o.keys.begin(), o.keys.end(), 0ull - seed_fixed) - o.keys.begin())
                         : 0u;
        if (rot == R) rot = 0u;
        return o.dev;
    }

    template <class Device>
    void release(Device &device)
    {
        for (auto &o : orders)
            if (o.second.dev) device.free(o.second.dev);
        orders.clear();
    }
};

}  // namespace cpd
