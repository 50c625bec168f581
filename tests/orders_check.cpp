// Host check of PointOrders (csrc/cpd_orders.h) on a device whose copies are carried out only when
// they are waited for.
// usage: orders_check early    <sizes>...       prints: given <orders handed out> early <before the device had them>
//        orders_check steady <one-off sizes>   prints: given <calls of a steady size that got an order, of 3 after those>
//                                                      kept <sizes kept when 100 come twice>
//        orders_check sorted   <R> <seeds>...   prints: points <n> misplaced <not in ascending order of the seed's points>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>
#include <string>
#include <vector>

#include "cpd_orders.h"

using namespace cpd;

struct LateDevice {
    struct Copy {
        uint32_t *dst;
        std::vector<uint32_t> data;
    };
    std::vector<Copy> pending;
    std::set<uint32_t *> owned;
    uint32_t *alloc(uint32_t n)
    {
        uint32_t *p = static_cast<uint32_t *>(std::malloc(4u * n));
        std::memset(p, 0xff, 4u * n);
        owned.insert(p);
        return p;
    }
    bool upload(uint32_t *dst, const uint32_t *src, uint32_t n)
    {
        pending.push_back(Copy{dst, {src, src + n}});
        return true;
    }
    bool wait()
    {
        for (Copy &c : pending) std::memcpy(c.dst, c.data.data(), 4u * c.data.size());
        pending.clear();
        return true;
    }
    void free(uint32_t *p)
    {
        owned.erase(p);
        std::free(p);
    }
};

int main(int argc, char **argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    LateDevice dev;
    PointOrders orders;
    if (what == "early") {
        long given = 0, early = 0;
        for (int i = 2; i < argc; i++) {
            const uint32_t R = (uint32_t)std::atoi(argv[i]);
            for (int call = 0; call < 3; call++) {
                uint32_t rot = 0;
                const uint32_t *o = orders.get(dev, R, 0, rot);
                if (!o) continue;
                given++;
                bool there = dev.pending.empty();
                std::vector<uint8_t> seen(R, 0);
                for (uint32_t k = 0; k < R && there; k++) {
                    there = o[k] < R && !seen[o[k]];
                    if (there) seen[o[k]] = 1;
                }
                early += !there;
            }
        }
        orders.release(dev);
        std::printf("given %ld early %ld left %zu\n", given, early, dev.owned.size());
    } else if (what == "steady" && argc > 2) {
        const uint32_t n = (uint32_t)std::atoi(argv[2]);
        uint32_t rot = 0;
        long given = 0, kept = 0;
        for (uint32_t i = 0; i < n; i++) orders.get(dev, 100u + i, 0, rot);
        for (int call = 0; call < 3; call++) given += orders.get(dev, 50u, 0, rot) != nullptr;
        for (int call = 0; call < 3; call++)
            for (uint32_t i = 0; i < 100u; i++) {
                orders.get(dev, 1000u + i, 0, rot);
                orders.get(dev, 1000u + i, 0, rot);
            }
        kept = (long)dev.owned.size();
        orders.release(dev);
        std::printf("given %ld kept %ld\n", given, kept);
    } else if (what == "sorted" && argc > 2) {
        const uint32_t R = (uint32_t)std::atoi(argv[2]);
        long n = 0, misplaced = 0;
        uint32_t rot = 0;
        orders.get(dev, R, 0, rot);
        for (int i = 3; i < argc; i++) {
            const double seed = std::atof(argv[i]);
            const uint32_t *o = orders.get(dev, R, (uint64_t)(seed * 18446744073709551616.0), rot);
            if (!o) return 1;
            double last = -1.0;
            for (uint32_t k = 0; k < R; k++, n++) {
                const uint32_t at = k + rot;
                const double u = x::seed_point(seed, o[at < R ? at : at - R] + 1u);
                misplaced += !(u > last) && u != 0.0;  // (a point that rounds to 0 is left to the host's table)
                last = u;
            }
        }
        orders.release(dev);
        std::printf("points %ld misplaced %ld\n", n, misplaced);
    } else {
        return 2;
    }
    return 0;
}
