/* PerDevice against a fake of the call that it makes once a device. */
#include <cstdio>
#include <thread>
#include <vector>

#include "fsph_per_device.h"

static int failures = 0;
#define CHECK(c)                                        \
    do {                                                \
        if (!(c)) {                                     \
            std::printf("line %d: %s\n", __LINE__, #c); \
            ++failures;                                 \
        }                                               \
    } while (0)

int main() {
    constexpr int kAll = fsph::PerDevice::kDevices;
    fsph::PerDevice once;
    int calls[kAll + 1] = {};
    auto good = [&](int dev) { return once.once(dev, [&] { return ++calls[dev], true; }); };
    CHECK(good(0) && good(0) && calls[0] == 1);
    CHECK(good(1) && good(0) && good(1) && calls[0] == 1 && calls[1] == 1); /* a second device has its own */
    int tries = 0;
    auto third = [&] { return ++tries == 3; };
    CHECK(!once.once(2, third) && !once.once(2, third) && once.once(2, third) && once.once(2, third) && tries == 3);
    CHECK(good(kAll - 1) && good(kAll - 1) && calls[kAll - 1] == 1);
    CHECK(good(kAll) && good(kAll) && calls[kAll] == 2); /* past the table: every time */
    int none = 0;
    CHECK(once.once(-1, [&] { return ++none, true; }) && once.once(-1, [&] { return ++none, true; }) && none == 2);

    fsph::PerDevice shared;
    int at[4] = {}; /* written under the lock only */
    std::vector<std::thread> ts;
    for (int t = 0; t < 8; ++t)
        ts.emplace_back([&, t] {
            for (int k = 0; k < 1000; ++k) shared.once((t + k) % 4, [&] { return ++at[(t + k) % 4], true; });
        });
    for (auto &t : ts) t.join();
    for (int n : at) CHECK(n == 1);
    return failures != 0;
}
