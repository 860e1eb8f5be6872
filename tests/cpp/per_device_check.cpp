// PerDevice (host/per_device.hpp): what is made on one device is not taken for another's, is made
// once a device whoever asks, and is tried again after a failure.
#include "host/per_device.hpp"

#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>

#define CHECK(x)                                              \
    do {                                                      \
        if (!(x)) {                                           \
            std::printf("failed at line %d: %s\n", __LINE__, #x); \
            return 1;                                         \
        }                                                     \
    } while (0)

int main() {
    psgb::PerDevice<int> table;
    std::vector<int> made(4, 0);
    const auto ask = [&](int device) {
        return table.of(device, [&] {
            ++made[static_cast<std::size_t>(device)];
            return 100 + device;
        });
    };
    // the second device makes its own, the first keeps what it has
    CHECK(ask(0) == 100 && ask(1) == 101 && ask(0) == 100 && ask(1) == 101);
    CHECK(made[0] == 1 && made[1] == 1 && made[2] == 0);
    // a device that failed is tried again, the others are untouched
    bool thrown = false;
    try {
        table.of(2, []() -> int { throw std::runtime_error("refused"); });
    } catch (const std::runtime_error&) {
        thrown = true;
    }
    CHECK(thrown && ask(2) == 102 && made[2] == 1 && made[0] == 1);
    // several threads: once a device
    psgb::PerDevice<int> shared;
    std::vector<int> count(4, 0), wrong(8, 0);
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t) {
        threads.emplace_back([&, t] {
            for (int k = 0; k < 4000; ++k) {
                const int device = (t + k) % 4;
                const int got = shared.of(device, [&] { return 10 * ++count[static_cast<std::size_t>(device)] + device; });
                if (got != 10 + device) ++wrong[static_cast<std::size_t>(t)];
            }
        });
    }
    for (std::thread& t : threads) t.join();
    for (int c : count) CHECK(c == 1);
    for (int w : wrong) CHECK(w == 0);
    std::puts("OK");
    return 0;
}
