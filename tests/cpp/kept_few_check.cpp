// KeptFew (host/kept_few.hpp): never more than its bound, the least recently used first to go,
// given back before another is made, nothing kept of one whose making throws.
#include "host/kept_few.hpp"

#include <cstdio>
#include <memory>
#include <stdexcept>
#include <vector>

#define CHECK(x)                                                  \
    do {                                                          \
        if (!(x)) {                                               \
            std::printf("failed at line %d: %s\n", __LINE__, #x); \
            return 1;                                             \
        }                                                         \
    } while (0)

namespace {
int alive = 0, most = 0, made = 0;
struct Plan {
    int key;
    explicit Plan(int k) : key(k) {
        ++made;
        most = ++alive > most ? alive : most;
    }
    ~Plan() { --alive; }
};
}  // namespace

int main() {
    {
        psgb::KeptFew<std::vector<int>, std::unique_ptr<Plan>, 4> kept;
        const auto ask = [&](int k) { return kept.of({k, k + 1}, [&] { return std::make_unique<Plan>(k); })->key; };
        for (int round = 0; round < 3; ++round)
            for (int k = 0; k < 40; ++k) CHECK(ask(k) == k);
        CHECK(made == 120 && most == 4 && alive == 4 && kept.size() == 4);
        // 36..39 are kept; 36 used again, so 37 goes first
        CHECK(ask(36) == 36 && made == 120);
        CHECK(ask(7) == 7 && made == 121);
        CHECK(ask(36) == 36 && ask(38) == 38 && ask(39) == 39 && made == 121);
        CHECK(ask(37) == 37 && made == 122 && alive == 4);
        bool thrown = false;
        try {
            kept.of({-1}, []() -> std::unique_ptr<Plan> { throw std::runtime_error("refused"); });
        } catch (const std::runtime_error&) {
            thrown = true;
        }
        CHECK(thrown && kept.size() == 3 && alive == 3);
        kept.clear();
        CHECK(alive == 0 && kept.size() == 0 && ask(1) == 1);
    }
    CHECK(alive == 0);
    std::puts("OK");
    return 0;
}
