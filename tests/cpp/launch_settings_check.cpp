// A level's launch shapes are the ones set, whatever its size: what a batch's settings report is
// what its launches take. Linked with the library; nothing here touches a device.
#include "autotune.hpp"
#include "planet.hpp"
#include "solver.hpp"

#include <cstdio>

int main() {
    for (std::uint32_t tiles : {1u, 304u, 2431u, 2432u, 2561u, 40000u}) {
        for (int stencil : {1, 2}) {
            for (int vector : {1, 4}) {
                psgb::Batch b;
                b.levels.resize(2);
                for (psgb::BatchLevel& L : b.levels) {
                    L.tiles = tiles;
                    L.rows = tiles * 256u;
                    L.width = 6;
                }
                psgb::Tuning t;
                t.pre = t.post = {1, 1};
                t.sets_stencil.assign(2, static_cast<std::uint8_t>(stencil));
                t.sets_vector.assign(2, static_cast<std::uint8_t>(vector));
                psgb::apply_tuning(b, t);
                const psgb::Tuning got = psgb::current_tuning(b);
                for (std::size_t l = 0; l < 2; ++l) {
                    const auto v32 = psgb::view32(b, l);
                    const auto v64 = psgb::view64(b, l);
                    if (got.sets_vector[l] != vector || got.sets_stencil[l] != stencil || v32.sets_vector != vector ||
                        v64.sets_vector != vector || v32.sets_stencil != stencil || v64.sets_stencil != stencil) {
                        std::printf("%u tiles, set %d and %d: reported %d and %d, launched %d and %d\n", tiles, stencil, vector,
                                    got.sets_stencil[l], got.sets_vector[l], v64.sets_stencil, v64.sets_vector);
                        return 1;
                    }
                }
            }
        }
    }
    std::puts("OK");
    return 0;
}
