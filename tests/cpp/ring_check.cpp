// Walks rings of stages whose copies land one after the other and compares what a drain waits for (ring.cuh) with what is in flight.
//   ring_check   prints "ok", or the first disagreement
#include <cstdio>
#include <vector>

#include "ring.cuh"

// An mbarrier as far as its parity test goes: `done` phases are complete, phase `done` is the current one.
struct Barrier {
    int done = 0;
    bool test(uint32_t parity) const { return ((uint32_t)done & 1u) != parity; }
};

int main() {
    for (int stages = 1; stages <= 7; ++stages)
        for (int steps = 0; steps <= 4 * stages + 1; ++steps)
            for (int landed = steps > stages ? steps - stages : 0; landed <= steps; ++landed) {  // a stage is armed again after its last copy was read
                std::vector<Barrier> full(stages);
                std::vector<int> armed(stages, 0);
                for (int i = 0; i < steps; ++i) {
                    ++armed[i % stages];
                    if (i < landed) ++full[i % stages].done;
                }
                for (int s = 0; s < stages; ++s) {
                    const int uses = lumen::ring_uses(steps, s, stages);
                    const bool in_flight = full[s].done < armed[s], waits = uses > 0 && !full[s].test(lumen::ring_last_parity(uses));
                    if (uses != armed[s] || waits != in_flight) {
                        std::printf("stages %d, steps %d, landed %d, stage %d: %d uses for %d, waits %d, in flight %d\n", stages, steps, landed, s, uses, armed[s],
                                    waits, in_flight);
                        return 1;
                    }
                }
            }
    std::puts("ok");
    return 0;
}
