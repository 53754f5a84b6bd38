// How zl_advance splits its steps between captured graphs and direct launches (host only).
#pragma once
#include <algorithm>

namespace zl {

// A graph holds an even number of background steps, which bring every level back to the same population
// layout, so it replays for any number of its multiples.
//
// Inside a graph the kernels follow one another as dependent launches, while a graph waits for the one before
// it.  Measured us per step, launched / in graphs of 4 / 8 / 16:
//   65^2 D2Q9 FP64   3.65 / 3.59 / 3.33 / 3.08 (in pairs 4.1)    257^2   3.94 / 4.10 / 4.08 / 3.84
//   64^3 FP32        6.70 / 7.17 / 6.67 / 6.56
//   faces in order, eight launches a step: 33 x 25 x 21 FP32 25.4 / 23.1 / 22.6 / 22.4 (in pairs 23.8),
//   97 x 65 x 65 41.3 / 39.8 / 39.4 / 39.1 (in pairs 40.4)
// So pairs pay where a step is several launches, and a step of one launch that fills no longer graph is
// launched by itself.  A graph of sixteen costs 0.17 ms to capture (0.5 ms with eight launches a step), what it
// gains in 140 to 300 steps on the smallest of these and in thousands on the others.  A context that runs
// a few dozen steps and is read out must not pay that, so a single level's long graph is captured once
// kLongGraphAfter steps have been asked for.  First call of 8 / 40 steps: 33^2 175 / 316 us with the long graph
// at once, 52 / 196 now; the ordered 33 x 25 x 21 464 / 1419 and 308 / 1081.
// Above kGraphMaxNodes a step of one launch outlasts the next one's launch and gains nothing from a graph
// (launched / in graphs of 16: 192^3 FP32 176 / 177, FP16 177.6 / 177.4, FP64 553 / 552; 256^3 FP32 398 / 399, FP64
// 1184 / 1184; below it the channel of 161 x 97 x 81 still gains 0.7 %), while instantiating one asks the driver
// for memory: a timed call that did so beside a starting nvidia-smi took 87 ms longer.  Such steps are always
// launched directly.
constexpr int kGraphSteps = 16, kGraphMinSteps = 8;
constexpr long long kLongGraphAfter = 128, kGraphMaxNodes = 1ll << 22;

struct GraphPlan {
    int run = 0;     // steps of the level's long graph (more than it holds now: capture it), 0: none
    int runs = 0;    // replays of it
    int pairs = 0;   // then replays of the graph of two steps
    int direct = 0;  // then steps launched directly
};

// seen: steps that earlier calls asked for since the last change of the set-up; have: steps that the
// long graph holds, 0 if there is none.  A multi-level step is dozens of launches and replays in pairs.
inline GraphPlan plan_graph(int steps, bool single_level, bool one_launch, long long nodes, long long seen, int have) {
    GraphPlan p;
    if (single_level && !(one_launch && nodes > kGraphMaxNodes)) {
        const int most = std::min(kGraphSteps, steps & ~1);
        p.run = seen + steps >= kLongGraphAfter && most >= kGraphMinSteps ? std::max(have, most) : have;
    }
    if (p.run > 0) p.runs = steps / p.run;
    const int rest = steps - p.runs * p.run;
    if (!(single_level && one_launch)) p.pairs = rest / 2;
    p.direct = rest - 2 * p.pairs;
    return p;
}

}  // namespace zl
