// Launch plans, host code: how many warps an SM holds, and which arenas each warp of a turn (arena_turn_kernel) works on.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include "rg_tick.cuh"

namespace rg {

// Warps of a kernel that are resident on an SM at once, by its registers per thread (65,536 an SM, allocated to a thread
// in eights), in blocks of `threads`.
inline int resident_warps(int registers, int threads) {
    return 65536 / ((registers + 7) / 8 * 8 * threads) * (threads / 32);
}

// A group of arenas that one warp of arena_turn_kernel works on: positions in the step order and in the active cars.
struct TurnGroup {
    int32_t arena_first, arena_count, car_first, car_count;
};

struct TurnPlan {
    // `count` groups; empty ones behind them up to as many as any earlier plan of the batch had
    std::vector<TurnGroup> groups;
    int count = 0;
    int car_room = 0, arena_room = 0;  // what a turn's block has room for, and its bytes of shared memory
    size_t shared = 0;
};

// The groups of a turn, along the step order: whole arenas, up to kTurnCars cars (or one arena). Fewer cars per group,
// down to one arena, while the chip has warps to spare (kTurnWarps resident per SM, by the kernel's registers), and no
// more groups than those while whole arenas allow it: a few groups more are a second wave (8,191 duels in 2,731 groups of
// three 119 us a turn, in 2,048 of four 75; 4,095 3v3 arenas one by one 131, by two 83). Groups of nine cars and more take
// so much shared memory that fewer are resident (twelve cars 17 KB, 13 per SM): between that number and kTurnWarps the
// rule still counts a second wave as one. At kTurnCars the count no longer decides: 177 us a turn at 16,384 mixed arenas;
// when it was 187, up to 32 cars took 221 and up to 8 (one arena of six, three of two) 216. 168 registers instead of 128
// gained 14 us there and lost 18 of 130 us at 4,095 3v3 arenas, where the warps count.
constexpr int kTurnWarps = 16, kTurnCars = 12, kTurnArenas = 16;
constexpr size_t kTurnSharedMax = 48 * 1024;
inline size_t turn_shared_bytes(int cars, int arenas, int pads) {
    const size_t room = static_cast<size_t>((cars + 3) / 4 * 4);
    return room * (sizeof(CarState) + sizeof(WheelRuntime)) +
           static_cast<size_t>(arenas) * static_cast<size_t>(pads) * sizeof(PadState);
}
// `plan` holds the batch's plan so far and gets the new one. `order`: the arenas in step order; `car_count` by arena.
inline void plan_turn(TurnPlan& plan, const std::vector<int32_t>& order, const std::vector<int32_t>& car_count,
                      int active_cars, int sms, int pads) {
    std::vector<TurnGroup>& groups = plan.groups;
    const size_t written = groups.size();
    const int64_t warps = static_cast<int64_t>(sms) * kTurnWarps;
    int share = static_cast<int>(std::min<int64_t>(kTurnCars, (active_cars + warps - 1) / warps));
    int cars_most = 0, arenas_most = 0;
    for (;; ++share) {
        groups.clear();
        cars_most = arenas_most = 0;
        TurnGroup g{0, 0, 0, 0};
        auto close = [&] {
            if (g.arena_count == 0) return;
            groups.push_back(g);
            cars_most = std::max(cars_most, g.car_count);
            arenas_most = std::max(arenas_most, g.arena_count);
            g = TurnGroup{g.arena_first + g.arena_count, 0, g.car_first + g.car_count, 0};
        };
        for (int32_t e : order) {
            const int n = car_count[e];
            if (g.arena_count == kTurnArenas || (g.car_count + n > share && g.car_count > 0) ||
                turn_shared_bytes(std::max(cars_most, g.car_count + n), std::max(arenas_most, g.arena_count + 1),
                                  pads) > kTurnSharedMax)
                close();
            ++g.arena_count;
            g.car_count += n;
        }
        close();
        if (share >= kTurnCars || static_cast<int64_t>(groups.size()) <= warps) break;
    }
    plan.count = static_cast<int>(groups.size());
    if (groups.size() < written) groups.resize(written, TurnGroup{0, 0, 0, 0});
    plan.car_room = (cars_most + 3) / 4 * 4;
    plan.arena_room = arenas_most;
    plan.shared = turn_shared_bytes(cars_most, arenas_most, pads);
}

}  // namespace rg
