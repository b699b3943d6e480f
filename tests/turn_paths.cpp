// Host build of the arena parts of a turn for test_turn_paths.py.
#include <cstring>
#include <random>
#include <vector>

#include "rg_tick.cuh"
#include "rg_turn.h"

namespace {

constexpr int kSlots = 6, kRoom = 16;  // room for every slot that four bits of a packed order can name

// One arena's state, in the middle of play: cars around the boost pads, some of them demolished.
struct Arena {
    rg::CarState slots[kRoom];
    rg::WheelRuntime wheels[kRoom];
    rg::CarConfig cfgs[kRoom];
    rg::PadState pads[64];
    rg::CarControls controls[kRoom];
    uint8_t teams[kRoom];
    rg::CarStage stages[kRoom];
    rg::BallState ball;
    rg::EnvState env;
    rg::BallWorldScratch ball_world;
    rg::Broadphase bp;
    rg::CarWorldScratch car_world[kRoom];
    rg::BallCarScratch ball_car[kRoom];
};

rg::PadLayout pad_layout() {
    rg::PadLayout l;
    memset(&l, 0, sizeof(l));
    l.count = 20;
    for (int p = 0; p < l.count; ++p) {
        l.pos[p] = rg::V3{600.0f * static_cast<float>(p % 5) - 1200.0f, 700.0f * static_cast<float>(p / 5) - 1000.0f, 70.0f};
        l.is_big[p] = p % 4 == 0;
    }
    return l;
}

rg::TickConfig tick_config() {
    rg::TickConfig tc{};
    tc.tick_dt = 1.0f / 120.0f;
    tc.frame_frac = 0.5f;
    tc.enable_boost_pads = 1;
    tc.boost_max = 100.0f;
    tc.boost_spawn_amount = 33.3f;
    tc.boost_pad_cooldown_big = 10.0f;
    tc.boost_pad_cooldown_small = 4.0f;
    tc.car_max_ang_speed = 5.5f;
    tc.max_cars = kSlots;
    return tc;
}

void fill(Arena& a, const rg::PadLayout& l, const rg::TickConfig& tc, unsigned seed) {
    memset(static_cast<void*>(&a), 0, sizeof(a));
    std::mt19937 g(seed);
    std::uniform_real_distribution<float> u(-1.0f, 1.0f);
    for (int i = 0; i < kRoom; ++i) {
        rg::CarState& c = a.slots[i];
        const rg::V3 p = l.pos[g() % l.count];
        c.pos_bt = rg::V3{p.x + 200.0f * u(g), p.y + 200.0f * u(g), 17.0f} * rg::kUuToBt;
        c.tick_start_pos_bt = c.pos_bt - rg::V3{0.3f * u(g), 0.3f * u(g), 0.0f};
        c.rot = rg::Q4{1.0f, 0.0f, 0.0f, 0.0f};
        c.boost = 50.0f + 50.0f * u(g);
        c.is_demoed = g() % 5 == 0;
        c.driving_disabled = static_cast<uint16_t>(g() % 3);
        c.boost_pad_touching = static_cast<uint8_t>(g() % (l.count + 1));
        a.cfgs[i].hitbox_size = rg::V3{118.0f, 84.0f, 36.0f};
        a.cfgs[i].hitbox_offset = rg::V3{13.9f, 0.0f, 20.8f};
        a.teams[i] = static_cast<uint8_t>(i & 1);
    }
    for (int p = 0; p < 64; ++p) {
        a.pads[p].is_active = g() % 3 != 0;
        a.pads[p].is_big = l.is_big[p];
        a.pads[p].cooldown = a.pads[p].is_active ? 0.0f : (g() % 2 ? 0.004f : 2.0f);
    }
    for (int i = 0; i < kRoom; ++i)
        rg::pad_contacts_stage(a.slots[i], a.cfgs[i], a.pads, l, tc, a.stages[i].pads);
}

rg::ArenaCars arena_cars(Arena& a, int count) {
    rg::ArenaCars A{};
    A.cars = A.slots = a.slots;
    A.wheels = a.wheels;
    A.cfgs = a.cfgs;
    A.pads = a.pads;
    A.controls = a.controls;
    A.teams = a.teams;
    A.count = count;
    A.max_cars = kSlots;
    return A;
}

}  // namespace

extern "C" {

// An arena with `count` active cars of six slots, visited in a packed order: a tick's start and tail (command 0) or a kickoff
// command and a tick's start (1), once on the batch's array and once with the active cars in a copy of their own. Returns 0, or what is
// wrong: 1 the copy's neighbours were written, 2 the results differ, 4 slots that the arena does not have were written.
int tp_visit_order(int command, int mode, uint32_t packed, int count, unsigned seed) {
    const rg::PadLayout l = pad_layout();
    const rg::TickConfig tc = tick_config();
    std::vector<Arena> both(2);
    Arena &a = both[0], &b = both[1];
    fill(a, l, tc, seed);
    a.env.car_visit_order_mode = static_cast<uint8_t>(mode);
    a.env.car_visit_order_packed = packed;
    a.env.car_visit_present_mask = 0xFF;
    memcpy(static_cast<void*>(&b), &a, sizeof(a));
    std::vector<rg::CarState> before(a.slots, a.slots + kRoom);
    rg::EnvCommand cmd;
    memset(&cmd, 0, sizeof(cmd));
    cmd.reset_to_kickoff = 1;
    cmd.kickoff_countdown_ticks = 7;
    auto run = [&](Arena& x, const rg::ArenaCars& A) {
        const rg::ArenaContactState cs{&x.ball_world, &x.bp, x.car_world, x.ball_car, nullptr, 0};
        rg::ArenaTickSnap snap;
        rg::bound_visit_order(x.env, count, kSlots);
        if (command)
            rg::apply_env_command(cmd, 0, x.env, x.ball, cs, A, x.controls, l, tc);
        rg::arena_tick_begin(x.env, x.ball, A, tc, snap, 0, 0);
        if (!command) rg::arena_tick_tail(x.env, x.ball, A, l, tc, x.stages);
    };
    run(a, arena_cars(a, count));
    std::vector<rg::CarState> packed_cars(kRoom + count + kRoom);
    memset(static_cast<void*>(packed_cars.data()), 0, packed_cars.size() * sizeof(rg::CarState));
    rg::ArenaCars A = arena_cars(b, count);
    A.cars = packed_cars.data() + kRoom;
    memcpy(static_cast<void*>(A.cars), b.slots, count * sizeof(rg::CarState));
    run(b, A);
    memcpy(static_cast<void*>(b.slots), A.cars, count * sizeof(rg::CarState));
    int wrong = 0;
    const rg::CarState zero = [] { rg::CarState z; memset(static_cast<void*>(&z), 0, sizeof(z)); return z; }();
    for (int i = 0; i < kRoom; ++i)
        if (memcmp(&packed_cars[i], &zero, sizeof(zero)) || memcmp(&packed_cars[kRoom + count + i], &zero, sizeof(zero)))
            wrong |= 1;
    if (memcmp(&a, &b, sizeof(a))) wrong |= 2;
    if (memcmp(a.slots + kSlots, before.data() + kSlots, (kRoom - kSlots) * sizeof(rg::CarState))) wrong |= 4;
    return wrong;
}

int tp_resident_warps(int registers, int threads) { return rg::resident_warps(registers, threads); }

// The packed order after bound_visit_order.
uint32_t tp_bound(int mode, uint32_t packed, int count, int max_cars) {
    rg::EnvState env;
    memset(&env, 0, sizeof(env));
    env.car_visit_order_mode = static_cast<uint8_t>(mode);
    env.car_visit_order_packed = packed;
    rg::bound_visit_order(env, count, max_cars);
    return env.car_visit_order_packed;
}

// The game's order after cars with the demolition flags `demoed` start a tick; `present` is the mask before and after.
uint32_t tp_update_order(uint32_t packed, uint8_t* present, int count, const uint8_t* demoed) {
    rg::EnvState env;
    memset(&env, 0, sizeof(env));
    env.car_visit_order_mode = 3;
    env.car_visit_order_packed = packed;
    env.car_visit_present_mask = *present;
    std::vector<rg::CarState> cars(count);
    for (int i = 0; i < count; ++i) cars[i].is_demoed = demoed[i];
    rg::update_game_visit_order(env, cars.data(), count);
    *present = env.car_visit_present_mask;
    return env.car_visit_order_packed;
}

// A tick's pad contacts and tail of an arena whose car 0 touches pad number `touching` (0: none): 0, or 1 when a pad past
// the layout's was read (one there takes cars, gives none) or changed.
int tp_touching(int touching, unsigned seed) {
    const rg::PadLayout l = pad_layout();
    const rg::TickConfig tc = tick_config();
    std::vector<rg::PadState> pads(2 * 256);  // the layout's, then other memory: in the second run all taken
    std::vector<rg::CarState> got[2];
    for (int k = 0; k < 2; ++k) {
        std::vector<Arena> one(1);
        Arena& a = one[0];
        fill(a, l, tc, seed);
        a.slots[0].boost_pad_touching = static_cast<uint8_t>(touching);
        a.slots[0].is_demoed = 0;
        memcpy(pads.data(), a.pads, l.count * sizeof(rg::PadState));
        for (size_t p = l.count; p < pads.size(); ++p) {
            memset(&pads[p], 0, sizeof(pads[p]));
            pads[p].is_active = k == 0;
            pads[p].is_big = k == 0;
        }
        const std::vector<rg::PadState> beyond(pads.begin() + l.count, pads.end());
        for (int i = 0; i < kSlots; ++i)
            rg::pad_contacts_stage(a.slots[i], a.cfgs[i], pads.data(), l, tc, a.stages[i].pads);
        rg::ArenaCars A = arena_cars(a, kSlots);
        A.pads = pads.data();
        rg::arena_tick_tail(a.env, a.ball, A, l, tc, a.stages);
        if (memcmp(beyond.data(), pads.data() + l.count, beyond.size() * sizeof(rg::PadState))) return 1;
        got[k].assign(a.slots, a.slots + kSlots);
    }
    return memcmp(got[0].data(), got[1].data(), kSlots * sizeof(rg::CarState)) != 0;
}

// Plans of a turn for `plans` rows of car counts of n arenas, one after another as a batch makes them. Returns 0, or what is
// wrong: 1 a plan's own groups do not hold every arena and active car once, in order and within the launch's room; 2 the
// grid of an earlier plan over a later plan's groups works on an arena twice.
int tp_plans(const int32_t* counts, int plans, int n, int sms, int pads) {
    rg::TurnPlan plan;
    std::vector<int> grids;
    int wrong = 0;
    for (int k = 0; k < plans; ++k) {
        const std::vector<int32_t> count(counts + static_cast<size_t>(k) * n, counts + static_cast<size_t>(k + 1) * n);
        std::vector<int32_t> order(n);
        for (int e = 0; e < n; ++e) order[e] = e;
        std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) { return count[x] > count[y]; });
        int active = 0;
        for (int32_t c : count) active += c;
        rg::plan_turn(plan, order, count, active, sms, pads);
        grids.push_back(plan.count);
        int arena = 0, car = 0;
        for (int g = 0; g < plan.count; ++g) {
            const rg::TurnGroup& t = plan.groups[g];
            int cars = 0;
            for (int j = 0; j < t.arena_count; ++j) cars += count[order[t.arena_first + j]];
            if (t.arena_first != arena || t.car_first != car || cars != t.car_count || t.arena_count < 1 ||
                t.arena_count > std::min(plan.arena_room, 32) || t.car_count > std::min(plan.car_room, 32))
                wrong |= 1;
            arena += t.arena_count;
            car += t.car_count;
        }
        if (arena != n || car != active || plan.car_room % 4 ||
            plan.shared != rg::turn_shared_bytes(plan.car_room, plan.arena_room, pads))
            wrong |= 1;
        for (int grid : grids) {
            std::vector<int> seen(n, 0);
            for (int g = 0; g < grid; ++g) {
                const rg::TurnGroup& t = plan.groups[g];
                for (int j = 0; j < t.arena_count; ++j)
                    if (++seen[order[t.arena_first + j]] > 1) wrong |= 2;
            }
        }
    }
    return wrong;
}

}  // extern "C"
