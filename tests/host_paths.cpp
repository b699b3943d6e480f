// Host build of the tick's headers for test_host_paths.py: entry points over plain arrays.
#include <vector>

#include "rg_tick.cuh"

namespace {
// A mesh's device view over its host tables.
rg::MeshDevice host_view(const rg::MeshHost& h) {
    rg::MeshDevice m;
    m.tris = h.dev_tris.data();
    m.tri_count = static_cast<int32_t>(h.dev_tris.size());
    m.quant = h.quant;
    m.aabb_min = h.aabb_min;
    m.aabb_max = h.aabb_max;
    m.grid_lo = h.grid_lo;
    for (int a = 0; a < 3; ++a) m.grid_dims[a] = h.grid_dims[a];
    m.inv_query_cell = 1.0f / h.query_cell;
    m.cell_start = h.cell_start.data();
    m.cell_entries = h.cell_entries.data();
    m.rank_entries = h.rank_entries.data();
    return m;
}
}  // namespace

extern "C" {

// n boxes against n triangles; out: hit, distance, point (5 floats per case)
void hp_box_triangle(const float* basis, const float* pos, const float* offset, const float* half, const float* tri,
                     float* out, int n) {
    using rg::V3;
    for (int i = 0; i < n; ++i) {
        auto v = [](const float* p, int k) { return V3{p[3 * k], p[3 * k + 1], p[3 * k + 2]}; };
        float d = 0.0f;
        V3 p{0.0f, 0.0f, 0.0f};
        const bool hit = rg::gjk::box_triangle_contact(v(basis, 3 * i), v(basis, 3 * i + 1), v(basis, 3 * i + 2),
                                                       v(pos, i), v(offset, i), v(half, i), v(tri, 3 * i),
                                                       v(tri, 3 * i + 1), v(tri, 3 * i + 2), d, p);
        const float o[5] = {hit ? 1.0f : 0.0f, d, p.x, p.y, p.z};
        memcpy(out + 5 * i, o, sizeof(o));
    }
}

// n boxes against n spheres; out: hit, distance, normal, the four relative / local points (17 floats per case)
void hp_ball_box(const float* basis, const float* pos, const float* offset, const float* half, const float* ball,
                 float* out, int n) {
    using rg::V3;
    for (int i = 0; i < n; ++i) {
        auto v = [](const float* p, int k) { return V3{p[3 * k], p[3 * k + 1], p[3 * k + 2]}; };
        rg::gjk::BallBoxContact c;
        memset(&c, 0, sizeof(c));
        const bool hit = rg::gjk::ball_box_contact(v(basis, 3 * i), v(basis, 3 * i + 1), v(basis, 3 * i + 2), v(pos, i),
                                                   v(offset, i), v(half, i), V3{1.0f, 0.0f, 0.0f},
                                                   V3{0.0f, 1.0f, 0.0f}, V3{0.0f, 0.0f, 1.0f}, v(ball, i),
                                                   1.8249998f, 0.04f, c);
        const V3 vs[5] = {c.normal, c.rel_ball_bt, c.rel_car_bt, c.ball_local_bt, c.car_local_bt};
        out[17 * i] = hit ? 1.0f : 0.0f;
        out[17 * i + 1] = c.distance_bt;
        memcpy(out + 17 * i + 2, vs, sizeof(vs));
    }
}

// n box queries (lo, hi per box) on a mesh: how many visit other triangles, or in another order, than a scan of all
// triangles in leaf order with the quantized overlap test; `cell` receives the query grid's cell size
int hp_query_boxes(const float* vertices_uu, long long nv, const int* indices, long long ni, const float* boxes, int n,
                   float* cell) {
    using rg::V3;
    const rg::MeshHost h = rg::build_mesh_host(vertices_uu, nv, indices, ni);
    const rg::MeshDevice m = host_view(h);
    *cell = h.query_cell;
    int wrong = 0;
    for (int i = 0; i < n; ++i) {
        const float* b = boxes + 6 * i;
        const V3 lo{b[0], b[1], b[2]}, hi{b[3], b[4], b[5]};
        std::vector<int> got, want;
        rg::mesh_query_box(m, lo, hi, [&](const rg::DevTri& t) { got.push_back(static_cast<int>(&t - m.tris)); });
        uint16_t qmin[3], qmax[3];
        rg::quantize_point(m.quant, lo, 0, qmin);
        rg::quantize_point(m.quant, hi, 1, qmax);
        for (int r = 0; r < m.tri_count; ++r) {
            const rg::DevTri& t = m.tris[r];
            bool over = true;
            for (int a = 0; a < 3; ++a) over = over && !(qmin[a] > t.qmax[a] || qmax[a] < t.qmin[a]);
            if (over) want.push_back(r);
        }
        wrong += got != want;
    }
    return wrong;
}

// ---- whole ticks on the host: the parts of a tick in order, one arena after another, one lane per car ------------------
struct HostBatch {
    int32_t envs, max_cars, pad_count;
    const int32_t* counts;
    const uint8_t* teams;
    const rg::CarConfig* cfgs;
    rg::CarState* cars;
    rg::BallState* balls;
    rg::EnvState* env_states;
    rg::PadState* pads;
    rg::WheelRuntime* wheels;
    rg::BallWorldScratch* ball_world;
    rg::Broadphase* broadphase;
    rg::CarWorldScratch* car_world;
    rg::BallCarScratch* ball_car;
    rg::CarCarManifold* pairs;
    const float* pad_pos;
    const uint8_t* pad_big;
    uint64_t kickoff_seed;
};

// `ticks` ticks of every arena under controls [ticks, envs * max_cars] and the default config (report fields after the
// last tick).
void hp_step(const HostBatch* b, const rg_sim_config* cfg, const float* vertices_uu, long long nv, const int* indices,
             long long ni, const rg::CarControls* controls, int ticks) {
    const rg::MeshHost h = rg::build_mesh_host(vertices_uu, nv, indices, ni);
    const rg::MeshDevice m = host_view(h);
    rg::TickConfig tc{};
    tc.tick_dt = cfg->tick_dt;
    tc.gravity_z = cfg->gravity_z;
    tc.ball_radius = cfg->ball_radius;
    tc.ball_mass = cfg->ball_mass;
    tc.ball_drag = cfg->ball_drag;
    tc.ball_drag_scale = rg::ucrt_powf(1.0f - cfg->ball_drag, cfg->tick_dt);
    tc.ball_friction = cfg->ball_friction;
    tc.ball_restitution = cfg->ball_restitution;
    tc.ball_max_speed = cfg->ball_max_speed;
    tc.ball_max_ang_speed = cfg->ball_max_ang_speed;
    tc.goal_base_threshold_y = cfg->goal_base_threshold_y;
    tc.frame_frac = 0.5f;
    tc.enable_scoring = cfg->enable_scoring;
    tc.enable_boost_pads = cfg->enable_boost_pads;
    tc.enable_car_car = cfg->enable_car_car_collisions;
    tc.enable_demos = cfg->enable_demos;
    tc.bump_force_scale = 1.0f;
    tc.bump_cooldown_time = 0.25f;
    tc.kickoff_seed = b->kickoff_seed;
    tc.max_cars = b->max_cars;
    tc.pad_count = b->pad_count;
    tc.car_mass = cfg->car_mass;
    tc.car_max_speed = cfg->car_max_speed;
    tc.car_max_ang_speed = cfg->car_max_ang_speed;
    rg::fill_car_constants(tc);
    tc.arena_friction = cfg->arena_friction;
    tc.arena_restitution = cfg->arena_restitution;
    rg::PadLayout layout{};
    layout.count = b->pad_count;
    for (int p = 0; p < b->pad_count; ++p) {
        layout.pos[p] = rg::V3{b->pad_pos[3 * p], b->pad_pos[3 * p + 1], b->pad_pos[3 * p + 2]};
        layout.is_big[p] = b->pad_big[p];
    }
    const int mc = b->max_cars, slots = mc * (mc - 1) / 2;
    std::vector<rg::CarTickRecord> recs(mc);
    std::vector<rg::CarStage> stages(mc);
    for (int e = 0; e < b->envs; ++e) {
        const int base = e * mc, count = b->counts[e];
        rg::BallState& ball = b->balls[e];
        rg::EnvState& env = b->env_states[e];
        for (int t = 0; t < ticks; ++t) {
            rg::ArenaCars A{};
            A.cars = A.slots = b->cars + base;
            A.wheels = b->wheels + base;
            A.cfgs = b->cfgs + base;
            A.pads = b->pads + static_cast<size_t>(e) * b->pad_count;
            A.controls = controls + static_cast<size_t>(t) * b->envs * mc + base;
            A.teams = b->teams + base;
            A.pairs = b->pairs + static_cast<size_t>(e) * slots;
            A.count = count;
            A.max_cars = mc;
            A.car_base = base;
            rg::ArenaTickSnap snap;
            rg::arena_tick_begin(env, ball, A, tc, snap, tc.kickoff_seed, e);
            for (int p = 0; p < layout.count; ++p) rg::pad_tick_begin(tc, count, A.pads, p);
            for (int i = 0; i < count; ++i) {
                rg::RespawnCtx rc{tc.kickoff_seed, e, env.tick, static_cast<uint32_t>(base + i + 1), A.teams[i]};
                rg::car_tick_pre(A.cars[i], A.controls[i], A.cfgs[i], tc, A.wheels[i], rc, recs[i]);
            }
            for (int i = 0; i < count; ++i) {
                rg::CarStage& st = stages[i];
                rg::car_mesh_stage(A.cars[i], A.cfgs[i], b->car_world[base + i], m, st);
                rg::car_proxy_ball_stage(ball, snap.ball_vel_bt, A.cars[i], A.cfgs[i], tc, recs[i].vel_bt,
                                         recs[i].ang_vel, b->ball_car[base + i], st);
                for (int w = 0; w < 4 && !A.cars[i].is_demoed; ++w) {
                    int met;
                    rg::wheel_mesh_ray_ahead(A.cars[i], A.cfgs[i], m, w, rg::WheelOthers{nullptr, nullptr, 0, i, 0u},
                                             st.wheel_mesh[w], met);
                }
            }
            rg::VehicleSlot slot;  // every vehicle update in the arena's car order
            rg::arena_cars_in_order(rg::OneLane{}, env, ball, b->broadphase[e], tc, m, A, recs.data(), stages.data(),
                                    (1u << count) - 1u, slot);
            rg::arena_tick_finish(env, ball, b->ball_world[e], b->broadphase[e], b->car_world + base,
                                  b->ball_car + base, tc, m, A, recs.data(), snap, stages.data());
            for (int i = 0; i < count; ++i)
                rg::car_tick_post(A.cars[i], stages[i].pre, A.controls[i], A.wheels[i], tc, t + 1 == ticks, A.cfgs[i],
                                  A.pads, layout, stages[i].pads);
            rg::arena_tick_tail(env, ball, A, layout, tc, stages.data());
        }
    }
}

}  // extern "C"
