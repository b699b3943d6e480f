// Host build of the tick's headers for test_host_paths.py: entry points over plain arrays.
#include "rg_tick.cuh"

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

}  // extern "C"
