// Host build of the tick's headers for test_host_paths.py: entry points over plain arrays.
#include <vector>

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

// n box queries (lo, hi per box) on a mesh: how many visit other triangles, or in another order, than a scan of all
// triangles in leaf order with the quantized overlap test; `cell` receives the query grid's cell size
int hp_query_boxes(const float* vertices_uu, long long nv, const int* indices, long long ni, const float* boxes, int n,
                   float* cell) {
    using rg::V3;
    const rg::MeshHost h = rg::build_mesh_host(vertices_uu, nv, indices, ni);
    rg::MeshDevice m;
    m.tris = h.dev_tris.data();
    m.tri_count = static_cast<int32_t>(h.dev_tris.size());
    m.quant = h.quant;
    m.grid_lo = h.grid_lo;
    for (int a = 0; a < 3; ++a) m.grid_dims[a] = h.grid_dims[a];
    m.inv_query_cell = 1.0f / h.query_cell;
    m.cell_start = h.cell_start.data();
    m.cell_entries = h.cell_entries.data();
    m.rank_entries = h.rank_entries.data();
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

}  // extern "C"
