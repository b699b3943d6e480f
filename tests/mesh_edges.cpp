// Triangles that share none to three vertices with one another, for test_mesh_edges.py: built with bounds checks that trap.
#include "rg_mesh.h"

int main() {
    const float v[] = {0, 0, 0, 1000, 0, 0, 0, 1000, 0, 1000, 1000, 0, 0, 0, 1000, 3000, 3000, 0};
    const int32_t idx[] = {0, 1, 2, 0, 1, 2, 2, 1, 0, 1, 3, 2, 0, 1, 4, 0, 5, 3, 3, 5, 4};
    const int64_t n = sizeof(idx) / sizeof(idx[0]);
    const rg::MeshHost h = rg::build_mesh_host(v, 6, idx, n);
    return h.dev_tris.size() == n / 3 ? 0 : 1;
}
