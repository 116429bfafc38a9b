// The uniform grid that near-neighbour searches go over (near_tour.cuh).
#pragma once
#include <cmath>
#include <cstdint>

namespace logo {

// Cells of the search grid: about two cities per cell; never more than this.
__host__ __device__ constexpr uint32_t near_cells_max(uint32_t n) { return n / 2 + 64; }

// The cells of the search grid: a coordinate x lies in column (x - x0) * inv,
// truncated.
struct NearGrid {
    int gx, gy;
    float x0, y0, inv;
    float side;  // 1 / inv
};
// Square cells of about two cities for n cities in a w x h box whose corner is
// (x0, y0); a thin box gets fewer, longer ones.
__host__ __device__ inline NearGrid near_grid(uint32_t n, float x0, float y0, float w, float h) {
    NearGrid g{1, 1, x0, y0, 0.f, 0.f};
    const float cap = (float)(n / 2 + 1);
    float side = fmaxf(sqrtf(w / cap * h), fmaxf(w, h) / cap);
    for (int t = 0; t < 64 && side > 0.f; ++t, side *= 1.125f) {
        const float inv = 1.0f / side;
        const int gx = (int)fminf(w * inv, 1.0e8f) + 1, gy = (int)fminf(h * inv, 1.0e8f) + 1;
        if ((uint64_t)gx * (uint64_t)gy <= near_cells_max(n)) {
            g.gx = gx;
            g.gy = gy;
            g.inv = inv;
            g.side = side;
            break;
        }
    }
    return g;
}

}  // namespace logo
