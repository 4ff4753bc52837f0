// The grid of a z-marching product (kuhn25.cuh): tiles of ox x oy owned nodes over the x and y planes, and
// segments of node layers along z, a CTA for each.  Plain C++, so that it can be checked without a GPU.
#pragma once

#include <cstdint>

namespace msfem {

struct ZmarchGrid {
    int tiles_x, tiles_y;
    int seg_len, n_seg;  // node layers of a segment (the last may be shorter), segments
    int64_t ctas() const { return (int64_t)tiles_x * tiles_y * n_seg; }
};

// nx, ny, nz: hexahedra; slots: CTAs resident on the device at once.  The segment count minimises waves x
// steps per CTA: a segment of s layers takes s + 1 steps, the CTAs run in ceil(tiles segments / slots) waves.
inline ZmarchGrid zmarch_grid(int nx, int ny, int nz, int ox, int oy, int64_t slots)
{
    ZmarchGrid g{(nx + ox) / ox, (ny + oy) / oy, nz + 1, 1};
    const int layers = nz + 1;
    const int64_t tiles = (int64_t)g.tiles_x * g.tiles_y;
    int64_t best = -1;
    for (int n_seg = 1; n_seg <= layers; n_seg++) {
        const int len = (layers + n_seg - 1) / n_seg;
        const int segs = (layers + len - 1) / len;
        const int64_t cost = (tiles * segs + slots - 1) / slots * (len + 1);
        if (best < 0 || cost < best) {
            best = cost;
            g.seg_len = len;
            g.n_seg = segs;
        }
    }
    return g;
}

}  // namespace msfem
