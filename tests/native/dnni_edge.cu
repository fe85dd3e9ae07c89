// dnni_edge.cu -- TEST INFRASTRUCTURE: host build of the batch plan, for
// tests/test_plan_host.py.
#include <cstdint>

#include "../../include/dnni.h"
#include "../../terranni_b200/csrc/dnni_plan.h"

using namespace dnni;

// A batch of n tiles of ncols x nrows cells each, points[k] points in tile k
// over its own grid: the binning regions listed per tile (strips, superblocks)
// into strips / whole, the tiles' bins into bins, and the most regions of a tile.
extern "C" int edge_batch_regions(int32_t n, const int32_t* ncols, const int32_t* nrows, int32_t cell,
                                  const int64_t* points, double target, int64_t* strips, int64_t* whole, int64_t* bins,
                                  int32_t* max_reg) {
    HostBatch hb;
    for (int k = 0; k < n; ++k) {
        dnni_workpackage wp{};
        wp.ncols = ncols[k];
        wp.nrows = nrows[k];
        wp.cell_size = cell;
        TileParams t;
        const char* msg;
        const dnni_status st = plan_geometry(&wp, points[k], 3, t, &msg);
        if (st) return st;
        const int32_t bb[6] = {INT32_MAX, INT32_MIN, INT32_MAX, INT32_MIN, 0, 0};
        plan_bins(bb, points[k], target, t);
        batch_add(hb, t, 0, 0, -1);
        strips[k] = hb.strip_base[k + 1] - hb.strip_base[k];
        whole[k] = hb.whole_base[k + 1] - hb.whole_base[k];
        bins[k] = t.bg.nbins;
    }
    *max_reg = hb.max_reg;
    return 0;
}

// The far pass's filter for one eighth of a group, as far_search forms it: four
// pixels (px, py relative to the group's corner, active where act) with their
// bounds d2, the group's extent, and a point (relative to the corner): hit.  The
// root is taken low by more than the device's estimate can be.
extern "C" void edge_circle(int64_t n, const int64_t* px, const int64_t* py, const uint8_t* act, const int64_t* d2,
                            const int64_t* ext, const int64_t* qx, const int64_t* qy, uint8_t* hit) {
    for (int64_t k = 0; k < n; ++k) {
        float cx0 = 3e38f, cx1 = -3e38f, cy0 = 3e38f, cy1 = -3e38f;
        int64_t m = 0;
        for (int64_t e = 4 * k; e < 4 * k + 4; ++e) {
            if (!act[e]) continue;
            cx0 = fminf(cx0, (float)px[e]);
            cx1 = fmaxf(cx1, (float)px[e]);
            cy0 = fminf(cy0, (float)py[e]);
            cy1 = fmaxf(cy1, (float)py[e]);
            m = d2[e] > m ? d2[e] : m;
        }
        const float half = far_half(cx1 - cx0, cy1 - cy0, (float)ext[k]);
        const float root = sqrtf((float)m) * (1.0f - 4.0f / (1 << 23));
        hit[k] = far_in_circle((float)qx[k], (float)qy[k], 0.5f * (cx0 + cx1), 0.5f * (cy0 + cy1),
                               far_circle_r2(root, half));
    }
}
