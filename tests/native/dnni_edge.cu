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
