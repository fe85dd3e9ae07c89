// dnni_est.cu -- TEST INFRASTRUCTURE: host build of the quotient estimates and
// the binning plan of dnni_search.cuh / dnni_plan.h, for tests/test_estimates_host.py.
#include <cstdint>

#include "../../include/dnni.h"
#include "../../terranni_b200/csrc/dnni_search.cuh"
#include "../../terranni_b200/csrc/dnni_plan.h"

using namespace dnni;

// kind 0: floor_div_est(x, u); 1: floor_div_u32(x, u); 2: r2_of32(x, u, cap = v)
extern "C" void est_eval(int kind, const uint32_t* x, const uint32_t* u, const uint32_t* v, int64_t n, int64_t* out) {
    for (int64_t k = 0; k < n; ++k) {
        const float inv = 1.0f / (float)u[k];
        if (kind == 0) out[k] = floor_div_est((int)x[k], (int)u[k], inv);
        else if (kind == 1) out[k] = floor_div_u32(x[k], u[k], inv);
        else out[k] = r2_of32(x[k], (int)u[k], 1.0f / ((float)u[k] * (float)u[k]), (int)v[k]);
    }
}

// The binning plan of n points over a w x h box: rsh, regions, bins.
extern "C" int est_regions(int64_t n, int32_t w, int32_t h, double target, int64_t* out) {
    dnni_workpackage wp{};
    wp.ncols = wp.nrows = 16;
    wp.cell_size = 1;
    TileParams t;
    const char* msg;
    const dnni_status st = plan_geometry(&wp, n, 3, t, &msg);
    if (st) return st;
    const int32_t bb[6] = {0, w - 1, 0, h - 1, 0, 0};
    plan_bins(bb, n, target, t);
    out[0] = t.rsh;
    out[1] = t.bg.nbins >> t.rsh;
    out[2] = t.bg.nbins;
    out[3] = kMaxRegions;
    out[4] = t.band;
    return 0;
}
