// The tile sweep's plan as its launcher asks for it (ss_tile.cu), for tests/test_tile_limits.py: "" or why it is refused.
#include <string>

#include "ss_tile_plan.hpp"

extern "C" const char *tile_limits_check(int n, int nlev, const int *prp, const int *pci, const int *ipos,
                                         const int *level, int lower, int elem, int lanes, long long device_bytes,
                                         long long *record_bytes) {
    static std::string why;
    const ssg::TileLimits lim = ssg::tile_limits(lanes, device_bytes);
    const ssg::TilePlanHost P =
        ssg::tile_plan_host(n, nlev, prp, pci, ipos, level, lower != 0, elem, lanes, 0,
                            ssg::tile_cluster(ssg::tile_count(n, lanes), lanes), nullptr, &lim);
    if (record_bytes) *record_bytes = P.ok ? P.rec_bytes : 0;
    why = P.ok ? "" : P.why;
    return why.c_str();
}
