// Host build of pointvortex_b200/csrc/pv_log.cuh for the CPU tests (tests/test_log.py).
#include <cstddef>

#include "../../pointvortex_b200/csrc/pv_log.cuh"

extern "C" {
// log_normal() of every value log_is_normal() accepts; returns how many it refused.
size_t pvl_log_many(const double *v, size_t n, double *out) {
    size_t refused = 0;
    for (size_t i = 0; i < n; ++i) {
        if (pvb::log_is_normal(v[i]))
            out[i] = pvb::log_normal(v[i], pvb::kLogTable);
        else
            ++refused;
    }
    return refused;
}
}
