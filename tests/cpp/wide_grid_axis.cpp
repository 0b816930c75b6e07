// ctypes shim over the two forms of wide_grid_axis (bvh_boxes.h) for tests/test_wide_grid_axis.py.
#include "bvh_boxes.h"

extern "C" void grid_axes(float const *lo, float const *hi, double const *step_min, int n, int single, uint32_t *e,
                          float *org, float *inv) {
    for (int k = 0; k < n; k++)
        e[k] = single ? e8g::wide_grid_axis(lo[k], hi[k], step_min[k], e8g::wide_exponent(step_min[k]), org[k], inv[k])
                      : e8g::wide_grid_axis_double(lo[k], hi[k], step_min[k], org[k], inv[k]);
}
