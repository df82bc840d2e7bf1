// Line pass instantiations for lines of 2^14 points with non-separable point-wise work (see
// line2.cuh).
#include "line2.cuh"

namespace srwg {
LineFn line2e_get_14(bool cols, int f1, int f2)
{
    return cols ? line2_select<14, true, true>(f1, f2) : line2_select<14, false, true>(f1, f2);
}
}  // namespace srwg
