// Line passes on pairs of lines (linep.cuh), one unit per (axis, mode) for the run-time schedules
// (-DSRWG_LINEP_COLS=<0|1> -DSRWG_LINEP=<mode>) and one per length for the fixed ones
// (-DSRWG_LINEF_N=<points>, linep_lengths.h).
#include "linep.cuh"
#include "linep_lengths.h"

#define SRWG_CAT3(a, b, c) a##b##_##c
#define SRWG_CAT(a, b, c) SRWG_CAT3(a, b, c)
#define SRWG_CAT2(a, b) a##b
#define SRWG_CATF(a, b) SRWG_CAT2(a, b)

namespace srwg {
// extra: 0 none, 1 the quartic angular term (two transforms), 2 any non-separable work
template <class Z, bool COLS, int MODE> static LineFn pick_extra(int extra)
{
    if (extra == 0) return linep_kernel<Z, COLS, MODE, 0>;
    if constexpr (MODE == 1)
        if (extra == 1) return linep_kernel<Z, COLS, MODE, 1>;
    if constexpr (MODE != 2)
        if (extra == 2) return linep_kernel<Z, COLS, MODE, 2>;
    return nullptr;
}
template <class Z, bool COLS> static LineFn pick(int mode, int extra)
{
    return mode == 2 ? pick_extra<Z, COLS, 2>(extra) : mode == 1 ? pick_extra<Z, COLS, 1>(extra) : pick_extra<Z, COLS, 0>(extra);
}

#ifdef SRWG_LINEF_N
#define SRWG_LINEF_CASE(N, A, B, C, D, T) template <> struct FixedOf<N> { typedef FShape<A, B, C, D, T> Z; };
template <int N> struct FixedOf;
SRWG_LINEF_LENGTHS(SRWG_LINEF_CASE)
LineFn SRWG_CATF(linef_get_, SRWG_LINEF_N)(bool cols, int mode, int extra)
{
    typedef FixedOf<SRWG_LINEF_N>::Z Z;
    static_assert(Z::N() == SRWG_LINEF_N, "schedule");
    return cols ? pick<Z, true>(mode, extra) : pick<Z, false>(mode, extra);
}
SampleFn SRWG_CATF(lines_get_, SRWG_LINEF_N)() { return linep_sample_kernel<FixedOf<SRWG_LINEF_N>::Z>; }
#else
LineFn SRWG_CAT(linep_get_, SRWG_LINEP_COLS, SRWG_LINEP)(int extra)
{
    return pick_extra<PShape, SRWG_LINEP_COLS != 0, SRWG_LINEP>(extra);
}
#if SRWG_LINEP == 2 && SRWG_LINEP_COLS == 0
SampleFn lines_get() { return linep_sample_kernel<PShape>; }
#endif
#endif
}  // namespace srwg
