// Division by a number whose reciprocal is at hand, rounded like v / d.
//
// Markstein's correction (P. Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", 1990): with y = RN(1 / d) and q within
// one ulp of v / d, RN(q + y RN(v - d q)) is RN(v / d). The product v y is
// within 1.5 ulp, one correction brings it within one, the second is the
// theorem's. It asks that no remainder underflows and nothing overflows, which
// holds for |v| in [2^-100, 2^100] and |d| in [2^-20, 2^20].
#pragma once

#include <math.h>

#include "frep/frep_math.h"

namespace frep {

FREP_HD float div_by(float v, float d, float y) {
    float q = v * y;
    q = fmaf(fmaf(-d, q, v), y, q);
    return fmaf(fmaf(-d, q, v), y, q);
}
constexpr float DIV_BY_MIN = 0x1p-100f, DIV_BY_MAX = 0x1p100f, DIV_BY_DMIN = 0x1p-20f, DIV_BY_DMAX = 0x1p20f;

}  // namespace frep
