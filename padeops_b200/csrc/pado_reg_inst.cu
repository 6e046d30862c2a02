// pado_reg_inst.cu -- instantiations of the register kernel for one stencil
// and segment length.  The library compiles this file once per pair, with
// -DPADO_RK=0..7 (cd06 d1, cd10 d1, cd10 d2, cf90; the staggered scheme's
// RHS_ST_*, along z only) and -DPADO_RM=8, 16 or 32;
// each defines the entry point pick_reg_rkN_M of pado_internal.h.
#include "pado_internal.h"

#if !defined(PADO_RK) || !defined(PADO_RM)
#error "compile with -DPADO_RK=<stencil 0..7> -DPADO_RM=<rows per segment>"
#endif
#define PADO_CAT4(a, b, c, d) a##b##c##d
#define PADO_CAT(a, b, c, d) PADO_CAT4(a, b, c, d)

namespace pado {

namespace {

template <bool PER, bool EVEN>
RegFn pick(int mode, int lines)
{
    constexpr int RK = PADO_RK, M = PADO_RM;
    if (mode == REG_ROWS) {
        if (lines == 32) return reg_kernel<RK, PER, M, EVEN, REG_ROWS, 32>;
        return lines == 16 ? reg_kernel<RK, PER, M, EVEN, REG_ROWS, 16> : reg_kernel<RK, PER, M, EVEN, REG_ROWS, 8>;
    }
    if (mode == REG_ODD) {
        if (lines == 32) return reg_kernel<RK, PER, M, EVEN, REG_ODD, 32>;
        return lines == 16 ? reg_kernel<RK, PER, M, EVEN, REG_ODD, 16> : reg_kernel<RK, PER, M, EVEN, REG_ODD, 8>;
    }
    if constexpr (reg_stagg(RK)) return nullptr;
    else if (mode == REG_SWZ)
        return lines == 16 ? reg_kernel<RK, PER, M, EVEN, REG_SWZ, 16> : reg_kernel<RK, PER, M, EVEN, REG_SWZ, 8>;
    else return lines == 16 ? reg_kernel<RK, PER, M, EVEN, REG_PACK, 16> : reg_kernel<RK, PER, M, EVEN, REG_PACK, 8>;
}

}  // namespace

RegFn PADO_CAT(pick_reg_rk, PADO_RK, _, PADO_RM)(bool per, bool even, int mode, int lines)
{
    if (!per) return pick<false, false>(mode, lines);
    return even ? pick<true, true>(mode, lines) : pick<true, false>(mode, lines);
}

}  // namespace pado
