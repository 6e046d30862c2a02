// pado_reg_emul.cu -- TEST ONLY.  Runs the register kernel's phase functions
// (padeops_b200/csrc/pado_reg.cuh) on the CPU, tile by tile, with the
// product's host-side constants (pado_reg_tables.cpp).
#include <cstring>
#include <vector>

#include "../../padeops_b200/csrc/pado_once.h"
#include "../../padeops_b200/csrc/pado_reg_tables.h"

using namespace pado;

namespace {

constexpr int LT = 8;

template <int RK, bool PER, int M, bool EVEN>
int run_mode(const RegParams &kp, int mode)
{
    if (mode == REG_ODD) emulate_reg<RK, PER, M, EVEN, REG_ODD, LT>(kp);
    else if (mode == REG_ROWS || reg_stagg(RK)) emulate_reg<RK, PER, M, EVEN, REG_ROWS, LT>(kp);
    else if constexpr (!reg_stagg(RK)) {
        if (mode == REG_SWZ) emulate_reg<RK, PER, M, EVEN, REG_SWZ, LT>(kp);
        else emulate_reg<RK, PER, M, EVEN, REG_PACK, LT>(kp);
    }
    return 0;
}

template <int RK, int M>
int run_cut(const RegParams &kp, bool per, bool even, int mode)
{
    if (!per) return run_mode<RK, false, M, false>(kp, mode);
    return even ? run_mode<RK, true, M, true>(kp, mode) : run_mode<RK, true, M, false>(kp, mode);
}

template <int RK>
int run_rk(const RegParams &kp, bool per, bool even, int m, int mode)
{
    switch (m) {
    case 8: return run_cut<RK, 8>(kp, per, even, mode);
    case 16: return run_cut<RK, 16>(kp, per, even, mode);
    case 32: return run_cut<RK, 32>(kp, per, even, mode);
    }
    return -1;
}

}  // namespace

// mode: RegMode.  Returns -2 when the line does not cut into segments of m
// rows, -3 when it is too short, else 0.
extern "C" int emul_reg(int scheme, int kind, int n, double dx, int periodic, int bc1, int bcn, int sbc1, int sbcn,
                        int m, int mode, int axis, int out_mode, double alpha, const double *f, double *df, long na,
                        long nb)
{
    if (n < REG_MIN_N) return -3;
    RegCut cut;
    if (!reg_cut(reg_rows(n, periodic != 0), m, reg_even_starts(axis, n), &cut)) return -2;
    RegParams kp;
    std::memset(&kp, 0, sizeof(kp));
    std::vector<double> segtab;
    reg_fill(RegBand::of(scheme, kind, n, periodic != 0), scheme, kind, dx, periodic != 0, bc1, bcn, sbc1, sbcn, cut, &kp, &segtab);
    kp.segtab = segtab.data();
    kp.in = f;
    kp.out = df;
    kp.axis = axis;
    kp.out_mode = out_mode;
    kp.out_alpha = alpha;
    kp.nlines = (long long)na * nb;
    kp.stages = 1;
    if (reg_strided(mode)) {
        kp.odd_rows = (n + 2) / 2 * (LT + 2);
        kp.na = (int)na;
        kp.xblocks = (int)((na + LT - 1) / LT);
        kp.ntiles = (long long)kp.xblocks * nb;
        kp.stride = axis == 2 ? na : na * (long long)nb;
        kp.pstride = axis == 2 ? na * (long long)n : na;
        kp.tile_doubles = mode == REG_ODD ? (2 * kp.odd_rows + 15) / 16 * 16 : n * LT;
    } else {
        kp.ntiles = (kp.nlines + LT - 1) / LT;
        kp.P = n | 1;
        kp.chunks = n / 16;
        kp.tile_doubles = mode == REG_SWZ ? (n + 15) / 16 * 16 * LT : ((kp.P * LT + 15) / 16 * 16);
    }
    switch (rhs_kind_of(scheme, kind)) {
    case RHS_CD06_D1: return run_rk<RHS_CD06_D1>(kp, periodic != 0, cut.even(), m, mode);
    case RHS_CD10_D1: return run_rk<RHS_CD10_D1>(kp, periodic != 0, cut.even(), m, mode);
    case RHS_CD10_D2: return run_rk<RHS_CD10_D2>(kp, periodic != 0, cut.even(), m, mode);
    default: return run_rk<RHS_CF90>(kp, periodic != 0, cut.even(), m, mode);
    }
}

// One operator of the staggered scheme on (n1, nin) lines along z; par: alpha,
// a, b, sign; lhs: lower, diagonal and upper rows; rows: closure rows.
extern "C" int emul_reg_stagg(int rk, int n, int nin, int periodic, int copy_first, const double *par, const double *lhs,
                              const double *rows, int m, int mode, const double *f, double *df, long n1)
{
    if (n < REG_MIN_N) return -3;
    RegCut cut;
    if (!reg_cut(reg_rows(n, periodic != 0), m, false, &cut)) return -2;
    RegStagg st;
    st.n = n;
    st.nin = nin;
    st.periodic = periodic != 0;
    st.copy_first = copy_first != 0;
    st.alpha = par[0];
    st.a = par[1];
    st.b = par[2];
    st.sign = par[3];
    st.lower = lhs;
    st.diag = lhs + n;
    st.upper = lhs + 2 * n;
    if (!st.periodic) std::memcpy(st.rows, rows, sizeof(st.rows));
    RegParams kp;
    std::memset(&kp, 0, sizeof(kp));
    std::vector<double> segtab;
    reg_fill_stagg(st, cut, &kp, &segtab);
    kp.segtab = segtab.data();
    kp.in = f;
    kp.out = df;
    kp.axis = 3;
    kp.nlines = kp.stride = n1;
    kp.stages = 1;
    kp.na = (int)n1;
    kp.xblocks = (int)((n1 + LT - 1) / LT);
    kp.ntiles = kp.xblocks;
    kp.pstride = n1;
    kp.odd_rows = (nin + 2) / 2 * (LT + 2);
    kp.tile_doubles = (2 * kp.odd_rows + 15) / 16 * 16;
    switch (rk) {
    case RHS_ST_EC: return run_rk<RHS_ST_EC>(kp, st.periodic, cut.even(), m, mode);
    case RHS_ST_CE: return run_rk<RHS_ST_CE>(kp, st.periodic, cut.even(), m, mode);
    case RHS_ST_D1: return run_rk<RHS_ST_D1>(kp, st.periodic, cut.even(), m, mode);
    default: return run_rk<RHS_ST_D2>(kp, st.periodic, cut.even(), m, mode);
    }
}

// Calls of one kernel on device dev[i], whose runtime would answer answer[i]:
// what each call got, and whether the runtime was asked.
extern "C" void emul_once_per_device(int calls, const int *dev, const int *answer, int *got, int *asked)
{
    OncePerDevice<const void *, int> once;
    for (int i = 0; i < calls; ++i) {
        asked[i] = 0;
        got[i] = once.get(nullptr, dev[i], [&] {
            asked[i] = 1;
            return answer[i];
        });
    }
}
