// pado_reg_tables.h -- host-side plan of the register kernel (pado_reg.cuh).
#pragma once

#include <vector>

#include "pado_reg.cuh"

namespace pado {

// Cut of the rows a segment covers on a line: S segments of M rows, neighbours
// sharing d1 rows at the first nd1 joints and d0 at the others.
struct RegCut {
    int M = 0, S = 0, d0 = 0, d1 = 0, nd1 = 0;
    bool even() const { return d0 == 0 && nd1 == 0; }
};
// The cut of `rows` rows into segments of M rows; false when the neighbours
// would have to share more than reg_overlap(M) rows.  even_starts: every overlap
// even.
bool reg_cut(int rows, int M, bool even_starts, RegCut *cut);

// x lines of even length: the swizzled tile moves two rows at a time.  The
// other copies of such a line (fields 8 bytes off a 16-byte boundary) take the
// same cut, so that a result's rounding does not depend on where its field
// lies; M and S are the same with any starts.
inline bool reg_even_starts(int axis, int n) { return axis == 1 && n % 2 == 0; }

// Rows of a line the segments cover.
inline int reg_rows(int n, bool periodic) { return periodic ? n : n - 2 * REG_EDGE; }

// Shortest line the kernel takes: the closure rows and stencils of the two
// ends stay apart.
constexpr int REG_MIN_N = 24;

// A left-hand side's interior on lines of n rows, in extended precision: what
// its operators of all closures and cuts share.
struct RegBand {
    struct M2 {
        long double a, b, c, d;  // row-major
    };
    int n = 0;
    long double c = 1, p1 = 0, p2 = 0;  // A = c L L^T
    std::vector<M2> tk;                 // T^k, k up to the rows the segments cover
    std::vector<long double> u;         // bounded: response of those rows to the y state before them
    RegBand(int n, bool periodic, long double al, long double be);
    static RegBand of(int scheme, int kind, int n, bool periodic);
};

// Fills every table of the launch parameters (not the geometry, pointers and
// copy descriptors) for one operator and cut, and the edge tables of bounded
// lines.  bc1/bcn: closures of the right-hand side; sbc1/sbcn: of the system
// solved (cd06: its init closures for both).
void reg_fill(const RegBand &rb, int scheme, int kind, double dx, bool periodic, int bc1, int bcn, int sbc1, int sbcn,
              const RegCut &cut, RegParams *kp, std::vector<double> *segtab);

// One operator of the staggered scheme.
struct RegStagg {
    int n = 0, nin = 0;         // solved rows, input rows
    bool periodic = false, copy_first = false;
    double alpha = 0.0, a = 0.0, b = 0.0, sign = 0.0;  // interior: band and stencil (taps a, b; sign of RHS_ST_EC / CE)
    const double *lower = nullptr, *diag = nullptr, *upper = nullptr;  // bounded: the left-hand side's rows
    double rows[REG_ROWTAB] = {0};  // bounded: closure rows [2][EDGE][GROUPS][coef, 8 muls]
};
void reg_fill_stagg(const RegStagg &st, const RegCut &cut, RegParams *kp, std::vector<double> *segtab);

}  // namespace pado
