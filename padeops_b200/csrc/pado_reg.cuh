// pado_reg.cuh -- the register kernel: one pass over shared memory per tile,
// the whole solve of a segment held in one thread's registers.
//
// Away from the line ends every left-hand side of this library is the
// symmetric band A = c L L^T, with L = 1 + p1 E^-1 + p2 E^-2 (E: shift by one
// row; Wiener-Hopf factors of the band's symbol, |roots| < 1), so the solve is
// two constant-coefficient recurrences,
//
//   y_i = r_i / c - p1 y_{i-1} - p2 y_{i-2}       x_i = y_i - p1 x_{i+1} - p2 x_{i+2},
//
// on cyclic lines exactly (a cyclic band is the product of its cyclic
// factors), on bounded lines for the rows [EDGE, n - EDGE).  A line is cut
// into S segments of M rows (neighbours overlap by a few rows when
// S M exceeds the rows to cover); thread (l, s) holds the M rows of segment s
// of line l in registers and never writes them to memory before the result:
//
//   sweep   stencil and both recurrences from zero states; publishes the y
//           state its successor starts from                        (barrier)
//   link    incoming y state P: T^k-weighted sum over the W segments before;
//           publishes the x state its predecessor starts from      (barrier)
//   close   incoming x state Q: the same over the W segments after
//   out     x_i = x_i(local) + W_i P + V_i Q, straight to df
//
// W_i, V_i (responses of a segment's rows to a unit incoming state) and T^k
// (the recurrence's transfer over a segment) are the same for every segment:
// constants of the launch.  The windows W end where T^k falls below half a
// unit of rounding.
//
// Bounded lines: the EDGE closure rows of each end are solved as a dense
// block.  With zero states at both ends, close leaves the rows next to each
// block known up to four numbers per line -- the y state entering row EDGE
// and the x state entering from row n - EDGE -- which the two blocks then
// fix (edge); every segment adds their effect through its own 2x2 tables.
//
// The cf90 filter solves for d = x - f instead of x: A d = (B - A) f, where
// B - A is the small high-pass part (an eighth difference inside, times
// 5e-6), so the near-singular A (condition number near 2000) amplifies the
// rounding of d and not that of f; f is added when d is complete.
//
// What bounds it: HBM, at 82-96% of the measured copy rate (6448 GB/s) for the
// derivatives of 512-row lines and 81-87% for cf90.  Per point the kernel issues the stencil (5
// to 10 FP64), 4 recurrence and 4 correction FMAs, 1 + 2 H / M shared loads (H
// the stencil's half width) and one store -- 31 (cd10 d1) to 56 (bounded cf90)
// instructions in all -- against 67 to 90 of the streaming kernel, which keeps
// the line in shared memory and passes over it four times.  B200, 512^3, x + y
// + z, streaming kernel -> this kernel: cd10 d1 1929 -> 1057 us, cd10 d2 1985
// -> 1106 us, cf90 2319 -> 1145 us; 1024x512x256 with walls in z: cd06 1664 ->
// 1107 us, cd10 d1 1999 -> 1099 us.
#pragma once

#include <cuda.h>
#include <vector_types.h>

#include <vector>

#include "pado_kernels.cuh"
#include "pado_stream.cuh"

namespace pado {

constexpr int REG_MAXM = 32;      // longest segment
constexpr int REG_MAXS = 64;      // most segments per line
constexpr int REG_EDGE = 4;       // closure rows solved as a block at each end
// Most rows two neighbouring segments of M share: with 8 of 32 every line of
// 104 rows or more between its closure blocks (112 points with walls) cuts into
// 32s, and some shorter ones (walls, along y: cd06 of 99 points 5100 -> 5660
// GB/s, cd10 d2 of 64 points 4820 -> 5780; with 4 such lines took 16s).
PADO_HD constexpr int reg_overlap(int M) { return M >= 32 ? 8 : 4; }
constexpr int REG_SEGTAB = 12;    // doubles per segment of the edge tables
// Closure rows of the staggered scheme, as its right-hand sides group them:
// up to 3 groups coef * (sum of mul * the 8 input rows next to the wall)
constexpr int REG_GROUPS = 3, REG_ROWTAB = 2 * REG_EDGE * REG_GROUPS * 9;
PADO_HD constexpr bool reg_stagg(int rk) { return rk >= RHS_ST_EC; }
PADO_HD constexpr int reg_edge_table(int rk, bool periodic, int S)
{
    return periodic ? 0 : S * REG_SEGTAB + (reg_stagg(rk) ? REG_ROWTAB : 0);
}

// How a tile of lines reaches and leaves shared memory.
enum RegMode {
    REG_ROWS = 0,   // strided lines: [row][L] tile (tensor copies, or per-element copies); results stored from registers
    REG_SWZ = 1,    // x lines: 16-row chunks [chunk][L][16] with the 128-byte swizzle, tensor copies in and out
    REG_ODD = 3,    // strided lines an odd number of elements apart: as REG_ROWS, the tile's even and odd rows copied
                    // apart (each 16-byte aligned), [2][rows][L + 2]
    REG_PACK = 2    // x lines of odd extent: [L][n], one bulk copy of the tile's span in and out; of any extent and
                    // alignment (async_copy): [L][P], P odd, per-element copies
};

PADO_HD constexpr bool reg_strided(int mode) { return mode == REG_ROWS || mode == REG_ODD; }

struct alignas(64) RegParams {
    CUtensorMap tin, tout;      // tensor copies (x lines: whole 16-row chunks)
    CUtensorMap tin2, tout2;    // x lines: the last, partial chunk
    const double *in;
    double *out;
    const double *segtab;       // bounded lines: [S][REG_SEGTAB] (staggered: then [2][EDGE][GROUPS][9], coef and muls)
    int *status;
    long long ntiles, nlines, stride, pstride;
    double out_alpha;
    int n, S, W, na, xblocks, axis, out_mode;
    int nin;                    // rows of the input (n but for the staggered scheme's cells and edges)
    int copy_first;             // the result's last row repeats its first (cyclic edges)
    int async_copy;             // REG_ROWS, REG_PACK: per-element copies
    int chunks;                 // REG_SWZ: whole chunks per line
    int odd_rows;               // REG_ODD: doubles from the even rows' part of a tile to the odd rows'
    int stages, tile_doubles, nbox, box_rows, P;
    int d0, d1, nd1;            // overlap at joint j (between segments j - 1 and j): d1 for 1 <= j <= nd1, else d0
    int cyc;                    // cyclic lines: the states pass round the line more than once (wrap)
    int bc1, bcn;
    double np1, np2;            // -p1, -p2
    double taps[5];             // interior stencil / c
    double phi[3][4];           // T^(M - d0), T^(M - d1), T^M (joint 0 of a cyclic line), row-major
    double wrap[4];             // (1 - T^n)^-1
    double w[REG_MAXM][2];      // response of row i to P
    double v[REG_MAXM][2];      // response of row i to Q
    // bounded lines, [0] left end, [1] right end
    double ctaps[16];           // RhsCoef::c of the closure rows
    double dtaps[2][REG_EDGE][8];  // cf90: rows of B - A on the 8 rows next to the wall
    double fr[2][2][REG_EDGE], fx[2][2][2];  // end state = fr r + fx (the two interior rows next to the block)
    double kinv[4][4];          // both ends together: (1 - K)^-1
    // closure rows, eliminated from the wall: x = xr r (its row's and those nearer the wall) + xx (the next two x inwards);
    // cf90's, solved: x = xr r + xx (the two interior rows)
    double xr[2][REG_EDGE][REG_EDGE], xx[2][REG_EDGE][2];
};
static_assert(sizeof(RegParams) <= 4096, "launch parameters");

// Shared-memory layout, offsets in doubles from a 1024-byte aligned base.
struct RegLayout {
    size_t tiles, ys, xs, edge, segtab, bars, total;
};
// doubles per line of the edge area: r (2 x EDGE), f (2 x EDGE), end states (4), last local rows (2)
constexpr int REG_EDGE_DOUBLES = 4 * REG_EDGE + 6;
PADO_HD PADO_INLINE RegLayout reg_layout(int L, int S, int stages, int tile_doubles, int edge_table)
{
    RegLayout o;
    o.tiles = 0;
    o.ys = (size_t)stages * tile_doubles;
    o.xs = o.ys + (size_t)S * L * 2;
    o.edge = o.xs + (size_t)S * L * 2;
    o.segtab = o.edge + (edge_table ? (size_t)L * REG_EDGE_DOUBLES : 0);
    o.bars = o.segtab + edge_table;
    o.total = o.bars + 2;
    return o;
}
PADO_HD PADO_INLINE size_t reg_smem_bytes(int L, int S, int stages, int tile_doubles, int edge_table)
{
    return reg_layout(L, S, stages, tile_doubles, edge_table).total * sizeof(double) + 1024;
}

struct RegSmem {
    double *tile;   // the buffer of this tile
    int first;      // REG_ODD: parity of the tile's first row in the field
    double2 *ys;    // [S][L] y state each segment hands on
    double2 *xs;    // [S][L] x state each segment hands back
    double *edge;   // [REG_EDGE_DOUBLES][L]
    const double *segtab;
};

// Rows of one line in a tile whose rows lie RS doubles apart: the segment's
// rows and the halo on either side, which wraps round a cyclic line (period
// n).  Staggered stencils (RK) centre row i of a segment on the first of its
// two nearest points: edge i for cell i, cell i - 1 for edge i.  Edge fields
// hold one row past the period, which is read and not its repeat.
template <int RS, int RK>
struct RowsAt {
    static constexpr int SHIFT = RK == RHS_ST_CE ? -1 : 0;
    static constexpr int LOW = RK == RHS_ST_CE ? 1 : 0;                      // rows below: wrapped at the start
    static constexpr int HIGH = RK == RHS_ST_EC || RK == RHS_ST_CE ? 1 : 0;  // rows from M + HIGH: at the end
    const double *p, *lo, *hi;
    PADO_HD PADO_INLINE RowsAt(const double *line, int n, int start, int m, bool cyclic)
    {
        p = line + (long long)(start + SHIFT) * RS;
        lo = cyclic && start == 0 ? p + (long long)n * RS : p;
        hi = cyclic && start + m == n ? p - (long long)n * RS : p;
    }
    // row k of the segment, k in [-H, M + H) known at compile time
    template <int M>
    PADO_HD PADO_INLINE double get(int k) const
    {
        return k < LOW ? lo[k * RS] : (k < M + HIGH ? p[k * RS] : hi[k * RS]);
    }
};

// The same where a tile's rows of either parity lie apart (REG_ODD): rows r of
// the tile at par[r & 1] + (r >> 1) (LT + 2).
template <int LT, int RK>
struct OddAt {
    static constexpr int RS = LT + 2;
    static constexpr int SHIFT = RowsAt<1, RK>::SHIFT, LOW = RowsAt<1, RK>::LOW, HIGH = RowsAt<1, RK>::HIGH;
    const double *p[2], *lo[2], *hi[2];  // rows of even and odd k
    PADO_HD PADO_INLINE static const double *place(const double *const (&par)[2], int r)
    {
        return (r & 1 ? par[1] : par[0]) + (r >> 1) * RS;  // r may be negative: floor
    }
    PADO_HD PADO_INLINE OddAt(const double *const (&par)[2], int n, int start, int m, bool cyclic)
    {
        const int r = start + SHIFT, rl = cyclic && start == 0 ? r + n : r, rh = cyclic && start + m == n ? r - n : r;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            p[k] = place(par, r + k);
            lo[k] = place(par, rl + k);
            hi[k] = place(par, rh + k);
        }
    }
    template <int M>
    PADO_HD PADO_INLINE double get(int k) const
    {
        if (k & 1) return (k < LOW ? lo[1] : (k < M + HIGH ? p[1] : hi[1]))[(k >> 1) * RS];
        return (k < LOW ? lo[0] : (k < M + HIGH ? p[0] : hi[0]))[(k >> 1) * RS];
    }
};

// The same in the swizzled x-line tile: 16-row chunks [chunk][LT][16], the
// 16-byte unit u of line l at unit u ^ (l & 7).  Segments start on even rows.
// The swizzle repeats every 8 units, so the places of the segment's first 8
// units give all the others by constant distances.
template <int LT>
struct SwzAt {
    static constexpr int CHUNK = LT * 16;
    const double *base;  // line l of chunk 0
    int x7, q, qlo, qhi; // (l & 7), first unit of the segment, and of its halos
    int off[8];          // places of units q .. q + 7
    PADO_HD PADO_INLINE SwzAt(const double *tile, int l, int n, int start, int m, bool cyclic)
    {
        base = tile + l * 16;
        x7 = l & 7;
        q = start >> 1;
        qlo = cyclic && start == 0 ? q + (n >> 1) : q;
        qhi = cyclic && start + m == n ? q - (n >> 1) : q;
#pragma unroll
        for (int j = 0; j < 8; ++j) off[j] = place(q + j);
    }
    PADO_HD PADO_INLINE int place(int u) const { return (u >> 3) * CHUNK + (((u & 7) ^ x7) << 1); }
    // unit k / 2 of the segment, k in [0, M) even and known at compile time
    PADO_HD PADO_INLINE double *unit(int k) const
    {
        return const_cast<double *>(base) + off[(k >> 1) & 7] + (k >> 4) * CHUNK;
    }
    template <int M>
    PADO_HD PADO_INLINE double2 get2(int k) const  // rows k, k + 1 (k even, known at compile time)
    {
        const double *p = k < 0 ? base + place(qlo + (k >> 1)) : (k < M ? unit(k) : base + place(qhi + (k >> 1)));
        return *reinterpret_cast<const double2 *>(p);
    }
};

// Per-thread state of one segment.
template <int M>
struct RegThread {
    double x[M];
    double2 xc;  // state handed back
    double2 P, Q;
};

template <int RK, bool PER, int M, bool EVEN>
struct RegLine {
    static constexpr int H = RK == RHS_CD06_D1 || reg_stagg(RK) ? 2 : (RK == RHS_CF90 ? 4 : 3);
    static constexpr bool TRI = RK == RHS_CD06_D1 || reg_stagg(RK);
    static constexpr bool DIFF = RK == RHS_CF90;
    using Th = RegThread<M>;

    PADO_HD PADO_INLINE static int overlap(const RegParams &kp, int joint)
    {
        if (EVEN) return 0;
        return joint < 1 || joint >= kp.S ? 0 : (joint <= kp.nd1 ? kp.d1 : kp.d0);
    }
    PADO_HD PADO_INLINE static int start(const RegParams &kp, int s)
    {
        if (EVEN) return s * M;
        const int e = s < kp.nd1 ? s : kp.nd1;  // joints 1..s: e with d1, the rest with d0
        return (PER ? 0 : REG_EDGE) + s * M - e * kp.d1 - (s - e) * kp.d0;
    }
    // T a: the state a carried across a joint, plus b
    PADO_HD PADO_INLINE static double2 carry(const double *t, double2 a, double2 b)
    {
        if (TRI) {
            b.x = fma(t[0], a.x, b.x);
            return b;
        }
        double2 r;
        r.x = fma(t[0], a.x, fma(t[1], a.y, b.x));
        r.y = fma(t[2], a.x, fma(t[3], a.y, b.y));
        return r;
    }

    // The state a carried across a joint, plus b.
    PADO_HD PADO_INLINE static double2 cross(const RegParams &kp, int joint, double2 a, double2 b)
    {
        if (EVEN || joint > kp.nd1) return carry(kp.phi[0], a, b);
        if (PER && joint == 0) return carry(kp.phi[2], a, b);
        return carry(kp.phi[1], a, b);
    }

    // Stencil and both recurrences with zero incoming states.  f: rows -H ..
    // M + H - 1 of the segment; od, op: rows shared with the next and the
    // previous segment.  again(i): f at row i once more (DIFF).  ys, xs: where
    // the states the neighbours start from go, taken on the way (a store under
    // a predicate is two instructions a row; held in registers they are five).
    template <class Load, class Again>
    PADO_HD PADO_INLINE static void sweep(const RegParams &kp, Th &t, int od, int op, const Load &load,
                                          const Again &again, double2 *ys, double2 *xs, double2 &last)
    {
        constexpr int OV = reg_overlap(M);
        double win[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) win[k] = 0.0;
        double f[M + 2 * H];
        load(f);
        double2 y;
        y.x = y.y = 0.0;
#pragma unroll
        for (int i = 0; i < M; ++i) {
#pragma unroll
            for (int o = -H; o <= H; ++o) win[4 + o] = f[i + H + o];
            double r = rhs_interior_fma(RK, PER, kp.taps, win);
            if (!TRI && i > 1) r = fma(kp.np2, y.y, r);
            if (i > 0) r = fma(kp.np1, y.x, r);
            t.x[i] = r;
            y.y = y.x;
            y.x = r;
            if (EVEN ? i == M - 1 : (i >= M - 1 - OV && i == M - 1 - od)) *ys = y;
        }
        double2 x;
        x.x = x.y = 0.0;
#pragma unroll
        for (int i = M - 1; i >= 0; --i) {
#ifdef __CUDA_ARCH__
            // no load of f moves up past here: all of the segment's would, and
            // spill 25 registers (cf90 on 512^3, x + y + z: 1326 us with the
            // spills, 1129 us without)
            if (DIFF && (i + 1) % 8 == 0) __syncwarp(__activemask());
#endif
            double d = t.x[i];
            if (!TRI && i < M - 2) d = fma(kp.np2, x.y, d);
            if (i < M - 1) d = fma(kp.np1, x.x, d);
            t.x[i] = DIFF ? d + again(i) : d;
            x.y = x.x;
            x.x = d;
            if (i == M - 2) last = x;
            if (!EVEN && i <= OV && i == op) *xs = x;
        }
        if (EVEN) t.xc = x;
    }

    // Incoming y state of segment s, and its x state as the predecessor
    // needs it (complete but for Q).
    PADO_HD PADO_INLINE static void link(const RegParams &kp, const RegSmem &sm, Th &t, int L, int l, int s, int op)
    {
        double2 a;
        a.x = a.y = 0.0;
        const int S = kp.S;
        int k = PER ? kp.W : (kp.W < s ? kp.W : s);
        int j = s - k;
        if (PER && j < 0) j += S;
        for (; k > 0; --k) {
            const double2 y = sm.ys[j * L + l];
            ++j;
            if (PER && j == S) j = 0;
            a = cross(kp, j, a, y);
        }
        if (PER && kp.cyc) {
            double2 z;
            z.x = z.y = 0.0;
            a = carry(kp.wrap, a, z);
        }
        t.P = a;
        if (!EVEN) t.xc = sm.xs[s * L + l];
        const double *w = kp.w[EVEN ? 0 : op];
        if (TRI) {
            t.xc.x = fma(w[0], a.x, t.xc.x);
        } else {
            t.xc.x = fma(w[0], a.x, fma(w[1], a.y, t.xc.x));
            t.xc.y = fma(w[2], a.x, fma(w[3], a.y, t.xc.y));
        }
    }

    // Incoming x state of segment s.
    PADO_HD PADO_INLINE static void close(const RegParams &kp, const RegSmem &sm, Th &t, int L, int l, int s)
    {
        double2 a;
        a.x = a.y = 0.0;
        const int S = kp.S;
        int k = PER ? kp.W : (kp.W < S - 1 - s ? kp.W : S - 1 - s);
        int j = s + k;
        if (PER && j >= S) j -= S;
        for (; k > 0; --k) {
            a = cross(kp, j, a, sm.xs[j * L + l]);
            --j;
            if (PER && j < 0) j = S - 1;
        }
        if (PER && kp.cyc) {
            double2 z;
            z.x = z.y = 0.0;
            a = carry(kp.wrap, a, z);
        }
        t.Q = a;
    }

    // Row i's correction for the incoming states.
    PADO_HD PADO_INLINE static double corrected(const RegParams &kp, const Th &t, int i, double x)
    {
        if (TRI) return fma(kp.w[i][0], t.P.x, fma(kp.v[i][0], t.Q.x, x));
        return fma(kp.w[i][0], t.P.x,
                   fma(kp.w[i][1], t.P.y, fma(kp.v[i][0], t.Q.x, fma(kp.v[i][1], t.Q.y, x))));
    }

    // ---- bounded lines ------------------------------------------------------
    PADO_HD PADO_INLINE static double *edge_r(const RegSmem &sm, int L, int l, int side)
    {
        return sm.edge + (side * REG_EDGE) * L + l;
    }
    PADO_HD PADO_INLINE static double *edge_f(const RegSmem &sm, int L, int l, int side)
    {
        return sm.edge + ((2 + side) * REG_EDGE) * L + l;
    }
    PADO_HD PADO_INLINE static double *edge_z(const RegSmem &sm, int L, int l) { return sm.edge + 4 * REG_EDGE * L + l; }

    // Right-hand sides of the closure rows of one end; g: the 8 rows next to
    // the wall, in line order.
    template <int SIDE>
    PADO_HD PADO_INLINE static void edge_rhs(const RegParams &kp, const RegSmem &sm, int L, int l, const double (&g)[8])
    {
        double *r = edge_r(sm, L, l, SIDE);
        if (DIFF) {
            double *f = edge_f(sm, L, l, SIDE);
#pragma unroll
            for (int i = 0; i < REG_EDGE; ++i) {
                double a = 0.0;
#pragma unroll
                for (int j = 0; j < 8; ++j) a = fma(kp.dtaps[SIDE][i][j], g[j], a);
                r[i * L] = a;
                f[i * L] = g[SIDE ? 4 + i : i];
            }
            return;
        }
        if constexpr (reg_stagg(RK)) {
            const double *c = sm.segtab + kp.S * REG_SEGTAB + SIDE * (REG_ROWTAB / 2);
#pragma unroll
            for (int i = 0; i < REG_EDGE; ++i) {
                double a = 0.0;
#pragma unroll
                for (int q = 0; q < REG_GROUPS; ++q) {
                    const double *m = c + (i * REG_GROUPS + q) * 9;
                    double b = 0.0;
#pragma unroll
                    for (int j = 0; j < 8; ++j) b = fma(m[1 + j], g[j], b);
                    a = fma(m[0], b, a);
                }
                r[i * L] = a;
            }
            return;
        }
        // a line of 16 rows whose first or last 8 are g: the closure rows
        // round like the reference's expressions
        double v[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            v[j] = g[j];
            v[8 + j] = g[j];
        }
        constexpr int CR = RK == RHS_CD06_D1 || RK == RHS_CD10_D2 ? 3 : 4;
#pragma unroll
        for (int i = 0; i < REG_EDGE; ++i) {
            const int row = SIDE ? 12 + i : i;
            const bool inside = SIDE ? i < REG_EDGE - CR : i >= CR;
            double a;
            if (inside) {
                double w[9];
#pragma unroll
                for (int k = 0; k < 9; ++k) w[k] = row + k - 4 >= 0 && row + k - 4 < 16 ? v[row + k - 4] : 0.0;
                a = rhs_interior(RK, 0, kp.ctaps, w);
            } else {
                a = rhs_closure_row(RK, kp.ctaps, v, 1, 16, row, kp.bc1, kp.bcn);
            }
            r[i * L] = a;
        }
    }

    // What one end's block makes of its right-hand sides and of the two
    // interior rows next to it (known but for the end states): b of
    // z = b + K z.
    template <int SIDE>
    PADO_HD PADO_INLINE static void edge_state(const RegParams &kp, const RegSmem &sm, int L, int l, double2 x)
    {
        const double *r = edge_r(sm, L, l, SIDE);
        double *z = edge_z(sm, L, l) + (2 * SIDE) * L;
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            double b = fma(kp.fx[SIDE][a][0], x.x, kp.fx[SIDE][a][1] * x.y);
#pragma unroll
            for (int j = 0; j < REG_EDGE; ++j) b = fma(kp.fr[SIDE][a][j], r[j * L], b);
            z[a * L] = b;
        }
    }
    // The rows next to the blocks, the end states left out: first two rows of
    // segment 0, last two rows of segment S - 1 (whose Q is then zero).
    PADO_HD PADO_INLINE static double2 next_left(const RegParams &kp, const Th &t)
    {
        double2 x;
        x.x = fma(kp.v[0][0], t.Q.x, fma(kp.v[0][1], t.Q.y, t.xc.x));
        x.y = fma(kp.v[1][0], t.Q.x, fma(kp.v[1][1], t.Q.y, t.xc.y));
        return x;
    }
    PADO_HD PADO_INLINE static double2 next_right(const RegParams &kp, const Th &t, double2 last)
    {
        double2 x;
        x.x = fma(kp.w[M - 2][0], t.P.x, fma(kp.w[M - 2][1], t.P.y, last.x));
        x.y = fma(kp.w[M - 1][0], t.P.x, fma(kp.w[M - 1][1], t.P.y, last.y));
        return x;
    }
    // Adds the end states to a segment's incoming ones.
    PADO_HD PADO_INLINE static void edge_add(const RegParams &kp, const RegSmem &sm, Th &t, int L, int l, int s)
    {
        if (s > kp.W && kp.S - 1 - s > kp.W) return;  // out of both ends' reach
        const double *b = edge_z(sm, L, l);
        double z[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            z[a] = kp.kinv[a][0] * b[0];
#pragma unroll
            for (int j = 1; j < 4; ++j) z[a] = fma(kp.kinv[a][j], b[j * L], z[a]);
        }
        const double *g = sm.segtab + s * REG_SEGTAB;
        t.P.x = fma(g[0], z[0], fma(g[1], z[1], t.P.x));
        t.P.y = fma(g[2], z[0], fma(g[3], z[1], t.P.y));
        t.Q.x = fma(g[4], z[0], fma(g[5], z[1], fma(g[8], z[2], fma(g[9], z[3], t.Q.x))));
        t.Q.y = fma(g[6], z[0], fma(g[7], z[1], fma(g[10], z[2], fma(g[11], z[3], t.Q.y))));
    }
    // x of the closure rows of one end, from the two interior rows next to it:
    // substitution towards the wall.  (As a product with the block's inverse,
    // every row of it from all four right-hand sides, the wall row's error was
    // up to 1.4 times an elimination's: it takes its neighbours' with weights
    // of 3 and 11.)  The filter's rows are that product: what it solves for is
    // small beside f, to which it is then added, and the chain of four rows
    // spills 8 bytes there (1024 rows along y and z, 220 -> 227 us).
    template <int SIDE>
    PADO_HD PADO_INLINE static void edge_rows(const RegParams &kp, const RegSmem &sm, int L, int l, double2 x,
                                              double (&out)[REG_EDGE])
    {
        const double *r = edge_r(sm, L, l, SIDE);
        if (DIFF) {
#pragma unroll
            for (int i = 0; i < REG_EDGE; ++i) {
                double a = fma(kp.xx[SIDE][i][0], x.x, kp.xx[SIDE][i][1] * x.y);
#pragma unroll
                for (int j = 0; j < REG_EDGE; ++j) a = fma(kp.xr[SIDE][i][j], r[j * L], a);
                out[i] = a + edge_f(sm, L, l, SIDE)[i * L];
            }
            return;
        }
#pragma unroll
        for (int k = REG_EDGE - 1; k >= 0; --k) {  // k-th row from the wall
            const int i = SIDE ? REG_EDGE - 1 - k : k;
            double a = fma(kp.xx[SIDE][i][0], x.x, kp.xx[SIDE][i][1] * x.y);
#pragma unroll
            for (int j = 0; j <= k; ++j) {
                const int c = SIDE ? REG_EDGE - 1 - j : j;
                a = fma(kp.xr[SIDE][i][c], r[c * L], a);
            }
            out[i] = a;
            if (SIDE) {
                x.x = x.y;
                x.y = a;
            } else {
                x.y = x.x;
                x.x = a;
            }
        }
    }
    // The rows next to the blocks, complete.
    PADO_HD PADO_INLINE static double2 full_left(const RegParams &kp, const Th &t, double2 xc)
    {
        // xc holds the local rows 0 and 1 plus their response to the P that link knew (zero)
        double2 x;
        x.x = corrected(kp, t, 0, xc.x);
        x.y = corrected(kp, t, 1, xc.y);
        return x;
    }
    PADO_HD PADO_INLINE static double2 full_right(const RegParams &kp, const Th &t, double2 last)
    {
        double2 x;
        x.x = corrected(kp, t, M - 2, last.x);
        x.y = corrected(kp, t, M - 1, last.y);
        return x;
    }
};

// Line l of tile t: its first element in the field (REG_ROWS: row 0 of line
// x0 + l of plane p) and whether it exists.
PADO_HD PADO_INLINE void reg_origin(const RegParams &kp, int LT, long long t, long long *x0, long long *p)
{
    if (kp.axis == 1) {
        *x0 = t * LT;
        *p = 0;
    } else {
        const unsigned tu = (unsigned)t, xb = (unsigned)kp.xblocks, q = tu / xb;
        *x0 = (long long)(tu - q * xb) * LT;
        *p = q;
    }
}

// Row i of a segment to its place: rows the predecessor also holds are its own.
template <int RK, bool PER, int M, bool EVEN, int MODE, int LT>
struct RegOut {
    using RL = RegLine<RK, PER, M, EVEN>;
    using Th = RegThread<M>;

    // strided lines: straight to df, in the launch's output mode
    PADO_HD PADO_INLINE static void rows(const RegParams &kp, const Th &t, double *dst, int op)
    {
        if (kp.out_mode == OUT_STORE) {
#pragma unroll
            for (int i = 0; i < M; ++i) {
                const double x = RL::corrected(kp, t, i, t.x[i]);
                if (EVEN || i >= reg_overlap(M) || i >= op) dst[i * kp.stride] = x;
            }
            return;
        }
        // df's values (already on their way to L2, reg_prefetch) are read 8 rows ahead
        const bool acc = kp.out_mode == OUT_ACC;
        double old[2][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) old[0][i] = acc ? dst[i * kp.stride] : 0.0;
#pragma unroll
        for (int c = 0; c < M; c += 8) {
            if (c + 8 < M) {
#pragma unroll
                for (int i = 0; i < 8; ++i) old[(c / 8 + 1) & 1][i] = acc ? dst[(c + 8 + i) * kp.stride] : 0.0;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const double x = RL::corrected(kp, t, c + i, t.x[c + i]);
                if (EVEN || c + i >= reg_overlap(M) || c + i >= op)
                    dst[(c + i) * kp.stride] = fma(kp.out_alpha, x, old[(c / 8) & 1][i]);
            }
        }
    }
    // x lines: into the tile
    PADO_HD PADO_INLINE static void tile(const RegParams &kp, const RegSmem &sm, const Th &t, int l, int start, int op)
    {
        if constexpr (MODE == REG_SWZ) {
            const SwzAt<LT> at(sm.tile, l, kp.n, start, M, false);
#pragma unroll
            for (int i = 0; i < M; i += 2) {
                double2 x;
                x.x = RL::corrected(kp, t, i, t.x[i]);
                x.y = RL::corrected(kp, t, i + 1, t.x[i + 1]);
                if (EVEN || i >= reg_overlap(M) || i >= op)
                    *reinterpret_cast<double2 *>(at.unit(i)) = x;
            }
        } else {
            double *p = sm.tile + (long long)l * kp.P + start;
#pragma unroll
            for (int i = 0; i < M; ++i) {
                const double x = RL::corrected(kp, t, i, t.x[i]);
                if (EVEN || i >= reg_overlap(M) || i >= op) p[i] = x;
            }
        }
    }
    // element r of line l in an x-line tile
    PADO_HD PADO_INLINE static double *at(const RegParams &kp, double *tile, int l, int r)
    {
        if constexpr (MODE == REG_SWZ) {
            return tile + l * 16 + (r >> 4) * (LT * 16) + ((((r >> 1) & 7) ^ (l & 7)) << 1) + (r & 1);
        } else {
            return tile + (long long)l * kp.P + r;
        }
    }
    // the closure rows of one end (row0: the first of them)
    PADO_HD PADO_INLINE static void edge(const RegParams &kp, const RegSmem &sm, const double (&e)[REG_EDGE], int l,
                                         int row0, double *line, bool live)
    {
        if constexpr (reg_strided(MODE)) {
            if (!live) return;
            // df's values first: one wait for the four of them
            double old[REG_EDGE];
#pragma unroll
            for (int i = 0; i < REG_EDGE; ++i) old[i] = kp.out_mode == OUT_ACC ? line[(row0 + i) * kp.stride] : 0.0;
#pragma unroll
            for (int i = 0; i < REG_EDGE; ++i)
                line[(row0 + i) * kp.stride] = kp.out_mode == OUT_STORE ? e[i] : fma(kp.out_alpha, e[i], old[i]);
        } else {
#pragma unroll
            for (int i = 0; i < REG_EDGE; ++i) *at(kp, sm.tile, l, row0 + i) = e[i];
        }
    }
};

// Phase functions of one thread (l, s), a barrier between consecutive ones.
template <int RK, bool PER, int M, bool EVEN, int MODE, int LT>
struct RegPhases {
    using RL = RegLine<RK, PER, M, EVEN>;
    using RO = RegOut<RK, PER, M, EVEN, MODE, LT>;
    using Th = RegThread<M>;
    static constexpr int H = RL::H;

    PADO_HD PADO_INLINE static void sweep(const RegParams &kp, const RegSmem &sm, Th &t, int l, int s)
    {
        const int st = RL::start(kp, s), od = RL::overlap(kp, s + 1), op = RL::overlap(kp, s);
        double2 last;
        if constexpr (MODE == REG_SWZ) {
            const SwzAt<LT> at(sm.tile, l, kp.n, st, M, PER);
            auto load = [&](double(&f)[M + 2 * H]) {
                constexpr int HP = (H + 1) / 2 * 2;
#pragma unroll
                for (int k = -HP; k < M + HP; k += 2) {
                    const double2 u = at.template get2<M>(k);
                    if (k >= -H && k < M + H) f[k + H] = u.x;
                    if (k + 1 >= -H && k + 1 < M + H) f[k + 1 + H] = u.y;
                }
            };
            double2 pair;
            auto again = [&](int i) {  // rows come in falling order
                if (i & 1) pair = *reinterpret_cast<const double2 *>(at.unit(i - 1));
                return i & 1 ? pair.y : pair.x;
            };
            RL::sweep(kp, t, od, op, load, again, sm.ys + (s * LT + l), sm.xs + (s * LT + l), last);
        } else if constexpr (MODE == REG_ODD) {
            const double *par[2];
            parities(kp, sm, l, par);
            const OddAt<LT, RK> at(par, kp.n, st, M, PER);
            auto load = [&](double(&f)[M + 2 * H]) {
#pragma unroll
                for (int k = -H; k < M + H; ++k) f[k + H] = at.template get<M>(k);
            };
            auto again = [&](int i) { return at.template get<M>(i); };
            RL::sweep(kp, t, od, op, load, again, sm.ys + (s * LT + l), sm.xs + (s * LT + l), last);
        } else {
            constexpr int RS = MODE == REG_ROWS ? LT : 1;
            const RowsAt<RS, RK> at(MODE == REG_ROWS ? sm.tile + l : sm.tile + (long long)l * kp.P, kp.n, st, M, PER);
            auto load = [&](double(&f)[M + 2 * H]) {
#pragma unroll
                for (int k = -H; k < M + H; ++k) f[k + H] = at.template get<M>(k);
            };
            auto again = [&](int i) { return at.template get<M>(i); };
            RL::sweep(kp, t, od, op, load, again, sm.ys + (s * LT + l), sm.xs + (s * LT + l), last);
        }
        if constexpr (!PER) {
            if (s == 0) {
                double g[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) g[j] = row(kp, sm, l, j);
                RL::template edge_rhs<0>(kp, sm, LT, l, g);
            }
            if (s == kp.S - 1) {
                double g[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) g[j] = row(kp, sm, l, kp.nin - 8 + j);
                RL::template edge_rhs<1>(kp, sm, LT, l, g);
                double *e = sm.edge + (4 * REG_EDGE + 4) * LT + l;
                e[0] = last.x;
                e[LT] = last.y;
            }
        }
    }
    // REG_ODD: rows 0 and 1 of line l (odd rows of the field sit one element further in)
    PADO_HD PADO_INLINE static void parities(const RegParams &kp, const RegSmem &sm, int l, const double *(&par)[2])
    {
        const double *even = sm.tile + l, *odd = sm.tile + kp.odd_rows + l + 1;
        par[0] = sm.first ? odd : even;
        par[1] = sm.first ? even : odd;
    }
    PADO_HD PADO_INLINE static double row(const RegParams &kp, const RegSmem &sm, int l, int r)
    {
        if constexpr (MODE == REG_ODD) {
            const double *par[2];
            parities(kp, sm, l, par);
            return *OddAt<LT, RK>::place(par, r);
        } else if constexpr (MODE == REG_ROWS) return sm.tile[r * LT + l];
        else return *RO::at(kp, sm.tile, l, r);
    }
    PADO_HD PADO_INLINE static double2 last_rows(const RegSmem &sm, int l)
    {
        const double *e = sm.edge + (4 * REG_EDGE + 4) * LT + l;
        double2 x;
        x.x = e[0];
        x.y = e[LT];
        return x;
    }
    PADO_HD PADO_INLINE static void link(const RegParams &kp, const RegSmem &sm, Th &t, int l, int s)
    {
        RL::link(kp, sm, t, LT, l, s, RL::overlap(kp, s));
        sm.xs[s * LT + l] = t.xc;
    }
    PADO_HD PADO_INLINE static void close(const RegParams &kp, const RegSmem &sm, Th &t, int l, int s)
    {
        RL::close(kp, sm, t, LT, l, s);
        if constexpr (!PER) {
            if (s == 0) RL::template edge_state<0>(kp, sm, LT, l, RL::next_left(kp, t));
            if (s == kp.S - 1) RL::template edge_state<1>(kp, sm, LT, l, RL::next_right(kp, t, last_rows(sm, l)));
        }
    }
    // dst: row 0 of the line in df (strided lines)
    PADO_HD PADO_INLINE static void out(const RegParams &kp, const RegSmem &sm, Th &t, int l, int s, double *dst, bool live)
    {
        const int st = RL::start(kp, s), op = RL::overlap(kp, s);
        if constexpr (!PER) {
            RL::edge_add(kp, sm, t, LT, l, s);
            double e[REG_EDGE];
            if (s == 0) {
                RL::template edge_rows<0>(kp, sm, LT, l, RL::full_left(kp, t, t.xc), e);
                RO::edge(kp, sm, e, l, 0, dst, live);
            }
            if (s == kp.S - 1) {
                RL::template edge_rows<1>(kp, sm, LT, l, RL::full_right(kp, t, last_rows(sm, l)), e);
                RO::edge(kp, sm, e, l, kp.n - REG_EDGE, dst, live);
            }
        }
        if constexpr (reg_strided(MODE)) {
            if (live) RO::rows(kp, t, dst + st * kp.stride, op);
            if constexpr (PER && (RK == RHS_ST_CE || RK == RHS_ST_D2))
                if (live && s == 0 && kp.copy_first) dst[kp.n * kp.stride] = RL::corrected(kp, t, 0, t.x[0]);
        } else {
            RO::tile(kp, sm, t, l, st, op);
        }
    }
};

#ifdef __CUDACC__
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, unsigned long long *bar, int c0, int c1)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];\n" ::"r"(smem_u32(dst)),
        "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, const void *src, int c0, int c1)
{
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];\n" ::"l"(map),
                 "r"(c0), "r"(c1), "r"(smem_u32(src))
                 : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, const void *src, int c0, int c1, int c2)
{
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];\n" ::"l"(map),
                 "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(src))
                 : "memory");
}

// Elements of the x-line tile from line x0.
template <int LT>
__device__ __forceinline__ int reg_span(const RegParams &kp, long long x0)
{
    const long long left = kp.nlines - x0;
    return (int)(left < LT ? left : LT) * kp.n;
}

// Tensor or bulk copies of tile t into `tile` (one thread, that which stores
// the results: what it writes itself is seen from the barrier before the sweep).
template <int MODE, int LT>
__device__ __forceinline__ void reg_load(const RegParams &kp, double *tile, unsigned long long *bar, long long t)
{
    long long x0, p;
    reg_origin(kp, LT, t, &x0, &p);
    if constexpr (MODE == REG_SWZ) {
        const bool part = kp.n & 15;
        mbar_expect_tx(bar, (unsigned)(kp.chunks + (part ? 1 : 0)) * LT * 128u);
        if (kp.chunks) tma_load_3d(tile, &kp.tin, bar, 0, (int)x0, 0);
        if (part) tma_load_2d(tile + (size_t)kp.chunks * LT * 16, &kp.tin2, bar, kp.chunks * 16, (int)x0);
    } else if constexpr (MODE == REG_ODD) {
        // rows p nin .. p nin + nin - 1 of the field, those of either parity from their own map
        const int r0 = kp.axis == 2 ? (int)p * kp.nin : 0;
        mbar_expect_tx(bar, 2u * kp.nbox * kp.box_rows * (LT + 2) * 8u);
        for (int b = 0; b < kp.nbox; ++b) {
            double *dst = tile + (size_t)b * kp.box_rows * (LT + 2);
            tma_load_2d(dst, &kp.tin, bar, (int)x0, ((r0 + 1) >> 1) + b * kp.box_rows);
            tma_load_2d(dst + kp.odd_rows, &kp.tin2, bar, (int)x0, (r0 >> 1) + b * kp.box_rows);
        }
    } else if constexpr (MODE == REG_PACK) {
        // whole 16-byte units of the span (tiles start on them: LT is even), and
        // the last element of a field of an odd number of them, by this thread
        // as well: it alone has waited for the tile's last results to be read
        const int total = reg_span<LT>(kp, x0);
        const unsigned bytes = ((unsigned)total * 8u) & ~15u;
        const double *src = kp.in + x0 * (long long)kp.n;
        mbar_expect_tx(bar, bytes);
        bulk_load(tile, src, bytes, bar);
        if (total & 1) tile[total - 1] = __ldg(src + total - 1);
    } else {
        mbar_expect_tx(bar, (unsigned)kp.nbox * kp.box_rows * LT * 8u);
        for (int b = 0; b < kp.nbox; ++b) {
            const int r0 = b * kp.box_rows;
            double *dst = tile + (size_t)r0 * LT;
            if (kp.axis == 2) tma_load_3d(dst, &kp.tin, bar, (int)x0, r0, (int)p);
            else tma_load_3d(dst, &kp.tin, bar, (int)x0, (int)p, r0);
        }
    }
}

// Per-element copies of tile t by every thread (8-byte cp.async, then one
// arrival each): strided lines thread by thread along rows, x lines along the
// tile's contiguous span.
template <int MODE, int LT>
__device__ __forceinline__ void reg_load_async(const RegParams &kp, double *tile, unsigned long long *bar, long long t,
                                               int tid, int nthreads)
{
    long long x0, p;
    reg_origin(kp, LT, t, &x0, &p);
    if constexpr (MODE == REG_PACK) {
        const int n = kp.n, pad = kp.P - n;
        const long long left = kp.nlines - x0;
        const int total = (int)(left < LT ? left : LT) * n;
        const double *src = kp.in + x0 * (long long)n + tid;
        const int l0 = tid / n;
        int r = tid - l0 * n;
        double *dst = tile + (size_t)l0 * kp.P + r;
        const int dl = nthreads / n, dr = nthreads - dl * n, dstep = dl * kp.P + dr;
        for (int e = tid; e < total; e += nthreads) {
            async_copy8(dst, src);
            src += nthreads;
            dst += dstep;
            r += dr;
            if (r >= n) {
                r -= n;
                dst += pad;
            }
        }
    } else if constexpr (MODE == REG_ROWS) {
        const int l = tid % LT;
        if (x0 + l < kp.na) {
            const int rstep = nthreads / LT;
            const long long sstep = (long long)rstep * kp.stride;
            const double *src = kp.in + (x0 + l) + p * kp.pstride + (long long)(tid / LT) * kp.stride;
            double *dst = tile + tid;
#pragma unroll 4
            for (int r = tid / LT; r < kp.nin; r += rstep) {
                async_copy8(dst, src);
                src += sstep;
                dst += nthreads;
            }
        }
    }
    async_arrive(bar);
}

// Accumulated output: tile t's part of df on its way to L2 while the tile's
// copies are, so that out() does not wait for HBM (divergence + laplacian on
// 384x256x192: 541 -> 525 us; with the reads 8 rows ahead of their use in
// RegOut::rows 515 us).
template <int MODE, int LT>
__device__ __forceinline__ void reg_prefetch(const RegParams &kp, long long t, int tid, int nthreads)
{
    long long x0, p;
    reg_origin(kp, LT, t, &x0, &p);
    if constexpr (reg_strided(MODE)) {
        constexpr int LINE = LT < 16 ? LT : 16, PER_ROW = LT / LINE;  // 128 bytes
        const int total = kp.n * PER_ROW;
        for (int i = tid; i < total; i += nthreads) {
            const int r = i / PER_ROW, c = (i % PER_ROW) * LINE;
            if (x0 + c < kp.na)
                asm volatile("prefetch.global.L2 [%0];\n" ::"l"(kp.out + x0 + c + p * kp.pstride + r * kp.stride));
        }
    } else {
        const long long left = kp.nlines - x0;
        const int total = (int)(left < LT ? left : LT) * kp.n;
        for (int i = tid * 16; i < total; i += nthreads * 16)
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(kp.out + x0 * (long long)kp.n + i));
    }
}

// Registers: a segment of 32 rows takes 64 for its values and about 45 more,
// so 512 threads fill an SM; the swizzled x-line tiles, two buffers to a CTA,
// leave room for 384 threads in shared memory anyway, and their kernels take
// the registers (bounded cf90 along x, n = 512: 28 spilled with 128, 4680 ->
// 5600 GB/s); shorter segments leave room for more threads.
PADO_HD constexpr int reg_max_threads(int M, int mode) { return M >= 32 && mode != REG_SWZ ? 512 : 384; }
PADO_HD constexpr int reg_min_ctas(int M) { return M >= 32 ? 1 : 2; }

template <int RK, bool PER, int M, bool EVEN, int MODE, int LT>
__global__ void __launch_bounds__(reg_max_threads(M, MODE), reg_min_ctas(M)) reg_kernel(const __grid_constant__ RegParams kp)
{
    using PH = RegPhases<RK, PER, M, EVEN, MODE, LT>;
    using RO = RegOut<RK, PER, M, EVEN, MODE, LT>;
    extern __shared__ double smem_raw[];
    double *base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u) / sizeof(double);
    const int S = kp.S, stages = reg_strided(MODE) ? 1 : kp.stages;
    const int edge_table = reg_edge_table(RK, PER, S);
    const RegLayout lay = reg_layout(LT, S, stages, kp.tile_doubles, edge_table);
    unsigned long long *bars = reinterpret_cast<unsigned long long *>(base + lay.bars);
    RegSmem sm;
    sm.ys = reinterpret_cast<double2 *>(base + lay.ys);
    sm.xs = reinterpret_cast<double2 *>(base + lay.xs);
    sm.edge = base + lay.edge;
    sm.segtab = base + lay.segtab;
    const int tid = threadIdx.x, nthreads = blockDim.x;
    const int l = tid % LT, s = tid / LT;
    const bool active = s < S;
    const bool async = (MODE == REG_ROWS || MODE == REG_PACK) && kp.async_copy;
    const long long G = gridDim.x;

    // the first copies start before the edge tables are staged
    if (tid == 0) {
        for (int b = 0; b < stages; ++b) mbar_init(&bars[b], async ? (unsigned)nthreads : 1u);
        mbar_fence_init();
        if (!async)
            for (int b = 0; b < stages; ++b)
                if (blockIdx.x + b * G < kp.ntiles)
                    reg_load<MODE, LT>(kp, base + (size_t)b * kp.tile_doubles, &bars[b], blockIdx.x + b * G);
    }
    if constexpr (!PER)
        for (int i = tid; i < edge_table; i += nthreads) base[lay.segtab + i] = __ldg(kp.segtab + i);
    __syncthreads();
    if (async && blockIdx.x < kp.ntiles) reg_load_async<MODE, LT>(kp, base, &bars[0], blockIdx.x, tid, nthreads);

    const bool acc = kp.out_mode == OUT_ACC;
    if (acc && blockIdx.x < kp.ntiles) reg_prefetch<MODE, LT>(kp, blockIdx.x, tid, nthreads);
    int b = 0;
    unsigned parity = 0;
    for (long long t = blockIdx.x; t < kp.ntiles; t += G) {
        bool arrived = true;
        if (tid < 32) arrived = mbar_wait(&bars[b], parity, STREAM_WAIT_NS);
        if (!__syncthreads_and(arrived)) {
            // record, let the copies in flight land, and leave
            if (tid == 0) {
                atomicExch(kp.status, PADO_STATUS_TIMEOUT);
                (void)mbar_wait(&bars[b], parity, STREAM_DRAIN_NS);
                if (stages == 2 && t + G < kp.ntiles)
                    (void)mbar_wait(&bars[b ^ 1], b ? parity ^ 1u : parity, STREAM_DRAIN_NS);
            }
            if (async) async_wait_all();
            else if (!reg_strided(MODE)) bulk_wait_all();
            return;
        }
        sm.tile = base + (size_t)b * kp.tile_doubles;
        long long x0, p;
        reg_origin(kp, LT, t, &x0, &p);
        sm.first = MODE == REG_ODD && kp.axis == 2 ? (int)(p * kp.nin & 1) : 0;
        RegThread<M> th;
        if (active) PH::sweep(kp, sm, th, l, s);
        __syncthreads();
        // every read of the tile is done: strided lines take the next one now,
        // x lines their other buffer, once its results have been read out
        if constexpr (reg_strided(MODE)) {
            if (t + G < kp.ntiles) {
                if (async) reg_load_async<MODE, LT>(kp, sm.tile, &bars[0], t + G, tid, nthreads);
                else if (tid == 0) reg_load<MODE, LT>(kp, sm.tile, &bars[0], t + G);
            }
        } else {
            if (stages == 2 && tid == 0 && t != blockIdx.x && t + G < kp.ntiles) {
                bulk_wait_read();
                reg_load<MODE, LT>(kp, base + (size_t)(b ^ 1) * kp.tile_doubles, &bars[b ^ 1], t + G);
            }
        }
        if (acc && t + G < kp.ntiles) reg_prefetch<MODE, LT>(kp, t + G, tid, nthreads);
        if (active) PH::link(kp, sm, th, l, s);
        __syncthreads();
        if (active) PH::close(kp, sm, th, l, s);
        if constexpr (!PER) __syncthreads();
        const bool live = !reg_strided(MODE) || x0 + l < kp.na;
        double *dst = reg_strided(MODE) ? kp.out + (live ? x0 + l + p * kp.pstride : 0) : nullptr;
        if (active) PH::out(kp, sm, th, l, s, dst, live);
        if constexpr (!reg_strided(MODE)) {
            const long long left = kp.nlines - x0;
            const int nl = (int)(left < LT ? left : LT), n = kp.n;
            if (!async && kp.out_mode != OUT_STORE) {
                // scaled or accumulated output: the tile takes df's values before it goes out
                __syncthreads();
                if constexpr (MODE == REG_SWZ) {
                    const int half = n >> 1, warp = tid >> 5, lane = tid & 31, nw = nthreads >> 5;
                    for (int ll = warp; ll < nl; ll += nw) {
                        const double2 *d = reinterpret_cast<const double2 *>(kp.out + (x0 + ll) * (long long)n);
                        for (int u = lane; u < half; u += 32) {
                            double2 *x = reinterpret_cast<double2 *>(RO::at(kp, sm.tile, ll, 2 * u));
                            double2 v = *x;
                            if (kp.out_mode == OUT_ACC) {
                                const double2 o = d[u];
                                v.x = fma(kp.out_alpha, v.x, o.x);
                                v.y = fma(kp.out_alpha, v.y, o.y);
                            } else {
                                v.x *= kp.out_alpha;
                                v.y *= kp.out_alpha;
                            }
                            *x = v;
                        }
                    }
                } else {
                    const double *d = kp.out + x0 * (long long)n;
                    for (int e = tid; e < nl * n; e += nthreads)
                        sm.tile[e] = kp.out_mode == OUT_ACC ? fma(kp.out_alpha, sm.tile[e], d[e]) : kp.out_alpha * sm.tile[e];
                }
            }
            if (!async) {
                fence_proxy_async();
                __syncthreads();
                if (tid == 0) {
                    if constexpr (MODE == REG_SWZ) {
                        if (kp.chunks) tma_store_3d(&kp.tout, sm.tile, 0, (int)x0, 0);
                        if (n & 15) tma_store_2d(&kp.tout2, sm.tile + (size_t)kp.chunks * LT * 16, kp.chunks * 16, (int)x0);
                    } else {
                        const int total = nl * n;
                        double *d = kp.out + x0 * (long long)n;
                        bulk_store(d, sm.tile, ((unsigned)total * 8u) & ~15u);
                        if (total & 1) d[total - 1] = sm.tile[total - 1];
                    }
                    bulk_commit();
                    if (stages == 1) {
                        bulk_wait_read();
                        if (t + G < kp.ntiles) reg_load<MODE, LT>(kp, sm.tile, &bars[0], t + G);
                    }
                }
            } else if constexpr (MODE == REG_PACK) {
                // the tile's lines are consecutive in global memory
                __syncthreads();
                const int pad = kp.P - n, total = nl * n;
                double *d = kp.out + x0 * (long long)n + tid;
                const int l0 = tid / n;
                int r = tid - l0 * n;
                const double *src = sm.tile + (size_t)l0 * kp.P + r;
                const int dl = nthreads / n, dr = nthreads - dl * n, sstep = dl * kp.P + dr;
                for (int e = tid; e < total; e += nthreads) {
                    const double x = *src;
                    *d = kp.out_mode == OUT_ACC ? fma(kp.out_alpha, x, *d)
                                                : (kp.out_mode == OUT_SCALE ? kp.out_alpha * x : x);
                    d += nthreads;
                    src += sstep;
                    r += dr;
                    if (r >= n) {
                        r -= n;
                        src += pad;
                    }
                }
                __syncthreads();
                if (t + G < kp.ntiles) reg_load_async<MODE, LT>(kp, sm.tile, &bars[0], t + G, tid, nthreads);
            }
        }
        if (stages == 2) {
            b ^= 1;
            if (!b) parity ^= 1u;
        } else {
            parity ^= 1u;
        }
    }
    if (!reg_strided(MODE) && !async) bulk_wait_all();
}
#endif  // __CUDACC__

// Host emulation (tests): the kernel's tile loop with plain copies in place
// of the tensor and asynchronous ones; phases in kernel order over all threads.
template <int RK, bool PER, int M, bool EVEN, int MODE, int LT>
inline void emulate_reg(const RegParams &kp)
{
    using PH = RegPhases<RK, PER, M, EVEN, MODE, LT>;
    using RO = RegOut<RK, PER, M, EVEN, MODE, LT>;
    const int edge_table = reg_edge_table(RK, PER, kp.S);
    const RegLayout lay = reg_layout(LT, kp.S, 1, kp.tile_doubles, edge_table);
    std::vector<double2> mem(lay.total / 2 + 1);
    double *base = reinterpret_cast<double *>(mem.data());
    RegSmem sm;
    sm.tile = base;
    sm.ys = reinterpret_cast<double2 *>(base + lay.ys);
    sm.xs = reinterpret_cast<double2 *>(base + lay.xs);
    sm.edge = base + lay.edge;
    sm.segtab = base + lay.segtab;
    if (!PER)
        for (int i = 0; i < edge_table; ++i) base[lay.segtab + i] = kp.segtab[i];
    std::vector<RegThread<M>> th((size_t)kp.S * LT);
    for (long long t = 0; t < kp.ntiles; ++t) {
        long long x0, p;
        reg_origin(kp, LT, t, &x0, &p);
        const long long lim = kp.axis == 1 ? kp.nlines : kp.na;
        sm.first = MODE == REG_ODD && kp.axis == 2 ? (int)(p * kp.nin & 1) : 0;
        for (int l = 0; l < LT && x0 + l < lim; ++l)
            for (int r = 0; r < kp.nin; ++r) {
                if (MODE == REG_ROWS) sm.tile[r * LT + l] = kp.in[x0 + l + p * kp.pstride + r * kp.stride];
                else if (MODE == REG_ODD)
                    sm.tile[((sm.first + r) & 1 ? kp.odd_rows + 1 : 0) + (r >> 1) * (LT + 2) + l] =
                        kp.in[x0 + l + p * kp.pstride + r * kp.stride];
                else *RO::at(kp, sm.tile, l, r) = kp.in[(x0 + l) * kp.n + r];
            }
        for (int ph = 0; ph < 4; ++ph)
            for (int s = 0; s < kp.S; ++s)
                for (int l = 0; l < LT; ++l) {
                    RegThread<M> &h = th[(size_t)s * LT + l];
                    const bool live = !reg_strided(MODE) || x0 + l < kp.na;
                    if (ph == 0) PH::sweep(kp, sm, h, l, s);
                    else if (ph == 1) PH::link(kp, sm, h, l, s);
                    else if (ph == 2) PH::close(kp, sm, h, l, s);
                    else PH::out(kp, sm, h, l, s, kp.out + (live ? x0 + l + p * kp.pstride : 0), live);
                }
        if (!reg_strided(MODE))
            for (int l = 0; l < LT && x0 + l < lim; ++l)
                for (int r = 0; r < kp.n; ++r) {
                    double *d = kp.out + (x0 + l) * kp.n + r;
                    const double x = *RO::at(kp, sm.tile, l, r);
                    *d = kp.out_mode == OUT_ACC ? fma(kp.out_alpha, x, *d)
                                                : (kp.out_mode == OUT_SCALE ? kp.out_alpha * x : x);
                }
    }
}

}  // namespace pado
