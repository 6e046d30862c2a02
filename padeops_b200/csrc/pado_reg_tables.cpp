// pado_reg_tables.cpp -- constants of the register kernel, in extended
// precision, rounded to double once.
#include "pado_reg_tables.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "pado_tables.h"

namespace pado {

namespace {

using ld = long double;

using M2 = RegBand::M2;

M2 mul(const M2 &x, const M2 &y)
{
    return {x.a * y.a + x.b * y.c, x.a * y.b + x.b * y.d, x.c * y.a + x.d * y.c, x.c * y.b + x.d * y.d};
}
void put(const M2 &m, double *o)
{
    o[0] = (double)m.a;
    o[1] = (double)m.b;
    o[2] = (double)m.c;
    o[3] = (double)m.d;
}

// Interior band of the left-hand side (1 on the diagonal) and stencil taps of
// the schemes (cd06.F90:14-20, cd10.F90:16-30, cf90.F90:16-24) for spacing dx.
// The derivatives' are fractions: formed in extended precision, so that each
// constant of the launch is rounded once.
void band(int scheme, int kind, ld *al, ld *be)
{
    *be = 0;
    if (scheme == CD06) {
        *al = (ld)1 / 3;
    } else if (scheme == CF90) {
        *al = Cf90Const().alpha;
        *be = Cf90Const().beta;
    } else if (kind == D2) {
        *al = (ld)334 / 899;
        *be = (ld)43 / 1798;
    } else {
        *al = (ld)1 / 2;
        *be = (ld)1 / 20;
    }
}
void interior_stencil(int scheme, int kind, ld dx, ld (&t)[5])
{
    for (ld &v : t) v = 0;
    if (scheme == CD06) {
        t[0] = (ld)7 / 9 / dx;
        t[1] = (ld)1 / 36 / dx;
    } else if (scheme == CF90) {
        // B - A: the first three taps cancel to 1e-4 of the filter's
        const Cf90Const k;
        t[0] = (ld)k.a - 1;
        t[1] = (ld)k.b - k.alpha;
        t[2] = (ld)k.c - k.beta;
        t[3] = k.d;
        t[4] = k.e;
    } else if (kind == D2) {
        t[0] = (ld)1065 / 1798 / dx / dx;
        t[1] = (ld)1038 / 3596 / dx / dx;
        t[2] = (ld)79 / 16182 / dx / dx;
    } else {
        t[0] = (ld)17 / 24 / dx;
        t[1] = (ld)101 / 600 / dx;
        t[2] = (ld)1 / 600 / dx;
    }
}

// Left-hand-side rows of a bounded line's closure block: A[side][i][j], j =
// columns 0 .. EDGE + 1 from the line's start (left) or the last EDGE + 2
// columns (right), in line order.
// A line of 16 rows tells both ends.
void edge_lhs(int scheme, int kind, int bc1, int bcn, ld A[2][REG_EDGE][REG_EDGE + 2])
{
    constexpr int n = 16;
    std::vector<double> bt(n, 0.0), b(n), d(n, 1.0), a(n), at(n, 0.0);
    if (scheme == CD06) {
        const Cd06Const k;
        std::fill(b.begin(), b.end(), k.alpha_hat);
        std::fill(a.begin(), a.end(), k.alpha_hat);
        const double W[3] = {k.w1, k.w2, k.w3}, R[3][3] = {{0.0, 1.0, k.alpha}, {k.alpha_p, 1.0, k.alpha_p},
                                                           {k.alpha_pp, 1.0, k.alpha_pp}};
        for (int r = 0; r < 3; ++r) {
            if (bc1 == 0) {
                b[r] = W[r] * R[r][0];
                d[r] = W[r] * R[r][1];
                a[r] = W[r] * R[r][2];
            }
            if (bcn == 0) {
                a[n - 1 - r] = W[r] * R[r][0];
                d[n - 1 - r] = W[r] * R[r][1];
                b[n - 1 - r] = W[r] * R[r][2];
            }
        }
    } else {
        const std::vector<double> P = penta_bounded(scheme, kind, n, bc1, bcn);
        for (int i = 0; i < n; ++i) {
            bt[i] = P[i];
            b[i] = P[(size_t)n + i];
            d[i] = P[2 * (size_t)n + i];
            a[i] = P[3 * (size_t)n + i];
            at[i] = P[4 * (size_t)n + i];
        }
    }
    for (int side = 0; side < 2; ++side)
        for (int i = 0; i < REG_EDGE; ++i) {
            const int row = side ? n - REG_EDGE + i : i, c0 = side ? n - REG_EDGE - 2 : 0;
            for (int j = 0; j < REG_EDGE + 2; ++j) {
                const int o = c0 + j - row;
                A[side][i][j] = o == -2 ? bt[row] : o == -1 ? b[row] : o == 0 ? d[row] : o == 1 ? a[row]
                                                                                                : o == 2 ? at[row] : 0.0;
            }
        }
}

// Gauss-Jordan with row pivoting: m (n x (n + k)) to [I | m^-1 rhs].
template <int N, int K>
void solve(ld (&m)[N][N + K])
{
    for (int c = 0; c < N; ++c) {
        int p = c;
        for (int r = c + 1; r < N; ++r)
            if (std::fabs(m[r][c]) > std::fabs(m[p][c])) p = r;
        for (int j = 0; j < N + K; ++j) std::swap(m[c][j], m[p][j]);
        const ld inv = 1 / m[c][c];
        for (int j = 0; j < N + K; ++j) m[c][j] *= inv;
        for (int r = 0; r < N; ++r) {
            if (r == c) continue;
            const ld f = m[r][c];
            for (int j = 0; j < N + K; ++j) m[r][j] -= f * m[c][j];
        }
    }
}

}  // namespace

// A = c L L^T: the limit of the factorization's pivots and multipliers
// (it converges with the square of the largest root, at most 0.67).
RegBand::RegBand(int n_, bool periodic, ld al, ld be) : n(n_)
{
    ld dm2 = 1, dm1 = 1 - al * al, l = al, d = dm1;
    for (int i = 0; i < 400; ++i) {
        const ld q = (al - be * l) / dm1, next = 1 - q * q * dm1 - (be / dm2) * be;
        const bool done = q == l && next == d && i > 2;
        d = next;
        l = q;
        dm2 = dm1;
        dm1 = d;
        if (done) break;
    }
    c = d;
    p1 = l;
    p2 = be / d;
    const int rows = std::max(reg_rows(n, periodic), REG_MAXM);
    const M2 T{-p1, -p2, 1, 0};
    tk.resize(rows + 1);
    tk[0] = M2{1, 0, 0, 1};
    for (int k = 1; k <= rows; ++k) tk[k] = mul(T, tk[k - 1]);
    if (periodic) return;
    const int N = reg_rows(n, false);
    u.assign((size_t)(N + 2) * 2, 0);
    for (int i = N - 1; i >= 0; --i) {
        u[2 * i] = tk[i + 1].a - p1 * u[2 * (i + 1)] - p2 * u[2 * (i + 2)];
        u[2 * i + 1] = tk[i + 1].b - p1 * u[2 * (i + 1) + 1] - p2 * u[2 * (i + 2) + 1];
    }
}

RegBand RegBand::of(int scheme, int kind, int n, bool periodic)
{
    ld al, be;
    band(scheme, kind, &al, &be);
    return RegBand(n, periodic, al, be);
}

bool reg_cut(int rows, int M, bool even_starts, RegCut *cut)
{
    if (rows < M) return false;
    const int S = (rows + M - 1) / M;
    const int step = even_starts ? 2 : 1;
    const int extra = S * M - rows;
    if (extra % step) return false;
    cut->M = M;
    cut->S = S;
    cut->d0 = cut->d1 = cut->nd1 = 0;
    if (extra == 0) return true;
    if (S < 2 || S > REG_MAXS) return false;
    const int units = extra / step, base = units / (S - 1);
    cut->d0 = base * step;
    cut->nd1 = units % (S - 1);
    cut->d1 = cut->nd1 ? (base + 1) * step : cut->d0;
    return std::max(cut->d0, cut->d1) <= reg_overlap(M);
}

namespace {

// Everything that follows from the left-hand side alone: its band and, on
// bounded lines, the closure rows A; solved: how RegParams::xr holds them.
void fill_system(const RegBand &rb, bool periodic, const ld (*A)[REG_EDGE][REG_EDGE + 2], bool solved, const RegCut &cut,
                 RegParams *kp, std::vector<double> *segtab)
{
    const int M = cut.M, S = cut.S, n = rb.n;
    const ld p1 = rb.p1, p2 = rb.p2;
    const std::vector<M2> &tk = rb.tk;
    kp->n = kp->nin = n;
    kp->S = S;
    kp->d0 = cut.d0;
    kp->d1 = cut.d1;
    kp->nd1 = cut.nd1;
    kp->np1 = (double)-p1;
    kp->np2 = (double)-p2;

    // W: backward recurrence over the response of y; V: over a zero y
    std::vector<ld> w((size_t)(M + 2) * 2, 0), v((size_t)(M + 2) * 2, 0);
    for (int i = M - 1; i >= 0; --i) {
        w[2 * i] = tk[i + 1].a - p1 * w[2 * (i + 1)] - p2 * w[2 * (i + 2)];
        w[2 * i + 1] = tk[i + 1].b - p1 * w[2 * (i + 1) + 1] - p2 * w[2 * (i + 2) + 1];
        v[2 * i] = tk[M - i].a;
        v[2 * i + 1] = tk[M - i].b;
    }
    for (int i = 0; i < M; ++i)
        for (int k = 0; k < 2; ++k) {
            kp->w[i][k] = (double)w[2 * i + k];
            kp->v[i][k] = (double)v[2 * i + k];
        }
    put(tk[M - cut.d0], kp->phi[0]);
    put(tk[M - cut.d1], kp->phi[1]);
    put(tk[M], kp->phi[2]);

    // coupling window: rows after which every state has decayed below half a unit of rounding
    const ld disc = p1 * p1 - 4 * p2;
    const ld rho = disc >= 0 ? (p1 + std::sqrt(disc)) / 2 : std::sqrt(p2);
    const ld reach = std::log((ld)5.5e-17) / std::log(rho);
    const int step = M - std::max(cut.d0, cut.d1);
    int W = (int)std::ceil(reach / step);
    kp->cyc = 0;
    if (periodic) {
        if (W >= S) {
            W = S;
            const M2 &tn = tk[n];
            const ld a = 1 - tn.a, d = 1 - tn.d, b = -tn.b, e = -tn.c, det = a * d - b * e;
            put(M2{d / det, -b / det, -e / det, a / det}, kp->wrap);
            kp->cyc = 1;
        }
        kp->W = W;
        segtab->clear();
        return;
    }
    kp->W = std::min(W, S - 1);

    // ---- bounded: the closure blocks and the line between them --------------
    const int N = n - 2 * REG_EDGE;
    // block rows, k-th from the wall: elimination inwards leaves each as its own
    // right-hand side's and those before it and the two x further in; with these
    // put in, all four right-hand sides and the two interior rows next to the block
    ld xr[2][REG_EDGE][REG_EDGE], xx[2][REG_EDGE][2];
    for (int side = 0; side < 2; ++side) {
        constexpr int E = REG_EDGE;
        auto at = [&](int k, int end) { return side ? end - 1 - k : k; };
        ld m[E][2 * E + 2], x[E][E + 2];
        for (int i = 0; i < E; ++i) {
            for (int j = 0; j < E + 2; ++j) m[i][j] = A[side][at(i, E)][at(j, E + 2)];
            for (int j = 0; j < E; ++j) m[i][E + 2 + j] = i == j ? 1 : 0;
        }
        for (int c = 0; c < E; ++c) {
            const ld inv = 1 / m[c][c];
            for (ld &v : m[c]) v *= inv;
            for (int i = c + 1; i < E; ++i) {
                const ld f = m[i][c];
                for (int j = 0; j < 2 * E + 2; ++j) m[i][j] -= f * m[c][j];
            }
        }
        for (int i = E - 1; i >= 0; --i)
            for (int j = 0; j < E + 2; ++j) {
                x[i][j] = j < E ? m[i][E + 2 + j] : (ld)0;
                for (int k = i + 1; k <= i + 2; ++k) x[i][j] -= m[i][k] * (k < E ? x[k][j] : (ld)(k == j));
            }
        for (int i = 0; i < E; ++i) {
            for (int j = 0; j < E; ++j) {
                xr[side][at(i, E)][at(j, E)] = x[i][j];
                kp->xr[side][at(i, E)][at(j, E)] = (double)(solved ? x[i][j] : m[i][E + 2 + j]);
            }
            for (int k = 0; k < 2; ++k) {
                xx[side][at(i, E)][at(k, 2)] = x[i][E + k];
                kp->xx[side][at(i, E)][at(k, 2)] = (double)(solved ? x[i][E + k] : -m[i][i + 1 + k]);
            }
        }
    }
    // end states: left (y_3, y_2) with y_i = x_i + p1 x_{i+1} + p2 x_{i+2};
    // right (x_{n-4}, x_{n-3})
    ld fr[2][2][REG_EDGE], fx[2][2][2];
    for (int j = 0; j < REG_EDGE; ++j) {
        fr[0][0][j] = xr[0][3][j];
        fr[0][1][j] = xr[0][2][j] + p1 * xr[0][3][j];
        fr[1][0][j] = xr[1][0][j];
        fr[1][1][j] = xr[1][1][j];
    }
    for (int k = 0; k < 2; ++k) {
        fx[0][0][k] = xx[0][3][k] + (k == 0 ? p1 : p2);
        fx[0][1][k] = xx[0][2][k] + p1 * xx[0][3][k] + (k == 0 ? p2 : (ld)0);
        fx[1][0][k] = xx[1][0][k];
        fx[1][1][k] = xx[1][1][k];
    }
    for (int side = 0; side < 2; ++side)
        for (int a = 0; a < 2; ++a) {
            for (int j = 0; j < REG_EDGE; ++j) kp->fr[side][a][j] = (double)fr[side][a][j];
            for (int k = 0; k < 2; ++k) kp->fx[side][a][k] = (double)fx[side][a][k];
        }
    const std::vector<ld> &u = rb.u;
    const M2 &tN = tk[N], &t2 = tk[2];
    // rows next to the blocks from z = (P0, Qlast): G[left 0..1, right 2..3][z]
    const ld G[4][4] = {{u[0], u[1], tN.a, tN.b},
                        {u[2], u[3], tN.c, tN.d},
                        {u[2 * (N - 2)], u[2 * (N - 2) + 1], t2.a, t2.b},
                        {u[2 * (N - 1)], u[2 * (N - 1) + 1], t2.c, t2.d}};
    ld m[4][8];
    for (int a = 0; a < 4; ++a) {
        const int side = a >> 1;
        for (int j = 0; j < 4; ++j) {
            ld k = 0;
            for (int q = 0; q < 2; ++q) k += fx[side][a & 1][q] * G[2 * side + q][j];
            m[a][j] = (a == j ? 1 : 0) - k;
            m[a][4 + j] = a == j ? 1 : 0;
        }
    }
    solve<4, 4>(m);
    for (int a = 0; a < 4; ++a)
        for (int j = 0; j < 4; ++j) kp->kinv[a][j] = (double)m[a][4 + j];
    segtab->assign((size_t)S * REG_SEGTAB, 0.0);
    for (int s = 0; s < S; ++s) {
        const int e = std::min(s, cut.nd1), start = s * M - e * cut.d1 - (s - e) * cut.d0, end = start + M;
        double *g = segtab->data() + (size_t)s * REG_SEGTAB;
        put(tk[start], g);
        put(M2{u[2 * end], u[2 * end + 1], u[2 * (end + 1)], u[2 * (end + 1) + 1]}, g + 4);
        put(tk[N - end], g + 8);
    }
}

}  // namespace

void reg_fill(const RegBand &rb, int scheme, int kind, double dx, bool periodic, int bc1, int bcn, int sbc1, int sbcn,
              const RegCut &cut, RegParams *kp, std::vector<double> *segtab)
{
    const ld c = rb.c;
    ld A[2][REG_EDGE][REG_EDGE + 2];
    if (!periodic) edge_lhs(scheme, kind, sbc1, sbcn, A);
    fill_system(rb, periodic, A, scheme == CF90, cut, kp, segtab);
    kp->bc1 = bc1;
    kp->bcn = bcn;
    const RhsCoef rc = make_rhs_coef(scheme, kind, dx, periodic);
    std::memcpy(kp->ctaps, rc.c, sizeof(kp->ctaps));
    ld t[5];
    interior_stencil(scheme, kind, dx, t);
    for (int k = 0; k < 5; ++k) kp->taps[k] = (double)(t[k] / c);
    if (scheme != CF90 || periodic) return;
    // the closure rows reach the 8 rows next to the wall: a line of 16 rows tells both ends
    constexpr int NL = 16;
    const std::vector<double> B = stencil_matrix(rc, NL, bc1, bcn);
    for (int side = 0; side < 2; ++side)
        for (int i = 0; i < REG_EDGE; ++i)
            for (int j = 0; j < 8; ++j) {
                const int row = side ? NL - REG_EDGE + i : i, col = side ? NL - 8 + j : j;
                const int aj = side ? j - (8 - REG_EDGE - 2) : j;
                const ld lhs = aj >= 0 && aj < REG_EDGE + 2 ? A[side][i][aj] : (ld)0;
                kp->dtaps[side][i][j] = (double)((ld)B[(size_t)row * NL + col] - lhs);
            }
}

void reg_fill_stagg(const RegStagg &st, const RegCut &cut, RegParams *kp, std::vector<double> *segtab)
{
    const int n = st.n;
    ld A[2][REG_EDGE][REG_EDGE + 2];
    for (int side = 0; side < 2 && !st.periodic; ++side)
        for (int i = 0; i < REG_EDGE; ++i) {
            const int row = side ? n - REG_EDGE + i : i, c0 = side ? n - REG_EDGE - 2 : 0;
            for (int j = 0; j < REG_EDGE + 2; ++j) {
                const int o = c0 + j - row;
                A[side][i][j] = o == -1 ? st.lower[row] : o == 0 ? st.diag[row] : o == 1 ? st.upper[row] : 0.0;
            }
        }
    const RegBand rb(n, st.periodic, st.alpha, 0);
    const ld c = rb.c;
    fill_system(rb, st.periodic, A, false, cut, kp, segtab);
    kp->nin = st.nin;
    kp->copy_first = st.copy_first;
    kp->taps[0] = (double)((ld)st.a / c);
    kp->taps[1] = (double)((ld)st.b / c);
    kp->taps[2] = st.sign;
    if (!st.periodic) segtab->insert(segtab->end(), st.rows, st.rows + REG_ROWTAB);
}

}  // namespace pado
