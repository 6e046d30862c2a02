"""CPU emulation of the register kernel: its phase functions
(padeops_b200/csrc/pado_reg.cuh) compiled for the host and run phase by phase
over every thread (tests/emul/pado_reg_emul.cu), against the oracle -- every
segment length and tile layout, line lengths at the edges of the cuts (one
segment, none, the most shared rows), closures, output modes.  Bar: 1e-12 of
max |oracle|, as everywhere."""
import ctypes
import itertools

import numpy as np
import pytest

import oracle

OPS = [(oracle.CD06, oracle.D1), (oracle.CD10, oracle.D1), (oracle.CD10, oracle.D2), (oracle.CF90, oracle.FILTER)]
ROWS, SWZ, PACK, ODD = 0, 1, 2, 3


@pytest.fixture(scope="module")
def emul():
    from tests.emul.build_reg import build

    lib = ctypes.CDLL(build())
    P, I, D, Lg = ctypes.c_void_p, ctypes.c_int, ctypes.c_double, ctypes.c_long
    lib.emul_reg.argtypes = [I, I, I, D, I, I, I, I, I, I, I, I, I, D, P, P, Lg, Lg]
    lib.emul_reg_stagg.argtypes = [I, I, I, I, I, P, P, P, I, I, P, P, Lg]
    return lib


def _run(emul, scheme, kind, n, dx, periodic, bc, solve, m, mode, axis, out_mode, alpha, f, out):
    na, nb = [s for a, s in enumerate(f.shape[::-1]) if a != axis - 1]
    return emul.emul_reg(scheme, kind, n, dx, int(periodic), *bc, *solve, m, mode, axis, out_mode, alpha, f.ctypes.data,
                out.ctypes.data, na, nb)


@pytest.mark.parametrize("scheme,kind", OPS)
@pytest.mark.parametrize("periodic", [True, False])
def test_register_kernel_emulated(emul, scheme, kind, periodic):
    rng = np.random.default_rng(31 + scheme + 5 * kind)
    dx = 0.37
    cuts = 0
    # 24: the shortest; 32, 64, 128: no shared rows; 40, 36: the most; 100, 129, 255, 512: both overlaps
    for n in (24, 25, 32, 36, 40, 64, 100, 129, 255, 512):
        bcs = [(0, 0)] if periodic or scheme == oracle.CD06 else [(0, 0), (1, -1), (-1, 1)]
        for bc in bcs:
            op = oracle.OracleOp(scheme, n, dx, periodic, *bc)
            for axis, mode in ((1, SWZ), (1, PACK), (2, ROWS), (3, ROWS), (2, ODD), (3, ODD)):
                f = rng.standard_normal({1: (3, 5, n), 2: (2, n, 11), 3: (n, 2, 11)}[axis])
                na, nb = [s for a, s in enumerate(f.shape[::-1]) if a != axis - 1]
                ref = op.apply(kind, axis, f, na, nb, *bc).reshape(f.shape)
                for m in (8, 16, 32):
                    if mode == SWZ and n % 2:
                        continue
                    out = np.full_like(f, np.nan)
                    rc = _run(emul, scheme, kind, n, dx, periodic, bc, bc, m, mode, axis, 0, 1.0, f, out)
                    if rc == -2:
                        continue  # the line does not cut into segments of m rows
                    assert rc == 0
                    cuts += 1
                    err = np.abs(out - ref).max() / np.abs(ref).max()
                    assert err <= 1e-12, (n, m, mode, axis, bc, err)
    assert cuts > 60


@pytest.mark.parametrize("scheme,kind", OPS)
def test_x_lines_round_alike_in_every_tile(emul, scheme, kind):
    """Even lengths whose cut shares rows: the swizzled and the packed tile give the same bits."""
    rng = np.random.default_rng(8 + scheme + kind)
    for n, m, periodic in itertools.product((50, 90, 200, 512, 1000), (8, 16, 32), (True, False)):
        f = rng.standard_normal((3, 5, n))
        outs = [np.full_like(f, np.nan) for _ in range(2)]
        rcs = [_run(emul, scheme, kind, n, 0.3, periodic, (0, 0), (0, 0), m, mode, 1, 0, 1.0, f, out)
               for mode, out in zip((SWZ, PACK), outs)]
        assert rcs[0] == rcs[1]
        if rcs[0] == 0:
            assert np.array_equal(*outs), (n, m, periodic)


def test_register_kernel_output_modes_emulated(emul):
    rng = np.random.default_rng(5)
    n = 72
    for scheme, kind in OPS:
        op = oracle.OracleOp(scheme, n, 0.2, False)
        for axis, mode in ((1, SWZ), (1, PACK), (3, ROWS)):
            f = rng.standard_normal({1: (3, 5, n), 3: (n, 2, 11)}[axis])
            na, nb = [s for a, s in enumerate(f.shape[::-1]) if a != axis - 1]
            ref = op.apply(kind, axis, f, na, nb).reshape(f.shape)
            df0 = rng.standard_normal(f.shape)
            for out_mode, beta in ((1, 0.0), (2, 1.0)):
                out = df0.copy()
                assert _run(emul, scheme, kind, n, 0.2, False, (0, 0), (0, 0), 16, mode, axis, out_mode, -0.75, f, out) == 0
                expect = -0.75 * ref + beta * df0
                assert np.abs(out - expect).max() / np.abs(expect).max() <= 1e-12, (scheme, kind, mode, out_mode)


def test_register_kernel_other_system_emulated(emul):
    """The complex z filter: closures in the right-hand side, the (0, 0) system solved."""
    from oracle import dense

    rng = np.random.default_rng(6)
    n = 60
    A = dense.lhs(dense.CF90, dense.FILTER, n, False, 0, 0)
    for bc in ((1, -1), (-1, 1), (0, 1)):
        D = np.linalg.solve(A, dense.rhs(dense.CF90, dense.FILTER, n, 1.0, False, *bc))
        f = rng.standard_normal((n, 2, 11))
        out = np.empty_like(f)
        assert _run(emul, dense.CF90, dense.FILTER, n, 1.0, False, bc, (0, 0), 16, ROWS, 3, 0, 1.0, f, out) == 0
        ref = dense.apply_axis(D, f, 3)
        assert np.abs(out - ref).max() / np.abs(ref).max() <= 1e-12, bc


@pytest.mark.parametrize("scheme,kind", OPS[:3])
def test_walls_lose_no_precision_emulated(emul, scheme, kind):
    """Smooth fields on lines with walls, whose error is the closure rows': against the operator formed in
    extended precision no further off than the oracle, which eliminates and substitutes in the reference's
    order -- by no more than 1% in the geometric mean of the lines, 10% (the luck of 64 fields' rounding)
    on any."""
    from perf import cases

    rng = np.random.default_rng(3)
    ratios = []
    for n in (24, 25, 33, 36, 40, 48, 50, 64, 77, 100, 127, 128, 191, 256):
        for bc in [(0, 0)] if scheme == oracle.CD06 else [(0, 0), (0, 1), (-1, 0)]:
            dx = 1.0 / (n - 1)
            t, c = np.linspace(0, 1, n)[:, None, None], rng.standard_normal((8, 1, 1, 64))
            f = np.ascontiguousarray(c[0] + c[1] * t + c[2] * t ** 2 + c[3] * t ** 3 + c[4] * np.sin(5 * t + c[5])
                                     + c[6] * np.cos(11 * t + c[7]))
            D = cases._dense({oracle.CD06: "cd06", oracle.CD10: "cd10"}[scheme], kind, n, dx, False, *bc)
            exact = np.tensordot(D.astype(np.longdouble), f.astype(np.longdouble), axes=(1, 0))
            ref = oracle.OracleOp(scheme, n, dx, False, *bc).apply(kind, 3, f, 64, 1, *bc).reshape(f.shape)
            out = np.full_like(f, np.nan)
            assert 0 in (_run(emul, scheme, kind, n, dx, False, bc, bc, m, ROWS, 3, 0, 1.0, f, out) for m in (32, 16, 8))
            err = [float(np.sqrt(np.square(v - exact).sum())) for v in (out, ref)]
            ratios.append(err[0] / err[1])
    assert np.exp(np.log(ratios).mean()) <= 1.01, ratios
    assert max(ratios) <= 1.1, ratios


# operator -> (RHS_ST_*, alpha, taps a, b, power of 1/dx, sign)
STAGG = {"ddz_E2C": (4, 9 / 62, 63 / 62, 17 / 186, 1, -1), "ddz_C2E": (5, 9 / 62, 63 / 62, 17 / 186, 1, -1),
         "InterpZ_E2C": (4, 0.3, 0.75, 0.05, 0, 1), "InterpZ_C2E": (5, 0.3, 0.75, 0.05, 0, 1),
         "ddz_C2C": (6, 1 / 3, 7 / 9, 1 / 36, 1, -1), "ddz_E2E": (6, 1 / 3, 7 / 9, 1 / 36, 1, -1),
         "d2dz2_C2C": (7, 2 / 11, 12 / 11, 3 / 44, 2, -1), "d2dz2_E2E": (7, 2 / 11, 12 / 11, 3 / 44, 2, -1)}


@pytest.mark.parametrize("name", STAGG)
@pytest.mark.parametrize("n", [24, 33, 64, 100])
def test_staggered_operators_emulated(emul, name, n):
    """The staggered operators' interior, end blocks (closure rows as one dense
    group each, taken from the oracle's right-hand side of unit fields) and
    cyclic wraps, against the oracle."""
    from oracle.stagg import Stagg

    rng = np.random.default_rng(n)
    rk, alpha, a, b, order, sign = STAGG[name]
    dx = 0.37
    setups = [(True,)] if name not in ("ddz_C2C", "ddz_E2E") else []
    setups += [(False, True, False, False, False), (False, False, True, False, False), (False, True, True, True, True)]
    for setup in setups:
        S = Stagg(n, dx, *setup)
        op = S.OPS[name]
        nin = n + 1 if name.split("_")[1].startswith("E") else n
        nout = n + 1 if name.endswith("E") else n
        f = rng.standard_normal((nin, 1, 13))
        ref = S.apply(name, f)
        rows = np.zeros((8, 3, 9))
        if setup[0]:
            lhs, solved = np.zeros((3, n)), n
        else:
            T = S.tri[op]  # lower / pivot, 1 / pivot, upper / pivot
            lower, upper = T[:, 0] / T[:, 1], T[:, 2] / T[:, 1]
            diag = 1 / T[:, 1] + np.concatenate([[0.0], lower[1:] * T[:-1, 2]])
            lhs, solved = np.stack([lower, diag, upper]), nout
            B = S._rhs_nonperiodic(op, np.eye(nin)[:, None, :])[:, 0, :]
            rows[:, 0, 0] = 1.0
            rows[:4, 0, 1:] = B[:4, :8]
            rows[4:, 0, 1:] = B[-4:, -8:]
        par = np.array([alpha, a / dx ** order, b / dx ** order, sign])
        lhs = np.ascontiguousarray(lhs)
        ran = 0
        for m, mode in itertools.product((8, 16, 32), (ROWS, ODD)):
            out = np.full_like(ref, np.nan)
            rc = emul.emul_reg_stagg(rk, solved, nin, int(setup[0]), int(setup[0] and nout > n), par.ctypes.data,
                                     lhs.ctypes.data, rows.ctypes.data, m, mode, f.ctypes.data, out.ctypes.data, 13)
            if rc == -2:
                continue
            assert rc == 0
            ran += 1
            err = np.abs(out - ref).max() / np.abs(ref).max()
            assert err <= 1e-12, (name, n, setup, m, mode, err)
        assert ran


def test_runtime_answers_are_kept_per_device(emul):
    """A kernel's shared-memory grant and occupancy: asked once on each device, again after a failure (0)."""
    V = ctypes.c_int * 6
    got, asked = V(), V()
    emul.emul_once_per_device(6, V(0, 0, 1, 1, 1, 0), V(3, 9, 0, 2, 9, 9), got, asked)
    assert list(got) == [3, 3, 0, 2, 2, 3]
    assert list(asked) == [1, 0, 1, 1, 0, 0]
