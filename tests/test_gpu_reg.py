"""GPU: the register kernel (the automatic choice for lines of 24 points and
more) against the oracle (1e-12 of max |oracle|): at line lengths on the edges
of its cuts -- no shared rows, the most, one segment -- with partial tiles and
chunks, and the same field through the streaming kernel, the path it replaced;
every tile layout and copy form on fields of more tiles than resident CTAs,
stored, scaled and accumulated.  Every case asserts that the kernel is the one
that would run."""
import numpy as np
import pytest

import oracle
from tests.fields import na_nb, rel_err
from tests.test_gpu_parity import OPS, _make, _oracle_apply

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _shape(n, axis, odd):
    e = 1 if odd else 0
    return {1: (61, 83, n), 2: (37, n, 70 + e), 3: (n, 37, 70 + e)}[axis]


@pytest.mark.parametrize("scheme,kind", OPS)
@pytest.mark.parametrize("n", [24, 31, 32, 50, 64, 72, 127, 128, 200])
def test_register_kernel(scheme, kind, n):
    import torch

    rng = np.random.default_rng(11 + n + 3 * scheme + kind)
    for periodic in (True, False):
        op = _make(scheme, n, 0.3, periodic)
        bc = (0, 0) if periodic or scheme == oracle.CD06 else [(0, 0), (1, -1), (-1, 1)][n % 3]
        for axis in (1, 2, 3):
            for odd in (False, True) if axis != 1 else (n % 2 == 1,):
                shape = _shape(n, axis, odd)
                f = rng.standard_normal(shape)
                ft = torch.from_numpy(f).cuda()
                na, nb = na_nb(shape, axis)
                out = torch.full_like(ft, float("nan"))
                plan = op.launch_plan(kind, axis, ft, out, na, nb, *bc)
                assert plan["variant"] == (6 if odd else 4) and plan["register"]
                op.apply(kind, axis, ft, out, na, nb, *bc)
                torch.cuda.synchronize()
                assert op.device_status() == 0
                ref = _oracle_apply(scheme, kind, axis, f, 0.3, periodic, *bc)
                assert rel_err(out.cpu().numpy(), ref) <= TOL, (periodic, axis, odd)
                general = torch.full_like(ft, float("nan"))
                op.set_variant(plan["variant"])
                assert not op.launch_plan(kind, axis, ft, general, na, nb, *bc)["register"]
                op.apply(kind, axis, ft, general, na, nb, *bc)
                op.set_variant(0)
                assert rel_err(out.cpu().numpy(), general.cpu().numpy()) <= TOL, (periodic, axis, odd)


@pytest.mark.parametrize("scheme,kind", OPS)
@pytest.mark.parametrize("n", [1000, 1024, 2048])
def test_register_kernel_long_lines(scheme, kind, n):
    import torch

    rng = np.random.default_rng(n + 3 * scheme + kind)
    for periodic in (True, False):
        op = _make(scheme, n, 0.3, periodic)
        for axis, shape in ((1, (3, 7, n)), (2, (2, n, 18)), (3, (n, 3, 18))):
            f = rng.standard_normal(shape)
            ft = torch.from_numpy(f).cuda()
            na, nb = na_nb(shape, axis)
            out = torch.full_like(ft, float("nan"))
            assert op.launch_plan(kind, axis, ft, out, na, nb)["register"]
            op.apply(kind, axis, ft, out, na, nb)
            torch.cuda.synchronize()
            assert op.device_status() == 0
            ref = _oracle_apply(scheme, kind, axis, f, 0.3, periodic, 0, 0)
            assert rel_err(out.cpu().numpy(), ref) <= TOL, (periodic, axis)


def _at(torch, a, offset):
    """A device copy of the array that starts `offset` elements past a 16-byte boundary."""
    t = torch.empty(a.size + offset, dtype=torch.float64, device="cuda")[offset:].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


# axis, rows, cross extent, elements past a 16-byte boundary, stages
TILES = [
    (1, 64, 83, 0, 2),     # swizzled, two buffers
    (1, 100, 83, 0, 2),    # the same with a partial chunk
    (1, 1800, 9, 0, 1),    # swizzled, one buffer
    (1, 127, 83, 0, 2),    # one span each way, two buffers
    (1, 511, 21, 0, 2),
    (1, 96, 83, 1, 1),     # per-element copies
    (2, 100, 70, 0, 1),    # boxes of rows
    (3, 512, 70, 0, 1),    # more rows than a box holds
    (2, 100, 71, 0, 1),    # rows of either parity apart: every plane starts on the same one
    (2, 101, 71, 0, 1),    # ... on another one each
    (3, 90, 71, 0, 1),
    (2, 100, 70, 1, 1),    # per-element copies
    (3, 129, 71, 1, 1),
]


@pytest.mark.parametrize("scheme,kind", OPS)
@pytest.mark.parametrize("axis,n,cross,offset,stages", TILES)
def test_register_kernel_many_tiles(scheme, kind, axis, n, cross, offset, stages):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(n + 7 * axis + 3 * scheme + kind)
    for periodic in (True, False):
        op = _make(scheme, n, 0.3, periodic)
        bc = (0, 0) if periodic or scheme == oracle.CD06 else (1, -1)
        planes = 9
        while True:  # as many planes as give every CTA two tiles and more
            shape = {1: (planes, cross, n), 2: (planes, n, cross), 3: (n, planes, cross)}[axis]
            na, nb = na_nb(shape, axis)
            ft = _at(torch, np.zeros(shape), offset)
            plan = op.launch_plan(kind, axis, ft, _at(torch, np.zeros(shape), offset), na, nb, *bc)
            assert plan["register"] and plan["stages"] == stages, plan
            L = plan["lines"]
            tiles = -(-na // L) * nb if axis == 2 else -(-na * nb // L)
            if tiles > 2 * plan["ctas_per_sm"] * sms:
                break
            planes = 2 * planes + 1
        f, df0 = rng.standard_normal(shape), rng.standard_normal(shape)
        ft = _at(torch, f, offset)
        ref = _oracle_apply(scheme, kind, axis, f, 0.3, periodic, *bc)
        for alpha, beta in ((1.0, 0.0), (-0.75, 0.0), (-0.75, 1.0)):
            out = _at(torch, df0 if beta else np.full(shape, np.nan), offset)
            op.apply(kind, axis, ft, out, na, nb, *bc, alpha=alpha, beta=beta)
            expect = alpha * ref + beta * df0
            assert rel_err(out.cpu().numpy(), expect) <= TOL, (periodic, alpha, beta)
        assert op.device_status() == 0


@pytest.mark.parametrize("scheme,kind", OPS)
@pytest.mark.parametrize("n,n2,n3", [(1023, 69, 35), (1701, 109, 11)])
def test_register_kernel_odd_lines_one_buffer(scheme, kind, n, n2, n3):
    """x lines of an odd length for which one tile buffer fits, a field of an odd number of elements (a last
    tile of 15 or 7 lines) and more tiles than CTAs: a CTA places the field's last element in the buffer whose
    results it has just handed to the copy engine.  Whole outputs, 50 times over."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(n + 3 * scheme + kind)
    f = rng.standard_normal((n3, n2, n))
    df0 = rng.standard_normal(f.shape)
    ft, df0t = torch.from_numpy(f).cuda(), torch.from_numpy(df0).cuda()
    for periodic in (True, False):
        op = _make(scheme, n, 0.3, periodic)
        out = torch.empty_like(ft)
        plan = op.launch_plan(kind, 1, ft, out, n2, n3)
        tiles = -(-n2 * n3 // plan["lines"])
        assert plan["register"] and plan["stages"] == 1 and tiles > plan["ctas_per_sm"] * sms, plan
        assert n2 * n3 % plan["lines"] == plan["lines"] - 1
        ref = _oracle_apply(scheme, kind, 1, f, 0.3, periodic, 0, 0)
        for alpha, beta in ((1.0, 0.0), (-0.75, 1.0)):
            first = None
            for _ in range(50):
                if beta:
                    out.copy_(df0t)
                else:
                    out.fill_(float("nan"))
                op.apply(kind, 1, ft, out, n2, n3, alpha=alpha, beta=beta)
                if first is None:
                    first = out.clone()
                    assert rel_err(first.cpu().numpy(), alpha * ref + beta * df0) <= TOL, (periodic, beta)
                assert torch.equal(out, first), (periodic, beta)
        assert op.device_status() == 0


@pytest.mark.parametrize("scheme,kind", OPS)
def test_refused_tiling_changes_nothing(scheme, kind):
    """Segments of 16 rows do not cover 1024: the call is refused, and the handle launches what it did."""
    import torch

    from padeops_b200 import PadoError

    op = _make(scheme, 1024, 0.3, True)
    ft = torch.zeros((4, 64, 1024), dtype=torch.float64, device="cuda")
    before = op.launch_plan(kind, 1, ft, torch.empty_like(ft), 64, 4)
    with pytest.raises(PadoError):
        op.set_tiling(16, 8)
    assert op.launch_plan(kind, 1, ft, torch.empty_like(ft), 64, 4) == before


@pytest.mark.parametrize("scheme,kind", OPS)
def test_rounding_does_not_depend_on_the_address(scheme, kind):
    """A field 8 bytes past a 16-byte boundary, input, output or both: other copies, the same bits."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(5 + scheme + kind)
    for n in (50, 64, 90, 129, 200, 512, 1000):
        for periodic in (True, False):
            op = _make(scheme, n, 0.3, periodic)
            for axis, cross in ((1, 22), (2, 22), (2, 21), (3, 22), (3, 21)):
                shape = {1: (9, 11, n), 2: (9, n, cross), 3: (n, 9, cross)}[axis]
                na, nb = na_nb(shape, axis)
                size = n * na * nb
                base = torch.randn(size, dtype=torch.float64, device="cuda", generator=g)
                outs = []
                for off_in, off_out in ((0, 0), (1, 0), (0, 1), (1, 1)):
                    f = torch.zeros(size + 1, dtype=torch.float64, device="cuda")[off_in:off_in + size]
                    f.copy_(base)
                    out = torch.full((size + 1,), float("nan"), dtype=torch.float64, device="cuda")[off_out:off_out + size]
                    op.apply(kind, axis, f, out, na, nb)
                    outs.append(out)
                for out in outs[1:]:
                    assert torch.equal(out, outs[0]), (n, periodic, axis, cross)
            assert op.device_status() == 0


@pytest.mark.parametrize("scheme,kind", OPS)
@pytest.mark.parametrize("n", [25, 64, 129])
def test_lines_across_a_field_one_point_wide(scheme, kind, n):
    """y lines of a field of extent 1 along x follow one another in memory: they are tiled as x lines, stored,
    accumulated and transposed, and give an x line's bits."""
    import torch

    rng = np.random.default_rng(n + scheme + kind)
    f = rng.standard_normal((2003, n, 1))
    ft = torch.from_numpy(f).cuda()
    for periodic in (True, False):
        op = _make(scheme, n, 0.3, periodic)
        outs = [torch.full_like(ft, float("nan")) for _ in range(2)]
        plans = [op.launch_plan(kind, axis, ft, out, na, nb)
                 for out, axis, na, nb in zip(outs, (2, 1), (1, 2003), (2003, 1))]
        assert plans[0]["register"] and plans[0] == plans[1]
        op.apply(kind, 2, ft, outs[0], 1, 2003)
        op.apply(kind, 1, ft, outs[1], 2003, 1)
        assert torch.equal(*outs)
        assert rel_err(outs[0].cpu().numpy(), _oracle_apply(scheme, kind, 2, f, 0.3, periodic, 0, 0)) <= TOL
        acc = [ft.clone(), ft.clone()]
        op.apply(kind, 2, ft, acc[0], 1, 2003, alpha=-0.5, beta=1.0)
        op.apply(kind, 1, ft, acc[1], 2003, 1, alpha=-0.5, beta=1.0)
        assert torch.equal(*acc)
        adj = torch.full_like(ft, float("nan"))
        op.apply(kind, 2, ft, adj, 1, 2003, adjoint=True)
        g = torch.from_numpy(rng.standard_normal(f.shape)).cuda()
        op.apply(kind, 2, g, outs[1], 1, 2003)
        bound = 1e-12 * float(outs[1].norm() * ft.norm())
        assert abs(float((outs[1] * ft).sum()) - float((g * adj).sum())) <= bound, periodic
        assert op.device_status() == 0
