"""FP64 residuals of the mixed form, each point against its own terms.

After one sweep the correction of a point that no other point of the first
colour reaches is omega / lhs times its residual: u's change shows the residual
to the last bits that u holds."""
import numpy as np
import pytest

import x2dhf_gb300 as xg

pytestmark = pytest.mark.gpu

LD = np.longdouble


@pytest.fixture(scope="module")
def ctx():
    c = xg.Context(0)
    yield c
    c.close()


def _first_points(nnu, nmu):
    """Ext indices of the points that are relaxed before any of their neighbours."""
    order, pts, tile, colour, level = xg.host_schedule(nnu, nmu)
    return pts[(colour == 0) & (level == 0)]


def _fields(nnu, nmu, rng):
    row, col = np.arange(nmu)[:, None], np.arange(nnu)[None, :]
    rand = lambda: rng.standard_normal((nmu, nnu))  # noqa: E731
    spikes = rand() * (rng.random((nmu, nnu)) < 0.01)
    return {"smooth": np.exp(-0.01 * row) * np.cos(0.01 * col), "random": rand(), "spikes": spikes,
            # one value in a hundred far above the others: the ends of many stencils
            "arms": spikes + 2.0 ** -14 * rand(),
            "steep": np.exp(-0.43 * (row % 100)) * (1.0 + 0.1 * rand()),
            "steeper": rand() * np.exp(-0.95 * (row % 50) - 0.5 * (col % 50)),
            "axis": np.sin(np.pi * col / (nnu - 1)) ** 2 * np.exp(-0.02 * row)}


def _extended(v, isym):
    """The field with its axis values and ghosts; odd functions vanish on the axes."""
    nmu, nnu = v.shape
    if isym == -1:
        v = v.copy()
        v[0] = v[:, 0] = v[:, -1] = 0.0
    u = np.zeros((nmu + 8, nnu + 8))
    u[4:nmu + 4, 4:nnu + 4] = v
    for k in range(1, 5):
        u[4:nmu + 4, 4 - k] = isym * v[:, k]
        u[4:nmu + 4, nnu + 3 + k] = isym * v[:, nnu - 1 - k]
        u[4 - k, 4:nnu + 4] = isym * v[k, :]
    return u


class Operator:
    """The potentials' operator on all points of a list (ext indices), in long double."""

    def __init__(self, g, nnu, nmu, points):
        self.hni, self.hmu = np.pi / (nnu - 1), np.arccosh(25.0) / (nmu - 1)
        self.f3, self.e, self.g, bpot, d = (g.table(k).reshape(nmu, nnu) for k in (7, 3, 9, 1, 2))
        self.row, self.col = points // (nnu + 8), points % (nnu + 8)
        self.ik = (self.row - 4, self.col - 4)
        self.b, self.d = bpot[self.ik], d[self.ik]

    def lhs(self, idel):
        return (self.f3 + idel * idel * self.e)[self.ik]

    def apply(self, u, idel):
        """A u, the sum of its terms' absolute values, and that of the weights' two parts."""
        a2, a1 = np.array([-9.0, 128, -1008, 8064]) / 5040.0, np.array([3.0, -32, 168, -672]) / 840.0
        au = LD(self.lhs(idel)) * LD(u[self.row, self.col])
        terms, parts = abs(au), LD(0)
        for q in range(4):
            for dr, dc, h, b in ((4 - q, 0, self.hmu, self.b), (0, 4 - q, self.hni, self.d)):
                w2, w1 = a2[q] / (h * h), a1[q] / h
                for s, w in ((-1, w2 + b * w1), (1, w2 - b * w1)):
                    x = LD(u[self.row + s * dr, self.col + s * dc])
                    au, terms, parts = au + LD(w) * x, terms + abs(w * x), parts + (abs(w2) + abs(b * w1)) * abs(x)
        return au, terms, parts

    def source(self, u, idel, start):
        """psa for which, with psb = 1, u solves the equation at the points to 53 bits of its terms."""
        psa = start.copy()
        psa[self.row, self.col] = (self.apply(u, idel)[0] / LD(self.g[self.ik])).astype(np.float64)
        return psa


# potentials on chip (both row pitches), and a grid that takes the persistent-band sweep
@pytest.mark.parametrize("nnu,nmu", [(91, 121), (361, 91), (811, 121)])
@pytest.mark.parametrize("mode", [True, False], ids=["fixed", "fma"])
def test_residual_of_every_point_in_terms_of_its_own(ctx, nnu, nmu, mode):
    """18 roundings to 53 bits of sums that the absolute terms bound, an FP32
    rounding of the residual, of omega / lhs (from two rounded terms and a fast
    reciprocal, 2^-21) and of their product, and u's own last bit.  (A sum in
    units of values a tile away, as a point left to it wrongly has, is off by
    up to 2^-42 of its terms.)"""
    torch = pytest.importorskip("torch")
    g = xg.Grid(ctx, nnu, nmu, 2.0, 25.0, 1.0, 1.0)
    dev, rng, omega = torch.device("cuda:0"), np.random.default_rng(nnu), 1.8
    op = Operator(g, nnu, nmu, _first_points(nnu, nmu))
    row, col = op.row, op.col
    one = torch.ones((nmu + 8) * (nnu + 8), dtype=torch.float64, device=dev)
    cases, jobs = [], []
    for name, v in _fields(nnu, nmu, rng).items():
        for idel, isym in ((0, 1), (1, -1), (2, 1)):
            u = _extended(v, isym)
            # near its solution, so that the residual is what the rounding leaves
            psa = op.source(u, idel, np.zeros_like(u))
            bare = u.copy()
            bare[0:4], bare[4:nmu + 4, 0:4], bare[4:nmu + 4, nnu + 4:] = 0.0, 0.0, 0.0  # ghosts are not the caller's
            du, dpsa = (torch.tensor(x.ravel(), device=dev) for x in (bare, psa))
            cases.append((name, idel, u, psa, du, dpsa))
            jobs.append(xg.Job(u=du.data_ptr(), psa=dpsa.data_ptr(), psb=one.data_ptr(), omega=omega, isym=isym, idel=idel,
                               kind=1))
    ctx.set_potential_clusters(mode)
    torch.cuda.synchronize()
    try:
        xg.relax(ctx, g, jobs, 1, xg.MIXED)
        ctx.synchronize()
    finally:
        ctx.set_potential_clusters("auto")
    eps = LD(2.0) ** -53
    for name, idel, u, psa, du, _ in cases:
        lhs = LD(op.lhs(idel))
        au, terms, parts = op.apply(u, idel)
        rhs = LD(psa[row, col]) * LD(op.g[op.ik])
        r, terms = rhs - au, terms + abs(rhs)
        # and the weights: formed here and there from steps that differ in their last bit, with four roundings
        off = 18 * eps * terms + 8 * eps * parts
        want = omega * r / lhs
        got = LD(du.cpu().numpy().reshape(u.shape)[row, col]) - LD(u[row, col])
        bound = abs(omega / lhs) * off + LD(2.0) ** -20 * abs(want) + eps * (abs(LD(u[row, col])) + abs(want))
        worst = float((abs(got - want) / (bound + LD(1e-300))).max())
        assert worst <= 1, (name, idel, worst)
    g.close()


@pytest.mark.parametrize("nnu,nmu", [(151, 241), (331, 481)])
@pytest.mark.parametrize("on_chip", [True, False])
def test_potential_does_not_depend_on_its_batch(ctx, nnu, nmu, on_chip):
    """Without the potentials' kernel a potential relaxed alone and among
    others is the same bit for bit, whatever the size of the batch."""
    torch = pytest.importorskip("torch")
    g = xg.Grid(ctx, nnu, nmu, 2.0, 25.0, 1.0, 1.0)
    dev, rng = torch.device("cuda:0"), np.random.default_rng(3)
    # at their solutions: the residual, and with it the result, is what its rounding leaves
    inner = (np.arange(5, nmu)[:, None] * (nnu + 8) + np.arange(5, nnu + 3)[None, :]).ravel()
    op = Operator(g, nnu, nmu, inner)
    fields = [_extended(rng.standard_normal((nmu, nnu)), 1) for _ in range(5)]
    u0 = [torch.tensor(u.ravel(), device=dev) for u in fields]
    psa = [torch.tensor(op.source(u, k % 3, np.zeros_like(u)).ravel(), device=dev) for k, u in enumerate(fields)]
    one = torch.ones_like(u0[0])

    def relaxed(groups):
        us = [u.clone() for u in u0]
        torch.cuda.synchronize()
        for group in groups:
            xg.relax(ctx, g, [xg.Job(u=us[k].data_ptr(), psa=psa[k].data_ptr(), psb=one.data_ptr(), omega=1.8, isym=1,
                                     idel=k % 3, kind=1) for k in group], 3, xg.MIXED)
        ctx.synchronize()
        return us

    ctx.set_potential_clusters(False)
    ctx.set_mixed_on_chip(on_chip)
    try:
        together, alone = relaxed([range(5)]), relaxed([[k] for k in range(5)])
    finally:
        ctx.set_potential_clusters("auto")
        ctx.set_mixed_on_chip(True)
    for k, (x, y) in enumerate(zip(together, alone)):
        assert torch.equal(x, y), k
    # and in the default, where one kernel takes both batches
    together, alone = relaxed([range(5)]), relaxed([[k] for k in range(5)])
    for k, (x, y) in enumerate(zip(together, alone)):
        assert torch.equal(x, y), k
    g.close()
