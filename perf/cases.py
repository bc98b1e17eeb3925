"""The work a user of this library has it do, as cases that can be timed and checked.

Three kinds of case, each through a public entry point:

  relax   one relaxation call, `x2dhf_gb300.relax`: a batch of functions on one grid, `sweeps` micro sweeps each, in the
          plain FP64 form, the mixed form or list-order SOR; the functions are potentials built from two orbitals or
          orbitals with their own lhs and rhs arrays
  host    the same call on host buffers, `x2dhf_gb300.mcsor_host` (what the reference's `mcsor_pthread_` does)
  scf     a whole SCF from its input deck: grid, hydrogenic start, iterations, energies and orbitals read back

The functions to relax are what an SCF under way holds: the analytic solution of the equation (the potential of a product
of two Slater functions; a hydrogenic orbital, part of its operator moved to the right-hand side) plus a smooth relative
error of 1e-5, with consistent axis values and ghost cells.  `exact` runs the same sweeps in 64 bits, colour by colour (or
level by level), in plain torch."""
import math

import numpy as np
import torch

import x2dhf_gb300 as xg

DEV = "cuda"

# grids (N_nu, N_mu), N = 1 (mod 30) as the reference rounds them, with (R, R_inf): He / H2 / Ne / LiH / N2 / KF sizes
# and the range of the serving stream (169..505 x 241..721 before rounding)
GRIDS = {(91, 121): (2.0, 35.0), (151, 241): (1.4, 40.0), (151, 181): (2.0, 35.0), (241, 301): (3.015, 60.0),
         (331, 481): (2.068, 40.0), (481, 721): (2.132, 40.0), (781, 1201): (4.1035, 60.0)}

H2_DECK = """title H2
method hf
nuclei  1.0 1.0  {r}
config 0
  1 sigma g end
grid {nnu} {nmu} 40.0
orbpot hydrogen
lcao
 1.0 1 0 1.0   1.0   1 0  1.0
scf  {iters} 0 12 14 1
mcsor
mcsor-ce
stop
"""

N2_DECK = """title N2
method hf
nuclei  7.0 7.0 {r}
config  0
  1 pi    u
  1 sigma g
  1 sigma u
  1 sigma g
  1 sigma u
  1 sigma g end
grid {nnu} {nmu} 40.0
orbpot hydrogen
lcao
  0.5   2 1 5.0     0.5   2 1 5.0
  1.5   2 1 5.0     0.0   2 1 5.0
  0.5   2 0 7.0    -0.5   2 0 7.0
  0.5   2 0 7.0     0.5   2 0 7.0
  0.5   1 0 7.0    -0.5   1 0 7.0
  0.5   1 0 7.0     0.5   1 0 7.0
scf {iters} 0 12 14 1
conv 5000
mcsor
mcsor-ce
stop
"""

# no mcsor card: list-order SOR for orbitals and potentials, the reference's default
NE_DECK = """title Ne
method hf
nuclei  10.0  0.0  {r}
config  0
1 pi
2 sigma
1 sigma   end
grid {nnu} {nmu} 35.0
orbpot hydrogen
lcao
1.0   2 1   6.0     0.0   1 0 9.0
1.0   2 1   8.0     0.0   1 0 9.0
1.0   2 0   9.0     0.0   1 0 9.0
1.0   1 0  10.0     0.0   1 0 9.0
scf {iters} 0 10 12 3
conv 2000
stop
"""

DECKS = {"h2": (H2_DECK, 1.4), "n2": (N2_DECK, 2.068), "ne": (NE_DECK, 2.0)}


def relax_case(what, form, nnu, nmu, jobs, sweeps=10, **more):
    return dict(more, kind="relax", what=what, form=form, nnu=nnu, nmu=nmu, jobs=jobs, sweeps=sweeps)


def scf_case(molecule, form, mode, nnu, nmu, iters, **more):
    return dict(more, kind="scf", molecule=molecule, form=form, mode=mode, nnu=nnu, nmu=nmu, iters=iters)


def listed():
    return [
        # the smallest call: one He orbital on host buffers, as a Fortran host program makes it
        dict(relax_case("orbital", "fp64", 91, 121, 1, name="host_orbital_he"), kind="host"),
        # one orbital of H2 in the mixed form: what an SCF of one orbital launches between two synchronisations
        relax_case("orbital", "mixed", 151, 241, 1, name="mixed_orbital_h2"),
        # the 6 orbitals and the 22 potentials of an N2 iteration in the mixed batched form
        relax_case("orbital", "mixed", 331, 481, 6, name="mixed_orbitals_n2"),
        relax_case("potential", "mixed", 331, 481, 22, name="mixed_potentials_n2"),
        # a batch of independent Poisson solves on that grid
        relax_case("potential", "mixed", 331, 481, 64, name="mixed_poisson_b64"),
        # the large grid, beyond one cluster's shared memory: half of KF's potentials, one more than a launch's job table
        relax_case("potential", "mixed", 781, 1201, 33, name="mixed_potentials_kf"),
        # plain FP64: one orbital's potentials in the reference's order (up to 7 at once on N2), and the batched form
        relax_case("potential", "fp64", 331, 481, 5, name="fp64_potentials_n2"),
        relax_case("potential", "fp64", 331, 481, 22, name="fp64_batch_n2"),
        # list-order SOR, the reference's default: an orbital on the N2 grid
        relax_case("orbital", "sor", 331, 481, 1, name="sor_orbital_n2"),
        # whole calls: H2 and N2 in the mixed batched form, Ne as its deck has it (FP64, SOR, reference order)
        scf_case("h2", "mixed", 2, 151, 241, 160, name="scf_h2_mixed"),
        scf_case("n2", "mixed", 2, 331, 481, 600, name="scf_n2_mixed"),
        scf_case("ne", "fp64", 0, 151, 181, 20, name="scf_ne_sor"),
    ]


def draw(rng):
    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return 30 * ((n - 1) // 30) + 1

    if rng.random() < 0.2:
        if rng.random() < 0.5:
            return scf_case("h2", "mixed", rng.choice((0, 1, 2)), size(121, 190), size(151, 310),
                            10 * rng.randint(18, 30))
        return scf_case("ne", "fp64", rng.choice((0, 1, 2)), size(121, 190), size(151, 220), rng.randint(8, 14))
    form = rng.choice(("mixed", "mixed", "mixed", "fp64", "sor"))
    what = rng.choice(("orbital", "potential"))
    if form == "mixed" and rng.random() < 0.25:
        nnu, nmu = size(421, 800), size(721, 1220)  # beyond one cluster's shared memory
        jobs = rng.randint(1, 24)
    else:
        nnu, nmu = size(91, 512), size(121, 730)
        jobs = int(round(math.exp(rng.uniform(0, math.log(40)))))
    sweeps = rng.choice((5, 10, 10, 10, 20))
    # at most a fifth of the largest listed relaxation's updates in the mixed form, less in FP64
    most = (2.5e8 if form == "mixed" else 6e7)
    jobs = max(1, min(jobs, int(most / (nnu * nmu * sweeps))))
    c = relax_case(what, form, nnu, nmu, jobs, sweeps)
    if form == "fp64" and jobs == 1:
        c.update(kind="host")
    return c


def geometry(case):
    """(R, R_inf) of a relaxation case: those of its grid's molecule, N2's elsewhere."""
    return GRIDS.get((case["nnu"], case["nmu"]), (2.068, 40.0))


class Operator:
    """The discretised operator of x2dhf on an (N_nu, N_mu) grid in 64 bits (src/initCBAllocArrays.F90 initCBlocks,
    initSuppl): coordinates, stencil coefficients and the tables the cases need, N_mu x N_nu tensors."""

    def __init__(self, nnu, nmu, r, rinf):
        f8 = dict(dtype=torch.float64, device=DEV)
        self.nnu, self.nmu, self.r = nnu, nmu, r
        hni = math.pi / (nnu - 1)
        hmu = math.acosh(2.0 * rinf / r) / (nmu - 1)
        xi = torch.cosh(torch.arange(nmu, **f8) * hmu)[:, None]
        eta = torch.cos(torch.arange(nnu, **f8) * hni)[None, :]
        xi1, eta1 = torch.sqrt((xi * xi - 1).clamp_min(0)), torch.sqrt((1 - eta * eta).clamp_min(0))
        self.xi, self.eta = xi, eta
        aa1 = torch.tensor([3.0, -32.0, 168.0, -672.0], **f8) / 840.0
        aa2 = torch.tensor([-9.0, 128.0, -1008.0, 8064.0], **f8) / 5040.0
        self.dmu1, self.dmu2, self.dni1, self.dni2 = aa1 / hmu, aa2 / hmu ** 2, aa1 / hni, aa2 / hni ** 2
        self.diag = -14350.0 / 5040.0 * (1 / hmu ** 2 + 1 / hni ** 2)
        inv1 = torch.where(xi1 > 0, 1 / xi1, torch.zeros_like(xi1))
        axis = eta1 < 2.3e-16
        self.b_orb = xi * inv1
        self.b_pot = torch.where(xi1 > 0, xi * inv1 - 2 * xi1 / xi, torch.zeros_like(xi))
        self.d = torch.where(axis, torch.zeros_like(eta), eta / eta1)
        self.f3 = -2.0 / xi ** 2 + self.diag
        self.e = torch.where(axis, torch.zeros_like(eta), -inv1 ** 2 - 1 / eta1 ** 2)
        w = xi * xi - eta * eta
        self.f1 = r * r * w / 2
        self.g = -(r ** 3) * math.pi * xi / 2 * w
        self.f4 = 0.5 * r * xi
        self.ra = (r / 2) * (xi + eta)  # distance from the first centre
        self.sin = torch.sqrt((1 - ((1 + xi * eta) / (xi + eta).clamp_min(1e-300)).clamp(-1, 1) ** 2).clamp_min(0))

    def extended(self, plain, isym):
        """(N_mu+8) x (N_nu+8) array with consistent axis values (even functions extrapolated, odd ones 0) and the
        mirrored ghost cells of putin."""
        nnu, nmu = self.nnu, self.nmu
        v = plain.clone()
        ex = [c / 126.0 for c in (210.0, -120.0, 45.0, -10.0, 1.0)]
        if isym == 1:
            v[0, 1:-1] = sum(c * v[k + 1, 1:-1] for k, c in enumerate(ex))
            v[:nmu - 4, 0] = sum(c * v[:nmu - 4, k + 1] for k, c in enumerate(ex))
            v[:nmu - 4, -1] = sum(c * v[:nmu - 4, -2 - k] for k, c in enumerate(ex))
        else:
            v[0, :] = 0
            v[:, 0] = 0
            v[:, -1] = 0
        u = torch.zeros(nmu + 8, nnu + 8, dtype=torch.float64, device=DEV)
        u[4:nmu + 4, 4:nnu + 4] = v
        for k in range(1, 5):
            u[4:nmu + 4, 4 - k] = isym * v[:, k]
            u[4:nmu + 4, nnu + 3 + k] = isym * v[:, nnu - 1 - k]
            u[4 - k, 4:nnu + 4] = isym * v[k, :]
        return u


def default_omega(nnu, nmu, charge):
    """setOmega: (orbitals, potentials)."""
    rho = 0.5 * (math.cos(math.pi / nmu) + math.cos(math.pi / nnu))
    w = 2.0 * 0.603 / (1.0 + math.sqrt(1.0 - rho * rho)) + 0.79
    return (w - 1.0) * w - 0.001 * charge, w


def functions(case, seed):
    """The functions of a relaxation case: per function its start u (extended), its inputs and its parameters."""
    nnu, nmu = case["nnu"], case["nmu"]
    r, rinf = geometry(case)
    op = Operator(nnu, nmu, r, rinf)
    rng = np.random.default_rng(seed)
    ni = torch.linspace(0, 1, nnu, dtype=torch.float64, device=DEV)[None, :]
    mi = torch.linspace(0, 1, nmu, dtype=torch.float64, device=DEV)[:, None]
    out = []
    for k in range(case["jobs"]):
        a, b, c = rng.uniform(-1, 1, 3)
        error = 1 + 1e-5 * (1 - mi * mi) * (a + b * torch.cos(math.pi * ni) + c * torch.cos(2 * math.pi * mi))
        m = int(k % 3 if case["what"] == "potential" else k % 4 == 1)
        isym = 1 if m % 2 == 0 else -1
        f = dict(m=m, isym=isym, op=op)
        if case["what"] == "potential":
            # psa = r^m sin^m e^(-za r), psb = e^(-zb r) on the first centre: their product's potential is analytic
            za, zb = rng.uniform(0.5, 4.0, 2)
            beta, rr = za + zb, op.ra.clamp_min(1e-9)
            ang = op.sin ** m
            x = beta * rr
            inner = math.gamma(2 * m + 3) * torch.special.gammainc(torch.full_like(x, 2 * m + 3), x)
            v = 4 * math.pi / (2 * m + 1) * ang * (rr ** (-m - 1) * inner / beta ** (2 * m + 3)
                                                   + rr ** m * (x + 1) * torch.exp(-x) / beta ** 2)
            norm = beta ** (2 * m + 3)  # potentials of order 1
            f["psa"] = op.extended(norm * rr ** m * ang * torch.exp(-za * rr), isym)
            f["psb"] = op.extended(torch.exp(-zb * rr), 1)
            f["omega"] = default_omega(nnu, nmu, 1.0)[1]
            f["u"] = op.extended(norm * v * op.f4 * error, isym)
        else:
            # hydrogenic 1s (m = 0) or 2p_pi (m = 1) of charge z on the first centre; a screening term s moved to
            # the right-hand side as s psi
            z = rng.uniform(1.0, 3.0)
            n = m + 1
            psi = (z ** 1.5) * (op.ra * op.sin) ** m * torch.exp(-z * op.ra / n)
            s = -0.3 * op.f1 * torch.exp(-0.5 * op.ra)
            f["lhs"] = ((r * (op.xi + -op.eta) * z - z * z / (2.0 * n * n) * op.f1 + s + m * m * op.e)
                        + op.diag).contiguous()
            f["rhs"] = (s * psi).contiguous()
            f["omega"] = default_omega(nnu, nmu, z)[0]
            f["u"] = op.extended(psi * error, isym)
        out.append(f)
    return out


_context = None


def context():
    """One library context per program, as a user's program keeps it."""
    global _context
    if _context is None:
        _context = xg.Context(0)
    return _context


FORMS = {"fp64": xg.FP64, "mixed": xg.MIXED, "sor": xg.SOR}


def prepare(case, seed):
    ctx = context()
    if case["kind"] == "scf":
        deck, r = DECKS[case["molecule"]]
        # the bond length (for the atom: the distance to the empty centre) near the deck's own
        r = round(r * (1 + 0.02 * np.random.default_rng(seed).uniform(-1, 1)), 6)
        text = deck.format(r=r, nnu=case["nnu"], nmu=case["nmu"], iters=case["iters"])
        return dict(case=case, ctx=ctx, deck=text)
    r, rinf = geometry(case)
    fs = functions(case, seed)
    state = dict(case=case, ctx=ctx, grid=xg.Grid(ctx, case["nnu"], case["nmu"], r, rinf))
    if case["kind"] == "host":
        f = fs[0]
        kind = 0
        if case["what"] == "potential":
            f["lhs"], f["rhs"], kind = *explicit(f), 1
        state.update(isym=f["isym"], job_kind=kind, omega=f["omega"], u=f["u"].cpu().numpy().ravel(),
                     lhs=f["lhs"].cpu().numpy().ravel(), rhs=f["rhs"].cpu().numpy().ravel())
        return state
    jobs = []
    for f in fs:
        j = xg.Job(u=f["u"].data_ptr(), omega=f["omega"], isym=f["isym"])
        if case["what"] == "potential":
            j.psa, j.psb, j.idel, j.kind = f["psa"].data_ptr(), f["psb"].data_ptr(), f["m"], 1
        else:
            j.lhs, j.rhs = f["lhs"].data_ptr(), f["rhs"].data_ptr()
        jobs.append(j)
        f.pop("op")
    state.update(functions=fs, jobs=jobs)
    torch.cuda.synchronize()  # the context's stream is not ordered after torch's
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    if case["kind"] == "scf":
        c = xg.parse_deck(state["deck"], precision=FORMS[case["form"]], batch_mode=case["mode"])
        s = xg.SCF(ctx, c)
        res = s.run()
        out = dict(energies=np.array([res.total_energy, res.electronic_energy, res.virial]),
                   orbital_energies=np.array(res.ee[:c.norb]), iterations=res.iterations,
                   orbitals=[s.orbital(i) for i in range(1, c.norb + 1)])
        s.close()
        return out
    if case["kind"] == "host":
        return xg.mcsor_host(ctx, state["grid"], state["isym"], state["job_kind"], state["omega"], case["sweeps"],
                             state["u"], state["lhs"], state["rhs"])
    xg.relax(ctx, state["grid"], state["jobs"], case["sweeps"], FORMS[case["form"]])
    return [f["u"] for f in state["functions"]]


def work(case):
    """Relaxation: each function and its inputs read once, the function written once; 54 operations per point update.
    SCF: the same for every relaxation of its iterations."""
    nnu, nmu = case["nnu"], case["nmu"]
    points = (nnu - 2) * (nmu - 5)
    if case["kind"] == "scf":
        orbitals, potentials = {"h2": (1, 1), "n2": (6, 22), "ne": (4, 11)}[case["molecule"]]
        calls = case["iters"] * (orbitals + potentials)
        return dict(bytes=32.0 * nnu * nmu * calls, flops=54.0 * points * 10 * calls)
    return dict(bytes=32.0 * nnu * nmu * case["jobs"], flops=54.0 * points * case["sweeps"] * case["jobs"])


# ----------------------------------------------------------------------
# the same sweeps in 64 bits
# ----------------------------------------------------------------------
def explicit(f):
    """lhs and rhs of a function's equation."""
    op = f["op"]
    if "lhs" in f:
        return f["lhs"], f["rhs"]
    inner = (slice(4, op.nmu + 4), slice(4, op.nnu + 4))
    lhs = (op.f3 + float(f["m"] ** 2) * op.e).contiguous()
    return lhs, f["psa"][inner] * f["psb"][inner] * op.g


def middle_list(nnu, nmu):
    """The interior points in the reference's "middle" order (mesh, src/initCBAllocArrays.F90:2503-2544) as indices of
    the extended array."""
    n8 = nnu + 8
    mx, nx = (nmu + 7) // 2, (nnu + 7) // 2
    rows = np.array([mx - i + 6 if i <= mx else i for i in range(6, nmu + 1)]) - 1
    cols = np.array([nx - j + 6 if j <= nx else j for j in range(6, nnu + 4)]) - 1
    return (rows[:, None] * n8 + cols[None, :]).ravel()


def steps_of(nnu, nmu, colours):
    """The list as sets of points that do not read one another: with 5 colours (list position mod 5, MCSOR) or one
    (SOR), each colour level by level, a point's level one above its latest same-colour neighbour earlier in the list."""
    order, n8 = middle_list(nnu, nmu), nnu + 8
    pos = [-1] * (n8 * (nmu + 8))
    for p, ij in enumerate(order.tolist()):
        pos[ij] = p
    offs = [s * k * t for k in range(1, 5) for s in (1, -1) for t in (1, n8)]
    level = [0] * len(order)
    for p, ij in enumerate(order.tolist()):
        near = [level[q] + 1 for q in (pos[ij + o] for o in offs) if 0 <= q < p and (q - p) % colours == 0]
        if near:
            level[p] = max(near)
    level, colour = np.array(level), np.arange(len(order)) % colours
    return [torch.from_numpy(order[(colour == c) & (level == n)]).to(DEV)
            for c in range(colours) for n in range(level[colour == c].max() + 1)]


def exact(case, seed):
    if case["kind"] == "scf":
        return None  # a whole SCF in plain torch would take minutes
    fs = functions(case, seed)
    op, nnu, nmu = fs[0]["op"], case["nnu"], case["nmu"]
    n8 = nnu + 8
    steps = steps_of(nnu, nmu, 1 if case["form"] == "sor" else 5)
    ex = [c / 126.0 for c in (210.0, -120.0, 45.0, -10.0, 1.0)]
    out = []
    for f in fs:
        lhs, rhs = (x.reshape(-1) for x in explicit(f))
        b = (op.b_pot if case["what"] == "potential" else op.b_orb).reshape(-1)
        d, w, even = op.d.reshape(-1), f["omega"], f["isym"] == 1
        u = f["u"].clone()
        flat = u.view(-1)
        for _ in range(case["sweeps"]):
            for ij in steps:
                row, col = ij // n8 - 4, ij % n8 - 4
                ik = row * nnu + col
                mu2, mu1, ni2, ni1 = 0, 0, 0, 0
                for q in range(4):
                    k = 4 - q
                    m, p, le, ri = flat[ij - k * n8], flat[ij + k * n8], flat[ij - k], flat[ij + k]
                    mu2, mu1 = mu2 + op.dmu2[q] * (m + p), mu1 + op.dmu1[q] * (m - p)
                    ni2, ni1 = ni2 + op.dni2[q] * (le + ri), ni1 + op.dni1[q] * (le - ri)
                cc = mu2 + b[row] * mu1 + ni2 + d[col] * ni1
                flat[ij] = w * (rhs[ik] - cc) / lhs[ik] + (1 - w) * flat[ij]
            v = u[4:nmu + 4, 4:nnu + 4]
            v[0, 1:-1] = sum(c * v[k + 1, 1:-1] for k, c in enumerate(ex)) if even else 0
            v[:nmu - 4, 0] = sum(c * v[:nmu - 4, k + 1] for k, c in enumerate(ex)) if even else 0
            v[:nmu - 4, -1] = sum(c * v[:nmu - 4, -2 - k] for k, c in enumerate(ex)) if even else 0
        out.append(u)
    return out[0].reshape(-1) if case["kind"] == "host" else out
