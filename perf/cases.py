"""Work that a user of this framework has it do, with the sizes it is done at.

The users are a Stokesian-dynamics driver that calls the fused step (or, one
by one, the three subroutines it replaces) every time step, an ensemble of
small systems, and the learned preconditioner's solve and training.  Inputs
are sphere packings in a Lees-Edwards cell, made on the GPU from a seed: a
cubic lattice (which stays periodic at skews that are whole numbers of its
cells) disordered by hard-sphere Monte Carlo sweeps in the sheared minimum
image.  One context and one set of lubrication tables serve every pass, as
in a driver's loop.
"""
import importlib
import math

import numpy as np
import torch

EWS, MU, DT, G_MIN = 1e-10, 1.0 / math.pi, 5e-4, 1e-4
_held = {}


def _rsd():
    """The package, and the context and tables that a program keeps."""
    if not _held:
        rsd = importlib.import_module("regularized-stokesian-dynamics_gb300")
        _held.update(rsd=rsd, ctx=rsd.Context(0), tab=rsd.LubTab(rsd.lubdat_dir()))
    return _held["rsd"], _held["ctx"], _held["tab"]


# ------------------------------------------------------------------- packings
_BASES = {"sc": (1, [[0, 0, 0]], 1.0),
          "bcc": (2, [[0, 0, 0], [.5, .5, .5]], math.sqrt(3) / 2),
          "fcc": (4, [[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]], math.sqrt(.5))}


def _lattice(N):
    """The cubic lattice with N sites or a few more and the widest spacing:
    (basis, cells per edge, spacing / L)."""
    best = None
    for per, basis, nn in _BASES.values():
        m = int(math.ceil((N / per) ** (1 / 3) - 1e-9))
        if best is None or nn / m > best[2]:
            best = (basis, m, nn / m)
    return best


def _phi_max(N, ratio):
    """The densest that the lattice start holds (the large spheres apart)."""
    L = (2 * max(1.0, ratio) + 0.01) / _lattice(N)[2]
    return _volume(N, ratio) / L ** 3


def _volume(N, ratio):
    return 4 / 3 * math.pi * ((N - N // 2) + (N // 2) * ratio ** 3)


def _min_image(d, L, skew):
    """Minimum images of separations (..., 3), right for those below L / 2."""
    n3 = torch.round(d[..., 2] / L)
    z = d[..., 2] - n3 * L
    y = d[..., 1] - torch.round(d[..., 1] / L) * L
    x = d[..., 0] - skew * L * n3
    x = x - torch.round(x / L) * L
    return x * x + y * y + z * z


def _packing(case, seed, sweeps=40):
    """Positions (N, 3) on the GPU, radii and box edge at the case's skew;
    every gap in the sheared cell is at least G_MIN."""
    N, ratio = case["N"], case["ratio"]
    L = (_volume(N, ratio) / case["phi"]) ** (1 / 3)
    basis, m, nn = _lattice(N)
    skew = case["shift"] / m
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    f64 = dict(dtype=torch.float64, device="cuda")
    a = torch.arange(m, **f64)
    cells = torch.stack(torch.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 1, 3)
    sites = ((cells + torch.tensor(basis, **f64) + 0.25) * (L / m)).reshape(-1, 3)
    x = sites[torch.randperm(len(sites), generator=g, device="cuda")[:N]]
    radii = torch.ones(N, **f64)
    radii[: N // 2] = ratio
    hard2 = (radii[:, None] + radii[None, :] + G_MIN) ** 2
    hard2.fill_diagonal_(-1.0)
    step = max(0.05, min(0.5, nn * L - 2 * max(1.0, ratio)))
    for _ in range(sweeps):
        p = x + (torch.rand(N, 3, generator=g, **f64) * 2 - 1) * step
        ok = (_min_image(p[:, None] - x[None], L, skew) >= hard2).all(1)
        ok &= (_min_image(p[:, None] - p[None], L, skew) >= hard2).all(1)
        x = torch.where(ok[:, None], p, x)
        if int(ok.sum()) * 3 < N:
            step *= 0.8
    n3 = torch.floor(x[:, 2] / L)
    z = x[:, 2] - n3 * L
    y = torch.remainder(x[:, 1], L)
    return torch.stack([torch.remainder(x[:, 0] - skew * L * n3, L), y, z], 1).contiguous(), radii, L, skew


# --------------------------------------------------------------------- cases
def _case(name, kind, N, phi, shift=0, ratio=1.0, gamma=1.0, forces=False, mode=""):
    c = dict(kind=kind, N=N, phi=phi, shift=shift, ratio=ratio, gamma=gamma, forces=forces, mode=mode)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest replica of an ensemble: launches and latency
        _case("step mixed N32", "mixed", 32, 0.20),
        # an ordinary replica, its size not a multiple of anything
        _case("step mixed N173", "mixed", 173, 0.35, shift=3, gamma=2.5),
        # the plain-against-mixed workload's size, with interparticle forces
        # from the host's contact model
        _case("step mixed N512 forces", "mixed", 512, 0.45, shift=2, forces=True),
        # the long dense run: the largest system stepped
        _case("step mixed N2048", "mixed", 2048, 0.50, shift=4),
        # two sizes of spheres
        _case("step mixed N300 bidisperse", "mixed", 300, 0.30, shift=3, ratio=1.4),
        # the plain method, in 64 bits, at its small and its ordinary size
        _case("step FP64 N64", "fp64", 64, 0.30, shift=1),
        _case("step FP64 N512", "fp64", 512, 0.45, shift=4),
        # the grand mobility alone, left on the GPU
        _case("mobility N1000", "mobility", 1000, 0.50, shift=0),
        # the reference's own sequence of subroutine calls on host arrays:
        # mobility, lubrication, resistance solve
        _case("subroutines N125", "subroutines", 125, 0.25, shift=2, forces=True),
        # the resistance solve by preconditioned conjugate gradients
        _case("PCG learned N500", "pcg", 500, 0.50, shift=1, mode="learned"),
        # one training step of the preconditioner's network
        _case("training N500", "train", 500, 0.50, shift=2),
    ]


_RANGE = {"mixed": (16, 2048), "fp64": (8, 512), "mobility": (8, 1000), "subroutines": (8, 125), "pcg": (64, 500),
          "train": (64, 500)}


def draw(rng):
    kind = rng.choice(["mixed"] * 8 + ["fp64"] * 3 + ["mobility"] * 3 + ["subroutines"] * 2 + ["pcg"] * 2 + ["train"])
    lo, hi = _RANGE[kind]
    N = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    ratio = rng.choice([1.0, 1.0, 1.0, round(rng.uniform(0.6, 1.6), 2)]) if kind in ("mixed", "fp64", "mobility") else 1.0
    if ratio != 1.0 and kind == "mixed":
        N = min(N, 300)  # where systems of unequal spheres are stepped
    phi = round(min(rng.uniform(0.10, 0.50), 0.97 * _phi_max(N, ratio)), 3)
    return _case("", kind, N, phi, shift=rng.randrange(_lattice(N)[1]), ratio=ratio,
                 gamma=round(math.exp(rng.uniform(math.log(0.1), math.log(10.0))), 3), forces=rng.random() < 0.4,
                 mode=rng.choice(["learned", "fsai"]) if kind == "pcg" else "")


# ------------------------------------------------------------------- passes
def prepare(case, seed):
    rsd, ctx, tab = _rsd()
    N, kind = case["N"], case["kind"]
    pos, radii, L, skew = _packing(case, seed)
    rng = np.random.default_rng(int(seed))
    s = dict(case=case, T=skew / case["gamma"], LB=[L, L, L])
    if kind in ("mixed", "fp64", "subroutines"):
        s.update(conf=pos.cpu().numpy(), radii=radii.cpu().numpy(), Fe=None)
        if case["forces"]:
            s["Fe"] = np.concatenate([rng.normal(size=3 * N), np.zeros(3 * N)])
    if kind == "subroutines":
        E = case["gamma"] * np.tile([0.0, 0.0, 0.0, -math.sqrt(0.5), 0.0], N)
        s.update(EIN=E, Fe=s["Fe"] if s["Fe"] is not None else np.zeros(6 * N))
    if kind == "mobility":
        s.update(pos=pos, radii=radii, out=torch.empty((11 * N, 11 * N), dtype=torch.float64, device="cuda"))
    if kind in ("pcg", "train"):
        prec = rsd.PREC_FP64 if kind == "pcg" else rsd.PREC_MIXED
        rpp, lat = rsd.resistance_pp_dev(ctx, tab, pos, radii, s["T"], s["LB"], case["gamma"], MU, EWS, precision=prec)
        s.update(pos=pos, radii=radii, rpp=rpp, lat=lat, net=rsd.LearnedPreconditioner.trained(0))
        if kind == "pcg":
            s["b"] = torch.tensor(rng.normal(size=6 * N), device="cuda")
    return s


def run(s):
    rsd, ctx, tab = _rsd()
    case = s["case"]
    kind = case["kind"]
    if kind in ("mixed", "fp64"):
        r = rsd.STEPPER_Stokesian(ctx, tab, s["conf"], s["radii"], s["T"], DT, s["LB"], case["gamma"], MU, EWS,
                                  Fe=s["Fe"], precision=rsd.PREC_MIXED if kind == "mixed" else rsd.PREC_FP64)
        return {k: r[k] for k in ("conf", "U_pos", "SijN", "yeta_mu")}
    if kind == "mobility":
        lat = rsd.SET_LATTICE_SKEW(s["T"], s["LB"], case["gamma"])
        return rsd.per_grpery_inv_fri_dev(ctx, s["pos"], s["radii"], lat, EWS, MU, out=s["out"])
    if kind == "subroutines":
        lat = rsd.SET_LATTICE_SKEW(s["T"], s["LB"], case["gamma"])
        mob = rsd.PER_GRPERY_INV_FRI(ctx, s["conf"], s["radii"], lat, EWS, MU)
        rfu, rfe, rse, contacts = rsd.lubmxcalc(ctx, tab, s["conf"], s["radii"], lat, MU)
        r = rsd.STEPPER_NOGmres(ctx, *mob, rfu, rfe, rse, s["Fe"], s["EIN"], s["Fe"], s["conf"])
        return [*mob, rfu, rfe, rse, contacts] + [r[k] for k in ("U_par", "SijN_hyd", "SijN_FP", "SijN_B", "RPP")]
    if kind == "pcg":
        mode = rsd.PC_LEARNED if case["mode"] == "learned" else rsd.PC_FSAI
        return rsd.pcg_dev(ctx, s["net"], mode, s["pos"], s["radii"], s["lat"], s["rpp"], s["b"], tol=1e-12, maxit=2000)[0]
    loss = s["net"].train_step(ctx, s["pos"], s["radii"], s["lat"], s["rpp"], 1e-4)
    return dict(loss=loss, grad=s["net"].grad(), params=s["net"].params())


# -------------------------------------------------------------- what it takes
def work(case):
    """Inputs read and results written once; of the arithmetic, the Cholesky
    factors and the inverse that the resistance needs (with n = 11 N unknowns
    of which 6 N are velocities: n^3 / 3, 2 (6 N)^3 / 3, (6 N)^3 / 3), and per
    pair 100 real images and 100 reciprocal vectors of 60 multiply-adds."""
    N, kind = case["N"], case["kind"]
    pairs = N * (N - 1) / 2 * 200 * 120.0
    dense = (11 * N) ** 3 / 3 + (6 * N) ** 3
    vec = 8.0 * (4 + 14 + (6 if case["forces"] else 0)) * N
    if kind in ("mixed", "fp64"):
        return dict(bytes=vec, flops=pairs + dense)
    if kind == "mobility":
        return dict(bytes=8.0 * (4 * N + (11 * N) ** 2), flops=pairs)
    if kind == "subroutines":  # six matrices out, the same six in, RPP out
        return dict(bytes=vec + 8.0 * N * N * (4 * 91 + 36), flops=pairs + dense + 2 / 3 * (6 * N) ** 3)
    if kind == "pcg":  # about 100 products with the matrix, which stays on the chip
        return dict(bytes=8.0 * (6 * N) ** 2, flops=100 * 2.0 * (6 * N) ** 2)
    # about 18 edges a particle; forward and backward over 3 layers and 2 heads
    edges = 18 * N
    return dict(bytes=4.0 * 36 * (N + edges), flops=6.0 * (edges * (3 * 192 * 64 + 192 * 36 + 40 * 64) + N * 4 * 128 * 64))


def exact(case, seed):
    """The solution of the PCG's system by a dense solve in 64 bits.  The
    mobilities, steps and the network's training have no plain 64-bit form
    short of writing the whole method again."""
    if case["kind"] != "pcg":
        return None
    s = prepare(case, seed)
    x = torch.linalg.solve(s["rpp"], s["b"])
    return x + torch.linalg.solve(s["rpp"], s["b"] - s["rpp"] @ x)
