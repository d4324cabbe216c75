"""Performance cases of the close-coupling solver, through its public entry points.

Every case is a scattering problem a user of the package solves: He-4 beams on
the square and hexagonal corrugated Morse surfaces and the He-LiF golden case
of the tests and the benchmark, from one small drop-in call to the 512-beam
sweep and the 81 x 81 x 300 grid.  ``kind`` says which entry point is called:

- ``dropin``   run_multiscat_fortran, the reference's f2py call (host arrays in, psi out);
- ``matrix``   get_scattering_matrix, one condition in, |S|^2 out;
- ``scan``     get_scattering_matrix over a list of potentials (a fit to measured data);
- ``state``    get_scattering_state and get_scattering_matrix_from_state;
- ``sweep``    get_scattering_matrices, many beams over one potential;
- ``plan``     ScatteringPlan.solve on a plan the program keeps;
- ``adjoint``  scattering_intensities and its backward pass, dL/dV_G(z).

The solves run to a residual of 2e-13 on plans and 1e-12 through the API (the
tolerances of the gradient tests and of the benchmark's adjoint line lie there),
so that the results are determined to about 1e-10 whichever way the iteration
takes; the node counts resolve the beams' waves on each z domain.  Beams, well depth, corrugation and
loss weights are drawn from the seed; the inputs are built here with numpy,
so ``exact`` shares no code with the package.
"""

import math

import numpy as np
import torch

import multiscat_b200 as mb
from multiscat_b200.adjoint import scattering_intensities
from multiscat_b200.solver import channel_subset_system, full_grid_system

HBAR = 1.054571817e-34
MEV = 1.602176634e-22
ANGSTROM = 1e-10
HE4 = 4.0026 * 1.66053906660e-27
ALPHA = 6.6446573450e-27
RTOL = 2e-13            # residual of the solves on plans (rounding level: 1e-15 to 5e-14)
PRECISION = 1e-9        # the API's precision (it solves to 1e-3 of that)
CUTOFF_MEV = 200.0      # closed-channel depth kept by the truncated sweeps

# lattice constant (A), corrugation h (A), z domain (A), mass
SURFACES = {
    "square": (2.54, 0.15, -1.5, 10.0, HE4),
    "hex": (3.16, 0.20, -1.5, 12.0, HE4),
    "deep": (2.54, 0.25, -2.0, 14.0, HE4),       # the large-grid square surface
    "helif": (2.84, 0.10, 0.0, 8.0, ALPHA),
}


def listed():
    return [
        # the smallest call: the f2py drop-in on an odd little grid, latency and set-up
        dict(name="dropin_hex_7x5x81", kind="dropin", surface="hex", nkx=7, nky=5, nz=81, modes=2,
             beams=1, precision="fp64"),
        # the reference user's everyday call (the tests' and smoke run's 11 x 11 x 100 grid)
        dict(name="matrix_square_11x11x100", kind="matrix", surface="square", nkx=11, nky=11,
             nz=100, modes=4, beams=1, precision="fp64"),
        # the reference's golden He-LiF case: few channels, a long z grid
        dict(name="matrix_helif_10x10x550", kind="matrix", surface="helif", nkx=10, nky=10,
             nz=550, modes=1, beams=1, precision="fp64"),
        # a fit: one beam over ten well depths, a new potential in every call
        dict(name="scan_square_11x11x100", kind="scan", surface="square", nkx=11, nky=11, nz=100,
             modes=4, beams=1, precision="fp64", potentials=10),
        # the full-state pair of calls (the reference's L psi convention), odd sizes
        dict(name="state_hex_9x9x91", kind="state", surface="hex", nkx=9, nky=9, nz=91, modes=3,
             beams=1, precision="fp64"),
        # one large beam on a kept plan, both precisions (the benchmark's single solve)
        dict(name="plan_hex_41x41x200_fp64", kind="plan", surface="hex", nkx=41, nky=41, nz=200,
             modes=4, beams=1, precision="fp64", truncated=False),
        dict(name="plan_hex_41x41x200_mixed", kind="plan", surface="hex", nkx=41, nky=41, nz=200,
             modes=4, beams=1, precision="mixed", truncated=False),
        # forward and backward of the benchmark's adjoint line
        dict(name="adjoint_hex_41x41x200", kind="adjoint", surface="hex", nkx=41, nky=41, nz=200,
             modes=4, beams=1, precision="mixed"),
        # a sweep through the API with the reference's n_channels truncation, odd node count
        dict(name="sweep_square_40x169x131", kind="sweep", surface="square", nkx=17, nky=17, nz=131,
             modes=4, beams=40, precision="mixed", n_channels=169),
        # the headline batch (512 truncated beams on a 32 x 32 torus), mixed, and a plain FP64 one
        dict(name="plan_square_512x150_mixed", kind="plan", surface="square", nkx=32, nky=32,
             nz=150, modes=4, beams=512, precision="mixed", truncated=True),
        dict(name="plan_square_128x150_fp64", kind="plan", surface="square", nkx=32, nky=32,
             nz=150, modes=4, beams=128, precision="fp64", truncated=True),
        # the large grid: 6561 channels, 300 nodes, 288 coupling taps, four azimuths
        dict(name="plan_deep_4x81x81x300_mixed", kind="plan", surface="deep", nkx=81, nky=81,
             nz=300, modes=8, beams=4, precision="mixed", truncated=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "matrix", "matrix", "scan", "state", "sweep", "plan", "plan",
                       "plan", "plan", "adjoint", "adjoint"])
    precision = rng.choice(["fp64", "mixed"])
    surface = rng.choice(["square", "hex"])
    c = dict(kind=kind, surface=surface, beams=1, precision=precision)
    if kind in ("dropin", "matrix", "scan", "state"):
        c.update(nkx=rng.randint(5, 13), nky=rng.randint(5, 13), nz=_log(rng, 80, 260))
        if kind == "matrix" and rng.random() < 0.34:
            c.update(surface="helif", nkx=rng.randint(8, 12), nky=rng.randint(8, 12),
                     nz=_log(rng, 250, 550))
        if kind != "matrix" or c["surface"] == "helif":
            c["precision"] = "fp64"
        if kind == "scan":
            c.update(potentials=rng.randint(9, 11), nz=_log(rng, 80, 150))
    elif kind == "sweep":
        nk = rng.randint(15, 21)
        c.update(nkx=nk, nky=nk, nz=rng.randint(90, 170), beams=_log(rng, 4, 96),
                 n_channels=rng.randint(90, 200))
    elif kind == "adjoint":
        c.update(nkx=rng.randint(11, 41), nky=rng.randint(11, 41), nz=rng.randint(90, 200))
    elif rng.random() < 0.5:
        c.update(nkx=32, nky=32, nz=rng.randint(100, 170), truncated=True,
                 beams=_log(rng, 2, 320 if precision == "mixed" else 128))
    else:
        top = 61 if precision == "mixed" else 45
        c.update(nkx=rng.randint(15, top), nky=rng.randint(15, top), nz=rng.randint(110, 300),
                 truncated=False)
        if rng.random() < 0.5:
            c["surface"] = "deep"
        c["beams"] = rng.randint(1, 3)
    m = {"helif": 1, "deep": 8}.get(c["surface"], 4)
    c["modes"] = min(m, (min(c["nkx"], c["nky"]) - 1) // 2)
    return c


# --------------------------------------------------------------------------- inputs
def _lobatto(z0, z1, n):
    """Gauss-Lobatto nodes and weights: the inner nodes are those of the Jacobi (1, 1) rule."""
    k = np.arange(1, n - 2, dtype=float)
    off = np.sqrt(k * (k + 2) / ((2 * k + 1) * (2 * k + 3)))
    inner = np.linalg.eigvalsh(np.diag(off, 1) + np.diag(off, -1))
    inner = 0.5 * (inner - inner[::-1])
    x = np.concatenate([[-1.0], inner, [1.0]])
    for _ in range(2):                     # Newton's steps on P'_{n-1}, then P_{n-1} itself
        p0, p1 = np.ones_like(x), x.copy()
        for j in range(2, n):
            p0, p1 = p1, ((2 * j - 1) * x * p1 - (j - 1) * p0) / j
        dp = (n - 1) * (p0[1:-1] - x[1:-1] * p1[1:-1])
        d2 = 2 * x[1:-1] * dp / (1 - x[1:-1] ** 2) - n * (n - 1) * p1[1:-1]
        x[1:-1] -= dp / d2
    p0, p1 = np.ones_like(x), x.copy()
    for j in range(2, n):
        p0, p1 = p1, ((2 * j - 1) * x * p1 - (j - 1) * p0) / j
    half = 0.5 * (z1 - z0)
    return 0.5 * (z0 + z1) + half * x, half * 2.0 / (n * (n - 1) * p1**2), x, p1


def _kinetic(x, p, w, half):
    """T_ij = sum_k w_k u_i'(z_k) u_j'(z_k), u_j = l_j / sqrt(w_j)."""
    n = x.size
    diff = x[:, None] - x[None, :]
    np.fill_diagonal(diff, 1.0)
    d = p[:, None] / p[None, :] / diff
    np.fill_diagonal(d, 0.0)
    d[0, 0], d[-1, -1] = -n * (n - 1) / 4.0, n * (n - 1) / 4.0
    u = d / half / np.sqrt(w)[None, :]
    t = u.T @ (w[:, None] * u)
    return 0.5 * (t + t.T)


def _modes(n):
    i = np.arange(n)
    return np.where(i <= (n - 1) // 2, i, i - n)


def _cell(surface):
    a = SURFACES[surface][0]
    if surface == "hex":
        return np.array([a, 0.0]), np.array([0.5 * a, 0.5 * math.sqrt(3.0) * a])
    return np.array([a, 0.0]), np.array([0.0, a])


def _potential(case, z, depth, h):
    """V_G(z) in meV, [nkx, nky, nz] in FFT order."""
    nkx, nky, m = case["nkx"], case["nky"], case["modes"]
    v = np.zeros((nkx, nky, z.size), complex)
    alpha = 1.1
    if case["surface"] == "helif":
        v[0, 0] = depth * (np.exp(2 * alpha * (3.0 - z)) - 2 * np.exp(alpha * (3.0 - z)))
        for i, j in ((1, 0), (nkx - 1, 0), (0, 1), (0, nky - 1)):
            v[i, j] = -depth * h * np.exp(-2 * alpha * (z - 3.0))
        return v
    cells = 128 if m > 4 else 64
    f = np.arange(cells) / cells
    fx, fy = np.meshgrid(2 * np.pi * f, 2 * np.pi * f, indexing="ij")
    if case["surface"] == "hex":
        xi = (h / 3.0) * (np.cos(fx) + np.cos(fy) + np.cos(fx + fy))
    else:
        xi = 0.5 * h * (np.cos(fx) + np.cos(fy))
    coef = np.fft.fft2(np.exp(2 * alpha * xi)) / cells**2
    k = np.arange(-m, m + 1)
    v[np.ix_(k % nkx, k % nky)] = (depth * np.exp(-2 * alpha * z))[None, None, :] * \
        coef[np.ix_(k % cells, k % cells)][:, :, None]
    v[0, 0] -= 2 * depth * np.exp(-alpha * z)
    return v


def _inputs(case, seed):
    """Everything a program has before it calls the solver, in natural units and in SI."""
    rng = np.random.default_rng(seed)
    _, h, z0, z1, mass = SURFACES[case["surface"]]
    factor = 2.0 * mass / HBAR**2 * MEV * ANGSTROM**2            # meV -> 1/A^2
    z, w, x, p = _lobatto(z0, z1, case["nz"])
    t = _kinetic(x, p, w, 0.5 * (z1 - z0))
    h = h * rng.uniform(0.9, 1.0)
    npot = case.get("potentials", 1)
    depths = 7.63 * (rng.uniform(0.95, 1.05) + 0.01 * np.arange(npot))
    nb = case["beams"]
    if case["surface"] == "helif":
        energy, theta, phi = 20.0 * rng.uniform(0.9, 1.1, nb), rng.uniform(25, 35, nb), rng.uniform(1, 10, nb)
    elif case["surface"] == "deep":                              # azimuths of one incidence
        energy, theta = np.full(nb, 100.0 * rng.uniform(0.95, 1.0)), np.full(nb, 45.0)
        phi = 3.0 * np.arange(nb) + rng.uniform(0.5, 2.5)
    elif nb > 1:                        # a survey of energies and angles, as set on the instrument
        energy, theta, phi = _survey(nb)
        energy = energy * rng.uniform(0.98, 1.0, nb)
        theta, phi = np.abs(theta + rng.uniform(-0.5, 0.5, nb)), phi + rng.uniform(-0.5, 0.5, nb)
    else:
        energy, theta, phi = rng.uniform(40, 64, nb), rng.uniform(20, 35, nb), rng.uniform(1, 20, nb)
    theta, phi = np.radians(theta), np.radians(phi)
    pkd = _pkd(case, factor, energy, theta, phi)
    weights = rng.uniform(0.0, 1.0, pkd.shape) * (pkd < 0)
    # channels each beam keeps, lowest pkd first: uneven on the truncated sets
    keep = np.full(nb, case.get("n_channels") or pkd[0].size)
    if case.get("truncated"):
        e0, th0, ph0 = _survey(nb)
        nominal = _pkd(case, factor, e0, np.radians(th0), np.radians(ph0))
        keep = (nominal <= factor * CUTOFF_MEV).reshape(nb, -1).sum(1)
    a1, a2 = _cell(case["surface"])
    return dict(z=z, w=w, t=t, factor=factor, mass=mass, z0=z0, z1=z1, energy=energy, theta=theta,
                phi=phi, a1=a1, a2=a2, pkd=pkd, weights=weights, keep=keep,
                v_mev=[_potential(case, z, d, h) for d in depths])


def _survey(nb):
    """Nominal energies (meV) and angles (degrees) of a sweep."""
    rng = np.random.default_rng(nb)
    return rng.uniform(8, 64, nb), rng.uniform(0, 60, nb), rng.uniform(0, 45, nb)


def _pkd(case, factor, energy, theta, phi):
    """|K + G|^2 - |k|^2 of every beam on the channel grid, [beams, nkx, nky]."""
    a1, a2 = _cell(case["surface"])
    area = a1[0] * a2[1] - a1[1] * a2[0]
    b1 = 2 * np.pi / area * np.array([a2[1], -a2[0]])
    b2 = 2 * np.pi / area * np.array([-a1[1], a1[0]])
    mx, my = _modes(case["nkx"])[:, None], _modes(case["nky"])[None, :]
    k = np.sqrt(factor * energy)
    kx, ky = k * np.sin(theta) * np.cos(phi), k * np.sin(theta) * np.sin(phi)
    gx, gy = mx * b1[0] + my * b2[0], mx * b1[1] + my * b2[1]
    return (kx[:, None, None] + gx) ** 2 + (ky[:, None, None] + gy) ** 2 - (k**2)[:, None, None]


def _waves(e, w, z0, z1):
    """Boundary waves a, b, c of channels with perpendicular energies -e (1/A^2)."""
    e = np.asarray(e, float)
    bw = 1.0 / math.sqrt(w[-1])
    dk = np.sqrt(np.abs(e))
    th = dk * ((z1 - z0) - z0)
    a = np.where(e < 0, np.exp(-2j * th), 0.0)
    b = np.where(e < 0, np.sqrt(dk) * np.exp(-1j * th), 0.0) * bw
    c = np.where(e < 0, 1j * dk, -dk) * bw**2
    return a, b, c


def _conditions(case, q, v_mev):
    md = mb.ScatteringMetadata(vectors=(q["a1"] * ANGSTROM, q["a2"] * ANGSTROM),
                               shape=(case["nkx"], case["nky"], case["nz"]),
                               z_delta=(q["z1"] - q["z0"]) * ANGSTROM, z_start=q["z0"] * ANGSTROM)
    v = v_mev * MEV
    return [mb.ScatteringCondition.from_angles(mass=q["mass"], theta=float(th), phi=float(ph),
                                               energy=float(e) * MEV, potential_values=v, metadata=md)
            for e, th, ph in zip(q["energy"], q["theta"], q["phi"])]


# --------------------------------------------------------------------------- the calls
def prepare(case, seed):
    q = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("matrix", "scan", "state", "sweep"):
        config = mb.OptimizationConfig(precision=PRECISION, max_iterations=2000,
                                       n_channels=case.get("n_channels"),
                                       precision_mode=case["precision"])
        sets = [_conditions(case, q, v) for v in q["v_mev"]]
        return dict(kind=kind, config=config, sets=sets)
    v = q["v_mev"][0] * q["factor"]
    if kind == "dropin":
        wa, wb, wc = _waves(q["pkd"][0], q["w"], q["z0"], q["z1"])
        return dict(kind=kind, args=(1, 9, v, q["pkd"][0], wa, wb, wc, q["t"]))
    waves = lambda e: _waves(e, q["w"], q["z0"], q["z1"])    # noqa: E731
    if kind == "adjoint":
        system = full_grid_system(q["pkd"][0], *waves(q["pkd"][0]))
        return dict(kind=kind, v=torch.as_tensor(v, device="cuda"), t=q["t"], systems=[system],
                    weights=torch.as_tensor(q["weights"].reshape(-1), device="cuda"),
                    precision=case["precision"])
    systems = [full_grid_system(e, *waves(e)) if not case["truncated"] else
               channel_subset_system(e, *(x.ravel() for x in waves(e)), n_channels=int(c))
               for e, c in zip(q["pkd"], q["keep"])]
    return dict(kind=kind, plan=mb.ScatteringPlan(v, q["t"], systems, rtol=RTOL,
                                                  precision=case["precision"]))


def run(state):
    kind = state["kind"]
    if kind == "plan":
        res = state["plan"].solve()
        return {"intensities": res.intensities, "psi": res.psi}
    if kind == "adjoint":
        v = state["v"].detach().requires_grad_(True)
        inten = scattering_intensities(v, state["t"], state["systems"], rtol=RTOL,
                                       precision=state["precision"])
        (state["weights"] * inten).sum().backward()
        return {"intensities": inten.detach(), "gradient": v.grad}
    if kind == "dropin":
        return {"psi": mb.run_multiscat_fortran(*state["args"])}
    config, first = state["config"], state["sets"][0]
    if kind == "sweep":
        return {"intensities": np.stack(mb.get_scattering_matrices(first, config))}
    if kind == "state":
        psi = mb.get_scattering_state(first[0], config)
        return {"state": psi, "intensities": mb.get_scattering_matrix_from_state(psi, first[0])}
    return {"intensities": np.stack([mb.get_scattering_matrix(s[0], config) for s in state["sets"]])}


# --------------------------------------------------------------------------- work
def _channels(case):
    """Channels per beam: the full grid, n_channels, or about those under the cutoff."""
    if case.get("n_channels"):
        return case["n_channels"]
    return 234 if case.get("truncated") else case["nkx"] * case["nky"]


def work(case):
    """One pass: inputs read and results written once; 25 Krylov steps of two n x n transforms
    and the coupling (two 1-D passes where the potential is a product) for each solve."""
    n, c, m = case["nz"], _channels(case), 2 * case["modes"] + 1
    taps = 4 if case["surface"] == "helif" else m * m - 1 if case["surface"] == "hex" else 2 * m + 1
    solves = case["beams"] * case.get("potentials", 1)
    steps = 25 * (2 if case["kind"] == "adjoint" else 1)
    flops = solves * c * steps * (8.0 * n * n + 8.0 * taps * n)
    size = case.get("potentials", 1) * (16.0 * m * m * n + 8.0 * n * n) + solves * c * 64.0
    if case["kind"] in ("plan", "dropin", "state"):
        size += solves * c * n * 16.0
    if case["kind"] == "adjoint":
        size += 2 * 16.0 * case["nkx"] * case["nky"] * n
        flops += 8.0 * c * c * n
    return {"bytes": size, "flops": flops}


# --------------------------------------------------------------------------- 64-bit values
class _Operator:
    """A = D + V_off on the channel torus (x: [b, nkx, nky, n]), its inverse diagonal blocks, and
    the conjugate transposes; the coupling is a circular convolution done by FFT."""

    def __init__(self, v, t, pkd, c, mask):
        self.v00 = v[0, 0].real
        voff = v.clone()
        voff[0, 0] = 0
        self.vk = torch.fft.fft2(voff, dim=(0, 1))[None]
        self.t, self.pkd, self.c, self.mask = t.to(v.dtype), pkd[..., None], c, mask[..., None]
        lam, e = torch.linalg.eigh(t + torch.diag(self.v00))
        self.e, self.en = e.to(v.dtype), e[-1].to(v.dtype)
        self.inv = 1.0 / (self.pkd + lam)
        self.fn = (self.inv * e[-1] ** 2).sum(-1)

    def couple(self, x, adj):
        vk = self.vk.conj() if adj else self.vk
        return torch.fft.ifft2(torch.fft.fft2(x, dim=(1, 2)) * vk, dim=(1, 2)) * self.mask

    def apply(self, x, adj):
        c = self.c.conj() if adj else self.c
        y = x @ self.t + (self.pkd + self.v00) * x + self.couple(x, adj)
        y[..., -1] -= c * x[..., -1]
        return y * self.mask

    def inverse_blocks(self, x, adj):
        c = self.c.conj() if adj else self.c
        xt = x @ self.e
        s = (xt * self.inv * self.en).sum(-1)
        beta = c * s / (1.0 - c * self.fn)
        return (((xt + beta[..., None] * self.en) * self.inv) @ self.e.T) * self.mask

    def solve(self, edge, adj=False, m=36, cycles=10):
        """x with A x = (edge at the last node), by restarted GMRES down to the rounding level."""
        nb, n = edge.shape[0], self.t.shape[0]
        rhs = torch.zeros(*edge.shape, n, dtype=self.t.dtype, device=edge.device)
        rhs[..., -1] = edge
        flat = lambda y: y.reshape(nb, -1)    # noqa: E731
        bn = torch.linalg.vector_norm(flat(rhs), dim=1)
        x, best = torch.zeros_like(rhs), None
        for _ in range(cycles):
            r = rhs - self.apply(x, adj)
            rn = torch.linalg.vector_norm(flat(r), dim=1)
            worst = float((rn / bn).max())
            if worst < 1e-15 or (best is not None and worst > 0.5 * best):
                break
            best = worst
            q = torch.empty(nb, m + 1, flat(r).shape[1], dtype=x.dtype, device=x.device)
            q[:, 0] = flat(r) / rn.clamp_min(1e-300)[:, None]
            hess = torch.zeros(nb, m + 1, m, dtype=x.dtype, device=x.device)
            for j in range(m):
                qj = q[:, j].reshape(x.shape)
                w = flat(qj + self.couple(self.inverse_blocks(qj, adj), adj))
                for _ in range(2):
                    hj = (q[:, : j + 1].conj() @ w[..., None])[..., 0]
                    w = w - (hj[:, None, :] @ q[:, : j + 1])[:, 0]
                    hess[:, : j + 1, j] += hj
                wn = torch.linalg.vector_norm(w, dim=1)
                hess[:, j + 1, j] = wn
                q[:, j + 1] = w / wn.clamp_min(1e-300)[:, None]
            g = torch.zeros(nb, m + 1, 1, dtype=x.dtype, device=x.device)
            g[:, 0, 0] = rn
            y = torch.linalg.lstsq(hess.cpu(), g.cpu()).solution.to(x.device)
            x = x + self.inverse_blocks((y.transpose(1, 2) @ q[:, :m])[:, 0].reshape(x.shape), adj)
        return x


def _solved(case, q, v_mev, beams, dev):
    """The torus solution psi [b, nkx, nky, n] of some of the beams, with its waves and mask."""
    pkd = q["pkd"][beams]
    a, b, c = (x.reshape(pkd.shape) for x in _waves(pkd, q["w"], q["z0"], q["z1"]))
    mask = np.ones(pkd.shape, bool)
    for k, keep in enumerate(q["keep"][beams]):
        mask[k].reshape(-1)[np.argsort(pkd[k].reshape(-1), kind="stable")[keep:]] = False
    T = lambda x: torch.as_tensor(x, device=dev)    # noqa: E731
    op = _Operator(T(v_mev * q["factor"]), T(q["t"]), T(pkd), T(c), T(mask))
    edge = torch.zeros(pkd.shape, dtype=torch.complex128, device=dev)
    edge[:, 0, 0] = T(b)[:, 0, 0]
    psi = op.solve(edge)
    s = 2j * T(b) * psi[..., -1]
    s[:, 0, 0] += T(a)[:, 0, 0]
    return psi, s, T(b), mask, op


def exact(case, seed):
    q = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "scan":
        out = [_solved(case, q, v, slice(0, 1), dev)[1].abs()[0] ** 2 for v in q["v_mev"]]
        return {"intensities": torch.stack(out).to(torch.complex128)}
    v = q["v_mev"][0]
    if kind in ("plan", "sweep"):
        per = max(1, int(2e7 / (case["nkx"] * case["nky"] * case["nz"])))
        inten, psis = [], []
        for b0 in range(0, case["beams"], per):
            psi, s, _, mask, _ = _solved(case, q, v, slice(b0, b0 + per), dev)
            for k in range(psi.shape[0]):
                if kind == "sweep":
                    inten.append((s[k].abs() ** 2 * torch.as_tensor(mask[k], device=dev)).to(s.dtype))
                    continue
                # plan rows: by pkd on truncated sets, row-major on the full grid
                rows = np.arange(mask[k].size)
                if case["truncated"]:
                    rows = np.argsort(q["pkd"][b0 + k].reshape(-1), kind="stable")
                    rows = rows[: q["keep"][b0 + k]]
                rows = torch.as_tensor(rows, device=dev)
                inten.append((s[k].abs() ** 2).reshape(-1)[rows])
                psis.append(psi[k].reshape(-1, case["nz"])[rows])
        if kind == "sweep":
            return {"intensities": torch.stack(inten)}
        return {"intensities": torch.cat(inten), "psi": torch.cat(psis)}
    psi, s, b, _, op = _solved(case, q, v, slice(0, 1), dev)
    if kind == "dropin":
        return {"psi": psi[0]}
    inten = s[0].abs() ** 2
    if kind == "matrix":
        return {"intensities": inten[None].to(s.dtype)}
    if kind == "adjoint":
        w = torch.as_tensor(q["weights"], device=dev)
        lam = op.solve(-1j * 2.0 * w * s * b.conj(), adj=True)
        fl, fp = torch.fft.fft2(lam, dim=(1, 2)), torch.fft.fft2(psi, dim=(1, 2))
        # K_D = sum_G conj(lambda_G) psi_{G - D}
        corr = torch.fft.ifft2((fl * fp.conj()), dim=(1, 2)).conj()[0]
        grad = -2.0 * corr.conj()
        grad[0, 0] = -2.0 * corr[0, 0].real
        return {"intensities": inten.reshape(-1), "gradient": grad}
    # state: L psi, L = D + the coupling to channels of lower pkd (the reference's ordering)
    nkx, nky, n = v.shape
    rank = np.empty(nkx * nky, int)
    rank[np.argsort(q["pkd"][0].reshape(-1))] = np.arange(nkx * nky)
    ix, iy = np.divmod(np.arange(nkx * nky), nky)
    out = op.apply(psi, False) - op.couple(psi, False)
    flat, vt = psi.reshape(-1, n), torch.as_tensor(v * q["factor"], device=dev)
    low = torch.zeros_like(flat)
    for j in range(nkx * nky):
        src = np.nonzero(rank < rank[j])[0]
        taps = vt[(ix[j] - ix[src]) % nkx, (iy[j] - iy[src]) % nky]
        low[j] = (taps * flat[src]).sum(0)
    return {"state": (out.reshape(-1, n) + low).reshape(v.shape), "intensities": inten.to(s.dtype)}
