"""The solver's measured workloads: what a hydro or SCF program has it do.

Every case is one call of the public Python mirror (the C ABI underneath) on
one grid, or on several for a plan.  `kind` is the call:

  step       potential_solver_device, tstep > 1: the five warm ADI steps of
             every hydro time step, density and potential resident on the GPU
  cold       potential_solver_device, tstep = 0: the twenty-step solve of a
             run's first density or of a client's first request
  host       potential_solver on pinned host arrays: the Fortran drop-in's
             call, copies both ways included
  batch      Batch.solve_device, warm: n models of a sweep on one grid
  plan       Plan.launch, warm: models on several grids as one graph
  converged  solve_converged_device, FP64, warm
  mixed      solve_converged_device(mixed=True), warm
  batch_converged / batch_mixed
             Batch.solve_converged_device of n models, warm

Warm calls start from the potential of the density one azimuthal zone away,
as a rotating binary's time step does: passes alternate between two such
densities, the first pass from the cold solution of the other one.
"""
import math

import numpy as np
import torch

import bipoly_hydro_b200 as bph

WARM, COLD = 5, 20  # ADI steps of potential_solver (tstep > 1, else)
CYCLE, TOL, MAX_CYCLES = 10, 1e-11, 60  # converged forms: steps per cycle, stopping update


def _grid(numr, numz, numphi, isym=2, mmax=30):
    return {"numr": numr, "numz": numz, "numphi": numphi, "isym": isym, "mmax": mmax}


# Grids of a plan: how many models on each.
_PLANS = {
    "uneven": (((66, 66, 64, 2, 30), 6), ((130, 98, 128, 2, 30), 6), ((130, 98, 256, 2, 30), 4),
               ((258, 194, 256, 2, 30), 1)),
    "small": (((34, 26, 64, 2, 30), 5), ((66, 66, 64, 2, 30), 3), ((51, 37, 32, 1, 12), 4)),
    "odd": (((67, 45, 64, 3, 12), 3), ((101, 75, 128, 2, 30), 3), ((130, 98, 128, 2, 30), 2)),
}


def listed():
    return [
        # a coarse run's time step: the smallest calls, where launches and latency count
        {"name": "step_66x66x64", "kind": "step", "n": 1, **_grid(66, 66, 64)},
        # a production run's time step
        {"name": "step_130x98x256", "kind": "step", "n": 1, **_grid(130, 98, 256)},
        # a full-z grid (no equatorial symmetry) with odd extents
        {"name": "step_101x75x128_full", "kind": "step", "n": 1, **_grid(101, 75, 128, isym=1, mmax=20)},
        # the largest grid's time step
        {"name": "step_258x194x512", "kind": "step", "n": 1, **_grid(258, 194, 512)},
        # the first solve of a run
        {"name": "cold_130x98x256", "kind": "cold", "n": 1, **_grid(130, 98, 256)},
        # the Fortran host's call
        {"name": "host_130x98x256", "kind": "host", "n": 1, **_grid(130, 98, 256)},
        # a sweep over mass ratio and separation on one grid
        {"name": "batch16_130x98x256", "kind": "batch", "n": 16, **_grid(130, 98, 256)},
        # the same over several grids at once
        {"name": "plan_uneven", "kind": "plan", "plan": "uneven"},
        # the converged potential of an SCF iteration, plain and mixed
        {"name": "converged_130x98x256", "kind": "converged", "n": 1, **_grid(130, 98, 256)},
        {"name": "mixed_130x98x256", "kind": "mixed", "n": 1, **_grid(130, 98, 256)},
        # converged sweeps
        {"name": "batch16_mixed_130x98x256", "kind": "batch_mixed", "n": 16, **_grid(130, 98, 256)},
        # the converged potential on the largest grid
        {"name": "mixed_258x194x512", "kind": "mixed", "n": 1, **_grid(258, 194, 512)},
    ]


_MOST_ZONES = 258 * 194 * 512


def draw(rng):
    kind = rng.choice(["step", "step", "step", "cold", "host", "batch", "plan", "converged", "mixed", "batch_converged",
                       "batch_mixed"])
    if kind == "plan" and rng.random() < 0.5:
        return {"kind": "plan", "plan": rng.choice(["small", "odd"])}
    if kind == "plan":
        kind = "step"
    while True:
        numr = int(round(math.exp(rng.uniform(math.log(18), math.log(258)))))
        numz = max(12, min(194, int(round(numr * rng.uniform(0.5, 1.1)))))
        numphi = rng.choice([16, 32, 64, 64, 128, 128, 256, 256, 512])
        isym = rng.choice([1, 2, 2, 2, 3])
        most = (numphi // 2 - 1) // (2 if isym == 3 else 1)
        mmax = max(2, min(30, most, rng.choice([8, 12, 20, 30, 30])))
        n = rng.choice([2, 3, 4, 7, 8, 16]) if kind.startswith("batch") else 1
        if n * numr * numz * numphi <= (_MOST_ZONES if kind in ("step", "cold", "host") else _MOST_ZONES // 2):
            break
    return {"kind": kind, "n": n, **_grid(numr, numz, numphi, isym, mmax)}


def _parts(case):
    """[(grid tuple, number of models)] of a case."""
    if case["kind"] == "plan":
        return _PLANS[case["plan"]]
    return (((case["numr"], case["numz"], case["numphi"], case["isym"], case["mmax"]), case["n"]),)


def _dr(numr):
    return 1.0 / (numr - 4)


def _device():
    return torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")


def _densities(case, seed):
    """Per part, a list of binaries [numphi, numz, numr] (the Fortran (numr, numz, numphi) order):
    two n = 1 polytropes with denser cores on the x axis, seeded mass ratio, separation, core
    jump, phase and noise, on a floor."""
    rng = np.random.Generator(np.random.PCG64(seed))
    gen = torch.Generator(device=_device())
    gen.manual_seed(int(seed))
    out = []
    for (numr, numz, numphi, isym, _), n in _parts(case):
        dr = _dr(numr)
        f = dict(dtype=torch.float64, device=_device())
        r = (torch.arange(numr, **f) - 0.5) * dr
        k = torch.arange(1, numz + 1, **f)
        z = (k - 1.5) * dr if isym != 1 else -(numz // 2) * dr + (k - 0.5) * dr
        phi = torch.arange(numphi, **f) * (2.0 * math.pi / numphi)
        height = min(1.0, float(z.abs().max()))
        models = []
        for _ in range(n):
            q, a, jump = rng.uniform(0.2, 1.0), rng.uniform(0.6, 1.0), rng.uniform(1.5, 3.0)
            phase = rng.uniform(0.0, 2.0 * math.pi)
            rho = torch.zeros(numphi, numz, numr, **f)
            for centre, size, weight in ((a * q / (1 + q), 0.3, 1.0), (-a / (1 + q), 0.22, q)):
                size = min(size, 0.8 * height)
                s2 = (r ** 2 + centre ** 2)[None, None, :] + (z ** 2)[None, :, None]
                s2 = s2 - 2.0 * centre * torch.cos(phi - phase)[:, None, None] * r[None, None, :]
                s = torch.sqrt(torch.clamp(s2, min=0.0))
                star = torch.where(s < size, torch.sinc(s / size), torch.zeros((), **f))
                rho += weight * torch.where(s < 0.4 * size, jump * star, star)
            rho = torch.clamp(rho, min=1e-10)
            noise = torch.rand(rho.shape, generator=gen, **f)
            models.append((rho * (1.0 + 1e-3 * (2.0 * noise - 1.0))).contiguous())
        out.append(models)
    return out


def _solver(grid):
    numr, numz, numphi, isym, mmax = grid
    solver = bph.PotentialSolver(numr, numz, numphi, _dr(numr), isym, mmax)
    solver.set_stream(torch.cuda.current_stream())
    return solver


def prepare(case, seed):
    kind = case["kind"]
    earlier = _densities(case, seed)
    now = [[torch.roll(rho, 1, dims=0) for rho in models] for models in earlier]
    pots = [[torch.empty_like(rho) for rho in models] for models in now]
    solvers = [_solver(grid) for grid, _ in _parts(case)]
    state = {"kind": kind, "solvers": solvers, "rho": (now, earlier), "pot": pots, "turn": 0}
    if kind in ("batch", "batch_converged", "batch_mixed", "plan"):
        state["batches"] = [bph.Batch(s, len(models)) for s, models in zip(solvers, now)]
        for batch, was, pot in zip(state["batches"], earlier, pots):
            batch.solve_device(was, pot, 0)
    elif kind != "cold":
        solvers[0].potential_solver_device(earlier[0][0], pots[0][0], 0)
    if kind == "plan":  # a plan's arrays are fixed: one plan per density
        state["plans"] = [bph.Plan(list(zip(state["batches"], rho, pots))) for rho in (now, earlier)]
    if kind == "host":
        state["host_rho"] = [_pinned(rho[0][0]) for rho in (now, earlier)]
        state["host_pot"] = _pinned(pots[0][0])
    torch.cuda.synchronize()
    return state


def _pinned(x):
    """A pinned host copy as a Fortran-ordered (numr, numz, numphi) array."""
    return torch.empty(x.shape, dtype=x.dtype, pin_memory=True).copy_(x).numpy().transpose(2, 1, 0)


def run(state):
    kind, solver, pot, turn = state["kind"], state["solvers"][0], state["pot"], state["turn"]
    state["turn"] = 1 - turn
    rho = state["rho"][turn]
    if kind == "host":
        return solver.potential_solver(state["host_rho"][turn], 2, out=state["host_pot"])
    if kind == "plan":
        state["plans"][turn].launch(2, torch.cuda.current_stream())
        return pot
    if kind == "batch":
        state["batches"][0].solve_device(rho[0], pot[0], 2)
        return pot
    if kind in ("batch_converged", "batch_mixed"):
        info = state["batches"][0].solve_converged_device(rho[0], pot[0], CYCLE, False, TOL, MAX_CYCLES,
                                                          mixed=kind == "batch_mixed")
    elif kind in ("converged", "mixed"):
        info = solver.solve_converged_device(rho[0][0], pot[0][0], CYCLE, False, TOL, MAX_CYCLES, mixed=kind == "mixed")
    else:
        solver.potential_solver_device(rho[0][0], pot[0][0], 0 if kind == "cold" else 2)
        return pot
    # The mixed form's cycle count is that of whichever refinement kernel the
    # set-up's timing chose, so only the plain form's is an output.
    return pot if kind.endswith("mixed") else {"pot": pot, "cycles": info.cycles}


def work(case):
    """Density read, potential written, warm potential read, and the distinct Green coefficients
    read once per grid; azimuthal transforms, boundary sums and tridiagonal steps."""
    total = {"bytes": 0, "flops": 0}
    for (numr, numz, numphi, isym, mmax), n in _parts(case):
        zones, nr, nz = numr * numz * numphi, numr - 2, numz - 2
        rows = nr + nz + (nr if isym == 1 else 0)
        # top (bottom) rows are symmetric in the two radii; side rows depend on height differences and sums
        tables = mmax * (nr * (nr + 1) // 2 * nz * (2 if isym == 1 else 1) + 2 * (2 * nz - 1) * nr)
        steps = COLD if case["kind"] == "cold" else CYCLE if "converged" in case["kind"] or "mixed" in case["kind"] else WARM
        total["bytes"] += 8 * (n * zones * (2 if case["kind"] == "cold" else 3) + tables)
        total["flops"] += n * (zones * (5 * math.log2(numphi) + 26 * steps) + 4 * mmax * rows * nr * nz)
    return total


# --------------------------------------------------------------------------
# The discrete solution in plain torch, 64 bits.


def _log_gamma(x):
    """Lanczos' approximation (gamma = 5, six terms): the tables are defined with it."""
    c = (76.18009172947146, -86.50532032941677, 24.01409824083091, -1.231739572450155, 0.1208650973866179e-2,
         -0.5395239384953e-5)
    series = 1.000000000190015 + sum(ci / (x + 1.0 + i) for i, ci in enumerate(c))
    return (x + 0.5) * math.log(x + 5.5) - (x + 5.5) + math.log(2.5066282746310005 * series / x)


def _elliptic(m1):
    """Complete K and E for complementary parameter m1 = 1 - k^2 (arithmetic-geometric mean)."""
    a, g = torch.ones_like(m1), torch.sqrt(m1)
    total, weight = (1.0 - m1) / 2.0, 0.5
    for _ in range(40):
        c = (a - g) / 2.0
        a, g = (a + g) / 2.0, torch.sqrt(a * g)
        weight *= 2.0
        total = total + weight * c * c
    k = math.pi / (2.0 * a)
    return k, k * (1.0 - total)


class _Toroidal:
    """Q_{fm m - 1/2}(x), m = 0 .. mmax - 1: recurrence below x = 1.025, a 111-term series above."""

    def __init__(self, isym, mmax, device):
        self.isym, self.mmax = isym, mmax
        self.order = [(2.0 * m if isym == 3 else float(m)) for m in range(mmax)]
        lead, terms = [], []
        for mm in self.order:
            a, b = 0.5 * (mm + 1.5), 0.5 * (mm + 0.5)
            lead.append(_log_gamma(0.5) + _log_gamma(mm + 0.5) - _log_gamma(a) - _log_gamma(b))
            terms.append([_log_gamma(a + i) + _log_gamma(b + i) - _log_gamma(mm + 1.0 + i) - _log_gamma(i + 1.0)
                          for i in range(111)])
        f = dict(dtype=torch.float64, device=device)
        self.lead, self.terms = torch.tensor(lead, **f), torch.exp(torch.tensor(terms, **f)).T.contiguous()
        self.half = torch.tensor(self.order, **f) + 0.5

    def __call__(self, x):
        """[len(x), mmax]"""
        powers = torch.exp(torch.log(x)[:, None] * (-2.0 * torch.arange(111, dtype=x.dtype, device=x.device)))
        q = torch.exp(self.lead - self.half * torch.log(2.0 * x)[:, None]) * (powers @ self.terms)
        near = torch.nonzero(x < 1.025).flatten()
        if near.numel():
            q[near] = self._near(x[near])
        return q

    def _near(self, x):
        mu, la = torch.sqrt(2.0 / (1.0 + x)), torch.sqrt(2.0 * (1.0 + x))
        k, e = _elliptic((1.0 - mu) * (1.0 + mu))
        q = [k * mu]
        if self.isym == 3:
            q.append((4.0 / 3.0 * x * x - 1.0 / 3.0) * mu * k - 4.0 / 3.0 * x * la * e)
            for m in range(2, self.mmax):
                n = 2.0 * m - 2.5
                down = (2.0 * n - 1.0) * (n + 2.0) * (n + 1.0)
                q.append(q[-1] * ((2 * n + 3) * (2 * n + 1) * x * x / ((n + 2) * (n + 1)) - (2 * n + 3) * n * n / down
                                  - (n + 1) / (n + 2)) - q[-2] * (2 * n + 3) * (n - 1) * n / down)
        else:
            q.append(x * mu * k - la * e)
            for m in range(2, self.mmax):
                n = m - 1.5
                q.append((2 * n + 1) / (n + 1) * x * q[-1] - n / (n + 1) * q[-2])
        return torch.stack(q[: self.mmax], dim=1)


class _Plain:
    """One grid's solve: boundary potential, then ADI on the azimuthal transform."""

    def __init__(self, grid, device):
        self.numr, self.numz, self.numphi, self.isym, self.mmax = grid
        self.dr, self.device = _dr(self.numr), device
        f = dict(dtype=torch.float64, device=device)
        N, dr = self.numphi, self.dr
        self.fm = 2 if self.isym == 3 else 1
        self.rhf = (torch.arange(self.numr, **f) - 0.5) * dr
        k = torch.arange(1, self.numz + 1, **f)
        self.zhf = (k - 1.5) * dr if self.isym != 1 else -(self.numz // 2) * dr + (k - 0.5) * dr
        self.dphi = 2.0 * math.pi / N
        J = torch.arange(1, self.numr - 1, **f)  # zero-based J of the interior, J = 2 .. numr-1
        self.alpha = -(J * dr) / self.rhf[1:-1] / dr ** 2  # r_g(J+1)
        self.beta = -((J - 1.0) * dr) / self.rhf[1:-1] / dr ** 2
        mode = torch.arange(N // 2 + 1, **f)
        mode = mode ** 2 if self.isym == 3 else mode
        az = 2.0 * (torch.cos(mode * self.dphi) - 1.0)[:, None] / self.dphi ** 2 / self.rhf[1:-1] ** 2
        self.diag = 2.0 / dr ** 2 - az
        first = 2.0 * self.beta[0] if self.isym == 3 else (1.0 - torch.where(mode % 2 == 0, 1.0, -1.0).to(**f)) * self.beta[0]
        self.diag[:, 0] = -self.alpha[0] - first - az[:, 0]
        self.gamma = 1.0 / dr ** 2

    def boundary(self, rho):
        """Boundary sums S[b, m, cos|sin] as rfft coefficients [b, N/2+1] of the boundary lines."""
        N, nr, nz = self.numphi, self.numr - 2, self.numz - 2
        f = dict(dtype=torch.float64, device=self.device)
        l = (torch.arange(1, N + 1, **f) - 0.5) * self.dphi
        m = torch.arange(self.mmax, **f) * self.fm
        trig = torch.stack([torch.cos(m[:, None] * l), torch.sin(m[:, None] * l)], dim=1)  # [m, 2, N]
        mom = (trig.reshape(-1, N) @ rho[:, 1:-1, 1:-1].reshape(N, -1)).reshape(self.mmax, 2, nz * nr)
        rs = self.rhf[1:-1].repeat(nz)
        zs = self.zhf[1:-1].repeat_interleave(nr)
        rows = [(self.rhf[j + 1], self.zhf[-1], self.isym != 1) for j in range(nr)]
        rows += [(self.rhf[-1], self.zhf[k + 1], self.isym != 1) for k in range(nz)]
        if self.isym == 1:
            rows += [(self.rhf[j + 1], self.zhf[0], False) for j in range(nr)]
        toroidal = _Toroidal(self.isym, self.mmax, self.device)
        sums = []
        for rb, zb, image in rows:
            coef = torch.sqrt(rs / rb) / math.pi
            q = toroidal(0.5 * ((zb - zs) ** 2 + rs ** 2 + rb ** 2) / (rs * rb))
            if image:
                q = q + toroidal(0.5 * ((zb + zs) ** 2 + rs ** 2 + rb ** 2) / (rs * rb))
            sums.append(torch.bmm(mom, (coef[:, None] * q).T.unsqueeze(2)).squeeze(2))
        S = torch.stack(sums)  # [b, m, 2]
        S[:, 0, 1] = 0.0
        S[:, 1:] *= 2.0
        line = S.reshape(len(rows), -1) @ trig.reshape(-1, N)
        factor = -(self.dr * self.dr * self.dphi) * (2.0 if self.isym == 3 else 1.0)
        return torch.fft.rfft(factor * line)

    @staticmethod
    def _thomas(lo, diag, up, rhs):
        """Systems along the first axis of rhs; lo/diag/up broadcast against its rows."""
        n = rhs.shape[0]
        ratio, y = [up[0] / diag[0]], [rhs[0] / diag[0]]
        for j in range(1, n):
            pivot = diag[j] - lo[j] * ratio[-1]
            ratio.append(up[j] / pivot)
            y.append((rhs[j] - lo[j] * y[-1]) / pivot)
        for j in range(n - 2, -1, -1):
            y[j] = y[j] - ratio[j] * y[j + 1]
        return torch.stack(y)

    def _schedule(self, steps):
        last = 4.0 / ((self.numr - 2) * self.dr) ** 2
        ratio = (float(self.numr - 2)) ** (2.0 / (steps - 1.0)) if steps > 1 else 1.0
        return [last * ratio ** (steps - 1 - i) for i in range(steps)]

    def _radial(self, x):
        """A_r x on [nr, nz, modes, 2]."""
        col = lambda v: v[:, None, None, None]  # noqa: E731
        out = self.diag.T[:, None, :, None] * x
        out[:-1] += col(self.alpha[:-1]) * x[1:]
        out[1:] += col(self.beta[1:]) * x[:-1]
        return out

    def _vertical(self, x):
        out = 2.0 * x
        if self.isym != 1:
            out[:, 0] -= x[:, 0]
        out[:, :-1] -= x[:, 1:]
        out[:, 1:] -= x[:, :-1]
        return self.gamma * out

    def sweep(self, phi, source, steps):
        """`steps` ADI steps on [nr, nz, modes, 2]."""
        lo, up = self.beta.clone(), self.alpha.clone()
        lo[0] = 0.0
        up[-1] = 0.0
        nz = self.numz - 2
        off = torch.full((nz,), -self.gamma, dtype=torch.float64, device=self.device)
        mid = torch.full_like(off, 2.0 * self.gamma)
        if self.isym != 1:
            mid[0] = self.gamma
        view = lambda v: v[:, None, None, None]  # noqa: E731
        for dt in self._schedule(steps):
            rhs = source + dt * phi - self._vertical(phi)
            phi = self._thomas(view(lo), (self.diag.T + dt)[:, None, :, None], view(up), rhs)
            rhs = (source + dt * phi - self._radial(phi)).transpose(0, 1).contiguous()
            phi = self._thomas(view(off), view(mid + dt), view(off), rhs).transpose(0, 1).contiguous()
        return phi

    def transform(self, rho):
        """(source with the Dirichlet terms [nr, nz, modes, 2], boundary coefficients)."""
        edge = self.boundary(rho)
        nr, nz = self.numr - 2, self.numz - 2
        inside = rho.clone()
        inside[:, -2:, :] = 0.0
        inside[:, :, -2:] = 0.0
        if self.isym == 1:
            inside[:, :2, :] = 0.0
        hat = torch.view_as_real(torch.fft.rfft(inside[:, 1:-1, 1:-1], dim=0))  # [modes, nz, nr, 2]
        source = (-4.0 * math.pi * hat).permute(2, 1, 0, 3).contiguous()
        real = torch.view_as_real(edge)
        source[:, -1] += self.gamma * real[:nr]
        source[-1] -= self.alpha[-1] * real[nr:nr + nz]
        if self.isym == 1:
            source[:, 0] += self.gamma * real[nr + nz:]
        return source, edge

    def potential(self, phi, edge):
        """[numphi, numz, numr] with the boundary planes, the axis and the equator."""
        N, nr, nz = self.numphi, self.numr - 2, self.numz - 2
        slots = torch.zeros(N // 2 + 1, self.numz, self.numr, dtype=torch.complex128, device=self.device)
        slots[:, 1:-1, 1:-1] = torch.view_as_complex(phi.permute(2, 1, 0, 3).contiguous())
        slots[:, -1, 1:-1] = edge[:nr].T
        slots[:, 1:-1, -1] = edge[nr:nr + nz].T
        if self.isym == 1:
            slots[:, 0, 1:-1] = edge[nr + nz:].T
        pot = torch.fft.irfft(slots, n=N, dim=0)
        pot[:, :, 0] = pot[:, :, 1] if self.isym == 3 else torch.roll(pot[:, :, 1], N // 2, dims=0)
        if self.isym != 1:
            pot[:, 0] = pot[:, 1]
        return pot

    def converge(self, phi, source, tol):
        weight = torch.full((self.numphi // 2 + 1, 1), 2.0, dtype=torch.float64, device=self.device)
        weight[0] = weight[-1] = 1.0
        for _ in range(MAX_CYCLES):
            new = self.sweep(phi, source, CYCLE)
            change = torch.sqrt((weight * (new - phi) ** 2).sum() / (weight * new ** 2).sum())
            phi = new
            if float(change) <= tol:
                break
        return phi


def exact(case, seed):
    kind, device = case["kind"], _device()
    out = []
    for (grid, _), models in zip(_parts(case), _densities(case, seed)):
        plain = _Plain(grid, device)
        out.append([])
        for rho in models:
            now, phi = torch.roll(rho, 1, dims=0), None
            if kind != "cold":
                source, _ = plain.transform(rho)
                phi = plain.sweep(torch.zeros_like(source), source, COLD)
            source, edge = plain.transform(now)
            if kind == "cold":
                phi = plain.sweep(torch.zeros_like(source), source, COLD)
            elif kind.endswith("converged"):
                phi = plain.converge(phi, source, TOL)
            elif kind.endswith("mixed"):  # the discrete solution itself, a little past the tolerance
                phi = plain.converge(phi, source, 1e-2 * TOL)
            else:
                phi = plain.sweep(phi, source, WARM)
            out[-1].append(plain.potential(phi, edge))
    if kind == "host":
        return out[0][0].permute(2, 1, 0)
    return {"pot": out, "cycles": None} if kind.endswith("converged") else out
