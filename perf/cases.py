"""The work that users of this framework have it do, as cases that can be timed.

Every case goes through the package's public entry points.  The synthetic workloads are the
package's own (`synth`: kind 0 the lattice with a central block, 1 the jittered lattice with
a perturbed sphere, 2 the permuted lattice with a screw, 3 the calibration cylinder, 4 an
ensemble member); `n` is the number of nodes along an edge.

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) what a program has in hand before the call
  run(state)          one pass and its outputs
  work(case)          bytes and flops that one pass cannot do without
  exact(case, seed)   run()'s outputs in 64 bits, by plain torch
"""
import ctypes as C
import importlib.util
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package (its directory name is not a Python identifier)."""
    if "nnpp_gb300" not in sys.modules:
        d = os.path.join(ROOT, "nnpp-mg-implant-corrosion-3d_gb300")
        spec = importlib.util.spec_from_file_location("nnpp_gb300", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["nnpp_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["nnpp_gb300"]


# ------------------------------------------------------------------------------ cases ----
def listed():
    return [
        # the plain FP64 method on the 8,000-node block: a short run from the initial state,
        # bound by launches and latency
        dict(name="explicit_fp64_8k", path="explicit", kind=0, n=20, precision="fp64", steps=100),
        # the same size in mixed precision: a quick look at a small sphere
        dict(name="explicit_mixed_8k", path="explicit", kind=1, n=20, precision="mixed", steps=100),
        # the headline workload: a run on the 512,000-node sphere
        dict(name="explicit_mixed_512k", path="explicit", kind=1, n=80, precision="mixed", steps=20),
        # the same lattice with the FP64 path, as a user checks a mixed run
        dict(name="explicit_fp64_512k", path="explicit", kind=1, n=80, precision="fp64", steps=5),
        # the largest: the permuted 2,000,376-node screw
        dict(name="explicit_mixed_2m", path="explicit", kind=2, n=126, precision="mixed", steps=5),
        # a host-side time loop that keeps the state in its own arrays: one call a step
        dict(name="step_host_64k", path="step_host", kind=1, n=40, precision="mixed", steps=10),
        # uneven instances with their own inclusions and parameters, stepped together
        dict(name="ensemble_mixed_8", path="ensemble", members=8, n_low=27, n_high=58, precision="mixed", steps=20),
        # one gradient of the calibration loop: forward with checkpoints, then backward
        dict(name="gradient_mixed_262k", path="gradient", n=64, precision="mixed", steps=40, every=10, sample=20),
        # the complete ten-species residual, arrays on the device
        dict(name="residual_ten_512k", path="residual_ten", kind=1, n=80),
        # a step of the complete model's implicit integration
        dict(name="implicit_ten_64k", path="implicit_ten", kind=1, n=40, steps=1),
        # a step of the four-species model's implicit integration
        dict(name="implicit_four_64k", path="implicit_four", kind=1, n=40, steps=1),
        # start-up: the neighbour lists of 512,000 nodes in the reference's order, host arrays
        dict(name="neighbours_512k", path="neighbours", kind=1, n=80, order="reference"),
    ]


def _log_int(rng, low, high):
    return int(round(low * (high / low) ** rng.random()))


def draw(rng):
    path = rng.choice(["explicit", "explicit", "explicit", "explicit", "step_host", "ensemble", "gradient",
                       "residual_ten", "implicit_ten", "implicit_four", "neighbours"])
    if path == "explicit":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        n = _log_int(rng, 12, 110 if precision == "mixed" else 80)
        budget = 6.0e6 if precision == "mixed" else 2.0e6  # node-steps
        steps = max(2, min(rng.randint(20, 80), int(budget / n ** 3)))
        return dict(path=path, kind=rng.choice([0, 1, 2, 4]), n=n, precision=precision, steps=steps)
    if path == "step_host":
        return dict(path=path, kind=rng.choice([0, 1, 4]), n=_log_int(rng, 14, 64),
                    precision=rng.choice(["mixed", "fp64"]), steps=rng.randint(3, 10))
    if path == "ensemble":
        low = rng.randint(18, 30)
        return dict(path=path, members=rng.randint(3, 10), n_low=low, n_high=low + rng.randint(4, 26),
                    precision=rng.choice(["mixed", "mixed", "fp64"]), steps=rng.randint(4, 12))
    if path == "gradient":
        return dict(path=path, n=_log_int(rng, 24, 64), precision="mixed", steps=rng.choice([20, 30, 40]),
                    every=rng.choice([7, 10, 25]), sample=rng.choice([5, 10, 20]))
    if path == "residual_ten":
        return dict(path=path, kind=rng.choice([0, 1, 4]), n=_log_int(rng, 12, 80))
    if path in ("implicit_ten", "implicit_four"):
        return dict(path=path, kind=rng.choice([1, 4]), n=_log_int(rng, 12, 40), steps=1)
    return dict(path=path, kind=rng.choice([1, 2, 4]), n=_log_int(rng, 12, 90),
                order=rng.choice(["reference", "canonical"]))


# ------------------------------------------------------------------------------ inputs ---
# The control vectors of the reference's data files (the .data2, .datac1..10 and .datac11
# values) that the ten-species cases use.
DATA2 = [0.0, 24192000.0, 10800.0, 2e-05, 2e-05, 2e-05, 6.000000000000001e-05, 66082.4, 2312.884, 142.0, 2.31, 34.88,
         1.39, 109.9, 15.97, 4.73, -4.49, -2.98, -1.8, 58.77, 13.61, 10.24, 12.32, 0.844, -0.477, 0.0451, 0.5, 0.5, 0.0,
         9.024499999999999e-21, 0.0, 7.0332e-09, 0.0, 7.0023e-10, 0.0, 0.010798, 0.0, 8.0037e-24, 0.0, 9.001e-16, 0.0,
         140.0, 0.0, 140.0, 0.0, 140.0, -0.5, 298.15, 8.3145, 96485.0, 4.79859938096492]
_K1, _K2 = 265258238.48649216, 88419412.82883072
DATAC = [[z, ds, dl, 0.0, 0.0, _K1, _K2] for z, ds, dl in (
    (2.0, 1e-15, 7.1e-10), (1.0, 9.31e-12, 9.31e-09), (-1.0, 5.27e-12, 5.27e-09), (-1.0, 1.19e-12, 1.19e-09),
    (-2.0, 9.230000000000002e-13, 9.230000000000001e-10), (-2.0, 6.9e-13, 6.9e-10),
    (-3.0, 6.120000000000001e-13, 6.120000000000001e-10), (2.0, 7.930000000000001e-13, 7.930000000000001e-10),
    (1.0, 1.3300000000000002e-12, 1.3300000000000002e-09), (-1.0, 2.03e-12, 2.03e-09))]
DATAC11 = [6100000.0, 6100000.0, 0.0, 265258238.48649216]
VOLN1REL = 0.3  # the relative volume at which the ten-species residual is evaluated


def _chem_lattice(case, seed):
    """A synthetic lattice and its phases at the node spacing of the reference's data files."""
    inp = _package().synth(case["kind"], case["n"], seed)
    dx = DATA2[3]
    nodes = np.ascontiguousarray(inp["nodes"] * (dx / inp["params"].dx))
    return inp, nodes, np.ascontiguousarray(inp["phase0"], dtype=np.int32), DATA2[6] * (1.0 + 1e-5), 10.0 * dx


def _chem_fields(N, seed):
    """Concentrations over the three decades that the model's species span, and potentials, at
    two time levels."""
    rng = np.random.default_rng(seed)
    Un = np.empty((11, N))
    Un[:10] = 10.0 ** rng.uniform(-5.0, -2.0, (10, N))
    Un[10] = 0.01 * rng.standard_normal(N)
    return Un * (1.0 + 1e-3 * rng.standard_normal((11, N))), Un


def _smooth_state(phase):
    """Uniform species in the liquid, the solid's Mg at 1."""
    U = np.zeros((11, phase.size))
    U[:10] = (1e-4 + 1e-5 * np.arange(10))[:, None]
    U[0][phase == 1] = 1.0
    return U


def _chem_boundary(inp, U):
    """Dirichlet values of the eleven fields on the workload's outer shell."""
    bv = -np.ones((11, U.shape[1]))
    bv[:4] = inp["bcvalues"][:4]
    bv[10] = inp["bcvalues"][4]
    on = (inp["bctypes"] == 0) & (inp["bcvalues"][0] != -1)
    bv[4:10, on] = U[4:10, on] * DATA2[7]
    return np.asarray(inp["bctypes"], dtype=np.int32), bv


def _member_sizes(case):
    """Edge lengths of an ensemble's members, spaced evenly in their logarithm."""
    lo, hi = case["n_low"], case["n_high"]
    return [int(round(lo * (hi / lo) ** (i / (case["members"] - 1)))) for i in range(case["members"])]


def _member_synth(case, seed):
    return [_package().synth(4, n, 1000 * (seed % 1000000) + i) for i, n in enumerate(_member_sizes(case))]


def _precision(case):
    nn = _package()
    return nn.FP64 if case["precision"] == "fp64" else nn.MIXED


def _simulation(inp):
    sim = _package().Simulation.from_synth(inp)
    sim.build_neighbours()
    return sim


def prepare(case, seed):
    nn = _package()
    path = case["path"]
    s = dict(case=case, nn=nn)
    if path in ("explicit", "step_host", "implicit_four"):
        inp = nn.synth(case["kind"], case["n"], seed)
        s["sim"] = _simulation(inp)
        if path == "step_host":
            s["c"], s["phase"] = inp["icvalues"][:4].copy(), inp["phase0"]
        if path == "implicit_four":  # the implicit step's use: time steps above the explicit limit
            p = inp["params"].copy()
            p.dt *= 10.0
            s["sim"].set_params(p)
    elif path == "ensemble":
        s["sims"] = [_simulation(inp) for inp in _member_synth(case, seed)]
        s["ensemble"] = nn.Ensemble(s["sims"])
    elif path == "gradient":
        inp = nn.synth(3, case["n"], seed)
        s["sim"], s["params"] = _simulation(inp), inp["params"]
        s["weights"] = torch.tensor(np.random.default_rng(seed).uniform(0.5, 1.5, case["steps"] // case["sample"]))
    elif path == "residual_ten":
        _, nodes, phase, r, cell = _chem_lattice(case, seed)
        clouds, lengths, ml = nn.build_clouds_hash(160, r, cell, cell, cell, nodes)
        U1, U0 = _chem_fields(phase.size, seed)
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        s.update(N=phase.size, nodes=dev(nodes), clouds=dev(clouds[:, :ml].T), lengths=dev(lengths), U1=dev(U1),
                 U0=dev(U0), phase=dev(phase), F=torch.empty((11, phase.size), dtype=torch.float64, device="cuda"))
        s["data"] = [np.ascontiguousarray(a, dtype=np.float64) for a in (DATA2, DATAC, DATAC11)]
    elif path == "implicit_ten":
        inp, nodes, phase, r, cell = _chem_lattice(case, seed)
        U = _smooth_state(phase)
        bt, bv = _chem_boundary(inp, U)
        clouds, lengths, ml = nn.build_clouds_hash(160, r, cell, cell, cell, nodes)
        s.update(U=U, phase=phase, chem=nn.ChemImplicit(nodes, clouds[:, :ml], lengths, bt, bv, DATA2, DATAC, DATAC11))
    elif path == "neighbours":
        inp = nn.synth(case["kind"], case["n"], seed)
        p = inp["params"]
        s.update(nodes=inp["nodes"], r=p.delta * (1.0 + 1e-5), cell=10.0 * p.dx,
                 order=nn.ORDER_REFERENCE if case["order"] == "reference" else nn.ORDER_CANONICAL)
    return s


# ------------------------------------------------------------------------------ runs -----
def run(s):
    case, nn = s["case"], s["nn"]
    path = case["path"]
    if path == "explicit":
        # a member of a parameter study: from the initial state through a number of steps
        sim = s["sim"]
        sim.reset()
        sim.forward(case["steps"], _precision(case))
        return _state(sim)
    if path == "step_host":
        sim = s["sim"]
        sim.reset()
        c, phase = s["c"], s["phase"]
        for _ in range(case["steps"]):
            c, phi, phase = sim.step_host(c, phase, _precision(case))
        return dict(c=c, phi=phi, phase=phase)
    if path == "ensemble":
        for sim in s["sims"]:
            sim.reset()
        s["ensemble"].forward(case["steps"], _precision(case))
        return [_state(sim) for sim in s["sims"]]
    if path == "gradient":
        sim = s["sim"]
        sim.set_params(s["params"])
        sim.reset()
        curve = sim.forward_ckpt(case["steps"], _precision(case), case["every"], case["sample"])
        gD, gk = sim.backward(s["weights"].numpy())
        return dict(curve=curve, gD=gD, gk=gk, state=_state(sim))
    if path == "residual_ten":
        d2, dc, d11 = s["data"]
        st = nn.lib().nnpp_residuals_full_device(
            s["N"], s["nodes"].data_ptr(), s["clouds"].data_ptr(), s["lengths"].data_ptr(), s["U1"].data_ptr(),
            s["U0"].data_ptr(), s["phase"].data_ptr(), VOLN1REL, nn._dp(d2), nn._dp(dc), nn._dp(d11),
            s["F"].data_ptr(), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st != 0:
            raise RuntimeError(nn.lib().nnpp_last_error())
        return s["F"]
    if path == "implicit_ten":
        ch = s["chem"]
        ch.set_state(s["U"], s["phase"], voln1rel=1.0)
        ch.step(case["steps"])
        U, phase, _ = ch.state()
        return dict(U=U, phase=phase)
    if path == "implicit_four":
        sim = s["sim"]
        sim.reset()
        sim.forward_implicit(case["steps"])
        return _state(sim)
    clouds, lengths, longest = nn.build_clouds_hash(160, s["r"], s["cell"], s["cell"], s["cell"], s["nodes"], s["order"])
    return dict(clouds=clouds, lengths=lengths, longest=longest)


def _state(sim):
    c, phi, phase = sim.state()
    return dict(c=c, phi=phi, phase=phase)


# ------------------------------------------------------------------------------ work -----
def _bonds(n):
    """Bonds of an n^3 lattice with the horizon 3.015 spacings (jitter leaves the mean)."""
    t = 0
    for i in range(-3, 4):
        for j in range(-3, 4):
            for k in range(-3, 4):
                if 0 < i * i + j * j + k * k <= 9:
                    t += max(0, n - abs(i)) * max(0, n - abs(j)) * max(0, n - abs(k))
    return t


def work(case):
    """A step reads the neighbour list (4 bytes a bond) and the node's fields and writes the
    new ones; its sums take 4 flops a bond and species for the two differences' products and
    sums, plus 2 for the potential's operator, applied once."""
    path = case["path"]
    if path == "ensemble":
        sizes = _member_sizes(case)
        N, nnz = float(sum(n ** 3 for n in sizes)), float(sum(_bonds(n) for n in sizes))
    else:
        N, nnz = float(case["n"] ** 3), float(_bonds(case["n"]))
    if path == "neighbours":
        return dict(bytes=24.0 * N + 4.0 * 160 * N + 4.0 * N, flops=8.0 * nnz)
    if path == "residual_ten":
        return dict(bytes=4.0 * nnz + N * (24 + 4 + 4 + 3 * 88), flops=100.0 * nnz)
    if path == "implicit_ten":
        # at least two Newton iterations (the test compares two updates' norms): residual,
        # and one product of the eleven tangents each
        return dict(bytes=2.0 * case["steps"] * (2 * 4.0 * nnz + N * (24 + 4 + 6 * 88)), flops=2.0 * case["steps"] * 122.0 * nnz)
    if path == "implicit_four":
        return dict(bytes=2.0 * case["steps"] * (2 * 4.0 * nnz + N * (4 + 6 * 40)), flops=2.0 * case["steps"] * 28.0 * nnz)
    b = 8 if case["precision"] == "fp64" else 4
    step = dict(bytes=4.0 * nnz + N * (2 * 5 * b + 2), flops=18.0 * nnz)
    passes = case["steps"] * (2 if path == "gradient" else 1)  # backward: the transposed sums
    extra = case["steps"] * N * 2 * 40.0 if path == "step_host" else 0.0
    return dict(bytes=passes * step["bytes"] + extra, flops=passes * step["flops"])


# ------------------------------------------------------------------------------ exact ----
# The model in 64 bits by plain torch: neighbours within the horizon as a padded table
# (N, K), the bond sums as sums over its second dimension.
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _table(nodes, r):
    """Neighbours within r (the node itself left out): columns (N, K) int64, the mask of
    the entries in use and the distances."""
    x = torch.as_tensor(nodes, dtype=torch.float64, device=_device()).T.contiguous()
    N = x.shape[0]
    cell = torch.floor((x - x.min(0).values) / (r * (1 + 1e-9))).long()
    dim = cell.max(0).values + 3
    cell = cell + 1
    key = (cell[:, 2] * dim[1] + cell[:, 1]) * dim[0] + cell[:, 0]
    total = int(dim[0] * dim[1] * dim[2])
    order = torch.argsort(key)
    count = torch.bincount(key, minlength=total)
    start = torch.cumsum(count, 0) - count
    m = int(count.max())
    member = torch.full((total, m), -1, dtype=torch.int64, device=x.device)
    slot = torch.arange(N, device=x.device) - start[key[order]]
    member[key[order], slot] = order
    near = torch.tensor([(k * int(dim[1]) + j) * int(dim[0]) + i for k in (-1, 0, 1) for j in (-1, 0, 1)
                         for i in (-1, 0, 1)], device=x.device)
    parts, widest = [], 0
    step = max(1, int(3e7) // (27 * m))
    for a in range(0, N, step):
        cand = member[key[a:a + step, None] + near].reshape(-1, 27 * m)
        d = (x[cand.clamp(min=0)] - x[a:a + step, None, :]).square().sum(2).sqrt()
        me = torch.arange(a, a + cand.shape[0], device=x.device)[:, None]
        ok = (cand >= 0) & (cand != me) & (d <= r)
        k = int(ok.sum(1).max())
        pick = torch.argsort(ok.to(torch.int8), dim=1, descending=True)[:, :k]
        parts.append((cand.gather(1, pick), ok.gather(1, pick), d.gather(1, pick)))
        widest = max(widest, k)
    pad = lambda t, v: torch.nn.functional.pad(t, (0, widest - t.shape[1]), value=v)  # noqa: E731
    ok = torch.cat([pad(p[1], False) for p in parts])
    col = torch.where(ok, torch.cat([pad(p[0], 0) for p in parts]), 0)
    return col, ok, torch.where(ok, torch.cat([pad(p[2], 1.0) for p in parts]), 1.0)


def _weights(ok, xi, delta, dx, dV):
    beta = ((delta + dx / 2 - xi) / dx).clamp(0.0, 1.0)
    return torch.where(ok, beta * dV / xi ** 3, 0.0)


class _Model:
    """The explicit step of the four-species model (kernel exponents 0)."""

    def __init__(self, inp):
        p = self.p = inp["params"]
        self.col, ok, xi = _table(inp["nodes"], p.delta * (1.0 + 1e-5))
        self.ok, self.w = ok, _weights(ok, xi, p.delta, p.dx, p.dx * p.dy * p.dz)
        dev = self.w.device
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        self.bc = t(inp["bcvalues"])
        self.dir = (t(inp["bctypes"]) == 0)[None, :] & (self.bc != -1)
        self.c, self.phase = t(inp["icvalues"][:4]), t(inp["phase0"]) != 0
        self.phi = t(inp["icvalues"][4])
        self.c0 = self.c[0].clone()
        self.past, self.op, self.sat = [], None, p.CSat / p.CSolid

    def operator(self):
        if self.op is None:
            solid = self.phase
            w = torch.where(solid[:, None] | solid[self.col], 0.0, self.w)
            free = ~self.dir[4] & (w != 0).any(1)
            diag = torch.where(free, w.sum(1), 1.0)
            self.op = torch.where(free[:, None], w, 0.0), diag, free
        return self.op

    def apply(self, x):
        w, diag, free = self.operator()
        return torch.where(free, diag * x - (w * x[self.col]).sum(1), 0.0)

    def solve(self, b, x, fixed):
        """A x = b on the unknowns (x carries the fixed values if `fixed`), Jacobi CG."""
        _, diag, free = self.operator()
        known = torch.where(free, 0.0, x) if fixed else torch.zeros_like(x)
        scale = float(torch.where(free, b - self.apply(known), 0.0).norm()) or 1.0
        x = torch.where(free, x, known)
        for _ in range(3):
            r = torch.where(free, b - self.apply(x), 0.0)
            if float(r.norm()) <= 1e-13 * scale:
                break
            z = r / diag
            p, rz = z, torch.dot(r, z)
            for it in range(4000):
                q = self.apply(p)
                alpha = rz / torch.dot(p, q)
                x, r = x + alpha * p, r - alpha * q
                if it % 8 == 7 and float(r.norm()) <= 1e-14 * scale:
                    break
                z = r / diag
                new = torch.dot(r, z)
                p, rz = z + (new / rz) * p, new
        return x

    def potential(self):
        p = self.p
        z = torch.tensor(list(p.z), dtype=torch.float64, device=self.c.device)
        b = p.F * p.CSolid / (p.K_phi * p.sigma) * (z[:, None] * self.c).sum(0)
        h = self.past
        x = self.phi if len(h) < 3 else 3 * h[-1] - 3 * h[-2] + h[-3]
        x = torch.where(self.dir[4], self.bc[4], torch.where(self.operator()[2], x, self.phi))
        self.phi = self.solve(b, x, True)
        self.past = h[-2:] + [self.phi]

    def diffusivity(self, k):
        """(N, K) diffusivity of species k on the bonds (vol_red is 0: BV = 1)."""
        p, a, n = self.p, self.phase[:, None], self.phase[self.col]
        D = torch.where(a | n, p.D_solid[k], torch.full_like(self.w, p.D_liquid[k]))
        return D if k == 0 else torch.where(a & n, 0.0, D)

    def switch(self):
        w = self.p.switch_width
        return torch.sigmoid((self.c[0] - self.sat) / w) if w > 0 else (self.c[0] > self.sat).double()

    def interface(self):
        return self.phase & (self.ok & ~self.phase[self.col]).any(1)

    def step(self):
        """One step; returns the mask of the clamped values."""
        p = self.p
        self.potential()
        dphi = self.phi[self.col] - self.phi[:, None]
        new, clamped = torch.empty_like(self.c), torch.zeros_like(self.c, dtype=torch.bool)
        for k in range(4):
            cn = self.c[k][self.col]
            f = p.K1[k] * (cn - self.c[k][:, None]) + p.K2[k] * p.z[k] * p.F / (p.R * p.T) * cn * dphi
            rate = (self.w * self.diffusivity(k) * f).sum(1)
            if k == 0:
                rate = rate - torch.where(self.interface(), p.k_diss * self.switch(), 0.0)
            v = torch.where(self.dir[k], self.bc[k] / p.CSolid, self.c[k] + p.dt * rate)
            clamped[k] = v < p.c_floor
            new[k] = v.clamp(min=p.c_floor)
        self.c = new
        flip = self.phase & (new[0] <= self.sat)
        if bool(flip.any()):
            self.phase, self.op = self.phase & ~flip, None
        return clamped

    def lost(self):
        return float((self.c0 - self.c[0]).sum()) * self.p.dx * self.p.dy * self.p.dz

    def state(self):
        return dict(c=self.c, phi=self.phi, phase=self.phase.to(torch.int32))


def _exact_gradient(case, seed):
    m = _Model(_package().synth(3, case["n"], seed))
    p = m.p
    curve, kept = [], []
    for s in range(1, case["steps"] + 1):
        c, phase = m.c, m.phase
        clamped = m.step()
        kept.append((c, m.phi, phase, clamped))
        if s % case["sample"] == 0:
            curve.append(m.lost())
    end = m.state()
    rng = np.random.default_rng(seed).uniform(0.5, 1.5, case["steps"] // case["sample"])
    dV = p.dx * p.dy * p.dz
    z = [float(v) for v in p.z]
    lam, gD, gk = torch.zeros_like(m.c), [0.0] * 4, 0.0
    psi = torch.zeros_like(m.phi)
    for s in range(case["steps"], 0, -1):
        if s % case["sample"] == 0:
            lam[0] -= dV * float(rng[s // case["sample"] - 1])
        m.c, m.phi, phase, clamped = kept[s - 1]
        if not torch.equal(phase, m.phase):
            m.phase, m.op = phase, None
        lh = torch.where(m.dir[:4] | clamped, 0.0, lam)
        dphi = m.phi[m.col] - m.phi[:, None]
        mu, nu = torch.empty_like(lam), torch.zeros_like(m.phi)
        for k in range(4):
            wD = m.w * m.diffusivity(k)
            K2 = p.K2[k] * z[k] * p.F / (p.R * p.T)
            ln, cn = lh[k][m.col], m.c[k][m.col]
            mu[k] = lh[k] + p.dt * (wD * (p.K1[k] * (ln - lh[k][:, None]) - K2 * ln * dphi)).sum(1)
            nu += p.dt * K2 * (m.c[k] * (wD * ln).sum(1) - lh[k] * (wD * cn).sum(1))
            rate = (wD * (p.K1[k] * (cn - m.c[k][:, None]) + K2 * cn * dphi)).sum(1)
            gD[k] += float((lh[k] * rate).sum()) * p.dt / p.D_liquid[k]
        on = m.interface() & ~m.dir[0]
        sw = m.switch()
        slope = sw * (1 - sw) / p.switch_width if p.switch_width > 0 else torch.zeros_like(sw)
        mu[0] -= torch.where(on, lh[0] * p.dt * p.k_diss * slope, 0.0)
        gk -= float(torch.where(on, lh[0] * p.dt * sw, 0.0).sum())
        psi = m.solve(nu, psi, False)
        free = m.operator()[2]
        f = p.F * p.CSolid / (p.K_phi * p.sigma)
        for k in range(4):
            mu[k] += torch.where(free, f * z[k] * psi, 0.0)
        lam = mu
    return dict(curve=np.array(curve), gD=np.array(gD), gk=gk, state=end)


def _exact_residual_ten(case, seed):
    _, nodes, phase, r, _ = _chem_lattice(case, seed)
    col, ok, xi = _table(nodes, r)
    U1, U0 = (torch.as_tensor(a, device=col.device) for a in _chem_fields(phase.size, seed))
    d = DATA2
    w = _weights(ok, xi, d[6], d[3], d[3] * d[4] * d[5])
    s = torch.as_tensor(phase, device=col.device) != 0
    a, n = s[:, None], s[col]
    iface, liq = s & (ok & ~s[col]).any(1), ~s
    act = iface | liq
    Cs, T, R, Fc = d[7], d[47], d[48], d[49]
    dphi = U0[10][col] - U0[10][:, None]
    F = torch.zeros_like(U1)
    for k in range(10):
        z, Ds, Dl, _, _, K1, K2 = DATAC[k]
        D = torch.where(a | n, Ds, torch.full_like(w, Dl))
        if k == 0:
            D = torch.where(a ^ n, Ds * 10.0 ** (-d[50] * (1.0 - VOLN1REL)), D)
        else:
            D = torch.where(a & n, 0.0, D)
        un = U1[k][col]
        F[k] = (U1[k] - U0[k]) / d[2] - (w * D * (K1 * (un - U1[k][:, None]) + K2 * z * Fc / (R * T) * un * dphi)).sum(1)
    lim = lambda i: 10.0 ** -d[i] / Cs  # noqa: E731
    over = lambda u, i: (u - lim(i)).clamp(min=0.0)  # noqa: E731
    k1, k2, k3, k4, k5, k6, k7, k8, k9 = (d[i] for i in (29, 31, 33, 35, 37, 39, 41, 43, 45))
    ca5 = lambda u: u * U0[7] ** 5 * U0[6] ** 3  # noqa: E731
    on = lambda m, v: torch.where(m, v, 0.0)  # noqa: E731
    po4 = k4 * over(U0[0] ** 3 * U0[5] ** 2, 17)
    F[0] += on(act, k1 * over(U1[0] * U0[2] ** 2, 14) + k2 * over(U1[0] * U0[4], 15) + k3 * over(U1[0] * U0[4], 16) + po4)
    phic = R * T / (Fc * DATAC[0][0]) * torch.log(U0[0] / (d[8] / Cs))
    source = d[46] / (DATAC[1][0] * Fc * Cs) * torch.exp(-d[27] * Fc * (d[23] + d[24] - U0[10] - phic) / (R * T))
    F[1] -= on(iface, source) + on(liq, k7 * (lim(20) - U1[1] * U0[2]) + k8 * (lim(21) - U1[1] * U0[4])
                                   + k9 * (lim(22) - U1[1] * U0[6]))
    F[2] += on(act, k1 * over(U0[2] ** 2 * U0[0], 14) + k6 * over(ca5(U1[2]), 19)) - on(liq, k7 * (lim(20) - U1[2] * U0[1]))
    F[3] -= on(liq, k8 * (lim(21) - U1[3] * U0[1]))
    F[4] += on(act, k2 * over(U1[4] * U0[0], 15) + k3 * over(U1[4] * U0[0], 16) + k5 * over(U1[4] * U0[7], 18)) \
        - on(liq, k8 * (lim(21) - U0[1] * U1[4]))
    F[5] += on(act, po4) - on(liq, k9 * (U0[6] * U0[1] - lim(22)))
    F[6] += on(act, k6 * over(ca5(U0[2]), 19)) - on(liq, k9 * (lim(22) - U1[6] * U0[1]))
    F[7] += on(act, k5 * over(U1[7] * U0[4], 18) + k6 * over(ca5(U0[2]), 19))
    ll = torch.where(a | n, 0.0, w)
    charge = sum(DATAC[k][0] * U0[k] for k in range(10))
    row = -(ll * (U1[10][col] - U1[10][:, None])).sum(1) - Fc * Cs * charge / (DATAC11[3] * DATAC11[1])
    F[10] = on((ok & ~a & ~n).any(1), row)
    return F


def exact(case, seed):
    path = case["path"]
    if path in ("explicit", "step_host"):
        m = _Model(_package().synth(case["kind"], case["n"], seed))
        for _ in range(case["steps"]):
            m.step()
        return m.state()
    if path == "ensemble":
        out = []
        for inp in _member_synth(case, seed):
            m = _Model(inp)
            for _ in range(case["steps"]):
                m.step()
            out.append(m.state())
        return out
    if path == "gradient":
        return _exact_gradient(case, seed)
    if path == "residual_ten":
        return _exact_residual_ten(case, seed)
    # the implicit steps return the iterate at which a truncated Krylov method stops (relative
    # residual 1e-5), the neighbour lists are whole numbers
    return None
