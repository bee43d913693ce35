"""The measured cases of the k-mesh response engine.

A case is one call that a program makes through the public entry points of
``wanniernlqg_b200.engine.ResponseEngine`` with a model and a compiled task in hand, from one rule of
an adaptive integrator on a 4-orbital model (where launches and latency count) to blocks of the
256^3 mesh of the 32-orbital model and 96-orbital transport.  ``exact`` evaluates the same formulas
in 64 bits with plain torch.

Case fields: ``entry`` (the call), ``responses`` ("kind:component,component;..."), ``nw`` and ``rmax``
(orbitals and the R cube |R_i| <= rmax of the seeded synthetic models), ``variant`` of the model,
``n`` points (or the whole ``mesh``), ``axis`` energies on the photon or Fermi axis up to ``top`` eV,
``width`` and ``kernel`` of the broadening, ``temperature`` and ``precision``.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from wanniernlqg_b200 import _abi
from wanniernlqg_b200.engine import ResponseEngine
from wanniernlqg_b200.model import kramers_doubled_model, synthetic_nonorthogonal_model, synthetic_orthogonal_model

KINDS = {"shift": _abi.SHIFT_CURRENT, "injection": _abi.INJECTION_CURRENT, "curvature": _abi.BERRY_CURVATURE,
         "metric": _abi.QUANTUM_METRIC, "ahc": _abi.INTRINSIC_AHC, "dipole": _abi.BERRY_DIPOLE,
         "shg": _abi.SECOND_HARMONIC, "jerk": _abi.JERK_CURRENT, "transport": _abi.LINEAR_TRANSPORT_BERRY}
OPTICAL = "shift:xyy;curvature:xy;metric:xx"
CURRENTS = "shift:xyy;injection:xyy"
TRANSPORT = "transport:xy;dipole:xyx"


def _case(entry, responses, nw, rmax, n, *, mesh=256, axis=128, top=3.0, width=0.02, kernel="lorentzian",
          temperature=0.0, precision="fp64", variant="orthogonal", depth=0, name=None):
    case = {"entry": entry, "responses": responses, "nw": nw, "rmax": rmax, "n": n, "mesh": mesh,
            "depth": depth or mesh, "axis": axis, "top": top, "width": width, "kernel": kernel,
            "temperature": temperature, "precision": precision, "variant": variant}
    return {"name": name, **case} if name else case


def listed():
    return [
        # One Genz-Malik rule of the adaptive integrator (33 nodes in 3D), the smallest call there is.
        _case("points", CURRENTS, 4, 2, 33, name="rule_nw4"),
        # The CPU-runnable workload as a whole: the 4-orbital model on its 32^3 mesh.
        _case("mesh", CURRENTS, 4, 2, 32 ** 3, mesh=32, name="mesh32_nw4"),
        # The workload of the throughput figure: a run of the 256^3 mesh, result left on the device.
        _case("mesh_device", OPTICAL, 32, 4, 32768, axis=512, top=4.0, width=0.01, name="block_nw32"),
        # The same run at mixed precision.
        _case("mesh_device", OPTICAL, 32, 4, 32768, axis=512, top=4.0, width=0.01, precision="mixed",
              name="block_nw32_mixed"),
        # Random sampling of the zone with weights, from host arrays.
        _case("weighted", OPTICAL, 32, 4, 8192, axis=512, top=4.0, width=0.01, name="random_nw32"),
        # One refinement round of the cell-adaptive integrator: point values at low photon energies.
        _case("points", "injection:xyz", 16, 2, 4913, axis=20, top=0.1, width=0.005, kernel="gaussian",
              precision="mixed", name="cells_nw16_mixed"),
        # Transport at finite temperature of a Kramers-doubled model (near-degenerate pairs).
        _case("mesh_device", TRANSPORT, 24, 3, 32768, mesh=128, axis=3, top=0.5, temperature=50.0,
              variant="kramers", name="transport_nw24"),
        # The largest orbital count of the batched workload.
        _case("mesh_device", TRANSPORT, 96, 2, 2048, mesh=64, axis=3, top=0.5, temperature=50.0,
              name="transport_nw96"),
        # A Fermi-level scan of the anomalous Hall conductivity of a film (one k layer).
        _case("mesh", "ahc:xy", 18, 2, 45 * 45, mesh=45, depth=1, axis=201, top=1.0, name="hall_scan_nw18"),
        # Nonorthogonal orbitals: both currents with the metric geometry.
        _case("mesh_device", CURRENTS, 64, 3, 1024, mesh=192, axis=256, variant="overlap", name="overlap_nw64"),
        # Second harmonic spectra on a whole small mesh.
        _case("mesh", "shg:xxx,xyz", 16, 2, 12 ** 3, mesh=12, axis=256, name="shg_nw16"),
        # Energies and eigenvectors along a band path (an odd number of points and orbitals).
        _case("spectrum", "curvature:xy", 31, 3, 601, name="bands_nw31"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["currents", "optical", "optical", "cells", "transport", "hall", "overlap", "shg", "jerk",
                         "bands"])
    precision = rng.choice(["fp64", "fp64", "mixed"])
    kernel = rng.choice(["lorentzian", "gaussian"])
    if family == "currents":
        n = _log(rng, 9, 16384)
        return _case("points" if n < 2000 else "weighted", CURRENTS, rng.randint(2, 8), 2, n, axis=_log(rng, 32, 512),
                     kernel=kernel, precision=precision)
    if family == "optical":
        nw = rng.randint(8, 48)
        n = max(1, min(_log(rng, 1024, 16384), 16384 * 512 // nw ** 2))
        return _case(rng.choice(["mesh_device", "weighted"]), OPTICAL, nw, rng.randint(2, 4), n,
                     mesh=rng.choice([64, 100, 256]), axis=_log(rng, 64, 512), top=4.0, width=0.01,
                     kernel=kernel, precision=precision)
    if family == "cells":
        return _case("points", "injection:xyz", rng.randint(6, 20), 2, _log(rng, 64, 8192), axis=rng.randint(10, 40),
                     top=0.1, width=0.005, kernel="gaussian", precision=precision)
    if family == "transport":
        nw = rng.choice([6, 8, 12, 16, 24, 32, 48, 64])
        n = max(64, min(_log(rng, 256, 16384), 16384 * 256 // nw ** 2))
        return _case("mesh_device", TRANSPORT, nw, rng.randint(2, 3), n, mesh=rng.choice([64, 96, 128]),
                     axis=rng.randint(1, 9), top=0.5, temperature=50.0, precision="fp64",
                     variant=rng.choice(["orthogonal", "kramers"]))
    if family == "hall":
        mesh = rng.randint(12, 64)
        return _case("mesh", "ahc:xy", rng.randint(4, 30), 2, mesh * mesh, mesh=mesh, depth=1,
                     axis=_log(rng, 11, 401), top=1.0)
    if family == "overlap":
        return _case("mesh_device", CURRENTS, rng.randint(10, 64), 2, _log(rng, 128, 1024), mesh=rng.choice([64, 192]),
                     axis=_log(rng, 64, 256), variant="overlap", precision=precision)
    if family == "shg":
        mesh = rng.randint(4, 12)
        return _case("mesh", rng.choice(["shg:xxx", "shg:xxx,xyz", "shg:xyy,yzx,zzz"]), rng.randint(4, 20), 2,
                     mesh ** 3, mesh=mesh, axis=_log(rng, 64, 256), kernel=kernel)
    if family == "jerk":
        return _case("points", "jerk:xyyx", rng.randint(4, 32), 2, _log(rng, 64, 2048), axis=_log(rng, 32, 256),
                     kernel=kernel)
    return _case("spectrum", "curvature:xy", rng.randint(4, 40), rng.randint(2, 3), _log(rng, 33, 1201))


def _model(case, seed):
    nw, rmax = case["nw"], case["rmax"]
    if case["variant"] == "overlap":
        return synthetic_nonorthogonal_model(nw, rmax, seed, full_position=True)
    if case["variant"] == "kramers":
        return kramers_doubled_model(synthetic_orthogonal_model(nw // 2, rmax, seed, full_position=True), 1e-3, seed)
    return synthetic_orthogonal_model(nw, rmax, seed, full_position=nw > 4)


def _responses(case):
    return [(part.split(":")[0], part.split(":")[1].split(",")) for part in case["responses"].split(";")]


def _task(case):
    fermi = any(kind in ("ahc", "dipole", "transport") for kind, _ in _responses(case))
    grid = np.linspace(-case["top"], case["top"], case["axis"]) if fermi else np.linspace(0.0, case["top"], case["axis"])
    return _abi.TaskArrays(
        [(KINDS[kind], comps) for kind, comps in _responses(case)],
        broadening_type=_abi.GAUSSIAN if case["kernel"] == "gaussian" else _abi.LORENTZIAN, broadening=case["width"],
        temperature=case["temperature"], degeneracy_threshold=1e-12 if fermi else 2e-3,
        photon_energies=() if fermi else grid, fermi_energies=grid if fermi else (),
        precision=_abi.PRECISION_MIXED if case["precision"] == "mixed" else _abi.PRECISION_FP64)


def _mesh(case):
    return (case["mesh"], case["mesh"], case["depth"])


def _block(case, seed):
    """A run of mesh indices that starts anywhere in the mesh."""
    total = int(np.prod(_mesh(case)))
    if case["entry"] == "mesh":
        return 0, total
    n = min(case["n"], total)
    begin = int(np.random.default_rng(seed + 1).integers(0, total - n + 1))
    return begin, begin + n


def _points(case, seed):
    rng = np.random.default_rng(seed + 2)
    if case["entry"] == "spectrum":   # a straight path between two points of the zone
        t = np.linspace(0.0, 1.0, case["n"])[:, None]
        return rng.random(3) * (1.0 - t) + rng.random(3) * t
    return rng.random((case["n"], 3))


def prepare(case, seed):
    task = _task(case)
    state = {"entry": case["entry"], "task": task, "mesh": _mesh(case)}
    n = int(np.prod(state["mesh"])) if case["entry"] == "mesh" else case["n"]
    state["engine"] = ResponseEngine(_model(case, seed), task, max_batch=n)
    if case["entry"] in ("points", "spectrum", "weighted"):
        state["k"] = _points(case, seed)
        state["w"] = np.full(case["n"], 1.0 / case["n"])
    if case["entry"] == "mesh_device":
        state["block"] = _block(case, seed)
        state["out"] = torch.zeros(state["engine"].value_count, dtype=torch.complex128, device="cuda")
    return state


def run(state):
    engine, entry = state["engine"], state["entry"]
    if entry == "mesh_device":
        engine.integrate_mesh_device(state["mesh"], *state["block"], state["out"].data_ptr(),
                                     torch.cuda.current_stream().cuda_stream)
        return [state["out"][off:off + n] for off, n in state["task"].block_offsets()]
    if entry == "spectrum":
        energies, vectors = engine.spectrum(state["k"])
        return {"energies": energies, "vectors": vectors}
    if entry == "points":
        return state["task"].split(engine.point_values(state["k"]))
    if entry == "weighted":
        return state["task"].split(engine.weighted_sum(state["k"], state["w"]))
    return state["task"].split(engine.integrate_mesh(state["mesh"]))


def work(case):
    """The real-space operators once, the k-points and the values once; per point a Hermitian
    eigensolve (30 nw^3), two nw^3 complex products per rotated operator and the spectral sums."""
    nw, nr, n = case["nw"], (2 * case["rmax"] + 1) ** 3, case["n"]
    values, products, sums, operators = 0, 0.0, 0.0, 1
    for kind, comps in _responses(case):
        nc, axis = len(comps), case["axis"]
        if kind == "shg":
            values += nc * axis * 14
            products += 24 * 2 + 9 * 8
            sums += nc * axis * 52 * nw * nw / 4
        elif kind in ("shift", "injection", "jerk"):
            values += nc * axis
            products += nc * {"shift": 10, "injection": 6, "jerk": 5}[kind]
            sums += nc * axis * 8 * nw * nw / 4
        else:
            values += nc * (axis if kind in ("ahc", "dipole", "transport") else 1)
            products += 0 if case["entry"] == "spectrum" else nc * 9
    operators = 1 if case["entry"] == "spectrum" else 4
    nbytes = operators * 16 * nr * nw * nw + 24 * n
    if case["entry"] == "spectrum":
        nbytes += n * (8 * nw + 16 * nw * nw)
    else:
        nbytes += 16 * values * (n if case["entry"] == "points" else 1)
    return {"bytes": float(nbytes), "flops": float(n * (30 * nw ** 3 + 8 * products * nw ** 3 + sums))}


# ---- the formulas in 64 bits -------------------------------------------------------------------

KB_EV = 8.617333262145e-5
CHARGE, HBAR_J, HBAR_EV = 1.602176634e-19, 1.054571817e-34, 6.582119569e-16


def _axes(component):
    return ["xyz".index(ch) for ch in component]


class _Geometry:
    """Band energies, vectors and operators of a batch of k-points (matrices [k, n, m])."""

    def __init__(self, model, k, eta):
        def on(a):
            return torch.from_numpy(np.ascontiguousarray(a)).cuda()
        self.nw, self.eta = model.num_orbitals, eta
        self.r = on(model.r_vectors.T.astype(np.float64))
        self.cart = self.r @ on(model.lattice)
        self.phase = torch.exp(2j * math.pi * (k @ self.r.T)) / on(model.r_degeneracies)
        self.h_r = on(model.hamiltonian_r.transpose(2, 0, 1))
        self.a_r = on(model.position_r.transpose(3, 2, 0, 1))
        self.s_r = None if model.overlap_r is None else on(model.overlap_r.transpose(2, 0, 1))
        self.kept = {}
        h = self.fourier("h")
        if self.s_r is None:
            self.e, self.u = torch.linalg.eigh(h)
        else:
            inv = torch.linalg.inv(torch.linalg.cholesky(self.fourier("s")))
            self.e, v = torch.linalg.eigh(inv @ h @ inv.mH)
            self.u = inv.mH @ v
        self.gap = self.e[:, :, None] - self.e[:, None, :]   # E_n - E_m
        self.off = ~torch.eye(self.nw, dtype=torch.bool, device="cuda")

    def fourier(self, op, *deriv):
        """sum_R exp(2 pi i k.R) (i R_d) ... X(R), X = h, s or the position axis 0-2."""
        x = self.h_r if op == "h" else self.s_r if op == "s" else self.a_r[:, op]
        f = self.phase
        for d in deriv:
            f = f * (1j * self.cart[:, d])
        return (f @ x.reshape(x.shape[0], -1)).reshape(-1, self.nw, self.nw)

    def band(self, op, *deriv):
        key = (op, *deriv)
        if key not in self.kept:
            self.kept[key] = self.u.mH @ self.fourier(op, *deriv) @ self.u
        return self.kept[key]

    def inverse(self):
        """Regularised 1 / (E_n - E_m)."""
        return self.gap / (self.gap ** 2 + self.eta ** 2)

    def d(self, a):
        return -self.band("h", a) * self.inverse()

    def connection(self, a):
        return self.metric(a)[2] if self.s_r is not None else self.band(a) + 1j * self.d(a)

    def velocity(self, a):
        if self.s_r is not None:
            return _diag(self.band("h", a)).real - self.e * _diag(self.band("s", a)).real
        return _diag(self.band("h", a)).real

    def derivative(self, p, d):
        """Generalised derivative of the connection r^p along d."""
        if self.s_r is not None:
            return self.metric_derivative(p, d)
        dd, dp, hp, ap = self.d(d), self.d(p), self.band("h", p), self.band(p)
        d_a, d_h = _differences(self.band(d)), _differences(self.band("h", d))
        h = self.band("h", p, d) + d_h * dp + hp @ dd - dd @ hp
        return self.band(p, d) + d_a * (dp - 1j * ap) + ap @ dd - dd @ ap - 1j * h * self.inverse()

    def metric(self, a):
        """Eigenvector derivative, source and Berry connection of nonorthogonal orbitals."""
        dh, ds = self.band("h", a), self.band("s", a)
        b = self.band(a) + 1j * ds
        mean = 0.5 * (self.e[:, :, None] + self.e[:, None, :])
        d = -0.5 * ds + (dh - mean * ds) * self.off * (-self.inverse())
        d = d + torch.diag_embed(1j * _diag(b).real)
        return d, b, 1j * d + b

    def metric_derivative(self, p, d):
        dd, bd, rd = self.metric(d)
        _, bp, rp = self.metric(p)
        hp, sp = self.band("h", p), self.band("s", p)
        mean = 0.5 * (self.e[:, :, None] + self.e[:, None, :])
        gap = -self.gap
        q = gap ** 2 + self.eta ** 2
        v = self.velocity(d)
        v_sum, v_diff = v[:, :, None] + v[:, None, :], v[:, None, :] - v[:, :, None]
        hd = dd.mH @ hp + hp @ dd + self.band("h", p, d)
        sd = dd.mH @ sp + sp @ dd + self.band("s", p, d)
        bd = dd.mH @ bp + bp @ dd + self.band(p, d) + 1j * self.band("s", p, d)
        nd = hd - mean * sd - 0.5 * v_sum * sp
        out = -0.5 * sd + nd * gap / q + (hp - mean * sp) * (self.eta ** 2 - gap ** 2) / q ** 2 * v_diff
        return (1j * out + bd - 1j * _differences(rd) * rp) * self.off

    def curvature_diagonal(self, a, b):
        """(U' (d_a A_b - d_b A_a) U)_nn - i [A_a, A_b]_nn."""
        aa, ab = self.band(a), self.band(b)
        return _diag(self.band(b, a) - self.band(a, b) - 1j * (aa @ ab - ab @ aa)).real


def _diag(x):
    return torch.diagonal(x, dim1=-2, dim2=-1)


def _differences(x):
    d = _diag(x)
    return d[:, :, None] - d[:, None, :]


def _step(e, mu):
    return (e <= mu).double()


def _logistic(e, mu, temperature):
    return torch.special.expit(-(e - mu) / (KB_EV * temperature))


def _delta(case, x):
    w = case["width"]
    if case["kernel"] == "gaussian":
        return torch.exp(-(x / w) ** 2) / (math.sqrt(math.pi) * w)
    return w / math.pi / (x * x + w * w)


def _pair_sum(weight, kernel):
    """sum over pairs of weight[k, pair] kernel[k, pair, energy], complex times real or complex."""
    parts = [kernel.real, kernel.imag] if kernel.is_complex() else [kernel]
    out = [torch.complex((weight.real[:, None] @ p)[:, 0], (weight.imag[:, None] @ p)[:, 0]) for p in parts]
    return out[0] + 1j * out[1] if len(out) == 2 else out[0]


def _energies(case):
    return torch.linspace(0.0, case["top"], case["axis"], dtype=torch.float64, device="cuda")


def _spectrum_of_pairs(case, weight, te, keep, screen):
    """sum over kept pairs of weight[k, pair] times the broadened delta at each photon energy."""
    om, w = _energies(case), case["width"]
    gauss = case["kernel"] == "gaussian"
    window = w * math.sqrt(200.0) if gauss and screen else 5.0 * w
    out = []
    step = max(1, 20_000_000 // (te.shape[1] * om.numel()))
    for t, q, kept in zip(te.split(step), weight.split(step), keep.split(step)):
        x = t[:, :, None] - om
        f = _delta(case, x)
        if screen:
            near = (x.abs() < window) & kept[:, :, None]
            f = f * (near if gauss else near.any(2).any(1)[:, None, None])
        else:
            f = f * (x.abs() <= window)
        out.append(_pair_sum(q * kept, f))
    return torch.cat(out)


def _pair_response(case, g, kind, comp):
    ax = _axes(comp)
    f = _step(g.e, 0.0)
    if kind == "jerk":
        a, b, c, d = ax
        hess = _diag(g.band("h", a, d)).real + 2.0 * ((g.band("h", a) * g.band("h", d).mT).real * g.inverse()
                                                       * g.off).sum(-1)
        fnm, te = f[:, None, :] - f[:, :, None], g.gap
        q = (hess[:, :, None] - hess[:, None, :]) * g.connection(b) * g.connection(c).mT
        keep = (te > 0) & (fnm != 0) & g.off
        return _spectrum_of_pairs(case, (q * fnm).flatten(1), te.flatten(1), keep.flatten(1), False)
    a, b, c = ax
    fnm, te = f[:, :, None] - f[:, None, :], -g.gap
    r_b, r_c = g.connection(b), g.connection(c)
    if kind == "shift":
        q = -1j * (g.derivative(c, a) * r_b.mT - g.derivative(b, a).mT * r_c)
        scale = -HBAR_EV * math.pi * CHARGE ** 3 / (2.0 * HBAR_J ** 2)   # cell volume 1
    else:
        v = g.velocity(a)
        q = (v[:, None, :] - v[:, :, None]) * r_c * r_b.mT
        scale = -math.pi * CHARGE ** 3 / HBAR_J ** 2
    keep = (fnm.abs() > 1e-10) & g.off
    return scale * _spectrum_of_pairs(case, (q * fnm).flatten(1), te.flatten(1), keep.flatten(1), True)


def _band_response(case, g, kind, comp):
    a, b = _axes(comp)[:2]
    r_a, r_b = g.connection(a), g.connection(b)
    if kind in ("curvature", "metric"):
        f = _step(g.e, 0.0)
        q = r_a * r_b.mT
        if kind == "metric":
            return (0.5 * (f[:, :, None] + f[:, None, :]) * q.real * g.off).sum((1, 2))[:, None].to(torch.complex128)
        pair = ((f[:, :, None] - f[:, None, :]) * (1j * q).real * g.off).sum((1, 2))
        return (pair + (f * g.curvature_diagonal(a, b)).sum(-1))[:, None].to(torch.complex128)
    diag = g.curvature_diagonal(a, b)
    out = []
    for mu in np.linspace(-case["top"], case["top"], case["axis"]):
        if kind == "dipole":
            z = torch.exp(-((g.e - mu) / (KB_EV * case["temperature"])).abs())
            slope = z / (KB_EV * case["temperature"] * (1.0 + z) ** 2)
            omega = diag - 2.0 * ((r_a * r_b.mT).imag * g.off).sum(-1)
            out.append((slope * omega * g.velocity(_axes(comp)[2])).sum(-1))
        elif kind == "transport":
            f = _logistic(g.e, mu, case["temperature"])
            pair = (f[:, :, None] - f[:, None, :]) * (1j * r_a * r_b.mT).real * g.off
            out.append(-(CHARGE ** 2 / HBAR_J * 1e-20) * ((f * diag).sum(-1) + pair.sum((1, 2))))
        else:
            f = _step(g.e, mu)
            inv = torch.where(g.off, 1.0 / g.gap, torch.zeros_like(g.gap))
            l_a, l_b = (g.band(x) - 1j * g.band("h", x) * inv for x in (a, b))
            pair = -(l_a * l_b.mT - l_b * l_a.mT).imag
            out.append((f * diag).sum(-1) + (f[:, :, None] * (1.0 - f[:, None, :]) * pair).sum((1, 2)))
    return torch.stack(out, 1).to(torch.complex128)


def _resonance(case, x):
    w = case["width"]
    lor = w / (x * x + w * w)
    return torch.complex(x / w * lor, math.sqrt(math.pi) / w * torch.exp(-(x / w) ** 2)
                         if case["kernel"] == "gaussian" else lor)


def _second_harmonic(case, g, comps):
    """[k, quantity, term, component, energy] of the five pair terms (T = 0: no one-band terms)."""
    nw, eta = g.nw, g.eta
    om = _energies(case)
    v, pos = [g.band("h", a) for a in range(3)], [g.band(a) for a in range(3)]
    rise = -g.gap                                        # E_m - E_n
    bare = torch.where(rise.abs() < 1e-7, torch.zeros_like(rise), 1.0 / rise)
    soft = rise / (rise ** 2 + eta ** 2)
    weight = eta ** 2 / (rise ** 2 + eta ** 2)
    r0, r_eta = [[p + 1j * x * w for p, x in zip(pos, v)] for w in (bare, soft)]

    def vertex(a, b):
        dr = v[b] * soft
        da, db = _differences(pos[a]), _differences(pos[b])
        va, vb = _differences(v[a]), _differences(v[b])
        d0a, d0b = v[a] * bare, v[b] * bare
        finite = g.band(a, b) + pos[a] @ dr - dr @ pos[a] - da * dr + da * d0b + db * d0a - 1j * pos[a] * db
        wv, wa = v[b] * weight * g.off, pos[b] * weight * g.off
        ao, bo = pos[a] * g.off, (v[a] + 1j * pos[a] * g.gap) * g.off
        corr = (ao @ wv - bo @ wa) - (wv @ ao - wa @ bo)
        num = 1j * (g.band("h", a, b) + v[a] @ dr - dr @ v[a] - va * dr + d0a * vb.real + d0b * va.real) + corr
        return finite + num * bare

    f = _step(g.e, 0.0)
    fo = f[:, :, None] - f[:, None, :]
    out = torch.zeros(g.e.shape[0], 2, 7, len(comps), om.numel(), dtype=torch.complex128, device="cuda")
    low = om / (om ** 2 + 0.025 ** 2)

    def principal(x):
        return x / (x ** 2 + eta ** 2)

    e_n, e_m, e_l = g.e[:, :, None, None], g.e[:, None, :, None], g.e[:, None, None, :]
    third_off = g.off[None, :, None, :] & g.off[None, None, :, :]
    k_f, k_1, k_2 = (principal(x) * third_off for x in (2 * e_l - e_n - e_m, 2 * e_n - e_m - e_l, 2 * e_m - e_l - e_n))
    for ic, comp in enumerate(comps):
        a, b, c = _axes(comp)
        dv = {x: -_differences(v[x]).real for x in (a, b, c)}   # V_mm - V_nn
        first = r0[a] * (vertex(b, c) + vertex(c, b)).mT
        second = vertex(a, b) * r0[c].mT + vertex(a, c) * r0[b].mT
        third = r0[a] * (r0[b].mT * dv[c] + r0[c].mT * dv[b]) * bare
        fourth = vertex(b, a) * r0[c].mT + vertex(c, a) * r0[b].mT
        fifth = -(r0[b] * r0[c].mT + r0[c] * r0[b].mT) * dv[a]
        through = torch.einsum("kml,kln,knml->knm", r_eta[b], r_eta[c], k_f.to(torch.complex128)) + \
            torch.einsum("kml,kln,knml->knm", r_eta[c], r_eta[b], k_f.to(torch.complex128))
        tf = r0[a] * through
        to = torch.einsum("kml,kln,knml->knm", r_eta[a], r_eta[b], k_1.to(torch.complex128)) * r0[c] + \
            torch.einsum("kml,kln,knml->knm", r_eta[a], r_eta[c], k_1.to(torch.complex128)) * r0[b] + \
            torch.einsum("kln,kml,knml->knm", r_eta[a], r_eta[c], k_2.to(torch.complex128)) * r0[b] + \
            torch.einsum("kln,kml,knml->knm", r_eta[a], r_eta[b], k_2.to(torch.complex128)) * r0[c]
        o = (fo * (fo.abs() >= 1e-10)).flatten(1)
        inv, q1, q2, q3, q4, q5, qt, qo = (x.flatten(1) for x in (bare, first, second, third, fourth, fifth, tf, to))
        oi, od = o * inv, o * rise.flatten(1)
        p = out[:, :, :, ic]
        step = max(1, 10_000_000 // (o.shape[1] * om.numel()))
        for s in (slice(i, i + step) for i in range(0, o.shape[0], step)):
            t = rise[s].flatten(1)[:, :, None]
            d1, d2, dn = (_resonance(case, x) for x in (t - om, t - 2 * om, -t - om))
            p[s, 0, 0] = 0.5j * (_pair_sum((2 * oi * q1)[s], d2) + _pair_sum((oi * q2)[s], d1))
            p[s, 0, 1] = 0.5j * _pair_sum((oi * q3)[s], d1 - 4 * d2)
            p[s, 0, 2] = 0.5 * (_pair_sum((2 * o * qt)[s], d2) + _pair_sum((o * qo)[s], dn))
            p[s, 0, 3] = -0.25j * _pair_sum((oi * q4)[s], d1)
            p[s, 0, 4] = -0.125j * low ** 2 * _pair_sum((o * q5)[s], d1)
            p[s, 1, 0] = _pair_sum((o * q1)[s], d2) + _pair_sum((o * q2)[s], d1)
            p[s, 1, 1] = _pair_sum((o * q3)[s], d1 - 2 * d2)
            p[s, 1, 2] = -1j * (_pair_sum((od * qt)[s], d2) - _pair_sum((od * qo)[s], dn))
            p[s, 1, 3] = -0.5 * _pair_sum((o * q4)[s], d1)
            p[s, 1, 4] = -0.25 * low * _pair_sum((o * q5)[s], d1)
        p[:, 0, 0] += 0.5j * ((q1 + q2) * oi).sum(1)[:, None] * low
        p[:, 0, 1] -= 0.5j * (q3 * oi).sum(1)[:, None] * low
        p[:, 0, 3] -= 0.25j * (q4 * oi).sum(1)[:, None] * low
    return out


def _values(case, model, k):
    """[k, values] of the task at k-points [k, 3], in the task's order."""
    g = _Geometry(model, k, 1e-3)
    parts = []
    for kind, comps in _responses(case):
        if kind == "shg":
            parts.append(_second_harmonic(case, g, comps).flatten(1))
            continue
        for comp in comps:
            pair = kind in ("shift", "injection", "jerk")
            parts.append((_pair_response if pair else _band_response)(case, g, kind, comp))
    return torch.cat(parts, 1)


def _canonical(u):
    """Each vector's largest component real and positive."""
    pivot = u.abs().argmax(1, keepdim=True)
    p = torch.gather(u, 1, pivot)
    return u * (p.conj() / p.abs())


def exact(case, seed):
    model, task = _model(case, seed), _task(case)
    mesh = _mesh(case)
    if case["entry"] in ("mesh", "mesh_device"):
        begin, end = _block(case, seed)
        i = np.arange(begin, end, dtype=np.int64)
        k = np.stack([(i % mesh[0]) / mesh[0], (i // mesh[0]) % mesh[1] / mesh[1], i // (mesh[0] * mesh[1]) / mesh[2]], 1)
    else:
        k = _points(case, seed)
    k = torch.from_numpy(k).cuda()
    step = min(4096, max(1, 40_000_000 // (case["nw"] ** 3 if "shg" in case["responses"] else 32 * case["nw"] ** 2)))
    if case["entry"] == "spectrum":
        got = [_Geometry(model, x, 0.0) for x in k.split(step)]
        return {"energies": torch.cat([x.e for x in got]).cpu().numpy(),
                "vectors": torch.cat([_canonical(x.u) for x in got]).cpu().numpy()}
    if case["entry"] == "points":
        return task.split(torch.cat([_values(case, model, x) for x in k.split(step)]).cpu().numpy())
    total = sum(_values(case, model, x).sum(0) for x in k.split(step))
    total = (total / (case["n"] if case["entry"] == "weighted" else int(np.prod(mesh)))).cpu().numpy()
    if case["entry"] == "mesh_device":
        return [total[off:off + n] for off, n in task.block_offsets()]
    return task.split(total)
