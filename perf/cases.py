"""The work a user of hv_b200 has it do, as cases that can be timed and checked.

Each case is one pass through the public entry points on synthetic nuclei
(uniform-sphere test particles, the Skyrme and Coulomb settings of the
package's workloads):

kind       entry point                         what it stands for
run        Session.run                         a window of time steps of a device-resident run
simulate   simulate                            a whole run from and to host buffers
batch      Batch.run                           many independent nuclei advanced together
adjoint    AdjointRun / dipole_series          the gradient of a D(t) objective
densities  Session.particle_densities          the pair sums of the Woods-Saxon initialisation
"""
import ctypes
import dataclasses
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "hyper-vlasov_b200"))

import hv_b200 as hv  # noqa: E402
from hv_b200 import _lib as lib  # noqa: E402
from hv_b200.adjoint import AdjointRun, dipole_series  # noqa: E402
from hv_b200.batch import Batch  # noqa: E402

NUCLEI = {"16O": (8, 8), "40Ca": (20, 20), "90Zr": (40, 50), "208Pb": (82, 126)}
HBAR_C, MC2, E2, RHO0 = 197.33, 935.0, 1.44, 0.16
K_FERMI = (3.0 * math.pi ** 2 * 0.08 / 2.0) ** (1.0 / 3.0)
SIGMA_R = 1.444 / (2.0 * math.sqrt(2.0 * math.log(2.0)))
THETA = (-2645.0, 15595.0, 1.0 / 6.0, 32.0)  # t0, t3, sigma, a_sym
FIELDS = {"density": lib.HV_FIELD_DENSITY, "potential": lib.HV_FIELD_POTENTIAL, "coulomb": lib.HV_FIELD_COULOMB,
          "force_x": lib.HV_FIELD_FORCE_X, "force_y": lib.HV_FIELD_FORCE_Y, "force_z": lib.HV_FIELD_FORCE_Z}
PAIR_LIMIT = 3.0e11  # pair sums of exact() that still take seconds


# ---- cases ------------------------------------------------------------------

def _run(nucleus, ppn, n, h, dt, steps, precision="f32", path="fused", deposit="atomic"):
    return {"kind": "run", "nucleus": nucleus, "ppn": ppn, "nx": n[0], "ny": n[1], "nz": n[2], "h": h, "dt": dt,
            "steps": steps, "precision": precision, "path": path, "deposit": deposit, "tol": 1e-6}


def listed():
    cases = [
        # the smallest run: 4,000 test particles, where launches and grid-wide waits count
        dict(_run("40Ca", 100, (32, 32, 32), 1.0, 0.5, 8), name="run-ca40-32"),
        # an ordinary run, 104,000 test particles
        dict(_run("208Pb", 500, (64, 64, 64), 0.5, 0.25, 16), name="run-pb208-64"),
        # the largest run, 2.08 M test particles
        dict(_run("208Pb", 10000, (128, 128, 128), 0.25, 0.2, 16), name="run-pb208-128"),
        # a box fitted to the nucleus: no axis a power of two or a multiple of eight
        dict(_run("90Zr", 400, (75, 61, 50), 0.4, 0.25, 8), name="run-zr90-odd"),
        # the reproducible mode: every node sums its particles in a fixed order
        dict(_run("208Pb", 10000, (128, 128, 128), 0.25, 0.2, 8, deposit="sorted"), name="sorted-pb208-128"),
        # the double-precision drop-in of the reference's step, small and ordinary
        dict(_run("40Ca", 100, (32, 32, 32), 1.0, 0.5, 4, "f64", "plain"), name="plain-ca40-32"),
        dict(_run("208Pb", 500, (64, 64, 64), 0.5, 0.25, 2, "f64", "plain"), name="plain-pb208-64"),
        # a whole short run through the one-call slot: upload, first field solve, steps, download
        dict(_run("208Pb", 500, (64, 64, 64), 0.5, 0.25, 20), kind="simulate", name="simulate-pb208-64"),
        # a parameter scan: sixteen nuclei of mixed sizes on one GPU
        {"kind": "batch", "instances": 16, "mix": 3, "cap": 8, "steps": 4, "name": "batch-16"},
        # the gradient of a D(t) objective, solved tightly enough to be compared with differences
        {"kind": "adjoint", "nucleus": "40Ca", "ppn": 100, "nx": 32, "ny": 32, "nz": 32, "h": 1.0, "dt": 0.5,
         "steps": 20, "every": 10, "tol": 1e-12, "name": "adjoint-ca40-32"},
        # the initialisation's pair sums in both precisions
        {"kind": "densities", "nucleus": "208Pb", "ppn": 500, "precision": "f64", "name": "densities-pb208-f64"},
        {"kind": "densities", "nucleus": "208Pb", "ppn": 2000, "precision": "f32", "name": "densities-pb208-f32"},
    ]
    return cases


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _box(rng, nucleus, lo, hi):
    """Grid extents (odd ones among them) and the spacing of a box around the nucleus."""
    radius = 1.2 * sum(NUCLEI[nucleus]) ** (1.0 / 3.0)
    n0 = _log(rng, lo, hi)
    if rng.random() < 0.35:
        g = min(hi, max(lo, 8 * round(n0 / 8)))
        n = (g, g, g)
    else:
        n = tuple(min(hi, max(lo, round(n0 * rng.uniform(0.85, 1.15)))) for _ in range(3))
    return n, round(2.0 * (radius + rng.uniform(4.5, 7.0)) / min(n), 4)


def draw(rng):
    kind = rng.choice(("run", "run", "run", "sorted", "plain", "simulate", "batch", "adjoint", "densities"))
    nucleus = rng.choice(sorted(NUCLEI))
    if kind == "batch":
        return {"kind": "batch", "instances": rng.randint(4, 24), "mix": rng.randrange(1 << 20),
                "cap": rng.choice((4, 8, 16)), "steps": rng.randint(2, 5)}
    if kind == "densities":
        return {"kind": "densities", "nucleus": nucleus, "ppn": round(_log(rng, 50, 2000)),
                "precision": rng.choice(("f32", "f64"))}
    if kind == "adjoint":
        n, h = _box(rng, nucleus, 24, 48)
        return {"kind": "adjoint", "nucleus": nucleus, "ppn": 2 * round(_log(rng, 25, 200)), "nx": n[0], "ny": n[1],
                "nz": n[2], "h": h, "dt": round(0.2 + 0.3 * min(h, 1.0), 3), "steps": rng.randint(6, 14),
                "every": rng.randint(3, 10), "tol": 1e-12}
    n, h = _box(rng, nucleus, 24, 64 if kind == "plain" else 128)
    ppn = round(_log(rng, 100, 1000 if kind in ("plain", "simulate") else 10000))
    dt = round(0.2 + 0.3 * min(h, 1.0), 3)
    if kind == "plain":
        return _run(nucleus, ppn, n, h, dt, rng.randint(1, 3), "f64", "plain")
    case = _run(nucleus, ppn, n, h, dt, rng.randint(4, 12), deposit="sorted" if kind == "sorted" else "atomic")
    return dict(case, kind="simulate") if kind == "simulate" else case


# ---- inputs -----------------------------------------------------------------

def _particles(z, n, ppn, seed, dtype):
    """x, y, z, kx, ky, kz: positions uniform in the ball of 1.2 A^(1/3) fm,
    wavenumbers uniform in the Fermi ball, protons first."""
    rng = np.random.default_rng(seed)
    total = (z + n) * ppn

    def ball(radius):
        v = rng.standard_normal((3, total))
        v *= radius * rng.random(total) ** (1.0 / 3.0) / np.sqrt((v * v).sum(0))
        return v

    return [np.ascontiguousarray(a, dtype=dtype)
            for a in (*ball(1.2 * (z + n) ** (1.0 / 3.0)), *ball(K_FERMI))]


def _dtype(case):
    return np.float64 if case.get("precision", "f64") == "f64" else np.float32


@dataclasses.dataclass
class _Box(hv.Workload):
    """A workload on a box of three different axes."""

    axes: tuple = (32, 32, 32)

    def world(self):
        w = lib.hv_world()
        for a in range(3):
            w.n[a] = self.axes[a]
            w.d_max[a] = 0.5 * self.axes[a] * self.h
        return w


def _workload(case):
    z, n = NUCLEI[case["nucleus"]]
    axes = (case.get("nx", 32), case.get("ny", 32), case.get("nz", 32))
    return _Box(case["nucleus"], Z=z, N=n, ppn=case["ppn"], n=axes[0], h=case.get("h", 1.0), dt=case.get("dt", 0.5),
                steps=case.get("steps", 1), sor_tol=case.get("tol", 1e-6), axes=axes,
                deposit_mode=hv.HV_DEPOSIT_SORTED if case.get("deposit") == "sorted" else hv.HV_DEPOSIT_ATOMIC)


class _Device:
    """A field of a session as torch sees it: the session's own buffer, which
    lives as long as the session, so the session is held here (and a tensor
    holds the object it was made from)."""

    def __init__(self, session, field):
        self.session = session
        p = ctypes.c_void_p()
        lib.check(session.lib.hv_field_device_ptr(session.handle, field, ctypes.byref(p)), "hv_field_device_ptr")
        n = session.G if field == lib.HV_FIELD_COULOMB else 2 * session.G
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": session.dtype.newbyteorder("<").str,
                                         "data": (p.value, False), "version": 3, "strides": None}


def _fields(session, names=tuple(FIELDS)):
    return {k: torch.as_tensor(_Device(session, FIELDS[k]), device="cuda") for k in names}


def _rows(obs, dtype):
    """The observable rows in the run's own precision."""
    return np.stack([obs[k] for k in ("t", "rms_p", "rms_n", "zcm_p", "zcm_n", "dipole")], axis=-1).astype(dtype)


def _batch_workloads(case):
    return hv.workloads.batch_workloads(case["instances"], seed=case["mix"], steps=case["steps"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sessions = []
        for i, w in enumerate(_batch_workloads(case)):
            s = hv.Session.from_workload(w, hv.HV_F32)
            s.upload_particles(*_particles(w.Z, w.N, w.ppn, (seed, i), np.float32))
            sessions.append(s)
        b = Batch(sessions)
        b.plan(case["cap"])  # few blocks per solve, so that several solves share a launch
        return {"kind": kind, "sessions": sessions, "batch": b, "steps": case["steps"],
                "fields": [_fields(s, ("density", "coulomb")) for s in sessions]}
    z, n = NUCLEI[case["nucleus"]]
    parts = _particles(z, n, case["ppn"], seed, _dtype(case))
    if kind == "adjoint":
        w = _workload(case)
        w.deposit_mode = hv.HV_DEPOSIT_SORTED  # the reproducible mode: gradients repeat
        run_ = AdjointRun(w, parts, case["steps"], case["every"], path=hv.HV_PATH_FUSED)
        t = torch.arange(case["steps"], dtype=torch.float64) * case["dt"]
        return {"kind": kind, "run": run_, "wave": torch.cos(15.0 / HBAR_C * t), "theta": torch.tensor(THETA, dtype=torch.float64)}
    if kind == "simulate":
        # pinned host buffers, advanced in place by the call; the start is kept
        # so that every pass simulates the same nucleus
        own = [torch.empty(p.shape, dtype=torch.float32, pin_memory=True).numpy() for p in parts]
        return {"kind": kind, "w": _workload(case), "start": parts, "own": own, "steps": case["steps"]}
    w = _workload(case)
    precision = hv.HV_F64 if case["precision"] == "f64" else hv.HV_F32
    s = hv.Session.from_workload(w, precision)
    s.upload_particles(*parts)
    if kind == "densities":
        return {"kind": kind, "session": s}
    path = hv.HV_PATH_PLAIN if case["path"] == "plain" else hv.HV_PATH_FUSED
    s.run(0, path)  # the fields of the initial positions
    return {"kind": kind, "session": s, "path": path, "steps": case["steps"], "fields": _fields(s)}


# ---- one pass ---------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "run":
        s = state["session"]
        return {"rows": _rows(s.run(state["steps"], state["path"]), s.dtype), **state["fields"]}
    if kind == "simulate":
        for dst, src in zip(state["own"], state["start"]):
            np.copyto(dst, src)
        obs = hv.simulate(state["w"], *state["own"], state["steps"], hv.HV_F32, hv.HV_PATH_FUSED)
        return {"rows": _rows(obs, np.float32), "particles": list(state["own"])}
    if kind == "batch":
        obs = state["batch"].run(state["steps"])
        return {"rows": _rows(obs, np.float32), "fields": state["fields"]}
    if kind == "adjoint":
        theta = state["theta"].clone().requires_grad_(True)
        d = dipole_series(theta, state["run"])
        (d * state["wave"]).sum().backward()
        return {"dipole": d.detach(), "gradient": theta.grad}
    return dict(zip(("density_p", "density_n"), state["session"].particle_densities()))


def work(case):
    """Per step: the particle state read and written once, and each node's
    density, potentials and forces written and read once; the smoothing,
    potential and field solve as a few operations a node."""
    if case["kind"] == "densities":
        z, n = NUCLEI[case["nucleus"]]
        total, b = (z + n) * case["ppn"], np.dtype(_dtype(case)).itemsize
        # partners within 4 sigma_r of a uniform ball, ten operations a pair
        share = min(1.0, (4.0 * SIGMA_R / (1.2 * (z + n) ** (1.0 / 3.0))) ** 3)
        return {"bytes": 5.0 * total * b, "flops": 10.0 * total * total * share}
    if case["kind"] == "batch":
        ws = _batch_workloads(case)
        particles, nodes, b, steps = sum(w.particles for w in ws), sum(w.G for w in ws), 4, case["steps"]
    else:
        z, n = NUCLEI[case["nucleus"]]
        particles, nodes = (z + n) * case["ppn"], case["nx"] * case["ny"] * case["nz"]
        b, steps = np.dtype(_dtype(case) if case["kind"] == "run" else np.float64 if case["kind"] == "adjoint"
                            else np.float32).itemsize, case["steps"] * (3 if case["kind"] == "adjoint" else 1)
    return {"bytes": float(steps * b * (12 * particles + 2 * 11 * nodes)),
            "flops": float(steps * (200 * particles + 150 * nodes))}


# ---- the same in 64 bits with plain torch ------------------------------------

class _Step:
    """The time step in double on torch tensors (differentiable in theta)."""

    def __init__(self, z, n, ppn, axes, h, dt, eta, theta):
        self.z, self.n, self.ppn, self.axes, self.h, self.dt, self.eta = z, n, ppn, axes, h, dt, eta
        self.theta = theta
        self.protons = z * ppn
        dev = dict(dtype=torch.float64, device="cuda")
        self.dev = dev
        pos = [0.5 * m * h * (2.0 * torch.arange(m, **dev) / m - 1.0) for m in axes]
        # smoothing: all node pairs within 4 sigma_r, as a zero-padded convolution
        lim = [min(int(4.0 * SIGMA_R / h) + 2, m - 1) for m in axes]
        self.pad = [m + q for m, q in zip(axes, lim)]
        off = [torch.arange(-q, q + 1, **dev) * h for q in lim]
        d2 = off[0][:, None, None] ** 2 + off[1][None, :, None] ** 2 + off[2][None, None, :] ** 2
        w = torch.where(d2 <= 16.0 * SIGMA_R ** 2, torch.exp(-d2 / (2.0 * SIGMA_R ** 2)), torch.zeros_like(d2))
        kernel = torch.zeros(self.pad, **dev)
        ix = [torch.remainder(torch.arange(-q, q + 1, device="cuda"), p) for q, p in zip(lim, self.pad)]
        kernel[ix[0][:, None, None], ix[1][None, :, None], ix[2][None, None, :]] = w
        self.kernel = torch.fft.rfftn(kernel)
        self.term = 1.0 / (ppn * (2.0 * math.pi * SIGMA_R ** 2) ** 1.5)
        # Coulomb: the monopole on the faces, the interior by sine transforms
        r = torch.sqrt(pos[0][:, None, None] ** 2 + pos[1][None, :, None] ** 2 + pos[2][None, None, :] ** 2)
        face = torch.ones(axes, dtype=torch.bool, device="cuda")
        face[1:-1, 1:-1, 1:-1] = False
        self.phi_face = torch.where(face, E2 * z / r.clamp(min=1e-300), torch.zeros_like(r))
        self.sines, lam = [], []
        for m in axes:
            k = torch.arange(1, m - 1, **dev)
            self.sines.append(torch.sin(math.pi * k[:, None] * k[None, :] / (m - 1)) * math.sqrt(2.0 / (m - 1)))
            lam.append((2.0 - 2.0 * torch.cos(math.pi * k / (m - 1))) / h ** 2)
        self.lam = lam[0][:, None, None] + lam[1][None, :, None] + lam[2][None, None, :]

    def corners(self, x):
        """(inside, nodes [8, N], weights [8, N]) of each particle's cell."""
        c = [0.5 * m * (q / (0.5 * m * self.h) + 1.0) for m, q in zip(self.axes, x)]
        inside = torch.ones_like(c[0], dtype=torch.bool)
        for m, q in zip(self.axes, c):
            inside &= (q >= 0) & (q < m)
        base = [torch.clamp(q.detach().floor().long(), 0, m - 1) for m, q in zip(self.axes, c)]
        frac = [q - b for q, b in zip(c, base)]
        nodes, weights = [], []
        for corner in range(8):
            bits = [(corner >> a) & 1 for a in range(3)]
            w, ok, at = 1.0, inside, 0
            for a in range(3):
                w = w * (frac[a] if bits[a] else 1.0 - frac[a])
                i = base[a] + bits[a]
                ok = ok & (i < self.axes[a])
                at = at * self.axes[a] + torch.clamp(i, max=self.axes[a] - 1)
            nodes.append(at)
            weights.append(torch.where(ok, w, torch.zeros_like(w)))
        return nodes, weights

    def sine_transform(self, f):
        """The orthonormal sine transform along the three axes, its own inverse."""
        for a in range(3):
            f = torch.movedim(torch.tensordot(self.sines[a], f, dims=([1], [a])), 0, a)
        return f

    def fields(self, x):
        """(density, potential with Coulomb merged, phi, forces, corners) of the positions."""
        nodes, weights = self.corners(x)
        G = self.axes[0] * self.axes[1] * self.axes[2]
        shift = torch.zeros(x[0].shape, dtype=torch.long, device="cuda")
        shift[self.protons:] = G
        raw = torch.zeros(2 * G, **self.dev)
        for at, w in zip(nodes, weights):
            raw = raw.index_add(0, at + shift, w)
        raw = raw.reshape(2, *self.axes)
        full = torch.fft.irfftn(torch.fft.rfftn(raw, s=self.pad, dim=(1, 2, 3)) * self.kernel, s=self.pad,
                                dim=(1, 2, 3))
        rho = torch.clamp(full[:, :self.axes[0], :self.axes[1], :self.axes[2]] * self.term, min=0.0)
        t0, t3, sigma, a_sym = self.theta
        t = (rho[0] + rho[1]) / RHO0
        a, b = 0.75 * t0 * RHO0, (sigma + 2.0) / 16.0 * t3 * RHO0 ** (sigma + 1.0)
        mean, iso = a * t + b * t ** (sigma + 1.0), 2.0 * a_sym * (rho[1] - rho[0]) / RHO0
        # lap phi = -4 pi e^2 rho_p with the face values moved to the right-hand side
        f = self.phi_face
        rhs = (4.0 * math.pi * E2 * rho[0] + (torch.roll(f, 1, 0) + torch.roll(f, -1, 0) + torch.roll(f, 1, 1)
               + torch.roll(f, -1, 1) + torch.roll(f, 1, 2) + torch.roll(f, -1, 2)) / self.h ** 2)[1:-1, 1:-1, 1:-1]
        inner = self.sine_transform(self.sine_transform(rhs) / self.lam)
        phi = f + torch.nn.functional.pad(inner, (1, 1, 1, 1, 1, 1))
        U = torch.stack([mean - iso + phi, mean + iso])
        force = []
        for axis in range(1, 4):
            m = self.axes[axis - 1]
            lo, hi = U.narrow(axis, 0, m - 2), U.narrow(axis, 2, m - 2)
            first = (U.narrow(axis, 1, 1) - U.narrow(axis, 0, 1)) / self.h
            last = (U.narrow(axis, m - 1, 1) - U.narrow(axis, m - 2, 1)) / self.h
            force.append(-torch.cat([first, (hi - lo) / (2.0 * self.h), last], axis))
        f = []
        for q in force:
            flat = q.reshape(-1)
            f.append(sum(w * flat[at + shift] for at, w in zip(nodes, weights)))
        return rho, U, phi, force, f

    def row(self, x, t):
        p = self.protons
        inside = torch.ones_like(x[0], dtype=torch.bool)
        r2 = 0.0
        for m, q in zip(self.axes, x):
            inside &= (q >= -0.5 * m * self.h) & (q <= 0.5 * m * self.h)
            r2 = r2 + q * q
        rms = [torch.sqrt((r2[s] * inside[s]).sum() / inside[s].sum()) for s in (slice(0, p), slice(p, None))]
        zp, zn = x[2][:p].mean(), x[2][p:].mean()
        d = self.n * self.z / (self.n + self.z) * (zp - zn)
        return torch.stack([torch.full_like(d, t), rms[0], rms[1], zp, zn, d])

    def advance(self, parts, steps):
        """(rows, x, k, fields) after the first field solve and `steps` steps."""
        x, k = [torch.as_tensor(np.asarray(p, np.float64), device="cuda") for p in parts[:3]], [
            torch.as_tensor(np.asarray(p, np.float64), device="cuda") for p in parts[3:]]
        out = self.fields(x)
        rows, kick, drift = [], self.dt / (2.0 * HBAR_C), self.dt * HBAR_C / MC2
        boost = torch.full_like(k[2], -self.eta * self.z / (self.z + self.n))
        boost[:self.protons] = self.eta * self.n / (self.z + self.n)
        for i in range(steps):
            rows.append(self.row(x, i * self.dt))
            if i == 0:
                k = [k[0], k[1], k[2] + boost]
            k = [a + kick * f for a, f in zip(k, out[4])]
            x = [a + drift * b for a, b in zip(x, k)]
            out = self.fields(x)
            k = [a + kick * f for a, f in zip(k, out[4])]
        return torch.stack(rows), x, k, out


def _pair_densities(parts, z, n, ppn):
    pos = torch.as_tensor(np.stack(parts[:3], 1).astype(np.float64), device="cuda")
    p, total = z * ppn, pos.shape[0]
    term = 1.0 / (ppn * (2.0 * math.pi * SIGMA_R ** 2) ** 1.5)
    out = torch.zeros(2, total, dtype=torch.float64, device="cuda")
    step = max(1, int(4.0e8 / total))
    for a in range(0, total, step):
        me = pos[a:a + step]
        d2 = sum((me[:, c, None] - pos[None, :, c]).square_() for c in range(3))
        w = torch.where(d2 <= 16.0 * SIGMA_R ** 2, torch.exp(-d2 / (2.0 * SIGMA_R ** 2)), 0.0)
        out[0, a:a + step] = w[:, :p].sum(1) * term
        out[1, a:a + step] = w[:, p:].sum(1) * term
    return out


def _numpy(t):
    return t.detach().reshape(-1).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    eta = 30.0 / HBAR_C
    if kind == "batch":
        rows, fields = [], []
        for i, w in enumerate(_batch_workloads(case)):
            parts = _particles(w.Z, w.N, w.ppn, (seed, i), np.float32)
            s = _Step(w.Z, w.N, w.ppn, (w.n,) * 3, w.h, w.dt, w.boost_mev / HBAR_C, (w.t0, w.t3, w.sigma, w.a_sym))
            r, _, _, out = s.advance(parts, case["steps"])
            rows.append(r.cpu().numpy())
            fields.append({"density": _numpy(out[0]), "coulomb": _numpy(out[2])})
        return {"rows": np.stack(rows), "fields": fields}
    z, n = NUCLEI[case["nucleus"]]
    parts = _particles(z, n, case["ppn"], seed, _dtype(case))
    if kind == "densities":
        if float(parts[0].size) ** 2 > PAIR_LIMIT:
            return None
        return dict(zip(("density_p", "density_n"), _pair_densities(parts, z, n, case["ppn"]).cpu().numpy()))
    axes = (case["nx"], case["ny"], case["nz"])
    if kind == "adjoint":
        theta = torch.tensor(THETA, dtype=torch.float64, device="cuda", requires_grad=True)
        s = _Step(z, n, case["ppn"], axes, case["h"], case["dt"], eta, theta)
        d = s.advance(parts, case["steps"])[0][:, 5]
        t = torch.arange(case["steps"], dtype=torch.float64, device="cuda") * case["dt"]
        (d * torch.cos(15.0 / HBAR_C * t)).sum().backward()
        return {"dipole": _numpy(d), "gradient": _numpy(theta.grad)}
    s = _Step(z, n, case["ppn"], axes, case["h"], case["dt"], eta, THETA)
    rows, x, k, (rho, U, phi, force, _) = s.advance(parts, case["steps"])
    if kind == "simulate":
        return {"rows": rows.cpu().numpy(), "particles": [_numpy(q) for q in (*x, *k)]}
    return {"rows": rows.cpu().numpy(), "density": _numpy(rho), "potential": _numpy(U), "coulomb": _numpy(phi),
            **{"force_" + c: _numpy(f) for c, f in zip("xyz", force)}}
