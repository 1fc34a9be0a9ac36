"""What the performance of this framework is measured on: RK3 steps of single simulations, batches of an
ensemble, and the statistics of a state, over the sizes, flows, precisions and particle counts that its
workloads, tests and benchmark use.

A case of kind "step" is a time loop over one resident simulation, "batch" the same over the members of one
batch class (the device side of the ensemble server), "stats" the statistics of a state beyond a step's own.
``exact`` repeats a case with plain torch in 64 bits, from the seeds: the seeded field, the forcing's random
numbers, the transforms (torch.fft), the products, the updates and the tracers' interpolation.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "pandora-2.0_b200"))

import pandora  # noqa: E402

LENGTHS = (24, 32, 40, 48, 56, 64, 80, 96, 112, 128, 160, 192, 224, 256, 320, 384, 448, 512)
BATCH_LENGTHS = (32, 48, 64, 96, 128, 192, 256)


def _step(name, flow, n, precision="fp64", steps=1, np_=0, order=4, dia=0.0, decide=False, form="bf-rot", particles=False):
    c = {"kind": "step", "flow": flow, "nx": n[0], "ny": n[1], "nz": n[2], "precision": precision, "steps": steps,
         "np": np_, "order": order, "dia": dia, "decide": decide, "form": form, "particles": particles}
    return dict(c, name=name) if name else c


def _batch(name, flow, n, members, precision="fp64", steps=20, np_=0):
    c = {"kind": "batch", "flow": flow, "nx": n, "ny": n, "nz": n, "members": members, "precision": precision,
         "steps": steps, "np": np_}
    return dict(c, name=name) if name else c


def _stats(name, flow, n, precision="fp64"):
    c = {"kind": "stats", "flow": flow, "nx": n[0], "ny": n[1], "nz": n[2], "precision": precision}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one synchronous step of the smallest grid and its statistics: a driver that looks at every step
        _step("decay_32_step", "decay", (32, 32, 32)),
        # the 64^3 decaying flow of the first workload, run without a look in between
        _step("decay_64_loop", "decay", (64, 64, 64), steps=20),
        # a ragged box (lengths with factors 5, 3 and 7), CFL-driven step, heavy particles of order 6, whose
        # positions are written out after some steps
        _step("forced_160x96x112_inertial", "forced", (160, 96, 112), steps=10, np_=32768, order=6, dia=0.01514314,
              decide=True, particles=True),
        # the convective Rogallo form, nine gradients through the transforms
        _step("shear_192_rconv", "shear", (192, 192, 192), form="r-conv"),
        # forced turbulence with 2^20 tracers, in both precisions
        _step("forced_256_tracers", "forced", (256, 256, 256), np_=1 << 20),
        _step("forced_256_tracers_mixed", "forced", (256, 256, 256), "fp32_mixed", np_=1 << 20),
        # the benchmark's default workload, in both precisions
        _step("shear_512_tracers", "shear", (512, 512, 512), np_=1 << 18),
        _step("shear_512_tracers_mixed", "shear", (512, 512, 512), "fp32_mixed", np_=1 << 18),
        # the largest grid
        _step("forced_1024_mixed", "forced", (1024, 1024, 1024), "fp32_mixed"),
        # members of the ensemble's smallest class, and of one of its larger ones, with tracers
        _batch("ensemble_32_decay", "decay", 32, 32, steps=40),
        _batch("ensemble_128_shear_mixed", "shear", 128, 4, "fp32_mixed", steps=30, np_=1 << 14),
        # moments and correlations of a state, as written every so many steps
        _stats("stats_256_forced", "forced", (256, 256, 256)),
    ]


def draw(rng):
    def near(values, x):
        return min(values, key=lambda v: abs(math.log(v / x)))

    kind = rng.choice(["step"] * 7 + ["batch"] * 2 + ["stats"])
    precision = rng.choice(["fp64", "fp64", "fp32_mixed"])
    flow = rng.choice(["decay", "forced", "shear", "shear"])
    if kind == "batch":
        n = rng.choice(BATCH_LENGTHS)
        members = max(1, min(40, int((192 ** 3 / n ** 3) * 2 ** rng.uniform(-2.0, 1.0))))
        steps = int(8.0e7 / (members * n ** 3) * rng.uniform(0.5, 1.0))
        return _batch(None, flow if flow != "forced" else "decay", n, members, precision,
                      max(4, min(40, steps)) + rng.randint(0, 5), rng.choice([0, 1 << 14, int(2.0 ** rng.uniform(8.0, 15.0))]))
    while True:
        base = 24.0 * (448.0 / 24.0) ** rng.random()
        n = tuple(near(LENGTHS, base * 2 ** rng.uniform(-0.8, 0.8)) for _ in range(3))
        points = n[0] * n[1] * n[2]
        if points <= 70e6:
            break
    if kind == "stats":
        return _stats(None, flow, n, precision)
    np_ = 0
    if rng.random() < 0.5:
        np_ = int(min(1 << 20, points / 8) ** rng.uniform(0.5, 1.0)) + 1
    dia = 0.01514314 if np_ and rng.random() < 0.25 else 0.0
    return _step(None, flow, n, precision, max(1, min(20, int(2.0e7 / points))), np_, rng.choice([2, 4, 4, 4, 5, 6]), dia,
                 flow != "shear" and rng.random() < 0.3, rng.choice(["bf-rot", "bf-rot", "r-rot", "r-conv"]) if flow == "shear" else "bf-rot",
                 bool(np_ and np_ <= 1 << 16))


# ---- the workloads' parameters ----
def _params(case, seed, member=0):
    base = {"decay": "iso_decay", "forced": "iso_forced_particles", "shear": "shear"}[case["flow"]]
    p = pandora.workload_params(base, case["nx"])
    p.nodes_x, p.nodes_y, p.nodes_z = case["nx"], case["ny"], case["nz"]
    if case["flow"] == "forced" and case["nx"] >= 1024:
        p.f_nu, p.rk3_dt = 0.0008, 0.001
    if case["flow"] == "decay":   # a stable step on the finer grids too
        p.rk3_dt = min(p.rk3_dt, 0.5 / max(case["nx"], case["ny"], case["nz"]))
    if case["kind"] == "batch":
        p.f_nu = 0.01 * (64.0 / case["nx"])
    p.precision = pandora.PREC_FP32_MIXED if case["precision"] == "fp32_mixed" else pandora.PREC_FP64
    np_ = case.get("np", 0)
    p.p_track_part, p.p_np_global = (1, np_) if np_ else (0, 0)
    p.p_interp_order, p.p_dia_vals = case.get("order", 4), case.get("dia", 0.0)
    if case.get("decide"):
        p.rk3_timestep = pandora.RK3_TIMESTEP_DECIDE
    p.ns_deformed = {"bf-rot": pandora.NS_BF_ROT, "r-rot": pandora.NS_R_ROT, "r-conv": pandora.NS_R_CONV}[case.get("form", "bf-rot")]
    s = seed * 64 + member
    p.seed_fluid, p.seed_force, p.seed_particles = 3 * s + 1, 3 * s + 2, 3 * s + 3
    return p


class _Buffer:
    """A device buffer of the library, for torch (no copy)."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


class _State:
    """What a program keeps; the library frees a simulation when its last view is gone."""

    def __init__(self, case, owner):
        self.case, self.owner = case, owner


def prepare(case, seed):
    if case["kind"] == "batch":
        b = pandora.Batch(_params(case, seed), case["members"])
        st = _State(case, b)
        st.slots = [b.admit(_params(case, seed, m)) for m in range(case["members"])]
        return st
    p = _params(case, seed)
    sim = pandora.Simulation(p)
    st = _State(case, sim)
    sim.init_fluid()
    if p.p_track_part:
        sim.init_particles()
    typestr = "<f4" if case["precision"] == "fp32_mixed" else "<f8"
    st.u = [torch.as_tensor(_Buffer(sim, a, sim.shape + (2,), typestr), device="cuda") for a in sim.device_state_ptrs()]
    return st


def _looked_at(case):
    """Members of a batch whose state is read back: copies to the host of about 5 MB, one member at least."""
    modes = (case["nx"] // 3 + 1) * (2 * (case["ny"] // 3) + 1) * (2 * (case["nz"] // 3) + 1)
    return max(1, min(case["members"], int(5e6 / (48 * modes + 104 * case["np"]))))


def _grouped(m):
    """The moments by their size, so that no large one hides the others."""
    groups = {"second": ("u1u1", "u2u2", "u3u3", "u1u2", "u1u3", "u2u3", "ucfl"), "rmsvort1": ("rmsvort1",),
              "vorticity": ("rmsvort2", "rmsvort3", "omegamax1", "omegamax2", "omegamax3", "lint11"),
              "shape": ("skew1", "skew2", "skew3", "flat1", "flat2", "flat3"),
              "shape_vorticity": ("skewvort2", "skewvort3", "flatvort2", "flatvort3")}
    return {g: np.array([m[k] for k in names]) for g, names in groups.items()}


def run(state):
    case = state.case
    if case["kind"] == "batch":
        b = state.owner
        b.step(case["steps"])
        out = {"stats": [], "u": []}
        for k, s in enumerate(state.slots):
            ek, tke, eps = b.last_step_stats(s)
            out["stats"].append(np.concatenate([ek, [tke, eps]]))
        out["stats"] = np.stack(out["stats"])
        # what the server hands back is the members' statistics; the state of those that are looked at as well
        out["u"] = np.stack([np.stack(b.get_state(s)) for s in state.slots[: _looked_at(case)]])
        if case["np"]:
            out["x"] = np.stack([b.get_particles(s)[0] for s in state.slots[: _looked_at(case)]])
        return out
    sim = state.owner
    if case["kind"] == "stats":
        ek, tke, eps, _ = sim.stats()
        r = sim.realspace_stats(corr=True)
        return dict(_grouped(r), ek=ek, tke=np.array([tke, eps]), r1i=r["r1i"])
    if case["steps"] == 1:
        sim.step()
    else:
        sim.advance(case["steps"])
    ek, tke, eps, ucfl = sim.stats(last_step=True)
    out = {"u": state.u, "ek": ek, "tke": np.array([tke, eps, ucfl])}
    if case["np"]:
        if case["particles"]:
            xp, up, _, _, _ = sim.get_particles()
            out["x"], out["v"] = xp, up
        else:   # the whole state stays on the device: the statistics that the particle code writes
            d = sim.particle_stats()
            out["particles"] = np.array([d[k] for k in ("u1u1", "u2u2", "u3u3", "u1u2", "u1u3", "u2u3", "tke")])
    return out


def work(case):
    """The state read and written once, with the particles' (positions and velocities); operations of the
    transforms at 2.5 N log2 N per real line and the products, per stage."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nki, nkj, nkk = nx // 3 + 1, 2 * (ny // 3) + 1, 2 * (nz // 3) + 1
    modes, points = nki * nkj * nkk, nx * ny * nz
    word = 8 if case["precision"] == "fp32_mixed" else 16
    inv = 9 if case.get("form") == "r-conv" else 6
    z = 5 * nz * math.log2(nz) * nki * nkj
    y = 5 * ny * math.log2(ny) * nki * nz
    x = 2.5 * nx * math.log2(nx) * ny * nz
    members, np_ = case.get("members", 1), case.get("np", 0)
    if case["kind"] == "stats":
        return {"bytes": 3 * modes * word, "flops": 6 * (x + y + z) + 60 * points}
    flops = 3 * (inv * (z + y) + (12 if inv == 9 else 6) * x + 3 * (x + y + z) + 12 * points + 80 * modes
                 + np_ * (6 * case.get("order", 4) ** 3 + 100))
    return {"bytes": members * (6 * modes * word + np_ * 8 * 12), "flops": case["steps"] * members * flops}


def tolerance(case):
    # about four times what the path is off from ``exact`` over a pass or two: 3e-16 to 1.5e-15 in 64 bits
    # (the statistics' sums), 5e-8 to 3e-7 in the mixed form (32-bit fields and transforms)
    return {"rel": 1.5e-6, "max": 6e-5} if case["precision"] == "fp32_mixed" else {"rel": 1e-14, "max": 4e-13}


# ---- the same in plain torch, 64 bits ----
_M = (1 << 64) - 1
_GOLDEN = 0x9E3779B97F4A7C15


def _mix64(z):
    if isinstance(z, np.ndarray):
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & _M
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _M
    return z ^ (z >> 31)


def _key(seed, tag):
    return _mix64((seed * _GOLDEN + tag * 0xD1B54A32D192ED03 + 0x632BE59BD9B4E019) & _M)


def _uniform(key, n):
    if isinstance(n, np.ndarray):
        return (_mix64(np.uint64(key) + (n + np.uint64(1)) * np.uint64(_GOLDEN)) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
    return (_mix64((key + (n + 1) * _GOLDEN) & _M) >> 11) * 2.0 ** -53


def _normal_pair(key, call):
    sub = _mix64((key + (call + 1) * _GOLDEN) & _M)
    for a in range(64):
        x, y = 2.0 * _uniform(sub, 2 * a) - 1.0, 2.0 * _uniform(sub, 2 * a + 1) - 1.0
        w = x * x + y * y
        if w < 1.0:
            w = math.sqrt(-2.0 * math.log(w) / w)
            return complex(x * w, y * w)
    return 0j


def _kvec(n, dev):
    a = torch.arange(n // 3 + 1, dtype=torch.float64, device=dev)
    b = torch.arange(2 * (n // 3) + 1, dtype=torch.float64, device=dev)
    return a, torch.where(b <= n // 3, b, b - b.numel())


class _Exact:
    """One simulation in plain torch: u[3] of shape (NKI, NKJ, NKK), complex128."""

    def __init__(self, p, dev):
        self.p, self.dev = p, dev
        self.n = (p.nodes_x, p.nodes_y, p.nodes_z)
        self.shear = p.f_type == pandora.params.F_SHEAR_DNS
        self.form = p.ns_deformed if self.shear else 0
        self.B = (p.b110, p.b220, p.b330) if self.shear else (1, 1, 1)
        self.S = p.f_deform_s if self.shear else 0.0
        self.k = (_kvec(self.n[0], dev)[0].view(-1, 1, 1), _kvec(self.n[1], dev)[1].view(1, -1, 1), _kvec(self.n[2], dev)[1].view(1, 1, -1))
        self.k2 = self.k[0] ** 2 + self.k[1] ** 2 + self.k[2] ** 2
        self.b13 = self.bi13 = 0.0
        self.t, self.t0, self.tstep, self.dt = 0.0, 0.0, 1, 0.0
        self.u = self._field()
        self.r = None
        self.nk = int(p.force_kf)
        self.f = np.zeros((3, self.nk + 1, 2 * self.nk + 1, 2 * self.nk + 1), complex)
        self.d = [2.0 * math.pi / m for m in self.n]
        if p.p_track_part:
            n = np.arange(p.p_np_global, dtype=np.uint64)
            key = _key(p.seed_particles, 3)
            x = np.stack([_uniform(key, n * np.uint64(3) + np.uint64(c)) * 2.0 * math.pi - self.d[c] * 0.5 for c in range(3)])
            self.x = torch.from_numpy(x).to(dev)
            self.v, self.rv, self.rx = (torch.zeros_like(self.x) for _ in range(3))

    # the seeded solenoidal field: three draws per mode, two triples per mode of the i = 0 plane
    def _mode(self, k, r, fdiv):
        p, tp = self.p, 2.0 * math.pi
        kmag = torch.sqrt(k[0] ** 2 + k[1] ** 2 + k[2] ** 2)
        k2d = k[0] ** 2 + k[1] ** 2
        ek = 16.0 * math.sqrt(2.0 / math.pi) * 1.5 * p.f_init_u0 * (kmag ** 4 / p.f_init_kp ** 5) * torch.exp(-2.0 * kmag ** 2 / p.f_init_kp ** 2)
        fac = torch.sqrt(ek / (4.0 * math.pi * kmag ** 2)) / fdiv
        a = fac * torch.cos(tp * r[2]) * torch.exp(1j * tp * r[0])
        b = fac * torch.sin(tp * r[2]) * torch.exp(1j * tp * r[1])
        den = kmag * torch.sqrt(k2d)
        t = [(a * kmag * k[1] + b * k[0] * k[2]) / den, (b * k[1] * k[2] - a * kmag * k[0]) / den, -(b * torch.sqrt(k2d)) / kmag]
        return [torch.where((k2d > 0) & (kmag > 0), c / self.B[i], torch.zeros_like(c)) for i, c in enumerate(t)]

    def _field(self):
        ki, kj, kk = (m // 3 for m in self.n)
        nkj, nkk = 2 * kj + 1, 2 * kk + 1
        key = _key(self.p.seed_fluid, 1)
        fdiv = math.sqrt(self.B[0] * self.B[1] * self.B[2])
        u = [torch.zeros(ki + 1, nkj, nkk, dtype=torch.complex128, device=self.dev) for _ in range(3)]
        to = lambda x: torch.from_numpy(x).to(self.dev)  # noqa: E731
        k1, k2, k3 = (self.k[c] / self.B[c] for c in range(3))
        n0 = (kj + 1) * 3 * nkk
        j, k = np.arange(nkj, dtype=np.uint64)[:, None], np.arange(nkk, dtype=np.uint64)[None, :]
        for i in range(1, ki + 1):
            n = np.uint64(n0) + np.uint64(3) * ((np.uint64(i - 1) * np.uint64(nkj + 1) + j) * np.uint64(nkk + 1) + k)
            t = self._mode((k1[i], k2[0], k3[0]), [to(_uniform(key, n + np.uint64(q))) for q in range(3)], fdiv)
            for c in range(3):
                u[c][i] = t[c]
        # the plane i = 0: j = 0..KJ, k = 0..KK, and their conjugates
        j, k = np.arange(kj + 1, dtype=np.uint64)[:, None], np.arange(kk + 1, dtype=np.uint64)[None, :]
        n = j * np.uint64(3 * nkk) + np.where(k == 0, np.uint64(0), np.uint64(3) + np.uint64(6) * (k - np.uint64(1)))
        jj = (nkj - np.arange(kj + 1)) % nkj
        kc = (nkk - np.arange(kk + 1)) % nkk
        zero = torch.zeros((), dtype=torch.float64, device=self.dev)
        kp = (zero, k2[0][: kj + 1], k3[0][:, : kk + 1])
        t = self._mode(kp, [to(_uniform(key, n + np.uint64(q))) for q in range(3)], fdiv)
        s = self._mode((zero, -k2[0][: kj + 1], k3[0][:, : kk + 1]), [to(_uniform(key, n + np.uint64(q))) for q in range(3, 6)], fdiv)
        for c in range(3):
            p = u[c][0]
            p[: kj + 1, : kk + 1] = t[c]
            p[jj[:, None], kc[None, :]] = t[c].conj()
            # the second triple, k != 0: (j', k) and the conjugate of it at (j, k')
            p[jj[:, None], np.arange(1, kk + 1)[None, :]] = s[c][:, 1:]
            p[np.arange(kj + 1)[:, None], kc[1:][None, :]] = s[c][:, 1:].conj()
        return u

    # transforms: spectral [i][j][k] <-> physical [z][y][x]
    def _phys(self, a):
        nx, ny, nz = self.n
        ki, kj, kk = nx // 3, ny // 3, nz // 3
        w = torch.zeros(nz, ny, nx // 2 + 1, dtype=torch.complex128, device=self.dev)
        a = a.permute(2, 1, 0)
        for zs, zd in ((slice(0, kk + 1), slice(0, kk + 1)), (slice(kk + 1, None), slice(nz - kk, None))):
            for ys, yd in ((slice(0, kj + 1), slice(0, kj + 1)), (slice(kj + 1, None), slice(ny - kj, None))):
                w[zd, yd, : ki + 1] = a[zs, ys]
        return torch.fft.irfftn(w, s=(nz, ny, nx), norm="forward")

    def _spec(self, r):
        nx, ny, nz = self.n
        ki, kj, kk = nx // 3, ny // 3, nz // 3
        w = torch.fft.rfftn(r, norm="forward")[:, :, : ki + 1]
        w = torch.cat([w[: kk + 1], w[nz - kk:]], 0)
        w = torch.cat([w[:, : kj + 1], w[:, ny - kj:]], 1)
        return w.permute(2, 1, 0).contiguous()

    def _frames(self):
        bm = np.diag([1.0 / b for b in self.B])
        bi = np.diag([float(b) for b in self.B])
        bm[0, 2], bi[0, 2] = self.b13, self.bi13
        return bm, bi

    def _klab(self):
        bm, _ = self._frames()
        return [self.k[0] * bm[0, 0], self.k[1] * bm[1, 1], self.k[2] * bm[2, 2] + self.k[0] * bm[0, 2]]

    def _vorticity(self):
        """The vorticity of the stored velocity (laboratory components)."""
        kl = self._klab()
        ul = self._ulab()
        return [1j * (kl[1] * ul[2] - kl[2] * ul[1]), 1j * (kl[2] * ul[0] - kl[0] * ul[2]), 1j * (kl[0] * ul[1] - kl[1] * ul[0])]

    def _ulab(self):
        if not self.shear or self.form != pandora.NS_BF_ROT:
            return self.u
        _, bi = self._frames()
        return [bi[0, 0] * self.u[0] + bi[0, 2] * self.u[2], bi[1, 1] * self.u[1], bi[2, 2] * self.u[2]]

    def _nonlinear(self):
        """The physical velocity and the nonlinear term (laboratory components) in wave space."""
        up = [self._phys(a) for a in self.u]
        if self.form == pandora.NS_R_CONV:
            bm, _ = self._frames()
            v = [bm[0, 0] * up[0] + bm[0, 2] * up[2], bm[1, 1] * up[1], bm[2, 2] * up[2]]
            nl = []
            for c in range(3):
                s = 0
                for d in range(3):
                    s = s + v[d] * self._phys(1j * self.k[d] * self.u[c])
                nl.append(self._spec(s))
            return up, nl
        ul = up
        if self.form == pandora.NS_BF_ROT:
            _, bi = self._frames()
            ul = [bi[0, 0] * up[0] + bi[0, 2] * up[2], bi[1, 1] * up[1], bi[2, 2] * up[2]]
        w = [self._phys(a) for a in self._vorticity()]
        return up, [self._spec(w[1] * ul[2] - w[2] * ul[1]), self._spec(w[2] * ul[0] - w[0] * ul[2]), self._spec(w[0] * ul[1] - w[1] * ul[0])]

    def _force(self, stage):
        """The Ornstein-Uhlenbeck forcing of this stage, projected, as a sparse list."""
        p, nk = self.p, self.nk
        fw = 2 * nk + 1
        calls = 3 * ((nk + 1) ** 2 + nk * (nk + 1)) + 3 * nk * fw * fw
        base = (self.tstep * 3 + stage - 1) * calls
        key = _key(p.seed_force, 2)
        r = [_normal_pair(key, base + c) for c in range(calls)]
        amp, decay = math.sqrt(2.0 * p.force_sigma ** 2 * self.dt / p.force_tf), 1.0 - self.dt / p.force_tf
        f, c = self.f, 0
        for jw in range(nk + 1):
            for kw in range(nk + 1):
                for a in ((jw, -jw) if jw else (jw,)):
                    for q in range(3):
                        f[q, 0, a + nk, kw + nk] = f[q, 0, a + nk, kw + nk] * decay + r[c + q] * amp
                        f[q, 0, -a + nk, -kw + nk] = f[q, 0, a + nk, kw + nk].conjugate()
                    c += 3
        for i in range(1, nk + 1):
            for a in range(fw):
                for b in range(fw):
                    for q in range(3):
                        f[q, i, a, b] = f[q, i, a, b] * decay + r[c + q] * amp
                    c += 3
        out = []
        for i in range(nk + 1):
            for jw in range(-nk, nk + 1):
                for kw in range(-nk, nk + 1):
                    k2 = float(i * i + jw * jw + kw * kw)
                    if 0.0 < math.sqrt(k2) <= p.force_kf:
                        v = f[:, i, jw + nk, kw + nk]
                        kd = i * v[0] + jw * v[1] + kw * v[2]
                        out.append((i, jw, kw, [v[q] - (i, jw, kw)[q] * kd / k2 for q in range(3)]))
        return out

    def _rhs(self, nl, stage):
        p = self.p
        if not self.shear:
            ik2 = torch.where(self.k2 > 0, 1.0 / self.k2.clamp(min=1.0), torch.zeros_like(self.k2))
            kd = self.k[0] * nl[0] + self.k[1] * nl[1] + self.k[2] * nl[2]
            tot = [-p.f_nu * self.k2 * self.u[c] - nl[c] + self.k[c] * ik2 * kd for c in range(3)]
            if self.tstep < p.force_stop:
                for i, j, k, v in self._force(stage):
                    for c in range(3):
                        tot[c][i, j, k] += v[c]
            return tot
        bm, bi = self._frames()
        kl = self._klab()
        p4 = kl[0] ** 2 + kl[1] ** 2 + kl[2] ** 2
        ip4 = torch.where(p4 > 0, 1.0 / torch.where(p4 > 0, p4, torch.ones_like(p4)), torch.zeros_like(p4))
        # the laboratory right-hand side; BF-rot carries twice the mean-shear source (its frame moves with it)
        ul = self._ulab()
        two = 2.0 if self.form == pandora.NS_BF_ROT else 1.0
        src = self.S * ul[2]
        div = kl[0] * nl[0] + kl[1] * nl[1] + kl[2] * nl[2] + kl[0] * two * src
        tot = [-p.f_nu * p4 * ul[c] - nl[c] + kl[c] * ip4 * div - (two * src if c == 0 else 0.0) for c in range(3)]
        if self.form == pandora.NS_BF_ROT:
            return [bm[0, 0] * tot[0] + bm[0, 2] * tot[2], bm[1, 1] * tot[1], bm[2, 2] * tot[2]]
        return tot

    def _fix(self):
        ik2 = torch.where(self.k2 > 0, 1.0 / self.k2.clamp(min=1.0), torch.zeros_like(self.k2))
        u = self.u
        bm, bi = self._frames()
        moving = self.shear and self.form != pandora.NS_BF_ROT
        if moving:
            u = [bm[0, 0] * u[0] + bm[0, 2] * u[2], bm[1, 1] * u[1], bm[2, 2] * u[2]]
        kd = (self.k[0] * u[0] + self.k[1] * u[1] + self.k[2] * u[2]) * ik2
        u = [u[c] - self.k[c] * kd for c in range(3)]
        if moving:
            u = [bi[0, 0] * u[0] + bi[0, 2] * u[2], bi[1, 1] * u[1], bi[2, 2] * u[2]]
        self.u = u

    def _interpolate(self, up):
        order, w, at = self.p.p_interp_order, [], []
        for c in range(3):
            d, nh = self.d[c], order // 2
            if order % 2 == 0:
                x = self.x[c] + (nh * d - 0.5 * d) + d + 0.5 * d
            else:
                x = self.x[c] + nh * d + 0.5 * d
            i0 = torch.trunc(x / d).long() - nh - nh
            node = [(i0 + m).double() * d for m in range(order)]
            w.append([math.prod([(self.x[c] - node[q]) / (node[m] - node[q]) for q in range(order) if q != m], start=torch.ones_like(x)) for m in range(order)])
            at.append([torch.remainder(i0 + m, self.n[c]) for m in range(order)])
        out = [torch.zeros_like(self.x[0]) for _ in range(3)]
        for a in range(order):
            for b in range(order):
                for e in range(order):
                    ww = w[2][a] * w[1][b] * w[0][e]
                    for c in range(3):
                        out[c] += ww * up[c][at[2][a], at[1][b], at[0][e]]
        return torch.stack(out)

    def _particles(self, up, stage, beta, gamma):
        p = self.p
        if self.tstep < p.p_ts_release:
            return
        uf = self._interpolate(up)
        x = self.x
        bfrot = self.shear and self.form == pandora.NS_BF_ROT
        bm, bi = self._frames()
        if bfrot:
            lab = lambda a: torch.stack([bi[0, 0] * a[0] + bi[0, 2] * a[2], bi[1, 1] * a[1], bi[2, 2] * a[2]])  # noqa: E731
            x, uf = lab(x), lab(uf)
        if self.tstep == p.p_ts_release and stage == 1:
            self.v, self.rv, self.rx = uf.clone(), torch.zeros_like(uf), torch.zeros_like(uf)
        if p.p_dia_vals > 0.0:
            tau = p.p_dia_vals ** 2 / (18.0 * p.f_nu) * (p.p_rho / p.f_rho)
            acc = (uf - self.v) / tau
            if bfrot:
                acc[0] -= self.S * self.v[2]
            self.rv = beta * self.rv + acc
            self.v = self.v + gamma * self.dt * self.rv
        else:
            self.v = uf
        self.rx = beta * self.rx + self.v
        x = x + gamma * self.dt * self.rx
        if bfrot:
            x = torch.stack([bm[0, 0] * x[0] + bm[0, 2] * x[2], bm[1, 1] * x[1], bm[2, 2] * x[2]])
        for c in range(3):
            lo, ln = -0.5 * self.d[c], 2.0 * math.pi
            y = torch.where(x[c] < lo, x[c] + ln, x[c])
            x[c] = torch.where(y >= lo + ln, y - ln, y)
        self.x = x

    def stats(self):
        """E(k), (tke, eps) of the state."""
        p = self.p
        ki, kj, kk = (m // 3 for m in self.n)
        B = self.B
        K = round(math.sqrt((ki / B[0]) ** 2 + (kj / B[1]) ** 2 + (kk / B[2]) ** 2))
        kl, ul = self._klab(), self._ulab()
        km = torch.sqrt(kl[0] ** 2 + kl[1] ** 2 + kl[2] ** 2)
        wgt = torch.full_like(km, 2.0)
        wgt[0] = 1.0
        e = 0.5 * wgt * sum(a.real ** 2 + a.imag ** 2 for a in ul)
        q = torch.floor(km + 0.5).long().clamp(0, K + 1).reshape(-1)
        se = torch.bincount(q, e.reshape(-1), K + 2)[1: K + 1].cpu().numpy()
        sd = torch.bincount(q, (2.0 * km * km * p.f_nu * e).reshape(-1), K + 2)[1: K + 1].cpu().numpy()
        sc = torch.bincount(q, wgt.reshape(-1), K + 2)[1: K + 1].cpu().numpy()
        sh = np.arange(1, K + 1)
        dens = sc / (4.0 / 3.0 * math.pi * ((sh + 0.5) ** 3 - (sh - 0.5) ** 3)) / (B[0] * B[1] * B[2])
        ek = np.where(dens != 0.0, se / np.where(dens != 0.0, dens, 1.0), se)
        return ek, np.array([float(e.sum()), float(sd[dens != 0.0].sum())])

    def step(self):
        p = self.p
        self.at_start = self.stats()
        self.r = [torch.zeros_like(a) for a in self.u]
        for stage, beta, gamma, ct in ((1, 0.0, 1.0 / 3.0, 1.0 / 3.0), (2, -5.0 / 9.0, 15.0 / 16.0, 0.75), (3, -153.0 / 128.0, 8.0 / 15.0, 1.0)):
            up, nl = self._nonlinear()
            if stage == 1:
                self.ucfl = float((up[0].abs() + up[1].abs() + up[2].abs()).max())
                if p.rk3_timestep == pandora.RK3_TIMESTEP_FIXED:
                    self.dt = p.rk3_dt
                elif self.shear:
                    self.dt = 0.5 / p.f_deform_s / p.f_remesh_t
                else:
                    self.dt = min(p.rk3_cfl * self.d[0] / self.ucfl, p.force_tf)
            if p.p_track_part:
                self._particles(up, stage, beta, gamma)
            tot = self._rhs(nl, stage)
            del up, nl
            self.r = [beta * self.r[c] + tot[c] for c in range(3)]
            self.u = [self.u[c] + gamma * self.dt * self.r[c] for c in range(3)]
            for a in self.u:
                a[0, 0, 0] = 0.0
            self._fix()
            self.t = self.t0 + ct * self.dt
            if self.shear:
                self.b13, self.bi13 = -self.S * self.t / self.B[0], self.S * self.t * self.B[2]
        self.t0, self.tstep = self.t, self.tstep + 1


def _pair(a):
    return torch.view_as_real(a.contiguous())


def exact(case, seed):
    points = case["nx"] * case["ny"] * case["nz"]
    if points * case.get("members", 1) * case.get("steps", 1) > 1.5e8:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "batch":
        out = {"stats": [], "u": []}
        x = []
        for m in range(case["members"]):
            e = _Exact(_params(case, seed, m), dev)
            for _ in range(case["steps"]):
                e.step()
            out["stats"].append(np.concatenate(e.at_start))
            if m < _looked_at(case):
                out["u"].append(np.stack([a.cpu().numpy() for a in e.u]))
                if case["np"]:
                    x.append(e.x.cpu().numpy().T)
        out["u"], out["stats"] = np.stack(out["u"]), np.stack(out["stats"])
        if case["np"]:
            out["x"] = np.stack(x)
        return out
    e = _Exact(_params(case, seed), dev)
    if case["kind"] == "stats":
        return _exact_stats(e)
    for _ in range(case["steps"]):
        e.step()
    out = {"u": [_pair(a) for a in e.u], "ek": e.at_start[0], "tke": np.append(e.at_start[1], e.ucfl)}
    if case["np"]:
        if case["particles"]:
            out["x"], out["v"] = e.x.cpu().numpy().T, e.v.cpu().numpy().T
        else:
            v = e.v
            d = [float((v[a] * v[b]).mean()) for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
            out["particles"] = np.array(d + [0.5 * (d[0] + d[1] + d[2])])
    return out


def _exact_stats(e):
    ek, te = e.stats()
    npts = float(e.n[0] * e.n[1] * e.n[2])
    u, w = [e._phys(a) for a in e._ulab()], [e._phys(a) for a in e._vorticity()]
    stored = e._phys(e.u[0])
    m = {}
    for a, b, k in ((0, 0, "u1u1"), (1, 1, "u2u2"), (2, 2, "u3u3"), (0, 1, "u1u2"), (0, 2, "u1u3"), (1, 2, "u2u3")):
        m[k] = float((u[a] * u[b]).mean())
    for c in range(3):
        uu = m[("u1u1", "u2u2", "u3u3")[c]]
        m["skew%d" % (c + 1)] = float((u[c] ** 3).mean()) / uu ** 1.5
        m["flat%d" % (c + 1)] = float((u[c] ** 4).mean()) / uu ** 2
        rms = math.sqrt(float((w[c] ** 2).mean()) * (npts if c == 0 else 1.0))
        m["rmsvort%d" % (c + 1)] = rms
        m["skewvort%d" % (c + 1)] = float((w[c] ** 3).mean()) / rms ** 3
        m["flatvort%d" % (c + 1)] = float((w[c] ** 4).mean()) / rms ** 4
        m["omegamax%d" % (c + 1)] = float(w[c].abs().max())
    m["ucfl"] = float((u[0].abs() + u[1].abs() + u[2].abs()).max())
    r = []
    fa, fb = torch.fft.rfft(u[0]), torch.fft.rfft(stored)
    corr = torch.fft.irfft((fa.conj() * fb).sum((0, 1)), n=e.n[0])
    for lag in range(e.n[0] // 2 + 1):
        r.append(float(corr[lag]) / (m["u1u1"] * npts))
    m["lint11"] = sum(r) * 2.0 * math.pi * e.p.b110 / e.n[0]
    return dict(_grouped(m), ek=ek, tke=te, r1i=np.array(r))
