"""Performance cases of the reconstruction engine: what its users have it do.

A user reconstructs tilt series: through the step-wise engine (prepared once, then outer
iterations of sweep or call, gain/offset and variance estimation, the cost, and the volume read
out), through whole runs from host buffers (one level, or the pipeline's resolution levels), by
projecting a volume, and by advancing several series together in a batch.  Tilt series come from
a microscope's files, so they are host arrays, as the engine's entry points take them; they are
generated on the GPU from the seed (ellipsoid particles over a slab, seeded noise) only because
that is quick.

Kinds of case
  step     a prepared engine, `outers` outer iterations, then cost, nuisance and volume
  run      create, upload, mbir_run with `outers` outer iterations, volume
  multires the pipeline's two resolution levels from host buffers (mbir_run_multires)
  project  a prepared engine holding a volume: forward projection, read out
  estimate a prepared engine holding a volume: gain/offset, variance, cost, error sinogram
  batch    several uneven prepared series, `outers` outer iterations together

Up to 64 views the engine has two voxel-group shapes and times both when it is prepared; the
cases name the shape it settles on (16 lanes x 4 views), so that every run takes the same visit
order and the same summation order.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "openmbir-tem_gb300"))
import mbir  # noqa: E402

DEV = "cuda:0"


def listed():
    return [
        # the smallest reconstruction of the smoke check: latency and launches
        dict(name="haadf-tiny-step", kind="step", mod="haadf", n_r=32, n_t=4, views=21,
             max_deg=60.0, n_z=16, outers=2),
        # the small HAADF configuration (128 x 32 x 64, 71 views, 20 iterations), from host
        # buffers to the volume
        dict(name="haadf-small-run", kind="run", mod="haadf", n_r=128, n_t=32, views=71,
             max_deg=70.0, n_z=64, outers=20),
        # the same series in the FP64 engine (precision studies)
        dict(name="haadf-small-fp64-step", kind="step", mod="haadf", n_r=128, n_t=32, views=71,
             max_deg=70.0, n_z=64, outers=2, fp64=True),
        # the HAADF form of the benchmark workload: one dense sweep, then zero-skipping sweeps
        dict(name="haadf-512-step", kind="step", mod="haadf", n_r=512, n_t=256, views=61,
             max_deg=60.0, n_z=128, outers=8),
        # many views on an odd detector: slices too large for shared memory stay in HBM
        dict(name="haadf-odd-141v-step", kind="step", mod="haadf", n_r=421, n_t=133, views=141,
             max_deg=67.0, n_z=91, outers=3),
        # the benchmark's default: bright field, one equivalent iteration of 20 NHICD calls with
        # the offset and variance updates that a run makes after each
        dict(name="bf-512-step", kind="step", mod="bf", n_r=512, n_t=256, views=61, max_deg=60.0,
             n_z=128, outers=20),
        # bright field with Bragg rejection on (the default threshold of 3), odd sizes
        dict(name="bf-odd-bragg-step", kind="step", mod="bf", n_r=333, n_t=97, views=75,
             max_deg=63.0, n_z=79, outers=20, bragg=3.0),
        # the two-level bright-field configuration, from host buffers to the volume
        dict(name="bf-512-multires", kind="multires", mod="bf", n_r=512, n_t=256, views=61,
             max_deg=60.0, n_z=128, outers=20),
        # the forward model on its own: a dense volume projected
        dict(name="haadf-512-project", kind="project", mod="haadf", n_r=512, n_t=256, views=61,
             max_deg=60.0, n_z=128, outers=1),
        # the estimates on their own, on the same volume
        dict(name="haadf-512-estimate", kind="estimate", mod="haadf", n_r=512, n_t=256, views=61,
             max_deg=60.0, n_z=128, outers=1),
        # uneven series of both modalities advanced together
        dict(name="batch-6-uneven", kind="batch", mod="mixed", n_r=384, n_t=160, views=121,
             max_deg=65.0, n_z=96, outers=6, series=6),
        # the precision workload's size, 121 views: the largest, slices in HBM
        dict(name="bf-1024-step", kind="step", mod="bf", n_r=1024, n_t=512, views=121,
             max_deg=60.0, n_z=256, outers=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["run", "multires", "project", "estimate", "batch"])
    mod = {"step": rng.choice(["haadf", "bf"]), "multires": "bf", "batch": "mixed",
           "run": rng.choice(["haadf", "bf"])}.get(kind, "haadf")
    c = dict(kind=kind, mod=mod, n_r=_log_int(rng, 32, 512), n_t=_log_int(rng, 4, 256),
             views=rng.randint(21, 141), max_deg=round(rng.uniform(55.0, 70.0), 1),
             n_z=2 * rng.randint(8, 64), outers=rng.randint(1, 12))
    if kind == "multires":  # both levels halve evenly
        c.update(n_r=c["n_r"] // 4 * 4, n_t=max(c["n_t"] // 4 * 4, 4), n_z=max(c["n_z"] // 4 * 4, 16))
    if kind == "batch":
        c["series"] = rng.randint(2, 6)
        c["outers"] = rng.randint(2, 6)
    if mod == "bf" and kind == "step" and rng.random() < 0.5:
        c["bragg"] = 3.0
    if kind == "step" and mod == "haadf" and c["n_r"] <= 128 and c["n_t"] <= 32 and \
            rng.random() < 0.3:
        c["fp64"] = True
        c["outers"] = min(c["outers"], 3)
    return c


# ---- synthetic series ------------------------------------------------------------------------
def _angles(case):
    return np.linspace(-case["max_deg"], case["max_deg"], case["views"]).astype(np.float32)


def _ellipsoids(case, rng):
    """Particles above a slab: centres and semi-axes in voxels, values U(0.5, 2)."""
    n_r, n_t, n_z = case["n_r"], case["n_t"], case["n_z"]
    n = max(3, (200 * n_r * n_t * (4 if n_r > 512 else 1)) // (512 * 256))
    top = min(15.0, n_r / 6.0, n_z / 5.0)
    ax = rng.uniform(3.0 if top > 4.0 else top / 2, max(top, 1.0), (n, 3))
    cx = rng.uniform(-1.0, 1.0, n) * (n_r / 2 - ax[:, 0])
    cy = rng.uniform(-0.5, 0.5, n) * n_t
    cz = rng.uniform(-0.5, 1.0, n) * (n_z / 2 - ax[:, 2])
    return np.column_stack([cx, cy, cz, ax, rng.uniform(0.5, 2.0, n)])


def _projection(case, rng):
    """Line integrals [theta][r][t] of the phantom (FP64, on the GPU)."""
    n_r, n_t, n_z = case["n_r"], case["n_t"], case["n_z"]
    th = torch.deg2rad(torch.from_numpy(_angles(case)).to(DEV).double())
    c, s = torch.cos(th)[:, None, None], torch.sin(th)[:, None, None]
    r = (torch.arange(n_r, device=DEV, dtype=torch.float64) - n_r / 2 + 0.5)[None, :, None]
    out = (0.1 * n_z / 8 / c).expand(-1, n_r, n_t).clone()  # the slab
    for cx, cy, cz, ax, ay, az, val in _ellipsoids(case, rng):
        lo, hi = max(0, int(cy - ay + n_t / 2)), min(n_t, int(cy + ay + n_t / 2) + 1)
        if hi <= lo:
            continue
        t = (torch.arange(lo, hi, device=DEV, dtype=torch.float64) - n_t / 2 + 0.5)[None, None, :]
        px, pz = r * c - cx, -r * s - cz
        A = (s / ax) ** 2 + (c / az) ** 2
        B = 2 * (px * s / ax ** 2 + pz * c / az ** 2)
        C = (px / ax) ** 2 + ((t - cy) / ay) ** 2 + (pz / az) ** 2 - 1
        out[:, :, lo:hi] += val * torch.sqrt(torch.clamp(B * B - 4 * A * C, min=0.0)) / A
    return out


def _series(case, seed):
    """(counts [theta][r][t] float32 on the host, tilts in degrees)."""
    rng = np.random.default_rng(seed)
    proj = _projection(case, rng)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    if case["mod"] == "bf":  # Poisson counts at 1e4 electrons, +-3% dose drift per view
        d = torch.from_numpy(1.0 + rng.uniform(-0.03, 0.03, case["views"])).to(DEV)
        lam = 1.0e4 * d[:, None, None] * torch.exp(-0.02 * proj)
        y = torch.poisson(lam.float(), generator=gen).clamp_(min=1.0)
    else:  # gain jitter, offset, signal-dependent Gaussian noise
        g = torch.from_numpy(1.0 + rng.uniform(-0.05, 0.05, case["views"])).to(DEV)
        sig = g[:, None, None] * proj
        noise = torch.randn(sig.shape, device=DEV, dtype=torch.float32, generator=gen)
        y = (sig + 0.1 + noise * torch.sqrt(0.05 * sig + 1e-3)).float()
    return y.cpu().numpy(), _angles(case)


def _volume(case, seed):
    """The phantom on the engine's grid, [z][x][y] float32 on the host."""
    n_r, n_t, n_z = case["n_r"], case["n_t"], case["n_z"]
    z, x, y = (torch.arange(n, device=DEV, dtype=torch.float32) - n / 2 + 0.5
               for n in (n_z, n_r, n_t))
    vol = torch.full((n_z, n_r, n_t), 0.1, device=DEV)
    for cx, cy, cz, ax, ay, az, val in _ellipsoids(case, np.random.default_rng(seed)):
        lo, hi = max(0, int(cy - ay + n_t / 2)), min(n_t, int(cy + ay + n_t / 2) + 1)
        if hi <= lo:
            continue
        d = (((z - cz) / az) ** 2)[:, None, None] + (((x - cx) / ax) ** 2)[None, :, None] + \
            (((y[lo:hi] - cy) / ay) ** 2)[None, None, :]
        vol[:, :, lo:hi] += val * (d <= 1.0)
    return vol.cpu().numpy()


def _params(case):
    if case["mod"] == "bf":
        p = mbir.default_params(mbir.BF)
        p.sigma_x = 0.02
        p.use_default_offset = 1
        p.default_dosage = 1.0e4
        p.bragg_threshold = case.get("bragg", 5.0e10)
    else:
        p = mbir.default_params()
        p.sigma_x = 0.2
    p.sample_thickness = case["n_z"] / 2.0
    p.diffuseness = 0.1
    p.num_resolutions = 2 if case["kind"] == "multires" else 1
    p.outer_iterations = case["outers"]
    p.inner_iterations = 1
    p.stop_threshold = 0.0
    p.precision = mbir.FP64 if case.get("fp64") else mbir.FP32
    p.lane_shape = 1 if case["views"] <= 64 else 0
    return p


# ---- the cases -------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        rng = np.random.default_rng(seed)
        batch, engines = mbir.Batch(0), []
        for k, sub in enumerate(_uneven(case, rng)):
            y, ang = _series(sub, seed * 64 + k)
            e = mbir.Engine(_params(sub))
            e.set_sinogram(y, ang)
            e.prepare()
            batch.add(e)
            engines.append(e)
        return dict(case=case, batch=batch, engines=engines)
    y, ang = _series(case, seed)
    if kind in ("run", "multires"):
        return dict(case=case, y=y, ang=ang, params=_params(case))
    e = mbir.Engine(_params(case))
    e.set_sinogram(y, ang)
    if kind in ("project", "estimate"):
        e.set_initial_volume(_volume(case, seed))
    e.prepare()
    return dict(case=case, engine=e)


def _uneven(case, rng):
    """The batch's series: sizes from a third of the case's to all of it, every third one bright
    field.  The sizes come from the case, the data from the seed."""
    out = []
    for k in range(case["series"]):
        f = 1.0 - 0.67 * k / max(case["series"] - 1, 1)
        g = 1.0 - 0.67 * ((k * 2) % case["series"]) / max(case["series"] - 1, 1)
        out.append(dict(kind="step", mod="bf" if k % 3 == 2 else "haadf",
                        n_r=max(32, int(case["n_r"] * f) | 1), n_t=max(4, int(case["n_t"] * g)),
                        views=max(21, int(case["views"] * g)), max_deg=case["max_deg"],
                        n_z=max(16, 2 * int(case["n_z"] * f / 2)), outers=case["outers"]))
    return out


def _state(e, cost=None):
    g, o, v = e.nuisance()
    out = {"volume": e.volume(), "gains": g, "offsets": o, "variances": v}
    if cost is not None:
        out["cost"] = float(cost)
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        with mbir.Engine(state["params"]) as e:
            e.set_sinogram(state["y"], state["ang"])
            e.run()
            return _state(e)
    if kind == "multires":
        return mbir.run_multires(state["params"], state["y"], state["ang"])
    if kind == "batch":
        _, costs = state["batch"].run(case["outers"], 0.0)
        return [dict(_state(e), cost=float(c)) for e, c in zip(state["engines"], costs)]
    e = state["engine"]
    if kind == "project":
        e.forward_project()
        return e.projection()
    if kind == "estimate":
        e.joint_estimation()
        e.update_weights()
        cost = e.cost()[0]
        g, o, v = e.nuisance()
        return {"error": e.error_sinogram(), "gains": g, "offsets": o, "variances": v,
                "cost": float(cost)}
    for k in range(case["outers"]):
        e.sweep(k, 0)
        e.joint_estimation()
        e.update_weights()
    return _state(e, e.cost()[0])


def work(case):
    """Bytes: the sinogram arrays and the volume read and written once per phase that has to pass
    over them, and the outputs; operations: the voxel updates that a dense sweep or a call makes
    (zero-skipped visits not counted: how many there are depends on the data)."""
    if case["kind"] == "batch":
        parts = [work(c) for c in _uneven(case, None)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    size = 8 if case.get("fp64") else 4
    voxels = case["n_r"] * case["n_t"] * case["n_z"]
    sino = case["n_r"] * case["n_t"] * case["views"]
    entries = 2.7 * case["views"]  # footprint entries of a voxel
    update = 8 * entries + 26 * 12
    forward = 2 * entries
    if case["kind"] == "project":
        return {"bytes": size * (voxels + 2 * sino), "flops": voxels * forward}
    if case["kind"] == "estimate":
        return {"bytes": size * (4 * sino + voxels) + 4 * sino, "flops": sino * 20 + voxels * 26 * 6}
    bf = case["mod"] == "bf"
    n = case["outers"]
    sweep = size * (2 * sino + 2 * voxels) + (sino * (size + 2) if bf else 0)
    estimates = size * 3 * sino + (sino * (2 * size + 2) if bf else 0)
    dense = n / 20.0 if bf else 1.0
    total = {"bytes": n * (sweep + estimates) + 4 * voxels, "flops": voxels * dense * update}
    if case["kind"] in ("run", "multires"):
        total["bytes"] += 4 * sino + size * (voxels + 2 * sino)
        total["flops"] += voxels * forward
    if case["kind"] == "multires":  # the coarse level: an eighth of the voxels, all detector bins
        total["bytes"] += n * (size * 4 * sino + size * voxels / 4)
        total["flops"] += voxels * dense * update / 8
    return total


# ---- 64-bit values ---------------------------------------------------------------------------
_WEIGHTS = (0.0302, 0.0370, 0.0302, 0.0370, 0.0523, 0.0370, 0.0302, 0.0370, 0.0302,
            0.0370, 0.0523, 0.0370, 0.0523, 0.0, 0.0523, 0.0370, 0.0523, 0.0370,
            0.0302, 0.0370, 0.0302, 0.0370, 0.0523, 0.0370, 0.0302, 0.0370, 0.0302)


class _Exact:
    """The HAADF model in 64 bits with torch: voxel size = detector pixel = 1, so that a voxel
    slice y meets detector row t = y alone, with response 1."""

    def __init__(self, case, y, ang):
        self.n_r, self.n_t, self.n_z = case["n_r"], case["n_t"], case["n_z"]
        self.views = case["views"]
        f64 = dict(device=DEV, dtype=torch.float64)
        rad = np.asarray(ang, np.float64) * np.pi / 180
        self.cos, self.sin = np.cos(rad), np.sin(rad)
        self.offset_r = (1 / np.sqrt(3.0) + 0.5) / 64
        self.kr = float(np.float32(1.0 / self.offset_r))
        H = self._response(rad)
        self.H = torch.from_numpy(np.concatenate([H, H[:, -1:]], 1)).to(DEV)
        self.u0 = ((-self.n_r / 2 + 0.5) * self.cos - (-self.n_z / 2 + 0.5) * self.sin +
                   self.n_r / 2)
        self.y = torch.from_numpy(y).to(DEV).double().permute(2, 0, 1).contiguous()  # [t][theta][r]
        # initial offset: constant term of the fit of the views' means against 1 / cos
        basis = np.stack([1.0 / self.cos, np.ones_like(self.cos)], 1)
        mean = self.y.mean(dim=(0, 2)).cpu().numpy()
        off = np.linalg.solve(basis.T @ basis, basis.T @ mean)[1]
        self.gain = torch.ones(self.views, **f64)
        self.mu = torch.full((self.views,), float(off), **f64)
        self.w = torch.ones(self.views, **f64)
        self.var = torch.ones(self.views, **f64)
        self.filt = torch.tensor(_WEIGHTS, **f64)
        self.P, self.Q, self.c, self.sigma = 2.0, 1.1, 0.001, 0.2

    def _response(self, rad):
        """Detector response [theta][64]: the voxel profile (its angle in radians twice, as the
        HAADF engine has it) against the beam profile."""
        n_prof, n_beam, bins = 1536, 512, 64
        a = rad * np.pi / 180
        a = np.where(a < 0, a + np.pi / 2, a)
        mv = np.where(a <= np.pi / 4, 1 / np.cos(a), 1 / np.cos(np.pi / 2 - a))
        k = np.cos(np.pi / 4)
        d1, d2 = k * np.cos(np.pi / 4 - a), k * np.abs(np.cos(np.pi / 4 + a))
        t = 2.0 * np.arange(n_prof) / n_prof
        lc, ln, rn, rc = (v[:, None] for v in (1 - d1, 1 - d2, 1 + d2, 1 + d1))
        m = mv[:, None]
        with np.errstate(divide="ignore", invalid="ignore"):
            prof = np.where((t <= lc) | (t >= rc), 0.0,
                            np.where(t > rn, m * (rc - t) / (rc - rn),
                                     np.where(t >= ln, m, m * (t - lc) / (ln - lc))))
        beam = 0.54 - 0.46 * np.cos((2 * np.pi / n_beam) * np.arange(n_beam))
        beam /= beam.sum()
        H = np.zeros((len(rad), bins))
        r = -0.5 + np.arange(n_beam) / n_beam
        for i in range(bins):
            rmin = i * self.offset_r - 1.0
            at = np.clip(np.floor((r - rmin) * (n_prof / 2.0)).astype(int), 0, n_prof - 1)
            H[:, i] = prof[:, at] @ np.where(r >= rmin, beam, 0.0)
        return H

    def column(self, z, xs):
        """A-column entries of the voxels (z, xs): bins and values [len(xs)][theta][3]."""
        u = torch.from_numpy(self.u0[None, :] - z * self.sin[None, :] +
                             np.asarray(xs, np.float64)[:, None] * self.cos[None, :]).to(DEV)
        lo = torch.floor(u - 1.0)
        j = lo[..., None] + torch.arange(3, device=DEV, dtype=torch.float64)
        ok = (j <= torch.floor(u + 1.0)[..., None]) & (j >= 0) & (j < self.n_r)
        xr = torch.abs(j + 0.5 - u[..., None]) * self.kr
        idx = xr.long()
        ok &= idx < 64
        idx = idx.clamp(max=63)
        t = xr - idx
        v = torch.arange(self.views, device=DEV)[None, :, None].expand_as(idx)
        a = (1 - t) * self.H[v, idx] + t * self.H[v, idx + 1]
        a = torch.where(ok & (a > 0), a, torch.zeros_like(a))
        return j.clamp(0, self.n_r - 1).long(), a

    def project(self, vol):
        """[t][theta][r] of vol [y][z][x] (without gains)."""
        out = torch.zeros_like(self.y)
        flat = out.view(self.n_t, -1)
        base = torch.arange(self.views, device=DEV)[None, :, None] * self.n_r
        for z in range(self.n_z):
            j, a = self.column(z, np.arange(self.n_r))
            A = torch.zeros(self.n_r, self.views * self.n_r, device=DEV, dtype=torch.float64)
            A.scatter_add_(1, (j + base).view(self.n_r, -1), a.view(self.n_r, -1))
            flat += vol[:, z, :] @ A
        return out

    def stride(self):
        """Smallest x distance at which no two voxels of a row share a detector bin."""
        eps = 1e-4
        u = (self.u0[:, None, None] - np.arange(self.n_z)[None, :, None] *
             self.sin[:, None, None] + np.arange(self.n_r)[None, None, :] *
             self.cos[:, None, None])
        s = 2
        while s < self.n_r:
            ua, ub = u[:, :, :-s], u[:, :, :-s] + s * self.cos[:, None, None]
            alo, ahi = (np.maximum(np.floor(ua - 1 - eps), 0),
                        np.minimum(np.floor(ua + 1 + eps), self.n_r - 1))
            blo, bhi = (np.maximum(np.floor(ub - 1 - eps), 0),
                        np.minimum(np.floor(ub + 1 + eps), self.n_r - 1))
            if not np.any((alo <= ahi) & (blo <= bhi) & ~((ahi < blo) | (bhi < alo))):
                break
            s += 1
        return max(2, min(s, max(self.n_r, 2)))

    def rows(self, sweep, seed=1):
        """The sweep's row order: a shuffle drawn from MT19937."""
        gen = np.random.MT19937()
        gen._legacy_seeding((seed * 2654435761 + sweep * 40503 + 17) % (1 << 32))
        order = list(range(self.n_z))
        for i, r in zip(range(self.n_z - 1, 0, -1), gen.random_raw(max(self.n_z - 1, 1))):
            k = int(r) % (i + 1)
            order[i], order[k] = order[k], order[i]
        return order

    def sweep(self, x, e, index, later, stride):
        """One sweep in the engine's order: colours in y, rows, conflict-free classes."""
        for colour in (0, 1):
            ys = torch.arange(colour, self.n_t, 2, device=DEV)
            if len(ys) == 0:
                continue
            es = e[ys].reshape(len(ys), -1)  # this colour's detector rows: disjoint, a copy
            for z in self.rows(index):
                for k in range(min(stride, self.n_r)):
                    self._class(x, es, ys, z, np.arange(k, self.n_r, stride), later)
            e[ys] = es.view(len(ys), self.views, self.n_r)

    def _class(self, x, es, ys, z, xs, later):
        xt = torch.from_numpy(xs).to(DEV)
        V = x[ys][:, z, :][:, xt]
        pad = self._pad  # volume padded by one voxel of NaN
        nb = torch.stack([pad[ys + 1 + dy][:, z + 1 + dz, :][:, xt + 1 + dx]
                          for dy in (-1, 0, 1) for dz in (-1, 0, 1) for dx in (-1, 0, 1)], -1)
        there = ~torch.isnan(nb)
        there[..., 13] = False
        nb = torch.where(there, nb, torch.zeros_like(nb))
        live = torch.ones_like(V, dtype=torch.bool)
        if later:
            live = ~((V == 0) & ~(nb > 0).any(-1))
            if not bool(live.any()):
                return
        d = (V[..., None] - nb).abs()
        t1 = d ** (self.P - self.Q) / self.sigma ** (self.P - self.Q)
        t3 = self.c + t1
        sp = self.sigma ** self.P
        coef = torch.where(d == 0, torch.full_like(d, self.P / (sp * self.c)),
                           (self.P - (self.P - self.Q) * t1 / t3) / (t3 * sp))
        coef = torch.where(there, coef * self.filt, torch.zeros_like(coef))
        s1, s2 = (coef * nb).sum(-1), coef.sum(-1)
        j, a = self.column(z, xs)
        at = (j + torch.arange(self.views, device=DEV)[None, :, None] * self.n_r).view(-1)
        pe = (a * self.gain[None, :, None]).view(len(xs), -1)
        pw = pe * self.w[None, :, None].expand(len(xs), -1, 3).reshape(len(xs), -1)
        ev = es[:, at].view(len(ys), len(xs), -1)
        th1 = -torch.einsum("yxe,xe->yx", ev, pw)
        th2 = (pe * pw).sum(-1)[None, :].expand_as(V)
        lo, hi = nb.amin(-1).clamp(max=0.0), nb.amax(-1).clamp(min=0.0)
        cand = torch.where(th2 != 0, V - th1 / th2, torch.zeros_like(V))
        lo = torch.where(th2 != 0, torch.minimum(lo, cand), lo)
        hi = torch.where(th2 != 0, torch.maximum(hi, cand), hi)
        u = (s1 + th2 * V - th1) / (s2 + th2)
        nv = torch.maximum(torch.minimum(V + 1.5 * (u - V), hi), lo).clamp(min=0.0)
        nv = torch.where(live, nv, V)
        dlt = nv - V
        es.index_add_(1, at, -(dlt[..., None] * pe[None]).reshape(len(ys), -1))
        yi, xi = ys[:, None].expand_as(nv), xt[None, :].expand_as(nv)
        x[yi, z, xi] = nv
        pad[yi + 1, z + 1, xi + 1] = nv

    def estimate(self, e):
        """Gain and offset per view, the error rebuilt, then the variances."""
        n = self.n_r * self.n_t
        yh = (self.y - e - self.mu[None, :, None]) / self.gain[None, :, None]
        w = self.w
        b_y, b_h = self.y.sum((0, 2)) * w, yh.sum((0, 2)) * w
        hy, hh = (yh * self.y).sum((0, 2)) * w, (yh * yh).sum((0, 2)) * w
        d1, d2 = b_y / (n * w), b_h / (n * w)
        den = hh - b_h * d2
        lm = (-self.views + ((hy - b_h * d1) / den).sum()) / (1 / den).sum()
        self.gain = (hy - b_h * d1 - lm) / den
        self.mu = d1 - d2 * self.gain
        e = self.y - self.mu[None, :, None] - self.gain[None, :, None] * yh
        self.var = (e * e).sum((0, 2)) / n
        self.w = 1.0 / self.var
        return e

    def cost(self, x, e):
        data = ((e * e).sum((0, 2)) * self.w).sum() / 2
        noise = (self.n_r * self.n_t * torch.log(2 * np.pi * self.var)).sum() / 2
        prior = 0.0
        for k in range(14, 27):  # every pair once
            dy, dz, dx = k // 9 - 1, (k // 3) % 3 - 1, k % 3 - 1

            def cut(v, sign):
                for dim, o in ((0, dy), (1, dz), (2, dx)):
                    lo, hi = max(0, -sign * o), min(v.shape[dim], v.shape[dim] - sign * o)
                    if hi <= lo:
                        return None
                    v = v.narrow(dim, lo, hi - lo)
                return v
            a, b = cut(x, 1), cut(x, -1)
            if a is None:
                continue
            d = (a - b).abs()
            prior = prior + _WEIGHTS[k] * (d ** self.P / self.sigma ** self.P /
                                           (self.c + (d / self.sigma) ** (self.P - self.Q))).sum()
        return float(data + noise + prior)

    def nuisance(self):
        return {"gains": self.gain.cpu().numpy(), "offsets": self.mu.cpu().numpy(),
                "variances": self.var.cpu().numpy()}


def exact(case, seed):
    """HAADF projection, estimates and single iterations in 64 bits.  Bright-field calls (their
    order comes from a sequential colouring), batches and long runs have none: they would take
    too long this way."""
    if case["mod"] != "haadf" or case["kind"] not in ("project", "estimate", "step"):
        return None
    steps = case["n_z"] * case["outers"]
    if case["kind"] == "step" and steps * max(1.0, case["n_r"] * case["n_t"] * case["views"] / 2e6) > 300:
        return None
    y, ang = _series(case, seed)
    m = _Exact(case, y, ang)
    if case["kind"] == "step":
        x = torch.zeros(m.n_t, m.n_z, m.n_r, device=DEV, dtype=torch.float64)
        e = m.y - m.mu[None, :, None]
        m._pad = torch.nn.functional.pad(x, (1,) * 6, value=float("nan"))
        stride = m.stride()
        for k in range(case["outers"]):
            m.sweep(x, e, k, k > 0, stride)
            e = m.estimate(e)
        return dict(m.nuisance(), volume=x.permute(1, 2, 0).contiguous().cpu().numpy(),
                    cost=m.cost(x, e))
    x = torch.from_numpy(_volume(case, seed)).to(DEV).double().permute(2, 0, 1).contiguous()
    proj = m.project(x)
    if case["kind"] == "project":
        return proj.permute(1, 2, 0).contiguous().cpu().numpy()
    e = m.estimate(m.y - proj - m.mu[None, :, None])
    return dict(m.nuisance(), error=e.permute(1, 2, 0).contiguous().cpu().numpy(),
                cost=m.cost(x, e))
