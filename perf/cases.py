"""Performance cases: the calls that programs using this framework spend
their time in, over the sizes that the repository's workloads, tests and
benchmark use.

A case is a dict of plain values:
  path       what one pass runs
               rhs       one right-hand side (Engine.rhs / Engine.rhs_device)
               rates     the out-scattering rates of a status (Engine.scattering_rates)
               dp45      an adaptive integration with dense output (Engine.dp45)
               ensemble  the same for many runs in one handle (BatchEngine.dp45)
               gradient  forward and backward of an integration (adjoint.DP45Solve)
  material   ee: one parabolic band, electron-electron scattering (four legs)
             eph: parabola and Dirac cone with one optical phonon and a field
                  (three legs and drift)
             eph3: three bands and two phonons (three legs)
  nx, ny     sections of the k mesh (2 nx ny triangles)
  umklapp    umklapp steps of every channel
  moments    fp64, or t40 / t48 / t32: the reduced-precision storage option
  exact_sums the deterministic mode (bit-reproducible sums)
  stream     four-leg tuples are enumerated in every evaluation, not stored
  pointers   host (NumPy arrays) or device (torch tensors on the GPU)
  t, dense   final time and dense-output step of an integration
  runs       runs of an ensemble

exact() restates the operator in plain torch, in FP64 and with every simplex
decision in the order of the reference's formulas (no FMA), because a tuple
whose points lie exactly on a face of the reference triangle is decided by
rounding.
"""
import itertools
import math

import numpy as np
import torch

from tortoise_b200 import adjoint as A
from tortoise_b200 import engine as E
from tortoise_b200 import workloads as W

_BASE = {"path": "rhs", "material": "eph", "nx": 16, "ny": 16, "umklapp": 0, "moments": "fp64", "exact_sums": False,
         "stream": False, "pointers": "host", "t": 0.0, "dense": 0.0, "runs": 1}


def _case(**kw):
    return dict(_BASE, **kw)


def listed():
    return [
        # a notebook, a test or a C++ host evaluating a small material once per call
        _case(name="rhs_eph_8", nx=8, ny=8),
        # the benchmark's mesh, state resident on the GPU (a user's own time stepper)
        _case(name="rhs_eph_64", nx=64, ny=64, pointers="device"),
        # the largest stored operator: three bands, two phonons, a non-square mesh
        _case(name="rhs_eph3_72x56", material="eph3", nx=72, ny=56, pointers="device"),
        # the mixed-precision option of single runs
        _case(name="rhs_t40_64", nx=64, ny=64, moments="t40", pointers="device"),
        # the deterministic option: bit-reproducible sums
        _case(name="rhs_exact_sums_32", nx=32, ny=32, exact_sums=True),
        # analysis of a status: the scattering rates, with umklapp channels
        _case(name="rates_eph_40x24", path="rates", nx=40, ny=24, umklapp=1),
        # the reference's own CPU case, 16x16 electron-electron: one right-hand side
        _case(name="rhs_ee_16", material="ee", pointers="device"),
        # a whole small electron-electron relaxation
        _case(name="dp45_ee_8", path="dp45", material="ee", nx=8, ny=8, t=10.0, dense=1.0),
        # a whole electron-phonon run from host buffers
        _case(name="dp45_eph_48", path="dp45", nx=48, ny=48, t=1.0, dense=0.25),
        # a parameter scan: many runs on several meshes in one handle
        _case(name="ensemble_48", path="ensemble", nx=32, ny=32, runs=48, t=0.5, dense=0.25),
        # fitting: gradients of an observable with respect to state and couplings
        _case(name="gradient_eph_24", path="gradient", nx=24, ny=24, t=0.5, dense=0.25, pointers="device"),
        # a four-leg channel whose tuples are not stored
        _case(name="stream_ee_12x10", material="ee", nx=12, ny=10, stream=True, pointers="device"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["rhs", "rhs", "rhs", "rhs", "rates", "dp45", "dp45", "ensemble", "gradient"])
    c = _case(path=path, pointers=rng.choice(["host", "device"]) if path in ("rhs", "gradient") else "host")
    c["material"] = rng.choice(["eph", "eph", "eph3", "ee"]) if path in ("rhs", "rates") else rng.choice(
        ["eph", "eph", "ee"]) if path == "dp45" else "eph"
    hi = {"rhs": 64, "rates": 48, "dp45": 40, "ensemble": 32, "gradient": 24}[path]
    if c["material"] == "ee":
        hi = 14 if path != "dp45" else 9
    c["nx"], c["ny"] = _log_int(rng, 5, hi), _log_int(rng, 5, hi)
    if c["material"] == "ee" and path == "rhs":
        c["stream"] = c["nx"] * c["ny"] <= 120 and rng.random() < 0.4
    if c["material"] != "ee" and path in ("rhs", "rates"):
        c["umklapp"] = 1 if c["nx"] * c["ny"] <= 1024 and rng.random() < 0.3 else 0
        if path == "rhs":
            c["moments"] = rng.choice(["fp64", "fp64", "fp64", "t40", "t48", "t32"])
            c["exact_sums"] = rng.random() < 0.2
    if path in ("dp45", "ensemble", "gradient"):
        c["t"] = rng.choice([0.25, 0.5, 1.0])
        c["dense"] = c["t"] / rng.choice([1, 2, 4])
    if path == "ensemble":
        c["runs"] = rng.randint(2, 48)
    return c


# ------------------------------------------------------------------ inputs
def _material(case, nx, ny, **kw):
    """The case's material on an nx x ny mesh (a host-side description only)."""
    bands, phonons, ee = {"ee": (("P",), (), True), "eph": (("P", "D"), (0.2,), False),
                          "eph3": (("P", "D", "H"), (0.15, 0.25), False)}[case["material"]]
    mat = W.build_material(max(nx, ny), bands, phonons, ee=ee, eph=not ee, field=(0.0, 0.0) if ee else (0.1, 0.0),
                           rtol=1e-6 if ee else 1e-8, atol=1e-9, mesh_nsplit=(nx, ny), **kw)
    for c in mat.channels:
        c.findUmklappVectors(case["umklapp"])
    return mat


def _runs(case, seed):
    """Materials and initial states of the case's runs: every run draws its
    temperature, coupling and hot-carrier bump; the meshes of an ensemble
    take turns between the case's, three quarters and half of it."""
    rng = np.random.default_rng([seed, 77])
    mats, states = [], []
    for r in range(case["runs"]):
        q = (4, 3, 2)[r % 3] if case["path"] == "ensemble" else 4
        kw = {"eph_amplitude": float(rng.uniform(0.5, 2.0))} if case["path"] in ("ensemble", "gradient") else {}
        m = _material(case, max(2, case["nx"] * q // 4), max(2, case["ny"] * q // 4), **kw)
        mats.append(m)
        states.append(W.initial_status(m, kT=float(rng.uniform(0.06, 0.2)), seed=int(rng.integers(1 << 30))).vec)
    return mats, states


def prepare(case, seed):
    mats, states = _runs(case, seed)
    opts = {"deterministic": case["exact_sums"], "stream_legs": 4 if case["stream"] else 0,
            "allow_fp32": {"fp64": 0, "t32": 1, "t40": 2, "t48": 3}[case["moments"]]}
    s = {"case": case}
    if case["path"] == "ensemble":
        s["engine"], s["f"] = E.BatchEngine(mats, **opts), np.concatenate(states)
        return s
    s["engine"], s["f"] = E.Engine(mats[0], **opts), states[0]
    if case["path"] == "gradient":
        dev = "cuda" if case["pointers"] == "device" else "cpu"
        s["f"] = torch.tensor(states[0], device=dev, requires_grad=True)
        s["amps"] = torch.tensor([c.amplitude for c in mats[0].channels], dtype=torch.float64, device=dev,
                                 requires_grad=True)
        s["w"] = torch.tensor(A.observable_weights(mats[0], 0, "energy"), device=dev)
    elif case["pointers"] == "device":
        s["f"] = torch.tensor(states[0], device="cuda")
        s["out"] = torch.empty_like(s["f"])
    return s


def run(s):
    """Integrations return their dense outputs, the trajectory that MaterialTimeStatus stores; the state after the
    last step lies at a time of the step control's own."""
    case, eng = s["case"], s["engine"]
    if case["path"] == "rhs":
        if case["pointers"] == "host":
            return eng.rhs(s["f"])
        eng.rhs_device(s["f"].data_ptr(), s["out"].data_ptr())
        return s["out"]
    if case["path"] == "rates":
        return eng.scattering_rates(s["f"])
    if case["path"] == "dp45":
        r = eng.dp45(s["f"], 0.0, case["t"], case["dense"])
        return {"dense": r["dense"], "attempts": r["attempts"]}
    if case["path"] == "ensemble":
        r = eng.dp45(s["f"], 0.0, case["t"], case["dense"])
        return {"dense": np.concatenate([q["dense"].ravel() for q in r["runs"]]),
                "attempts": np.array([q["attempts"] for q in r["runs"]])}
    s["f"].grad = s["amps"].grad = None
    fo = A.DP45Solve.apply(s["f"], s["amps"], eng, 0.0, case["t"], case["dense"])
    j = (s["w"] * fo).sum()
    j.backward()
    return {"observable": j.detach(), "f_obs": fo.detach(), "grad_f": s["f"].grad, "grad_amps": s["amps"].grad}


def work(case):
    """What a pass cannot do without: per evaluation the element ids of every
    tuple with a contribution, the state once in and once out, and the
    integrand with its first moments at the points inside the simplices
    (6 L + 14 operations each).  Tuples grow as (nx ny)^1.5 for three legs
    and (nx ny)^2.5 for four; their counts and points per tuple are those of
    the enumeration on square meshes."""
    L, per, kept, points, bands = {"ee": (4, 55.0, 0.71, 2.8, 1), "eph": (3, 37.4, 0.88, 5.2, 3),
                                   "eph3": (3, 77.0, 0.88, 4.9, 5)}[case["material"]]
    sizes = [1.0] if case["path"] != "ensemble" else [(1.0, 0.75, 0.5)[r % 3] for r in range(case["runs"])]
    evals = 1.0
    if case["path"] in ("dp45", "ensemble"):
        evals = 6.0 * (6 + 14 * case["t"]) + 1
    elif case["path"] == "gradient":
        evals = 3 * 6.0 * (6 + 14 * case["t"])
    elif case["path"] == "rates":
        evals = float(L)
    tuples = dofs = 0.0
    for s in sizes:
        sec = case["nx"] * case["ny"] * s * s
        tuples += per * sec ** (1.5 if L == 3 else 2.5)
        dofs += 6 * sec * bands
    return {"bytes": evals * (tuples * kept * 4 * (L + 1) + 16 * dofs), "flops": evals * tuples * points * (6 * L + 14)}


# ------------------------------------------------- the operator, in plain torch
_GW, _GA, _GB = 0.33333333333333, 0.16666666666667, 0.66666666666667
_G1 = (0.2113248654051871, 0.7886751345948129)
_VERT = torch.tensor([[[0., 0.], [1., 0.], [1., 1.]], [[0., 0.], [0., 1.], [1., 1.]]], dtype=torch.float64)


class _Mesh:
    """Vertices, P1 coefficients of kx and ky, mass matrix and section boxes of one mesh."""

    def __init__(self, mesh, dev):
        self.nx, self.ny = mesh.nsplit
        self.ne, self.vol = 2 * self.nx * self.ny, float(mesh.elemVolume)
        self.o, self.G = [float(x) for x in mesh.origin], [[float(x) for x in r] for r in mesh.dG]
        self.rel = [float(x) for x in mesh.rel_origin]
        G = self.G
        inv = 1.0 / (G[0][0] * G[1][1] - G[0][1] * G[1][0])
        self.iG = [[G[1][1] * inv, -G[0][1] * inv], [-G[1][0] * inv, G[0][0] * inv]]
        e = torch.arange(self.ne, device=dev)
        s = torch.div(e, 2, rounding_mode="floor")
        p = torch.stack([s % self.nx, torch.div(s, self.nx, rounding_mode="floor")], -1).double()[:, None, :]
        p = p + _VERT.to(dev)[e % 2]
        self.local = [G[i][0] * p[..., 0] + G[i][1] * p[..., 1] for i in range(2)]   # relative to the origin
        self.k = []
        for i in range(2):
            v = self.o[i] + self.local[i]
            self.k.append(torch.stack([v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]], -1))
        phi = torch.tensor([[1., 1., 1.], [_GA, _GB, _GA], [_GA, _GA, _GB]], dtype=torch.float64, device=dev)
        self.minv = torch.linalg.inv(self.vol * _GW * (phi @ phi.T))

    def boxes(self, d, dev):
        """[nx ny, 2 (low, high), 2] of every section, shrunk by 1e-8, times d."""
        s = torch.arange(self.nx * self.ny, device=dev)
        xy = [s % self.nx, torch.div(s, self.nx, rounding_mode="floor")]
        ends = []
        for shift, eps in ((0, 0.00000001), (1, -0.00000001)):
            a, b = [(q + shift).double() + eps for q in xy]
            ends.append(torch.stack([self.o[i] + (self.G[i][0] * a + self.G[i][1] * b) for i in range(2)], -1) * d)
        return torch.stack(ends if d > 0 else ends[::-1], 1)


def _det_and_inverse(a):
    """det by the expansion along row 0; the inverse by cofactors over the expansion along column 0."""
    det = (a[0][0] * (a[1][1] * a[2][2] - a[1][2] * a[2][1]) - a[0][1] * (a[1][0] * a[2][2] - a[1][2] * a[2][0])
           + a[0][2] * (a[1][0] * a[2][1] - a[1][1] * a[2][0]))
    cof = [[a[(i + 1) % 3][(j + 1) % 3] * a[(i + 2) % 3][(j + 2) % 3]
            - a[(i + 1) % 3][(j + 2) % 3] * a[(i + 2) % 3][(j + 1) % 3] for j in range(3)] for i in range(3)]
    inv = 1.0 / ((cof[0][0] * a[0][0] + cof[1][0] * a[1][0]) + cof[2][0] * a[2][0])
    return det, [[cof[j][i] * inv for j in range(3)] for i in range(3)]


class _Reference:
    def __init__(self, mat, dev):
        self.dev, self.mat = dev, mat
        self.meshes = {id(b.mesh): _Mesh(b.mesh, dev) for b in mat.bands}
        self.mesh = [self.meshes[id(b.mesh)] for b in mat.bands]
        self.off, self.n = mat.band_offsets()
        self.E = [torch.tensor(b.dispersion_coeffs, device=dev).reshape(-1, 3) for b in mat.bands]
        nod = [torch.stack([e[:, 0], e[:, 1] + e[:, 0], e[:, 2] + e[:, 0]], -1) for e in self.E]
        self.lo, self.hi = [x.min(1).values for x in nod], [x.max(1).values for x in nod]
        self.kept = None

    # -- the points inside the simplices of every tuple
    def points(self):
        """(channel, element ids [L, p], reference coordinates [L, 2, p], weight [p]) of the (tuple, point) pairs
        that contribute, in parts."""
        if self.kept is not None:
            yield from self.kept
            return
        for ci, c in enumerate(self.mat.channels):
            for ids, umk in self._candidates(c):
                yield from self._inside(ci, c, ids, umk)

    def keep_points(self):
        """Finds the pairs once, for many evaluations."""
        parts = list(self.points())
        self.kept = []
        for ci in range(len(self.mat.channels)):
            mine = [q for q in parts if q[0] == ci]
            if mine:
                self.kept.append((ci,) + tuple(torch.cat([q[j] for q in mine], -1) for j in (1, 2, 3)))
        return self

    def _candidates(self, c):
        """Element ids inside the energy window, in chunks of about a million."""
        L, dev, d, b = c.nlegs, self.dev, c.legDirection, c.legBandNumber
        ms, last = [self.mesh[x] for x in b], self.mesh[b[-1]]
        nsec = [m.nx * m.ny for m in ms[:-1]]
        total = math.prod(nsec)
        box = [m.boxes(float(d[l]), dev) for l, m in enumerate(ms[:-1])]
        g = np.asarray(self.mat.region.gvec)
        ids_out, umk_out, have = [], [], 0
        for ui, u in enumerate(np.asarray(c.umklappUnitVectors, dtype=np.float64).reshape(-1, 2)):
            gu = [float(g[i, 0] * u[0] + g[i, 1] * u[1]) for i in range(2)]
            for first in range(0, total, 1 << 22):
                r = torch.arange(first, min(total, first + (1 << 22)), device=dev)
                sec = []
                for n in reversed(nsec):
                    sec.insert(0, r % n)
                    r = torch.div(r, n, rounding_mode="floor")
                acc = box[0][sec[0]]
                for l in range(1, L - 1):
                    acc = acc + box[l][sec[l]]
                acc = (acc + torch.tensor(gu, device=dev, dtype=torch.float64)) * -float(d[-1])
                if d[-1] > 0:
                    acc = acc.flip(1)
                lo, width = [], []
                for i in range(2):
                    x, y = acc[..., 0] - last.o[0], acc[..., 1] - last.o[1]
                    t = torch.floor(last.iG[i][0] * x + last.iG[i][1] * y)
                    n = (last.nx, last.ny)[i]
                    lo.append(t[:, 0].clamp(0, n).long())
                    width.append((t[:, 1] + 1.0).clamp(0, n).long() - lo[i])
                for dy, dx in itertools.product(range(int(width[1].max())), range(int(width[0].max()))):
                    sel = ((dx < width[0]) & (dy < width[1])).nonzero()[:, 0]
                    end = 2 * (lo[0][sel] + dx + (lo[1][sel] + dy) * last.nx)
                    s = [q[sel] for q in sec]
                    for comb in itertools.product((0, 1), repeat=L):
                        e = [2 * s[l] + comb[l] for l in range(L - 1)] + [end + comb[-1]]
                        mn = mx = 0.0
                        for l in range(L):
                            a, z = self.lo[b[l]][e[l]], self.hi[b[l]][e[l]]
                            mn, mx = (mn + a, mx + z) if d[l] > 0 else (mn + -z, mx + -a)
                        ok = (mn <= 0.0) & (mx >= 0.0)
                        ids_out.append(torch.stack([q[ok] for q in e]))
                        umk_out.append(torch.full((ids_out[-1].shape[1],), ui, device=dev))
                        have += ids_out[-1].shape[1]
                        if have > 1_000_000:
                            yield torch.cat(ids_out, 1), torch.cat(umk_out)
                            ids_out, umk_out, have = [], [], 0
        if have:
            yield torch.cat(ids_out, 1), torch.cat(umk_out)

    def _inside(self, ci, c, ids_all, umk_all):
        dev, L, d, b = self.dev, c.nlegs, c.legDirection, c.legBandNumber
        n_mc, fact = c.numMCPoints, 2.0 ** (L - 2)
        umk_vec = torch.tensor(np.asarray(c.umklappUnitVectors), device=dev).reshape(-1, 2)
        g = np.asarray(self.mat.region.gvec)
        vol = 1.0
        for l in range(L):
            vol *= self.mesh[b[l]].vol * 2.0
        for a in range(0, ids_all.shape[1], 1 << 22):
            ids, umk = ids_all[:, a:a + (1 << 22)], umk_all[a:a + (1 << 22)]
            tab = lambda l: (self.mesh[b[l]].k[0], self.mesh[b[l]].k[1], self.E[b[l]])  # noqa: E731

            def geometry(ids, umk):
                D, N = [[None] * (2 * L) for _ in range(3)], [0.0, 0.0, 0.0]
                for l in range(L):
                    for i, t in enumerate(tab(l)):
                        v = t[ids[l]] * float(d[l])
                        N[i] = N[i] - v[:, 0]
                        D[i][2 * l], D[i][2 * l + 1] = v[:, 1], v[:, 2]
                for i in range(2):
                    for j in range(2):
                        N[i] = N[i] - umk_vec[umk][:, j] * float(g[i, j])
                det, Ci = _det_and_inverse([[D[i][2 * L - 3 + j] for j in range(3)] for i in range(3)])
                return D, N, det.abs(), Ci

            def point(D, N, Ci, q):
                r = []
                for i in range(3):
                    s = 0.0
                    for l in range(L - 2):
                        s = s + (D[i][2 * l] * q[2 * l] + D[i][2 * l + 1] * q[2 * l + 1])
                    r.append((s + D[i][2 * L - 4] * q[-1]) - N[i])
                al = [-((Ci[i][0] * r[0] + Ci[i][1] * r[1]) + Ci[i][2] * r[2]) for i in range(3)]
                ok = (al[0] > 0) & (al[0] + q[-1] < 1) & (al[1] > 0) & (al[2] > 0) & (al[1] + al[2] < 1)
                return al, (ok & (q[-1] > 0))

            D, N, det, Ci = geometry(ids, umk)
            prodc, sums = 1.0, torch.zeros_like(det)
            for _ in range(L):
                prodc *= math.sqrt(2.0)
            for q in c.mc_points_precalc.tolist():
                sums = sums + point(D, N, Ci, q)[1] * prodc
            live = (det >= c.minimumDeterminant) & (((1.0 / (fact * n_mc * det)) * sums * vol).abs()
                                                    > c.scattElemeThreshold)
            ids, umk = ids[:, live], umk[live]
            D, N, det, Ci = geometry(ids, umk)
            weight = vol / (fact * n_mc * det)
            for q in c.mc_points.tolist():
                al, ok = point(D, N, Ci, q)
                at = ok.nonzero()[:, 0]
                if not at.numel():
                    continue
                p = [torch.full((2, at.numel()), 0.0, dtype=torch.float64, device=dev) for _ in range(L)]
                for l in range(L - 2):
                    p[l][0], p[l][1] = q[2 * l], q[2 * l + 1]
                p[L - 2][0], p[L - 2][1] = q[-1], al[0][at]
                p[L - 1][0], p[L - 1][1] = al[1][at], al[2][at]
                yield ci, ids[:, at], torch.stack(p), weight[at]

    # -- the right-hand side
    def collisions(self, f, amps=None, rates=False):
        acc = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        for ci, ids, p, w in self.points():
            c = self.mat.channels[ci]
            amp = c.amplitude if amps is None else amps[ci]
            base = [3 * ids[l] + self.off[bd] for l, bd in enumerate(c.legBandNumber)]
            form = []
            for l, bd in enumerate(c.legBandNumber):
                s, sign = self.mat.bands[bd].statistics, -1.0 if l == 0 else 1.0
                t = f[base[l]] + f[base[l] + 1] * p[l][0] + f[base[l] + 2] * p[l][1]
                loss, gain = (t, 1.0 + s * t) if c.legDirection[l] > 0 else (1.0 + s * t, t)
                unit = (2.0, 2.0 * s) if c.legDirection[l] > 0 else (2.0 * s, 2.0)
                form.append((sign * loss, gain, sign * unit[0], unit[1]))
            for l in range(c.nlegs):
                if not rates and l:
                    v = w * amp * common
                else:
                    a = g = 1.0
                    for m in range(c.nlegs):
                        u = rates and m == l
                        a, g = a * form[m][2 if u else 0], g * form[m][3 if u else 1]
                    common = a + g
                    v = w * amp * common
                v = v * (-c.legDirection[l] if rates else c.legDirection[l])
                acc = acc.index_add(0, base[l], v)
                acc = acc.index_add(0, base[l] + 1, v * p[l][0])
                acc = acc.index_add(0, base[l] + 2, v * p[l][1])
        return acc

    def drift(self, f):
        """Volume minus upwind surface term of the DG transport operator."""
        out = []
        for bi, band in enumerate(self.mat.bands):
            m, v = self.mesh[bi], band.drift_velocity
            c = f[self.off[bi]:self.off[bi] + 3 * m.ne].reshape(-1, 3)
            if v[0] == 0.0 and v[1] == 0.0:
                out.append(torch.zeros(3 * m.ne, dtype=torch.float64, device=self.dev))
                continue
            e = torch.arange(m.ne, device=self.dev)
            odd = (e % 2) == 1
            x, y = [m.rel[i] + m.local[i] for i in range(2)]
            two_area = (x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) - (x[:, 2] - x[:, 0]) * (y[:, 1] - y[:, 0])
            zero = torch.zeros_like(two_area)
            gx = torch.stack([zero, (y[:, 2] - y[:, 0]) / two_area, -(y[:, 1] - y[:, 0]) / two_area], -1)
            gy = torch.stack([zero, -(x[:, 2] - x[:, 0]) / two_area, (x[:, 1] - x[:, 0]) / two_area], -1)
            mean = c[:, 0] * (3 * _GW) + (c[:, 1] + c[:, 2]) * ((2 * _GA + _GB) * _GW)
            r = m.vol * mean[:, None] * (v[0] * gx + v[1] * gy)
            sx, sy = torch.div(e, 2, rounding_mode="floor") % m.nx, torch.div(e, 2 * m.nx, rounding_mode="floor")
            element = lambda i, j, k: 2 * (i % m.nx + (j % m.ny) * m.nx) + k  # noqa: E731
            # face k joins vertices 1-2, 2-0 and 0-1 for k = 0, 1, 2; neighbours of even and odd elements
            across = [(element(sx + 1, sy, 1), element(sx, sy + 1, 0)),
                      (element(sx, sy, 1), element(sx, sy, 0)),
                      (element(sx, sy - 1, 1), element(sx - 1, sy, 0))]
            point = lambda k, g: ((1 - g, g), (0.0, g), (g, 0.0))[k]  # noqa: E731
            for k in range(3):
                i, j, o = (k + 1) % 3, (k + 2) % 3, k
                nx, ny = y[:, j] - y[:, i], x[:, i] - x[:, j]
                inward = (nx * (x[:, o] - x[:, i]) + ny * (y[:, o] - y[:, i])) > 0
                flux = (v[0] * nx + v[1] * ny) * torch.where(inward, -1.0, 1.0)   # velocity . normal x length
                nb = torch.where(odd, across[k][1], across[k][0])
                for g in _G1:
                    (a0, a1), (b0, b1) = point(k, g), point(2 - k, g)
                    own = c[:, 0] + c[:, 1] * a0 + c[:, 2] * a1
                    other = c[nb, 0] + c[nb, 1] * b0 + c[nb, 2] * b1
                    t = 0.5 * flux * torch.where(flux > 0, own, other)
                    r = r - t[:, None] * torch.tensor([1.0, a0, a1], dtype=torch.float64, device=self.dev)
            out.append(r.reshape(-1))
        return torch.cat(out)

    def inverse_mass(self, acc):
        return torch.cat([(acc[o:o + 3 * m.ne].reshape(-1, 3) @ m.minv).reshape(-1) for o, m in zip(self.off, self.mesh)])

    def rhs(self, f, amps=None):
        return self.inverse_mass(self.collisions(f, amps) + self.drift(f))

    # -- Dormand-Prince 5(4)
    def norm(self, err, p):
        worst = 0.0
        nodal = lambda x: torch.stack([x[:, 0], x[:, 1] + x[:, 0], x[:, 2] + x[:, 0]], -1)  # noqa: E731
        for b, o, m in zip(self.mat.bands, self.off, self.mesh):
            n, q = nodal(err[o:o + 3 * m.ne].reshape(-1, 3)), nodal(p[o:o + 3 * m.ne].reshape(-1, 3))
            scale = torch.minimum(q.abs(), (1.0 - q).abs()) if b.statistics < 0 else q
            n = n / (b.relativeErrorTolerance * scale + b.absoluteErrorTolerance)
            at = lambda x, y: n[:, 0] * (1 - x - y) + n[:, 1] * x + n[:, 2] * y  # noqa: E731
            sq = _GW * (at(_GA, _GA) ** 2 + at(_GB, _GA) ** 2 + at(_GA, _GB) ** 2)
            worst = max(worst, math.sqrt(float(sq.sum()) / m.ne))
        return worst

    def integrate(self, f, tf, dense, amps=None):
        """(y, dense outputs, attempts, accepted dt, (step, fraction) of the last output)."""
        rhs = lambda y: self.rhs(y, amps)  # noqa: E731
        t, dt, old, rejected, next_dense = 0.0, dense, 1.0, False, dense
        y, k1, outs, attempts, dts, last = f, rhs(f), [], 0, [], None
        dt = min(dt, (t + dt) - t)
        while t < tf:
            attempts += 1
            k = _stages(rhs, y, k1, dt)
            y5 = _combine(y, k, [dt * b for b in _B5])
            k.append(rhs(y5))
            err = self.norm(y5 - _combine(y, k, [dt * b for b in _B4]), y5)
            if err <= 1.0:
                while next_dense <= t + 1.0001 * dt and next_dense <= tf + .0001 * dt:
                    s = (next_dense - t) / dt
                    outs.append(_combine(y, k, [s * dt * b for b in _dense_weights(s)]))
                    last = (len(dts), s)
                    next_dense += dense
                t, y, k1 = t + dt, y5, k[6]
                dts.append(dt)
                scale = 3.0 if err == 0 else min(max(0.98 * (1 / err) ** (0.7 / 5) * old ** (0.4 / 5), 0.333333), 3.0)
                dt *= min(1.0, scale) if rejected else scale
                dt = min(dt, (t + dt) - t)
                rejected, old = False, err
            else:
                dt *= min(max(0.98 * (1 / err) ** (1 / 5.), 0.333333), 3.0)
                rejected = True
        return y, outs, attempts, dts, last


_A = [[], [1 / 5.], [3 / 40., 9 / 40.], [44 / 45., -56 / 15., 32 / 9.],
      [19372 / 6561., -25360 / 2187., 64448 / 6561., -212 / 729.],
      [9017 / 3168., -355 / 33., 46732 / 5247., 49 / 176., -5103 / 18656.]]
_B5 = [35 / 384., 0., 500 / 1113., 125 / 192., -2187 / 6784., 11 / 84.]
_B4 = [5179 / 57600., 0., 7571 / 16695., 393 / 640., -92097 / 339200., 187 / 2100., 1 / 40.]


def _dense_weights(s):
    return [-(435. * s ** 3 - 1184. * s ** 2 + 1098. * s - 384.) / 384., 0.,
            500. * s * (6. * s * s - 14. * s + 9.) / 1113., -125. * s * (9. * s * s - 16. * s + 6.) / 192.,
            729. * s * (35. * s * s - 64. * s + 26.) / 6784., -11. * s * (3. * s - 2.) * (5. * s - 6.) / 84.,
            s * (s - 1.) * (5. * s - 3.) / 2.]


def _combine(y, k, c):
    for kj, cj in zip(k, c):
        if cj != 0.0:
            y = y + cj * kj
    return y


def _stages(rhs, y, k1, dt):
    k = [k1]
    for row in _A[1:]:
        k.append(rhs(_combine(y, k, [dt * a for a in row])))
    return k


def _gradient(ref, case, f, amps, w):
    """Gradients of <w, f_obs> over the steps that the integration takes, step sizes held fixed: reverse over the
    steps, torch differentiating one right-hand side at a time."""
    with torch.no_grad():
        _, outs, _, dts, (m, s) = ref.integrate(f, case["t"], case["dense"])
        ys = [f]
        for dt in dts[:m]:
            ys.append(_combine(ys[-1], _stages(ref.rhs, ys[-1], ref.rhs(ys[-1]), dt), [dt * b for b in _B5]))

    def back(y, co):
        """(dF/dy)^T co and dF/damps . co"""
        with torch.enable_grad():
            a, b = y.detach().requires_grad_(), amps.detach().requires_grad_()
            return torch.autograd.grad(ref.rhs(a, b), (a, b), co)

    ga = torch.zeros_like(amps)
    lam = torch.zeros_like(f)
    for n in range(m, -1, -1):
        y, dt = ys[n], dts[n]
        with torch.no_grad():
            k, inp = [], []
            for i in range(6):
                inp.append(_combine(y, k, [dt * a for a in _A[i]]))
                k.append(ref.rhs(inp[-1]))
            inp.append(_combine(y, k, [dt * b for b in _B5]))
        # the co-states of the stages, from the next state (lam) and, in the last step, the observed output
        co = [dt * b * lam for b in _B5] + [torch.zeros_like(f)]
        if n == m:
            co = [x + s * dt * c * w for x, c in zip(co, _dense_weights(s))]
            lam = lam + w
        for i in range(6 if n == m else 5, -1, -1):
            nu, g = back(inp[i], co[i])
            lam, ga = lam + nu, ga + g
            for j, a in enumerate(_A[i] if i < 6 else _B5):
                co[j] = co[j] + dt * a * nu
    return {"observable": (w * outs[-1]).sum(), "f_obs": outs[-1], "grad_f": lam, "grad_amps": ga}


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    mats, states = _runs(case, seed)
    states = [torch.tensor(f, device=dev) for f in states]
    if case["path"] == "ensemble":
        refs, dense = {}, []
        for m, f in zip(mats, states):   # runs on the same mesh differ in their couplings and states only
            key = m.bands[0].mesh.nsplit
            if key not in refs:
                refs[key] = _Reference(m, dev).keep_points()
            amps = [c.amplitude for c in m.channels]
            dense += refs[key].integrate(f, case["t"], case["dense"], amps)[1]
        return {"dense": torch.cat(dense), "attempts": None}
    ref, f = _Reference(mats[0], dev), states[0]
    if case["path"] == "rhs":
        return ref.rhs(f)
    if case["path"] == "rates":
        return ref.inverse_mass(ref.collisions(f, rates=True))
    ref.keep_points()
    if case["path"] == "dp45":
        return {"dense": torch.stack(ref.integrate(f, case["t"], case["dense"])[1]), "attempts": None}
    amps = torch.tensor([c.amplitude for c in mats[0].channels], dtype=torch.float64, device=dev)
    w = torch.tensor(A.observable_weights(mats[0], 0, "energy"), device=dev)
    return _gradient(ref, case, f, amps, w)
