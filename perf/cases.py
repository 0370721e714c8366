"""The work that programs have this framework do, as cases that can be timed and compared.

A case is one simulation, one batch or one burst of requests through the public entry points:

  run       valomc_gb300.run(problem): host arrays in, fluence and exitance out, the equivalent
            of one MC2Dmex / MC3Dmex call or one run of the executables (mesh set-up included)
  resident  valomc_gb300.run_batch on one mesh that stays on the device
  batch     valomc_gb300.run_batch of several problems, each on its own resident mesh
  serve     a burst of requests to valomc_gb300.Server on resident meshes

in both forms (32: FP32 tracking, 64: plain FP64), continuous wave and frequency domain, on the
triangle and tetrahedron meshes that the benchmark, the tests and the examples use.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import valomc_gb300 as V
from valomc_gb300 import meshgen as mg

OUTPUTS = ("ER", "EI", "EBR", "EBI", "DEBR", "DEBI")


def _case(name, entry, mesh, photons, bits=32, nx=0, ny=0, nz=0, source="", hz=0.0, jobs=1):
    case = {"entry": entry, "mesh": mesh, "photons": photons, "bits": bits, "nx": nx, "ny": ny, "nz": nz,
            "source": source, "hz": hz, "jobs": jobs}
    return {"name": name, **case} if name else case


def listed():
    return [
        # the smallest call: a first look at the 10 x 10 mm square of the 2D example, 1e4 photons
        _case("square2d_1e4", "run", "square", 10_000, nx=10, ny=10, source="cosinic"),
        # the 2D example at the usual photon count, in the tracking form
        _case("square2d_1e6", "run", "square", 1_000_000, nx=10, ny=10, source="cosinic"),
        # the same in the reference's arithmetic
        _case("square2d_1e6_fp64", "run", "square", 1_000_000, bits=64, nx=10, ny=10, source="cosinic"),
        # two inclusions with index jumps on an uneven 2D mesh (as the NetGen example), modulated source
        _case("uneven2d_fd", "run", "uneven", 333_337, nx=57, source="gaussian", hz=100e6),
        # a quick preview on a small resident cube (48k tetrahedra): the smallest served request's size
        _case("cube20_1e5", "resident", "phantom", 100_000, nx=20, ny=20, nz=20, source="disk"),
        # one MEX-like call on the 648k-tetrahedron inclusion phantom, 1e6 photons, host arrays in and out
        _case("phantom_1e6_run", "run", "phantom", 1_000_000, nx=60, ny=60, nz=30, source="gaussian"),
        # a production run on the resident phantom
        _case("phantom_1e7", "resident", "phantom", 10_000_000, nx=60, ny=60, nz=30, source="gaussian"),
        # frequency domain on the phantom with per-tetrahedron optics
        _case("phantom_fd_1e6", "resident", "phantom", 1_000_000, nx=60, ny=60, nz=30, source="gaussian", hz=100e6),
        # the plain FP64 form on the phantom, as a check run beside the tracking form
        _case("phantom_1e5_fp64", "resident", "phantom", 100_000, bits=64, nx=60, ny=60, nz=30, source="gaussian"),
        # a small uneven tetrahedral mesh with an inclusion of another index, FP64, modulated source
        _case("jitter3d_fd_fp64", "run", "jitter", 30_011, bits=64, hz=100e6),
        # several instances of different size and optics in one launch
        _case("batch_cubes", "batch", "cubes", 2_000_000, nx=20, ny=48, jobs=10),
        # a burst of requests of mixed size on four resident cubes
        _case("serve_burst", "serve", "cubes", 1_000_000, nx=20, ny=44, jobs=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["2d", "2d", "3d", "3d", "3d", "batch", "serve"])
    bits = rng.choice([32, 32, 64])
    hz = rng.choice([0.0, 0.0, 100e6])
    if kind == "2d":
        photons = _log(rng, 1e4, 1e6 if bits == 32 else 2e5)
        source = rng.choice(["cosinic", "gaussian", "isotropic"])
        if rng.random() < 0.5:
            return _case("", "run", "square", photons, bits, rng.randint(5, 60), rng.randint(5, 60), 0, source, hz)
        return _case("", "run", "uneven", photons, bits, rng.randint(9, 80), 0, 0, source, hz)
    if kind == "3d":
        photons = _log(rng, 1e4, 3e6) if bits == 32 else _log(rng, 5e3, 6e4)
        return _case("", rng.choice(["run", "resident"]), "phantom", photons, bits, rng.randint(12, 60),
                     rng.randint(12, 60), rng.randint(10, 30), rng.choice(["gaussian", "disk", "pencil"]), hz)
    lo = rng.randint(12, 24)
    if kind == "batch":
        return _case("", "batch", "cubes", _log(rng, 1e5, 2e6), 32, lo, rng.randint(lo + 4, 48), 0, "", 0.0,
                     rng.randint(2, 10))
    return _case("", "serve", "cubes", _log(rng, 1e5, 1e6), 32, lo, rng.randint(lo + 4, 44), 0, "", 0.0,
                 rng.randint(4, 20))


# ---------------------------------------------------------------------------------------------
# problems
# ---------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def _geometry(mesh, nx, ny, nz):
    if mesh == "square":
        return mg.rectangular_mesh(nx, ny, 1)
    if mesh == "uneven":
        return mg.uneven_mesh_2d(nx, 10.0)
    if mesh == "jitter":
        p = mg.jittered_box_3d()
        return p.r, p.H, p.BH
    return mg.box_mesh_3d(nx, ny, nz)


def _two_circles(cen):
    return (np.hypot(cen[:, 0] + 2.0, cen[:, 1] + 1.5) < 1.6) | (np.hypot(cen[:, 0] - 2.2, cen[:, 1] - 1.8) < 1.2)


def _problem_2d(case, rng):
    r, H, BH = _geometry(case["mesh"], case["nx"], case["ny"], 0)
    ne, nb = len(H), len(BH)
    vary = rng.uniform(0.9, 1.1, 2)
    types = np.full(nb, ord("a"), np.uint8)
    if case["mesh"] == "square":
        mua, mus, g, n = (np.full(ne, v) for v in (0.01 * vary[0], 1.0 * vary[1], 0.9, 1.3))
        lit = (np.arange(nb) >= 3) & (np.arange(nb) < min(7, case["ny"]))
    else:
        inside = _two_circles(r[H].mean(axis=1))
        mua = np.where(inside, 0.09, 0.01) * vary[0]
        mus = np.full(ne, 1.3 * vary[1])
        g = np.where(inside, 0.5, 0.9)
        n = np.where(inside, 1.5, 1.3)
        lit = r[BH].mean(axis=1)[:, 0] < -5.0 + 1e-9
    types[lit] = ord({"cosinic": "c", "gaussian": "g", "isotropic": "i"}[case["source"]])
    return mg.Problem(dim=2, H=H, BH=BH, r=r, mua=mua, mus=mus, g=g, n=n, BCType=types, BCn=np.ones(nb),
                      GaussianSigma=np.full(nb, 0.2) if case["source"] == "gaussian" else None)


def _light(p, source, cx, cy):
    """Marks the source of a box problem around (cx, cy) on its z = 0 face."""
    if source == "gaussian":
        p.BCType, p.BCIntensity = mg.gaussian_footprint(p.r, p.BH, cx, cy, sigma=1.0)
    elif source == "disk":
        p.BCType = mg.cosinic_disk(p.r, p.BH, cx, cy, radius=1.0)
    else:  # a pencil beam entering at a point of a top triangle (its centroid)
        mid = p.r[p.BH].mean(axis=1)
        tri = int(np.argmin(np.where(mg.top_face_mask(p.r, p.BH), np.hypot(mid[:, 0] - cx, mid[:, 1] - cy), np.inf)))
        p.BCType = np.full(p.Nb, ord("a"), np.uint8)
        p.BCType[tri] = ord("p")
        p.BCLightDirectionType = np.full(p.Nb, ord("n"), np.uint8)
        p.BCLightDirectionType[tri] = ord("p")
        p.BCLNormal = np.zeros((p.Nb, 3))
        p.BCLNormal[tri] = mid[tri]
    return p


def _problem_3d(case, rng):
    if case["mesh"] == "jitter":
        p = mg.jittered_box_3d()
        vary = rng.uniform(0.9, 1.1, 2)
        p.mua, p.mus = p.mua * vary[0], p.mus * vary[1]
        return p
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r, H, BH = _geometry("phantom", nx, ny, nz)
    ne, nb = len(H), len(BH)
    vary = rng.uniform(0.9, 1.1, 2)
    if case["hz"] > 0:  # optics of every element drawn
        mua = rng.lognormal(math.log(0.01) - 0.045, 0.3, ne) * vary[0]
        mus = rng.uniform(8.0, 12.0, ne) * vary[1]
    else:
        ball = ((r[H].mean(axis=1) - [nx / 2.0, ny / 2.0, nz / 3.0]) ** 2).sum(1) < (nz / 6.0) ** 2
        mua = np.where(ball, 0.05, 0.01) * vary[0]
        mus = np.full(ne, 10.0 * vary[1])
    p = mg.Problem(dim=3, H=H, BH=BH, r=r, mua=mua, mus=mus, g=np.full(ne, 0.9), n=np.full(ne, 1.4),
                   BCType=np.zeros(nb, np.uint8), BCn=np.ones(nb))
    return _light(p, case["source"], nx / 2.0, ny / 2.0)


def _problem(case, seed):
    rng = np.random.default_rng([seed, 17])
    p = _problem_2d(case, rng) if case["mesh"] in ("square", "uneven") else _problem_3d(case, rng)
    p.f = float(case["hz"])
    p.Nphoton = int(case["photons"])
    p.seed, p.seedflag = int(rng.integers(1 << 31)), 1
    return p


def _edges(case):
    """Edges of the cubes of a batch (one per job) or of a server's four meshes."""
    count = case["jobs"] if case["entry"] == "batch" else 4
    return [int(round(v)) for v in np.geomspace(case["nx"], case["ny"], count)]


def _requests(case, seed):
    """(mesh index, problem) of every job: homogeneous optics and a source of its own each,
    photon counts spread over a factor of 20 up to the case's."""
    rng = np.random.default_rng([seed, 19])
    edges = _edges(case)
    counts = rng.permutation(np.geomspace(case["photons"] / 20, case["photons"], case["jobs"])).astype(int)
    out = []
    for i in range(case["jobs"]):
        k = i % len(edges)
        L = edges[k]
        r, H, BH = _geometry("phantom", L, L, L)
        ne, nb = len(H), len(BH)
        p = mg.Problem(dim=3, H=H, BH=BH, r=r, mua=np.full(ne, rng.uniform(0.005, 0.1)),
                       mus=np.full(ne, rng.uniform(5, 20)), g=np.full(ne, rng.uniform(0.8, 0.95)),
                       n=np.full(ne, rng.uniform(1.33, 1.45)), BCType=np.zeros(nb, np.uint8), BCn=np.ones(nb),
                       Nphoton=int(counts[i]), seed=int(rng.integers(1 << 31)), seedflag=1)
        source = "pencil" if case["entry"] == "batch" else ("disk", "gaussian")[int(rng.integers(2))]
        out.append((k, _light(p, source, rng.uniform(0.5, L - 0.5), rng.uniform(0.5, L - 0.5))))
    return out


def prepare(case, seed):
    bits = V.VMC_FP64 if case["bits"] == 64 else V.VMC_FP32
    state = {"case": case, "precision": bits}
    if case["entry"] in ("run", "resident"):
        state["problem"] = _problem(case, seed)
        if case["entry"] == "resident":
            state["mesh"] = V.Mesh(state["problem"], precision=bits)
        return state
    jobs = _requests(case, seed)
    state["problems"] = [p for _, p in jobs]
    first = {}
    for k, p in jobs:
        first.setdefault(k, p)
    meshes = {k: V.Mesh(p, precision=bits) for k, p in first.items()}
    if case["entry"] == "batch":
        state["meshes"] = [meshes[k] for k, _ in jobs]
    else:
        state["server"] = V.Server(precision=bits, max_slots=32)
        ids = {k: state["server"].add_mesh(m) for k, m in meshes.items()}
        state["ids"] = [ids[k] for k, _ in jobs]
    return state


def _fields(result, names=OUTPUTS):
    return {k: getattr(result, k) for k in names}


def run(state):
    entry = state["case"]["entry"]
    if entry == "run":
        return _fields(V.run(state["problem"], precision=state["precision"]))
    if entry == "resident":
        results, _ = V.run_batch([state["mesh"]], [state["problem"]], precision=state["precision"])
        return _fields(results[0])
    # the boxes of a batch and of a burst run in continuous wave: their imaginary parts are zero
    if entry == "batch":
        results, _ = V.run_batch(state["meshes"], state["problems"], precision=state["precision"])
        return [_fields(r, ("ER", "EBR")) for r in results]
    server = state["server"]
    tickets = [server.submit(k, p) for k, p in zip(state["ids"], state["problems"])]
    return [_fields(server.wait(t), ("ER", "EBR")) for t in tickets]


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------

def _steps_per_photon(dim, edge, cell, mua, mus, g):
    """Element steps of a photon: its path until it is absorbed or has left a body of thickness
    `edge`, times the scatters and the faces crossed per mm (7.6 faces per mm of a 1 mm grid of
    tetrahedra, 2.2 of triangles).  Gives 1420 for the phantom and 32 for the square, which are
    measured."""
    leave = 1.0 / (0.6 * edge * (1.0 + 0.75 * mus * (1.0 - g) * edge))
    return (mus + (7.6 if dim == 3 else 2.2) / cell) / (mua + leave)


def _body(case):
    """(dimension, thickness, cell size, elements, mua, mus, g) of a one-problem case."""
    if case["mesh"] == "square":
        return 2, min(case["nx"], case["ny"]), 1.0, 2 * case["nx"] * case["ny"], 0.01, 1.0, 0.9
    if case["mesh"] == "uneven":
        return 2, 10.0, 10.0 / case["nx"], 2 * case["nx"] ** 2, 0.02, 1.3, 0.85
    if case["mesh"] == "jitter":
        return 3, 6.0, 1.0, 2304, 0.03, 5.8, 0.84
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return 3, min(nx, ny, nz), 1.0, 6 * nx * ny * nz, 0.01, 10.0, 0.9


def work(case):
    """Bytes: nodes of the elements, their neighbours and optics read once, the outputs written
    once.  Operations: per element step the distances to all faces (7 per coordinate and face),
    the advance, the deposit and the crossing (about 25), and for the scatters among them the
    sampled angles and the rotation (about 60, half of the steps)."""
    if case["entry"] in ("run", "resident"):
        bodies = [(_body(case), case["photons"])]
    else:
        edges = _edges(case)
        counts = np.geomspace(case["photons"] / 20, case["photons"], case["jobs"])
        bodies = [((3, edges[i % len(edges)], 1.0, 6 * edges[i % len(edges)] ** 3, 0.05, 12.0, 0.88), float(c))
                  for i, c in enumerate(counts)]
    nbytes = flops = 0.0
    word = 8 if case["bits"] == 64 else 4
    for (dim, edge, cell, ne, mua, mus, g), photons in bodies:
        steps = photons * _steps_per_photon(dim, edge, cell, mua, mus, g)
        nbytes += ne * ((dim + 1) * (dim * word + 4) + 4 * word + 16)
        flops += steps * ((dim + 1) * 7 * dim + 25 + 30 + (20 if case["hz"] > 0 else 0))
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------------------------
# 64-bit values, in plain torch
# ---------------------------------------------------------------------------------------------

def exact(case, seed):
    """The photons of a plain FP64 run followed one element step at a time in float64 tensors,
    from the same counter-based uniforms.  None for the FP32 form, whose walks leave these at the
    first rounded draw, and where the walk takes too long this way (the large boxes)."""
    if case["bits"] != 64 or case["entry"] != "run" or case["mesh"] not in ("square", "uneven", "jitter"):
        return None
    if case["source"] not in ("", "cosinic", "isotropic"):
        return None
    return _Walk(_problem(case, seed)).outputs()


M32 = 0xFFFFFFFF


def _mul32(a, b):
    """(high, low) 32-bit words of the product of the 32-bit values in a (int64 tensor) and b."""
    t = a * (b & 0xFFFF)                 # below 2^48
    u = a * (b >> 16) + (t >> 16)        # below 2^49
    return (u >> 16) & M32, ((u & 0xFFFF) << 16) | (t & 0xFFFF)


def _philox(key, photon, block):
    """Philox4x32-10 of the counters (photon low, photon high, block, 0)."""
    x = [photon & M32, photon >> 32, block, torch.zeros_like(photon)]
    a, b = key & M32, (key >> 32) & M32
    for _ in range(10):
        hi0, lo0 = _mul32(x[0], 0xD2511F53)
        hi1, lo1 = _mul32(x[2], 0xCD9E8D57)
        x = [hi1 ^ x[1] ^ a, lo1, hi0 ^ x[3] ^ b, lo0]
        a, b = (a + 0x9E3779B9) & M32, (b + 0xBB67AE85) & M32
    return torch.stack(x, 1)


class _Walk:
    """All photons of a problem, advanced together."""

    def __init__(self, p):
        self.p, self.dim = p, p.dim
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        D = self.dim
        self.faces = [(0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3)] if D == 3 else [(0, 1), (1, 2), (2, 0)]
        self.HN = self._neighbours()
        put = lambda a, t=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device=self.dev)  # noqa: E731
        self.vert = put(p.r[p.H])
        self.nbr = put(self.HN, torch.int64)
        self.opt = put(np.stack([p.mua, p.mus, p.g, p.n], 1))
        self.bcn = put(p.BCn)
        self.omega_c = 2.0 * math.pi * p.f / 2.99792458e11
        self.fd = p.f > 0
        self.sums = {k: torch.zeros(p.Ne if k in ("ER", "EI") else p.Nb, dtype=torch.float64, device=self.dev)
                     for k in OUTPUTS}

    def _neighbours(self):
        """Element or -1 - boundary element behind each face."""
        p, D = self.p, self.dim
        nf = len(self.faces)
        of = np.concatenate([np.sort(p.H[:, f], axis=1) for f in self.faces] + [np.sort(p.BH, axis=1)])
        _, key = np.unique(of, axis=0, return_inverse=True)
        order = np.argsort(key, kind="stable")
        owner = np.concatenate([np.tile(np.arange(p.Ne), nf), -1 - np.arange(p.Nb)])
        pairs = order.reshape(-1, 2)  # every face has two sides in a closed mesh
        other = np.empty(len(of), np.int64)
        other[pairs[:, 0]], other[pairs[:, 1]] = owner[pairs[:, 1]], owner[pairs[:, 0]]
        return other[: nf * p.Ne].reshape(nf, p.Ne).T

    def _measure(self, nodes):
        """Length / area / volume of the simplices with these nodes."""
        e = self.p.r[nodes[:, 1:]] - self.p.r[nodes[:, :1]]
        return np.sqrt(np.linalg.det(e @ e.transpose(0, 2, 1))) / math.factorial(nodes.shape[1] - 1)

    def _sources(self):
        p, D = self.p, self.dim
        el, f = np.nonzero((self.HN < 0) & np.isin(p.BCType[np.maximum(0, -1 - self.HN)], [ord(c) for c in "lci"]))
        ib = -1 - self.HN[el, f]
        w = self._measure(p.BH)[ib] * (1.0 if p.BCIntensity is None else p.BCIntensity[ib])
        cdf = np.cumsum(w)
        e = p.r[p.BH[ib]]
        if D == 3:
            n = np.cross(e[:, 1] - e[:, 0], e[:, 2] - e[:, 0])
        else:
            d = e[:, 1] - e[:, 0]
            n = np.stack([d[:, 1], -d[:, 0]], 1)
        n /= np.linalg.norm(n, axis=1, keepdims=True)
        inward = p.r[p.H[el]].mean(axis=1) - e.mean(axis=1)
        n *= np.where((n * inward).sum(1) < 0, -1.0, 1.0)[:, None]
        return el, f, e, n, cdf / cdf[-1], p.BCType[ib]

    # ---- uniforms: words of blocks 0, 1, ... of each photon's counter ----
    def _word(self, m):
        """The next word of the photons in m (indices)."""
        dry = m[self.left[m] == 0]
        if len(dry):
            self.buf[dry] = _philox(int(self.p.seed), self.ph[dry], self.block[dry])
            self.block[dry] += 1
            self.left[dry] = 4
        w = self.buf[m, 4 - self.left[m]]
        self.left[m] -= 1
        return w.double()

    def _closed(self, m):
        return self._word(m) / 4294967295.0

    def _open(self, m):
        return (self._word(m) + 0.5) / 4294967296.0

    def _half(self, m):
        return self._word(m) / 4294967296.0

    def _launch(self):
        p, D, dev = self.p, self.dim, self.dev
        N = p.Nphoton
        self.ph = torch.arange(N, device=dev)
        self.block = torch.zeros(N, dtype=torch.int64, device=dev)
        self.left = torch.zeros(N, dtype=torch.int64, device=dev)
        self.buf = torch.zeros(N, 4, dtype=torch.int64, device=dev)
        every = torch.arange(N, device=dev)
        el, f, e, n, cdf, kind = (torch.as_tensor(a, device=dev) for a in self._sources())
        s = torch.searchsorted(cdf, self._closed(every), right=True).clamp(max=len(cdf) - 1)
        self.el, self.face = el[s], f[s]
        r1 = self._open(every)
        if D == 3:
            r2, sr = self._open(every), r1.sqrt()
            self.pos = ((1.0 - sr)[:, None] * e[s, 0] + (sr * (1.0 - r2))[:, None] * e[s, 1]
                        + (sr * r2)[:, None] * e[s, 2])
            self.dir = n[s].clone()
        else:
            self.pos = e[s, 0] + r1[:, None] * (e[s, 1] - e[s, 0])
            phi = torch.where(kind[s] == ord("c"), 0.0, 1.0)
            u = self._open(every)
            phi = torch.atan2(n[s, 1], n[s, 0]) + torch.where(phi == 0.0, torch.asin(2.0 * u - 1.0), math.pi * (u - 0.5))
            self.dir = torch.stack([phi.cos(), phi.sin()], 1)
        self.w = torch.ones(N, dtype=torch.float64, device=dev)
        self.phase = torch.zeros(N, dtype=torch.float64, device=dev)
        self.prop = -torch.log(self._open(every)) / self.opt[self.el, 1]

    def _exit(self):
        """Distance to and number of the face that each photon leaves its element through: the
        first in order that its ray meets ahead of it, other than the face it stands on."""
        V, D = self.vert[self.el], self.dim
        dist = torch.zeros_like(self.w)
        nf = torch.full_like(self.el, -1)
        for f, fv in enumerate(self.faces):
            a = V[:, fv[0]]
            if D == 3:
                e1, e2 = V[:, fv[1]] - a, V[:, fv[2]] - a
                pv = torch.linalg.cross(self.dir, e2)
                det = (e1 * pv).sum(1)
                tv = self.pos - a
                u = (tv * pv).sum(1) / det
                qv = torch.linalg.cross(tv, e1)
                v = (self.dir * qv).sum(1) / det
                t = (e2 * qv).sum(1) / det
                hit = (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1)
            else:
                d, b = self.dir, V[:, fv[1]]
                det = d[:, 0] * (a[:, 1] - b[:, 1]) - d[:, 1] * (a[:, 0] - b[:, 0])
                q = self.pos - a
                s = (d[:, 1] * q[:, 0] - d[:, 0] * q[:, 1]) / det
                t = (q[:, 1] * (a[:, 0] - b[:, 0]) - q[:, 0] * (a[:, 1] - b[:, 1])) / det
                hit = (s >= 0) & (s <= 1)
            hit &= (det.abs() >= 2.220446049250313e-16) & (t > 0) & (self.face != f) & (nf < 0)
            dist, nf = torch.where(hit, t, dist), torch.where(hit, f, nf)
        return dist, nf

    def _normal(self, m, f):
        V = self.vert[self.el[m]]
        idx = torch.tensor(self.faces, device=self.dev)[f]
        a = V[torch.arange(len(m), device=self.dev)[:, None], idx]
        if self.dim == 3:
            n = torch.linalg.cross(a[:, 1] - a[:, 0], a[:, 2] - a[:, 0])
        else:
            d = a[:, 1] - a[:, 0]
            n = torch.stack([d[:, 1], -d[:, 0]], 1)
        return n / n.norm(dim=1, keepdim=True)

    def _fresnel(self, m, nf, eta, boundary):
        """Reflects or refracts the photons m at their face nf; True where reflected."""
        if not len(m):
            return torch.zeros(0, dtype=torch.bool, device=self.dev)
        nor = self._normal(m, nf)
        ci = -(self.dir[m] * nor).sum(1)
        s = 1.0 - eta * eta * (1.0 - ci * ci)
        ct = s.clamp(min=0).sqrt()
        thi, tht = ci.abs().acos(), ct.acos()
        sp = (thi + tht).sin()
        flat = ((eta - 1.0) / (eta + 1.0)) ** 2
        R = torch.where(sp > 2.220446049250313e-16,
                        0.5 * (((thi - tht).sin() / sp) ** 2 + ((thi - tht).tan() / (thi + tht).tan()) ** 2), flat)
        refl = s <= 0.0
        ask = torch.nonzero(~refl).flatten()
        refl[ask] = self._closed(m[ask]) <= R[ask]
        back = self.dir[m] + 2.0 * ci[:, None] * nor
        k = eta * ci - torch.copysign(ct, ci)
        on = self.dir[m] if boundary and self.dim == 2 else eta[:, None] * self.dir[m] + k[:, None] * nor
        self.dir[m] = torch.where(refl[:, None], back, on)
        self.face[m[refl]] = nf[refl]
        return refl

    def _scatter(self, m):
        if not len(m):
            return
        g, d = self.opt[self.el[m], 2], self.dir[m]
        if self.dim == 2:
            th = 2.0 * torch.atan(torch.tan(math.pi * self._half(m)) * (1.0 - g) / (1.0 + g))
            d = d / d.norm(dim=1, keepdim=True)
            c, s = th.cos(), th.sin()
            self.dir[m] = torch.stack([d[:, 0] * c - d[:, 1] * s, d[:, 1] * c + d[:, 0] * s], 1)
        else:
            q = (1.0 - g * g) / (1.0 - g * (1.0 - 2.0 * self._closed(m)))
            ct = (1.0 + g * g - q * q) / (2.0 * g)
            st = (1.0 - ct * ct).sqrt()
            phi = 2.0 * math.pi * self._closed(m)
            cp, sp = phi.cos(), phi.sin()
            x, y, z = d.unbind(1)
            sq = (1.0 - z * z).clamp(min=0).sqrt()
            new = torch.stack([st * (x * z * cp - y * sp) / sq + x * ct, st * (y * z * cp + x * sp) / sq + y * ct,
                               -st * cp * sq + z * ct], 1)
            new = torch.where((z.abs() > 0.999)[:, None], torch.stack([st * cp, st * sp, ct * z.sign()], 1), new)
            self.dir[m] = new / new.norm(dim=1, keepdim=True)

    def _keep(self, alive):
        for k in ("ph", "block", "left", "buf", "el", "face", "pos", "dir", "w", "phase", "prop"):
            setattr(self, k, getattr(self, k)[alive])

    def _step(self):
        S = self.sums
        dist, nf = self._exit()
        if bool((nf < 0).any()):  # lost at an edge by rounding
            self._keep(nf >= 0)
            return
        mua, mus, _, n = self.opt[self.el].unbind(1)
        ds = torch.minimum(self.prop, dist)
        self.pos = self.pos + self.dir * ds[:, None]
        att = torch.exp(-mua * ds)
        if self.fd:
            ph = self.phase + self.omega_c * n * ds
            S["ER"].index_add_(0, self.el, self.w * (self.phase.cos() - ph.cos() * att))
            S["EI"].index_add_(0, self.el, self.w * (-self.phase.sin() + ph.sin() * att))
            self.phase = ph
        else:
            S["ER"].index_add_(0, self.el, torch.where(mua > 0, -torch.expm1(-mua * ds) * self.w, self.w * ds))
        self.w = self.w * att
        self.prop = self.prop - ds
        stay = self.prop <= 0.0
        m = torch.nonzero(stay).flatten()
        self.left[m] = 0  # every scatter takes its words from a new block
        self._scatter(m)
        self.face[m] = -1
        self.prop[m] = -torch.log(self._open(m)) / mus[m]
        nxt = self.nbr[self.el, nf.clamp(min=0)]
        dead = torch.zeros_like(stay)
        # boundary: reflected, or out
        m = torch.nonzero(~stay & (nxt < 0)).flatten()
        ib = -1 - nxt[m]
        refl = self._fresnel(m, nf[m], n[m] / self.bcn[ib], True)
        m, ib = m[~refl], ib[~refl]
        dead[m] = True
        c, s = (self.phase[m].cos(), -self.phase[m].sin()) if self.fd else (1.0, None)
        S["EBR"].index_add_(0, ib, self.w[m] * c)
        if self.fd:
            S["EBI"].index_add_(0, ib, self.w[m] * s)
        if self.dim == 2 and len(m):
            nor = self._normal(m, nf[m])
            inside = self.vert[self.el[m]].mean(1) - self.pos[m]
            dn = (self.dir[m] * nor).sum(1) * torch.where((nor * inside).sum(1) > 0, -1.0, 1.0)
            S["DEBR"].index_add_(0, ib, self.w[m] * c / dn)
            if self.fd:
                S["DEBI"].index_add_(0, ib, self.w[m] * s / dn)
        # the next element: roulette, then its interface
        m = torch.nonzero(~stay & (nxt >= 0)).flatten()
        low = m[self.w[m] < 0.001]
        out = self._closed(low) > 0.1
        dead[low[out]] = True
        self.w[low[~out]] = self.w[low[~out]] / 0.1
        m = m[~dead[m]]
        n2 = self.opt[nxt[m], 3]
        jump = n[m] != n2
        refl = torch.zeros_like(jump)
        refl[jump] = self._fresnel(m[jump], nf[m[jump]], (n[m] / n2)[jump], False)
        m = m[~refl]
        self.prop[m] = self.prop[m] * (mus[m] / self.opt[nxt[m], 1])
        came = self.el[m]
        self.el[m] = nxt[m]
        self.face[m] = (self.nbr[nxt[m]] == came[:, None]).int().argmax(1)
        if bool(dead.any()):
            self._keep(~dead)

    def outputs(self):
        p = self.p
        self._launch()
        while len(self.ph):
            self._step()
        put = lambda a: torch.as_tensor(a, dtype=torch.float64, device=self.dev)  # noqa: E731
        vol, area, N = put(self._measure(p.H)), put(self._measure(p.BH)), float(p.Nphoton)
        S, mua = self.sums, self.opt[:, 0]
        if self.fd:
            k = self.omega_c * self.opt[:, 3]
            er = (S["EI"] * k + S["ER"] * mua) / (k * k + mua * mua) / N / vol
            ei = -(S["ER"] * k - S["EI"] * mua) / (k * k + mua * mua) / N / vol
        else:
            er, ei = S["ER"] / torch.where(mua > 0, mua, 1.0) / N / vol, S["EI"]
        out = {"ER": er, "EI": ei}
        for key in ("EBR", "EBI", "DEBR", "DEBI"):
            out[key] = S[key] / (N * area)
        return {k: v.cpu().numpy() for k, v in out.items()}
