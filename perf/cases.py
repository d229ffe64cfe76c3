"""The work that users of the library have it do, as measurable cases.

A case is one call pattern of a user's program (mr-lbm_b200/mrlbm.py): a
domain set up from host fields, then one pass = one `step(n)` call (or a whole
job with its transfers).  The outputs of a stepping pass are the domain's own
moments on the device, viewed through the plane pointers that the library
hands out (mrlbm_zslab_plane): moment pair p is a plane stack
[z][y + 1][x + 4][2] of the buffer that the next step reads.

`exact` is a plain torch restatement in 64 bits of the same time steps:
regularised reconstruction, streaming, lattice sums, the moment-space wall
system, power-law / Bingham viscosity, the thermal scalar on D3G19.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "mr-lbm_b200"))
import mrlbm  # noqa: E402

X_OFFSET = 4  # padded column of x = 0 (csrc/domain.h)
STORAGE = {"f32": mrlbm.F32, "f16": mrlbm.F16, "bf16": mrlbm.BF16, "f16u": mrlbm.F16U}
TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
BATCH_MEMBERS = 40


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # one step per call on a small lid cavity: a program that couples the
        # flow to something else after every step (launch latency)
        dict(name="cavity32_q19_step1", kind="cavity", nx=32, ny=32, nz=32, q=19, storage="f32", steps=1),
        # the shipped lid-driven cavity (64^3, D3Q19), stepped between reports
        dict(name="cavity64_q19", kind="cavity", nx=64, ny=64, nz=64, q=19, storage="f32", steps=50),
        # a resolved lid cavity, walls on six faces
        dict(name="cavity128_q19", kind="cavity", nx=128, ny=128, nz=128, q=19, storage="f32", steps=20),
        # the headline: the periodic vortex box of bench.py
        dict(name="vortex256_q27", kind="vortex", nx=256, ny=256, nz=256, q=27, storage="f32", steps=10),
        # a periodic box with ragged sides on the smaller lattice
        dict(name="vortex_ragged_q19", kind="vortex", nx=203, ny=173, nz=121, q=19, storage="f32", steps=20),
        # the 512^3 box of the storage-precision study, 16-bit moments
        dict(name="vortex512_q27_f16", kind="vortex", nx=512, ny=512, nz=512, q=27, storage="f16", steps=3),
        # velocity inlet, no-slip sides, outflow outlet (mounted-cube kind of case)
        dict(name="channel_q27", kind="channel", nx=96, ny=80, nz=180, q=27, storage="f32", steps=20),
        # power-law duct with 5 % scattered obstacles, driven by a force
        dict(name="duct128_powerlaw", kind="duct", nx=128, ny=128, nz=128, q=19, storage="f32", steps=10),
        # one served request: a split-fp16 duct advanced, then its fields read
        dict(name="served_duct72_f16u", kind="served", nx=72, ny=72, nz=72, q=19, storage="f16u", steps=200),
        # Rayleigh-Benard cell: thermal scalar, hot and cold walls in x
        dict(name="thermal160_q19", kind="thermal", nx=160, ny=160, nz=160, q=19, storage="f32", steps=10),
        # many lid cavities of uneven sizes advanced together
        dict(name="batch40_cavities_f16", kind="batch", nx=24, ny=24, nz=96, q=19, storage="f16", steps=16),
        # a whole job from and to host memory, with kinetic-energy reports
        dict(name="job128_q27", kind="job", nx=128, ny=128, nz=128, q=27, storage="f32", steps=100),
    ]


def _edge(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vortex", "vortex", "vortex", "cavity", "cavity", "cavity", "channel", "duct", "plates", "served",
                       "thermal", "batch", "job"])
    hi = {"vortex": 340, "cavity": 256, "channel": 180, "duct": 160, "plates": 160, "served": 96, "thermal": 200,
          "batch": 96, "job": 144}[kind]
    lo = 32 if kind != "batch" else 24
    c = dict(kind=kind, nx=_edge(rng, lo, hi), ny=_edge(rng, lo, hi), nz=_edge(rng, lo, hi))
    c["q"] = rng.choice([19, 27]) if kind in ("vortex", "cavity", "channel", "job") else 19
    c["storage"] = {"vortex": rng.choice(["f32", "f32", "f16", "bf16"]), "cavity": rng.choice(["f32", "f32", "f16"]),
                    "served": "f16u", "batch": rng.choice(["f32", "f16"])}.get(kind, "f32")
    if kind == "batch":  # nx .. nz are the smallest and the largest edge of the members
        c["nx"] = c["ny"] = min(c["nx"], c["nz"])
        c["nz"] = max(c["nx"] + 8, c["nz"])
    if kind == "job":    # the reference's layout wants multiples of 8
        for a in ("nx", "ny", "nz"):
            c[a] = (c[a] + 7) // 8 * 8
    if kind == "vortex":
        c["force"] = rng.random() < 0.25
    n = c["nx"] * c["ny"] * c["nz"]
    c["steps"] = {"served": 200, "job": 100, "batch": 16}.get(kind) or max(1, min(60, int(8e7 / n)))
    if kind == "cavity" and rng.random() < 0.2:
        c["steps"] = 1
    return c


def _fluid_nodes(c):
    return c["nx"] * c["ny"] * c["nz"]


def _moments(c):
    return 14 if c["kind"] == "thermal" else 11 if c["kind"] in ("duct", "served", "plates") else 10


def work(case):
    """Every step reads and writes each node's moments once (and its class
    byte where there are walls); a job or a served request also writes the
    fields it returns (and reads those it starts from)."""
    nm = _moments(case)
    words = nm + (4 if case["storage"] == "f16u" else 0)
    size = 4 if case["storage"] == "f32" else 2
    walls = case["kind"] not in ("vortex", "job")
    nodes = _fluid_nodes(case)
    if case["kind"] == "batch":
        nodes = sum(int(np.prod(s)) for s, _ in _batch_members(case, 0))
    b = case["steps"] * nodes * (2 * words * size + (1 if walls else 0))
    if case["kind"] == "served":
        b += nodes * nm * 4
    if case["kind"] == "job":
        b += 2 * nodes * nm * 4
    flops = case["steps"] * nodes * (300 if case["q"] == 27 else 220)
    return {"bytes": b, "flops": flops * (2 if case["kind"] == "thermal" else 1)}


def tolerance(case):
    """About four times the largest difference measured between the path and
    `exact`.  32-bit moments: 2e-5 to 8e-5 (sums of O(1) populations rounded
    into second moments of O(u^2)), 1.4e-4 in the omega iteration's second
    moments.  16-bit moments carry their own rounding: 6e-4 in a cavity from a
    uniform start, 1e-2 in the small density waves of a box; split fp16 2e-3
    after 200 steps of a power-law duct."""
    if case["storage"] == "f16u":
        return {"rel": 8e-3}
    if case["storage"] != "f32":
        return {"rel": 3e-3 if case["kind"] == "batch" else 3e-2}
    return {"rel": 6e-4 if case["kind"] in ("duct", "plates") else 4e-4}


# --------------------------------------------------------------------- inputs

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _rand(seed, *salt):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, *salt])


def _modes(case, seed, dtype=torch.float32):
    """rho, ux, uy, uz (z, y, x) float32: a mean flow plus a few smooth
    divergence-free waves of the box, density waves of O(u^2)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = _rand(seed, 1)
    dev = _device()
    ax = [torch.arange(n, device=dev, dtype=torch.float64) * (2 * math.pi / n) for n in (nx, ny, nz)]
    mean = 0.004 * r.uniform(0.5, 1.0, 3)
    out = [torch.full((nz, ny, nx), float(v), device=dev, dtype=torch.float32) for v in (1.0, *mean)]
    for _ in range(4):
        k = r.integers(1, 4, 3) * r.choice([-1, 1], 3)
        kk = np.array([k[0] / nx, k[1] / ny, k[2] / nz])
        d = np.cross(kk, r.normal(size=3))
        d *= 0.012 / np.linalg.norm(d)
        ph = r.uniform(0, 2 * math.pi)
        # cos(a + b + c) as a product form: two outer products, no 64-bit field
        e = [torch.exp(1j * float(k[a]) * ax[a]).to(torch.complex64) for a in range(3)]
        plane = (e[1][:, None] * e[0][None, :]) * complex(math.cos(ph), math.sin(ph))
        cosz, sinz = e[2].real[:, None, None], e[2].imag[:, None, None]
        for a in range(3):
            out[1 + a] += float(d[a]) * (plane.real * cosz - plane.imag * sinz)
        out[0] += 2e-4 * (plane.imag * cosz + plane.real * sinz)
    return out


def _host(t):
    return t.cpu().numpy()


def _lid(case, seed):
    r = _rand(seed, 2)
    re = r.uniform(50.0, 1000.0)
    return float(r.uniform(0.03, 0.05)), float(re)


def _solid(case, seed):
    """5 % scattered obstacles on the interior of the duct's cross-section."""
    r = _rand(seed, 3)
    s = np.zeros((case["nz"], case["ny"], case["nx"]), dtype=np.uint8)
    s[:, 1:-1, 1:-1] = r.random((case["nz"], case["ny"] - 2, case["nx"] - 2), dtype=np.float32) < 0.05
    return s


def _faces(case, axes):
    """Octant masks of the domain's faces on the given axes (0, 1, 2 = x, y, z)."""
    lo, hi = (mrlbm.WEST, mrlbm.SOUTH, mrlbm.BACK), (mrlbm.EAST, mrlbm.NORTH, mrlbm.FRONT)
    t = np.zeros((case["nz"], case["ny"], case["nx"]), dtype=np.uint32)
    for a in axes:
        v = [slice(None)] * 3
        v[2 - a] = 0
        t[tuple(v)] |= lo[a]
        v[2 - a] = -1
        t[tuple(v)] |= hi[a]
    return t


def _setup(case, seed):
    """(descriptor, node types or None, initial fields or None for rest)."""
    kind, q, st = case["kind"], case["q"], STORAGE[case["storage"]]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if kind in ("vortex", "job"):
        r = _rand(seed, 4)
        f = tuple(float(v) for v in 1e-6 * r.uniform(0.5, 1.0, 3)) if case.get("force") else (0.0, 0.0, 0.0)
        return mrlbm.make_desc(nx, ny, nz, lattice=q, storage=st, tau=float(r.uniform(0.51, 0.6)), force=f), None, True
    if kind == "cavity":
        lid, re = _lid(case, seed)
        d = mrlbm.lid_cavity_desc(nx, re=re, lid_u=lid, storage=st, lattice=q, ny=ny, nz=nz)
        return d, mrlbm.lid_cavity_node_types(nx, ny, nz, 1), True
    if kind == "channel":
        t = _faces(case, (0, 1))
        inside = t[0] == 0
        zf = (mrlbm.BACK, mrlbm.FRONT)
        for k, z in enumerate((0, -1)):
            t[z][~inside] |= zf[k]
        t[0][inside] = mrlbm.BACK | mrlbm.BC_VELOCITY_WALL | mrlbm.BC_VELOCITY_INDEX(0)
        t[-1][inside] = mrlbm.FRONT | mrlbm.BC_OUTFLOW
        u = float(_rand(seed, 5).uniform(0.02, 0.03))
        return mrlbm.make_desc(nx, ny, nz, lattice=q, storage=st, periodic=(0, 0, 0), tau=0.7,
                               bc_velocity=[(0.0, 0.0, u)]), t, "along z"
    if kind in ("duct", "served"):
        n = float(_rand(seed, 6).uniform(0.8, 1.2))
        h = min(nx, ny) - 1
        f = 0.05 * 0.1 / (0.0737 * h * h)
        d = mrlbm.make_desc(nx, ny, nz, lattice=q, storage=st, periodic=(0, 0, 1), tau=0.8, force=(0.0, 0.0, f),
                            rheology=mrlbm.POWERLAW, nnf_n=n)
        return d, mrlbm.voxel_node_types(_solid(case, seed), (0, 0, 1)), "along z"
    if kind == "plates":
        d = mrlbm.make_desc(nx, ny, nz, lattice=q, storage=st, periodic=(1, 0, 1), tau=0.6, force=(0.0, 0.0, 2e-6),
                            rheology=mrlbm.BINGHAM, nnf_yield=float(_rand(seed, 7).uniform(0.5, 1.0)) * 1e-6)
        return d, _faces(case, (1,)), True
    if kind == "thermal":
        r = _rand(seed, 8)
        tau = 0.55
        nu = (tau - 0.5) / 3
        alpha = nu / 10.0
        gb = 1e5 * alpha * nu / nx ** 3
        th = dict(diffusivity=alpha, reference=1.0, gravity_beta=(gb, 0.0, 0.0),
                  wall=(float(r.uniform(1.3, 1.5)), float(r.uniform(0.5, 0.7))))
        t = np.zeros((nz, ny, nx), dtype=np.uint32)
        rule = mrlbm.THERMAL_RULE(mrlbm.THERMAL_DIRICHLET_FLUX)
        t[:, :, 0] = mrlbm.WEST | rule | mrlbm.THERMAL_INDEX(0)
        t[:, :, -1] = mrlbm.EAST | rule | mrlbm.THERMAL_INDEX(1)
        return mrlbm.make_desc(nx, ny, nz, lattice=q, storage=st, periodic=(0, 1, 1), tau=tau, thermal=th), t, True
    raise ValueError(kind)


def _fields(case, seed, how):
    f = _modes(case, seed)
    if how == "along z":  # a channel's or duct's flow is mostly along it
        f[3] += 0.01
    return f


def _batch_members(case, seed):
    """(nx, ny, nz) and Reynolds number of each member: the sizes are the
    case's, the Reynolds numbers the seed's."""
    r = np.random.default_rng([77, case["nx"], case["nz"]])
    re = _rand(seed, 9).uniform(50.0, 1000.0, BATCH_MEMBERS)
    sizes = r.integers(case["nx"], case["nz"] + 1, size=(BATCH_MEMBERS, 3))
    return [(tuple(int(v) for v in s), float(e)) for s, e in zip(sizes, re)]


# ------------------------------------------------- device views of the moments

class _Bytes:
    """A range of a domain's device memory; keeps the domain alive."""

    def __init__(self, ptr, nbytes, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (int(nbytes),), "typestr": "|u1", "data": (int(ptr), False),
                                         "version": 2}


def _pairs(dom, case, owner, split):
    """The moments of the buffer that the next step reads: one view
    [z][y][x][2] per moment pair, or one [pair][z][y][x][2]."""
    first, last = dom.zplane(mrlbm.ZPLANE_FIRST), dom.zplane(mrlbm.ZPLANE_LAST)
    nz, ny, nx = dom.shape
    dt = TORCH[case["storage"]]
    es = 4 if dt == torch.float32 else 2
    plane = first["bytes"] // es
    stride = first["pair_stride"] // es
    pitch = plane // (2 * (ny + 2))
    n = (first["npairs"] - 1) * first["pair_stride"] + (last["base"] - first["base"]) + first["bytes"]
    flat = torch.as_tensor(_Bytes(first["base"], n, owner), device="cuda").view(dt)
    at = 2 * (pitch + X_OFFSET)
    nm = _moments(case)
    if not split:
        return {"m": flat.as_strided((nm // 2, nz, ny, nx, 2), (stride, plane, 2 * pitch, 2, 1), at)}
    v = {}
    for p in range((nm + 1) // 2):
        size = (nz, ny, nx, 2) if 2 * p + 1 < nm else (nz, ny, nx, 1)
        v["m%02d" % (2 * p)] = flat.as_strided(size, (plane, 2 * pitch, 2, 1), at + p * stride)
    return v


def _views(dom, case, start):
    """The views of both moment buffers, by the parity of the steps done; the
    domain is back at its start afterwards."""
    both = [_pairs(dom, case, dom, True)]
    dom.step(1)
    both.append(_pairs(dom, case, dom, True))
    start()
    return both


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = mrlbm.Batch(case["q"], STORAGE[case["storage"]])
        mem = []
        for (nx, ny, nz), re in _batch_members(case, seed):
            m = b.add(mrlbm.lid_cavity_desc(nx, re=re, lid_u=0.05, storage=STORAGE[case["storage"]], ny=ny, nz=nz))
            m.set_node_types(mrlbm.lid_cavity_node_types(nx, ny, nz, 1))
            m.init_uniform((0.005, 0.002, 0.003))
            mem.append(m)
        views = [[_pairs(m, case, (b, m), False) for m in mem]]
        b.step(1)
        views.append([_pairs(m, case, (b, m), False) for m in mem])
        for m in mem:
            m.init_uniform((0.005, 0.002, 0.003))
        return dict(case=case, batch=b, members=mem, views=views, done=0)
    d, types, how = _setup(case, seed)
    dom = mrlbm.Domain(d)
    if types is not None:
        dom.set_node_types(types)
    fields = [_host(f) for f in _fields(case, seed, how)]
    dom.init_flow(*fields)
    if kind == "served":
        return dict(case=case, dom=dom)
    if kind == "job":
        n = dom.nm * case["nx"] * case["ny"] * case["nz"]
        a, b = (torch.empty(n, dtype=torch.float32, pin_memory=True) for _ in range(2))
        a.numpy()[:] = dom.moments_ref_layout()
        return dict(case=case, dom=dom, start=a, end=b)
    return dict(case=case, dom=dom, views=_views(dom, case, lambda: dom.init_flow(*fields)), done=0)


def run(state):
    case = state["case"]
    kind, n = case["kind"], case["steps"]
    if kind == "served":
        state["dom"].step(n)
        return {"m": state["dom"].moments()}
    if kind == "job":
        dom = state["dom"]
        dom.set_moments_ref_layout(state["start"].numpy())
        energy = []
        for _ in range(0, n, 50):
            dom.step(50)
            s = dom.sums()
            energy.append(s["kinetic_energy"])
        end = state["end"].numpy()
        mrlbm.check(mrlbm.lib().mrlbm_get_moments_ref_layout(dom.h, end.ctypes.data_as(mrlbm.FP)))
        return {"m": state["end"], "kinetic_energy": np.array(energy)}
    state["done"] += n
    if kind == "batch":
        state["batch"].step(n)
    else:
        state["dom"].step(n)
    return state["views"][state["done"] & 1]


# ------------------------------------------------------------- in 64 bits

CX = [0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0, 1, -1, 1, -1, 1, -1, -1, 1]
CY = [0, 0, 0, 1, -1, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 1, -1, 1, -1, 1, -1, -1, 1, 1, -1]
CZ = [0, 0, 0, 0, 0, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0, -1, 1, -1, 1, 1, -1, -1, 1, 1, -1, 1, -1]
SECOND = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]


def _w(q, i):
    n = abs(CX[i]) + abs(CY[i]) + abs(CZ[i])
    return ((1 / 3, 1 / 18, 1 / 36) if q == 19 else (8 / 27, 2 / 27, 1 / 54, 1 / 216))[n]


def _f64(v):
    """A descriptor value as the step kernels hold it (32-bit), in 64 bits."""
    return float(np.float32(v))


def _h(i):
    c = (CX[i], CY[i], CZ[i])
    return [c[a] * c[b] - (1 / 3 if a == b else 0.0) for a, b in SECOND]


def _wall_class(q, mq, word, uvel, omega0):
    """The wall system of one node type: known directions, A(omega0)^-1 and
    the rank-one dependence on omega (A = A0 + (omega - omega0) e0 q^T)."""
    oct_, kind, idx = word & 0xFF, (word >> 8) & 7, (word >> 11) & 3
    known = []
    for i in range(q):
        d = (-CX[i], -CY[i], -CZ[i])
        all_marked = True
        for o in range(8):
            s = (1 if o & 1 else -1, 1 if o & 2 else -1, 1 if o & 4 else -1)
            if all(d[a] == 0 or d[a] == s[a] for a in range(3)) and not (oct_ >> o) & 1:
                all_marked = False
        known.append(not all_marked)
    axis, side, faces = 3, 0, 0
    for a in range(3):
        for sd in range(2):
            if all((oct_ >> o) & 1 for o in range(8) if ((o >> a) & 1) == sd):
                axis, side, faces = a, 1 if sd else -1, faces + 1
    u = np.array([float(v) for v in uvel[idx]]) if kind == 1 else np.zeros(3)
    A, qv = np.zeros((7, 7)), np.zeros(7)
    for i in range(mq):
        if not known[i]:
            continue
        w, h = _w(mq, i), np.array(_h(i))
        g = np.array([4.5, 9.0, 9.0, 4.5, 9.0, 4.5]) * h
        cu = 3.0 * (CX[i] * u[0] + CY[i] * u[1] + CZ[i] * u[2])
        guu = float(sum(g[k] * u[a] * u[b] for k, (a, b) in enumerate(SECOND)))
        A[0, 0] += w * (1 + cu + omega0 * guu)
        A[0, 1:] += (1 - omega0) * w * g
        A[1:, 0] += w * h * (1 + cu)
        A[1:, 1:] += w * np.outer(h, g)
        qv[0] += w * guu
        qv[1:] -= w * g
    inv = np.eye(7) if kind == 2 else np.linalg.inv(A)
    return dict(known=known, inv=inv, v=inv[:, 0], qa=qv @ inv, s=float((qv @ inv)[0]), u=u, outflow=kind == 2,
                axis=axis if faces == 1 else 3, side=side)


class _Exact:
    """The time steps of one domain in 64 bits."""

    def __init__(self, d, types, fields, dev):
        self.d, self.q, self.dev = d, d.lattice, dev
        self.shape = (d.nz, d.ny, d.nx)
        self.rho0 = float(d.rho0)
        self.omega0 = 1.0 / d.tau
        self.F = [float(d.force[a]) for a in range(3)]
        self.per = [bool(d.periodic[a]) for a in range(3)]
        self.th, self.rheo = bool(d.thermal), d.rheology
        self.nm = 14 if self.th else 11 if self.rheo else 10
        m = torch.zeros((self.nm,) + self.shape, dtype=torch.float64, device=dev)
        rho, u = fields[0].to(dev, torch.float64), [f.to(dev, torch.float64) for f in fields[1:4]]
        uu = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        for i in range(19):  # the initial second moments: D3Q19 sums, weights of the lattice times rho0
            if i == 0:
                continue
            uc = 3 * (u[0] * CX[i] + u[1] * CY[i] + u[2] * CZ[i])
            f = _w(self.q, i) * self.rho0 * ((1 - 1.5 * uu) + uc * (1 + 0.5 * uc))
            c = (CX[i], CY[i], CZ[i])
            for k, (a, b) in enumerate(SECOND):
                if c[a] * c[b]:
                    m[4 + k] += f * (c[a] * c[b])
        for k, (a, b) in enumerate(SECOND):
            m[4 + k] = 4.5 * (m[4 + k] / rho - 1 / 3) if a == b else 9.0 * m[4 + k] / rho
        m[0] = rho - self.rho0
        for a in range(3):
            m[1 + a] = 3 * u[a]
        if self.rheo:
            m[10] = self.omega0
        if self.th:
            m[10] = d.t_reference
            a = 3.0 * (d.t_diffusivity - 1 / 6)
            self.coef = a / (1 + a)
        self.m = m
        w19 = sum(_w(self.q, i) * CX[i] ** 2 for i in range(19))
        self.ext = [0.0] * 4 + [4.5 * (w19 - 1 / 3), 0, 0, 4.5 * (w19 - 1 / 3), 0, 4.5 * (w19 - 1 / 3)]
        if self.nm > 10:
            self.ext += [float(d.t_reference), 0, 0, 0] if self.th else [self.omega0]
        self._walls(types)

    def _walls(self, types):
        d, dev = self.d, self.dev
        self.idx = None
        if types is None:
            return
        t = torch.from_numpy(types.astype(np.int64).reshape(-1)).to(dev)
        self.solid = ((t & 0xFF) == 0xFF).reshape(self.shape)
        self.idx = torch.nonzero(((t & 0xFF) != 0) & ((t & 0xFF) != 0xFF)).reshape(-1)
        words, inv = torch.unique(t[self.idx], return_inverse=True)
        uvel = [[d.bc_velocity[k][a] for a in range(3)] for k in range(4)]
        cl = [_wall_class(self.q, d.bc_matrix_q or (19 if self.q == 27 else self.q), int(w) & 0x1FFF, uvel, self.omega0)
              for w in words.tolist()]

        def at(f):
            return torch.tensor(np.array([f(c) for c in cl], dtype=np.float64), device=dev)[inv]
        self.known = at(lambda c: c["known"])
        self.inv, self.v, self.qa, self.s = at(lambda c: c["inv"]), at(lambda c: c["v"]), at(lambda c: c["qa"]), at(
            lambda c: c["s"])
        self.uw = at(lambda c: c["u"])
        self.out = at(lambda c: c["outflow"]) > 0
        stride = (1, d.nx, d.nx * d.ny, 0)
        # the inward neighbour, for the classes that read it
        near = [c["side"] * stride[c["axis"]] if c["outflow"] or self.th else 0 for c in cl]
        self.inward = self.idx - torch.tensor(near, device=dev)[inv]
        if self.th:
            words = words.to(dev)[inv]
            self.rule, self.tidx = (words >> 13) & 3, (words >> 15) & 3
            self.axis = at(lambda c: c["axis"]).long()
            assert bool((self.rule == 2).all())

    def _padded(self, k):
        a = self.m[k]
        for ax in range(3):  # z, y, x: periodic axes first
            if self.per[2 - ax]:
                n = a.shape[ax]
                a = torch.cat([a.narrow(ax, n - 1, 1), a, a.narrow(ax, 0, 1)], ax)
        pad = []
        for ax in range(3):
            pad += [0, 0] if self.per[ax] else [1, 1]
        return torch.nn.functional.pad(a, pad, value=self.ext[k]) if any(pad) else a

    def _src(self, p, i):
        nz, ny, nx = self.shape
        return p[1 - CZ[i]:1 - CZ[i] + nz, 1 - CY[i]:1 - CY[i] + ny, 1 - CX[i]:1 - CX[i] + nx]

    def step(self):
        q = self.q
        P = [self._padded(k) for k in range(self.nm)]
        pics = 1 - (P[4] + P[7] + P[9]) / 3
        S = [torch.zeros(self.shape, dtype=torch.float64, device=self.dev) for _ in range(10)]
        walls = self.idx is not None
        fw = torch.empty((q, self.idx.numel()), dtype=torch.float64, device=self.dev) if walls else None
        for i in range(q):
            c = (CX[i], CY[i], CZ[i])
            t = self._src(pics, i).clone()
            for a in range(3):
                if c[a]:
                    t += c[a] * self._src(P[1 + a], i)
            for k, (a, b) in enumerate(SECOND):
                if c[a] * c[b]:
                    t += (c[a] * c[b]) * self._src(P[4 + k], i)
            t *= (self._src(P[0], i) + self.rho0) * _w(q, i)
            S[0] += t
            for a in range(3):
                if c[a]:
                    S[1 + a] += c[a] * t
            for k, (a, b) in enumerate(SECOND):
                if c[a] * c[b]:
                    S[4 + k] += (c[a] * c[b]) * t
            if walls:
                fw[i] = t.reshape(-1)[self.idx]
        F = self.F
        cq = None
        if self.th:
            cq, F = self._thermal(P)
        ir = 1 / S[0]
        mac = [S[0]] + [S[1 + a] * ir for a in range(3)] + [
            S[4 + k] * ir - (1 / 3 if a == b else 0) for k, (a, b) in enumerate(SECOND)]
        omega = self.m[10].clone() if self.rheo else torch.full((), self.omega0, dtype=torch.float64, device=self.dev)
        if walls:
            self._solve(fw, mac, omega)
        new = self._collide(mac, omega, F)
        if cq is not None:
            new += cq
        out = torch.stack(new)
        if walls:
            out = torch.where(self.solid, self.m, out)
        self.m = out

    def _solve(self, fw, mac, omega):
        f = fw * self.known.t()
        b = torch.zeros((7, self.idx.numel()), dtype=torch.float64, device=self.dev)
        for i in range(self.q):
            b[0] += f[i]
            for k, h in enumerate(_h(i)):
                if h:
                    b[1 + k] += h * f[i]
        X = torch.einsum("nij,jn->in", self.inv, b)
        om = omega.reshape(-1)[self.idx] if omega.dim() else omega
        dw = om - self.omega0
        X = X - (dw * (self.qa.t() * b).sum(0) / (1 + dw * self.s)) * self.v.t()
        new = [X[0]] + [self.uw[:, a] for a in range(3)] + [X[1 + k] / X[0] for k in range(6)]
        old = [self.m[k].reshape(-1)[self.inward] for k in range(10)]
        scale = (0, 3, 3, 3, 4.5, 9, 9, 4.5, 9, 4.5)
        for k in range(10):
            o = self.rho0 + old[0] if k == 0 else old[k] / scale[k]
            mac[k].reshape(-1)[self.idx] = torch.where(self.out, o, new[k])

    def _omega(self, mac, omega, F):
        d = self.d
        rho, u = mac[0], mac[1:4]
        s = 0
        for k, (a, b) in enumerate(SECOND):
            g = rho * (mac[4 + k] - u[a] * u[b]) + 0.5 * (u[a] * F[b] + u[b] * F[a])
            s = s + (1 if a == b else 2) * g * g
        s = torch.sqrt(0.5 * s)
        if self.rheo == mrlbm.BINGHAM:
            return (d.nnf_omega_p or self.omega0) * torch.clamp(1 - d.nnf_yield / s, min=0.0)
        n = _f64(d.nnf_n)
        K = d.nnf_k or self.rho0 * (d.tau - 0.5) / 3
        om = omega.clone()
        a = K * (s / (self.rho0 / 3)) ** n
        live = torch.ones_like(s, dtype=torch.bool)
        for _ in range(7):
            dx = (a * om ** n + 0.5 * s * om - s) / (a * n * om ** (n - 1) + 0.5 * s)
            live = live & (dx.abs() >= 1e-6)
            om = torch.where(live, om - dx, om)
        return torch.where(s < 1e-6, torch.zeros_like(om), om)

    def _collide(self, mac, omega, F):
        rho, ir = mac[0], 1 / mac[0]
        if self.rheo:
            omega = self._omega(mac, omega, F)
        u = [3 * mac[1 + a] + 3 * ir * F[a] for a in range(3)]
        new = [rho - self.rho0] + u
        for k, (a, b) in enumerate(SECOND):
            if a == b:
                new.append((1 - omega) * 4.5 * mac[4 + k] + 0.5 * omega * u[a] * u[a] + 1.5 * ir * (1 - 0.5 * omega)
                           * 2 * F[a] * u[a])
            else:
                new.append((1 - omega) * 9 * mac[4 + k] + omega * u[a] * u[b] + 3 * (1 - 0.5 * omega) * ir
                           * (F[a] * u[b] + F[b] * u[a]))
        return new + ([omega] if self.rheo else [])

    def _thermal(self, P):
        d = self.d
        v = [P[1 + a] + self.coef * (P[11 + a] / P[10] - P[1 + a]) for a in range(3)]
        C = torch.zeros(self.shape, dtype=torch.float64, device=self.dev)
        qf = [torch.zeros_like(C) for _ in range(3)]
        for i in range(19):
            c = (CX[i], CY[i], CZ[i])
            g = 1 + sum(c[a] * self._src(v[a], i) for a in range(3) if c[a])
            g = g * self._src(P[10], i) * _w(19, i)
            C += g
            for a in range(3):
                if c[a]:
                    qf[a] += 3 * c[a] * g
        C += d.t_source
        bulk = torch.ones_like(C)
        bulk.reshape(-1)[self.idx] = 0.0
        F = [self.F[a] + bulk * (d.t_gravity_beta[a] * self.rho0) * (C - d.t_reference) for a in range(3)]
        tw = torch.tensor([_f64(d.t_wall[k]) for k in range(4)], dtype=torch.float64, device=self.dev)
        C.reshape(-1)[self.idx] = tw[self.tidx]
        for a in range(3):
            near = self.m[11 + a].reshape(-1)[self.inward]
            qf[a].reshape(-1)[self.idx] = torch.where(self.axis == a, near, torch.zeros_like(near))
        return [C] + qf, F


SCALES = [256.0] + [8.0] * 3 + [64.0] * 6


def _exact_domain(d, types, fields, steps):
    e = _Exact(d, types, fields, _device())
    for _ in range(steps):
        e.step()
    return e


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for (nx, ny, nz), re in _batch_members(case, seed):
            d = mrlbm.lid_cavity_desc(nx, re=re, lid_u=0.05, ny=ny, nz=nz)
            f = [torch.full((nz, ny, nx), v, dtype=torch.float32) for v in (1.0, 0.005, 0.002, 0.003)]
            m = _exact_domain(d, mrlbm.lid_cavity_node_types(nx, ny, nz, 1), f, case["steps"]).m
            if case["storage"] == "f16":
                m = m * torch.tensor(SCALES, dtype=torch.float64, device=m.device)[:, None, None, None]
            out.append({"m": torch.stack([m[0::2], m[1::2]], -1)})
        return out
    d, types, how = _setup(case, seed)
    fields = _fields(case, seed, how)
    if kind == "job":
        return _exact_job(case, d, fields)
    m = _exact_domain(d, types, fields, case["steps"]).m
    if kind == "served":
        return {"m": m}
    if case["storage"] == "f16":
        for k in range(10):
            m[k] *= SCALES[k]
    return {"m%02d" % k: torch.stack([m[k], m[k + 1]], -1) if k + 1 < len(m) else m[k][..., None]
            for k in range(0, len(m), 2)}


def _exact_job(case, d, fields):
    e = _Exact(d, None, fields, _device())
    energy = []
    for s in range(case["steps"]):
        e.step()
        if (s + 1) % 50 == 0:
            rho, u = e.rho0 + e.m[0], e.m[1:4] / 3
            energy.append(float((0.5 * rho * (u * u).sum(0)).sum()))
    nz, ny, nx = e.shape
    # the reference's layout: 8^3 blocks, moments of a block together
    v = e.m.reshape(10, nz // 8, 8, ny // 8, 8, nx // 8, 8).permute(1, 3, 5, 0, 2, 4, 6)
    return {"m": v.reshape(-1), "kinetic_energy": np.array(energy)}
