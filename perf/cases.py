"""The work a user has this library do, as cases that can be timed and compared.

Every case is water (three sites, TIP3P charges) with or without 0.15 M NaCl at
1 g/cm^3, the boxes of the benchmark and the tests, in one of the uses the
library has:

  force    one force evaluation of the engine on the caller's coordinates (an
           external integrator's step, or a print step with energy and virial)
  md       graph-replayed NVE steps of the engine, flexible (0.5 fs) or rigid
           water (SETTLE, 2 fs), then the velocities rescaled to 300 K
  host     the same steps for a caller that keeps its state in host memory
  soft     the same steps with the soft-core pair kernel and a solute
  batch    the same steps for many independent boxes in one engine
  module   one step through the module entry points, as a program that
           replaces its NEIGHBOR_LIST, LJ and Particle_Mesh modules calls them
  pme      the reciprocal part alone (Particle_Mesh)

`exact` is each case in plain torch, 64 bits throughout.
"""

import ctypes
import math

import numpy as np
import torch

from sponge_b200 import capi

TIME = 20.455           # internal time units per ps
KB = 0.00198716         # kcal/mol/K
SCALE = 18.2223         # charge unit
WATER_A3 = 29.9150      # volume of one water at 1 g/cm^3
IONS_PER_A3 = 0.15 * 6.02214076e23 * 1e-27
SIGMA = np.array([3.1507, 0.0, 2.439, 4.478])    # O, H, Na, Cl
EPS = np.array([0.1521, 0.0, 0.0874, 0.0355])
MASS = np.array([15.9994, 1.008, 22.98977, 35.453])
CHARGE = np.array([-0.834, 0.417, 1.0, -1.0])
R_OH, T_HOH = 0.9572, math.radians(104.52)
R_HH = 2 * R_OH * math.sin(T_HOH / 2)
BOND_K, ANGLE_K = 553.0, 100.0
SOFT = {"soft_core_alpha": 0.5, "soft_core_powfer": 1.0, "soft_core_sigma": 3.0,
        "soft_core_sigma_min": 0.0}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: the 648-atom box of the tests, forces only
        dict(name="force_648", kind="force", waters=216, ions=False, cutoff=8.0, energy=False),
        # a print step of the 9,000-atom box: energy and virial too
        dict(name="force_energy_9k", kind="force", waters=3000, ions=False, cutoff=8.0,
             energy=True),
        # the benchmark's small box, 40 MD steps
        dict(name="md_9k", kind="md", waters=3000, ions=False, cutoff=8.0, rigid=False, steps=40),
        # the headline box (99,639 atoms), 20 MD steps
        dict(name="md_100k", kind="md", waters=33333, ions=True, cutoff=10.0, rigid=False,
             steps=20),
        # rigid water at 2 fs in a mid-size box
        dict(name="md_rigid_36k", kind="md", waters=12000, ions=False, cutoff=9.0, rigid=True,
             steps=20),
        # many small boxes in one engine, as the benchmark's batch (U[200, 2000] waters)
        dict(name="batch_64", kind="batch", boxes=64, least=200, most=2000, cutoff=8.0, steps=10),
        # the decoupling window of the ~1M-atom soft-core box: the largest
        dict(name="soft_1m", kind="soft", waters=332000, solute=64, cutoff=10.0, lam=0.5, steps=4),
        # the state in host memory, one call per step
        dict(name="host_30k", kind="host", waters=10000, ions=True, cutoff=10.0, steps=1, calls=4),
        # module entry points on the headline box: list kept, forces only
        dict(name="module_100k", kind="module", waters=33333, ions=True, cutoff=10.0,
             energy=False, rebuild=False, skew=False),
        # module entry points, list rebuilt, energies and virials wanted
        dict(name="module_energy_24k", kind="module", waters=8000, ions=True, cutoff=9.0,
             energy=True, rebuild=True, skew=False),
        # module entry points in a skewed cell
        dict(name="module_skew_18k", kind="module", waters=6000, ions=False, cutoff=8.0,
             energy=True, rebuild=False, skew=True),
        # the reciprocal part alone on a ragged grid, energy and virial wanted
        dict(name="pme_ragged_45k", kind="pme", nx=20, ny=25, nz=30, k0=63, k1=75, k2=98,
             energy=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cutoff(rng, waters):
    half = 0.5 * (waters * WATER_A3) ** (1 / 3) - 0.4
    return round(rng.uniform(min(7.5, half), min(11.0, half)), 2)


def draw(rng):
    kind = rng.choice(["force", "md", "md", "soft", "batch", "host", "module", "module", "pme"])
    if kind == "force":
        w = _log(rng, 200, 33333)
        return dict(kind=kind, waters=w, ions=rng.random() < 0.5, cutoff=_cutoff(rng, w),
                    energy=rng.random() < 0.5)
    if kind == "md":
        w = _log(rng, 216, 40000)
        return dict(kind=kind, waters=w, ions=rng.random() < 0.5, cutoff=_cutoff(rng, w),
                    rigid=rng.random() < 0.4, steps=rng.randint(5, 16))
    if kind == "soft":
        w = _log(rng, 1000, 100000)
        return dict(kind=kind, waters=w, solute=rng.randint(1, 64), cutoff=_cutoff(rng, w),
                    lam=rng.choice([0.0, 0.25, 0.5, 0.75, 1.0]), steps=rng.randint(2, 8))
    if kind == "batch":
        lo = _log(rng, 200, 1000)
        return dict(kind=kind, boxes=rng.randint(2, 64), least=lo,
                    most=lo + rng.randint(0, 1000), cutoff=round(rng.uniform(7.0, 8.5), 2),
                    steps=rng.randint(3, 10))
    if kind == "host":
        w = _log(rng, 216, 33333)
        return dict(kind=kind, waters=w, ions=rng.random() < 0.5, cutoff=_cutoff(rng, w),
                    steps=rng.randint(1, 5), calls=rng.randint(1, 3))
    if kind == "module":
        skew = rng.random() < 0.3
        w = _log(rng, 1500 if skew else 300, 12000 if skew else 33333)
        return dict(kind=kind, waters=w, ions=rng.random() < 0.5,
                    cutoff=min(_cutoff(rng, w), 8.0) if skew else _cutoff(rng, w),
                    energy=rng.random() < 0.5, rebuild=rng.random() < 0.5, skew=skew)
    n = [_log(rng, 6, 32) for _ in range(3)]
    k = [rng.choice([g for g in _grids() if 2.9 * m <= g <= 4.2 * m and (d < 2 or g % 2 == 0)])
         for d, m in enumerate(n)]
    return dict(kind="pme", nx=n[0], ny=n[1], nz=n[2], k0=k[0], k1=k[1], k2=k[2],
                energy=rng.random() < 0.5)


def _grids():
    out = []
    for n in range(16, 141):
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            out.append(n)
    return out


# ----------------------------------------------------------------- the boxes
class Water:
    """Boxes of water (and ions), one after another in every array."""


def _lattice(rng, waters):
    side = math.ceil(waters ** (1 / 3) - 1e-9)
    return dict(waters=waters, dims=(side, side, side),
                cell=np.eye(3) * (waters * WATER_A3) ** (1 / 3))


def _boxes(specs, rng, ions, clear=0.0):
    """Waters on a jittered lattice of each box, uniformly random orientations
    redrawn where a hydrogen would sit within 1.6 A of another molecule, 0.15 M
    NaCl in the place of randomly chosen waters (none within `clear` of the
    centre)."""
    dev = "cuda"
    o_pos, kind, nbr, cells, box_of, base = [], [], [], [], [], 0
    off = np.array([(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)
                    if (i, j, k) != (0, 0, 0)])
    off = torch.from_numpy(off).to(dev)
    for b, s in enumerate(specs):
        nx, ny, nz = s["dims"]
        w = s["waters"]
        sites = np.sort(rng.permutation(nx * ny * nz)[:w])
        ijk = np.stack([sites // (ny * nz), sites // nz % ny, sites % nz], 1)
        cell = s["cell"]
        x = ((ijk + 0.5) / np.array([nx, ny, nz])) @ cell
        o_pos.append(x + rng.uniform(-0.3, 0.3, x.shape))
        kd = np.zeros(w, np.int64)
        if ions:
            pairs = int(round(IONS_PER_A3 * abs(np.linalg.det(cell))))
            free = np.flatnonzero(np.linalg.norm(o_pos[-1] - cell.sum(0) / 2, axis=1) >= clear)
            pick = rng.choice(free, 2 * pairs, replace=False)
            kd[pick[:pairs]], kd[pick[pairs:]] = 2, 3
        kind.append(kd)
        where = torch.full((nx * ny * nz,), -1, dtype=torch.int64, device=dev)
        where[torch.from_numpy(sites).to(dev)] = torch.arange(base, base + w, device=dev)
        t = torch.from_numpy(ijk).to(dev)[:, None, :] + off
        t = t % torch.tensor([nx, ny, nz], device=dev)
        nbr.append(where[(t[..., 0] * ny + t[..., 1]) * nz + t[..., 2]])
        cells.append(cell)
        box_of.append(np.full(w, b))
        base += w
    o = torch.from_numpy(np.concatenate(o_pos)).to(dev)
    kind, box_of = np.concatenate(kind), np.concatenate(box_of)
    water = torch.from_numpy(kind == 0).to(dev)
    nbr = torch.cat(nbr)
    H = torch.from_numpy(np.stack(cells)).to(dev)
    Hi = torch.linalg.inv(H)
    bx = torch.from_numpy(box_of).to(dev)
    one = len(specs) == 1
    local = torch.tensor([[math.sin(T_HOH / 2), 0, math.cos(T_HOH / 2)],
                          [-math.sin(T_HOH / 2), 0, math.cos(T_HOH / 2)]],
                         dtype=torch.float64, device=dev) * R_OH

    def hydrogens(n):
        q = torch.from_numpy(rng.normal(size=(n, 4))).to(dev)
        q = q / q.norm(dim=1, keepdim=True)
        w, x, y, z = q.unbind(1)
        R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                         2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                         2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)],
                        1).reshape(-1, 3, 3)
        return torch.einsum("nij,kj->nki", R, local)

    h = hydrogens(len(kind))                       # relative to the oxygen
    todo = torch.nonzero(water)[:, 0]
    for _ in range(300):
        if not len(todo):
            break
        bad = torch.zeros(len(kind), dtype=torch.bool, device=dev)
        for part in todo.split(200_000):
            m = nbr[part]
            there = m >= 0
            m = m.clamp(min=0)
            d = o[m] - o[part][:, None]            # centre to centre, nearest image
            if one:
                d = d - torch.round(d @ Hi[0]) @ H[0]
            else:
                g = torch.einsum("nmi,nij->nmj", d, Hi[bx[part]])
                d = d - torch.einsum("nmi,nij->nmj", torch.round(g), H[bx[part]])
            near = torch.zeros_like(there)
            far = torch.zeros_like(there)
            for k in (0, 1):
                mine = h[part, k][:, None]
                near |= (d - mine).square().sum(-1) < 2.56          # my H, their centre
                for l in (0, 1):
                    c = ((d + h[m, l] - mine).square().sum(-1) < 2.56) & water[m]
                    near |= c
                    far |= c
                far |= ((d + h[m, k]).square().sum(-1) < 2.56) & water[m]  # their H, my centre
            bad[part] |= (near & there).any(1)
            bad[m[far & there]] = True
        todo = torch.nonzero(bad & water)[:, 0]
        h[todo] = hydrogens(len(todo))
    sites = np.where(kind == 0, 3, 1)
    first = np.concatenate([[0], np.cumsum(sites)])[:-1]
    n = int(sites.sum())
    crd = torch.empty((n, 3), dtype=torch.float64, device=dev)
    ft = torch.from_numpy(first).to(dev)
    crd[ft] = o
    wf = ft[water]
    crd[wf + 1] = o[water] + h[water, 0]
    crd[wf + 2] = o[water] + h[water, 1]
    s = Water()
    s.n = n
    s.crd = crd.float().cpu().numpy()
    s.type = np.ones(n, np.int32)
    s.type[first] = kind
    s.o = first[kind == 0].astype(np.int32)
    s.n_types = 4
    s.A, s.B = _tables(SIGMA, EPS)
    s.charge = (CHARGE[s.type] * SCALE).astype(np.float32)
    s.mass = MASS[s.type].astype(np.float32)
    s.mol = np.repeat(np.arange(len(kind)), sites).astype(np.int64)
    s.box_of = np.repeat(box_of, sites).astype(np.int64)
    s.counts = np.bincount(s.box_of, minlength=len(specs)).astype(np.int32)
    s.cells = np.stack(cells).astype(np.float32)
    v = rng.normal(size=(n, 3)) * np.sqrt(KB * 300.0 / MASS[s.type])[:, None]
    v -= (v * s.mass[:, None]).sum(0) / s.mass.sum()
    s.vel = v.astype(np.float32)
    s.en = np.zeros(n, np.int32)
    s.en[s.o], s.en[s.o + 1] = 2, 1
    s.es = np.concatenate([[0], np.cumsum(s.en)])[:-1].astype(np.int32)
    s.el = np.stack([s.o + 1, s.o + 2, s.o + 2], 1).reshape(-1).astype(np.int32)
    return s


def _tables(sigma, eps):
    """A' = 12 A and B' = 6 B per triangular type pair, Lorentz-Berthelot."""
    T = len(sigma)
    a, b = np.tril_indices(T)
    e = np.sqrt(eps[a] * eps[b])
    sg = np.where(e > 0, 0.5 * (sigma[a] + sigma[b]), 0.0)
    return ((4 * e * sg ** 12).astype(np.float32) * np.float32(12),
            (4 * e * sg ** 6).astype(np.float32) * np.float32(6))


def _reach(sites):
    """Radius of the cluster of LJ sites."""
    return max(4.0, 1.4 * sites ** (1 / 3) * 2.5 / 1.6)


def _solute(s, rng, sites):
    """A compact cluster of LJ sites without charge in the centre (the LJ stage
    of a decoupling): the nearest waters give way, as many as a sphere 0.8 A
    larger holds.  State B has its LJ switched off."""
    centre = s.cells[0].diagonal().astype(np.float64) / 2
    radius = _reach(sites)
    got = []
    while len(got) < sites:
        p = rng.uniform(-radius, radius, 3)
        if np.linalg.norm(p) <= radius and all(np.linalg.norm(p - q) >= 2.5 for q in got):
            got.append(p)
    x = np.asarray(got) + centre
    close = s.o[np.linalg.norm(s.crd[s.o] - centre, axis=1) < radius + 6.0]
    near = np.minimum.reduce([np.linalg.norm(s.crd[close + k][:, None] - x[None], axis=2).min(1)
                              for k in (0, 1, 2)])
    give = int(4 / 3 * math.pi * (radius + 0.8) ** 3 / WATER_A3)
    gone = np.isin(s.mol, s.mol[close[np.argsort(near)[:give]]])
    keep = np.flatnonzero(~gone)
    new = np.cumsum(~gone) - 1
    s.o = new[s.o[~gone[s.o]]].astype(np.int32)
    for k in ("crd", "vel", "type", "charge", "mass", "mol", "box_of", "en"):
        setattr(s, k, getattr(s, k)[keep])
    m = len(keep)
    s.crd = np.concatenate([s.crd, x.astype(np.float32)])
    v = rng.normal(size=(sites, 3)) * math.sqrt(KB * 300.0 / 12.011)
    s.vel = np.concatenate([s.vel, v.astype(np.float32)])
    s.type_A = np.concatenate([s.type, 4 + np.arange(sites)]).astype(np.int32)
    s.type_B = np.concatenate([s.type, np.full(sites, 4)]).astype(np.int32)
    s.type = s.type_A
    s.charge = np.concatenate([s.charge, np.zeros(sites, np.float32)])
    s.mass = np.concatenate([s.mass, np.full(sites, 12.011, np.float32)])
    s.mol = np.concatenate([s.mol, s.mol.max() + 1 + np.arange(sites)])
    s.box_of = np.zeros(m + sites, np.int64)
    s.mask = np.concatenate([np.zeros(m, np.int32), np.ones(sites, np.int32)])
    s.n = m + sites
    s.en = np.concatenate([s.en, np.zeros(sites, np.int32)]).astype(np.int32)
    s.es = np.concatenate([[0], np.cumsum(s.en)])[:-1].astype(np.int32)
    s.el = np.stack([s.o + 1, s.o + 2, s.o + 2], 1).reshape(-1).astype(np.int32)
    sig, eps = rng.uniform(3.0, 4.0, sites), rng.uniform(0.05, 0.2, sites)
    s.A, s.B = _tables(np.concatenate([SIGMA, sig]), np.concatenate([EPS, eps]))
    s.BA, s.BB = _tables(np.append(SIGMA, 0.0), np.append(EPS, 0.0))
    s.n_types, s.n_types_B = 4 + sites, 5
    return s


def _system(case, seed):
    rng = np.random.default_rng([seed, 7])
    kind = case["kind"]
    if kind == "batch":
        sizes = np.random.default_rng(case["boxes"])  # the same boxes for every seed
        w = sizes.integers(case["least"], case["most"] + 1, case["boxes"])
        return _boxes([_lattice(rng, int(x)) for x in w], rng, True)
    if kind == "pme":
        n = np.array([case["nx"], case["ny"], case["nz"]])
        return _boxes([dict(waters=int(n.prod()), dims=tuple(int(x) for x in n),
                            cell=np.diag(n * WATER_A3 ** (1 / 3)))], rng, False)
    spec = _lattice(rng, case["waters"])
    if case.get("skew"):
        a = spec["cell"][0, 0]
        spec["cell"] = np.array([[a, 0, 0], [0.2 * a, a, 0], [-0.1 * a, 0.15 * a, a]])
    s = _boxes([spec], rng, case.get("ions", True),
               _reach(case["solute"]) + 6.0 if kind == "soft" else 0.0)
    return _solute(s, rng, case["solute"]) if kind == "soft" else s


# -------------------------------------------------------------- the handles
def _np(a, dt):
    return np.ascontiguousarray(a, dt)


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _boundary(cell):
    c = cell.astype(np.float64)
    r = np.linalg.inv(c)
    low = lambda m: [m[0, 0], m[1, 0], m[1, 1], m[2, 0], m[2, 1], m[2, 2]]  # noqa: E731
    return capi.boundary(np.float32(low(c)), np.float32(low(r)))


class State:
    """What a user's program keeps: device buffers and library handles."""

    def __init__(self):
        self.lib = capi.load()
        self.owned = []

    def own(self, destroy, h):
        self.owned.append((destroy, h))
        return h

    def __del__(self):
        if self.owned:
            torch.cuda.synchronize()
        for destroy, h in reversed(self.owned):
            getattr(self.lib, destroy)(h)


def _engine(st, s, case):
    lib, h = st.lib, ctypes.c_void_p()
    o = capi.options(cutoff=case["cutoff"], skin=2.0)
    t, A, B, q = _np(s.type, np.int32), _np(s.A, np.float32), _np(s.B, np.float32), s.charge
    arrays = (t.ctypes.data, A.ctypes.data, B.ctypes.data, q.ctypes.data, s.es.ctypes.data,
              s.en.ctypes.data, s.el.ctypes.data, len(s.el), ctypes.byref(h))
    if case["kind"] == "batch":
        L = _np([c.diagonal() for c in s.cells], np.float32)
        capi.check(lib.snb_batch_create(ctypes.byref(o), len(s.cells), s.counts.ctypes.data,
                                        L.ctypes.data, s.n_types, *arrays), "batch_create")
    else:
        capi.check(lib.snb_engine_create(ctypes.byref(o), s.n, _boundary(s.cells[0]),
                                         s.n_types, *arrays), "engine_create")
    st.own("snb_engine_destroy", h)
    w = len(s.o)
    if case["kind"] == "force":
        return h
    if case.get("rigid"):
        ai = _np(np.stack([s.o, s.o, s.o + 1], 1).reshape(-1), np.int32)
        aj = _np(np.stack([s.o + 1, s.o + 2, s.o + 2], 1).reshape(-1), np.int32)
        r0 = _np(np.tile([R_OH, R_OH, R_HH], w), np.float32)
        g = ctypes.c_void_p()
        capi.check(lib.snb_settle_create(s.n, 3 * w, ai.ctypes.data, aj.ctypes.data,
                                         r0.ctypes.data, s.mass.ctypes.data, ctypes.byref(g)),
                   "settle_create")
        st.own("snb_settle_destroy", g)
        capi.check(lib.snb_engine_set_settle(h, g), "set_settle")
        return h
    ba, bb = _np(np.repeat(s.o, 2), np.int32), _np(np.stack([s.o + 1, s.o + 2], 1).reshape(-1),
                                                   np.int32)
    bk, br = np.full(2 * w, BOND_K, np.float32), np.full(2 * w, R_OH, np.float32)
    aa, ab, ac = _np(s.o + 1, np.int32), _np(s.o, np.int32), _np(s.o + 2, np.int32)
    ak, at = np.full(w, ANGLE_K, np.float32), np.full(w, T_HOH, np.float32)
    capi.check(lib.snb_engine_set_bonded(h, 2 * w, *[x.ctypes.data for x in (ba, bb, bk, br)], w,
                                         *[x.ctypes.data for x in (aa, ab, ac, ak, at)]),
               "set_bonded")
    if case["kind"] == "soft":
        g = ctypes.c_void_p()
        o = capi.options(cutoff=case["cutoff"], lambda_lj=case["lam"], **SOFT)
        x = [_np(s.type_A, np.int32), _np(s.type_B, np.int32), A, B, s.BA, s.BB,
             _np(s.mask, np.int32)]
        capi.check(lib.snb_lj_soft_create(ctypes.byref(o), s.n, s.n_types, s.n_types_B,
                                          *[v.ctypes.data for v in x], case["cutoff"],
                                          ctypes.byref(g)), "lj_soft_create")
        st.own("snb_lj_soft_destroy", g)
        capi.check(lib.snb_engine_set_soft_core(h, g), "set_soft_core")
    return h


def _modules(st, s, case):
    lib, rc = st.lib, case.get("cutoff", 9.0)
    st.bnd = _boundary(s.cells[0])
    keys = dict(cutoff=rc, skin=2.0)
    if case["kind"] == "pme":
        keys.update(PM_fftx=case["k0"], PM_ffty=case["k1"], PM_fftz=case["k2"])
    o = capi.options(**keys)
    L = _np(s.cells[0].diagonal(), np.float32)
    st.pme = ctypes.c_void_p()
    capi.check(lib.snb_pme_create(ctypes.byref(o), s.n, st.bnd, L.ctypes.data, rc,
                                  ctypes.byref(st.pme)), "pme_create")
    st.own("snb_pme_destroy", st.pme)
    st.beta = ctypes.c_float(lib.snb_pme_beta(st.pme))
    if case["kind"] == "pme":
        return
    st.nl, st.lj = ctypes.c_void_p(), ctypes.c_void_p()
    capi.check(lib.snb_nl_create(ctypes.byref(o), s.n, rc, 2.0, st.bnd, ctypes.byref(st.nl)),
               "nl_create")
    st.own("snb_nl_destroy", st.nl)
    t = _np(s.type, np.int32)
    capi.check(lib.snb_lj_create(ctypes.byref(o), s.n, s.n_types, t.ctypes.data, s.A.ctypes.data,
                                 s.B.ctypes.data, rc, ctypes.byref(st.lj)), "lj_create")
    st.own("snb_lj_destroy", st.lj)
    st.es, st.en, st.el = (torch.from_numpy(x).cuda() for x in (s.es, s.en, s.el))
    _update(st, 1)


def _update(st, forced):
    capi.check(st.lib.snb_nl_update(st.nl, None, st.n, 0, _p(st.crd), st.bnd, 0, forced,
                                    _p(st.es), _p(st.el), _p(st.en), st.sp), "nl_update")


def prepare(case, seed):
    s = _system(case, seed)
    st = State()
    st.case, st.n, st.step = case, s.n, 0
    st.stream = torch.cuda.Stream()
    st.sp = ctypes.c_void_p(st.stream.cuda_stream)
    st.crd = torch.from_numpy(s.crd.reshape(-1)).cuda()
    st.charge = torch.from_numpy(s.charge).cuda()
    kind = case["kind"]
    if kind in ("md", "soft", "batch", "host"):
        both = torch.cat([st.crd, torch.from_numpy(s.vel.reshape(-1)).cuda()])
        st.crd, st.vel = both[:3 * s.n], both[3 * s.n:]
        st.both = both
        m = torch.from_numpy(s.mass).cuda()
        st.mass = m[:, None]
        st.invm = 1.0 / m
        st.dt = 1e-3 * TIME * (2.0 if case.get("rigid") else 0.5)
        st.kt3 = (2 * s.n if case.get("rigid") and not case["ions"] else
                  6 * len(s.o) + 3 * (s.n - 3 * len(s.o)) if case.get("rigid") else
                  3 * s.n) * KB * 300.0
    if kind in ("force", "md", "soft", "batch", "host"):
        st.engine = _engine(st, s, case)
    if kind == "host":
        st.host = torch.empty(6 * s.n, dtype=torch.float32, pin_memory=True)
        st.host.copy_(st.both)
    torch.cuda.synchronize()
    if kind in ("module", "pme"):
        _modules(st, s, case)
    st.frc = torch.zeros(3 * s.n, device="cuda")
    if case.get("energy"):
        st.totals = torch.zeros(14, dtype=torch.float64, device="cuda")
        st.ene, st.cou = (torch.zeros(s.n, device="cuda") for _ in range(2))
        st.vir = torch.zeros((s.n, 6), device="cuda")
        st.pot, st.pvir = torch.zeros(1, device="cuda"), torch.zeros(6, device="cuda")
    torch.cuda.synchronize()
    return st


def run(st):
    case, lib = st.case, st.lib
    kind = case["kind"]
    on = int(bool(case.get("energy")))
    with torch.cuda.stream(st.stream):
        if kind in ("md", "soft", "batch"):
            capi.check(lib.snb_engine_md_steps_graph(
                st.engine, _p(st.crd), _p(st.vel), _p(st.invm), ctypes.c_float(st.dt), st.step,
                case["steps"], st.sp), "md_steps_graph")
            st.step += case["steps"]
            v = st.vel.view(-1, 3)
            v.mul_(torch.sqrt(st.kt3 / (v.square() * st.mass).sum(dtype=torch.float64)).float())
            return {"crd": st.crd, "vel": st.vel}
        if kind == "host":
            for _ in range(case["calls"]):
                capi.check(lib.snb_engine_md_steps_host(
                    st.engine, _p(st.host), ctypes.c_void_p(st.host.data_ptr() + 12 * st.n),
                    _p(st.crd), _p(st.vel), _p(st.invm), ctypes.c_float(st.dt), st.step,
                    case["steps"], st.sp), "md_steps_host")
                st.step += case["steps"]
            return {"crd": st.host[:3 * st.n], "vel": st.host[3 * st.n:]}
        st.frc.zero_()
        if kind == "force":
            capi.check(lib.snb_engine_force(st.engine, _p(st.crd), _p(st.frc), st.step, on, on,
                                            _p(st.totals) if on else None, st.sp),
                       "engine_force")
            st.step += 1
            return {"frc": st.frc, "totals": st.totals} if on else {"frc": st.frc}
        if on:
            for x in (st.ene, st.cou, st.vir, st.pot, st.pvir):
                x.zero_()
        more = [_p(x) for x in (st.ene, st.vir, st.cou, st.pvir, st.pot)] if on else [None] * 5
        e, v, c, pv, pe = more
        if kind == "module":
            _update(st, int(case["rebuild"]))
            capi.check(lib.snb_lj_pme_direct_force(
                st.lj, st.n, st.n, 0, 0, _p(st.crd), _p(st.charge), _p(st.frc), st.bnd, st.nl,
                st.beta, on, e, on, v, c, st.sp), "lj_pme_direct_force")
            capi.check(lib.snb_pme_excluded_force(
                st.pme, st.n, None, None, _p(st.crd), st.bnd, _p(st.charge), _p(st.es),
                _p(st.el), _p(st.en), _p(st.frc), on, e, on, v, st.sp), "pme_excluded_force")
        capi.check(lib.snb_pme_reciprocal_force(
            st.pme, _p(st.crd), st.bnd, _p(st.charge), _p(st.frc), on, on, pv, pe, 0, st.sp),
            "pme_reciprocal_force")
        out = {"frc": st.frc}
        if on:
            out.update(pot=st.pot, pvir=st.pvir)
            if kind == "module":
                out.update(ene=st.ene, cou=st.cou, vir=st.vir)
        return out


# ----------------------------------------------------- what it cannot do without
def _sizes(case):
    """(atoms, grid points, pairs within the cutoff) about."""
    k = case["kind"]
    if k == "pme":
        return 3 * case["nx"] * case["ny"] * case["nz"], case["k0"] * case["k1"] * case["k2"], 0
    if k == "batch":
        w = case["boxes"] * (case["least"] + case["most"]) / 2
    else:
        w = case["waters"]
    pairs = 0.5 * 3 * w * (4 / 3 * math.pi * case["cutoff"] ** 3) * 3 / WATER_A3
    return 3 * w, w * WATER_A3, pairs


def work(case):
    n, grid, pairs = _sizes(case)
    steps = case.get("steps", 1) * case.get("calls", 1)
    per_pair = 47 + (25 if case.get("energy") else 0)
    fft = 2 * 2.5 * grid * math.log2(max(grid, 2))
    flops = steps * (pairs * per_pair + fft + n * 64 * 12)
    io = 12 + 4 + 4 + 12                       # coordinates, charge, type in; forces out
    if case["kind"] in ("md", "soft", "batch", "host"):
        io = 24 + 24 + 12                      # state in and out, charge, type, mass
    if case.get("energy"):
        io += 32 if case["kind"] == "module" else 0
    return {"bytes": float(n * io), "flops": float(flops)}


def tolerance(case):
    """About four times what the library differs by from `exact` over the
    ranges: forces and energies as 32-bit sums give them, trajectories as the
    rounding of the coordinates lets them."""
    if case["kind"] in ("md", "soft", "batch", "host"):
        return {"rel": 6e-4, "max": 5e-2}
    if case["kind"] == "pme":
        return {"rel": 2.5e-5, "max": 2.5e-3}
    return {"rel": 1e-5, "max": 1e-3}


# ------------------------------------------------------------------ in 64 bits
def _beta(rc, tol=1e-5):
    """The reference's bisection, in 32-bit floats."""
    f = np.float32
    erfc = lambda b: f(math.erfc(float(f(b) * f(rc)))) / f(rc)  # noqa: E731
    hi, n = f(1), 50
    while erfc(hi) > f(tol):
        hi, n = f(hi * f(2)), n + 1
    lo = f(0)
    for _ in range(n):
        mid = f((lo + hi) / f(2))
        if erfc(mid) >= f(tol):
            lo = mid
        else:
            hi = mid
    return float(mid)


def _fft_size(length):
    t = (math.ceil(np.float32(length) + 3) >> 2) << 2
    for lo, hi, v in ((60, 68, 64), (120, 136, 128), (240, 272, 256)):
        if lo <= t <= hi:
            t = v
    while t not in _GRID4:
        t += 4
    return t


_GRID4 = {a * b * c * d for a in (4, 8, 16, 32, 64, 128, 256) for b in (1, 3, 9, 27, 81)
          for c in (1, 5, 25, 125) for d in (1, 7, 49)}


def _pairs(x, H, rc):
    """All pairs i < j within rc, nearest image."""
    n, dev = len(x), x.device
    Hi = torch.linalg.inv(H)
    u = x @ Hi
    u = u - torch.floor(u)
    w = u @ H
    heights = 1 / Hi.norm(dim=0)
    nb = [int(v) for v in torch.floor(heights / rc).tolist()]
    out = []
    if min(nb) < 3 or n < 4000:
        step = max(1, 30_000_000 // n)
        for a in range(0, n, step):
            d = w[a:a + step, None] - w[None]
            d = d - torch.round(d @ Hi) @ H
            m = d.square().sum(-1) < rc * rc
            m &= torch.arange(a, min(a + step, n), device=dev)[:, None] < torch.arange(
                n, device=dev)[None]
            i, j = torch.nonzero(m, as_tuple=True)
            out.append(torch.stack([i + a, j]))
        return torch.cat(out, 1)
    nbt = torch.tensor(nb, device=dev)
    c = torch.minimum((u * nbt).long(), nbt - 1)
    cid = (c[:, 0] * nb[1] + c[:, 1]) * nb[2] + c[:, 2]
    order = torch.argsort(cid)
    counts = torch.bincount(cid, minlength=nb[0] * nb[1] * nb[2])
    start = torch.cumsum(counts, 0) - counts
    M = int(counts.max())
    slot = torch.arange(M, device=dev)
    table = (start[:, None] + slot).clamp(max=n - 1)
    table = torch.where(slot < counts[:, None], order[table], torch.full_like(table, -1))
    ids = torch.arange(len(counts), device=dev)
    cx, cy, cz = ids // (nb[1] * nb[2]), ids // nb[2] % nb[1], ids % nb[2]
    offs = [(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)
            if (i, j, k) >= (0, 0, 0)]
    step = max(1, 20_000_000 // (M * M))
    for o in offs:
        to = ((cx + o[0]) % nb[0] * nb[1] + (cy + o[1]) % nb[1]) * nb[2] + (cz + o[2]) % nb[2]
        for a in range(0, len(counts), step):
            A, B = table[a:a + step], table[to[a:a + step]]
            d = w[A][:, :, None] - w[B][:, None]
            d = d - torch.round(d @ Hi) @ H
            m = d.square().sum(-1) < rc * rc
            m &= (A >= 0)[:, :, None] & (B >= 0)[:, None]
            if o == (0, 0, 0):
                m &= A[:, :, None] < B[:, None]
            k, p, q = torch.nonzero(m, as_tuple=True)
            out.append(torch.stack([A[k, p], B[k, q]]))
    return torch.cat(out, 1)


def _image(d, H):
    return d - torch.round(d @ torch.linalg.inv(H)) @ H


def _six(f, d):
    return torch.stack([f[:, 0] * d[:, 0], f[:, 0] * d[:, 1] + f[:, 1] * d[:, 0],
                        f[:, 1] * d[:, 1], f[:, 0] * d[:, 2] + f[:, 2] * d[:, 0],
                        f[:, 1] * d[:, 2] + f[:, 2] * d[:, 1], f[:, 2] * d[:, 2]], 1)


class Exact:
    """One box in 64 bits."""

    def __init__(self, s, case, box=0):
        dev = "cuda"
        f64 = lambda a: torch.from_numpy(np.asarray(a, np.float64)).to(dev)  # noqa: E731
        at = np.flatnonzero(s.box_of == box)
        self.case, self.n = case, len(at)
        self.H = f64(s.cells[box])
        self.rc = float(np.float32(case.get("cutoff", 9.0)))
        self.beta = _beta(self.rc)
        self.x, self.v = f64(s.crd[at]), f64(s.vel[at])
        self.q = f64(s.charge[at])
        self.mass = f64(s.mass[at])[:, None]
        self.invm = f64(np.float32(1) / s.mass[at])[:, None]
        self.type = torch.from_numpy(s.type[at].astype(np.int64)).to(dev)
        self.mol = torch.from_numpy(s.mol[at]).to(dev)
        self.o = torch.from_numpy(s.o[np.isin(s.o, at)].astype(np.int64) - at[0]).to(dev)
        self.A, self.B = f64(s.A), f64(s.B)
        self.soft = case["kind"] == "soft"
        if self.soft:
            self.type_B = torch.from_numpy(s.type_B.astype(np.int64)).to(dev)
            self.BA, self.BB = f64(s.BA), f64(s.BB)
        L = s.cells[box].diagonal()
        self.K = ([case["k0"], case["k1"], case["k2"]] if case["kind"] == "pme" else
                  [_fft_size(v) for v in L])
        self.pairs = None

    def list(self, margin):
        p = _pairs(self.x, self.H, self.rc + margin).sort(0)[0]   # i < j
        self.pairs = p[:, self.mol[p[0]] != self.mol[p[1]]]

    def _terms(self, i, j):
        """Force / r, LJ energy and Coulomb energy of pairs, with r_j - r_i."""
        d = _image(self.x[j] - self.x[i], self.H)
        r2 = d.square().sum(1)
        k = r2 < self.rc ** 2
        i, j, d, r2 = i[k], j[k], d[k], r2[k]
        r = r2.sqrt()
        qq, b = self.q[i] * self.q[j], self.beta
        pick = lambda t, T: T[torch.maximum(t[i], t[j]) * (torch.maximum(t[i], t[j]) + 1) // 2  # noqa
                              + torch.minimum(t[i], t[j])]
        lj_f = lambda A, B, r: (B - A * r ** -6) * r ** -8  # noqa: E731
        lj_e = lambda A, B, r: (A / 12 * r ** -6 - B / 6) * r ** -6  # noqa: E731
        g = 2 / math.sqrt(math.pi)
        cf = lambda r: (b * r * g * torch.exp(-(b * r) ** 2) + torch.erfc(b * r)) * r ** -3  # noqa
        ce = lambda r: torch.erfc(b * r) / r  # noqa: E731
        A, B = pick(self.type, self.A), pick(self.type, self.B)
        if not self.soft:
            return i, j, d, lj_f(A, B, r) - qq * cf(r), lj_e(A, B, r), qq * ce(r)
        C, D = pick(self.type_B, self.BA), pick(self.type_B, self.BB)
        lam = float(np.float32(self.case["lam"]))
        fs = (1 - lam) * lj_f(A, B, r) + lam * lj_f(C, D, r) - qq * cf(r)
        s = torch.nonzero((C * A == 0) & (C + A != 0))[:, 0]
        if len(s):
            s6 = SOFT["soft_core_sigma"] ** 6
            A, B, C, D, r, qq = (t[s] for t in (A, B, C, D, r, qq))
            sig = lambda A, B: torch.where((A == 0) | (B == 0), torch.full_like(A, s6),  # noqa
                                           0.5 * A / B.clamp(min=1e-300))
            got = 0
            for w, l, P, Q in ((1 - lam, lam, A, B), (lam, 1 - lam, C, D)):
                rs = (r ** 6 + SOFT["soft_core_alpha"] * l * sig(P, Q)) ** (1 / 6)
                got = got + w * r ** 4 * ((Q - P * rs ** -6) * rs ** -12
                                          - qq * cf(rs) * rs ** -4)
            fs[s] = got
        return i, j, d, fs, None, None

    def direct(self, energy):
        f = torch.zeros_like(self.x)
        e = torch.zeros(self.n, 2, dtype=torch.float64, device=self.x.device)
        v = torch.zeros(self.n, 6, dtype=torch.float64, device=self.x.device)
        for part in self.pairs.split(10_000_000, 1):
            i, j, d, fs, el, ec = self._terms(part[0], part[1])
            g = fs[:, None] * d
            f.index_add_(0, i, g)
            f.index_add_(0, j, -g)
            if energy:
                e.index_add_(0, i, torch.stack([el, ec], 1))
                v.index_add_(0, i, -_six(g, d))
        return f, e, v

    def excluded(self):
        i = torch.cat([self.o, self.o, self.o + 1])
        j = torch.cat([self.o + 1, self.o + 2, self.o + 2])
        d = _image(self.x[j] - self.x[i], self.H)
        r = d.norm(dim=1)
        b, qq = self.beta * r, self.q[i] * self.q[j]
        fs = -qq * (2 / math.sqrt(math.pi) * b * torch.exp(-b * b) + torch.erfc(b) - 1) / r ** 3
        g = fs[:, None] * d
        f = torch.zeros_like(self.x).index_add_(0, i, g).index_add_(0, j, -g)
        e = torch.zeros_like(self.q).index_add_(0, i, -qq * torch.erf(b) / r)
        return f, e, torch.zeros(self.n, 6, dtype=torch.float64,
                                 device=g.device).index_add_(0, i, -_six(g, d))

    def recip(self):
        dev, K = self.x.device, self.K
        Hi = torch.linalg.inv(self.H)
        u = self.x @ Hi
        u = (u - torch.floor(u)) * torch.tensor(K, device=dev, dtype=torch.float64)
        base = torch.minimum(u.long(), torch.tensor(K, device=dev) - 1)
        t = u - base
        w = torch.stack([t ** 3 / 6, -t ** 3 / 2 + t ** 2 / 2 + t / 2 + 1 / 6,
                         t ** 3 / 2 - t ** 2 + 4 / 6, -t ** 3 / 6 + t ** 2 / 2 - t / 2 + 1 / 6])
        dw = torch.stack([t ** 2 / 2, -1.5 * t ** 2 + t + 0.5, 1.5 * t ** 2 - 2 * t,
                          -t ** 2 / 2 + t - 0.5])
        Q = torch.zeros(K[0] * K[1] * K[2], dtype=torch.float64, device=dev)
        pts = [(a, b, c) for a in range(4) for b in range(4) for c in range(4)]
        at = lambda a, b, c: (((base[:, 0] - a) % K[0]) * K[1] + (base[:, 1] - b) % K[1]  # noqa
                              ) * K[2] + (base[:, 2] - c) % K[2]
        for a, b, c in pts:
            Q.index_add_(0, at(a, b, c), self.q * w[a, :, 0] * w[b, :, 1] * w[c, :, 2])
        F = torch.fft.rfftn(Q.view(*K))
        kk = [torch.fft.fftfreq(K[0], 1 / K[0], device=dev, dtype=torch.float64),
              torch.fft.fftfreq(K[1], 1 / K[1], device=dev, dtype=torch.float64),
              torch.arange(K[2] // 2 + 1, device=dev, dtype=torch.float64)]
        for k, n in zip(kk[:2], K[:2]):
            k[k == -n / 2] = n / 2
        gx, gy, gz = torch.meshgrid(*kk, indexing="ij")
        m = torch.stack([gx * Hi[0, 0], gx * Hi[1, 0] + gy * Hi[1, 1],
                         gx * Hi[2, 0] + gy * Hi[2, 1] + gz * Hi[2, 2]])
        m2 = m.square().sum(0)
        m2[0, 0, 0] = 1
        V = float(torch.linalg.det(self.H))
        pre = (math.pi / self.beta) ** 2
        bc = torch.exp(-pre * m2) / (math.pi * V * m2)
        for d, n in enumerate(K):
            z = torch.arange(n, device=dev, dtype=torch.float64) * (2 * math.pi / n)
            mod = 1 / ((1 / 6 + 4 / 6 * torch.cos(z) + 1 / 6 * torch.cos(2 * z)) ** 2
                       + (4 / 6 * torch.sin(z) + 1 / 6 * torch.sin(2 * z)) ** 2)
            shape = [1, 1, 1]
            shape[d] = -1
            bc = bc * mod[:gz.shape[2] if d == 2 else n].view(shape)
        bc[0, 0, 0] = 0
        half = torch.ones(gz.shape[2], device=dev, dtype=torch.float64)
        half[0] = half[-1] = 0.5
        ew = half * 0.5 * bc * (F.real ** 2 + F.imag ** 2)
        c = 2 / m2 * (1 + pre * m2)
        vir = torch.stack([-(ew * ((1.0 if a == b else 0.0) - c * m[a] * m[b])).sum()
                           for a, b in ((0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2))])
        phi = torch.fft.irfftn(F * bc, s=K, norm="forward").reshape(-1)
        e = 0.5 * (Q * phi).sum()
        g = torch.zeros_like(self.x)
        for a, b, c in pts:
            p = -self.q * phi[at(a, b, c)]
            g += p[:, None] * torch.stack([dw[a, :, 0] * w[b, :, 1] * w[c, :, 2] * K[0],
                                           w[a, :, 0] * dw[b, :, 1] * w[c, :, 2] * K[1],
                                           w[a, :, 0] * w[b, :, 1] * dw[c, :, 2] * K[2]], 1)
        own = (-self.beta / math.sqrt(math.pi) * self.q.square().sum()
               - 0.5 * math.pi / (self.beta ** 2 * V) * self.q.sum() ** 2)
        return g @ Hi.T, e, own, vir

    def bonded(self):
        o, f = self.o, torch.zeros_like(self.x)
        arm = [_image(self.x[o + k] - self.x[o], self.H) for k in (1, 2)]
        r = [a.norm(dim=1, keepdim=True) for a in arm]
        r0, t0 = float(np.float32(R_OH)), float(np.float32(T_HOH))
        for k in (0, 1):
            g = 2 * BOND_K * (r[k] - r0) / r[k] * arm[k]
            f[o] += g
            f[o + 1 + k] -= g
        c = ((arm[0] * arm[1]).sum(1, keepdim=True) / (r[0] * r[1])).clamp(-0.999999, 0.999999)
        k = 2 * ANGLE_K * (torch.acos(c) - t0) / torch.sqrt(1 - c * c)
        ga = k * (arm[1] / (r[0] * r[1]) - c * arm[0] / r[0] ** 2)
        gb = k * (arm[0] / (r[0] * r[1]) - c * arm[1] / r[1] ** 2)
        f[o + 1] += ga
        f[o + 2] += gb
        f[o] -= ga + gb
        return f

    def settle(self, old, dt):
        o, x = self.o, self.x
        sets = ((o, o + 1, R_OH), (o, o + 2, R_OH), (o + 1, o + 2, R_HH))
        was = [_image(old[j] - old[i], self.H) for i, j, _ in sets]
        for _ in range(200):
            worst = 0.0
            for (i, j, r0), w in zip(sets, was):
                d = _image(x[j] - x[i], self.H)
                off = d.square().sum(1, keepdim=True) - float(np.float32(r0)) ** 2
                g = off / (2 * (self.invm[i] + self.invm[j]) * (d * w).sum(1, keepdim=True))
                for a, sign in ((i, 1.0), (j, -1.0)):
                    x[a] += sign * g * self.invm[a] * w
                    self.v[a] += sign * g * self.invm[a] * w / dt
                worst = max(worst, float(off.abs().max()))
            if worst < 1e-13:
                break

    def md(self, steps, dt, rigid):
        for k in range(steps):
            if k % 10 == 0:
                self.list(1.0)
            f = self.direct(False)[0] + self.excluded()[0] + self.recip()[0]
            if not rigid:
                f = f + self.bonded()
            old = self.x.clone()
            self.v = self.v + dt * f * self.invm
            self.x = self.x + dt * self.v
            if rigid:
                self.settle(old, dt)


def exact(case, seed):
    n, _, pairs = _sizes(case)
    kind = case["kind"]
    steps = case.get("steps", 1) * case.get("calls", 1)
    if pairs * steps > 1e9 or kind == "batch" and case["boxes"] * steps > 700:
        return None
    s = _system(case, seed)
    if kind in ("md", "soft", "batch", "host"):
        dt = float(np.float32(1e-3 * TIME * (2.0 if case.get("rigid") else 0.5)))
        boxes = [Exact(s, case, b) for b in range(len(s.cells))]
        for b in boxes:
            b.md(steps, dt, bool(case.get("rigid")))
        x, v, m = (torch.cat([getattr(b, k) for b in boxes]) for k in ("x", "v", "mass"))
        if kind == "host":
            return {"crd": x.reshape(-1).cpu(), "vel": v.reshape(-1).cpu()}
        dof = 3 * s.n
        if case.get("rigid"):
            dof = 2 * s.n if not case["ions"] else 6 * len(s.o) + 3 * (s.n - 3 * len(s.o))
        v = v * torch.sqrt(dof * KB * 300.0 / (v.square() * m).sum())
        return {"crd": x.reshape(-1), "vel": v.reshape(-1)}
    b = Exact(s, case)
    on = bool(case["energy"])
    f, e, own, vir = b.recip()
    if kind == "pme":
        out = {"frc": f.reshape(-1)}
        if on:
            out.update(pot=(e + own).reshape(1), pvir=vir)
        return out
    b.list(0.0)
    fd, ed, vd = b.direct(on)
    fx, ex, vx = b.excluded()
    f = (f + fd + fx).reshape(-1)
    if not on:
        return {"frc": f}
    if kind == "module":
        return {"frc": f, "pot": (e + own).reshape(1), "pvir": vir, "ene": ed.sum(1) + ex,
                "cou": ed[:, 1], "vir": vd + vx}
    cnt = np.bincount(s.type, minlength=s.n_types).astype(np.float64)
    i, j = np.tril_indices(s.n_types)
    c6 = float((np.where(i == j, 1.0, 2.0) * cnt[i] * cnt[j] * s.B.astype(np.float64)).sum())
    tail = -2.0 / 3.0 * math.pi * c6 / b.rc ** 3 / 6.0 / float(torch.linalg.det(b.H))
    t = torch.zeros(14, dtype=torch.float64, device=f.device)
    t[0], t[1], t[2], t[3] = ed[:, 0].sum(), tail, ed[:, 1].sum(), ex.sum()
    t[4], t[5] = e, own
    t[7] = t[:7].sum()
    t[8:] = vd.sum(0) + vx.sum(0) + vir
    t[[8, 10, 13]] += 2 * tail
    return {"frc": f, "totals": t}
