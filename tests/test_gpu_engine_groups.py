"""The engine's grouped rows (k_group_search, k_lj_groups) where they can go
wrong: boxes so small that each pair is imaged by itself, groups of every size
from one atom to eight, rows of less than a batch and of several, a cutoff at
which beta r leaves the erfc polynomial, more than two exclusions per atom, and
charges and LJ types that differ inside a group.

The pair set must be the oracle's bit for bit.  Forces: each pair's terms are
32-bit (relative error below 1.1e-6, the erfc polynomial's), summed in 32 bits
over at most 64 partners of a lane, so 1e-5 relative RMS against FP64 leaves a
factor of five; energies within 2e-6, as in test_gpu_engine.py."""

import ctypes
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    import torch
    assert torch.cuda.is_available(), "GPU tests need CUDA"
    from tests import gpu_helpers
    return gpu_helpers


def _pairs(g, e):
    import torch
    lib = g.capi.load()
    cnt = ctypes.c_longlong(0)
    g.capi.check(lib.snb_engine_stats(e, None, ctypes.byref(cnt), g.stream()), "stats")
    n = cnt.value
    pi = torch.empty(max(n, 1), dtype=torch.int32, device="cuda")
    pj = torch.empty(max(n, 1), dtype=torch.int32, device="cuda")
    got = ctypes.c_longlong(0)
    g.capi.check(lib.snb_engine_export_pairs(e, g.ptr(pi), g.ptr(pj), n, ctypes.byref(got),
                                             g.stream()), "export")
    assert got.value == n
    p = np.stack([pi[:n].cpu().numpy(), pj[:n].cpu().numpy()], 1).astype(np.int64)
    return p[np.lexsort((p[:, 1], p[:, 0]))]


def _want(oracle, s, cutoff, tol=1e-5):
    """FP64 forces of the engine's terms over the oracle's pairs."""
    from sponge_b200 import systems
    rs, cols = oracle.nl_pairs_system(s, cutoff, 2.0)
    beta = oracle.get_beta(cutoff, tol)
    return (oracle.direct_f64(s, cutoff, beta, rs, cols)["frc"] +
            oracle.excluded_f64(s, beta)["frc"] +
            oracle.pme_f64(s, (systems.fft_size(s.box),) * 3, beta)["frc"])


def _spread_and_packed(waters=1000, factor=1.8):
    """The same molecules twice in one large box: drawn apart over all of it,
    and as a dense block in one corner, whose rows outgrow the capacity that
    the mean density gave."""
    from sponge_b200 import systems
    s = systems.water_box(waters, seed=21)
    o = np.repeat(s.crd[::3], 3, axis=0)
    apart = (s.crd - o) + o * np.float32(factor)
    return (dataclasses.replace(s, crd=apart.astype(np.float32), box=s.box * factor),
            dataclasses.replace(s, box=s.box * factor))


def _check(g, oracle, s, cutoff, tol=1e-5):
    import torch
    from sponge_b200 import systems
    lib = g.capi.load()
    e = g.engine_create(s, cutoff, PM_Direct_Tolerance=tol)
    crd = g.dev(s.crd.reshape(-1), np.float32)
    frc = torch.zeros(3 * s.n, dtype=torch.float32, device="cuda")
    only = torch.zeros(3 * s.n, dtype=torch.float32, device="cuda")
    tot = torch.zeros(16, dtype=torch.float64, device="cuda")
    try:
        g.capi.check(lib.snb_engine_force(e, g.ptr(crd), g.ptr(frc), 0, 1, 1, g.ptr(tot),
                                          g.stream()), "engine_force")
        g.capi.check(lib.snb_engine_force(e, g.ptr(crd), g.ptr(only), 1, 0, 0, None, g.stream()),
                     "engine_force")
        got = _pairs(g, e)
    finally:
        lib.snb_engine_destroy(e)
    rs, cols = oracle.nl_pairs_system(s, cutoff, 2.0)
    assert np.array_equal(got, g.csr_to_pairs(rs, cols))
    beta = oracle.get_beta(cutoff, tol)
    d, x = oracle.direct_f64(s, cutoff, beta, rs, cols), oracle.excluded_f64(s, beta)
    p = oracle.pme_f64(s, (systems.fft_size(s.box),) * 3, beta)
    want = d["frc"] + x["frc"] + p["frc"]
    assert g.rel_rms(frc.cpu().numpy().reshape(s.n, 3), want) <= 1e-5
    assert g.rel_rms(only.cpu().numpy().reshape(s.n, 3), want) <= 1e-5
    t = tot.cpu().numpy()
    assert abs(t[0] - d["lj_energy"].sum()) <= 2e-6 * np.abs(d["lj_energy"]).sum()
    assert abs(t[2] - d["coulomb_energy"].sum()) <= 2e-6 * np.abs(d["coulomb_energy"]).sum()
    vir = d["virial"].sum(0) + x["virial"].sum(0) + p["virial"]
    lrc = oracle.lrc_factor(s, cutoff) / float(np.float32(s.box)) ** 3
    vir[[0, 2, 5]] += 2 * lrc
    assert np.abs(t[8:14] - vir).max() <= 2e-6 * np.abs(vir).max()


@pytest.mark.parametrize("waters,cutoff,tol", [
    (200, 8.0, 1e-5),    # half the box 9.07 A: every pair imaged, 3 cells per axis
    (231, 9.0, 1e-5),    # the cutoff just below half the box
    (200, 10.0, 1e-5),   # the cutoff beyond half the box: nearest images only
    (700, 7.3, 1e-5),    # 5 cells per axis: trimmed runs, some groups imaged
    (1500, 9.0, 1e-9),   # beta * cutoff = 4.3: beyond the polynomial
    (2600, 6.1, 1e-5),   # narrow cells: groups of a few atoms
    (1400, 15.0, 1e-5),  # rows beyond the search's buffer, eight warps per group
    (1700, 15.0, 1e-5),  # the same with four
])
def test_groups_match_fp64(g, oracle, waters, cutoff, tol):
    from sponge_b200 import systems
    s = systems.water_box(waters, seed=waters, ion_pairs=None)
    _check(g, oracle, s, cutoff, tol)


@pytest.mark.parametrize("waters", [1, 2, 5])
def test_smallest_boxes(g, oracle, waters):
    """One group or a few, in a box of empty cells.  A water's excluded and
    reciprocal forces on itself nearly cancel (each about 4 kcal/mol/A, their
    sum 0.03), so the error is held to the terms' sizes: 1e-5 of them, the
    reciprocal part going through a float FFT and a grid in steps of 2^-22
    (up to 6e-6 of its size against FP64 on a full box)."""
    from sponge_b200 import systems
    s = dataclasses.replace(systems.water_box(waters, seed=2), box=26.0)
    lib = g.capi.load()
    e = g.engine_create(s, 8.0)
    try:
        got = _force_of(g, e, g.dev(s.crd.reshape(-1), np.float32), s.n, 0)
        pairs = _pairs(g, e)
    finally:
        lib.snb_engine_destroy(e)
    rs, cols = oracle.nl_pairs_system(s, 8.0, 2.0)
    assert np.array_equal(pairs, g.csr_to_pairs(rs, cols))
    beta = oracle.get_beta(8.0)
    terms = [oracle.direct_f64(s, 8.0, beta, rs, cols)["frc"],
             oracle.excluded_f64(s, beta)["frc"],
             oracle.pme_f64(s, (systems.fft_size(s.box),) * 3, beta)["frc"]]
    size = sum(np.linalg.norm(t) for t in terms)
    assert np.linalg.norm(got - sum(terms)) <= 1e-5 * size


def test_long_rows_of_a_large_box(g, oracle):
    """Rows beyond the search's buffer where one warp takes a group."""
    from sponge_b200 import systems
    s = systems.water_box(19500, seed=4, ion_pairs=None)
    lib = g.capi.load()
    e = g.engine_create(s, 15.0)
    try:
        got = _force_of(g, e, g.dev(s.crd.reshape(-1), np.float32), s.n, 0)
    finally:
        lib.snb_engine_destroy(e)
    assert g.rel_rms(got, _want(oracle, s, 15.0)) <= 1e-5


def test_sparse_and_dense_cells(g, oracle):
    """Most waters in one corner: empty cells, cells of one molecule and cells
    of many groups; rows from empty to regrown."""
    from sponge_b200 import systems
    s = systems.water_box(900, seed=5)
    rng = np.random.default_rng(5)
    keep = np.ones(s.n, bool)
    o = s.crd[::3] - np.floor(s.crd[::3] / s.box) * s.box
    far = (o.max(1) > 0.55 * s.box) & (rng.random(len(o)) < 0.93)
    keep = np.repeat(~far, 3)
    _check(g, oracle, systems._subset(s, keep), 6.5)


def test_many_exclusions_and_types(g, oracle):
    """Chains of 24 waters excluded from one another (up to 71 partners, beyond
    the 16 that the build keeps per atom) and four LJ types dealt out at
    random."""
    from sponge_b200 import systems
    s = systems.water_box(1000, seed=8)
    rng = np.random.default_rng(8)
    lists = []
    for i in range(s.n):
        end = min(s.n, (i // 72 + 1) * 72)
        lists.append(np.arange(i + 1, end) if (i // 72) % 3 == 0 else
                     np.arange(i + 1, (i // 3 + 1) * 3))
    numbers = np.array([len(x) for x in lists], np.int32)
    start = np.concatenate([[0], np.cumsum(numbers)[:-1]]).astype(np.int32)
    s = dataclasses.replace(s, excl_start=start, excl_numbers=numbers,
                            excl_list=np.concatenate(lists).astype(np.int32))
    s.lj_type[::3] = rng.choice([0, 2, 3], len(s.lj_type[::3]))
    _check(g, oracle, s, 7.0)


def _force_of(g, e, crd, n, step, sp=None):
    import torch
    frc = torch.zeros(3 * n, dtype=torch.float32, device="cuda")
    g.capi.check(g.capi.load().snb_engine_force(e, g.ptr(crd), g.ptr(frc), step, 0, 0, None,
                                                sp or g.stream()), "engine_force")
    torch.cuda.synchronize()
    return frc.cpu().numpy().reshape(n, 3)


@pytest.mark.parametrize("ask", ["stats", "export"])
def test_overflow_seen_between_steps_rebuilds(g, oracle, ask):
    """A later rebuild outgrows the rows and a call between steps is the first
    to see it: the count is the new frame's, the export is refused, and the
    next force on the same coordinates and the next graph steps (captured
    before with the old rows) build the list again."""
    import torch
    from sponge_b200 import systems
    spread, packed = _spread_and_packed()
    lib = g.capi.load()
    e = g.engine_create(spread, 7.0)
    g.engine_set_water_bonded(e, spread)
    state = g.dev(spread.crd.reshape(-1), np.float32)
    vel = torch.zeros_like(state)
    invm = g.dev((1.0 / spread.mass).astype(np.float32))
    dense = g.dev(packed.crd.reshape(-1), np.float32)
    dt = ctypes.c_float(1e-4 * systems.TIME_CONVERSION)
    st = torch.cuda.Stream()
    sp = ctypes.c_void_p(st.cuda_stream)
    pi = torch.empty(1, dtype=torch.int32, device="cuda")
    count = ctypes.c_longlong(0)

    def steps(first):
        g.capi.check(lib.snb_engine_md_steps_graph(e, g.ptr(state), g.ptr(vel), g.ptr(invm), dt,
                                                   first, 3, sp), "md")
        st.synchronize()

    try:
        torch.cuda.synchronize()
        steps(1)
        _force_of(g, e, dense, packed.n, 1, sp)
        if ask == "stats":
            g.capi.check(lib.snb_engine_stats(e, None, ctypes.byref(count), sp), "stats")
        else:
            assert lib.snb_engine_export_pairs(e, g.ptr(pi), g.ptr(pi), 1, ctypes.byref(count),
                                               sp) != 0
        rs, cols = oracle.nl_pairs_system(packed, 7.0, 2.0)
        assert count.value == len(cols)
        assert lib.snb_engine_export_pairs(e, g.ptr(pi), g.ptr(pi), count.value,
                                           ctypes.byref(count), sp) != 0
        assert b"builds them again" in lib.snb_last_error()
        got = _force_of(g, e, dense, packed.n, 1, sp)
        assert g.rel_rms(got, _want(oracle, packed, 7.0)) <= 1e-5
        assert np.array_equal(_pairs(g, e), g.csr_to_pairs(rs, cols))
        before = state.clone()
        steps(4)
        assert torch.isfinite(state).all() and not torch.equal(state, before)
    finally:
        lib.snb_engine_destroy(e)


def test_module_list_overflow_between_updates_rebuilds(g, oracle):
    """The modules' rows likewise: emptied by the count that found them too
    short, refused to the export, built by the next conditional update."""
    spread, packed = _spread_and_packed()
    lib = g.capi.load()
    box, dense = g.Box(spread), g.Box(packed)
    h = g.make_nl(box, 7.0, 2.0)
    import torch
    pi = torch.empty(1, dtype=torch.int32, device="cuda")
    count = ctypes.c_longlong(0)
    try:
        g.nl_update(h, box)
        g.nl_update(h, dense)
        g.capi.check(lib.snb_nl_pair_count(h, ctypes.byref(count), g.stream()), "count")
        rs, cols = oracle.nl_pairs_system(packed, 7.0, 2.0)
        assert count.value == len(cols)
        assert lib.snb_nl_export_pairs(h, g.ptr(pi), g.ptr(pi), count.value,
                                       ctypes.byref(count), g.stream()) != 0
        assert b"builds them again" in lib.snb_last_error()
        g.nl_update(h, dense, forced=0)
        assert np.array_equal(g.nl_pairs(h), g.csr_to_pairs(rs, cols))
    finally:
        lib.snb_nl_destroy(h)


def test_regrown_rows_beside_default_stream_work(g, oracle):
    """Rows regrown in the first build, and the pruned rows' bytes made by a
    new margin, while the legacy default stream is busy: a non-blocking stream
    does not wait for that one, so clears left on it could land after the
    rebuild's or the prune pass's writes."""
    import torch
    from sponge_b200 import systems
    spread, packed = _spread_and_packed()
    lib = g.capi.load()
    e = g.engine_create(spread, 7.0)
    dense = g.dev(packed.crd.reshape(-1), np.float32)
    vel = torch.zeros_like(dense)
    invm = g.dev((1.0 / packed.mass).astype(np.float32))
    dt = ctypes.c_float(1e-4 * systems.TIME_CONVERSION)
    st = torch.cuda.Stream()
    sp = ctypes.c_void_p(st.cuda_stream)
    frc = torch.zeros(3 * packed.n, dtype=torch.float32, device="cuda")
    want = _want(oracle, packed, 7.0)
    try:
        for _ in range(2):
            torch.cuda.synchronize()
            frc.zero_()
            torch.cuda._sleep(20_000_000)  # about 10 ms
            st.wait_stream(torch.cuda.default_stream())
            torch.cuda._sleep(20_000_000)
            g.capi.check(lib.snb_engine_force(e, g.ptr(dense), g.ptr(frc), 0, 0, 0, None, sp),
                         "engine_force")
            torch.cuda.synchronize()
            assert g.rel_rms(frc.cpu().numpy().reshape(-1, 3), want) <= 1e-5
            moved = dense.clone()
            vel.zero_()
            torch.cuda.synchronize()
            torch.cuda._sleep(20_000_000)
            g.capi.check(lib.snb_engine_set_prune_margin(e, ctypes.c_float(0.5)), "margin")
            g.capi.check(lib.snb_engine_md_steps_graph(e, g.ptr(moved), g.ptr(vel), g.ptr(invm),
                                                       dt, 1, 2, sp), "md")
            torch.cuda.synchronize()
            kick = dt.value * want
            got = (vel.cpu().numpy() * packed.mass.repeat(3)).reshape(-1, 3)
            assert g.rel_rms(got, 2 * kick) <= 0.05  # two short steps along the force
    finally:
        lib.snb_engine_destroy(e)


@pytest.mark.parametrize("waters,cutoff", [(900, 8.0), (300, 8.0)])
def test_kept_list_holds_only_its_pairs(g, oracle, waters, cutoff):
    """A list that is older than the displacement rule allows (rebuilt at an
    interval instead): the forces are those of the pairs within cutoff + skin
    at the build, whatever has come within the cutoff since beside them."""
    from sponge_b200 import systems
    s = systems.water_box(waters, seed=13)
    rng = np.random.default_rng(13)
    shift = np.repeat(rng.uniform(-0.25, 0.25, (s.n // 3 + 1, 3)), 3, axis=0)[:s.n]
    moved = dataclasses.replace(s, crd=(s.crd + shift).astype(np.float32))
    lib = g.capi.load()
    e = g.engine_create(s, cutoff, skin=0.05, neighbor_list_refresh_interval=1000)
    try:
        _force_of(g, e, g.dev(s.crd.reshape(-1), np.float32), s.n, 0)
        got = _force_of(g, e, g.dev(moved.crd.reshape(-1), np.float32), s.n, 1)
    finally:
        lib.snb_engine_destroy(e)
    rs, cols = oracle.nl_pairs_system(s, cutoff, 0.05)
    new_rs, new_cols = oracle.nl_pairs_system(moved, cutoff, 0.05)
    beta = oracle.get_beta(cutoff)
    other = (oracle.excluded_f64(moved, beta)["frc"] +
             oracle.pme_f64(moved, (systems.fft_size(s.box),) * 3, beta)["frc"])
    want = oracle.direct_f64(moved, cutoff, beta, rs, cols)["frc"] + other
    fresh = oracle.direct_f64(moved, cutoff, beta, new_rs, new_cols)["frc"] + other
    assert g.rel_rms(got, want) <= 1e-5
    assert g.rel_rms(fresh, want) >= 5e-5  # the list's age shows at this tolerance


def test_box_beyond_32_bit_rows_is_refused(g):
    """1.2 M atoms at a cutoff of 20 A (2,230 pairs per atom): the list would
    hold more than 2^31 pairs.  A row per atom never took such a box, and the
    grouped rows do not either."""
    lib = g.capi.load()
    n, box = 1_200_000, (1_200_000 / 0.1) ** (1 / 3)
    L = np.float32(box)
    cell = np.array([L, 0, L, 0, 0, L], np.float32)
    rcell = np.array([1 / L, 0, 1 / L, 0, 0, 1 / L], np.float32)
    h = ctypes.c_void_p()
    o = g.capi.options(cutoff=20.0, skin=2.0)
    zero, none = np.zeros(n, np.int32), np.zeros(1, np.float32)
    q = np.zeros(n, np.float32)
    rc = lib.snb_engine_create(ctypes.byref(o), n, g.capi.boundary(cell, rcell), 1,
                               zero.ctypes.data, none.ctypes.data, none.ctypes.data,
                               q.ctypes.data, zero.ctypes.data, zero.ctypes.data,
                               zero.ctypes.data, 0, ctypes.byref(h))
    if rc == 0:
        lib.snb_engine_destroy(h)
    assert rc != 0 and b"32-bit offsets" in lib.snb_last_error()


def test_droplet_in_a_large_box_takes_rows_by_atoms(g, oracle):
    """1,000 waters in a box of 85,000 cells: right, and held in rows for the
    3,000 atoms (n / 8 + n rows of some 600 entries, 8 MB) instead of rows for
    the cells (0.2 GB)."""
    import torch
    from sponge_b200 import systems
    lib = g.capi.load()
    s = dataclasses.replace(systems.water_box(1000, seed=3), box=200.0)
    crd = g.dev(s.crd.reshape(-1), np.float32)

    def run():
        e = g.engine_create(s, 7.0, PM_grid_spacing=6.0)
        _force_of(g, e, crd, s.n, 0)
        return e

    lib.snb_engine_destroy(run())  # modules loaded
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    e = run()
    try:
        used = free - torch.cuda.mem_get_info()[0]
        got = _pairs(g, e)
    finally:
        lib.snb_engine_destroy(e)
    rs, cols = oracle.nl_pairs_system(s, 7.0, 2.0)
    assert np.array_equal(got, g.csr_to_pairs(rs, cols))
    assert used < 100e6
