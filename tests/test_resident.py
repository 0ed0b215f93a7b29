"""Runs of many steps with the state held on chip (lfm_leapfrog_run_f32).

The on-chip run computes the single steps' arithmetic, so every result is compared
with single steps bit for bit: at the smallest and largest lattices it takes, at odd
edges and at edges that are no multiple of the two cells a thread owns, at even and
odd step counts, across several launches and on two streams at once.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from lfm_b200 import _lib
from lfm_b200.config import gravity_em, gravity_only

REAL, COMPLEX = 0, 1
FIELD_FLOATS = {REAL: 22656, COMPLEX: 16448}
SMEM_LIMIT = 227 * 1024 - 1024


def plan(level, N, sms=148):
    v = (ctypes.c_int * 8)()
    if _lib.load().lfm_leapfrog_run_plan(level, N, sms, v) != _lib.LFM_OK:
        return None
    return dict(zip(("nbi", "nbj", "NI", "NJ", "V", "segs", "threads", "smem"), v))


@pytest.mark.parametrize("level", [REAL, COMPLEX])
def test_plan_cuts_every_lattice_that_fits(level):
    """Blocks within the SMs, threads and shared memory; every cell in one thread's march."""
    fits = []
    for N in range(8, 129):
        p = plan(level, N)
        if p is None:
            continue
        fits.append(N)
        assert p["nbi"] * p["nbj"] <= 148 and p["threads"] <= 512 and p["smem"] <= SMEM_LIMIT
        RS = (N + 3) // 4 * 4 + 4
        rows = 2 * p["NI"] * p["NJ"] + 2 * (p["NJ"] + 2) + 2 * p["NI"]
        assert 4 + rows * RS <= FIELD_FLOATS[level]
        groups = -(-N // p["V"])
        for nb, most in ((p["nbi"], p["NI"]), (p["nbj"], p["NJ"])):
            cut = [b * N // nb for b in range(nb + 1)]
            assert cut[0] == 0 and cut[-1] == N
            assert all(1 <= b - a <= most for a, b in zip(cut, cut[1:]))
        assert p["segs"] * p["NJ"] * groups <= p["threads"]
        for ni in {(b + 1) * N // p["nbi"] - b * N // p["nbi"] for b in range(p["nbi"])}:
            seg = [s * ni // p["segs"] for s in range(p["segs"] + 1)]
            assert seg[0] == 0 and seg[-1] == ni
    assert fits == list(range(8, 109 if level == REAL else 97))
    assert plan(2, 32) is None and plan(level, 7) is None
    assert plan(level, 16, sms=1) is not None  # one block, its own neighbour


# ------------------------------------------------------------------ on the GPU
def _evolver(level, N, seed, be):
    from lfm_b200 import Evolver

    ev = Evolver((gravity_em if level else gravity_only)(N), backend=be)
    rng = np.random.default_rng(seed)
    f = lambda a: (a * rng.standard_normal((N, N, N))).astype(np.float32)  # noqa: E731
    ev.set_psi_real(f(0.5))
    ev.set_psi_real_prev(f(0.5))
    if level:
        ev.set_psi_imag(f(0.5))
        ev.set_psi_imag_prev(f(0.5))
    ev.set_chi((19.0 + f(1e-2)).astype(np.float32))
    return ev


def _same(a, b):
    import torch

    sa, sb = a.device_state(), b.device_state()
    sa["chi_prev"], sb["chi_prev"] = a._buf("chi_prev_A"), b._buf("chi_prev_A")
    assert sa.keys() == sb.keys()
    for k in sa:
        assert torch.equal(sa[k].view(torch.int32), sb[k].view(torch.int32)), k
    assert (a.step, a._use_buffer_A, a._cur) == (b.step, b._use_buffer_A, b._cur)


@pytest.fixture(scope="module")
def be(cuda_device):
    from lfm_b200 import B200Backend
    from lfm_b200.build import build_library

    build_library()
    return B200Backend(cuda_device)


@pytest.mark.gpu
@pytest.mark.parametrize("level,N", [(REAL, n) for n in (8, 9, 15, 30, 32, 33, 63, 66, 96, 97, 107,
                                                         108, 109)]
                         + [(COMPLEX, n) for n in (8, 9, 15, 30, 32, 33, 63, 66, 95, 96, 97)])
def test_run_equals_single_steps(be, level, N):
    a, b = _evolver(level, N, N, be), _evolver(level, N, N, be)
    b.use_graphs = False
    fits = plan(level, N) is not None
    for steps in (4, 5, 9):  # the first from undamped previous fields; both slot parities
        a.evolve(steps)
        b.evolve(steps)
        assert (a._run_sync is not None and a._run_sync.numel() > 0) == fits
        _same(a, b)
    a.run_block = 6  # several launches, and a single step left over
    a.evolve(19)
    b.evolve(19)
    _same(a, b)
    a.synchronize()


@pytest.mark.gpu
def test_forced_path_and_tile_keep_the_single_steps(be):
    a, b = _evolver(REAL, 32, 1, be), _evolver(REAL, 32, 1, be)
    b.use_graphs = False
    try:
        for path in (_lib.PATH_DIRECT, _lib.PATH_FUSED):
            _lib.set_step_path(path)
            assert not a._run_on_chip(4)
            a.evolve(6)
            b.evolve(6)
            _same(a, b)
    finally:
        _lib.set_step_path(_lib.PATH_AUTO)
    _lib.tune_set(REAL, 32, 8, 3, 8, 4)
    try:
        assert not a._run_on_chip(4)
    finally:
        _lib.tune_set(REAL, 32, 0, 0)
    assert not a._run_on_chip(1)


@pytest.mark.gpu
def test_no_memory_for_the_workspace_keeps_the_single_steps(be, monkeypatch):
    import torch

    a, b = _evolver(COMPLEX, 16, 3, be), _evolver(COMPLEX, 16, 3, be)

    def no_memory(*args, **kwargs):
        raise torch.OutOfMemoryError("planted")

    with monkeypatch.context() as m:
        m.setattr(torch, "zeros", no_memory)
        a.evolve(9)
    assert a._run_sync.numel() == 0
    b.use_graphs = False
    b.evolve(9)
    _same(a, b)


@pytest.mark.gpu
def test_two_lattices_on_two_streams(be):
    """Launches that wait on one another's CTAs only: two at a time do not mix."""
    import torch

    pairs = [(_evolver(REAL, 64, 3, be), _evolver(REAL, 64, 3, be)),
             (_evolver(COMPLEX, 96, 4, be), _evolver(COMPLEX, 96, 4, be))]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(be.device) for _ in pairs]
    for _ in range(4):
        for (a, _), s in zip(pairs, streams):
            with torch.cuda.stream(s):
                a.evolve(50)
    torch.cuda.synchronize()
    for a, b in pairs:
        b.use_graphs = False
        b.evolve(200)
        _same(a, b)
        a.synchronize()


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [[(8, REAL), (108, REAL), (96, COMPLEX), (12, COMPLEX)],
                                   [(32, REAL)] * 40 + [(32, COMPLEX)] * 35,
                                   [(96, REAL), (64, COMPLEX), (80, COMPLEX), (48, REAL)] * 2])
def test_batch_waves_equal_single_steps(be, sizes):
    """Smallest and largest lattices, more than a wave's lattices, mixed waves: each lattice
    comes out as the one-step batch kernel gives it, at odd and even step counts."""
    import torch

    from lfm_b200.batch import BatchedLattices

    cfgs = [(gravity_em if lv else gravity_only)(n, kappa=(1 + i % 3) / 63.0)
            for i, (n, lv) in enumerate(sizes)]
    a, b = BatchedLattices(cfgs, backend=be), BatchedLattices(cfgs, backend=be)
    b._on_chip = False
    rng = np.random.default_rng(len(sizes))
    for i, (n, lv) in enumerate(sizes):
        f = [(0.5 * rng.standard_normal((n, n, n))).astype(np.float32) for _ in range(3)]
        for e in (a, b):
            e.set_psi_real(i, f[0])
            e.set_psi_real_prev(i, f[2])
            if lv:
                e.set_psi_imag(i, f[1])
            e.set_chi(i, (19.0 + 1e-2 * f[2]).astype(np.float32))
    a.run_block = 6
    for steps in (4, 5, 13):
        a.evolve(steps)
        b.evolve(steps)
        assert (a._cur, a.step) == (b._cur, b.step)
        for i in range(len(sizes)):
            sa, sb = a.device_state(i), b.device_state(i)
            for k in sa:
                assert torch.equal(sa[k].view(torch.int32), sb[k].view(torch.int32)), (i, k)
    a.get_chi(0)  # raises if a wait gave up


@pytest.mark.gpu
def test_batch_keeps_single_steps_where_it_must(be):
    from lfm_b200.batch import BatchedLattices

    big = BatchedLattices([gravity_only(112), gravity_only(32)], backend=be)
    assert not big._run_on_chip(4)  # 112^3 does not fit
    assert not BatchedLattices([gravity_only(32)], backend=be, tuning={"threads": 256})._on_chip
    small = BatchedLattices([gravity_only(32)], backend=be)
    assert not small._run_on_chip(1)
    _lib.set_step_path(_lib.PATH_DIRECT)
    try:
        assert not small._run_on_chip(4)
    finally:
        _lib.set_step_path(_lib.PATH_AUTO)


@pytest.mark.gpu
def test_a_workspace_made_under_capture_is_not_kept(be):
    """Its zeroes come with the graph's replays: runs outside the graph need their own."""
    import torch

    from lfm_b200 import adjoint

    a, b = _evolver(COMPLEX, 32, 5, be), _evolver(COMPLEX, 32, 5, be)
    b.use_graphs = False
    a.evolve(3)
    b.evolve(3)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a.evolve(8)
    a.step -= 8  # nothing has run yet
    assert a._run_sync is None
    for again in (lambda: a.evolve(8), g.replay, lambda: a.evolve(8), g.replay):
        again()
        b.evolve(8)
        a.step = b.step
        _same(a, b)
    assert a._run_sync.numel() > 0
    a.synchronize()

    lat = adjoint._lattice_for(gravity_em(36, kappa=1.25 / 63.0), be)
    state = [t.clone().reshape(36, 36, 36) for t in lat.state()]
    g = torch.cuda.CUDAGraph()
    with torch.no_grad():
        with torch.cuda.graph(g):
            adjoint.leapfrog(lat.config, state, 6, backend=be)
        assert lat.run_sync is None
        adjoint.leapfrog(lat.config, state, 6, backend=be)
    assert lat.run_sync.numel() > 0


@pytest.mark.gpu
def test_warm_graphs_captures_what_evolve_replays(be):
    """Graphs for lattices that take single steps; for the others the workspace."""
    import torch

    from lfm_b200.batch import BatchedLattices

    graphs = lambda ev: len(getattr(ev, "_graphs", {}))  # noqa: E731
    for n, forced in ((32, False), (110, False), (32, True)):
        ev = _evolver(REAL, n, 1, be)
        ev.evolve(1)
        if forced:
            _lib.tune_set(REAL, n, 8, 3, 8, 4)
        try:
            ev.warm_graphs()
            fits = n == 32 and not forced
            assert graphs(ev) == (0 if fits else 2)
            assert (ev._run_sync is not None and ev._run_sync.numel() > 0) == fits
            before = torch.cuda.memory_stats(be.device)["allocation.all.allocated"]
            ev.evolve(9)
            assert torch.cuda.memory_stats(be.device)["allocation.all.allocated"] == before
            assert graphs(ev) == (0 if fits else 2)
        finally:
            _lib.tune_set(REAL, n, 0, 0)
    for tuning in (None, dict(threads=128)):
        B = BatchedLattices([gravity_only(32), gravity_em(16)], backend=be, tuning=tuning)
        B.evolve(1)
        B.warm_graphs()
        assert len(B._graphs) == (0 if tuning is None else 4)


@pytest.mark.parametrize("level", [REAL, COMPLEX])
def test_blocks_of_small_lattices_share_an_sm(level):
    """Shared memory by what a small lattice needs, so that runs on several streams find
    room beside one another (REAL takes 144 registers a thread, COMPLEX 160)."""
    for N in range(8, 37):
        p = plan(level, N)
        assert 2 * (p["smem"] + 1024) <= 227 * 1024
        assert 2 * p["threads"] * (160 if level else 144) <= 65536


@pytest.mark.gpu
@pytest.mark.parametrize("level", [REAL, COMPLEX])
def test_many_small_lattices_on_many_streams(be, level):
    import torch

    sizes = [8, 15, 24, 32, 33, 36, 37, 48, 16, 32, 36, 20]
    pairs = [(_evolver(level, n, n, be), _evolver(level, n, n, be)) for n in sizes]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(be.device) for _ in pairs]
    for _ in range(3):
        for (a, _), s in zip(pairs, streams):
            with torch.cuda.stream(s):
                a.evolve(200)
    torch.cuda.synchronize()
    for a, b in pairs:
        b.use_graphs = False
        b.evolve(600)
        _same(a, b)
        a.synchronize()
