"""The marching kernel for lattices without 16-byte rows against the direct kernel.

Both evaluate lfm_cells.cuh's arithmetic, so results agree bit for bit: around the
smallest lattice it takes (32^3), odd and even edges and fields that start off an
8-byte boundary (one and two cells a load), one to four planes a march, every step
form, and slabs.
"""

from __future__ import annotations

import numpy as np
import pytest

from lfm_b200 import _lib
from lfm_b200.config import gravity_em, gravity_only

pytestmark = pytest.mark.gpu
REAL, COMPLEX = 0, 1


@pytest.fixture(scope="module")
def be(cuda_device):
    from lfm_b200 import B200Backend
    from lfm_b200.build import build_library

    build_library()
    return B200Backend(cuda_device)


def _direct(run):
    """run() on the direct kernel, then on the kernel the library chooses."""
    _lib.set_step_path(_lib.PATH_DIRECT)
    try:
        a = run()
    finally:
        _lib.set_step_path(_lib.PATH_AUTO)
    return a, run()


def _fields(rng, count, n):
    f = [(0.5 * rng.standard_normal(n)).astype(np.float32) for _ in range(count - 2)]
    return f + [(19.0 + 0.1 * rng.standard_normal(n)).astype(np.float32) for _ in range(2)]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("level", [REAL, COMPLEX])
@pytest.mark.parametrize("N", [2, 3, 5, 31, 32, 33, 34, 35, 46, 62])
def test_protocol_steps(be, level, N, shift):
    import torch

    n, count = N**3, 4 if level == REAL else 6
    rng = np.random.default_rng(N)
    ins = _fields(rng, count, n) + [rng.random(n).astype(np.float32)]

    def dev(a):
        t = torch.zeros(n + shift, dtype=torch.float32, device=be.device)
        t[shift:] = torch.from_numpy(a).to(be.device)
        return t[shift:]

    def run():
        out = [dev(np.zeros(n, np.float32)) for _ in range(count)]
        step = be.step_real if level == REAL else be.step_complex
        extra = () if level == REAL else (0.1,)
        step(*[dev(a) for a in ins], *out, N, 4e-4, 1 / 63, 4 / 31, 19.0, 0.01, *extra)
        return [be.to_numpy(o).view(np.uint32) for o in out]

    for a, b in zip(*_direct(run)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kind", ["plain", "split", "comp"])
@pytest.mark.parametrize("level", [REAL, COMPLEX])
@pytest.mark.parametrize("N", [9, 33, 50, 110])
def test_evolver_steps(be, level, N, kind):
    from lfm_b200 import Evolver, SplitChiEvolver
    from lfm_b200.compensated import CompensatedEvolver

    cls = {"plain": Evolver, "split": SplitChiEvolver, "comp": CompensatedEvolver}[kind]
    rng = np.random.default_rng(N)
    shape = (N, N, N)
    pr, pi = ((0.5 * rng.standard_normal(shape)).astype(np.float32) for _ in range(2))
    chi = (19.0 + 1e-2 * rng.standard_normal(shape)).astype(np.float32)

    def run():
        ev = cls((gravity_em if level else gravity_only)(N), backend=be)
        ev.use_graphs = False
        ev.set_psi_real(pr)
        if level:
            ev.set_psi_imag(pi)
        ev.set_chi(chi)
        ev.evolve(3)  # the first from undamped previous fields
        return [ev.get_psi_real(), ev.get_chi()] + ([ev.get_psi_imag()] if level else [])

    for a, b in zip(*_direct(run)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("level", [REAL, COMPLEX])
@pytest.mark.parametrize("N,ranks", [(33, 2), (34, 5), (50, 3)])
def test_slabs(be, level, N, ranks):
    """Slabs read their ghost planes: every rank's planes equal the whole lattice's."""
    from lfm_b200 import Evolver
    from lfm_b200.slab import SlabEvolver, evolve_local, gather_local

    rng = np.random.default_rng(N)
    cfg = (gravity_em if level else gravity_only)(N)
    pr, pi = ((0.5 * rng.standard_normal((N,) * 3)).astype(np.float32) for _ in range(2))
    chi = (19.0 + 1e-2 * rng.standard_normal((N,) * 3)).astype(np.float32)
    slabs = [SlabEvolver(cfg, backend=be, rank=r, world=ranks) for r in range(ranks)]
    ev = Evolver(cfg, backend=be)
    for e in slabs + [ev]:
        e.set_psi_real(pr)
        if level:
            e.set_psi_imag(pi)
        e.set_chi(chi)
    evolve_local(slabs, 4)
    _lib.set_step_path(_lib.PATH_DIRECT)
    try:
        ev.use_graphs = False
        ev.evolve(4)
    finally:
        _lib.set_step_path(_lib.PATH_AUTO)
    got = np.asarray(gather_local(slabs, "psi_r"))
    assert np.array_equal(got.view(np.uint32), ev.get_psi_real().view(np.uint32))


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("N", [44, 45, 46, 72, 110])
def test_color_steps(be, N, shift):
    """COLOR around its smallest marching lattice, odd and even, one and several planes a
    march, with every coupling (S_a apart, which enters both kernels as the same array)."""
    import torch

    n = N**3
    rng = np.random.default_rng(N)
    psi = [(0.5 * rng.standard_normal(3 * n)).astype(np.float32) for _ in range(4)]
    ins = psi + _fields(rng, 2, n) + [rng.random(n).astype(np.float32)]

    def dev(a):
        t = torch.zeros(a.size + shift, dtype=torch.float32, device=be.device)
        t[shift:] = torch.from_numpy(a).to(be.device)
        return t[shift:]

    def run():
        out = [dev(np.zeros_like(a)) for a in ins[:6]]
        sa = dev(np.zeros(3 * n, np.float32))
        be.step_color(*[dev(a) for a in ins], *out, N, 4e-4, 1 / 63, 4 / 31, 19.0, 0.01, 0.1,
                      1 / 189, 2 / 17, kappa_string=1 / 189, kappa_tube=30 / 63,
                      sa_fields_out=sa)
        return [be.to_numpy(o).view(np.uint32) for o in out + [sa]]

    for a, b in zip(*_direct(run)):
        assert np.array_equal(a, b)


def _three_steps(be, kind, level, N):
    """Fields after three steps of an evolver (the first from undamped previous fields)."""
    from lfm_b200 import Evolver, SplitChiEvolver
    from lfm_b200.compensated import CompensatedEvolver

    make = {"plain": Evolver, "split": SplitChiEvolver, "comp": CompensatedEvolver,
            "ab": lambda cfg, backend: Evolver(cfg, backend=backend, buffers="ab")}[kind]
    rng = np.random.default_rng(N)
    pr, pi, chi = (rng.standard_normal((N, N, N), dtype=np.float32) for _ in range(3))
    ev = make((gravity_em if level else gravity_only)(N), backend=be)
    ev.use_graphs = False
    ev.set_psi_real(0.5 * pr)
    if level:
        ev.set_psi_imag(0.5 * pi)
    ev.set_chi(19.0 + np.float32(1e-2) * chi)
    ev.evolve(3)
    return [ev.get_psi_real(), ev.get_chi()] + ([ev.get_psi_imag()] if level else [])


@pytest.mark.parametrize("kind", ["plain", "split", "comp", "ab"])
@pytest.mark.parametrize("level", [REAL, COMPLEX])
@pytest.mark.parametrize("N", [150, 163])
def test_marches_of_more_planes_than_the_queue_holds(be, level, N, kind):
    """Five planes a march and more (the queue's slots come round again), the last march of
    a column shorter than the others."""
    for a, b in zip(*_direct(lambda: _three_steps(be, kind, level, N))):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("kind", ["plain", "split", "comp", "ab"])
@pytest.mark.parametrize("level", [REAL, COMPLEX])
@pytest.mark.parametrize("N", [24, 48, 160, 240])
def test_run_time_tiles_at_every_size(be, level, N, kind):
    """The fused kernel's run-time tiles, also where another kernel is the faster one and
    they run only when asked for."""
    if (N, level) == (24, REAL) and kind != "split":
        pytest.skip("no tile: rows of six threads")
    _lib.set_step_path(_lib.PATH_FUSED)
    try:
        tile = _three_steps(be, kind, level, N)
    finally:
        _lib.set_step_path(_lib.PATH_AUTO)
    for other in _direct(lambda: _three_steps(be, kind, level, N)):
        for a, b in zip(tile, other):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("N", [112, 150, 192])
def test_color_steps_on_every_kernel(be, N):
    """COLOR with a streamed mask where the chosen kernel is a tile (112, 192) or marches
    (150: four planes a march), against the direct kernel."""
    rng = np.random.default_rng(N)
    n = N**3
    f = lambda k: be.from_numpy(rng.standard_normal(k * n, dtype=np.float32))  # noqa: E731
    ins = [f(3) * 0.5 for _ in range(4)] + [19.0 + 0.1 * f(1) for _ in range(2)]
    mask = be.from_numpy(rng.random(n, dtype=np.float32))

    def run():
        import torch

        out = [torch.empty_like(a) for a in ins]
        be.step_color(*ins, mask, *out, N, 4e-4, 1 / 63, 4 / 31, 19.0, 0.01, 0.1, 1 / 189, 2 / 17)
        return [be.to_numpy(o).view(np.uint32) for o in out]

    for a, b in zip(*_direct(run)):
        assert np.array_equal(a, b)
