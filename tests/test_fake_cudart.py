"""The library's launch code on a CUDA runtime without a GPU (fake_cudart.cpp): two devices
in one process, and cooperative launches that are refused.  The library's own objects are
linked against it; a launch is checked and counted, and runs nothing."""

from __future__ import annotations

import ctypes
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from lfm_b200 import _lib
from lfm_b200.build import LIB_DIR, build_library, sources
from lfm_b200.mask import MaskTable

REAL, COMPLEX, COLOR = 0, 1, 2
STEP = (4e-4, 1 / 63, 0.0, 19.0, 0.0)  # dt2, kappa, lambda_self, chi0, e0_sq


@pytest.fixture(scope="module")
def fake_path(tmp_path_factory):
    build_library()
    objs = [LIB_DIR / "obj" / f"{s.stem}.o" for s in sources()]
    if not all(o.exists() for o in objs):
        build_library(force=True)
    out = tmp_path_factory.mktemp("fake") / "liblfm_fake.so"
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic",
                           "-I/usr/local/cuda/include", "-o", str(out),
                           str(ROOT / "tests" / "fake_cudart.cpp"), *map(str, objs)])
    return out


@pytest.fixture
def fake(fake_path, monkeypatch):
    """The linked library, in the package's place, as a process finds it at its start."""
    lib = ctypes.CDLL(str(fake_path))
    for name, args in _lib._SIGNATURES.items():
        getattr(lib, name).argtypes = args
    lib.fake_last_kernel.restype = ctypes.c_char_p
    lib.lfm_strerror.restype = lib.lfm_last_error_detail.restype = ctypes.c_char_p
    monkeypatch.setattr(_lib, "_lib", lib)
    lib.fake_reset()
    return lib


class Lattice:
    """Host buffers in the place of a lattice's device memory."""

    def __init__(self, level, N):
        self.level, self.N = level, N
        per = 3 if level == COLOR else 1
        self.bufs = [np.zeros(per * N**3 + 4, np.float32) for _ in range(6)]
        self.p = [(b.ctypes.data + 15) & ~15 for b in self.bufs]
        self.pr, self.pi, self.chi = self.p[:2], self.p[2:4] if level else (None, None), self.p[4:]
        self.table = MaskTable.for_lattice(N, 0.3)
        self.t = np.ascontiguousarray(self.table.table, np.float32)
        self.mask = (self.t.ctypes.data, ctypes.byref(self.table.desc))
        words = ctypes.c_longlong()
        _lib.call("lfm_leapfrog_run_words", min(level, 1), N, ctypes.byref(words))
        self.sync = np.zeros(words.value + 4, np.int32)

    def run(self, steps=4):
        return _lib.run_steps("lfm_leapfrog_run_f32", self.level, steps, *self.pr, *self.pi,
                              *self.chi, *self.mask, 0, self.N, *STEP, 0.1, None,
                              (self.sync.ctypes.data + 15) & ~15, None)

    def step(self):
        if self.level == REAL:
            _lib.call("lfm_leapfrog_real_f32", *self.pr, *self.chi, *self.mask, 0, self.N, *STEP,
                      None)
        elif self.level == COMPLEX:
            _lib.call("lfm_leapfrog_complex_f32", *self.pr, *self.pi, *self.chi, *self.mask, 0,
                      self.N, *STEP, 0.1, None)
        else:
            _lib.call("lfm_leapfrog_color_f32", *self.pr, *self.pi, *self.chi, *self.mask, 0,
                      self.N, *STEP, *([0.1] * 5), None, None)

    def masked_step(self):
        """The protocol's step: a mask beside the fields, every output apart."""
        n = self.N**3
        f = [np.zeros(n + 4, np.float32) for _ in range(13)]
        p = [(b.ctypes.data + 15) & ~15 for b in f]
        if self.level == REAL:
            _lib.call("lfm_step_real_f32", *p[:9], self.N, *STEP, None)
        else:
            _lib.call("lfm_step_complex_f32", *p, self.N, *STEP, 0.1, None)

    def comp_step(self):
        f = [np.zeros(self.N**3 + 4, np.float32) for _ in range(9)]
        p = [(b.ctypes.data + 15) & ~15 for b in f]
        if self.level == REAL:
            _lib.call("lfm_leapfrog_real_comp_f32", *p[:6], *self.mask, self.N, *STEP, None)
        else:
            _lib.call("lfm_leapfrog_complex_comp_f32", *p, *self.mask, self.N, *STEP, 0.1, None)

    def split_step(self):
        f = [np.zeros(self.N**3 + 4, np.float32) for _ in range(8)]
        p = [(b.ctypes.data + 15) & ~15 for b in f]
        name, n = (("lfm_leapfrog_real_split_f32", 6) if self.level == REAL
                   else ("lfm_leapfrog_complex_split_f32", 8))
        _lib.call(name, *p[:n], *self.mask, 0, self.N, *STEP,
                  *(() if self.level == REAL else (0.1,)), None)

    def desc(self):
        d = _lib.LatticeDesc()
        d.N, d.level = self.N, self.level
        for s in range(2):
            d.psi_r[s], d.psi_i[s], d.chi[s] = self.pr[s], self.pi[s], self.chi[s]
        d.mask_table, d.lut = self.t.ctypes.data, self.table.desc
        d.dt2, d.kappa, d.lambda_self, d.chi0, d.e0_sq = STEP
        return d


def batch(lattices, **tuning):
    descs = (_lib.LatticeDesc * len(lattices))(*[x.desc() for x in lattices])
    h, t = ctypes.c_void_p(), _lib.BatchTuning(**tuning)
    _lib.call("lfm_batch_create", descs, len(lattices), ctypes.byref(t), ctypes.byref(h))
    return h


def solve_sa(N):
    ctx = ctypes.c_void_p()
    _lib.call("lfm_context_create", ctypes.byref(ctx))
    e, s = (np.zeros(3 * N**3, np.float32) for _ in range(2))
    _lib.call("lfm_helmholtz_sa_from_energy_f32", ctx, e.ctypes.data, s.ctypes.data, N, 0.1, 4.9,
              None)


@pytest.mark.parametrize("what", ["run", "color", "fused", "batch", "s_a"])
def test_shared_memory_limits_are_raised_on_every_device(fake, what):
    """The limit of a kernel's dynamic shared memory belongs to the device: what a process
    launches on its first GPU it can launch on its second."""
    call = {"run": lambda: Lattice(REAL, 32).run(), "color": Lattice(COLOR, 128).step,
            "fused": Lattice(REAL, 128).step,
            "batch": lambda: _lib.call("lfm_batch_step", batch([Lattice(REAL, 96)]), 0, 0, None),
            "s_a": lambda: solve_sa(512)}[what]
    for device in (0, 1, 0):
        fake.cudaSetDevice(device)
        before = fake.fake_launches()
        call()
        assert fake.fake_launches() > before and fake.fake_refusals() == 0


def test_a_refused_run_leaves_the_lattice_to_single_steps(fake):
    """Blocks that cannot all be resident at once (a context with a part of the SMs): the
    run answers that it is not supported, and has launched nothing."""
    lat = Lattice(REAL, 32)
    fake.fake_free_sms(60)
    assert lat.run() is False
    assert fake.fake_launches() == 0 and fake.fake_refusals() == 1 and fake.fake_last_error() == 0
    lat.step()
    fake.fake_free_sms(148)
    assert lat.run() is True


@pytest.mark.parametrize("sizes", [[(8, REAL), (96, COMPLEX)], [(96, REAL), (8, COMPLEX)]])
def test_a_refused_wave_leaves_the_batch_to_single_steps(fake, sizes):
    """A batch's largest wave is refused before any other has run."""
    lats = [Lattice(level, n) for n, level in sizes]
    h = batch(lats)
    before = fake.fake_launches()
    fake.fake_free_sms(100)
    assert _lib.run_steps("lfm_batch_run", h, 4, 0, 0, None) is False
    assert fake.fake_launches() == before and fake.fake_last_error() == 0
    _lib.call("lfm_batch_step", h, 0, 0, None)
    fake.fake_free_sms(148)
    assert _lib.run_steps("lfm_batch_run", h, 4, 0, 0, None) is True


@pytest.mark.parametrize("level,form,tiles,marches", [
    (REAL, "step", (128, 192, 240, 256), (96, 176, 288, 352)),
    (COMPLEX, "step", (128, 256), (96, 160, 240, 288)),
    (COLOR, "step", (112, 128, 192, 224, 256), (72, 96, 144, 160, 288)),
    (REAL, "masked_step", (160, 192, 256, 352), (128, 144, 288)),
    (COMPLEX, "masked_step", (128, 240, 256), (96, 192, 224, 288)),
    (REAL, "comp_step", (240, 256), (128, 224, 288)),
    (COMPLEX, "comp_step", (256,), (128, 192, 240, 288))])
def test_a_lattice_takes_the_kernel_that_measured_faster(fake, level, form, tiles, marches):
    """The fused kernel (its tile lies in shared memory) against the marching one."""
    for n in tiles + marches:
        getattr(Lattice(level, n), form)()
        assert (fake.fake_dynamic_smem() > 0) == (n in tiles), n


def test_a_tuned_batch_plans_its_waves_when_a_run_comes(fake):
    """retune() and a tuning search make batches that step with the tile kernel."""
    lats = [Lattice(REAL, 32), Lattice(COMPLEX, 16)]
    start = fake.fake_allocations()
    plain = batch(lats)
    with_waves = fake.fake_allocations() - start
    tuned = batch(lats, threads=128)
    assert fake.fake_allocations() - start == 2 * with_waves - 1
    _lib.call("lfm_batch_step", tuned, 0, 0, None)
    fake.fake_capture(1)
    assert _lib.run_steps("lfm_batch_run", plain, 4, 0, 0, None) is True
    assert _lib.run_steps("lfm_batch_run", tuned, 4, 0, 0, None) is False
    fake.fake_capture(0)
    assert _lib.run_steps("lfm_batch_run", tuned, 4, 0, 0, None) is True
    assert fake.fake_allocations() - start == 2 * with_waves


@pytest.mark.parametrize("level,form,direct,marches", [
    (REAL, "step", (31,), (32, 33, 41, 48)),
    (REAL, "comp_step", (31, 33, 41), (32, 34, 43)),
    (REAL, "split_step", (31, 33, 41), (32, 34, 43)),
    (COMPLEX, "step", (31, 33, 41), (32, 34, 43)),
    (COMPLEX, "masked_step", (31, 33, 41), (32, 34, 43)),
    (COMPLEX, "comp_step", (31,), (32, 33, 41)),
    (COMPLEX, "split_step", (31, 33, 41), (32, 34, 43)),
    (COLOR, "step", (33, 44, 51, 52, 53, 55, 57), (45, 48, 50, 54, 56, 59, 61))])
def test_the_smallest_lattices_take_the_direct_kernel(fake, level, form, direct, marches):
    for n in direct + marches:
        getattr(Lattice(level, n), form)()
        want = b"direct_step_kernel" if n in direct else (
            b"march_color_kernel" if level == COLOR else b"march_step_kernel")
        assert want in fake.fake_last_kernel(), (n, fake.fake_last_kernel())
