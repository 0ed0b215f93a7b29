"""What the step calls refuse, without a GPU: the checks of their arrays."""

from __future__ import annotations

import pytest
import torch

from lfm_b200 import _lib, backend

N = 4


class OnCpu(backend.B200Backend):
    def __init__(self):
        self.device = torch.device("cpu")


@pytest.fixture
def calls(monkeypatch):
    seen = []
    monkeypatch.setattr(_lib, "call", lambda name, *a: seen.append((name, a)))
    monkeypatch.setattr(backend, "_stream_handle", lambda device: 0)
    return seen


def arrays(level, wrap):
    n = N**3
    sizes = {0: [n] * 9, 1: [n] * 13,
             2: [3 * n] * 4 + [n] * 3 + [3 * n] * 4 + [n] * 2}[level]
    return [wrap(torch.zeros(s)) for s in sizes]


def step(level, arrs, **kw):
    be = OnCpu()
    f = (be.step_real, be.step_complex, be.step_color)[level]
    f(*arrs, N, 4e-4, 1 / 63, 0.0, 19.0, 0.0, *(() if level == 0 else (0.1,)), **kw)


@pytest.mark.parametrize("wrap", [lambda t: t, backend.device_array])
@pytest.mark.parametrize("level", [0, 1, 2])
def test_step_calls_check_every_array(calls, level, wrap):
    good = arrays(level, wrap)
    step(level, good)
    name, args = calls.pop()
    at = 0 if level < 2 else 1  # the COLOR call starts with the context
    assert list(args[at:at + len(good)]) == [t.data_ptr() for t in good]
    names = (backend._REAL_ARGS, backend._COMPLEX_ARGS,
             backend._COLOR_IN + backend._COLOR_CHI_IN + backend._COLOR_OUT
             + backend._COLOR_CHI_OUT)[level]
    assert len(names) == len(good)
    for i, t in enumerate(good):
        n = t.numel()
        bad = [(None, TypeError, "expected a torch"), (t.double(), TypeError, "expected float32"),
               (wrap(torch.zeros(n + 1)), ValueError, "elements, expected"),
               (wrap(torch.zeros(2 * n)[::2]), ValueError, "must be contiguous"),
               (torch.empty(n, device="meta"), ValueError, "tensor on meta")]
        for b, error, text in bad:
            with pytest.raises(error, match=f"{names[i]}: .*{text}|{names[i]}: {text}"):
                step(level, good[:i] + [b] + good[i + 1:])
    assert not calls


def test_the_optional_s_a_fields_are_checked_too(calls):
    good, sa = arrays(2, lambda t: t), torch.zeros(3 * N**3)
    step(2, good, sa_fields_in=sa, sa_fields_out=sa)
    assert sa.data_ptr() in calls.pop()[1]
    for name in ("sa_fields_in", "sa_fields_out"):
        with pytest.raises(ValueError, match=f"{name}: "):
            step(2, good, **{name: sa[1:]})
