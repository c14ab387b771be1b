"""Facet staging for a device that is not the current one: the library's kernel
is launched with the facets' device current and on that device's stream. The
CUDA runtime is replaced by a record of what was current at the launch."""

import contextlib
from types import SimpleNamespace

import numpy as np
import torch

from radar_sounder_simulator_gb300 import _lib, coherent


def test_staging_makes_the_facets_device_current(monkeypatch):
    now, seen = [torch.device("cuda", 0)], []

    @contextlib.contextmanager
    def device(d):
        now.append(torch.device(d))
        yield
        now.pop()

    def stream(d=None):
        return SimpleNamespace(cuda_stream=100 + (
            now[-1] if d is None else torch.device(d)).index)

    def stage(*args):
        seen.append((now[-1].index, args[-1]))
        return 0

    def empty(shape, dtype=None, device=None):
        return SimpleNamespace(device=torch.device(device), shape=shape,
                               data_ptr=lambda: 64)
    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(torch.cuda, "current_stream", stream)
    monkeypatch.setattr(torch, "empty", empty)
    monkeypatch.setattr(_lib, "lib",
                        lambda: SimpleNamespace(ss_stage_facets=stage))
    n = 5
    cols = [torch.from_numpy(np.zeros(3 * n))] * 4 + [
        torch.from_numpy(np.zeros(n))]
    for index in (1, 0):
        fac = coherent.stage_facets(None, None, None, None, None,
                                    torch.arange(n), f"cuda:{index}",
                                    uploaded=cols)
        assert fac.n == n and fac.soa.shape == (13, n)
    assert seen == [(1, 101), (0, 100)]
    assert now == [torch.device("cuda", 0)]
