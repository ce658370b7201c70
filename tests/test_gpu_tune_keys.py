"""The autotuner's keys name what was timed: choices for the transforms' Y pass, from
a cache file that knows no direct solve, are not taken for it, and fields of another
width are timed for themselves."""
import importlib

import pytest

pytestmark = pytest.mark.gpu


def _tuned(ib, monkeypatch, tmp_path, cache_lines, nx):
    abi = importlib.import_module(ib.__name__ + "._abi")
    cache = tmp_path / f"tune_{nx}.txt"
    cache.write_text(cache_lines)
    monkeypatch.delenv("IBPM_TUNE_FORCE_NG", raising=False)
    monkeypatch.setenv("IBPM_TUNE_CACHE", str(cache))
    monkeypatch.setenv("IBPM_TUNE", "1")
    h = 4.0 / 72
    prob = ib.configs.cylinder(h, (-1.0, -1.0 + nx * h), (-2.0, 2.0), 2, 40, 100.0, 0.2 * h)
    ib.create_solver(ib.State(prob))
    added = [line.rsplit(" ", 1) for line in cache.read_text()[len(cache_lines):].splitlines()]
    assert all(abi.tune_table()[k] == int(v) for k, v in added)
    return added


def test_direct_solves_are_timed_for_themselves(ib, monkeypatch, tmp_path):
    import torch

    name = torch.cuda.get_device_name(0)
    old = "".join(f"{name} ypass M=72 fp64 batch={b} 8\n" for b in range(5))
    first = _tuned(ib, monkeypatch, tmp_path, old, 120)
    second = _tuned(ib, monkeypatch, tmp_path, old, 200)
    assert first and second and not {k for k, _ in first} & {k for k, _ in second}
    assert all(int(v) in (1, 2, 4) for _, v in first + second)
    assert all("ypass M=72 fp64" in k for k, _ in first + second)
