"""Tile shapes cached by a build with other kernels (another key version) are not
applied: a file with such an entry for the plan's own key leaves the choice to a
new tuning."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import nfftgb300 as nf  # noqa: E402


def test_entries_of_an_earlier_version_are_not_used(tmp_path, monkeypatch):
    k = (np.random.default_rng(4).random((3, 20000)) - 0.5).astype(np.float32)

    def tuned(path, use_cache):
        monkeypatch.setenv("NFFT_GB300_TUNE_CACHE", str(path))
        p = nf.plan_nfft(k, (40, 36, 32), m=4, sigma=2.0, precompute=nf.TENSOR)
        p.autotune(use_cache=use_cache)
        return tuple(p.params.blockSize)

    tuned(tmp_path / "new.txt", False)
    key = (tmp_path / "new.txt").read_text().split()[0]
    version, rest = key.split("_", 1)
    stale = tmp_path / "stale.txt"
    stale.write_text(f"v{int(version[1:]) - 1}_{rest} 5 6 7 1\nv2_{rest} 5 6 7 1\n")
    assert tuned(stale, True) != (5, 6, 7)
    same = tmp_path / "same.txt"
    same.write_text(f"{key} 5 6 7 1\n")
    assert tuned(same, True) == (5, 6, 7)
