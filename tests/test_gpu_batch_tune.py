"""The batched form's autotuner: what it stores holds for every axis of that
length."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(code, cache):
    """In a process of its own (widths are read once a process)."""
    env = dict(os.environ, SHAFFT_SM100_TUNE_CACHE=str(cache))
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout


def _widths(cache):
    return dict(line.split() for line in cache.read_text().splitlines())


def test_width_does_not_depend_on_the_batch_dimension_it_was_met_with(tmp_path):
    """16 points met first with two columns: the stored width is one a batch of
    many columns would choose from (tiles of at least 1024 points)."""
    cache = tmp_path / "tune.txt"
    _run("from shafft_b200 import _sm100; _sm100.Batch([(16, 2)], 0, autotune=True)", cache)
    w = {k: int(v) for k, v in _widths(cache).items() if k.startswith("c64:L=16:col")}
    assert len(w) == 1 and min(w.values()) >= 64, w
