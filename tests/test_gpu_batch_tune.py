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


def test_widths_of_another_kernel_revision_are_not_used(tmp_path):
    """Entries without the revision (those of the kernel before) and of another
    one leave the default widths in place; an entry of this one is used."""
    code = "from shafft_b200 import _sm100; print(_sm100.Batch([(64, 96)], 0).describe()['tiles'])"
    none = int(_run(code, tmp_path / "none.txt"))
    old = tmp_path / "old.txt"
    old.write_text("c64:L=96:row 2\nc64:L=64:col 2\nc64:L=96:row:r1:t128 2\nc64:L=64:col:r1:t128 2\n")
    assert int(_run(code, old)) == none
    tuned = tmp_path / "tuned.txt"
    _run("from shafft_b200 import _sm100; _sm100.Batch([(64, 96)], 0, autotune=True)", tuned)
    keys = [k for k in _widths(tuned) if k.startswith("c64:L=96:row")]
    assert len(keys) == 1
    tuned.write_text(f"{keys[0]} 2\n")
    assert int(_run(code, tuned)) > none
