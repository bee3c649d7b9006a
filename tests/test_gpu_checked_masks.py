"""The suites that store through the sorted ranges (hit masks of differentiable frames, batches that share a launch,
the emit's partitions) under the checked build, and on the CPU that the hit masks' words of a frame's tiles fit
their plane and do not meet."""
import subprocess
import sys

import numpy as np
import pytest

from test_gpu_checked import ROOT, _env

SUITES = ["test_gpu_backward_reduction.py", "test_gpu_backward_views.py", "test_gpu_batch_runs.py",
          "test_gpu_raster_lists.py", "test_gpu_emit_partitions.py", "test_gpu_differentiable_memory.py"]


@pytest.mark.gpu
def test_suites_pass_under_the_checked_build():
    cmd = [sys.executable, "-m", "pytest", "-m", "gpu", "-x", "-q", "-p", "no:cacheprovider", "-k",
           "not needs_no_more_memory", *[str(ROOT / "tests" / f) for f in SUITES]]
    proc = subprocess.run(cmd, cwd=ROOT, env=_env(), capture_output=True, text=True, timeout=1800)
    assert proc.returncode == 0, proc.stdout[-4000:] + proc.stderr[-2000:]
    assert " passed" in proc.stdout


@pytest.mark.parametrize("seed", range(20))
def test_mask_words_of_the_tiles_fit_and_do_not_meet(seed):
    """gs_kernels.h: a tile's first word is start / 32 + tile, one word per 32 positions; a plane holds
    max_instance / 32 + tiles + 1 words."""
    rng = np.random.default_rng(seed)
    tiles = int(rng.integers(1, 400))
    lengths = rng.integers(0, rng.choice([1, 2, 40, 200]) + 1, tiles) * (rng.random(tiles) < rng.choice([0.1, 0.6, 1.0]))
    ends = np.cumsum(lengths)
    max_instance = int(ends[-1]) + int(rng.integers(0, 2)) * int(rng.integers(0, 100))
    used = np.zeros(max_instance // 32 + tiles + 1, int)
    for tile, (end, length) in enumerate(zip(ends, lengths)):
        base = (int(end - length) >> 5) + tile
        words = used[base:base + (int(length) + 31) // 32]
        assert len(words) == (length + 31) // 32
        words += 1
    assert used.max(initial=0) <= 1
