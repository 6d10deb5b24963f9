"""Shapes tuned for other kernels: entries of a cache file whose keys do not name the
present kernels are not taken for the workload's own, so that the sampler tunes it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import math
import numpy as np
from theboss_gb300 import _native
from theboss_gb300.utilities import haar_unitary
n, m = 16, 32
S = np.array([1] * n + [0] * (m - n), dtype=np.int32)
np.random.seed(1)
_native.gccb_sample(haar_unitary(m, 1), S, [math.comb(n, l) / 2 ** n for l in range(n + 1)], 200)
"""


def test_entries_of_other_kernels_are_not_used(tmp_path):
    import torch

    cache, name = tmp_path / "tune.txt", torch.cuda.get_device_name()
    # every level and sample count, keyed by arithmetic, level and sample count alone
    old = [f"{name}|{(1 << 32) | (k << 16) | b}|3|0\n" for k in range(2, 33) for b in range(20)]
    cache.write_text("".join(old))
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, BOSS_TUNE_CACHE=str(cache), BOSS_AUTOTUNE="1", PYTHONPATH=root)
    subprocess.run([sys.executable, "-c", CHILD], check=True, env=env, cwd=root)
    lines = cache.read_text().splitlines(keepends=True)
    assert not set(lines) & set(old)
    tuned = {int(l.split("|")[1]) >> 16 & 0xFFFF for l in lines if "pipeline" not in l}
    assert tuned and tuned <= set(range(2, 17))
