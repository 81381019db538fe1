"""The library's scratch pool is given back (B200).

Host drivers take their scratch from a pool that keeps up to 1 GiB between
calls; the end of the last operator of any kind and the clearing of the
operator cache return it to the driver.  Each case is a process of its own: an
operator elsewhere would keep the pool.
"""

import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import numpy as np, torch
import aspher_b200 as asb
from aspher_b200 import _lib as L
def held(call, after=lambda: None):
    # device memory that stays after a call, once its code is loaded
    call(); after(); torch.cuda.synchronize(); torch.cuda.empty_cache()
    a = torch.cuda.mem_get_info()[0]
    return a
x = torch.zeros(1, device="cuda")
"""

TANGENTIAL = HEAD + """
def run(n):
    op = asb.TangentialOperator(n)
    op.solve(0.01 + 0.02 * np.random.default_rng(1).random(n * n), target=(0.01, 0.0), tol=1e-2,
             max_iter=3)
    del op
small = held(lambda: run(700))
big = held(lambda: run(1500))
print("held", (small - big) / 2**20)
"""

CACHE = HEAD + """
own = asb.Operator("periodic", 64)   # a live operator of the program's own
def run(n, coarsest):
    g = torch.from_numpy(asb.self_affine_gap(n, hurst=0.8, rms=0.002, seed=3)).cuda()
    asb.solve_nested(n, g, 0.01, tol=1e-3, coarsest=coarsest, backend="fft", light_result=True)
clear = lambda: L.check(L.lib().aspher_operator_cache_clear())
small = held(lambda: run(256, 64), clear)
big = held(lambda: run(2048, 512), clear)
print("held", (small - big) / 2**20)
"""


@pytest.mark.parametrize("program", [TANGENTIAL, CACHE], ids=["tangential", "cache"])
def test_scratch_goes_back(program):
    """After a large call no more memory stays than after a small one, but for
    modules loaded late (less than 24 MiB; the kept scratch was 32 and 64)."""
    p = subprocess.run([sys.executable, "-c", program], cwd=ROOT, capture_output=True, text=True,
                       env=dict(os.environ, PYTHONPATH=ROOT), timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    held = float(p.stdout.split("held")[1])
    assert held < 24.0, held
