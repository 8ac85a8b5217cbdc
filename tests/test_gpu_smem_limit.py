"""Launches whose dynamic shared memory is just under 48 KB: with the kernel's static
part they are over, and the launch has to ask for more.  Each in a fresh process, as a
larger launch before it would have asked already; and a call after a refused one is
not refused for it."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CALL = """
import numpy as np, sys
sys.path.insert(0, {root!r})
import wideanglepropagation_b200 as wap
from oracle import propagation_oracle as O
ny, nx, B, K = {shape}
rng = np.random.default_rng(1)
V = (40.0 * rng.uniform(0, 1, (2, ny, nx)) ** 3).astype(np.float32)
psi = (rng.normal(size=(ny, nx)) + 1j * rng.normal(size=(ny, nx))).astype(np.complex64)
pos = np.stack([rng.integers(0, ny, B), rng.integers(0, nx, B)], 1).astype(np.int32)
got = wap.simulate_wpm(V, psi, 1.0, 300e3, (0.05, 0.05), n_bins=K, power_spacing=1.5, positions=pos)
ref = O.simulate_wpm(V, O.move_probe(psi, tuple(pos[-1])), 1.0, 300e3, (0.05, 0.05), n_bins=K, power_spacing=1.5)
assert all(O.rel_l2(g[-1].cpu().numpy(), r) < 1e-5 for g, r in zip(got, ref))
"""


@pytest.mark.parametrize("shape", [(240, 300, 1, 16), (240, 45, 16, 32), (100, 72, 16, 16)])
def test_just_under_the_default_limit(shape):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, "-c", CALL.format(root=ROOT, shape=shape)], capture_output=True, text=True,
                       timeout=240)
    assert r.returncode == 0, r.stderr[-1500:]
