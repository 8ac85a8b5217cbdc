"""Modes that are evanescent in vacuum and propagate in the medium: strong potentials
in thick slices on grids that reach beyond k0.  Their vacuum factor decays to some
1e-28 within a slice and is divided out again.

Bar: rel-L2 <= 1e-5 against the FP64 oracle, as on the other paths.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nx,B,K,power", [(100, 60, 1, 16, 1.0), (256, 256, 1, 16, 2.0), (128, 128, 30, 3, 1.3),
                                             (101, 64, 2, 7, 1.0), (64, 512, 1, 33, 2.0)])
@pytest.mark.parametrize("energy", [300e3, 80e3])
def test_modes_across_the_edge(ny, nx, B, K, power, energy):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import wideanglepropagation_b200 as wap
    from oracle import propagation_oracle as O
    rng = np.random.default_rng(ny + nx)
    V = (600.0 * rng.uniform(0, 1, (2, ny, nx)) ** 3).astype(np.float32)
    psi = (rng.normal(size=(ny, nx)) + 1j * rng.normal(size=(ny, nx))).astype(np.complex64)
    pos = np.stack([rng.integers(0, ny, B), rng.integers(0, nx, B)], 1).astype(np.int32)
    got = wap.simulate_wpm(V, psi, 4.0, energy, (0.01, 0.01), K, power, positions=pos)
    for b in {0, B - 1}:
        ref = O.simulate_wpm(V, O.move_probe(psi, tuple(pos[b])), 4.0, energy, (0.01, 0.01), K, power)
        for g, r in zip(got, ref):
            assert O.rel_l2(g[b].cpu().numpy(), r) < 1e-5
