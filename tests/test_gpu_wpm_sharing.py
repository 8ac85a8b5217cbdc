"""Wide-angle slices without interpolation nodes, on power-of-two grids just short of
the evanescent edge: their reference fields are shared out to more blocks where the
pass alone leaves the chip idle, and the last block of a row tile finishes it.
Slices with and without nodes in one call, several draws and probes, one and several
thread groups, shares of unequal size, bins that no pixel wants.

Bar: rel-L2 <= 1e-5 of exit wave, pattern and wavefronts against the FP64 oracle,
as on the other paths; repeated calls agree bit for bit (every pixel has one owner).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.fixture(scope="module")
def wap():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import wideanglepropagation_b200 as w
    return w


@pytest.mark.parametrize("ny,nx,B,K,power", [
    (32, 32, 1, 128, 2.0), (64, 64, 1, 16, 1.0), (64, 64, 40, 33, 2.0), (128, 128, 2, 64, 1.5), (256, 256, 1, 40, 2.0),
    (32, 512, 1, 17, 1.0), (1024, 64, 1, 24, 2.0), (64, 1024, 1, 24, 1.0), (2048, 32, 1, 16, 2.0), (32, 2048, 2, 31, 2.0),
    (64, 64, 600, 16, 1.0)])   # the last fills the chip: no shares
def test_slices_without_nodes(wap, ny, nx, B, K, power):
    from oracle import propagation_oracle as O
    rng = np.random.default_rng(ny + 3 * nx + K)
    ps, dz, E, N = 0.01397, 1.0, 300e3, 4
    V = rng.uniform(0, 1, (2, N, ny, nx)) ** 3 * np.array([600.0, 5.0, 0.0, 400.0])[None, :, None, None]
    V[1] = 0.5 * V[1, ::-1]
    V = V.astype(np.float32)
    psi = (rng.normal(size=(ny, nx)) + 1j * rng.normal(size=(ny, nx))).astype(np.complex64)
    pos = np.stack([rng.integers(0, ny, B), rng.integers(0, nx, B)], 1).astype(np.int32)
    draw = (np.arange(B) % 2).astype(np.int32)
    stack = B < 100

    def call():
        return wap.simulate_wpm(V, psi, dz, E, (ps, ps), n_bins=K, power_spacing=power, positions=pos, draw=draw,
                                return_wavefronts=stack)

    got, again = call(), call()
    for g, a in zip(got, again):
        assert (g is None and a is None) or torch.equal(g, a)
    for b in {0, B - 1}:
        ref = O.simulate_wpm(V[draw[b]], O.move_probe(psi, tuple(pos[b])), dz, E, (ps, ps), n_bins=K,
                             power_spacing=power, return_wavefronts=stack)
        for g, r in zip(got, ref):
            if g is not None:
                assert O.rel_l2(g[b].cpu().numpy(), r) < TOL
