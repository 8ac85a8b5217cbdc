"""Wide-angle steps on grids that are not powers of two, by line kind: Bluestein
lines of every transform length (64 .. 2048), both element counts per thread, one
and several thread groups per row, beside mixed-radix and power-of-two sides; the
fields of interpolation nodes and, on grids that reach the evanescent edge or
with strong slices close to it, of the K reference indices.

Bar: rel-L2 <= 1e-5 of exit wave, pattern and wavefronts against the FP64 oracle,
as on the other paths.
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


def _check(wap, ny, nx, B, K, ps, amp=40.0, N=2, power=1.5, wave="random"):
    from oracle import propagation_oracle as O
    rng = np.random.default_rng(ny * 31 + nx + B)
    dz, E = 1.0, 300e3
    V = (amp * rng.uniform(0, 1, (N, ny, nx)) ** 3).astype(np.float32)
    psi = np.ones((ny, nx), np.complex64)
    if wave == "random":
        psi = (rng.normal(size=(ny, nx)) + 1j * rng.normal(size=(ny, nx))).astype(np.complex64)
    pos = np.stack([rng.integers(0, ny, B), rng.integers(0, nx, B)], 1).astype(np.int32)
    got = wap.simulate_wpm(V, psi, dz, E, (ps, ps), n_bins=K, power_spacing=power, positions=pos)
    for b in {0, B - 1}:
        ref = O.simulate_wpm(V, O.move_probe(psi, tuple(pos[b])), dz, E, (ps, ps), n_bins=K, power_spacing=power)
        for g, r in zip(got, ref):
            assert O.rel_l2(g[b].cpu().numpy(), r) < TOL


SHAPES = [(31, 19, 1), (33, 37, 3), (64, 67, 2), (67, 100, 1), (97, 41, 5), (129, 22, 2), (257, 38, 1), (23, 517, 1),
          (1021, 19, 1), (19, 1021, 2), (37, 37, 520), (101, 101, 48), (202, 26, 200), (509, 33, 80), (1021, 1021, 1)]


@pytest.mark.parametrize("ny,nx,B", SHAPES)
def test_nodes(wap, ny, nx, B):
    _check(wap, ny, nx, B, 6, 0.05)


@pytest.mark.parametrize("ny,nx,B", SHAPES[:-1] + [(100, 60, 1), (45, 70, 3), (128, 100, 2), (30, 30, 40)])
@pytest.mark.parametrize("ps,amp", [(0.01, 40.0), (0.01397, 600.0)])   # beyond the edge; short of it, strong slices
def test_reference_fields(wap, ny, nx, B, ps, amp):
    _check(wap, ny, nx, B, 3 if B > 100 else 7, ps, amp)
