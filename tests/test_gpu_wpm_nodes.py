"""WPM by interpolation nodes (csrc/wap_wpm_nodes.cuh) against the FP64 oracle:
light to heavy atoms (few to many nodes), ranges of the index that need none,
negative potentials, slices of different ranges in one call, several draws and
probes, and the smallest and largest tiles.

Bar: rel-L2 <= 1e-5 of exit wave, pattern and wavefronts, the bar of the other
paths (float32 rounding of the chain is ~1e-6 here; the interpolation adds at
most 1e-9 per slice).
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


def _atoms(ny, nx, N, seed, amp, ps, dz, sigma=0.25):
    import wideanglepropagation_b200.synthetic as S
    rng = np.random.default_rng(seed)
    return np.stack([S.gaussian_slice(ny, nx, ps, rng.uniform(0, 1, (12, 2)) * [ny * ps, nx * ps], amp, sigma)
                     for _ in range(N)]) / dz


def _check(wap, V, probe, dz, E, ps, K, p, **kw):
    from oracle import propagation_oracle as O
    V = V.astype(np.float32)
    got = wap.simulate_wpm(V, probe, dz, E, (ps, ps), n_bins=K, power_spacing=p, **kw)
    ref = O.simulate_wpm(V, probe, dz, E, (ps, ps), n_bins=K, power_spacing=p)
    for g, r in zip(got, ref):
        assert O.rel_l2(g.cpu().numpy(), r) < TOL


@pytest.mark.parametrize("ny,nx,K,p,amp,E,ps,dz", [
    (32, 64, 5, 1.0, 25.0, 300e3, 0.05, 2.0),
    (64, 32, 128, 2.0, 400.0, 200e3, 0.05, 3.0),
    (128, 128, 16, 1.0, 4000.0, 300e3, 0.05, 2.0),     # radians per slice: many nodes
    (256, 128, 6, 2.0, 3000.0, 80e3, 0.05, 1.5),       # as many nodes as bins: the reference fields
    (256, 256, 64, 2.0, 60.0, 80e3, 0.04, 2.0),        # wide spread of 1 / kz over the grid
    (32, 1024, 8, 1.0, 50.0, 300e3, 0.1, 1.0),
    (2048, 32, 7, 1.0, 50.0, 300e3, 0.1, 1.0),
    (100, 64, 16, 1.0, 80.0, 300e3, 0.05, 2.0),        # a side that is not a power of two
])
def test_nodes_match_oracle(wap, ny, nx, K, p, amp, E, ps, dz):
    import wideanglepropagation_b200.synthetic as S
    V = _atoms(ny, nx, 4, ny + 3 * nx + K, amp, ps, dz)
    probe = S.aperture_probe(ny, nx, ps, E, 25.0, -30.0, dtype=np.complex64)
    _check(wap, V, probe, dz, E, ps, K, p)


@pytest.mark.parametrize("n", [64, 90])
def test_ranges_of_a_slice(wap, n):
    """One call with slices of a single value (zero and not), of a large offset
    with little contrast, negative, and of atoms."""
    import wideanglepropagation_b200.synthetic as S
    ps, dz, E = 0.05, 2.0, 300e3
    atoms = _atoms(n, n, 2, 5, 300.0, ps, dz)
    flat = np.zeros((n, n))
    V = np.stack([flat, atoms[0], flat + 150.0, flat + 1000.0 + 1e-3 * atoms[1], -0.5 * atoms[1], atoms[1]])
    probe = S.aperture_probe(n, n, ps, E, 25.0, -30.0, dtype=np.complex64)
    _check(wap, V, probe, dz, E, ps, 16, 2.0)


def test_draws_and_probes(wap):
    """Draws of different ranges in one launch, probes of each, against one-probe calls."""
    import wideanglepropagation_b200.synthetic as S
    from oracle import propagation_oracle as O
    n, ps, dz, E, N = 128, 0.05, 2.0, 300e3, 3
    V = np.stack([_atoms(n, n, N, 1, 25.0, ps, dz), _atoms(n, n, N, 2, 2000.0, ps, dz)]).astype(np.float32)
    probe = S.aperture_probe(n, n, ps, E, 25.0, -30.0, dtype=np.complex64)
    pos = np.array([[64, 64], [3, 120], [77, 20]], np.int32)
    draw = np.array([1, 0, 1], np.int32)
    ex, dp, _ = wap.simulate_wpm(V, probe, dz, E, (ps, ps), n_bins=32, positions=pos, draw=draw,
                                 return_wavefronts=False)
    for b in range(3):
        rex, rdp, _ = O.simulate_wpm(V[draw[b]], O.move_probe(probe, tuple(pos[b])), dz, E, (ps, ps), n_bins=32,
                                     return_wavefronts=False)
        assert O.rel_l2(ex[b].cpu().numpy(), rex) < TOL
        assert O.rel_l2(dp[b].cpu().numpy(), rdp) < TOL


def test_values_without_an_index_are_left_out(wap):
    """Pixels whose potential has no real index do not enter the slice's range
    and take the first reference, as a NaN index does in searchsorted(left)
    followed by the clip."""
    import wideanglepropagation_b200.synthetic as S
    n, ps, dz, E = 64, 0.05, 2.0, 300e3
    V = _atoms(n, n, 2, 9, 80.0, ps, dz).astype(np.float32)
    probe = S.aperture_probe(n, n, ps, E, 25.0, dtype=np.complex64)
    low = V.copy()
    low[0, 5, 7] = low[0].min()
    want = wap.simulate_wpm(low, probe, dz, E, (ps, ps), n_bins=16)
    for bad in (np.nan, np.inf, -np.inf):
        W = low.copy()
        W[0, 5, 7] = bad
        got = wap.simulate_wpm(W, probe, dz, E, (ps, ps), n_bins=16)
        assert torch.isfinite(torch.view_as_real(got[0])).all()
        assert float((got[0] - want[0]).norm() / want[0].norm()) < 1e-6
