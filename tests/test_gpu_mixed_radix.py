"""Mixed-radix and Bluestein lines (csrc/wap_mixed.cuh) against the FP64 oracle on
sides that reach every radix (2 .. 8), one to five stages, the turn at each end
radix, primes (Bluestein, smallest and largest), and a power-of-two side beside
them; several probes with draws in one call.

Bar: rel-L2 <= 1e-5 of exit wave, pattern and wavefronts, as on the other grids
(measured ~1e-6; the transforms' constants carry hi + lo parts).
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


def _case(ny, nx, N, D=1):
    import wideanglepropagation_b200.synthetic as S
    ps, dz, E = 0.1, 2.0, 200e3
    rng = np.random.default_rng(ny * 7 + nx)
    V = np.stack([np.stack([S.gaussian_slice(ny, nx, ps, rng.uniform(0, 1, (8, 2)) * [ny * ps, nx * ps], 30.0, 0.3)
                            for _ in range(N)]) for _ in range(D)]) / dz
    return V.astype(np.float32), S.aperture_probe(ny, nx, ps, E, 20.0, -30.0, dtype=np.complex64), ps, dz, E


@pytest.mark.parametrize("ny,nx", [
    (17, 18), (20, 49), (24, 60), (35, 98), (30, 30), (75, 36), (48, 100), (125, 64), (243, 21), (625, 32),
    (686, 40), (32, 720), (997, 33), (1000, 24), (19, 1021), (1023, 20), (64, 972), (1024, 48)])
def test_sides_match_oracle(wap, ny, nx):
    from oracle import propagation_oracle as O
    V, probe, ps, dz, E = _case(ny, nx, 3)
    H = O.angular_spectrum_propagation_kernel(ny, nx, (ps, ps), dz, E)
    got = wap.simulate_fresnel_as(V[0], probe, H, dz, E)
    ref = O.simulate_fresnel_as(V[0], probe, H, dz, E)
    for g, r in zip(got, ref):
        assert O.rel_l2(g.cpu().numpy(), r) < TOL
    got = wap.simulate_wpm(V[0], probe, dz, E, (ps, ps), n_bins=9, power_spacing=1.5)
    ref = O.simulate_wpm(V[0], probe, dz, E, (ps, ps), n_bins=9, power_spacing=1.5)
    for g, r in zip(got, ref):
        assert O.rel_l2(g.cpu().numpy(), r) < TOL


@pytest.mark.parametrize("B", [1, 3, 40])
def test_probes_and_draws(wap, B):
    """Blocks of several lines, lines beyond the grid's edge, probes of two draws."""
    from oracle import propagation_oracle as O
    ny, nx, N = 45, 70, 4
    V, probe, ps, dz, E = _case(ny, nx, N, D=2)
    rng = np.random.default_rng(B)
    pos = np.stack([rng.integers(0, ny, B), rng.integers(0, nx, B)], 1).astype(np.int32)
    draw = (np.arange(B) % 2).astype(np.int32)
    H = O.angular_spectrum_propagation_kernel(ny, nx, (ps, ps), dz, E)
    ex, dp, st = wap.simulate_fresnel_as(V, probe, H, dz, E, positions=pos, draw=draw)
    wx, wp, ws = wap.simulate_wpm(V, probe, dz, E, (ps, ps), n_bins=12, positions=pos, draw=draw)
    for b in {0, B // 2, B - 1}:
        p0 = O.move_probe(probe, tuple(pos[b]))
        for got, ref in (((ex, dp, st), O.simulate_fresnel_as(V[draw[b]], p0, H, dz, E)),
                         ((wx, wp, ws), O.simulate_wpm(V[draw[b]], p0, dz, E, (ps, ps), n_bins=12))):
            for g, r in zip(got, ref):
                assert O.rel_l2(g[b].cpu().numpy(), r) < TOL
