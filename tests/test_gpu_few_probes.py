"""Pass launch shapes of small grids and few probes (fewer rows and columns per
block, plans without a tuned shape), and the counts on either side of the
hand-over to the persistent scheduler, against the FP64 oracle.

Bar: rel-L2 <= 1e-5, as on the other paths; probes on the two sides of the
hand-over agree to 8e-6 (the scheduler's stage twiddles are float32 up to 160
slices: at most 4.9e-6 from FP64 there, the passes 2.4e-6).
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


def _case(ny, nx, N):
    import wideanglepropagation_b200.synthetic as S
    ps, dz, E = 0.1, 2.0, 200e3
    rng = np.random.default_rng(ny * 3 + nx)
    V = np.stack([S.gaussian_slice(ny, nx, ps, rng.uniform(0, 1, (8, 2)) * [ny * ps, nx * ps], 30.0, 0.3)
                  for _ in range(N)]) / dz
    return V.astype(np.float32), S.aperture_probe(ny, nx, ps, E, 20.0, -30.0, dtype=np.complex64), ps, dz, E


@pytest.mark.parametrize("ny,nx,B", [(32, 32, 1), (64, 64, 1), (64, 64, 3), (32, 256, 1), (512, 128, 2), (2048, 32, 1),
                                     (128, 64, 5), (256, 256, 1), (256, 256, 4), (256, 256, 8), (128, 128, 16),
                                     (256, 512, 6)])
def test_shapes_match_oracle(wap, ny, nx, B):
    from oracle import propagation_oracle as O
    V, probe, ps, dz, E = _case(ny, nx, 4)
    pos = np.array([[7 * b % ny, 11 * b % nx] for b in range(B)], np.int32)
    H = O.angular_spectrum_propagation_kernel(ny, nx, (ps, ps), dz, E)
    ex, dp, st = wap.simulate_fresnel_as(V, probe, H, dz, E, positions=pos)
    for b in range(B):
        ref = O.simulate_fresnel_as(V, O.move_probe(probe, tuple(pos[b])), H, dz, E)
        for g, r in zip((ex, dp, st), ref):
            assert O.rel_l2(g[b].cpu().numpy(), r) < TOL


@pytest.mark.parametrize("n", [128, 256])
def test_scheduler_hand_over(wap, n):
    from wideanglepropagation_b200.propagation import SCAN_FROM_PROBES
    V, probe, ps, dz, E = _case(n, n, 6)
    H = wap.angular_spectrum_propagation_kernel(n, n, (ps, ps), dz, E)
    many = SCAN_FROM_PROBES[n]
    pos = np.random.default_rng(n).integers(0, n, (many, 2)).astype(np.int32)
    out = []
    for B in (many - 1, many):   # passes, scheduler
        ex, dp, _ = wap.simulate_fresnel_as(V, probe, H, dz, E, positions=pos[:B], return_wavefronts=False)
        out.append((ex[:many - 1], dp[:many - 1]))
    for a, b in zip(*out):
        assert float((a - b).norm() / b.norm()) < 8e-6
