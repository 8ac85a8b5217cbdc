"""Repeated scans on the persistent scheduler agree bit for bit (nothing in a forward
scan depends on the order of its tiles).  Scans whose groups put few tiles of a pass
on each block, so that a block's row tiles often follow its column tiles while some
of its warps are still in those: there a warp's row exchange once overwrote what
another had yet to read, in one call in sixty of the first case's shape.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,B,N,repeats", [(512, 71, 40, 200), (512, 9, 60, 100), (256, 90, 60, 100),
                                           (128, 200, 60, 60), (1024, 9, 12, 40)])
def test_scans_repeat_bit_for_bit(n, B, N, repeats):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import wideanglepropagation_b200 as wap
    import wideanglepropagation_b200.synthetic as S
    g = torch.Generator(device="cuda").manual_seed(n + B)
    ps, dz, E = 0.069, 3.9, 80e3
    V = 60.0 * torch.rand((2, N, n, n), device="cuda", generator=g) ** 4
    probe = torch.from_numpy(S.aperture_probe(n, n, ps, E, 20.0, -30.0, dtype=np.complex64)).cuda()
    pos = torch.randint(0, n, (B, 2), device="cuda", generator=g, dtype=torch.int32)
    draw = (np.arange(B) % 2).astype(np.int32)
    H = wap.angular_spectrum_propagation_kernel(n, n, (ps, ps), dz, E)

    def run():
        return wap.simulate_fresnel_as(V, probe, H, dz, E, positions=pos, draw=draw, return_wavefronts=False)[:2]

    first = run()
    for _ in range(repeats):
        for a, b in zip(run(), first):
            assert torch.equal(a, b)
