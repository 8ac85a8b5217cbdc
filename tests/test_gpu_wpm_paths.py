"""Instances that the size rules pick and other tests do not reach, against the FP64
oracle: the reference-field kernels of grids that reach the evanescent edge in every
launch shape and bin split, the interpolating kernels with one thread group per line,
Bluestein lines with 16 elements per thread, and a plane wave on general grids.

Bar: rel-L2 <= 1e-5 as on the other paths.  The plane wave's pattern is one number,
the square of its mean: 1e-6, between the 2e-7 of 100 slices with the constant part of
the k_x = 0 column carried beside it and their 3e-6 to 5e-6 without.
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


def _inputs(ny, nx, N, B, seed=0):
    rng = np.random.default_rng(ny * 17 + nx + seed)
    V = (60.0 * rng.uniform(0, 1, (N, ny, nx)) ** 2).astype(np.float32)
    psi = (rng.normal(size=(ny, nx)) + 1j * rng.normal(size=(ny, nx))).astype(np.complex64)
    pos = np.stack([rng.integers(0, ny, B), rng.integers(0, nx, B)], 1).astype(np.int32)
    return V, psi, pos


def _check(got, ref, b):
    from oracle import propagation_oracle as O
    for g, r in zip(got, ref):
        if r is not None:
            assert O.rel_l2(g[b].cpu().numpy(), r) < TOL


def test_reference_fields_every_launch_shape(wap):
    from oracle import propagation_oracle as O
    from wideanglepropagation_b200 import _lib, autotune
    n, K, ps = 128, 24, 0.01
    V, psi, pos = _inputs(n, n, 2, 1)
    ref = O.simulate_wpm(V, O.move_probe(psi, tuple(pos[0])), 1.0, 300e3, (ps, ps), K, 1.5)
    plan = wap.get_plan(n, n, 1, _lib.WAP_OP_WPM, K)
    old = plan.config()
    shapes = 0
    try:
        for cfg in autotune.candidates(n, n):
            if cfg[0] < 8 or cfg[1] < 8:
                continue   # 4 elements per thread: Fresnel/AS plans only
            plan.set_config(*cfg)
            _check(wap.simulate_wpm(V, psi, 1.0, 300e3, (ps, ps), K, 1.5, positions=pos), ref, 0)
            shapes += 1
    finally:
        plan.hint_config(*old)
    assert shapes > 8


@pytest.mark.parametrize("ny,nx,B,K", [(256, 256, 1, 16), (256, 256, 1, 100), (64, 512, 2, 24), (512, 64, 1, 9),
                                       (128, 128, 20, 7), (32, 32, 300, 12)])
def test_reference_fields_bin_split(wap, ny, nx, B, K):
    from oracle import propagation_oracle as O
    V, psi, pos = _inputs(ny, nx, 3, B)
    got = wap.simulate_wpm(V, psi, 1.0, 300e3, (0.01, 0.01), K, 2.0, positions=pos)
    for b in {0, B - 1}:
        _check(got, O.simulate_wpm(V, O.move_probe(psi, tuple(pos[b])), 1.0, 300e3, (0.01, 0.01), K, 2.0), b)


@pytest.mark.parametrize("ny,nx,B", [(512, 512, 2), (1024, 1024, 1), (256, 256, 6), (32, 32, 900)])
def test_nodes_one_group_per_line(wap, ny, nx, B):
    from oracle import propagation_oracle as O
    V, psi, pos = _inputs(ny, nx, 2, B)
    got = wap.simulate_wpm(V, psi, 2.0, 300e3, (0.05, 0.05), 8, 1.0, positions=pos)
    for b in {0, B - 1}:
        _check(got, O.simulate_wpm(V, O.move_probe(psi, tuple(pos[b])), 2.0, 300e3, (0.05, 0.05), 8, 1.0), b)


@pytest.mark.parametrize("ny,nx,B", [(31, 19, 1000), (37, 37, 600), (101, 101, 48), (257, 22, 120), (509, 41, 60),
                                     (1021, 1021, 1)])
def test_bluestein_sixteen_elements(wap, ny, nx, B):
    from oracle import propagation_oracle as O
    V, psi, pos = _inputs(ny, nx, 3, B)
    H = O.angular_spectrum_propagation_kernel(ny, nx, (0.1, 0.1), 2.0, 200e3)
    got = wap.simulate_fresnel_as(V, psi, H, 2.0, 200e3, positions=pos)
    for b in {0, B - 1}:
        _check(got, O.simulate_fresnel_as(V, O.move_probe(psi, tuple(pos[b])), H, 2.0, 200e3), b)


@pytest.mark.parametrize("ny,nx", [(100, 100), (101, 64), (60, 97)])
def test_plane_wave_on_general_grids(wap, ny, nx):
    from oracle import propagation_oracle as O
    V, _, _ = _inputs(ny, nx, 60, 1)
    psi = np.ones((ny, nx), np.complex64)
    ex, dp, _ = wap.simulate_wpm(V, psi, 1.0, 300e3, (0.05, 0.05), 8, 1.0, return_wavefronts=False)
    rex, rdp, _ = O.simulate_wpm(V, psi, 1.0, 300e3, (0.05, 0.05), 8, 1.0, return_wavefronts=False)
    assert O.rel_l2(ex.cpu().numpy(), rex) < TOL
    assert O.rel_l2(dp.cpu().numpy(), rdp) < 1e-6
