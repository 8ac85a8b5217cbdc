"""Calls captured in a CUDA graph and replayed, against the same calls made
eagerly: inputs that the graph's own kernels write, and later calls on the same
cached plan.

Bar: rel-L2 <= 1e-6 (the same kernels; a captured call may evaluate the
transmission in the passes, with the table's function).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-6


@pytest.fixture(scope="module")
def wap():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import wideanglepropagation_b200 as w
    return w


def _case(wap, ny, nx, N, seed=0):
    import wideanglepropagation_b200.synthetic as S
    ps, dz, E = 0.1, 2.0, 200e3
    rng = np.random.default_rng(seed + ny)
    V = torch.from_numpy((S.random_gaussian_stack(rng, N, ny, nx, ps, 8, 30.0, 0.3) / dz).astype(np.float32)).cuda()
    probe = torch.from_numpy(S.aperture_probe(ny, nx, ps, E, 20.0, -30.0, dtype=np.complex64)).cuda()
    H = wap.angular_spectrum_propagation_kernel(ny, nx, (ps, ps), dz, E).to(torch.complex64)
    return V, probe, H, dz, E


def _close(a, b):
    return float((a - b).norm() / b.norm()) <= TOL


def _captured(fn):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        out = fn()
    return g, out


@pytest.mark.parametrize("ny,nx", [(100, 60), (67, 101)])   # mixed radix, Bluestein
def test_positions_written_just_before_the_call(wap, ny, nx):
    """The call's first pass directly follows the kernel that writes the
    positions (their cast to int32), with no table kernel between the two."""
    V, probe, H, dz, E = _case(wap, ny, nx, 4)
    rng = np.random.default_rng(1)
    sets = [torch.from_numpy(rng.integers(0, min(ny, nx), (5, 2))).cuda() for _ in range(3)]
    pos = sets[0].clone()

    def call(p, n=4):
        return wap.simulate_fresnel_as(V[:n], probe, H, dz, E, positions=p, return_wavefronts=False)[:2]

    call(pos, 1)   # the plan, with a table too small for the captured call
    g, out = _captured(lambda: call(pos))
    for s in sets:
        pos.copy_(s)
        g.replay()
        torch.cuda.synchronize()
        got = [o.clone() for o in out]
        for a, b in zip(got, call(s)):
            assert _close(a, b)


def test_general_grid_goes_without_the_plans_table(wap):
    """A captured call on a grid that is not a power of two reads no memory of
    the plan that another call writes: no table kernel (2 N + 1 passes)."""
    from wideanglepropagation_b200 import _lib
    V, probe, H, dz, E = _case(wap, 48, 60, 3)

    def call():
        return wap.simulate_fresnel_as(V, probe, H, dz, E, return_wavefronts=False)[:2]

    want = call()
    n0 = _lib.launch_count()
    g, out = _captured(call)
    assert _lib.launch_count() - n0 == 2 * 3 + 1
    g.replay()
    torch.cuda.synchronize()
    for a, b in zip(out, want):
        assert _close(a, b)


def _wpm(wap, V, probe, dz, E, **kw):
    return wap.simulate_wpm(V, probe, dz, E, (0.1, 0.1), 6, 1.0, return_wavefronts=False, **kw)[:2]


@pytest.mark.parametrize("kind", ["scan", "wpm"])
def test_larger_calls_leave_a_captured_one_valid(wap, kind):
    """Later calls on the cached plan with more slices (its table and records are
    replaced by larger ones) and with more probes (the plan is)."""
    n, B = (128, 16) if kind == "scan" else (64, 3)
    V, probe, H, dz, E = _case(wap, n, n, 12)
    pos = torch.from_numpy(np.random.default_rng(2).integers(0, n, (B, 2)).astype(np.int32)).cuda()
    many = pos.repeat(5, 1)

    def call(k, p=pos):
        if kind == "wpm":
            return _wpm(wap, V[:k], probe, dz, E, positions=p)
        return wap.simulate_fresnel_as(V[:k], probe, H, dz, E, positions=p, return_wavefronts=False)[:2]

    want = [o.clone() for o in call(3)]
    g, out = _captured(lambda: call(3))
    call(12)
    if kind == "wpm":
        _wpm(wap, V, probe, dz, E, positions=many)
    else:   # 80 different waves: past the cached plan's 64
        wap.simulate_fresnel_as(V, probe.repeat(80, 1, 1), H, dz, E, return_wavefronts=False)
    fill = [torch.full((1 << 20,), float("nan"), device="cuda") for _ in range(8)]
    for o in out:
        o.zero_()
    g.replay()
    torch.cuda.synchronize()
    del fill
    for a, b in zip(out, want):
        assert _close(a, b)
    del g
    wap.release_caches()
