"""Launch shapes of plans: one that the caller sets is launched as it is, a hinted
one may give way to shorter lines per thread where a pass is small.

Shapes of different element counts have different radices, so their results
differ in the last bits; passes of one shape agree bit for bit.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wap():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import wideanglepropagation_b200 as w
    return w


@pytest.mark.parametrize("n,B", [(256, 1), (512, 1)])
def test_set_shape_is_the_launched_one(wap, n, B):
    from wideanglepropagation_b200 import _lib
    from wideanglepropagation_b200.propagation import Plan
    rng = np.random.default_rng(n)
    V = torch.from_numpy(rng.uniform(0, 30, (1, 3, n, n)).astype(np.float32)).cuda()
    psi = torch.from_numpy((rng.normal(size=(B, n, n)) + 1j * rng.normal(size=(B, n, n))).astype(np.complex64)).cuda()
    H = wap.fresnel_propagation_kernel(n, n, (0.1, 0.1), 2.0, 200e3).to(torch.complex64)
    plan = Plan(n, n, 8, _lib.WAP_OP_FRESNEL_AS)

    def run():
        ex = torch.empty_like(psi)
        stack = torch.empty((B, 3, n, n), dtype=torch.complex64, device="cuda")
        p = lambda t: t.data_ptr()   # noqa: E731
        _lib.check(_lib.lib().wap_multislice_fwd(plan.handle, p(V), 3, 1, None, p(psi), B, 1, None, p(H), None, 2.0,
                                                 200e3, p(ex), None, p(stack), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        return ex

    out = {}
    for cfg in ((8, 8, 8), (16, 8, 8), (8, 16, 8), (16, 16, 8)):
        plan.set_config(*cfg)
        assert plan.config() == cfg
        out[cfg] = run()
    got = list(out.values())
    for i in range(4):
        for j in range(i):
            assert not torch.equal(got[i], got[j]), (i, j)
            assert float((got[i] - got[j]).norm() / got[j].norm()) < 2e-6
    plan.hint_config(16, 16, 16)
    assert torch.equal(run(), out[(8, 8, 8)])   # both passes are small
    plan.close()
