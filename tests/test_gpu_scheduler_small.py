"""The scheduler's tests of small scans, on the scheduler.

Scans of few probes go to the pass kernels where those are the faster way
(``SCAN_FROM_PROBES``, ``SCAN_GRAD_FROM_PROBES``: up to 63 probes on 128^2), and the
tests below, written for the scheduler, with them.  Here they run once more with the
hand-over at eight probes on every grid, and each has to reach the scheduler.
"""
import pytest

torch = pytest.importorskip("torch")

from test_gpu_detector import (test_fused_crop_persistent_scan, test_gradient_through_the_window,  # noqa: E402,F401
                               test_gradient_window_and_exit_loss)
from test_gpu_edges import (test_inference_mode_complex128_transfer, test_one_slice,  # noqa: E402,F401
                            test_release_caches_frees_and_recovers, test_wrapping_positions_both_paths)
from test_gpu_grad import (test_persistent_gradient_exit_wave_loss, test_persistent_gradient_matches_autograd,  # noqa: E402,F401
                           test_persistent_gradient_two_pending_graphs, wap)
from test_gpu_probe_accumulate import test_accumulate_draws_per_position  # noqa: E402,F401
from test_gpu_streams import test_gradient_scans_on_two_streams  # noqa: E402,F401

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def hand_over_at_eight(request, monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wideanglepropagation_b200 import autograd as A
    from wideanglepropagation_b200 import propagation as P
    for n in (128, 256):
        monkeypatch.setitem(P.SCAN_FROM_PROBES, n, 8)
        monkeypatch.setitem(P.SCAN_GRAD_FROM_PROBES, n, 8)
    runs = []
    scan_run, acquire = P._scan_run, A._acquire
    monkeypatch.setattr(P, "_scan_run", lambda *a, **k: (runs.append("forward"), scan_run(*a, **k))[1])
    monkeypatch.setattr(A, "_acquire", lambda *a, **k: (runs.append("gradient"), acquire(*a, **k))[1])
    yield
    few = {"n_side": (2,), "B": (7,)}   # the cases of four and seven probes are the pass kernels'
    params = getattr(request.node, "callspec", None)
    if not any(params.params.get(k) in v for k, v in few.items()) if params else True:
        assert runs, "the scheduler was not reached"
