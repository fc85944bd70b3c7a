"""Plans given up while a CUDA graph is being captured, and while their work still runs."""
import threading
import time

import pytest

from imaging2d_wlsq_b200 import migration, synthetic
from imaging2d_wlsq_b200._lib import lib

pytestmark = pytest.mark.gpu


def _plan():
    """A plan with buffers large enough for the pool of released blocks."""
    return migration.Plan.for_workload(synthetic.plain_medium(nx=1024, nz=64, nf=16, ns=16))


@pytest.mark.parametrize("mode", ["relaxed", "thread_local"])
def test_closing_a_plan_leaves_a_capture_valid(mode):
    """In the capturing thread (relaxed mode) or in another one (thread-local mode): freeing device memory
    is allowed there, so giving up a plan is."""
    import torch
    plan = _plan()
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode=mode):
        x.add_(1)
        if mode == "relaxed":
            plan.close()
        else:
            t = threading.Thread(target=plan.close)
            t.start()
            t.join()
        x.add_(1)
    graph.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 2000.0
    lib().img2d_release_host_cache()


@pytest.mark.parametrize("what", ["plan", "scratch"])
def test_giving_up_blocks_waits_for_the_work_on_them(what):
    """A block that another plan may take next has nobody using it: giving it up returns after the
    device's queued work (here 0.2 s of it on another stream).  "scratch" gives up one large block."""
    import torch
    plan = _plan()
    migration.fp32_peak_tflops()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(400_000_000)
    t = time.perf_counter()
    if what == "plan":
        plan.close()
    else:
        migration.fp32_peak_tflops()
    assert side.query() and time.perf_counter() - t > 0.1
    plan.close()
    lib().img2d_release_host_cache()
