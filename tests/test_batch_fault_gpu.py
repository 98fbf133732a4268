"""A fault that a prefix scan recorded (a bounded wait that ran out) ends a batch's
round where its compaction reads the counters, and batches made later run."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAMO_ERR_DEVICE = 4


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def test_batch_compaction_reports_a_scan_fault(torch_cuda):
    import pamo_b200
    from pamo_b200 import _lib
    from pamo_b200 import meshgen as mg
    from pamo_b200.batch import simplify_many

    ctx = pamo_b200.Context(0)
    stream = ctypes.c_void_p(torch_cuda.cuda.current_stream().cuda_stream)
    for _ in range(2):
        assert _lib.lib().pamo_debug_wait_timeout(ctx.handle, 0, 4096, stream) == PAMO_ERR_DEVICE
    V, F = mg.displaced_icosphere(4, 3)
    V, F = V.astype(np.float32), F.astype(np.int32)
    (v, f), = simplify_many([(V, F)], ratio=0.1, min_verts=0)
    wv, wf, _ = pamo_b200.stage2_run(pamo_b200.Context(0), torch_cuda.from_numpy(V).cuda(),
                                     torch_cuda.from_numpy(F).cuda(), int(0.1 * len(F)))
    assert np.array_equal(f, wf.cpu().numpy())
    assert np.array_equal(v.view(np.uint32), wv.cpu().numpy().view(np.uint32))
