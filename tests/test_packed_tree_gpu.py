"""The packed tree's query (pamo_self_intersect's candidate pairs) at the sizes
where its levels and padding change: the pairs of live faces with overlapping
boxes that share fewer than two vertices, counted by brute force."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _pairs(V, F):
    P = V[np.maximum(F, 0)]
    lo, hi = P.min(1), P.max(1)
    live = F[:, 0] >= 0
    n = 0
    for f in range(len(F)):
        if not live[f]:
            continue
        g = np.arange(f + 1, len(F))
        g = g[live[g] & (lo[g] <= hi[f]).all(1) & (hi[g] >= lo[f]).all(1)]
        n += int(((F[g][:, :, None] == F[f][None, None, :]).sum((1, 2)) < 2).sum())
    return n


# 8 leaves a group, 512 a tile, 8 tiles before the next level starts
@pytest.mark.parametrize("m", [1, 2, 7, 8, 9, 64, 65, 511, 512, 513, 4095, 4096, 4097])
@pytest.mark.parametrize("dead", [False, True])
def test_candidate_pairs_match_brute_force(torch_cuda, m, dead):
    import pamo_b200

    rng = np.random.default_rng(m)
    n = 3 * m + 3
    V = rng.random((n, 3)).astype(np.float32)
    F = rng.integers(0, n, (m, 3)).astype(np.int32)
    # mostly small faces about their first corner, neighbours sharing one or two corners
    F[:, 1:] = np.minimum(F[:, :1] + rng.integers(1, 3, (m, 2)), n - 1)
    V = (np.cumsum(rng.normal(size=(n, 3)), 0) * 0.05).astype(np.float32)
    if dead:
        F[::5] = -1
    want = _pairs(V, F)
    ctx = pamo_b200.Context(0)
    for _ in range(2):  # the second call reuses the buffers
        _, got = pamo_b200.self_intersect(ctx, torch_cuda.from_numpy(V).cuda(), torch_cuda.from_numpy(F).cuda())
        assert got == want
