"""The edge cost by groups of eight lanes where a one-ring does not fit one step:
whole stage-2 loops on spheres whose pole rings have 7 to 40 faces, equal to the
oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _globe(segments, rings, seed):
    """A latitude / longitude sphere, slightly displaced: its two poles have `segments` faces each."""
    rng = np.random.default_rng(seed)
    th = np.pi * (np.arange(rings) + 1) / (rings + 1)
    ph = 2 * np.pi * np.arange(segments) / segments
    T, P = np.meshgrid(th, ph, indexing="ij")
    V = np.stack([np.sin(T) * np.cos(P), np.sin(T) * np.sin(P), np.cos(T)], -1).reshape(-1, 3)
    V = np.concatenate([V, [[0, 0, 1], [0, 0, -1]]])
    V *= 1 + 0.02 * rng.normal(size=(len(V), 1))
    n, s = len(V) - 2, len(V) - 1
    F = []
    for j in range(segments):
        k = (j + 1) % segments
        F.append((n, j, k))
        F.append((s, (rings - 1) * segments + k, (rings - 1) * segments + j))
        for i in range(rings - 1):
            a, b, c, d = i * segments + j, (i + 1) * segments + j, (i + 1) * segments + k, i * segments + k
            F += [(a, b, c), (a, c, d)]
    return V.astype(np.float32), np.asarray(F, np.int32)


@pytest.mark.parametrize("segments", [7, 8, 9, 16, 17, 24, 40])
def test_high_valence_rings_match_oracle(torch_cuda, segments):
    import pamo_b200
    from oracle import oracle as O

    V, F = _globe(segments, 14, segments)
    ctx = pamo_b200.Context(0)
    v, f, rounds = pamo_b200.stage2_run(ctx, torch_cuda.from_numpy(V).cuda(), torch_cuda.from_numpy(F).cuda(),
                                        int(0.1 * len(F)))
    ov, of, orounds = O.pamo_run_stage2(V, F, 0.1, min_verts=0)
    assert rounds == orounds
    assert np.array_equal(f.cpu().numpy(), of)
    assert np.array_equal(v.cpu().numpy().view(np.uint32), ov.view(np.uint32))
