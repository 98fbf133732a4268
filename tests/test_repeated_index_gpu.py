"""Faces that repeat an index, as scanned and exported meshes hold them: a collapse
that takes such a vertex away removes the face, round by round as the oracle does."""
import numpy as np
import pytest

from helpers import bits, compact

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _open_grid(k, n_repeats, seed):
    """A k x k grid with a boundary (its edges start at cost 0, so they collapse
    whatever they touch) and faces (a, a, b), (a, b, a), (b, a, a), (a, a, a) in it."""
    rng = np.random.default_rng(seed)
    x, y = np.meshgrid(np.arange(k), np.arange(k))
    V = np.stack([x.ravel(), y.ravel(), 0 * x.ravel()], 1) + 0.05 * rng.normal(size=(k * k, 3))
    i = np.arange(k * k).reshape(k, k)
    q = [i[:-1, :-1].ravel(), i[:-1, 1:].ravel(), i[1:, 1:].ravel(), i[1:, :-1].ravel()]
    F = np.concatenate([np.stack([q[0], q[1], q[2]], 1), np.stack([q[0], q[2], q[3]], 1)])
    more = []
    for t in F[rng.integers(0, len(F), n_repeats)]:
        a, b = t[rng.permutation(3)[:2]]
        more.append([(a, a, b), (a, b, a), (b, a, a), (a, a, a)][rng.integers(0, 4)])
    F = np.concatenate([F, more])
    return V.astype(np.float32), F[rng.permutation(len(F))].astype(np.int32)


def _rounds(V, F, n_rounds):
    """The oracle's rounds, and how many collapses took a face with the vertex in it twice."""
    from oracle import oracle as O

    orc = O.Stage2Oracle()
    scale = float((V.max(0) - V.min(0)).max())
    undo = np.zeros(0, np.int32)
    P, T = V, O.shuffle_faces(F)
    out, hits = [], 0
    for _ in range(n_rounds):
        r = orc.forward(P, T, undo, len(undo), scale, 1e-3, 0)
        out.append((P, T, undo, r))
        for u, v in orc.edges()[orc.collapsed()]:
            if r[2][v] == 0:
                hits += int((((T == v).sum(1) > 1) & ((T == u).sum(1) == 0)).sum())
        undo = r[4]
        P, T = compact(*r[:4])
    return out, scale, hits


@pytest.mark.parametrize("k,n_repeats,seed", [(5, 6, 2), (8, 40, 21), (8, 40, 24), (14, 12, 0), (14, 12, 22),
                                              (20, 300, 18)])
def test_rounds_with_repeated_indices_match_oracle(torch_cuda, k, n_repeats, seed):
    import pamo_b200

    V, F = _open_grid(k, n_repeats, seed)
    want, scale, hits = _rounds(V, F, 4)
    assert hits > 0  # the case is there
    gpu = pamo_b200.CUDSP_Free()
    dev = lambda x: torch_cuda.from_numpy(np.ascontiguousarray(x)).cuda()
    for r, (P, T, undo, (op, ot, oo, om, ou)) in enumerate(want):
        g = gpu.forward(dev(P), dev(F if r == 0 else T), dev(undo), len(undo), scale, 1e-3, False, r == 0)
        gv, gt, go, gm, gu = [x.cpu().numpy() for x in g]
        assert np.array_equal(gt, ot), f"round {r}: faces differ"
        assert np.array_equal(go, oo), f"round {r}: occupancy differs"
        assert np.array_equal(bits(gv), bits(op)), f"round {r}: points differ"
        assert np.array_equal(gm, om) and np.array_equal(gu, ou), f"round {r}: map or undo list differ"
