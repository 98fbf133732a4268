"""The mesh distance's two walks, a group of eight lanes per sample up to 40,000 samples
and a thread per sample beyond, against a plain search, at the sizes where the rule and
the hierarchies turn; and with faces that have no distance."""
import numpy as np
import pytest

from test_nonfinite_gpu import _closest, _soup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _plain_search(P, V, F):
    d2 = np.full(len(P), np.inf)
    with np.errstate(all="ignore"):
        for t in F:
            a, b, c = (np.broadcast_to(V[i].astype(np.float64), P.shape) for i in t)
            d2 = np.fmin(d2, ((P - _closest(P, a, b, c)) ** 2).sum(1))
    return np.sqrt(d2)


# 39,903 samples a face at 281 steps an edge, 40,186 at 282
@pytest.mark.parametrize("m,subdiv", [(1, 281), (1, 282), (2, 282), (3, 282), (87, 281), (87, 282), (513, 282)])
@pytest.mark.parametrize("bad", [None, "nan", "inf"])
def test_both_walks_match_plain_search(torch_cuda, m, subdiv, bad):
    from oracle import check_oracle as C
    from pamo_b200 import metrics

    rng = np.random.default_rng(m)
    V, F = _soup(rng, m)
    if bad and m > 1:
        hit = rng.choice(m, max(1, m // 10), replace=False)
        V.reshape(m, 3, 3)[hit, rng.integers(0, 3, len(hit)), rng.integers(0, 3, len(hit))] = float(bad)
    F = F.copy()
    if m > 80:
        F[5] = -1  # a removed face
    A, FA = _soup(rng, 1)
    got = metrics.mesh_distance(A, FA, V, F, subdiv=subdiv)
    P = C.face_samples(A, FA, subdiv)
    assert got["samples"] == len(P)
    d = _plain_search(P, V, F[F[:, 0] >= 0])
    assert d.max() < 4
    # FP64 on both sides: some dozen roundings a distance, and 40,000 in the sum
    assert abs(got["max"] - d.max()) < 1e-12
    assert abs(got["mean_sq"] - (d**2).mean()) < 40_186 * 2.3e-16 * 16
