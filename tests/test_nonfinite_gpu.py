"""Meshes with NaN and infinite coordinates in the acceptance checks: a distance
to such a mesh is the least over the faces that have one, as a plain search over
all faces finds it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _soup(rng, m):
    """m small triangles about random points, no two sharing a vertex."""
    V = (rng.random((m, 1, 3)) + 0.05 * rng.normal(size=(m, 3, 3))).astype(np.float32).reshape(-1, 3)
    return V, np.arange(3 * m, dtype=np.int32).reshape(-1, 3)


def _closest(p, a, b, c):
    """The closest points of the triangles to p (Ericson, Real-Time Collision Detection, 5.1.5)."""
    dot = lambda x, y: (x * y).sum(1)
    ab, ac, ap, bp, cp = b - a, c - a, p - a, p - b, p - c
    d1, d2, d3, d4, d5, d6 = dot(ab, ap), dot(ac, ap), dot(ab, bp), dot(ac, bp), dot(ab, cp), dot(ac, cp)
    vc, vb, va = d1 * d4 - d3 * d2, d5 * d2 - d1 * d6, d3 * d6 - d5 * d4
    col = lambda x: x[:, None]
    den = 1.0 / (va + vb + vc)
    cond = [(d1 <= 0) & (d2 <= 0), (d3 >= 0) & (d4 <= d3), (vc <= 0) & (d1 >= 0) & (d3 <= 0), (d6 >= 0) & (d5 <= d6),
            (vb <= 0) & (d2 >= 0) & (d6 <= 0), (va <= 0) & (d4 - d3 >= 0) & (d5 - d6 >= 0)]
    pick = [a, b, a + col(d1 / (d1 - d3)) * ab, c, a + col(d2 / (d2 - d6)) * ac,
            b + col((d4 - d3) / ((d4 - d3) + (d5 - d6))) * (c - b)]
    q = a + ab * col(vb * den) + ac * col(vc * den)
    for k in range(5, -1, -1):
        q = np.where(col(cond[k]), pick[k], q)
    return q


def _plain_search(P, V, F):
    a, b, c = (V[F[:, k]].astype(np.float64) for k in range(3))
    with np.errstate(all="ignore"):
        return np.array([np.sqrt(np.fmin.reduce(((p - _closest(p, a, b, c)) ** 2).sum(1))) for p in P])


# 8 leaves a group, 512 a tile; one bad face in a group of eight, and most of them
@pytest.mark.parametrize("bad", ["nan", "inf", "-inf"])
@pytest.mark.parametrize("m,n_bad", [(8, 1), (9, 5), (40, 7), (513, 30), (6000, 300)])
def test_distance_of_non_finite_mesh_matches_plain_search(torch_cuda, m, n_bad, bad):
    from oracle import check_oracle as C
    from pamo_b200 import metrics

    rng = np.random.default_rng(m)
    V, F = _soup(rng, m)
    hit = rng.choice(m, n_bad, replace=False)
    V.reshape(m, 3, 3)[hit, rng.integers(0, 3, n_bad), rng.integers(0, 3, n_bad)] = float(bad)
    A, FA = _soup(rng, 60)
    got = metrics.mesh_distance(A, FA, V, F, subdiv=2)
    d = _plain_search(C.face_samples(A, FA, 2), V, F)
    assert np.isfinite(d).all()
    # FP64 on both sides, some dozen roundings of values below 10
    assert abs(got["max"] - d.max()) < 1e-12
    assert abs(got["mean_sq"] - (d**2).mean()) < 1e-12


def _boundless(V, F, kind):
    """Face 0's box made NaN, or all of space, on every axis."""
    V = V.copy()
    V[F[0]] = np.nan if kind == "nan" else np.array([[-np.inf] * 3, [np.inf] * 3, [0] * 3], np.float32)
    return V


def _overlaps(V, F):
    """Pairs f < g whose boxes are not apart."""
    P = V[F]
    lo, hi = P.min(1), P.max(1)
    n = 0
    for f in range(len(F)):
        apart = (hi[f + 1:] < lo[f]) | (hi[f] < lo[f + 1:])
        n += int((~apart.any(1)).sum())
    return n


# the ends of a group, a tile and a level, where padding starts
@pytest.mark.parametrize("kind", ["nan", "inf"])
@pytest.mark.parametrize("m", [1, 2, 8, 9, 63, 65, 512, 513, 4095, 4097, 33000])
def test_face_apart_from_nothing_meets_every_face_once(torch_cuda, m, kind):
    import pamo_b200
    from pamo_b200 import metrics

    V, F = _soup(np.random.default_rng(m), m)
    V = _boundless(V, F, kind)
    want = _overlaps(V, F)
    assert want >= m - 1
    ctx = pamo_b200.Context(0)
    _, got = pamo_b200.self_intersect(ctx, torch_cuda.from_numpy(V).cuda(), torch_cuda.from_numpy(F).cuda())
    assert got == want
    res = metrics.check_mesh(V, F)
    assert res["degenerate_faces"] in (0, 1)  # such a face may count as degenerate, and is then not tested
    assert res["candidate_pairs"] == want - (m - 1) * res["degenerate_faces"]


@pytest.mark.parametrize("m", [1, 9, 513, 4097, 33000])
def test_sample_without_coordinates_is_at_no_distance(torch_cuda, m):
    from pamo_b200 import metrics

    rng = np.random.default_rng(m)
    V, F = _soup(rng, m)
    A, FA = _soup(rng, 5)
    A[FA[2]] = np.nan
    got = metrics.mesh_distance(A, FA, V, F, subdiv=2)
    assert got["samples"] == 30
    assert got["max"] == np.sqrt(np.finfo(np.float64).max)
