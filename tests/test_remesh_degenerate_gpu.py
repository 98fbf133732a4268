"""The remesh of meshes with triangles without an area: their distances are not
distances (none on one side of their line), so the short reach of the distance pass
does not hold and the whole band is walked.  Against the CPU restatement with such
values dropped from the minimum, bit for bit; the short reach would give other bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _restated(V, F, R, voxels, monkeypatch):
    """The restatement whose triangles reach this many voxels (the band: 3)."""
    from oracle import s1_oracle as S1

    def unsigned_distance(tris, R, band):
        tris = np.asarray(tris, np.float64)
        reach = band if voxels == 3 else voxels / R
        d2 = np.full((R, R, R), band * band)
        lo = np.clip(np.floor((tris.min(1) - reach) * R - 0.5).astype(np.int64), 0, R - 1)
        hi = np.clip(np.ceil((tris.max(1) + reach) * R - 0.5).astype(np.int64), 0, R - 1)
        for (a, b, c), l, h in zip(tris, lo, hi):
            z, y, x = np.meshgrid(*(np.arange(l[k], h[k] + 1) for k in (2, 1, 0)), indexing="ij")
            P = (np.stack([x, y, z], -1) + 0.5) / R
            box = np.maximum(np.maximum(np.minimum(np.minimum(a, b), c) - P, P - np.maximum(np.maximum(a, b), c)), 0)
            with np.errstate(all="ignore"):
                dd = np.where((box**2).sum(-1) < reach * reach, S1._point_tri_d2(P, a, b, c), np.inf)
            sub = d2[l[2]:h[2] + 1, l[1]:h[1] + 1, l[0]:h[0] + 1]
            np.fmin(sub, dd, out=sub)
        return np.sqrt(d2)

    monkeypatch.setattr(S1, "unsigned_distance", unsigned_distance)
    return S1.remesh(V, F, R)


def _mesh(kind, seed):
    """Triangles along a random walk, every other one replaced by one of the kind named."""
    rng = np.random.default_rng(seed)
    n = 60
    V = np.cumsum(rng.normal(size=(n, 3)), 0) * 0.1
    if kind == "twice":  # most faces repeat an index: (a, a, b), (a, b, a), (b, a, a), (a, a, a)
        return V.astype(np.float32), np.minimum(np.arange(n)[:, None] + rng.integers(0, 3, (n, 3)), n - 1).astype(np.int32)
    F = np.minimum(np.arange(n)[:, None] + rng.permuted(np.tile(np.arange(4), (n, 1)), axis=1)[:, :3], n - 1)
    F = F[(F[:, 0] != F[:, 1]) & (F[:, 1] != F[:, 2]) & (F[:, 2] != F[:, 0])]
    a, b, F = F[1::2, 0], F[1::2, 1], F[::2]
    if kind == "points":
        more = np.stack([a, a, a], 1)
    else:  # a third corner on the edge, exactly, or off it by `kind` of its length
        V = np.round(V * 1024) / 1024  # so that halves are exact in float32
        off = 0.0 if kind == "collinear" else kind
        e = V[b] - V[a]
        side = np.cross(e, rng.normal(size=e.shape))
        side *= np.linalg.norm(e, axis=1, keepdims=True) / np.linalg.norm(side, axis=1, keepdims=True)
        more = np.stack([a, b, len(V) + np.arange(len(a))], 1)
        V = np.concatenate([V, V[a] + 0.5 * e + off * side])
    return V.astype(np.float32), np.concatenate([F, more]).astype(np.int32)


@pytest.mark.parametrize("kind,seed,R", [("twice", 2, 49), ("twice", 3, 23), ("twice", 17, 32), ("collinear", 3, 23),
                                         ("collinear", 4, 49), ("points", 5, 32), (1e-6, 6, 32), (1e-4, 7, 49), (1e-2, 8, 32)])
def test_remesh_with_degenerate_faces_matches_restatement(torch_cuda, monkeypatch, kind, seed, R):
    import pamo_b200

    V, F = _mesh(kind, seed)
    v, f, _ = pamo_b200.remesh(pamo_b200.Context(0), torch_cuda.from_numpy(V).cuda(), torch_cuda.from_numpy(F).cuda(), R)
    ov, of, _ = _restated(V, F, R, 3, monkeypatch)
    assert np.array_equal(f.cpu().numpy(), of)
    assert np.array_equal(v.cpu().numpy().view(np.uint32), ov.view(np.uint32))
    if kind == "twice":  # the case is there: two voxels are not enough
        sv, sf, _ = _restated(V, F, R, 2, monkeypatch)
        assert not (np.array_equal(sf, of) and np.array_equal(sv, ov))
