"""The remesh's flood on a grid it needs thousands of launches for: a corridor one
sample wide that winds through the whole grid, so that the outside reaches its end
one tile crossing at a time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R = 64


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _maze():
    """Walls through the samples of even x and of even z, given in sample numbers.  In
    each layer the corridors run along y and join at alternating ends; layers join at
    alternating corners, and the first is open to the outside."""
    scale = R * R / (R + 6)  # samples across the mesh's extent, which starts at sample `lo`
    lo = 3 * R / (R + 6) - 0.5
    hi = lo + scale
    V, F = [], []

    def wall(axis, at, u0, u1, v0, v1):
        p = np.array([[u0, v0], [u1, v0], [u1, v1], [u0, v1]])
        q = np.insert(p, axis, at, axis=1)
        n = len(V) * 4
        V.append(q)
        F.extend([(n, n + 1, n + 2), (n, n + 2, n + 3)])

    def floor(at, corner):
        """A wall across z, open over the samples about (3, 3) (corner 0) or (59, 60) (corner 1)."""
        if corner == 0:
            wall(2, at, 4, hi, lo, hi)
            wall(2, at, lo, 4, 4, hi)
        else:
            wall(2, at, lo, 58, lo, hi)
            wall(2, at, 58, hi, lo, 59)

    wall(0, lo, lo, hi, lo, hi)
    wall(0, hi, lo, hi, lo, hi)
    wall(1, lo, lo, hi, lo, hi)
    wall(1, hi, lo, hi, lo, hi)
    wall(2, hi, lo, hi, lo, hi)
    floor(lo, 0)
    for j in range(28):
        wall(0, 4 + 2 * j, *((lo, 59) if j % 2 == 0 else (4, hi)), lo, hi)
        floor(4 + 2 * j, 1 if j % 2 == 0 else 0)
    wall(0, 60, lo, hi, lo, hi)
    wall(2, 60, lo, hi, lo, hi)
    return (np.concatenate(V) - lo).astype(np.float32), np.array(F, np.int32)


def test_flood_follows_a_path_through_the_whole_grid(torch_cuda):
    import pamo_b200
    from oracle import s1_oracle as S1

    V, F = _maze()
    ctx = pamo_b200.Context(0)
    v, f, _ = pamo_b200.remesh(ctx, torch_cuda.from_numpy(V).cuda(), torch_cuda.from_numpy(F).cuda(), R)
    ov, of, _ = S1.remesh(V, F, R)
    assert len(of) > 100_000  # the corridors are outside: their walls have surface on both sides
    assert np.array_equal(f.cpu().numpy(), of)
    assert np.array_equal(v.cpu().numpy().view(np.uint32), ov.view(np.uint32))
