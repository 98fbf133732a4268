"""The remesh where its words of 32 samples, its 8-row tiles and the two-voxel
reach can go wrong: resolutions about a word's end, the smallest grids, surfaces
with thin gaps (free samples enclosed, cells with several patches) and large
triangles, equal to the CPU restatement bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _soup(seed, n):
    """Random triangles of all sizes, crossing each other."""
    rng = np.random.default_rng(seed)
    c = rng.random((n, 1, 3))
    V = (c + rng.normal(size=(n, 3, 3)) * 10.0 ** rng.uniform(-2.5, -0.5, (n, 1, 1))).reshape(-1, 3)
    return V.astype(np.float32), np.arange(3 * n, dtype=np.int32).reshape(-1, 3)


def _shape(kind, R):
    from pamo_b200 import meshgen as mg

    if kind == "sphere":
        return mg.displaced_icosphere(2, R)
    if kind == "shell":
        return mg.thin_shell_pair(2000, 2.5 / R, R)
    return _soup(R, 60)


@pytest.mark.parametrize("R", [8, 15, 16, 17, 31, 32, 33, 63, 65])
@pytest.mark.parametrize("kind", ["sphere", "shell", "soup"])
def test_remesh_matches_oracle_about_word_and_tile_ends(torch_cuda, kind, R):
    import pamo_b200
    from oracle import s1_oracle as S1

    V, F = _shape(kind, R)
    ctx = pamo_b200.Context(0)
    v, f, _ = pamo_b200.remesh(ctx, torch_cuda.from_numpy(V).cuda(), torch_cuda.from_numpy(F).cuda(), R)
    ov, of, _ = S1.remesh(V, F, R)
    v, f = v.cpu().numpy(), f.cpu().numpy()
    assert np.array_equal(f, of)
    assert np.array_equal(v.view(np.uint32), ov.view(np.uint32))
