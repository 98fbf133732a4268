"""The two forms of the edge cost, a thread per edge above 100,000 faces (50,000 in
quality mode) and a group of eight lanes per edge up to there, give the same bits: a
mesh that crosses the limit against the oracle round by round, meshes packed beyond
it against the same meshes alone, and a quality-mode mesh alone and beside another."""
import numpy as np
import pytest

from helpers import bits, compact, prepare

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def test_rounds_across_the_limit_match_oracle(torch_cuda):
    import pamo_b200
    from oracle import oracle as O
    from pamo_b200 import meshgen as mg

    P, F, scale, _ = prepare(*mg.noisy_torus(232, 232, 5))
    T = O.shuffle_faces(F)
    orc, gpu = O.Stage2Oracle(), pamo_b200.CUDSP_Free()
    dev = lambda x: torch_cuda.from_numpy(np.ascontiguousarray(x)).cuda()
    undo = np.zeros(0, np.int32)
    sizes = []
    for r in range(4):
        sizes.append(len(T))
        op, ot, oo, om, ou = orc.forward(P, T, undo, len(undo), scale, 1e-3, 0)
        g = gpu.forward(dev(P), dev(F if r == 0 else T), dev(undo), len(undo), float(scale), 1e-3, False, r == 0)
        gv, gt, go, gm, gu = [x.cpu().numpy() for x in g]
        assert np.array_equal(bits(gv), bits(op)) and np.array_equal(gt, ot), f"round {r}"
        assert np.array_equal(go, oo) and np.array_equal(gm, om) and np.array_equal(gu, ou), f"round {r}"
        undo = ou
        P, T = compact(op, ot, oo, om)
    assert sizes[1] > 100_000 > sizes[-1], sizes  # two rounds above, and below


def test_packed_meshes_match_the_same_alone(torch_cuda):
    import pamo_b200
    from pamo_b200 import meshgen as mg
    from pamo_b200.batch import simplify_many

    meshes = [mg.noisy_torus(n, n, n) for n in (150, 152, 154)]
    meshes = [(V.astype(np.float32), F.astype(np.int32)) for V, F in meshes]
    sizes = [len(F) for _, F in meshes]
    assert max(sizes) < 50_000 and sum(sizes) > 130_000
    got = simplify_many(meshes, ratio=0.6, min_verts=0)
    for (V, F), (v, f) in zip(meshes, got):
        ctx = pamo_b200.Context(0)
        wv, wf, _ = pamo_b200.stage2_run(ctx, torch_cuda.from_numpy(V).cuda(), torch_cuda.from_numpy(F).cuda(),
                                         int(0.6 * len(F)))
        assert np.array_equal(f, wf.cpu().numpy())
        assert np.array_equal(bits(v), bits(wv.cpu().numpy()))


def test_quality_mesh_alone_and_beside_another(torch_cuda):
    """Faces keep their order, so the first mesh's edges keep their numbers and, as the
    meshes are apart, its rounds do not depend on the second one."""
    import pamo_b200
    from pamo_b200 import _lib
    from pamo_b200 import meshgen as mg

    V, F = mg.noisy_torus(150, 150, 7)
    W, G = mg.noisy_torus(152, 152, 8)
    scale = 2.7
    V, F = V.astype(np.float32), F.astype(np.int32)
    both = np.concatenate([V, (W + 5).astype(np.float32)]), np.concatenate([F, (G + len(V)).astype(np.int32)])
    assert len(F) < 50_000 and len(both[1]) > 85_000

    def rounds(P, T):
        gpu = pamo_b200.CUDSP_Free()
        assert _lib.lib().pamo_set_quality(gpu.ctx.handle, 1) == 0
        dev = lambda x: torch_cuda.from_numpy(np.ascontiguousarray(x)).cuda()
        none = dev(np.zeros(0, np.int32))
        out = []
        for _ in range(3):
            size = len(T)
            r = [x.cpu().numpy() for x in gpu.forward(dev(P), dev(T), none, 0, scale, 1e-3, False, False)]
            out.append((size, r))
            P, T = compact(*r[:4])
        return out

    n, m = len(V), len(F)
    for (size, a), (size2, b) in zip(rounds(V, F), rounds(*both)):
        assert size < 50_000 < size2
        gone = (a[2] == 0).sum()
        assert gone > 500
        assert np.array_equal(bits(a[0]), bits(b[0][:n])) and np.array_equal(a[1], b[1][:m])
        assert np.array_equal(a[2], b[2][:n]) and np.array_equal(a[3], b[3][:n])
        n -= int(gone)
        m = int((a[1][:, 0] >= 0).sum())
