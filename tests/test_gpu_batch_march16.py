"""GPU: the marching sweep of periodic isotropic batches in both tile shapes
(32 x 8 and 16 x 16 columns, 16 planes a chunk) forced on every level: boxes
smaller than a tile, one more than a tile or a chunk, one node short of it,
cells that are not cubes.  Every problem reaches 1e-9 by the oracle's residual
of the GPU solution (zero-mean parts: the boxes are singular; margin 1e-4 of it
for the rounding of the two residuals)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [5, 6])
@pytest.mark.parametrize("precision,krylov,fmg", [(0, 0, 0), (1, 0, 0), (1, 8, 4)])
def test_batch_march_shapes(gpu_lib, monkeypatch, shape, precision, krylov, fmg):
    from alamo_gb300.batch import Batch
    monkeypatch.setenv("AGB_BATCH_SHAPE", str(shape))
    boxes = [(34, 18, 14), (16, 16, 18), (30, 34, 16), (6, 10, 4)]
    rng = np.random.default_rng(17)
    bt = Batch(boxes, precision=precision, krylov=krylov, max_fmg_iter=fmg)
    probs = []
    for q, n in enumerate(boxes):
        z, y, x = np.meshgrid(*[np.arange(k + 1) * 2 * np.pi / k for k in n[::-1]], indexing="ij")
        ddw = np.stack([1.2 + 0.3 * np.cos(x + q) * np.sin(z), 0.8 + 0.2 * np.cos(y) * np.cos(x + z)], axis=-1)
        bt.SetModel(q, ddw.reshape(-1))
        probs.append((n, ddw.reshape(-1), rng.uniform(-0.02, 0.02, (3, 3))))
    bt.SetEigenstrain(np.stack([p[2] for p in probs]))
    assert bt.solve(1e-9, 0.0).status == 0
    for q, (n, ddw, F0) in enumerate(probs):
        g = O.make_grid(list(n), sym=O.ISO, periodic=(1, 1, 1))
        N = O.nodes(g)
        rhs = O.newton_rhs(g, ddw, np.tile(F0.reshape(9), N), np.zeros(3 * N), np.zeros(3 * N))

        def stored(a):
            return a.reshape(3, n[2] + 1, n[1] + 1, n[0] + 1)[:, :n[2], :n[1], :n[0]]

        def zero_mean(a):
            a = stored(a)
            return a - a.mean(axis=(1, 2, 3), keepdims=True)
        pb = (rhs.reshape(3, -1) - stored(rhs).mean(axis=(1, 2, 3))[:, None]).reshape(-1)
        r = np.abs(zero_mean(O.residual(g, ddw, bt.solution(q), pb))).max()
        scale = np.abs(zero_mean(rhs)).max()
        assert r <= 1e-9 * scale * 1.0001, (q, r, scale)
    bt.close()
