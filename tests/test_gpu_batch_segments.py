"""GPU: the batched solve's elementwise and reducing kernels work on runs of
consecutive elements of one component: boxes whose nodes are no multiple of a
run or of a vector (padded rows), boxes of more than one run, and a box with
nothing to solve beside others that go on.  Every problem reaches its tolerance
by the oracle's residual of the GPU solution (zero-mean parts: the boxes are
singular), with a margin of 1e-4 of it for the rounding of the two residuals,
and the displacement is zero-mean to rounding."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,krylov,fmg", [(0, 0, 0), (1, 0, 0), (1, 8, 0), (1, 8, 4)])
def test_batch_segments(gpu_lib, precision, krylov, fmg):
    from alamo_gb300.batch import Batch
    boxes = [(6, 10, 14), (20, 12, 8), (36, 28, 20), (4, 4, 4)]
    rng = np.random.default_rng(11)
    bt = Batch(boxes, precision=precision, krylov=krylov, max_fmg_iter=fmg)
    probs = []
    for q, n in enumerate(boxes):
        z, y, x = np.meshgrid(*[np.arange(k + 1) * 2 * np.pi / k for k in n[::-1]], indexing="ij")
        wave = np.cos(x + q) * np.cos(y) * np.cos(z)
        ddw = np.stack([1.2 + 0.3 * wave, 0.8 + 0.2 * wave], axis=-1).reshape(-1)
        F0 = rng.uniform(-0.02, 0.02, (3, 3)) if q != 3 else np.zeros((3, 3))   # box 3: nothing to solve
        bt.SetModel(q, ddw)
        probs.append((n, ddw, F0))
    bt.SetEigenstrain(np.stack([p[2] for p in probs]))
    assert bt.solve(1e-9, 0.0).status == 0
    for q, (n, ddw, F0) in enumerate(probs):
        g = O.make_grid(list(n), sym=O.ISO, periodic=(1, 1, 1))
        N = O.nodes(g)
        rhs = O.newton_rhs(g, ddw, np.tile(F0.reshape(9), N), np.zeros(3 * N), np.zeros(3 * N))
        u = bt.solution(q)
        assert np.all(np.isfinite(u))

        def stored(a):
            return a.reshape(3, n[2] + 1, n[1] + 1, n[0] + 1)[:, :n[2], :n[1], :n[0]]

        def zero_mean(a):
            a = stored(a)
            return a - a.mean(axis=(1, 2, 3), keepdims=True)
        pb = (rhs.reshape(3, -1) - stored(rhs).mean(axis=(1, 2, 3))[:, None]).reshape(-1)
        r = np.abs(zero_mean(O.residual(g, ddw, u, pb))).max()
        scale = np.abs(zero_mean(rhs)).max()
        assert r <= 1e-9 * scale * 1.0001, (q, r, scale)
        assert np.abs(stored(u).mean(axis=(1, 2, 3))).max() <= 1e-12 * np.abs(u).max()
    bt.close()
