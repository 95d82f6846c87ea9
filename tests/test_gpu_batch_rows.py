"""GPU: the batched FP32 cycles' coarsest solve on stored rows.

Boxes whose coarsest levels have 2 nodes in a direction (a node is its own two
neighbours' neighbour), odd counts, exactly and just above the number of
unknowns the stored rows serve (512: 5 x 5 x 6 nodes are 450, 5 x 5 x 7 are
525), cells that are not cubes, both symmetries.  With a single level the
coarsest solve is the whole cycle, so a converged solve shows the rows are the
operator's: every problem reaches 1e-9 by the oracle's residual of the GPU
solution (zero-mean parts; margin 1e-4 of it for the rounding of the two
residuals)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def zero_mean(a, n):
    a = a.reshape(3, n[2] + 1, n[1] + 1, n[0] + 1)[:, :n[2], :n[1], :n[0]]
    return a - a.mean(axis=(1, 2, 3), keepdims=True)


@pytest.mark.parametrize("sym", ["isotropic", "majorminor"])
@pytest.mark.parametrize("boxes,levels", [([(2, 2, 2), (3, 4, 5), (5, 5, 6), (5, 5, 7), (2, 9, 3)], 0),
                                          ([(4, 8, 16), (10, 12, 20), (20, 20, 28), (6, 6, 6)], -1)])
def test_batch_bottom_rows(gpu_lib, sym, boxes, levels):
    from alamo_gb300.batch import Batch
    from alamo_gb300 import microstructure as M
    rng = np.random.default_rng(5)
    bt = Batch(boxes, sym=sym, precision=1, krylov=8, max_coarsening_level=levels)
    C = np.array(M.cubic(1.68, 1.21, 0.75))
    probs = []
    for q, n in enumerate(boxes):
        z, y, x = np.meshgrid(*[np.arange(k + 1) * 2 * np.pi / k for k in n[::-1]], indexing="ij")
        wave = 1.0 + 0.2 * np.cos(x + q) + 0.1 * np.sin(y) * np.cos(z)
        base = np.array([1.2, 0.8]) if sym == "isotropic" else C
        ddw = (wave[..., None] * base).reshape(-1)
        bt.SetModel(q, ddw)
        probs.append((n, ddw, rng.uniform(-0.02, 0.02, (3, 3))))
    bt.SetEigenstrain(np.stack([p[2] for p in probs]))
    assert bt.solve(1e-9, 0.0).status == 0
    for q, (n, ddw, F0) in enumerate(probs):
        g = O.make_grid(list(n), sym=O.ISO if sym == "isotropic" else O.MAJORMINOR, periodic=(1, 1, 1))
        N = O.nodes(g)
        rhs = O.newton_rhs(g, ddw, np.tile(F0.reshape(9), N), np.zeros(3 * N), np.zeros(3 * N))
        mean = rhs.reshape(3, n[2] + 1, n[1] + 1, n[0] + 1)[:, :n[2], :n[1], :n[0]].mean(axis=(1, 2, 3))
        pb = (rhs.reshape(3, -1) - mean[:, None]).reshape(-1)
        r = np.abs(zero_mean(O.residual(g, ddw, bt.solution(q), pb), n)).max()
        scale = np.abs(zero_mean(rhs, n)).max()
        if scale == 0:   # on two cells both neighbours are one node: no gradient, nothing to solve
            assert np.abs(bt.solution(q)).max() < 1e-15
            continue
        assert r <= 1e-9 * scale * 1.0001, (q, n, r, scale)
    bt.close()
