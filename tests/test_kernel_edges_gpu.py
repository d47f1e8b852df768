"""The force kernels at the sizes where their tiles, ranges and queues can go
wrong, against the FP64 oracle.  Tolerances: the per-particle bounds of the
other parity tests (acceleration and potential 1e-6, jerk 1e-5 relative), which
the FP32 pair math on hi/lo differences with double-single sums meets at any
size; neighbour lists identical."""
import ctypes as C

import numpy as np
import pytest

from parity import rel_err_vec

pytestmark = pytest.mark.gpu


# tile of 128 bodies, i-tile of 128 (256 once ni >= 4736), order from 1e9 pairs
@pytest.mark.parametrize("n,i0,ni", [(127, 0, 127), (257, 129, 128), (4736, 0, 4736), (5001, 265, 4735),
                                     (33000, 0, 30304), (33000, 2696, 30304), (40007, 14997, 25010),
                                     (65537, 65537 - 15361, 15361), (40960, 0, 40960)])
def test_potential_ranges(nb6, orc, n, i0, ni):
    """Ranges of the set on both sides of the rule that orders it, at its
    start, inside and at its end, whole and ragged tiles."""
    from nb6b200 import ics
    cl = ics.plummer(n, seed=n + i0, imf=True)
    x = cl.pos.copy()
    x[i0] = x[(i0 + 1) % n]                       # a coincident pair
    p = nb6.gpupot(cl.mass, x, istart=i0 + 1, ni=ni)
    sel = np.unique(np.concatenate([[0, ni - 1], np.random.default_rng(n).integers(0, ni, 300)]))
    po = np.array([orc.pot(cl.mass, x, i0 + 1 + int(k), 1)[0] for k in sel])
    assert np.all(p > 0)
    assert rel_err_vec(p[sel], po).max() <= 1e-6


# 32 samples per CTA and round; 296 CTAs, so a second round from 9,473 samples
@pytest.mark.parametrize("n", [31, 32, 33, 1000, 9472, 9473, 20011])
def test_mlp_gradient_sample_counts(n):
    """The gradient's sample streams at full and ragged rounds against the
    FP64 oracle: within 2e-5 of its norm (FP32 sums over the batch)."""
    import mlp_oracle as M
    from nb6b200 import mlp
    rng = np.random.default_rng(n)
    model = np.zeros(M.NPARAM + M.NNORM, dtype=np.float32)
    model[:M.NPARAM] = rng.normal(size=M.NPARAM) * 0.15
    model[M.NPARAM + M.IN:M.NPARAM + 2 * M.IN] = 1.0
    model[-1] = 0.5
    mlp.set_model(model)
    x = rng.normal(size=(n, 5)).astype(np.float32)
    y = rng.normal(size=n).astype(np.float32)
    g, loss = mlp.grad(x, y)
    gr, lr = M.grad(model, x, y)
    assert abs(loss - lr) <= 1e-5 * lr
    assert np.linalg.norm(g - gr) <= 2e-5 * np.linalg.norm(gr)
