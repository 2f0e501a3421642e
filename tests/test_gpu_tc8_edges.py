"""The split-FP8 contraction and its operand terms at the edges of their tiles:
rows around 128 (a tile), K around 256 (a stage) and around 16 (a chunk of
terms), widths around the 16-column blocks, the widths of one and of two
accumulator copies, with and without the indicator.  Bounds as in test_gpu_tc."""
import numpy as np
import pytest

import simdata
from test_gpu_tc import _check, exact_g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p,w", [(5, 9, 1), (15, 127, 7), (17, 128, 15), (127, 129, 16), (129, 16, 17),
                                   (255, 257, 31), (256, 256, 33), (257, 255, 48), (511, 385, 64), (513, 300, 65),
                                   (1025, 140, 100), (300, 1100, 128)])
@pytest.mark.parametrize("transposed", [False, True])
def test_edges(engine, n, p, w, transposed):
    c = simdata.simulate(n, p, miss=0.04, seed=n + p + w)
    geno = engine.upload(c.packed, n)
    K = p if transposed else n
    W = np.random.default_rng(w).normal(size=(K, w))
    g = exact_g(c) if transposed else exact_g(c).T
    _check(geno.contract_raw(W, transposed=transposed), g, W, "fp8")
    if w <= 32:
        gm = g + (np.isnan(c.raw) if transposed else np.isnan(c.raw).T)
        _check(geno.contract_raw(W, transposed=transposed, missing_as_one=True), gm, W, "fp8")
    geno.free()
