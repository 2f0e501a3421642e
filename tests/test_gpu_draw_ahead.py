"""The sketch that a fit draws ahead of Step 0 on the device (k_draw.cu), against
the host's draw injected as omega: sizes around a block's 1920 outputs and
around the 4096 values up to which a draw that nobody started ahead is the
host's, bit for bit.  And draws around that line made at once."""
import numpy as np
import pytest

import simdata

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,l", [(137, 14), (240, 8), (113, 17), (273, 15), (256, 16), (241, 17), (700, 12)])
def test_drawn_ahead_equals_injected(n, l):
    import schnellfmm_gb300 as sg
    c = simdata.simulate(n, 600, k_pop=3, fst=0.1, miss=0.01, d=2, n_causal=10, seed=n)
    eng = sg.Engine()
    try:
        geno = eng.upload(c.packed, n)
        for seed in range(6):
            cfg = sg.Lfmm2Config(k=3, oversampling=l - 3, seed=seed)
            drawn = sg.estimate_factors(geno, sg.SubsetSpec.all(), c.x, cfg, engine=eng)
            given = sg.estimate_factors(geno, sg.SubsetSpec.all(), c.x, cfg, omega=sg.reference_normal(seed, n, l),
                                        engine=eng)
            np.testing.assert_array_equal(drawn.view(np.uint64), given.view(np.uint64))
        geno.free()
    finally:
        eng.close()


@pytest.mark.parametrize("count", [4095, 4096, 4097, 5759, 5761])
def test_at_once(count):
    import schnellfmm_gb300 as sg
    eng = sg.Engine()
    try:
        for seed in range(8):
            got = eng.generate_omega(seed, count, 1)
            np.testing.assert_array_equal(got.view(np.uint64), sg.reference_normal(seed, count, 1).view(np.uint64))
    finally:
        eng.close()
