"""The ChaCha8 sketch draw on the device (k_draw.cu) against the host's
(slfmm_reference_normal), bit for bit: sizes around a block's 1920 outputs and
the carry of draws over block edges (wedge and tail draws fall on an edge in
some of the seeds), the smallest, and one with hundreds of tail draws."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,l,seeds", [(1, 1, 64), (3, 2, 16), (1895, 1, 16), (1919, 1, 16), (1921, 1, 16),
                                       (240, 16, 16), (5003, 20, 4), (60_000, 33, 2)])
def test_draw_equals_host_stream(n, l, seeds):
    import schnellfmm_gb300 as sg
    eng = sg.Engine()
    try:
        for s in range(seeds):
            seed = 7919 * s + n + l
            got = eng.generate_omega(seed, n, l)
            np.testing.assert_array_equal(got.view(np.uint64), sg.reference_normal(seed, n, l).view(np.uint64))
    finally:
        eng.close()
