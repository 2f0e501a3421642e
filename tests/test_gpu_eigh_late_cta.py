"""The clustered eigen-solve (k_jacobi_svd above 32 columns) with one of its
eight CTAs late to every round: the angles are formed from elements in other
CTAs' shared memory, which those rotate in the same round, so the late CTA
reads rotated ones unless every read is ordered before the first write.  The
result must not depend on the CTAs' pace: the same bits as without."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [33, 34, 57, 100, 115, 256])
def test_late_cta_changes_nothing(engine, m):
    import schnellfmm_gb300 as sg
    rng = np.random.default_rng(m)
    x = rng.standard_normal((3 * m, m)) * rng.uniform(0.1, 10, m)
    a = x.T @ x
    sig, v = engine.small_eigh(a)
    for cycles in (3_000, 20_000):   # about an angle's five divisions and square roots, and well past them
        engine.check(engine.lib.slfmm_debug_hold_next_solve(engine.h, cycles))
        late_sig, late_v = engine.small_eigh(a)
        np.testing.assert_array_equal(late_sig, sig)
        np.testing.assert_array_equal(late_v, v)
    assert engine.lib.slfmm_debug_hold_next_solve(engine.h, 0) == sg.ERR_BAD_ARG
    assert engine.lib.slfmm_debug_hold_next_solve(engine.h, 1_000_001) == sg.ERR_BAD_ARG
