"""Association statistics that leave in chunks of SNPs (page-locked results)
against the same pass in one piece (pageable results), bit for bit, in every
form of the statistics: the thread per SNP (to 4 covariates), the 16-trait and
the 64-trait tiles, with the indicator operand (to 32 columns) and without, designs of
more than 128 columns among them.
The sizes follow the rule for the chunks (whole waves of one 128-row tile per
SM, 8 MB of results at least in each); the number of launches is checked, so
that a change of the rule cannot leave nothing to compare.  SNPs without
variance lie in every chunk: t and beta are exactly 0 there and nowhere else."""
import numpy as np
import pytest

from oracle import lfmm_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,p", [(1, 700_001), (3, 470_000), (5, 300_007), (12, 200_000), (16, 190_123), (17, 150_000),
                                 (40, 100_001), (70, 60_000), (127, 60_000), (140, 60_000), (200, 60_000)])
def test_chunks_equal_one_piece(engine, d, p):
    import schnellfmm_gb300 as sg
    n, k, apart = 96 if d < 90 else 260, 2, 4999
    rng = np.random.default_rng(d)
    codes = rng.choice(np.array([0, 1, 2, 3], dtype=np.uint8), size=(p, n), p=[0.4, 0.02, 0.38, 0.2])
    codes[::apart] = rng.choice(np.array([0, 2, 3], dtype=np.uint8), size=(len(codes[::apart]), 1))
    codes[apart::2 * apart, ::7] = 1            # without variance, and with missing calls
    packed = O.pack_codes(codes)
    x = rng.standard_normal((n, d))
    cfg = sg.Lfmm2Config(k=k, oversampling=6, norm=sg.SnpNorm.EIGENSTRAT)
    shapes = dict(u_hat=(n, k), beta=(p, d), tstat=(p, d), pvalue=(p, d), r2=(p, 3), gif_per_trait=(d,))
    pinned = {m: sg.PinnedArray(s, np.float64) for m, s in shapes.items()}
    launches = []
    try:
        engine.profile(True)
        a = sg.fit_lfmm2_host(packed, n, x, cfg, engine=engine, out={m: v.array for m, v in pinned.items()})
        launches.append(engine.profile_read("assoc_epilogue")["launches"])
        engine.profile(True)
        b = sg.fit_lfmm2_host(packed, n, x, cfg, engine=engine)
        launches.append(engine.profile_read("assoc_epilogue")["launches"])
    finally:
        engine.profile(False)
    assert launches[0] >= 3 and launches[1] == 1, launches
    for m in shapes:
        np.testing.assert_array_equal(getattr(a, m), getattr(b, m))
    flat = np.zeros(p, dtype=bool)
    flat[::apart] = True
    for m in ("tstat", "beta"):
        v = getattr(a, m)
        np.testing.assert_array_equal(v.astype(np.float32).astype(np.float64), v)   # FP32 values, widened
        assert (v[flat] == 0).all() and ((v[~flat] != 0).sum(axis=1) > 0).all()
    del a
    for v in pinned.values():
        v.free()
