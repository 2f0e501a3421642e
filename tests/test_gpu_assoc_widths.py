"""Fits against the FP64 oracle where the small kernels change form: designs of
1 + d + K columns on both sides of each form of the Cholesky with its inverse
(22, 31, 44, 67, 127 and 236 columns), of the inverses in place (112) and of the
singularity probe (160); traits of the thread-per-SNP statistics (to 4), of the 16-trait tiles
(to 16) and of the 64-trait tiles; and statistics that leave in several chunks."""
import numpy as np
import pytest

from oracle import lfmm_oracle as O
from parity import check_fit
import simdata

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 4, 5, 16, 17, 18, 19, 27, 28, 40, 41, 63, 64, 108, 109, 123, 124, 157, 232, 233])
def test_widths_match_oracle(engine, d):
    import schnellfmm_gb300 as sg
    n, p, k = 900, 1500, 3
    c = simdata.simulate(n, p, k_pop=4, fst=0.08, miss=0.02, d=d, n_causal=25, seed=300 + d)
    cfg = sg.Lfmm2Config(k=k, lambda_=1e-3, oversampling=5, norm=sg.SnpNorm.EIGENSTRAT)
    omega = O.rng_normal_matrix(7, n, k + 5)
    geno = engine.upload(c.packed, n)
    res = sg.fit_lfmm2(geno, sg.SubsetSpec.all(), geno, c.x, cfg, omega=omega, engine=engine)
    ref = O.fit_oracle64(c.raw, c.raw, c.x, k=k, lam=1e-3, oversampling=5, norm=O.NORM_EIGENSTRAT, omega=omega)
    check_fit(res, ref.assoc, ref.u_hat)
    geno.free()


@pytest.mark.parametrize("d", [3, 40])
def test_chunks_equal_one_piece(engine, d):
    """Statistics that leave in chunks (page-locked results) and in one piece."""
    import schnellfmm_gb300 as sg
    n, p, k = 200, 1_000_000 // d, 2
    c = simdata.simulate(n, p, k_pop=3, fst=0.08, miss=0.01, d=d, seed=d)
    cfg = sg.Lfmm2Config(k=k, oversampling=6)
    shapes = dict(u_hat=(n, k), beta=(p, d), tstat=(p, d), pvalue=(p, d), r2=(p, 3), gif_per_trait=(d,))
    pinned = {m: sg.PinnedArray(s, np.float64) for m, s in shapes.items()}
    a = sg.fit_lfmm2_host(c.packed, n, c.x, cfg, engine=engine, out={m: v.array for m, v in pinned.items()})
    b = sg.fit_lfmm2_host(c.packed, n, c.x, cfg, engine=engine)
    for m in shapes:
        np.testing.assert_array_equal(getattr(a, m), getattr(b, m))
    del a
    for v in pinned.values():
        v.free()


@pytest.mark.parametrize("d", [38, 45, 130])
def test_singular_wide_design(engine, capfd, d):
    """A constant covariate: the elimination finds an exactly zero pivot, adds
    eps and starts again, in one CTA (38) and in clusters, and the covariate
    gets t = 0."""
    import schnellfmm_gb300 as sg
    c = simdata.simulate(500, 1200, k_pop=3, fst=0.1, miss=0.01, d=d, n_causal=20, seed=40 + d)
    x = 0.5 * c.x
    x[:, 7] = 2.5
    omega = O.rng_normal_matrix(5, c.n, 13)
    geno = engine.upload(c.packed, c.n)
    capfd.readouterr()
    res = sg.fit_lfmm2(geno, sg.SubsetSpec.all(), geno, x, sg.Lfmm2Config(k=3, norm=sg.SnpNorm.EIGENSTRAT),
                       omega=omega, engine=engine)
    assert "is singular, adding epsilon" in capfd.readouterr().err
    ref = O.fit_oracle64(c.raw, c.raw, x, k=3, norm=O.NORM_EIGENSTRAT, omega=omega)
    check_fit(res, ref.assoc, ref.u_hat)
    assert (res.tstat[:, 7] == 0).all() and (ref.assoc.tstat[:, 7] == 0).all()
    geno.free()
