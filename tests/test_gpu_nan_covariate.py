"""A covariate with a value that is not finite, in one CTA's and a cluster's
elimination (to 40 columns and above), in the LU's solves (above 112) and in
the status-only eliminations: X^T X is NaN, which is no zero pivot.  As in
the reference, whose inversions pass NaN on and whose t_test returns 0 for
what is not finite (src/testing.rs:1036-1048), the call succeeds: U_hat is
that of a fit without covariates to project out, every t is 0 and every beta
that a NaN reaches is NaN."""
import numpy as np
import pytest

from oracle import lfmm_oracle as O
import simdata

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("d,j", [(1, 0), (3, 1), (20, 7), (40, 39), (45, 7), (113, 0), (120, 100),
                                 (200, 3)])
def test_not_finite_covariate(engine, capfd, d, j, bad):
    import schnellfmm_gb300 as sg
    c = simdata.simulate(400, 1500, k_pop=3, fst=0.1, miss=0.01, d=d, n_causal=10, seed=d)
    x = c.x.copy()
    x[5, j] = bad
    omega = O.rng_normal_matrix(9, c.n, 13)
    cfg = sg.Lfmm2Config(k=3, norm=sg.SnpNorm.EIGENSTRAT)
    geno = engine.upload(c.packed, c.n)
    capfd.readouterr()
    res = sg.fit_lfmm2(geno, sg.SubsetSpec.all(), geno, x, cfg, omega=omega, engine=engine)
    assert "singular" not in capfd.readouterr().err
    none = O.fit_oracle64(c.raw, c.raw, c.x[:, :1], k=3, lam=1e30, norm=O.NORM_EIGENSTRAT, omega=omega)
    assert O.principal_angles_sin_max(res.u_hat, none.u_hat) < 1e-3
    assert (res.tstat == 0).all()
    assert np.isnan(res.beta[res.beta != 0]).all()
    assert np.isfinite(res.pvalue).all()
    # the same context on the covariates without it
    good = sg.fit_lfmm2(geno, sg.SubsetSpec.all(), geno, c.x, cfg, omega=omega, engine=engine)
    assert np.isfinite(good.beta).all() and np.abs(good.tstat).max() > 1
    geno.free()


def test_nothing_left_to_invert(engine):
    """NaN from the first column on is refused (to 112 columns: the LU of wider
    matrices passes it on): the factors of a sketch that broke down are NaN
    altogether, and a fit on them has no tests to give."""
    import schnellfmm_gb300 as sg
    rng = np.random.default_rng(4)
    c = simdata.simulate(300, 1500, k_pop=3, fst=0.1, miss=0.01, d=45, n_causal=10, seed=4)
    geno = engine.upload(c.packed, c.n)
    for d in (2, 20, 45):
        x = c.x[:, :d].copy()
        x[5, 0] = np.nan
        with pytest.raises(sg.SchnelGpuError, match=r"X\^T X \+ .* inversion failed") as e:
            sg.fit_lfmm2(geno, sg.SubsetSpec.all(), geno, x, sg.Lfmm2Config(k=3), engine=engine)
        assert e.value.code == sg.ERR_SINGULAR
    for k in (2, 16, 41):
        u = rng.standard_normal((c.n, k))
        u[7] = np.nan
        with pytest.raises(sg.SchnelGpuError, match=r"U_hat\^T U_hat inversion failed") as e:
            sg.test_associations(geno, c.x[:, :2], u, sg.Lfmm2Config(k=k), engine=engine)
        assert e.value.code == sg.ERR_SINGULAR
        u[7, 0] = 1.0
        res = sg.test_associations(geno, c.x[:, :2], u, sg.Lfmm2Config(k=k), engine=engine)
        assert (res.tstat == 0).all() and np.isnan(res.beta[res.beta != 0]).all()
    geno.free()
