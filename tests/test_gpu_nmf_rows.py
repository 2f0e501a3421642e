"""The NMF corrections with fill rows read 4, 16 and 32 bytes at a time (ranks off,
on 4 and on 8), rank bounds 16 and 32 and sketches of 8, 16, 32 and more columns,
against the FP64 oracle.  Bounds as in test_gpu_nmf."""
import numpy as np
import pytest

from oracle import lfmm_oracle as O
from test_gpu_nmf import _cohort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,over", [(3, 3), (4, 10), (8, 4), (8, 20), (16, 10), (24, 30)])
def test_nmf_rank_and_width(engine, k, over):
    import schnellfmm_gb300 as sg
    raw, packed, x = _cohort()
    n = raw.shape[0]
    it, rate, chunk, seed = 3, 0.01, 1000, 42
    cfg = sg.Lfmm2Config(k=3, lambda_=1e-5, oversampling=over, norm=sg.SnpNorm.EIGENSTRAT,
                         impute=sg.ImputeStrategy.NMF, chunk_size=chunk, seed=seed,
                         nmf=sg.NmfConfig(k=k, n_iter=it, eps=1e-16, cv_rate=rate))
    omega = O.rng_normal_matrix(9, n, 3 + over)
    geno = engine.upload(packed, n)
    res = sg.fit_lfmm2(geno, sg.SubsetSpec.all(), geno, x, cfg, omega=omega, engine=engine)
    ref = O.fit_oracle64(raw, raw, x, k=3, lam=1e-5, oversampling=over, seed=seed, norm=O.NORM_EIGENSTRAT,
                         omega=omega, nmf=dict(k=k, n_iter=it, eps=1e-16, cv_rate=rate), chunk=chunk)
    np.testing.assert_allclose(res.nmf_cv, ref.nmf.cv_mae_per_iter, rtol=2e-3, atol=0)
    assert O.principal_angles_sin_max(res.u_hat, ref.u_hat) < 2e-3
    dt = np.abs(res.tstat - ref.assoc.tstat).max()
    assert dt <= 1e-3, f"max|dt| = {dt}"
    geno.free()
