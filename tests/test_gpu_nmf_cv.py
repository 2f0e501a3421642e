"""The NMF cross-validation kernels (k_nmf_cv, k_nmf_gwas_cv) against the FP64
oracle on the same mask streams, at the sizes where a draw can go to the wrong
call: sample counts off the eight draws of a block and the 256 of a warp's
step, chunks that end inside a block, ranks read as 16-byte vectors and not,
more held-out calls per SNP than a warp lists (512), both streams.  Held-out
count exact, mean-fill errors to 1e-9, the errors of the FP32 fills to 2e-3 as
in test_gpu_nmf."""
import numpy as np
import pytest

from oracle import lfmm_oracle as O
import simdata

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p,k,rate,chunk,rng", [
    (37, 400, 3, 0.05, 7, "chacha8"), (256, 300, 4, 0.01, 300, "chacha8"), (257, 301, 8, 0.1, 100, "chacha8"),
    (1203, 150, 5, 0.6, 64, "chacha8"), (1203, 150, 20, 0.9, 149, "chacha8"), (521, 260, 4, 0.3, 33, "counter"),
])
def test_held_out_calls_equal_the_oracles(n, p, k, rate, chunk, rng):
    import schnellfmm_gb300 as sg
    c = simdata.simulate(n, p, k_pop=3, fst=0.12, miss=0.04, d=1, seed=n + k)
    eng = sg.Engine(rng=sg.SketchRng.CHACHA8 if rng == "chacha8" else sg.SketchRng.COUNTER)
    try:
        cfg = sg.Lfmm2Config(k=2, lambda_=1e-5, oversampling=6, norm=sg.SnpNorm.EIGENSTRAT,
                             impute=sg.ImputeStrategy.NMF, chunk_size=chunk, seed=42,
                             nmf=sg.NmfConfig(k=k, n_iter=2, eps=1e-16, cv_rate=rate))
        geno = eng.upload(c.packed, n)
        res = sg.fit_lfmm2(geno, sg.SubsetSpec.all(), geno, c.x, cfg, engine=eng)
        more = dict(rng="chacha8") if rng == "chacha8" else {}
        ref = O.fit_oracle64(c.raw, c.raw, c.x, k=2, lam=1e-5, oversampling=6, seed=42, norm=O.NORM_EIGENSTRAT,
                             nmf=dict(k=k, n_iter=2, eps=1e-16, cv_rate=rate), chunk=chunk, **more)
        mae, mmae, cnt = ref.gwas_cv
        assert res.nmf_gwas_cv_count == cnt > 0
        assert res.nmf_cv_mean == pytest.approx(ref.nmf.cv_mae_mean_impute, rel=1e-9)
        assert res.nmf_gwas_cv_mean_mae == pytest.approx(mmae, rel=1e-9)
        np.testing.assert_allclose(res.nmf_cv, ref.nmf.cv_mae_per_iter, rtol=2e-3, atol=0)
        assert res.nmf_gwas_cv_mae == pytest.approx(mae, rel=2e-3)
        geno.free()
    finally:
        eng.close()
