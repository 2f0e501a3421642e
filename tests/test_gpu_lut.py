"""The FP32 contractions (k_row_lut, k_col_lut) through fits against the FP64
oracle: sample counts around a stage (128), SNP counts around a block (64, 128)
and a split's stage (32, 64), both forms of the row pass, operands of one, two
and nine blocks of 16 columns.  Bounds as in test_gpu_fit."""
import numpy as np
import pytest

from oracle import lfmm_oracle as O
from parity import check_fit
import simdata

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p,d", [(127, 1023, 1), (128, 1024, 2), (129, 1057, 3), (257, 1000, 20), (520, 641, 100),
                                   (200, 40_001, 2), (150, 12_000, 30)])
def test_fp32_fit_matches_oracle(engines, n, p, d):
    import schnellfmm_gb300 as sg
    eng = engines["fp32"]
    c = simdata.simulate(n, p, k_pop=4, fst=0.1, miss=0.02, d=d, n_causal=20, seed=n + p + d)
    cfg = sg.Lfmm2Config(k=3, lambda_=1e-3, oversampling=5, norm=sg.SnpNorm.EIGENSTRAT)
    omega = O.rng_normal_matrix(7, n, 8)
    geno = eng.upload(c.packed, n)
    res = sg.fit_lfmm2(geno, sg.SubsetSpec.all(), geno, c.x, cfg, omega=omega, engine=eng)
    ref = O.fit_oracle64(c.raw, c.raw, c.x, k=3, lam=1e-3, oversampling=5, norm=O.NORM_EIGENSTRAT, omega=omega)
    check_fit(res, ref.assoc, ref.u_hat)
    geno.free()
