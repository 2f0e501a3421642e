"""The missing-call corrections over lists of every length class -- none, part of
a batch of 32, whole batches, batches and a rest -- and sketches of one and two
columns per lane (k_colfix_mean, k_rowfix_mean4), through BF16 fits against the
FP64 oracle.  Bounds as in test_gpu_fit."""
import numpy as np
import pytest

from oracle import lfmm_oracle as O
from parity import check_fit
import simdata

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p,miss,k,over", [(300, 900, 0.0, 3, 5), (300, 900, 0.01, 3, 5), (321, 1100, 0.1, 4, 28),
                                             (321, 1100, 0.1, 4, 29), (640, 2500, 0.2, 6, 34), (500, 3000, 0.03, 4, 60)])
def test_bf16_fit_matches_oracle(engines, n, p, miss, k, over):
    import schnellfmm_gb300 as sg
    eng = engines["bf16"]
    c = simdata.simulate(n, p, k_pop=k + 1, fst=0.1, miss=miss, d=2, n_causal=20, seed=n + p + over)
    raw = c.raw
    cfg = sg.Lfmm2Config(k=k, lambda_=1e-3, oversampling=over, norm=sg.SnpNorm.EIGENSTRAT)
    omega = O.rng_normal_matrix(7, n, k + over)
    geno = eng.upload(c.packed, n)
    res = sg.fit_lfmm2(geno, sg.SubsetSpec.all(), geno, c.x, cfg, omega=omega, engine=eng)
    ref = O.fit_oracle64(raw, raw, c.x, k=k, lam=1e-3, oversampling=over, norm=O.NORM_EIGENSTRAT, omega=omega)
    check_fit(res, ref.assoc, ref.u_hat)
    geno.free()
