"""The host side of the API under a stand-in CUDA runtime (fake_cudart.cpp,
preloaded): a copy to the device may read its pageable source until the stream
is synchronised, so every source has to be there, unchanged, until then, and no
copy may outlive the call that was given its source.  Freed memory is filled by
the allocator, so a source that went out of scope too early shows as changed."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent

CALLS = r'''
import ctypes as C, sys
import numpy as np
import schnellfmm_gb300 as sg
fake = C.CDLL(sys.argv[1])
fake.fake_launches.argtypes = [C.c_char_p]
rng = np.random.default_rng(3)
n, p, k = 400, 2000, 3
packed = rng.integers(0, 256, size=(p, n // 4), dtype=np.uint8)
cfg = sg.Lfmm2Config(k=k, lambda_=1e-3, oversampling=5, norm=sg.SnpNorm.EIGENSTRAT)
alls = sg.SubsetSpec.all()

def done(what):
    assert fake.fake_changed_sources() == 0, what + ": a copy's source was gone or changed before the copy was over"
    assert fake.fake_pending() == 0, what + ": copies in flight when the call returned"

for d in (1, 120):
    x = rng.standard_normal((n, d))
    with sg.Engine() as eng:
        geno = eng.upload(packed, n); done("upload")
        sub = eng.upload(packed, n, sample_keep=range(0, n, 2)); done("upload of some samples")
        sg.fit_lfmm2(geno, alls, geno, x, cfg, engine=eng); done("fit")
        u = sg.estimate_factors(geno, alls, x, cfg, omega=rng.standard_normal((n, 8)), engine=eng); done("factors")
        sg.test_associations(geno, x, u + rng.standard_normal(u.shape), cfg, engine=eng); done("tests")
        sg.fit_lfmm2_traits(geno, x, rng.random((n, d)) < 0.9, cfg, engine=eng); done("traits")
        sg.fit_lfmm2_many([(packed, n, x, cfg)] * 3, engine=eng); done("many fits")
        nmf = sg.Lfmm2Config(k=k, oversampling=5, impute=sg.ImputeStrategy.NMF, nmf=sg.NmfConfig(k=4, n_iter=2))
        sg.fit_lfmm2(geno, alls, geno, x, nmf, engine=eng); done("fit with NMF")
        sg.fit_lfmm2_host(packed, n, x, cfg, engine=eng); done("fit from the host")
        eng.generate_omega(5, 70_000, 20); done("draw")
        eng.center_covariates(x, True); done("centring")
        eng.small_eigh(x.T @ x); done("eigen-solve")
        geno.free(); sub.free()
    done("close")
assert fake.fake_launches(b"k_jacobi_svd") > 0 and fake.fake_launches(b"k_draw_tails") > 0
assert fake.fake_sources_compared() > 50
print("ran")
'''


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    from schnellfmm_gb300 import build
    build.build()
    include = Path(build.nvcc()).resolve().parent.parent / "include"
    lib = tmp_path_factory.mktemp("fake") / "libfake_cudart.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{include}", str(HERE / "fake_cudart.cpp"),
                    "-o", str(lib)], check=True)
    return lib


def run_with(fake, script, *args):
    # freed memory is filled, and stays mapped
    env = dict(os.environ, LD_PRELOAD=str(fake), MALLOC_PERTURB_="165", MALLOC_MMAP_MAX_="0",
               MALLOC_TRIM_THRESHOLD_=str(1 << 40), PYTHONPATH=str(HERE.parent))
    r = subprocess.run([sys.executable, "-c", script, str(fake), *args], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "ran" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]


def test_sources_outlive_their_copies(fake):
    run_with(fake, CALLS)
