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


REFUSED = r'''
import ctypes as C, mmap, sys
import numpy as np
import schnellfmm_gb300 as sg
fake = C.CDLL(sys.argv[1])
libc = C.CDLL(None, use_errno=True)
rng = np.random.default_rng(3)
p, size = 4000, 64 << 20

def attempt(what, d, want, n=400, fit=True, tests=True, **cfg):
    packed = rng.integers(0, 256, size=(p, n // 4), dtype=np.uint8)
    args = dict(k=3, lambda_=1e-3, oversampling=5)
    args.update(cfg)
    c = sg.Lfmm2Config(**args)._c()
    x, u = rng.standard_normal((n, max(d, 1))), rng.standard_normal((n, args["k"]))
    g = eng.upload(packed, n)
    calls = []
    if fit:
        calls.append(lambda r: eng.lib.slfmm_fit(eng.h, g.h, g.h, x.ctypes.data, d, C.byref(c), None, C.byref(r)))
        calls.append(lambda r: eng.lib.slfmm_fit_host(eng.h, packed.ctypes.data, n, p, None, 0, None, x.ctypes.data, d,
                                                      C.byref(c), None, C.byref(r)))
    if tests:
        calls.append(lambda r: eng.lib.slfmm_test_associations(eng.h, g.h, x.ctypes.data, d, u.ctypes.data, C.byref(c),
                                                               C.byref(r)))
    for i, call in enumerate(calls):
        r, maps = sg._Results(), []
        for f in ("beta", "tstat", "pvalue", "r2"):
            m = mmap.mmap(-1, size, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
            buf = (C.c_char * size).from_buffer(m)
            setattr(r, f, C.cast(buf, C.POINTER(C.c_double)))
            maps.append((f, m, buf))
        rc = call(r)
        assert rc == want, f"{what}, call {i}: {rc}"
        assert fake.fake_pending() == 0, f"{what}, call {i}: copies in flight when the call returned"
        assert fake.fake_changed_sources() == 0, f"{what}, call {i}: a source was gone before its copy was over"
        for f, m, buf in maps:
            there = (C.c_ubyte * (size // mmap.PAGESIZE))()
            assert libc.mincore(C.c_void_p(C.addressof(buf)), C.c_size_t(size), there) == 0
            touched = sum(b & 1 for b in there)
            assert touched == 0 or rc == 0, f"{what}, call {i}: {touched} pages of {f} touched"
    g.free()

with sg.Engine() as eng:
    attempt("accepted", 60, sg.OK)
    attempt("too many covariates", 257, sg.ERR_BAD_ARG)
    attempt("too wide a design", 253, sg.ERR_BAD_ARG)
    attempt("no degrees of freedom", 238, sg.ERR_DF_NONPOSITIVE, n=240)
    attempt("no penalty", 60, sg.ERR_BAD_ARG, lambda_=0.0)
    attempt("too wide a sketch", 60, sg.ERR_BAD_ARG, tests=False, k=30, oversampling=35)
    attempt("no covariates", 0, sg.ERR_BAD_ARG)
    attempt("NMF rank", 60, sg.ERR_BAD_ARG, tests=False, impute=sg.ImputeStrategy.NMF, nmf=sg.NmfConfig(k=33, n_iter=2))
print("ran")
'''


def test_refused_calls_leave_the_results_alone(fake):
    """Result arrays that the process has not touched are made present while a
    call runs: not by a call that is refused, whose arrays may be smaller than
    its d says."""
    run_with(fake, REFUSED)


SCARCE = r'''
import ctypes as C, sys
import numpy as np
import schnellfmm_gb300 as sg
fake = C.CDLL(sys.argv[1])
rng = np.random.default_rng(3)
n, p, d = 400, 2000, 2
packed = rng.integers(0, 256, size=(p, n // 4), dtype=np.uint8)
x, u, mask = rng.standard_normal((n, d)), rng.standard_normal((n, 3)), rng.random((n, d)) < 0.9
cfg, alls = sg.Lfmm2Config(k=3, oversampling=5), sg.SubsetSpec.all()
calls = {
    "fit": lambda: sg.fit_lfmm2(geno, alls, geno, x, cfg, engine=eng),
    "fit from the host": lambda: sg.fit_lfmm2_host(packed, n, x, cfg, engine=eng),
    "tests": lambda: sg.test_associations(geno, x, u, cfg, engine=eng),
    "traits": lambda: sg.fit_lfmm2_traits(geno, x, mask, cfg, engine=eng),
    "many fits": lambda: sg.fit_lfmm2_many([(packed, n, x, cfg)], engine=eng, n_streams=1),
    "draw": lambda: eng.generate_omega(3, 10_000, 3),
}
with sg.Engine() as eng:
    for name, call in calls.items():
        geno = eng.upload(packed, n)
        fake.fake_fail_allocation(0)
        call()
        count = fake.fake_allocations()
        refused = 0
        for k in range(1, count + 1):
            fake.fake_fail_allocation(k)
            try:
                call()
            except sg.SchnelGpuError as e:
                assert e.code == sg.ERR_NOMEM, f"{name}, allocation {k}: {e}"
                refused += 1
            fake.fake_fail_allocation(0)
            assert fake.fake_pending() == 0, f"{name}, allocation {k}: copies in flight when the call returned"
            assert fake.fake_changed_sources() == 0, f"{name}, allocation {k}: a source was gone before its copy"
            call()   # the context goes on
        # the sketch's scratch is done without
        assert refused >= count - 8 and refused > 0, (name, refused, count)
        geno.free()
print("ran")
'''


def test_every_allocation_may_fail(fake):
    """A call that runs out of device memory, at any of its allocations, says so
    and leaves neither copies in flight nor an error behind."""
    run_with(fake, SCARCE)
