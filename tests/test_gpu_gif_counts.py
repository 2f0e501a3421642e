"""The median of the t^2 histogram (k_gif) over more values than 32 bits
count, all in one group of 128 bins that the kernel sums first."""
import ctypes as C

import numpy as np
import pytest

from oracle import lfmm_oracle as O

pytestmark = pytest.mark.gpu


def test_more_than_32_bits_of_values():
    torch = pytest.importorskip("torch")
    import schnellfmm_gb300 as sg
    first, nbins = 390, 64                 # bins 384 .. 511 are one group
    each = 2**26 + 1000                    # values per bin: 2**32 + 64 000 in all, 17 GB
    eng = sg.Engine()
    try:
        # bin centres in t^2; a warp's values fall into bins side by side
        centres = (np.arange(first, first + nbins) + 0.5) * 0.001
        t = torch.tensor(np.sqrt(centres).astype(np.float32), device="cuda").repeat(each)
        out = torch.full((1,), -1.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        eng.check(eng.lib.slfmm_gif_noalloc(eng.h, C.c_void_p(t.data_ptr()), t.numel(), 1,
                                            C.c_void_p(out.data_ptr())))
        torch.cuda.synchronize()
        # an even count, half of it in the bins up to the middle one
        median = (centres[nbins // 2 - 1] + centres[nbins // 2]) / 2
        assert out.item() == pytest.approx(median / O.GIF_DIVISOR, rel=1e-12)
    finally:
        eng.close()
        t = None
        torch.cuda.empty_cache()
