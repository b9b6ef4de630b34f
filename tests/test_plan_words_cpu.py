"""The allocation-free row plan serves every problem whose histogram per 256 slots, first rows and totals fit its array (what
its documentation has always promised), however few slots there are per bin."""

import ctypes

import pytest
import torch  # noqa: F401  (libtorch must be loaded before the extension)

from composed_mixture_of_experts_engine_b200.ops import _ext

WORDS = 1 << 20  # CMOE_NOALLOC_SCRATCH_WORDS


@pytest.mark.parametrize("per_k", [0, 1])
@pytest.mark.parametrize("n_slots", [1, 8, 256, 257, 1000, 3328, 4096, 4104, 8192, 8200, 40000, 1 << 20])
def test_nothing_that_fits_is_refused(n_slots, per_k):
    _ext.ext()
    fn = ctypes.CDLL(str(_ext.BUILD_DIR / f"{_ext.EXT_NAME}.so")).cmoe_moe_plan_noalloc_words
    fn.restype, fn.argtypes = ctypes.c_size_t, [ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_int]
    K = 8
    units = (n_slots + 255) // 256
    for n_local in (1, 64, 350, 512, 1400, 3900, 3940, 8192, 25600, 25608, 80000, 116000, 200000, 349525, 400000):
        bins = n_local * (K if per_k else 1)
        if (units + 2) * bins <= WORDS:
            assert fn(n_slots, n_local, K, per_k) <= WORDS, (n_slots, n_local)
