"""matmul_host: results in page-locked buffers that come back to a pool, both layouts, every kernel that can serve the call.
Exact on integers; results that are still held must not be overwritten by later calls."""
import numpy as np
import pytest

import oracle
from conftest import random_ternary
from ternaryllm_b200 import PackedWeight, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pin", [-1, 0])                       # the default choice, and the gather kernel (whose result is turned)
@pytest.mark.parametrize("dtype", [np.float32, np.float16, np.int8])
def test_layouts_and_lifetime(dtype, pin):
    rng = np.random.default_rng(1)
    K, N = 333, 150
    w = random_ternary(rng, K, N, 0.6)
    pw = PackedWeight.from_dense(w)
    prev = _lib.lib().tllm_set_mma_min_rows(pin)
    try:
        held = []
        for M in (1, 2, 7, 33, 131):
            x = rng.integers(-3, 4, size=(M, K)).astype(dtype)
            want = oracle.dense_f64(x.astype(np.float64), w)
            for xc in (False, True):
                for yc in (False, True):
                    y = pw.matmul_host(np.ascontiguousarray(x.T) if xc else x, col_major=xc, y_col_major=yc)
                    assert y.shape == ((N, M) if yc else (M, N)) and y.dtype == (np.int32 if dtype == np.int8 else dtype) and y.flags.writeable
                    held.append((y, want.T if yc else want))
        for y, want in held:
            assert np.array_equal(y.astype(np.float64), want)
    finally:
        _lib.lib().tllm_set_mma_min_rows(prev)
        pw.close()
