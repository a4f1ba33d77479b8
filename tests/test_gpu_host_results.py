"""matmul_host: both layouts, every kernel that can serve the call.  Exact on integers; results that are still held must not be
overwritten by later calls, and are ordinary numpy arrays of their own memory."""
import ctypes as C

import numpy as np
import pytest
import torch

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


@pytest.mark.parametrize("threads", [1, 8])                     # one: no page-locked block in between
def test_results_are_ordinary_arrays(threads):
    """Pageable memory of their own: a copy of one to the GPU has read its source when it returns, even with non_blocking=True,
    so that the array may be dropped or written at once; and a program that keeps many of them locks no memory."""
    rng = np.random.default_rng(2)
    K, N, M = 256, 2048, 512                                    # 4 MB a result
    w = random_ternary(rng, K, N, 0.5)
    pw = PackedWeight.from_dense(w)
    xs = [rng.integers(-3, 4, size=(M, K)).astype(np.float32) for _ in range(3)]
    before = torch.get_num_threads()
    torch.set_num_threads(threads)
    try:
        for x in xs:
            y = pw.matmul_host(x)
            assert y.flags.owndata and y.flags.c_contiguous and y.flags.writeable
            assert not torch.from_numpy(y).is_pinned()
        on_gpu = [torch.from_numpy(pw.matmul_host(x)).to("cuda", non_blocking=True) for x in xs]
        for x, y in zip(xs, on_gpu):
            assert np.array_equal(y.double().cpu().numpy(), oracle.dense_f64(x.astype(np.float64), w))
    finally:
        torch.set_num_threads(before)
        pw.close()


def test_results_under_a_dispatch_mode():
    """The call works on numpy arrays: what intercepts torch's operations has nothing to do with it."""
    from torch._subclasses.fake_tensor import FakeTensorMode

    rng = np.random.default_rng(3)
    K, N, M = 96, 1024, 256                                     # 1 MB: through the page-locked block
    w = random_ternary(rng, K, N, 0.5)
    pw = PackedWeight.from_dense(w)
    x = rng.integers(-3, 4, size=(M, K)).astype(np.float32)
    before = torch.get_num_threads()
    torch.set_num_threads(8)
    try:
        with FakeTensorMode():
            y = pw.matmul_host(x)
        assert np.array_equal(y.astype(np.float64), oracle.dense_f64(x.astype(np.float64), w))
    finally:
        torch.set_num_threads(before)
        pw.close()


def test_more_rows_than_a_grid_is_high():
    """Column-major results that are turned on the device (here behind a bias): one row more than 65535 tiles
    of 32."""
    rng = np.random.default_rng(4)
    K, N, M = 16, 3, 65535 * 32 + 1
    w = random_ternary(rng, K, N, 0.5)
    pw = PackedWeight.from_dense(w)
    x = rng.integers(-3, 4, size=(M, K)).astype(np.float16)
    bias = np.array([1.0, -2.0, 5.0], np.float16)
    want = (x.astype(np.float32) @ w.astype(np.float32)).T + bias[:, None].astype(np.float32)
    y = np.empty((N, M), np.float16)
    try:
        rc = _lib.lib().tllm_spmm_host_bias(pw._h, _lib.np_ptr(x), _lib.F16, _lib.ROW_MAJOR, M, _lib.np_ptr(bias), _lib.np_ptr(y), _lib.F16, _lib.COL_MAJOR)
        assert rc == 0, _lib.lib().tllm_last_error()
        assert np.array_equal(y.astype(np.float32), want)
    finally:
        pw.close()


# results in one piece, several, as many as there are, ragged last ones, and too large to be staged; activations staged and not; threads that copy and none
@pytest.mark.parametrize("threads", [1, 8])
@pytest.mark.parametrize("M,K,N", [(64, 512, 1024), (33, 1000, 2051), (131, 257, 1111), (256, 300, 3001), (301, 1024, 3500), (512, 64, 8200)])
def test_staged_buffers(M, K, N, threads):
    rng = np.random.default_rng(N)
    w = random_ternary(rng, K, N, 0.5)
    pw = PackedWeight.from_dense(w)
    before = torch.get_num_threads()
    torch.set_num_threads(threads)
    try:
        for dtype in (np.float32, np.float16, np.int8):
            x = rng.integers(-3, 4, size=(M, K)).astype(dtype)
            want = x.astype(np.float32) @ w.astype(np.float32)
            assert np.array_equal(pw.matmul_host(x).astype(np.float32), want)
            assert np.array_equal(pw.matmul_host(np.ascontiguousarray(x.T), col_major=True, y_col_major=True).astype(np.float32), want.T)
    finally:
        torch.set_num_threads(before)
        pw.close()


# Pieces of a result in the order of their bytes, more of them than it has blocks of 4096 bytes too; a refused call reports none
def test_results_in_pieces():
    L = _lib.lib()
    rng = np.random.default_rng(3)
    K, N = 128, 520
    w = random_ternary(rng, K, N, 0.5)
    pw = PackedWeight.from_dense(w)
    seen = []
    ready = C.CFUNCTYPE(None, C.c_void_p, C.c_size_t, C.c_size_t)(lambda arg, begin, end: seen.append((begin, end)))
    for M in (1, 9, 64):
        x = rng.integers(-3, 4, size=(M, K)).astype(np.float32)
        y = np.full((M, N), -1, np.float32)

        def call(parts, rows=M, y_type=_lib.F32, function=ready):
            seen.clear()
            return L.tllm_spmm_host_parts(pw._h, x.ctypes.data, _lib.F32, _lib.ROW_MAJOR, rows, y.ctypes.data, y_type, _lib.ROW_MAJOR, parts, C.cast(function, C.c_void_p), None)

        for parts in (1, 3, 8):
            y[:] = -1
            assert call(parts) == 0 and len(seen) == parts
            assert [b for b, _ in seen] == [0] + [e for _, e in seen[:-1]] and seen[-1][1] == y.nbytes
            assert np.array_equal(y, oracle.dense_f64(x.astype(np.float64), w))
        assert call(0) != 0 and call(9) != 0 and call(2, rows=0) != 0 and call(2, y_type=77) != 0 and not seen
        assert call(2, function=None) != 0
    pw.close()


# Staged copies are dealt out in elements of one to eight bytes: sizes that are multiples of eight and not, above and below the least that is staged
@pytest.mark.parametrize("threads", [4, 5, 6, 7, 12])
@pytest.mark.parametrize("dtype", [np.float32, np.float16, np.int8])
def test_staging_by_threads(dtype, threads):
    rng = np.random.default_rng(4)
    before = torch.get_num_threads()
    torch.set_num_threads(threads)
    try:
        for M, K, N in ((64, 4096, 512), (255, 1001, 1037), (511, 515, 2051)):
            w = random_ternary(rng, K, N, 0.5)
            pw = PackedWeight.from_dense(w)
            x = rng.integers(-1, 2, size=(M, K)).astype(dtype)
            want = x.astype(np.float32) @ w.astype(np.float32)          # exact: sums below 4097
            y = pw.matmul_host(x)
            assert np.array_equal(y, want.astype(np.float16) if dtype == np.float16 else want)
            assert np.array_equal(pw.matmul_host(np.ascontiguousarray(x.T), col_major=True, y_col_major=True), y.T)
            pw.close()
    finally:
        torch.set_num_threads(before)
