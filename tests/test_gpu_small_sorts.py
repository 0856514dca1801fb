"""The sorts of few entries: one cluster (radix), one block (bitonic), at the
edges of their blocks and tiles."""
import ctypes

import numpy as np
import pytest

from fluid_step import _abi
from fluid_step.pipelines import sort_pairs_host

pytestmark = pytest.mark.gpu


def _keys(n, bits, kind):
    rng = np.random.default_rng(n + bits)
    if kind == "ones":                       # every digit the padding's
        return np.full(n, (1 << bits) - 1, np.uint64).astype(np.uint32)
    k = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    if kind == "ties":
        k &= np.uint32(7)
    return k


@pytest.mark.parametrize("kind", ["random", "ties", "ones"])
@pytest.mark.parametrize("bits", [32, 17, 8, 1])
@pytest.mark.parametrize("n", [2, 31, 512, 2047, 2048, 2049, 4097, 16385, 32767, 32768, 32769,
                               65535, 65536, 65537])
def test_small_radix_sort_is_stable(n, bits, kind):
    k = _keys(n, bits, kind)
    v = np.arange(n, dtype=np.uint32)[::-1].copy()
    ks, vs = sort_pairs_host(k, v, key_bits=bits)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(ks, k[order]) and np.array_equal(vs, v[order])


def test_small_sort_clears_the_error_word_in_order():
    import torch
    lib = _abi.load_library()
    big = torch.randint(0, 1 << 30, (100000,), dtype=torch.int32, device="cuda")
    bv = torch.arange(100000, dtype=torch.int32, device="cuda")
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for n in (100000, 1000, 100000, 1000):
        assert lib.fe_sort_pairs(ctypes.c_void_p(big.data_ptr()), ctypes.c_void_p(bv.data_ptr()),
                                 n, 32, _abi.FE_SORT_RADIX, st) == _abi.FE_OK
        flags = torch.full((1,), 7, dtype=torch.int32, device="cuda")
        assert lib.fe_sort_flags(ctypes.c_void_p(flags.data_ptr()), st) == _abi.FE_OK
        assert int(flags.item()) == 0
        assert bool((big[1:n] >= big[:n - 1]).all())


@pytest.mark.parametrize("n", [2, 4, 32, 64, 128, 512, 4096, 8192, 16384, 32768])
@pytest.mark.parametrize("ties", [False, True])
def test_bitonic_network_of_every_tile(oracle_mod, n, ties):
    k = _keys(n, 32, "ties" if ties else "random")
    v = np.arange(n, dtype=np.uint32)
    ks, vs = sort_pairs_host(k, v, algorithm=_abi.FE_SORT_BITONIC)
    rk, rv = oracle_mod.sort_bitonic(k, v)
    assert np.array_equal(ks, rk) and np.array_equal(vs, rv)


@pytest.mark.parametrize("n", [1000, 40000, 100000])
def test_a_sort_clears_an_error_word_that_was_raised(n):
    """The error word is one call's: a wait that ran out raises it, and the next
    sort, by one cluster or in passes, clears it in stream order."""
    import torch
    lib = _abi.load_library()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    k = torch.randint(0, 1 << 30, (n,), dtype=torch.int32, device="cuda")
    v = torch.arange(n, dtype=torch.int32, device="cuda")

    def sort():
        assert lib.fe_sort_pairs(ctypes.c_void_p(k.data_ptr()), ctypes.c_void_p(v.data_ptr()), n,
                                 32, _abi.FE_SORT_RADIX, st) == _abi.FE_OK

    def word():
        f = torch.full((1,), 7, dtype=torch.int32, device="cuda")
        assert lib.fe_sort_flags(ctypes.c_void_p(f.data_ptr()), st) == _abi.FE_OK
        return int(f.item())

    sort()
    assert word() == 0
    assert lib.fe_debug_sort_wait_timeout(500, st) == _abi.FE_OK
    assert word() == _abi.FE_STATS_LOOKBACK_TIMEOUT
    sort()
    assert word() == 0
    assert lib.fe_debug_sort_wait_timeout(0, st) == _abi.FE_ERR_INVALID_ARGUMENT
