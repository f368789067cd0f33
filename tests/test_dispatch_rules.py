"""Rules by which the launchers choose a kernel, as far as they can be asked without a GPU."""
import pytest

from qwb200.ops import lib as qlib


@pytest.fixture
def lib():
    L = qlib.load()
    if L is None:
        pytest.skip("the kernel library is not built")
    return L


@pytest.mark.parametrize("nt", [1, 8, 15, 17, 100, 255, 257, 272, 4096])
def test_exchanged_tiles_of_other_sizes_are_refused(lib, nt):
    """A tile's tokens have to be a multiple of 16 up to 256; anything else leaves the setting as it is."""
    old = lib.qwk_gemm_tc_exchange_nt(48)
    try:
        assert lib.qwk_gemm_tc_exchange_nt(nt) == 48
        assert lib.qwk_gemm_tc_exchanged(777, 16480, 2560) == 48
    finally:
        lib.qwk_gemm_tc_exchange_nt(old)
    assert lib.qwk_gemm_tc_exchange_nt(old) == old
