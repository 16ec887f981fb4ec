"""How the GEMM of few rows divides an SM: host arithmetic, no device (CPU)."""
import ctypes as C

import pytest

from brain_b200.ops import _cuda

SM_KB, TMEM_COLUMNS = 228, 512


@pytest.mark.parametrize("int8", [0, 1])
@pytest.mark.parametrize("slices,smem_kb", [(0, 0), (1, 32), (2, 74), (8, 110), (4, 226)])
def test_ctas_of_an_sm_fit_its_tensor_memory(int8, slices, smem_kb):
    """CTAs that wait for tensor memory while their cluster waits for them can wait for ever: as many as share an SM by
    their shared memory, of any sizes, must find their columns."""
    lib, out = _cuda.lib(), (C.c_int * 3)()
    for M in (1, 16, 17, 32, 33, 48, 64, 65, 100, 128, 129, 160, 224, 255):
        for N, glu in ((64, 0), (1024, 0), (3072, 1), (24576, 0)):
            for K in (16, 64, 128, 256, 512, 1024, 2056, 4096, 12288):
                rc = lib.bb_gemm_rows_plan(M, N, K, int8, N if glu else 0, 148, slices, smem_kb, out)
                if rc != 0:
                    assert (slices, smem_kb) == (1, 32) and M > 64      # a stage does not fit: the call is refused
                    continue
                s, smem, columns = out
                assert 1 <= s <= 8 and columns >= M and smem <= 227 * 1024
                assert columns * (SM_KB * 1024) <= TMEM_COLUMNS * (smem + 1024), (M, N, K, smem, columns)
