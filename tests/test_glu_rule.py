"""Which form gate, up and SwiGLU of 256 rows and more take: the rule against both sides as measured (CPU: no launch)."""
import pytest

from brain_b200.ops import _cuda

# int8, rows, ff, K, us as product + pass, us in one kernel; sizes at which the two differ by 5 % or more
MEASURED = [(0, 300, 6144, 2048, 25.6, 39.1), (0, 512, 512, 512, 8.2, 10.7), (0, 1072, 2048, 1024, 14.7, 19.2), (0, 256, 256, 256, 8.9, 11.9),
            (0, 1300, 2048, 1024, 21.4, 19.3), (0, 2200, 3072, 1024, 31.4, 25.7), (0, 8192, 6144, 2048, 375.2, 340.6),
            (0, 8192, 1024, 512, 29.4, 26.4), (0, 256, 12288, 4096, 71.7, 66.4), (0, 4096, 9728, 2560, 354.3, 325.8),
            (1, 256, 256, 256, 7.3, 13.0), (1, 8192, 1024, 512, 33.9, 42.2), (1, 1072, 3072, 1024, 21.8, 24.5), (1, 1072, 6144, 2048, 38.8, 44.9),
            (1, 8192, 3072, 1024, 98.9, 104.8), (1, 512, 12288, 4096, 56.1, 53.0), (1, 300, 12288, 4096, 47.6, 51.0),
            (1, 4096, 12288, 4096, 366.1, 328.4), (1, 8192, 12288, 4096, 702.8, 649.9)]


@pytest.mark.parametrize("int8,rows,ff,k,apart,fused", MEASURED)
def test_the_faster_form_is_taken(int8, rows, ff, k, apart, fused):
    assert bool(_cuda.lib().bb_glu_on_pairs(int8, rows, ff, k)) == (fused < apart)


@pytest.mark.parametrize("rows,ff,k", [(255, 6144, 2048), (8192, 255, 2048), (8192, 6144, 255)])
def test_sizes_that_pairs_do_not_serve(rows, ff, k):
    assert not _cuda.lib().bb_glu_on_pairs(0, rows, ff, k) and not _cuda.lib().bb_glu_on_pairs(1, rows, ff, k)
