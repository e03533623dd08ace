"""Which kernel serves more than 16 rows of the linear module: lines taken from timings of both."""
from bitmtp_b200 import ops


def test_few_rows_of_a_narrow_deep_weight_go_through_the_gemv():
    for N, K in ((512, 1024), (4096, 1024), (512, 2048), (2048, 2560), (4096, 4096), (512, 9728), (4096, 9728), (8, ops.GEMV_MAX_K)):
        assert [ops.gemv_serves_rows(T, N, K) for T in (1, 16, 17, 32, 33, 333)] == [False, False, True, True, False, False]


def test_the_rest_goes_through_the_many_row_kernel():
    for N, K in ((6144, 1024), (4104, 9728), (12288, 2048), (512, 512), (512, 768), (512, 1152), (512, 9600),
                 (512, ops.GEMV_MAX_K + 256), (8, 51200)):
        assert not any(ops.gemv_serves_rows(T, N, K) for T in (17, 24, 32, 33, 64))
