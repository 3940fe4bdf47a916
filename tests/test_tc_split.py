"""The rule that says how many CTAs of a cluster share K in the Q40 tensor-core GEMM (host code of the CUDA library: no GPU needed)."""
import pytest

from dllama_b200.ops import kernels as K


@pytest.mark.parametrize("d,n,rows,want", [
    # a rank's part of models of width 2048, 4096 and 8192: few columns or few inputs (times beside the rule)
    (768, 4096, (4, 8, 16, 32), 8), (512, 2048, (4, 16, 32), 8), (1024, 2048, (4, 32), 8), (1280, 8192, (8, 32, 64), 8), (1536, 4096, (4, 8, 32), 8),
    (4096, 512, (4, 32, 64, 128), 1), (4096, 1024, (4, 32), 4), (4096, 1024, (64, 128, 256), 1), (4096, 1792, (4, 32), 4), (8192, 1024, (4, 32), 2),
    (8192, 1024, (64, 128), 1), (8192, 2048, (4, 32), 2), (8192, 2048, (128,), 1), (2048, 1024, (128, 256), 1), (1536, 4096, (384,), 2), (2048, 512, (4, 32), 1),
    # whole models
    (4096, 4096, (4, 32, 64, 128), 4), (4096, 14336, (4, 32, 128), 4), (2048, 8192, (4, 32, 128), 4), (4096, 2048, (4, 32, 64), 4), (2048, 2048, (4, 32, 64), 4),
    (6144, 4096, (4, 32, 128), 2), (28672, 4096, (4, 128, 700), 1)])
def test_split_of_measured_products(d, n, rows, want):
    assert [K.choose_tc_split(d, n, M, 148) for M in rows] == [want] * len(rows)


def test_split_stays_within_what_finds_room():
    for d in (128, 300, 512, 1280, 4096, 8192, 28672, 128256):
        for n in (128, 256, 640, 2048, 14336):
            for M in (1, 4, 16, 17, 33, 64, 65, 128, 129, 300, 512, 767):
                S = K.choose_tc_split(d, n, M, 148)
                assert S in (1, 2, 4, 8) and S <= n // 128
                nt = K.tc_tile(d, n, M, 1 << 30, S)
                assert S == 1 or (d + 127) // 128 * -(-M // nt) * S <= {2: 148, 4: 128, 8: 96}[S]
