"""Which kernel a prompt's projections take (csrc/gemm_tcgen05.cu): sizes at which one of the three was measured to be faster than the
others by 4 % and more, around where the choice has its borders.  The times are the fastest kernel's and what the others took."""
import pytest

pytestmark = pytest.mark.gpu

MEASURED = [  # rows, outputs, K, gated, kernel; us of the persistent kernel, the clusters and the pairs
    (1777, 8192, 28672, False, "pairs"),   # 680 / 713 / 545
    (2048, 8192, 28672, False, "pairs"),   # 774 / 856 / 696
    (900, 57344, 8192, True, "pairs"),     # 710 / 787 / 636
    (2048, 57344, 8192, True, "pairs"),    # 1455 / 1717 / 1345
    (4096, 57344, 8192, True, "pairs"),    # 2922 / 3556 / 2741
    (301, 28672, 4096, True, "rows"),      # 84 / 76 / 82
    (336, 28672, 4096, True, "persistent"),  # 85 / 95 / 83
    (400, 28672, 4096, True, "pairs"),     # 112 / 112 / 91
    (301, 8192, 8192, False, "rows"),      # 60 / 41 / 44
    (400, 4096, 14336, False, "rows"),     # 90 / 44 / 50
    (450, 4096, 4096, False, "pairs"),     # 32 / 22 / 19
    (2048, 256, 4096, False, "rows"),      # narrow: the pairs 27 % slower
    # qkv projections, with the rotation in the epilogue (without it they take the same kernel)
    (129, 10240, 8192, False, "rows"),     # 67 / 37 / 49
    (301, 6144, 4096, False, "rows"),      # 38 / 22 / 28
    (384, 6144, 4096, False, "rows"),      # 38 / 23 / 28
    (600, 6144, 4096, False, "pairs"),     # 38 / 30 / 29
    (1024, 6144, 4096, False, "pairs"),    # 59 / 54 / 39
    (512, 10240, 8192, False, "pairs"),    # 104 / 92 / 72
]


@pytest.mark.parametrize("M,N,K,gated,kernel", MEASURED)
def test_the_kernel_measured_to_be_faster(cuda, M, N, K, gated, kernel):
    from dli_b200 import ops

    if ops.sm_count() != 148:
        pytest.skip("the choice counts SMs")
    assert ops.gemm_plan(M, N, K, gated)[0] == kernel
