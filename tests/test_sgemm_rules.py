"""How a float32 product of many rows is cut into calls: the rule alone, without a GPU."""
import ctypes

import pytest


@pytest.mark.parametrize("K", [512, 2048, 12288, 25600, 40000, 300001])
@pytest.mark.parametrize("batch", [1, 3, 128])
def test_scratch_of_a_call_stays_within_its_limit(K, batch):
    """Every row of every product once, and no call's scratch above the limit but a lone tile's."""
    from binfer_b200.csrc import ops
    scratch = ops.lib().bf_sgemm_split_scratch
    scratch.restype = ctypes.c_longlong
    for M in (0, 1, 16, 17, 112, 113, 333, 1232, 4096, 70001):
        seen = set()
        for b, nb, m0, m in ops._sgemm_split_calls(M, K, batch):
            rows = {(x, m0) for x in range(b, b + nb)}
            assert not rows & seen and nb > 0 and b + nb <= batch and m0 + m <= M
            seen |= rows
            for N in (8, 4096, 151936):
                n = scratch(m, N, K, nb, batch, 0)
                assert n <= ops.SGEMM_SPLIT_MAX_BYTES or (nb == 1 and m <= 112), (M, m, nb, n)
        starts = {m0: m for _, _, m0, m in ops._sgemm_split_calls(M, K, batch)}
        assert sum(starts.values()) == M and len(seen) == batch * len(starts)
