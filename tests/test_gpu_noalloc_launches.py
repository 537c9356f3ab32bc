"""The launch counter counts every blind-rotation launch of a call without allocations, as of one with them: the
descriptors are the one kernel more."""
import numpy as np
import pytest

import tfhe_b200 as tb
from test_zz_no_alloc import noalloc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 200, 330])  # 200 split bootstraps are two waves of one per SM
def test_counted_launches(count):
    sk, ck = tb.keygen(tb.default_params(), seed=61)
    ck.to_device(0, precisions=(tb.SPLIT_FP32,))
    a = torch.from_numpy(sk.encrypt(np.zeros(count, np.int64), seed=62)).cuda()
    out = torch.zeros_like(a)
    counts = []
    for call in (lambda: ck.gate_device(tb.api.NAND, a, a, None, out, count, precision=tb.SPLIT_FP32),
                 lambda: noalloc(ck, tb.api.NAND, tb.SPLIT_FP32, count, a, a, None, out)):
        before = tb.kernel_launches()
        call()
        ck.synchronize()
        counts.append(tb.kernel_launches() - before)
    assert counts[1] == counts[0] + 1
    assert counts[0] == (5 if count == 200 else 4)
