"""Batches that leave the last CTA of a packed kernel partly empty, as they come: bit for bit the first listed variant
run in whole waves, on every ring and form; and such a batch's key stream stalled."""
import numpy as np
import pytest

import tfhe_b200 as tb
from test_gpu_variant_choice import make_key, operands, rotate, whole_waves

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# 148 SMs: one and two SMs per bootstrap, one per SM; two, three and four per CTA, the last one with one bootstrap, or
# lacking one; beyond four per SM the packed kernel of eight at N = 1024 (1037 = 129 x 8 + 5)
FEW = [1, 73, 75, 147, 149, 295, 298, 443, 445, 446, 447, 591]


@pytest.mark.parametrize("N,l,Bgbit,counts", [(1024, 3, 7, FEW + [1037, 1041, 1183]), (1024, 2, 10, FEW + [1037, 1041, 1183]),
                                              (2048, 3, 8, FEW)])
@pytest.mark.parametrize("precision", [tb.FP64, tb.SPLIT_FP32])
def test_partly_empty_ctas(precision, N, l, Bgbit, counts):
    acc, bara = operands(N, max(counts), N + l)
    bara.flat[:5] = [0, 1, N - 1, N, 2 * N - 1]  # the ends of the rotation's range
    want = whole_waves(N, l, Bgbit, precision, acc, bara)
    ck = make_key(N, l, Bgbit, precision)
    for count in counts:
        assert (rotate(ck, precision, acc, bara, count) == want[:count]).all(), count


@pytest.mark.parametrize("N,counts", [(1024, [298, 447, 1041]), (2048, [446, 592])])
@pytest.mark.parametrize("precision", [tb.FP64, tb.SPLIT_FP32])
def test_stalled_key_stream(precision, N, counts):
    ck = make_key(N, 3, 7, precision)
    acc, bara = operands(N, max(counts), 7)
    want = rotate(ck, precision, acc, bara, max(counts))
    ck.set_wait_timeout(0.02)
    for count in counts:
        ck.test_stall_key_stream(True)
        with pytest.raises(tb.api.TfhebError) as exc:
            rotate(ck, precision, acc, bara, count)
        assert exc.value.status == tb.api.TIMEOUT
        ck.test_stall_key_stream(False)
        assert (rotate(ck, precision, acc, bara, count) == want[:count]).all()
