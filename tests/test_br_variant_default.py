"""A key's blind-rotation variant can be set to any listed one and back to the default rule (-1)."""
import numpy as np
import pytest

import tfhe_b200 as tb


@pytest.mark.parametrize("precision", [tb.FP64, tb.SPLIT_FP32])
def test_accepted_variants(precision):
    sk, ck = tb.keygen(tb.make_params(6, 1024, 1, 3, 7, 8, 2), seed=51)
    n = len(ck.br_variants(precision)[0])
    for v in range(-1, n):
        ck.set_br_variant(precision, v)
    for v in (-2, n):
        with pytest.raises(tb.api.TfhebError):
            ck.set_br_variant(precision, v)


@pytest.mark.gpu
@pytest.mark.parametrize("tune", [False, True])
def test_back_to_the_default(tune):
    # a packed wave of the default's variant is one launch, of entry 0 a wave and a rest
    torch = pytest.importorskip("torch")
    sk, ck = tb.keygen(tb.make_params(6, 1024, 1, 3, 7, 8, 2), seed=52)
    ck.to_device(0)
    count = 8 * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(53)
    acc = torch.from_numpy(rng.integers(-2**31, 2**31, (count, 2, 1024)).astype(np.int32)).cuda()
    bara = torch.from_numpy(rng.integers(0, 2048, (count, 6)).astype(np.int32)).cuda()

    def launches():
        out, before = acc.clone(), tb.kernel_launches()
        torch.cuda.synchronize()
        ck.blind_rotate_device(bara, out, count, 6, precision=tb.SPLIT_FP32)
        ck.synchronize()
        return tb.kernel_launches() - before, out

    default, want = launches()
    if tune:
        ck.autotune(tb.SPLIT_FP32, boots=count)
    ck.set_br_variant(tb.SPLIT_FP32, 0)
    other, out = launches()
    assert (default, other) == (1, 2) and torch.equal(out, want)
    ck.set_br_variant(tb.SPLIT_FP32, -1)
    again, out = launches()
    assert again == 1 and torch.equal(out, want)
