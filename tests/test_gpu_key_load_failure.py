"""A cloud key whose loading ran out of device memory half-way is not loaded: calls that need it are refused before
anything is launched, and loading it again gives a whole key."""
import numpy as np
import pytest

import tfhe_b200 as tb

pytestmark = pytest.mark.gpu
NOMEM = 3  # TFHEB_ERR_NOMEM


def gate(ck, a, precision):
    return ck.gate(tb.api.NAND, a, a, precision=precision)


# allocations: the coefficients and tables for the transform, the key, its second layout where there is one, its tables
@pytest.mark.parametrize("N,precision,allocations", [(1024, tb.FP64, 4), (1024, tb.SPLIT_FP32, 6), (2048, tb.FP64, 5),
                                                     (2048, tb.SPLIT_FP32, 6), (512, tb.SPLIT_FP32, 5)])
def test_failed_allocation(N, precision, allocations):
    p = tb.make_params(6, N, 1, 3, 7, 8, 2)
    sk, ck = tb.keygen(p, seed=21)
    a = sk.encrypt(np.array([0, 1, 1]), seed=22)
    ck.to_device(0, precisions=(precision,))
    want = gate(ck, a, precision)
    for nth in range(allocations + 1):
        ck = tb.keygen(p, seed=21)[1]
        ck.test_fail_device_alloc(nth)
        if nth == allocations:  # one more than there are
            ck.to_device(0, precisions=(precision,))
        else:
            with pytest.raises(tb.api.TfhebError) as exc:
                ck.to_device(0, precisions=(precision,))
            assert exc.value.status == NOMEM
            with pytest.raises(tb.api.TfhebError):
                ck.fft_key(precision)
            with pytest.raises(tb.api.TfhebError):
                gate(ck, a, precision)
            ck.to_device(0, precisions=(precision,))
        assert (gate(ck, a, precision) == want).all()


def test_failed_change_of_the_split():
    # the key is remade for another split of its words: if that fails, the former one is gone too
    sk, ck = tb.keygen(tb.make_params(6, 1024, 1, 3, 7, 8, 2), seed=23)
    a = sk.encrypt(np.array([0, 1, 1]), seed=24)
    ck.to_device(0)
    fp64 = gate(ck, a, tb.FP64)
    ck.test_fail_device_alloc(3)
    with pytest.raises(tb.api.TfhebError):
        ck.to_device(0, precisions=(tb.SPLIT_FP32,), split_shift=25)
    with pytest.raises(tb.api.TfhebError):
        gate(ck, a, tb.SPLIT_FP32)
    assert (gate(ck, a, tb.FP64) == fp64).all()
    ck.to_device(0, precisions=(tb.SPLIT_FP32,), split_shift=25)
    assert (sk.decrypt(gate(ck, a, tb.SPLIT_FP32))[0] == [1, 0, 0]).all()
