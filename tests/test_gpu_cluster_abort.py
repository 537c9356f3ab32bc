"""A bootstrap on two SMs whose key stream stalls gives up in its first or its last step (they are the same where a
rotation has one): the call reports the timeout, both CTAs have received what they were sent before they exit, and
the next rotations are right."""
import numpy as np
import pytest

import tfhe_b200 as tb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def rotate(ck, precision, acc, bara):
    out = torch.from_numpy(acc).cuda()
    ck.blind_rotate_device(torch.from_numpy(np.ascontiguousarray(bara)).cuda(), out, len(acc), bara.shape[1], precision=precision)
    ck.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("N,l", [(1024, 3), (1024, 2), (2048, 3)])
@pytest.mark.parametrize("nsteps", [1, 2, 3, 9])
@pytest.mark.parametrize("precision", [tb.FP64, tb.SPLIT_FP32])
def test_stalled_pair_of_ctas(precision, nsteps, N, l):
    sk, ck = tb.keygen(tb.make_params(9, N, 1, l, 7, 8, 2), seed=31)
    ck.to_device(0, precisions=(precision,))
    rng = np.random.default_rng(nsteps)
    acc = rng.integers(-2**31, 2**31, (74, 2, N)).astype(np.int32)
    bara = rng.integers(0, 2 * N, (74, nsteps)).astype(np.int32)
    want = rotate(ck, precision, acc, bara)
    ck.set_wait_timeout(0.02)
    for count in (1, 74):
        ck.test_stall_key_stream(True)
        with pytest.raises(tb.api.TfhebError) as exc:
            rotate(ck, precision, acc[:count], bara[:count])
        assert exc.value.status == tb.api.TIMEOUT
        ck.test_stall_key_stream(False)
        assert (rotate(ck, precision, acc[:count], bara[:count]) == want[:count]).all()
