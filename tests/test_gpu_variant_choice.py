"""Which compiled blind-rotation kernel serves a batch must not show in its bits.  The reference here is the team
kernel by itself: a batch of whole waves of the first listed variant, which is then cut nowhere."""
import numpy as np
import pytest

import tfhe_b200 as tb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

STEPS = 6


def make_key(N, l, Bgbit, precision, seed=41):
    sk, ck = tb.keygen(tb.make_params(STEPS, N, 1, l, Bgbit, 8, 2), seed=seed)
    ck.to_device(0, precisions=(precision,))
    return ck


def operands(N, count, seed):
    rng = np.random.default_rng(seed)
    return rng.integers(-2**31, 2**31, (count, 2, N)).astype(np.int32), rng.integers(0, 2 * N, (count, STEPS)).astype(np.int32)


def rotate(ck, precision, acc, bara, count):
    out = torch.from_numpy(acc[:count]).cuda()
    ck.blind_rotate_device(torch.from_numpy(np.ascontiguousarray(bara[:count])).cuda(), out, count, STEPS, precision=precision)
    ck.synchronize()
    return out.cpu().numpy()


def whole_waves(N, l, Bgbit, precision, acc, bara):
    """All rows through the first listed variant, which `N` and `l` have as a kernel of one team per bootstrap."""
    ck = make_key(N, l, Bgbit, precision)
    wave = torch.cuda.get_device_properties(0).multi_processor_count * int(ck.br_variants(precision)[0][0])
    pad = -len(acc) % wave
    ck.set_br_variant(precision, 0)
    acc, bara = (np.concatenate([x, np.repeat(x[:1], pad, 0)]) for x in (acc, bara))
    return rotate(ck, precision, acc, bara, len(acc))[:len(acc) - pad]


# digits wider than the split form of the warp kernels holds: l Bgbit = 24, 30, 24, 32
@pytest.mark.parametrize("l,Bgbit", [(3, 8), (3, 10), (2, 12), (2, 16)])
def test_autotuned_wide_digits(l, Bgbit):
    precision = tb.SPLIT_FP32
    acc, bara = operands(1024, 592, 10 * l + Bgbit)
    want = whole_waves(1024, l, Bgbit, precision, acc, bara)
    ck = make_key(1024, l, Bgbit, precision)
    ck.autotune(precision, boots=1184)
    for count in (20, 100, 200, 300, 444, 592):  # every number of bootstraps per SM up to four
        assert (rotate(ck, precision, acc, bara, count) == want[:count]).all(), count


# FP64 sums of products near 2^50 and beyond do not round to exact integers, so their order shows; the other sets' do
@pytest.mark.parametrize("N,l,Bgbit", [(1024, 2, 11), (1024, 2, 12), (1024, 2, 14), (1024, 2, 16), (1024, 3, 10), (2048, 3, 10)])
@pytest.mark.parametrize("tuned", [False, True])
def test_wide_digits_in_fp64(N, l, Bgbit, tuned):
    precision = tb.FP64
    acc, bara = operands(N, 1184, 100 + Bgbit)
    want = whole_waves(N, l, Bgbit, precision, acc, bara)
    ck = make_key(N, l, Bgbit, precision)
    if tuned:
        ck.autotune(precision, boots=1184)
    for count in (1, 74, 100, 200, 300, 592, 1184):
        assert (rotate(ck, precision, acc, bara, count) == want[:count]).all(), count


# a launch costs as much as a step or two: a rotation of one step is cut into no more launches than pay for themselves
@pytest.mark.parametrize("N,l,Bgbit,precision,count,launches", [
    (1024, 3, 7, tb.SPLIT_FP32, 700, 1), (1024, 3, 7, tb.SPLIT_FP32, 1500, 1), (1024, 3, 7, tb.SPLIT_FP32, 296, 1),
    (1024, 3, 7, tb.FP64, 600, 1), (1024, 2, 10, tb.SPLIT_FP32, 700, 1), (2048, 3, 8, tb.SPLIT_FP32, 148, 1),
    # a second packed wave takes 18.6 us, the rest in a launch of its own 7.7 + 7
    (2048, 3, 8, tb.FP64, 700, 2)])
def test_one_step_in_few_launches(N, l, Bgbit, precision, count, launches):
    ck = make_key(N, l, Bgbit, precision)
    acc, bara = operands(N, count, count)
    got = torch.from_numpy(acc).cuda()
    one = torch.from_numpy(np.ascontiguousarray(bara[:, :1])).cuda()
    before = tb.kernel_launches()
    ck.blind_rotate_device(one, got, count, 1, precision=precision)
    ck.synchronize()
    assert tb.kernel_launches() - before == launches
    # the same step of the packed kernel: a whole wave of it
    G = ck.br_variants(precision)[0]
    wave = torch.cuda.get_device_properties(0).multi_processor_count * int(G[0])
    pad = -count % wave
    want = torch.from_numpy(np.concatenate([acc, np.repeat(acc[:1], pad, 0)])).cuda()
    bara1 = np.concatenate([bara[:, :1], np.repeat(bara[:1, :1], pad, 0)])
    ck.set_br_variant(precision, 0)
    ck.blind_rotate_device(torch.from_numpy(bara1).cuda(), want, count + pad, 1, precision=precision)
    ck.synchronize()
    assert (got.cpu().numpy() == want[:count].cpu().numpy()).all()
