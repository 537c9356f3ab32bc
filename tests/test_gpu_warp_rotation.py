"""The one-warp-per-bootstrap blind rotation (eight bootstraps per CTA, FFT exchanges in tensor memory): bit for
bit the rotation of the team kernels, which the oracle pins, with full, partly filled and single CTAs, over
the fewest steps, on both gadget lengths; its form with two warps per bootstrap and the kernels for a few
bootstraps (one per SM, one per cluster of two) against it; their forms for the larger ring; the cut of a batch into waves; digits too wide for the split form; stalled key streams."""
import numpy as np
import pytest

import tfhe_b200 as tb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def make(l, Bgbit, n=24):
    return tb.make_params(n, 1024, 1, l, Bgbit, 8, 2)


@pytest.fixture(scope="module")
def keys():
    made = {}

    def get(l, Bgbit):
        if (l, Bgbit) not in made:
            made[l, Bgbit] = tb.keygen(make(l, Bgbit), seed=77)
            made[l, Bgbit][1].to_device(0)
        return made[l, Bgbit]
    return get


@pytest.fixture(scope="module")
def large_keys():
    sk, ck = tb.keygen(tb.make_params(9, 2048, 1, 3, 8, 8, 2), seed=79)
    ck.to_device(0)
    return sk, ck


def packed_eight(ck, precision):
    G, _ = ck.br_variants(precision)
    return int(np.flatnonzero(G == 8)[0])


def rotate(ck, precision, variant, bara, acc, nsteps):
    out = torch.from_numpy(acc).cuda()
    ck.set_br_variant(precision, variant)
    ck.blind_rotate_device(torch.from_numpy(bara).cuda(), out, len(acc), nsteps, precision=precision)
    ck.synchronize()
    return out.cpu().numpy()


# 8 per CTA: one warp, a full CTA, one warp beyond, and a wave of 148 CTAs but for one warp
@pytest.mark.parametrize("count", [1, 8, 9, 1183])
@pytest.mark.parametrize("nsteps", [1, 2, 5])
@pytest.mark.parametrize("precision", [tb.FP64, tb.SPLIT_FP32])
@pytest.mark.parametrize("l,Bgbit", [(3, 7), (2, 10)])
def test_rotation_equals_the_team_kernel(keys, l, Bgbit, precision, nsteps, count):
    sk, ck = keys(l, Bgbit)
    rng = np.random.default_rng(count + nsteps)
    acc = rng.integers(-2**31, 2**31, (count, 2, 1024)).astype(np.int32)
    bara = rng.integers(0, 2048, (count, nsteps)).astype(np.int32)
    bara.flat[:4] = [0, 1, 1023, 1024][:min(4, bara.size)]  # the ends of the rotation's range
    want = rotate(ck, precision, 0, bara, acc, nsteps)
    # a batch of these sizes would be cut into waves of other variants: pad it to whole CTAs' worth of one wave
    pad = 1184 - count
    big = np.concatenate([acc, np.repeat(acc[:1], pad, 0)])
    got = rotate(ck, precision, packed_eight(ck, precision), np.concatenate([bara, np.repeat(bara[:1], pad, 0)]), big, nsteps)
    assert (got[:count] == want).all()
    assert (got[count:] == want[0]).all()
    ck.set_br_variant(precision, 0)


# N = 2048, two warps per bootstrap, four bootstraps per CTA
@pytest.mark.parametrize("count", [1, 4, 5, 591])
@pytest.mark.parametrize("nsteps", [1, 2, 3])
@pytest.mark.parametrize("precision", [tb.FP64, tb.SPLIT_FP32])
def test_large_ring_rotation_equals_the_team_kernel(large_keys, precision, nsteps, count):
    sk, ck = large_keys
    rng = np.random.default_rng(3 * count + nsteps)
    acc = rng.integers(-2**31, 2**31, (592, 2, 2048)).astype(np.int32)
    bara = rng.integers(0, 4096, (592, nsteps)).astype(np.int32)
    bara.flat[:5] = [0, 1, 2047, 2048, 4095]  # the ends of the rotation's range, both parities
    acc[count:], bara[count:] = acc[:1], bara[:1]
    G, D = ck.br_variants(precision)
    got = rotate(ck, precision, int(np.flatnonzero(G == 4)[0]), bara, acc, nsteps)
    want = rotate(ck, precision, 0, bara[:count], acc[:count], nsteps)
    assert (got[:count] == want).all() and (got[count:] == want[0]).all()


# one bootstrap on two SMs (at most 74 of 148), one per SM, both in turn, and two warps for each of 3 or 4 per SM
@pytest.mark.parametrize("count", [1, 2, 74, 75, 148, 149, 230, 443, 589, 592])
@pytest.mark.parametrize("nsteps", [1, 2, 3, 7])
@pytest.mark.parametrize("precision", [tb.FP64, tb.SPLIT_FP32])
@pytest.mark.parametrize("l,Bgbit", [(3, 7), (2, 10)])
def test_few_bootstraps_equal_a_packed_wave(keys, l, Bgbit, precision, nsteps, count):
    sk, ck = keys(l, Bgbit)
    rng = np.random.default_rng(10 * count + nsteps)
    acc = rng.integers(-2**31, 2**31, (1184, 2, 1024)).astype(np.int32)
    bara = rng.integers(0, 2048, (1184, nsteps)).astype(np.int32)
    bara.flat[:4] = [0, 1, 1023, 1024][:min(4, bara.size)]
    eight = packed_eight(ck, precision)
    want = rotate(ck, precision, eight, bara, acc, nsteps)
    assert (rotate(ck, precision, eight, bara[:count], acc[:count], nsteps) == want[:count]).all()
    ck.set_br_variant(precision, 0)


# N = 2048: one bootstrap on two SMs (at most 74 of 148); a step takes six rows through a ring of five, or three
@pytest.mark.parametrize("count", [1, 2, 73, 74, 75, 148])
@pytest.mark.parametrize("nsteps", [1, 2, 5, 9])
@pytest.mark.parametrize("precision", [tb.FP64, tb.SPLIT_FP32])
def test_large_ring_few_bootstraps_equal_a_packed_wave(large_keys, precision, nsteps, count):
    sk, ck = large_keys
    rng = np.random.default_rng(7 * count + nsteps)
    acc = rng.integers(-2**31, 2**31, (592, 2, 2048)).astype(np.int32)
    bara = rng.integers(0, 4096, (592, nsteps)).astype(np.int32)
    bara.flat[:5] = [0, 1, 2047, 2048, 4095]
    four = int(np.flatnonzero(ck.br_variants(precision)[0] == 4)[0])
    want = rotate(ck, precision, four, bara, acc, nsteps)
    assert (rotate(ck, precision, four, bara[:count], acc[:count], nsteps) == want[:count]).all()


# around the waves' ends: all of the last wave's choices, and a last CTA with one of eight warps at work
@pytest.mark.parametrize("count", [1033, 1177, 1184, 1185, 1500, 1777])
@pytest.mark.parametrize("precision", [tb.FP64, tb.SPLIT_FP32])
@pytest.mark.parametrize("l,Bgbit", [(3, 7), (2, 10), (3, 8)])  # 24 digit bits: the split form's other kernel
def test_batches_cut_into_waves(l, Bgbit, precision, count):
    sk, ck = tb.keygen(make(l, Bgbit, n=12), seed=78)
    ck.to_device(0, precisions=(precision,))
    rng = np.random.default_rng(count)
    x, y = rng.integers(0, 2, count), rng.integers(0, 2, count)
    a, b = sk.encrypt(x, seed=1), sk.encrypt(y, seed=2)
    got = ck.gate(tb.api.NAND, a, b, precision=precision)  # the default rule
    ck.set_br_variant(precision, 0)
    assert (got == ck.gate(tb.api.NAND, a, b, precision=precision)).all()
    assert (sk.decrypt(got)[0] == 1 - (x & y)).all()


# a packed wave, two warps per bootstrap, one bootstrap per SM, one per two SMs (both CTAs of a cluster give up)
@pytest.mark.parametrize("count", [1184, 592, 100, 3])
@pytest.mark.parametrize("precision", [tb.FP64, tb.SPLIT_FP32])
def test_stalled_key_stream(keys, precision, count):
    sk, ck = keys(3, 7)
    rng = np.random.default_rng(5)
    x = rng.integers(0, 2, count)
    a = sk.encrypt(x, seed=9)
    ck.set_br_variant(precision, packed_eight(ck, precision))
    ck.set_wait_timeout(0.05)
    ck.test_stall_key_stream(True)
    with pytest.raises(tb.api.TfhebError) as exc:
        ck.gate(tb.api.NAND, a, a, precision=precision)
    assert exc.value.status == tb.api.TIMEOUT
    ck.test_stall_key_stream(False)
    ck.set_wait_timeout(1.0)
    assert (sk.decrypt(ck.gate(tb.api.NAND, a, a, precision=precision))[0] == 1 - x).all()
    ck.set_br_variant(precision, 0)


@pytest.mark.parametrize("precision", [tb.FP64, tb.SPLIT_FP32])
def test_stalled_key_stream_large_ring(large_keys, precision):
    sk, ck = large_keys
    bara, acc = np.zeros((3, 2), np.int32), np.zeros((3, 2, 2048), np.int32)
    ck.set_wait_timeout(0.05)
    ck.test_stall_key_stream(True)
    with pytest.raises(tb.api.TfhebError) as exc:
        rotate(ck, precision, 0, bara, acc, 2)
    assert exc.value.status == tb.api.TIMEOUT
    ck.test_stall_key_stream(False)
    ck.set_wait_timeout(1.0)
    rotate(ck, precision, 0, bara, acc, 2)
