"""The calls by which the engine's speed is measured: batches of bootstrapped gates, bootstraps, keyswitches
and netlists, from one gate to thousands, through the public entry points of tfhe_b200.

A case is a dict of plain values:
  name     (listed cases only)
  kind     the entry point: "device" (gate batch on device buffers), "host" (the same on host buffers),
           "mixed" (several gate types over rows of a device wire array), "woks" (bootstrap without
           keyswitch), "keyswitch", or "netlist" (a levelled circuit, replayed as a CUDA graph)
  params   "128" (n=630, N=1024, l=3, the default set), "80" (n=500, N=1024, l=2) or "2048" (n=800, N=2048, l=3)
  form     "split" (FP32 limbs) or "fp64"; a keyswitch has no form
  gate     a gate's name, for "device" and "host"
  count    gates, samples, or (netlist) the widest level
  levels   levels of a netlist, else 0
"""
import ctypes
import math

import numpy as np
import torch

import tfhe_b200 as tb
from tfhe_b200 import api

GATES = api.GATE_NAMES[:11]  # the bootstrapped ones
FORMS = {"fp64": tb.FP64, "split": tb.SPLIT_FP32}


def case(name, kind, params, form, gate, count, levels=0):
    return {"name": name, "kind": kind, "params": params, "form": form, "gate": gate, "count": count, "levels": levels}


def listed():
    return [
        # one gate at a time, as a program that chains single gate calls has it: launches and one
        # bootstrap's serial chain count; from device buffers, and from host buffers as the drop-in calls it
        case("gate-1-split", "device", "128", "split", "NAND", 1),
        case("gate-1-host-fp64", "host", "128", "fp64", "AND", 1),
        # a few dozen concurrent callers combined into one host call
        case("gates-64-host-split", "host", "128", "split", "XOR", 64),
        # one step of a circuit evaluator: all gate types in one batch, less than one wave of an SM's room
        case("mixed-333-split", "mixed", "128", "split", "", 333),
        # bootstraps whose extracted samples are used as they are (no keyswitch), several per SM
        case("woks-600-fp64", "woks", "128", "fp64", "", 600),
        # a ragged batch of a few per cent over a whole number of waves, or under it
        case("gates-1500-host-split", "host", "128", "split", "ORNY", 1500),
        # the throughput workload, both forms
        case("nand-4096-split", "device", "128", "split", "NAND", 4096),
        case("nand-4096-fp64", "device", "128", "fp64", "NAND", 4096),
        # the 80-bit set, in its usual form, two bootstraps per gate
        case("mux-700-80bit-fp64", "device", "80", "fp64", "MUX", 700),
        # the larger ring at its throughput batch
        case("mux-1024-n2048-split", "device", "2048", "split", "MUX", 1024),
        # keyswitches of extracted samples alone (after sums of bootstraps without keyswitch)
        case("keyswitch-4096", "keyswitch", "128", "", "", 4096),
        # a circuit of levels of very different widths, replayed on one wire array
        case("netlist-10x1200-split", "netlist", "128", "split", "", 1200, 10),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["device", "device", "device", "host", "host", "mixed", "woks", "keyswitch", "netlist"])
    params = rng.choice(["128", "128", "128", "80", "2048"])
    form = "" if kind == "keyswitch" else rng.choice(["split", "split", "fp64"])
    gate = rng.choice(GATES) if kind in ("device", "host") else ""
    levels = 0
    if kind == "netlist":
        params, levels = "128", rng.randint(3, 8)
        count = _log_uniform(rng, 20, 1000 if form == "split" else 600)
    elif kind == "keyswitch":
        count = _log_uniform(rng, 1, 4096 if params != "2048" else 2048)
    else:
        # bootstraps of a listed case's cost at most (a MUX, like the mixed batch's, takes two)
        most = {"128": 4096, "80": 4096, "2048": 2048 if form == "split" else 1200}[params]
        count = _log_uniform(rng, 1, most // 2 if gate == "MUX" else most * 4 // 5 if kind == "mixed" else most)
    return {"kind": kind, "params": params, "form": form, "gate": gate, "count": count, "levels": levels}


def _params(c):
    return api.large_params() if c["params"] == "2048" else api.default_params(int(c["params"]))


def _circuit(c):
    """A netlist's wiring: widths from a few gates to the widest, operands from the two levels before."""
    rng = np.random.default_rng(c["count"])
    return api.random_netlist(rng, c["levels"], max(1, c["count"] // 16), c["count"])


def _mixed(c, rng):
    """Every gate type, MUX rarer; rows 0 .. 2 count - 1 are operands, gate g writes row 2 count + g."""
    n = c["count"]
    codes = rng.choice(13, size=n, p=np.array([3, 2, 2, 3, 2, 1, 1, 1, 1, 1, 2, .5, .5]) / 20)
    idx = rng.integers(0, 2 * n, (3, n))
    return [x.astype(np.int32) for x in (codes, *idx, 2 * n + np.arange(n))]


_streams = []


def _stream():
    """The program's one stream: what it asks of several keys runs in turn."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return ctypes.c_void_p(_streams[0].cuda_stream)


def prepare(c, seed):
    p, kind, n = _params(c), c["kind"], c["count"]
    rng = np.random.default_rng(seed)
    sk, ck = tb.keygen(p, seed=seed)
    form = FORMS.get(c["form"], tb.SPLIT_FP32)
    ck.to_device(0, precisions=(form,))
    s = {"kind": kind, "ck": ck, "form": form, "count": n, "stream": _stream()}
    if kind in ("device", "host"):
        s["gate"] = api.GATE_NAMES.index(c["gate"])
        cts = [sk.encrypt(rng.integers(0, 2, n), seed=seed + 1 + i) for i in range(3 if c["gate"] == "MUX" else 2)]
        cts = cts + [None] * (3 - len(cts))
        s["in"] = cts if kind == "host" else [None if x is None else torch.from_numpy(x).cuda() for x in cts]
        if kind == "device":
            s["out"] = torch.zeros((n, p.n + 1), dtype=torch.int32, device="cuda")
    elif kind == "woks":
        s["in"] = torch.from_numpy(sk.encrypt(rng.integers(0, 2, n), seed=seed + 1)).cuda()
        s["out"] = torch.zeros((n, p.k * p.N + 1), dtype=torch.int32, device="cuda")
    elif kind == "keyswitch":  # masks and phases of bootstrapped samples are uniform
        x = rng.integers(-2**31, 2**31, (n, p.k * p.N + 1)).astype(np.int32)
        s["in"] = torch.from_numpy(x).cuda()
        s["out"] = torch.zeros((n, p.n + 1), dtype=torch.int32, device="cuda")
    elif kind == "mixed":
        s["plan"] = _mixed(c, rng)
        s["out"] = torch.zeros((3 * n, p.n + 1), dtype=torch.int32, device="cuda")
        s["out"][:2 * n] = torch.from_numpy(sk.encrypt(rng.integers(0, 2, 2 * n), seed=seed + 1))
    else:
        ni, gates, ia, ib, ic = _circuit(c)
        s["netlist"] = api.Netlist(ck, ni, gates, ia, ib, ic)
        s["out"] = torch.zeros((ni + len(gates), p.n + 1), dtype=torch.int32, device="cuda")
        s["out"][:ni] = torch.from_numpy(sk.encrypt(rng.integers(0, 2, ni), seed=seed + 1))
    torch.cuda.synchronize()  # the inputs are ready before the engine's stream reads them
    return s


def run(s):
    ck, kind, n, form, stream = s["ck"], s["kind"], s["count"], s["form"], s["stream"]
    if kind == "host":
        return ck.gate(s["gate"], *s["in"], precision=form)
    if kind == "device":
        ck.gate_device(s["gate"], *s["in"], s["out"], n, precision=form, stream=stream)
    elif kind == "woks":
        ck.bootstrap_woks_device(s["in"], s["out"], n, mu=1 << 29, precision=form, stream=stream)
    elif kind == "keyswitch":
        ck.keyswitch_device(s["in"], s["out"], n, stream=stream)
    elif kind == "mixed":
        ck.gate_mixed_device(*s["plan"], s["out"], len(s["out"]), precision=form, stream=stream)
    else:
        s["netlist"].run(s["out"], precision=form, use_graph=True, stream=stream)
    return s["out"]


def _bootstraps(c):
    """(bootstraps, keyswitches, ciphertexts read, ciphertexts written) of one pass."""
    n = c["count"]
    if c["kind"] == "mixed":  # one gate in ten is a MUX, one in twenty needs no bootstrap
        return n * 1.05, n * .95, 2 * n, n
    if c["kind"] == "netlist":
        gates = c["levels"] * n * 17 / 32  # widths uniform between a sixteenth and the whole
        return 1.1 * gates, gates, n * 17 / 32, gates
    if c["kind"] == "keyswitch":
        return 0, n, n, n
    if c["kind"] == "woks":
        return n, 0, n, n
    return (2 * n, n, 3 * n, n) if c["gate"] == "MUX" else (n, n, 2 * n, n)


def work(c):
    """The two keys once, the ciphertexts in and out, and the arithmetic of the textbook algorithm: a
    bootstrap is n external products, each (k+1)l forward transforms, the products of their spectra
    with the key's, and an inverse transform per output (and limb); a keyswitch subtracts the rows of
    the non-zero digits, three in four."""
    p = _params(c)
    boots, switches, ins, outs = _bootstraps(c)
    M, rows, limbs = p.N // 2, (p.k + 1) * p.l, 2 if c["form"] == "split" else 1
    transform = 5 * M * math.log2(M) + 6 * M
    step = (rows + (p.k + 1) * limbs) * transform + rows * (p.k + 1) * limbs * M * 8
    small, large = 4 * (p.n + 1), 4 * (p.k * p.N + 1)
    nbytes = ins * (large if c["kind"] == "keyswitch" else small) + outs * (large if c["kind"] == "woks" else small)
    nbytes += p.n * rows * (p.k + 1) * M * 16 * (boots > 0) + p.k * p.N * p.ks_t * 3 * small * (switches > 0)
    return {"bytes": nbytes, "flops": boots * p.n * step + switches * p.k * p.N * p.ks_t * .75 * (p.n + 1)}


# ---- the same results in plain numpy, 64-bit integers and floats -----------------------------------

def _negacyclic(digits, key):
    """Sum over rows of digits[row] * key[row, v] in Z[X]/(X^N+1), mod 2^32: exact, as the key's two
    16-bit halves keep every coefficient below 2^40."""
    N = digits.shape[-1]
    twist = np.exp(-1j * np.pi * np.arange(N) / N)
    fd = np.fft.fft(digits * twist)[:, None]
    out = 0
    for half, shift in ((key & 0xffff, 0), (key >> 16, 16)):
        c = np.fft.ifft((fd * np.fft.fft(half * twist)).sum(0)) * twist.conj()
        out = out + (np.rint(c.real).astype(np.int64) << shift)
    return out & 0xffffffff


def _bootstrap(p, bsk, x, mu):
    """Gate bootstrap of one sample x [n+1] without keyswitch: the extracted sample [kN+1], k = 1."""
    N, two = p.N, 2 * p.N
    bar = (((x.astype(np.int64) & 0xffffffff) * two + (1 << 31)) >> 32) % two
    j = np.arange(N)

    def rotated(poly, a):  # X^a poly
        e = (j - a) % two
        return np.where(e < N, poly[..., e % N], -poly[..., e % N]) & 0xffffffff

    acc = np.zeros((2, N), np.int64)
    acc[1] = rotated(np.full(N, mu, np.int64), two - bar[p.n])
    half = 1 << (p.Bgbit - 1)
    offset = sum(half << (32 - (q + 1) * p.Bgbit) for q in range(p.l))
    for i in range(p.n):
        d = (rotated(acc, bar[i]) - acc + offset) & 0xffffffff
        digits = [((d[u] >> (32 - (q + 1) * p.Bgbit)) & (2 * half - 1)) - half for u in range(2) for q in range(p.l)]
        acc = (acc + _negacyclic(np.array(digits), bsk[i].astype(np.int64))) & 0xffffffff
    return np.concatenate([acc[0, :1], -acc[0, :0:-1], acc[1, :1]]) & 0xffffffff


def _keyswitch(p, ksk, x):
    out = np.zeros(p.n + 1, np.int64)
    out[p.n] = x[-1]
    a = (x[:-1].astype(np.int64) + (1 << (31 - p.ks_basebit * p.ks_t))) & 0xffffffff
    for q in range(p.ks_t):
        h = (a >> (32 - (q + 1) * p.ks_basebit)) & ((1 << p.ks_basebit) - 1)
        out -= (ksk[np.arange(len(h)), q, h].astype(np.int64) * (h != 0)[:, None]).sum(0)
    return out


def _torus32(rows):
    return torch.from_numpy((np.stack(rows) & 0xffffffff).astype(np.uint32).view(np.int32).copy())


#: Linear combinations of the gates (eighths, sign of a, sign of b)
_FORM = {"NAND": (1, -1, -1), "OR": (1, 1, 1), "AND": (-1, 1, 1), "XOR": (2, 2, 2), "XNOR": (-2, -2, -2),
         "NOR": (-1, -1, -1), "ANDNY": (-1, -1, 1), "ANDYN": (-1, 1, -1), "ORNY": (1, -1, 1), "ORYN": (1, 1, -1)}


def exact(c, seed):
    """Keyswitches, and single gates and a few bootstraps in FP64 (whose products round to the exact
    integers).  The split form's low limb is rounded in FP32 and every rounding changes the masks of
    all later steps, so its ciphertexts have no such value; large batches would take too long."""
    p = _params(c)
    if c["kind"] == "keyswitch" and c["count"] <= 256:
        ksk = tb.keygen(p, seed=seed)[1].export()[1]
        x = np.random.default_rng(seed).integers(-2**31, 2**31, (c["count"], p.k * p.N + 1)).astype(np.int32)
        return _torus32([_keyswitch(p, ksk, row) for row in x])
    if c["form"] != "fp64" or c["gate"] not in _FORM or c["count"] > 4:
        return None
    sk, ck = tb.keygen(p, seed=seed)
    bsk, ksk = ck.export()
    rng = np.random.default_rng(seed)
    a, b = (sk.encrypt(rng.integers(0, 2, c["count"]), seed=seed + 1 + i).astype(np.int64) for i in range(2))
    const, sa, sb = _FORM[c["gate"]]
    x = sa * a + sb * b
    x[:, p.n] += const << 29
    return _torus32([_keyswitch(p, ksk, _bootstrap(p, bsk, row, 1 << 29)) for row in x])
