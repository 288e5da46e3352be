"""Payloads that no compressor writes.  A tree in which nodes have two parents
decodes as a walk over it says.  Damage that the Huffman stage finds is refused, and
the caller's output stays as it was."""
import struct

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import faz_gb300 as F

pytestmark = pytest.mark.gpu

N = 20001  # of the field; the odd points hold 0 or 2 at a bound of 1


def _payload():
    """A payload of two symbols: the bytes before its tree, the two states, the symbol
    of each code, the field."""
    bit = np.random.default_rng(2).integers(0, 2, N // 2)
    x = np.zeros(N, np.float32)
    x[1::2] = 2.0 * bit
    conf = F.Config(N)
    conf.cmprAlgo, conf.errorBoundMode, conf.absErrorBound = F.ALGO_INTERP, F.EB_ABS, 1.0
    conf.interpAlgo = F.INTERP_ALGO_LINEAR
    payload = bytes(F.compress_payload_device(conf, torch.from_numpy(x).cuda())[0])
    # dims, block size, interpolator, direction, alpha, beta, maxStep, list length (0),
    # block-wise, fixed block, cross block, trim, block order; quantiser id, bound, radius
    head = 8 + 4 * 3 + 8 * 3 + 4 + 1 + 4 + 8 + 4 + 4 + 1 + 8 + 4
    nunpred, = struct.unpack_from("<Q", payload, head)
    assert nunpred == 0
    tree = head + 8
    nodes, = struct.unpack_from(">I", payload, tree + 4)
    assert nodes == 3
    states = struct.unpack_from("<3i", payload, tree + 12 + 1 + 6)
    left, right = payload[tree + 13], payload[tree + 16]
    nbytes, = struct.unpack_from("<Q", payload, tree + 12 + 1 + 6 + 12 + 3)
    bits = payload[len(payload) - nbytes:]
    codes = np.unpackbits(np.frombuffer(bits, np.uint8))[:N]
    return payload[:tree], payload[tree:tree + 4], (states[left], states[right]), codes, x


def _tree(offset, left, right, states, leaf):
    n = len(left)
    return (offset + struct.pack(">2I", n, 2) + b"\0" + bytes(left) + bytes(right) + struct.pack(f"<{n}i", *states)
            + bytes(leaf))


def _decode(payload, out):
    F.decompress_payload_device(1, payload, out)
    return out.cpu().numpy()


@pytest.mark.parametrize("depth", [1, 11, 12, 13, 20, 21, 40])
def test_nodes_with_two_parents(depth):
    """Node i names i + 1 as both children, but for the last: codewords of `depth` bits
    of which the last counts."""
    head, offset, states, codes, x = _payload()
    left = list(range(1, depth)) + [depth, 0, 0]
    right = list(range(1, depth)) + [depth + 1, 0, 0]
    tree = _tree(offset, left, right, [0] * depth + list(states), [0] * depth + [1, 1])
    bits = np.random.default_rng(depth).integers(0, 2, (N, depth)).astype(np.uint8)
    bits[:, -1] = codes
    string = np.packbits(bits.reshape(-1)).tobytes()
    payload = head + tree + struct.pack("<Q", len(string)) + string
    got = _decode(payload, torch.full((N,), 7.0, device="cuda"))
    assert np.abs(got - x).max() <= 1.0
    assert np.array_equal(got, np.where(x > 0, 2.0, 0.0).astype(np.float32))


# one CTA's levels alone, sweep launches with an anchor grid, the block kernel
# (float64), the plane kernel
FIELDS = [((20001,), {}, np.float32), ((90, 80, 70), dict(maxStep=16, alpha=1.5, beta=2.0), np.float32),
          ((231, 230, 229), {}, np.float64), ((231, 262, 264), {}, np.float32)]


@pytest.mark.parametrize("damage", ["string cut", "one value less", "one value more", "negative state"])
@pytest.mark.parametrize("dims,kw,dtype", FIELDS)
def test_damage_leaves_the_output(dims, kw, dtype, damage):
    rng = np.random.default_rng(sum(dims))
    x = rng.normal(0, 3, dims).astype(dtype)
    x.reshape(-1)[rng.integers(0, x.size, 50)] = 1e9  # unpredictable values
    conf = F.Config(*dims)
    conf.cmprAlgo, conf.errorBoundMode, conf.absErrorBound = F.ALGO_INTERP, F.EB_ABS, 0.5
    for k, v in kw.items():
        setattr(conf, k, v)
    good = bytes(F.compress_payload_device(conf, torch.from_numpy(x).cuda())[0])
    head = 8 * len(dims) + 4 * 3 + 8 * 3 + 4 + 1 + 4 + 8 + 4 + 4 + 1 + 8 + 4
    nunpred, = struct.unpack_from("<Q", good, head)
    assert nunpred > 0
    tree = head + 8 + nunpred * x.itemsize
    nodes, = struct.unpack_from(">I", good, tree + 4)
    assert 3 < nodes <= 256  # one-byte indices
    at = tree + 13 + 2 * nodes + 4 * nodes + nodes
    nbytes, = struct.unpack_from("<Q", good, at)
    assert at + 8 + nbytes == len(good)
    if damage == "string cut":
        bad = good[:at] + struct.pack("<Q", nbytes // 2) + good[at + 8:at + 8 + nbytes // 2]
    elif damage == "one value less":
        bad = good[:head] + struct.pack("<Q", nunpred - 1) + good[head + 8:tree - x.itemsize] + good[tree:]
    elif damage == "one value more":
        bad = good[:head] + struct.pack("<Q", nunpred + 1) + good[head + 8:tree] + good[tree - x.itemsize:]
    else:  # of a rare symbol, one with a long codeword
        types = good[tree + 13 + 6 * nodes:at]
        left, right = good[tree + 13:tree + 13 + nodes], good[tree + 13 + nodes:tree + 13 + 2 * nodes]
        depth = [0] * nodes
        for i in range(nodes):
            if not types[i]:
                depth[left[i]] = depth[right[i]] = depth[i] + 1
        leaf = max((d, i) for i, d in enumerate(depth) if types[i])[1]
        assert depth[leaf] > 12
        state = tree + 13 + 2 * nodes + 4 * leaf
        bad = good[:state] + struct.pack("<i", -1) + good[state + 4:]
    out = torch.full(dims, 7.0, dtype=torch.from_numpy(x).dtype, device="cuda")
    with pytest.raises(F.FazError) as e:
        F.decompress_payload_device(len(dims), bad, out)
    assert e.value.code == -4
    assert bool((out == 7.0).all())
    F.decompress_payload_device(len(dims), good, out)
    assert np.abs(out.cpu().numpy() - x).max() <= 0.5
