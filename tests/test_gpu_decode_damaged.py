"""Payloads that no compressor writes.  A tree in which nodes have two parents
decodes as a walk over it says."""
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
