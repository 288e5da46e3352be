"""Chunks whose bits begin and end on the words of the string (k_scan_chunks in
huffman.cu clears the words that two chunks share): two symbols of one bit each, so
that every chunk of 4096 codes is 128 words, one symbol alone, and the same in a
string that goes through the encoder in slices."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import faz_gb300 as F

import oracle.oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def system_zstd():
    O.set_zstd(None)
    yield


def _conf(dims):
    conf = F.Config(*dims)
    conf.cmprAlgo, conf.errorBoundMode, conf.absErrorBound = F.ALGO_INTERP, F.EB_ABS, 0.5
    return conf


@pytest.mark.parametrize("n", [4095, 4096, 4097, 3 * 4096, 1 << 20, (1 << 20) + 17])
@pytest.mark.parametrize("spikes", [(), (-2,), (1, -2)])
def test_word_aligned_chunks(n, spikes):
    x = np.zeros(n, np.float32)
    for s in spikes:
        x[s - (n & 1)] = 3.0
    conf = _conf((n,))
    t = torch.from_numpy(x).cuda()
    junk = torch.full((4 * n,), 255, dtype=torch.uint8, device="cuda")  # the pool's memory is not zero
    del junk
    payload, _ = F.compress_payload_device(conf, t)
    _, want = O.compress(conf, x)
    assert bytes(payload) == want


def test_word_aligned_chunks_in_slices():
    """16 MB of one-bit codes."""
    dims = (512, 512, 520)
    t = torch.zeros(dims, device="cuda")
    t[101, 203, 301] = 3.0
    t[511, 511, 519] = 3.0
    payload, _ = F.compress_payload_device(_conf(dims), t)
    assert len(payload) >= 16 << 20
    out = torch.empty_like(t)
    F.decompress_payload_device(3, payload, out)
    assert (out - t).abs().max().item() <= 0.5
