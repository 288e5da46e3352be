"""The plane kernel of the finest level with a line to a lane (finest.cu), at
fields of enough blocks for it to run by default (two blocks per SM or more),
and the calls that go to the block kernel instead.

Blocks whose two in-plane extents are 32 or 33 points take the lines; the first
and the last blocks of an axis, shorter ones and one-point ones take single
targets.  Codes move in runs of 16-byte pieces whose alignment depends on the
code count of all earlier blocks.  Streams equal the oracle's byte for byte and
the block kernel's (FAZ_FINEST_PLANES=0), decompressed arrays bit for bit: the
arithmetic is the reference's, so no tolerance.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import faz_gb300 as F
from faz_gb300.fields import spectral_field
from conftest import mask_first_size

import oracle.oracle as O

pytestmark = pytest.mark.gpu

LIN, CUB = F.INTERP_ALGO_LINEAR, F.INTERP_ALGO_CUBIC


@pytest.fixture(scope="module", autouse=True)
def system_zstd():
    O.set_zstd(None)
    yield


def _conf(dims, interp, direction, **kw):
    c = F.Config(*dims)
    c.cmprAlgo = F.ALGO_INTERP
    c.interpAlgo, c.interpDirection = interp, direction
    for k, v in kw.items():
        setattr(c, k, v)
    return c


REL3 = dict(errorBoundMode=F.EB_REL, relErrorBound=1e-3)
REL6 = dict(errorBoundMode=F.EB_REL, relErrorBound=1e-6, quantbinCnt=1024)
HALF = dict(errorBoundMode=F.EB_ABS, absErrorBound=0.5)
CASES = [
    # first and last blocks of 33 and 32 points in the plane; an odd plane count
    ((2463, 64, 64), CUB, 0, REL3, "plain"),
    ((64, 2464, 64), LIN, 2, REL3, "plain"),
    # last blocks of one point to 26: code runs at every alignment
    ((161, 258, 264), CUB, 0, REL3, "plain"),
    ((250, 161, 260), CUB, 2, REL3, "plain"),
    ((130, 271, 260), LIN, 0, REL3, "plain"),
    # unpredictable targets in lines and single ones
    ((161, 258, 264), CUB, 0, REL6, "spikes"),
    ((250, 161, 260), LIN, 2, REL6, "spikes"),
    # whole numbers at a bound of one half: differences on the bins' edges, targets
    # that only the double computation decides
    ((161, 258, 264), LIN, 0, HALF, "whole"),
    ((250, 161, 260), CUB, 2, HALF, "whole"),
    # rows that are no multiple of 16 bytes, and blocks of edge 16: the block kernel;
    # one block in four full in the plane: it decompresses
    ((161, 258, 263), CUB, 0, REL3, "plain"),
    ((161, 130, 132), CUB, 0, dict(REL3, interpBlockSize=16), "plain"),
    ((2464, 40, 40), CUB, 0, REL3, "plain"),
]


@pytest.mark.parametrize("dims,interp,direction,kw,kind", CASES)
def test_lines_match_block_kernel_and_oracle(dims, interp, direction, kw, kind, monkeypatch):
    x = spectral_field(dims, slope=-3.0, noise=0.02, seed=sum(dims) + direction)
    if kind == "spikes":
        x[np.random.default_rng(3).random(dims) < 0.01] *= 40.0
    elif kind == "whole":
        x = np.rint(x).astype(np.float32)
    conf = _conf(dims, interp, direction, **kw)
    monkeypatch.delenv("FAZ_FINEST_PLANES", raising=False)
    s = F.SZ_compress(conf, x)
    d, _ = F.SZ_decompress(None, s, dtype=x.dtype)
    monkeypatch.setenv("FAZ_FINEST_PLANES", "0")
    assert s == F.SZ_compress(conf, x)
    ref, _ = O.compress(conf, x)
    assert mask_first_size(s) == mask_first_size(ref)
    ref_dec, _ = O.decompress(ref)
    assert np.array_equal(d.view(np.uint32), ref_dec.view(np.uint32))


def test_unaligned_buffers_match_aligned():
    """Input and output four bytes off a 16-byte boundary: the block kernel."""
    dims = (161, 258, 264)
    n = int(np.prod(dims))
    x = torch.from_numpy(spectral_field(dims, slope=-3.0, noise=0.02, seed=4)).cuda()
    conf = _conf(dims, CUB, 0, **REL3)
    off = torch.empty(n + 1, dtype=torch.float32, device="cuda")[1:].view(dims)
    off.copy_(x)
    s = F.compress_device(conf, x)
    assert s == F.compress_device(conf, off)
    a, b = torch.empty_like(x), torch.empty(n + 1, dtype=torch.float32, device="cuda")[1:].view(dims)
    F.decompress_device(s, a)
    F.decompress_device(s, b)
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
