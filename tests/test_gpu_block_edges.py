"""Blocks of every edge (interpBlockSize) in the block kernel: more than 16 targets a
line above an edge of 32, odd remainders, one block, and fields of enough blocks for
that kernel by default.  Payloads equal the oracle's byte for byte and decoded fields
bit for bit (the arithmetic is the reference's, so no tolerance), by the default route,
in the block kernel throughout (FAZ_FINEST_PLANES=0 for the finest level), and for
float32 in a batch."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import faz_gb300 as F
from faz_gb300.fields import spectral_field

import oracle.oracle as O

pytestmark = pytest.mark.gpu

LIN, CUB = F.INTERP_ALGO_LINEAR, F.INTERP_ALGO_CUBIC


@pytest.fixture(scope="module", autouse=True)
def system_zstd():
    O.set_zstd(None)
    yield


CASES = [((100000,), e, 0) for e in (2, 30, 34, 62, 64, 66, 100, 1000, 4096)] + [
    ((300, 301), 34, 0), ((300, 301), 64, 1), ((513, 400), 100, 0), ((130, 140), 128, 1), ((700, 650), 200, 0),
    ((2000, 1100), 64, 1), ((97, 90, 100), 34, 0), ((97, 90, 100), 38, 3), ((60, 61, 100), 40, 5),
    ((300, 290, 310), 36, 4), ((33, 300, 34), 40, 2)]


def _check(dims, dtype, monkeypatch, **kw):
    x = spectral_field(dims, slope=-3.0, noise=0.02, seed=sum(dims)).astype(dtype)
    conf = F.Config(*dims)
    conf.cmprAlgo, conf.errorBoundMode, conf.relErrorBound = F.ALGO_INTERP, F.EB_REL, 1e-3
    for k, v in kw.items():
        setattr(conf, k, v)
    stream, want = O.compress(conf, x)
    ref, _ = O.decompress(stream, dtype=x.dtype)
    t = torch.from_numpy(x).cuda()
    for mode in (None, "0"):
        if mode:
            monkeypatch.setenv("FAZ_FINEST_PLANES", mode)
        payload, _ = F.compress_payload_device(conf, t)
        assert bytes(payload) == want
        out = torch.full_like(t, 7.0)
        F.decompress_payload_device(len(dims), payload, out)
        assert out.cpu().numpy().tobytes() == ref.tobytes()
    monkeypatch.delenv("FAZ_FINEST_PLANES")
    streams = F.compress_batch([conf, conf], [t, t])
    assert streams[0] == streams[1] == F.compress_device(conf, t)


@pytest.mark.parametrize("interp", [LIN, CUB])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims,edge,direction", CASES)
def test_block_edge(dims, edge, direction, dtype, interp, monkeypatch):
    if dtype is np.float64 and len(dims) == 3 and edge > 34:
        pytest.skip("does not fit in shared memory")
    _check(dims, dtype, monkeypatch, interpAlgo=interp, interpDirection=direction, interpBlockSize=edge)


@pytest.mark.parametrize("dims,step,block", [((700, 901), 16, 64), ((700, 901), 8, 48), ((65, 70, 200), 8, 40)])
def test_fixed_blocks(dims, step, block, monkeypatch):
    """fixBlockSize: one block size for every level, the finest one's edge."""
    _check(dims, np.float32, monkeypatch, maxStep=step, alpha=1.5, beta=2.0, fixBlockSize=block)
