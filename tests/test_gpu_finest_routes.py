"""Each kernel of the finest level on fields of every size.  By default small 3-D and
large 2-D fields take the sweep launches; FAZ_FINEST_PLANES sends the finest level of
any field to the block kernel (0), or to the plane kernel wherever that can run (2).
Payloads equal the oracle's byte for byte, decoded fields bit for bit (the arithmetic is
the reference's, so no tolerance), and the launch counts say which kernel ran: three
sweeps (two of a 2-D field), or one launch."""
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


def _run(conf, t, ref_payload, ref, monkeypatch, mode):
    if mode is None:
        monkeypatch.delenv("FAZ_FINEST_PLANES", raising=False)
    else:
        monkeypatch.setenv("FAZ_FINEST_PLANES", mode)
    payload, _ = F.compress_payload_device(conf, t)
    n = [F.last_timings()["kernel_launches"]]
    assert bytes(payload) == ref_payload
    out = torch.empty_like(t)
    F.decompress_payload_device(t.ndim, payload, out)
    n.append(F.last_timings()["kernel_launches"])
    assert out.cpu().numpy().tobytes() == ref.tobytes()
    return n


def _check(dims, interp, direction, dtype, modes, monkeypatch, fewer=(2, 2), **kw):
    x = spectral_field(dims, slope=-3.0, noise=0.02, seed=sum(dims) + direction).astype(dtype)
    conf = F.Config(*dims)
    conf.cmprAlgo, conf.errorBoundMode, conf.relErrorBound = F.ALGO_INTERP, F.EB_REL, 1e-3
    conf.interpAlgo, conf.interpDirection = interp, direction
    for k, v in kw.items():
        setattr(conf, k, v)
    stream, payload = O.compress(conf, x)
    ref, _ = O.decompress(stream, dtype=x.dtype)
    t = torch.from_numpy(x).cuda()
    sweeps = _run(conf, t, payload, ref, monkeypatch, None)
    for mode in modes:
        one = _run(conf, t, payload, ref, monkeypatch, mode)
        assert [a - b for a, b in zip(sweeps, one)] == list(fewer)


@pytest.mark.parametrize("direction", range(6))
@pytest.mark.parametrize("interp", [LIN, CUB])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims", [(97, 66, 70), (65, 64, 33)])
def test_block_kernel(dims, dtype, interp, direction, monkeypatch):
    _check(dims, interp, direction, dtype, ["0"], monkeypatch)


# fields on either side of the rule between the sweeps and a CTA per block: launches that
# one launch saves in compression and in decompression
@pytest.mark.parametrize("dims,dtype,edge,fewer", [
    # 2-D: 2^20 points, two blocks across, each range of edges
    ((1024, 1024), np.float32, 32, (1, 1)), ((1024, 1023), np.float32, 32, (0, 0)),
    ((1024, 1024), np.float64, 16, (1, 1)), ((300, 700), np.float64, 16, (1, 1)), ((300, 700), np.float64, 32, (0, 0)),
    ((64, 17000), np.float32, 32, (1, 1)), ((63, 17000), np.float32, 32, (0, 0)),
    ((17000, 63), np.float32, 32, (0, 0)), ((1025, 1030), np.float32, 4, (0, 0)),
    ((1025, 1030), np.float32, 14, (0, 1)), ((300, 400), np.float64, 8, (1, 1)),
    ((300, 400), np.float64, 6, (0, 0)), ((192, 320), np.float64, 64, (1, 1)), ((640, 641), np.float32, 64, (1, 1)),
    # 3-D: 2^21 points, two blocks an SM
    ((128, 128, 127), np.float32, 32, (2, 2)), ((128, 128, 128), np.float32, 32, (0, 0)),
    ((130, 129, 128), np.float32, 38, (2, 2)), ((128, 128, 128), np.float64, 32, (2, 2)),
    ((160, 192, 320), np.float64, 32, (2, 2)), ((170, 192, 320), np.float64, 32, (0, 0))])
def test_rule(dims, dtype, edge, fewer, monkeypatch):
    _check(dims, CUB, 1, dtype, ["0"], monkeypatch, fewer, interpBlockSize=edge)


@pytest.mark.parametrize("interp", [LIN, CUB])
@pytest.mark.parametrize("direction", [0, 2])
@pytest.mark.parametrize("dims,kw", [((66, 97, 68), {}), ((100, 64, 100), {}), ((70, 60, 52), dict(interpBlockSize=16)),
                                     ((66, 50, 52), dict(interpBlockSize=12)),
                                     ((96, 64, 64), dict(maxStep=16, alpha=1.5, beta=3.0))])
def test_plane_kernel(dims, kw, direction, interp, monkeypatch):
    _check(dims, interp, direction, np.float32, ["0", "2"], monkeypatch, **kw)


@pytest.mark.parametrize("mode", [None, "0", "2"])
@pytest.mark.parametrize("interp", [LIN, CUB])
@pytest.mark.parametrize("whole", [True, False])
def test_verified(whole, interp, mode, monkeypatch):
    """FAZ_VERIFY_FASTPATH in each kernel of the finest level: the call fails where the
    float proofs and the double computation differ.  Whole numbers at a bound of one
    half lie on the bins' edges.  Blocks of 32 and 33 points, whose lines the plane
    kernel keeps in registers, and shorter ones."""
    dims = (97, 100, 132)
    x = spectral_field(dims, slope=-3.0, noise=0.02, seed=11)
    conf = F.Config(*dims)
    conf.cmprAlgo, conf.interpAlgo, conf.errorBoundMode = F.ALGO_INTERP, interp, F.EB_ABS
    conf.absErrorBound = 0.5 if whole else 0.013
    if whole:
        x = np.rint(x).astype(np.float32)
    monkeypatch.setenv("FAZ_VERIFY_FASTPATH", "1")
    if mode is None:
        monkeypatch.delenv("FAZ_FINEST_PLANES", raising=False)
    else:
        monkeypatch.setenv("FAZ_FINEST_PLANES", mode)
    stream, want = O.compress(conf, x)
    ref, _ = O.decompress(stream)
    t = torch.from_numpy(x).cuda()
    payload, _ = F.compress_payload_device(conf, t)
    assert bytes(payload) == want
    out = torch.empty_like(t)
    F.decompress_payload_device(3, payload, out)
    assert out.cpu().numpy().tobytes() == ref.tobytes()
