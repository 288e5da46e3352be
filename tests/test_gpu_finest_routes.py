"""Each kernel of the finest level on fields of every size.  By default few-block
fields take the sweep launches; FAZ_FINEST_PLANES sends the finest level of any field
to the block kernel (0), or to the plane kernel wherever that can run (2).  Payloads
equal the oracle's byte for byte, decoded fields bit for bit (the arithmetic is the
reference's, so no tolerance), and the launch counts say that another kernel ran:
three sweeps, or one launch."""
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


def _check(dims, interp, direction, dtype, modes, monkeypatch, **kw):
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
        # three sweeps (two of a 2-D field, one of a 1-D one) or one launch
        assert [a - b for a, b in zip(sweeps, one)] == [len(dims) - 1] * 2


@pytest.mark.parametrize("direction", range(6))
@pytest.mark.parametrize("interp", [LIN, CUB])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims", [(97, 66, 70), (65, 64, 33)])
def test_block_kernel(dims, dtype, interp, direction, monkeypatch):
    _check(dims, interp, direction, dtype, ["0"], monkeypatch)


@pytest.mark.parametrize("dims", [(700, 300), (65, 1000), (129, 97)])
@pytest.mark.parametrize("direction", [0, 1])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_block_kernel_flat(dims, dtype, direction, monkeypatch):
    _check(dims, CUB, direction, dtype, ["0"], monkeypatch)


@pytest.mark.parametrize("interp", [LIN, CUB])
@pytest.mark.parametrize("direction", [0, 2])
@pytest.mark.parametrize("dims,kw", [((66, 97, 68), {}), ((100, 64, 100), {}), ((70, 60, 52), dict(interpBlockSize=16)),
                                     ((66, 50, 52), dict(interpBlockSize=12)),
                                     ((96, 64, 64), dict(maxStep=16, alpha=1.5, beta=3.0))])
def test_plane_kernel(dims, kw, direction, interp, monkeypatch):
    _check(dims, interp, direction, np.float32, ["0", "2"], monkeypatch, **kw)
