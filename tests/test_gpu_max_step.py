"""Anchor grids coarser than the field, up to the largest power of two that fits the
header: one anchor, and a call that ends.  (A step of 2^63 made the search for its
logarithm go on for ever.)"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import faz_gb300 as F

import oracle.oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,kw", [((70, 90), {}), ((33, 40, 50), {}), ((64, 64), dict(fixBlockSize=128))])
@pytest.mark.parametrize("log2", [10, 40, 62, 63])
def test_step(log2, dims, kw):
    x = np.random.default_rng(log2).normal(0, 3, dims).astype(np.float32)
    conf = F.Config(*dims)
    conf.cmprAlgo, conf.errorBoundMode, conf.absErrorBound = F.ALGO_INTERP, F.EB_ABS, 0.5
    conf.maxStep, conf.alpha, conf.beta = 1 << log2, 1.5, 2.0
    for k, v in kw.items():
        setattr(conf, k, v)
    t = torch.from_numpy(x).cuda()
    payload = bytes(F.compress_payload_device(conf, t)[0])
    if log2 < 63:
        assert payload == O.compress(conf, x)[1]
    out = torch.empty_like(t)
    F.decompress_payload_device(len(dims), payload, out)
    assert np.abs(out.cpu().numpy() - x).max() <= 0.5


@pytest.mark.parametrize("step", [(1 << 63) + 1, (1 << 64) - 1])
def test_step_not_a_power_of_two(step):
    conf = F.Config(30, 40)
    conf.cmprAlgo, conf.absErrorBound, conf.maxStep = F.ALGO_INTERP, 0.5, step
    with pytest.raises(F.FazError) as e:
        F.compress_payload_device(conf, torch.zeros(30, 40, device="cuda"))
    assert e.value.code == -2
