"""The level dispatch and the Huffman encoder where their rules and tiles end:
fields of one sub-chunk (2048 codes) and of one packing chunk (4096) and one value
to either side, levels on either side of the one-CTA rule and of the two blocks an
SM, thin and flat fields (blocks of one point, one axis alone), zero inside the
histogram's window (few bins), symbols outside it (many), codes longer than 32
bits, strings on either side of the sliced copy (16 MB).  Payloads against the
oracle's."""
import numpy as np
import pytest

import faz_gb300 as F

import oracle.oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def system_zstd():
    O.set_zstd(None)
    yield


def _check(x, eb, **kw):
    import torch
    conf = F.Config(*x.shape)
    conf.cmprAlgo, conf.errorBoundMode, conf.absErrorBound = F.ALGO_INTERP, F.EB_ABS, eb
    for k, v in kw.items():
        setattr(conf, k, v)
    t = torch.from_numpy(x).cuda()
    payload, _ = F.compress_payload_device(conf, t)
    _, want = O.compress(conf, x)
    assert bytes(payload) == want
    out = torch.empty_like(t)
    F.decompress_payload_device(x.ndim, payload, out)
    assert np.abs(out.cpu().numpy().astype(np.float64) - x.astype(np.float64)).max() <= eb


def _noise(dims, scale, dtype=np.float32, seed=0):
    return np.random.default_rng(seed).normal(0, scale, dims).astype(dtype)


@pytest.mark.parametrize("dims", [(2047,), (2048,), (2049,), (4095,), (4096,), (4097,), (65537,), (1, 1, 4097),
                                  (1, 300), (300, 1), (2, 3, 5), (1, 1), (33, 65), (513, 1025), (97, 33, 1),
                                  (1, 97, 161), (65, 65, 65), (129, 130, 131), (212, 213, 214), (5, 400, 401)])
def test_sizes(dims):
    if int(np.prod(dims)) == 1:
        pytest.skip("the reference aborts on one value")
    _check(_noise(dims, 4.0, seed=sum(dims)), 0.5)


@pytest.mark.parametrize("dims", [(65, 66, 67), (700, 700), (90000,)])
@pytest.mark.parametrize("bins,scale", [(16, 30.0), (4096, 3000.0), (8192, 9000.0), (65536, 20000.0)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_alphabets(dims, bins, scale, dtype):
    _check(_noise(dims, scale, dtype, seed=bins), 1.0, quantbinCnt=bins)


def test_codes_beyond_32_bits():
    """34 symbols with Fibonacci counts: codes of 33 bits."""
    fib = [1, 1]
    while len(fib) < 34:
        fib.append(fib[-1] + fib[-2])
    sym = np.repeat(np.arange(34), fib)
    np.random.default_rng(5).shuffle(sym)
    x = np.zeros(2 * sym.size + 1, np.float32)
    x[1::2] = 2.0 * sym
    _check(x, 1.0, interpAlgo=F.INTERP_ALGO_LINEAR)


@pytest.mark.parametrize("n", [12000000, 14500000])
def test_sliced_copy(n):
    """About 9.3 bits a value: 14 and 17 MB."""
    _check(np.random.default_rng(n).uniform(-500, 500, n).astype(np.float32), 1.0)
