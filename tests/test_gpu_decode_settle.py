"""The Huffman decoder's second part: unit starts that the first passes leave wrong.
Three symbols, of one, two and two bits; one of the two-bit codewords repeats one bit
(11 or 00), so a decode that starts at its second bit never falls in step with a run of
it.  Runs longer than several CTAs' units, which begin at an odd bit, then take a link
pass for each CTA, and the codes, zero positions and levels are queued again.  The
fields are whole steps of the bound, which the compressors reproduce exactly; launches
beyond those of the same symbols in random order say that the part ran."""
import numpy as np
import pytest

import faz_gb300 as F

pytestmark = pytest.mark.gpu


def _launches(conf, x):
    s = F.SZ_compress(conf, x)
    got, _ = F.SZ_decompress(None, s, dtype=x.dtype)
    assert got.tobytes() == x.tobytes()
    return F.last_timings()["kernel_launches"]


def _extra(conf, make, symbols, rng):
    shuffled = symbols.copy()
    rng.shuffle(shuffled)
    return _launches(conf, make(symbols)) - _launches(conf, make(shuffled))


# units of 5 words (40,960 bits a CTA) and, from 2^25 bits on, of 17 (139,264)
@pytest.mark.parametrize("n,run", [(600001, 40000), (40000001, 300000)])
@pytest.mark.parametrize("unpredictable", [0, 37])
def test_interpolation(n, run, unpredictable):
    """The odd points, predicted as 0 from the even ones, are -2, 0 or 2 at a bound of 1;
    after `shift` points of 0 come the runs.  Of two neighbouring shifts one begins a
    run at an odd bit."""
    conf = F.Config(n)
    conf.cmprAlgo, conf.errorBoundMode, conf.absErrorBound = F.ALGO_INTERP, F.EB_ABS, 1.0
    conf.interpAlgo = F.INTERP_ALGO_LINEAR
    rng = np.random.default_rng(n)

    def make(symbols):
        x = np.zeros(n, np.float32)
        x[1::2] = symbols
        if unpredictable:  # in the codes, and so in the zero positions, on both sides of the runs
            x[1::2][:: symbols.size // unpredictable] = 1e9
        return x

    extra = []
    for shift in (1000, 1001):
        symbols = np.zeros(n // 2, np.float32)
        symbols[shift:shift + run] = 2.0
        symbols[shift + run:shift + 2 * run] = -2.0
        extra.append(_extra(conf, make, symbols, rng))
    assert max(extra) >= 2 * 2  # two link passes and their outcomes, at least


@pytest.mark.parametrize("block,bins", [(6, 65536), (4, 65536), (6, 131072)])
def test_lorenzo(block, bins):
    """The residuals of the one-layer predictor, by planes."""
    dims = (95, 101, 103)
    conf = F.Config(*dims)
    conf.cmprAlgo, conf.errorBoundMode, conf.absErrorBound = F.ALGO_LORENZO_REG, F.EB_ABS, 0.5
    conf.lorenzo, conf.lorenzo2, conf.regression, conf.regression2 = 1, 0, 0, 0
    conf.blockSize, conf.quantbinCnt = block, bins
    rng = np.random.default_rng(block)

    def make(symbols):
        x = symbols.reshape(dims)
        for axis in range(3):
            x = np.cumsum(x, axis=axis)
        assert np.abs(x).max() < 1 << 24
        return x.astype(np.float32)

    extra = []
    for shift in (24, 25):
        symbols = np.zeros(dims, np.int64)
        symbols[shift:shift + 24] = 1
        symbols[shift + 24:shift + 48] = -1
        extra.append(_extra(conf, make, symbols.reshape(-1), rng))
    assert max(extra) >= 2 * 2
