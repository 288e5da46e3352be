"""The Huffman decoder where its passes meet edges: strings of one unit and of
one unit more than a CTA's, short and long units (the rule is the string's
length), codewords beyond both lookup tables (up to 40 bits), a codeword repeated
over many units (which a decode started between two of them never falls in step
with), one symbol alone, and unpredictable values at the ends of the ranges they
are counted in.  Decoded fields are compared with the oracle's bit for bit."""
import numpy as np
import pytest

import faz_gb300 as F

import oracle.oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def system_zstd():
    O.set_zstd(None)
    yield


def _round_trip(x, eb, **kw):
    conf = F.Config(*x.shape)
    conf.cmprAlgo, conf.errorBoundMode, conf.absErrorBound = F.ALGO_INTERP, F.EB_ABS, eb
    for k, v in kw.items():
        setattr(conf, k, v)
    s = F.SZ_compress(conf, x)
    got, c = F.SZ_decompress(None, s, dtype=x.dtype)
    want, _ = O.decompress(s, dtype=x.dtype)
    assert got.tobytes() == want.tobytes()
    assert np.abs(got.astype(np.float64) - x.astype(np.float64)).max() <= eb


# noise of +-7 bounds: about 3 bits a value, so the bit strings cross the ends of
# units (160 and 544 bits), CTAs (256 units) and the rule's 2^25 bits
@pytest.mark.parametrize("n", [2, 40, 53, 54, 55, 13600, 13700, 27400, 400000, 11000000, 12500000])
def test_string_lengths(n):
    rng = np.random.default_rng(n)
    _round_trip(rng.uniform(-7, 7, n).astype(np.float32), 1.0)


def test_long_codewords():
    """Counts in Fibonacci proportion give a tree as deep as its symbols are many."""
    fib = [1, 1]
    while len(fib) < 27:
        fib.append(fib[-1] + fib[-2])
    sym = np.repeat(np.arange(27), fib)
    np.random.default_rng(5).shuffle(sym)
    n = sym.size
    # linear prediction of a field whose even points are zero: every other value codes itself
    x = np.zeros(2 * n + 1, np.float32)
    x[1::2] = 2.0 * sym
    _round_trip(x, 1.0, interpAlgo=F.INTERP_ALGO_LINEAR, interpBlockSize=32)


@pytest.mark.parametrize("dims,step", [((200, 190, 180), 4), ((700, 900), 8)])
def test_repeated_codeword(dims, step):
    rng = np.random.default_rng(1)
    x = rng.normal(0, 3, dims).astype(np.float64)
    _round_trip(x, 1.0, maxStep=step, alpha=1.5, beta=2.0)


@pytest.mark.parametrize("value", [0.0, 3.5])
def test_constant_field(value):
    _round_trip(np.full((70, 60, 50), value, np.float32), 0.25)


@pytest.mark.parametrize("every", [1, 2, 8192, 4099])
def test_unpredictable_positions(every):
    x = np.zeros((90, 80, 70), np.float32)
    x.reshape(-1)[::every] = np.linspace(1e9, 2e9, x.reshape(-1)[::every].size)
    _round_trip(x, 1e-3)
