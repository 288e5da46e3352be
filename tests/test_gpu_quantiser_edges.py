"""The quantiser and the stencils where their exact shortcuts meet edges:
differences on odd multiples of the bound, zeros of both signs (negative
differences of half index 0, stencil sums of 0), denormals, values far beyond
the code range and powers of two, for float and double data and both
interpolators.  Payloads are bytes and decoded fields bit patterns, so the
comparison with the oracle is for equality."""
import numpy as np
import pytest

import faz_gb300 as F
from conftest import mask_first_size

import oracle.oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def system_zstd():
    O.set_zstd(None)
    yield


def _edge_field(dims, dtype, seed):
    rng = np.random.default_rng(seed)
    eb = 2.0 ** -5
    x = rng.integers(-6, 7, dims) * eb                      # odd multiples of eb
    m = rng.random(dims)
    x = np.where(m < 0.25, 0.0, x)
    x = np.where((m >= 0.25) & (m < 0.45), -0.0, x)
    x = np.where((m >= 0.45) & (m < 0.5), -1e-310 if dtype == np.float64 else -1e-40, x)
    x = np.where((m >= 0.5) & (m < 0.52), 2.0 ** rng.integers(-8, 20, dims), x)
    x = np.where((m >= 0.52) & (m < 0.54), 1e30, x)
    x = np.where((m >= 0.54) & (m < 0.56), np.nextafter(dtype(eb), dtype(0)), x)
    return np.ascontiguousarray(x.astype(dtype)), eb


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("interp", [F.INTERP_ALGO_LINEAR, F.INTERP_ALGO_CUBIC])
@pytest.mark.parametrize("dims", [(40, 36, 44), (67, 130), (33, 35, 37)])
def test_quantiser_edges_match_oracle(dims, interp, dtype):
    x, eb = _edge_field(dims, dtype, sum(dims))
    conf = F.Config(*dims)
    conf.cmprAlgo, conf.interpAlgo = F.ALGO_INTERP, interp
    conf.errorBoundMode, conf.absErrorBound = F.EB_ABS, eb
    s = F.SZ_compress(conf, x)
    ref, _ = O.compress(conf, x)
    assert mask_first_size(s) == mask_first_size(ref)
    got, _ = F.SZ_decompress(None, s, dtype=dtype)
    want, _ = O.decompress(ref, dtype=dtype)
    assert got.tobytes() == want.tobytes()
