"""The QoZ tuner's error sums (k_qz_line_sums, k_qz_sum in qoz.cu) on sampled
blocks of few and many lines: below one chunk of the chain kernel and across one
chunk's end, one block and several.  The sums decide the
interpolators, directions, alpha and beta, which the stream records: streams
equal the oracle's byte for byte."""
import numpy as np
import pytest

import faz_gb300 as F
from faz_gb300.fields import spectral_field
from conftest import mask_first_size

import oracle.oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def system_zstd():
    O.set_zstd(None)
    yield


CASES = [
    ((60, 70, 52), 16, 0.02, np.float32),     # 17^3: 767 lines and less
    ((100, 101, 99), 32, 0.1, np.float32),    # 33^3: 2.6 thousand
    ((100, 101, 99), 32, 0.1, np.float64),
    ((210, 333), 32, 0.2, np.float32),        # 33^2: a hundred
]


@pytest.mark.parametrize("dims,sbs,rate,dtype", CASES)
def test_sums_match_oracle(dims, sbs, rate, dtype):
    conf = F.Config(*dims)
    conf.QoZ = 1
    conf.errorBoundMode, conf.relErrorBound = F.EB_REL, 1e-3
    conf.sampleBlockSize = sbs
    conf.autoTuningRate = conf.predictorTuningRate = rate
    x = spectral_field(dims, slope=-3.0, noise=0.01, seed=sum(dims) + sbs, dtype=dtype)
    stream = F.SZ_compress(conf, x)
    ref, _ = O.compress(conf, x)
    assert mask_first_size(stream) == mask_first_size(ref)
