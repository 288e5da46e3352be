"""The Lorenzo wavefront's block paths against the oracle: edges with the fast
path (5 and 6) and without (1, 4, 8), fields of full blocks only, with clipped
blocks on every axis and of one block, regression and Lorenzo blocks side by side
(smooth ramps beside noise, so that neither kind fills the field), unpredictable
values inside fast blocks, float and double."""
import numpy as np
import pytest

import faz_gb300 as F
from conftest import mask_fast_frontend_padding

import oracle.oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def system_zstd():
    O.set_zstd(None)
    yield


def _field(dims, dtype, spikes, seed):
    rng = np.random.default_rng(seed)
    g = np.meshgrid(*[np.arange(n, dtype=np.float64) for n in dims], indexing="ij")
    ramp = 0.7 * g[0] - 0.4 * g[1] + 0.9 * g[2] + rng.normal(0, 0.4, dims)
    rough = 3 * np.sin(g[0] / 3) * np.cos(g[1] / 4 + g[2] / 5)
    x = np.where((g[0] // 11 + g[1] // 13 + g[2] // 17) % 2 == 0, ramp, rough)
    if spikes:
        x[rng.random(dims) < 0.01] *= 1e7
    return np.ascontiguousarray(x.astype(dtype))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("dims,bs,lo2", [((36, 42, 48), 6, 0), ((37, 44, 53), 6, 0), ((6, 6, 6), 6, 0),
                                         ((35, 40, 45), 5, 0), ((36, 41, 47), 5, 1), ((38, 43, 50), 6, 1),
                                         ((33, 34, 35), 8, 0), ((30, 31, 33), 4, 1), ((9, 10, 11), 1, 1)])
@pytest.mark.parametrize("spikes", [False, True])
def test_wavefront_blocks_match_oracle(dims, bs, lo2, dtype, spikes):
    x = _field(dims, dtype, spikes, sum(dims) + bs)
    conf = F.Config(*dims)
    conf.cmprAlgo, conf.blockSize, conf.lorenzo2 = F.ALGO_LORENZO_REG, bs, lo2
    conf.errorBoundMode, conf.absErrorBound = F.EB_ABS, 0.05
    s = F.SZ_compress(conf, x)
    ref, ref_payload = O.compress(conf, x)
    _, payload = O.read_stream(s)
    assert mask_fast_frontend_padding(payload, x.itemsize) == mask_fast_frontend_padding(ref_payload, x.itemsize)
    got, _ = F.SZ_decompress(None, s, dtype=dtype)
    want, _ = O.decompress(ref, dtype=dtype)
    assert got.tobytes() == want.tobytes()
