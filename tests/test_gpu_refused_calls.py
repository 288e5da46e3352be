"""A payload buffer that is too small: the call refuses it, writes nothing, and
leaves no work behind that a call on another stream could meet."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import faz_gb300 as F
from faz_gb300.api import FAZ_FLOAT, library
from faz_gb300.config import FazConfigStruct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", [F.ALGO_INTERP, F.ALGO_LORENZO_REG])
def test_small_buffer(algo):
    """17 MB of bits, packed in slices by the interpolation compressor."""
    dims = (145, 316, 317)
    rng = np.random.default_rng(1)
    x = torch.from_numpy(rng.uniform(-500, 500, dims).astype(np.float32)).cuda()
    conf = F.Config(*dims)
    conf.cmprAlgo, conf.errorBoundMode, conf.absErrorBound = algo, F.EB_ABS, 1.0
    want = bytes(F.compress_payload_device(conf, x)[0])
    assert len(want) > 16 << 20
    small = torch.full((1 << 20,), 7, dtype=torch.uint8, pin_memory=True)
    size, tm = ctypes.c_size_t(), F.api.FazTimings()
    for _ in range(5):
        a, b = torch.cuda.Stream(), torch.cuda.Stream()
        torch.cuda.synchronize()
        rc = library().faz_compress_device_payload(
            ctypes.byref(conf.to_struct()), FAZ_FLOAT, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(a.cuda_stream),
            ctypes.c_void_p(small.data_ptr()), small.numel(), ctypes.byref(size), ctypes.byref(FazConfigStruct()),
            ctypes.byref(tm))
        assert a.query()
        assert rc == -1 and size.value == len(want)
        assert bool((small == 7).all())
        assert bytes(F.compress_payload_device(conf, x, stream=b)[0]) == want
