"""The calls whose time is measured: fields compressed to their payload on the
GPU, payloads decoded on the GPU, and whole calls from a host array to a
stream and back.

A payload is what the compressor hands to zstd (compress_payload_device /
decompress_payload_device): the path that runs on the GPU, with the payload
copied to or from the caller's pinned memory.  Whole calls (SZ_compress,
SZ_decompress) add the host copies and the host zstd frame.  Fields are seeded
spectral Gaussian fields (power law, anisotropy, white noise) on [-50, 80].
"""
import math

import numpy as np
import torch

import faz_gb300 as F

ALGOS = {"interp": F.ALGO_INTERP, "default": F.ALGO_INTERP_LORENZO, "qoz": F.ALGO_INTERP_LORENZO,
         "lorenzo": F.ALGO_LORENZO_REG}


def _case(op, dims, dtype="f32", rel=1e-3, algo="interp", linear=False, direction=0, anchors=False, slope=-3.0,
          noise=0.01, name=None):
    c = {"op": op, "dims": "x".join(str(d) for d in dims), "dtype": dtype, "rel": rel, "algo": algo,
         "linear": linear, "direction": direction, "anchors": anchors, "slope": slope, "noise": noise}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the repository's benchmark field, plain cubic interpolation: the compressor alone, both directions
        _case("compress", (512, 512, 512), slope=-3.5, name="compress_512_f32"),
        _case("decompress", (512, 512, 512), slope=-3.5, name="decompress_512_f32"),
        # the same field as a caller who sets nothing compresses it: the default sampled autotune, then the choice
        _case("compress", (512, 512, 512), algo="default", slope=-3.5, name="compress_512_f32_default"),
        # float64 simulation output at a tight and a usual bound, in the configuration a QoZ-tuned user keeps
        # (anchor grid, per-level lists, alpha / beta)
        _case("compress", (256, 384, 384), "f64", 1e-6, anchors=True, noise=0.0, name="compress_256x384x384_f64"),
        _case("decompress", (256, 384, 384), "f64", 1e-4, anchors=True, noise=0.0,
              name="decompress_256x384x384_f64"),
        # 2-D climate fields: high resolution in, a quarter-degree grid (odd extent, loose bound, linear) out
        _case("compress", (1800, 3600), name="compress_1800x3600_f32"),
        _case("decompress", (721, 1440), rel=1e-2, linear=True, name="decompress_721x1440_f32"),
        # the smallest calls: one ragged tile of a domain decomposition, where latency and launches count
        _case("compress", (33, 47, 61), direction=5, name="compress_33x47x61_f32"),
        _case("decompress", (33, 47, 61), direction=5, name="decompress_33x47x61_f32"),
        # a 100x500x500 weather field through the Lorenzo / regression compressor, and its stream back to a host array
        _case("compress", (100, 500, 500), algo="lorenzo", name="compress_100x500x500_lorenzo"),
        _case("stream_decompress", (100, 500, 500), algo="lorenzo", name="stream_decompress_100x500x500_lorenzo"),
        # the drop-in call from a host array to a stream with the QoZ autotune (the tool's -q)
        _case("stream_compress", (256, 256, 256), algo="qoz", name="stream_compress_256_qoz"),
    ]


def _extents(rng, lo, hi, ndim, least):
    """ndim extents whose product is log-uniform in [lo, hi], none below
    `least`, aspect ratios up to about 4, odd values among them."""
    while True:
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        w = [math.exp(rng.uniform(-0.7, 0.7)) for _ in range(ndim)]
        g = (n / math.prod(w)) ** (1.0 / ndim)
        d = [max(least, round(g * v)) for v in w]
        if rng.random() < 0.3:  # sizes as programs allocate them
            d = [max(least, 16 * round(v / 16)) for v in d]
        if math.prod(d) <= hi:
            return d


def draw(rng):
    def bound(lo, hi):
        return float("%.2g" % math.exp(rng.uniform(math.log(lo), math.log(hi))))

    field = {"slope": round(rng.uniform(-4.0, -2.5), 2), "noise": rng.choice([0.0, 0.01, 0.02])}
    how = {"linear": rng.random() < 0.35}
    kind = rng.choice(["f32", "f32", "f32", "f64", "2d", "2d", "default", "lorenzo", "qoz"])
    op = rng.choice(["compress", "decompress"])
    if kind == "f32":
        return _case(op, _extents(rng, 8e4, 1.3e8, 3, 24), "f32", bound(1e-5, 1e-2), direction=rng.randrange(6),
                     **how, **field)
    if kind == "f64":
        return _case(op, _extents(rng, 3e5, 3.7e7, 3, 40), "f64", bound(1e-6, 1e-3), anchors=rng.random() < 0.6,
                     direction=rng.choice([0, 5]), **how, **field)
    if kind == "2d":
        return _case(op, _extents(rng, 4e4, 6.5e6, 2, 100), "f32", bound(1e-4, 1e-2), direction=rng.randrange(2),
                     **how, **field)
    if kind == "default":
        return _case("compress", _extents(rng, 5e5, 1.3e8, 3, 64), "f32", bound(1e-4, 1e-2), "default", **field)
    if kind == "lorenzo":
        return _case("compress" if op == "compress" else "stream_decompress", _extents(rng, 2e5, 2.5e7, 3, 32), "f32",
                     bound(1e-4, 1e-2), "lorenzo", **field)
    return _case("stream_compress", _extents(rng, 5e5, 1e7, 3, 64), "f32", bound(1e-3, 1e-2), "qoz", **field)


def _dims(case):
    return tuple(int(d) for d in case["dims"].split("x"))


def _field(case, seed):
    """Spectral Gaussian field: white noise filtered by |k|^(slope/2) with
    correlation lengths 1, 2, 4 along the axes, plus white noise."""
    shape = _dims(case)
    g = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7fffffff)
    spec = torch.fft.rfftn(torch.randn(shape, generator=g, device="cuda"))
    k2 = torch.zeros((), device="cuda")
    for ax, n in enumerate(shape):
        last = ax == len(shape) - 1
        f = (torch.fft.rfftfreq(n, device="cuda") if last else torch.fft.fftfreq(n, device="cuda")) * float(1 << ax)
        k2 = k2 + (f * f).reshape([-1 if i == ax else 1 for i in range(len(shape))])
    k2.view(-1)[0] = 1.0
    amp = k2.pow(case["slope"] / 4.0)
    amp.view(-1)[0] = 0.0
    x = torch.fft.irfftn(spec * amp, s=shape, dim=tuple(range(len(shape))))
    if case["noise"] > 0:
        x = x + torch.randn(shape, generator=g, device="cuda") * (case["noise"] * x.std())
    x = x.to(torch.float64 if case["dtype"] == "f64" else torch.float32)
    lo, hi = x.min(), x.max()
    return ((x - lo) / (hi - lo) * 130.0 - 50.0).contiguous()


def _conf(case):
    c = F.Config(*_dims(case))
    c.cmprAlgo = ALGOS[case["algo"]]
    c.errorBoundMode, c.relErrorBound = F.EB_REL, case["rel"]
    if case["algo"] == "qoz":
        c.QoZ = 1
    if case["algo"] == "interp":
        c.interpAlgo = F.INTERP_ALGO_LINEAR if case["linear"] else F.INTERP_ALGO_CUBIC
        c.interpDirection = case["direction"]
        if case["anchors"]:  # what the QoZ tuner typically settles on
            c.maxStep, c.alpha, c.beta = 32, 1.5, 2.0
            c.interpAlgo_list = [c.interpAlgo] * 4
            c.interpDirection_list = [case["direction"]] * 4
    return c


def prepare(case, seed):
    x, conf = _field(case, seed), _conf(case)
    s = {"op": case["op"], "conf": conf, "N": len(_dims(case)),
         "dtype": np.float64 if case["dtype"] == "f64" else np.float32}
    if case["op"] == "compress":
        s["x"] = x
        s["buf"] = torch.zeros(x.numel() * x.element_size() + (1 << 20), dtype=torch.uint8, pin_memory=True)
    elif case["op"] == "decompress":
        pl, _ = F.compress_payload_device(conf, x)
        s["payload"] = torch.empty(len(pl), dtype=torch.uint8, pin_memory=True)
        s["payload"].numpy()[:] = np.frombuffer(pl, dtype=np.uint8)
        s["out"] = torch.empty_like(x)
    elif case["op"] == "stream_compress":
        s["host"] = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
        s["host"].copy_(x)
        s["file"] = np.zeros(x.numel() * x.element_size() + (1 << 20), dtype=np.uint8)
    else:
        s["stream"] = F.compress_device(conf, x)
        s["host"] = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
    return s


def run(state):
    op = state["op"]
    if op == "compress":
        payload, _ = F.compress_payload_device(state["conf"], state["x"], out=state["buf"])
        return {"size": len(payload), "payload": state["buf"]}
    if op == "decompress":
        F.decompress_payload_device(state["N"], memoryview(state["payload"].numpy()), state["out"])
        return state["out"]
    if op == "stream_compress":
        stream = F.SZ_compress(state["conf"], state["host"].numpy())
        state["file"][:len(stream)] = np.frombuffer(stream, dtype=np.uint8)  # as a writer's buffer takes it
        return {"size": len(stream), "stream": state["file"]}
    out, _ = F.SZ_decompress(None, state["stream"], dtype=state["dtype"], out=state["host"].numpy())
    return out


def work(case):
    """The field's bytes once (read or written); the payload's, a fraction of
    them that depends on the field, are not counted."""
    n = math.prod(_dims(case))
    return {"bytes": n * (8 if case["dtype"] == "f64" else 4), "flops": 0}


def exact(case, seed):
    """A decoded field stands for the field that was compressed.  Payloads and
    streams are bytes and have no such value."""
    if case["op"] not in ("decompress", "stream_decompress"):
        return None
    return _field(case, seed).double()
