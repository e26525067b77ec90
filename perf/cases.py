"""The work that users of this codec have it do, as cases of one call (or one
round trip) each, over the range of sizes and options in use.

A case names its kind and its sizes; prepare() makes the inputs on the GPU from
the seed, and what a program keeps between calls (an instance, a volume batch,
output buffers); run() is one pass through the public entry points.

Inputs: float volumes are Gaussian fields with a k^(-5/3) amplitude spectrum,
unit standard deviation (the statistics of turbulence_field); heightfields are
fractal terrain of 12 bits and more; images are smooth RGB(A) pictures with
noise; symbol streams are quantized-coefficient-like (zero runs, geometric
magnitudes).  Quantization steps span the benchmark's range, 0.002 (bricks) or 0.003 to 0.05 std.
"""
import math
import random

import torch

import cudacompress_b200 as cc
from cudacompress_b200 import image as ci


def listed():
    return [
        # one brick of a streamed volume, the smallest edge served: latency and launches
        dict(name="brick-32-encode", kind="volume_encode", nx=32, ny=32, nz=32, levels=2, q0=0.01),
        # one uneven brick on its way to a renderer
        dict(name="brick-uneven-decode", kind="volume_decode", nx=64, ny=48, nz=24, levels=2, q0=0.01, channels=1),
        # an ordinary volume, one call
        dict(name="volume-128-encode", kind="volume_encode", nx=128, ny=128, nz=128, levels=3, q0=0.01),
        # the three components of a ragged vector field, one multi-channel call
        dict(name="vector-ragged-decode", kind="volume_decode", nx=200, ny=136, nz=88, levels=3, q0=0.01, channels=3),
        # a large component at the finest quantization in use: the largest code tables
        dict(name="volume-256-fine-encode", kind="volume_encode", nx=256, ny=256, nz=256, levels=3, q0=0.003),
        # the flagship workload, each direction: three 256^3 components as one batch
        dict(name="vector-256-encode", kind="batch_encode", nx=256, ny=256, nz=256, levels=3, q0=0.01, count=3),
        dict(name="vector-256-decode", kind="batch_decode", nx=256, ny=256, nz=256, levels=3, q0=0.01, count=3),
        # a bricked volume: thousands of uneven bricks, each with its own step, one batch there and back
        dict(name="bricks-4096", kind="bricks", count=4096, levels=2),
        # lossless terrain, there and back
        dict(name="heightfield-2048", kind="heightfield", nx=2048, ny=2048, levels=4),
        # one level of an image pyramid, there and back
        dict(name="image-1024", kind="image", nx=1024, ny=768, channels=3, q0=4.0),
        # the entropy coder alone on a caller's own symbols (odd count), there and back through a host bit stream
        dict(name="streams-rlhuff", kind="streams", count=7, n=100003, bits=16),
        # the transform alone, there and back
        dict(name="dwt-float-256", kind="dwt", nx=256, ny=256, nz=256, dtype="float32"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _size(rng, lo, hi, step):
    return max(lo, int(_log(rng, lo, hi)) // step * step)


def draw(rng):
    kind = rng.choice(["volume_encode", "volume_decode", "batch_encode", "batch_decode", "bricks", "heightfield",
                       "image", "streams", "dwt"])
    if kind in ("volume_encode", "volume_decode", "batch_encode", "batch_decode"):
        levels = rng.choice([1, 2, 2, 3, 3])
        f = 1 << levels
        lo = 32
        c = dict(kind=kind, levels=levels, q0=round(_log(rng, 0.003, 0.05), 5))
        for k in ("nx", "ny", "nz"):
            c[k] = _size(rng, lo, 200 if kind == "volume_decode" else 250, f)
        if kind == "volume_decode":
            c["channels"] = rng.choice([1, 1, 2, 3])
        if kind.startswith("batch"):
            c["count"] = rng.choice([1, 2, 3, 4])
        return c
    if kind == "bricks":
        return dict(kind=kind, count=int(_log(rng, 32, 3000)), levels=2)
    if kind == "heightfield":
        levels = rng.choice([1, 2, 3, 4])
        return dict(kind=kind, nx=_size(rng, 256, 2048, 64), ny=_size(rng, 256, 2048, 64), levels=levels)
    if kind == "image":
        return dict(kind=kind, nx=_size(rng, 128, 1500, 2), ny=_size(rng, 128, 1500, 2), channels=rng.choice([3, 4]),
                    q0=round(_log(rng, 1.0, 16.0), 3))
    if kind == "streams":
        return dict(kind=kind, count=rng.choice([1, 3, 7, 14]), n=int(_log(rng, 1000, 400000)) | 1,
                    bits=rng.choice([16, 16, 32]))
    if rng.random() < 0.5:
        return dict(kind=kind, nx=_size(rng, 32, 250, 2), ny=_size(rng, 32, 250, 2), nz=_size(rng, 32, 250, 2),
                    dtype=rng.choice(["float32", "float32", "int16"]))
    return dict(kind=kind, nx=_size(rng, 256, 4000, 64), ny=_size(rng, 256, 4000, 64), nz=1,
                dtype=rng.choice(["float32", "int16"]))


# ------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _field(n, g):
    """n^3 float32 field, zero mean, unit std, amplitudes |k|^(-5/3) for 1 <= |k| <= n / 4."""
    k = torch.fft.fftfreq(n, 1.0 / n, device="cuda")
    r = torch.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, : n // 2 + 1] ** 2)
    amp = torch.where((r >= 1.0) & (r <= n / 4), r.clamp(min=1.0) ** (-5.0 / 3.0), torch.zeros_like(r))
    noise = torch.randn(n, n, n // 2 + 1, 2, device="cuda", generator=g)
    f = torch.fft.irfftn(torch.view_as_complex(noise) * amp, s=(n, n, n))
    return (f - f.mean()) / f.std()


def _volume(nx, ny, nz, g):
    n = max(nx, ny, nz)
    n += -n % 8
    return _field(n, g)[:nz, :ny, :nx].contiguous()


def _terrain(nx, ny, g):
    """int16 fractal terrain over -2000 .. 8000 m: octaves of smoothly interpolated lattice noise."""
    acc = torch.zeros(ny, nx, dtype=torch.float64, device="cuda")
    n = max(nx, ny)
    for o in range(10):
        cells = 2 << o
        lat = torch.rand(cells + 1, cells + 1, dtype=torch.float64, device="cuda", generator=g) * 2 - 1

        def axis(m):
            t = torch.arange(m, dtype=torch.float64, device="cuda") * cells / n
            i = t.floor().long()
            f = t - i
            return i, f * f * (3 - 2 * f)

        (iy, fy), (ix, fx) = axis(ny), axis(nx)
        fy, fx = fy[:, None], fx[None, :]
        top = lat[iy[:, None], ix[None, :]] * (1 - fx) + lat[iy[:, None], ix[None, :] + 1] * fx
        bot = lat[iy[:, None] + 1, ix[None, :]] * (1 - fx) + lat[iy[:, None] + 1, ix[None, :] + 1] * fx
        acc += 2.0 ** (-0.8 * o) * (top * (1 - fy) + bot * fy)
    acc = (acc - acc.min()) / (acc.max() - acc.min())
    return torch.round(-2000 + 10000 * acc).to(torch.int16)


def _picture(nx, ny, channels, g):
    """uint8 picture: smooth waves per channel with sensor-like noise."""
    y = torch.arange(ny, device="cuda", dtype=torch.float32)[:, None]
    x = torch.arange(nx, device="cuda", dtype=torch.float32)[None, :]
    out = torch.empty(ny, nx, channels, dtype=torch.uint8, device="cuda")
    for c in range(channels):
        k = torch.rand(4, device="cuda", generator=g) * 0.12 + 0.01
        v = 128 + 70 * torch.sin(k[0] * x + k[1] * y) + 35 * torch.cos(k[2] * x - k[3] * y)
        v = v + 4 * torch.randn(ny, nx, device="cuda", generator=g)
        out[..., c] = v.round().clamp(0, 255).to(torch.uint8)
    return out


def _symbols(n, bits, density, g):
    """Symbols as a deadzone quantizer leaves them: mostly 0, geometric magnitudes."""
    u = torch.rand(n, device="cuda", generator=g)
    mag = 1 + torch.floor(-torch.log(torch.rand(n, device="cuda", generator=g).clamp(min=1e-7)) * 3.0)
    s = torch.where(u < density, mag, torch.zeros_like(mag))
    return s.to(torch.int16 if bits == 16 else torch.int32)


def _bricks(count, g):
    """Uneven bricks (edges 16 .. 64 per axis) cut from four fields, a log-uniform step each."""
    n = 256 if count > 512 else 128
    src = [_field(n, g) for _ in range(4)]
    r = torch.rand(count, 8, generator=g, device="cuda").tolist()
    shape = random.Random(count)                        # the bricking is the data set's, not the field's
    bricks, steps = [], []
    for u in r:
        ex, ey, ez = (shape.choice((16, 24, 32, 48, 64)) for _ in range(3))
        ox, oy, oz = int(u[3] * (n - ex)), int(u[4] * (n - ey)), int(u[5] * (n - ez))
        bricks.append(src[min(3, int(u[6] * 4))][oz:oz + ez, oy:oy + ey, ox:ox + ex].contiguous())
        steps.append(math.exp(math.log(0.002) + u[7] * math.log(25.0)))
    return bricks, steps


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    g = _gen(seed)
    s = dict(case)
    kind = case["kind"]
    if kind in ("volume_encode", "volume_decode"):
        nx, ny, nz, L, q0 = (case[k] for k in ("nx", "ny", "nz", "levels", "q0"))
        ch = case.get("channels", 1)
        s["inst"] = cc.Instance(0, 7 * ch, (nx // 2) * (ny // 2) * (nz // 2), 128, 14)
        vols = [_volume(nx, ny, nz, g) for _ in range(ch)]
        cap = cc.volume_stream_capacity_words(nx, ny, nz)
        words = [torch.zeros(cap, dtype=torch.int32, device="cuda") for _ in range(ch)]
        if kind == "volume_encode":
            s["volume"], s["words"] = vols[0], words[0]
        else:
            s["bits"] = [cc.compress_volume_float(s["inst"], v, L, q0, w)[1] for v, w in zip(vols, words)]
            s["words"] = words
            s["outs"] = torch.empty(ch, nz, ny, nx, device="cuda")
    elif kind in ("batch_encode", "batch_decode", "bricks"):
        if kind == "bricks":
            s["volumes"], steps = _bricks(case["count"], g)
        else:
            s["volumes"] = [_volume(case["nx"], case["ny"], case["nz"], g) for _ in range(case["count"])]
            steps = [case["q0"]] * case["count"]
        s["inst"] = cc.Instance(0, 7, 1 << 12, 64 if kind == "bricks" else 128, 14)
        s["batch"] = cc.VolumeBatch(s["inst"], [v.shape for v in s["volumes"]], case["levels"], steps, graph=True)
        total = sum(v.numel() for v in s["volumes"])
        if kind == "batch_encode":
            s["host_words"] = torch.zeros(total // 2 + 65536, dtype=torch.int32).pin_memory()
            s["host_extents"] = torch.zeros(2 * len(s["volumes"]), dtype=torch.int64).pin_memory()
        else:
            s["out"] = torch.empty(total, device="cuda")
            at, s["outs"] = 0, []
            for v in s["volumes"]:
                s["outs"].append(s["out"][at:at + v.numel()].view(v.shape))
                at += v.numel()
            if kind == "batch_decode":
                s["batch"].compress(s["volumes"])
                s["batch"].status()
    elif kind == "heightfield":
        nx, ny = case["nx"], case["ny"]
        s["image"] = _terrain(nx, ny, g)
        s["inst"] = cc.Instance(0, 5, (nx // 2) * (ny // 2), 128, 14)
        s["words"] = torch.zeros(nx * ny + 64 * 1024, dtype=torch.int32, device="cuda")
        s["out"] = torch.empty_like(s["image"])
    elif kind == "image":
        nx, ny, ch = case["nx"], case["ny"], case["channels"]
        s["image"] = _picture(nx, ny, ch, g)
        s["lowpass"] = ci.get_lowpass_image(s["image"], ch)
        s["inst"] = cc.Instance(0, 4 * ch, (nx // 2) * (ny // 2), 128, 14)
        s["words"] = torch.zeros(ci.image_stream_capacity_words(nx, ny, ch), dtype=torch.int32, device="cuda")
        s["coded"], s["out"] = torch.empty_like(s["image"]), torch.empty_like(s["image"])
    elif kind == "streams":
        n, count = case["n"], case["count"]
        s["inst"] = cc.Instance(0, count, n, 128, 14 if case["bits"] == 16 else 18)
        pitch = n + -n % 64
        flat = torch.zeros(count, pitch, dtype=torch.int16 if case["bits"] == 16 else torch.int32, device="cuda")
        for i in range(count):
            flat[i, :n] = _symbols(n, case["bits"], 0.05 + 0.6 * (i + 1) / count, g)
        s["symbols"] = [flat[i, :n] for i in range(count)]
        s["out"] = torch.empty_like(flat).zero_()
        s["outs"] = [s["out"][i, :n] for i in range(count)]
    elif kind == "dwt":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        if case["dtype"] == "float32":
            src = _volume(nx, ny, nz, g) if nz > 1 else (_terrain(nx, ny, g).float() / 1000.0)[None].contiguous()
        else:
            src = (_volume(nx, ny, nz, g) * 1000).to(torch.int16) if nz > 1 else _terrain(nx, ny, g)[None].contiguous()
        s["src"] = src
        for k in ("coef", "back", "buf1", "buf2"):
            s[k] = torch.empty_like(src)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "volume_encode":
        words, bits = cc.compress_volume_float(s["inst"], s["volume"], s["levels"], s["q0"], s["words"])
        return [words, bits]
    if kind == "volume_decode":
        if len(s["outs"]) == 1:
            cc.decompress_volume_float(s["inst"], s["outs"][0], s["levels"], s["q0"], s["words"][0], s["bits"][0])
        else:
            cc.decompress_volume_float_multichannel(s["inst"], list(s["outs"]), s["words"], s["bits"],
                                                    [s["q0"]] * len(s["outs"]), s["levels"])
        return s["outs"]
    if kind == "batch_encode":
        s["batch"].compress(s["volumes"])
        s["batch"].download_streams(s["host_words"], s["host_extents"])
        return [s["host_words"], s["host_extents"]]
    if kind == "batch_decode":
        s["batch"].decompress(s["outs"])
        return s["out"]
    if kind == "bricks":
        s["batch"].compress(s["volumes"])
        s["batch"].decompress(s["outs"])
        return s["out"]
    if kind == "heightfield":
        words, bits = cc.compress_heightfield(s["inst"], s["image"], s["levels"], s["words"])
        cc.decompress_heightfield(s["inst"], s["out"], s["levels"], words, bits)
        return [words, bits, s["out"]]
    if kind == "image":
        # compressing leaves the reconstruction in its argument
        ch = s["channels"]
        s["coded"].copy_(s["image"])
        words, bits = ci.compress_image_one_level(s["inst"], s["coded"], ch, s["lowpass"], s["q0"], s["words"])
        ci.decompress_image_one_level(s["inst"], s["out"], ch, s["lowpass"], s["q0"], words, bits)
        return [words, bits, s["coded"], s["out"]]
    if kind == "streams":
        bs = cc.BitStream()
        ok = cc.encode_rlhuff(s["inst"], bs, s["symbols"], s["n"])
        bs.set_bit_position(0)
        ok = cc.decode_rlhuff(s["inst"], bs, s["outs"], s["n"]) and ok
        return [bool(ok), bs.words, bs.bit_size, s["out"]]
    nx, ny, nz = s["nx"], s["ny"], s["nz"]
    if s["dtype"] == "float32":
        cc.dwt_float_forward(s["coef"], s["buf2"], s["buf1"], s["src"], nx, ny, nz)
        cc.dwt_float_inverse(s["back"], s["buf2"], s["buf1"], s["coef"], nx, ny, nz)
    else:
        cc.dwt_int_forward(s["coef"], s["buf1"], s["src"], nx, ny, nz)
        cc.dwt_int_inverse(s["back"], s["buf1"], s["coef"], nx, ny, nz)
    return [s["coef"], s["back"]]


# --------------------------------------------------------------------- work
def work(case):
    """Raw samples and coded bytes, each in and out once (an estimate of the coded size stands for it)."""
    kind = case["kind"]
    if kind in ("volume_encode", "volume_decode", "batch_encode", "batch_decode"):
        raw = 4.0 * case["nx"] * case["ny"] * case["nz"] * case.get("channels", 1) * case.get("count", 1)
        return {"bytes": raw * 1.1, "flops": raw / 4 * 54 * 8 / 7}     # 9 taps x 3 axes x 2, all levels
    if kind == "bricks":
        raw = 4.0 * 36.8 ** 3 * case["count"]
        return {"bytes": 2 * raw * 1.1, "flops": 2 * raw / 4 * 54 * 8 / 7}
    if kind == "heightfield":
        raw = 2.0 * case["nx"] * case["ny"]
        return {"bytes": 2 * raw * 1.3, "flops": 0.0}
    if kind == "image":
        raw = 1.0 * case["nx"] * case["ny"] * case["channels"]
        return {"bytes": raw * (1 + 0.25 + 1 + 1.25 + 0.5), "flops": 3 * raw * 36}
    if kind == "streams":
        raw = case["bits"] / 8.0 * case["n"] * case["count"]
        return {"bytes": 2 * raw * 1.3, "flops": 0.0}
    n = case["nx"] * case["ny"] * case["nz"]
    axes = 3 if case["nz"] > 1 else 2
    if case["dtype"] == "float32":
        return {"bytes": 16.0 * n, "flops": 2.0 * n * 18 * axes}
    return {"bytes": 8.0 * n, "flops": 0.0}


# -------------------------------------------------------------------- exact
# CDF 9/7 analysis (even / odd output) and synthesis taps, centre tap index 4,
# as the codec's format fixes them (single-precision constants).
_ANALYSIS = [[0.0267488, -0.0168641, -0.0782233, 0.2668641, 0.6029490, 0.2668641, -0.0782233, -0.0168641, 0.0267488],
             [0.0, 0.0456359, -0.0287718, -0.2956359, 0.5575435, -0.2956359, -0.0287718, 0.0456359, 0.0]]
_SYNTHESIS = [[0.0, 0.0337282, -0.0575435, -0.5337281, 1.1150871, -0.5337281, -0.0575435, 0.0337282, 0.0],
              [0.0534975, -0.0912718, -0.1564465, 0.5912718, 1.2058980, 0.5912718, -0.1564465, -0.0912718, 0.0534975]]


def _axis64(a, dim, taps):
    """out[i] = sum_t taps[i & 1][t] * a[mirror(i + t - 4)] along dim, in 64 bits."""
    n = a.shape[dim]
    x = a.movedim(dim, -1)
    taps = torch.tensor(taps, dtype=torch.float32).double().to(a.device)
    i = torch.arange(n, device=a.device)
    out = torch.zeros_like(x)
    for t in range(9):
        j = (i + t - 4).abs()
        j = torch.where(j > n - 1, 2 * (n - 1) - j, j)
        out += x[..., j] * taps[i & 1, t]
    return out.movedim(-1, dim)


def exact(case, seed):
    """The float transform in 64 bits; the other outputs are integers, or depend on quantization decisions."""
    if case["kind"] != "dwt" or case["dtype"] != "float32":
        return None
    a = prepare(case, seed)["src"].double()
    dims = [2, 1, 0] if case["nz"] > 1 else [2, 1]
    coef = a
    for d in dims:
        v = _axis64(coef, d, _ANALYSIS).movedim(d, -1)
        coef = torch.cat([v[..., 0::2], v[..., 1::2]], -1).movedim(-1, d)
    back = coef
    for d in reversed(dims):
        v = back.movedim(d, -1)
        h = v.shape[-1] // 2
        back = _axis64(torch.stack([v[..., :h], v[..., h:]], -1).flatten(-2).movedim(-1, d), d, _SYNTHESIS)
    return [coef, back]
