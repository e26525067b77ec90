"""Edges of the kernels' size, alignment and length rules, each against the
oracle, bit for bit: tile borders of the transform passes, sources and streams
at odd addresses, code words longer than the staged window, and symbol tables
on both sides of each builder's capacity."""
import numpy as np
import pytest

from helpers import Oracle, symbol_streams

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import cudacompress_b200 as cc  # noqa: E402
from cudacompress_b200 import fields  # noqa: E402


@pytest.fixture(scope="module")
def oracle():
    return Oracle()


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy()


def same(a, b):
    return a.shape == b.shape and np.ascontiguousarray(a).tobytes() == np.ascontiguousarray(b).tobytes()


def pitched(a, row, rows, shift):
    """A device copy of `a` (z, y, x) whose rows are `row` and slices
    `row * rows` elements apart, its first element `shift` past an aligned
    address.  Returns (view to pass on, function reading it back)."""
    nz, ny, nx = a.shape
    base = torch.zeros(nz * row * rows + shift, dtype=torch.from_numpy(a[:1, :1, :1]).dtype, device="cuda")
    view = base[shift:].view(nz, rows, row)
    view[:, :ny, :nx] = dev(a)
    return view, lambda: host(view[:, :ny, :nx])


# ------------------------------------------------------------- transforms
# The plane pass works on tiles of 64 x 64 outputs: one below, at and above a
# tile in x and y, the smallest level, several tiles, and the 2D form.
FLOAT_SHAPES = [(8, 8, 8), (8, 10, 12), (8, 62, 64), (10, 66, 62), (8, 64, 66), (12, 72, 136), (8, 8, 130), (8, 130, 8),
                (1, 8, 8), (1, 66, 130), (1, 128, 64), (66, 8, 10)]


@pytest.mark.parametrize("shape", FLOAT_SHAPES)
@pytest.mark.parametrize("pad,shift", [(0, 0), (1, 0), (2, 2), (4, 1)])
def test_float_transform_at_tile_edges(oracle, shape, pad, shift):
    """Both directions, with rows padded by `pad` elements and arrays starting
    `shift` elements past an aligned address."""
    rng = np.random.default_rng(sum(shape) + pad)
    a = rng.standard_normal(shape).astype(np.float32)
    nz, ny, nx = shape
    row, rows = nx + pad, ny + (1 if pad else 0)
    pitches = (row, row * rows, row, row * rows)
    zero = np.zeros_like(a)
    src, _ = pitched(a, row, rows, shift)
    dst, read = pitched(zero, row, rows, shift)
    b1, _ = pitched(zero, row, rows, shift)
    b2, _ = pitched(zero, row, rows, shift)
    cc.dwt_float_forward(dst, b2, b1, src, nx, ny, nz, 1, *pitches)
    fwd = read()
    assert same(fwd, oracle.dwt_float(a))
    back, read_back = pitched(zero, row, rows, shift)
    cc.dwt_float_inverse(back, b2, b1, dst, nx, ny, nz, 1, *pitches)
    assert same(read_back(), oracle.dwt_float(fwd, inverse=True))


@pytest.mark.parametrize("shape", [(1, 8, 8), (1, 66, 130), (1, 200, 72)])
def test_float_transform_in_place_2d(oracle, shape):
    """A 2D transform whose destination is its source: tiles overlap their
    neighbours' inputs, so it goes through the buffer."""
    rng = np.random.default_rng(3)
    a = rng.standard_normal(shape).astype(np.float32)
    _, ny, nx = shape
    t, b1, b2 = dev(a), dev(np.zeros_like(a)), dev(np.zeros_like(a))
    cc.dwt_float_forward(t, b2, b1, t, nx, ny, 1)
    fwd = host(t)
    assert same(fwd, oracle.dwt_float(a))
    cc.dwt_float_inverse(t, b2, b1, t, nx, ny, 1)
    assert same(host(t), oracle.dwt_float(fwd, inverse=True))


@pytest.mark.parametrize("shape", [(8, 8, 8), (10, 62, 130), (66, 72, 64)])
@pytest.mark.parametrize("alias", ["buf2=src", "buf2=dst"])
def test_float_transform_3d_aliases(oracle, shape, alias):
    """Arrays that a plane pass would read and write at once: the source in
    the second buffer (forward), the second buffer in the destination
    (inverse); X and Y then go through the first one."""
    rng = np.random.default_rng(sum(shape))
    a = rng.standard_normal(shape).astype(np.float32)
    nz, ny, nx = shape
    fwd = oracle.dwt_float(a)
    src, dst, b1 = dev(a), dev(np.zeros_like(a)), dev(np.zeros_like(a))
    if alias == "buf2=src":
        cc.dwt_float_forward(dst, src, b1, src, nx, ny, nz)
        assert same(host(dst), fwd)
    else:
        cc.dwt_float_inverse(dst, dst, b1, dev(fwd), nx, ny, nz)
        assert same(host(dst), oracle.dwt_float(fwd, inverse=True))


@pytest.mark.parametrize("shape", [(8, 8, 8), (1, 8, 8), (8, 10, 12), (1, 34, 66), (1, 66, 258), (10, 66, 34), (34, 8, 8),
                                   (1, 258, 520)])
@pytest.mark.parametrize("pad,shift", [(0, 0), (1, 1), (2, 2), (4, 4)])
def test_int_transform_at_tile_edges(oracle, shape, pad, shift):
    rng = np.random.default_rng(sum(shape) + pad)
    a = rng.integers(-2000, 8000, shape).astype(np.int16)
    nz, ny, nx = shape
    row, rows = nx + pad, ny + (1 if pad else 0)
    pitches = (row, row * rows, row, row * rows)
    zero = np.zeros_like(a)
    src, _ = pitched(a, row, rows, shift)
    dst, read = pitched(zero, row, rows, shift)
    buf, _ = pitched(zero, row, rows, shift)
    cc.dwt_int_forward(dst, buf, src, nx, ny, nz, *pitches)
    assert same(read(), oracle.dwt_int(a))
    back, read_back = pitched(zero, row, rows, shift)
    cc.dwt_int_inverse(back, buf, dst, nx, ny, nz, *pitches)
    assert same(read_back(), a)


@pytest.mark.parametrize("shape", [(8, 8, 8), (16, 10, 48), (64, 48, 64), (34, 66, 130), (1, 48, 64), (1, 64, 48), (1, 300, 520),
                                   (8, 8, 2000)])
@pytest.mark.parametrize("alias", ["dst=src", "buf=src", "dst=buf", "dst=buf=src"])
@pytest.mark.parametrize("pad", [0, 3])
def test_int_transform_in_place(oracle, shape, alias, pad):
    """A pass whose destination is its source stages whole lines: lines within
    and across a warp's eight-sample groups, a CTA's rows of pairs, and 32
    lines to a CTA or fewer."""
    rng = np.random.default_rng(sum(shape))
    a = rng.integers(-2000, 8000, shape).astype(np.int16)
    nz, ny, nx = shape
    row, rows = nx + pad, ny + (1 if pad else 0)
    pitches = (row, row * rows, row, row * rows)
    fwd = oracle.dwt_int(a)
    for run, given, expect in ((cc.dwt_int_forward, a, fwd), (cc.dwt_int_inverse, fwd, a)):
        src, read = pitched(given, row, rows, 0)
        dst, read_dst = (src, read) if "dst" in alias and "src" in alias else pitched(np.zeros_like(a), row, rows, 0)
        buf = {"dst=src": None, "buf=src": src, "dst=buf": dst, "dst=buf=src": src}[alias]
        if buf is None:
            buf, _ = pitched(np.zeros_like(a), row, rows, 0)
        run(dst, buf, src, nx, ny, nz, *pitches)
        assert same(read_dst(), expect)


def test_int_transform_of_a_very_tall_image(oracle):
    """More groups of pairs along Y than a grid has rows (65535)."""
    shape = (1, 2 * 8 * 65535 + 10, 8)
    a = np.random.default_rng(4).integers(-2000, 8000, shape).astype(np.int16)
    src, dst, buf, back = dev(a), dev(a * 0), dev(a * 0), dev(a * 0)
    cc.dwt_int_forward(dst, buf, src, shape[2], shape[1])
    assert same(host(dst), oracle.dwt_int(a))
    cc.dwt_int_inverse(back, buf, dst, shape[2], shape[1])
    assert same(host(back), a)


@pytest.mark.parametrize("shape,levels", [((20, 28), 1), ((16, 16), 1), ((40, 24), 2), ((64, 136), 2), ((66, 260), 1)])
def test_heightfield_sizes(oracle, shape, levels):
    """Band widths that are and are not multiples of four symbols."""
    img = np.ascontiguousarray(fields.fbm_heightfield(512, seed=31)[: shape[0], : shape[1]])
    n = max(4096, img.size)
    with cc.Instance(0, 3, n, 128, 14) as inst:
        words, bits = cc.compress_heightfield(inst, dev(img), levels)
        ref_words, ref_bits = oracle.compress_heightfield(img, levels)
        assert bits == ref_bits
        assert np.array_equal(host(words)[: (bits + 31) // 32].view(np.uint32), ref_words)
        out = torch.zeros(shape, dtype=torch.int16, device="cuda")
        cc.decompress_heightfield(inst, out, levels, words, bits)
        assert np.array_equal(host(out), img)


@pytest.mark.parametrize("z_chunk", [0, 8, 12, 32, 64])
@pytest.mark.parametrize("shape", [(16, 16, 16), (48, 80, 136), (144, 32, 32)])
def test_forward_level_depths(oracle, z_chunk, shape):
    """The forward level's tile depth, chosen by the rule (0) or given, does
    not show in the streams; levels smaller and larger than a tile."""
    vol = np.ascontiguousarray(fields.turbulence_field(144, 256, 36, seed=77)[: shape[0], : shape[1], : shape[2]])
    ref_words, ref_bits = oracle.compress_volume(vol, 1, 0.01)
    ref = oracle.decompress_volume(ref_words, ref_bits, shape, 1, 0.01)
    with cc.Instance(0, 8, vol.size, 128, 14) as inst, \
            cc.VolumeBatch(inst, [shape], 1, [0.01], z_chunk=z_chunk) as batch:
        batch.compress([dev(vol)])
        words, bits = batch.read_stream(0)
        assert bits == ref_bits and np.array_equal(words, ref_words)
        out = torch.zeros(shape, dtype=torch.float32, device="cuda")
        batch.decompress([out])
        batch.status()
        assert same(host(out), ref)


# ---------------------------------------------------------- entropy coder
def roundtrip(oracle, inst, kind, streams, cb=128, log2max=14, shift=0):
    """Encodes views `shift` elements into larger buffers, compares with the
    oracle, decodes the oracle's words into such views."""
    S, n = streams.shape
    signed, tsigned = (np.int16, torch.int16) if streams.dtype == np.uint16 else (np.int32, torch.int32)
    pitch = (n + 16) // 8 * 8
    buf = torch.zeros(S * pitch + 16, dtype=tsigned, device="cuda")
    views = [buf[i * pitch + shift: i * pitch + shift + n] for i in range(S)]
    for v, s in zip(views, streams):
        v.copy_(dev(s.view(signed)))
    bs = cc.BitStream()
    enc, dec = (cc.encode_rlhuff, cc.decode_rlhuff) if kind == 0 else (cc.encode_huff, cc.decode_huff)
    assert enc(inst, bs, views, n), cc.last_error()
    words, bits, _ = oracle.encode(kind, streams, cb=cb, log2max=log2max)
    assert bs.bit_size == bits
    assert np.array_equal(bs.raw(), words)
    buf.fill_(-1)
    assert dec(inst, cc.BitStream(words, bits), views, n), cc.last_error()
    assert cc.decode_status(inst) == 0
    for v, s in zip(views, streams):
        assert np.array_equal(host(v).view(streams.dtype), s)
    guard = torch.ones_like(buf, dtype=torch.bool)
    for i in range(S):
        guard[i * pitch + shift: i * pitch + shift + n] = False
    assert bool((buf[guard] == -1).all())


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("n", [31, 33, 1023, 1025, 4097, 20011])
def test_streams_at_odd_addresses(oracle, kind, shift, n):
    """Symbol arrays aligned to 16, 2 and 8 bytes; lengths around a lane's
    group, a warp's and a block's tile."""
    with cc.Instance(0, 3, 20011, 128, 14) as inst:
        roundtrip(oracle, inst, kind, symbol_streams("laplace", 3, n, seed=n), shift=shift)


@pytest.mark.parametrize("n", [31 * 2048 + 1, 32 * 2048, 32 * 2048 + 1, 130 * 2048 + 77])
def test_streams_around_a_step_of_the_tile_scan(oracle, n):
    """32 run-length tiles of 2048 symbols are one step of a stream's scan;
    the third stream's only nonzero is its last symbol."""
    streams = symbol_streams("sparse", 3, n, seed=n)
    streams[2] = 0
    streams[2, -1] = 3
    with cc.Instance(0, 3, n, 128, 14) as inst:
        roundtrip(oracle, inst, 0, streams)


@pytest.mark.parametrize("zeros,dense", [(2303, 2048), (2304, 2048), (2305, 2047), (2056 * 256 - 1, 1), (2056 * 256, 1),
                                         (2056 * 256 + 255, 1), (1 << 20, 1200)])
def test_tiles_around_the_write_stage(oracle, zeros, dense):
    """A tile of 2048 symbols with 2056 entries, which its stage holds, and
    with more: `dense` nonzeros from its start on after a run of `zeros`."""
    rng = np.random.default_rng(zeros + dense)
    start = (zeros + 1 + 2047) // 2048 * 2048
    n = start + 3 * 2048 + 11
    streams = np.zeros((2, n), np.uint16)
    streams[0, start - zeros - 1] = 9
    streams[0, start:start + dense] = rng.integers(1, 30, dense)
    streams[1] = np.roll(streams[0], 5)   # compact arrays that start off a 16-byte boundary
    with cc.Instance(0, 2, n, 128, 14) as inst:
        roundtrip(oracle, inst, 0, streams)


@pytest.mark.parametrize("S,tiles", [(1, 128), (1, 129), (2, 511), (2, 512), (2, 513), (1, 1090), (33, 64), (33, 65), (64, 65),
                                     (65, 64), (65, 65)])
def test_long_streams_of_the_tile_scan(oracle, S, tiles):
    """Both sides of the rule for a block per stream, and of a block's step of
    512 tiles; the first stream is dense, the second has runs across many
    tiles, the last one nonzero near its end."""
    n = tiles * 2048 - 5
    rng = np.random.default_rng(tiles + S)
    streams = np.zeros((S, n), np.uint16)
    for i in range(S):
        at = np.unique(rng.integers(0, n, 37 if i == 1 else 3 * tiles))
        streams[i, at] = rng.integers(1, 40, len(at))
    streams[-1] = 0
    streams[-1, -3] = 7
    if S > 1:
        streams[0] = rng.integers(0, 4, n)
    with cc.Instance(0, S, n, 128, 14) as inst:
        roundtrip(oracle, inst, 0, streams)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("cb", [32, 64, 128, 256])
@pytest.mark.parametrize("n", [3000, 40000])
def test_code_words_longer_than_the_staged_window(oracle, kind, cb, n):
    """One stream of near-uniform symbols over the whole alphabet (13 to 14
    bits each: read from global memory), one whose second half is sparse (a
    stream with both kinds of warps), one of zeros (no code words)."""
    rng = np.random.default_rng(cb + n)
    streams = np.zeros((3, n), np.uint16)
    streams[0] = rng.integers(1, 1 << 14, n)
    streams[1, : n // 2] = rng.integers(1, 1 << 14, n // 2)
    streams[1, n // 2:] = (rng.random(n - n // 2) < 0.05) * 3
    with cc.Instance(0, 3, n, cb, 14) as inst:
        roundtrip(oracle, inst, kind, streams, cb=cb)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("leaves", [256, 257, 1024, 1025, 2048, 2049, 12287, 12288, 12289, 16383])
@pytest.mark.parametrize("S", [1, 33])
def test_table_sizes_around_each_builder(oracle, kind, leaves, S):
    """A stream of exactly `leaves` distinct symbols, alone (one call's few
    tables) and with small ones (the tiers by leaf count)."""
    rng = np.random.default_rng(leaves)
    n = 20000
    streams = symbol_streams("laplace", S, n, seed=leaves)
    v = rng.permutation(np.concatenate([np.arange(1, leaves + 1), rng.integers(1, leaves + 1, n - leaves)]))
    streams[S // 2] = v
    assert len(np.unique(streams[S // 2])) == leaves
    with cc.Instance(0, S, n, 128, 14) as inst:
        roundtrip(oracle, inst, kind, streams)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("S", [1, 31, 32, 33, 63, 64, 65, 130])
@pytest.mark.parametrize("cb", [32, 128])
def test_stream_counts_around_the_plans(oracle, kind, S, cb):
    """Stream and table counts on both sides of the one-CTA plans' 64."""
    with cc.Instance(0, S, 5000, cb, 14) as inst:
        roundtrip(oracle, inst, kind, symbol_streams("sparse", S, 4675, seed=S), cb=cb)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("n", [33, 4097, 20000])
@pytest.mark.parametrize("shift", [0, 1])
def test_wide_symbols(oracle, kind, n, shift):
    """32-bit symbols of a 20-bit alphabet, dense and sparse, at 16- and
    4-byte aligned addresses."""
    rng = np.random.default_rng(n)
    streams = rng.integers(0, 1 << 19, (2, n)).astype(np.uint32)
    streams[1] *= rng.random(n) < 0.2
    with cc.Instance(0, 2, 20000, 128, 20) as inst:
        roundtrip(oracle, inst, kind, streams, log2max=20, shift=shift)


@pytest.mark.parametrize("kind,S", [(0, 7), (0, 74), (0, 75), (0, 296), (0, 297), (1, 1), (1, 148), (1, 149), (1, 592),
                                    (1, 593)])
def test_wide_symbol_tables_of_many_streams(oracle, kind, S):
    """Decode tables of 32-bit symbols, whose table kernel has no barrier
    between the symbols and the block offsets: both CTA widths (up to 148
    tables and more), tables of one leaf to hundreds, several times over.
    No warp may miss its share of a table: a guard reads the table's state
    while another warp goes on to its block offsets."""
    rng = np.random.default_rng(S)
    n = 700
    streams = (rng.integers(0, 1 << 18, (S, n)) * (rng.random((S, n)) < rng.random((S, 1)))).astype(np.uint32)
    streams[0] = 5
    with cc.Instance(0, S, n, 32, 18) as inst:
        words, bits, _ = oracle.encode(kind, streams, cb=32, log2max=18)
        outs = torch.empty((S, n + 4), dtype=torch.int32, device="cuda")
        dec = cc.decode_rlhuff if kind == 0 else cc.decode_huff
        for _ in range(8):
            outs.fill_(-1)
            assert dec(inst, cc.BitStream(words, bits), [outs[i, :n] for i in range(S)], n), cc.last_error()
            assert cc.decode_status(inst) == 0
            assert np.array_equal(host(outs[:, :n]).view(np.uint32), streams)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("bits", [16, 32])
def test_counts_of_large_symbols(oracle, kind, bits):
    """Symbols counted by slots of their low byte: one value throughout, a few
    neighbours, many that share a low byte, the whole upper range, and both
    sides of the first symbol that is not counted by bin."""
    rng = np.random.default_rng(bits + kind)
    n, top = 9000, 1 << (14 if bits == 16 else 20)
    streams = np.zeros((7, n), np.uint16 if bits == 16 else np.uint32)
    streams[0] = 2000
    streams[1] = 1500 + rng.integers(0, 4, n)
    streams[2] = 1024 + 7 + 256 * rng.integers(0, (top - 1100) // 256, n)
    streams[3] = rng.integers(1024, top, n)
    streams[4] = rng.integers(1016, 1032, n) * (rng.random(n) < 0.5)
    streams[5] = top - 1 - 256 * (np.arange(n) % 3)
    streams[6] = 760 + rng.integers(0, 16, n)
    with cc.Instance(0, 7, n, 128, 14 if bits == 16 else 20) as inst:
        roundtrip(oracle, inst, kind, streams, log2max=14 if bits == 16 else 20)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("S", [1, 40])
@pytest.mark.parametrize("top", [31, 32, 63, 511, 512, 513, 4095, 4096, 4097, 65536, 300001])
def test_leaves_spread_over_an_alphabet(oracle, kind, S, top):
    """Few symbols in an alphabet of `top` + 1 bins, at the borders of the
    warps' ranges and of their steps, the largest in the last bin."""
    rng = np.random.default_rng(top)
    at = np.array([1, 30, 31, 32, 33, 255, 256, 257, 511, 512, 1023, 8191, 8192, top // 2, top - 1, top])
    at = np.unique(at[(at >= 1) & (at <= top)])
    streams = rng.choice(at, (S, 600)).astype(np.uint32)
    streams[:, 0] = top
    with cc.Instance(0, S, 600, 128, 20) as inst:
        roundtrip(oracle, inst, kind, streams, log2max=20)


@pytest.mark.parametrize("leaves", [26626, 26627, 26628, 53254, 53255])
def test_tables_around_the_sequential_builders_area(oracle, leaves):
    """Leaf counts around what the builder's shared memory holds as a heap (8
    bytes each) and as sort keys (4 bytes)."""
    rng = np.random.default_rng(leaves)
    n = 60000
    v = rng.permutation(np.concatenate([np.arange(1, leaves + 1), rng.integers(1, 200, n - leaves)]))
    with cc.Instance(0, 1, n, 128, 17) as inst:
        roundtrip(oracle, inst, 1, v.astype(np.uint32)[None], log2max=17)


@pytest.mark.parametrize("cb", [32, 128])
@pytest.mark.parametrize("streams", [1, 3])
def test_zero_counts_past_a_byte(oracle, cb, streams):
    """Streams with zero counts up to 65535, which the encoder does not write
    (it splits runs at 256) but the format's tables can hold: rounds of 32
    entries within 65536 positions, and longer ones.  A run-length stream is
    its entry count and the two arrays' Huff streams."""
    rng = np.random.default_rng(cb)
    parts, expect, n = [], [], 1 << 21
    for k in range(streams):
        zc = np.concatenate([np.full(32, 2046), [0, 65535], rng.integers(0, 40000, 30), rng.integers(0, 256, 64),
                             [65535], np.full(31, 0), rng.integers(200, 3000, 77 + k)]).astype(np.uint16)
        sym = rng.integers(1, 50, len(zc)).astype(np.uint16)
        at = np.cumsum(zc.astype(np.int64) + 1) - 1
        assert at[-1] < n and int((zc[:32].astype(int) + 1).sum()) <= 65536 < int((zc[32:64].astype(int) + 1).sum())
        out = np.zeros(n, np.uint16)
        out[at] = sym
        expect.append(out)
        parts.append(np.array([len(zc)], np.uint32))
        for a in (sym, zc):
            words, bits, _ = oracle.encode(1, a[None], cb=cb, log2max=16)
            parts.append(words[: (bits + 31) // 32])
    words = np.concatenate(parts).astype(np.uint32)
    with cc.Instance(0, streams, n, cb, 16) as inst:
        outs = torch.full((streams, n), -1, dtype=torch.int16, device="cuda")
        assert cc.decode_rlhuff(inst, cc.BitStream(words, 32 * len(words)), list(outs), n), cc.last_error()
        assert cc.decode_status(inst) == 0
        assert np.array_equal(host(outs).view(np.uint16), np.stack(expect))


def test_forward_depths_of_uneven_levels(oracle):
    """Batches whose levels take different tile depths by the rule: with 148
    multiprocessors 8 volumes of 64^3 and near it 8 slices at every level, 24
    take 16 at level 0, 40 take 32, 100 also 16 at level 1."""
    shapes = [(64, 64, 64), (64, 48, 64), (48, 64, 56), (64, 64, 40)]
    field = fields.turbulence_field(64, 256, 21, seed=5)
    distinct = [np.ascontiguousarray(field[: s[0], : s[1], : s[2]]) for s in shapes]
    refs = [oracle.compress_volume(v, 3, 0.01) for v in distinct]
    for count in (8, 24, 40, 100):
        vols = [dev(distinct[i % 4]) for i in range(count)]
        with cc.Instance(0, 8, 64 ** 3, 128, 14) as inst, \
                cc.VolumeBatch(inst, [tuple(v.shape) for v in vols], 3, [0.01] * count) as batch:
            batch.compress(vols)
            batch.status()
            for i in range(count):
                words, bits = batch.read_stream(i)
                assert bits == refs[i % 4][1] and np.array_equal(words, refs[i % 4][0])


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("S,blocks", [(3, 1023), (3, 1024), (80, 5), (160, 5), (300, 5), (2, 9000)])
def test_block_scans_by_length(oracle, kind, S, blocks):
    """Both sides of the rules for a block per stream in the scans over coding
    blocks and in the table kernel: lengths and stream counts."""
    n = 32 * blocks - 3
    with cc.Instance(0, S, n, 32, 14) as inst:
        roundtrip(oracle, inst, kind, symbol_streams("sparse", S, n, seed=S + blocks), cb=32)
