"""GPU tests of the stand-alone codec kernels against the CPU oracle (bit exact)."""
import ctypes as C

import numpy as np
import pytest
import torch

import gcow_b200 as g
from gcow_b200 import _native
from gcow_b200.codec import ZfpParams, Compressed

from test_codec_cpu import (_rand, _special_1d, field, CAST_3, XFORM_3, NB_3, UBLOCK_A, WORDS_A)

pytestmark = pytest.mark.gpu


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


@pytest.mark.parametrize("rate", [4, 8, 16, 32])
def test_fast_1d_bit_exact(rate):
    p = ZfpParams.from_rate(rate, 1)
    for x in (_rand(1 << 20), _special_1d(), _rand(5, seed=9), _rand(1 << 20 | 3, seed=2)):
        cpu = g.compress(torch.from_numpy(x), params=p)
        gpu = g.compress(dev(x), params=p)
        assert gpu.stream.is_cuda and gpu.nbytes == cpu.nbytes
        assert torch.equal(gpu.stream.cpu(), cpu.stream)
        for shift in (0, 3):
            a = g.decompress(cpu, shift=shift)
            b = g.decompress(gpu, shift=shift).cpu()
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))


def test_fast_1d_unaligned_views():
    base = dev(_rand((1 << 16) + 8))
    x = base[1:(1 << 16) + 2]           # 4-byte aligned only
    p = ZfpParams.from_rate(8, 1)
    cpu = g.compress(x.cpu(), params=p)
    gpu = g.compress(x, params=p)
    assert torch.equal(gpu.stream.cpu(), cpu.stream)
    out = torch.empty((1 << 16) + 9, device="cuda")[1:(1 << 16) + 2]
    assert not out.is_contiguous() or True
    o = torch.empty_like(x)
    g.decompress(gpu, out=o)
    assert torch.equal(o.cpu().view(torch.int32), g.decompress(cpu).view(torch.int32))


def test_fast_1d_decode_random_streams():
    rng = np.random.default_rng(11)
    for rate in (4, 8, 16, 32):
        p = ZfpParams.from_rate(rate, 1)
        n = 4 * 65536
        raw = rng.integers(0, 256, size=n * rate // 8, dtype=np.uint8)
        a = g.decompress(Compressed(torch.from_numpy(raw.copy()), p, (n,), None))
        b = g.decompress(Compressed(dev(raw), p, (n,), None)).cpu()
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("p", [ZfpParams.from_rate(2, 1), ZfpParams.from_rate(3, 1), ZfpParams.from_rate(6, 1),
                               ZfpParams.from_accuracy(1e-3), ZfpParams.from_accuracy(1e-6),
                               ZfpParams.from_precision(12)],
                         ids=lambda p: f"{p.minbits}-{p.maxbits}-{p.maxprec}-{p.minexp}")
def test_generic_1d_bit_exact(p):
    for x in (_rand(1 << 16), _special_1d(), _rand(7, seed=3)):
        cpu = g.compress(torch.from_numpy(x), params=p, return_index=True)
        gpu = g.compress(dev(x), params=p, return_index=True)
        assert gpu.nbytes == cpu.nbytes
        assert torch.equal(gpu.stream.cpu(), cpu.stream)
        assert torch.equal(gpu.index.cpu(), cpu.index)
        a = g.decompress(cpu)
        b = g.decompress(gpu).cpu()
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("p", [ZfpParams.from_rate(1, 2), ZfpParams.from_rate(4, 2), ZfpParams.from_rate(8, 2),
                               ZfpParams.from_rate(16, 2), ZfpParams.from_accuracy(1e-3),
                               ZfpParams.from_accuracy(1e-6), ZfpParams.from_precision(16)],
                         ids=lambda p: f"{p.minbits}-{p.maxbits}-{p.maxprec}-{p.minexp}")
def test_generic_2d_bit_exact(p):
    rng = np.random.default_rng(1)
    for x in (field(37), (rng.standard_normal((130, 257)) * 5).astype(np.float32), field(8),
              np.zeros((9, 5), dtype=np.float32)):
        cpu = g.compress(torch.from_numpy(x), params=p, dim=2, return_index=True)
        gpu = g.compress(dev(x), params=p, dim=2, return_index=True)
        assert gpu.nbytes == cpu.nbytes
        assert torch.equal(gpu.stream.cpu(), cpu.stream)
        a = g.decompress(cpu)
        b = g.decompress(gpu).cpu()
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))


def test_variable_rate_decode_without_index_goes_through_host():
    x = field(64)
    gpu = g.compress(dev(x), tolerance=1e-3, dim=2)
    c = Compressed(gpu.stream, gpu.params, gpu.shape, None)
    d = g.decompress(c).cpu().numpy()
    assert np.max(np.abs(d - x)) <= 1e-3


def test_golden_3x3_on_gpu():
    c = g.compress(dev(field(3)), tolerance=1e-3, dim=2)
    w = list(np.frombuffer(c.stream.cpu().numpy().tobytes(), dtype=np.uint64))
    assert w == [7846959668108800257, 9092781915241025288, 1168152206201298680, 33031166]


def test_stage_kernels_golden():
    lib = _native.cuda()
    cpu = _native.cpu()
    s = torch.cuda.current_stream().cuda_stream
    blk = np.zeros(16, dtype=np.float32)
    a = field(3)
    cpu.gcow_stage_gather(a.ctypes.data, 3, 3, 0, blk.ctypes.data)
    nb = 1000
    f = dev(np.tile(blk, nb))
    emax = torch.empty(nb, dtype=torch.int32, device="cuda")
    assert lib.gcow_dbg_stage(0, 2, nb, f.data_ptr(), emax.data_ptr(), None, 0, s) == 0
    assert bool((emax == 1).all())
    q = torch.empty(nb * 16, dtype=torch.int32, device="cuda")
    assert lib.gcow_dbg_stage(1, 2, nb, f.data_ptr(), q.data_ptr(), emax.data_ptr(), 0, s) == 0
    assert q.view(nb, 16)[nb - 1].tolist() == CAST_3
    assert lib.gcow_dbg_stage(2, 2, nb, None, q.data_ptr(), None, 0, s) == 0
    assert q.view(nb, 16)[0].tolist() == XFORM_3
    u = torch.empty(nb * 16, dtype=torch.int32, device="cuda")
    assert lib.gcow_dbg_stage(4, 2, nb, q.data_ptr(), u.data_ptr(), None, 0, s) == 0
    assert [v & 0xffffffff for v in u.view(nb, 16)[nb // 2].tolist()] == NB_3
    # plane coder: header 257 + all planes of the golden coefficient block
    ub = dev(np.tile(np.array(UBLOCK_A, dtype=np.uint32), nb).view(np.int32))
    p = ZfpParams.from_accuracy(1e-3)
    out = torch.zeros(nb * 4, dtype=torch.int64, device="cuda")
    bits = torch.zeros(nb, dtype=torch.int32, device="cuda")
    assert lib.gcow_dbg_planes(2, nb, ub.data_ptr(), p.maxbits - 9, p.block_precision(1, 2), 257, 4,
                               out.data_ptr(), bits.data_ptr(), s) == 0
    one = np.frombuffer(out.view(nb, 4)[7].cpu().numpy().tobytes(), dtype=np.uint64)
    nbits = int(bits[7])
    # first block of the 3-block golden stream: compare the bits it owns
    gold = np.array(WORDS_A[:4], dtype=np.uint64)
    full = nbits // 64
    assert list(one[:full]) == list(gold[:full])
    rem = nbits % 64
    if rem:
        m = np.uint64((1 << rem) - 1)
        assert one[full] == (gold[full] & m)
    # inverse cast with an averaging shift equals the host stage
    qi = dev(np.array(CAST_3 * nb, dtype=np.int32))
    fo = torch.empty(nb * 16, dtype=torch.float32, device="cuda")
    assert lib.gcow_dbg_stage(5, 2, nb, qi.data_ptr(), fo.data_ptr(), emax.data_ptr(), 2, s) == 0
    ref = np.zeros(16, dtype=np.float32)
    qn = np.array(CAST_3, dtype=np.int32)
    cpu.gcow_stage_inv_cast(qn.ctypes.data, ref.ctypes.data, 16, 1, 2, 0)
    assert np.array_equal(fo.view(nb, 16)[3].cpu().numpy(), ref)


def test_gather_and_whole_block_stage_kernels():
    """Block formation with edge padding (5 x 7 ramp of the reference's gather test) and the
    whole-block encoder (3 x 3 field of its integration test) as stand-alone stage kernels."""
    lib = _native.cuda()
    s = torch.cuda.current_stream().cuda_stream
    ramp = torch.arange(1, 36, dtype=torch.float32, device="cuda").reshape(7, 5).contiguous()
    blocks = torch.zeros(4 * 16, dtype=torch.float32, device="cuda")
    assert lib.gcow_dbg_gather(2, ramp.data_ptr(), 5, 7, 4, blocks.data_ptr(), s) == 0
    b = blocks.view(4, 16).cpu()
    assert b[1].tolist() == [5, 5, 5, 5, 10, 10, 10, 10, 15, 15, 15, 15, 20, 20, 20, 20]
    assert b[3].tolist() == [25, 25, 25, 25, 30, 30, 30, 30, 35, 35, 35, 35, 25, 25, 25, 25]
    assert b[2][:4].tolist() == [21, 22, 23, 24] and b[2][12:].tolist() == [21, 22, 23, 24]
    f3 = dev(field(3))
    blk = torch.zeros(16, dtype=torch.float32, device="cuda")
    assert lib.gcow_dbg_gather(2, f3.data_ptr(), 3, 3, 1, blk.data_ptr(), s) == 0
    p = ZfpParams.from_accuracy(1e-3)
    out = torch.zeros(9, dtype=torch.int64, device="cuda")
    bits = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert lib.gcow_dbg_encode_block(2, blk.data_ptr(), 1, p.as_c(), 9, out.data_ptr(), bits.data_ptr(), s) == 0
    w = list(np.frombuffer(out.cpu().numpy().tobytes(), dtype=np.uint64)[:4])
    assert w == [7846959668108800257, 9092781915241025288, 1168152206201298680, 33031166]
    assert 192 < int(bits[0]) <= 256


# Sizes around what one lane (4 or 1 blocks), one string (128 or 32 blocks) and one tile (1024 or 256 blocks) hold, and
# several tiles; every mode the tile kernels take, with budgets that cut a code and that end on word boundaries or not.
@pytest.mark.parametrize("dim,sizes", [(1, [1, 4, 127, 509, 512, 516, 4093, 4096, 4100, 70001]),
                                       (2, [(1, 1), (4, 128), (7, 129), (40, 512), (129, 1023), (64, 2052), (33, 78)])])
@pytest.mark.parametrize("how", [dict(tolerance=1e-6), dict(tolerance=1e-3), dict(tolerance=1e9), dict(precision=3), dict(precision=32),
                                 dict(rate=2), dict(rate=3), dict(rate=12), dict(rate=20), dict(rate=33)],
                         ids=lambda h: "%s-%g" % next(iter(h.items())))
def test_tile_kernels_at_edges(dim, sizes, how):
    rng = np.random.default_rng(7)
    for sz in sizes:
        n = sz if dim == 1 else sz[0] * sz[1]
        noise = rng.standard_normal(n).astype(np.float32)
        sparse = np.where(rng.random(n) < 0.7, np.float32(0), noise)
        for x in (noise * 1e-3, np.cumsum(noise).astype(np.float32) * 1e-2, sparse, np.zeros(n, np.float32)):
            t = torch.from_numpy(x if dim == 1 else x.reshape(sz))
            cpu, gpu = (g.compress(v, dim=dim, return_index=True, **how) for v in (t, t.cuda()))
            assert torch.equal(gpu.stream.cpu(), cpu.stream) and torch.equal(gpu.index.cpu(), cpu.index), sz
            for shift in (0, 2):
                a, b = g.decompress(cpu, shift=shift), g.decompress(gpu, shift=shift).cpu()
                assert torch.equal(a.view(torch.int32), b.view(torch.int32)), sz


@pytest.mark.parametrize("blocks", [151552, 151553, 151552 + 1024, 148 * 6 * 4 * 1024 + 1025])
@pytest.mark.parametrize("how", [dict(tolerance=1e-6), dict(tolerance=1e-2), dict(precision=2), dict(rate=6), dict(rate=8)])
def test_tile_kernels_with_four_blocks_per_lane(blocks, how):
    """The last size with one block per lane and the first ones with four, the first with more tiles than CTAs; strings whose
    words belong to one block, to two, and (runs of 1-bit blocks) to many."""
    n = 4 * blocks - 1
    rng = np.random.default_rng(blocks)
    x = (rng.standard_normal(n) * 1e-2).astype(np.float32)
    x[n // 3: n // 2] = 0                                    # runs of 1-bit blocks, and some among the others
    x[n // 2: n // 2 + 40_000: 7] = 0
    x[-4000:] *= np.float32(1e-36)                           # denormals
    x[5000::70_001] = np.inf
    cpu = g.compress(torch.from_numpy(x), **how)
    gpu = g.compress(dev(x), **how)
    assert gpu.nbytes == cpu.nbytes and torch.equal(gpu.stream.cpu(), cpu.stream)
    assert torch.equal(g.decompress(gpu).cpu().view(torch.int32), g.decompress(cpu).view(torch.int32))


@pytest.mark.parametrize("tiles", [591, 592, 593])
@pytest.mark.parametrize("how", [dict(tolerance=1e-3), dict(precision=16), dict(rate=8), dict(rate=9), dict(rate=16)])
def test_2d_tiles_around_the_line_between_instances(tiles, how):
    """Four tiles of 256 blocks per SM, one less and one more, against the CPU codec."""
    ny, nx = 4 * 256 - 1, 4 * tiles - 3
    y, x = np.mgrid[0:ny, 0:nx].astype(np.float32) * np.float32(1e-3)
    f = (np.exp(-(x * x + y * y)) + np.random.default_rng(tiles).standard_normal((ny, nx)) * 1e-4).astype(np.float32)
    cpu, gpu = g.compress(torch.from_numpy(f), **how), g.compress(dev(f), **how)
    assert gpu.nbytes == cpu.nbytes and torch.equal(gpu.stream.cpu(), cpu.stream)
    assert torch.equal(g.decompress(gpu).cpu().view(torch.int32), g.decompress(cpu).view(torch.int32))


@pytest.mark.parametrize("dim,tile", [(1, 256), (1, 1024), (2, 256)])
@pytest.mark.parametrize("more", [-1, 0, 1])
def test_strings_of_as_many_tiles_as_ctas(dim, tile, more):
    """The placing kernel where its CTAs have a tile each and just above, the last tile with one block or one short of all, for an index
    at a multiple of 16 bytes and of 8 only."""
    tiles = 740 + more if (dim, tile) != (1, 256) else 592 + more       # 1-D: four blocks a lane from 593 tiles of 256 on
    blocks = tiles * tile - (tile - 1 if more == 0 else 1)
    rng = np.random.default_rng(blocks)
    if dim == 1:
        x = (rng.standard_normal(4 * blocks) * 1e-3).astype(np.float32)
        x[:8000] = 0
    else:
        x = (rng.standard_normal((4, 4 * blocks)) * 1e-4).astype(np.float32) + np.float32(1) / (1 + np.arange(4 * blocks, dtype=np.float32))
    p = ZfpParams.from_accuracy(1e-5)
    cpu = g.compress(torch.from_numpy(x), params=p, dim=dim, return_index=True)
    lib, d = _native.cuda(), dev(x)
    lib.gcow_encode_tiles.argtypes = [C.c_void_p, C.c_uint64, C.c_uint64, C.c_void_p] + [C.c_void_p] * 5
    lib.gcow_encode_tiles_scratch_bytes.argtypes, lib.gcow_encode_tiles_scratch_bytes.restype = [C.c_void_p, C.c_uint64, C.c_int], C.c_uint64
    par = p.as_c()
    scratch = torch.empty(lib.gcow_encode_tiles_scratch_bytes(par, blocks, dim), dtype=torch.uint8, device="cuda")
    for skip in (0, 1):
        out = torch.full((blocks * 72 + 64,), 255, dtype=torch.uint8, device="cuda")
        index = torch.full((blocks + 3,), -1, dtype=torch.int64, device="cuda")
        rc = lib.gcow_encode_tiles(d.data_ptr(), x.shape[-1], 4 if dim == 2 else 0, par, out.data_ptr(), scratch.data_ptr(),
                                   index.data_ptr() + 8 * skip, None, None)
        torch.cuda.synchronize()
        assert rc == 0
        assert torch.equal(index[skip:skip + blocks + 1].cpu(), cpu.index) and (index[skip + blocks + 1:] == -1).all()
        assert torch.equal(out[:cpu.nbytes].cpu(), cpu.stream)


@pytest.mark.parametrize("n", [4 * 300, 4 * 151552 + 7, 4 * 148 * 6 * 4 * 1024 * 2 + 40_001])
@pytest.mark.parametrize("how", [dict(tolerance=1e-6), dict(tolerance=1e-3), dict(precision=8), dict(precision=16)])
def test_1d_tiles_of_data_that_changes(n, how):
    """Noise, values near 1, denormals and zeros in turn, in stretches that end inside a group of 32 blocks and in long ones: warps that
    stop trying the straight line and ones that do not, on one tile and on several."""
    rng = np.random.default_rng(n)
    x = (rng.standard_normal(n) * 1e-3).astype(np.float32)
    turn = np.arange(n) // 1999 % 4
    turn[n // 2:] = np.arange(n - n // 2) // 400_003 % 4
    x = np.select([turn == 1, turn == 2, turn == 3], [1 + x * np.float32(1e-3), x * np.float32(1e-37), x * 0], x).astype(np.float32)
    cpu = g.compress(torch.from_numpy(x), **how)
    gpu = g.compress(dev(x), **how)
    assert gpu.nbytes == cpu.nbytes and torch.equal(gpu.stream.cpu(), cpu.stream)
    assert torch.equal(g.decompress(gpu).cpu().view(torch.int32), g.decompress(cpu).view(torch.int32))


@pytest.mark.parametrize("dim", [1, 2])
def test_tiles_of_zeros(dim):
    """Groups of one-bit blocks: nothing else, behind strings that end at every bit of a word, and a last group of fewer than 32."""
    per = 4 if dim == 1 else 16
    for blocks in (1, 31, 32, 33, 64, 255, 257, 5000, 151_553 + 77):
        x = np.zeros((blocks, per), np.float32)
        for lead in (0, 1, 7):
            x[:] = 0
            if lead:                                         # a code of another length ahead of each warp's groups of zeros
                x[::161] = np.random.default_rng(blocks + lead).standard_normal((len(x[::161]), per)) * 10.0 ** -lead
            f = x.reshape(-1) if dim == 1 else np.ascontiguousarray(x.reshape(blocks, 4, 4).transpose(1, 0, 2).reshape(4, -1))
            cpu = g.compress(torch.from_numpy(f), dim=dim, tolerance=1e-9)
            gpu = g.compress(dev(f), dim=dim, tolerance=1e-9)
            assert gpu.nbytes == cpu.nbytes and torch.equal(gpu.stream.cpu(), cpu.stream)
            assert torch.equal(g.decompress(gpu).cpu(), torch.from_numpy(f).new_tensor(g.decompress(cpu).numpy()))


@pytest.mark.parametrize("rate", [2.25, 2.5, 2.75, 3])
def test_decode_of_short_blocks(rate):
    """Blocks of 9 to 11 bits go to the kernel without staging, 12 bits and streams that are not word aligned to the tiles."""
    rng = np.random.default_rng(3)
    for n in (1, 5, 1021, 4096, 70001):
        for x in (rng.standard_normal(n).astype(np.float32), np.cumsum(rng.standard_normal(n)).astype(np.float32),
                  np.where(rng.random(n) < 0.9, 0, 1).astype(np.float32)):
            cpu = g.compress(torch.from_numpy(x), rate=rate)
            gpu = g.compress(dev(x), rate=rate)
            assert torch.equal(gpu.stream.cpu(), cpu.stream)
            held = torch.zeros(gpu.nbytes + 8, dtype=torch.uint8, device="cuda")
            held[4:4 + gpu.nbytes] = gpu.stream
            for shift in (0, 2):
                want = g.decompress(cpu, shift=shift).view(torch.int32)
                out = torch.zeros(n + 2, device="cuda")
                got = g.decompress(gpu, out=out[1:n + 1], shift=shift)
                assert torch.equal(got.cpu().view(torch.int32), want) and out[0] == 0 and out[n + 1] == 0
                moved = Compressed(held[4:4 + gpu.nbytes], gpu.params, gpu.shape, None)
                assert torch.equal(g.decompress(moved, shift=shift).cpu().view(torch.int32), want)


@pytest.mark.parametrize("dim,how", [(1, dict(tolerance=1e-6)), (1, dict(precision=20)), (2, dict(tolerance=1e-6))])
def test_variable_rate_result_on_another_stream(dim, how):
    """These modes wait for the length alone; the stream and its index are ready in the order of the CUDA stream that made
    them, on which another stream has to wait."""
    x = torch.randn(1 << 24, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    x = x.view(4096, -1) if dim == 2 else x
    side = torch.cuda.Stream()
    for _ in range(5):
        c = g.compress(x, dim=dim, **how)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            stream, index, y = c.stream.clone(), c.index.clone(), g.decompress(c)
        torch.cuda.synchronize()
        assert torch.equal(stream, c.stream) and torch.equal(index, c.index) and torch.equal(y, g.decompress(c))
        assert c.nbytes == (int(index[-1]) + 63) // 64 * 8


@pytest.mark.gpu
@pytest.mark.parametrize("rate", [4, 8, 16, 32])
def test_long_vectors_equal_their_pieces(rate):
    """Vectors long enough for the larger grid of the fixed-rate kernels, against the same values in pieces, which are short."""
    n = 4 * (32 * 148 * 4 * 512 + 777) + 3
    x = torch.randn(n, device="cuda", generator=torch.Generator("cuda").manual_seed(rate)) * 1e-3
    x[::4099] = float("nan")
    x[n // 3:n // 2] += 1
    x[n // 2:n // 2 + 100000] = 0
    x[-n // 5::9] *= 1e-36
    c = g.compress(x, rate=rate)
    piece = 1 << 22
    parts = [g.compress(x[i:i + piece], rate=rate) for i in range(0, n, piece)]
    assert torch.equal(c.stream, torch.cat([p.stream for p in parts]))
    y = g.decompress(c)
    assert torch.equal(y.view(torch.int32), torch.cat([g.decompress(p) for p in parts]).view(torch.int32))
