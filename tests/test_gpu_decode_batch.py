"""decode_batch on the GPU against the CPU oracle (mirrors the reference's own
GPU tests, tests/test_lmz.py:2272-2390 and :2538-2570 in the reference tree)."""
import numpy as np
import pytest

from helpers import DISTRIBUTIONS, SHAPES, distribution, pack_streams, shaped

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True, params=[0, 2, 3, 4, -1], ids=["narrow", "compact", "wide1", "wide13", "auto"])
def table_mode(request, gpu):
    """Every test runs with each per-stream table layout forced: k_stream's, k_solo's two."""
    lib = gpu.library()
    assert lib.lmz_gpu_set_table_mode(request.param) == 0
    yield request.param
    lib.lmz_gpu_set_table_mode(-1)


def _check(gpu, orc, plains, header=None, freqs=None):
    nstr, plane = len(plains), plains[0].size
    if header is None:
        streams = [orc.rans_encode(p) for p in plains]
    else:
        streams = [orc.rans_encode_shared(p, freqs) for p in plains]
    blob, offs = pack_streams(streams)
    out = gpu.decode_batch(blob, offs, nstr, plane, header=header)
    assert out is not None, gpu.last_error()
    out = np.frombuffer(out, dtype=np.uint8).reshape(nstr, plane)
    for i, p in enumerate(plains):
        assert (out[i] == p).all(), f"stream {i} differs"
        if header is None:
            assert (orc.rans_decode(streams[i], plane) == p).all()


def test_matches_cpu_64x4096(gpu, orc):
    plains = [shaped("skewed", 4096, 100 + i) for i in range(64)]
    _check(gpu, orc, plains)


@pytest.mark.parametrize("name", list(SHAPES))
@pytest.mark.parametrize("plane", [1, 2, 7, 8, 9, 17, 127, 128, 129, 4096, 4097, 65537])
def test_shapes_and_ragged_planes(gpu, orc, name, plane):
    for nstr in (1, 17, 129):
        if plane > 4097 and nstr > 17:
            continue
        plains = [shaped(name, plane, hash((name, plane, nstr, i)) & 0xFFFF) for i in range(nstr)]
        _check(gpu, orc, plains)


@pytest.mark.parametrize("dist", DISTRIBUTIONS)
@pytest.mark.parametrize("n", [1, 17, 4096, 65536, 1 << 20])
def test_stress_distributions_per_stream_and_shared(gpu, orc, dist, n):
    nstr = 7 if n >= 65536 else 64
    plains = [distribution(dist, n, 7 * i + n) for i in range(nstr)]
    _check(gpu, orc, plains)
    counts = np.sum([np.bincount(p, minlength=256) for p in plains], axis=0)
    freqs = orc.rans_freqs(counts)
    header = b"R1\0\0" + freqs.astype("<u2").tobytes()
    _check(gpu, orc, plains, header=header, freqs=freqs)


def test_large_batches_are_sorted_by_alphabet_on_the_device(gpu, orc, table_mode):
    """12 000 short streams, every seventh with more live symbols than the dense instance
    of the throughput kernel holds: in automatic mode the library counts alphabets on the
    device and splits the launch; results must not depend on it."""
    if table_mode not in (-1, 2):
        pytest.skip("only the throughput kernel takes batches this large")
    pool = [distribution("uniform" if i % 7 == 0 else "exponent", 640, 900 + i) for i in range(70)]
    streams = [orc.rans_encode(p) for p in pool]
    n = 12000
    blob, offs = pack_streams([streams[i % 70] for i in range(n)])
    out = np.frombuffer(gpu.decode_batch(blob, offs, n, 640), dtype=np.uint8).reshape(n, 640)
    assert (out == np.stack([pool[i % 70] for i in range(n)])).all()
    bad = bytearray(blob)
    bad[int(np.frombuffer(offs, dtype="<u8")[2 * 777])] = ord("X")      # one stream's magic
    with pytest.raises(ValueError):
        gpu.decode_batch(bytes(bad), offs, n, 640)


def test_declines_and_errors(gpu, orc):
    plains = [shaped("skewed", 4096, i) for i in range(2)]
    blob, offs = pack_streams([orc.rans_encode(p) for p in plains])
    assert bytes(gpu.decode_batch(blob, offs, 0, 4096)) == b""
    with pytest.raises(ValueError):
        gpu.decode_batch(blob, offs, -1, 4096)
    with pytest.raises(ValueError):
        gpu.decode_batch(blob, offs[:16], 2, 4096)
    with pytest.raises(ValueError):
        gpu.decode_batch(blob, offs, 2, 4096, header=b"x" * 10)
    broken = bytearray(blob)
    broken[0] = ord("X")
    with pytest.raises(ValueError):
        gpu.decode_batch(bytes(broken), offs, 2, 4096)
    broken = bytearray(blob)
    broken[4] ^= 1                      # frequencies no longer sum to 4096
    with pytest.raises(ValueError):
        gpu.decode_batch(bytes(broken), offs, 2, 4096)
    # the superset: a plane that is not a multiple of 128 decodes
    out = gpu.decode_batch(blob, offs, 2, 4095)
    assert bytes(out[:4095]) == plains[0][:4095].tobytes()
    # truncated stream: the reference CPU decoder rejects it, so does this
    short = orc.rans_encode(shaped("flat", 4096, 9))
    cut = short[:len(short) - 200]
    b2, o2 = pack_streams([cut])
    with pytest.raises(ValueError):
        orc.rans_decode(cut, 4096)
    with pytest.raises(ValueError):
        gpu.decode_batch(b2, o2, 1, 4096)


def test_cuda_tensor_path(gpu, orc):
    import torch
    plains = [shaped("tail", 4099, i) for i in range(33)]
    blob, offs = pack_streams([orc.rans_encode(p) for p in plains])
    t = torch.frombuffer(bytearray(blob), dtype=torch.uint8).cuda()
    out = gpu.decode_batch(t, offs, 33, 4099)
    assert out.is_cuda
    assert out.cpu().numpy().tobytes() == b"".join(p.tobytes() for p in plains)


def test_verify_reports_ok(gpu):
    r = gpu.verify(quick=True)
    assert r["ok"], r
    assert r["checked"] >= 5 and r["gbps"] > 0


@pytest.mark.parametrize("dist", ["exponent", "uniform", "two"])
def test_stress_extremes_long_streams_and_wide_batches(gpu, orc, dist, table_mode):
    """The corners of the decoder stress matrix: 4 MiB streams (batch 1 and 7) and a
    4096-stream batch, per-stream and shared tables.  The wide batch cycles a pool of
    256 distinct streams so the CPU encoder stays out of the way."""
    if table_mode in (0, 3, -1) and dist != "exponent":
        pytest.skip("one distribution is enough for the narrow and wide-per-stream kernels")
    big = [distribution(dist, 4 << 20, 1000 + i) for i in range(7)]
    _check(gpu, orc, big[:1])
    _check(gpu, orc, big)
    pool = [distribution(dist, 4096, 50 + i) for i in range(256)]
    plains = [pool[i % 256] for i in range(4096)]
    streams = [orc.rans_encode(p) for p in pool]
    blob, offs = pack_streams([streams[i % 256] for i in range(4096)])
    out = np.frombuffer(gpu.decode_batch(blob, offs, 4096, 4096), dtype=np.uint8).reshape(4096, 4096)
    assert (out == np.stack(plains)).all()
    counts = np.sum([np.bincount(p, minlength=256) for p in pool], axis=0)
    freqs = orc.rans_freqs(counts)
    header = b"R1\0\0" + freqs.astype("<u2").tobytes()
    shared = [orc.rans_encode_shared(p, freqs) for p in pool]
    blob, offs = pack_streams([shared[i % 256] for i in range(4096)])
    out = np.frombuffer(gpu.decode_batch(blob, offs, 4096, 4096, header=header),
                        dtype=np.uint8).reshape(4096, 4096)
    assert (out == np.stack(plains)).all()


@pytest.mark.parametrize("nstr,plane", [(1, 1), (3, 4097), (40, 65537)])
def test_results_in_lent_memory_stay_their_callers_own(gpu, orc, nstr, plane, table_mode):
    """Results of host batches come in memory the library takes back when they are dropped:
    one that is still held must not change under later calls, from this thread or others."""
    if table_mode != -1:
        pytest.skip("the memory does not depend on the table layout")
    from concurrent.futures import ThreadPoolExecutor
    sets = []
    for s in range(4):
        plains = [shaped("skewed", plane, 31 * s + i) for i in range(nstr)]
        sets.append((pack_streams([orc.rans_encode(p) for p in plains]), b"".join(p.tobytes() for p in plains)))
    held = [gpu.decode_batch(*sets[s][0], nstr, plane) for s in range(2)]
    with ThreadPoolExecutor(6) as pool:
        got = list(pool.map(lambda i: bytes(gpu.decode_batch(*sets[i % 4][0], nstr, plane)), range(24)))
    assert all(g == sets[i % 4][1] for i, g in enumerate(got))
    assert [bytes(h) for h in held] == [sets[0][1], sets[1][1]]
    part = held[0][:1]
    del held
    gpu.trim()
    gpu.decode_batch(*sets[2][0], nstr, plane)
    assert bytes(part) == sets[0][1][:1]


@pytest.mark.parametrize("lead,tail", [(0, 0), (0, 63), (0, 64), (1, 0), (3, 200), (16, 64)])
def test_device_batches_wherever_they_lie(gpu, orc, lead, tail, table_mode):
    """A tensor that starts anywhere in its memory and ends where that does (it is then copied
    for the kernel's reading ahead) or before; offsets outside it are refused."""
    if table_mode != -1:
        pytest.skip("where the bytes lie does not depend on the table layout")
    import torch
    plains = [shaped("skewed", 1001, i) for i in range(9)]
    blob, offs = pack_streams([orc.rans_encode(p) for p in plains])
    whole = torch.zeros(lead + len(blob) + tail, dtype=torch.uint8, device="cuda")
    t = whole[lead:lead + len(blob)]
    t.copy_(torch.frombuffer(bytearray(blob), dtype=torch.uint8))
    out = gpu.decode_batch(t, offs, 9, 1001)
    assert out.cpu().numpy().tobytes() == b"".join(p.tobytes() for p in plains)
    table = np.frombuffer(offs, dtype="<u8").copy()
    for at, value in ((16, len(blob) - 100), (16, 1 << 63), (17, len(blob) - int(table[16]) + 1), (17, 1 << 32)):
        bad = table.copy()
        bad[at] = value
        with pytest.raises(ValueError):
            gpu.decode_batch(t, bad.tobytes(), 9, 1001)


@pytest.mark.parametrize("kind", ["int8", "int32", "int64", "strided"])
def test_device_batches_of_bytes_in_other_tensors(gpu, orc, kind, table_mode):
    """Byte values in a tensor of another type are taken by value, a strided tensor in its own order."""
    if table_mode != -1:
        pytest.skip("what the bytes come in does not depend on the table layout")
    import torch
    plains = [shaped("skewed", 1001, i) for i in range(9)]
    blob, offs = pack_streams([orc.rans_encode(p) for p in plains])
    t = torch.frombuffer(bytearray(blob), dtype=torch.uint8).cuda()
    if kind == "strided":
        two = torch.zeros(t.numel(), 2, dtype=torch.uint8, device="cuda")
        two[:, 1] = t
        t = two[:, 1]
    else:
        t = t.to(getattr(torch, kind))
    out = gpu.decode_batch(t, offs, 9, 1001)
    assert out.cpu().numpy().tobytes() == b"".join(p.tobytes() for p in plains)


@pytest.mark.parametrize("where", ["on its start", "on its end", "on what is read ahead", "beside it"])
def test_device_batches_decoded_over_their_own_streams(gpu, orc, where, table_mode):
    """`out` may share memory with the streams: they are read as they were."""
    if table_mode != -1:
        pytest.skip("where the result goes does not depend on the table layout")
    import torch
    plains = [shaped("flat", 4097, i) for i in range(40)]
    blob, offs = pack_streams([orc.rans_encode(p) for p in plains])
    n, size = len(blob), 40 * 4097
    whole = torch.zeros(3 * n + 4096, dtype=torch.uint8, device="cuda")
    at = n + 512
    whole[at:at + n] = torch.frombuffer(bytearray(blob), dtype=torch.uint8).cuda()
    lo = {"on its start": at - size + 1000, "on its end": at + n - 1000, "on what is read ahead": at + n + 3, "beside it": at - size}[where]
    out = gpu.decode_batch(whole[at:at + n], offs, 40, 4097, out=whole[lo:lo + size])
    assert out.data_ptr() == whole.data_ptr() + lo
    assert out.cpu().numpy().tobytes() == b"".join(p.tobytes() for p in plains)


@pytest.mark.parametrize("on_device", [False, True])
def test_sizes_beyond_32_bits_are_refused(gpu, orc, on_device, table_mode):
    """Never taken modulo 2^32: the stream would decode, to a part of what was asked for."""
    if table_mode != -1:
        pytest.skip("refused before any table")
    import torch
    blob, offs = pack_streams([orc.rans_encode(shaped("skewed", 64, 1))])
    src = torch.frombuffer(bytearray(blob), dtype=torch.uint8).cuda() if on_device else blob
    for plane in ((1 << 32) + 64, (1 << 63) + 1, 1 << 70):
        with pytest.raises(ValueError):
            gpu.decode_batch(src, offs, 1, plane)
    with pytest.raises(ValueError):
        gpu.decode_batch(src, offs, (1 << 32) + 1, 64)


@pytest.mark.parametrize("nstr,plane", [(5, 4097), (40, 65537)])
def test_a_refused_batch_leaves_out_alone(gpu, orc, nstr, plane, table_mode):
    """Whatever the caller's buffer is: its own, or an earlier result brought back."""
    if table_mode != -1:
        pytest.skip("the memory does not depend on the table layout")
    plains = [shaped("skewed", plane, i) for i in range(nstr)]
    want = b"".join(p.tobytes() for p in plains)
    others = [shaped("flat", plane, 77 + i) for i in range(nstr)]
    blob, offs = pack_streams([orc.rans_encode(p) for p in plains])
    streams = [orc.rans_encode(p) for p in others]
    good, good_offs = pack_streams(streams)
    bad, bad_offs = pack_streams(streams[:-1] + [streams[-1][:-200]])
    for out in (gpu.decode_batch(blob, offs, nstr, plane), bytearray(want)):
        with pytest.raises(ValueError):
            gpu.decode_batch(bad, bad_offs, nstr, plane, out=out)
        assert bytes(out) == want
        got = gpu.decode_batch(good, good_offs, nstr, plane, out=out)
        assert bytes(got) == bytes(out) == b"".join(p.tobytes() for p in others)
        if not isinstance(out, bytearray):
            assert gpu.decode_batch(blob, offs, nstr, plane, out=out[1:]) is not None       # too short: memory of its own


@pytest.mark.parametrize("nstr", [148 * 76 + 1, 13024, 28577])
@pytest.mark.parametrize("wide", ["none", "every seventh", "all"])
def test_device_batches_sorted_by_alphabet(gpu, orc, nstr, wide, table_mode):
    """More streams in one launch than full-size tables have room for (the counts are those of 148 SMs): alphabets
    are counted on the device and each class gets its instance, one of them for none or for all.  A host
    batch of this size may run in slices that are each below the line."""
    if table_mode != -1:
        pytest.skip("sorted only where the library chooses")
    import torch
    plane = 331
    every = {"none": 0, "every seventh": 7, "all": 1}[wide]
    pool = [distribution("uniform" if every and i % every == 0 else "exponent", plane, 40 + i) for i in range(70)]
    streams = [orc.rans_encode(p) for p in pool]
    live = [len(np.unique(p)) for p in pool]
    assert max(live) > 104 if every else max(live) <= 104
    blob, offs = pack_streams([streams[i % 70] for i in range(nstr)])
    t = torch.frombuffer(bytearray(blob), dtype=torch.uint8).cuda()
    want = torch.from_numpy(np.stack(pool)).cuda()[torch.arange(nstr, device="cuda") % 70].reshape(-1)
    assert torch.equal(gpu.decode_batch(t, offs, nstr, plane), want)
    for at in (0, nstr // 2, nstr - 1):                   # one stream's last word is missing
        bad = np.frombuffer(offs, dtype="<u8").copy()
        bad[2 * at + 1] -= 2
        with pytest.raises(ValueError):
            gpu.decode_batch(t, bad.tobytes(), nstr, plane)


@pytest.mark.parametrize("table_mode", [-1], ids=["auto"], indirect=True)
@pytest.mark.parametrize("per_sm", [1, 6, 7, 20, 21])
@pytest.mark.parametrize("plane", [63, 511, 513, 1031])
def test_batches_around_the_lines_between_kernels(gpu, orc, per_sm, plane, table_mode):
    """As many streams per SM as a warp with a table entry per slot each, a warp each and four to a warp take, and one
    more; planes around the eight steps and the 512 symbols that a warp takes at a time.  Uniform bytes take more
    words in eight steps than a round translates, a single symbol none."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nstr = sms * per_sm - sms // 2
    kinds = ("exponent", "uniform", "single", "two")
    pool = [distribution(kinds[i % 4], plane, 31 * i + plane) for i in range(61)]
    streams = [orc.rans_encode(p) for p in pool]
    blob, offs = pack_streams([streams[i % 61] for i in range(nstr)])
    out = np.frombuffer(gpu.decode_batch(blob, offs, nstr, plane), dtype=np.uint8).reshape(nstr, plane)
    want = np.stack([pool[i % 61] for i in range(nstr)])
    bad = np.nonzero((out != want).any(axis=1))[0]
    assert bad.size == 0, bad[:10]


@pytest.mark.parametrize("table_mode", [-1], ids=["auto"], indirect=True)
@pytest.mark.parametrize("nstr", [148 * 20, 148 * 20 + 1, 148 * 28 - 1, 148 * 28 + 1])
@pytest.mark.parametrize("plane", [1, 17, 129, 1000, 4097])
def test_device_batches_around_the_lines_between_kernels(gpu, nstr, plane, table_mode):
    """20 and 28 streams per SM (of 148) and one more: a warp each, byte tables for four to a warp, compact tables; planes
    that end anywhere in a tile, alphabets of one symbol to all of them, and one stream a word short."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(nstr + plane)
    u = torch.rand((nstr, plane), generator=gen, device="cuda")
    kind = (torch.arange(nstr, device="cuda") % 5)[:, None]
    flat, few = (u * 256).to(torch.int32), torch.log2(1 / (1 - u)).clamp_(max=40).to(torch.int32)
    planes = torch.where(kind == 0, flat, torch.where(kind == 1, few + 100, torch.where(kind == 2, torch.full_like(flat, 7),
                         torch.where(kind == 3, (flat > 250).to(torch.int32), (flat * flat) >> 8)))).to(torch.uint8)
    streams, offsets = gpu.encode_batch(planes.reshape(-1), nstr, plane)
    assert torch.equal(gpu.decode_batch(streams, offsets, nstr, plane).view(nstr, plane), planes)
    if plane >= 129:
        short = offsets.clone()
        short[2 * (nstr - nstr % 5 - 5) + 1] -= 2              # (a flat one)
        with pytest.raises(ValueError):
            gpu.decode_batch(streams, short, nstr, plane)


@pytest.mark.parametrize("table_mode", [-1], ids=["auto"], indirect=True)
@pytest.mark.parametrize("plane", [331, 2048])
def test_byte_tables_of_any_alphabet_are_built_in_little_time(gpu, plane, table_mode):
    """24 streams per SM of short planes with large alphabets, where a stream's table is most of what it takes: as long as with
    compact tables or less, and half as much again at the very most (with symbols filled in one by one 2.3 and 1.3 times)."""
    import torch
    lib, nstr = gpu.library(), 24 * torch.cuda.get_device_properties(0).multi_processor_count
    planes = torch.randint(0, 256, (nstr * plane,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(plane)).to(torch.uint8)
    streams, offsets = gpu.encode_batch(planes, nstr, plane)
    out = torch.empty_like(planes)
    cs = torch.cuda.current_stream().cuda_stream

    def took(mode):
        assert lib.lmz_gpu_set_table_mode(mode) == 0
        each = []
        for _ in range(30):
            torch.cuda._sleep(200_000)                    # (the launches are queued by the time the first one runs)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                assert lib.lmz_gpu_decode_batch_dev(None, streams.data_ptr(), offsets.data_ptr(), nstr, plane, out.data_ptr(), cs, 0) == 0
            b.record()
            b.synchronize()
            each.append(a.elapsed_time(b))
        assert torch.equal(out, planes)
        return sorted(each)[len(each) // 2]

    assert took(-1) < (1.5 if plane < 1000 else 1.15) * took(2)
