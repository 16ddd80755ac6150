"""GPU batch encoder against the CPU oracle's encoder (itself held byte-identical to the
reference's, tests/test_oracle_golden.py): the streams must be the same bytes, and they
must decode back through the GPU decoder."""
import numpy as np
import pytest

from helpers import DISTRIBUTIONS, distribution, shaped, SHAPES

pytestmark = pytest.mark.gpu


def _check(gpu, orc, plains):
    nstr, plane = len(plains), plains[0].size
    got = gpu.encode_batch(b"".join(p.tobytes() for p in plains), nstr, plane)
    assert got is not None, gpu.last_error()
    streams, offsets = got
    offs = np.frombuffer(offsets, dtype="<u8").reshape(nstr, 2)
    pos = 0
    for i, p in enumerate(plains):
        want = orc.rans_encode(p)
        o, n = int(offs[i, 0]), int(offs[i, 1])
        assert o == pos, f"stream {i} is not packed behind its predecessor"
        assert n == len(want), f"stream {i}: {n} bytes, the reference writes {len(want)}"
        assert streams[o:o + n] == want, f"stream {i} differs from the reference's bytes"
        pos += n
    assert pos == len(streams)
    back = gpu.decode_batch(streams, offsets, nstr, plane)
    assert bytes(back) == b"".join(p.tobytes() for p in plains)


@pytest.mark.parametrize("name", list(SHAPES))
@pytest.mark.parametrize("plane", [1, 7, 8, 9, 127, 128, 129, 4096, 4097, 65537])
def test_shapes_and_ragged_planes(gpu, orc, name, plane):
    for nstr in (1, 5, 33):
        if plane > 4097 and nstr > 5:
            continue
        _check(gpu, orc, [shaped(name, plane, hash((name, plane, nstr, i)) & 0xFFFF) for i in range(nstr)])


@pytest.mark.parametrize("dist", DISTRIBUTIONS)
@pytest.mark.parametrize("n", [1, 17, 4096, 65536, 1 << 20])
def test_stress_distributions(gpu, orc, dist, n):
    nstr = 3 if n >= 65536 else 40
    _check(gpu, orc, [distribution(dist, n, 7 * i + n) for i in range(nstr)])


def test_device_tensors_round_trip(gpu, orc):
    import torch
    plains = [distribution("exponent", 32768, i) for i in range(200)]
    t = torch.from_numpy(np.concatenate(plains)).cuda()
    streams, offs = gpu.encode_batch(t, 200, 32768)
    assert streams.is_cuda and offs.is_cuda and offs.numel() == 400
    back = gpu.decode_batch(streams, offs, 200, 32768)
    assert torch.equal(back, t)
    o = offs.cpu().numpy().reshape(200, 2)
    s = streams.cpu().numpy()
    assert s[o[17, 0]:o[17, 0] + o[17, 1]].tobytes() == orc.rans_encode(plains[17])


def test_arguments(gpu):
    assert gpu.encode_batch(b"", 0, 16) == (b"", b"")
    with pytest.raises(ValueError):
        gpu.encode_batch(b"abc", 2, 16)
    with pytest.raises(ValueError):
        gpu.encode_batch(b"abc", 1, 0)


def test_random_round_trips(gpu, orc):
    """Seeded random planes - alphabet size, skew, length and batch size all drawn - through
    encode_batch and back through decode_batch in every table mode; the first stream of
    every batch is also held to the oracle's encoder."""
    rng = np.random.default_rng(20261125)
    lib = gpu.library()
    try:
        for trial in range(60):
            plane = int(rng.choice([1, 3, 64, 129, 1000, 4096, 20000, 70001]))
            nstr = int(rng.choice([1, 2, 9, 33, 130])) if plane <= 4096 else int(rng.choice([1, 3, 7]))
            live = int(rng.integers(1, 257))
            syms = rng.choice(256, live, replace=False)
            weights = rng.random(live) ** rng.integers(1, 8)
            weights /= weights.sum()
            data = syms[rng.choice(live, size=nstr * plane, p=weights)].astype(np.uint8)
            streams, offsets = gpu.encode_batch(data.tobytes(), nstr, plane)
            o = np.frombuffer(offsets, dtype="<u8").reshape(nstr, 2)
            assert streams[:int(o[0, 1])] == orc.rans_encode(data[:plane])
            lib.lmz_gpu_set_table_mode([0, 2, 3, -1][trial % 4])
            assert bytes(gpu.decode_batch(streams, offsets, nstr, plane)) == data.tobytes(), (trial, plane, nstr, live)
    finally:
        lib.lmz_gpu_set_table_mode(-1)


@pytest.mark.parametrize("plane", [511_999, 512_000, 512_001, 1_024_016])
@pytest.mark.parametrize("dist", ["single", "two", "uniform"])
def test_counts_past_one_stretch_of_the_lanes_counters(gpu, orc, dist, plane):
    """Planes around the lengths at which the encoder sums its 16-bit counters: all of one
    symbol (a lane's counter at its fullest), next to all of one, and every symbol."""
    _check(gpu, orc, [distribution(dist, plane, 5 * i + plane) for i in range(3)])


def test_device_results_are_there_when_they_are_returned(gpu, orc):
    """Streams and offsets may be read at once on any stream, in any thread."""
    import torch
    plain = distribution("exponent", 65536, 3)
    want = torch.frombuffer(bytearray(orc.rans_encode(plain)), dtype=torch.uint8).cuda()
    t = torch.from_numpy(np.tile(plain, 2000)).cuda()
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        streams, offs = gpu.encode_batch(t, 2000, 65536)
        assert torch.cuda.current_stream().query()
        with torch.cuda.stream(other):
            same = torch.equal(streams.reshape(2000, -1), want.expand(2000, -1))
        assert same and offs.numel() == 4000


def test_strided_device_planes(gpu, orc):
    import torch
    plains = [distribution("exponent", 5000, i) for i in range(3)]
    two = torch.zeros(15000, 2, dtype=torch.uint8, device="cuda")
    two[:, 1] = torch.from_numpy(np.concatenate(plains)).cuda()
    streams, _offs = gpu.encode_batch(two[:, 1], 3, 5000)
    assert streams.cpu().numpy().tobytes() == b"".join(orc.rans_encode(p) for p in plains)


@pytest.mark.parametrize("lead", [0, 1, 2, 7])
@pytest.mark.parametrize("plane", [127, 128, 129, 511, 640, 2049])
def test_tiles_that_fill_their_buffer(gpu, orc, lead, plane):
    """Next to each other in a warp: planes whose every tile fills two pieces (each symbol once or twice), one piece every
    few tiles, none at all; both halves of the alphabet, wherever the planes lie in memory."""
    import torch
    rng = np.random.default_rng(plane + lead)
    plains = [rng.permutation(np.arange(plane) % 256).astype(np.uint8), distribution("exponent", plane, lead),
              np.full(plane, 255, np.uint8), rng.choice([127, 128], plane).astype(np.uint8), distribution("uniform", plane, 5)]
    t = torch.zeros(lead + 5 * plane, dtype=torch.uint8, device="cuda")
    t[lead:] = torch.from_numpy(np.concatenate(plains)).cuda()
    streams, _offs = gpu.encode_batch(t[lead:], 5, plane)
    assert streams.cpu().numpy().tobytes() == b"".join(orc.rans_encode(p) for p in plains)
