"""The save path: BF16 safetensors bytes in HBM -> an lmz archive, chunk payloads framed on the
device.  The file must be, byte for byte in its payload and chunk records, what the checker's
writer produces for the same input -- and that writer is held to the reference's own
`lmz.api.compress` output by tests/test_oracle_vs_reference.py -- and it must decode back,
on the device and on the CPU, to the source."""
import numpy as np
import pytest

from oracle import archive as oa, synth

pytestmark = pytest.mark.gpu


def _same_as_checker(path, files, **kw):
    theirs = np.fromfile(path, dtype=np.uint8)
    ours = np.frombuffer(oa.write_archive(files, **kw), dtype=np.uint8)
    a, b = oa.Archive(ours), oa.Archive(theirs)
    assert a.records.size == b.records.size
    bad = np.nonzero(a.records != b.records)[0]
    assert bad.size == 0, (int(bad[0]), a.records[bad[0]], b.records[bad[0]])
    ta = int(np.frombuffer(ours[-40:-32].tobytes(), dtype="<u8")[0])
    tb = int(np.frombuffer(theirs[-40:-32].tobytes(), dtype="<u8")[0])
    assert ta == tb and (ours[:ta] == theirs[:tb]).all()
    return theirs


def _cases():
    rng = np.random.default_rng(2)
    shard = synth.llama_shard([0], 5, scale=0.25, vocab=2000, embed=True)            # weights + all-ones norms
    noise = rng.integers(0, 65536, 300_001, dtype=np.uint16).astype("<u2").view(np.uint8)   # nothing to gain: stored chunks
    e = (120 + rng.integers(0, 3, 200_000)).astype(np.uint16)                          # both planes low-entropy
    m = rng.integers(0, 4, 200_000).astype(np.uint16)
    narrow = ((e << 7) | m).astype("<u2").view(np.uint8)
    odd = synth.safetensors_bytes([("n", "BF16", (300_001,), noise), ("w", "BF16", (200_000,), narrow),
                                   ("t", "BF16", (7,), synth.normal_bf16((7,), 3))])
    return {"shard": shard, "odd": odd}


@pytest.mark.parametrize("name", ["shard", "odd"])
@pytest.mark.parametrize("kw", [dict(mapped=True), dict(chunk_size=1 << 20), dict(chunk_size=(1 << 18) + 2)],
                         ids=["mapped", "1MiB", "256KiB+2"])
def test_device_written_archive_equals_the_checkers(gpu, tmp_path, name, kw):
    import torch
    from lmz_b200 import decode, save
    src = _cases()[name]
    files = [("m.safetensors", src)]
    path = str(tmp_path / "out.lmz")
    stats = {}
    n = save.save_archive(path, [("m.safetensors", torch.from_numpy(src.copy()).cuda())],
                          chunk_size=kw.get("chunk_size", 64 << 10), mapped=bool(kw.get("mapped")), stats=stats)
    blob = _same_as_checker(path, files, **kw)
    assert n == blob.size and stats["payload_bytes"] > 0
    assert (oa.decode_archive(blob) == src).all()
    assert (decode.decode_archive(path).cpu().numpy() == src).all()


def test_two_members_and_what_the_writer_declines(gpu, tmp_path):
    import torch
    from lmz_b200 import decode, save
    a = synth.llama_shard([0], 5, scale=0.125, vocab=1000, embed=True)
    b = synth.llama_shard([1], 6, scale=0.125)
    path = str(tmp_path / "two.lmz")
    save.save_archive(path, [("a.safetensors", torch.from_numpy(a).cuda()), ("b.safetensors", torch.from_numpy(b).cuda())])
    _same_as_checker(path, [("a.safetensors", a), ("b.safetensors", b)], mapped=True, delta=False)
    assert (decode.decode_archive(path).cpu().numpy() == np.concatenate([a, b])).all()
    f32 = synth.safetensors_bytes([("f", "F32", (100,), np.zeros(400, np.uint8))])
    with pytest.raises(ValueError, match="BF16"):
        save.save_archive(path, [("f.safetensors", torch.from_numpy(f32).cuda())])
    with pytest.raises(ValueError, match="chunk_size"):
        save.save_archive(path, [("a.safetensors", torch.from_numpy(a).cuda())], chunk_size=8 << 20)


@pytest.mark.parametrize("before", ["a longer archive", "a shorter one", "other bytes"])
def test_over_what_was_there(gpu, tmp_path, before):
    """A save over an existing file leaves the file that a save to a new one does; one that fails leaves it empty."""
    import torch
    from lmz_b200 import archive, decode, save
    a = synth.llama_shard([0], 5, scale=0.25, vocab=2000, embed=True)
    b = synth.llama_shard([1], 6, scale=0.125)
    small, large = (("b.safetensors", b), ("a.safetensors", a))
    old, new = (large, small) if before == "a longer archive" else (small, large)
    path, fresh = tmp_path / "over.lmz", tmp_path / "fresh.lmz"
    if before == "other bytes":
        path.write_bytes(bytes(range(256)) * 40000)
    else:
        save.save_archive(str(path), [(old[0], torch.from_numpy(old[1].copy()).cuda())])
    member = [(new[0], torch.from_numpy(new[1].copy()).cuda())]
    assert save.save_archive(str(path), member) == save.save_archive(str(fresh), member) == path.stat().st_size
    assert path.read_bytes() == fresh.read_bytes()
    assert (decode.load_archive(str(path)).cpu().numpy() == new[1]).all()
    with pytest.raises(ValueError):
        save.save_archive(str(path), member + [("c", torch.zeros(100, device="cuda"))])
    assert path.stat().st_size == 0
    with pytest.raises(ValueError):                       # (nothing to map)
        archive.Archive(str(path))


@pytest.mark.parametrize("mib", [20, 22])
def test_checksums_of_a_tensor_that_ends_where_its_memory_does(gpu, mib):
    """A tensor of whole 2 MiB pages fills an allocation of its own to the last byte: the checksum
    kernel reads no further."""
    import ctypes
    import zlib
    import torch
    from lmz_b200 import decode
    lib = gpu.library()
    torch.cuda.empty_cache()
    data = torch.randint(0, 256, (mib << 20,), dtype=torch.uint8, device="cuda")
    meta = torch.zeros((mib * 16, 4), dtype=torch.int32, device="cuda")
    tabs = decode._crc_tables(lib, torch.device("cuda", torch.cuda.current_device()))
    assert lib.lmz_gpu_crc32_chunks_dev(data.data_ptr(), data.numel(), 65536, tabs.data_ptr(), meta.data_ptr(),
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    got = meta[:, 3].cpu().numpy().view(np.uint32)
    host = data.cpu().numpy().reshape(-1, 65536)
    assert [int(v) for v in got] == [zlib.crc32(row) for row in host]
