"""The staged MD5 streams and the folded CRC32 at their edges: message lengths
around the 64-byte copy units, the 1,024-byte fold groups and the 16 KiB parts, every 4-byte start within a 16-byte quad, warps whose
lanes differ in length, and stream counts around a warp, a CTA and the
switch to 256 lanes a CTA (more than 148 x 128 streams)."""
import ctypes as C
import hashlib
import zlib

import pytest

pytestmark = pytest.mark.gpu


def _device(n, seed):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=g)


# slice sizes around the ring's units (64 B), its depth (12 units, 8 ahead) and one block
SLICES = [(1, 4, 4, 0), (31, 60, 64, 0), (33, 64, 64, 0), (129, 68, 68, 4), (40, 124, 128, 8), (200, 508, 512, 0),
          (257, 576, 580, 12), (64, 772, 776, 4), (130, 1028, 1040, 0), (128, 4092, 4096, 0), (19000, 132, 132, 0)]


@pytest.mark.parametrize("count,size,stride,off", SLICES)
def test_slice_streams(p2g, gpu, count, size, stride, off):
    import torch

    src = _device(off + count * stride, count + size)
    out = torch.zeros(20 * count, dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert p2g.lib().p2g_slice_checksums(src.data_ptr() + off, stride, count, size, out.data_ptr(),
                                         p2g.DEVICE_POINTERS, st) == 0
    host = src.cpu().numpy()[off:]
    want = b"".join(hashlib.md5(s).digest() + zlib.crc32(s).to_bytes(4, "little")
                    for s in (host[i * stride:i * stride + size].tobytes() for i in range(count)))
    assert out.cpu().numpy().tobytes() == want


@pytest.mark.parametrize("count,size,stride,off", SLICES)
def test_packet_streams(p2g, gpu, count, size, stride, off):
    """The same rows behind the packet's 36-byte prefix (set id, type, exponent)."""
    import torch

    src = _device(off + count * stride, count + 3 * size)
    out = torch.zeros(16 * count, dtype=torch.uint8, device="cuda")
    sid = bytes(range(16))
    st = torch.cuda.current_stream().cuda_stream
    assert p2g.lib().p2g_recovery_packet_md5(sid, src.data_ptr() + off, stride, count, size, 7, out.data_ptr(),
                                             p2g.DEVICE_POINTERS, st) == 0
    host = src.cpu().numpy()[off:]
    want = b"".join(hashlib.md5(sid + b"PAR 2.0\0RecvSlic" + (7 + i).to_bytes(4, "little") +
                                host[i * stride:i * stride + size].tobytes()).digest() for i in range(count))
    assert out.cpu().numpy().tobytes() == want


def test_file_streams_of_mixed_lengths(p2g, gpu):
    """Lanes of one warp with different lengths and starts 4 bytes apart."""
    import torch

    lengths = [1, 3, 55, 56, 63, 64, 65, 119, 128, 191, 1000, 4095, 16383, 16384, 16385, 40001] * 9
    pitch = 40960 + 4
    src = _device(len(lengths) * pitch + 16, 5)
    n = len(lengths)
    ptrs = (C.c_void_p * n)(*[src.data_ptr() + i * pitch for i in range(n)])
    lens = (C.c_uint64 * n)(*lengths)
    out = torch.zeros(32 * n, dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert p2g.lib().p2g_file_hashes(ptrs, lens, n, out.data_ptr(), out.data_ptr() + 16 * n, p2g.DEVICE_POINTERS,
                                     st) == 0
    host = src.cpu().numpy()
    data = [host[i * pitch:i * pitch + k].tobytes() for i, k in enumerate(lengths)]
    got = out.cpu().numpy().tobytes()
    assert got[:16 * n] == b"".join(hashlib.md5(d).digest() for d in data)
    assert got[16 * n:] == b"".join(hashlib.md5(d[:16384]).digest() for d in data)


@pytest.mark.parametrize("pitch", [40960, 40976])
def test_file_streams_that_all_start_16_byte_aligned(p2g, gpu, pitch):
    """The unshifted ring of device-pointer file hashes, lanes of different lengths."""
    import torch

    lengths = [1, 63, 64, 65, 575, 576, 577, 767, 768, 16383, 16384, 16385, 40001] * 11
    src = _device(len(lengths) * pitch, pitch)
    n = len(lengths)
    ptrs = (C.c_void_p * n)(*[src.data_ptr() + i * pitch for i in range(n)])
    assert all(p % 16 == 0 for p in ptrs)
    lens = (C.c_uint64 * n)(*lengths)
    out = torch.zeros(32 * n, dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert p2g.lib().p2g_file_hashes(ptrs, lens, n, out.data_ptr(), out.data_ptr() + 16 * n, p2g.DEVICE_POINTERS,
                                     st) == 0
    host = src.cpu().numpy()
    data = [host[i * pitch:i * pitch + k].tobytes() for i, k in enumerate(lengths)]
    assert out.cpu().numpy().tobytes() == b"".join(hashlib.md5(d).digest() for d in data) + b"".join(
        hashlib.md5(d[:16384]).digest() for d in data)


# around 1, 2, 3, 4 and more fold groups of 1,024 B; around 2, 4, 8 and 16 parts of a slice (16 KiB each at least)
CRC_SIZES = [(3, 1020), (3, 1024), (3, 1028), (2, 2048), (2, 2052), (5, 3076), (4, 4092), (4, 4100), (1, 32764),
             (17, 32768), (2, 32772), (3, 65540), (1, 131076), (9, 262144), (2, 262148), (1, 1048580), (2400, 1032)]


@pytest.mark.parametrize("count,size", CRC_SIZES)
def test_slice_crc(p2g, gpu, count, size):
    src = _device(count * size, size).cpu().numpy()
    got = p2g.slice_checksums(src, size)
    for i in range(count):
        s = src[i * size:(i + 1) * size].tobytes()
        assert got[i].crc32 == zlib.crc32(s) and got[i].md5 == hashlib.md5(s).digest(), i


def test_slice_crc_in_device_job(p2g, gpu):
    """CRC items of one slice to a warp and of several warps to a slice."""
    import torch

    for size, slices in ((1 << 20, 5), (16388, 300), (65536, 70)):
        src = _device(slices * size + 16, size)
        bufs = p2g.run_device_job(src, [slices * size - 5], [b"f"], size, 1, skip_hash_full=True)
        torch.cuda.synchronize()
        host = src.cpu().numpy()
        got = bufs.checksums.cpu().numpy().reshape(slices, 20)
        for i in range(slices):
            s = host[i * size:(i + 1) * size].tobytes()
            assert got[i].tobytes() == hashlib.md5(s).digest() + zlib.crc32(s).to_bytes(4, "little"), (size, i)


def test_staged_host_uploads(p2g, gpu, oracle):
    """Pageable inputs around the staging chunks (1 MiB): one run of bytes,
    many pieces with gaps between them, and rows padded to another stride."""
    import numpy as np

    rng = np.random.default_rng(9)
    for size, count in ((1 << 20, 1), ((1 << 20) + 4, 3), (262140, 21), (1028, 4097)):
        src = rng.integers(0, 256, size * count, dtype=np.uint8)
        got = p2g.slice_checksums(src, size)
        assert [(c.md5, c.crc32) for c in got] == [
            (hashlib.md5(s).digest(), zlib.crc32(s)) for s in (src[i * size:(i + 1) * size].tobytes() for i in range(count))]
    lengths = [1, (1 << 20) - 1, 15, (1 << 20) + 1, 3 << 20, 0, 7, 700_001]
    files = [rng.integers(0, 256, n, dtype=np.uint8).tobytes() for n in lengths]
    assert p2g.file_hashes(files) == [(hashlib.md5(f).digest(), hashlib.md5(f[:16384]).digest()) for f in files]
    assert p2g.file_hashes([bytearray(f) for f in files]) == p2g.file_hashes(files)
    S, size, R = 130, 16388, 3  # 16,400-byte rows on the device
    src = rng.integers(0, 256, S * size, dtype=np.uint8)
    assert np.array_equal(p2g.encode(src, size, R), oracle.encode_fast(src, S, size, R))


@pytest.mark.parametrize("size", [4096, 1 << 20])  # the driver's copy, the staged one
def test_null_host_buffers_are_refused(p2g, gpu, size):
    out, one = (C.c_uint8 * 4096)(), C.create_string_buffer(size)
    lib, lens = p2g.lib(), (C.c_uint64 * 2)(size, size)
    files = (C.c_void_p * 2)(C.addressof(one), None)
    job = p2g._ffi.p2g_encode_job(src=None, src_stride=size, input_count=2, slice_size=size, recovery_count=1,
                                  first_exponent=0, recovery=C.addressof(one), recovery_stride=size,
                                  flags=p2g.HOST_POINTERS, stream=None)
    calls = [lambda: lib.p2g_slice_checksums(None, size, 2, size, out, p2g.HOST_POINTERS, None),
             lambda: lib.p2g_recovery_packet_md5(bytes(16), None, size, 2, size, 0, out, p2g.HOST_POINTERS, None),
             lambda: lib.p2g_file_hashes(files, lens, 2, out, out, p2g.HOST_POINTERS, None),
             lambda: lib.p2g_encode(C.byref(job))]
    for call in calls:
        with pytest.raises(p2g.CudaError):
            p2g._check(call())
