"""Which kernel an encode call runs on: the rule by shape (CPU), and where its
first choice cannot run (GPU): inside a stream capture, or with the device too
full for the coefficient image.  Each GPU test is a process of its own, since
the library keeps its scratch."""
import os
import subprocess
import sys
import textwrap
import time

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(code, **env):
    head = """
        import sys
        sys.path.insert(0, %r)
        import numpy as np, torch
        import par2rust_b200 as p2g
        from oracle import oracle
        from par2rust_b200.workloads import file_bytes

        def encode(src, S, size, rows, **kw):
            rec = torch.zeros((rows, size), dtype=torch.uint8, device="cuda")
            p2g.encode_device(src.data_ptr(), size, S, size, rows, rec.data_ptr(), size,
                              torch.cuda.current_stream().cuda_stream, **kw)
            return rec
    """ % ROOT
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(head) + textwrap.dedent(code)], cwd=ROOT,
                       env=dict(os.environ, **env), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_rule_counts_the_waves_of_the_given_gpu(p2g):
    """32 slices of 1 MiB, 4 rows: 2,048 tensor tiles, 14 waves of 148 SMs and 32
    of 64, against one wave of lookup tiles."""
    assert p2g.plan_encode(1 << 20, 32, 4, ctas=148) == p2g.ENCODE_TENSOR
    assert p2g.plan_encode(1 << 20, 32, 4, ctas=64) == p2g.ENCODE_LUT


# (slice, slices, rows, us on the lookup kernel, us on the tensor cores), one B200
MEASURED = [
    (100016, 8, 2, 16.3, 11.4), (1048576, 32, 2, 42.6, 34.5), (262144, 32, 32, 42.6, 36.9),
    (1048576, 16, 100, 179.2, 258.0), (4096, 1024, 1, 771.2, 38.6), (1048576, 7, 2, 18.2, 28.3),
    (65536, 8, 20, 16.3, 14.3), (1048576, 8, 8, 20.3, 34.8), (262144, 64, 32, 72.8, 49.4),
    (262144, 32, 100, 95.6, 86.3), (65536, 64, 8, 60.9, 14.6), (1048576, 8, 50, 65.3, 133.1),
    (16384, 8, 100, 16.4, 14.6),
]


@pytest.mark.parametrize("size,S,rows,lut,mma", MEASURED)
def test_rule_picks_the_kernel_that_is_faster(p2g, size, S, rows, lut, mma):
    assert p2g.plan_encode(size, S, rows) == (p2g.ENCODE_LUT if lut < mma else p2g.ENCODE_TENSOR)


def test_rule_costs_little_for_long_slices(p2g):
    """It runs on every encode call, whose launches take ~15 us."""
    p2g.plan_encode(64 << 20, 8, 4)
    t = time.perf_counter()
    for _ in range(200):
        p2g.plan_encode(64 << 20, 8, 4)
    assert (time.perf_counter() - t) / 200 < 20e-6


@pytest.mark.gpu
@pytest.mark.parametrize("warm,S,size,rows", [("LUT", 64, 16384, 20), ("TENSOR", 4, 1024, 3), ("LUT", 4, 1024, 3),
                                              ("TENSOR", 64, 16384, 20)])
def test_capture_after_one_kernel_ran(p2g, gpu, warm, S, size, rows):
    """A program that has only run one of the kernels captures a call of a
    smaller shape, whichever kernel the rule would give it."""
    _run("""
        S, size, rows = %d, %d, %d
        big = torch.from_numpy(file_bytes(1, 256 * 1024).copy()).cuda()
        encode(big, 256, 1024, 200, variant=p2g.ENCODE_%s)
        data = file_bytes(2, S * size)
        src = torch.from_numpy(data.copy()).cuda()
        g = torch.cuda.CUDAGraph()
        rec = torch.zeros((rows, size), dtype=torch.uint8, device="cuda")
        with torch.cuda.graph(g):
            p2g.encode_device(src.data_ptr(), size, S, size, rows, rec.data_ptr(), size,
                              torch.cuda.current_stream().cuda_stream)
        for _ in range(2):
            rec.zero_()
            g.replay()
            torch.cuda.synchronize()
            assert np.array_equal(rec.cpu().numpy().ravel(), oracle.encode_fast(data, S, size, rows))
    """ % (S, size, rows, warm))


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", ["LUT", "TENSOR"])
def test_replay_after_the_scratch_grew(p2g, gpu, kernel):
    """A captured call's scratch outlives its growth by later calls: here it
    grows twice, and what a free would have given back is overwritten."""
    _run("""
        S, size, rows = 64, 16384, 20
        kw = dict(variant=p2g.ENCODE_%s)
        data = file_bytes(2, S * size)
        src = torch.from_numpy(data.copy()).cuda()
        encode(src, S, size, rows, **kw)
        g = torch.cuda.CUDAGraph()
        rec = torch.zeros((rows, size), dtype=torch.uint8, device="cuda")
        with torch.cuda.graph(g):
            p2g.encode_device(src.data_ptr(), size, S, size, rows, rec.data_ptr(), size,
                              torch.cuda.current_stream().cuda_stream, **kw)
        want = oracle.encode_fast(data, S, size, rows)
        for S2, rows2 in ((1024, 100), (2048, 200)):
            big = file_bytes(3, S2 * 512)
            got = encode(torch.from_numpy(big.copy()).cuda(), S2, 512, rows2, **kw)
            hogs = [torch.full((1 << 20,), 0xAB, dtype=torch.uint8, device="cuda") for _ in range(64)]
            rec.zero_()
            g.replay()
            torch.cuda.synchronize()
            assert np.array_equal(rec.cpu().numpy().ravel(), want)
            assert np.array_equal(got.cpu().numpy().ravel(), oracle.encode_fast(big, S2, 512, rows2))
            assert all(bool((h == 0xAB).all()) for h in hogs)
    """ % kernel)


FULL = """
    S, size, rows = 32768, 64, 512  # image 2.2 GB, bases 0.5 GB
    data = file_bytes(2, S * size)
    src = torch.from_numpy(np.concatenate([data, np.zeros(16, np.uint8)])).cuda()
    bufs = p2g.DeviceJobBuffers(S, 1, size, rows, src.device)
    want = oracle.encode_rows(data, S, size, [0, 1, 300, 511])
    small = encode(src, 64, size, 20, variant=p2g.ENCODE_TENSOR)  # the library is up, a small image is held
    torch.cuda.synchronize()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (1500 << 20), dtype=torch.uint8, device="cuda")

    def check(rec):
        torch.cuda.synchronize()
        assert np.array_equal(rec.view(rows, -1)[[0, 1, 300, 511], :size].cpu().numpy(), want)

    def refused(call):
        try:
            call()
        except p2g.OutOfMemory:
            return
        raise AssertionError("accepted")

    def job(**kw):
        bufs.recovery.zero_()
        return p2g.run_device_job(src, [S * size], [b"f"], size, rows, bufs, skip_hash_full=True, **kw).recovery

    def batch(flags=0):
        bufs.recovery.zero_()
        b = p2g.Batch([p2g.BatchJobSpec(src, [S * size], [b"f"], size, rows, bufs)], flags)
        b.launch()
        torch.cuda.synchronize()
        b.check()
        b.close()
        return bufs.recovery
"""


@pytest.mark.gpu
def test_image_that_does_not_fit(p2g, gpu):
    """Left to the rule, an encode, a job and a batch run on the lookup kernel
    then; the forced tensor kernel reports that memory is short."""
    _run(FULL + """
    check(encode(src, S, size, rows))
    check(job())
    check(batch())
    refused(lambda: encode(src, S, size, rows, variant=p2g.ENCODE_TENSOR))
    refused(lambda: job(variant=p2g.ENCODE_TENSOR))
    refused(lambda: batch(p2g.BATCH_TENSOR))
    """)


@pytest.mark.gpu
def test_image_that_does_not_fit_forced_by_the_environment(p2g, gpu):
    _run(FULL + """
    refused(lambda: encode(src, S, size, rows))
    refused(job)
    refused(batch)
    """, P2G_ENCODE_VARIANT="tensor")
