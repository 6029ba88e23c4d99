"""The tensor-core tile at its edges: row tiles of 13 rows and the even split
of a few more, symbol tiles of 256 with a last one of 8 or 248, the 16-slice
input stages, and the dual-basis form of the coefficient matrices."""
import numpy as np
import pytest

SHAPES = [  # (S, slice, R, first_exponent)
    (1, 512, 13, 0), (4, 512, 14, 0), (15, 528, 12, 0), (16, 1008, 26, 3), (17, 1024, 27, 0), (31, 4, 1, 0),
    (33, 1040, 39, 65000), (80, 2544, 40, 0), (97, 512, 5, 0), (129, 4612, 8, 0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("S,slice_,R,fe", SHAPES)
def test_tensor_tile_edges(p2g, gpu, oracle, S, slice_, R, fe):
    from par2rust_b200.workloads import file_bytes

    src = file_bytes(3 * S + R, S * slice_)
    got = p2g.encode(src, slice_, R, first_exponent=fe, variant=p2g.ENCODE_TENSOR).reshape(R, slice_)
    if fe == 0:
        want = oracle.encode_fast(src, S, slice_, R).reshape(R, slice_)
    else:
        want = oracle.encode_rows(src, S, slice_, [fe + r for r in range(R)])
    assert np.array_equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("slices,tiles", [(33, 1), (48, 1), (400, 300), (32768, 40)])
def test_tile_that_gives_up(p2g, gpu, oracle, slices, tiles):
    """A stage that never arrives (the last one; one after which the input
    ring wraps, with a next tile's stages asked for; one with 2,045 behind it):
    every role gives up, the call reports it soon, and the next encode is right."""
    import time

    from par2rust_b200.workloads import file_bytes

    t0 = time.time()
    with pytest.raises(p2g.DeviceTimeout):
        p2g.check_tile_wait(slices, tiles)
    assert time.time() - t0 < 5
    src = file_bytes(slices, 40 * 1024)
    assert np.array_equal(p2g.encode(src, 1024, 15, variant=p2g.ENCODE_TENSOR), oracle.encode_fast(src, 40, 1024, 15))


def test_rows_of_the_multiplication_matrix_are_trace_runs():
    """Bit i of c * 2^j is Tr(2^(log c + log d_i + j)), d_i the basis dual to 1, 2, .., 2^15."""
    al = np.zeros(65535, np.int64)
    v = 1
    for k in range(65535):
        al[k] = v
        v = (v << 1) ^ (0x1100B if v & 0x8000 else 0)
    lg = np.zeros(65536, np.int64)
    lg[al] = np.arange(65535)
    tr = al.copy()
    z = al.copy()
    for _ in range(15):  # z -> z^2, z never 0
        z = al[2 * lg[z] % 65535]
        tr ^= z
    assert set(np.unique(tr)) <= {0, 1}
    g = np.array([[tr[(i + j) % 65535] for j in range(16)] for i in range(16)], dtype=np.int64)
    a = np.concatenate([g, np.eye(16, dtype=np.int64)], axis=1)
    for c in range(16):
        p = next(r for r in range(c, 16) if a[r, c])
        a[[c, p]] = a[[p, c]]
        for r in range(16):
            if r != c and a[r, c]:
                a[r] ^= a[c]
    dual = [int(sum(int(b) << j for j, b in enumerate(a[i, 16:]))) for i in range(16)]
    rng = np.random.default_rng(1)
    for lc in list(rng.integers(0, 65535, 200)) + [0, 65534]:
        for i in range(16):
            k = (lc + lg[dual[i]] + np.arange(16)) % 65535
            assert np.array_equal(tr[k], al[(lc + np.arange(16)) % 65535] >> i & 1)
