"""GPU parity at the edges of the kernels' variants: tile and vector remainders,
row alignments and the sizes at which a dispatch changes kernel.  Same oracle,
canaries and bounds as test_gpu_parity.py."""
import numpy as np
import pytest

from test_gpu_parity import GUARD, Guarded, bits, run, softmax_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import fe2o3_b200 as fe
    ctx = fe.GpuContext(0)
    return fe, ctx, ctx.default_stream()


# ---- exact-order GEMM: 32 x 64 tiles, k in blocks of 32
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (32, 64, 32), (33, 65, 33), (31, 63, 31), (65, 1, 64), (1, 130, 97), (100, 68, 64),
                                   # 16 x 64 and 32 x 64 tiles, rows on 16 bytes and not; three tiles of k in flight
                                   (1600, 1532, 70), (1601, 1533, 31), (520, 516, 100), (500, 700, 97)])
def test_scalar_gemm_tile_edges_bit_exact(gpu, orc, m, n, k):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    a, b = synth.uniform_f32(0, 1, m * k), synth.uniform_f32(0, 2, k * n)
    A, B = Guarded(fe, stream, a), Guarded(fe, stream, b)
    Cb = Guarded(fe, stream, np.full(m * n, np.nan, np.float32))
    run(fe, ctx, stream, "scalar_gemm_v1", a=A.slice, b=B.slice, c=Cb.slice, m=m, n=n, k=k)
    assert (bits(Cb.read()) == bits(orc.gemm_f32(m, n, k, a, b))).all()
    A.unchanged(); B.unchanged()


# bf16 operands: products that are exact in f32 are fused with their sum, tiles with values that may leave its range are not
@pytest.mark.parametrize("low,high", [(65, 189), (60, 189), (65, 192), (1, 254), (0, 255)])
@pytest.mark.parametrize("m,n,k,pad", [(33, 65, 100, 0), (70, 200, 64, 3), (1700, 1500, 40, 1)])
def test_exact_bf16_gemm_any_exponent_bit_exact(gpu, orc, m, n, k, pad, low, high):
    fe, ctx, stream = gpu
    rng = np.random.default_rng(low * 1000 + high)
    lda, ldb = k + pad, n + pad

    def values(count):
        v = (rng.integers(0, 2, count) << 15 | rng.integers(low, high + 1, count) << 7 | rng.integers(0, 128, count)).astype(np.uint16)
        v[rng.random(count) < 0.05] = 0
        return v
    a, b = values((m - 1) * lda + k), values((k - 1) * ldb + n)
    c = values(2 * m * n).view(np.float32)
    c[~np.isfinite(c)] = 1.0
    A, B, Cb = Guarded(fe, stream, a), Guarded(fe, stream, b), Guarded(fe, stream, c)
    run(fe, ctx, stream, "tiled_gemm_general_v1", schedule=fe.SCHEDULE_EXACT_ORDER, a=A.slice, b=B.slice, c=Cb.slice, m=m, n=n, k=k,
        lda=lda, ldb=ldb, ldc=n, alpha=0.5, beta=-0.25)
    want = orc.gemm_bf16(m, n, k, a, b, lda=lda, ldb=ldb, ldc=n, alpha=0.5, beta=-0.25, c=c)
    got = Cb.read()
    assert (np.isnan(got) == np.isnan(want)).all()
    assert (bits(got) == bits(want))[~np.isnan(want)].all()


# f32 operands: the tile is the one that was measured to be the fastest (launch_gemm_exact), with rows on 16 bytes and not
@pytest.mark.parametrize("rows,m,n,k", [(16, 301, 1036, 100), (16, 801, 804, 100), (16, 1001, 1001, 65), (32, 768, 768, 64), (32, 900, 900, 36),
                                        (32, 701, 701, 65), (32, 1201, 1201, 33), (64, 2301, 2300, 252), (64, 2301, 2297, 251)])
def test_scalar_gemm_takes_the_fastest_tile_bit_exact(gpu, orc, rows, m, n, k):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    a, b = synth.uniform_f32(0, 1, m * k), synth.uniform_f32(0, 2, k * n)
    A, B, Cb = Guarded(fe, stream, a), Guarded(fe, stream, b), Guarded(fe, stream, np.full(m * n, np.nan, np.float32))
    prepared = fe.prepare(ctx, "scalar_gemm_v1", a=A.slice, b=B.slice, c=Cb.slice, m=m, n=n, k=k)
    assert prepared.geometry.grid[0] == -(-m // rows) * -(-n // 64)
    for _ in range(3):   # (the later ones start early)
        prepared.launch(stream)
    prepared.launch_and_wait(stream)
    assert (bits(Cb.read()) == bits(orc.gemm_f32(m, n, k, a, b))).all()
    A.unchanged(); B.unchanged()


# bf16 operands, a case for each tile: 16 x 32, 32 x 64 and 64 x 64, with and without old values; rows at odd addresses too
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("rows,cols,m,n,k", [(16, 32, 304, 1008, 112), (32, 64, 512, 2000, 80), (64, 64, 1712, 1504, 48)])
def test_exact_bf16_gemm_every_tile_bit_exact(gpu, orc, rows, cols, m, n, k, offset):
    fe, ctx, stream = gpu
    rng = np.random.default_rng(m + offset)
    values = lambda count: (rng.normal(0, 1, count).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    a, b, c = values(m * k), values(k * n), rng.normal(0, 1, m * n).astype(np.float32)
    A, B = (Guarded(fe, stream, np.concatenate([np.zeros(offset, np.uint16), v])) for v in (a, b))
    for update in (False, True):
        # an odd size where the shape allows one
        mm, nn, kk = (m - 1, n - 3, k - 1) if update and offset else (m, n, k)
        Cb = Guarded(fe, stream, c[:mm * nn])
        args = dict(schedule=fe.SCHEDULE_EXACT_ORDER, a=A.buf.view(GUARD + offset, mm * kk), b=B.buf.view(GUARD + offset, kk * nn), c=Cb.slice,
                    m=mm, n=nn, k=kk)
        if update:
            prepared = fe.prepare(ctx, "tiled_gemm_general_v1", lda=kk, ldb=nn, ldc=nn, alpha=0.5, beta=-0.25, **args)
            want = orc.gemm_bf16(mm, nn, kk, a[:mm * kk], b[:kk * nn], lda=kk, ldb=nn, ldc=nn, alpha=0.5, beta=-0.25, c=c[:mm * nn])
        else:
            prepared = fe.prepare(ctx, "tiled_gemm_v1", **args)
            want = orc.gemm_bf16_rows(mm, nn, kk, a, b).ravel()
        assert prepared.geometry.grid[0] == -(-mm // rows) * -(-nn // cols)
        prepared.launch_and_wait(stream)
        assert (bits(Cb.read()) == bits(want.ravel())).all()


# more tiles in one direction than a second grid dimension holds (65535)
@pytest.mark.parametrize("m,n", [(1, 5_000_000), (5_000_000, 1), (2, 65535 * 64 + 1)])
def test_scalar_gemm_long_results_bit_exact(gpu, m, n):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    a, b = synth.uniform_f32(0, 1, m), synth.uniform_f32(0, 2, n)
    A, B = Guarded(fe, stream, a), Guarded(fe, stream, b)
    Cb = Guarded(fe, stream, np.full(m * n, np.nan, np.float32))
    run(fe, ctx, stream, "scalar_gemm_v1", a=A.slice, b=B.slice, c=Cb.slice, m=m, n=n, k=1)
    want = np.float32(0) + a[:, None] * b[None, :]   # one product, added to +0
    assert (bits(Cb.read()) == bits(want).ravel()).all()


# ---- tensor-core GEMM: outputs that the copy engine does not write (alpha/beta form, C at any alignment)
@pytest.mark.parametrize("m,n,k,ldc,offset", [(129, 40, 64, 40, 0), (128, 256, 64, 257, 0), (200, 136, 96, 140, 1), (257, 300, 72, 304, 0),
                                              (16, 1000, 128, 1001, 3)])
def test_gemm_tcgen05_direct_output_exact(gpu, orc, m, n, k, ldc, offset):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    lda, ldb = (k + 7) // 8 * 8, (n + 7) // 8 * 8
    a = synth.gemm_inputs_v1((m - 1) * lda + k, 1, 1, 5)[0]   # dyadic alphabet: every summation order is exact
    b = synth.gemm_inputs_v1(1, (k - 1) * ldb + n, 1, 6)[1]
    size = (m - 1) * ldc + n
    c = synth.uniform_f32(0, 9, size)
    A, B = Guarded(fe, stream, a), Guarded(fe, stream, b)
    for alpha, beta in ((2.0, -1.0), (1.0, 0.0)):
        Cb = Guarded(fe, stream, np.concatenate([np.zeros(offset, np.float32), c]))
        run(fe, ctx, stream, "tiled_gemm_general_v1", schedule=fe.SCHEDULE_TCGEN05, a=A.slice, b=B.slice,
            c=Cb.buf.view(GUARD + offset, size), m=m, n=n, k=k, lda=lda, ldb=ldb, ldc=ldc, alpha=alpha, beta=beta)
        want = orc.gemm_bf16(m, n, k, a, b, lda=lda, ldb=ldb, ldc=ldc, alpha=alpha, beta=beta, c=c)
        got = Cb.read()[offset:]
        for r in range(m):
            assert (bits(got[r * ldc:r * ldc + n]) == bits(want[r * n:(r + 1) * n])).all(), r
            assert (bits(got[r * ldc + n:(r + 1) * ldc]) == bits(c[r * ldc + n:(r + 1) * ldc])).all(), r


# ---- tensor-core GEMM tile shapes: 64, 128 and 256 columns, and pairs of SMs (k above 1024) whose second half has
# no rows or no columns
@pytest.mark.parametrize("m,n,k,ldc,beta", [(1, 130, 1025, 131, -1.0), (129, 72, 520, 72, 0.0), (1000, 1000, 96, 1003, 0.5),
                                            (1100, 2050, 64, 2052, 0.0), (1281, 1912, 1032, 1912, 0.0), (1281, 2000, 1100, 2003, -1.0),
                                            (700, 3400, 1040, 3400, 0.0), (700, 3400, 72, 3400, 0.0),
                                            # 192 columns: C in vectors and by elements, tiles that end inside
                                            (1000, 3001, 1100, 3004, -0.25), (1000, 2900, 200, 2903, 1.0)])
def test_gemm_tile_shapes_exact(gpu, orc, m, n, k, ldc, beta):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    lda, ldb = (k + 7) // 8 * 8, (n + 7) // 8 * 8
    a = synth.gemm_inputs_v1((m - 1) * lda + k, 1, 1, 5)[0]   # dyadic alphabet: every summation order is exact
    b = synth.gemm_inputs_v1(1, (k - 1) * ldb + n, 1, 6)[1]
    c = synth.uniform_f32(0, 9, (m - 1) * ldc + n)
    A, B, Cb = Guarded(fe, stream, a), Guarded(fe, stream, b), Guarded(fe, stream, c)
    run(fe, ctx, stream, "tiled_gemm_general_v1", schedule=fe.SCHEDULE_TCGEN05, a=A.slice, b=B.slice, c=Cb.slice, m=m, n=n, k=k,
            lda=lda, ldb=ldb, ldc=ldc, alpha=1.0, beta=beta)
    want = orc.gemm_bf16(m, n, k, a, b, lda=lda, ldb=ldb, ldc=ldc, alpha=1.0, beta=beta, c=c)
    got = Cb.read()
    for r in range(m):
        assert (bits(got[r * ldc:r * ldc + n]) == bits(want[r * n:(r + 1) * n])).all(), r
        assert (bits(got[r * ldc + n:(r + 1) * ldc]) == bits(c[r * ldc + n:(r + 1) * ldc])).all(), r


# packed operands, one size for each tile shape: 64, 128, 192, 256 columns and pairs
@pytest.mark.parametrize("m,n,k", [(512, 512, 512), (1536, 1536, 512), (1008, 3008, 1104), (2048, 2048, 512), (2304, 2304, 1104)])
def test_tiled_gemm_v1_tile_shapes_exact(gpu, m, n, k):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    a, b = synth.gemm_inputs_v1(m * k, 1, 1, 5)[0], synth.gemm_inputs_v1(1, k * n, 1, 6)[1]
    A, B = Guarded(fe, stream, a), Guarded(fe, stream, b)
    Cb = Guarded(fe, stream, np.zeros(m * n, np.float32))
    run(fe, ctx, stream, "tiled_gemm_v1", a=A.slice, b=B.slice, c=Cb.slice, m=m, n=n, k=k)
    wide = lambda v: (v.astype(np.uint32) << 16).view(np.float32)
    want = wide(a).reshape(m, k) @ wide(b).reshape(k, n)   # dyadic alphabet: every summation order is exact
    assert (Cb.read().reshape(m, n) == want).all()


# ring lengths: fewer k blocks than stages, as many, and a ring that ends inside a tile, two rounds of tiles
@pytest.mark.parametrize("k", [8, 64, 448, 520, 576, 1088])
@pytest.mark.parametrize("m,n", [(100, 100), (2600, 2600), (1300, 5000)])
def test_gemm_ring_lengths_exact(gpu, m, n, k):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    a, b = synth.gemm_inputs_v1(m * k, 1, 1, 5)[0], synth.gemm_inputs_v1(1, k * ((n + 7) // 8 * 8), 1, 6)[1]
    ldb = (n + 7) // 8 * 8
    A, B = Guarded(fe, stream, a), Guarded(fe, stream, b[:(k - 1) * ldb + n])
    Cb = Guarded(fe, stream, np.zeros(m * n, np.float32))
    run(fe, ctx, stream, "tiled_gemm_general_v1", schedule=fe.SCHEDULE_TCGEN05, a=A.slice, b=B.slice, c=Cb.slice, m=m, n=n, k=k,
        lda=k, ldb=ldb, ldc=n, alpha=1.0, beta=0.0)
    wide = lambda v: (v.astype(np.uint32) << 16).view(np.float32)
    want = wide(a).reshape(m, k) @ wide(b).reshape(k, ldb)[:, :n]   # dyadic alphabet: every summation order is exact
    assert (Cb.read().reshape(m, n) == want).all()


# Every tile shape with an edge inside its last tiles, by the count of its blocks: rows x columns of a tile, and blocks a tile.
# Pairs of SMs: the last pair's second block has no rows or 42 of them, and no columns or two.
SHAPES = {64: (128, 64, 1), 128: (128, 128, 1), 192: (128, 192, 1), 256: (128, 256, 1), "pair": (256, 256, 2)}


def shape_is(geometry, shape, m, n):
    rows, cols, blocks = SHAPES[shape]
    tiles = -(-m // rows) * -(-n // cols)
    return geometry.grid[0] == blocks * min(tiles, 148 // blocks)


def exact_product(a, b, m, n, k, lda, ldb):   # dyadic alphabet: every summation order is exact
    wide = lambda v: (v.astype(np.uint32) << 16).view(np.float32)
    full = lambda v, rows, ld: np.concatenate([wide(v), np.zeros(rows * ld - v.size, np.float32)]).reshape(rows, ld)
    return full(a, m, lda)[:, :k] @ full(b, k, ldb)[:, :n]


@pytest.mark.parametrize("pad,offset", [(4, 0), (3, 1)])   # C in vectors, and by elements
@pytest.mark.parametrize("shape,m,n,k", [(64, 300, 3001, 700), (128, 1281, 1400, 300), (192, 1281, 2300, 300), (256, 1281, 2700, 300),
                                         ("pair", 1281, 2900, 1500), ("pair", 1281, 2946, 1500), ("pair", 1450, 2946, 1500),
                                         ("pair", 2200, 2400, 1500)])   # (two rounds)
def test_gemm_update_every_tile_shape_exact(gpu, shape, m, n, k, pad, offset):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    lda, ldb, ldc = (k + 7) // 8 * 8, (n + 7) // 8 * 8, (n + 3) // 4 * 4 + pad
    a = synth.gemm_inputs_v1((m - 1) * lda + k, 1, 1, 5)[0]
    b = synth.gemm_inputs_v1(1, (k - 1) * ldb + n, 1, 6)[1]
    size = (m - 1) * ldc + n
    c = synth.uniform_f32(0, 9, size)
    A, B, Cb = Guarded(fe, stream, a), Guarded(fe, stream, b), Guarded(fe, stream, np.concatenate([np.zeros(offset, np.float32), c]))
    prepared = fe.prepare(ctx, "tiled_gemm_general_v1", schedule=fe.SCHEDULE_TCGEN05, a=A.slice, b=B.slice, c=Cb.buf.view(GUARD + offset, size),
                          m=m, n=n, k=k, lda=lda, ldb=ldb, ldc=ldc, alpha=0.5, beta=-0.25)
    assert shape_is(prepared.geometry, shape, m, n)
    prepared.launch_and_wait(stream)
    rows = lambda v: np.concatenate([v, np.zeros(ldc - n, np.float32)]).reshape(m, ldc)
    got, old = rows(Cb.read()[offset:]), rows(c)
    want = np.float32(0.5) * exact_product(a, b, m, n, k, lda, ldb) + np.float32(-0.25) * old[:, :n]
    assert (bits(got[:, :n].ravel()) == bits(want.ravel())).all()
    assert (bits(got[:, n:].ravel()) == bits(old[:, n:].ravel())).all()


# few rows: copies of A of 32, 64 and 128 rows, most of them past the last one
@pytest.mark.parametrize("m", [1, 8, 31, 32, 33, 64, 65])
@pytest.mark.parametrize("n,k,pad", [(130, 40, 3), (1000, 1100, 4), (9473, 200, 0)])
def test_gemm_few_rows_exact(gpu, m, n, k, pad):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    lda, ldb, ldc = (k + 7) // 8 * 8, (n + 7) // 8 * 8, n + pad
    a = synth.gemm_inputs_v1((m - 1) * lda + k, 1, 1, 5)[0]
    b = synth.gemm_inputs_v1(1, (k - 1) * ldb + n, 1, 6)[1]
    c = synth.uniform_f32(0, 9, (m - 1) * ldc + n)
    A, B, Cb = Guarded(fe, stream, a), Guarded(fe, stream, b), Guarded(fe, stream, c)
    run(fe, ctx, stream, "tiled_gemm_general_v1", schedule=fe.SCHEDULE_TCGEN05, a=A.slice, b=B.slice, c=Cb.slice, m=m, n=n, k=k, lda=lda, ldb=ldb,
        ldc=ldc, alpha=0.5, beta=-0.25)
    rows = lambda v: np.concatenate([v, np.zeros(pad, np.float32)]).reshape(m, ldc)
    got, old = rows(Cb.read()), rows(c)
    want = np.float32(0.5) * exact_product(a, b, m, n, k, lda, ldb) + np.float32(-0.25) * old[:, :n]
    assert (bits(got[:, :n].ravel()) == bits(want.ravel())).all()
    assert (bits(got[:, n:].ravel()) == bits(old[:, n:].ravel())).all()


@pytest.mark.parametrize("offset", [0, 1])   # C by the copy engine, and by elements
@pytest.mark.parametrize("shape,m,n,k", [("pair", 1296, 2832, 1504), ("pair", 1296, 2960, 1504), (256, 1296, 2704, 304), (192, 1296, 2320, 304),
                                         (128, 1296, 1424, 304), (64, 304, 3008, 704), (64, 16, 3008, 704),
                                         (64, 48, 3008, 704)])
def test_tiled_gemm_v1_every_tile_shape_exact(gpu, shape, m, n, k, offset):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    a, b = synth.gemm_inputs_v1(m * k, 1, 1, 5)[0], synth.gemm_inputs_v1(1, k * n, 1, 6)[1]
    A, B, Cb = Guarded(fe, stream, a), Guarded(fe, stream, b), Guarded(fe, stream, np.zeros(m * n + offset, np.float32))
    prepared = fe.prepare(ctx, "tiled_gemm_v1", a=A.slice, b=B.slice, c=Cb.buf.view(GUARD + offset, m * n), m=m, n=n, k=k)
    assert shape_is(prepared.geometry, shape, m, n)
    prepared.launch_and_wait(stream)
    got = Cb.read()
    assert (got[:offset] == 0).all() and (got[offset:].reshape(m, n) == exact_product(a, b, m, n, k, k, n)).all()


@pytest.mark.parametrize("T,d,f,E,cap", [(1000, 1088, 1152, 4, 2000), (1040, 1152, 1088, 4, 500),
                                         # few rows a group: copies of 32 and 64 rows, groups without rows
                                         (1, 128, 256, 8, 2), (40, 128, 256, 4, 3), (90, 192, 320, 4, 180),
                                         (64, 128, 128, 32, 128)])
def test_moe_tile_shapes(gpu, orc, T, d, f, E, cap):
    from test_gpu_parity import assert_close, moe_pipeline
    compact, want_compact, out, want_out, accepted = moe_pipeline(gpu, orc, T, d, f, E, cap)
    assert_close(out, want_out, 2e-2, 2e-3, "combined output")
    assert_close(compact[: accepted * d], want_compact[: accepted * d], 2e-2, 2e-3, "compact expert output")


@pytest.mark.parametrize("d,f,rows", [(64, 64, 128), (64, 64, 77), (128, 200, 300), (64, 384, 33)])
def test_expert_ffn_gelu_values(gpu, d, f, rows):
    """Hidden activations of chosen arguments (W1 copies column c of the row to columns c, c + d, ...): half a bf16 step, and
    1e-6 for the tail's polynomial (8.3e-8), its evaluation and the exponential (a few f32 roundings of at most 1.2)."""
    import math
    fe, ctx, stream = gpu
    B = lambda a: fe.DeviceBuffer.from_host(stream, a)
    rng = np.random.default_rng(7)
    x = np.concatenate([rng.normal(0, 2, rows * d - 12), [0.0, -0.0, 10, -10, 10.5, -10.5, 64, -64, 3e38, -3e38, 1e-39, -5.5]]).astype(np.float32)
    xb = (x.view(np.uint32) >> 16).astype(np.uint16)
    x = (xb.astype(np.uint32) << 16).view(np.float32).astype(np.float64).reshape(rows, d)
    w1 = np.zeros((d, f), np.uint16)
    w1[np.arange(f) % d, np.arange(f)] = 0x3f80
    HID = Guarded(fe, stream, np.zeros(rows * f, np.uint16))
    run(fe, ctx, stream, "moe_expert_ffn_v1", x=B(xb), w1=B(w1.ravel()), w2=B(np.zeros(f * d, np.uint16)),
        permutation=B(np.arange(0, 2 * rows, 2, dtype=np.uint32)), expert_offsets=B(np.array([0, rows], np.uint32)),
        compact_x=B(np.zeros(rows * d, np.uint16)), hidden=HID.slice, compact_output=B(np.zeros(rows * d, np.float32)),
        tokens=rows, d_model=d, d_ff=f, experts=1)
    got = (HID.read().astype(np.uint32) << 16).view(np.float32).astype(np.float64).reshape(rows, f)
    arg = x[:, np.arange(f) % d]
    want = 0.5 * arg * np.vectorize(math.erfc)(-arg / math.sqrt(2))
    assert (np.abs(got - want) <= np.abs(want) * 2.0 ** -8 + 1e-6).all()


def test_expert_ffn_without_tokens(gpu):
    """No token to gather, and a table that claims rows all the same: rows of zeros, and no launch for an empty output."""
    fe, ctx, stream = gpu
    d, f, rows = 128, 64, 200
    B = lambda a: fe.DeviceBuffer.from_host(stream, a)
    X, W1, W2 = B(np.ones(64, np.uint16)), B(np.ones(d * f, np.uint16)), B(np.ones(f * d, np.uint16))
    PERM, OFF = B(np.arange(rows, dtype=np.uint32)), B(np.array([0, rows], np.uint32))
    CX, HID = B(np.ones(rows * d, np.uint16)), B(np.ones(rows * f, np.uint16))
    CO = Guarded(fe, stream, np.ones(rows * d, np.float32))
    common = dict(w1=W1, w2=W2, permutation=PERM, expert_offsets=OFF, hidden=HID, tokens=0, d_model=d, d_ff=f, experts=1)
    run(fe, ctx, stream, "moe_expert_ffn_v1", x=X.view(0, 0), compact_x=CX, compact_output=CO.slice, **common)
    assert (CO.read() == 0).all()
    run(fe, ctx, stream, "moe_expert_ffn_combine_v1", x=X.view(0, 0), route_weights=CO.buf.view(GUARD, 0),
        combined_output=CO.buf.view(GUARD, 0), **common)
    assert (CO.read() == 0).all()


# ---- gate, first launch of a process: sizes at which its blocks ask for shared memory that only together with the
# kernel's own passes the limit without opt-in, so that an earlier launch of another size would hide a missing one
@pytest.mark.parametrize("T,E", [(2048, 8), (1000, 16), (4000, 4)])
def test_moe_gate_first_launch_of_a_process(T, E):
    import os
    import subprocess
    import sys
    code = """
import sys
sys.path.insert(0, %r)
import numpy as np, fe2o3_b200 as fe, oracle
from fe2o3_b200 import synth
T, E, d = %d, %d, 128
ctx = fe.GpuContext(0); s = ctx.default_stream()
x, wg = synth.normal_bf16(1, 1, T * d, 1.0), synth.normal_bf16(1, 2, d * E, 0.1)
X, W, L = fe.DeviceBuffer.from_host(s, x), fe.DeviceBuffer.from_host(s, wg), fe.DeviceBuffer.zeroed(s, T * E, np.float32)
fe.prepare(ctx, "moe_gate_v1", x=X, wg=W, logits=L, tokens=T, d_model=d, experts=E).launch_and_wait(s)
assert (L.to_host_vec(s).view(np.uint32) == oracle.moe_gate_logits(x, wg, T, d, E).view(np.uint32)).all()
print("ok")
""" % (os.path.dirname(os.path.dirname(os.path.abspath(__file__))), T, E)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr


# ---- gate fed by warps of products: half chunks, one block to one per SM (148) and the first count beyond
@pytest.mark.parametrize("d", [64, 128, 192, 448, 2048])
@pytest.mark.parametrize("T,E", [(1, 4), (9, 4), (1, 8), (5, 8), (592, 8), (593, 8), (3, 16), (296, 16), (297, 16)])
def test_moe_gate_small_batches_bit_exact(gpu, orc, T, E, d):
    from fe2o3_b200 import synth
    fe, ctx, stream = gpu
    if d * E * 4 > 96 * 1024:
        d = 1472
    x, wg = synth.normal_bf16(4, d, T * d, 1.0), synth.normal_bf16(4, d + 1, d * E, 0.1)
    X, W, L = Guarded(fe, stream, x), Guarded(fe, stream, wg), Guarded(fe, stream, np.full(T * E, np.nan, np.float32))
    run(fe, ctx, stream, "moe_gate_v1", x=X.slice, wg=W.slice, logits=L.slice, tokens=T, d_model=d, experts=E)
    assert (bits(L.read()) == bits(orc.moe_gate_logits(x, wg, T, d, E))).all()


# ---- routing in one launch: one warp to eight blocks of two passes, and the sizes around each step
@pytest.mark.parametrize("T,E,cap,bad", [(1, 2, 1, 0), (33, 8, 100, 0), (1000, 5, 300, 0), (1024, 16, 2048, 0), (1025, 8, 200, 0),
                                         (2049, 32, 4098, 0), (4097, 8, 900, 0), (8192, 8, 2100, 0), (8193, 16, 16386, 0),
                                         (16384, 8, 4000, 0), (16385, 8, 4000, 0), (5000, 8, 10000, 1)])
def test_moe_routing_one_launch_bit_exact(gpu, orc, T, E, cap, bad):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    logits = (np.round(synth.normal_f32(5, T + E, T * E, 1.0) * 8) / 8).astype(np.float32)   # ties between experts
    if bad:
        logits[T * E - 1] = np.inf
    L = Guarded(fe, stream, logits)
    R = 2 * T
    outs = {k: Guarded(fe, stream, np.full(n, 0x12345678, np.uint32)) for k, n in
            [("top2_experts", R), ("requested_counts", E), ("admitted_counts", E), ("expert_offsets", E + 1),
             ("route_slots", R), ("permutation", R), ("inverse", R)]}
    p = fe.prepare(ctx, "moe_top2_v1", logits=L.slice, tokens=T, experts=E, capacity=cap, **{k: g.slice for k, g in outs.items()})
    if bad:   # refused, with every block's outputs as they were
        with pytest.raises(fe.Fe2o3Error):
            p.launch_and_wait(stream)
        assert p.kernel_status == 2 and all((g.read() == 0x12345678).all() for g in outs.values())
        return
    p.launch_and_wait(stream)
    _, want = orc.moe_top2_route(logits, T, E, cap)
    for k, g in outs.items():
        assert (g.read() == want[k]).all(), k


def test_moe_layer_of_few_tokens_many_passes(gpu):
    """Groups of a few rows: gather warps without rows must stay in step with the ring.  No wait may run out and every
    pass gives the same bits."""
    fe, ctx, stream = gpu
    import torch
    from fe2o3_b200.moe import MoeTop2Layer
    layers = [MoeTop2Layer(ctx, stream, T, 1024, 2048, 8) for T in (16, 33)]
    for layer in layers:
        for t in (layer.x, layer.wg, layer.w1, layer.w2):
            t.normal_(0, 0.1)
    want = [layer.forward().clone() for layer in layers]
    for _ in range(1500):
        for layer in layers:
            layer.forward()
    torch.cuda.synchronize()
    assert ctx.take_kernel_status(stream) == 0
    for layer, w in zip(layers, want):
        assert (layer.out.view(torch.int32) == w.view(torch.int32)).all()


# ---- prefix sum: one tile a block up to four tiles an SM (592 on 148), the ring beyond; last tiles of every kind, aligned and not
@pytest.mark.parametrize("n,offset", [(8191, 0), (8193, 1), (592 * 8192, 0), (592 * 8192 + 1, 0), (593 * 8192 + 8190, 0), (594 * 8192, 0),
                                      (593 * 8192 + 4, 1)])
def test_device_scan_tile_edges(gpu, orc, n, offset):
    fe, ctx, stream = gpu
    rng = np.random.default_rng(n)
    v = rng.integers(0, 2**32, n + offset, dtype=np.uint64).astype(np.uint32)
    V = fe.DeviceBuffer.from_host(stream, v)
    O = Guarded(fe, stream, np.full(n + offset, 0xdeadbeef, np.uint32))
    for exclusive in (0, 1):
        run(fe, ctx, stream, "device_scan_u32", values=V.view(offset, n), output=O.buf.view(GUARD + offset, n), exclusive=exclusive)
        assert (O.read()[offset:] == orc.scan_sum_u32(v[offset:], bool(exclusive))).all()
    f = (v % 7).astype(np.float32) / 8   # sums of at most 2^26 eighths: within the bound the header states
    F = fe.DeviceBuffer.from_host(stream, f)
    G = Guarded(fe, stream, np.full(n + offset, np.nan, np.float32))
    want, mag = orc.scan_sum_f32(f[offset:], False)
    for _ in range(2):
        run(fe, ctx, stream, "device_scan_f32", values=F.view(offset, n), output=G.buf.view(GUARD + offset, n), exclusive=0)
        assert (np.abs(G.read()[offset:].astype(np.float64) - want) <= (128 + n / 8192 / 192) * 2.0 ** -24 * mag + 1e-30).all()


def test_first_scan_of_a_context_on_its_own_stream(gpu, orc):
    """The counters a scan starts from are zero before a context is handed out: nothing orders a non-blocking stream
    behind clears that are still under way."""
    fe, _, stream = gpu
    v = np.arange(1, 700 * 8192 + 1, dtype=np.uint32)
    V = fe.DeviceBuffer.from_host(stream, v)
    want = orc.scan_sum_u32(v, False)
    for _ in range(10):
        O = fe.DeviceBuffer.from_host(stream, np.zeros(v.size, np.uint32))
        ctx = fe.GpuContext(0)
        own = ctx.create_stream()
        p = fe.prepare(ctx, "device_scan_u32", values=V, output=O, exclusive=0)
        p.launch_and_wait(own)
        assert (O.to_host_vec(stream) == want).all()


@pytest.mark.parametrize("n,tickets", [(3 * 8192, 5), (3 * 8192, 1 << 31), (700 * 8192, 1 << 31)])
def test_scan_reports_and_recovers_from_disordered_counters(gpu, orc, n, tickets):
    """Counters that are not those between two launches (here: tickets that nobody should have drawn) are reported by the
    next scan, which writes nothing, and put right when that status is taken."""
    import ctypes as C
    fe, _, stream = gpu
    ctx = fe.GpuContext(0)   # its own counters
    own = ctx.create_stream()
    state = C.c_uint64.from_address(ctx._h.value + 64).value   # fe2o3_ctx::scan_scratch; the low half of its first word counts tickets
    v = np.arange(1, n + 1, dtype=np.uint32)
    V, one = fe.DeviceBuffer.from_host(stream, v), fe.DeviceBuffer.from_host(stream, np.ones(1, np.uint32))
    O = fe.DeviceBuffer.from_host(stream, np.full(n, 0xdeadbeef, np.uint32))
    p = fe.prepare(ctx, "device_scan_u32", values=V, output=O, exclusive=0)
    planted = fe.DeviceBuffer.from_host(stream, np.array([tickets], np.uint32))
    fe.prepare(ctx, "masked_reduce_u32", values=planted, active=one, output=(state, 1)).launch_and_wait(own)
    with pytest.raises(fe.Fe2o3Error):
        p.launch_and_wait(own)
    assert p.kernel_status == 6 and (O.to_host_vec(stream) == 0xdeadbeef).all()
    for _ in range(2):
        p.launch_and_wait(own)
        assert (O.to_host_vec(stream) == orc.scan_sum_u32(v, False)).all()


def test_scan_beside_other_kernels(gpu, orc):
    """More register tiles than are resident at once, while another stream's kernels hold the SMs: a block only waits for
    tiles that have started."""
    fe, ctx, stream = gpu
    side = ctx.create_stream()
    n = 592 * 8192 - 5
    v = np.arange(7, n + 7, dtype=np.uint32)
    V, O = fe.DeviceBuffer.from_host(stream, v), fe.DeviceBuffer.from_host(stream, np.zeros(n, np.uint32))
    m = 2048
    A, B = (fe.DeviceBuffer.from_host(stream, np.zeros(m * m, np.uint16)) for _ in range(2))
    C = fe.DeviceBuffer.zeroed(stream, m * m, np.float32)
    gemm = fe.prepare(ctx, "tiled_gemm_v1", a=A, b=B, c=C, m=m, n=m, k=m)
    scan = fe.prepare(ctx, "device_scan_u32", values=V, output=O, exclusive=0)
    for _ in range(20):
        for _ in range(3):
            gemm.launch(side)
        scan.launch(stream)
    stream.synchronize()
    side.synchronize()
    assert ctx.take_kernel_status(stream) == 0
    assert (O.to_host_vec(stream) == orc.scan_sum_u32(v, False)).all()


# ---- row softmax: lanes per row 8 to 128, one to nine vectors per lane, rows at every phase of a 16-byte vector
@pytest.mark.parametrize("cols", [3, 29, 32, 33, 61, 64, 65, 125, 129, 256, 513, 1021, 1024, 1025, 2045, 2048, 2050, 3001, 4093, 4094, 4095, 4096])
def test_row_softmax_widths(gpu, orc, cols):
    from fe2o3_b200 import synth
    rows = 37
    x = synth.normal_f32(2, cols, rows * cols, 2.0).reshape(rows, cols)
    softmax_case(gpu, orc, x)
    mask = (synth.u32_below(2, 5000 + cols, rows * cols, 4) != 0).reshape(rows, cols)
    mask[:, cols // 2] = True
    got = softmax_case(gpu, orc, x, mask)
    assert (bits(got[~mask]) == 0).all()


# every number of vectors a thread, at its fewest and most columns, aligned and not; a bad row's neighbours share its vectors
@pytest.mark.parametrize("cols", [c for lanes, nvs in ((32, range(2, 9)), (64, range(5, 9)), (128, range(5, 9))) for nv in nvs
                                  for c in (4 * lanes * (nv - 1) + 4, 4 * lanes * nv - 3, 4 * lanes * nv)])
def test_row_softmax_vectors_a_thread(gpu, orc, cols):
    from fe2o3_b200 import synth
    fe, ctx, stream = gpu
    rows = 9
    x = synth.normal_f32(2, 70 + cols, rows * cols, 2.0).reshape(rows, cols)
    x[4, 0] = x[4, cols - 1] = np.inf
    good = [r for r in range(rows) if r != 4]
    for mask in (None, (synth.u32_below(2, 6000 + cols, rows * cols, 4) != 0).reshape(rows, cols)):
        i, o = Guarded(fe, stream, x), Guarded(fe, stream, np.full(x.size, -1, np.float32))
        m = Guarded(fe, stream, mask.astype(np.uint8)) if mask is not None else None
        p = fe.prepare(ctx, "row_softmax_v1", input=i.slice, output=o.slice, mask=m.slice if m else None, rows=rows, cols=cols)
        with pytest.raises(fe.Fe2o3Error):
            p.launch_and_wait(stream)
        got = o.read().reshape(rows, cols)
        _, want = orc.row_softmax(x[good], None if mask is None else mask[good])
        assert (np.abs(got[good] - want) <= 1e-5 * np.abs(want)).all()
        assert (got[4] == -1).all()


@pytest.mark.parametrize("cols", [20, 64, 1000, 1023, 4095])
@pytest.mark.parametrize("in_at,out_at", [(1, 1), (2, 3)])   # the same phase in a vector, and different ones
def test_row_softmax_views_and_bad_rows(gpu, orc, cols, in_at, out_at):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    rows = 11
    x = synth.normal_f32(2, 9000 + cols, rows * cols, 2.0).reshape(rows, cols)
    mask = np.ones((rows, cols), np.uint8)
    x[3, cols - 1] = np.inf      # refused although it is masked: the physical input counts
    mask[3, cols - 1] = 0
    mask[7] = 0                  # no active element
    n = rows * cols
    i = Guarded(fe, stream, np.concatenate([np.zeros(in_at, np.float32), x.ravel()]))
    o = Guarded(fe, stream, np.full(out_at + n, -1, np.float32))
    m = Guarded(fe, stream, np.concatenate([np.zeros(in_at, np.uint8), mask.ravel()]))
    p = fe.prepare(ctx, "row_softmax_v1", input=i.buf.view(GUARD + in_at, n), output=o.buf.view(GUARD + out_at, n),
                   mask=m.buf.view(GUARD + in_at, n), rows=rows, cols=cols)
    with pytest.raises(fe.Fe2o3Error):
        p.launch_and_wait(stream)
    assert p.kernel_status == 2
    got = o.read()[out_at:].reshape(rows, cols)
    good = [r for r in range(rows) if r not in (3, 7)]
    _, want = orc.row_softmax(x[good], mask[good] != 0)
    assert (np.abs(got[good] - want) <= 1e-5 * np.abs(want)).all()
    assert (got[[3, 7]] == -1).all()
    i.unchanged(); m.unchanged()


# ---- attention with f32-precision probabilities (head sizes other than 64): 128-row tiles, 64-key blocks
@pytest.mark.parametrize("B,H,S,D,causal", [(1, 1, 1, 128, False), (1, 3, 63, 128, True), (2, 1, 65, 96, True), (1, 2, 129, 72, False),
                                            (1, 1, 257, 32, True), (1, 5, 300, 128, True), (1, 1, 600, 8, False), (2, 13, 500, 56, True),
                                            # more units than SMs: several rounds, dealt in both directions
                                            (4, 50, 200, 128, False), (4, 45, 400, 40, True)])
def test_attention_split_probabilities(gpu, orc, B, H, S, D, causal):
    from fe2o3_b200 import synth
    from test_gpu_parity import attn_run
    fe = gpu[0]
    n = B * H * S * D
    q, k, v = (synth.normal_bf16(3, d, n, 1.0).reshape(B, H, S, D) for d in (1, 2, 3))
    got, _ = attn_run(gpu, q, k, v, 1.0 / np.sqrt(D), causal, fe.DTYPE_BF16)
    v32 = synth.bf16_to_f32(v)
    _, want = orc.flash_attention(synth.bf16_to_f32(q), synth.bf16_to_f32(k), v32, 1.0 / np.sqrt(D), causal)
    # probabilities are exact sums of three bf16 terms.  What rounds: the score (8 accumulations of at most
    # 128 products, below 1e-5 absolute after scaling), its exponential (1e-6 relative) and 3 * S / 16 <= 113
    # accumulations of p * v at 2^-23 each: together below 2.5e-5 of the largest |v|
    assert np.isfinite(got).all()
    assert np.abs(got - want).max() <= 2.5e-5 * np.abs(v32).max()


def attention_f64(q, k, v, scale, causal):
    scores = q.astype(np.float64) @ k.astype(np.float64).transpose(0, 2, 1) * np.float64(np.float32(scale))
    if causal:
        scores[:, np.triu(np.ones(scores.shape[1:], bool), 1)] = -np.inf
    top = scores.max(-1, keepdims=True)
    w = np.exp(scores - top)
    return w @ v.astype(np.float64) / w.sum(-1, keepdims=True), np.abs(scores[np.isfinite(scores)]).max()


# ---- attention at head size 64: units of two tiles, or of two streams, by the number of units, the length and the limit
@pytest.mark.parametrize("B,H,S,causal", [(1, 1, 1, False), (1, 2, 128, True), (1, 3, 129, False), (1, 2, 257, True), (1, 1, 640, False),
                                          (1, 147, 200, False), (1, 148, 200, False), (4, 40, 300, False), (4, 40, 300, True),
                                          (1, 100, 600, False), (2, 90, 520, True), (1, 320, 100, True), (1, 330, 64, False)])
def test_attention_bf16_tiles_and_streams(gpu, B, H, S, causal):
    from fe2o3_b200 import synth
    from test_gpu_parity import attn_run
    fe = gpu[0]
    D = 64
    q, k, v = (synth.normal_bf16(5, d, B * H * S * D, 1.0).reshape(B, H, S, D) for d in (1, 2, 3))
    got, _ = attn_run(gpu, q, k, v, 1.0 / np.sqrt(D), causal, fe.DTYPE_BF16)
    q32, k32, v32 = (synth.bf16_to_f32(x).reshape(B * H, S, D) for x in (q, k, v))
    want, _ = attention_f64(q32, k32, v32, 1.0 / np.sqrt(D), causal)
    size, _ = attention_f64(q32, k32, np.abs(v32), 1.0 / np.sqrt(D), causal)
    # a probability is cut to eight bits, by less than 2^-7 of itself, and the centring gives back 2^-9
    assert (np.abs(got.reshape(want.shape) - want) <= 2.0 ** -7 * size).all()


# ... and in the 2-norm, where a lost centring would show: the cut leaves 2^-9 - 2^-7 U / m of a probability, U uniform in [0, 1)
# and m log-uniform in [1, 2): 1.95e-3 root mean square, 3.3e-3 without the centring.  Independent from key to key, these add up
# in squares.
@pytest.mark.parametrize("B,H,S,causal", [(1, 1, 1, False), (1, 2, 128, True), (1, 3, 129, False), (1, 2, 257, True), (1, 1, 640, False),
                                          (1, 148, 200, False), (4, 40, 300, False), (4, 40, 300, True), (1, 100, 600, False),
                                          (2, 90, 520, True), (1, 320, 100, True), (1, 330, 64, False),
                                          # two-tile units of which the last few are split into single tiles
                                          (1, 150, 200, False), (3, 50, 512, False),
                                          # one whole key block
                                          (1, 2, 128, False), (1, 100, 128, False)])
def test_attention_bf16_error_norm(gpu, B, H, S, causal):
    from fe2o3_b200 import synth
    from test_gpu_parity import attn_run
    D = 64
    q, k, v = (synth.normal_bf16(5, d, B * H * S * D, 1.0).reshape(B, H, S, D) for d in (1, 2, 3))
    got, _ = attn_run(gpu, q, k, v, 1.0 / np.sqrt(D), causal, gpu[0].DTYPE_BF16)
    q64, k64, v64 = (synth.bf16_to_f32(x).reshape(B * H, S, D).astype(np.float64) for x in (q, k, v))
    scores = q64 @ k64.transpose(0, 2, 1) / np.sqrt(D)
    if causal:
        scores[:, np.triu(np.ones((S, S), bool), 1)] = -np.inf
    weights = np.exp(scores - scores.max(-1, keepdims=True))
    weights /= weights.sum(-1, keepdims=True)
    expected = 1.95e-3 * np.sqrt((weights ** 2 @ v64 ** 2).sum())
    assert np.linalg.norm(got.reshape(B * H, S, D) - weights @ v64) <= expected   # (less for a row's largest probability, which is exact)


# The kernel that a call without a causal limit takes is the faster one (figures in attention_tc_plan): shared memory tells which.
@pytest.mark.parametrize("H,S,streams", [(5, 1900, True), (12, 1900, False), (18, 1900, False), (16, 2048, False), (64, 2048, False),
                                         (9, 4096, False), (4, 4096, True), (36, 1024, False), (118, 256, False), (74, 256, True),
                                         (81, 129, False), (150, 200, False), (150, 512, False), (74, 512, False), (40, 300, True),
                                         (162, 300, False), (49, 640, False), (108, 640, True), (57, 2048, False), (458, 100, False),
                                         (2, 128, False), (148, 128, False), (281, 128, False), (330, 128, False), (2, 127, False), (1, 1, False),
                                         (100, 100, True), (148, 100, False)])
def test_attention_bf16_takes_the_faster_kernel(gpu, H, S, streams):
    fe, ctx, stream = gpu
    n = H * S * 64
    q, k, v = (fe.DeviceBuffer.zeroed(stream, n, np.uint16) for _ in range(3))
    o = fe.DeviceBuffer.zeroed(stream, n, np.float32)
    used = [fe.prepare(ctx, "flash_attention_v1", q=q, k=k, v=v, output=o, batch=1, heads=H, seq=S, dim=64, scale=0.125, causal=causal,
                       input_dtype=fe.DTYPE_BF16).geometry.dynamic_shared_bytes for causal in (0, 1)]
    assert (used[0] == used[1]) == streams   # with a limit it is always streams


@pytest.mark.parametrize("S,D,causal", [(333, 128, True), (1025, 72, False), (1900, 128, True), (1900, 48, False), (4096, 128, False)])
def test_attention_split_error_is_not_above_the_cuda_cores(gpu, S, D, causal):
    """The tensor core truncates its running sum at every accumulation; the kernel may not let that build up over a row.
    The same values given as f32 take the CUDA-core kernel, which serves as the measure."""
    from fe2o3_b200 import synth
    from test_gpu_parity import attn_run
    fe = gpu[0]
    q, k, v = (synth.normal_bf16(3, d, 2 * S * D, 1.0).reshape(1, 2, S, D) for d in (1, 2, 3))
    wide = [synth.bf16_to_f32(x) for x in (q, k, v)]
    want, _ = attention_f64(*(x[0] for x in wide), 1.0 / np.sqrt(D), causal)
    err = [np.linalg.norm(attn_run(gpu, *x, 1.0 / np.sqrt(D), causal, dtype)[0][0] - want)
           for x, dtype in (((q, k, v), fe.DTYPE_BF16), (wide, fe.DTYPE_F32))]
    assert err[0] <= err[1]


@pytest.mark.parametrize("S,D,causal", [(1900, 48, False), (1900, 128, True), (2100, 72, False)])
def test_attention_split_rising_scores(gpu, S, D, causal):
    """Scores that grow along the keys: the reference exponent moves in the first block of a group and inside one."""
    from fe2o3_b200 import synth
    from test_gpu_parity import attn_run
    fe = gpu[0]
    q, k, v = (synth.normal_bf16(3, d, 2 * S * D, 1.0).reshape(1, 2, S, D) for d in (1, 2, 3))
    ramp = synth.bf16_to_f32(k) * np.linspace(0.0, 20.0, S, dtype=np.float32)[:, None]
    k = (ramp.view(np.uint32) >> 16).astype(np.uint16)
    q32, k32, v32 = (synth.bf16_to_f32(x)[0] for x in (q, k, v))
    want, top = attention_f64(q32, k32, v32, 1.0 / np.sqrt(D), causal)
    got, _ = attn_run(gpu, q, k, v, 1.0 / np.sqrt(D), causal, fe.DTYPE_BF16)
    # a score is wrong by up to D / 16 + 2 roundings of its size, a weight by as much relatively, and a result by twice that
    assert np.abs(got[0] - want).max() <= 2 * top * (D / 16 + 2) * 2.0 ** -23 * np.abs(v32).max() + 2.5e-5


@pytest.mark.parametrize("S,D,causal", [(200, 128, False), (300, 40, True)])
def test_attention_split_goes_on_after_rows_that_are_settled(gpu, S, D, causal):
    """A head with a non-finite key among several rounds of units: its blocks settle rows and then take further units."""
    from fe2o3_b200 import synth
    fe, ctx, stream = gpu
    B, H = 1, 160
    q, k, v = (synth.normal_bf16(3, d, H * S * D, 1.0).reshape(H, S, D) for d in (1, 2, 3))
    for h in (0, 77, 159):
        k[h, S - 3, 5] = 0xff80   # -Inf
    Q, K, V = (Guarded(fe, stream, x) for x in (q, k, v))
    O = Guarded(fe, stream, np.full(H * S * D, 7.0, np.float32))
    p = fe.prepare(ctx, "flash_attention_v1", q=Q.slice, k=K.slice, v=V.slice, output=O.slice, batch=B, heads=H, seq=S, dim=D,
                   scale=1.0 / np.sqrt(D), causal=int(causal), input_dtype=fe.DTYPE_BF16)
    with pytest.raises(fe.Fe2o3Error):
        p.launch_and_wait(stream)
    got = O.read().reshape(H, S, D)
    want, _ = attention_f64(*(synth.bf16_to_f32(np.where(x == 0xff80, 0, x).astype(np.uint16)) for x in (q, k, v)), 1.0 / np.sqrt(D), causal)
    spared = S - 3 if causal else 0   # rows that do not admit the bad key
    for h in range(H):
        rows = spared if h in (0, 77, 159) else S
        assert np.abs(got[h, :rows] - want[h, :rows]).max(initial=0.0) <= 2.5e-5 * 6, h   # |v| below 6
        assert (got[h, rows:] == 7.0).all(), h


@pytest.mark.parametrize("causal", [False, True])
def test_attention_split_leaves_bad_rows_unwritten(gpu, orc, causal):
    from fe2o3_b200 import synth
    fe, ctx, stream = gpu
    B, H, S, D = 1, 3, 150, 128
    q, k, v = (synth.normal_bf16(3, d, B * H * S * D, 1.0).reshape(B, H, S, D) for d in (1, 2, 3))
    k[0, 1, 70, 17] = 0x7f80   # +inf: scores of both signs of infinity, so some probabilities are 0 and the sums finite
    Q, K, V = Guarded(fe, stream, q), Guarded(fe, stream, k), Guarded(fe, stream, v)
    O = Guarded(fe, stream, np.full(q.size, -7, np.float32))
    p = fe.prepare(ctx, "flash_attention_v1", q=Q.slice, k=K.slice, v=V.slice, output=O.slice, batch=B, heads=H, seq=S, dim=D,
                   scale=1.0 / np.sqrt(D), causal=int(causal), input_dtype=fe.DTYPE_BF16)
    with pytest.raises(fe.Fe2o3Error):
        p.launch_and_wait(stream)
    assert p.kernel_status == 2
    got = O.read().reshape(B, H, S, D)
    bad = np.zeros((B, H, S), bool)
    bad[0, 1, 70 if causal else 0:] = True
    k[0, 1, 70, 17] = 0
    _, want = orc.flash_attention(*(synth.bf16_to_f32(x) for x in (q, k, v)), 1.0 / np.sqrt(D), causal)
    assert (got[bad] == -7).all()
    assert np.abs(got - want)[~bad].max() <= 2.5e-5 * 6


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("S,D,key,bad", [(150, 128, 70, 0x7f80), (700, 72, 383, 0x7fc0), (260, 32, 256, 0xff80), (65, 8, 1, 0x7f80)])
def test_attention_split_bad_value_spares_rows_that_do_not_admit_it(gpu, orc, S, D, key, bad, causal):
    """The tensor core multiplies the values of masked keys too, by probabilities of 0: rows before a non-finite value
    are written all the same, as the CUDA-core kernel writes them."""
    from fe2o3_b200 import synth
    fe, ctx, stream = gpu
    B, H = 1, 3
    q, k, v = (synth.normal_bf16(3, d, B * H * S * D, 1.0).reshape(B, H, S, D) for d in (1, 2, 3))
    _, want = orc.flash_attention(*(synth.bf16_to_f32(x) for x in (q, k, v)), 1.0 / np.sqrt(D), causal)
    v[0, 1, key, D - 1] = bad
    Q, K, V = Guarded(fe, stream, q), Guarded(fe, stream, k), Guarded(fe, stream, v)
    O = Guarded(fe, stream, np.full(q.size, -7, np.float32))
    p = fe.prepare(ctx, "flash_attention_v1", q=Q.slice, k=K.slice, v=V.slice, output=O.slice, batch=B, heads=H, seq=S, dim=D,
                   scale=1.0 / np.sqrt(D), causal=int(causal), input_dtype=fe.DTYPE_BF16)
    with pytest.raises(fe.Fe2o3Error):
        p.launch_and_wait(stream)
    assert p.kernel_status == 2
    got = O.read().reshape(B, H, S, D)
    lost = np.zeros((B, H, S), bool)
    lost[0, 1, key if causal else 0:] = True
    assert (got[lost] == -7).all()
    assert np.abs(got - want)[~lost].max() <= 2.5e-5 * 6   # as above: largest |v| below 6


# ---- launches that start early: inside a graph behind copies and clears, and where two streams join
def test_early_launches_in_a_captured_graph(gpu):
    import torch
    fe, ctx, _ = gpu
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    src = torch.rand(512 * 512, generator=gen, device="cuda")
    x, y, z, c, total = (torch.zeros_like(src) for _ in range(5))
    a, b = (torch.rand(256 * 256, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
    g32 = torch.zeros(256 * 256, device="cuda")
    soft = fe.prepare(ctx, "row_softmax_v1", input=x, output=y, rows=512, cols=512)
    scan = fe.prepare(ctx, "device_scan_f32", values=y, output=z, exclusive=0)
    exact = fe.prepare(ctx, "scalar_gemm_v1", a=y, b=y, c=c, m=512, n=512, k=512)
    gemm = fe.prepare(ctx, "tiled_gemm_v1", a=a, b=b, c=g32, m=256, n=256, k=256)
    last = fe.prepare(ctx, "device_scan_f32", values=total, output=x, exclusive=0)
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    s, o = ctx.wrap_stream(side.cuda_stream), ctx.wrap_stream(other.cuda_stream)

    def work():
        x.copy_(src)
        soft.launch(s)
        other.wait_stream(side)
        with torch.cuda.stream(other):
            exact.launch(o)
            gemm.launch(o)
            c.mul_(2.0)
            gemm.launch(o)
        scan.launch(s)
        total.zero_()
        side.wait_stream(other)
        soft.launch(s)   # behind a clear and a kernel of the other stream
        exact.launch(s)
        torch.add(c, z, out=total)
        last.launch(s)

    with torch.cuda.stream(side):
        work()
        side.synchronize()
        outs = (x, y, z, c, g32, total)
        want = [t.clone() for t in outs]
        side.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        work()
    for _ in range(3):
        for t in outs:
            t.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert ctx.take_kernel_status(s) == 0
        for t, w in zip(outs, want):
            assert (t.view(torch.int32) == w.view(torch.int32)).all()
