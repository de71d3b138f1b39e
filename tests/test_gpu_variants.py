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
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (32, 64, 32), (33, 65, 33), (31, 63, 31), (65, 1, 64), (1, 130, 97), (100, 68, 64)])
def test_scalar_gemm_tile_edges_bit_exact(gpu, orc, m, n, k):
    fe, ctx, stream = gpu
    from fe2o3_b200 import synth
    a, b = synth.uniform_f32(0, 1, m * k), synth.uniform_f32(0, 2, k * n)
    A, B = Guarded(fe, stream, a), Guarded(fe, stream, b)
    Cb = Guarded(fe, stream, np.full(m * n, np.nan, np.float32))
    run(fe, ctx, stream, "scalar_gemm_v1", a=A.slice, b=B.slice, c=Cb.slice, m=m, n=n, k=k)
    assert (bits(Cb.read()) == bits(orc.gemm_f32(m, n, k, a, b))).all()
    A.unchanged(); B.unchanged()
