"""GPU parity of the register-operand GEMV (csrc/gemv_reg.cuh: gs = 2, up to 64 rows) at the sizes where it can go wrong:
one and a few K blocks (four to a ring stage, two teams), ragged tiles of 256 columns, the edges of the eight-row
n-tiles, matrices that one thread block covers and matrices that many share -- against the float64 oracle.  Up to 16 rows
matrices of one wave are the direct kernels': cabi.pipelined() keeps them here."""

import numpy as np
import pytest
import torch

from conftest import F32_REL_FRO_TOL, MAX_ABS_REL_TOL, REL_FRO_TOL
from oracle import msaq_oracle as orc
from test_gpu_give_up import _short_waits, _status

pytestmark = pytest.mark.gpu


def _case(rng, OUT, K, u, M):
    W = orc.to_bf16((rng.standard_normal((OUT, K)) * rng.uniform(0.005, 0.08, (OUT, 1))).astype(np.float32))
    X = orc.to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    return X, orc.pack_weight(W, u, 2)


@pytest.mark.parametrize("u", (2, 3, 4))
@pytest.mark.parametrize("M,OUT,K", [(1, 16, 32), (8, 240, 96), (9, 256, 160), (16, 272, 4096), (17, 528, 288), (31, 16, 8224),
                                     (32, 1040, 1312), (33, 256, 128),
                                     (33, 144, 96), (61, 400, 8224), (64, 1040, 544), (65, 128, 64),
                                     (5, 272, 4096), (8, 528, 288), (7, 1040, 1312), (5, 9616, 32), (8, 9616, 544), (9, 9616, 96),
                                     (16, 9616, 1312)])
def test_edges(rng, u, M, OUT, K):
    import cabi
    X, p = _case(rng, OUT, K, u, M)
    with cabi.pipelined():
        got, gotf = cabi.gemv("batched", cabi.bf16_dev(X), cabi.planes_to_dev(p), M=M)
    cabi.check_output(got, gotf, orc.wonly_matmul(p, X), MAX_ABS_REL_TOL, REL_FRO_TOL, F32_REL_FRO_TOL)


@pytest.mark.parametrize("u,M", [(2, 3), (3, 8), (4, 9), (4, 32)])
def test_misaligned_activations_and_smallest_workspace(rng, u, M):
    """X off a 16-byte boundary, and a workspace of the size the tensor-memory kernel needs, take that kernel: the same
    result to fp32 rounding of the sums."""
    import cabi
    from ms_kernel_b200 import _lib
    L = _lib.lib()
    OUT, K = 4096, 512
    X, p = _case(rng, OUT, K, u, M)
    pd = cabi.planes_to_dev(p)
    ref = orc.wonly_matmul(p, X)
    buf = torch.empty(M * K + 1, dtype=torch.bfloat16, device="cuda")
    buf[1:] = cabi.bf16_dev(X).reshape(-1)
    got, gotf = cabi.gemv("batched", buf[1:], pd, M=M)
    cabi.check_output(got, gotf, ref, MAX_ABS_REL_TOL, REL_FRO_TOL, F32_REL_FRO_TOL)

    full = L.msaq_wonly_gemv_workspace(M, OUT, K // 32, u, 2)
    y = torch.empty((M, OUT), dtype=torch.bfloat16, device="cuda")
    x = cabi.bf16_dev(X)
    ws = torch.empty(full, dtype=torch.uint8, device="cuda")
    served = []
    for size in range(full, 0, -max(256, full // 64)):
        with cabi.pipelined():
            rc = L.msaq_wonly_gemv_batched(x.data_ptr(), pd["scale_exp"].data_ptr(), pd["upper_cm"].data_ptr(),
                                           pd["shared_cm"].data_ptr(), y.data_ptr(), None, M, OUT, K // 32, u, 2, ws.data_ptr(),
                                           size, torch.cuda.current_stream().cuda_stream)
        if rc:
            assert rc == -3
            break
        served.append(y.float().cpu().numpy())
    for s in served:
        assert orc.rel_fro(s, got) < 1e-3           # a few roundings to bf16 at most


@pytest.mark.parametrize("u,M,OUT,K", [(3, 5, 1024, 2048), (4, 8, 10256, 1056), (2, 12, 7120, 1056), (4, 40, 1040, 2048)])
def test_bits_do_not_depend_on_the_workspace_contents(rng, u, M, OUT, K):
    import cabi
    X, p = _case(rng, OUT, K, u, M)
    pd = cabi.planes_to_dev(p)
    x = cabi.bf16_dev(X)
    with cabi.pipelined():
        first = cabi.gemv("batched", x, pd, M=M, fill=0)[1]
        for fill in (0xFF, 0x5A, 0x7F):
            assert np.array_equal(cabi.gemv("batched", x, pd, M=M, fill=fill)[1], first)


@pytest.mark.parametrize("u,M", [(3, 2), (4, 12), (4, 50)])
def test_wait_gives_up_and_next_call_is_correct(rng, u, M):
    import cabi
    OUT, K = 2048, 2048
    X, p = _case(rng, OUT, K, u, M)
    pd = cabi.planes_to_dev(p)
    x = cabi.bf16_dev(X)
    ref = orc.wonly_matmul(p, X)
    _status()
    with _short_waits(0):
        _, gotf = cabi.gemv("batched", x, pd, M=M)
    assert _status() & 1
    assert np.isnan(gotf).any()
    with cabi.pipelined():
        got2, gotf2 = cabi.gemv("batched", x, pd, M=M)
    cabi.check_output(got2, gotf2, ref, MAX_ABS_REL_TOL, REL_FRO_TOL, F32_REL_FRO_TOL)
    assert _status() == 0


@pytest.mark.parametrize("bad", (float("inf"), float("-inf"), float("nan")))
@pytest.mark.parametrize("M,OUT,K", [(5, 9616, 96), (8, 9616, 1056), (6, 9616, 544)])
def test_non_finite_activation_gives_a_nan_row(rng, bad, M, OUT, K):
    """u = 4, five to eight rows, more columns than one wave of the direct kernels: the row is NaN as a whole, as everywhere
    up to eight rows of u = 4; the other rows are untouched."""
    import cabi
    X, p = _case(rng, OUT, K, 4, M)
    X[M - 2, K - 3] = bad
    _, gotf = cabi.gemv("batched", cabi.bf16_dev(X), cabi.planes_to_dev(p), M=M)
    assert np.isnan(gotf[M - 2]).all() and np.isfinite(np.delete(gotf, M - 2, 0)).all()


@pytest.mark.parametrize("u,M", [(4, 3), (4, 5), (4, 8), (4, 9), (3, 1), (3, 12), (2, 6), (2, 30)])
@pytest.mark.parametrize("OUT,K", [(256, 96), (9616, 96)])
def test_largest_finite_weights(rng, u, M, OUT, K):
    """Weights of 2^127 and more (block exponent 121, the largest that finite values give), direct and register kernels."""
    import cabi
    W = rng.standard_normal((OUT, K)) * 0.05
    huge = np.sign(W[::3, :32]) * 2.0 ** 127 * rng.uniform(1.0, 1.99, W[::3, :32].shape)
    W[::3, :32] = huge * (rng.random(huge.shape) < 0.7)
    X = orc.to_bf16(rng.standard_normal((M, K)).astype(np.float32) * np.float32(2.0 ** -60))
    p = orc.pack_weight(orc.to_bf16(W.astype(np.float32)), u, 2)
    assert p["scale_exp"].max() == 121
    got, gotf = cabi.gemv("batched", cabi.bf16_dev(X), cabi.planes_to_dev(p), M=M)
    cabi.check_output(got, gotf, orc.wonly_matmul(p, X), MAX_ABS_REL_TOL, REL_FRO_TOL, F32_REL_FRO_TOL)


@pytest.mark.parametrize("u,M,OUT,K,launches", [(4, 33, 6144, 4096, 2), (4, 33, 4096, 11008, 2), (4, 33, 14336, 3072, 3), (4, 40, 4096, 14336, 3),
                                                (4, 44, 14336, 2048, 2), (4, 48, 4096, 14336, 2), (4, 48, 14336, 3072, 3), (4, 49, 14336, 4096, 3), (4, 56, 14880, 3072, 2),
                                                (4, 64, 14336, 4096, 2), (4, 64, 57344, 512, 2), (3, 37, 47056, 256, 2), (3, 54, 42272, 1088, 3),
                                                (3, 64, 12288, 4096, 2), (3, 64, 14336, 4096, 3), (2, 36, 57344, 512, 2), (2, 36, 28672, 1536, 3),
                                                (2, 17, 57344, 512, 2)])
def test_row_counts_where_the_kernels_take_turns(u, M, OUT, K, launches):
    """On either side of each line between this kernel (itself and the sum of its partials) and the tensor-memory kernel
    (staging, itself, the sum), where their times cross; the two agree to the rounding of the sums."""
    from ms_kernel_b200 import _lib, ops, pack
    g = torch.Generator(device="cuda").manual_seed(M + OUT)
    W = (torch.randn((OUT, K), generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    lin = ops.PackedLinear(pack.pack_weight(W, u, 2), "cuda")
    buf = torch.randn(M * K + 1, generator=g, device="cuda").to(torch.bfloat16)
    x = buf[:M * K].reshape(M, K)
    n0 = _lib.lib().msaq_launch_count()
    y = lin.fwd(x)
    assert _lib.lib().msaq_launch_count() - n0 == launches
    off = torch.empty_like(buf)[1:].reshape(M, K)            # off a 16-byte boundary: always the tensor-memory kernel
    off.copy_(x)
    want = lin.fwd(off)
    assert float((y.float() - want.float()).norm() / want.float().norm()) < 2e-3
