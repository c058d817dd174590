"""The gs = 2 quantiser in fp32 (csrc/quant8.cuh) against the float64 kernels it stands in for, byte for byte: half-way
points, residual sums that fp32 rounds onto them, infinities, NaN, subnormals, the largest and smallest magnitudes; the
weight packer at ragged sizes; the cache writers at every head size.  A plane off the alignment that the fast kernels
need takes the float64 kernel, which gives the comparison."""

import numpy as np
import pytest
import torch

from oracle import msaq_oracle as orc

pytestmark = pytest.mark.gpu


def _adversarial(rng, n):
    """n blocks of 32 fp32 values."""
    b = (rng.standard_normal((n, 32)) * np.exp2(rng.integers(-20, 20, (n, 1)))).astype(np.float32)
    # multiples of half the grid step, so that upper codes and shared codes fall on half-way points
    k = n // 4
    grid = np.exp2(np.floor(np.log2(np.abs(b[:k]).max(1, keepdims=True))) - 6)
    b[:k] = (np.round(b[:k] / (grid / 4)) * (grid / 4)).astype(np.float32)
    # ... and the same moved by one place of the last digit, or with a partner far below it
    b[k:2 * k] = np.nextafter(b[:k], np.float32(np.inf) * rng.choice([-1, 1], b[:k].shape).astype(np.float32))
    b[2 * k:3 * k] = b[:k]
    b[2 * k:3 * k, 1::2] = (b[:k, 1::2] * np.exp2(rng.integers(-60, 0, (k, 16)))).astype(np.float32)
    b[0] = 0
    b[1] = np.float32(1e-30)
    b[2] = np.float32(1e-38) * rng.standard_normal(32).astype(np.float32)
    b[3, :] = np.float32(3e38)
    b[4, 3], b[5, 7], b[6, 0] = np.inf, -np.inf, np.nan
    b[7, ::2], b[7, 1] = np.nan, np.inf
    b[8] = np.float32(2.0) ** 127
    b[8, ::3] *= -1.9
    b[9, 1:] = b[8, 1:]
    b[9, 0] = np.inf
    return b


def _pack(W, u, shift):
    """pack_weight through the C ABI with the shared column-major plane `shift` bytes off its alignment."""
    from ms_kernel_b200 import _lib
    L = _lib.lib()
    OUT, K = W.shape
    nb, UB, SB = K // 32, 4 * (8 - u), 2 * u
    n = OUT * nb
    mk = lambda size: torch.full((size + 16,), 0x5A, dtype=torch.uint8, device="cuda")   # noqa: E731
    planes = [mk(n), mk(n * UB), mk(n * SB), mk(n * UB), mk(n * SB)]
    ptr = [p.data_ptr() for p in planes]
    ptr[4] += shift
    rc = L.msaq_pack_weight(W.data_ptr(), int(W.dtype == torch.bfloat16), *ptr, OUT, K, u, 2, torch.cuda.current_stream().cuda_stream)
    _lib.check(rc)
    torch.cuda.synchronize()
    sizes = [n, n * UB, n * SB, n * UB, n * SB]
    out = []
    for i, (p, s) in enumerate(zip(planes, sizes)):
        off = shift if i == 4 else 0
        a = p.cpu().numpy()
        assert (a[:off] == 0x5A).all() and (a[off + s:] == 0x5A).all(), "bytes outside the plane were written"
        out.append(a[off:off + s])
    return out


@pytest.mark.parametrize("u", (2, 3, 4))
@pytest.mark.parametrize("OUT,nb", [(1, 1), (127, 5), (128, 4), (132, 3), (200, 9), (514, 2), (1024, 16)])
def test_weight_packer_bytes(rng, u, OUT, nb):
    W = _adversarial(rng, max(OUT * nb, 16))[: OUT * nb].reshape(OUT, nb * 32)
    for t in (torch.from_numpy(W).cuda(), torch.from_numpy(W).cuda().to(torch.bfloat16)):
        for a, b in zip(_pack(t, u, 0), _pack(t, u, 1)):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("u", (2, 3, 4))
def test_weight_packer_leaves_out_planes(rng, u):
    from ms_kernel_b200 import _lib
    L = _lib.lib()
    W = torch.randn((300, 96), device="cuda").to(torch.bfloat16)
    ref = _pack(W, u, 0)
    for keep in range(5):
        planes = [torch.empty(r.size, dtype=torch.uint8, device="cuda") if i == keep else None for i, r in enumerate(ref)]
        _lib.check(L.msaq_pack_weight(W.data_ptr(), 1, *[None if p is None else p.data_ptr() for p in planes], 300, 96, u, 2,
                                      torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert np.array_equal(planes[keep].cpu().numpy(), ref[keep])


@pytest.mark.parametrize("u", (2, 3, 4))
@pytest.mark.parametrize("D", (32, 64, 128, 256))
@pytest.mark.parametrize("rot", (0, 1))
def test_cache_writer_bytes(rng, u, D, rot):
    """msaq_kv_write_rope, fast kernel against float64 kernel (shared plane one byte off)."""
    from ms_kernel_b200 import _lib
    L = _lib.lib()
    H, Lr, Lcap, key0, NB, UB, SB = 3, 37, 48, 5, D // 32, 4 * (8 - u), 2 * u
    X = torch.from_numpy(_adversarial(rng, H * Lr * NB).reshape(H, Lr, D)).cuda().to(torch.bfloat16)
    if rot:
        X = torch.where(torch.isfinite(X) & (X.abs() < 1e30), X, torch.ones_like(X))
    cos = torch.randn((Lcap, D // 2), device="cuda")
    sin = torch.randn((Lcap, D // 2), device="cuda")
    n = H * NB * Lcap
    for rope in (False, True):
        res = []
        for shift in (0, 1):
            s, up, sh = (torch.full((n * k + 16,), 0x5A, dtype=torch.uint8, device="cuda") for k in (1, UB, SB))
            _lib.check(L.msaq_kv_write_rope(X.data_ptr(), s.data_ptr(), up.data_ptr(), sh.data_ptr() + shift, H, Lr, D, NB, key0, Lcap, u, 2,
                                            rot, cos.data_ptr() if rope else None, sin.data_ptr() if rope else None,
                                            Lcap if rope else 0, torch.cuda.current_stream().cuda_stream))
            torch.cuda.synchronize()
            a = sh.cpu().numpy()
            res.append((s.cpu().numpy(), up.cpu().numpy(), a[shift:shift + n * SB], a[:shift], a[shift + n * SB:]))
        for a, b in zip(res[0][:3], res[1][:3]):
            assert np.array_equal(a, b)
        assert all((t == 0x5A).all() for r in res for t in r[3:])


def test_oracle_bytes_of_adversarial_blocks(rng):
    import cabi
    W = _adversarial(rng, 4096)
    W = np.where(np.isfinite(W), W, np.float32(1.0)).reshape(512, 256)
    for u in (2, 3, 4):
        ref = orc.pack_weight(W, u, 2)
        got = cabi.pack_weight(cabi.dev(W), u, 2)
        for k in ("scale_exp", "upper", "shared", "upper_cm", "shared_cm"):
            assert np.array_equal(got[k].cpu().numpy(), ref[k]), (u, k)


@pytest.mark.parametrize("u,gs", [(u, gs) for u in (2, 3, 4) for gs in (2, 4, 8, 16, 32)])
@pytest.mark.parametrize("OUT,nb", [(5, 3), (512, 2), (1028, 1)])
def test_dequant_is_exact_at_every_exponent(rng, u, gs, OUT, nb):
    """Every exponent byte, random codes: exactly q * 2^e rounded to bf16 (an overflow becomes an infinity)."""
    UB, SB = 4 * (8 - u), ((32 // gs) * u + 7) // 8
    se = rng.integers(-127, 128, (nb, OUT)).astype(np.int8)
    up = rng.integers(0, 256, (nb, OUT, UB)).astype(np.uint8)
    sh = rng.integers(0, 256, (nb, OUT, SB)).astype(np.uint8)
    bits = lambda a: np.unpackbits(a, axis=-1, bitorder="little").astype(np.int64)      # noqa: E731

    def codes(a, width, n):
        v = (bits(a)[..., : n * width].reshape(nb, OUT, n, width) << np.arange(width)).sum(-1)
        return v - ((v >> (width - 1)) << width)

    q = codes(up, 8 - u, 32) * (1 << u) + np.repeat(codes(sh, u, 32 // gs), gs, -1)
    with np.errstate(over="ignore"):
        ref = torch.from_numpy((q * np.exp2(se.astype(np.float64))[..., None]).astype(np.float32)).to(torch.bfloat16)
    got = torch.ops.msaq.ms_dequant_bf16(torch.from_numpy(se).cuda(), torch.from_numpy(up).cuda(), torch.from_numpy(sh).cuda(),
                                         OUT, nb * 32, nb, u, gs).cpu()
    ref = ref.permute(0, 2, 1).reshape(nb * 32, OUT)
    assert torch.equal(got, ref)
