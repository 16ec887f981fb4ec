"""GEMM of few rows (csrc/kernels/gemm_rows.cu): every branch of its split against a product in 64 bits."""
import ctypes as C

import pytest
import torch

from brain_b200.ops import _cuda

pytestmark = pytest.mark.gpu

# rows around the padding to 16 and the limits of the split (48, 64, 128, 255); channels around a tile of 128 and over
# more tiles than half the SMs; k-blocks fewer than the slices, ragged (K % 64), long
SIZES = [(1, 1, 64), (1, 1000, 72), (3, 130, 200), (16, 1024, 2048), (17, 4096, 1024), (48, 129, 4096), (49, 12288, 512),
         (64, 2048, 2048), (65, 640, 2048), (128, 3000, 4096), (129, 6144, 4104), (255, 1024, 2056), (40, 40000, 136), (224, 24576, 512), (200, 6144, 4096)]


def _p(t):
    return C.c_void_p(t.data_ptr() if t is not None else None)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("M,N,K", SIZES)
def test_bf16(M, N, K, mode):
    g = torch.Generator("cuda").manual_seed(M + N + K)
    a = torch.randn(M, K + 8, device="cuda", generator=g).bfloat16()          # a pitch wider than K
    b = torch.randn(N, K, device="cuda", generator=g).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)
    ldc = N + 3                                                               # rows that no vector store fits
    out = torch.full((M, ldc), 7.0, device="cuda", dtype=torch.float32 if mode in (1, 2) else torch.bfloat16)
    rc = _cuda.lib().bb_gemm_bf16(_p(a), _p(b), _p(out), _p(bias), M, N, K, K + 8, K, ldc, 0, 0, mode, C.c_float(0.125), 0, 0, _stream())
    assert rc == 0
    _cuda.check_error()
    want = 0.125 * (a[:, :K].double() @ b.double().t()) + bias.double()
    if mode == 2:
        want = want + 7.0
    if mode == 3:
        want = torch.nn.functional.gelu(want, approximate="tanh")
    # fp32 sums of K products of size ~1 (error ~ sqrt(K) 2^-24 of their scale sqrt(K) / 8), one rounding to bf16; the tanh
    # of the device's fast unit is good to 2^-11 of 1
    tol = 1e-5 * K ** 0.5 if mode in (1, 2) else 0.0
    err = (out[:, :N].double() - want).abs()
    bound = tol + (0 if mode in (1, 2) else 2 ** -8) * want.abs() + 1e-5 * K ** 0.5 + (2 ** -10 * want.abs() + 1e-3 if mode == 3 else 0)
    assert bool((err <= bound).all()), float((err - bound).max())
    assert bool((out[:, N:] == 7.0).all())


@pytest.mark.parametrize("M,N,K", [(m, n, -(-k // 16) * 16) for m, n, k in SIZES])
def test_int8(M, N, K):
    g = torch.Generator("cuda").manual_seed(M + N + K)
    a = torch.randint(-127, 128, (M, K), device="cuda", dtype=torch.int8, generator=g)
    b = torch.randint(-127, 128, (N, K), device="cuda", dtype=torch.int8, generator=g)
    sm, sn = torch.rand(M, device="cuda", generator=g) * 1e-2, torch.rand(N, device="cuda", generator=g) * 1e-2
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    assert _cuda.lib().bb_gemm_i8(_p(a), _p(b), _p(out), _p(sm), _p(sn), M, N, K, K, K, N, 0, 0, _stream()) == 0
    _cuda.check_error()
    # whole sums, then two fp32 products and a rounding to bf16
    want = ((a.double() @ b.double().t()) * sm.double()[:, None] * sn.double()).float()
    err = (out.float() - want).abs()
    assert bool((err <= 2 ** -8 * 1.01 * want.abs()).all()), float(err.max())


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("slices,smem_kb", [(1, 74), (4, 110), (8, 220)])
@pytest.mark.parametrize("M,N,K", SIZES)
def test_splits_that_the_choice_by_size_leaves_out(M, N, K, slices, smem_kb, int8):
    """Every size under given slices of K, also where the general call takes another kernel; sums of whole numbers are exact."""
    g = torch.Generator("cuda").manual_seed(M + N + K)
    K = -(-K // 16) * 16
    a, b = (torch.randint(-8, 9, (r, K), device="cuda", dtype=torch.int8, generator=g) for r in (M, N))
    one = torch.ones(max(M, N), device="cuda")
    x, w = (a, b) if int8 else (a.bfloat16(), b.bfloat16())
    out = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16 if int8 else torch.float32)
    rc = _cuda.lib().bb_gemm_rows(_p(x), _p(w), _p(out), _p(None), _p(one if int8 else None), _p(one if int8 else None), M, N, K, K, K, N,
                                  int(int8), 0 if int8 else 1, C.c_float(1.0), slices, smem_kb, 0, _stream())
    assert rc == 0
    _cuda.check_error()
    want = a.double() @ b.double().t()                                        # below 2^24: exact in fp32
    assert torch.equal(out, want.to(out.dtype))


def test_same_sum_every_run():
    a = torch.randn(33, 4096, device="cuda").bfloat16()
    b = torch.randn(1024, 4096, device="cuda").bfloat16()
    outs = [torch.empty(33, 1024, device="cuda") for _ in range(3)]
    for o in outs:
        assert _cuda.lib().bb_gemm_bf16(_p(a), _p(b), _p(o), _p(None), 33, 1024, 4096, 4096, 4096, 1024, 0, 0, 1, C.c_float(1.0), 0, 0, _stream()) == 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("M,ff,K", [(1, 64, 64), (5, 3072, 1024), (48, 72, 2048), (64, 6144, 2048), (130, 200, 4096), (224, 12288, 512)])
def test_glu_is_the_product_and_its_activation(M, ff, K, int8):
    """Bit for bit the two kernels that it stands for."""
    g = torch.Generator("cuda").manual_seed(M + ff + K)
    bias = None
    if int8:
        a = torch.randint(-127, 128, (M, K), device="cuda", dtype=torch.int8, generator=g)
        b = torch.randint(-127, 128, (2 * ff, K), device="cuda", dtype=torch.int8, generator=g)
        sm, sn = torch.rand(M, device="cuda", generator=g) * 1e-2, torch.rand(2 * ff, device="cuda", generator=g) * 1e-2
    else:
        a, b = (torch.randn(r, K, device="cuda", generator=g).bfloat16() for r in (M, 2 * ff))
        sm = sn = None
        bias = torch.randn(2 * ff, device="cuda", generator=g)
    gu = torch.empty(M, 2 * ff, device="cuda", dtype=torch.bfloat16)
    want, got = (torch.empty(M, ff, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    lib = _cuda.lib()
    rc = lib.bb_gemm_rows_glu(_p(a), _p(b), _p(got), _p(bias), _p(sm), _p(sn), M, ff, K, K, K, ff, int(int8), 0, _stream())
    if rc == -3:
        pytest.skip("left to the general kernel")
    assert rc == 0
    # the general call at this size cuts K into the same slices
    assert lib.bb_gemm_rows(_p(a), _p(b), _p(gu), _p(bias), _p(sm), _p(sn), M, 2 * ff, K, K, K, 2 * ff, int(int8), 0, C.c_float(1.0), 0, 0, 0, _stream()) == 0
    assert lib.bb_swiglu_fwd(_p(gu), _p(want), C.c_long(M), ff, _stream()) == 0
    _cuda.check_error()
    assert torch.equal(got, want)


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("M,ff,K", [(256, 256, 256), (300, 264, 320), (700, 3072, 1024), (1072, 1000, 512), (513, 384, 4096)])
def test_pair_glu_is_the_product_and_its_activation(M, ff, K, int8):
    """Bit for bit the product on CTA pairs and the activation of its bf16 values; columns behind ff stay as they were."""
    g = torch.Generator("cuda").manual_seed(M + ff + K)
    if int8:
        a = torch.randint(-127, 128, (M, K), device="cuda", dtype=torch.int8, generator=g)
        b = torch.randint(-127, 128, (2 * ff, K), device="cuda", dtype=torch.int8, generator=g)
        sm, sn = torch.rand(M, device="cuda", generator=g) * 1e-2, torch.rand(2 * ff, device="cuda", generator=g) * 1e-2
    else:
        a, b = (torch.randn(r, K, device="cuda", generator=g).bfloat16() for r in (M, 2 * ff))
        sm = sn = None
    gu = torch.empty(M, 2 * ff, device="cuda", dtype=torch.bfloat16)
    want = torch.empty(M, ff, device="cuda", dtype=torch.bfloat16)
    got = torch.full((M, ff + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    lib = _cuda.lib()
    assert lib.bb_gemm_pair_glu(_p(a), _p(b), _p(got), _p(sm), _p(sn), M, ff, K, K, K, ff + 8, _stream()) == 0
    if int8:
        assert lib.bb_gemm_i8_pair(_p(a), _p(b), _p(gu), _p(sm), _p(sn), M, 2 * ff, K, K, K, 2 * ff, 0, _stream()) == 0
    else:
        assert lib.bb_gemm_bf16_pair(_p(a), _p(b), _p(gu), M, 2 * ff, K, K, K, 2 * ff, 0, 0, 0, C.c_float(1.0), 1, 0, _stream()) == 0
    assert lib.bb_swiglu_fwd(_p(gu), _p(want), C.c_long(M), ff, _stream()) == 0
    _cuda.check_error()
    assert torch.equal(got[:, :ff], want) and bool((got[:, ff:] == 7.0).all())


def test_products_are_planned_alike_from_the_first_on():
    """The number of CTA pairs that forms are chosen by is the device's, in a process that has launched none and after it."""
    import subprocess
    import sys
    code = """
import ctypes as C, torch
from brain_b200.ops import _cuda
lib = _cuda.lib()
a = torch.zeros(256, 256, device="cuda", dtype=torch.int8)
one = torch.ones(256, device="cuda")
out = torch.empty(256, 256, device="cuda", dtype=torch.bfloat16)
before = lib.bb_gemm_pair_clusters()
p = lambda t: C.c_void_p(t.data_ptr())
assert lib.bb_gemm_i8_pair(p(a), p(a), p(out), p(one), p(one), 256, 256, 256, 256, 256, 256, 0, None) == 0
torch.cuda.synchronize()
assert 0 < before == lib.bb_gemm_pair_clusters(), (before, lib.bb_gemm_pair_clusters())
print("pairs", before)
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
