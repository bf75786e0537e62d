"""mm / addmm / bmm on the tcgen05 tensor-core path: every operand layout the kernel takes
without copying (A row- or column-major, B as [K,N] or as a transposed [N,K] view), ragged
tile edges, batches, the fused bias / alpha / beta epilogue -- against an fp64 product of the
same bf16 / f16 inputs. The device status word must stay clean (no bounded wait gave up)."""

import pytest
import torch

from backendbench_b200 import _abi, ops
from backendbench_b200.eval import compare

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(params=[1, 0], ids=["small-path-on", "small-path-off"])
def small_path(request):
    """Small 16-bit products normally take the mma.sync kernel; with the path switched off the
    same shapes exercise the tcgen05 / CUDA-core kernels (ragged tiles, every layout)."""
    prev = _abi.lib().b200_gemm_small_path(request.param)
    try:
        yield request.param
    finally:
        _abi.lib().b200_gemm_small_path(prev)


def _uses_tc(a, b, batch, M, N, K, sa, sb):
    return bool(_abi.lib().b200_gemm_uses_tensor_cores(batch, M, N, K, sa[0], sa[1], sa[2], sb[0], sb[1], sb[2], _abi.BF16 if a.dtype == torch.bfloat16 else _abi.F16, a.data_ptr(), b.data_ptr(), a.data_ptr()))


def _rand(shape, dtype, g, std):
    return (torch.randn(shape, generator=g, device=DEV) * std).to(dtype)


def _check(got, exact, dtype):
    # fp32 accumulation + one rounding to a 16-bit type: relative 2^-8 (bf16) / 2^-11 (f16) of the value, plus accumulation noise
    ok, ea, er = compare(exact.to(dtype), got, 2e-2 if dtype == torch.bfloat16 else 4e-3, 1e-2)
    assert ok, (ea, er)


SHAPES = [(128, 256, 64), (128, 256, 256), (256, 512, 128), (130, 264, 72), (33, 48, 64), (1, 256, 512), (257, 8, 4096), (512, 1000, 136), (384, 768, 2048)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, False), (True, True)])
def test_mm_all_layouts(dtype, a_t, b_t, small_path):
    g = torch.Generator(device=DEV).manual_seed(5)
    for M, N, K in SHAPES:
        Mp, Kp, Np = (M + 7) // 8 * 8, (K + 7) // 8 * 8, (N + 7) // 8 * 8
        a = _rand((Kp, Mp), dtype, g, K**-0.5).t()[:M, :K] if a_t else _rand((Mp, Kp), dtype, g, K**-0.5)[:M, :K]
        b = _rand((Np, Kp), dtype, g, 1.0).t()[:K, :N] if b_t else _rand((Kp, Np), dtype, g, 1.0)[:K, :N]
        assert _uses_tc(a, b, 1, M, N, K, (0, a.stride(0), a.stride(1)), (0, b.stride(0), b.stride(1))), (M, N, K, a.stride(), b.stride())
        got = ops.mm_default(a, b)
        ops.check_device_status()
        assert got.shape == (M, N) and got.dtype == dtype and got.is_contiguous()
        _check(got, a.double() @ b.double(), dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_addmm_epilogue_variants(dtype, small_path):
    g = torch.Generator(device=DEV).manual_seed(6)
    M, N, K = 300, 520, 192
    a, b = _rand((M, K), dtype, g, K**-0.5), _rand((K, N), dtype, g, 1.0)
    exact = a.double() @ b.double()
    for bias_shape in [(N,), (M, N), (1, N), (M, 1), ()]:
        bias = _rand(bias_shape, dtype, g, 1.0)
        _check(ops.addmm_default(bias, a, b), exact + bias.double(), dtype)
        _check(ops.addmm_default(bias, a, b, beta=0.5, alpha=2), 2 * exact + 0.5 * bias.double(), dtype)
    nan_bias = torch.full((N,), float("nan"), dtype=dtype, device=DEV)
    _check(ops.addmm_default(nan_bias, a, b, beta=0), exact, dtype)  # beta = 0 ignores the bias
    ops.check_device_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_bmm_batches_and_strided_views(dtype, small_path):
    g = torch.Generator(device=DEV).manual_seed(7)
    for B, M, K, N in [(3, 128, 64, 256), (5, 200, 72, 136), (32, 256, 128, 320), (2, 64, 1024, 64)]:
        a, b = _rand((B, M, K), dtype, g, K**-0.5), _rand((B, K, N), dtype, g, 1.0)
        _check(ops.bmm_default(a, b), a.double() @ b.double(), dtype)
        bt = _rand((B, N, K), dtype, g, 1.0).transpose(1, 2)  # K-major B, as attention scores use it
        _check(ops.bmm_default(a, bt), a.double() @ bt.double(), dtype)
        at = _rand((B, K, M), dtype, g, K**-0.5).transpose(1, 2)
        _check(ops.bmm_default(at, b), at.double() @ b.double(), dtype)
    ops.check_device_status()


def test_layouts_the_tensor_core_path_declines_still_work():
    """K stride off the 16-byte grid, fp32 operands, unaligned bases: the CUDA-core kernel."""
    g = torch.Generator(device=DEV).manual_seed(8)
    a, b = _rand((64, 100), torch.bfloat16, g, 0.1), _rand((100, 50), torch.bfloat16, g, 1.0)
    assert not _uses_tc(a, b, 1, 64, 50, 100, (0, 100, 1), (0, 50, 1))
    _check(ops.mm_default(a, b), a.double() @ b.double(), torch.bfloat16)
    a32, b32 = torch.randn(96, 200, device=DEV, generator=g), torch.randn(200, 72, device=DEV, generator=g)
    ok, ea, er = compare((a32.double() @ b32.double()).float(), ops.mm_default(a32, b32), 1e-4, 1e-4)
    assert ok, (ea, er)
    av = _rand((65, 129), torch.float16, g, 0.1)[1:, 1:]  # base pointer 2 bytes off alignment
    bv = _rand((128, 64), torch.float16, g, 1.0)
    _check(ops.mm_default(av, bv), av.double() @ bv.double(), torch.float16)
    ops.check_device_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_large_misaligned_operands_are_repitched_onto_tensor_cores(dtype):
    """Row pitches / bases off the 16-byte grid (K = 2049, N = 127, sliced views): large
    products get their operands re-pitched by the library's copy kernel and still match."""
    g = torch.Generator(device=DEV).manual_seed(9)
    a, b = _rand((1024, 2049), dtype, g, 2049**-0.5), _rand((2049, 127), dtype, g, 1.0)
    _check(ops.mm_default(a, b), a.double() @ b.double(), dtype)
    at = _rand((2049, 1030), dtype, g, 2049**-0.5).t()[1:, :]  # M-major A with an odd base offset
    _check(ops.mm_default(at, b), at.double() @ b.double(), dtype)
    bias = _rand((127,), dtype, g, 1.0)
    _check(ops.addmm_default(bias, a, b, beta=2, alpha=0.5), 0.5 * (a.double() @ b.double()) + 2 * bias.double(), dtype)
    x, y = _rand((4, 300, 1001), dtype, g, 1001**-0.5), _rand((4, 260, 1001), dtype, g, 1.0).transpose(1, 2)  # K-major B, K = 1001
    _check(ops.bmm_default(x, y), x.double() @ y.double(), dtype)
    ops.check_device_status()


def _check32(got, a, b, extra=None, alpha=1.0, beta=1.0):
    """fp32 result against the fp64 product. The tensor core truncates each of its K/16
    additions into the accumulator (half a unit in the last place of the running sum on
    average, always toward zero), so the allowed error is K/16 such units of a running sum
    as large as the result or four standard deviations of it."""
    K = a.shape[-1]
    exact = alpha * (a.double() @ b.double())
    spread = abs(alpha) * ((a.double() ** 2) @ (b.double() ** 2)).sqrt()
    if extra is not None:
        exact = exact + beta * extra.double()
    err = (got.double() - exact).abs()
    bound = 2.0**-24 * (K / 16 + 4) * (exact.abs() + 4 * spread) + 1e-30
    assert got.dtype == torch.float32 and bool((err <= bound).all()), float((err / bound).max())


@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, False), (True, True)])
def test_large_fp32_products_take_split_bf16_planes_on_tensor_cores(a_t, b_t):
    """fp32 mm / addmm / bmm above the size threshold: operands split into three bf16 planes,
    six plane products accumulated in fp32 by the tcgen05 kernel. Every operand layout, ragged
    M / N / K (K padded to 64 inside the planes), bias with alpha / beta, batches."""
    g = torch.Generator(device=DEV).manual_seed(12)
    for M, N, K in [(512, 512, 512), (446, 2048, 1024), (130, 1000, 1111), (1000, 36, 4099), (33, 8192, 300)]:
        assert M * N * K >= ops.F32_SPLIT_MIN_MACS
        a = torch.randn((K, M) if a_t else (M, K), generator=g, device=DEV)
        b = torch.randn((N, K) if b_t else (K, N), generator=g, device=DEV)
        a = a.t() if a_t else a
        b = b.t() if b_t else b
        _check32(ops.mm_default(a, b), a, b)
        bias = torch.randn(N, generator=g, device=DEV)
        _check32(ops.addmm_default(bias, a, b, beta=0.5, alpha=-1.5), a, b, bias.expand(M, N), -1.5, 0.5)
    B, M, N, K = 4, 200, 264, 640
    a = torch.randn((B, K, M) if a_t else (B, M, K), generator=g, device=DEV)
    b = torch.randn((B, N, K) if b_t else (B, K, N), generator=g, device=DEV)
    a = a.transpose(1, 2) if a_t else a
    b = b.transpose(1, 2) if b_t else b
    _check32(ops.bmm_default(a, b), a, b)
    ops.check_device_status()


def test_split_fp32_product_keeps_special_values_and_wide_ranges():
    g = torch.Generator(device=DEV).manual_seed(13)
    a = torch.randn(512, 512, generator=g, device=DEV) * torch.logspace(-20, 20, 512, device=DEV)  # columns spanning 40 decades
    b = torch.randn(512, 512, generator=g, device=DEV) * torch.logspace(20, -20, 512, device=DEV).unsqueeze(1)
    _check32(ops.mm_default(a, b), a, b)
    a = torch.randn(512, 512, generator=g, device=DEV)
    b = torch.randn(512, 512, generator=g, device=DEV)
    a[3, 7] = float("inf")
    a[5, 9] = float("nan")
    a[8, 1] = 3.4e38  # rounds to infinity as bf16: must stay finite
    b[1] *= 1e-3      # ... and its products stay below the fp32 maximum
    got, want = ops.mm_default(a, b), a @ b
    assert bool(torch.isnan(got[5]).all()) and bool(torch.isinf(got[3]).all()) and bool((got[3] == want[3]).all())
    assert bool(torch.isfinite(got[8]).all()) and bool(((got[8] - want[8]).abs() <= 1e-5 * want[8].abs()).all())
    b[:, 11] = float("-inf")  # a whole output column: -inf * a, NaN where a is 0 or NaN
    a[40, :] = 0.0
    got, want = ops.mm_default(a, b), a @ b
    assert bool((torch.isnan(got[:, 11]) == torch.isnan(want[:, 11])).all()) and bool((got[:, 11][~torch.isnan(want[:, 11])] == want[:, 11][~torch.isnan(want[:, 11])]).all())
    rest = [i for i in range(512) if i not in (3, 5, 8)]
    cols = [j for j in range(512) if j != 11]
    _check32(got[rest][:, cols], a[rest], b[:, cols])
    ops.check_device_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_odd_output_widths_on_the_tensor_core_path(dtype):
    """N off the 8-element grid: B is re-pitched, C rows start at odd addresses, and the
    epilogue writes them row by row from its staging buffer (every column tail length, a
    ragged last row block, batches, bias and scaling)."""
    g = torch.Generator(device=DEV).manual_seed(15)
    for M, N, K in [(300, 513, 192), (1000, 127, 1024), (129, 65, 2048), (4100, 255, 64), (257, 1, 4096), (640, 71, 512)]:
        a, b = _rand((M, K), dtype, g, K**-0.5), _rand((K, N), dtype, g, 1.0)
        exact = a.double() @ b.double()
        _check(ops.mm_default(a, b), exact, dtype)
        bias = _rand((N,), dtype, g, 1.0)
        _check(ops.addmm_default(bias, a, b, beta=0.5, alpha=2), 2 * exact + 0.5 * bias.double(), dtype)
    a3, b3 = _rand((5, 700, 256), dtype, g, 1 / 16), _rand((5, 256, 127), dtype, g, 1.0)
    _check(ops.bmm_default(a3, b3), a3.double() @ b3.double(), dtype)
    ops.check_device_status()


def test_many_rows_few_columns_take_the_row_per_thread_kernel():
    """fp32 (and 16-bit below the re-pitch threshold) products with at most 16 output columns
    and some hundred thousand rows: both accumulator counts (8, 16), K tails that are not whole
    16-byte vectors, K longer than one chunk of B, batches, bias and scaling, specials; and
    the same shapes just outside the kernel's range (19 and 32 columns, few rows)."""
    g = torch.Generator(device=DEV).manual_seed(16)
    for M, K, N in [(80000, 256, 8), (76000, 300, 13), (100000, 64, 1), (16384, 1024, 19), (9473, 2060, 32), (12000, 600, 13)]:
        a32, b32, bias = torch.randn(M, K, generator=g, device=DEV), torch.randn(K, N, generator=g, device=DEV), torch.randn(1, N, generator=g, device=DEV)
        _check32(ops.mm_default(a32, b32), a32, b32)
        _check32(ops.addmm_default(bias, a32, b32, beta=2, alpha=0.5), a32, b32, extra=bias.expand(M, N), alpha=0.5, beta=2.0)
    wide = torch.randn(90000, 132, generator=g, device=DEV)
    a32, b32 = wide[:, :130], torch.randn(130, 5, generator=g, device=DEV)  # rows 16-byte aligned, K = 130 leaves a tail of 2
    _check32(ops.mm_default(a32, b32), a32, b32)
    a3, b3 = torch.randn(16, 8192, 96, generator=g, device=DEV), torch.randn(16, 96, 5, generator=g, device=DEV)
    a3[3, 100, 7] = float("inf")
    b3[9, 50, 2] = float("nan")
    got, ref = ops.bmm_default(a3, b3), torch.bmm(a3, b3)
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.isinf(got), torch.isinf(ref))
    fin = torch.isfinite(ref)
    assert torch.allclose(got[fin], ref[fin], atol=1e-4, rtol=1e-4)
    for dt in (torch.bfloat16, torch.float16):
        h, w = _rand((90000, 64), dt, g, 1 / 8), _rand((64, 6), dt, g, 1.0)
        _check(ops.mm_default(h, w), h.double() @ w.double(), dt)
    ops.check_device_status()


def test_long_contractions_with_small_outputs_leave_the_single_cta_path():
    """K in the thousands with a handful of outputs: 16-bit operands are re-pitched onto the
    tensor cores whatever their alignment, fp32 operands share K among the CTAs of a cluster
    (every cluster size from 2 to 8, a K that leaves the last CTAs of the cluster empty)."""
    g = torch.Generator(device=DEV).manual_seed(14)
    a, b, bias = _rand((32, 4096), torch.bfloat16, g, 4096**-0.5), _rand((4096, 31), torch.bfloat16, g, 1.0), _rand((32, 1), torch.bfloat16, g, 1.0)
    _check(ops.addmm_default(bias, a, b), a.double() @ b.double() + bias.double(), torch.bfloat16)
    a32, b32 = torch.randn(16, 8192, generator=g, device=DEV), torch.randn(8192, 40, generator=g, device=DEV)
    _check32(ops.mm_default(a32, b32), a32, b32)
    a32, b32 = torch.randn(1, 4096, generator=g, device=DEV), torch.randn(4096, 1024, generator=g, device=DEV)
    _check32(ops.mm_default(a32, b32), a32, b32)
    for M, K, N in [(2, 130, 256), (55, 200, 70), (100, 257, 33), (33, 330, 130), (7, 400, 9), (140, 450, 20), (64, 513, 64), (3, 2048, 17), (165, 4096, 32), (44, 2072, 1024)]:
        a32, b32, bias = torch.randn(M, K, generator=g, device=DEV), torch.randn(K, N, generator=g, device=DEV), torch.randn(M, 1, generator=g, device=DEV)
        _check32(ops.mm_default(a32, b32), a32, b32)
        _check32(ops.mm_default(a32.t().contiguous().t(), b32.t().contiguous().t()), a32, b32)  # both operands in the other memory order
        _check32(ops.addmm_default(bias, a32, b32, beta=2, alpha=0.5), a32, b32, extra=bias.expand(M, N), alpha=0.5, beta=2.0)
    a3, b3 = torch.randn(5, 21, 1024, generator=g, device=DEV), torch.randn(5, 1024, 40, generator=g, device=DEV)
    a3[2, 3, 100] = float("inf")
    b3[4, 7, 5] = float("nan")
    got, ref = ops.bmm_default(a3, b3), torch.bmm(a3, b3)
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.isinf(got), torch.isinf(ref))
    fin = torch.isfinite(ref)
    assert torch.allclose(got[fin], ref[fin], atol=1e-3, rtol=1e-4)
    for dt in (torch.float16, torch.bfloat16):  # 16-bit operands off the 16-byte grid, K below the re-pitch threshold
        h, w = _rand((9, 1000), dt, g, 1000**-0.5), _rand((1000, 7), dt, g, 1.0)
        _check(ops.mm_default(h, w), h.double() @ w.double(), dt)
    ops.check_device_status()


def test_a_wait_that_cannot_complete_ends_in_a_status_not_a_hang():
    """The failure-detection form this kernel has: every mbarrier wait carries a time limit.
    The probe entry withholds one K slab (so the MMA warp's wait for it can never complete)
    with a 1 ms limit; the kernel must come back by itself, report B200_DEV_WAIT_TIMEOUT in
    the status word, and leave the context and the tensor memory usable for the next product."""
    import time

    g = torch.Generator(device=DEV).manual_seed(9)
    a = _rand((512, 1024), torch.bfloat16, g, 1024**-0.5)
    b = _rand((1024, 768), torch.bfloat16, g, 1.0)
    c = torch.empty(512, 768, dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    rc = _abi.lib().b200_gemm_wait_probe(a.data_ptr(), b.data_ptr(), c.data_ptr(), 512, 768, 1024, _abi.BF16, 1000, status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0, rc
    torch.cuda.synchronize()
    took = time.perf_counter() - t0
    assert int(status.item()) & _abi.DEV_WAIT_TIMEOUT
    assert took < 1.0, took  # a handful of 1 ms limits, not the 2 s of an ordinary call
    # limits outside 50 us .. 0.1 s are refused, as are operands that would not reach the kernel
    assert _abi.lib().b200_gemm_wait_probe(a.data_ptr(), b.data_ptr(), c.data_ptr(), 512, 768, 1024, _abi.BF16, 5_000_000, status.data_ptr(), 0) < 0
    assert _abi.lib().b200_gemm_wait_probe(a.data_ptr(), b.data_ptr(), c.data_ptr(), 512, 768, 1024, _abi.F32, 1000, status.data_ptr(), 0) < 0
    # the same context, the same tensor memory: an ordinary product right behind it is correct
    got = ops.mm_default(a, b)
    ops.check_device_status()
    _check(got, a.double() @ b.double(), torch.bfloat16)


PAIR_SHAPES = [(256, 256, 320), (300, 520, 640), (1000, 1000, 1000), (129, 130, 4096), (2048, 384, 512), (513, 257, 328)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, False), (True, True)])
def test_cta_pair_tiles_every_layout_and_ragged_edge(dtype, a_t, b_t):
    """Products of more than 128 rows and columns with more than four K slabs run on CTA pairs
    (256 x 256 tiles, tcgen05 cta_group::2): rows that end in the first or in the second CTA of
    the last pair, columns that end in either half of B, K off the 64 grid, all four operand
    layouts -- against the fp64 product, and bit for bit against the single-CTA kernel's rule
    (fp32 accumulation, one rounding) through the tolerance of `_check`."""
    g = torch.Generator(device=DEV).manual_seed(21)
    for M, N, K in PAIR_SHAPES:
        Mp, Kp, Np = (M + 7) // 8 * 8, (K + 7) // 8 * 8, (N + 7) // 8 * 8
        a = _rand((Kp, Mp), dtype, g, K**-0.5).t()[:M, :K] if a_t else _rand((Mp, Kp), dtype, g, K**-0.5)[:M, :K]
        b = _rand((Np, Kp), dtype, g, 1.0).t()[:K, :N] if b_t else _rand((Kp, Np), dtype, g, 1.0)[:K, :N]
        got = ops.mm_default(a, b)
        ops.check_device_status()
        assert got.shape == (M, N) and got.dtype == dtype
        _check(got, a.double() @ b.double(), dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_cta_pair_epilogue_and_batches(dtype):
    g = torch.Generator(device=DEV).manual_seed(22)
    M, N, K = 300, 520, 704
    a, b = _rand((M, K), dtype, g, K**-0.5), _rand((K, N), dtype, g, 1.0)
    exact = a.double() @ b.double()
    for bias_shape in [(N,), (M, N), (1, N), (M, 1), ()]:
        bias = _rand(bias_shape, dtype, g, 1.0)
        _check(ops.addmm_default(bias, a, b), exact + bias.double(), dtype)  # alpha = beta = 1: the single-add epilogue
        _check(ops.addmm_default(bias, a, b, beta=0.5, alpha=2), 2 * exact + 0.5 * bias.double(), dtype)
    for B, M, K, N in [(3, 256, 384, 256), (5, 200, 520, 136), (2, 640, 1024, 300)]:
        x, y = _rand((B, M, K), dtype, g, K**-0.5), _rand((B, K, N), dtype, g, 1.0)
        _check(ops.bmm_default(x, y), x.double() @ y.double(), dtype)
        yt = _rand((B, N, K), dtype, g, 1.0).transpose(1, 2)
        _check(ops.bmm_default(x, yt), x.double() @ yt.double(), dtype)
    ops.check_device_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_long_contraction_with_few_tiles_is_split_along_k(dtype):
    """A handful of output tiles and K >= 1024: the contraction runs as up to 32 ranges side by
    side and the fp32 partial products are added in a fixed order. Same answer as the unsplit
    product to rounding, bit-identical from run to run, every operand layout, bias and scales
    applied once, and shapes the split declines (K not divisible) fall through."""
    g = torch.Generator(device=DEV).manual_seed(15)
    dt = _abi.BF16 if dtype == torch.bfloat16 else _abi.F16
    for M, N, K, split in [(5, 512, 4096, True), (45, 2048, 4096, True), (12, 512, 2048, True), (44, 32, 4096, True), (130, 264, 1096, False), (1, 7, 4104, True), (300, 200, 8200, True)]:
        a, b = _rand((M, K), dtype, g, K**-0.5), _rand((K, N), dtype, g, 1.0)
        c = torch.empty(M, N, dtype=dtype, device=DEV)
        need = _abi.lib().b200_gemm_splitk_scratch_bytes(a.data_ptr(), b.data_ptr(), c.data_ptr(), 1, M, N, K, 0, K, 1, 0, N, 1, dt)
        if N % 8 == 0:  # B [K, N] with rows off the 16-byte grid never reaches the tensor cores
            assert (need > 0) == split, (M, N, K, need)
        exact = a.double() @ b.double()
        got = ops.mm_default(a, b)
        _check(got, exact, dtype)
        assert torch.equal(got, ops.mm_default(a, b))
        bias = _rand((N,), dtype, g, 1.0)
        _check(ops.addmm_default(bias, a, b, beta=0.5, alpha=2), 2 * exact + 0.5 * bias.double(), dtype)
        at = _rand((K, (M + 7) // 8 * 8), dtype, g, K**-0.5).t()[:M]  # M-major A
        bt = _rand(((N + 7) // 8 * 8, K), dtype, g, 1.0).t()[:, :N]   # K-major B
        _check(ops.mm_default(at, bt), at.double() @ bt.double(), dtype)
    ops.check_device_status()


def test_fp32_products_with_a_narrow_result():
    """C of at most 16 columns under a long row-major fp32 A: a warp per row of A (16-byte
    pieces of the row per lane, B in shared memory, the lanes' partial sums folded by a halving
    exchange). Ragged K, every N up to 16, batches, bias and scales, rows that do not fill the
    last CTA; against an fp64 product."""
    g = torch.Generator(device=DEV).manual_seed(23)
    for B, M, K, N in [(1, 2000, 280, 8), (1, 1500, 128, 16), (1, 5001, 1000, 3), (3, 700, 260, 9), (1, 16384, 256, 8), (2, 1999, 2052, 16), (1, 1300, 132, 1)]:
        a = torch.randn(B, M, K, generator=g, device=DEV) * K**-0.5
        b = torch.randn(B, K, N, generator=g, device=DEV)
        exact = a.double() @ b.double()
        got = ops.bmm_default(a, b)
        assert got.shape == (B, M, N) and got.dtype == torch.float32
        ok, ea, er = compare(exact.float(), got, 1e-4, 1e-4)
        assert ok, (B, M, K, N, ea, er)
        assert torch.equal(got, ops.bmm_default(a, b))  # fixed order of additions
        bias = torch.randn(M, N, generator=g, device=DEV)
        got = ops.addmm_default(bias, a[0], b[0], beta=0.5, alpha=2)
        ok, ea, er = compare((2 * exact[0] + 0.5 * bias.double()).float(), got, 1e-4, 1e-4)
        assert ok, (M, K, N, ea, er)
    ops.check_device_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_small_products_on_the_mma_kernel(dtype):
    """Few 64 x 64 tiles and a short contraction: the four-warp mma.sync kernel when both
    operands are on the 16-byte grid (all four layout pairs, ragged M / N / K, batches, bias and
    scales); offset bases, odd pitches and operands with no unit stride go to the other kernels."""
    g = torch.Generator(device=DEV).manual_seed(29)
    dt = _abi.BF16 if dtype == torch.bfloat16 else _abi.F16

    def prefers(a, b, B, M, N, K):
        sa = (a.stride(0) if B > 1 else 0, a.stride(-2), a.stride(-1))
        sb = (b.stride(0) if B > 1 else 0, b.stride(-2), b.stride(-1))
        return _abi.lib().b200_gemm_prefers_small(a.data_ptr(), b.data_ptr(), B, M, N, K, sa[0], sa[1], sa[2], sb[0], sb[1], sb[2], dt)

    for B, M, N, K in [(1, 41, 64, 256), (64, 2, 64, 64), (1, 367, 264, 40), (1, 227, 72, 256), (1, 36, 24, 32), (32, 15, 8, 256), (2, 4, 72, 64), (1, 1, 8, 200), (3, 136, 72, 104), (1, 64, 64, 8),
                       (1, 5, 8, 248), (8, 6, 16, 40), (1, 17, 9 * 8, 136), (2, 49, 40, 72)]:
        for a_t in (False, True):
            for b_t in (False, True):
                Mp = (M + 7) // 8 * 8
                a = _rand((B, K, Mp), dtype, g, K**-0.5).transpose(1, 2)[:, :M] if a_t else _rand((B, M, K), dtype, g, K**-0.5)
                b = _rand((B, N, K), dtype, g, 1.0).transpose(1, 2) if b_t else _rand((B, K, N), dtype, g, 1.0)
                assert prefers(a, b, B, M, N, K) == 1, (B, M, N, K, a.stride(), b.stride())
                got = ops.bmm_default(a, b)
                assert got.shape == (B, M, N) and got.dtype == dtype and got.is_contiguous()
                _check(got, a.double() @ b.double(), dtype)
        a2, b2 = _rand((M, K), dtype, g, K**-0.5), _rand((K, N), dtype, g, 1.0)
        for bias_shape in [(N,), (M, N), (M, 1), ()]:
            bias = _rand(bias_shape, dtype, g, 1.0)
            _check(ops.addmm_default(bias, a2, b2, beta=0.5, alpha=2), 2 * (a2.double() @ b2.double()) + 0.5 * bias.double(), dtype)
        nan_bias = torch.full((N,), float("nan"), dtype=dtype, device=DEV)
        _check(ops.addmm_default(nan_bias, a2, b2, beta=0), a2.double() @ b2.double(), dtype)
        # off the grid: an offset base, an odd pitch, no unit stride -- other kernels, same answer
        shifted = _rand((M, K + 8), dtype, g, K**-0.5)[:, 3 : K + 3]
        every_other = _rand((M, 2 * K), dtype, g, K**-0.5)[:, ::2]
        for a3 in (shifted, every_other):
            assert prefers(a3, b2, 1, M, N, K) == 0
            _check(ops.mm_default(a3, b2), a3.double() @ b2.double(), dtype)
    ops.check_device_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [1, 2, 7, 8, 9, 15, 16, 17])
def test_few_rows_against_weights_along_k(dtype, M):
    """Row counts on both sides of 8 and 16, N and K at the edges of a CTA's columns, a step, a
    batch of steps and the warps' shares, row pitches, every form of bias, poison outside the rows. Small N with
    K > 256 and short K with many columns: the other small products are a different kernel's."""
    from backendbench_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M)
    rnd = lambda *shape: torch.randn(shape, device="cuda", generator=g).to(dtype)
    eps = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-11
    for N, K, pad in [(1, 264, 0), (7, 520, 0), (16, 264, 8), (17, 1032, 0), (9601, 64, 0), (9601, 136, 8), (250, 1024, 0), (33, 1032, 16), (4099, 2056, 0), (130, 7168, 0), (130, 16384, 0), (64, 16392, 0), (9600, 256, 0)]:
        x, w = rnd(M, K + pad)[:, :K], rnd(N, K + pad)[:, :K]
        if pad:  # what lies between the rows must not be read as part of them
            x._base[:, K:] = float("nan")
            w._base[:, K:] = float("nan")
        assert _abi.lib().b200_gemm_prefers_small(x.data_ptr(), w.data_ptr(), 1, M, N, K, 0, K + pad, 1, 0, 1, K + pad, _abi.BF16 if dtype == torch.bfloat16 else _abi.F16) == 0
        prod, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
        for bias, alpha, beta in [(None, 1, 1), (rnd(N), 1, 1), (rnd(M, 1), 0.5, 2), (rnd(M, N), 1, 1), (torch.full((N,), float("nan"), device="cuda", dtype=dtype), 1, 0)]:
            got = ops.mm_default(x, w.t()) if bias is None else ops.addmm_default(bias, x, w.t(), beta=beta, alpha=alpha)
            want = alpha * prod + (beta * bias.double() if bias is not None and beta else 0)
            # fp32 accumulation (truncating adds: 2^-23 of the running sum each) and one rounding
            bound = want.abs() * eps + (K + 8) * 2.0**-23 * size + 1e-7
            assert got.shape == (M, N) and bool(((got.double() - want).abs() <= bound).all()), (M, N, K)


def test_products_of_few_rows_and_columns_leave_a_long_k_to_ranges():
    """Which of two kernels takes a 16-bit product of at most 16 rows: the one that walks all of K in a CTA asks for no
    scratch, the K-split for 256 bytes and one fp32 copy of the result per range. Where few columns leave the first only a
    handful of CTAs, a long K is cut into ranges (nothing is launched here, the pointers are never followed)."""
    lib = _abi.lib()
    a, b, c = 1 << 20, 1 << 21, 1 << 22
    need = lambda M, N, K: lib.b200_gemm_splitk_scratch_bytes(a, b, c, 1, M, N, K, 0, K, 1, 0, 1, K, _abi.BF16)
    for M, N, K in [(16, 64, 16384), (4, 512, 12288), (2, 128, 8192), (16, 1024, 16384), (8, 1536, 16384), (16, 256, 9216)]:
        ranges, left = divmod(need(M, N, K) - 256, M * N * 4)
        assert ranges >= 2 and left == 0, (M, N, K)
    for M, N, K in [(16, 4096, 11008), (1, 2048, 16384), (16, 64, 4096), (4, 512, 8192), (8, 1536, 12288), (16, 1024, 11008), (16, 8, 11008)]:
        assert need(M, N, K) == 0, (M, N, K)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_few_rows_carry_infinities_and_nan_to_their_own_results(dtype):
    """An infinity or a NaN in one row of x or of the weights reaches that row or column of the result, as in aten, and no other."""
    g = torch.Generator(device=DEV).manual_seed(1)
    x, w = torch.randn(5, 1032, device=DEV, generator=g).to(dtype), torch.randn(300, 1032, device=DEV, generator=g).to(dtype)
    x[1, 1031], x[3, 0], w[7, 515], w[299, 5] = float("inf"), float("nan"), float("-inf"), float("nan")
    got, want = ops.mm_default(x, w.t()).float(), x.double() @ w.double().t()
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got[torch.isinf(want)].double(), want[torch.isinf(want)])
    assert int(torch.isfinite(got).sum()) == 3 * 298


@pytest.mark.parametrize("M,N,K", [(16, 64, 16384), (40, 129, 20000), (45, 2048, 4096), (256, 1030, 4096), (100, 1000, 3000)])
def test_sums_over_ranges_of_k_are_complete(M, N, K):
    """Few and many outputs, few and many ranges of K: with integers whose sums are exact in fp32 a range left out, added twice
    or read past the last one shows in the result."""
    g = torch.Generator(device=DEV).manual_seed(M)
    x, w = (torch.randint(-3, 4, (n, K), device=DEV, generator=g).to(torch.bfloat16) for n in (M, N))
    need = _abi.lib().b200_gemm_splitk_scratch_bytes(x.data_ptr(), w.data_ptr(), x.data_ptr(), 1, M, N, K, 0, K, 1, 0, 1, K, _abi.BF16)
    assert need >= 2 * M * N * 4  # the K-split is what runs
    bias = torch.randint(-3, 4, (N,), device=DEV, generator=g).to(torch.bfloat16)
    exact = x.double() @ w.double().t()  # at most 9 K in size, below 2^24
    assert torch.equal(ops.mm_default(x, w.t()), exact.to(torch.bfloat16))
    assert torch.equal(ops.addmm_default(bias, x, w.t(), beta=2), (exact + 2 * bias.double()).to(torch.bfloat16))



@pytest.mark.parametrize("M,N,K", [(129, 129, 4100), (129, 1029, 4100), (700, 33, 4100), (257, 260, 1027), (300, 515, 1027), (1531, 2050, 1027), (130, 1024, 1030), (513, 1027, 2050)])
def test_fp32_rows_of_c_on_and_off_the_16_byte_grid(M, N, K):
    """The fp32 epilogue writes C row by row from its staging buffer where rows are off the 16-byte grid, straight from registers
    where they are on it: N odd, even, a multiple of 4 and of the tile, at most 32 columns past a multiple of it, ragged M, a bias of each form, batches, transposed operands."""
    g = torch.Generator(device=DEV).manual_seed(M + N)
    for batch in (1, 2):
        a, b = torch.randn(batch, M, K, device=DEV, generator=g), torch.randn(batch, N, K, device=DEV, generator=g).transpose(1, 2)
        exact, size = a.double() @ b.double(), a.double().abs() @ b.double().abs()
        # accumulation adds truncate: at most K / 16 + 8 of them carry the full running sum
        bound = (K / 16 + 32) * 2.0**-23 * size
        if batch == 2:
            assert bool(((ops.bmm_default(a, b).double() - exact).abs() <= bound).all())
            continue
        assert bool(((ops.mm_default(a[0], b[0]).double() - exact[0]).abs() <= bound[0]).all())
        for bias in (torch.randn(N, device=DEV, generator=g), torch.randn(M, 1, device=DEV, generator=g), torch.randn(M, N, device=DEV, generator=g)):
            got = ops.addmm_default(bias, a[0], b[0], beta=0.5, alpha=2.0)
            assert bool(((got.double() - (2 * exact[0] + 0.5 * bias.double())).abs() <= 2 * bound[0] + 2.0**-20 * (1 + bias.double().abs())).all())
    ops.check_device_status()


@pytest.mark.parametrize("M,N,K", [(129, 300, 28000), (1531, 1027, 2050), (2050, 1027, 1531), (256, 256, 20000), (257, 1000, 513), (1000, 1000, 4096)])
def test_fp32_products_cut_into_ranges_of_k(M, N, K):
    """Few tiles and a long K: fp32 partial products over ranges of K (the last one short), added in
    order; the operands in both layouts, a bias, and an infinity, which sends the product to the
    CUDA-core kernel and must leave nothing of the partial products behind."""
    g = torch.Generator(device=DEV).manual_seed(K)
    for ta, tb in ((False, False), (True, True)):
        a = torch.randn(K, M, device=DEV, generator=g).t() if ta else torch.randn(M, K, device=DEV, generator=g)
        b = torch.randn(K, N, device=DEV, generator=g) if tb else torch.randn(N, K, device=DEV, generator=g).t()
        bias = torch.randn(N, device=DEV, generator=g)
        exact, size = a.double() @ b.double(), a.double().abs() @ b.double().abs()
        bound = (K / 16 + 32) * 2.0**-23 * size + 1e-6
        got = ops.mm_default(a, b)
        assert bool(((got.double() - exact).abs() <= bound).all()) and torch.equal(got, ops.mm_default(a, b))
        assert bool(((ops.addmm_default(bias, a, b, beta=2.0, alpha=0.5).double() - (0.5 * exact + 2.0 * bias.double())).abs() <= bound + 1e-5).all())
    # integers of nine bits take two planes each; with 24 terms every sum is exact, so a slab walked twice or left out shows
    ai, bi = torch.zeros(M, K, device=DEV), torch.zeros(K, N, device=DEV)
    ks = torch.cat([torch.arange(8, device=DEV), torch.arange(K - 8, K, device=DEV), torch.arange(K // 2 - 4, K // 2 + 4, device=DEV)])
    ai[:, ks] = torch.randint(257, 512, (M, 24), device=DEV, generator=g).float()
    bi[ks] = torch.randint(257, 512, (24, N), device=DEV, generator=g).float()
    assert torch.equal(ops.mm_default(ai, bi).double(), ai.double() @ bi.double())
    b = b.contiguous()
    b[K // 2, 7] = float("inf")
    got = ops.mm_default(a, b)
    assert bool(torch.isinf(got[:, 7]).all()) and bool((torch.isfinite(got).sum(1) == N - 1).all())
    ops.check_device_status()


def _within_rounding(got, a, b, extra=None):
    """One rounding to the result's type (half a unit in the last of 8 or 11 places: 2^-8 of the value for bf16, 2^-11 for f16), and
    in front of it K additions, each truncated at fp32 (2^-23 of the sum of magnitudes at most)."""
    exact, mass = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    if extra is not None:
        exact, mass = exact + extra.double(), mass + extra.double().abs()
    half_ulp = 2.0**-8 if got.dtype == torch.bfloat16 else 2.0**-11
    bound = exact.abs() * half_ulp * 1.01 + mass * (a.shape[-1] + 2) * 2.0**-23 + 2.0**-25  # (the last: subnormal f16)
    assert bool(((got.double() - exact).abs() <= bound).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N", [1, 500, 4091, 6141, 8185, 11003, 11009])
def test_few_rows_in_every_width_of_a_cta(dtype, N):
    """One to five fragments of eight columns to a CTA, the last CTA cut short, K that ends within a step, within the first
    round of the warps and beyond it, one row up to sixteen, with a bias and after a kernel that is still writing A."""
    g = torch.Generator(device=DEV).manual_seed(N)
    for M, K in [(1, 72), (9, 392), (16, 1032), (7, 2056)]:
        x, w = _rand((M, K), dtype, g, K**-0.5), _rand((N, K), dtype, g, 1.0)
        bias = _rand((N,), dtype, g, 1.0)
        a = ops.relu(x)
        _within_rounding(ops.mm_default(a, w.t()), a, w.t())
        _within_rounding(ops.addmm_default(bias, a, w.t()), a, w.t(), bias)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("b_along_k", [False, True])
@pytest.mark.parametrize("batch,M,K,N", [(1, 1, 64, 1), (1, 4, 65, 33), (1, 5, 255, 64), (3, 8, 257, 65), (1, 9, 2049, 31), (1, 16, 511, 130), (2, 17, 513, 32), (1, 40, 1000, 97), (1, 41, 4097, 63), (2, 100, 7173, 70)])
def test_few_outputs_and_a_long_contraction(dtype, b_along_k, batch, M, K, N, small_path):
    """Rows and columns on both sides of a tile, K that leaves warps or whole CTAs of a cluster without a step or cuts
    the last one, A along K and along M, strides on neither side, a bias, and NaN beside the operands that no lane may pick up."""
    g = torch.Generator(device=DEV).manual_seed(K + N)

    def view(rows, cols, turned, step=1):  # a window into a buffer of NaN
        buf = torch.full((batch, (cols if turned else rows) * step + 2, (rows if turned else cols) * step + 3), float("nan"), dtype=dtype, device=DEV)
        v = buf[:, 1:-1:step, 1:-2:step] if step > 1 else buf[:, 1:-1, 1:-2]
        v = v.transpose(1, 2) if turned else v
        return v.copy_(_rand((batch, rows, cols), dtype, g, 1.0))

    for a_turned, step in ((False, 1), (True, 1), (False, 2)):
        a, b = view(M, K, a_turned), view(K, N, b_along_k, step)
        bias = _rand((M, N), dtype, g, 1.0)
        got = ops.bmm_default(a, b)
        if dtype == torch.float32:
            # one chain of K multiply-adds at most, each rounded to nearest (2^-24 of the sum of magnitudes so far); the bf16 planes
            # of larger products truncate (2^-23) six of them
            mass = a.double().abs() @ b.double().abs()
            assert bool(((got.double() - a.double() @ b.double()).abs() <= mass * (K + 8) * 2.0**-23).all())
            got = ops.addmm_default(bias, a[0], b[0], beta=0.5, alpha=2.0)
            want = 0.5 * bias.double() + 2.0 * (a[0].double() @ b[0].double())
            assert bool(((got.double() - want).abs() <= (2.0 * mass[0] + bias.double().abs()) * (K + 8) * 2.0**-23).all())
        else:
            _within_rounding(got, a, b)
            _within_rounding(ops.addmm_default(bias, a[0], b[0]), a[0], b[0], bias)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N", [129, 130, 132, 191, 250, 255, 257, 514, 770])
def test_rows_of_c_between_two_words(dtype, N):
    """16-bit results whose rows start anywhere: whole and partial chunks of 64 columns, row blocks cut short, batches (the
    parity of a row's first element goes on through them), a bias vector on and off the 16-byte grid and a bias matrix."""
    g = torch.Generator(device=DEV).manual_seed(31)
    for batch, M, K in [(1, 33, 320), (1, 257, 320), (3, 130, 128), (2, 129, 520)]:
        a, b = _rand((batch, M, K), dtype, g, K**-0.5), _rand((batch, N, K), dtype, g, 1.0).transpose(1, 2)
        _within_rounding(ops.bmm_default(a, b), a, b)
        row, col = _rand((N + 1,), dtype, g, 1.0), _rand((M, 1), dtype, g, 1.0)
        for bias in (row[:N], row[1:], _rand((M, N), dtype, g, 1.0), col):
            _within_rounding(ops.addmm_default(bias, a[0], b[0]), a[0], b[0], bias)
    ops.check_device_status()


@pytest.mark.parametrize("M,N,K", [(17, 152, 7221), (61, 64, 3966), (14, 888, 3342), (250, 250, 4096), (129, 255, 1537), (40, 129, 12345), (128, 1030, 2049)])
def test_any_k_is_cut_into_ranges(M, N, K):
    """Ranges of whole slabs, the last one shorter and its end off the slab grid; partial sums with rows off the 16-byte grid."""
    g = torch.Generator(device=DEV).manual_seed(37)
    for dtype in (torch.bfloat16, torch.float16):
        a, w, bias = _rand((M, K), dtype, g, K**-0.5), _rand((N, K), dtype, g, 1.0), _rand((N,), dtype, g, 1.0)
        _within_rounding(ops.addmm_default(bias, a, w.t()), a, w.t(), bias)
        _within_rounding(ops.mm_default(a.t().contiguous().t(), w.t().contiguous()), a, w.t())
        assert torch.equal(ops.mm_default(a, w.t()), ops.mm_default(a, w.t()))
    ops.check_device_status()


@pytest.mark.parametrize("M,N,K", [(257, 129, 320), (1280, 1800, 640), (513, 385, 384), (1300, 960, 330), (2537, 920, 512), (300, 6700, 328), (4100, 193, 328)])
def test_pair_tiles_of_every_width(M, N, K):
    """Tiles of 256, 192 or 128 columns, whichever makes fewest rounds: the last one cut short in each of its chunks of 64
    columns, B along K (any width) and along N, 16-bit and fp32 results."""
    g = torch.Generator(device=DEV).manual_seed(41)
    for dtype in (torch.bfloat16, torch.float16):
        a, w, bias = _rand((M, K), dtype, g, K**-0.5), _rand((N, K), dtype, g, 1.0), _rand((N,), dtype, g, 1.0)
        _within_rounding(ops.mm_default(a, w.t()), a, w.t())
        _within_rounding(ops.addmm_default(bias, a, w.t().contiguous()), a, w.t(), bias)
    a, w = torch.randn((M, K), generator=g, device=DEV) * K**-0.5, torch.randn((N, K), generator=g, device=DEV)
    _check32(ops.mm_default(a, w.t()), a, w.t())
    _check32(ops.mm_default(a, w.t().contiguous()), a, w.t())
    ops.check_device_status()
