"""Backward neighbours of the row operators (`_softmax_backward_data`,
`_log_softmax_backward_data`; BackendBench/backends/flag_gems.py:196,233) against aten CUDA on
the same device tensors and against the CPU oracle, at full size and on the ragged /
non-last-dim / mixed-dtype geometries the fallback kernel serves."""

import pytest
import torch

import oracle
from backendbench_b200 import ops
from backendbench_b200.backends import B200Backend
from backendbench_b200.cases import named_case, scaled_down
from backendbench_b200.eval import compare
from backendbench_b200.opregistry import get_operator

pytestmark = pytest.mark.gpu
DEV = "cuda"
SOFT = "_softmax_backward_data.default"
LOGSOFT = "_log_softmax_backward_data.default"


@pytest.fixture(scope="module")
def backend():
    return B200Backend()


def _tol(dtype):
    return (1e-2, 1e-2) if dtype in (torch.bfloat16, torch.float16) else (1e-5, 1e-5)


@pytest.mark.parametrize("name", ["softmax_backward_bf16_8192x4096", "log_softmax_backward_bf16_8192x4096", "softmax_backward_f32_65536x1024", "log_softmax_backward_f32_65536x1024"])
def test_full_size_matches_aten_cuda_and_oracle_rows(backend, name):
    c = named_case(name)
    op = get_operator(c.op)
    args, kwargs = c.build(DEV)
    got = backend[op](*args, **kwargs)
    want = op(*args, **kwargs)
    atol, rtol = _tol(got.dtype)
    ok, ea, er = compare(want, got, atol, rtol)
    assert ok and got.dtype == want.dtype and got.shape == want.shape, (ea, er)
    head = [a[:64].cpu() if isinstance(a, torch.Tensor) else a for a in args]
    ok, ea, er = compare(oracle.run(c.op, head, {}).to(DEV), got[:64], atol, rtol)
    assert ok, (ea, er)
    # rows of a softmax gradient sum to zero: sum_j (g_j - s) y_j = s - s
    if c.op == SOFT:
        assert float(got.float().sum(-1).abs().max()) < (2e-2 if got.dtype != torch.float32 else 1e-4)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_ragged_non_last_dim_and_strided_inputs(backend, dtype):
    g = torch.Generator(device=DEV).manual_seed(6)
    atol, rtol = _tol(dtype)
    for shape, dim in [((300, 67), -1), ((5, 1000, 9), 1), ((40, 7, 33), 0), ((1, 8192), 1), ((3, 0, 4), 2), ((2049,), 0)]:
        x = torch.randn(shape, device=DEV, generator=g)
        grad = torch.randn(shape, device=DEV, generator=g).to(dtype)
        for spec, fwd in ((SOFT, torch.softmax), (LOGSOFT, torch.log_softmax)):
            y = fwd(x, dim).to(dtype)
            op = get_operator(spec)
            ok, ea, er = compare(op(grad, y, dim, dtype), backend[op](grad, y, dim, dtype), atol, rtol)
            assert ok, (spec, shape, dim, ea, er)
    x = torch.randn(64, 96, device=DEV, generator=g)
    grad_t = torch.randn(96, 64, device=DEV, generator=g).to(dtype).t()  # a transposed incoming gradient
    y = torch.softmax(x, -1).to(dtype)
    op = get_operator(SOFT)
    ok, ea, er = compare(op(grad_t, y, -1, dtype), backend[op](grad_t, y, -1, dtype), atol, rtol)
    assert ok, (ea, er)
    ops.check_device_status()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cols", [1025, 2048 + 1, 8199, 33000, 50257, 65536])
def test_long_rows_off_the_grid_or_past_the_registers(backend, dtype, cols):
    """Rows that start at every offset from the 16-byte grid, bases on and off it (grad, output and
    result alike, or the base of one of them differently), against the fp64 formulas."""
    g = torch.Generator(device=DEV).manual_seed(cols)
    for rows, shift_g, shift_y in ((9, 0, 0), (5, 1, 1), (3, 0, 1)):
        grad = torch.randn(rows * cols + 1, device=DEV, generator=g).to(dtype)[shift_g : shift_g + rows * cols].view(rows, cols)
        x = torch.randn(rows, cols, device=DEV, generator=g)
        for spec, fwd in ((SOFT, torch.softmax), (LOGSOFT, torch.log_softmax)):
            y = torch.empty(rows * cols + 1, device=DEV, dtype=dtype)[shift_y : shift_y + rows * cols].view(rows, cols).copy_(fwd(x, -1))
            got = backend[get_operator(spec)](grad, y, -1, dtype)
            gd, yd = grad.double(), y.double()
            want = gd - yd.exp() * gd.sum(-1, keepdim=True) if spec == LOGSOFT else (gd - (gd * yd).sum(-1, keepdim=True)) * yd
            # an fp32 sum of n terms is off by n 2^-24 sum|terms| at most; ex2 by 2^-21 of its value (argument and unit); one rounding of the result
            terms = gd if spec == LOGSOFT else gd * yd
            off = (cols * 2.0**-24 * terms.abs().sum(-1, keepdim=True) + (2.0**-20 * terms.sum(-1, keepdim=True).abs() if spec == LOGSOFT else 0)) * (yd.exp() if spec == LOGSOFT else yd)
            bound = off + want.abs() * {torch.float32: 2.0**-21, torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11}[dtype] + gd.abs() * 2.0**-22 * (1 if spec == LOGSOFT else yd) + (2.0**-24 if dtype == torch.float16 else 0)
            assert bool(((got.double() - want).abs() <= bound).all()), (spec, rows, float(((got.double() - want).abs() - bound).max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("outer,dim,inner", [(1, 1, 1024), (1, 3, 1025), (1, 65, 4096), (1, 700, 1023), (1, 130, 2050), (3, 129, 700), (40, 33, 64), (1, 4100, 2111)])
def test_softmax_backward_along_a_leading_dim(backend, dtype, outer, dim, inner):
    """Columns in pairs and singly, rows that fill some, all and many trips of the warps, tiles that
    reach past the last column, a base off the word grid; against the fp64 formulas."""
    g = torch.Generator(device=DEV).manual_seed(dim * inner)
    for shift in (0, 1):
        n = outer * dim * inner
        grad = torch.randn(n + 1, device=DEV, generator=g).to(dtype)[shift : shift + n].view(outer, dim, inner)
        x = torch.randn(outer, dim, inner, device=DEV, generator=g)
        for spec, fwd in ((SOFT, torch.softmax), (LOGSOFT, torch.log_softmax)):
            y = fwd(x, 1).to(dtype)
            got = backend[get_operator(spec)](grad, y, 1, dtype).double()
            gd, yd = grad.double(), y.double()
            terms = gd if spec == LOGSOFT else gd * yd
            total = terms.sum(1, keepdim=True)
            want = gd - yd.exp() * total if spec == LOGSOFT else (gd - total) * yd
            # fp32 sums of dim terms in any order, ex2 to 2^-20 of its value, one rounding of the result
            scale = yd.exp() if spec == LOGSOFT else yd
            bound = (dim * 2.0**-24 * terms.abs().sum(1, keepdim=True) + 2.0**-20 * total.abs()) * scale + gd.abs() * 2.0**-22 * (1 if spec == LOGSOFT else yd)
            bound = bound + want.abs() * {torch.float32: 2.0**-21, torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11}[dtype] + (2.0**-24 if dtype == torch.float16 else 0)
            assert bool(((got - want).abs() <= bound).all()), (spec, shift, float(((got - want).abs() - bound).max()))


def test_float_gradients_for_a_half_input(backend):
    """The half_to_float form: fp32 grad_output / output, 16-bit grad_input."""
    g = torch.Generator(device=DEV).manual_seed(7)
    for shape in [(128, 4096), (77, 130)]:
        x = torch.randn(shape, device=DEV, generator=g)
        grad = torch.randn(shape, device=DEV, generator=g)
        for spec, fwd in ((SOFT, torch.softmax), (LOGSOFT, torch.log_softmax)):
            op = get_operator(spec)
            for dt in (torch.float16, torch.bfloat16):
                # aten CUDA takes this form for an f16 input only; the bf16 result is checked against the fp32 one, rounded
                want = op(grad, fwd(x, -1), -1, dt) if dt == torch.float16 else op(grad, fwd(x, -1), -1, torch.float32).to(dt)
                got = backend[op](grad, fwd(x, -1), -1, dt)
                ok, ea, er = compare(want, got, 1e-2, 1e-2)
                assert ok and got.dtype == dt, (spec, shape, dt, ea, er)


LNB = "native_layer_norm_backward.default"


def _check_tuple(want, got, atol, rtol, tag):
    assert len(want) == len(got), tag
    for i, (w_, g_) in enumerate(zip(want, got)):
        if w_ is None or g_ is None:
            assert w_ is None and g_ is None, (tag, i)
            continue
        assert w_.shape == g_.shape and w_.dtype == g_.dtype, (tag, i, w_.shape, g_.shape, w_.dtype, g_.dtype)
        ok, ea, er = compare(w_, g_, atol, rtol)
        assert ok, (tag, i, ea, er)


@pytest.mark.parametrize("name", ["layer_norm_backward_bf16_8192x4096", "layer_norm_backward_f32_65536x1024"])
def test_full_size_layer_norm_backward(backend, name):
    c = named_case(name)
    op = get_operator(c.op)
    args, kwargs = c.build(DEV)
    got = backend[op](*args, **kwargs)
    want = op(*args, **kwargs)
    # dx to the dtype's tolerance; dw / db are sums over thousands of rows: compare at the size of those sums
    atol, rtol = _tol(got[0].dtype)
    _check_tuple(want[:1], got[:1], atol, rtol, name)
    scale = float(want[1].float().abs().max())
    _check_tuple(want[1:], got[1:], max(atol, 2e-3 * scale), 1e-2 if got[0].dtype != torch.float32 else 1e-3, name)
    head = [a[:64].cpu() if isinstance(a, torch.Tensor) and a.dim() == 2 and a.shape[0] == args[0].shape[0] else (a.cpu() if isinstance(a, torch.Tensor) else a) for a in args]
    head[-1] = [True, False, False]
    _check_tuple(oracle.run(c.op, head, {})[:1], (got[0][:64].cpu(),), atol, rtol, name + "/oracle")
    ops.check_device_status()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_layer_norm_backward_geometries_and_masks(backend, dtype):
    g = torch.Generator(device=DEV).manual_seed(9)
    atol, rtol = (3e-2, 2e-2) if dtype != torch.float32 else (1e-4, 1e-4)
    op = get_operator(LNB)
    for shape, nd in [((300, 67), 1), ((5, 40, 1000), 1), ((6, 8, 5), 2), ((64, 8200), 1), ((3, 16384), 1), ((1, 96), 1), ((2000, 17), 1)]:
        x = torch.randn(shape, device=DEV, generator=g).to(dtype)
        dy = torch.randn(shape, device=DEV, generator=g).to(dtype)
        ns = list(shape[-nd:])
        w, b = torch.randn(ns, device=DEV, generator=g).to(dtype), torch.randn(ns, device=DEV, generator=g).to(dtype)
        _, mean, rstd = torch.ops.aten.native_layer_norm.default(x, ns, w, b, 1e-5)
        for weight, bias, mask in [(w, b, [True, True, True]), (w, None, [True, True, False]), (None, None, [True, False, False]), (w, b, [False, True, True]), (w, b, [True, False, False])]:
            want = op(dy, x, ns, mean, rstd, weight, bias, mask)
            got = backend[op](dy, x, ns, mean, rstd, weight, bias, mask)
            rows = x.numel() // max(1, int(torch.tensor(ns).prod()))
            _check_tuple(want[:1], got[:1], atol, rtol, (shape, mask))
            _check_tuple(want[1:], got[1:], atol * max(1.0, rows**0.5), rtol, (shape, mask))
    # fp32 parameters with 16-bit activations (autocast-style)
    if dtype != torch.float32:
        x = torch.randn(128, 512, device=DEV, generator=g).to(dtype)
        dy = torch.randn(128, 512, device=DEV, generator=g).to(dtype)
        w32 = torch.randn(512, device=DEV, generator=g)
        xf = x.float()
        mean, rstd = xf.mean(-1, keepdim=True), torch.rsqrt(xf.var(-1, unbiased=False, keepdim=True) + 1e-5)
        got = backend[op](dy, x, [512], mean, rstd, w32, w32, [True, True, True])
        xhat = (xf - mean) * rstd
        gy = dy.float() * w32
        dx = rstd * (gy - gy.mean(-1, keepdim=True) - xhat * (gy * xhat).mean(-1, keepdim=True))
        _check_tuple((dx.to(dtype), (dy.float() * xhat).sum(0), dy.float().sum(0)), got, 3e-2, 2e-2, "fp32 params")
    ops.check_device_status()


EMB = "embedding_dense_backward.default"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_embedding_backward_matches_oracle_bit_for_bit_and_aten_closely(backend, dtype):
    """Rows are added in ascending position in fp32 and rounded once: the CPU oracle does the
    same, so results agree bit for bit (and run to run); aten CUDA agrees to tolerance."""
    g = torch.Generator().manual_seed(10)
    op = get_operator(EMB)
    impl = backend[op]
    for n_shape, V, D, hot in [((500,), 97, 64, None), ((40, 50), 300, 257, None), ((5000,), 50, 96, 3), ((70000,), 8, 40, 2), ((3,), 1000, 8, None), ((0,), 10, 16, None)]:
        idx = torch.randint(0, V, n_shape, generator=g)
        if hot is not None:  # most positions on a few rows: the many-contributions path
            idx[torch.rand(n_shape, generator=g) < 0.9] = hot
        grad = torch.randn(n_shape + (D,), generator=g).to(dtype)
        pad = 1 if V > 1 else -1
        got = impl(grad.to(DEV), idx.to(DEV), V, pad, False)
        want = oracle.embedding_backward(grad, idx, V, pad, False)
        from conftest import bits_equal

        assert got.shape == (V, D) and got.dtype == dtype and bits_equal(want, got.cpu()), (n_shape, V, D)
        assert bits_equal(got, impl(grad.to(DEV), idx.to(DEV).int(), V, pad, False))  # int32 indices, and reproducible
        ref = op(grad.to(DEV), idx.to(DEV), V, pad, False)
        contributions = max(1, idx.numel() // V if hot is None else idx.numel())
        ok, ea, er = compare(ref, got, (2e-2 if dtype != torch.float32 else 1e-5) * contributions**0.5, 2e-2 if dtype != torch.float32 else 1e-4)
        assert ok, (n_shape, V, D, ea, er)
    ops.check_device_status()
    idx = torch.tensor([1, 5, 99, 2], device=DEV)
    impl(torch.randn(4, 8, device=DEV).to(dtype), idx, 10, -1, False)
    with pytest.raises(IndexError):
        ops.check_device_status()


@pytest.mark.parametrize("dtype,D", [(torch.float32, 33), (torch.float32, 264), (torch.bfloat16, 1), (torch.bfloat16, 67), (torch.float16, 66), (torch.bfloat16, 264), (torch.float16, 4104)])
def test_embedding_backward_at_the_edges_of_its_batches_and_windows(backend, dtype, D):
    """Rows with counts on both sides of the long-row limit (32), of the batch of loads and of the
    CTA's width, and positions on both sides of a sorting window (2^17), bit for bit."""
    from conftest import bits_equal

    g = torch.Generator().manual_seed(D)
    counts = [0, 1, 2, 3, 4, 5, 15, 16, 17, 31, 32, 33, 34, 47, 48, 49, 63, 64, 65, 96, 97, 255, 257, 1000]
    idx = torch.repeat_interleave(torch.arange(len(counts)) * 7, torch.tensor(counts))
    if D == 33:  # long rows that cross from one window of positions into the next
        idx = torch.cat([idx, torch.full((2**17,), 3), idx[-1300:], torch.full((2,), 3)])
    else:
        idx = idx[torch.randperm(idx.numel(), generator=g)]
    grad = torch.randn((idx.numel(), D), generator=g).to(dtype)
    V = 7 * len(counts) + 5
    got = backend[get_operator(EMB)](grad.to(DEV), idx.to(DEV), V, 7, False)
    assert bits_equal(oracle.embedding_backward(grad, idx, V, 7, False), got.cpu())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V,n,D", [(1, 1, 1), (2, 33, 4), (32768, 1024, 9), (32769, 1024, 9), (40000, 1025, 12), (9, 1024, 67), (5, 1025, 67), (3000, 65, 11), (70, 64, 4), (1030, 1000, 5)])
def test_embedding_backward_of_few_tokens(backend, dtype, V, n, D):
    """Both sides of the limits below which one CTA sorts the tokens, and tables off the 16-byte grid that are
    written 16 bytes at a time (a word over two rows, long rows among them), padding and rows out of range, bit for bit."""
    from conftest import bits_equal

    g = torch.Generator().manual_seed(V + n)
    idx = torch.randint(0, V, (n,), generator=g)
    if n >= 64:
        idx[torch.randperm(n, generator=g)[: n - 20]] = V - 1  # a long row; its neighbour is written by another thread
    grad = torch.randn((n, D), generator=g).to(dtype)
    pad = int(idx[-1]) if n == 33 else -1
    got = backend[get_operator(EMB)](grad.to(DEV), idx.to(DEV), V, pad, False)
    ops.check_device_status()
    assert bits_equal(oracle.embedding_backward(grad, idx, V, pad, False), got.cpu())
    if n >= 64:
        idx[3] = V
        backend[get_operator(EMB)](grad.to(DEV), idx.to(DEV), V, pad, False)
        with pytest.raises(IndexError):
            ops.check_device_status()


@pytest.mark.parametrize("V,n,D", [(1, 5000, 9), (3, 40000, 64), (40, 3000, 192), (256, 20000, 63), (256, 20000, 200), (1000, 40000, 8)])
def test_embedding_backward_of_short_tables_under_many_tokens(backend, V, n, D):
    """More rows of many contributions than groups of 256 table rows: they are sorted by CTAs of their own."""
    from conftest import bits_equal

    g = torch.Generator().manual_seed(V)
    for dtype in (torch.float32, torch.bfloat16):
        idx, grad = torch.randint(0, V, (n,), generator=g), torch.randn(n, D, generator=g).to(dtype)
        got = backend[get_operator(EMB)](grad.to(DEV), idx.to(DEV), V, -1, False)
        assert bits_equal(oracle.embedding_backward(grad, idx, V, -1, False), got.cpu())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_softmax_backward_of_streamed_rows_and_columns_with_infinities_and_nan(backend, dtype):
    """Rows off the 16-byte grid from one trip of a CTA to many, few and many of them, and columns by tiles of every size: a NaN or an infinity in
    the gradient spoils its own row (column) and no other, as in aten."""
    g = torch.Generator(device=DEV).manual_seed(8)
    atol, rtol = _tol(dtype)
    one_trip = 2048 * (16 // dtype.itemsize)
    for shape, dim in [((160, 1025), -1), ((9, 1025), -1), ((150, one_trip + 1), -1), ((150, one_trip + 17), -1), ((5, 50257), -1), ((3, 2000), 0), ((8, 1030), 0), ((40, 1025), 0), ((300, 1100), 0), ((20, 70, 64), 1), ((130, 20000), 0)]:
        x = torch.randn(shape, device=DEV, generator=g)
        grad = torch.randn(shape, device=DEV, generator=g).to(dtype)
        for spec, fwd in ((SOFT, torch.softmax), (LOGSOFT, torch.log_softmax)):
            y = fwd(x, dim).to(dtype)
            got = backend[get_operator(spec)](grad, y, dim, dtype)
            ok, ea, er = compare(get_operator(spec)(grad, y, dim, dtype), got, atol, rtol)
            assert ok, (spec, shape, dim, ea, er)
            rows_got, rows_grad = got.movedim(dim, -1).reshape(-1, shape[dim]), grad.clone()
            lines = rows_grad.movedim(dim, -1)
            lines = lines.reshape(-1, shape[dim])  # (a copy where dim is not the last)
            bad = {0: float("nan"), 2: float("inf"), lines.shape[0] - 1: float("-inf")}
            for r, v in bad.items():
                lines[r, (0, shape[dim] // 2, shape[dim] - 1)[r % 3]] = v
            spoiled = lines.reshape(*[n for i, n in enumerate(shape) if i != dim % len(shape)], shape[dim]).movedim(-1, dim).contiguous()
            again = backend[get_operator(spec)](spoiled, y, dim, dtype).movedim(dim, -1).reshape(-1, shape[dim])
            clean = torch.ones(lines.shape[0], dtype=torch.bool, device=DEV)
            for r in bad:
                clean[r] = False
                assert not bool(torch.isfinite(again[r].float()).all()), (spec, shape, r)
            assert torch.equal(again[clean], rows_got[clean]), (spec, shape)


def test_log_softmax_backward_of_columns_is_as_exact_as_its_chains(backend):
    """With y = 0 the result is grad minus the column's sum. In chains of c fp32 additions, of which n / c are added as a tree, that sum is off
    (root mean square) by at most 2^-24 / sqrt 3 sqrt(c / 2 + log2(n / c) + 1) of its size, and the result is rounded once more; c = n / 32."""
    n, cols = 4096, 9600
    grad = torch.randn(n, cols, device=DEV, generator=torch.Generator(device=DEV).manual_seed(2))
    got = backend[get_operator(LOGSOFT)](grad, torch.zeros_like(grad), 0, torch.float32)[:64].double()
    exact = grad[:64].double() - grad.double().sum(0)
    error = float((got - exact).norm() / exact.norm())
    assert error < 2.0**-24 / 3**0.5 * (n / 32 / 2 + 5 + 1 + 1) ** 0.5, error


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cols", [256, 512, 4096])
def test_layer_norm_backward_of_a_constant_gradient(backend, dtype, cols):
    """One value g everywhere under weights of one: what is left of rstd (g - mean g - xhat mean(g xhat)) is next to nothing. The sums of g are exact,
    so the error is that of an fp32 mean of g xhat, about 2^-27 g rstd; rounding rstd mean g, 2^-24 / sqrt 12 of rstd g times the place of
    rstd g in its binade, would show above 2^-26 (both as root mean squares)."""
    g = torch.Generator(device=DEV).manual_seed(cols)
    x = (0.6 * torch.randn(500, cols, device=DEV, generator=g)).to(dtype)
    mean, var = x.double().mean(1, keepdim=True), x.double().var(1, unbiased=False, keepdim=True)
    mean, rstd = mean.float(), (var + 1e-5).rsqrt().float()
    one = torch.ones(cols, device=DEV, dtype=dtype)
    dx = backend[get_operator("native_layer_norm_backward.default")](torch.full_like(x, 0.703125), x, [cols], mean, rstd, one, one, [True, True, True])[0].double()
    xhat = (x.double() - mean.double()) * rstd.double()
    exact = rstd.double() * 0.703125 * (-xhat * xhat.mean(1, keepdim=True))
    assert float(((dx - exact) / (0.703125 * rstd.double())).pow(2).mean().sqrt()) < 2.0**-26


def test_full_size_embedding_backward(backend):
    c = named_case("embedding_backward_bf16_128256x4096_16384")
    op = get_operator(c.op)
    args, kwargs = c.build(DEV)
    got, want = backend[op](*args, **kwargs), op(*args, **kwargs)
    ok, ea, er = compare(want, got, 2e-2, 2e-2)
    assert ok and got.shape == want.shape and got.dtype == want.dtype, (ea, er)
    touched = torch.zeros(128256, dtype=torch.bool, device=DEV)
    touched[args[1]] = True
    assert float(got[~touched].abs().max()) == 0.0  # rows nobody indexed are exactly zero


def test_autograd_through_registered_overrides():
    """With the kernels registered through torch.library, a softmax forward + backward of an
    ordinary autograd graph runs on them and matches aten."""
    import backendbench_b200 as bb

    x = torch.randn(200, 512, device=DEV, requires_grad=True)
    w = torch.randn(200, 512, device=DEV)
    (torch.softmax(x, -1) * w).sum().backward()
    want = x.grad.clone()
    x.grad = None
    bb.enable()
    try:
        (torch.softmax(x, -1) * w).sum().backward()
    finally:
        bb.disable()
    torch.testing.assert_close(x.grad, want, rtol=1e-5, atol=1e-6)
    # layer norm forward + backward, parameters included
    ln = torch.nn.LayerNorm(512).to(DEV)
    x.grad = None
    (ln(x) * w).sum().backward()
    want = [x.grad.clone(), ln.weight.grad.clone(), ln.bias.grad.clone()]
    x.grad = ln.weight.grad = ln.bias.grad = None
    bb.enable()
    try:
        (ln(x) * w).sum().backward()
    finally:
        bb.disable()
    for got_t, want_t in zip([x.grad, ln.weight.grad, ln.bias.grad], want):
        torch.testing.assert_close(got_t, want_t, rtol=1e-4, atol=1e-4)
    # embedding forward + backward
    emb = torch.nn.Embedding(1000, 64).to(DEV)
    tok = torch.randint(0, 1000, (32, 50), device=DEV)
    up = torch.randn(32, 50, 64, device=DEV)
    (emb(tok) * up).sum().backward()
    want_w = emb.weight.grad.clone()
    emb.weight.grad = None
    bb.enable()
    try:
        (emb(tok) * up).sum().backward()
    finally:
        bb.disable()
    torch.testing.assert_close(emb.weight.grad, want_w, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cols", [1, 2, 9, 31, 33, 62, 63, 65, 66, 126, 127, 129, 250, 255, 256, 257, 258, 511, 513, 1023, 1026, 2047, 2934, 8190, 8191])
def test_layer_norm_of_ragged_rows(backend, dtype, cols):
    """Rows off the 16-byte grid, and short ones on it: whole rows in chunks of one or two elements or a vector, a warp or a CTA to a
    row, rows that start between two words, more and fewer rows than there are warps. Each result is within its own
    rounding (2^-24, 2^-8, 2^-11 of the value and a binade) plus a few fp32 roundings of the terms it is made of."""
    g = torch.Generator(device=DEV).manual_seed(cols)
    unit = {torch.float32: 2.0**-23, torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11}[dtype]
    forward, backward = backend[get_operator("native_layer_norm.default")], backend[get_operator("native_layer_norm_backward.default")]

    def within(got, exact, scale):
        assert bool(((got.double() - exact).abs() <= unit * exact.abs() + 2.0**-19 * scale + (2.0**-24 if dtype == torch.float16 else 0)).all())

    for rows in (5, 700) + ((4099,) if cols < 300 else ()):
        x, dy = (torch.randn(rows * cols + 1, device=DEV, generator=g).to(dtype)[k : k + rows * cols].view(rows, cols) for k in (1, 0))
        for params in (dtype, torch.float32):
            w, b = (torch.randn(cols, device=DEV, generator=g) * 0.3 + 1).to(params), torch.randn(cols, device=DEV, generator=g).to(params)
            y, mean, rstd = forward(x, [cols], w, b, 1e-3)
            X, W = x.double(), w.double()
            mu = X.mean(1, keepdim=True)
            rs = (X.sub(mu).square().mean(1, keepdim=True) + 1e-3).rsqrt()
            assert bool(((mean.double() - mu).abs() <= 2.0**-20 * X.abs().mean(1, keepdim=True)).all()) and bool(((rstd.double() / rs - 1).abs() <= 2.0**-18).all())
            within(y, (X - mu) * rs * W + b.double(), ((X - mu).abs() * rs + (X.abs().mean(1, keepdim=True)) * rs + 1) * (W.abs() + b.double().abs() + 1))
            dx, dw, db = backward(dy, x, [cols], mean, rstd, w, b, [True, True, True])
            D, M, R = dy.double(), mean.double(), rstd.double()
            xh, gy = (X - M) * R, D * W
            within(dx, R * (gy - gy.mean(1, keepdim=True) - xh * (gy * xh).mean(1, keepdim=True)), R * (gy.abs() + gy.abs().mean(1, keepdim=True) + xh.abs() * (gy * xh).abs().mean(1, keepdim=True) + 1))
            within(dw, (D * xh).sum(0), (D * xh).abs().sum(0) + rows)
            within(db, D.sum(0), D.abs().sum(0))
            only = backward(dy, x, [cols], mean, rstd, w, b, [True, False, False])
            assert torch.equal(only[0], dx) and only[1] is None and only[2] is None
            assert all(torch.equal(p, q) for p, q in zip(backward(dy, x, [cols], mean, rstd, w, b, [False, True, True])[1:], (dw, db)))
