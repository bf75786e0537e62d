"""The native calls (csrc/host.cpp) beside the host wrappers they stand in front of: the same bits, the same refusals, and no
call served natively that the dispatcher would have handled in another way."""

import threading

import pytest
import torch

from backendbench_b200 import _native, backward, custom_ops, ops
from backendbench_b200.backends import B200Backend
from backendbench_b200.eval import compare_enqueue, decode_record
from backendbench_b200.opregistry import get_operator
from conftest import bits_equal

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def backend():
    assert _native.module() is not None, "the host module has not been built"
    return B200Backend()


def _wrapper(name):
    return {**ops.OP_TABLE, **backward.BACKWARD_TABLE}[name]


def _outcome(fn, args, kwargs):
    try:
        r = fn(*args, **kwargs)
        ops.check_device_status()
    except Exception as e:
        return type(e)
    return r


def _same(a, b):
    if isinstance(a, type) or isinstance(b, type):
        # (an argument too many: Python's own refusal on the one side, the operator schema's on the other)
        return a is b or {a, b} == {TypeError, RuntimeError}
    if isinstance(a, (tuple, list)):
        return len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    if a is None or b is None:
        return a is b
    return a.shape == b.shape and a.dtype == b.dtype and a.device == b.device and a.stride() == b.stride() and bits_equal(a, b)


def _calls():
    g = torch.Generator(device=DEV).manual_seed(1)

    def r(*s, dt=torch.float32):
        return torch.randn(s, generator=g, device=DEV).to(dt)

    def i(high, *s):
        return torch.randint(0, high, s, generator=g, device=DEV)

    x, y, h, w = r(33, 65), r(33, 65), r(33, 65, dt=torch.float16), r(7, 5, 3, 4)
    shapes = [x, x.t(), x[:, 3:], x[::2], r(), r(1), r(0, 4), r(4, 1, 6).expand(4, 5, 6), w, w.permute(3, 1, 0, 2), h, h[:, 1:], r(2, 3, 4, 5, 6, 1, 2, 2, 1, 2), i(9, 4, 4), r(5, 5).double()]
    for t in shapes:
        yield "relu.default", (t,), {}
        for o in (t, 2, -0.5, True, torch.tensor(3.0), torch.tensor(2.0, device=DEV)):
            yield "mul.Tensor", (t, o), {}
            yield "add.Tensor", (t, o), {"alpha": 0.5}
        for d in (0, -1, 1, 7):
            yield "_softmax.default", (t, d, False), {}
            yield "_log_softmax.default", (t, d, False), {}
            yield "argmax.default", (t, d), {}
            yield "sum.dim_IntList", (t, [d]), {}
        yield "argmax.default", (t,), {"keepdim": True}
        yield "argmax.default", (t, -1, True), {}
        for dims in ([0, 1], [-1, 0], [0, 0], [], None):
            yield "sum.dim_IntList", (t, dims, True), {}
        yield "sum.dim_IntList", (t, [0]), {"dtype": torch.float32}
    yield "_softmax.default", (h, -1, True), {}
    yield "_softmax.default", (r(200, 3), 0, False), {}
    yield "add.Tensor", (x, r(65)), {}
    yield "add.Tensor", (x, r(33, 1)), {"alpha": 2}
    yield "add.Tensor", (x, h), {}
    yield "add.Tensor", (x, r(64)), {}
    yield "add.Tensor", (x, y, 2), {}
    yield "add.Tensor", (2.0, x), {}
    yield "mul.Tensor", (x.t(), r(33)), {}
    yield "add.Tensor", (r(4, 1, 3), r(5, 1)), {}
    c = x > 0
    for args in ((c, x, y), (c.t(), x.t(), y.t()), (c[:1], x, y), (c, x, r(65)), (c, x, h), (c, x, 0.0), (c.to(torch.uint8), x, y), (c, i(3, 33, 65), i(3, 33, 65)), (x, x, y)):
        yield "where.self", args, {}
    for t, ns in ((x, [65]), (x, [33, 65]), (h, [65]), (x.t(), [33]), (x, [64]), (r(3, 4, 5), [4, 5]), (r(0, 5), [5]), (x, [])):
        for p in (None, 1):
            wt = None if p is None else torch.ones(ns, device=DEV, dtype=t.dtype)
            yield "native_layer_norm.default", (t, ns, wt, wt, 1e-5), {}
            yield "native_layer_norm.default", (t, ns, wt, None, 1e-5), {}
    m, s = r(33, 1), r(33, 1).abs()
    for mask in ([True] * 3, [True, False, False], [False, True, False], [False, False, True]):
        yield "native_layer_norm_backward.default", (x, y, [65], m, s, r(65), r(65), mask), {}
        yield "native_layer_norm_backward.default", (h, h, [65], m, s, None, None, mask), {}
        yield "native_layer_norm_backward.default", (x.t(), y.t(), [33], r(65, 1), r(65, 1), r(33), None, mask), {}
    for name in ("_softmax_backward_data.default", "_log_softmax_backward_data.default"):
        yield name, (x, y, -1, torch.float32), {}
        yield name, (x, y, 0, torch.float32), {}
        yield name, (h, h, -1, torch.float32), {}
        yield name, (x, y.t(), -1, torch.float32), {}
        yield name, (x.t(), y.t(), 1, torch.float32), {}
    ix = i(33, 20)
    yield "embedding.default", (x, ix), {}
    yield "embedding.default", (x, ix.int(), -1, False, False), {}
    yield "embedding.default", (w, i(7, 2, 2)), {}
    yield "embedding.default", (x.t(), i(65, 3)), {}
    yield "embedding.default", (i(9, 40, 3), ix), {}
    yield "embedding.default", (x, ix.float()), {}
    yield "embedding.default", (x, torch.tensor([0, 40], device=DEV)), {}
    for pad in (-1, 3):
        yield "embedding_dense_backward.default", (r(20, 8), ix, 33, pad, False), {}
    yield "embedding_dense_backward.default", (r(20, 8), ix, 33, -1, True), {}
    yield "embedding_dense_backward.default", (r(21, 8), ix, 33, -1, False), {}
    yield "embedding_dense_backward.default", (r(2, 3, 8, dt=torch.float16), i(9, 2, 3).int(), 9, -1, False), {}
    for d, n in ((0, 33), (1, 65), (-1, 65), (2, 1)):
        yield "index_select.default", (x, d, i(n, 9)), {}
        yield "index_select.default", (x.t(), d, i(33, 9)), {}
    yield "index_select.default", (r(), 0, i(1, 1)), {}
    yield "index_select.default", (x, 0, i(33, 2, 2)), {}
    yield "index_select.default", (i(9, 40, 3), 0, ix), {}
    yield "index_select.default", (x, 0, torch.tensor([-1], device=DEV)), {}
    for d in (0, 1):
        lim = (33, 65)[d]
        for t, index in ((x, i(lim, 33, 65)), (x, i(lim, 20, 30)), (x.t(), i(33, 40, 20)), (x, i(lim, 33, 66)), (x, i(lim, 33)), (x, i(lim, 33, 65).int()), (x, i(lim, 0, 65)), (x, i(lim, 33, 65) + 1)):
            yield "gather.default", (t, d, index), {}
            yield "gather.default", (t, d, index), {"sparse_grad": False}
            yield "scatter_add.default", (t, d, index, y), {}
            yield "scatter_add.default", (h, d, index, h), {}
    yield "scatter_add.default", (r(), 0, i(1), r()), {}
    for dt in (torch.float32, torch.bfloat16):
        for M, K, N in ((5, 7, 9), (64, 64, 64), (130, 300, 200), (1, 1024, 8), (300, 257, 1000), (40, 2049, 33), (300, 520, 400), (0, 4, 4), (4, 0, 4)):
            a, b = r(M, K, dt=dt), r(K, N, dt=dt)
            for p, q in ((a, b), (a.t().contiguous().t(), b), (a, b.t().contiguous().t()), (torch.cat([a, a], 1)[:, :K], b)):
                yield "mm.default", (p, q), {}
                yield "bmm.default", (p.expand(3, M, K), q.expand(3, K, N).contiguous()), {}
                for bias in (r(N, dt=dt), r(M, N, dt=dt), r(M, 1, dt=dt), r(dt=dt), r(N + 1, dt=dt), r(1, M, N, dt=dt)):
                    yield "addmm.default", (bias, p, q), {}
                yield "addmm.default", (r(N, dt=dt), p, q), {"beta": 0.5, "alpha": 2}
    yield "mm.default", (x, y), {}
    yield "mm.default", (x, h.t()), {}
    yield "mm.default", (x, r(3, 65, 2)), {}
    yield "bmm.default", (r(2, 3, 4), r(3, 4, 5)), {}


def test_every_call_is_answered_as_the_wrapper_answers_it(backend):
    seen, n = set(), 0
    for name, args, kwargs in _calls():
        impl = backend[get_operator(name)]
        want, got = _outcome(_wrapper(name), args, kwargs), _outcome(impl, args, kwargs)
        assert _same(want, got), (name, [getattr(a, "shape", a) for a in args], kwargs, want, got)
        seen.add(name)
        n += 1
    assert len(seen) == len(custom_ops.OPERATORS) and n > 1000


def test_arguments_that_a_call_does_not_use_are_looked_at_all_the_same(backend):
    """What the operator's schema refuses is refused by the native call, too."""
    x, ix = torch.randn(9, 4, device=DEV), torch.zeros(9, 4, dtype=torch.int64, device=DEV)
    embedding, gather = backend[get_operator("embedding.default")], backend[get_operator("gather.default")]
    for call in (lambda: embedding(x, ix, "3"), lambda: embedding(x, ix, -1, "no"), lambda: embedding(x, ix, -1, False, ix), lambda: embedding(x, ix, padding_idx=None), lambda: gather(x, 0, ix, sparse_grad="no")):
        with pytest.raises((RuntimeError, TypeError)):
            call()
    assert bits_equal(embedding(x, ix, 3, False, True), embedding(x, ix)) and bits_equal(gather(x, 0, ix, sparse_grad=True), gather(x, 0, ix))


class _Seen(torch.Tensor):
    calls = 0

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        cls.calls += 1
        return super().__torch_function__(func, types, args, kwargs or {})


def test_what_the_dispatcher_would_handle_in_its_own_way_goes_through_it(backend):
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.utils._python_dispatch import TorchDispatchMode

    impl, op = backend[torch.ops.aten.mul.Tensor], torch.ops.b200.mul.default
    x, y = torch.randn(8, 8, device=DEV), torch.randn(8, 8, device=DEV)
    with FakeTensorMode() as mode:
        assert type(impl(mode.from_tensor(x), mode.from_tensor(y))) is type(mode.from_tensor(x))
    impl(x.as_subclass(_Seen), y)
    assert _Seen.calls > 0

    class Log(TorchDispatchMode):
        names = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.names.append(str(func))
            return func(*args, **(kwargs or {}))

    with Log():
        impl(x, y)
    assert any("b200.mul" in n for n in Log.names)
    p = torch.nn.Parameter(x.clone())
    assert impl(p, y).requires_grad == op(p, y).requires_grad
    with torch.no_grad():
        assert impl(p, y).requires_grad == op(p, y).requires_grad and bits_equal(impl(p, y), op(p, y))
    with torch.inference_mode():
        z = impl(x, y)
        assert z.is_inference() == op(x, y).is_inference() and bits_equal(z, op(x, y))

    def outcome(f):
        try:
            return f()
        except Exception as e:
            return type(e)

    assert _same(outcome(lambda: torch.vmap(op)(x, y)), outcome(lambda: torch.vmap(impl)(x, y)))
    with torch.autograd.forward_ad.dual_level():
        d = torch.autograd.forward_ad.make_dual(x, y)
        a, b = outcome(lambda: torch.autograd.forward_ad.unpack_dual(op(d, y)).tangent is None), outcome(lambda: torch.autograd.forward_ad.unpack_dual(impl(d, y)).tangent is None)
        assert a == b
    with torch.profiler.profile() as prof:
        impl(x, y)
    assert any("b200::mul" in e.key for e in prof.key_averages())
    with pytest.raises(ops.UnsupportedByB200):
        impl(x.cpu(), y.cpu())


def test_streams_threads_capture_and_scratch(backend):
    """A sum that needs scratch on several streams and threads at once, and in a captured graph."""
    impl, x = backend[torch.ops.aten.sum.dim_IntList], torch.randn(1 << 20, 3, device=DEV)
    want = ops.sum_dim_IntList(x, [0])
    got, errors = {}, []

    def work(k):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                for _ in range(20):
                    r = impl(x, [0])
                s.synchronize()
            got[k] = r
        except Exception as e:  # pragma: no cover
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors and len(got) == 6 and all(bits_equal(want, r) for r in got.values())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        r = impl(x, [0])
    x.mul_(2)
    graph.replay()
    torch.cuda.synchronize()
    assert bits_equal(ops.sum_dim_IntList(x, [0]), r)


@pytest.mark.parametrize("native", [True, False])
def test_threads_that_share_a_stream(backend, native):
    """Operators of several launches and scratch between them, each thread with results of its own, all on one stream."""
    g = torch.Generator(device=DEV).manual_seed(3)

    def one(k):
        x = torch.randn(3000 + k, 33, generator=g, device=DEV)
        i = torch.randint(0, 3000 + k, (3000, 33), generator=g, device=DEV)
        t = torch.randint(0, 500 + k, (4000,), generator=g, device=DEV)
        a, b = torch.randn(40, 3000 + 8 * k, generator=g, device=DEV).half(), torch.randn(3000 + 8 * k, 64, generator=g, device=DEV).half()
        ones, m, s = torch.ones(33, device=DEV), x.mean(1, keepdim=True), 1 / x.std(1, keepdim=True)
        return [("scatter_add.default", (x, 0, i, x[:3000].contiguous())), ("sum.dim_IntList", (x, [0])), ("embedding_dense_backward.default", (x[:3000], t[:3000], 500 + k, -1, False)),
                ("mm.default", (a, b)), ("native_layer_norm_backward.default", (x, x, [33], m, s, ones, ones, [True, True, True]))]

    work = [one(k) for k in range(6)]
    call = {n: backend[get_operator(n)] if native else _wrapper(n) for n, _ in work[0]}
    want = [[call[n](*args) for n, args in calls] for calls in work]
    ops.check_device_status()
    wrong = []

    def run(k):
        try:
            for _ in range(30):
                got = [call[n](*args) for n, args in work[k]]
                wrong.extend((k, n) for (n, _), w, r in zip(work[k], want[k], got) if not _same(w, r))
        except Exception as e:  # pragma: no cover
            wrong.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(6)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    ops.check_device_status()
    assert not wrong, wrong
    ops.release_scratch()
    for calls, w in zip(work, want):
        assert all(_same(x, call[n](*args)) for (n, args), x in zip(calls, w))


def test_comparisons_queued_natively_give_the_same_records(monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(2)
    x = torch.randn(1000, 33, generator=g, device=DEV)
    near = x + 1e-3 * torch.randn(1000, 33, generator=g, device=DEV)
    cases = [(x, x), (x, near), ((x, x[0]), (near, x[0])), (x.half(), near.half()), (x, near.t().contiguous().t()), (x, x[:, :5]), (x, x.half()), (x[:0], x[:0]), (x.long(), near.long()), ((x, 3), (x, 3)), (x, None)]
    for ref, res in cases:
        records = []
        for native in (True, False):
            if not native:
                monkeypatch.setattr(_native, "module", lambda: None)
            rec = torch.full((8,), 7, dtype=torch.int32, device=DEV)
            try:
                ok = compare_enqueue(ref, res, 1e-4, 1e-4, rec)
            except Exception as e:
                ok = type(e)
            records.append((ok, decode_record(rec.tolist())))
            monkeypatch.undo()
        assert records[0][0] == records[1][0] and str(records[0][1]) == str(records[1][1]), (records, ref)
