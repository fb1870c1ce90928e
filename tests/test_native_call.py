"""The calls from Python into the compiled library (csrc/native_call.cpp): arguments as the launchers get them, tensors checked as
the Python check does; on a GPU the library's product as `torch.mm` forms it."""

import ctypes

import pytest
import torch

from ullm_b200.csrc import launchers, ops
from ullm_b200.csrc.build import load_native


@pytest.fixture(scope="module")
def native():
    module = load_native()
    module.set_slow_need(ops._checked)
    return module


def test_arguments_arrive_as_ctypes_passes_them(native):
    """Each kind of argument, past the registers too, in the order and width of a launcher's declaration."""
    seen = []
    kinds = {launchers.P: ctypes.c_void_p, launchers.I: ctypes.c_int, launchers.F: ctypes.c_float, launchers.LL: ctypes.c_longlong}
    name = "ullm_window_attention"  # the longest mixed list
    types = launchers.LAUNCHERS[name]
    target = ctypes.CFUNCTYPE(ctypes.c_int, *[kinds[t] for t in types])(lambda *a: seen.append(a) or -7)
    fn = native.bind(name, ctypes.cast(target, ctypes.c_void_p).value)
    t = torch.zeros(5)
    given = [{"P": 1 << 40 | i, "I": -i, "F": 0.1 * i, "LL": -(1 << 40) - i}[k] for i, k in enumerate(types)]
    pointers = [i for i, k in enumerate(types) if k == "P"]
    given[pointers[0]], given[pointers[1]], given[types.index("I")] = None, t, (1 << 32) + 3  # (an int is cut to 32 bits)
    assert fn(*given) == -7
    want = list(given)
    want[pointers[1]], want[types.index("I")] = t.data_ptr(), 3
    want = [ctypes.c_float(w).value if k == "F" else w for w, k in zip(want, types)]
    assert list(seen[0]) == want
    for wrong in (given[:-1], given + [0], ["x", *given[1:]], [1.5, *given[1:]]):
        with pytest.raises(TypeError):
            fn(*wrong)
    with pytest.raises(TypeError):
        fn(*given[:-1], last=0)
    with pytest.raises(KeyError):
        native.bind("ullm_no_such_launcher", 1)


def test_addresses_and_checks(native):
    t = torch.zeros(4, 6)
    assert native.ptr(None) is None and native.ptr(t[1:]) == t.data_ptr() + 24
    for args, kw in (((t, "x"), {}), ((t, "x", torch.float32), {}), ((t, "x"), {"dtype": torch.int32, "contiguous": False})):
        with pytest.raises(ops.KernelError, match="x is on cpu"):
            native.need(*args, **kw)
    with pytest.raises(AttributeError):
        native.need(None, "x")
    with pytest.raises(TypeError):
        native.need(t)


def test_every_entry_of_the_table_is_in_the_library(native):
    from ullm_b200.csrc.build import build

    dll = ctypes.CDLL(build(verbose=False))
    for name in (*launchers.LAUNCHERS, *launchers.QUERIES):
        native.bind(name, ctypes.cast(getattr(dll, name), ctypes.c_void_p).value)


@pytest.mark.gpu
@pytest.mark.needs_cuda
def test_checks_on_the_device(native):
    t = torch.zeros(4, 6, device="cuda")
    assert native.need(t, "x") is None and native.need(t, "x", torch.float32, False) is None
    assert native.need(t[:, 1:], "x", torch.float32, contiguous=False) is None
    with pytest.raises(ops.KernelError, match="dtype"):
        native.need(t, "x", torch.bfloat16)
    with pytest.raises(ops.KernelError, match="contiguous"):
        native.need(t[:, 1:], "x", dtype=torch.float32)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert native.stream() == side.cuda_stream
    assert native.stream() == torch.cuda.current_stream().cuda_stream


@pytest.mark.gpu
@pytest.mark.needs_cuda
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("M,N,K", [(2, 2, 2), (17, 8, 7), (33, 1000, 129), (511, 4096, 1024), (1426, 1024, 3072), (2048, 8, 2048)])
def test_the_product_is_torchs(native, M, N, K, wide):
    torch.manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda").bfloat16()
    w = torch.randn(N, K, device="cuda").bfloat16()
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float32 if wide else torch.bfloat16)
    assert native.mm(x, w, out) is True
    want = torch.mm(x, w.t(), out_dtype=torch.float32) if wide else torch.mm(x, w.t())
    assert torch.equal(out, want)


@pytest.mark.gpu
@pytest.mark.needs_cuda
def test_what_the_product_leaves_to_torch(native):
    x, w = torch.zeros(4, 8, device="cuda").bfloat16(), torch.zeros(6, 8, device="cuda").bfloat16()
    out = torch.ones(4, 6, device="cuda").bfloat16()
    for a, b, c in ((x[:1], w, out[:1]), (x[:, 1:], w[:, 1:], out), (x, w[:, ::2], out), (x.float(), w, out), (x, w.half(), out),
                    (x, w, out.t().contiguous().t()), (x, w, out.half()), (x[:0], w, out[:0]), (x[:, :0], w[:, :0], out), (x.cpu(), w, out),
                    (x[None], w, out), (x, w[:5], out)):
        assert native.mm(a, b, c) is False
    before = torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction
    torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
    try:
        assert native.mm(x, w, out) is False
    finally:
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = before
    assert torch.equal(out, torch.ones_like(out))


def recorded(native, fn, calls):
    native.record()
    try:
        for c in calls:
            fn(*c)
    finally:
        tape = native.recorded()
    return tape


def test_lists_of_launches_run_with_other_tensors(native):
    """A list runs with the addresses inside one layer's tensors moved to another's and everything else as it was; layers whose
    lists differ in any other way, and launches that answer an error, are not alike."""
    seen = []
    target = ctypes.CFUNCTYPE(ctypes.c_int, *[{"P": ctypes.c_void_p, "I": ctypes.c_int, "F": ctypes.c_float, "LL": ctypes.c_longlong}[t]
                                              for t in launchers.LAUNCHERS["ullm_add_rmsnorm"]])(lambda *a: seen.append(a) or 0)
    fn = native.bind("ullm_add_rmsnorm", ctypes.cast(target, ctypes.c_void_p).value)
    a, b, c = ((torch.zeros(8, 4), torch.zeros(3)) for _ in range(3))
    step = torch.zeros(100)

    def launch(layer, rows=7, eps=0.25, other=step):
        return [(1, other, layer[0].data_ptr() + 20, None, layer[1], rows, -1, eps, 5), (0, layer[0], other, layer[1], None, rows, 2, 1.5, None)]

    ta, tb = recorded(native, fn, launch(a)), recorded(native, fn, launch(b))
    assert native.alike(ta, a, tb, b)
    seen.clear()
    assert native.replay(tb, c) == 0
    want = [tuple(x.data_ptr() if isinstance(x, torch.Tensor) else x for x in call) for call in launch(c)]
    assert seen == want
    for other in (launch(b, rows=8), launch(b, eps=0.5), launch(b)[:1], launch(b, other=torch.zeros(100)), launch((b[1], b[0]))):
        assert not native.alike(ta, a, recorded(native, fn, other), b)
    assert not native.alike(ta, a, tb, (b[0], torch.zeros(4)))
    assert not native.alike(ta, a, tb, b[:1])
    with pytest.raises(ValueError):
        native.replay(recorded(native, fn, launch(b)), c)  # (not compared)
    with pytest.raises(ValueError):
        native.replay(tb, (c[0][:1], c[1]))
    native.record()
    fn(*launch(a)[0])
    native.unlisted()
    assert native.recorded() is None
    native.record()
    assert native.recorded() is None  # (nothing ran)
    failing = ctypes.CFUNCTYPE(ctypes.c_int, *[ctypes.c_longlong] * 6)(lambda *x: 4)
    bad = native.bind("ullm_argmax", ctypes.cast(failing, ctypes.c_void_p).value)
    assert recorded(native, bad, [(None, 1, 2, 3, None, None)]) is None


def test_a_list_refuses_tensors_of_other_sizes(native):
    """The launches take sizes and types from the recorded layer: a shorter tensor would be read past its end, also where the recorded
    address is its first."""
    seen = []
    target = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_float, ctypes.c_void_p)(lambda *a: seen.append(a) or 0)
    fn = native.bind("ullm_softcap_f32", ctypes.cast(target, ctypes.c_void_p).value)
    a, b, c = ((torch.zeros(8),) for _ in range(3))
    ta, tb = (recorded(native, fn, [(t[0], 8, 1.0, None)]) for t in (a, b))
    assert native.alike(ta, a, tb, b)
    seen.clear()
    for other in ((c[0][:7],), (torch.zeros(9),), (torch.zeros(8, 2)[:, 0],), (), (c[0], c[0]), (c[0].view(torch.int32),)):
        with pytest.raises(ValueError):
            native.replay(tb, other)
    assert not seen
    assert native.replay(tb, c) == 0 and seen[0][0] == c[0].data_ptr()


def test_a_tensor_without_storage_is_an_exception(native):
    """As `Tensor.data_ptr` says it, from every way in."""
    t = torch.zeros(2, 2).to_sparse()
    never = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_float, ctypes.c_void_p)(lambda *a: pytest.fail("called"))
    fn = native.bind("ullm_softcap_f32", ctypes.cast(never, ctypes.c_void_p).value)
    with pytest.raises(RuntimeError, match="doesn't have storage"):
        native.ptr(t)
    with pytest.raises(RuntimeError, match="doesn't have storage"):
        fn(t, 4, 1.0, None)


def test_lists_of_tensors_without_storage_are_an_exception(native):
    quiet = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_float, ctypes.c_void_p)(lambda *a: 0)
    fn = native.bind("ullm_softcap_f32", ctypes.cast(quiet, ctypes.c_void_p).value)
    a, b, t = torch.zeros(3), torch.zeros(3), torch.zeros(2, 2).to_sparse()
    ta, tb = (recorded(native, fn, [(x, 3, 1.0, None)]) for x in (a, b))
    with pytest.raises(RuntimeError, match="doesn't have storage"):
        native.alike(ta, (a, t), tb, (b, t))
    assert native.alike(ta, (a,), tb, (b,))
    with pytest.raises(RuntimeError, match="doesn't have storage"):
        native.replay(tb, (t,))


@pytest.mark.gpu
@pytest.mark.needs_cuda
def test_the_product_is_torchs_where_somebody_watches_or_chooses(native):
    """Profilers, modes and subclasses see `torch.mm`; another preferred library and tunable operations decide in it."""
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Sub(torch.Tensor):
        pass

    x, w = torch.randn(4, 8, device="cuda").bfloat16(), torch.randn(6, 8, device="cuda").bfloat16()
    out = torch.ones(4, 6, device="cuda").bfloat16()
    with Function():
        assert native.mm(x, w, out) is False
    with Dispatch():
        assert native.mm(x, w, out) is False
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]):
        assert native.mm(x, w, out) is False
    assert native.mm(x.as_subclass(Sub), w, out) is False and native.mm(x, torch.nn.Parameter(w), out) is False
    before = torch.backends.cuda.preferred_blas_library()
    torch.backends.cuda.preferred_blas_library("cublaslt")
    try:
        assert native.mm(x, w, out) is False
    finally:
        torch.backends.cuda.preferred_blas_library(before)
    torch.cuda.tunable.enable(True)
    try:
        assert native.mm(x, w, out) is False
    finally:
        torch.cuda.tunable.enable(False)
    assert torch.equal(out, torch.ones_like(out))
    assert native.mm(x, torch.nn.Parameter(w, requires_grad=False), out) is True


@pytest.mark.gpu
@pytest.mark.needs_cuda
def test_a_profiler_sees_the_products_of_the_engine():
    from ullm_b200.csrc import kernels

    K = kernels()
    x, w = torch.randn(400, 2048, device="cuda").bfloat16(), torch.randn(4096, 2048, device="cuda").bfloat16()
    out = torch.empty(400, 4096, device="cuda").bfloat16()
    K.linear(x, w, out)
    want = out.clone()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as seen:
        K.linear(x, w, out)
    assert any(e.key == "aten::mm" for e in seen.key_averages()) and torch.equal(out, want)


def test_without_headers_the_library_is_called_through_ctypes(monkeypatch):
    """Where the extension module cannot be built, the kernels run all the same: a warning, the same arguments, nothing listed."""
    from ullm_b200.csrc import build as b

    def missing(*a, **kw):
        raise RuntimeError("g++ failed on native_call.cpp: Python.h: No such file or directory")

    monkeypatch.setattr(b, "load_native", missing)
    monkeypatch.setattr(b, "build_native", missing)
    assert b.build(verbose=False).endswith(b.LIB_NAME)
    with pytest.warns(UserWarning, match="Python.h"):
        plain = b.calls()
    plain.set_slow_need(ops._checked)
    seen = []
    target = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_float, ctypes.c_void_p)(lambda *a: seen.append(a) or 3)
    fn = plain.bind("ullm_softcap_f32", ctypes.cast(target, ctypes.c_void_p).value)
    t = torch.zeros(3)
    assert fn(t, 1 << 40, 0.5, None) == 3 and fn(plain.ptr(t), 1, 0.5, 1 << 41) == 3
    assert seen == [(t.data_ptr(), 1 << 40, 0.5, None), (t.data_ptr(), 1, 0.5, 1 << 41)]
    assert plain.mm(t, t, t) is False and plain.record() is None and plain.unlisted() is None and plain.recorded() is None
    with pytest.raises(ops.KernelError, match="x is on cpu"):
        plain.need(t, "x")
    for wrong in ((t, 1, 0.5), ("x", 1, 0.5, None)):
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            fn(*wrong)


@pytest.mark.gpu
@pytest.mark.needs_cuda
def test_a_kernel_called_through_ctypes(monkeypatch):
    from ullm_b200.csrc import build as b
    from ullm_b200.csrc.plain_call import PlainCalls

    x = torch.randn(5, 64, device="cuda").bfloat16()
    w, want = torch.rand(64, device="cuda"), torch.empty(5, 64, device="cuda").bfloat16()
    names = ("_native", "_ptr", "_need", "_stream")
    for n in names:
        monkeypatch.setattr(ops, n, getattr(ops, n))  # (put back afterwards)
    ops.Kernels().add_rmsnorm(x, None, w, 1e-6, want)
    monkeypatch.setattr(ops, "calls", PlainCalls)
    k, out = ops.Kernels(), torch.empty_like(want)
    assert isinstance(ops._native, PlainCalls)
    k.add_rmsnorm(x, None, w, 1e-6, out)
    product = torch.empty(5, 64, device="cuda").bfloat16()
    k.linear(x, torch.eye(64, device="cuda").bfloat16(), product)
    k.raise_on_status()
    assert torch.equal(out, want) and torch.equal(product, x)
