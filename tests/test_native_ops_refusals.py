"""The native module of the operators hands everything unusual back to Python, and what its
allocations throw arrives as torch's own exception."""
import gc
import os
import threading
import time

import pytest
import torch

from raf_b200 import _lib, build, op


def calls(t):
    return [lambda: op.sgd(t, t, t, 0.1, 0.9), lambda: op.group_cast([t], "float16"), lambda: op.fuse_tensor([t]),
            lambda: op.defuse_tensor(t, [t.numel()], [t.numel()], [1])]


@pytest.mark.parametrize("which", range(4))
def test_cpu_tensors_are_refused(which):
    with pytest.raises(ValueError, match="no CPU path"):
        calls(torch.zeros(4))[which]()


def test_null_tensors_are_refused_before_a_launch():
    lib = _lib.load()
    addr, n = _lib.ptr_array([4096, 0]), _lib.i64_array([8, 8])
    at = _lib.i64_array([0, 8])
    other = _lib.ptr_array([8192, 16384])
    for src, dst in ((addr, other), (other, addr)):
        assert lib.rafb200_group_cast(2, src, _lib.F32, dst, _lib.F16, n, None) == 1
    assert lib.rafb200_fuse_tensor(2, addr, n, at, 4, 8192, None) == 1
    assert lib.rafb200_defuse_tensor(2, addr, n, at, 4, 8192, None) == 1


def test_operators_work_without_the_native_module(monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "_ops", None)
    monkeypatch.setattr(build, "ops_path", lambda: str(tmp_path / "missing.so"))
    monkeypatch.setattr(build.subprocess, "run", lambda *a, **k: (_ for _ in ()).throw(FileNotFoundError("no g++")))
    with pytest.warns(UserWarning, match="no g\\+\\+"):
        assert _lib.ops().sgd(1, 2, 3, 4, 5) is None
    with pytest.raises(ValueError, match="no CPU path"):
        calls(torch.zeros(4))[0]()


def test_a_build_puts_a_whole_module_in_place_or_none(monkeypatch, tmp_path):
    out = tmp_path / "ops.so"
    out.write_text("the one before")
    os.utime(out, (0, 0))
    monkeypatch.setattr(build, "ops_path", lambda: str(out))

    def link(cmd, **kw):  # dies half way
        with open(cmd[cmd.index("-o") + 1], "w") as f:
            f.write("half")
        assert out.read_text() == "the one before"
        return build.subprocess.CompletedProcess(cmd, code, "", "")

    monkeypatch.setattr(build.subprocess, "run", link)
    code = 1
    with pytest.raises(RuntimeError):
        build.build_ops()
    assert out.read_text() == "the one before" and len(list(tmp_path.iterdir())) == 1
    code = 0
    build.build_ops()
    assert out.read_text() == "half" and len(list(tmp_path.iterdir())) == 1


def test_the_module_is_named_after_the_versions_it_is_built_for(monkeypatch):
    before = build.ops_path()
    monkeypatch.setattr(torch, "__version__", "9.9")
    assert build.ops_path() != before


@pytest.mark.gpu
@pytest.mark.parametrize("which", range(4))
def test_without_the_native_module_the_results_are_the_same(monkeypatch, which):
    t = torch.arange(5000, device="cuda", dtype=torch.float32) / 7
    want = calls(t)[which]()
    monkeypatch.setattr(_lib, "_ops", _lib._GeneralWay())
    got = calls(t)[which]()
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("which", range(4))
def test_out_of_memory_is_torchs_exception(which):
    gc.collect()
    torch.cuda.empty_cache()
    t = torch.zeros((64 << 20) + torch.cuda.memory_reserved(), device="cuda")  # no cached block holds its copy
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (1 << 20)) / total)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            calls(t)[which]()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,shapes,indices", [
    ([0], [1 << 32, 1 << 32], [2]),  # the product is 2^64: 0 in 64 bits
    ([4], [(1 << 62) + 1, 4], [2]),  # 2^64 + 4
    ([(1 << 62) + 1] * 4, [(1 << 62) + 1] * 4, [1, 2, 3, 4]),  # the sum is 2^64 + 4
])
def test_defuse_tensor_sizes_beyond_64_bits(sizes, shapes, indices):
    flat = torch.zeros(8, device="cuda")
    assert _lib.ops().defuse_tensor(flat, sizes, shapes, indices, None) is None
    with pytest.raises(RuntimeError):  # torch.empty's, in front of any launch
        op.defuse_tensor(flat, sizes, shapes, indices)


class Sub(torch.Tensor):
    pass


@pytest.mark.gpu
def test_subclasses_stay_what_they_are():
    x = torch.ones(5, device="cuda")
    s = x.as_subclass(Sub)
    assert all(type(t) is Sub for t in op.sgd(s, x, s, 0.1, 0.9)) and type(op.group_cast([s], "float16")[0]) is Sub
    p = torch.nn.Parameter(x, requires_grad=False)
    assert all(type(t) is torch.Tensor for t in _lib.ops().sgd(p, x, x, 0.1, 0.9))


@pytest.mark.gpu
def test_strides_of_single_elements_are_kept():
    x = torch.empty_strided((64, 32, 1, 1), (32, 1, 32, 32), device="cuda").zero_()  # channels_last
    y = torch.zeros(64, 32, 1, 1, device="cuda")
    v1, x1 = op.sgd(x, y, y, 0.1, 0.9)
    assert x.is_contiguous() and x1.stride() == x.clone().stride() and v1.stride() == y.clone().stride()
    assert op.group_cast([x], "float16")[0].stride() == torch.empty_like(x).stride()
    for shape in ((0,), (0, 3), (), (1,), (1, 0, 2)):
        e = torch.zeros(shape, device="cuda")
        assert op.group_cast([e], "float16")[0].stride() == torch.empty_like(e).stride()
        assert op.sgd(e, e, e, 0.1, 0.9)[0].shape == e.shape


@pytest.mark.gpu
def test_sgd_on_parameters():
    """Without grad mode the result is data; with it, what torch's own clone makes of a parameter."""
    p, x = torch.nn.Parameter(torch.ones(5, device="cuda")), torch.full((5,), 2.0, device="cuda")
    with torch.no_grad():
        v1, x1 = _lib.ops().sgd(p, x, x, 0.5, 0.5)
    assert not x1.requires_grad and v1.tolist() == [3.0] * 5 and x1.tolist() == [-0.5] * 5
    assert _lib.ops().sgd(p, x, x, 0.5, 0.5) is None
    assert op.sgd(p, x, x, 0.5, 0.5)[1].grad_fn is not None


@pytest.mark.gpu
def test_a_full_launch_queue_stalls_no_other_thread():
    x = torch.ones(5, device="cuda")
    _lib.ops().sgd(x, x, x, 0.1, 0.9)
    torch.cuda.synchronize()
    torch.cuda._sleep(1_000_000_000)  # half a second; what follows waits behind it
    start = last = time.perf_counter()
    caller = threading.Thread(target=lambda: [_lib.ops().sgd(x, x, x, 0.1, 0.9) for _ in range(3000)])
    caller.start()
    longest = 0.0
    while caller.is_alive():
        time.sleep(1e-3)
        now = time.perf_counter()
        longest, last = max(longest, now - last), now
    caller.join()
    assert last - start > 0.3, "the queue never filled"
    assert longest < 0.15


@pytest.mark.gpu
def test_defuse_tensor_of_too_few_elements():
    with pytest.raises(ValueError, match="9 elements"):
        op.defuse_tensor(torch.zeros(8, device="cuda"), [4, 5], [4, 5], [1, 2])


def native(t):
    """Every function of the module on one tensor, as the operators call it."""
    ops, n = _lib.ops(), t.numel()
    return [ops.sgd(t, t, t, 0.1, 0.9), ops.sgd_step([(t, t)], 0.1, 0.9), ops.group_cast([t], 1, None),
            ops.lans([t, t, t, t], 1, 1e-3, 0.9, 0.999, 1e-6, 1, 0.01, 1, 1, True), ops.fuse_tensor([t], None),
            ops.defuse_tensor(t, [n], [n], [1], None)]


def test_cpu_and_fake_tensors_are_handed_back():
    from torch._subclasses.fake_tensor import FakeTensorMode

    with FakeTensorMode():
        fake = torch.empty(4, device="cuda")
    for t in (torch.zeros(4), fake):
        t.grad = torch.zeros_like(t)
        assert native(t) == [None] * 6
    with pytest.raises(ValueError, match="no CPU path"):
        op.lans([torch.zeros(4)] * 4, 1, 1e-3, 0.9, 0.999, 1e-6, 1, 0.01, 1, 1, True)


@pytest.mark.gpu
def test_tensors_that_stand_for_others_are_handed_back():
    """Under a dispatch mode, inside torch.func's transforms, with a lazy negation, as efficient zeros: no
    function looks at the address."""
    from torch.utils._python_dispatch import TorchDispatchMode

    x = torch.ones(3, 4, device="cuda")
    seen = []

    def look(t):
        seen.append(native(t))
        return t.sum()

    torch.func.vmap(look)(x)
    torch.func.grad(look)(x)
    torch.func.functionalize(look)(x)
    look(torch._neg_view(torch.ones(4, device="cuda")))
    look(torch._efficientzerotensor(4, device="cuda"))

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    y = torch.ones(4, device="cuda")
    y.grad = torch.ones(4, device="cuda")
    with Mode():
        seen.append(native(y))
    assert seen == [[None] * 6] * 6
    assert y.tolist() == [1.0] * 4


@pytest.mark.gpu
def test_autograd_and_forward_mode_take_torchs_calls():
    import torch.autograd.forward_ad as fwd

    x = torch.ones(4, device="cuda")
    with fwd.dual_level():
        dual = fwd.make_dual(x, x)
        assert _lib.ops().sgd(dual, x, x, 0.1, 0.9) is None
        assert fwd.unpack_dual(op.sgd(dual, x, x, 0.1, 0.9)[1]).tangent is not None
    for i in range(3):
        args = [x.clone().requires_grad_(j == i) for j in range(3)]
        assert _lib.ops().sgd(*args, 0.1, 0.9) is None
