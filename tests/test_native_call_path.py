"""The operators' native call path (csrc/host_ops.cpp) against the Python autograd Functions it stands in for."""
import subprocess
import sys
import warnings

import pytest
import torch

import lightning_attention_b200 as la
from lightning_attention_b200 import _lib
from lightning_attention_b200.ops.cuda.srmsnorm import _SrmsNorm, _SrmsNormGate

DEV = "cuda"


def test_cpu_tensors_are_left_to_the_python_operators():
    x = torch.zeros(1, 2, 16, 16, dtype=torch.bfloat16)
    H = _lib.host()
    assert H.attn(x, x, x, torch.zeros(2)) is None and H.attn_no_decay(x, x, x) is None and H.prefill(x, x, x, None, None) is None
    assert H.decode(x, x, x, None, x) is None and H.norm(x, 1e-6) is None and H.norm_gate(x, x, 1e-6) is None
    for call in (lambda: la.lightning_attn2(x, x, x, torch.zeros(2)), lambda: la.SimpleRMSNorm(16)(x), lambda: la.srmsnorm_sigmoid_gate(x, x)):
        with pytest.raises(RuntimeError, match="CUDA tensors only"):
            call()


@pytest.mark.parametrize("kind", ["missing", "garbage", "no string", "other torch"])
def test_a_native_path_that_cannot_be_used_costs_one_warning(monkeypatch, tmp_path, kind):
    path = tmp_path / "_host_ops.so"
    if kind == "garbage":
        path.write_bytes(b"not a library")
    elif kind != "missing":
        src = tmp_path / "x.c"
        src.write_text("int x;" if kind == "no string" else 'const char* lab200_host_built_for(void) { return "torch 1.0"; }')
        subprocess.run(["gcc", "-shared", "-fPIC", str(src), "-o", str(path)], check=True)
    assert _lib.host_built_for() == _lib.host_abi()  # the file in the tree
    monkeypatch.setattr(_lib, "HOST_PATH", str(path))
    monkeypatch.setattr(_lib, "_host", None)
    x = torch.zeros(1, 2, 16, 16, dtype=torch.bfloat16)
    with pytest.warns(UserWarning, match="slower Python path"):
        assert _lib.host().attn(x, x, x, torch.zeros(2)) is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        for call in (lambda: la.lightning_attn2(x, x, x, torch.zeros(2)), lambda: la.lightning_attn_decode(x, x, x, None, x), lambda: la.SimpleRMSNorm(16)(x)):
            with pytest.raises(RuntimeError, match="CUDA tensors only"):
                call()


def test_the_build_sees_another_torch(monkeypatch):
    """The native path is compiled anew when it was built for another torch, whatever the times of the files say."""
    from lightning_attention_b200 import build

    runs = []
    monkeypatch.setattr(build, "build_host", lambda verbose=False: runs.append(1))
    monkeypatch.setattr(build, "_newer", lambda *a: True)
    build.build()
    assert not runs
    monkeypatch.setattr(_lib, "host_abi", lambda: "torch 99")
    build.build()
    assert runs == [1]


def test_the_build_runs_by_its_path_as_well():
    from lightning_attention_b200 import build

    r = subprocess.run([sys.executable, build.__file__], capture_output=True, text=True)  # up to date: nothing is compiled
    assert r.returncode == 0 and r.stdout.strip() == build.LIB_PATH, r.stderr


def _tensors(b, h, n, d, e, bnhd, dtype=torch.bfloat16):
    torch.manual_seed(31)
    def one(dim):
        if bnhd:
            return torch.randn(b, n, h, dim, device=DEV, dtype=dtype).transpose(1, 2)
        return torch.randn(b, h, n, dim, device=DEV, dtype=dtype)
    return [one(d).requires_grad_(), one(d).requires_grad_(), one(e).requires_grad_()], one(e)


def _grads(fn, ts, do, **kw):
    o = fn(*ts)
    return (o,) + torch.autograd.grad(o, ts, do, **kw)


def _same(got, ref):
    for x, y in zip(got, ref):
        assert x.shape == y.shape and x.stride() == y.stride() and x.dtype == y.dtype and torch.equal(x, y)


SHAPES = [(1, 4, 256, 64, 64, False), (1, 4, 1000, 128, 128, False), (1, 4, 1000, 128, 128, True), (2, 3, 300, 64, 96, True),
          (4, 32, 130, 128, 128, True), (1, 2, 700, 192, 192, False), (2, 3, 1, 16, 16, False)]


@pytest.mark.gpu
@pytest.mark.parametrize("b,h,n,d,e,bnhd", SHAPES)
@pytest.mark.parametrize("decay", [True, False])
def test_attention_equals_the_python_function(cuda_lib, b, h, n, d, e, bnhd, decay):
    ts, do = _tensors(b, h, n, d, e, bnhd)
    s = la._build_slope_tensor(h).to(DEV) if decay else None
    fast = (lambda q, k, v: la.lightning_attn2(q, k, v, s)) if decay else la.lightning_attn2_no_decay
    slow = (lambda q, k, v: la.LightningAttention2.apply(q, k, v, s)) if decay else la.LightningAttention2NoDecay.apply
    assert (_lib.host().attn(*ts, s) if decay else _lib.host().attn_no_decay(*ts)) is not None
    ref = _grads(slow, ts, do)
    _same(_grads(fast, ts, do), ref)
    # a gradient in another layout, the graph used twice
    odd = do.transpose(2, 3).contiguous().transpose(2, 3)
    o = fast(*ts)
    _same(torch.autograd.grad(o, ts, odd, retain_graph=True), ref[1:])
    _same(torch.autograd.grad(o, ts, do), ref[1:])
    # saved-tensor hooks: what they return is what the backward pass reads
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(1) or t.clone(), lambda t: t):
        o = fast(*ts)
    assert packed
    _same(torch.autograd.grad(o, ts, do), ref[1:])
    with torch.no_grad():
        assert not fast(*ts).requires_grad


@pytest.mark.gpu
@pytest.mark.parametrize("b,h,n,d", [(1, 4, 1000, 128), (4, 32, 130, 64)])
def test_native_path_with_a_dispatch_mode_another_stream_and_two_threads(cuda_lib, b, h, n, d):
    """A dispatch mode sees the Python functions' operations; a backward pass of a forward on a side stream runs there; two threads may
    run the backward pass of one retained graph."""
    import threading

    from torch.utils._python_dispatch import TorchDispatchMode

    ts, do = _tensors(b, h, n, d, d, False)
    s = la._build_slope_tensor(h).to(DEV)
    op = lambda q, k, v: la.lightning_attn2(q, k, v, s)
    ref = _grads(op, ts, do)

    class Seen(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            names.append(str(func))
            return func(*args, **(kwargs or {}))

    names = []
    with Seen():
        assert _lib.host().attn(*ts, s) is None
        o = op(*ts)
    assert any("empty" in x for x in names)
    _same((o,) + torch.autograd.grad(o, ts, do), ref)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        # the copies are late on the side stream: a backward pass on another one would read them too early
        torch.cuda._sleep(20_000_000)
        late = [t.detach().clone().requires_grad_() for t in ts]
        o = op(*late)
    got = torch.autograd.grad(o, late, do)  # called with the default stream current
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    _same((o,) + got, ref)

    o, res = op(*ts), [None, None]
    def run(i):
        res[i] = [torch.autograd.grad(o, ts, do, retain_graph=True) for _ in range(20)]
    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for r in res:
        for g in r:
            _same(g, ref[1:])


def _odd_strides(t):
    """The same values with the second dimension innermost (one-dimensional and byte tensors as they are)."""
    return t.transpose(1, -1).contiguous().transpose(1, -1) if t.dim() > 1 else t


@pytest.mark.gpu
@pytest.mark.parametrize("b,h,n,d,e,bnhd", [(1, 4, 1000, 128, 128, True), (1, 4, 1000, 128, 128, False), (2, 3, 300, 64, 96, True),
                                            (4, 32, 130, 128, 128, True), (1, 2, 700, 192, 192, False)])
@pytest.mark.parametrize("decay", [True, False])
@pytest.mark.parametrize("cls", [False, True], ids=["native", "class"])
def test_saved_tensor_hooks_that_return_another_layout(cuda_lib, b, h, n, d, e, bnhd, decay, cls):
    """Cut into chunks and not; what comes back has the values that were packed, in other strides: the gradients are the same."""
    ts, do = _tensors(b, h, n, d, e, bnhd)
    s = la._build_slope_tensor(h).to(DEV) if decay else None
    if cls:
        op = (lambda q, k, v: la.LightningAttention2.apply(q, k, v, s)) if decay else la.LightningAttention2NoDecay.apply
    else:
        op = (lambda q, k, v: la.lightning_attn2(q, k, v, s)) if decay else la.lightning_attn2_no_decay
    assert (_lib.host().attn(*ts, s) if decay else _lib.host().attn_no_decay(*ts)) is not None
    ref = _grads(op, ts, do)
    hooks = [torch.autograd.graph.saved_tensors_hooks(lambda t: t, f) for f in (lambda t: t.contiguous().clone(), _odd_strides)]
    hooks += [torch.autograd.graph.save_on_cpu(pin_memory=True), torch.autograd.graph.save_on_cpu()]
    for ctx in hooks:
        with ctx:
            o = op(*ts)
        _same(torch.autograd.grad(o, ts, do, retain_graph=True), ref[1:])
        _same(torch.autograd.grad(o, ts, do), ref[1:])
    from torch.utils.checkpoint import checkpoint

    w = torch.ones((), device=DEV, dtype=ts[0].dtype)  # the recomputed k and v are other tensors than the forward pass had
    _same(torch.autograd.grad(checkpoint(lambda q, k, v: op(q * w, k * w, v * w), *ts, use_reentrant=False), ts, do), ref[1:])
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t.float()):
        o = op(*ts)
    with pytest.raises(RuntimeError, match="hooks returned another"):
        torch.autograd.grad(o, ts, do)


@pytest.mark.gpu
def test_other_forms_take_the_python_function(cuda_lib):
    ts, do = _tensors(1, 4, 200, 64, 64, False)
    s = la._build_slope_tensor(4).to(DEV)
    H = _lib.host()
    odd = [t.detach().transpose(2, 3).contiguous().transpose(2, 3).requires_grad_() for t in ts]
    assert H.attn(*odd, s) is None and H.attn(*ts, s.cpu()) is None and H.attn(*ts, s.double()) is None
    ref = _grads(lambda *t: la.lightning_attn2(*t, s), ts, do)
    _same(_grads(lambda *t: la.lightning_attn2(*t, s.cpu()), odd, do), ref)
    import torch.autograd.forward_ad as fwAD
    with fwAD.dual_level():
        dual = fwAD.make_dual(ts[0].detach(), torch.ones_like(ts[0]))
        assert H.attn(dual, ts[1], ts[2], s) is None
        with pytest.raises(RuntimeError):
            la.lightning_attn2(dual, ts[1], ts[2], s)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda x: la.lightning_attn2(x, x, x, s))(torch.stack([ts[0].detach()] * 2))
    with pytest.raises(AttributeError):
        la.lightning_attn2(*ts, None)
    with pytest.raises(RuntimeError, match="share one dtype"):
        la.lightning_attn2(ts[0], ts[1].half(), ts[2], s)
    with pytest.raises(RuntimeError, match="need at least"):
        la.lightning_attn2(*ts, s[:2])
    flat = torch.zeros(ts[0].numel() + 1, device=DEV, dtype=torch.bfloat16)[1:].view(ts[0].shape)
    with pytest.raises(RuntimeError, match="code 6"):
        la.lightning_attn2(flat, flat, flat, s)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(64,), (5, 33), (3, 7, 512), (2, 4096)])
def test_norms_equal_the_python_functions(cuda_lib, dtype, shape):
    torch.manual_seed(32)
    x, g, dy = (torch.randn(shape, device=DEV, dtype=dtype) for _ in range(3))
    x.requires_grad_(), g.requires_grad_()
    assert _lib.host().norm(x, 1e-6) is not None
    for eps in (1e-6, 1e-3):
        _same(_grads(lambda t: la.SimpleRMSNorm(shape[-1], eps)(t), [x], dy), _grads(lambda t: _SrmsNorm.apply(t, eps), [x], dy))
        if shape[-1] % 8 == 0:
            _same(_grads(lambda t, u: la.srmsnorm_sigmoid_gate(t, u, eps), [x, g], dy), _grads(lambda t, u: _SrmsNormGate.apply(t, u, eps), [x, g], dy))
    wide = torch.randn(shape + (2,), device=DEV, dtype=dtype)[..., 0]
    _same(_grads(la.SimpleRMSNorm(shape[-1]), [x], wide), _grads(lambda t: _SrmsNorm.apply(t, 1e-6), [x], wide))
    assert la.SimpleRMSNorm(shape[-1])(wide).shape == wide.shape


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("cls", [False, True], ids=["native", "class"])
def test_norms_under_saved_tensor_hooks_that_return_another_layout(cuda_lib, dtype, cls):
    x, g, dy = (torch.randn((6, 5, 512), device=DEV, dtype=dtype) for _ in range(3))
    x.requires_grad_(), g.requires_grad_()
    norm = (lambda t: _SrmsNorm.apply(t, 1e-6)) if cls else la.SimpleRMSNorm(512)
    gated = (lambda t, u: _SrmsNormGate.apply(t, u, 1e-6)) if cls else la.srmsnorm_sigmoid_gate
    ref = _grads(norm, [x], dy)[1:], _grads(gated, [x, g], dy)[1:]
    apart = lambda t: torch.stack([t, t], -1)[..., 0]  # every second element: no dimension is contiguous
    off = lambda t: torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view(t.shape)  # contiguous, not 16-byte aligned
    for unpack in (_odd_strides, apart, off):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            y, z = norm(x), gated(x, g)
        # rows that lost their alignment are reduced by another kernel, in another order: one rounding of the 16-bit result may differ
        for a, b in zip(torch.autograd.grad(y, [x], dy) + torch.autograd.grad(z, [x, g], dy), ref[0] + ref[1]):
            assert torch.linalg.vector_norm((a - b).float()) <= (2.0 ** -8 if dtype == torch.bfloat16 else 1e-6) * torch.linalg.vector_norm(b.float())


class _Marked(torch.Tensor):
    """A subclass without a dispatch key of its own."""


@pytest.mark.gpu
@pytest.mark.parametrize("dim", [64, 33])
def test_norms_keep_the_type_of_a_tensor_subclass(cuda_lib, dim):
    x, g, dy = (torch.randn((4, dim), device=DEV) for _ in range(3))
    calls = [lambda t: la.SimpleRMSNorm(dim)(t), lambda t: la.srmsnorm_sigmoid_gate(t, g.as_subclass(type(t)))]
    for call in calls:
        ref = call(x)
        assert type(ref) is torch.Tensor and type(call(torch.nn.Parameter(x))) is torch.Tensor
        t = x.as_subclass(_Marked).requires_grad_()
        y = call(t)
        assert type(y) is _Marked and torch.equal(y.as_subclass(torch.Tensor), ref)
        p = x.clone().requires_grad_()
        assert torch.equal(torch.autograd.grad(y, t, dy)[0].as_subclass(torch.Tensor), torch.autograd.grad(call(p), p, dy)[0])


@pytest.mark.gpu
@pytest.mark.parametrize("bnhd", [False, True])
def test_inference_calls_equal_the_general_product(cuda_lib, bnhd):
    ts, _ = _tensors(2, 3, 333, 64, 64, bnhd)
    s = la._build_slope_tensor(3).to(DEV)
    o, st = la.lightning_attn_prefill(*ts, s)
    assert not o.requires_grad and _lib.host().prefill(*ts, s, st) is not None
    _same((o, st), la.la_generic(*[t.detach() for t in ts], s, want_state=True))
    _same(la.lightning_attn_prefill(*ts, s, st), la.la_generic(*[t.detach() for t in ts], s, state_in=st, want_state=True))
    q, k, v = (t.detach()[:, :, :1].contiguous() for t in ts)
    st3, st4 = st.clone(), st.clone()
    o4 = la.lightning_attn_decode(q, k, v, s, st4)
    o3 = la.lightning_attn_decode(q[:, :, 0], k[:, :, 0], v[:, :, 0], s.double(), st3)  # fp64 slopes: the Python operator
    assert o4.shape == v.shape
    _same((o4[:, :, 0], st4), (o3, st3))
