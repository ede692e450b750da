"""The host path of small calls: parameter blocks packed in one go, and custom ops bypassed only where their dispatch would do
nothing but call the body."""
import ctypes as C
import random

import pytest
import torch

import fa_b200_capi as capi


@pytest.mark.parametrize("cls,block", [(capi.FwdParams, capi.FWD_BLOCK), (capi.BwdParams, capi.BWD_BLOCK)])
def test_packed_block_equals_the_structure_field_by_field(cls, block):
    rng = random.Random(3)
    p, leaves = cls(), []

    def fill(obj, fields):
        for name, kind in fields:
            if hasattr(kind, "_fields_"):
                fill(getattr(obj, name), kind._fields_)
                continue
            x = {C.c_void_p: lambda: rng.choice([0, rng.randrange(1, 2 ** 48)]), C.c_size_t: lambda: rng.randrange(2 ** 40),
                 C.c_int64: lambda: rng.randrange(-2 ** 40, 2 ** 40), C.c_int32: lambda: rng.randrange(-2 ** 31, 2 ** 31),
                 C.c_float: lambda: rng.uniform(-5, 5)}[kind]()
            setattr(obj, name, x)
            leaves.append(x)

    fill(p, cls._fields_)
    buf = block.new(*leaves)
    assert bytes(buf) == bytes(p) and block.size == C.sizeof(cls)
    ws = torch.empty(64, dtype=torch.uint8)
    capi.set_workspace(block, buf, ws, 48)
    p.workspace, p.workspace_bytes = ws.data_ptr(), 48
    assert bytes(buf) == bytes(p)


def test_cpu_tensors_take_the_op_and_are_refused():
    import flash_attn_npu as fa
    import flash_attn_npu_3 as fa3
    q = torch.randn(1, 8, 2, 64).half()
    assert not capi.plain(q)
    for f in (fa.flash_attn_func, fa3.flash_attn_func):
        with pytest.raises(RuntimeError):                    # NotImplementedError of the dispatcher is one
            f(q, q, q)


def _inputs(dt=torch.bfloat16, d=64):
    g = torch.Generator(device="cuda").manual_seed(1)
    return [torch.randn(2, 130, 2, d, device="cuda", dtype=dt, generator=g) for _ in range(4)]


@pytest.mark.gpu
def test_plain_names_what_the_dispatcher_would_act_on():
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode
    q = _inputs()[0]
    assert capi.plain(q, None) and capi.plain(torch.nn.Parameter(q.clone()).detach())
    assert not capi.plain(q.clone().requires_grad_(True))
    with torch.no_grad():
        assert capi.plain(q.clone().requires_grad_(True))
    assert not capi.plain(torch._neg_view(q))
    with TorchDispatchMode():
        assert not capi.plain(q)
    with TorchFunctionMode():
        assert not capi.plain(q)
    with FakeTensorMode() as mode:
        assert not capi.plain(mode.from_tensor(q))
    seen = []
    torch.func.vmap(lambda t: seen.append(capi.plain(t)) or t)(q)
    with torch.autograd.forward_ad.dual_level():
        seen.append(capi.plain(q))
    assert seen == [False, False]


@pytest.mark.gpu
@pytest.mark.parametrize("version", [2, 3])
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("d", [64, 96, 100])
def test_both_routes_give_the_same_bits(version, packed, d, monkeypatch):
    """The direct route and the op, forward and backward, with saved-tensor hooks around; an int softcap takes the op."""
    import flash_attn_npu as fa2
    import flash_attn_npu_3 as fa3
    from flash_attn_npu import flash_attn_npu_interface as i2
    from flash_attn_npu_3 import flash_attn_npu_interface as i3
    fa = fa2 if version == 2 else fa3
    q, k, v, do = _inputs(d=d)
    cu = torch.tensor([0, 130, 260], dtype=torch.int32, device="cuda")

    def step(softcap):
        x = [t.clone().requires_grad_(True) for t in (q, k, v)]
        packs = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: packs.append(t.shape) or t, lambda t: t):
            if packed:
                out = fa.flash_attn_varlen_func(*[t.flatten(0, 1) for t in x], cu, cu, 130, 130, causal=True, softcap=softcap)
            else:
                out = fa.flash_attn_func(*x, causal=True, softcap=softcap)
        g = torch.autograd.grad(out, x, do.reshape(out.shape))
        assert len(packs) >= 5
        return (out,) + g

    direct = step(0.0)
    assert all(torch.equal(a, b) for a, b in zip(direct, step(0)))
    for m in (i2, i3):
        monkeypatch.setattr(m, "_plain", lambda *t: False)
    assert all(torch.equal(a, b) for a, b in zip(direct, step(0.0)))


@pytest.mark.gpu
def test_transforms_behave_as_with_the_op(monkeypatch):
    """What autograd functions refuse stays refused with the same exception, whichever route a plain call takes."""
    import flash_attn_npu as fa
    from flash_attn_npu import flash_attn_npu_interface as i2
    q, k, v, do = _inputs()

    def twice():
        x = q.clone().requires_grad_(True)
        (g,) = torch.autograd.grad(fa.flash_attn_func(x, k, v), x, do, create_graph=True)
        torch.autograd.grad(g.float().sum(), x)

    def forward_mode():
        with torch.autograd.forward_ad.dual_level():
            fa.flash_attn_func(torch.autograd.forward_ad.make_dual(q, q), k, v)

    calls = (twice, forward_mode, lambda: torch.func.vmap(lambda a: fa.flash_attn_func(a, k, v))(q[None]),
             lambda: torch.func.grad(lambda a: fa.flash_attn_func(a, k, v).float().sum())(q))

    def kinds():
        out = []
        for c in calls:
            try:
                c()
                out.append(None)
            except Exception as e:  # noqa: BLE001
                out.append(type(e))
        return out

    here = kinds()
    monkeypatch.setattr(i2, "_plain", lambda *t: False)
    assert here == kinds()


@pytest.mark.parametrize("name", ["_len_torch_dispatch_stack", "_len_torch_function_stack", "_get_tracing_state"])
def test_a_torch_without_one_of_the_names_takes_the_op(name, monkeypatch):
    assert not capi._dispatch_state()()
    monkeypatch.delattr(torch._C, name)
    acts = capi._dispatch_state()
    monkeypatch.undo()
    assert acts()


def test_a_profiler_is_something_the_dispatch_acts_for():
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]):
        assert capi._dispatch_acts()
    assert not capi._dispatch_acts()


@pytest.mark.gpu
@pytest.mark.parametrize("version", [2, 3])
def test_a_profiler_sees_the_ops(version):
    import flash_attn_npu as fa2
    import flash_attn_npu_3 as fa3
    fa = fa2 if version == 2 else fa3
    q, k, v, do = _inputs()
    x = [t.requires_grad_(True) for t in (q, k, v)]
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        torch.autograd.grad(fa.flash_attn_func(*x), x, do)
    names = {e.name for e in prof.events()}
    pkg = "flash_attn_npu" if version == 2 else "flash_attn_npu_3"
    assert {f"{pkg}::_flash_attn_forward", f"{pkg}::_flash_attn_backward"} <= names
