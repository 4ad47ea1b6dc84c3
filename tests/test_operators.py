"""Which calls of an operator may run its Python function directly and which belong to torch's dispatcher; on CPU."""
import pytest
import torch
import torch.utils._python_dispatch as python_dispatch

from hawk_b200 import ops

OPERATORS = sorted(k for k, v in vars(ops).items() if isinstance(v, ops._Operator))


class _Passes(torch.overrides.TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class _Dispatches(python_dispatch.TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("context", [_Passes, _Dispatches, torch.autograd.forward_ad.dual_level, torch.profiler.profile,
                                     torch.autograd.profiler.profile])
def test_contexts_of_the_dispatcher(context):
    assert ops._plain_call(()) is False
    with context():
        assert ops._plain_call(()) is None
    assert ops._plain_call(()) is False


def test_transforms_and_tracing_belong_to_the_dispatcher():
    seen = []

    def f(x):
        seen.append(ops._plain_call(()))
        return (x * x).sum()
    torch.func.grad(f)(torch.ones(3))
    torch.vmap(f)(torch.ones(2, 3))
    torch.jit.trace(f, torch.ones(3), check_trace=False)
    assert len(seen) >= 3 and all(s is None for s in seen)


def test_arguments_of_the_dispatcher():
    class Sub(torch.Tensor):
        pass
    cpu = torch.ones(2)
    for args in [(cpu,), (torch.nn.Parameter(cpu),), (cpu.as_subclass(Sub),), (torch.ones(2, device="meta"),), ("text",),
                 ([cpu],), (torch.fx.Proxy(torch.fx.Graph().placeholder("x")),)]:
        assert ops._plain_call(args) is None
    assert ops._plain_call((None, 1, 1.0, True, torch.bfloat16)) is False


def test_a_torch_without_the_private_names_takes_the_dispatcher(monkeypatch):
    monkeypatch.delattr(torch._C, "_len_torch_function_stack")
    assert ops._probes() is None
    monkeypatch.setattr(ops, "_PROBES", None)
    assert ops._plain_call(()) is None


def test_fx_records_an_operator_as_one_node():
    def f(x, w, b):
        return ops.conv1d_fwd(ops.cast_bf16(x), w, b, torch.bfloat16)
    targets = [str(n.target) for n in torch.fx.symbolic_trace(f).graph.nodes if n.op == "call_function"]
    assert [t.split(".")[:2] for t in targets] == [["hawk_b200", "cast_bf16"], ["hawk_b200", "conv1d_fwd"]]


def test_operators_are_torch_library_operators():
    assert len(OPERATORS) >= 34
    for name in OPERATORS:
        op = getattr(ops, name)
        assert isinstance(op, torch.library.CustomOpDef) and op.direct, name
        assert all(hasattr(op, m) for m in ("register_vmap", "register_kernel", "register_torch_dispatch"))


def test_a_registered_kernel_is_used(monkeypatch):
    @ops._operator("hawk_b200_test::twice", mutates_args=())
    def twice(x: torch.Tensor) -> torch.Tensor:
        return 2 * x
    x = torch.ones(3)
    monkeypatch.setattr(ops, "_plain_call", lambda args: False)  # as for a plain CUDA tensor
    assert torch.equal(twice(x), 2 * x)
    twice.register_kernel("cpu")(lambda x: 3 * x)
    assert torch.equal(twice(x), 3 * x)


def test_defaults_left_out(monkeypatch):
    @ops._operator("hawk_b200_test::affine", mutates_args=())
    def affine(x: torch.Tensor, a: float = 2.0, b: float = 1.0) -> torch.Tensor:
        return a * x + b
    x = torch.ones(3)
    seen = []
    for direct in (None, False):  # the dispatcher, the direct way
        monkeypatch.setattr(ops, "_plain_call", lambda args: (seen.append(args[1:]), direct)[1])
        assert [float(affine(x, *rest)[0]) for rest in ((), (3.0,), (3.0, 5.0))] == [3.0, 4.0, 8.0]
        assert float(affine(x, b=5.0)[0]) == 7.0
        with pytest.raises((TypeError, RuntimeError)):
            affine()
    assert seen == 2 * [(2.0, 1.0), (3.0, 1.0), (3.0, 5.0)]


def test_a_registered_vmap_rule_is_used():
    @ops._operator("hawk_b200_test::thrice", mutates_args=())
    def thrice(x: torch.Tensor) -> torch.Tensor:
        return 3 * x
    thrice.register_vmap(lambda info, dims, x: (5 * x, dims[0]))
    assert torch.equal(torch.vmap(thrice)(torch.ones(2, 3)), torch.full((2, 3), 5.0))


def test_linear_ce_sizes_are_asked_on_the_operands_device(monkeypatch):
    """The K splits of the gradient GEMMs follow the current device's SM count, so the calls that size their scratch belong
    under the same device guard as the calls that use it."""
    inside = []

    class Guard:
        def __init__(self, *args):
            pass

        def __enter__(self):
            inside.append(1)

        def __exit__(self, *exc):
            inside.pop()

    class Lib:
        def __getattr__(self, name):
            def call(*args):
                assert inside or name == "hawk_linear_ce_saved_bytes", name
                return 256 if name.endswith("_bytes") else 0
            return call
    monkeypatch.setattr(ops._lib, "load", Lib)
    monkeypatch.setattr(ops, "_on", Guard)
    monkeypatch.setattr(ops, "_stream", lambda t: 0)
    monkeypatch.setattr(ops, "_status_word", lambda device: torch.zeros(1, dtype=torch.int32))
    w, act, labels = torch.ones(4, 8, requires_grad=True), torch.ones(3, 8, requires_grad=True), torch.zeros(3, dtype=torch.long)
    torch.autograd.grad(ops.fused_cross_entropy(w, act, labels), (w, act))
    ops.linear_ce(w.detach(), act.detach(), labels)
