"""Direct calls of the operators against the dispatcher's way through the same functions: modes, subclasses, hooks, double
backward, profiler."""
import pytest
import torch
import torch.utils._python_dispatch as python_dispatch

from hawk_b200 import ops

pytestmark = pytest.mark.gpu


class _Functions(torch.overrides.TorchFunctionMode):
    def __init__(self):
        self.seen = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.seen.append(str(func))
        return func(*args, **(kwargs or {}))


class _Dispatches(python_dispatch.TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.seen.append(str(func))
        return func(*args, **(kwargs or {}))


class _Sub(torch.Tensor):
    pass


def _cases():
    g = torch.Generator(device="cuda").manual_seed(0)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    labels = torch.randint(0, 96, (60,), generator=g, device="cuda")
    return {
        "scan": (lambda x, gx, ga, lam: ops.fused_linear_scan(x, gx, ga, lam), [rn(2, 40, 64), rn(2, 40, 64), rn(2, 40, 64), rn(64)]),
        "norm": (lambda x, w: ops.rms_norm(x, w, 1e-6), [rn(7, 64), rn(64)]),
        "add_norm": (lambda x, d, w: sum(ops.add_rms_norm(x, d, w, 1e-6)), [rn(7, 64), rn(7, 64), rn(64)]),
        "geglu": (ops.geglu, [rn(9, 128)]),
        "conv": (lambda x, w, b: ops.conv1d_fwd(x, w, b, torch.float32), [rn(2, 30, 64), rn(4, 64), rn(64)]),
        "loss": (lambda w, a: ops.fused_cross_entropy(w, a, labels), [rn(96, 64), rn(60, 64)]),
        "drop_last": (ops.drop_last, [rn(2, 5, 64)]),
    }


NAMES = ["scan", "norm", "add_norm", "geglu", "conv", "loss", "drop_last"]


def _run(fn, inputs, **kw):
    ins = [t.detach().clone().requires_grad_() for t in inputs]
    out = fn(*ins)
    go = torch.linspace(-1, 1, out.numel(), device="cuda").view(out.shape).to(out.dtype)
    return [out.detach(), *(t.detach() for t in torch.autograd.grad(out, ins, go, **kw))]


@pytest.mark.parametrize("name", NAMES)
def test_dispatcher_and_direct_calls_agree(name, monkeypatch):
    fn, inputs = _cases()[name]
    direct = _run(fn, inputs)
    monkeypatch.setattr(ops, "_PROBES", None)
    through = _run(fn, inputs)
    assert all(torch.equal(a, b) for a, b in zip(direct, through))


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("mode", [_Functions, _Dispatches])
def test_modes_see_the_operators(name, mode):
    fn, inputs = _cases()[name]
    direct = _run(fn, inputs)
    with mode() as m:
        inside = _run(fn, inputs)
    assert all(torch.equal(a, b) for a, b in zip(direct, inside))
    assert any("hawk_b200" in s for s in m.seen), m.seen


@pytest.mark.parametrize("name", NAMES)
def test_subclasses_and_hooks(name):
    fn, inputs = _cases()[name]
    direct = _run(fn, inputs)
    out = fn(*(t.as_subclass(_Sub) for t in inputs))
    assert isinstance(out, _Sub) and torch.equal(out.as_subclass(torch.Tensor), direct[0])
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(1), t.cpu())[1], lambda t: t.cuda()):
        offloaded = _run(fn, inputs)
    assert all(torch.equal(a, b) for a, b in zip(direct, offloaded))
    assert packed or name == "drop_last"


@pytest.mark.parametrize("name", NAMES)
def test_create_graph_leaves_the_gradients_as_they_are(name):
    fn, inputs = _cases()[name]
    assert all(torch.equal(a, b) for a, b in zip(_run(fn, inputs), _run(fn, inputs, create_graph=True)))


def test_profiler_shows_operator_names():
    fn, inputs = _cases()["norm"]
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        _run(fn, inputs)
    assert any("hawk_b200::rms_norm_fwd" in e.key for e in prof.key_averages())


def test_opcheck():
    g = torch.Generator(device="cuda").manual_seed(0)
    x, w, b = (torch.randn(*s, generator=g, device="cuda") for s in ((2, 30, 64), (4, 64), (64,)))
    labels = torch.randint(0, 96, (60,), generator=g, device="cuda")
    utils = ("test_schema", "test_faketensor", "test_autograd_registration")
    torch.library.opcheck(ops.cast_bf16, (x,), test_utils=utils)
    torch.library.opcheck(ops.conv1d_fwd, (x.requires_grad_(), w.requires_grad_(), b.requires_grad_(), torch.float32), test_utils=utils)
    torch.library.opcheck(ops.linear_ce, (torch.randn(96, 64, device="cuda", requires_grad=True),
                                          torch.randn(60, 64, device="cuda", requires_grad=True), labels), test_utils=utils)
