"""The chained decode kernels: a projection at the edges of its tiles, splits and token counts, and a whole cached token
against the same modules called one by one."""
import pytest
import torch

import hawk_b200.ops as ops
from conftest import rel_l2
from hawk_b200.generate import GraphedDecoder
from hawk_b200.model import HawkConfig, HawkModel, Linear

pytestmark = pytest.mark.gpu


# rows: one, a full and a ragged group of 8 and of 16 (the most that decode_rows_kernel takes), the fewest of the other kernel,
# more than one of its reduction passes (two of 128), the most
# (H, N): one K block and one tile; K not a multiple of 64 with a ragged tile; every K split up to 8; more tiles than SMs
@pytest.mark.parametrize("rows", [1, 8, 11, 16, 17, 129, 256])
@pytest.mark.parametrize("H,N", [(64, 8), (72, 136), (520, 200), (1000, 264), (1536, 768), (2048, 20000)])
@pytest.mark.parametrize("wdt,rdt", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32)])
def test_norm_linear(rows, H, N, wdt, rdt):
    torch.manual_seed(rows + H + N)
    res = torch.randn(rows, 1, H, device="cuda").to(rdt)
    pend = torch.randn(rows, 1, H, device="cuda").bfloat16()
    norm = torch.rand(H, device="cuda") + 0.5
    w = (torch.randn(N, H, device="cuda") / H**0.5).to(wdt)
    for p in (None, pend):
        out = ops.decode_norm_linear(res, p, norm, 1e-6, w, False)
        s = res if p is None else (res.float() + p.float()).to(rdt)
        s = s.double()
        x = (s * torch.rsqrt((s * s).mean(-1, keepdim=True) + 1e-6) * norm.double()).float().bfloat16().double()
        ref = x @ w.bfloat16().double().t()
        # the result is one rounding to bf16 (2^-9 relative at most); x's own roundings can differ in ties only
        assert out.shape == (rows, 1, N) and rel_l2(out, ref) < 3e-3
    ops.check_device_status()


def _model(vocab, hidden, inter, layers, blocks):
    with torch.device("cuda"):
        model = HawkModel(HawkConfig(vocab, hidden, inter, layers, hidden, blocks, 4), use_cache=True)
    with torch.no_grad():
        for p in model.parameters():
            if p.dim() == 2 and float(p.abs().max()) == 0.0:
                p.normal_(0.0, p.shape[1] ** -0.5)
    return model


CASES = [(64, 72, 4, b, half) for b in (1, 13, 19, 32) for half in (True, False)]
CASES += [(256, 768, 16, b, half) for b in (1, 13, 19, 32) for half in (True, False)]
CASES += [(2048, 6144, 16, b, True) for b in (1, 8, 16, 32)] + [(2048, 6144, 16, b, False) for b in (1, 13, 64)]
CASES += [(1024, 3072, 16, b, True) for b in (2, 11)]


@pytest.mark.parametrize("hidden,inter,blocks,batch,half", CASES)
def test_cached_token_against_modules(hidden, inter, blocks, batch, half):
    torch.manual_seed(hidden + batch)
    model = _model(1000, hidden, inter, 2, blocks)
    if half:
        model = model.bfloat16()
    dec = GraphedDecoder(model, batch, autocast=not half, use_graph=False)
    ids = torch.randint(0, 1000, (batch, 6), device="cuda")
    outs = []
    for hooked in (False, True):
        # a hook on a module keeps its layer (and the head) on the module-by-module path
        handles = [m.register_forward_hook(lambda *_: None) for m in model.modules() if isinstance(m, torch.nn.Linear)] if hooked else []
        dec.prefill(ids[:, :4])
        ops.LOG.reset()
        logits = [dec.step(ids[:, t:t + 1]) for t in (4, 5)]
        counts = dict(ops.LOG.counts)
        ops.LOG.reset(enabled=False)
        assert ("decode_layer" in counts) == (not hooked) and ("decode_norm_linear" in counts) == (not hooked)
        outs.append((logits, [(c.recc_state.clone(), c.conv_state.clone()) for c in dec.caches]))
        for h in handles:
            h.remove()
    (la, ca), (lb, cb) = outs
    # both are bf16 computations that differ in the order of fp32 sums: a few bf16 roundings (2^-9 each) of two layers
    for a, b in zip(la, lb):
        assert a.dtype == b.dtype and a.shape == b.shape and rel_l2(a, b) < 2e-2
    for (ra, ka), (rb, kb) in zip(ca, cb):
        assert rel_l2(ra, rb) < 2e-2 and rel_l2(ka, kb) < 2e-2
    ops.check_device_status()


def test_graph_replay_equals_direct_calls():
    torch.manual_seed(0)
    model = _model(1000, 256, 512, 3, 16).bfloat16()
    ids = torch.randint(0, 1000, (5, 12), device="cuda")
    res = []
    for graph in (False, True):
        dec = GraphedDecoder(model, 5, autocast=False, use_graph=graph)
        dec.prefill(ids[:, :4])
        res.append(torch.cat([dec.step(ids[:, t:t + 1]).clone() for t in range(4, 12)], 1))
    assert torch.equal(res[0], res[1])  # the same kernels in the same order of sums


@pytest.mark.parametrize("how", ["assign", "data"])
def test_cached_token_after_replaced_weights(how):
    """A bf16 model given other weights decodes as a model built with them (the converted copies of its small parameters
    follow a replaced parameter, whatever its version)."""
    torch.manual_seed(5)
    model, other = (_model(500, 128, 256, 2, 4).bfloat16() for _ in range(2))
    with torch.no_grad():
        for p in other.parameters():
            p.add_(0.05 * torch.randn_like(p))
    state = {k: v.clone() for k, v in other.state_dict().items()}
    ids = torch.randint(0, 500, (3, 6), device="cuda")

    def run(m):
        dec = GraphedDecoder(m, 3, autocast=False, use_graph=False)
        return [dec.prefill(ids[:, :4]).clone(), dec.step(ids[:, 4:5]).clone()]
    if how == "assign":  # twice: the parameters of both loads are at version 0
        model.load_state_dict({k: v.clone() for k, v in model.state_dict().items()}, assign=True)
    run(model)
    if how == "assign":
        model.load_state_dict(state, assign=True)
    else:
        for k, p in model.named_parameters():
            p.data = state[k]
    for a, b in zip(run(model), run(other)):
        assert torch.equal(a, b)


# an fp32 residual with bf16 weights, as decoding under autocast has it once an optimiser has left bf16 copies: both kernels, a
# ragged group of each size, K at and past 512 and in more than one step
@pytest.mark.parametrize("rows", [1, 8, 11, 16, 17])
@pytest.mark.parametrize("H,N", [(256, 136), (512, 200), (520, 264), (2048, 768), (4096, 136)])
@pytest.mark.parametrize("wdt,rdt", [(torch.bfloat16, torch.float32), (torch.float32, torch.bfloat16)])
def test_norm_linear_of_mixed_types(rows, H, N, wdt, rdt):
    test_norm_linear(rows, H, N, wdt, rdt)


@pytest.mark.parametrize("hidden,inter,blocks,batch", [(64, 72, 4, 3), (256, 768, 16, 13), (256, 768, 16, 19), (1024, 3072, 16, 2)])
def test_cached_token_with_bf16_copies(hidden, inter, blocks, batch):
    """Under autocast, with the bf16 copies that FusedAdamW leaves on the projections: the chain reads them and its results
    are those of the modules."""
    torch.manual_seed(hidden + batch)
    model = _model(1000, hidden, inter, 2, blocks)
    for m in model.modules():
        if isinstance(m, Linear):
            m.weight_bf16, m.weight_bf16_version = m.weight.detach().bfloat16(), m.weight._version
    dec = GraphedDecoder(model, batch, use_graph=False)
    ids = torch.randint(0, 1000, (batch, 6), device="cuda")
    outs = []
    for hooked in (False, True):
        handles = [m.register_forward_hook(lambda *_: None) for m in model.modules() if isinstance(m, torch.nn.Linear)] if hooked else []
        dec.prefill(ids[:, :4])
        ops.LOG.reset()
        outs.append([dec.step(ids[:, t:t + 1]) for t in (4, 5)])
        assert ("decode_layer" in ops.LOG.counts) == (not hooked)
        ops.LOG.reset(enabled=False)
        for h in handles:
            h.remove()
    for a, b in zip(*outs):
        assert a.dtype == b.dtype and rel_l2(a, b) < 2e-2
    ops.check_device_status()


def test_methods_replaced_on_an_object_are_called():
    """A layer's `step`, or a method of one of its modules, replaced on the object: a cached token calls it too."""
    torch.manual_seed(1)
    model = _model(500, 128, 256, 2, 4).bfloat16()
    ids = torch.randint(0, 500, (3, 6), device="cuda")
    dec = GraphedDecoder(model, 3, autocast=False, use_graph=False)
    for module, name in [(model.layers[1], "step"), (model.layers[0].input_norm, "add_forward"), (model.norm, "add_forward"),
                         (model.layers[0].recc, "_decode")]:
        calls, own = [], getattr(module, name)
        setattr(module, name, lambda *args, own=own, calls=calls: (calls.append(1), own(*args))[1])
        dec.prefill(ids[:, :4])
        calls.clear()
        dec.step(ids[:, 4:5])
        assert len(calls) == 1, name
        delattr(module, name)


@pytest.mark.parametrize("batch", [2, 40])  # the chained kernels, the modules
def test_caches_on_another_device_are_refused(batch):
    model = _model(500, 128, 256, 2, 4).bfloat16()
    caches = model.new_caches(batch, device="cpu")
    for c in caches:
        c.recc_state.zero_()
        c.conv_state.zero_()
        c.current_cache_size = 1
    with torch.no_grad(), pytest.raises(RuntimeError, match="tensors on cuda:0 and cpu"):
        model(torch.zeros(batch, 1, dtype=torch.long, device="cuda"), layer_past=caches)
