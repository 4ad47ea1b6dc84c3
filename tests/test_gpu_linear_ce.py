"""Parity of the tcgen05 fused linear + cross-entropy (through the C ABI) with the CPU oracle.

The op computes like the reference under bf16 autocast (bf16 operands and logits, fp32 softmax), so it
is held to 2e-2 (norm-wise) against the fp64 oracle on bf16-rounded operands, and compared with the
oracle's own bf16 emulation of the reference."""
import math

import pytest
import torch

from conftest import load_golden, max_rel, rel_l2
from oracle import linear_ce as oce

pytestmark = pytest.mark.gpu
TOL = 2e-2


def _run(w, act, labels, upstream=1.0, dtype=torch.float32):
    from hawk_b200 import check_device_status, fused_cross_entropy
    wd = w.to("cuda", dtype).requires_grad_(True)
    ad = act.to("cuda", dtype).requires_grad_(True)
    loss = fused_cross_entropy(wd, ad, labels.cuda())
    assert loss.dtype == torch.float32 and loss.dim() == 0
    (upstream * loss).backward()
    check_device_status()
    return loss.detach().cpu(), wd.grad.float().cpu(), ad.grad.float().cpu()


def _case(N, H, V, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    w = (scale * torch.randn(V, H, generator=g) / math.sqrt(H)).bfloat16().float()
    act = torch.randn(N, H, generator=g).bfloat16().float()
    labels = torch.randint(0, V, (N,), generator=g)
    labels[0], labels[-1] = 0, V - 1
    return w, act, labels


@pytest.mark.parametrize("N,H,V", [(128, 64, 256), (200, 64, 300), (1, 64, 257), (2100, 32, 97), (513, 512, 1000),
                                   (4096, 512, 4096), (2047, 2048, 2048)])
def test_linear_ce_matches_oracle(N, H, V):
    w, act, labels = _case(N, H, V, seed=N + H + V, scale=4.0)
    loss, dw, da = _run(w, act, labels, upstream=1.7)
    l64, dw64, da64 = oce.linear_ce_direct(w, act, labels)
    assert abs(float(loss) - float(l64)) <= TOL * abs(float(l64))
    assert rel_l2(dw, 1.7 * dw64) <= TOL and rel_l2(da, 1.7 * da64) <= TOL
    assert max_rel(dw, 1.7 * dw64) <= TOL and max_rel(da, 1.7 * da64) <= TOL


def test_linear_ce_matches_reference_fixture_and_bf16_emulation():
    g = load_golden("linear_ce_ref.npz")
    loss, dw, da = _run(g["w"], g["act"], g["labels"], upstream=float(g["upstream"]))
    assert abs(float(loss) - float(g["loss"])) <= TOL * float(g["loss"])
    assert rel_l2(dw, g["dw"]) <= TOL and rel_l2(da, g["dact"]) <= TOL
    # closer still to the oracle's emulation of the reference under bf16 autocast
    l16, dw16, da16 = oce.linear_ce_fwd_bwd(g["w"], g["act"], g["labels"], autocast_bf16=True)
    up = float(g["upstream"])
    assert abs(float(loss) - float(l16)) <= 2e-3 * float(l16)
    assert rel_l2(dw, up * dw16) <= 1e-2 and rel_l2(da, up * da16) <= 1e-2


def test_linear_ce_zero_weight_gives_log_vocab():
    """The reference initialises lm_head to zero: loss = ln V exactly, d act = 0."""
    N, H, V = 300, 64, 1000
    g = torch.Generator().manual_seed(0)
    act = torch.randn(N, H, generator=g)
    labels = torch.randint(0, V, (N,), generator=g)
    loss, dw, da = _run(torch.zeros(V, H), act, labels)
    assert abs(float(loss) - math.log(V)) < 1e-5
    assert float(da.abs().max()) == 0.0
    _, dw64, _ = oce.linear_ce_direct(torch.zeros(V, H), act.bfloat16().float(), labels)
    assert rel_l2(dw, dw64) <= TOL


def test_linear_ce_bf16_inputs_and_determinism():
    w, act, labels = _case(777, 128, 515, seed=5)
    a = _run(w, act, labels, dtype=torch.bfloat16)
    b = _run(w, act, labels, dtype=torch.bfloat16)
    c = _run(w, act, labels, dtype=torch.float32)
    assert all(torch.equal(p, q) for p, q in zip(a, b))
    assert abs(float(a[0]) - float(c[0])) < 1e-6
    assert rel_l2(a[1], c[1]) <= 1e-2  # bf16 gradients are rounded on return


def test_linear_ce_config2_shape_properties():
    """N = 16*2047, H = 512, V = 32000 (too large for the CPU oracle in seconds): size-independent checks.
    Row sums of dprobs vanish => d weight summed over the vocabulary is ~0; the loss of a sampled row
    subset recomputed in fp64 agrees; every gradient row of an untouched label direction is finite."""
    from hawk_b200 import check_device_status
    from hawk_b200.ops import linear_ce
    N, H, V = 16 * 2047, 512, 32000
    g = torch.Generator(device="cuda").manual_seed(0)
    w = (torch.randn(V, H, generator=g, device="cuda") / math.sqrt(H)).bfloat16().float()
    act = torch.randn(N, H, generator=g, device="cuda").bfloat16().float()
    labels = torch.randint(1, V, (N,), generator=g, device="cuda")
    loss, dw, da = linear_ce(w, act, labels)
    check_device_status()
    assert torch.isfinite(dw).all() and torch.isfinite(da).all()
    # sum_v dprobs[n, v] = 0  =>  sum_v dW[v, :] = 0 up to bf16 rounding of dprobs
    assert float(dw.sum(0).abs().max()) <= 2e-2 * float(dw.abs().sum(0).max())
    idx = torch.arange(0, N, 997, device="cuda")
    logits = (act[idx].double() @ w.double().T)
    ref_rows = torch.logsumexp(logits, -1) - logits.gather(1, labels[idx][:, None]).squeeze(1)
    full = torch.nn.functional.cross_entropy((act.bfloat16() @ w.bfloat16().T).float(), labels)
    assert abs(float(loss) - float(full)) <= 2e-3 * float(full)
    da_ref = ((torch.softmax(logits, -1) - torch.nn.functional.one_hot(labels[idx], V)) @ w.double()) / N
    assert rel_l2(da[idx].cpu(), da_ref.cpu()) <= TOL
    assert float(ref_rows.mean()) > 0


def test_label_outside_the_vocabulary_is_visible_in_the_loss():
    """The reference's gather raises on a label outside [0, V) (hawk/fused_cross_entropy.py:37-39; it has no
    ignore_index).  The kernel cannot raise: such a label makes the loss non-finite instead of silently wrong."""
    from hawk_b200 import ops
    g = torch.Generator().manual_seed(2)
    w = (torch.randn(300, 64, generator=g) / 8).cuda()
    act = torch.randn(200, 64, generator=g).cuda()
    labels = torch.randint(0, 300, (200,), generator=g).cuda()
    assert bool(torch.isfinite(ops.fused_cross_entropy(w, act, labels)))
    labels[17] = -100
    assert not bool(torch.isfinite(ops.fused_cross_entropy(w, act, labels)))
    labels[17] = 300
    assert not bool(torch.isfinite(ops.fused_cross_entropy(w, act, labels)))
    ops.check_device_status()


def test_backward_as_a_threads_first_cuda_call():
    """The backward runs on autograd's thread, where it can be the first call that needs a context (its buffers come from the
    allocator's pool): the tensor maps must not fail to encode there."""
    import threading

    import hawk_b200.ops as ops
    torch.manual_seed(0)
    w, act = torch.randn(1000, 64, device="cuda"), torch.randn(300, 64, device="cuda")
    labels = torch.randint(0, 1000, (300,), device="cuda")
    _, saved = ops.linear_ce_fwd(w, act, labels, True)
    one = torch.ones((), device="cuda")
    want = ops.linear_ce_bwd(w, act, saved, one, True, True)
    got = []
    stream = torch.cuda.current_stream()
    torch.cuda.synchronize()

    def run():
        with torch.cuda.stream(stream):
            got.extend(ops.linear_ce_bwd(w, act, saved, one, True, True))
    t = threading.Thread(target=run)
    t.start()
    t.join()
    assert len(got) == 2 and all(torch.equal(a, b) for a, b in zip(got, want))


# tile heights and K splits that plan_grad chooses: one K block and one ragged pair tile; many splits of a ragged tile; two
# halves per pair with and without splits, both ragged, in either gradient; mixed operand types
@pytest.mark.parametrize("N,H,V", [(1, 8, 2), (255, 72, 257), (513, 264, 1031), (300, 72, 5000), (4000, 520, 9000)])
@pytest.mark.parametrize("wdt,adt", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32)])
def test_linear_ce_tiles_and_splits(N, H, V, wdt, adt):
    from hawk_b200 import check_device_status, fused_cross_entropy
    g = torch.Generator(device="cuda").manual_seed(N + V)
    w = (torch.randn(V, H, generator=g, device="cuda") / math.sqrt(H)).bfloat16()
    act = torch.randn(N, H, generator=g, device="cuda").bfloat16()
    labels = torch.randint(0, V, (N,), generator=g, device="cuda")
    wd, ad = w.to(wdt).requires_grad_(), act.to(adt).requires_grad_()
    loss = fused_cross_entropy(wd, ad, labels)
    (1.7 * loss).backward()
    check_device_status()
    w64, a64 = w.detach().double().requires_grad_(), act.detach().double().requires_grad_()
    ref = torch.nn.functional.cross_entropy(a64 @ w64.t(), labels)
    (1.7 * ref).backward()
    assert wd.grad.dtype == wdt and ad.grad.dtype == adt and abs(float(loss) - float(ref)) <= TOL * float(ref)
    assert rel_l2(wd.grad, w64.grad) <= TOL and rel_l2(ad.grad, a64.grad) <= TOL


@pytest.mark.parametrize("wdt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("adt", [torch.float16, torch.float64])
def test_act_of_other_types_is_converted_to_the_weights(wdt, adt):
    from hawk_b200 import fused_cross_entropy
    w, act, labels = _case(200, 64, 300, seed=1)
    w, labels = w.to("cuda", wdt).requires_grad_(), labels.cuda()
    other = act.to("cuda", adt).requires_grad_()
    same = other.detach().to(wdt).requires_grad_()
    losses = [fused_cross_entropy(w, a, labels) for a in (other, same)]
    grads = [torch.autograd.grad(1.7 * loss, (w, a)) for loss, a in zip(losses, (other, same))]
    assert torch.equal(losses[0], losses[1]) and torch.equal(grads[0][0], grads[1][0])
    assert grads[0][1].dtype == adt and torch.equal(grads[0][1], grads[1][1].to(adt))


@pytest.mark.parametrize("wdt,adt", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32)])
def test_act_of_the_other_type_at_any_address(wdt, adt):
    from hawk_b200 import fused_cross_entropy
    N, H = 200, 64
    w, act, labels = _case(N, H, 300, seed=2)
    w, labels = w.to("cuda", wdt).requires_grad_(), labels.cuda()
    flat = torch.empty(1 + N * H, dtype=adt, device="cuda")
    flat[1:] = act.to("cuda", adt).view(-1)
    odd = flat[1:].view(N, H).requires_grad_()
    even = odd.detach().clone().requires_grad_()
    assert odd.data_ptr() % 16 and not even.data_ptr() % 16
    res = []
    for a in (odd, even):
        loss = fused_cross_entropy(w, a, labels)
        res.append([loss, *torch.autograd.grad(1.7 * loss, (w, a))])
    assert all(torch.equal(p, q) for p, q in zip(*res))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_loss_waiting_for_its_backward(dtype):
    """Between the loss and backward(): the operands may be written, and what is held is no larger than the fp32 gradients
    (an [N,V] tensor would be 2 N V = 15 MB here, the gradients are 2.6 MB)."""
    from hawk_b200 import fused_cross_entropy
    N, H, V = 2500, 64, 3000
    w, act, labels = _case(N, H, V, seed=3)
    w, act, labels = w.to("cuda", dtype).requires_grad_(), act.to("cuda", dtype).requires_grad_(), labels.cuda()
    want = torch.autograd.grad(1.7 * fused_cross_entropy(w, act, labels), (w, act))
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    loss = fused_cross_entropy(w, act, labels)
    held = torch.cuda.memory_allocated() - before
    assert held <= 4 * H * (N + V) + 4096, held
    with torch.no_grad():
        w.zero_()
        act.mul_(3)
    twice = [torch.autograd.grad(1.7 * loss, (w, act), retain_graph=keep) for keep in (True, False)]
    assert all(torch.equal(a, b) for got in twice for a, b in zip(got, want))


@pytest.mark.parametrize("which", [0, 1])
def test_gradient_of_one_operand_only(which):
    from hawk_b200 import fused_cross_entropy
    w, act, labels = _case(300, 64, 500, seed=4)
    both = [w.cuda().requires_grad_(), act.cuda().requires_grad_()]
    want = torch.autograd.grad(fused_cross_entropy(*both, labels.cuda()), both)[which]
    one = [t.detach().requires_grad_(i == which) for i, t in enumerate(both)]
    fused_cross_entropy(*one, labels.cuda()).backward()
    assert torch.equal(one[which].grad, want) and one[1 - which].grad is None
    with torch.no_grad():
        assert not fused_cross_entropy(*both, labels.cuda()).requires_grad


@pytest.mark.parametrize("n", [1, 7, 8, 2047, 2048, 5001])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_scaled(n, dtype):
    from hawk_b200 import ops
    flat = torch.randn(n + 1, device="cuda")
    g = torch.tensor(1.7, device="cuda")
    for x in (flat[:n], flat[1:]):  # at an aligned and an odd address
        assert torch.equal(ops.scaled(x, g, dtype), (g * x).to(dtype))


@pytest.mark.parametrize("shift", [0.0, 300.0, -1000.0])
def test_loss_of_shifted_logits(shift):
    """The loss does not depend on a shift common to a row's logits, and its error is that of rounding each row's log-sum-exp
    to fp32 (half an ulp of the shift, independent from row to row), not one common to all rows."""
    from hawk_b200 import fused_cross_entropy
    N, H, V = 2000, 512, 8000
    g = torch.Generator(device="cuda").manual_seed(0)
    w = (torch.randn(V, H, generator=g, device="cuda") / math.sqrt(H)).bfloat16()
    act = torch.randn(N, H, generator=g, device="cuda").bfloat16()
    if shift:
        w[:, 0], act[:, 0] = shift, 1.0
    labels = torch.randint(0, V, (N,), generator=g, device="cuda")
    want = float(torch.nn.functional.cross_entropy((act @ w.t()).double(), labels))  # from the same bf16 logits on
    ulp = 2.0 ** (math.floor(math.log2(max(abs(shift), 9.0))) - 23)
    # the mean of N roundings, at four standard deviations, and fp32 sums of N terms and of the loss itself (a few ulp of it)
    bound = 4 * ulp / math.sqrt(12 * N) + 1.5e-6
    assert abs(float(fused_cross_entropy(w, act, labels)) - want) <= bound


# K unsplit in both gradient GEMMs, split in one, split in both; each gradient alone, bf16 operands
@pytest.mark.parametrize("N,H,V", [(60, 64, 64), (513, 264, 1031), (300, 72, 5000), (4000, 520, 9000)])
@pytest.mark.parametrize("dtype,which", [(torch.float32, (0, 1)), (torch.bfloat16, (0, 1)), (torch.float32, (0,)), (torch.float32, (1,)),
                                         (torch.float32, ())])
def test_launches_are_counted(N, H, V, dtype, which):
    """What LOG counts for the loss is what a profiler sees of this library's kernels."""
    from hawk_b200 import fused_cross_entropy, ops
    w, act, labels = _case(N, H, V, seed=6)
    t = [w.to("cuda", dtype), act.to("cuda", dtype)]
    for i in which:
        t[i].requires_grad_()
    labels = labels.cuda()

    def step():
        loss = fused_cross_entropy(*t, labels)
        if which:
            torch.autograd.grad(loss, [t[i] for i in which])
    step()
    torch.cuda.synchronize()
    ops.LOG.reset()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        step()
        torch.cuda.synchronize()
    counted = ops.LOG.total_launches()
    ops.LOG.reset(enabled=False)
    assert counted == sum(e.count for e in prof.key_averages() if "hawk::" in e.key)
