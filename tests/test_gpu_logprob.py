"""Losses and continuation scores from materialised logits against fp64."""
import pytest
import torch

from gpt_moe_b200.evaluation.hellaswag import continuation_scores
from gpt_moe_b200.ops import cuda_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,vocab,pitch", [(1, 1, 1), (5, 7, 7), (3, 1000, 1003), (64, 8192, 8192), (33, 50304, 50304)])
def test_row_losses(rows, vocab, pitch):
    torch.manual_seed(1)
    logits = (6 * torch.randn(rows, pitch, device="cuda")).bfloat16()[:, :vocab]
    if vocab > 4:
        logits[0, :3] = float("-inf")
        logits[-1, 2] = 80.0                                   # one entry far above the rest
    targets = torch.randint(min(3, vocab - 1), vocab, (rows,), device="cuda")
    if rows > 4:
        targets[2] = -100
    got = cuda_ops.cross_entropy(logits, targets, -100)
    want = torch.nn.functional.cross_entropy(logits.double(), targets, ignore_index=-100)
    # fp32 sums of up to 50304 exponentials with 2-ulp exponentials: 1e-6 of a loss of a few units
    assert abs(got.item() - want.item()) < 1e-5 * max(1.0, abs(want.item()))
    assert torch.isnan(cuda_ops.cross_entropy(logits, torch.full_like(targets, -100), -100))      # nothing to average, as in torch
    cuda_ops.check_status()


@pytest.mark.parametrize("spread,offset", [(0.5, 20.0), (3.0, -40.0), (10.0, 20.0), (30.0, 0.0)])
@pytest.mark.parametrize("vocab", [1003, 50304])
def test_row_losses_are_as_exact_as_torchs(spread, offset, vocab):
    torch.manual_seed(9)
    logits = (spread * torch.randn(512, vocab, device="cuda") + offset).bfloat16()
    targets = torch.randint(0, vocab, (512,), device="cuda")
    exact = torch.nn.functional.cross_entropy(logits.double(), targets, reduction="none")
    mine = cuda_ops.ext().row_nll(logits, targets, -100).double() - exact
    torchs = torch.nn.functional.cross_entropy(logits.float(), targets, reduction="none").double() - exact
    assert mine.norm() < 1.25 * torchs.norm() and mine.norm() < 1e-7 * exact.norm()


def test_target_outside_the_vocabulary_is_reported():
    logits = torch.randn(2, 64, device="cuda").bfloat16()
    assert torch.isnan(cuda_ops.cross_entropy(logits, torch.tensor([3, 64], device="cuda"), -100))
    with pytest.raises(RuntimeError):
        cuda_ops.check_status()


@pytest.mark.parametrize("vocab", [64, 56960, 60000, 1003])           # rows in shared memory up to 56960 columns, streamed beyond and for odd widths
@pytest.mark.parametrize("bad", [-1, 0, 7, 1 << 20, -(1 << 40), (1 << 62)])          # distance from the vocabulary's end; negative: from its start
def test_target_outside_the_vocabulary_in_the_training_loss(vocab, bad):
    if cuda_ops.ext().bounds_checked():
        pytest.skip("the bounds-checked build ignores such a row and records code 905")
    torch.manual_seed(6)
    logits = torch.randn(4, (vocab + 7) // 8 * 8, device="cuda").bfloat16()[:, :vocab]
    targets = torch.randint(0, vocab, (4,), device="cuda")
    targets[1] = bad if bad < 0 else vocab + bad
    before = logits.double()
    loss = cuda_ops.ext().ce_fwd_bwd(logits, targets, torch.ones(1, device="cuda"), -100, True)
    keep = torch.tensor([0, 2, 3], device="cuda")
    want = torch.nn.functional.cross_entropy(before[keep], targets[keep], reduction="none")
    assert torch.isnan(loss[1]) and torch.allclose(loss[keep].double(), want, rtol=1e-5, atol=1e-5)
    assert (logits[1] == 0).all() and (logits[keep] != 0).any(dim=1).all()
    with pytest.raises(RuntimeError, match="701"):
        cuda_ops.check_status()


def test_tangents_and_vmap_run_through_torch():
    torch.manual_seed(7)
    logits, v = torch.randn(4, 6, 64, device="cuda").bfloat16(), torch.randn(4, 6, 64, device="cuda").bfloat16()
    ids = torch.randint(0, 64, (4, 6), device="cuda")
    plain = torch.nn.functional.cross_entropy
    with torch.no_grad():
        out, tangent = torch.func.jvp(lambda x: cuda_ops.cross_entropy(x, ids[0], -100), (logits[0],), (v[0],))
        want = torch.func.jvp(lambda x: plain(x.double(), ids[0]), (logits[0],), (v[0],))
        assert abs(out.item() - want[0].item()) < 1e-4 and abs(tangent.item() - want[1].item()) < 1e-2
        rows = torch.func.vmap(lambda x, t: cuda_ops.cross_entropy(x, t, -100))(logits, ids)
        assert torch.allclose(rows.double(), torch.stack([plain(x.double(), t) for x, t in zip(logits, ids)]), atol=1e-4)
        tangent = torch.func.jvp(lambda x: continuation_scores(x, ids, [1, 2, 3, 1], [6, 5, 4, 2]), (logits,), (v,))[1]
        want = torch.func.jvp(lambda x: continuation_scores(x, ids.cpu(), [1, 2, 3, 1], [6, 5, 4, 2]), (logits.cpu().float(),), (v.cpu().float(),))[1]
        assert torch.allclose(tangent.cpu().float(), want, atol=2e-2)
        traced = torch.jit.trace(lambda x: cuda_ops.cross_entropy(x, ids[0], -100), logits[0], check_trace=False)
        assert abs(traced(v[0]).item() - plain(v[0].double(), ids[0]).item()) < 1e-4


def test_gradients_still_run_through_torch():
    logits = torch.randn(4, 64, device="cuda").bfloat16().requires_grad_()
    cuda_ops.cross_entropy(logits, torch.tensor([1, 2, 3, 4], device="cuda"), -100).backward()
    assert logits.grad is not None and logits.grad.abs().sum() > 0


@pytest.mark.parametrize("n,t,vocab", [(1, 2, 9), (4, 17, 1000), (6, 33, 50304)])
def test_continuation_scores(n, t, vocab):
    torch.manual_seed(2)
    logits = (3 * torch.randn(n, t, vocab, device="cuda")).bfloat16()
    ids = torch.randint(0, vocab, (n, t), device="cuda")
    prefix = [min(i, t) for i in range(n)]                     # from the very first position on, where there is no prediction
    true = [min(prefix[i] + 4 * i + 1, t) for i in range(n)]
    true[-1] = t + 5 if n > 1 else true[-1]                    # past the end
    if n > 3:
        true[1] = prefix[1]                                    # empty
    got = continuation_scores(logits, ids, prefix, true)
    want = continuation_scores(logits.cpu().float(), ids.cpu(), prefix, true)
    assert torch.allclose(got.cpu(), want, rtol=2e-5, atol=2e-5)
    cuda_ops.check_status()


def test_continuation_bounds_of_any_kind():
    torch.manual_seed(5)
    logits, ids = torch.randn(3, 9, 128, device="cuda").bfloat16(), torch.randint(0, 128, (3, 9), device="cuda")
    prefix, true = [2, 1, 4], [9, 3, 8]
    want = continuation_scores(logits, ids, prefix, true)
    for p in (prefix, torch.tensor(prefix), torch.tensor(prefix, device="cuda"), torch.tensor(prefix, dtype=torch.int32)):
        for t in (true, torch.tensor(true, device="cuda")):
            assert torch.equal(continuation_scores(logits, ids, p, t), want)
    with pytest.raises(RuntimeError):                           # ids that lie elsewhere than the logits are refused, as by torch's ops
        continuation_scores(logits, ids.cpu(), prefix, true)


# one 16-byte unit, fewer units than pieces, units that do not divide into pieces, the training vocabulary, both sides of the shared-memory limit
@pytest.mark.parametrize("vocab", [8, 24, 40, 4104, 50304, 56960, 56968, 50301])
@pytest.mark.parametrize("write_grad", [True, False])
def test_loss_and_gradient_in_place(vocab, write_grad):
    torch.manual_seed(3)
    pitch = (vocab + 15) // 8 * 8
    store = torch.randn(9, pitch, device="cuda").mul_(4).bfloat16()
    logits = store[:, :vocab]
    logits[1, 0] = float("-inf")
    logits[2, vocab - 1] = 90.0
    targets = torch.randint(0, vocab, (9,), device="cuda")
    targets[1], targets[3], targets[4] = vocab - 1, 0, -100
    before, tail = logits.clone(), store[:, vocab:].clone()
    scale = torch.tensor([0.25], device="cuda")
    loss = cuda_ops.ext().ce_fwd_bwd(logits, targets, scale, -100, write_grad)
    exact = before.double()
    want = torch.nn.functional.cross_entropy(exact, targets, ignore_index=-100, reduction="none")
    assert torch.allclose(loss.double(), want, rtol=1e-5, atol=1e-5)
    if write_grad:
        grad = torch.softmax(exact, dim=-1)
        keep = targets != -100
        grad[keep, targets[keep]] -= 1.0
        grad[~keep] = 0.0
        assert torch.allclose(logits.double(), grad * 0.25, rtol=2 ** -8, atol=1e-7)       # one rounding to bf16
    else:
        assert torch.equal(logits, before)
    assert torch.equal(store[:, vocab:], tail)
    cuda_ops.check_status()
