"""Branches of the kernel dispatch at the sizes where they begin, end or leave a remainder, against plain PyTorch in fp32 / fp64."""
import math
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch

from llmq_b200.ops import kernels as K
from llmq_b200.ops import lib as L

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16
F8 = torch.float8_e4m3fn


@pytest.fixture(autouse=True)
def _check_status():
    yield
    torch.cuda.synchronize()
    K.check_status(torch.device(DEV, 0))


def rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return ((a - b).norm() / b.norm().clamp_min(1e-30)).item()


# dQ with one head per CTA (few items), parts of a group, whole groups (many items); one query tile without a second
@pytest.mark.parametrize("HS", [64, 128])
@pytest.mark.parametrize("B,T,Hq,Hkv", [(1, 1, 2, 1), (1, 63, 3, 1), (2, 64, 4, 2), (1, 65, 14, 2), (1, 128, 7, 1), (3, 129, 5, 1), (1, 257, 8, 1),
                                        (1, 300, 16, 1), (2, 384, 6, 3), (1, 1000, 4, 4), (24, 130, 14, 7), (8, 1200, 12, 6)])
def test_attention_head_splits(HS, B, T, Hq, Hkv):
    g = torch.Generator(device=DEV).manual_seed(T)
    qkv = torch.randn(B, T, Hq + 2 * Hkv, HS, device=DEV, generator=g).to(BF)
    dout = torch.randn(B, T, Hq, HS, device=DEV, generator=g).to(BF)
    out, lse = torch.full((B, T, Hq, HS), 9.0, device=DEV, dtype=BF), torch.empty(B, Hq, T, device=DEV)
    dqkv, scratch = torch.full_like(qkv, 9.0), torch.empty(B * Hq * T, device=DEV)
    K.attention_forward(out, lse, qkv, Hq, Hkv)
    K.attention_backward(dqkv, scratch, dout, out, lse, qkv, Hq, Hkv)
    again = torch.empty_like(dqkv)
    K.attention_backward(again, scratch, dout, out, lse, qkv, Hq, Hkv)
    assert torch.equal(dqkv, again)                       # no order depends on the schedule
    x = qkv.float().requires_grad_(True)
    o, l = K._attention_ref(x, Hq, Hkv)
    o.backward(dout.float())
    # 16-bit probabilities and score gradients (2^-9 each, random signs) and the 16-bit outputs
    assert rel(out, o.detach()) < 1e-2 and (lse - l.detach()).abs().max() < 2e-3
    if T > 1:
        assert rel(dqkv[:, :, :Hq], x.grad[:, :, :Hq]) < 1.2e-2
        assert rel(dqkv[:, :, Hq:Hq + Hkv], x.grad[:, :, Hq:Hq + Hkv]) < 1.2e-2
    assert rel(dqkv[:, :, Hq + Hkv:], x.grad[:, :, Hq + Hkv:]) < 1.2e-2


# Forward, many items per CTA: even and odd numbers of items with both query tiles (their extra key tile alternates between the pipelines), items without a second tile before them, an
# output that is aligned to 16 bytes only
@pytest.mark.parametrize("HS", [64, 128])
@pytest.mark.parametrize("B,T,Hq,Hkv", [(3, 256, 50, 10), (12, 256, 50, 10), (3, 300, 60, 30), (5, 513, 32, 8), (6, 640, 40, 8)])
def test_attention_forward_items(HS, B, T, Hq, Hkv):
    g = torch.Generator(device=DEV).manual_seed(T)
    qkv = torch.randn(B, T, Hq + 2 * Hkv, HS, device=DEV, generator=g).to(BF)
    out, lse, absmax = torch.full((B, T, Hq, HS), 9.0, device=DEV, dtype=BF), torch.empty(B, Hq, T, device=DEV), torch.zeros(1, device=DEV)
    K.attention_forward(out, lse, qkv, Hq, Hkv, absmax=absmax)
    shifted, lse2 = torch.full((out.numel() + 8,), 9.0, device=DEV, dtype=BF)[8:].view_as(out), torch.empty_like(lse)
    assert shifted.data_ptr() % 32 == 16
    K.attention_forward(shifted, lse2, qkv, Hq, Hkv)
    assert torch.equal(out, shifted) and torch.equal(lse, lse2) and absmax.item() == out.float().abs().max().item()
    for b in range(B):
        o, l = K._attention_ref(qkv[b:b + 1].float(), Hq, Hkv)
        # 16-bit probabilities (2^-9 each, random signs) and the 16-bit output
        assert rel(out[b:b + 1], o) < 1e-2 and (lse[b:b + 1] - l).abs().max() < 2e-3


# A gradient that is aligned to 16 bytes only, without and with dK / dV parts
@pytest.mark.parametrize("HS", [64, 128])
@pytest.mark.parametrize("B,T,Hq,Hkv", [(2, 100, 6, 2), (1, 300, 8, 1)])
def test_attention_backward_alignment(HS, B, T, Hq, Hkv):
    g = torch.Generator(device=DEV).manual_seed(T)
    qkv = torch.randn(B, T, Hq + 2 * Hkv, HS, device=DEV, generator=g).to(BF)
    dout, out = torch.randn(B, T, Hq, HS, device=DEV, generator=g).to(BF), torch.empty(B, T, Hq, HS, device=DEV, dtype=BF)
    lse, scratch = torch.empty(B, Hq, T, device=DEV), torch.empty(B * Hq * T, device=DEV)
    K.attention_forward(out, lse, qkv, Hq, Hkv)
    dqkv, shifted = torch.full_like(qkv, 9.0), torch.full((qkv.numel() + 8,), 9.0, device=DEV, dtype=BF)[8:].view_as(qkv)
    assert dqkv.data_ptr() % 32 == 0 and shifted.data_ptr() % 32 == 16
    for d in (dqkv, shifted):
        K.attention_backward(d, scratch, dout, out, lse, qkv, Hq, Hkv)
    assert torch.equal(dqkv, shifted)


# dK / dV of head size 128: CTAs per item on both sides of the steps of the rule (one CTA, clusters of two to eight, odd shares of the heads)
@pytest.mark.parametrize("T", [70, 200])
@pytest.mark.parametrize("Hq,Hkv", [(6, 1), (10, 2), (9, 1)])
def test_attention_backward_shared_heads(T, Hq, Hkv):
    per = (T + 127) // 128 * Hkv                          # items per sequence
    counts = [n // per for n in (296, 148, 98, 74, 59, 49, 37, 6)]
    g = torch.Generator(device=DEV).manual_seed(T)
    most = counts[0]
    qkv = torch.randn(most, T, Hq + 2 * Hkv, 128, device=DEV, generator=g).to(BF)
    dout = torch.randn(most, T, Hq, 128, device=DEV, generator=g).to(BF)
    want = None
    for B in counts:
        out, lse, dqkv = torch.empty(B, T, Hq, 128, device=DEV, dtype=BF), torch.empty(B, Hq, T, device=DEV), torch.full_like(qkv[:B], 9.0)
        K.attention_forward(out, lse, qkv[:B], Hq, Hkv)
        K.attention_backward(dqkv, torch.empty(B * Hq * T, device=DEV), dout[:B], out, lse, qkv[:B], Hq, Hkv)
        if want is None:
            want = dqkv
        assert torch.equal(dqkv[:, :, :Hq], want[:B, :, :Hq])            # dQ has one order
        # the same products summed in another order in fp32, then one rounding to bf16: neighbours at most, where the sum does not cancel
        d = (dqkv.float() - want[:B].float()).abs()
        assert (d <= want[:B].float().abs() * 2**-7 + 1e-4 * want.float().abs().max()).all()


# the CTAs that share the heads of an item: short walks and many items alone, every size of a cluster; each against the same sequences in a batch
# whose items are walked by one CTA
@pytest.mark.parametrize("T,B,Hq,Hkv,parts", [(16, 9, 28, 4, 1), (64, 2, 40, 8, 1), (128, 16, 28, 4, 2), (70, 1, 6, 1, 3), (70, 1, 7, 1, 4), (70, 1, 9, 1, 5),
                                              (200, 1, 6, 1, 6), (130, 1, 7, 1, 7), (130, 1, 8, 1, 8), (1000, 12, 8, 1, 2)])
def test_attention_backward_parts_of_an_item(T, B, Hq, Hkv, parts):
    lib, most = L.kernels(), 300 // ((T + 127) // 128 * Hkv)
    assert torch.cuda.get_device_properties(0).multi_processor_count != 148 or lib.llmq_attention_dkdv_parts(B, T, Hq, Hkv, 128) == parts
    assert lib.llmq_attention_dkdv_parts(most, T, Hq, Hkv, 128) == 1 and lib.llmq_attention_dkdv_parts(B, T, Hq, Hkv, 64) == 1
    g = torch.Generator(device=DEV).manual_seed(T)
    qkv = torch.randn(most, T, Hq + 2 * Hkv, 128, device=DEV, generator=g).to(BF)
    dout = torch.randn(most, T, Hq, 128, device=DEV, generator=g).to(BF)
    got = []
    for n in (B, most):
        out, lse, dqkv = torch.empty(n, T, Hq, 128, device=DEV, dtype=BF), torch.empty(n, Hq, T, device=DEV), torch.full_like(qkv[:n], 9.0)
        K.attention_forward(out, lse, qkv[:n], Hq, Hkv)
        K.attention_backward(dqkv, torch.empty(n * Hq * T, device=DEV), dout[:n], out, lse, qkv[:n], Hq, Hkv)
        got.append(dqkv[:B].float())
    # one CTA: the same bits; a cluster: fp32 sums in another order, then one rounding to bf16
    d = (got[0] - got[1]).abs()
    assert torch.equal(got[0], got[1]) if parts == 1 else (d <= got[1].abs() * 2**-7 + 1e-4 * got[1].abs().max()).all()


# dK / dV and dQ CTAs in one grid: the last cluster filled up with blocks that have nothing to do (dQ CTAs that are no multiple of the cluster size),
# one and two key blocks on both sides of the rule, groups that the dQ CTAs cut unevenly; each against the walk of a batch that has no clusters
@pytest.mark.parametrize("HS", [64, 128])
@pytest.mark.parametrize("B,T,Hq,Hkv", [(1, 70, 9, 1), (1, 128, 28, 4), (1, 129, 28, 4), (1, 333, 12, 2), (3, 257, 5, 1), (2, 683, 28, 4), (1, 1024, 32, 8), (9, 100, 32, 8)])
def test_attention_backward_one_grid(HS, B, T, Hq, Hkv):
    most = max(B, 300 // ((T + 127) // 128 * Hkv) + 1)
    assert L.kernels().llmq_attention_dkdv_parts(most, T, Hq, Hkv, HS) == 1
    g = torch.Generator(device=DEV).manual_seed(T)
    qkv = torch.randn(most, T, Hq + 2 * Hkv, HS, device=DEV, generator=g).to(BF)
    dout = torch.randn(most, T, Hq, HS, device=DEV, generator=g).to(BF)
    got = []
    for n in (B, most):
        out, lse, dqkv = torch.empty(n, T, Hq, HS, device=DEV, dtype=BF), torch.empty(n, Hq, T, device=DEV), torch.full_like(qkv[:n], 9.0)
        K.attention_forward(out, lse, qkv[:n], Hq, Hkv)
        K.attention_backward(dqkv, torch.empty(n * Hq * T, device=DEV), dout[:n], out, lse, qkv[:n], Hq, Hkv)
        got.append(dqkv[:B].float())
    assert torch.equal(got[0][:, :, :Hq], got[1][:, :, :Hq])             # dQ has one order
    # head size 64: one order; 128: fp32 sums of a cluster in another order, then one rounding to bf16
    d = (got[0] - got[1]).abs()
    assert torch.equal(got[0], got[1]) if HS == 64 else (d <= got[1].abs() * 2**-7 + 1e-4 * got[1].abs().max()).all()
    x = qkv[:B].float().requires_grad_(True)
    o, _ = K._attention_ref(x, Hq, Hkv)
    o.backward(dout[:B].float())
    assert rel(got[0], x.grad) < 1.2e-2                                  # 16-bit probabilities and score gradients, 16-bit outputs


# sequences of one query tile: a head per CTA and, with more heads than SMs, two heads of a group (the last one of an odd group alone)
@pytest.mark.parametrize("HS", [64, 128])
@pytest.mark.parametrize("T", [1, 33, 64, 65, 127, 128])
@pytest.mark.parametrize("Hq,Hkv", [(14, 2), (8, 4), (5, 1), (4, 4)])
def test_attention_of_short_sequences(HS, T, Hq, Hkv):
    few, many = 148 // Hq, 420 // Hq
    g = torch.Generator(device=DEV).manual_seed(T)
    qkv = torch.randn(many, T, Hq + 2 * Hkv, HS, device=DEV, generator=g).to(BF)
    got = []
    for B in (few, many):
        out, lse, am = torch.full((B, T, Hq, HS), 9.0, device=DEV, dtype=BF), torch.full((B, Hq, T), 9.0, device=DEV), torch.zeros(1, device=DEV)
        K.attention_forward(out, lse, qkv[:B], Hq, Hkv, absmax=am)
        assert am.item() == out.float().abs().max().item()
        got.append((out, lse))
    assert torch.equal(got[0][0], got[1][0][:few]) and torch.equal(got[0][1], got[1][1][:few])
    o, l = K._attention_ref(qkv.float(), Hq, Hkv)
    assert rel(got[1][0], o) < 1e-2 and (got[1][1] - l).abs().max() < 2e-3


@pytest.mark.parametrize("HS", [64, 128])
def test_attention_with_growing_row_maxima(HS):
    """Scores whose row maximum grows by more than 2^8 after the first key tiles, in some rows of a warp and not in others: the
    output accumulator and the row sum are rescaled on the way."""
    B, T, Hq, Hkv = 2, 700, 4, 2
    g = torch.Generator(device=DEV).manual_seed(HS)
    qkv = torch.randn(B, T, Hq + 2 * Hkv, HS, device=DEV, generator=g)
    t = torch.arange(T, device=DEV)
    qkv[:, :, Hq:Hq + Hkv] *= (1 + t / 48)[None, :, None, None]
    qkv[:, ::3, :Hq] *= 0.05
    qkv = qkv.to(BF)
    dout = torch.randn(B, T, Hq, HS, device=DEV, generator=g).to(BF)
    q, k = qkv[:, :, :Hq].float().transpose(1, 2), qkv[:, :, Hq:Hq + Hkv].float().transpose(1, 2).repeat_interleave(Hq // Hkv, 1)
    s = (q @ k.transpose(-1, -2) * (math.log2(math.e) / math.sqrt(HS))).masked_fill(t[:, None] < t, -math.inf)
    first64, first = s[..., :64].amax(-1), s[..., :128].amax(-1)
    grows = s.amax(-1) - first > 8
    assert (first - first64 > 8).any() and grows.any() and (~grows[..., 256:]).any()       # each way of choosing the reference
    out, lse = torch.full((B, T, Hq, HS), 9.0, device=DEV, dtype=BF), torch.empty(B, Hq, T, device=DEV)
    dqkv, scratch = torch.full_like(qkv, 9.0), torch.empty(B * Hq * T, device=DEV)
    K.attention_forward(out, lse, qkv, Hq, Hkv)
    K.attention_backward(dqkv, scratch, dout, out, lse, qkv, Hq, Hkv)
    x = qkv.float().requires_grad_(True)
    o, l = K._attention_ref(x, Hq, Hkv)
    o.backward(dout.float())
    # as above; fp32 scores of up to 200 carry 2^-17 of absolute error into lse
    assert rel(out, o.detach()) < 1e-2 and (lse - l.detach()).abs().max() < 2e-3
    for part in (slice(0, Hq), slice(Hq, Hq + Hkv), slice(Hq + Hkv, None)):
        assert rel(dqkv[:, :, part], x.grad[:, :, part]) < 1.2e-2


# less than a vector per thread of the cluster's two CTAs, whole rounds of four vectors a thread (32768) and not, tails behind the
# last whole vector
@pytest.mark.parametrize("V", [3, 8, 13, 4096, 4103, 4104, 8192, 8200, 32768, 32776, 40967, 128256, 151936, 163847, 200000])
@pytest.mark.parametrize("z_reg", [0.0, 1e-3])
def test_fused_classifier_row_splits(V, z_reg):
    rows, ld = 5, (V + 7) // 8 * 8
    g = torch.Generator().manual_seed(V)
    buf = torch.randn(rows, ld, generator=g).mul_(3).to(BF)
    buf[3, 1:V] = -math.inf                               # one finite logit
    buf[2, : V // 2] = torch.finfo(BF).min                # masked by the type's lowest value
    guarded = torch.full((rows + 2, ld), 7.0, device=DEV, dtype=BF)
    guarded[1:-1] = buf.to(DEV)
    logits = guarded[1:-1, :V]
    tg = torch.tensor([V - 1, -100, V // 2, 0, (V - 1) // 8 * 8], dtype=torch.int32)
    losses, lse = torch.full((rows,), 0.5, device=DEV), torch.empty(rows, device=DEV)
    K.fused_classifier(logits, losses, lse, tg.to(DEV), 0.25, z_reg * 0.25, True)
    x = buf[:, :V].double()
    ok, safe = tg >= 0, tg.clamp_min(0).long()
    l = torch.logsumexp(x, -1)
    want_loss = 0.5 + torch.where(ok, l - x[torch.arange(rows), safe], torch.zeros_like(l))
    p = torch.exp(x - l[:, None]) * (0.25 * (1 + z_reg * l))[:, None]
    p[torch.arange(rows), safe] -= 0.25
    p[~ok] = 0
    assert (losses.cpu().double() - want_loss).abs().max() < 2e-5 * (1 + want_loss.abs().max())
    assert (lse.cpu().double() - torch.where(ok, l, torch.zeros_like(l))).abs().max() < 2e-5 * (1 + l[ok].abs().max())
    # one bf16 rounding (2^-9 of the value); the target's entry keeps the fp32 error of p next to its -0.25
    assert ((logits.cpu().double() - p).abs() <= p.abs() * 2 ** -8 + 1e-6).all()
    # nothing behind the vocabulary, before the first row or after the last one was touched
    assert torch.equal(guarded[1:-1, V:].cpu(), buf[:, V:]) and bool((guarded[[0, -1]] == 7.0).all())


@pytest.mark.parametrize("dtype", [BF, torch.float32])
def test_fused_classifier_keeps_subnormal_gradients(dtype):
    """Probabilities below 2^-126 are subnormal numbers in the gradient, not zero: whole vectors of them, single ones and the tail."""
    V = 4101
    x = torch.zeros(2, 4104)
    x[0, 1:] = -torch.linspace(80.0, 95.0, 4103)              # dloss * p: 2^-117 to 2^-139, the smallest bf16 is 2^-133
    x[1, 9::16] = -87.0
    x[1, V - 1] = -86.0
    x = x.to(dtype)
    logits = x.to(DEV)[:, :V]
    losses, lse = torch.zeros(2, device=DEV), torch.zeros(2, device=DEV)
    K.fused_classifier(logits, losses, lse, torch.zeros(2, dtype=torch.int32, device=DEV), 0.25)
    p = torch.softmax(x[:, :V].double(), -1) * 0.25
    p[:, 0] -= 0.25
    got = logits.cpu().double()
    assert ((got[:, 1:] != 0) & (got[:, 1:].abs() < 2.0 ** -126)).sum() > 1000
    # a rounding of the storage type, or half of its smallest step; fp32 exponents near -128 carry 2^-17 of the value
    half_step = 2.0 ** (-134 if dtype == BF else -150)
    assert ((got - p).abs() <= p.abs() * (2 ** -8 if dtype == BF else 2 ** -15) + 1.01 * half_step)[:, 1:].all()


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("rows", [2, 200])
def test_fused_classifier_with_masked_columns_in_front(dtype, rows):
    """-inf up to a finite logit that the same thread meets later, and in the tail: probability 0, not NaN."""
    V = 16389
    x = torch.randn(rows, V).mul_(3)
    x[:, :9000] = -math.inf
    x[1, V - 3:] = -math.inf
    x = x.to(dtype)
    buf = torch.zeros(rows, 16392, dtype=dtype, device=DEV)
    buf[:, :V] = x.to(DEV)
    logits, losses, lse = buf[:, :V], torch.zeros(rows, device=DEV), torch.zeros(rows, device=DEV)
    tg = torch.full((rows,), 12000, dtype=torch.int32)
    K.fused_classifier(logits, losses, lse, tg.to(DEV), 0.5)
    l = torch.logsumexp(x.double(), -1)
    p = torch.exp(x.double() - l[:, None]) * 0.5
    p[:, 12000] -= 0.5
    assert (lse.cpu().double() - l).abs().max() < 1e-4 and (losses.cpu().double() - (l - x[:, 12000].double())).abs().max() < 1e-4
    assert ((logits.cpu().double() - p).abs() <= p.abs() * (2 ** -8 if dtype == BF else 1e-5) + 1e-6).all()


def test_fused_classifier_takes_more_rows_than_a_grid_has_pairs_of_blocks():
    rows, V = 2 ** 30 + 5, 8
    if torch.cuda.mem_get_info()[0] < 40e9:
        pytest.skip("needs 26 GB of device memory")
    logits = torch.zeros(rows, V, device=DEV, dtype=BF)
    targets = torch.full((rows,), -100, device=DEV, dtype=torch.int32)
    at = torch.tensor([0, 5, 6, 2 ** 30 - 1, 2 ** 30, rows - 1], device=DEV)      # the first launch takes the rows from 6 on
    targets[at] = 3
    losses = torch.zeros(rows, device=DEV)
    K.fused_classifier(logits, losses, None, targets, 1.0)
    assert (losses[at] - math.log(8)).abs().max() < 1e-6 and int((losses != 0).sum()) == len(at)
    want = torch.full((len(at), V), 0.125, device=DEV, dtype=BF)
    want[:, 3] = -0.875
    assert torch.equal(logits[at], want) and int((logits[:, 0] != 0).sum()) == len(at)
    del logits, targets, losses
    torch.cuda.empty_cache()


@pytest.mark.parametrize("dtype", [BF, torch.float32])
def test_fused_classifier_rows_without_a_finite_maximum(dtype):
    V = 30000
    x = torch.full((4, V), -math.inf)
    x[1, 7] = math.inf
    x[2] = 0.0
    x[2, 5] = math.nan
    x[3] = torch.finfo(dtype).min
    losses, lse = torch.zeros(4, device=DEV), torch.zeros(4, device=DEV)
    K.fused_classifier(x.to(dtype).to(DEV), losses, lse, torch.tensor([1, 2, 3, 4], dtype=torch.int32, device=DEV), 1.0)
    assert lse[3].item() == torch.finfo(dtype).min
    assert lse[0].item() == -math.inf and math.isnan(lse[1].item()) and math.isnan(lse[2].item())


# forward: rows of 1 .. 8 vectors per thread with 64 and with 256 threads, the two-pass kernel beyond; backward: 1, 2, 4 and 8 vectors
@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("C", [8, 264, 512, 896, 2056, 3584, 4096, 4104, 8192, 8200, 16384])
@pytest.mark.parametrize("rows", [1, 37, 700])
def test_rmsnorm_row_splits(dtype, C, rows):
    if dtype == torch.float32 and C > 8192:
        pytest.skip("longer than the backward kernel takes")
    g = torch.Generator().manual_seed(C + rows)
    r = lambda *s: torch.randn(*s, generator=g).to(dtype)
    x, y, w, dy, dres, dw0 = r(rows, C), r(rows, C), r(C), r(rows, C), r(rows, C), r(C)
    res, out, rstd = torch.empty(rows, C, dtype=dtype, device=DEV), torch.empty(rows, C, dtype=dtype, device=DEV), torch.empty(rows, device=DEV)
    am, amb = torch.zeros(1, device=DEV), torch.zeros(1, device=DEV)
    K.rmsnorm_forward(out, rstd, x.to(DEV), w.to(DEV), 1e-6, residual_out=res, inp2=y.to(DEV), absmax=am)
    s = (x.float() + y.float()).to(dtype)
    assert torch.equal(res.cpu(), s)
    rs = torch.rsqrt(s.double().square().mean(-1, keepdim=True) + 1e-6)
    want = s.double() * rs * w.double()
    eps = 2 ** -8 if dtype == BF else 2 ** -22            # half a unit of the last place of the storage type; fp32: a few ulp
    assert ((out.cpu().double() - want).abs() <= 2.1 * eps * want.abs() + 1e-30).all()        # x * rstd and its product with w are rounded
    assert am.item() == out.float().abs().max().item()
    assert (rstd.cpu().double() / rs[:, 0] - 1).abs().max() < 1e-6
    plain = torch.empty_like(out)
    K.rmsnorm_forward(plain, None, res, w.to(DEV), 1e-6)
    assert torch.equal(plain, out)
    dinp, dw = dres.to(DEV), dw0.to(DEV)
    scratch = torch.full((K.rmsnorm_backward_scratch_elems(C, DEV),), math.nan, device=DEV)
    K.rmsnorm_backward(dinp, dw, scratch, dy.to(DEV), res, w.to(DEV), rstd, absmax=amb)
    xh, wdy = s.double() * rs, w.double() * dy.double()
    gx = dres.double() + (wdy - xh * (wdy * xh).mean(-1, keepdim=True)) * rs
    gw = dw0.double() + (dy.double() * xh).sum(0)
    assert rel(dinp, gx) < eps and rel(dw, gw) < eps
    assert amb.item() == dinp.float().abs().max().item()


@pytest.mark.parametrize("N", [300, 301, 896])            # whole vectors of four columns, and not
@pytest.mark.parametrize("out_dt", [BF, torch.float32])
def test_split_k_reduce(N, out_dt):
    g = torch.Generator().manual_seed(N)
    M, Kd = 200, 4096
    a, b, bias = torch.randn(M, Kd, generator=g).to(BF), torch.randn(N, Kd, generator=g).to(BF), torch.randn(N, generator=g).to(BF)
    prev = torch.randn(M, N, generator=g).to(out_dt)
    out, am = prev.to(DEV), torch.zeros(1, device=DEV)
    K.gemm(out, a.to(DEV), b.to(DEV), bias=bias.to(DEV), accumulate=True, alpha=0.5, absmax=am)
    want = 0.5 * (a.double() @ b.double().t()) + bias.double() + prev.double()
    assert rel(out, want) < (2 ** -8 if out_dt == BF else 1e-5)
    assert abs(am.item() - want.abs().max().item()) < 1e-3 * want.abs().max().item()


def _through_the_second_kernel(M, N, Kd, out, a, b, **kw):
    """The same GEMM into a view that is not aligned to four columns, whose parts therefore go through the workspace."""
    view = torch.full((M + 1, N + 4), 9.0, device=DEV, dtype=out.dtype)[:M, 1:N + 1]
    view.copy_(out)
    assert L.calls().llmq_gemm_split_mode(view, M, N, Kd, a.element_size(), view.stride(0), int(out.dtype != BF), 148) == 2
    K.gemm(view, a, b, **kw)
    return view


# K cut into 2 to 8 parts that a cluster adds up, uneven shares of its rows (3, 5, 6, 7 parts), ragged last tiles, both tile widths; one tile more than clusters
# reside (36 of 4 parts, 28 of 5, 16 of 8) and N = 301 go through the second kernel
@pytest.mark.parametrize("M,N,Kd,parts", [(1001, 896, 1152, 2), (130, 8196, 2048, 2), (339, 3584, 3584, 3), (64, 2048, 1536, 3), (200, 2052, 2048, 4), (1152, 896, 2048, 4),
                                          (385, 1280, 3584, 7), (848, 896, 2560, 5), (385, 1024, 3072, 6), (97, 304, 4096, 8), (256, 2048, 4096, 8), (97, 301, 4096, 8)])
@pytest.mark.parametrize("dt,out_dt", [(BF, BF), (F8, BF), (BF, torch.float32), (torch.float32, torch.float32)])
def test_split_k_parts(M, N, Kd, parts, dt, out_dt):
    Kd *= {1: 2, 2: 1, 4: 1}[dt.itemsize]                    # as many K steps of 128 bytes (fp32: twice as many, so the same parts or more)
    floats = L.kernels().llmq_gemm_splitk_floats(M, N, Kd, dt.itemsize, 148)
    assert floats == parts * M * N or dt == torch.float32 and floats >= parts * M * N
    g = torch.Generator(device=DEV).manual_seed(M)
    a, b = torch.randn(M, Kd, device=DEV, generator=g).to(dt), torch.randn(N, Kd, device=DEV, generator=g).to(dt)
    bias, prev, scale = torch.randn(N, device=DEV, generator=g).to(BF), torch.randn(M, N, device=DEV, generator=g).to(out_dt), torch.full((1,), 0.5, device=DEV)
    rows = torch.full((M + 1, N), 9.0, device=DEV, dtype=out_dt)
    am = torch.zeros(1, device=DEV)
    plain, added = rows[:M], prev.clone()
    two = _through_the_second_kernel(M, N, Kd, plain, a, b), _through_the_second_kernel(M, N, Kd, prev, a, b, bias=bias, accumulate=True, scale_a=scale)
    K.gemm(plain, a, b)
    K.gemm(added, a, b, bias=bias, accumulate=True, scale_a=scale, absmax=am)
    K.check_status(torch.device(DEV, 0))
    assert torch.equal(plain, two[0]) and torch.equal(added, two[1])             # the parts are added up in one order
    prod = a.double() @ b.double().t()
    want = 0.5 * prod + bias.double() + prev.double()
    # fp32 sums; products of fp32 operands have 10-bit mantissas (tf32 truncates: 2^-10 an operand); one rounding to bf16 of the outputs
    eps = 2e-3 if dt == torch.float32 else 1e-5
    eps += 2 ** -8 if out_dt == BF else 0
    assert rel(plain, prod) < eps and rel(added, want) < eps
    assert (rows[M] == 9).all()
    assert abs(am.item() - want.abs().max().item()) < 4e-3 * want.abs().max().item()


# split K of outputs that fill their tiles partly: fewer rows than parts, rows and columns around the shares of a cluster's CTAs, 8 to 64 pieces of four columns
@pytest.mark.parametrize("M,N", [(1, 16), (5, 264), (16, 32), (31, 40), (130, 72), (208, 136), (257, 304)])
@pytest.mark.parametrize("Kd", [1216, 4096])
@pytest.mark.parametrize("out_dt", [BF, torch.float32])
def test_split_k_narrow(M, N, Kd, out_dt):
    assert L.kernels().llmq_gemm_splitk_floats(M, N, Kd, 2, 148) > 0
    g = torch.Generator(device=DEV).manual_seed(M)
    a, b = torch.randn(M, Kd, device=DEV, generator=g).to(BF), torch.randn(N, Kd, device=DEV, generator=g).to(BF)
    rows = torch.full((M + 1, N), 9.0, device=DEV, dtype=out_dt)
    prev = torch.randn(M, N, device=DEV, generator=g).to(out_dt)
    added = prev.clone()
    two = _through_the_second_kernel(M, N, Kd, prev, a, b), _through_the_second_kernel(M, N, Kd, prev, a, b, accumulate=True)
    K.gemm(rows[:M], a, b)
    K.gemm(added, a, b, accumulate=True)
    K.check_status(torch.device(DEV, 0))
    assert torch.equal(rows[:M], two[0]) and torch.equal(added, two[1])
    prod = a.double() @ b.double().t()
    eps = 1e-5 + (2 ** -8 if out_dt == BF else 0)             # fp32 sums, one rounding of the outputs
    assert rel(rows[:M], prod) < eps and rel(added, prod + prev.double()) < eps
    assert (rows[M] == 9).all()


# the kernel for a plain GEMM on both sides of each line of the rule for rows that start with a 128-byte line: short K (8 and 9 steps of 128 bytes), one round of tiles (64 / 65 steps, both
# operands MN-major 16 / 17), more than half of the SMs idle (47 / 48 steps, from where K is cut in two); odd edges of the last tiles
@pytest.mark.parametrize("M,N,steps,mn,ctas,parts", [(9728, 912, 8, 0, 1, 1), (9728, 912, 9, 0, 2, 1), (2320, 1168, 64, 0, 1, 1), (2320, 1168, 65, 0, 2, 1), (2040, 2064, 16, 1, 1, 1),
                                                     (2040, 2064, 17, 1, 2, 1), (1064, 2032, 47, 0, 2, 1), (1064, 2032, 48, 0, 1, 2)])
@pytest.mark.parametrize("dt", [BF, F8])
def test_gemm_kernel_choice(M, N, steps, mn, ctas, parts, dt):
    lib, step = L.kernels(), 128 // dt.itemsize
    Kd = steps * step - 8 * (2 // dt.itemsize)                # the last step is not whole
    if mn and dt == F8:
        M, N = M // 16 * 16, N // 16 * 16
    assert lib.llmq_gemm_splitk_floats(M, N, Kd, dt.itemsize, 148) == (parts * M * N if parts > 1 else 0)
    assert lib.llmq_gemm_tile_ctas(M, N, Kd, dt.itemsize, mn, 128, 0, 1, 148) == ctas
    g = torch.Generator(device=DEV).manual_seed(M + steps)
    shapes = [(Kd, r) if mn else (r, Kd) for r in (M, N)]
    a, b = (torch.randn(rows, -(-cols // 128) * 128, device=DEV, generator=g).to(dt)[:, :cols] for rows, cols in shapes)
    got = []
    try:
        for mode in (0, 1, 2):
            lib.llmq_gemm_set_mode(mode)
            out = torch.full((M, N), 9.0, device=DEV, dtype=BF)
            cut = lib.llmq_gemm_splitk_floats(M, N, Kd, dt.itemsize, 148) > 0
            K.gemm(out, a, b, a_mn=bool(mn), b_mn=bool(mn))
            got.append((out, cut))
    finally:
        lib.llmq_gemm_set_mode(0)
    ad, bd = (x.double().t() if mn else x.double() for x in (a, b))
    assert rel(got[0][0], ad @ bd.t()) < 2**-8                # fp32 sums, one rounding to bf16
    assert all(torch.equal(got[0][0], out) for out, cut in got if cut == (parts > 1))            # one order of the sum over K, cut or not


# bf16 outputs that are added to: up to 32 columns, blocks of 64 columns and remainders of 16, 32 and 48, ragged rows, tiles of 224 and 256 columns, several tiles per CTA in both kernels
@pytest.mark.parametrize("M,N,Kd", [(130, 16, 64), (300, 32, 192), (20000, 32, 64), (300, 48, 64), (130, 336, 64), (1000, 1008, 128), (300, 65, 64), (4100, 912, 640), (4096, 896, 1280), (9000, 2096, 192), (9000, 2096, 1216)])
@pytest.mark.parametrize("dt", [BF, F8])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_gemm_added_to(M, N, Kd, dt, mode):
    g = torch.Generator(device=DEV).manual_seed(N)
    a, b = torch.randn(M, Kd, device=DEV, generator=g).to(dt), torch.randn(N, Kd, device=DEV, generator=g).to(dt)
    bias, scale = torch.randn(N, device=DEV, generator=g).to(BF), torch.full((1,), 0.5, device=DEV)
    whole = torch.randn(M + 1, N, device=DEV, generator=g).to(BF)
    before = whole.clone()
    out, am = whole[:M], torch.zeros(1, device=DEV)
    try:
        L.kernels().llmq_gemm_set_mode(mode)
        K.gemm(out, a, b, bias=bias, accumulate=True, scale_a=scale, absmax=am)
    finally:
        L.kernels().llmq_gemm_set_mode(0)
    want = 0.5 * (a.double() @ b.double().t()) + bias.double() + before[:M].double()
    # one rounding to bf16 and fp32 sums of Kd products of a few units
    assert ((out.double() - want).abs() <= want.abs() * 2**-8 + 1e-4 * Kd**0.5).all()
    assert torch.equal(whole[M], before[M])
    assert abs(am.item() - want.abs().max().item()) < 1e-4 * want.abs().max().item()


def _split_k_operands(n, seed, N):
    """n GEMMs of one shape (8 parts; 2 MB of partial sums each where N is no multiple of 4, clusters add them up where it is) and what each gives by itself."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    a, b = torch.randn(n, 200, 8192, device=DEV, generator=g).to(BF), torch.randn(n, N, 8192, device=DEV, generator=g).to(BF)
    want = torch.empty(n, 200, N, device=DEV)
    assert L.calls().llmq_gemm_split_mode(want[0], 200, N, 8192, 2, N, 1, 148) == (2 if N % 4 else 1)
    for i in range(n):
        K.gemm(want[i], a[i], b[i])
        torch.cuda.synchronize()
    assert rel(want, a.double() @ b.double().transpose(1, 2)) < 1e-5
    return a, b, want


@pytest.mark.parametrize("how", ["streams", "threads", "graphs"])
@pytest.mark.parametrize("N", [301, 304])
def test_split_k_on_several_streams(how, N):
    """GEMMs that cut K, side by side on four streams (of one thread, of four threads, of four captured graphs): the partial sums of
    one are never those of another."""
    n, lanes = 16, 4
    a, b, want = _split_k_operands(n, 3, N)
    out, streams = torch.zeros_like(want), [torch.cuda.Stream() for _ in range(lanes)]
    torch.cuda.synchronize()

    def lane(j):
        with torch.cuda.stream(streams[j]):
            torch.zeros(1, device=DEV)                       # gives the thread a CUDA context
            for i in range(j, n, lanes):
                K.gemm(out[i], a[i], b[i])

    for _ in range(3):
        out.zero_()
        torch.cuda.synchronize()
        if how == "threads":
            with ThreadPoolExecutor(lanes) as pool:
                list(pool.map(lane, range(lanes)))
        elif how == "streams":
            for i in range(n):
                with torch.cuda.stream(streams[i % lanes]):
                    K.gemm(out[i], a[i], b[i])
        else:
            graphs = [torch.cuda.CUDAGraph() for _ in range(lanes)]
            for j, graph in enumerate(graphs):
                with torch.cuda.graph(graph):                # all captured on the same stream
                    for i in range(j, n, lanes):
                        K.gemm(out[i], a[i], b[i])
            for j, graph in enumerate(graphs):
                with torch.cuda.stream(streams[j]):
                    graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


def test_split_k_workspaces_kept_by_a_thread_are_bounded():
    a, b, want = _split_k_operands(2, 4, 301)
    out = torch.zeros_like(want)
    with ThreadPoolExecutor(1) as pool:
        def many():
            torch.zeros(1, device=DEV)
            for _ in range(2 * K.SPLITK_KEPT):
                with torch.cuda.stream(torch.cuda.Stream()):
                    K.gemm(out[0], a[0], b[0])
                    K.gemm(out[1, :100], a[1, :100], b[1])   # a smaller one takes the same
                torch.cuda.synchronize()
                assert torch.equal(out[0], want[0]) and torch.equal(out[1, :100], want[1, :100])
            return {k: v.numel() for k, v in K._thread.splitk.items()}
        kept = pool.submit(many).result()
    assert 1 <= len(kept) <= K.SPLITK_KEPT and set(kept.values()) == {8 * 200 * 301}


def test_split_k_added_up_by_clusters_takes_no_workspace():
    a, b, want = _split_k_operands(1, 5, 304)
    out, graph = torch.zeros_like(want), torch.cuda.CUDAGraph()
    with ThreadPoolExecutor(1) as pool:
        def one():
            torch.zeros(1, device=DEV)
            K.gemm(out[0], a[0], b[0])
            torch.cuda.synchronize()
            return dict(K._thread.__dict__.get("splitk", {}))
        assert pool.submit(one).result() == {} and torch.equal(out, want)
    with torch.cuda.graph(graph):
        K.gemm(out[0], a[0], b[0])
        used = torch.cuda.memory_allocated()
        K.gemm(out[0], a[0], b[0])
        assert torch.cuda.memory_allocated() == used
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


@pytest.mark.parametrize("op", ["gemm_fp32", "attention_fp32", "encoder_backward"])
def test_scratch_of_calls_on_several_streams(op):
    """Calls that need scratch for a conversion or a sort, of one shape and side by side, give what each gives by itself."""
    n, g = 8, torch.Generator(device=DEV).manual_seed(1)
    r = lambda *s: torch.randn(n, *s, device=DEV, generator=g)
    if op == "gemm_fp32":
        a, b = r(1024, 512), r(1024, 768)
        new, call = (lambda: torch.zeros(n, 512, 768, device=DEV)), (lambda o, i: K.gemm(o[i], a[i], b[i], a_mn=True, b_mn=True))
    elif op == "attention_fp32":
        qkv, dout = r(2, 256, 8, 64), r(2, 256, 4, 64)
        new = lambda: torch.zeros(n, 2, 256, 8, 64, device=DEV)

        def call(o, i):
            out, lse, scratch = torch.empty_like(dout[i]), torch.empty(2, 4, 256, device=DEV), torch.empty(2 * 4 * 256, device=DEV)
            K.attention_forward(out, lse, qkv[i], 4, 2)
            K.attention_backward(o[i], scratch, dout[i], out, lse, qkv[i], 4, 2)
    else:
        d, tokens = r(4096, 64).to(BF), torch.randint(0, 500, (n, 4096), device=DEV, generator=g, dtype=torch.int32)
        new, call = (lambda: torch.zeros(n, 500, 64, device=DEV, dtype=BF)), (lambda o, i: K.encoder_backward(o[i], d[i], tokens[i]))
    want, streams = new(), [torch.cuda.Stream() for _ in range(4)]
    for i in range(n):
        call(want, i)
        torch.cuda.synchronize()
    for _ in range(3):
        got = new()
        torch.cuda.synchronize()
        for i in range(n):
            with torch.cuda.stream(streams[i % 4]):
                call(got, i)
        torch.cuda.synchronize()
        assert torch.equal(got, want)


# short rows go to 256 threads up to 1184 rows (and from 1777 to 4096 with more than 448 vectors of 16 bytes), else to 64
@pytest.mark.parametrize("dtype,C,rows", [(BF, 896, 1184), (BF, 2048, 1184), (BF, 2056, 1184), (BF, 3072, 1184), (BF, 3584, 1184), (BF, 3592, 1776),
                                          (BF, 4096, 4096), (torch.float32, 448, 1184), (torch.float32, 1024, 1184), (torch.float32, 2048, 4096)])
def test_rmsnorm_of_few_and_many_rows_has_the_same_bits(dtype, C, rows):
    g = torch.Generator(device=DEV).manual_seed(C)
    x, y = (torch.randn(rows + 1, C, device=DEV, generator=g).to(dtype) for _ in range(2))
    w = torch.randn(C, device=DEV, generator=g).to(dtype)
    got = []
    for n in (rows, rows + 1):
        o, r, rs, am = torch.empty(n, C, dtype=dtype, device=DEV), torch.empty(n, C, dtype=dtype, device=DEV), torch.empty(n, device=DEV), torch.zeros(1, device=DEV)
        K.rmsnorm_forward(o, rs, x[:n], w, 1e-6, residual_out=r, inp2=y[:n], absmax=am)
        assert am.item() == o.float().abs().max().item()
        got.append((o[:rows], r[:rows], rs[:rows]))
    assert all(torch.equal(a, b) for a, b in zip(*got))
    s = (x.float() + y.float()).to(dtype)[:rows].double()
    rs = torch.rsqrt(s.square().mean(-1, keepdim=True) + 1e-6)
    eps = 2 ** -8 if dtype == BF else 2 ** -22
    assert ((got[0][0].double() - s * rs * w.double()).abs() <= 2.1 * eps * (s * rs * w.double()).abs() + 1e-30).all()


@pytest.mark.parametrize("n", [8, 8 * 512 * 512 - 8, 8 * 512 * 512 * 4 + 8, 12345679])
@pytest.mark.parametrize("dtype", [BF, torch.float32])
def test_norm_squared_sizes(n, dtype):
    x = torch.randn(n, device=DEV).to(dtype)
    part, out = torch.full((512,), 0.25, device=DEV), torch.empty(1, device=DEV)
    K.norm_squared(part, x)
    K.deterministic_sum(out, part)
    want = 128.0 + x.double().square().sum().item()
    assert abs(out.item() - want) < 1e-5 * want
    # block by block: thread t of block b adds up vectors b * 512 + t, + 512 * 512, ... (the tail belongs to block 0)
    width = 16 // x.element_size()
    vecs = x[: n // width * width].double().square().view(-1, width).sum(1)
    blocks = torch.zeros(512, dtype=torch.float64, device=DEV).index_add_(0, torch.arange(len(vecs), device=DEV) // 512 % 512, vecs)
    blocks[0] += x[n // width * width:].double().square().sum()
    assert ((part.double() - 0.25 - blocks).abs() <= 1e-5 * blocks + 1e-6).all()


def test_adamw_stores_non_finite_values_as_they_are():
    n = 256
    p, m, v = (torch.zeros(n, device=DEV, dtype=BF) for _ in range(3))
    g = torch.ones(n, device=DEV, dtype=BF)
    g[3], g[10], g[17] = math.inf, -math.inf, math.nan
    K.adamw(p, g, m, v, lr=0.1, beta1=0.9, beta2=0.95, step=1, eps=1e-8, weight_decay=0.0, seed=3)
    assert m[3].item() == math.inf and m[10].item() == -math.inf and math.isnan(m[17].item()) and math.isnan(p[17].item())
    assert v[3].item() == math.inf and v[10].item() == math.inf and math.isnan(v[17].item())
    ok = torch.ones(n, dtype=torch.bool, device=DEV)
    ok[[3, 10, 17]] = False
    assert (p[ok].float() + 0.1).abs().max() < 1e-3 and torch.isfinite(m[ok]).all()


# MN-major operands whose extent is whole 128-byte chunks (one 3-D load per stage), the last tile partly outside the matrix, and
# extents with a ragged last chunk (2-D boxes); one-CTA kernel and CTA pairs (from 2^21 outputs)
@pytest.mark.parametrize("M,N,Kd", [(320, 448, 200), (64, 192, 72), (128, 384, 65), (2112, 1088, 136), (2112, 1152, 264), (2080, 1040, 130)])
@pytest.mark.parametrize("dt", [BF, torch.float8_e4m3fn])
@pytest.mark.parametrize("a_mn,b_mn", [(1, 0), (0, 1), (1, 1)])
def test_gemm_mn_major_chunks(M, N, Kd, dt, a_mn, b_mn):
    if not (a_mn and b_mn):
        Kd = (Kd + 15) // 16 * 16                          # rows of a K-major operand start at multiples of 16 bytes
    g = torch.Generator().manual_seed(M + N)
    a, b = torch.randn(M, Kd, generator=g).to(dt), torch.randn(N, Kd, generator=g).to(dt)
    sa = a.float().t().contiguous().to(dt) if a_mn else a
    sb = b.float().t().contiguous().to(dt) if b_mn else b
    out = torch.full((M, N), 5.0, dtype=torch.float32, device=DEV)
    K.gemm(out, sa.to(DEV), sb.to(DEV), a_mn=bool(a_mn), b_mn=bool(b_mn))
    assert rel(out, a.double() @ b.double().t()) < 1e-5    # exact products, fp32 sums


# 128-column tiles with and without a split of K, shapes on both sides of the line to 256-column tiles (148 tiles of 128 columns)
@pytest.mark.parametrize("M,N,Kd", [(1, 8, 16), (129, 136, 320), (1001, 896, 1152), (896, 896, 4096), (1000, 2304, 208), (1152, 2048, 96), (9600, 256, 64),
                                    (9472, 256, 64), (640, 2048, 1024), (1152, 896, 4096)])
@pytest.mark.parametrize("dt", [BF, torch.float8_e4m3fn])
@pytest.mark.parametrize("accumulate", [False, True])
def test_gemm_tile_widths(M, N, Kd, dt, accumulate):
    g = torch.Generator().manual_seed(M + N + Kd)
    a, b = torch.randn(M, Kd, generator=g).to(dt), torch.randn(N, Kd, generator=g).to(dt)
    bias, prev = torch.randn(N, generator=g).to(BF), torch.randn(M, N, generator=g)
    out, am = prev.to(DEV), torch.zeros(1, device=DEV)
    K.gemm(out, a.to(DEV), b.to(DEV), bias=bias.to(DEV), accumulate=accumulate, absmax=am)
    want = a.double() @ b.double().t() + bias.double() + (prev.double() if accumulate else 0)
    assert rel(out, want) < 1e-5                           # exact products, fp32 sums
    assert abs(am.item() - want.abs().max().item()) < 1e-4 * want.abs().max().item()


@pytest.mark.parametrize("types", [(BF, BF, BF, BF), (BF, BF, torch.float32, torch.float32), (BF, BF, torch.float8_e4m3fn, BF), (torch.float32,) * 4])
@pytest.mark.parametrize("sizes", [[128], [16384, 128, 16384 + 128, 896, 3 * 16384, 16384 - 128], [128 * (i + 1) for i in range(50)]])
@pytest.mark.parametrize("scalars", ["values", "device"])
def test_adamw_and_norm_of_all_tensors_in_one_launch(types, sizes, scalars):
    """Bit for bit the launches per tensor: sizes around one chunk of the table, more tensors than one round of the norm, the
    step's scalars by value and from device memory (as captured launches read them)."""
    g = torch.Generator(device=DEV).manual_seed(len(sizes))
    r = lambda n, dt, s=1.0: (torch.randn(n, device=DEV, generator=g) * s).to(dt)
    f8 = types[2] == torch.float8_e4m3fn

    def rows():
        g.manual_seed(len(sizes))
        return [{"param": r(n, types[0]), "grad": r(n, types[1], 0.1), "m": r(n, types[2], 0.1), "v": r(n, torch.float32, 0.1).square().to(types[3]),
                 "m_scales": r(n // 128, torch.float32).abs() + 0.1 if f8 else None, "absmax": torch.zeros(1, device=DEV) if i % 2 else None,
                 "elem_offset": 128 * i, "seed": 7919 * i, "decay": i % 3 == 0} for i, n in enumerate(sizes)]

    one, each = rows(), rows()
    table = K.AdamTable(one, DEV)
    assert table.matches(one) and not table.matches(each)
    a, b = torch.full((512,), 0.5, device=DEV), torch.full((512,), 0.5, device=DEV)
    K.norm_squared_multi(a, table)
    for t in each:
        K.norm_squared(b, t["grad"])
    assert torch.equal(a, b)
    scale, hyper = torch.full((1,), 0.7, device=DEV), dict(lr=1e-2, beta1=0.9, beta2=0.95, step=3, eps=1e-8)
    if scalars == "values":
        K.adamw_multi(table, weight_decay=0.1, grad_scale=scale, seed=11, **hyper)
    else:
        host = torch.zeros(8, pin_memory=True)
        K.adamw_hyper(host, weight_decay=0.1, seed=11, **hyper)
        K.adamw_multi(table, lr=0.0, beta1=0.0, beta2=0.0, step=1, eps=0.0, weight_decay=1.0, grad_scale=scale, hyper=host.to(DEV))
    for t in each:
        K.adamw(t["param"], t["grad"], t["m"], t["v"], weight_decay=0.1 if t["decay"] else 0.0, grad_scale=scale, absmax=t["absmax"],
                m_scales=t["m_scales"], seed=11 + t["seed"], elem_offset=t["elem_offset"], **hyper)
    for x, y in zip(one, each):
        for k in ("param", "m", "v", "m_scales", "absmax"):
            if x[k] is not None:
                assert torch.equal(x[k].view(torch.uint8), y[k].view(torch.uint8)), k


# CTA-pair tiles of 224 columns (K-major B) against 256: whole and ragged last tiles, a last half block of 32 columns; the same bits
@pytest.mark.parametrize("f8", [False, True])
@pytest.mark.parametrize("M,N,depth", [(4096, 896, 64), (2300, 1120, 200), (4096, 680, 136), (8448, 264, 128), (256, 8256, 96)])
@pytest.mark.parametrize("accumulate,bias", [(False, True), (True, False)])
def test_gemm_pair_tile_columns(f8, M, N, depth, accumulate, bias):
    dt = torch.float8_e4m3fn if f8 else BF
    if f8:
        depth = (depth + 15) // 16 * 16
    g = torch.Generator(device=DEV).manual_seed(M + N)
    a, b = (torch.randn(r, depth, device=DEV, generator=g).to(dt) for r in (M, N))
    old = torch.randn(M, N, device=DEV, generator=g).to(BF)
    bi = torch.randn(N, device=DEV, generator=g).to(BF) if bias else None
    lib, got = L.kernels(), []
    try:
        for bn in (256, 224):
            lib.llmq_gemm_set_pair_bn(bn)
            wide = torch.full((M, N + 32), 9.0, device=DEV, dtype=BF)
            c, am = wide[:, :N], torch.zeros(1, device=DEV)
            c.copy_(old)
            K.gemm(c, a, b, bias=bi, accumulate=accumulate, absmax=am)
            assert (wide[:, N:] == 9).all()               # nothing beyond the row
            got.append((c.clone(), am.item()))
    finally:
        lib.llmq_gemm_set_pair_bn(0)
    assert torch.equal(got[0][0], got[1][0]) and got[0][1] == got[1][1]
    ref = a.float() @ b.float().t() + (old.float() if accumulate else 0) + (bi.float() if bias else 0)
    assert rel(got[1][0], ref) < 4e-3                     # bf16 rounding: 2^-9 of a value at most


# outputs in whole 32-byte sectors or not: ragged widths, row pitches and addresses on both sides of the rule, in both kernels
@pytest.mark.parametrize("M,N", [(130, 48), (300, 272), (300, 264), (4096, 560), (2304, 1160)])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("pitch,offset", [(0, 0), (16, 0), (8, 0), (16, 8)])
def test_gemm_output_sectors(M, N, accumulate, pitch, offset):
    g = torch.Generator(device=DEV).manual_seed(M + N)
    a, b = (torch.randn(r, 136, device=DEV, generator=g).to(BF) for r in (M, N))
    old = torch.randn(M, N, device=DEV, generator=g).to(BF)
    ld = N + pitch
    flat = torch.full((M * ld + 16,), 9.0, device=DEV, dtype=BF)
    c = flat[offset:offset + M * ld].view(M, ld)[:, :N]
    c.copy_(old)
    K.gemm(c, a, b, accumulate=accumulate)
    assert rel(c, a.float() @ b.float().t() + (old.float() if accumulate else 0)) < 4e-3
    rest = torch.ones_like(flat, dtype=torch.bool)
    rest[offset:offset + M * ld].view(M, ld)[:, :N] = False
    assert (flat[rest] == 9).all()


# as many rounds of pair tiles as of 128-row tiles, and more: the kernel that the rule picks gives the bits of the other one
@pytest.mark.parametrize("M,N,depth", [(896, 4864, 128), (896, 4608, 128), (1152, 3840, 192)])
def test_gemm_rounds_of_tiles(M, N, depth):
    g = torch.Generator(device=DEV).manual_seed(M)
    a, b = (torch.randn(depth, r, device=DEV, generator=g).to(BF) for r in (M, N))
    lib, got = L.kernels(), []
    try:
        for mode in (0, 1, 2):
            lib.llmq_gemm_set_mode(mode)
            c = torch.empty(M, N, device=DEV, dtype=BF)
            K.gemm(c, a, b, a_mn=True, b_mn=True)
            got.append(c)
    finally:
        lib.llmq_gemm_set_mode(0)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    assert rel(got[0], a.float().t() @ b.float()) < 4e-3


def test_chained_launches_see_what_the_kernel_before_wrote():
    """Kernels that start while their predecessor runs, each reading scalars or rows that the one before it writes: the results of back-to-back
    launches and of a captured graph are those of launches with a synchronisation in between."""
    g = torch.Generator(device=DEV).manual_seed(3)
    n, B, T, Hq, Hkv, HS = 1 << 20, 2, 200, 6, 2, 64
    C = (Hq + 2 * Hkv) * HS
    x0, w = torch.randn(B * T, 256, device=DEV, generator=g).to(BF), (torch.randn(C, 256, device=DEV, generator=g) * 0.06).to(BF)
    p0, fr = torch.randn(n, device=DEV, generator=g).to(BF), torch.randn(T, HS // 2, 2, device=DEV, generator=g)
    dout, grad = torch.randn(B, T, Hq, HS, device=DEV, generator=g).to(BF), torch.randn(n, device=DEV, generator=g).to(BF)

    def chain(between):
        x, p = x0.clone(), p0.clone()
        m, v, parts, io = torch.zeros_like(p), torch.zeros_like(p), torch.zeros(512, device=DEV), torch.zeros(2, device=DEV)
        qkv, rot = torch.empty(B * T, C, device=DEV, dtype=BF), torch.empty(B, T, Hq + 2 * Hkv, HS, device=DEV, dtype=BF)
        out, lse = torch.empty(B, T, Hq, HS, device=DEV, dtype=BF), torch.empty(B, Hq, T, device=DEV)
        dqkv, scratch, dw, dx = torch.empty_like(rot), torch.empty(B * Hq * T, device=DEV), torch.empty(C, 256, device=DEV, dtype=BF), torch.empty_like(x)

        def body():
            for step in range(4):
                for f in (lambda: K.gemm(qkv, x, w), lambda: K.rope(rot, qkv.view_as(rot), fr, Hq, Hkv),
                          lambda: K.attention_forward(out, lse, rot, Hq, Hkv), lambda: K.attention_backward(dqkv, scratch, dout, out, lse, rot, Hq, Hkv),
                          lambda: K.gemm(dw, dqkv.view(B * T, C), x, a_mn=True, b_mn=True), lambda: K.gemm(dx, dqkv.view(B * T, C), w, b_mn=True),
                          lambda: parts.zero_(), lambda: K.norm_squared(parts, p), lambda: K.deterministic_sum(io[0:1], parts), lambda: K.norm_finish(io, 1.0),
                          lambda: K.adamw(p, grad, m, v, lr=1e-2, beta1=0.9, beta2=0.95, step=step + 1, eps=1e-8, weight_decay=0.1, grad_scale=io[1:2], seed=step),
                          lambda: x.add_(dx, alpha=0.1)):
                    f()
                    if between:
                        torch.cuda.synchronize()
        return body, (qkv, out, lse, dqkv, dw, dx, p, m, v, io, x)

    body, want = chain(True)
    body()
    for _ in range(5):
        body, got = chain(False)
        torch.cuda.synchronize()
        body()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    body, got = chain(False)
    start = [t.clone() for t in got]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        body()                                                 # workspaces and attributes exist before the capture
        with torch.cuda.graph(graph, stream=side):
            body()
    torch.cuda.current_stream().wait_stream(side)
    for _ in range(3):
        for t, s in zip(got, start):
            t.copy_(s)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))


def _same_with_and_without_waits(chain):
    """``chain()`` gives (launches, tensors they write).  Launched back to back and replayed from a graph, they leave the bits that they leave with
    a synchronisation after every launch."""
    launches, want = chain()
    start = [t.clone() for t in want]
    for f in launches:
        f()
        torch.cuda.synchronize()
    for _ in range(4):
        launches, got = chain()
        torch.cuda.synchronize()
        for f in launches:
            f()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        with torch.cuda.graph(graph, stream=side):
            for f in launches:
                f()
    torch.cuda.current_stream().wait_stream(side)
    for _ in range(3):
        for t, s in zip(got, start):
            t.copy_(s)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))


# the norm starts while the GEMM or the update that writes its tensor runs: one and four loads in flight, fp32 beyond the L2
@pytest.mark.parametrize("dtype,M,N", [(BF, 1001, 896), (BF, 2048, 2048), (torch.float32, 520, 1000), (torch.float32, 2048, 1024), (torch.float32, 8192, 4104)])
def test_norm_right_behind_the_kernel_that_writes_its_tensor(dtype, M, N):
    g = torch.Generator(device=DEV).manual_seed(N)
    a, b = torch.randn(M, 192, device=DEV, generator=g).to(BF), torch.randn(N, 192, device=DEV, generator=g).to(BF)
    p0, grad = torch.randn(M * N, device=DEV, generator=g).to(dtype), torch.randn(M * N, device=DEV, generator=g).to(dtype)

    def chain():
        dw, p = torch.full((M, N), 100.0, device=DEV, dtype=dtype), p0.clone()
        m, v, parts, parts2, io = torch.zeros_like(p), torch.zeros_like(p), torch.zeros(512, device=DEV), torch.zeros(512, device=DEV), torch.zeros(4, device=DEV)
        return [lambda: K.gemm(dw, a, b), lambda: K.norm_squared(parts, dw), lambda: K.deterministic_sum(io[0:1], parts),
                lambda: K.adamw(p, grad, m, v, lr=0.1, beta1=0.9, beta2=0.95, step=1, eps=1e-8, weight_decay=0.1, seed=5),
                lambda: K.norm_squared(parts2, p), lambda: K.deterministic_sum(io[2:3], parts2)], (dw, p, m, v, parts, parts2, io)

    _same_with_and_without_waits(chain)


def test_second_passes_and_tables_see_what_the_kernel_before_wrote():
    """The other kernels that start while their predecessor runs, each right behind the one that writes its rows or its scale: split-K and its sum, the
    bias and norm weight sums, the embedding and its gradient, the loss statistics, the update of a table."""
    g = torch.Generator(device=DEV).manual_seed(11)
    r = lambda *s, std=1.0: (torch.randn(*s, device=DEV, generator=g) * std).to(BF)
    B, T, C, V = 4, 512, 256, 300
    tok = torch.randint(0, V, (B * T,), device=DEV, generator=g, dtype=torch.int32)
    wte0, w0, wn0, b0 = r(V, C), r(C, C, std=0.06), r(C), r(C, std=0.1)

    def chain():
        p = [t.clone() for t in (wte0, w0, wn0)]
        d = [torch.zeros_like(t) for t in p]
        m, v = [torch.zeros_like(t) for t in p], [torch.zeros_like(t) for t in p]
        wte, w, wn = p
        x, h, dx = (torch.zeros(B * T, C, device=DEV, dtype=BF) for _ in range(3))
        f32, rstd, db = torch.zeros(B, T, device=DEV), torch.zeros(B * T, device=DEV), b0.clone()
        st, gl, parts, io = torch.zeros(2, device=DEV), torch.zeros(T // 64, device=DEV), torch.zeros(512, device=DEV), torch.ones(2, device=DEV)
        s1, s2 = torch.zeros(64 * C, device=DEV), torch.zeros(K.rmsnorm_backward_scratch_elems(C, torch.device(DEV, 0)), device=DEV)
        table = K.AdamTable([dict(param=a.view(-1), grad=b.view(-1), m=c.view(-1), v=e.view(-1), elem_offset=0, seed=i, decay=True)
                             for i, (a, b, c, e) in enumerate(zip(p, d, m, v))], DEV)
        hyper = dict(lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, seed=7)
        launches = []
        for step in range(3):
            launches += [lambda: parts.zero_(), lambda: K.encoder_forward(x, tok, wte), lambda: K.gemm(h, x, w, bias=db),
                         lambda: K.bias_backward(db, h, s1, scale_a=io[1:2], accumulate=False),
                         lambda: K.gemm(d[1], h, x, a_mn=True, b_mn=True),                  # cut into parts of K = 2048 tokens
                         lambda: K.gemm(f32, x[:B], x[:T]), lambda: K.lse_stats(st, f32), lambda: K.gemm(f32, h[:B], x[:T]),
                         lambda: K.grouped_loss_sum(gl, f32, 64),
                         lambda: K.rmsnorm_forward(dx, rstd, h, wn, 1e-6), lambda: K.gemm(dx, h, w, b_mn=True, alpha=0.01),
                         lambda: K.rmsnorm_backward(dx, d[2], s2, x, h, wn, rstd, accumulate_dweight=False), lambda: K.gemm(dx, h, w, b_mn=True, alpha=0.02),
                         lambda: K.encoder_backward(d[0], dx, tok), lambda: K.norm_squared_multi(parts, table),
                         lambda: K.deterministic_sum(io[0:1], parts), lambda: K.norm_finish(io, 1.0),
                         lambda step=step: K.adamw_multi(table, grad_scale=io[1:2], step=step + 1, **hyper)]
        return launches, (*p, *d, *m, *v, x, h, dx, f32, rstd, db, st, gl, parts, io)

    assert L.kernels().llmq_gemm_splitk_floats(C, C, B * T, 2, K.num_sms(torch.device(DEV, 0))) > 0
    _same_with_and_without_waits(chain)


# blocks per SM of the backward kernel on both sides of the rule (7 and 24 rows per SM, three or four vectors a thread), as many rows as blocks and one more
@pytest.mark.parametrize("C", [1024, 1032, 3584, 4096, 4104])
@pytest.mark.parametrize("rows", [1, 2, 148, 149, 1036, 1037, 3552, 3553])
def test_rmsnorm_backward_blocks(C, rows):
    g = torch.Generator(device=DEV).manual_seed(C + rows)
    x, w, dy, dres, dw0 = (torch.randn(*s, device=DEV, generator=g).to(BF) for s in ((rows, C), (C,), (rows, C), (rows, C), (C,)))
    rs = torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6)
    dinp, dw, am = dres.clone(), dw0.clone(), torch.zeros(1, device=DEV)
    scratch = torch.full((K.rmsnorm_backward_scratch_elems(C, torch.device(DEV, 0)),), math.nan, device=DEV)
    K.rmsnorm_backward(dinp, dw, scratch, dy, x, w, rs[:, 0].float().contiguous(), absmax=am)
    xh, wdy = x.double() * rs, w.double() * dy.double()
    gx = dres.double() + (wdy - xh * (wdy * xh).mean(-1, keepdim=True)) * rs
    # every element: one rounding to bf16 (2^-9 of it) and fp32 arithmetic on terms of a few units
    assert ((dinp.double() - gx).abs() <= gx.abs() * 2**-8 + 1e-5 * (1 + wdy.abs() * rs)).all()
    assert rel(dw, dw0.double() + (dy.double() * xh).sum(0)) < 2**-8 and am.item() == dinp.float().abs().max().item()


# short rows on both sides of two rows per block: one vector per thread, blocks of the whole GPU (three per SM) and of C > 1024 (one per SM)
@pytest.mark.parametrize("C", [8, 256, 1000, 1024, 2048])
@pytest.mark.parametrize("rows", [1, 296, 297, 444, 445, 888, 889])
@pytest.mark.parametrize("dt", [BF, torch.float32])
def test_rmsnorm_backward_few_rows(C, rows, dt):
    g = torch.Generator(device=DEV).manual_seed(C + rows)
    x, w, dy, dres, dw0 = (torch.randn(*s, device=DEV, generator=g).to(dt) for s in ((rows, C), (C,), (rows, C), (rows, C), (C,)))
    rs = torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6)
    dinp, dw, am = dres.clone(), dw0.clone(), torch.zeros(1, device=DEV)
    scratch = torch.full((K.rmsnorm_backward_scratch_elems(C, torch.device(DEV, 0)),), math.nan, device=DEV)
    K.rmsnorm_backward(dinp, dw, scratch, dy, x, w, rs[:, 0].float().contiguous(), absmax=am)
    xh, wdy = x.double() * rs, w.double() * dy.double()
    gx = dres.double() + (wdy - xh * (wdy * xh).mean(-1, keepdim=True)) * rs
    # as above: one rounding of the output, fp32 arithmetic on terms of a few units
    eps = 2**-8 if dt == BF else 2**-20
    assert ((dinp.double() - gx).abs() <= gx.abs() * eps + 1e-5 * (1 + wdy.abs() * rs)).all()
    assert rel(dw, dw0.double() + (dy.double() * xh).sum(0)) < (2**-8 if dt == BF else 1e-5) and am.item() == dinp.float().abs().max().item()


# the bias gradient in one launch (columns in fours) against the two kernels that take unaligned gradients: the same sums in the same order; rows around
# multiples of 8 and 512, columns around multiples of 16 and 128
@pytest.mark.parametrize("rows", [1, 7, 65, 511, 513, 1001, 3000])
@pytest.mark.parametrize("C", [4, 124, 128, 148, 1152])
@pytest.mark.parametrize("dt,out_dt", [(BF, BF), (torch.float32, torch.float32), (F8, BF), (torch.float8_e5m2, torch.float32)])
def test_bias_backward_one_launch(rows, C, dt, out_dt):
    g = torch.Generator(device=DEV).manual_seed(rows + C)
    dout = torch.randn(rows, C, device=DEV, generator=g).to(dt)
    shifted = torch.empty(rows * C + 8, device=DEV, dtype=dt)[4 // dt.itemsize or 1:][:rows * C].view(rows, C)
    shifted.copy_(dout)
    assert dout.data_ptr() % 16 == 0 and shifted.data_ptr() % 16 != 0
    sa, sb, d0 = torch.full((1,), 0.5, device=DEV), torch.full((1,), 3.0, device=DEV), torch.randn(C, device=DEV, generator=g).to(out_dt)
    for acc in (False, True):
        got = []
        for d in (dout, shifted):
            db, scratch = d0.clone(), torch.full((64 * C,), math.nan, device=DEV)
            K.bias_backward(db, d, scratch, scale_a=sa, scale_b=sb, accumulate=acc)
            got.append(db)
        assert torch.equal(*got)
        want = 1.5 * dout.double().sum(0) + (d0.double() if acc else 0)
        assert ((got[0].double() - want).abs() <= want.abs() * (2**-8 if out_dt == BF else 1e-6) + 1e-5 * rows**0.5 * (448 if dt.itemsize == 1 else 1)).all()


# on both sides of the rows up to which one launch is taken, and numbers of partial sums (one per 8 rows) that are no multiples of 16, in the two-launch form
@pytest.mark.parametrize("rows,C", [(1536, 128), (1537, 128), (1792, 256), (1793, 256), (2048, 1152), (2049, 1152), (8, 2432), (100, 2432), (129, 2432), (500, 2432)])
@pytest.mark.parametrize("dt", [BF, F8])
def test_bias_backward_lines(rows, C, dt):
    g = torch.Generator(device=DEV).manual_seed(rows + C)
    dout, db = torch.randn(rows, C, device=DEV, generator=g).to(dt), torch.full((C,), 9.0, device=DEV)
    K.bias_backward(db, dout, torch.full((64 * C,), math.nan, device=DEV), accumulate=False)
    # fp32 sums of numbers of a few units
    assert ((db.double() - dout.double().sum(0)).abs() <= 1e-5 * rows**0.5).all()


# the sum of the partial squares and the clipping factor in one launch: fewer and more partials than threads, no clipping, a norm that is not finite
@pytest.mark.parametrize("n", [1, 31, 512, 513, 2000])
@pytest.mark.parametrize("clip,bad", [(0.0, None), (1.0, None), (1e6, None), (1.0, math.inf), (1.0, math.nan)])
def test_norm_sum_finish(n, clip, bad):
    x = torch.rand(n, device=DEV, generator=torch.Generator(device=DEV).manual_seed(n))
    if bad is not None:
        x[n // 2] = bad
    io, two = torch.full((3,), 9.0, device=DEV), torch.full((3,), 9.0, device=DEV)
    K.norm_sum_finish(io, x, clip, io[2:3])
    K.deterministic_sum(two[0:1], x)
    K.norm_finish(two, clip, two[2:3])
    assert torch.equal(io.view(torch.int32), two.view(torch.int32))
    if bad is None:
        assert abs(io[0].item() - x.double().sum().sqrt().item()) < 1e-5 * io[0].item()


# SwiGLU where the sigmoid of the gate goes under or over: large gates of both signs, zeros, infinities.  Rounding the exponent g x log2(e) to fp32 alone makes the sigmoid of a negative
# gate wrong by up to |g| 2^-24 of its value (up to a gate of 104, beyond which both are 0), a few more operations by 2^-24 each.  Below -88 the sigmoid is less than 2^-126 and may be 0.
# up x gate, which is taken first, stays finite for the negative gates
@pytest.mark.parametrize("dt", [BF, torch.float32])
def test_swiglu_gate_extremes(dt):
    gates = torch.tensor([0.0, -0.0, 1e-30, -1e-30, 1.0, -1.0, 17.0, -17.0, 60.0, -60.0, 87.0, -87.0, 89.0, -89.0, 104.0, -104.0, 1e4, -1e4, 3e38, -1e38, math.inf, -20.0, 20.0, 5.5])
    gate = gates.to(DEV).to(dt).repeat(3, 8)
    inp = torch.cat([torch.full_like(gate, 1.5), gate], 1)
    out = torch.empty_like(gate)
    K.swiglu_forward(out, inp)
    want = 1.5 * gate.double() * torch.sigmoid(gate.double())
    finite = want.isfinite() & (want.abs() < torch.finfo(dt).max)
    tol = (2**-8 if dt == BF else 0) + (8 + gate.double().abs().clamp(max=104)) * 2**-24
    assert ((out.double() - want).abs()[finite] <= (tol * want.abs() + 1e-34)[finite]).all()
    assert (out[~finite] == math.inf).all()


# the sigmoid 1 / (1 + 2^(-g log2 e)) at every bf16 gate, and at fp32 gates of random bits, with the bound above and the error of log2 e as an fp32 number (1.3e-8 of it, 0.23 x 2^-24), by which the
# sigmoid is wrong by another 0.23 |g| 2^-24
@pytest.mark.parametrize("dt", [BF, torch.float32])
def test_swiglu_every_gate(dt):
    if dt == BF:
        gate = torch.arange(-32768, 32768, device=DEV).to(torch.int16).view(BF)
    else:
        gate = torch.randint(-2**31, 2**31, (1 << 21,), device=DEV, generator=torch.Generator(device=DEV).manual_seed(1)).to(torch.int32).view(torch.float32)
    gate = gate.view(-1, 512)
    out = torch.empty_like(gate)
    K.swiglu_forward(out, torch.cat([torch.ones_like(gate), gate], 1))
    want = gate.double() * torch.sigmoid(gate.double())
    assert torch.equal(out.isnan(), want.isnan())
    finite = want.isfinite() & (want.abs() < torch.finfo(dt).max)
    tol = (2**-8 if dt == BF else 0) + (8 + 1.25 * gate.double().abs().clamp(max=104)) * 2**-24
    assert ((out.double() - want).abs()[finite] <= (tol * want.abs() + 1e-34)[finite]).all()


# RoPE, a head of a token per thread (small calls) and two: odd and even numbers of heads (the last thread of a token has one), head sizes whose halves are 1, 2, 3, 4 and 8 vectors, one token, in
# place with and without the abs-max (value heads are then only read), angles that are not aligned to 16 bytes
@pytest.mark.parametrize("B,T,Hq,Hkv,HS", [(1, 1, 1, 1, 16), (2, 7, 2, 1, 32), (3, 33, 3, 2, 48), (1, 100, 14, 2, 64), (2, 65, 5, 2, 128), (1, 257, 1, 3, 128),
                                           (2, 701, 11, 2, 64), (3, 999, 3, 1, 48), (1, 1301, 2, 3, 128)])
@pytest.mark.parametrize("dt", [BF, torch.float32])
@pytest.mark.parametrize("backward", [False, True])
def test_rope_heads(B, T, Hq, Hkv, HS, dt, backward):
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn(B, T, Hq + 2 * Hkv, HS, device=DEV, generator=g).to(dt)
    table = K.rope_table(T, HS, 1e4, torch.device(DEV, 0))
    shifted = torch.empty(table.numel() + 1, device=DEV)[1:].view_as(table).copy_(table)
    assert shifted.data_ptr() % 16 == 4
    cos, sin = table[:, :, 0].double()[None, :, None], table[:, :, 1].double()[None, :, None] * (-1 if backward else 1)
    a, b = x.double()[..., :HS // 2], x.double()[..., HS // 2:]
    want = torch.cat([torch.cat([a * cos - b * sin, b * cos + a * sin], -1)[:, :, :Hq + Hkv], x.double()[:, :, Hq + Hkv:]], 2)
    eps = 2**-8 if dt == BF else 1e-6
    for freqs in (table, shifted):
        for absmax in (None, torch.zeros(1, device=DEV)):
            for in_place in (False, True):
                src = x.clone()
                out = src if in_place else torch.full_like(x, 9.0)
                if absmax is not None:
                    absmax.zero_()
                K.rope(out, src, freqs, Hq, Hkv, backward=backward, absmax=absmax)
                assert ((out.double() - want).abs() <= eps * want.abs() + 1e-6 * (1 + x.double().abs().max())).all()
                assert absmax is None or absmax.item() == out.float().abs().max().item()


# e4m3 first moments rounded in pairs: blocks of zeros, of values far below the largest (subnormal quotients beside normal ones), of subnormal and of huge gradients
@pytest.mark.parametrize("n", [128, 1152, 128 * 1001])
def test_adamw_e4m3_scales_and_rounding(n):
    g = torch.Generator(device=DEV).manual_seed(n)
    grad = torch.randn(n // 128, 128, device=DEV, generator=g) * torch.logspace(-30, 30, n // 128, device=DEV)[:, None]
    grad *= 10 ** -(6 * torch.rand(n // 128, 128, device=DEV, generator=g))
    grad[0] = 0
    grad = grad.to(BF).view(-1)
    p, v = torch.zeros(n, device=DEV, dtype=BF), torch.ones(n, device=DEV, dtype=BF)
    m, ms = torch.zeros(n, device=DEV, dtype=F8), torch.ones(n // 128, device=DEV)
    K.adamw(p, grad, m, v, lr=0.0, beta1=0.0, beta2=0.5, step=1, eps=1e-8, weight_decay=0.0, m_scales=ms, seed=11)      # beta1 = 0: the moment is the gradient
    want = grad.float().view(-1, 128)
    top = want.abs().amax(-1)
    assert torch.equal(ms, (top.clamp_min(1e-30).double() / 448).float())        # the rounded quotient
    q, x = m.float().view(-1, 128), want.double() / ms.double()[:, None]
    quantum = torch.exp2(torch.floor(torch.log2(x.abs().clamp_min(2.0**-6))) - 3)
    assert ((q.double() - x).abs() < quantum * (1 + 1e-5)).all()                              # stochastic rounding: one of the two neighbours
    assert abs((q.double() - x).div(quantum).mean().item()) < 4 / n**0.5                      # and unbiased


# the ring of the backward kernel turns: more rows per block than it has stages, one vector a thread (four stages) and three or four (two)
@pytest.mark.parametrize("C", [896, 2048, 4104, 5120, 8192])
@pytest.mark.parametrize("rows", [1001, 1777, 3000])
def test_rmsnorm_backward_ring_turns(C, rows):
    g = torch.Generator(device=DEV).manual_seed(C + rows)
    x, w, dy, dres, dw0 = (torch.randn(*s, device=DEV, generator=g).to(BF) for s in ((rows, C), (C,), (rows, C), (rows, C), (C,)))
    rs = torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6)
    dinp, dw, am = dres.clone(), dw0.clone(), torch.zeros(1, device=DEV)
    scratch = torch.full((K.rmsnorm_backward_scratch_elems(C, torch.device(DEV, 0)),), math.nan, device=DEV)
    K.rmsnorm_backward(dinp, dw, scratch, dy, x, w, rs[:, 0].float().contiguous(), absmax=am)
    xh, wdy = x.double() * rs, w.double() * dy.double()
    gx = dres.double() + (wdy - xh * (wdy * xh).mean(-1, keepdim=True)) * rs
    # every element: one rounding to bf16 (2^-9 of it) and fp32 arithmetic on terms of a few units
    assert ((dinp.double() - gx).abs() <= gx.abs() * 2**-8 + 1e-5 * (1 + wdy.abs() * rs)).all()
    assert rel(dw, dw0.double() + (dy.double() * xh).sum(0)) < 2**-8 and am.item() == dinp.float().abs().max().item()


# the entry points through ctypes, for installations whose extension module does not load: the same kernels and results
def test_calls_through_ctypes(monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(3)
    a, b = torch.randn(130, 512, device=DEV, generator=g).to(BF), torch.randn(96, 512, device=DEV, generator=g).to(BF)
    qkv, table = torch.randn(1, 70, 8, 64, device=DEV, generator=g).to(BF), K.rope_table(70, 64, 1e4, torch.device(DEV, 0))
    got = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(L, "_calls", None)
            monkeypatch.setattr(L, "binding", lambda: None)
        out, rot, am = torch.zeros(130, 96, device=DEV, dtype=BF), torch.empty_like(qkv), torch.zeros(1, device=DEV)
        att, lse = torch.empty(1, 70, 4, 64, device=DEV, dtype=BF), torch.empty(1, 4, 70, device=DEV)
        K.gemm(out, a, b, alpha=0.5, absmax=am)
        K.rope(rot, qkv, table, 4, 2)
        K.attention_forward(att, lse, rot, 4, 2)
        got.append((out, rot, am, att, lse))
    assert all(torch.equal(x, y) for x, y in zip(*got)) and got[0][2].item() > 0


# on both sides of the lines between the kernels of short rows: bf16 768 channels (more than two rows a block), fp32 32 MB, 96 MB; the ring of per-thread copies turns
@pytest.mark.parametrize("C,rows,dt", [(8, 5001, BF), (264, 4099, BF), (768, 1333, BF), (776, 1333, BF), (512, 32768, BF), (512, 32769, BF), (1024, 2730, torch.float32),
                                       (1024, 2731, torch.float32), (200, 1001, torch.float32)])
def test_rmsnorm_backward_short_rows(C, rows, dt):
    test_rmsnorm_backward_few_rows(C, rows, dt)


# a row whose copies never come (a build of the kernel that does not issue those of row 300, with a limit of 20 ms): the block that waits for it ends, the status word and NaNs in the weight
# gradient and in all rows of that block say so, and no other row differs
@pytest.mark.parametrize("C,rows", [(896, 2000), (3584, 1001), (5120, 700)])
def test_rmsnorm_backward_lost_copy(C, rows):
    import ctypes
    from llmq_b200.build import build_lost_row
    g = torch.Generator(device=DEV).manual_seed(C)
    x, w, dy, dres = (torch.randn(*s, device=DEV, generator=g).to(BF) for s in ((rows, C), (C,), (rows, C), (rows, C)))
    rs = torch.rsqrt(x.float().square().mean(-1) + 1e-6)
    want, scratch = dres.clone(), torch.zeros(K.rmsnorm_backward_scratch_elems(C, torch.device(DEV, 0)), device=DEV)
    K.rmsnorm_backward(want, torch.zeros_like(w), scratch, dy, x, w, rs)
    lossy = L._through_ctypes(ctypes.CDLL(str(build_lost_row(300))).llmq_rmsnorm_backward, L.SIGNATURES["llmq_rmsnorm_backward"])
    sms = K.num_sms(torch.device(DEV, 0))
    blocks = sms if C > 1024 else 3 * sms                    # rows per block: see the kernel's launch
    for status in (torch.zeros(1, dtype=torch.int32, device=DEV), None):
        dinp, dw, am = dres.clone(), torch.zeros_like(w), torch.zeros(1, device=DEV)
        assert lossy(dinp, dw, scratch, dy, x, w, rs, rows, C, 0, am, 0, 3 * sms, status) == 0
        torch.cuda.synchronize()
        lost = torch.zeros(rows, dtype=torch.bool, device=DEV)
        lost[300 % blocks::blocks] = True
        assert dinp[lost].isnan().all() and torch.equal(dinp[~lost], want[~lost]) and dw.isnan().all()
        assert status is None or status.item() == 32
        assert am.item() <= want.float().abs().max().item()
    again = dres.clone()
    K.rmsnorm_backward(again, torch.zeros_like(w), scratch, dy, x, w, rs)
    assert torch.equal(again, want)
    K.check_status(torch.device(DEV, 0))


# e4m3 first moments of gradients that are not finite: the scale of a block with an infinity is infinite, its finite moments are 0 and the infinity and a NaN are NaN; a NaN alone leaves its
# neighbours and their scale as they are; the largest finite gradients have a finite scale
def test_adamw_e4m3_not_finite():
    n, big = 128 * 6, torch.finfo(BF).max
    grad = torch.randn(6, 128, device=DEV, generator=torch.Generator(device=DEV).manual_seed(7))
    grad[0, 5], grad[1, 127], grad[2, 64], grad[3, 0] = math.inf, -math.inf, math.nan, big
    grad[4, 1], grad[4, 2] = math.inf, math.nan
    p, v = torch.zeros(n, device=DEV, dtype=BF), torch.ones(n, device=DEV, dtype=BF)
    m, ms = torch.zeros(n, device=DEV, dtype=F8), torch.ones(6, device=DEV)
    K.adamw(p, grad.to(BF).view(-1), m, v, lr=0.0, beta1=0.0, beta2=0.5, step=1, eps=1e-8, weight_decay=0.0, m_scales=ms, seed=11)
    want, q = grad.to(BF).float(), m.float().view(6, 128)
    top = want.abs().nan_to_num(0.0, math.inf).amax(-1)
    assert torch.equal(ms, (top.double() / 448).float())
    for b in (0, 1, 4):
        assert torch.equal(q[b].isnan(), ~want[b].isfinite()) and (q[b][want[b].isfinite()] == 0).all()
    for b in (2, 3, 5):
        ok = ~want[b].isnan()
        x = want[b].double() / ms[b].double()
        assert torch.equal(q[b].isnan(), ~ok)
        assert ((q[b].double() - x).abs()[ok] < (torch.exp2(torch.floor(torch.log2(x.abs().clamp_min(2.0**-6))) - 3) * (1 + 1e-5))[ok]).all()


# gradients below the smallest normal number still move a parameter that is 0: they are divided by eps
@pytest.mark.parametrize("params,moments", [(BF, BF), (BF, F8), (BF, torch.float32), (torch.float32, BF), (torch.float32, torch.float32)])
@pytest.mark.parametrize("eps", [1e-8, 1e-39])
def test_adamw_subnormal_gradients(params, moments, eps):
    n = 256
    grad = (2.0 ** -torch.arange(120, 133, device=DEV, dtype=torch.float64)).repeat(20)[:n].to(BF)
    assert (grad > 0).all() and (grad.float() < torch.finfo(torch.float32).tiny).any()
    p, v = torch.zeros(n, device=DEV, dtype=params), torch.zeros(n, device=DEV, dtype=torch.float32 if moments == torch.float32 else BF)
    ms = torch.ones(n // 128, device=DEV) if moments == F8 else None
    K.adamw(p, grad, torch.zeros(n, device=DEV).to(moments), v, lr=1.0, beta1=0.0, beta2=0.0, step=1, eps=eps, weight_decay=0.0, m_scales=ms, seed=3)
    want = grad.double() / torch.tensor(eps, dtype=torch.float32).double().item()
    # the fp32 quotient, a few units in the last place; bf16 parameters are rounded up or down
    assert ((p.double() + want).abs() <= (2**-7 if params == BF else 1e-6) * want).all()


# short sequences: the older rule's pair is kept or left by the estimate of that pair (12 sequences of 128 tokens leave it, 16 keep it)
@pytest.mark.parametrize("B,T,Hq,Hkv,parts", [(12, 128, 28, 4, 1), (16, 128, 28, 4, 2), (7, 33, 12, 2, 1), (8, 20, 16, 2, 4)])
def test_attention_backward_parts_of_short_sequences(B, T, Hq, Hkv, parts):
    assert torch.cuda.get_device_properties(0).multi_processor_count != 148 or L.kernels().llmq_attention_dkdv_parts(B, T, Hq, Hkv, 128) == parts
    test_attention_head_splits(128, B, T, Hq, Hkv)
