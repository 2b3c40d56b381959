"""PyTorch paths of the kernel wrappers that have no model-level CPU coverage: they are what the CPU tests of the model run
and what the GPU kernels are compared with, so they are checked against the formulas directly."""
import pytest
import torch

from llmq_b200.ops import kernels as K
from llmq_b200.ops import lib as L

F8 = torch.float8_e4m3fn


def _swiglu_grad(dout, inp):
    D = inp.shape[-1] // 2
    x = inp.float()
    up, gate = x[:, :D], x[:, D:]
    s = torch.sigmoid(gate)
    d = dout.float()
    return torch.cat([d * gate * s, d * up * s * (1 + gate * (1 - s))], -1)


def test_swiglu_backward_two_pass_fallbacks_match_the_separate_kernels():
    torch.manual_seed(0)
    rows, D = 48, 80
    inp = (torch.randn(rows, 2 * D) * 1.5).bfloat16()
    dout = (torch.randn(rows, D) * 0.7).bfloat16()
    want = _swiglu_grad(dout, inp).bfloat16()
    # pass 1: abs-max of the gradient as it would be stored
    am = torch.zeros(1)
    K.swiglu_backward_stats(am, dout, inp)
    assert am.item() == want.float().abs().max().item()
    # ... and, on request, the transposed e4m3 SwiGLU output under a known abs-max
    act = torch.empty(rows, D, dtype=torch.bfloat16)
    act_am = torch.zeros(1)
    K.swiglu_forward(act, inp, absmax=act_am)
    act_t, act_sc = torch.zeros(D, rows, dtype=F8), torch.zeros(1)
    am2 = torch.zeros(1)
    K.swiglu_backward_stats(am2, dout, inp, act_t=act_t, act_absmax=act_am, act_scale=act_sc)
    assert am2.item() == am.item()
    assert act_sc.item() == pytest.approx(act_am.item() / 448.0, rel=1e-6)
    back = act_t.float().t() * act_sc
    assert (back - act.float()).abs().max().item() <= 0.07 * act_am.item()          # e4m3: 3 mantissa bits
    # pass 2: e4m3 rows and their transpose, same bytes as quantising the stored gradient
    q, qt, sc = torch.zeros(rows, 2 * D, dtype=F8), torch.zeros(2 * D, rows, dtype=F8), torch.zeros(1)
    K.swiglu_backward_quant(q, qt, sc, dout, inp, am)
    q_ref, qt_ref, sc_ref = torch.zeros(rows, 2 * D, dtype=F8), torch.zeros(2 * D, rows, dtype=F8), torch.zeros(1)
    K.quantize_transpose(q_ref, qt_ref, sc_ref, want, am)
    assert sc.item() == sc_ref.item() == pytest.approx(am.item() / 448.0, rel=1e-6)
    assert torch.equal(q.view(torch.uint8), q_ref.view(torch.uint8))
    assert torch.equal(qt.view(torch.uint8), q.view(torch.uint8).t())


def test_quantize_transpose_fallback_is_quantise_then_transpose():
    torch.manual_seed(1)
    x = torch.randn(32, 48).bfloat16()
    am = x.float().abs().max().reshape(1)
    q, qt, sc = torch.zeros(32, 48, dtype=F8), torch.zeros(48, 32, dtype=F8), torch.zeros(1)
    K.quantize_transpose(q, qt, sc, x, am)
    assert torch.equal(qt.view(torch.uint8), q.view(torch.uint8).t())
    assert (q.float() * sc - x.float()).abs().max().item() <= 0.07 * am.item()
    # 1-byte input: a plain transpose
    qt2 = torch.zeros(48, 32, dtype=F8)
    K.quantize_transpose(None, qt2, None, q, None)
    assert torch.equal(qt2.view(torch.uint8), q.view(torch.uint8).t())


@pytest.mark.skipif(not L.have_kernels(), reason="native library not built")
@pytest.mark.parametrize("elem_bytes", [1, 2, 4])
def test_split_k_workspace_rule(elem_bytes):
    """The workspace of a GEMM is asked for per call (no pointer is bound to a thread): whole parts of M x N floats, each with a K step."""
    lib = L.kernels()
    assert not hasattr(lib, "llmq_gemm_set_splitk_workspace")
    sms, bk, seen = 148, 128 // elem_bytes, set()
    for M in (1, 128, 200, 896, 1001, 1152, 2304, 4096, 9472):
        for N in (8, 256, 300, 896, 1152, 2048, 4608):
            for K in (64, 1001, 1024, 1152, 4096, 65536, 151936):
                floats = lib.llmq_gemm_splitk_floats(M, N, K, elem_bytes, sms)
                parts, rest = divmod(floats, M * N)
                tiles, steps = -(-M // 128) * -(-N // 256), -(-K // bk)
                seen.add(parts)
                assert rest == 0 and (parts == 0 or 2 <= parts <= 8) and floats <= 16 << 20
                if parts:
                    assert tiles * 2 <= sms and tiles * parts <= sms and (parts - 1) * -(-steps // parts) < steps and steps >= 8 * parts
                elif tiles * 2 <= sms and steps >= 16 and 2 * M * N <= 16 << 20:
                    assert elem_bytes != 4 and M >= 256 and M * N >= 32 * 256 * 256       # the CTA-pair kernel
    assert {0, 2, 3, 8} <= seen
    assert lib.llmq_gemm_splitk_floats(0, 8, 8, elem_bytes, sms) == 0


# one or two CTAs per tile on both sides of each line of the rule: few output elements, short K, one round of tiles (both by the bytes that rows start at multiples of), half of the SMs idle with
# and without a workspace to cut K with
@pytest.mark.skipif(not L.have_kernels(), reason="native library not built")
@pytest.mark.parametrize("M,N,steps,both_mn,may_cut,ctas", [(255, 16384, 40, 0, 1, 1), (1024, 2047, 40, 0, 1, 1), (9728, 904, 6, 0, 1, 1), (9728, 904, 7, 0, 1, 1), (9728, 904, 8, 0, 1, 1), (9728, 904, 9, 0, 1, 2),
                                                            (2320, 1160, 12, 0, 1, 1), (2320, 1160, 13, 0, 1, 1), (2320, 1160, 24, 0, 1, 1), (2320, 1160, 25, 0, 1, 1), (2320, 1160, 32, 0, 1, 1),
                                                            (2320, 1160, 33, 0, 1, 1), (2320, 1160, 64, 0, 1, 1), (2320, 1160, 65, 0, 1, 2), (2040, 2064, 16, 1, 1, 1), (2040, 2064, 17, 1, 1, 2),
                                                            (1064, 2040, 47, 0, 1, 2), (1064, 2040, 48, 0, 1, 1), (1064, 2040, 48, 0, 0, 1), (1064, 2040, 47, 1, 0, 2),
                                                            (1064, 2040, 48, 1, 1, 1), (1064, 2040, 48, 1, 0, 2)])
@pytest.mark.parametrize("elem_bytes", [1, 2])
def test_gemm_tile_rule(M, N, steps, both_mn, may_cut, ctas, elem_bytes):
    lib, K = L.kernels(), steps * (128 // elem_bytes)
    assert lib.llmq_gemm_tile_ctas(M, N, K, elem_bytes, both_mn, 128, 0, may_cut, 148) == ctas
    if may_cut and steps >= 47:
        assert (lib.llmq_gemm_splitk_floats(M, N, K, elem_bytes, 148) > 0) == (ctas == 1 and steps == 48)
    assert lib.llmq_gemm_tile_ctas(M, N, K * elem_bytes // 4, 4, both_mn, 128, 0, may_cut, 148) == 1      # fp32 operands
    if (M, N) in ((2320, 1160), (2040, 2064), (9728, 904)):
        assert lib.llmq_gemm_tile_ctas(M, N, K, elem_bytes, both_mn, 128, 1, may_cut, 148) == 2              # bf16 that is not made of whole sectors
        assert lib.llmq_gemm_tile_ctas(M, N, K, elem_bytes, both_mn, 128, 2, may_cut, 148) == (2 if steps > 32 else ctas)        # fp32
    for line, walk, short in ((64, 32, 8), (32, 24, 8), (16, 12, 6)):
        if (M, N) in ((2320, 1160), (2040, 2064)):           # one round
            assert lib.llmq_gemm_tile_ctas(M, N, K, elem_bytes, both_mn, line, 0, may_cut, 148) == (1 if steps <= (min(walk, 16) if both_mn else walk) else 2)
        if (M, N) == (9728, 904):
            assert lib.llmq_gemm_tile_ctas(M, N, K, elem_bytes, both_mn, line, 0, may_cut, 148) == (1 if steps <= short else 2)


@pytest.mark.skipif(not L.have_kernels(), reason="native library not built")
@pytest.mark.parametrize("change,message", [
    (dict(m_scales=None), "need m_scales"), (dict(m_scales=torch.ones(1)), "m_scales holds 2"), (dict(m_scales=torch.ones(2).bfloat16()), "m_scales holds"),
    (dict(m_scales=torch.ones(4)[::2]), "m_scales holds"), (dict(absmax=torch.zeros(1).double()), "absmax holds"), (dict(absmax=torch.zeros(0)), "absmax holds"),
    (dict(param=torch.zeros(128).bfloat16()), "one size"), (dict(), "one CUDA device")])
def test_optimizer_table_refuses_rows_that_its_kernel_cannot_take(change, message):
    """The launch reads the rows' addresses on the GPU, so everything is checked before one is written down."""
    row = {"param": torch.zeros(256).bfloat16(), "grad": torch.zeros(256).bfloat16(), "m": torch.zeros(256).to(F8), "v": torch.zeros(256).bfloat16(),
           "m_scales": torch.ones(2), "absmax": torch.zeros(1), "elem_offset": 0, "seed": 0, "decay": True}
    with pytest.raises(ValueError, match=message):
        K.AdamTable([{**row, **change}], "cpu")


def test_tile_width_of_the_pair_gemm_is_checked():
    lib = L.kernels()
    try:
        assert [lib.llmq_gemm_set_pair_bn(n) for n in (224, 256, 0)] == [0, 0, 0]
        assert [lib.llmq_gemm_set_pair_bn(n) for n in (-1, 1, 128, 225, 512)] == [-1] * 5
    finally:
        lib.llmq_gemm_set_pair_bn(0)
