"""The tensor-bound CTA-pair GEMM (csrc/gemm_tc.cu: tcgen05 cta_group::2, 256 weight rows x <= 256 tokens per tile,
persistent, two TMEM accumulators) against a torch fp32 reference of the same contraction.  bf16 inputs are exact
in fp32, so the only difference is the fp32 summation order: relative tolerance 2e-5 of the row scale."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(x, w):
    return x.float() @ w.float().T


@pytest.mark.parametrize("M,N,K,ksplit", [
    (576, 1024, 1024, 0),        # 3 token tiles of 192, 4 weight pair-tiles
    (576, 8192, 3696, 0),        # 72B down projection shard at TP = 8 (K not a multiple of 64)
    (300, 1344, 1000, 0),        # ragged everything: 2 token tiles of 160, N not a multiple of 256, K % 64 != 0
    (257, 512, 4096, 3),         # forced 3-way K split: slices summed in order
    (1024, 2560, 8192, 0),       # 4 token tiles of 256: both accumulators full width
    (40, 256, 512, 1),           # smallest legal tile (32 tokens), single unit
])
def test_tc_linear_matches_fp32_reference(M, N, K, ksplit):
    from asd_b200.ops import linear_bf16_tc
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = (torch.randn(M, K, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    got = linear_bf16_tc(x, w, 0, ksplit)
    ref = _ref(x, w)
    tol = 2e-5 * ref.abs().max().item() * (K ** 0.5) / 8 + 1e-6
    assert (got - ref).abs().max().item() <= tol, ((got - ref).abs().max().item(), tol)


@pytest.mark.parametrize("M,ff,K", [(576, 3696, 1024), (320, 1000, 768)])
def test_tc_swiglu_matches_reference(M, ff, K):
    from asd_b200.ops import interleave_gate_up, linear_bf16_tc
    g = torch.Generator(device="cuda").manual_seed(ff)
    x = (torch.randn(M, K, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    wg = (torch.randn(ff, K, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    wu = (torch.randn(ff, K, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    got = linear_bf16_tc(x, interleave_gate_up(wg, wu), 2)[:, :ff].float()
    ref = torch.nn.functional.silu(_ref(x, wg)) * _ref(x, wu)
    err = (got - ref).abs().max().item()
    assert err <= 1e-2 * ref.abs().max().item() + 1e-3, err      # bf16 output rounding


def test_tc_agrees_with_weight_streaming_kernel():
    from asd_b200.ops import linear_bf16, linear_bf16_tc
    g = torch.Generator(device="cuda").manual_seed(1)
    x = (torch.randn(576, 2048, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    w = (torch.randn(1536, 2048, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    a, b = linear_bf16_tc(x, w, 0), linear_bf16(x, w, 3)
    assert (a - b).abs().max().item() <= 1e-3 * b.abs().max().item()


@pytest.mark.parametrize("M,N,K,ksplit", [(300, 1001, 512, 1), (300, 1001, 1032, 2), (257, 130, 1024, 1), (520, 97, 264, 1)])
@pytest.mark.parametrize("shift", [0, 1])
def test_tc_linear_stores_directly_where_no_tensor_map_fits(M, N, K, ksplit, shift):
    """fp32 rows that are no multiple of 16 bytes, or a result that starts 4 bytes off: a store per lane and token instead of TMA
    boxes, and nothing written beside them"""
    import ctypes
    from asd_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = (torch.randn(M, K, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    buf = torch.full((1 + ksplit * M * N + 64,), 7.0, device="cuda")
    used = ctypes.c_int(0)
    check(lib().asd_linear_bf16_tc(x.data_ptr(), w.data_ptr(), buf.data_ptr() + 4 * shift, M, N, K, 0, ksplit, 0, ctypes.byref(used),
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "tc")
    assert used.value == ksplit
    got = buf[shift:shift + ksplit * M * N].view(ksplit, M, N).sum(0)
    ref = _ref(x, w)
    tol = 2e-5 * ref.abs().max().item() * (K ** 0.5) / 8 + 1e-6
    assert (got - ref).abs().max().item() <= tol
    assert (buf[:shift] == 7).all() and (buf[shift + ksplit * M * N:] == 7).all()


@pytest.mark.parametrize("pad", [3, 4, 64])
def test_logits_of_a_large_step_keep_to_their_columns(pad):
    """300 rows of logits, vocab + pad floats apart: TMA boxes clipped at the vocabulary (pad 4 and 64), direct stores (pad 3)"""
    from asd_b200._lib import lib
    from asd_b200.engine import QwenEngine
    from asd_b200.models.qwen2 import tiny_config
    cfg = tiny_config(num_hidden_layers=1, vocab_size=500)
    eng = QwenEngine(cfg, max_seqs=30, max_seq_len=16, max_tokens=300).load_random(seed=2)
    ids = torch.randint(0, 500, (30, 10), generator=torch.Generator().manual_seed(3), dtype=torch.int32).cuda()
    slots = torch.arange(30, dtype=torch.int32, device="cuda")
    start = torch.zeros(30, dtype=torch.int32, device="cuda")
    want = eng.forward_uniform(ids, start, slots, 10)
    out = torch.full((300, 500 + pad), 7.0, device="cuda")
    before = lib().asd_kernel_launches(b"gemm_pair")
    eng.forward_uniform(ids, start, slots, 10, logits_out=out, logits_ld=500 + pad)
    assert lib().asd_kernel_launches(b"gemm_pair") > before
    assert torch.equal(out[:, :500], want.view(300, 500)) and (out[:, 500:] == 7).all()
    eng.close()
