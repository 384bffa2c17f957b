"""GPU: a one-token step in one launch (one_step.cu): widths, head sizes and contexts at the edges of its panels and key shares."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from test_engine_gpu import MAX_ABS, Qwen2Config, _launched, check, qwen2_forward, random_hf_weights  # noqa: E402


@pytest.mark.parametrize("cfg,page,contexts", [
    (Qwen2Config(896, 3, 14, 2, 4864, 1531, head_dim=64, name="step-896"), 16, (0, 1, 63, 254, 256, 700)),     # one share of keys, two, three
    (Qwen2Config(1536, 2, 12, 2, 8960, 999, head_dim=128, name="step-1536"), 24, (5, 126, 127, 128, 300)),     # two pieces of k, eight panels
    (Qwen2Config(960, 2, 5, 5, 1232, 515, head_dim=64, name="step-odd"), 8, (40, 129)),      # pieces of 960 and 272, no grouping, few rows
    (Qwen2Config(160, 2, 8, 1, 512, 300, head_dim=128, name="step-least"), 16, (17, 300)),   # one or two rows a CTA
])
def test_one_token_in_one_launch(cfg, page, contexts):
    """three steps in a row behind every context, so that each reads what the ones before appended: against the oracle and the chain of
    kernels, which rounds at the same points"""
    from asd_b200._lib import lib
    from asd_b200.engine import QwenEngine
    w = random_hf_weights(cfg, seed=31, logit_std=0.4)
    top = max(contexts) + 3
    ids = torch.randint(0, cfg.vocab_size, (1, top), generator=torch.Generator().manual_seed(7))
    ref = qwen2_forward(w, cfg, ids)
    idc, slot = ids.cuda().to(torch.int32), torch.zeros(1, dtype=torch.int32, device="cuda")
    for n in contexts:
        got = {}
        for mode in (1, 2):
            eng = QwenEngine(cfg, max_seqs=1, max_seq_len=top + 5, max_tokens=64, page_size=page).load_hf_weights(w)
            eng.set_option("one_token", mode)
            if n:
                eng.prefill(idc[:, :n].contiguous(), slot, want_logits=False)

            def steps():
                got[mode] = torch.cat([eng.forward_uniform(idc[:, i:i + 1].contiguous(), slot + i, slot, i + 1) for i in range(n, n + 3)]).cpu()

            before = lib().asd_kernel_launches(b"gemv")
            assert _launched("one_step", steps) == (3 if mode == 1 else 0)
            assert lib().asd_kernel_launches(b"gemv") - before == 3 * (1 if mode == 1 else 4 * cfg.num_hidden_layers + 1)      # 1: the logits
            eng.close()
        check(got[1], ref[0, n:n + 3])
        assert (got[1] - got[2]).abs().max().item() <= MAX_ABS


@pytest.mark.parametrize("cfg", [
    Qwen2Config(256, 2, 4, 2, 256, 300, head_dim=64, name="step-narrow-ffn"),      # 128 pairs of gate and up rows: fewer than CTAs
    Qwen2Config(256, 2, 2, 1, 512, 300, head_dim=64, name="step-narrow-qkv"),      # 128 pairs of query, key and value rows
])
def test_narrow_models_stay_a_chain(cfg):
    """a model whose matrices leave CTAs without rows takes a kernel a projection, as larger steps do"""
    from asd_b200.engine import QwenEngine
    w = random_hf_weights(cfg, seed=37, logit_std=0.4)
    ids = torch.randint(0, cfg.vocab_size, (1, 20), generator=torch.Generator().manual_seed(9))
    ref = qwen2_forward(w, cfg, ids)
    eng = QwenEngine(cfg, max_seqs=1, max_seq_len=32, max_tokens=16).load_hf_weights(w)
    idc, slot, got = ids.cuda().to(torch.int32), torch.zeros(1, dtype=torch.int32, device="cuda"), []

    def steps():
        for i in range(20):
            got.append(eng.forward_uniform(idc[:, i:i + 1].contiguous(), slot + i, slot, i + 1))

    assert _launched("one_step", steps) == 0
    check(torch.cat(got).cpu(), ref[0])
    eng.check_device()
    eng.close()


def test_one_launch_again_and_again():
    """many steps on one engine, with and without logits between them, and on two engines in turn: always the same results"""
    from asd_b200.engine import QwenEngine
    cfg = Qwen2Config(896, 2, 14, 2, 4864, 1000, head_dim=64, name="step-again")
    w = random_hf_weights(cfg, seed=33, logit_std=0.4)
    engines = [QwenEngine(cfg, max_seqs=1, max_seq_len=64, max_tokens=16).load_hf_weights(w) for _ in range(2)]
    slot = torch.zeros(1, dtype=torch.int32, device="cuda")
    ids = torch.randint(0, cfg.vocab_size, (1, 20), generator=torch.Generator().manual_seed(8)).cuda().to(torch.int32)
    pos, cu = slot.clone(), torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    first = None
    for _ in range(10):
        for eng in engines:
            out = []
            for i in range(20):
                tok = ids[0, i:i + 1].contiguous()
                if i % 3 == 1:
                    eng.forward(tok, pos + i, slot, cu, slot, 1, i + 1, want_logits=False)
                else:
                    out.append(eng.forward(tok, pos + i, slot, cu, slot, 1, i + 1).clone())
            out = torch.cat(out)
            first = out if first is None else first
            assert torch.equal(out, first)
    for eng in engines:
        eng.close()


def test_one_launch_on_two_streams_and_under_capture():
    """steps of two engines enqueued on two streams at once end (one such grid at a time), and a captured step stays a chain of kernels"""
    from asd_b200.engine import QwenEngine
    cfg = Qwen2Config(896, 2, 14, 2, 4864, 1000, head_dim=64, name="step-streams")
    w = random_hf_weights(cfg, seed=35, logit_std=0.4)
    engines = [QwenEngine(cfg, max_seqs=1, max_seq_len=64, max_tokens=16).load_hf_weights(w) for _ in range(2)]
    slot = torch.zeros(1, dtype=torch.int32, device="cuda")
    tok, pos, cu = slot + 7, slot.clone(), torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    out = [torch.empty(1, cfg.vocab_size, device="cuda") for _ in range(2)]
    want = engines[0].forward(tok, pos, slot, cu, slot, 1, 1).clone()
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(50):
        for eng, s, o in zip(engines, streams, out):
            with torch.cuda.stream(s):
                eng.forward(tok, pos, slot, cu, slot, 1, 1, logits_out=o)
    torch.cuda.synchronize()
    assert torch.equal(out[0], want) and torch.equal(out[1], want)
    graph = torch.cuda.CUDAGraph()

    def captured():
        with torch.cuda.graph(graph):
            engines[0].forward(tok, pos, slot, cu, slot, 1, 1, logits_out=out[0])
    assert _launched("one_step", captured) == 0
    out[0].zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert (out[0] - want).abs().max().item() <= MAX_ABS
    for eng in engines:
        eng.check_device()
        eng.close()


def test_one_launch_beside_a_persistent_forward():
    """steps of two engines on two streams, one in one launch and one in the persistent forward kernel (both wait for their own CTAs), end with the
    right results; a captured step of either is a chain of kernels"""
    from asd_b200.engine import QwenEngine
    cfg = Qwen2Config(896, 2, 14, 2, 4864, 1000, head_dim=64, name="step-persist")
    w = random_hf_weights(cfg, seed=39, logit_std=0.4)
    engines = [QwenEngine(cfg, max_seqs=1, max_seq_len=64, max_tokens=16).load_hf_weights(w) for _ in range(2)]
    engines[1].set_option("persist", 1)
    slot = torch.zeros(1, dtype=torch.int32, device="cuda")
    tok, pos, cu = slot + 7, slot.clone(), torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    out = [torch.empty(1, cfg.vocab_size, device="cuda") for _ in range(2)]
    want = [eng.forward(tok, pos, slot, cu, slot, 1, 1).clone() for eng in engines]
    check(torch.cat(want).cpu(), qwen2_forward(w, cfg, torch.tensor([[7]]))[0].expand(2, -1))
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()

    def steps():
        for _ in range(50):
            for eng, s, o in zip(engines, streams, out):
                with torch.cuda.stream(s):
                    eng.forward(tok, pos, slot, cu, slot, 1, 1, logits_out=o)
        torch.cuda.synchronize()

    assert _launched("one_step", steps) == 50
    for eng, o, x in zip(engines, out, want):
        assert (o - x).abs().max().item() <= MAX_ABS
        eng.check_device()
        graph = torch.cuda.CUDAGraph()

        def captured():
            with torch.cuda.graph(graph):
                eng.forward(tok, pos, slot, cu, slot, 1, 1, logits_out=o)

        assert _launched("gemv", captured) > 0
        o.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert (o - x).abs().max().item() <= MAX_ABS
        eng.close()
