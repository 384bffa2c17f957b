"""A wait inside a kernel that runs out: it ends, is reported through mapped host memory, and nothing made from its results
reaches the host (the waits of these tests have a limit of two seconds)."""
import pytest
import torch

from asd_b200._lib import AsdError, check, lib
from asd_b200.models.qwen2 import tiny_config

pytestmark = pytest.mark.gpu


def _engine(name):
    from asd_b200 import engine
    from asd_b200.models import mezilix, rivetar
    kw = dict(max_seqs=2, max_seq_len=64, max_tokens=32)
    if name == "qwen":
        return engine.QwenEngine(tiny_config(), **kw).load_random(seed=1)
    if name == "mezilix":
        return engine.MezilixEngine(mezilix.sized_config(256, 1, 2, ff=256), ring=8, **kw).load_random(seed=1)
    return engine.RivetarEngine(rivetar.sized_config(256, 3, 2, ff=768), ring=8, **kw).load_random(seed=1)


def _step(eng):
    slots = torch.arange(2, dtype=torch.int32, device="cuda")
    return eng.prefill(torch.ones(2, 5, dtype=torch.int32, device="cuda"), slots)


@pytest.mark.parametrize("name", ["qwen", "mezilix", "rivetar"])
def test_engine_refuses_after_a_wait_ran_out(name):
    eng, other = _engine(name), _engine("qwen")
    _step(eng)
    eng.check_device()
    eng.set_option("debug_wait", 1)
    with pytest.raises(AsdError, match="bounded wait"):
        eng.check_device()
    for _ in range(2):                      # and it stays refused: its caches hold what the launch left
        with pytest.raises(AsdError, match="bounded wait"):
            _step(eng)
    want = _step(other)                     # the GPU and the other engines go on
    assert torch.equal(_step(other), want)
    other.check_device()
    eng.close()
    other.close()


def test_decoder_hands_nothing_to_the_host_after_a_wait_ran_out():
    from asd_b200.engine import SpecDecoder
    eng = _engine("qwen")
    dec = SpecDecoder(eng, None, 2, 0, 0.0)
    dec.prefill(torch.ones(2, 5, dtype=torch.int64))
    host = torch.zeros(3, 2, dtype=torch.int32).pin_memory()
    host.copy_(torch.stack([dec.last_tok, dec.prev_tok, dec.pos]))
    toks, acc = torch.zeros(2, 1, dtype=torch.int32).pin_memory(), torch.zeros(2, dtype=torch.int32).pin_memory()
    step = dec._step

    def last_kernel_waits():
        out = step()
        eng.set_option("debug_wait", 1)
        return out

    dec._step = last_kernel_waits
    with pytest.raises(AsdError, match="bounded wait"):
        dec.step_host(host, toks, acc)
    eng.close()


def test_sampler_call_is_refused_once():
    from asd_b200.ops import RejectionSampler
    s = RejectionSampler(2, 0)
    args = (torch.randn(2, 1, 4096, device="cuda"), None, torch.zeros(2, 0, dtype=torch.int32, device="cuda"),
            torch.zeros(2, 0, dtype=torch.float64, device="cuda"), torch.full((2,), 0.5, dtype=torch.float64, device="cuda"), 0.7)
    want = s(*args)["out_tokens"].clone()
    check(lib().asd_debug_wait_expiry(torch.cuda.current_stream().cuda_stream), "asd_debug_wait_expiry")
    torch.cuda.synchronize()
    with pytest.raises(AsdError, match="bounded wait"):
        s(*args)
    assert torch.equal(s(*args)["out_tokens"], want) and lib().asd_wait_error() == 0
