"""GPU: the few-token projection (csrc/linear_few.cu) against a torch fp32 product of the same bf16 operands."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def few(x, w):
    from asd_b200._lib import check, lib
    out = torch.full((x.shape[0], w.shape[0]), float("nan"), device="cuda")
    check(lib().asd_linear_bf16_few(x.data_ptr(), w.data_ptr(), out.data_ptr(), x.shape[0], w.shape[0], x.shape[1],
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "few")
    return out


# rows that no group of 16 fills, k that no piece of 32, warp or block of eight pieces fills, several groups a CTA,
# both sides of the line between two blocks an SM and one, the longest k
@pytest.mark.parametrize("N,K", [(1, 8), (16, 40), (25, 256), (100, 1000), (2051, 2048), (6144, 2048), (9000, 264), (48, 3000), (2816, 2816), (4000, 2824), (6000, 4096),
                                 (2048, 6144)])
def test_few_tokens_match_and_do_not_depend_on_their_number(N, K):
    g = torch.Generator(device="cuda").manual_seed(N + K)
    x = (torch.randn(16, K, device="cuda", generator=g) * 0.5).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16()
    ref = (x.double() @ w.double().T).float()
    # fp32 sums of K products in another order: as tests/test_gemm_tc_gpu.py
    tol = 2e-5 * ref.abs().max().item() * max(1.0, K ** 0.5 / 8) + 1e-6
    one = few(x[:1].contiguous(), w)
    for M in (1, 3, 8, 9, 16):
        got = few(x[:M].contiguous(), w)
        assert (got - ref[:M]).abs().max().item() <= tol
        assert torch.equal(got[:1], one)


def test_few_tokens_refuse_what_they_cannot_take():
    from asd_b200._lib import AsdError
    x, w = torch.zeros(17, 64, device="cuda").bfloat16(), torch.zeros(64, 64, device="cuda").bfloat16()
    with pytest.raises(AsdError):
        few(x, w)
    with pytest.raises(AsdError):
        few(x[:1, :60].contiguous(), w[:, :60].contiguous())
