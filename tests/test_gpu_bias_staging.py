"""Biased 16-bit problems at the edges of the bias staging (and short ones, on the kernels below it): rows on 16-byte boundaries (N a multiple of 4) and off them, key
tails of one key up to a full tile, an offset base address, a broadcast and a dense bias, and the dense bias gradient, which
the kernels store without a cleared tensor."""
import pytest
import torch

import elsa_b200 as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 49, 64, 130, 512, 513, 516, 639, 642, 772])
@pytest.mark.parametrize("d", [64, 40, 128])
@pytest.mark.parametrize("kind", ["hnn", "bhnn", "offset"])
@pytest.mark.parametrize("causal", [False, True])
def test_biased_forward_and_gradients_match_fp64(n, d, kind, causal):
    b, h = 2, 2
    gen = torch.Generator(device="cuda").manual_seed(n + d)
    q, k, v, do = (torch.randn((b, h, n, d), generator=gen, device="cuda").half() for _ in range(4))
    if kind == "offset":       # a contiguous bias whose first element is 4 bytes past a 16-byte boundary
        bias = torch.randn(h * n * n + 1, generator=gen, device="cuda")[1:].view(1, h, n, n)
    else:
        bias = torch.randn((h, n, n) if kind == "hnn" else (b, h, n, n), generator=gen, device="cuda")
    x = [t.detach().requires_grad_(True) for t in (q, k, v, bias)]
    out = E.twopass_attention_train(x[0], x[1], x[2], bias=x[3], is_causal=causal)
    poison = torch.full_like(bias, float("nan"))   # what an uncleared gradient tensor would be made of
    del poison
    got = torch.autograd.grad(out, x, do)
    y = [t.detach().double().requires_grad_(True) for t in (q, k, v, bias)]
    s = y[0] @ y[1].transpose(-1, -2) * d ** -0.5 + y[3]
    if causal:
        s = s.masked_fill(torch.ones(n, n, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    ref = torch.softmax(s, -1) @ y[2]
    want = torch.autograd.grad(ref, y, do.double())
    for g, w in zip((out.detach(),) + got, (ref.detach(),) + want):
        # P, dS and the outputs are rounded to fp16 (2^-12 relative on average, a few of them in a row)
        assert (g.double() - w).norm() <= 2e-3 * w.norm()
