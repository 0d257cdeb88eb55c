"""The bias gradient at its contract: every entry stored where nothing is summed and the problem is not causal, and rows of the
bias that leave no key."""
import pytest
import torch

import elsa_b200 as E
from elsa_b200 import _lib

pytestmark = pytest.mark.gpu

DTYPES = [torch.float16, torch.bfloat16, torch.float32]


def _fp64(q, k, v, bias, grad_out):
    x = [t.detach().double().requires_grad_(True) for t in (q, k, v, bias)]
    s = x[0] @ x[1].mT * q.shape[-1] ** -0.5 + x[3]
    out = torch.softmax(s, -1) @ x[2]
    return torch.autograd.grad(out, x, grad_out.double())


def _problem(b, h, n, d, dtype):
    gen = torch.Generator(device="cuda").manual_seed(n + d)
    q, k, v, do = (torch.randn((b, h, n, d), generator=gen, device="cuda").to(dtype) for _ in range(4))
    return q, k, v, do, torch.randn((b, h, n, n), generator=gen, device="cuda")


# a few roundings of P, dS and the results to the input type in a row, 2^-12 (fp16) and 2^-9 (bf16) on average; fp32 sums
LIMIT = {torch.float16: 2e-3, torch.bfloat16: 1.5e-2, torch.float32: 1e-5}


# one size per kernel family and edge: windows / FP32-FMA one-launch, FP32-FMA, five contractions, wide heads, fp32 planes
@pytest.mark.parametrize("n,d", [(1, 64), (49, 32), (64, 64), (65, 64), (130, 40), (130, 36), (513, 64), (640, 24), (513, 128), (130, 72)])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("flags", [0, _lib.FLAG_REPEATABLE, _lib.FLAG_FORCE_SIMT])
def test_a_dense_gradient_is_stored_entry_by_entry(n, d, dtype, flags):
    lib = _lib.load()
    b, h = 2, 3
    q, k, v, do, bias = _problem(b, h, n, d, dtype)
    out, row_m, row_z = E.twopass_attention_with_state(q, k, v, bias=bias)
    dq, dk, dv = (torch.full_like(q, float("nan")) for _ in range(3))
    dbias = torch.full_like(bias, float("nan"))
    dt = _lib.dtype_code(dtype)
    need = lib.elsa_backward_workspace_bytes(dt, b, h, n, d, 1, 0, flags)
    ws = torch.empty(max(need, 256), device="cuda", dtype=torch.uint8)
    strides = bias.stride()
    rc = lib.elsa_twopass_backward(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), do.data_ptr(), row_m.data_ptr(), row_z.data_ptr(),
                                   bias.data_ptr(), *strides, dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dbias.data_ptr(), *strides,
                                   ws.data_ptr(), ws.numel(), dt, b, h, n, d, 0, flags, _lib.raw_stream(q.device))
    assert rc == 0
    for g, w in zip((dq, dk, dv, dbias), _fp64(q, k, v, bias, do)):
        if n == 1:                                   # one key: P = 1, dS = 0, and only dv is not 0
            assert (g.double() - w).abs().max() <= LIMIT[dtype] * do.abs().max()
        else:
            assert (g.double() - w).norm() <= LIMIT[dtype] * w.norm()


@pytest.mark.parametrize("n,d", [(49, 32), (130, 64), (640, 40), (513, 128)])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shared", [False, True])
def test_rows_without_a_key_get_zero_gradients(n, d, dtype, shared):
    q, k, v, do, bias = _problem(2, 2, n, d, dtype)
    if shared:
        bias = bias[:1].clone()
    rows = [0, 7, n // 2, n - 1]
    bias[..., rows, :] = float("-inf")
    bias[..., 3, : n - 1] = float("-inf")             # and one row with a single key
    x = [t.detach().requires_grad_(True) for t in (q, k, v, bias)]
    got = torch.autograd.grad(E.twopass_attention_train(x[0], x[1], x[2], bias=x[3]), x, do)
    assert float(got[0][:, :, rows].abs().max()) == 0.0 and float(got[3][..., rows, :].abs().max()) == 0.0
    # against fp64 with those rows taken out of the problem
    keep = torch.ones(n, device="cuda", dtype=torch.bool)
    keep[rows] = False
    y = [t.detach().double().requires_grad_(True) for t in (q, k, v, bias)]
    s = y[0][:, :, keep] @ y[1].mT * d ** -0.5 + y[3][..., keep, :]
    want = torch.autograd.grad(torch.softmax(s, -1) @ y[2], y, do.double()[:, :, keep])
    for g, w in zip(got, want):
        assert torch.isfinite(g).all()
        assert (g.double() - w).norm() <= LIMIT[dtype] * w.norm()


@pytest.mark.parametrize("n,part_width", [(512, 0), (516, 128), (520, 0), (527, 256), (639, 128), (1025, 384)])
@pytest.mark.parametrize("form", ["rows", "offset", "transposed"])
@pytest.mark.parametrize("causal", [False, True])
def test_fp32_tensor_core_fold_reads_a_bias_of_any_alignment(n, part_width, form, causal):
    """16 keys at a time: whole sectors on 32-byte boundaries, single loads off them, clamped ones at a partition's end and for a
    bias whose keys are not contiguous (C ABI only)."""
    lib = _lib.load()
    b, h, d = 1, 2, 64
    q, k, v, _, bias = _problem(b, h, n, d, torch.float32)
    if form == "offset":
        bias = torch.cat([bias.new_zeros(1), bias.reshape(-1)])[1:].view_as(bias)
    elif form == "transposed":
        bias = bias.mT.contiguous().mT
    out, row_m, row_z = torch.full_like(q, float("nan")), q.new_empty(b * h, n), q.new_empty(b * h, n)
    need = lib.elsa_forward_workspace_bytes(0, 0, b, h, n, d, 1, int(causal), part_width, 0, 0)
    ws = torch.empty(max(need, 256), device="cuda", dtype=torch.uint8)
    rc = lib.elsa_twopass_forward(q.data_ptr(), k.data_ptr(), v.data_ptr(), bias.data_ptr(), *bias.stride(), out.data_ptr(), row_m.data_ptr(),
                                  row_z.data_ptr(), ws.data_ptr(), ws.numel(), 0, 0, b, h, n, d, int(causal), part_width, 0, 0, _lib.raw_stream(q.device))
    assert rc == 0
    s = q.double() @ k.double().mT * d ** -0.5 + bias.double()
    if causal:
        s = s.masked_fill(torch.ones(n, n, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    want = torch.softmax(s, -1) @ v.double()
    assert (out.double() - want).norm() <= 1e-6 * want.norm()      # the bound of the unbiased fold


@pytest.mark.parametrize("n,d", [(516, 64), (640, 64), (1025, 40), (130, 64)])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("form", ["rows", "offset", "transposed"])
def test_a_dense_gradient_of_any_alignment(n, d, dtype, form):
    """As `test_a_dense_gradient_is_stored_entry_by_entry`, with bias and gradient off 16-byte boundaries or key by key."""
    lib = _lib.load()
    b, h = 1, 2
    q, k, v, do, bias = _problem(b, h, n, d, dtype)
    out, row_m, row_z = E.twopass_attention_with_state(q, k, v, bias=bias)

    def laid_out(t):
        if form == "offset":
            return torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view_as(t)
        return t.mT.contiguous().mT if form == "transposed" else t

    used, dbias = laid_out(bias), laid_out(torch.full_like(bias, float("nan")))
    dq, dk, dv = (torch.full_like(q, float("nan")) for _ in range(3))
    dt = _lib.dtype_code(dtype)
    ws = torch.empty(max(lib.elsa_backward_workspace_bytes(dt, b, h, n, d, 1, 0, 0), 256), device="cuda", dtype=torch.uint8)
    rc = lib.elsa_twopass_backward(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), do.data_ptr(), row_m.data_ptr(), row_z.data_ptr(),
                                   used.data_ptr(), *used.stride(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dbias.data_ptr(), *dbias.stride(),
                                   ws.data_ptr(), ws.numel(), dt, b, h, n, d, 0, 0, _lib.raw_stream(q.device))
    assert rc == 0
    for g, w in zip((dq, dk, dv, dbias), _fp64(q, k, v, bias, do)):
        assert (g.double() - w).norm() <= LIMIT[dtype] * w.norm()
