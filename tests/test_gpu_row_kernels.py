"""Row forms of the block's elementwise kernels at the sizes where their dispatch changes, against fp64 torch.

Tolerances: the result differs from fp64 by its own rounding (half an ulp: at most 2^-8 of the value for bf16, 2^-11 for fp16, 2^-24 for
fp32) plus fp32 arithmetic on values of order one (1e-5)."""

import pytest
import torch

pytestmark = pytest.mark.gpu

ULP = {torch.bfloat16: 2 ** -7, torch.float16: 2 ** -10, torch.float32: 2 ** -23}  # spacing at one


def _close(got, ref, dtype):
    got = got.double().cpu()
    assert torch.isfinite(got).all()
    assert ((got - ref).abs() <= 0.51 * ULP[dtype] * ref.abs() + 2e-5).all(), (got - ref).abs().max().item()


# columns: below / at / above one block's vectors, odd vector counts, two vectors per thread, beyond the column form
@pytest.mark.parametrize("C", [64, 508, 512, 1000, 1536, 3080, 4096, 5120, 8192])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("B,L", [(1, 1), (2, 5), (3, 130)])
def test_layernorm_and_gate(C, dtype, B, L):
    from chitudiffusion_b200 import ops

    gen = torch.Generator().manual_seed(C + L)
    x = (torch.randn(B, L, C, generator=gen) * 2 + 0.5).to(dtype)
    mul, add, gate = (torch.randn(B, C, generator=gen) for _ in range(3))
    y = torch.randn(B, L, C, generator=gen).to(torch.float16 if dtype == torch.float16 else torch.bfloat16)
    xd = x.double()
    norm = (xd - xd.mean(-1, keepdim=True)) / (xd.var(-1, unbiased=False, keepdim=True) + 1e-6).sqrt()
    out = ops.layernorm_modulate(x.cuda(), mul.cuda(), add.cuda(), add_one=True)
    _close(out, norm * (1 + mul.double()[:, None]) + add.double()[:, None], torch.bfloat16)
    _close(ops.layernorm_modulate(x.cuda(), out_dtype=torch.float16), norm, torch.float16)
    xc = x.cuda()
    ops.gate_residual(xc, y.cuda(), gate.cuda())
    _close(xc, xd + y.double() * gate.double()[:, None], dtype)
    xc = x.cuda()
    ops.gate_residual(xc, y.cuda())
    _close(xc, xd + y.double(), dtype)


def test_gate_of_a_branch_at_an_odd_address():
    """y eight bytes off a 16-byte boundary is accepted and takes the general kernel."""
    from chitudiffusion_b200 import ops

    flat = torch.randn(4 + 3 * 256, dtype=torch.float32).to(torch.bfloat16).cuda()
    y = flat[4:].view(1, 3, 256)
    x = torch.randn(1, 3, 256).cuda()
    ref = x.double().cpu() + y.double().cpu()
    ops.gate_residual(x, y)
    _close(x, ref, torch.float32)


@pytest.mark.parametrize("B,S,H", [(1, 1, 1), (2, 3, 5), (1, 130, 12), (3, 257, 7)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_lse_combine_rows(B, S, H, dtype):
    from chitudiffusion_b200 import ops

    gen = torch.Generator().manual_seed(S)
    outs = [torch.randn(B, S, H, 128, generator=gen).to(dtype) for _ in range(3)]
    lses = [torch.randn(B, H, S, generator=gen) * 4 for _ in range(3)]
    acc = torch.empty(B, S, H, 128, device="cuda")
    acc_lse = torch.empty(B, S, H, 1, device="cuda")
    for i in range(3):
        ops.lse_combine(acc, acc_lse, outs[i].cuda(), lses[i].cuda(), first=i == 0)
    l64 = torch.stack([l.double().permute(0, 2, 1).unsqueeze(-1) for l in lses])
    w = torch.softmax(l64, 0)
    ref = sum(w[i] * outs[i].double() for i in range(3))
    assert (acc.double().cpu() - ref).abs().max().item() <= 2e-6 * ref.abs().max().item() + 1e-6
    assert (acc_lse.double().cpu() - torch.logsumexp(l64, 0)).abs().max().item() <= 1e-5


# where the dispatch changes hands: narrow rows, few and many; one and two rows in very many batches (a warp's and a
# block's worth of columns); fp32 rows of 512 vectors below and above the machine's fill; a last batch that is not whole
@pytest.mark.parametrize("C,dtype,B,L", [
    (128, torch.float32, 1, 300), (128, torch.float32, 1, 2048), (256, torch.bfloat16, 3, 700), (1536, torch.float32, 400, 1),
    (3072, torch.bfloat16, 400, 2), (3072, torch.float32, 160, 1), (5120, torch.bfloat16, 160, 1), (2048, torch.float32, 1, 1499),
    (2048, torch.float32, 3, 501), (4096, torch.bfloat16, 1, 1600), (512, torch.float32, 520, 3), (1024, torch.bfloat16, 520, 3),
    (64, torch.float16, 700, 2),
])
def test_layernorm_and_gate_where_forms_change(C, dtype, B, L):
    test_layernorm_and_gate(C, dtype, B, L)
