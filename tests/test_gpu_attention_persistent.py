"""The persistent attention kernel: several query blocks per CTA, and blocks cut along the keys and merged.

Tolerances as in test_gpu_attention.py (bf16 inputs, fp32 oracle on the same inputs); two schedules of the same
arithmetic differ by the 16-bit rounding of the result (2^-8 relative) at most.
"""

import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _inputs(B, Sq, Sk, H, dtype, seed):
    gen = torch.Generator().manual_seed(seed)
    return (torch.randn(B, Sq, H, 128, generator=gen).to(dtype), torch.randn(B, Sk, H, 128, generator=gen).to(dtype),
            torch.randn(B, Sk, H, 128, generator=gen).to(dtype))


def _need(B, Sq, Sk, H):
    from chitudiffusion_b200 import _lib

    return int(_lib.load().chitu_b200_attn_balanced_workspace_bytes(B, Sq, Sk, H))


# (B, Sq, Sk, H, dtype, cut): one key tile per block (masked and full); many blocks per CTA; a last block of one tile;
# cut last waves whose bundles start inside, end inside and span two blocks
@pytest.mark.parametrize("B,Sq,Sk,H,dtype,cut", [
    (1, 2500, 77, 40, torch.bfloat16, False),
    (2, 1100, 128, 37, torch.float16, False),
    (1, 4097, 129, 24, torch.bfloat16, False),
    (1, 1100, 1500, 37, torch.bfloat16, True),
    (1, 1300, 1409, 26, torch.float16, True),
    (2, 513, 2049, 50, torch.bfloat16, True),
])
def test_matches_the_oracle(B, Sq, Sk, H, dtype, cut):
    from chitudiffusion_b200 import ops

    q, k, v = _inputs(B, Sq, Sk, H, dtype, Sq + Sk)
    ref, ref_lse = oracle.sdpa_fp32(q, k, v, return_lse=True)
    assert (_need(B, Sq, Sk, H) > 0) == cut
    qc, kc, vc = q.cuda(), k.cuda(), v.cuda()
    ws = torch.zeros(max(_need(B, Sq, Sk, H), 65536), dtype=torch.uint8, device="cuda")
    for _ in range(2):  # the second call finds the first one's scratch
        out, lse = ops.attn_fwd(qc, kc, vc, return_lse=True, workspace=ws)
        assert (out.float().cpu() - ref).abs().max().item() <= 2e-2 * ref.abs().max().item()
        assert (lse.cpu() - ref_lse).abs().max().item() <= 1e-3
    assert int(ws[:65536].max().item()) == 0  # the counters are back at zero
    whole, lse1 = ops.attn_fwd(qc, kc, vc, return_lse=True, n_splits=1)
    assert (out.float() - whole.float()).abs().max().item() <= 2 ** -7 * ref.abs().max().item()
    assert (lse - lse1).abs().max().item() <= 1e-4
    ops.check_status()


def test_a_fragment_without_a_finite_score_carries_no_weight():
    """Keys whose scores are -inf for every row: wherever the cuts fall, the others decide alone."""
    from chitudiffusion_b200 import ops

    q, k, v = _inputs(1, 1100, 1500, 37, torch.bfloat16, 3)
    q[..., 0] = 1.0
    for lo, hi in ((0, 700), (900, 1500), (128, 256)):
        kk = k.clone()
        kk[:, lo:hi, :, 0] = float("-inf")
        keep = torch.tensor([i for i in range(1500) if not lo <= i < hi])
        ref, ref_lse = oracle.sdpa_fp32(q, kk[:, keep], v[:, keep], return_lse=True)
        for n_splits in (None, 1, 2, 3):
            out, lse = ops.attn_fwd(q.cuda(), kk.cuda(), v.cuda(), return_lse=True, n_splits=n_splits)
            assert (out.float().cpu() - ref).abs().max().item() <= 2e-2 * ref.abs().max().item()
            assert (lse.cpu() - ref_lse).abs().max().item() <= 1e-3


def test_a_row_without_any_finite_score_is_undefined():
    from chitudiffusion_b200 import ops

    q, k, v = _inputs(1, 1100, 1500, 37, torch.bfloat16, 5)
    q[..., 0] = 1.0
    k[..., 0] = float("-inf")
    for n_splits in (None, 1, 3):
        out, _ = ops.attn_fwd(q.cuda(), k.cuda(), v.cuda(), n_splits=n_splits)
        assert torch.isnan(out).all()


def test_a_captured_call_keeps_its_query_blocks_whole():
    """Inside a capture no scratch of the stream is used: a replay may run beside eager calls that use it."""
    from chitudiffusion_b200 import ops

    q, k, v = (t.cuda() for t in _inputs(1, 1100, 1500, 37, torch.bfloat16, 4))
    whole, _ = ops.attn_fwd(q, k, v, n_splits=1)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ops.attn_fwd(q, k, v)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out, _ = ops.attn_fwd(q, k, v)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, whole)


def test_a_replayed_key_split_call_beside_eager_cut_calls():
    """A graph captured on one stream, replayed on another beside eager calls of the first: no scratch in common, and
    none of it is first zeroed by the replay."""
    from chitudiffusion_b200 import ops

    q, k, v = (t.cuda() for t in _inputs(1, 300, 1500, 5, torch.bfloat16, 6))
    big = [t.cuda() for t in _inputs(1, 1100, 1500, 37, torch.bfloat16, 7)]
    want, _ = ops.attn_fwd(q, k, v, n_splits=3)
    want_big, _ = ops.attn_fwd(*big)
    torch.cuda.synchronize()
    one, other = torch.cuda.Stream(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=one):  # the stream's first key-split call is a captured one
        out, _ = ops.attn_fwd(q, k, v, n_splits=3)
    with torch.cuda.stream(one):
        early, _ = ops.attn_fwd(q, k, v, n_splits=3)
    torch.cuda.synchronize()
    assert torch.equal(early, want)
    for _ in range(4):
        with torch.cuda.stream(one):
            eager = [ops.attn_fwd(*big)[0] for _ in range(4)]
        with torch.cuda.stream(other):
            for _ in range(8):
                graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
        assert all(torch.equal(e, want_big) for e in eager)
    ops.check_status()


def test_any_workspace_is_taken_by_a_call_on_one_key_range():
    from chitudiffusion_b200 import ops

    q, k, v = (t.cuda() for t in _inputs(1, 1100, 1500, 37, torch.bfloat16, 8))
    whole, _ = ops.attn_fwd(q, k, v, n_splits=1)
    big = torch.zeros(2 * _need(1, 1100, 1500, 37) + 16, dtype=torch.uint8, device="cuda")
    for ws in (big[8:], big[:16], big.view(-1, 2)[:, 0], torch.zeros(0, dtype=torch.uint8, device="cuda")):
        out, _ = ops.attn_fwd(q, k, v, workspace=ws)
        assert torch.equal(out, whole)
    assert int(big.max().item()) == 0


# fewer bundles than SMs behind one, two and three waves of whole blocks; one bundle per SM; one-tile query blocks among the cut
@pytest.mark.parametrize("B,Sq,Sk,H", [(1, 2560, 2100, 15), (1, 2500, 1700, 30), (1, 3840, 1800, 31), (1, 1500, 2500, 37), (2, 300, 2200, 40)])
def test_bundles_behind_whole_blocks(B, Sq, Sk, H):
    from chitudiffusion_b200 import ops

    q, k, v = _inputs(B, Sq, Sk, H, torch.bfloat16, Sq)
    ref, ref_lse = oracle.sdpa_fp32(q, k, v, return_lse=True)
    need = _need(B, Sq, Sk, H)
    assert need > 0
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
    ws[65536:] = 0xff  # NaN wherever a fragment is read that was not written
    for _ in range(2):
        out, lse = ops.attn_fwd(q.cuda(), k.cuda(), v.cuda(), return_lse=True, workspace=ws)
        assert (out.float().cpu() - ref).abs().max().item() <= 2e-2 * ref.abs().max().item()
        assert (lse.cpu() - ref_lse).abs().max().item() <= 1e-3
    assert int(ws[:65536].max().item()) == 0
    ops.check_status()


def test_a_cut_that_does_not_pay_is_not_taken():
    """Few key tiles: two epilogues and the merge cost more than the last wave's idle SMs."""
    assert _need(1, 1664, 1100, 24) == 0  # 168 blocks x 9 tiles: 39 us whole, 46 us cut
    assert _need(1, 2560, 2048, 24) == 0  # 240 x 16: 64, 67
    assert _need(1, 4608, 4608, 24) == 0  # 432 x 36: 202, 213
    assert _need(1, 2560, 8192, 15) > 0  # 150 x 64: 209, 140


def test_two_streams_cut_at_once():
    from chitudiffusion_b200 import ops

    sets = [[t.cuda() for t in _inputs(1, 1100, 1500, 37, torch.bfloat16, seed)] for seed in (11, 12)]
    want = [ops.attn_fwd(*s)[0] for s in sets]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in sets]
    outs = [[], []]
    for _ in range(8):
        for i, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                outs[i].append(ops.attn_fwd(*sets[i])[0])
    torch.cuda.synchronize()
    for i in range(2):
        assert all(torch.equal(o, want[i]) for o in outs[i])
    ops.check_status()


@pytest.mark.parametrize("H,n_splits", [(40, None), (2, 3)])
def test_the_first_call_of_a_process_may_be_a_captured_one(H, n_splits):
    """Status word and scratch come into being inside the capture; a child process, so that this is its first call."""
    import os
    import subprocess
    import sys

    code = f"""
import torch
from chitudiffusion_b200 import ops
q, k, v = (torch.randn(1, s, {H}, 128, device="cuda").bfloat16() for s in (1100, 1500, 1500))
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    out, _ = ops.attn_fwd(q, k, v, n_splits={n_splits})
graph.replay()
torch.cuda.synchronize()
ref, _ = ops.attn_fwd(q, k, v, n_splits=1)
assert (out.float() - ref.float()).abs().max().item() <= 2 ** -7 * ref.float().abs().max().item()
ops.check_status()
"""
    root = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
    done = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
