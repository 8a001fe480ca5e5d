"""Which scratch an attention call gets: host-side rules, with CPU buffers in the place of device memory."""

import types

import pytest
import torch


class Cuda:
    """The current stream and its capture state, as the code under test sees them."""

    stream = 11
    capturing = False


@pytest.fixture
def cuda(monkeypatch):
    from chitudiffusion_b200 import ops

    state = Cuda()
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: types.SimpleNamespace(cuda_stream=state.stream))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state.capturing)
    monkeypatch.setattr(ops, "_stream_ptr", lambda dev: state.stream)
    monkeypatch.setattr(ops, "_device_key", lambda dev: dev.index or 0)
    monkeypatch.setattr(ops, "_on", lambda dev: ops._NO_GUARD)
    monkeypatch.setattr(ops, "_workspaces", {})
    monkeypatch.setattr(ops, "_retired_workspaces", [])
    monkeypatch.setattr(ops, "_cut_scratches", {})
    return state


CPU = torch.device("cpu")


def _header_is_zero(ws):
    return int(ws[:65536].max()) == 0


def test_a_cut_never_uses_the_key_split_buffer(cuda):
    """The key-split buffer of a stream may be part of a captured graph that is replayed beside eager calls."""
    from chitudiffusion_b200 import ops

    split = ops.splitkv_workspace(CPU, 50 << 20)  # larger than any cut needs
    cut = ops._cut_scratch(CPU, 1 << 20)
    assert cut.data_ptr() != split.data_ptr()
    assert _header_is_zero(cut)
    assert ops._cut_scratch(CPU, 30 << 20) is cut  # made once, at the size of the largest cut
    assert not ops._retired_workspaces


def test_the_cut_pool_is_bounded(cuda):
    from chitudiffusion_b200 import ops

    seen = {}
    for stream in range(3 * ops.CUT_SCRATCH_STREAMS):
        cuda.stream = stream
        seen[stream] = ops._cut_scratch(CPU, 1 << 20)
    assert len(ops._cut_scratches) == ops.CUT_SCRATCH_STREAMS
    assert len({t.data_ptr() for t in ops._cut_scratches.values()}) == ops.CUT_SCRATCH_STREAMS
    assert ops._cut_scratch(CPU, 1 << 20) is seen[stream]
    # 148 bundles, two fragments of two 128-row tiles each
    assert ops.CUT_SCRATCH_BYTES == 65536 + 148 * 2 * 2 * 128 * 129 * 4


def test_a_captured_split_call_has_scratch_of_its_own(cuda):
    from chitudiffusion_b200 import ops

    eager = ops._split_scratch(CPU, 2 << 20)
    assert ops._split_scratch(CPU, 2 << 20) is eager  # eager calls of a stream share one buffer
    cuda.capturing = True
    first, second = ops._split_scratch(CPU, 2 << 20), ops._split_scratch(CPU, 3 << 20)
    assert len({t.data_ptr() for t in (eager, first, second)}) == 3
    assert _header_is_zero(first) and first.numel() >= 2 << 20
    # what a capture zeroes is not zero before the first replay: nothing of it reaches an eager call
    cuda.capturing = False
    cuda.stream = 12
    before = dict(ops._workspaces)
    cuda.capturing = True
    ops._split_scratch(CPU, 2 << 20)
    assert ops._workspaces == before and not ops._cut_scratches


def test_a_reported_timeout_takes_the_scratch_out_of_use(cuda, monkeypatch):
    """The call that gave up may have left counters behind; the next one must not find them."""
    import ctypes

    from chitudiffusion_b200 import _lib, ops

    monkeypatch.setattr(torch.cuda, "synchronize", lambda dev=None: None)
    word = ctypes.c_int32(0)
    monkeypatch.setattr(ops, "_status_words", {0: (None, word), 1: (None, ctypes.c_int32(0))})
    split, cut = ops.splitkv_workspace(CPU, 1 << 20), ops._cut_scratch(CPU, 1 << 20)
    ops._cut_scratches[(1, 5)] = other = torch.empty(8, dtype=torch.uint8)
    ops.poll_status(torch.device("cuda", 0))  # nothing reported: the buffers stay
    assert ops._cut_scratch(CPU, 1 << 20) is cut and ops.splitkv_workspace(CPU, 1 << 20) is split
    for raising in (ops.poll_status, ops.check_status):
        for ws in (split, cut):
            ws[:4].fill_(1)
        word.value = 3
        with pytest.raises(_lib.ChituB200Error, match="softmax"):
            raising(torch.device("cuda", 0))
        assert word.value == 0
        fresh_split, fresh_cut = ops.splitkv_workspace(CPU, 1 << 20), ops._cut_scratch(CPU, 1 << 20)
        assert _header_is_zero(fresh_split) and _header_is_zero(fresh_cut)
        split, cut = fresh_split, fresh_cut
    assert ops._cut_scratches[(1, 5)] is other  # another device's buffers are not touched


def test_a_callers_buffer_that_will_not_do_is_left_alone():
    """Too small, off its alignment or with gaps: the call runs its query blocks whole instead of being refused."""
    from chitudiffusion_b200 import ops

    raw = torch.zeros(4096 + 64, dtype=torch.uint8)
    base = raw[(-raw.data_ptr()) % 16:][:4096]
    assert ops._holds(base, 4096, CPU)
    assert not ops._holds(base, 4097, CPU)
    assert not ops._holds(raw[(-raw.data_ptr()) % 16 + 8:], 1024, CPU)
    assert not ops._holds(base.view(64, 64)[:, :32], 1024, CPU)
    assert not ops._holds(base, 1024, torch.device("cuda", 0))
