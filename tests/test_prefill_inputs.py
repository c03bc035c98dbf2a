"""Inputs of a prefill chunk (ModelRunner._prefill_inputs) and the pinned buffers they are staged in."""
from types import SimpleNamespace

import pytest
import torch

from skein_b200.runtime.runner import ModelRunner, _Staging


def _runner(device, slots=0, blocks=6):
    return ModelRunner(SimpleNamespace(device=torch.device(device), num_state_slots=slots), max_blocks_per_seq=blocks, use_graphs=False)


def _check(inp, seqs, blocks, want=None, slots=None):
    lens = [len(s[0]) for s in seqs]
    start = [sum(lens[:i]) for i in range(len(seqs))]
    flat = lambda v: [int(x) for x in v]      # noqa: E731
    assert flat(inp.token_ids) == [int(t) for s in seqs for t in s[0]]
    assert flat(inp.positions) == [s[2] + i for s in seqs for i in range(len(s[0]))]
    assert flat(inp.seq_of_token) == [i for i, n in enumerate(lens) for _ in range(n)]
    assert flat(inp.q_start) == start and flat(inp.q_len) == lens and flat(inp.seq_lens) == [s[2] + n for s, n in zip(seqs, lens)]
    assert flat(inp.kv_start) == [sum(s[2] + len(s[0]) for s in seqs[:i]) for i in range(len(seqs))]
    assert (inp.max_q_len, inp.kv_total, inp.max_cached) == (max(lens), sum(s[2] + n for s, n in zip(seqs, lens)), max(s[2] for s in seqs))
    assert inp.block_table.tolist() == [[int(b) for b in s[1]] + [0] * (blocks - len(s[1])) for s in seqs]
    assert inp.logit_rows.dtype == torch.int64
    assert flat(inp.logit_rows) == ([a + n - 1 for a, n in zip(start, lens)] if want is None else [start[i] + j for i, w in enumerate(want) for j in w])
    assert (inp.slots is None) if slots is None else flat(inp.slots) == slots


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_forms(device):
    """Tokens and pages as lists and as tensors, several wanted places of a sequence and none, given state slots and default ones."""
    seqs = [([5, 6, 7], [2, 1], 4), (torch.tensor([9]), torch.tensor([3, 4, 5], dtype=torch.int32), 33), (tuple(range(20)), (0,), 0)]
    r = _runner(device)
    _check(r._prefill_inputs(seqs, None)[0], seqs, 6)
    _check(r._prefill_inputs(seqs, None, [[0, 2], [], [19]])[0], seqs, 6, [[0, 2], [], [19]])
    s = _runner(device, slots=8)
    _check(s._prefill_inputs(seqs, None)[0], seqs, 6, slots=[0, 1, 2])
    given = [(*q, i) for q, i in zip(seqs, (7, 0, 3))]
    _check(s._prefill_inputs(given, None)[0], given, 6, slots=[7, 0, 3])
    with pytest.raises(Exception):
        r._prefill_inputs([([1], list(range(7)), 0)], None)          # more pages than the table holds


def test_cpu_inputs_of_two_chunks_are_apart():
    r = _runner("cpu")
    a, b = [([1, 2], [0], 0)], [([3, 4], [1], 5)]
    x, y = r._prefill_inputs(a, None)[0], r._prefill_inputs(b, None)[0]
    _check(x, a, 6)
    _check(y, b, 6)


def _chunk(i, n):
    return [(list(range(100 * i, 100 * i + n)), [i, i + 1], i), ([7 * i], [i + 2], 2 * i)]


@pytest.mark.gpu
def test_a_chunk_takes_no_pinned_memory_of_its_own(monkeypatch):
    r = _runner("cuda")
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **kw: pytest.fail("pinned allocation") if kw.get("pin_memory") else empty(*a, **kw))
    for i, n in enumerate((37, 4000, 1, 37)):
        seqs = _chunk(i, n)
        _check(r._prefill_inputs(seqs, None)[0], seqs, 6)
        torch.cuda.synchronize()


@pytest.mark.gpu
def test_chunks_behind_a_busy_device():
    """Their copies wait, so that a buffer taken too early would be overwritten; more chunks than the ring holds, and one larger than its buffers."""
    r, got = _runner("cuda"), []
    torch.cuda._sleep(40_000_000)
    for i in range(_Staging.RING - 1):
        seqs = _chunk(i, 50 + i)
        got.append((seqs, r._prefill_inputs(seqs, None)[0]))
    assert len(r.staging.ring) > 2
    for i, n in enumerate((40, 25000, 30, 20, 10), start=20):
        seqs = _chunk(i, n)
        got.append((seqs, r._prefill_inputs(seqs, None)[0]))
    assert len(r.staging.ring) <= _Staging.RING
    for seqs, inp in got:
        _check(inp, seqs, 6)


@pytest.mark.gpu
def test_one_buffer_grows_for_large_chunks():
    r = _runner("cuda")
    for i in range(3):
        seqs = _chunk(i, 30000)
        _check(r._prefill_inputs(seqs, None)[0], seqs, 6)
        torch.cuda.synchronize()
    assert [s[0].numel() > _Staging.WORDS for s in r.staging.ring] == [True]
