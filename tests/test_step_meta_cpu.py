"""Step metadata from Python lengths against a plain statement, under any default device."""
import pytest
import torch

from tensorrt_edge_llm_b200.ops import build_step_meta


def _plain(q_lens, pasts):
    start = [sum(q_lens[:i]) for i in range(len(q_lens) + 1)]
    return start, [p + j for q, p in zip(q_lens, pasts) for j in range(q)], [i for i, q in enumerate(q_lens) for _ in range(q)]


@pytest.mark.parametrize("q_lens,pasts", [([1], [0]), ([3, 0, 2], [5, 7, 0]), ([1] * 9, list(range(9))), ([700, 1], [64, 3]), ([], [])])
def test_step_meta_matches_lists(q_lens, pasts):
    n = len(q_lens)
    start, pos, sid = _plain(q_lens, pasts)
    table = torch.arange(4 * n, dtype=torch.int64).reshape(n, 4)
    m = build_step_meta(q_lens, pasts, table, 64, slot_ids=[n - i for i in range(n)])
    for got, want in ((m.q_start, start), (m.q_len, q_lens), (m.past_len, pasts), (m.positions, pos), (m.seq_ids, sid),
                      (m.slot_ids, [n - i for i in range(n)]), (m.logits_idx, [s - 1 for s in start[1:]])):
        assert got.dtype == torch.int32 and got.tolist() == want
    assert torch.equal(m.page_table.long(), table) and m.page_table.dtype == torch.int32
    assert (m.num_seqs, m.num_tokens, m.max_q_len, m.host_lens) == (n, sum(q_lens), max(q_lens, default=0), tuple(zip(q_lens, pasts)))
    assert build_step_meta(q_lens, pasts, table, 64, logits_all=True).logits_idx.tolist() == list(range(sum(q_lens)))
    assert build_step_meta(q_lens, pasts, table, 64, logits_rows=[2, 0]).logits_idx.tolist() == [2, 0]
    assert build_step_meta(q_lens, pasts, table, 64, positions=[7] * sum(q_lens)).positions.tolist() == [7] * sum(q_lens)


def test_step_meta_under_a_default_device():
    """The host's part stays on the host wherever new tensors go by default; no device given means that one."""
    table = torch.zeros(2, 3, dtype=torch.int32)
    with torch.device("meta"):
        m = build_step_meta([1, 2], [3, 4], table, 64, device="cpu")
        assert build_step_meta([1, 2], [3, 4], table, 64, device=None).positions.device.type == "meta"
    assert m.positions.tolist() == [3, 4, 5]
    assert build_step_meta([1, 2], [3, 4], table, 64, device=None).positions.tolist() == [3, 4, 5]


@pytest.mark.gpu
@pytest.mark.parametrize("q_lens,pasts", [([1], [0]), ([3, 0, 2], [5, 7, 0]), ([700, 1], [64, 3])])
def test_step_meta_on_the_gpu_equals_the_host(q_lens, pasts):
    table = torch.arange(5 * len(q_lens), dtype=torch.int32).reshape(len(q_lens), 5)
    a = build_step_meta(q_lens, pasts, table, 64)
    with torch.device("cuda"):
        metas = [build_step_meta(q_lens, pasts, t, 64, device=d) for t in (table, table.cuda()) for d in ("cuda", 0, None)]
    for m in metas:
        for f in ("q_start", "q_len", "past_len", "positions", "seq_ids", "page_table", "slot_ids", "logits_idx"):
            t = getattr(m, f)
            assert t.is_cuda and torch.equal(t.cpu(), getattr(a, f)), f
