"""The 32-bit attention's scratch, without a GPU: what a step asks the workspace for, and that its passes serve every token."""

import pytest
import torch

from jax_llm_examples_b200.kernels import api as K
from jax_llm_examples_b200.parts import LayerCache, PagedAttention, Runtime, StepContext
from jax_llm_examples_b200.parts.attention import plan_attention_tiles
from jax_llm_examples_b200.parts.base import StepShape

LIMIT = 1 << 26  # float32 elements: 256 MB


class Asked:
    def __init__(self):
        self.most = {}

    def get(self, name, numel, dtype):
        self.most[name] = max(self.most.get(name, 0), numel)
        return torch.empty(numel, dtype=dtype, device="meta")


@pytest.mark.parametrize("heads, kv_heads", [(16, 4), (40, 8), (32, 1)])
@pytest.mark.parametrize("lens, kv", [([2048, 1], 131072), ([1], 131072), ([1] * 5, 1 << 20), ([17, 1, 1, 30], 65536), ([128], 65536), ([512], 65536),
                                      ([5], 1 << 21), ([2048], 2048), ([300, 1], 700)])
def test_the_partial_results_of_a_step_are_bounded(monkeypatch, heads, kv_heads, lens, kv):
    calls, dh, asked = [], 128, Asked()
    monkeypatch.setattr(K, "sm_count", lambda: 148)
    monkeypatch.setattr(K, "attention_f32_supported", lambda *a: True)
    monkeypatch.setattr(K, "attention_mma_supported", lambda *a: False)

    def attention_f32(q, pages, bt, req, pos, out, scale, chunk, window, a, f, status, n_items, items, max_count, rows, splits, per_split, part_o, part_ml, *rest):
        assert q.shape[0] == out.shape[0] == req.shape[0] == pos.shape[0]
        ranges = -(-kv // 256)
        if splits > 1:
            kept = min(q.shape[0], n_items * max_count) * heads * splits * per_split
            assert splits * per_split >= ranges and part_o.numel() >= kept * dh and part_ml.numel() >= kept * 2
        calls.append([(int(x), int(c)) for x, c in items.view(-1, 2)] if items is not None else
                     [(int(x), 1) for x in (rows if rows is not None else pos)])
        assert len(calls[-1]) == n_items

    monkeypatch.setattr(K, "attention_f32", attention_f32)
    n, rows = sum(lens), (heads + 2 * kv_heads) * dh
    mixer = PagedAttention(torch.empty(rows, 1, device="meta"), torch.empty(1, heads * dh, device="meta"), heads, kv_heads, dh, None)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32)  # noqa: E731
    ctx = StepContext(Runtime(torch.float32, torch.device("cpu")), n, len(lens), i32([0] * n), i32(list(range(n))), i32([0] * n), i32([0]), i32([0]), i32(lens),
                      i32([0]), i32([]), 0, i32([0]), max_q_len=max(lens), max_kv_len=kv, workspace=asked)
    for name, a in plan_attention_tiles(StepShape(tuple(lens), (0,) * len(lens), 64, kv)).items():
        ctx.host_arrays[name], ctx.arrays[name] = a, i32(a.reshape(-1).tolist())
    q = torch.empty(n, heads, dh, device="meta")
    for workspace in (asked, None):  # a step made by hand may have no workspace: its scratch is made for the call
        ctx.workspace = workspace
        calls.clear()
        mixer.attend(ctx, q, LayerCache(None, None, True, None), torch.empty_like(q), 0.0, 1.0)
        served = sorted(row + i for call in calls for row, count in call for i in range(count))
        assert served == list(range(n))
    assert sum(asked.most.values()) <= LIMIT + LIMIT // 32
