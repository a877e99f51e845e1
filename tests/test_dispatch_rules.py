"""The host-side rules that choose a kernel or a split, at the sizes where the choice was measured to matter."""
import types

import pytest


def _splits(rows, pages, kv_heads=8):
    from openagents_b200.models.paged import PagedEngine
    return PagedEngine._attn_splits(types.SimpleNamespace(attn_target_ctas=0, max_splits=64), rows // kv_heads, kv_heads, pages)


# us by split count, 32 query heads on 8 of size 128 (rows = sequences x 8) unless said otherwise
MEASURED = {
    (8, 32): {1: 8.66, 2: 8.20, 4: 6.84, 8: 6.36}, (8, 128): {1: 26.85, 5: 10.45, 8: 8.46, 12: 8.65, 16: 8.74, 24: 9.84},
    (56, 63): {1: 15.00, 2: 12.42, 4: 10.90, 6: 10.91, 12: 14.14}, (56, 128): {1: 27.25, 3: 17.80, 5: 14.76, 6: 14.11, 7: 15.12, 12: 17.49},
    (128, 40): {1: 12.78, 3: 11.70, 4: 15.57, 6: 14.96}, (128, 94): {1: 26.39, 3: 18.44, 6: 22.57},
    (160, 63): {1: 20.66, 2: 16.35, 3: 21.27, 8: 23.42}, (256, 63): {1: 25.66, 2: 34.07, 3: 30.82}, (256, 94): {1: 35.41, 2: 45.82, 3: 39.95},
    (512, 63): {1: 53.47, 2: 52.73, 4: 52.73, 8: 66.52}, (512, 128): {1: 100.58, 2: 92.20, 4: 90.47, 8: 95.57},
}
# 64 query heads on 8 of size 64: a split costs the same and saves half as much
MEASURED_64 = {(8, 32): {1: 6.88, 2: 9.36}, (32, 32): {1: 7.01, 2: 9.80}, (128, 32): {1: 9.03, 2: 12.23}, (8, 8): {1: 4.5, 2: 8.35}}


@pytest.mark.parametrize("table,slack", [(MEASURED, 1.4), (MEASURED_64, 1.02)])
def test_attention_splits_are_near_the_best_measured_ones(table, slack):
    """A short context of small heads is never split (which cost up to twice the time); elsewhere the choice stays near the best."""
    for (rows, pages), us in table.items():
        s = _splits(rows, pages)
        near = min(us, key=lambda k: abs(k - s))
        assert us[near] <= slack * min(us.values()), (rows, pages, s)


def test_attention_splits_follow_a_layers_window():
    from openagents_b200.models.engine import LlamaEngine
    from openagents_b200.models.paged import PagedEngine
    eng = types.SimpleNamespace(attn_target_ctas=0, max_splits=64, Hkv=8)
    eng._attn_splits = types.MethodType(PagedEngine._attn_splits, eng)
    assert LlamaEngine._splits(eng, 1, 256, 0) > 8                 # a long context is split
    assert LlamaEngine._splits(eng, 1, 256, 128) == 1              # ten pages of it are not
    assert LlamaEngine._splits(eng, 1, 20, 4096) == LlamaEngine._splits(eng, 1, 20, 0)


# us on tcgen05 and on mma.sync, head size 64: (query heads, prompts, tokens of each, tokens ahead of them)
PROMPTS_64 = {
    (64, 1, 40, 0): (5.9, 4.1), (64, 1, 128, 0): (6.7, 5.5), (64, 1, 320, 0): (14.6, 12.2), (64, 1, 512, 0): (19.0, 22.7), (64, 1, 1200, 0): (58.4, 76.6),
    (64, 4, 256, 0): (27.6, 21.5), (64, 4, 512, 0): (60.2, 55.4), (64, 4, 1024, 0): (150.0, 174.0), (8, 1, 300, 0): (8.4, 9.2), (8, 1, 100, 0): (6.1, 5.2),
    (8, 4, 512, 0): (10.4, 16.2), (64, 1, 16, 2000): (23.3, 42.8), (64, 4, 64, 2000): (51.7, 56.5), (64, 8, 128, 0): (24.7, 14.1),
}


def test_prefill_attention_of_head_size_64_takes_the_faster_kernel():
    from openagents_b200.models.engine import LlamaEngine
    layer = lambda window: types.SimpleNamespace(window=window)
    for (heads, prompts, tokens, past), (tc05, mma) in PROMPTS_64.items():
        eng = types.SimpleNamespace(hd=64, Hq=heads, prefill_tc05=True)
        assert LlamaEngine._tc05_prefill(eng, layer(0), prompts, tokens, tokens + past) == (tc05 < mma), (heads, prompts, tokens, past)
        assert not LlamaEngine._tc05_prefill(eng, layer(128), prompts, tokens, tokens + past)
    assert LlamaEngine._tc05_prefill(types.SimpleNamespace(hd=128, Hq=32, prefill_tc05=True), layer(0), 1, 1, 1)
    assert not LlamaEngine._tc05_prefill(types.SimpleNamespace(hd=128, Hq=32, prefill_tc05=False), layer(0), 1, 4096, 4096)
    assert not LlamaEngine._tc05_prefill(types.SimpleNamespace(hd=256, Hq=32, prefill_tc05=True), layer(0), 1, 4096, 4096)
