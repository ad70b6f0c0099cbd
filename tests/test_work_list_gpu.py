"""Work list of the tensor-core attention kernel, from the kernel's own device code (``come_attn_work_list``): every query row
of every (segment, head) belongs to exactly one item, and the query tiles per item and the split of the last round are those
of a plain restatement of the rule."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STEP = [0, 70, 80, 96, 115]  # cost of a key step with that many query tiles
TILE, KEYS = 128, 64


def _device_list(lengths, heads, ctas, rows=None, bound=None, device_bound=None):
    from come_b200 import _lib
    from come_b200._torch_util import ptr, stream_ptr
    ends = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    lo, hi = rows or (0, int(ends[-1]))
    cu = torch.from_numpy(ends).cuda()
    capacity = int(sum((n // TILE + 2) for n in lengths) + 8) * heads * 2
    if len(lengths) > 2048:
        capacity = len(lengths) * heads * (-(-max(lengths) // (4 * TILE)) + 1)
    out = torch.zeros(4 + 8 * capacity, dtype=torch.int32, device="cuda")
    md = None if device_bound is None else torch.tensor([device_bound], dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib().come_attn_work_list(ptr(cu), len(lengths), heads, lo, hi, int(bound or max(lengths)), ptr(md), ctas,
                                              ptr(out), capacity, stream_ptr(cu.device)))
    out = out.cpu().numpy()
    total, height, first_split, parts = out[:4]
    assert 0 < total <= capacity
    return ends, (lo, hi), height, first_split, parts, out[4: 4 + 8 * total].reshape(-1, 8)


def _tail(height, rest, ctas):
    if height > 1 and rest * height <= ctas:
        return 1
    return 2 if height > 2 and rest * 2 <= ctas else height


def _plans(ends, span, heads, ctas, table):
    """``{height: (cost, first split item, parts)}``."""
    lo, hi = span
    segs = []
    for s0, s1 in zip(ends[:-1], ends[1:]):
        rows = min(s1, hi) - max(s0, lo)
        segs.append((-(-(s1 - s0) // KEYS), -(-max(rows, 0) // TILE)))
    if not table:
        segs.sort(key=lambda s: -s[0])  # stable
    plans = {}
    for h in (1, 2, 3, 4):
        first, cost, owner = 0, 0.0, (0, 0.0)
        items = sum(-(-n // h) for _, n in segs) * heads
        rest = items % ctas
        weight = sum(k * (n // h * STEP[h] + STEP[n % h]) for k, n in segs) * heads / max(items, 1)
        for k, n in segs:
            blocks = -(-n // h)
            mean = k * (n // h * STEP[h] + STEP[n % h]) / max(blocks, 1)
            end = first + blocks * heads
            cost += (-(-end // ctas) - -(-first // ctas)) * mean
            if first <= items - rest < end:
                owner = (k, mean)
            first = end
        if table:
            cost, owner = -(-items // ctas) * weight, (weight / STEP[h], weight)
        low, parts, split = _tail(h, rest, ctas), 1, items
        if rest and low != h:
            cost += STEP[low] * owner[0] - owner[1]
            parts, split = -(-h // low), items - rest
        plans[h] = (cost, split, parts)
    return plans


def _check(lengths, heads, ctas, rows=None, bound=None, device_bound=None):
    ends, span, height, split, parts, items = _device_list(lengths, heads, ctas, rows, bound, device_bound)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    most = -(-min(max(lengths), span[1] - span[0]) // TILE)
    ctas = min(ctas, most * len(lengths) * heads)  # no more CTAs than tiles could exist
    seen = np.zeros((heads, span[1] - span[0]), np.int32)
    starts = {int(s): i for i, s in enumerate(ends[:-1]) if ends[i + 1] > s}
    for i, (head, s0, s1, row, end, tiles, key_tiles, slot) in enumerate(items):
        if tiles == 0:
            continue
        seg = starts[int(s0)]
        assert s1 == ends[seg + 1] and key_tiles == -(-(s1 - s0) // KEYS)
        assert max(s0, span[0]) <= row < end == min(s1, span[1])
        low = height if i < split else (1 if parts == height else 2)
        assert 1 <= tiles <= low
        assert slot == ((i // ctas) % 4 if height == 1 else 0) and slot + tiles <= 4
        seen[head, row - span[0]: min(end, row + tiles * TILE) - span[0]] += 1
    assert (seen == 1).all()
    table = 16 <= len(lengths) <= 2048 and most > 1
    on_device = (table or 2 <= len(lengths) <= 15) and not (most == 1 or (not table and most * len(lengths) * heads <= min(ctas, sms)))
    if len(lengths) == 1 or on_device:
        plans = _plans(ends, span, heads, ctas, table)
        assert plans[height][0] <= min(p[0] for p in plans.values()) * (1 + 1e-5)  # float32 sums on the device
        assert (split, parts) == plans[height][1:]
        if not table:  # rounds of like length: keys never rise along the list
            assert (np.diff(items[items[:, 5] > 0][:, 6]) <= 0).all()
    return int(height), int(parts)


SHAPES = {
    "one": [6456], "one tile": [100], "short one": [897], "equal": [1374] * 8, "falling": [12000, 6000, 3000, 1500, 750, 375],
    "rising": [375, 750, 1500, 3000], "one long": [300] * 14 + [9000], "edges": [1, 128, 129, 256, 257, 384, 385, 511, 512, 513],
    "empty between": [700, 0, 300, 0, 5], "table": [60 + 31 * i for i in range(17)], "table long": [4000] + [90] * 20,
    "all short": [100] * 15, "many short": [64] * 300, "more than the table": [33] * 2049, "more, one longer": [33] * 2100 + [700],
}


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("heads", [1, 6, 16])
def test_every_row_once(shape, heads):
    for ctas in (1, 3, 7, 20, 148):
        _check(SHAPES[shape], heads, ctas)


def test_row_slices_and_device_bounds():
    """A slice of the query rows (segments without rows in it, segments cut by it) and a loose bound with the true one on the
    device."""
    for rows in [(0, 100), (650, 1400), (1300, 6725), (6000, 6725)]:
        for ctas in (4, 148):
            _check([700, 420, 901, 130, 4574], 4, ctas, rows=rows)
            _check([6725], 4, ctas, rows=rows)
    _check([1374] * 5, 4, 20, bound=6870, device_bound=1374)
    _check([1374], 4, 5, bound=2748, device_bound=1374)


def test_loose_bound_does_not_count():
    """2048 segments of 8192 tokens x 16 heads are 2 million items; with the sum of all lengths as the bound of the longest one
    2^32 slots could exist, which no launch holds."""
    from come_b200 import _lib
    from come_b200._torch_util import ptr, stream_ptr
    cu = torch.arange(0, 2049, dtype=torch.int32, device="cuda") * 8192
    total = 2048 * 8192
    out = torch.zeros(4 + 8, dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib().come_attn_work_list(ptr(cu), 2048, 16, 0, total, total, None, 0, ptr(out), 1, stream_ptr(cu.device)))
    assert out[1].item() == 4 and 2048 * 16 * 16 <= out[0].item() < 2048 * 16 * 16 + 4 * 148


def test_all_heights_and_splits_are_reached():
    """The lengths of the attention tests that compare bits over the number of CTAs take every height and every split."""
    reached = set()
    for lengths in ([897], SHAPES["edges"], SHAPES["table"]):
        for ctas in (1, 2, 3, 4, 5, 6, 8, 10, 14, 20, 40):
            reached.add(_check(lengths, 2, ctas))
    assert {h for h, _ in reached} == {1, 2, 3, 4}, reached
    # items of two tiles split into one each never win: enumerated over 2 to 59 tiles, 1 to 16 heads and 1 to 148 CTAs
    assert {(4, 4), (4, 2), (3, 2)} <= reached | {_check([n], 2, c) for n in (1153, 1700, 2300) for c in range(4, 30)}, reached
