"""The work lists of omc_latent_attn_mma and omc_window_attn_mma: the library builds what a loop in Python says, and that covers every key of every row once."""
import random

import pytest

from omchat_b200.seqlib import MMA_ROWS, WINDOW_ALL, LatentAttnPlan, load, window_attn_items


def _portions(rng):
    out, row = [], 0
    for slot in range(rng.choice([0, 1, 2, 5])):
        n = rng.choice([0, 1, 3, 64, rng.randint(1, 300)])
        out.append((row, n, slot, rng.choice([0, 1, 63, 64, rng.randint(0, 5000)])))
        row += n
    return out


def _lists(portions, H, tok, base, target_ctas, min_keys, window):
    """items of eight numbers and merges of four in one list, and how many items, merges and partial results."""
    items, merges, part = [], [], 0
    for first_row, n, slot, p0 in portions:
        for start in range(0, n, tok):
            ntok, first = min(tok, n - start), p0 + start
            low = max(0, first - window + 1)                            # first key the tile's first row sees
            keys = first + ntok - low                                   # ... up to the end of what its last row sees
            want = 1
            if base < target_ctas // 2:
                want = max(1, min(-(-keys // min_keys), -(-target_ctas // base), LatentAttnPlan.MAX_PARTS))
            if want == 1:
                items.append((first_row + start, ntok, slot, first, low, low + keys, -1, 0))
                continue
            span = -(-(-(-keys // want)) // MMA_ROWS) * MMA_ROWS        # keys per part, a multiple of 64
            ends = [min(keys, at + span) for at in range(0, keys, span)]
            merges += [(first_row + start) * H, ntok * H, part, len(ends)]
            for i, end in enumerate(ends):
                items.append((first_row + start, ntok, slot, first, low + i * span, low + end, part + i, 0))
            part += len(ends)
    items.sort(key=lambda it: it[4] - it[5])    # those with the most keys first
    return [x for it in items for x in it] + merges, len(items), len(merges) // 4, part


def _case(seed):
    rng = random.Random(seed)
    portions, H = _portions(rng), rng.choice([1, 3, 8, 16, 33, 64])
    target, min_keys, window = rng.choice([2, 148, 296]), rng.choice([64, 128, 256]), rng.choice([1, 33, 256, 1024, WINDOW_ALL])
    tok = MMA_ROWS // H
    return portions, H, tok, target, min_keys, window, _lists(portions, H, tok, sum(-(-n // tok) for _, n, _, _ in portions), target, min_keys, window)


@pytest.mark.parametrize("seed", range(60))
def test_the_lists_cover_every_key_of_every_row_once(seed):
    portions, H, tok, _, _, window, (numbers, n_items, n_merges, n_parts) = _case(seed)
    seen, parts = {}, {}
    for i in range(n_items):
        row, ntok, slot, first, lo, hi, part, zero = numbers[8 * i:8 * i + 8]
        assert 1 <= ntok <= tok and lo < hi and zero == 0
        seen.setdefault((row, ntok, slot, first), []).append((lo, hi))
        if part >= 0:
            assert part not in parts
            parts[part] = row
    assert sorted(parts) == list(range(n_parts))
    want = {(r + s, min(tok, n - s), slot, p0 + s) for r, n, slot, p0 in portions for s in range(0, n, tok)}
    assert set(seen) == want
    for (row, ntok, slot, first), ranges in seen.items():
        ranges.sort()
        assert ranges[0][0] == max(0, first - window + 1) and ranges[-1][1] == first + ntok
        assert all(x[1] == y[0] for x, y in zip(ranges, ranges[1:]))
    for i in range(n_merges):
        qrow, rows, part, n = numbers[8 * n_items + 4 * i:8 * n_items + 4 * i + 4]
        assert rows <= MMA_ROWS and 1 <= n <= LatentAttnPlan.MAX_PARTS and all(parts[part + j] * H == qrow for j in range(n))


@pytest.mark.parametrize("seed", range(40))
def test_the_library_builds_the_lists_of_the_loop(seed):
    portions, H, tok, target, min_keys, window, (numbers, n_items, n_merges, n_parts) = _case(1000 + seed)
    plan = LatentAttnPlan(portions, H, "cpu", target_ctas=target, min_keys=min_keys, window=window)
    assert (plan.n_items, plan.n_merges, plan.n_parts) == (n_items, n_merges, n_parts)
    assert plan.items.tolist() + (plan.merges.tolist() if plan.merges is not None else []) == list(numbers)
    assert plan.max_rows == max((min(tok, n) for _, n, _, _ in portions), default=1) * H


@pytest.mark.parametrize("seed", range(20))
def test_windowed_items_cover_every_row_once_and_end_where_chunks_do(seed):
    rng = random.Random(seed)
    portions, rep, chunk = _portions(rng), rng.choice([1, 3, 4, 64]), rng.choice([33, 64, 100, 512, WINDOW_ALL])
    items = window_attn_items(portions, rep, "cpu", chunk).tolist()
    tok, want = MMA_ROWS // rep, []
    for first_row, n, slot, p0 in portions:
        row = 0
        while row < n:
            m = min(tok, n - row)
            if MMA_ROWS <= chunk < WINDOW_ALL:       # tiles count from the portion's or the chunk's begin
                m = min(m, chunk - (p0 + row) % chunk)
            want.append([first_row + row, m, slot, p0 + row])
            row += m
    assert items == want


def test_what_lists_take_and_refuse():
    portions = [(0, 100, 0, 5), (100, 3, 1, 2000)]
    plain = window_attn_items(portions, 4, "cpu").tolist()
    for chunk in (-3, 0, 33, 1 << 40):       # no chunks, or shorter ones than a key tile
        assert window_attn_items(portions, 4, "cpu", chunk).tolist() == plain
    assert LatentAttnPlan(portions, 8, "cpu", window=1 << 40).items.tolist() == LatentAttnPlan(portions, 8, "cpu").items.tolist()
    assert LatentAttnPlan([], 8, "cpu").n_items == 0
    for odd in ([(0, 1, 2)], [(0, 1, 2), (0, 1, 2, 3, 4)]):
        with pytest.raises(ValueError):
            window_attn_items(odd, 4, "cpu")
        with pytest.raises(ValueError):
            LatentAttnPlan(odd, 8, "cpu")


def test_a_list_without_items_asks_nothing_of_addresses():
    call = lambda n: load().omc_latent_attn_mma_rows(8, 0, 16, 512, 64, 8, 16, 1, 64, 16, n, 64, None, 0, None, 1, None, 0, 1.0, 16, 1, None, None, None)  # noqa: E731
    assert call(0) == 0 and call(1) != 0     # with one the addresses are refused: rows are read by 16 bytes
