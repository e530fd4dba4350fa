"""The radix sort and the scans behind a dump, at the edges of their tiles:
1024-pair sort tiles below 1024 pairs per SM, 3840-pair tiles from there on, and
4096-item scan tiles."""
import numpy as np
import pytest

from trinityrnaseq_gb300 import KmerTable

pytestmark = pytest.mark.gpu

BIG = 152 * 1024   # pairs from which the larger tiles are taken on 152 SMs


def distinct_keys(n, k, seed):
    rng = np.random.default_rng(seed)
    keys = np.unique(rng.integers(0, 1 << (2 * k), size=n + n // 4 + 64, dtype=np.uint64))
    return rng.permutation(keys)[:n]


@pytest.mark.parametrize("n,k", [(1, 25), (2, 31), (1023, 25), (1024, 31), (1025, 5 + 8), (4095, 25), (4096, 21),
                                 (4097, 25), (40_000, 31), (BIG - 1, 25), (BIG, 25), (BIG + 1, 31),
                                 (42 * 3840 - 1, 17), (42 * 3840, 31), (42 * 3840 + 1, 25), (2_000_003, 25)])
def test_dump_order_at_tile_edges(ctx, n, k):
    keys = distinct_keys(n, k, n)
    counts = (np.arange(keys.size, dtype=np.uint32) * 7919) % 100_003 + 1
    t = KmerTable(ctx, k, False)
    t.load_pairs(keys, counts)
    gk, gc = t.dump(1)
    order = np.argsort(keys)
    assert np.array_equal(gk, keys[order]) and np.array_equal(gc, counts[order])
    # the text: every record's place is the scan of the lengths before it
    text = np.frombuffer(t.dump_fasta(1), np.uint8)
    digits = np.char.str_len(counts[order].astype(str))
    assert text.size == int((digits + k + 3).sum())
    starts = np.concatenate([[0], np.cumsum(digits + k + 3)[:-1]])
    assert np.all(text[starts] == ord(">")) and np.all(text[starts + digits + 1] == ord("\n"))
    last = text[int(starts[-1]):].tobytes()
    want = "".join("ACGT"[int(keys[order][-1]) >> (2 * (k - 1 - i)) & 3] for i in range(k))
    assert last == b">%d\n%s\n" % (int(counts[order][-1]), want.encode())


def test_sort_of_keys_with_one_digit_apart(ctx):
    """Every pass but one sees a single digit: one digit's run spans every tile."""
    n, k = 45 * 3840 + 17, 25
    keys = (np.arange(n, dtype=np.uint64) << np.uint64(8)) | np.uint64(5)
    t = KmerTable(ctx, k, False)
    t.load_pairs(keys[::-1].copy(), np.arange(n, 0, -1).astype(np.uint32))
    gk, gc = t.dump(1)
    assert np.array_equal(gk, keys) and np.array_equal(gc, np.arange(1, n + 1))


@pytest.mark.parametrize("k,low", [(25, 10), (24, 8), (31, 6), (13, 10), (9, 10), (5, 2)])
@pytest.mark.parametrize("lens", [[1, 2, 3], [63, 64], [65, 66, 1], [700, 1024, 5], [1024]])
def test_runs_of_keys_alike_but_for_their_last_bits(ctx, k, low, lens):
    """Keys that agree in all but the bits no radix pass sorts: runs shorter and
    longer than those ranked by comparing (64), whole and across the edges of
    tiles (1024), and tables with every key of the last bits."""
    rng = np.random.default_rng(k)
    tops = min(1 << (2 * k - low), 3 * 152 if max(lens) > 64 else 3000)
    parts = []
    for i in range(tops):
        n = min(int(lens[i % len(lens)]), 1 << low)
        parts.append((np.uint64(i * 7 % (1 << (2 * k - low))) << np.uint64(low)) + rng.choice(1 << low, n, replace=False).astype(np.uint64))
    keys = rng.permutation(np.unique(np.concatenate(parts)))
    counts = (np.arange(keys.size, dtype=np.uint32) * 31) % 10_007 + 1
    t = KmerTable(ctx, k, False)
    t.load_pairs(keys, counts)
    gk, gc = t.dump(1)
    order = np.argsort(keys)
    assert np.array_equal(gk, keys[order]) and np.array_equal(gc, counts[order])


@pytest.mark.parametrize("off", [-1, 0, 1])
def test_dump_order_where_the_tiles_change(ctx, off):
    """1024 pairs per SM of this device."""
    import torch
    n = torch.cuda.get_device_properties(ctx.device).multi_processor_count * 1024 + off
    keys = distinct_keys(n, 25, n)
    t = KmerTable(ctx, 25, False)
    t.load_pairs(keys, np.arange(1, n + 1, dtype=np.uint32))
    gk, gc = t.dump(1)
    order = np.argsort(keys)
    assert np.array_equal(gk, keys[order]) and np.array_equal(gc, np.arange(1, n + 1, dtype=np.uint32)[order])
