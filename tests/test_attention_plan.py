"""The work lists of the tensor-core attention (``kernels.ops.plan_attention_work``) are host
arithmetic: which (request, token tile) a CTA of the prompt kernel takes, and into how many key
slices a decode row is cut.  Checked here without a GPU: every token of every request is covered
exactly once, slices and their result slots neither overlap nor leave holes, and a graph replay's
lists depend on the bound only."""
import random

import pytest

from blackwellllm_b200.kernels.ops import plan_attention_f32, plan_attention_work


def random_batch(rng, R, G):
    q_len, q_start, kv_len = [], [], []
    for _ in range(R):
        kind = rng.choice(("decode", "portion", "few"))
        n = 1 if kind == "decode" else (rng.randint(2, 16 // G) if kind == "few" and 16 // G >= 2 else rng.randint(2, 700))
        start = rng.choice((0, 0, rng.randint(0, 9000)))
        q_len.append(n); q_start.append(start); kv_len.append(start + n)
    return q_len, q_start, kv_len


@pytest.mark.parametrize("G,nkv,hd,rows_tile,page", [(4, 8, 128, 128, 16), (3, 1, 32, 64, 8), (1, 5, 64, 128, 64),
                                                     (7, 4, 128, 128, 16), (16, 2, 80, 64, 16), (2, 2, 256, 128, 32)])
@pytest.mark.parametrize("window", (None, 48, 300))
def test_every_token_once_and_slices_without_holes(G, nkv, hd, rows_tile, page, window):
    rng = random.Random(G * 1000 + hd + (window or 0))
    for trial in range(40):
        R = rng.randint(1, 70)
        q_len, q_start, kv_len = random_batch(rng, R, G)
        rows, keys, merge, n_slots = plan_attention_work(q_len, q_start, kv_len, G, nkv, window, hd, rows_tile, page)
        tpt = rows_tile // G
        assert tpt >= 1
        # prompt portions: tiles of tpt tokens cover each long segment exactly once
        covered = {}
        for r, t0, a, b in rows:
            assert (a, b) == (0, 0) and q_len[r] * G > 16 and 0 <= t0 < q_len[r] and t0 % tpt == 0
            assert t0 not in covered.setdefault(r, set())
            covered[r].add(t0)
        for r in range(R):
            if q_len[r] * G > 16:
                assert covered.get(r) == set(range(0, q_len[r], tpt)), (r, q_len[r])
            else:
                assert r not in covered
        # longest first: the keys a tile walks never grow along the list
        walk = [q_start[r] + t0 for r, t0, _, _ in rows]
        assert walk == sorted(walk, reverse=True)
        # decode rows: slices 0..n-1 of each short segment, result slots contiguous and disjoint
        by_req = {}
        for r, s, n, first in keys:
            by_req.setdefault(r, []).append((s, n, first))
        slot = 0
        for r in range(R):
            if q_len[r] * G > 16:
                assert r not in by_req
                continue
            items = by_req[r]
            n = items[0][1]
            assert [s for s, _, _ in items] == list(range(n)) and all(it[1:] == (n, slot) for it in items)
            span = kv_len[r] if not window else min(kv_len[r], window + q_len[r])
            assert 1 <= n <= 64 and (n == 1 or 2 * n <= -(-span // 64))   # a slice has at least two key tiles
            assert ((r, 0, n, slot) in merge) == (n > 1)
            slot += n
        assert slot == n_slots and len(merge) == sum(1 for v in by_req.values() if v[0][1] > 1)


def test_a_graph_replay_depends_on_the_bound_only():
    q_len, q_start = [1] * 8, [100, 5000, 8191, 17, 0, 640, 4096, 77]
    a = plan_attention_work(q_len, q_start, [s + 1 for s in q_start], 4, 8, None, 128, 128, 16, static_bound=8192)
    b = plan_attention_work(q_len, [8191] * 8, [8192] * 8, 4, 8, None, 128, 128, 16, static_bound=8192)
    assert a == b and a[3] > 8          # cut into slices although some requests are short
    alone = plan_attention_work([1], [8191], [8192], 4, 8, None, 128, 128, 16)
    many = plan_attention_work([1] * 64, [8191] * 64, [8192] * 64, 4, 8, None, 128, 128, 16)
    assert alone[3] > many[3] // 64 >= 1   # fewer slices a request when more requests fill the GPU


@pytest.mark.parametrize("G,nkv", ((1, 32), (3, 2), (4, 8), (16, 1), (20, 1), (64, 1)))
@pytest.mark.parametrize("window,chunk", [(None, None), (48, None), (9000, None), (None, 100), (None, 9000), (20000, 30000)])
def test_float32_work(G, nkv, window, chunk):
    """The float32 kernel's lists: every token in one tile, every slice that a tile's rows may see in one block (counted as the kernel
    counts), and results of slices that neither overlap nor leave the scratch."""
    rng = random.Random(G)
    first = lambda pos: max(0, pos - window + 1 if window else 0, pos - pos % chunk if chunk else 0)
    keys_of = lambda pos: 128 * -(-(pos + 1 - first(pos)) // 8192)
    for trial in range(60):
        q_len, q_start, _ = random_batch(rng, rng.randint(1, 20), G)
        if trial % 4 == 3:
            q_len = [rng.choice((1, 20, 45)) for _ in q_len[:2]]
        if trial % 2:
            q_start = [s + rng.choice((0, 8185, 16380, 40000, 120000)) for s in q_start]
        bound = None
        if trial % 3 == 0:
            q_len, bound = [1] * len(q_len), max(q_start) + 1 + rng.randint(0, 100000)
        q_start = q_start[:len(q_len)]
        (rows, wide, keys, merge), part_rows, merge_rows = plan_attention_f32(q_len, q_start, G, nkv, window, chunk, 128, 64, 148, bound)
        merged, covered, parts = {(r, t0): (n, w) for r, t0, n, w in merge}, [], []
        assert len(merged) == len(merge)
        for r, t0, _, _ in rows:
            covered.append((r, t0, min(64 // G, q_len[r] - t0)))
        for items, tile in ((wide, 64), (keys, 16)):
            tiles = {}
            for r, t0, z, where in items:
                tiles.setdefault((r, t0), []).append((z & 0xffff, z >> 16, where))
            for (r, t0), blocks in tiles.items():
                n = min(tile // G, q_len[r] - t0)
                covered.append((r, t0, n))
                B, where = blocks[0][1:]
                assert 1 <= B <= 66 and blocks == [(i, B, where) for i in range(B)] and n * G <= tile
                sizes = {keys_of(q_start[r] + t0 + i) for i in range(n)}
                assert len(sizes) == 1
                size = sizes.pop()
                base = first(q_start[r] + t0) // size * size
                real = -(-(q_start[r] + t0 + n - base) // size)
                share = -(-real // B)
                assert share * B >= real
                if (r, t0) not in merged:
                    assert real <= 1 and B == 1
                else:
                    assert merged[(r, t0)] == (n * G, where) and n * G <= merge_rows <= 64
                    parts.append((where, where + real * n * G))
        covered.sort()
        for r, n_q in enumerate(q_len):
            at = 0
            for _, t0, n in (c for c in covered if c[0] == r):
                assert t0 == at
                at += n
            assert at == n_q
        parts.sort()
        assert all(a[1] <= b[0] for a, b in zip(parts, parts[1:])) and (not parts or parts[-1][1] <= part_rows)


@pytest.mark.parametrize("bound", (131072, 340000))
@pytest.mark.parametrize("R,G,nkv", [(64, 4, 8), (64, 1, 32), (8, 4, 8), (2, 64, 1)])
def test_float32_decode_graphs_stay_small(bound, R, G, nkv):
    """A decode graph's lists are made for the longest context: its blocks and partial results are bounded all the same."""
    (rows, wide, keys, merge), part_rows, _ = plan_attention_f32([1] * R, [700] * R, G, nkv, None, None, 128, 64, 148, bound)
    assert len(rows + wide + keys) * nkv <= 8 * 148 + R * nkv
    assert part_rows <= 64 * R * G and 4 * part_rows * nkv * (128 + 2) <= 70e6


def test_float32_prompts_scratch_is_bounded():
    for nkv, n in ((1, 500), (2, 250), (8, 64), (37, 16)):
        (rows, wide, keys, merge), part_rows, _ = plan_attention_f32([n], [100000], 4, nkv, None, None, 128, 64)
        assert 4 * part_rows * nkv * 258 <= 64e6
