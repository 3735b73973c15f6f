"""The 32-bit path's products and its tiled attention, at the edges of their tiles, against 64 bits and against the
general kernels that take every other form."""
import math

import pytest
import torch

from test_kernels_gpu import FakeBatch, paged_case, plain_rows

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from blackwellllm_b200.kernels import ops as o
    return o


@pytest.fixture(autouse=True)
def no_wait_gave_up(ops):
    yield
    assert ops.gemm_f32_tc_status() == 0


def rand(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


# tokens on both sides of the widths of a tile and of its columns in tensor memory; ragged features; channels that leave the last
# stage ragged; tiles in one part, in several and both in one launch; tokens in one launch and in two
@pytest.mark.parametrize("M", [1, 2, 9, 16, 17, 33, 65, 128, 129, 257, 513])
@pytest.mark.parametrize("N,K", [(128, 256), (130, 260), (200, 1028), (1024, 4100), (4096, 2048), (20000, 260)])
def test_split_products(ops, M, N, K):
    x, w, b, base = rand(M, K + 4, seed=1)[:, 4:], rand(N, K, seed=2), rand(N, seed=3), rand(M, N + 1, seed=4)
    assert ops.gemm_f32_tc_supports(x, w)
    want = x.double() @ w.double().T
    size = float(want.pow(2).mean().sqrt())
    err = lambda out, ref: float((out.double() - ref).pow(2).mean().sqrt()) / size
    plain = ops.gemm_f32(x, w)
    # no further off than one chain of float32 FMAs, whose error grows with the root of K (over at least 128 sums: few of them, from 256
    # channels, may lie 20 % apart by chance)
    assert err(plain, want) <= 1.2 * err(ops.gemm_simt(x, w), want)
    # products off by up to 2^-22 each add up like their root: at most 2^-22 of the result's size, and the largest of 1e6 is five times that
    assert float((plain.double() - want).abs().max()) / size <= 2 ** -22 * 8 + 2 ** -24 * math.sqrt(K)
    out = base.clone()
    ops.gemm_f32(x, w, b.bfloat16(), out=out[:, :N], accumulate=True)
    assert err(out[:, :N], want + b.bfloat16().double() + base[:, :N].double()) <= 3e-7 * max(1.0, 1.0 / size)
    assert torch.equal(out[:, N], base[:, N])
    assert torch.equal(ops.gemm_f32(x, w), plain)
    for rows in (slice(0, 1), slice(M - 1, M), slice(M // 3, M // 3 + 20)):        # a row is the same bits whatever is beside it
        assert torch.equal(ops.gemm_f32(x[rows], w), plain[rows])


@pytest.mark.parametrize("M,N,K", [(301, 6144, 4096), (301, 4096, 4096), (128, 4096, 2048), (17, 6144, 4096), (1500, 1024, 512)])
def test_queued_products_repeat_themselves(ops, M, N, K):
    """Products right behind other kernels, nothing waited for in between: every one the bits of the same product by itself.  (The
    product's blocks start beside those of the kernels before, whose memory traffic holds up their reads of shared memory.)"""
    gain, xs, w = torch.ones(K, device=DEV), [rand(M, K, seed=s) for s in (1, 2)], rand(N, K, seed=3)
    alone = []
    for x in xs:
        torch.cuda.synchronize()
        y = ops.rmsnorm(x, gain, 1e-5, torch.float32)
        torch.cuda.synchronize()
        alone.append(ops.gemm_f32(y, w))
    for _ in range(8):
        queued = [ops.gemm_f32(ops.rmsnorm(xs[i % 2], gain, 1e-5, torch.float32), w) for i in range(300)]
        assert all(torch.equal(out, alone[i % 2]) for i, out in enumerate(queued))


def test_queued_steps_repeat_themselves():
    """Whole float32 steps of two engines in turn, queued: the logits of a step that was waited for.  (A step's prompt gets its pages
    in another order each time, and everything it reads was written by the steps right before it.)"""
    from blackwellllm_b200 import Engine, StepEntry
    raw = {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "hidden_size": 4096, "num_attention_heads": 32,
           "num_key_value_heads": 8, "head_dim": 128, "intermediate_size": 14336, "num_hidden_layers": 2, "vocab_size": 32064,
           "rope_theta": 500000.0, "rms_norm_eps": 1e-5, "tie_word_embeddings": False}
    n = 301
    engines = [Engine.from_config(raw, seed=s, dtype="float32", num_pages=24, max_requests=2, max_batch_tokens=512, max_context=384)
               for s in (0, 1)]
    entry = StepEntry("p", torch.randint(0, 32064, (n,), generator=torch.Generator().manual_seed(5)).tolist(), list(range(n)))

    def step(e):
        logits = e.step([entry])
        e.end_request("p")
        return logits

    alone = []
    for e in engines:
        for _ in range(2):
            torch.cuda.synchronize()
            logits = step(e)
            torch.cuda.synchronize()
        alone.append(logits)
    for _ in range(10):
        queued = [step(engines[i % 2]) for i in range(60)]
        assert all(torch.equal(out, alone[i % 2]) for i, out in enumerate(queued))


def test_split_products_over_the_range_of_float32(ops):
    """Products of magnitudes from 1e-30 to 1e30: the split is relative to each value.  (Smaller ones:
    test_single_products_and_small_magnitudes.)"""
    for scale_x, scale_w in ((1e-15, 1e-15), (1e15, 1e15), (1e-18, 1e18)):
        x, w = rand(40, 512, seed=1) * scale_x, rand(256, 512, seed=2) * scale_w
        want = x.double() @ w.double().T
        assert float((ops.gemm_f32(x, w).double() - want).abs().max()) <= 1e-6 * float(want.abs().max())


# results in tiles of one range, in shared tiles, and both
@pytest.mark.parametrize("M,N,K", [(3, 130, 260), (40, 1024, 4100), (5, 20000, 260)])
def test_split_products_of_infinities(ops, M, N, K):
    """Operands that are not finite, or whose parts would not be, give what a chain of FMAs gives; other rows keep their bits."""
    x, w, b, base = rand(M, K, seed=1), rand(N, K, seed=2), rand(N, seed=3), rand(M, N, seed=4)
    plain = ops.gemm_f32(x, w)
    inf, top = float("inf"), 3.4028e38
    w[7] = w[7].to(torch.bfloat16).float()                # a weight without a second part, a zero, an infinity, a NaN
    w[5, 11], w[N - 1, 200], w[64, 30] = 0.0, -inf, float("nan")
    touched = torch.zeros(M, N, dtype=torch.bool, device=DEV)
    touched[:, [5, 7, 64, N - 1]] = True
    for fill in ({(1, 11): inf}, {(1, 11): -inf, (1, 12): inf}, {(2, 5): float("nan")}, {(M - 1, K - 1): top / 2, (M - 1, 3): top},
                 {(0, 4): -top}):
        y, rows = x.clone(), sorted({r for r, _ in fill})
        for at, v in fill.items():
            y[at] = v
        hit = touched.clone()
        hit[rows] = True
        # near the largest value: what overflows depends on the order of a sum, so the other entries and weights stay small there
        scale = 1e-4 if any(abs(v) == top for v in fill.values()) else 1.0
        got, want = ops.gemm_f32(y, w * scale), ops.gemm_simt(y, w * scale)
        assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
        known = hit & torch.isfinite(want)
        assert torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
        # sums of K products in two orders: each off by 2^-24 K of the largest at most
        size = want.nan_to_num(0.0, 0.0, 0.0).abs().amax(1, keepdim=True)
        assert bool(((got - want).abs() <= 2 ** -24 * K * size)[known].all())
        if scale == 1.0:
            assert torch.equal(got[~hit], plain[~hit])
        out = base.clone()
        ops.gemm_f32(y, w * scale, b, out=out, accumulate=True)
        assert torch.equal(out.nan_to_num(), (got + b + base).nan_to_num()) and torch.equal(torch.isnan(out), torch.isnan(got))


def test_single_products_and_small_magnitudes(ops):
    """What splitting in two loses where float32 FMAs lose next to nothing: bounds, derived from the parts' 11 bits each."""
    N, K, M = 256, 512, 40
    x, w, at = torch.zeros(M, K, device=DEV), rand(N, K, seed=2), torch.arange(M) * 3
    x[torch.arange(M), at] = 1.0
    assert bool(((ops.gemm_f32(x, w) - w[:, at].T).abs() <= 2 ** -23 * w[:, at].T.abs()).all())
    x[torch.arange(M), at] = rand(M, seed=3)
    want = x.double() @ w.double().T
    assert bool(((ops.gemm_f32(x, w).double() - want).abs() <= (2 ** -21 + 2 ** -24) * want.abs()).all())
    x = rand(M, K, seed=4)
    for scale in (1e-30, 1e-34, 1e-36, 1e-38):
        for a, b in ((x * scale, w), (x, w * scale)):
            want, sizes = a.double() @ b.double().T, a.double().abs() @ b.double().abs().T
            # products of 512 channels as everywhere (see test_split_products), and operands whose lo keeps multiples of 2^-136 only
            other = w if b is w else x
            bound = 2 ** -21 * sizes + 2 ** -135 * K * float(other.abs().max())
            assert bool(((ops.gemm_f32(a, b).double() - want).abs() <= bound).all())


@pytest.mark.parametrize("nh,nkv,hd,page", [(4, 2, 16, 16), (3, 1, 20, 8), (8, 8, 64, 16), (32, 8, 128, 16), (14, 2, 132, 4),
                                            (6, 2, 256, 32), (17, 1, 32, 16), (64, 1, 8, 16), (5, 5, 80, 24)])
@pytest.mark.parametrize("window,chunk", [(None, None), (1, None), (50, None), (None, 96), (40, 64)])
def test_tiled_attention(ops, nh, nkv, hd, page, window, chunk):
    # prompt portions (from position 0, continuing, ragged), single tokens at 1 and at many keys, a two-token portion
    q_lens, kv_lens = [70, 1, 33, 2, 1, 130], [70, 900, 97, 64, 1, 400]
    q, kp, vp, table, refs = paged_case(q_lens, kv_lens, nh, nkv, hd, page, torch.float32, seed=hd)
    batch = FakeBatch(q_lens, kv_lens)
    assert ops.attention_f32_supports(q, kp, vp, nh)
    out = ops.attention_f32(q, kp, vp, batch, table, nh, window, hd ** -0.5, chunk)
    general = ops.attention_simt(q, kp, vp, batch.positions, batch.req_of_token, table, nh, window, hd ** -0.5, chunk=chunk)
    assert not torch.isnan(out).any()
    # both are float32 softmaxes over at most 900 keys: scores up to |s| < 8 off by 2^-22 |s| sqrt(hd) move a weight by 2e-5 at most
    assert float((out - general).abs().max()) <= 2e-5 * float(general.abs().max())
    # the rows of a request are the same bits alone, a few at a time, and in a portion; whatever bound the slices were made for
    for r, at in ((0, 0), (2, 33 + 38), (5, 107)):
        sees = kv_lens[r] - q_lens[r]
        for i, n in ((0, 1), (q_lens[r] - 1, 1), (q_lens[r] // 2, min(16, q_lens[r] // 2))):
            alone = FakeBatch([n], [sees + i + n])
            alone.static_bound = 1000 if n == 1 else None
            rows = slice(at + i, at + i + n)
            assert torch.equal(ops.attention_f32(q[rows].contiguous(), kp, vp, alone, table[r:r + 1].contiguous(), nh, window, hd ** -0.5, chunk),
                               out[rows])
    if chunk is None:
        ref = plain_rows(refs, window, nh, hd)
        assert float((out.double().cpu() - ref).abs().max()) <= 2e-5 * float(ref.abs().max())
    # a table entry without a page hides its keys in both kernels
    table[1, 3] = -1
    out = ops.attention_f32(q, kp, vp, batch, table, nh, window, hd ** -0.5, chunk)
    general = ops.attention_simt(q, kp, vp, batch.positions, batch.req_of_token, table, nh, window, hd ** -0.5, chunk=chunk)
    assert float((out - general).abs().max()) <= 2e-5 * float(general.abs().max())


@pytest.mark.parametrize("window,chunk", [(None, None), (9000, None), (None, 8500), (8193, 16500)])
def test_slices_that_grow_with_the_context(ops, window, chunk):
    """Beyond 64 slices of 128 keys a row's slices get longer: the same bits in a portion, in a few tokens and by itself, on both sides
    of the place where they do."""
    nh, nkv, hd, page = 4, 2, 16, 32
    q_lens, kv_lens = [40, 3, 1, 90], [8212, 8194, 16385, 17020]
    q, kp, vp, table, _ = paged_case(q_lens, kv_lens, nh, nkv, hd, page, torch.float32, seed=7)
    batch = FakeBatch(q_lens, kv_lens)
    out = ops.attention_f32(q, kp, vp, batch, table, nh, window, hd ** -0.5, chunk)
    general = ops.attention_simt(q, kp, vp, batch.positions, batch.req_of_token, table, nh, window, hd ** -0.5, chunk=chunk)
    assert float((out - general).abs().max()) <= 2e-5 * float(general.abs().max())      # (see test_tiled_attention)
    for r, at, places in ((0, 0, (0, 18, 19, 20, 21, 39)), (1, 40, (0, 1, 2)), (3, 44, (0, 24, 55, 56, 68, 89))):
        for i in places:
            for n in (1, 2):
                if i + n > q_lens[r]:
                    continue
                alone = FakeBatch([n], [kv_lens[r] - q_lens[r] + i + n], 131072 if n == 1 else None)
                rows = slice(at + i, at + i + n)
                assert torch.equal(ops.attention_f32(q[rows].contiguous(), kp, vp, alone, table[r:r + 1].contiguous(), nh, window, hd ** -0.5,
                                                     chunk), out[rows])


@pytest.mark.parametrize("nh,nkv,hd", [(8, 2, 64), (32, 8, 128), (6, 2, 132), (4, 4, 256)])
@pytest.mark.parametrize("q_lens,kv_lens", [([385], [385]), ([257, 65], [257, 640]), ([512], [512])])
def test_tiles_whose_slices_are_dealt_out(ops, monkeypatch, nh, nkv, hd, q_lens, kv_lens):
    """A block for each slice of every tile: the bits of a block per tile (which slices there are does not depend on it), and float32's
    distance from the general kernel (see test_tiled_attention)."""
    q, kp, vp, table, _ = paged_case(q_lens, kv_lens, nh, nkv, hd, 16, torch.float32, seed=hd)
    starts = [k - n for n, k in zip(q_lens, kv_lens)]
    assert ops.plan_attention_f32(q_lens, starts, nh // nkv, nkv, None, None, 128, 64)[0][1]
    batch = FakeBatch(q_lens, kv_lens)
    out = ops.attention_f32(q, kp, vp, batch, table, nh, None, hd ** -0.5)
    general = ops.attention_simt(q, kp, vp, batch.positions, batch.req_of_token, table, nh, None, hd ** -0.5)
    assert float((out - general).abs().max()) <= 2e-5 * float(general.abs().max())
    monkeypatch.setattr(ops, "num_sms", lambda device: 1)       # one SM: every tile is a block's
    assert torch.equal(ops.attention_f32(q, kp, vp, FakeBatch(q_lens, kv_lens), table, nh, None, hd ** -0.5), out)


@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 16), (8, 2, 128), (3, 1, 132)])
@pytest.mark.parametrize("window,chunk", [(None, None), (40, None), (None, 64)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_values_of_hidden_keys_are_not_read_into_a_result(ops, nh, nkv, hd, window, chunk, bad):
    """A value that is no number reaches the rows that see its key, and leaves the bits of all others."""
    q_lens, kv_lens, page = [70, 1, 3], [90, 200, 150], 16
    q, kp, vp, table, _ = paged_case(q_lens, kv_lens, nh, nkv, hd, page, torch.float32, seed=hd)
    batch = FakeBatch(q_lens, kv_lens)
    whole = ops.attention_f32(q, kp, vp, batch, table, nh, window, hd ** -0.5, chunk)
    for r, pos in ((0, 89), (0, 47), (1, 150), (1, 10), (2, 149), (2, 109)):
        v2 = vp.clone()
        v2[table[r, pos // page], :, pos % page] = bad
        out = ops.attention_f32(q, kp, v2, batch, table, nh, window, hd ** -0.5, chunk)
        general = ops.attention_simt(q, kp, v2, batch.positions, batch.req_of_token, table, nh, window, hd ** -0.5, chunk=chunk)
        at = batch.positions
        sees = (batch.req_of_token == r) & (at >= pos)
        if window:
            sees &= pos > at - window
        if chunk:
            sees &= pos >= at // chunk * chunk
        assert torch.equal(out[~sees], whole[~sees])
        assert not torch.isfinite(out[sees]).any()
        assert torch.equal(torch.isnan(out), torch.isnan(general)) and torch.equal(torch.isinf(out), torch.isinf(general))


def test_rows_off_16_bytes_go_to_the_general_kernel(ops):
    q, kp, vp, table, refs = paged_case([5, 1], [5, 40], 4, 2, 18, 16, torch.float32, seed=3)
    assert not ops.attention_f32_supports(q, kp, vp, 4)                   # a head size that is no multiple of four
    out = ops.paged_attention(q, kp, vp, FakeBatch([5, 1], [5, 40]), table, 4, None, 18 ** -0.5)
    assert float((out.double().cpu() - plain_rows(refs, None, 4, 18)).abs().max()) <= 2e-5
