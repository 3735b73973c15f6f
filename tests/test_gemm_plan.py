"""The tensor-core product's planner (``bw_gemm_tc_plan`` in csrc/gemm_tc.cu) is host code:
which orientation, which tile width and how many K splits a product gets.  Its
decisions are checked here without a GPU, over the shapes the engine's layers produce and
over odd ones: every decision must be one the kernels are built for, and a split must fit
the scratch it is given."""
import ctypes
import itertools

import pytest

BM, BK, NUM_SMS = 128, 64, 148          # csrc/gemm_tc.cu: tile rows, k-block, CTAs of the persistent grid
WIDTHS_TOKENS_WIDE = (16, 32, 64, 128, 256)   # features in the 128-row dimension: tokens rounded up to a power of two
WIDTHS_FEATURES_WIDE = (128, 224, 240, 256)   # tokens in the 128-row dimension


@pytest.fixture(scope="module")
def plan():
    from blackwellllm_b200.kernels.build import load_library
    lib = load_library("gemm_tc")
    fn = lib.bw_gemm_tc_plan
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_longlong,
                   ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_int)]

    def call(M, N, K, swiglu=0, workspace=1 << 24, counters=1 << 14):
        tr, bn = ctypes.c_int(-1), ctypes.c_int(-1)
        splits = fn(M, N, K, swiglu, workspace, counters, ctypes.byref(tr), ctypes.byref(bn))
        return splits, tr.value, bn.value
    return call


def ceil_div(a, b):
    return -(-a // b)


TOKENS = (1, 2, 3, 7, 8, 16, 17, 33, 64, 65, 100, 128, 255, 256, 257, 300, 512, 1000, 1024, 2048, 2049, 8192)
# (features, inner size): q/k/v, o, gate/up, down and head of the three layer shapes the bench knows, and odd ones
PRODUCTS = ((6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336), (128256, 4096),
            (4608, 3584), (3584, 3584), (37888, 3584), (3584, 18944), (152064, 3584),
            (7168, 5120), (5120, 5120), (27648, 5120), (5120, 13824),
            (16, 8), (48, 24), (100, 72), (352, 64), (1000, 1000), (33, 4096))


@pytest.mark.parametrize("swiglu", (0, 1))
def test_every_decision_is_one_the_kernels_are_built_for(plan, swiglu):
    for M, (N, K) in itertools.product(TOKENS, PRODUCTS):
        if swiglu and N % 32:
            continue
        splits, tr, bn = plan(M, N, K, swiglu)
        what = f"M={M} N={N} K={K} swiglu={swiglu}: splits={splits} transposed={tr} bn={bn}"
        assert tr == (1 if M <= 256 else 0), what
        if tr:
            assert bn in WIDTHS_TOKENS_WIDE and bn >= M and (bn == 16 or bn // 2 < M), what
        else:
            assert bn in WIDTHS_FEATURES_WIDE, what
            assert not swiglu or bn % 32 == 0, what      # the SwiGLU epilogue pairs 16 gate with 16 up features
        kb_total = ceil_div(K, BK)
        assert 1 <= splits <= max(1, kb_total), what
        tiles = ceil_div(N, BM) * ceil_div(M, bn) if tr else ceil_div(M, BM) * ceil_div(N, bn)
        if tiles >= NUM_SMS:
            assert splits == 1, what                        # enough tiles for every CTA: no partial sums
        if splits > 1:
            assert splits <= 16 and kb_total // splits >= 8, what
            assert M <= 64 or splits * 8 * M <= K, what     # partial sums stay well below the weight bytes


def test_a_split_fits_the_scratch_it_is_given(plan):
    for M, (N, K) in itertools.product((1, 8, 16, 64, 200), PRODUCTS):
        free, tr, bn = plan(M, N, K)
        tiles = ceil_div(N, BM) * ceil_div(M, bn)
        for workspace, counters in ((0, 0), (M * N, 1 << 14), (3 * M * N, 1 << 14), (1 << 24, 4 * tiles - 1),
                                    (1 << 24, 4 * tiles)):
            splits, tr2, bn2 = plan(M, N, K, 0, workspace, counters)
            assert (tr2, bn2) == (tr, bn)                   # scratch changes the split only
            assert 1 <= splits <= free
            if splits > 1:
                assert splits * M * N <= workspace and tiles * 4 <= counters


def test_decode_shapes_fill_the_gpu(plan):
    """The products of a decode step at batch 1 to 64 on the 8B layer sizes: with fewer tiles than
    CTAs the K splits bring the items of a round to at least half of the CTAs."""
    for M in (1, 8, 64):
        for N, K in ((6144, 4096), (4096, 4096), (4096, 14336)):
            splits, tr, bn = plan(M, N, K)
            tiles = ceil_div(N, BM) * ceil_div(M, bn)
            assert tr == 1 and tiles < NUM_SMS
            assert NUM_SMS // 2 <= tiles * splits <= NUM_SMS, (M, N, K, splits)


@pytest.fixture(scope="module")
def route(plan):
    from blackwellllm_b200.kernels.build import load_library
    fn = load_library("gemm_tc").bw_gemm_tc_route
    fn.argtypes = [ctypes.c_int] * 6 + [ctypes.c_longlong] + [ctypes.POINTER(ctypes.c_int)] * 3

    def call(M, N, K, kind, mode=1, force=0, workspace=1 << 24):
        planned, tr0, bn0 = plan(M, N, K, int(kind == 1), workspace)
        tr, bn, splits = ctypes.c_int(tr0), ctypes.c_int(bn0), ctypes.c_int(planned)
        pairs = fn(M, N, K, kind, mode, force, workspace, ctypes.byref(tr), ctypes.byref(bn), ctypes.byref(splits))
        return pairs, tr.value, bn.value, splits.value
    return call


@pytest.mark.parametrize("kind", (0, 1, 2))
def test_pair_plan_splits_k_only_where_the_pairs_would_idle(route, kind):
    """CTA pairs split K only where it was measured to pay: in two halves, a long K (the down projection) at a few hundred tokens, when
    both halves of every tile fit one round of the 74 pairs."""
    for M in (200, 300, 512, 1024, 2048, 8192):
        for N, K in PRODUCTS[:14]:
            pairs, tr, bn, sp = route(M, N, K, kind)
            if not pairs:
                continue
            kb = ceil_div(K, BK)
            tiles = ceil_div(M, 2 * BM) * ceil_div(N, bn)
            if sp > 1:   # two halves of a long K whose items fit one round of the 74 pairs, planes within the scratch
                assert not tr and sp == 2 and kb >= 128 and tiles * 2 <= NUM_SMS // 2 and sp * M * N <= 1 << 24
            assert route(M, N, K, kind, workspace=0)[3] == 1            # no scratch, no split
    if kind != 1:
        assert route(512, 4096, 14336, kind) == (1, 0, 256, 2)          # down at 512 tokens: 32 tiles for 74 pairs
        assert route(700, 520, 2240, kind, force=3)[3] == 3             # a forced split is taken as it is
    assert route(512, 4096, 4096, kind)[3] == 1 and route(768, 4096, 14336, kind)[3] == 1
    assert route(2048, 28672, 4096, kind)[3] == 1                       # gate/up at 2,048 tokens: rounds of whole tiles


def test_pairs_of_129_to_256_tokens_only_where_they_are_faster(route):
    """Products measured on single CTAs and on CTA pairs: a weight of few features and a long K leaves most pairs idle."""
    single = {0: [(161, 512, 4096), (161, 256, 4096), (160, 4096, 4096), (200, 4096, 14336)], 4: [(161, 512, 4096), (161, 4096, 4096), (129, 1024, 8192)],
              1: [(161, 1024, 4096), (200, 1024, 8192), (129, 4096, 4096), (256, 512, 8192)],
              2: [(161, 768, 4096), (161, 1536, 14336), (256, 768, 14336), (129, 1536, 8192)]}
    pairs = {0: [(200, 512, 2048), (200, 4096, 4096), (256, 12288, 4096)], 4: [(200, 512, 2048), (256, 4096, 4096)],
             1: [(161, 28672, 4096), (161, 11264, 4096), (256, 8192, 4096), (129, 512, 1024)],
             2: [(161, 6144, 4096), (200, 6144, 8192), (129, 768, 2048), (256, 4608, 14336)]}
    for kind in (0, 1, 2, 4):
        for case in single[kind]:
            assert route(*case, kind)[:2] == (0, 1), (kind, case)
            assert kind in (0, 4) or route(*case, kind, mode=2)[0] == 1
        for case in pairs[kind]:
            assert route(*case, kind)[0] == 1, (kind, case)


def test_few_channels_on_pairs_only_where_they_are_faster(route):
    """Below 2,048 channels a tile's epilogue and the pairs' start count; a written result on tiles of 240 columns goes out value by value."""
    for kind in (0, 2, 4):
        for case in ((300, 5120, 1024), (257, 6144, 1024), (257, 3072, 512), (300, 4096, 512)):
            assert route(*case, kind)[0] == 0, (kind, case)
        for case in ((512, 5120, 1024), (300, 5120, 4096), (400, 6144, 1024), (300, 3072, 1024)):
            assert route(*case, kind)[0] == 1, (kind, case)
    assert route(1024, 4096, 1024, 0)[0] == 1 and route(1024, 4096, 512, 0)[0] == 1


@pytest.mark.parametrize("kind", (0, 1, 2, 3, 4))
def test_every_route_is_one_the_kernels_are_built_for(plan, kind):
    """``bw_gemm_tc_route``: single CTAs in either orientation or CTA pairs (kind 0 plain, 1 SwiGLU, 2 rotary, 3 sums left open, 4 added
    into float32, in equal ranges of k-blocks where that is faster)."""
    from blackwellllm_b200.kernels.build import load_library
    fn = load_library("gemm_tc").bw_gemm_tc_route
    fn.argtypes = [ctypes.c_int] * 6 + [ctypes.c_longlong] + [ctypes.POINTER(ctypes.c_int)] * 3
    for M, (N, K), mode, force in itertools.product(TOKENS + (129, 160, 161, 200, 640), PRODUCTS, (0, 1, 2), (0, 3)):
        if kind == 1 and N % 32 or kind == 3 and M > 256:
            continue
        for workspace in (0, 3 * M * N, 1 << 24):
            planned, tr0, bn0 = plan(M, N, K, int(kind == 1), workspace)
            tr, bn, splits = ctypes.c_int(tr0), ctypes.c_int(bn0), ctypes.c_int(planned)
            pairs = fn(M, N, K, kind, mode, force, workspace, ctypes.byref(tr), ctypes.byref(bn), ctypes.byref(splits))
            what = f"M={M} N={N} K={K} kind={kind} mode={mode} force={force}: pairs={pairs} {tr.value} {bn.value} {splits.value}"
            assert splits.value == 1 or splits.value * M * N <= workspace, what
            if pairs:
                assert mode and M > 128 and kind != 3, what
                if tr.value:        # the SwiGLU of 256 features x bn tokens
                    assert kind == 1 and bn.value in (96, 128, 160, 192, 224, 256) and splits.value == 1 and not force, what
                else:
                    assert bn.value in (128, 192, 224, 256), what
                assert not force or M > 256, what
                if pairs > 1:       # ranges of half a tile of features or longer, and of 16 k-blocks; no planes
                    ranges, tiles = pairs - 1, ceil_div(N, 256)
                    assert kind == 4 and M > 256 and not force and (tr.value, bn.value, splits.value) == (0, 256, 1), what
                    assert ranges * ceil_div(M, 2 * BM) <= NUM_SMS // 2 and ranges <= 2 * tiles, what
                    assert tiles * ceil_div(K, BK) >= 16 * ranges, what
            elif (tr.value, bn.value, splits.value) != (tr0, bn0, planned):
                assert kind == 1 and 64 < M <= 128 and tr.value == 0 and bn.value in (224, 256) and splits.value == 1, what


def test_each_stream_has_counters_of_its_own_for_products_that_add_in_turns(monkeypatch):
    """Products of more than 256 tokens added into float32 may run on several streams at once: the parts of a tile are counted per stream,
    the counters of the last streams are kept (a bounded number), a recorded graph has its own."""
    import torch
    from blackwellllm_b200.kernels import ops
    at, capturing, device = [1], [False], torch.device("cpu")
    monkeypatch.setattr(ops, "_stream", lambda: at[0])
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    monkeypatch.setattr(ops, "_turns", type(ops._turns)())
    first = ops._turn_counters(device)
    assert first.numel() == ops._COUNTERS and not bool(first.any())
    at[0] = 2
    second = ops._turn_counters(device)
    assert second.data_ptr() != first.data_ptr()
    at[0] = 1
    assert ops._turn_counters(device) is first
    capturing[0] = True
    assert all(ops._turn_counters(device).data_ptr() not in (first.data_ptr(), second.data_ptr()) for _ in range(2))
    capturing[0] = False
    for at[0] in range(2, 40):      # the streams used longest ago go; stream 1's was used before the others
        ops._turn_counters(device)
    assert len(ops._turns) == ops._TURN_STREAMS and (device, 1) not in ops._turns and (device, 39) in ops._turns


@pytest.mark.parametrize("status", (0, 35))
def test_counters_that_a_product_left_in_between_are_cleared_with_its_status(monkeypatch, status):
    import types
    import torch
    from blackwellllm_b200.kernels import ops
    mine = [types.SimpleNamespace(device=types.SimpleNamespace(index=i), zeroed=0) for i in (0, 0, 1)]
    for m in mine:
        m.zero_ = lambda m=m: setattr(m, "zeroed", m.zeroed + 1)
    monkeypatch.setattr(ops, "_workspaces", {"cuda:0": (None, mine[0])})
    monkeypatch.setattr(ops, "_turns", {("cuda:0", 7): mine[1], ("cuda:1", 7): mine[2]})
    monkeypatch.setattr(ops, "load_library", lambda *a: types.SimpleNamespace(bw_gemm_tc_status=type("F", (), {"__call__": lambda self: status})()))
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    assert ops.gemm_tc_status() == status
    assert [m.zeroed for m in mine] == ([1, 1, 0] if status else [0, 0, 0])
