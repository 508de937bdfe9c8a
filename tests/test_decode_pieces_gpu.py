"""Decode attention by a list of even pieces, its merge of many chunks, and the head-by-head preparation of queries, keys and
values by 16-byte loads: each against the form that it stands beside."""

from __future__ import annotations

import dataclasses

import pytest
import torch

import kernel_refs
from mlx_omnia_b200.parts.base import KVSpec, KVView
from test_kernels_gpu import close, make_kv, ops, rand, step_of  # noqa: F401

pytestmark = pytest.mark.gpu


def _cache(seq_lens, nkv, d, page, seed):
    pages, table = make_kv(seq_lens, nkv, d, page, torch.bfloat16, 1 + sum(-(-n // page) for n in seq_lens), seed=seed)
    pages.copy_(rand(*pages.shape, dtype=torch.bfloat16, seed=seed + 1))
    return pages, table


def _reference(q, view, step, scale, gate=None, sink=None, run=0, cap=0.0, difference=None, keep=0):
    """A decode step's attention in 64 bits, request by request."""
    nq, nkv = q.shape[1], view.pages.shape[2]
    out = []
    for s, n in enumerate(step.seq_lens_host):
        j = torch.arange(n, device="cuda")
        sees = (j >= n - view.window) | (j < keep) if view.window else j >= 0
        if run:
            sees &= j >= (n - 1) - (n - 1) % run
        pages = view.block_table[s].long()[j // view.page_size]
        k, v = (view.pages[pages, w, :, j % view.page_size].double().repeat_interleave(nq // nkv, dim=1) for w in (0, 1))
        z = torch.einsum("hd,jhd->hj", q[s].double(), k) * scale
        z = (cap * torch.tanh(z / cap) if cap else z).masked_fill(~sees, -torch.inf)
        if sink is not None:
            z = torch.cat([z, sink.double()[:, None]], dim=1)
        p = torch.softmax(z, dim=1)[:, :n]
        o = torch.einsum("hj,jhd->hd", p, v)
        if difference is not None:
            o = (o[0::2] - difference.lam * o[1::2])[:, : difference.dv]
            o = o * torch.rsqrt((o * o).sum(1, keepdim=True) / difference.dv + difference.eps) * difference.factor
        out.append(o.reshape(-1))
    out = torch.stack(out)
    return out if gate is None else out * torch.sigmoid(gate.double())


def _near(got, want):
    """Each request within 2^-7 of its own largest value: weights and result are rounded to bfloat16 (2^-9 each), and a sum of
    weighted values is as uncertain as its largest entry's rounding, some 3 deviations of it."""
    worst = ((got.double() - want).abs().amax(1) / want.abs().amax(1)).tolist()
    assert max(worst) <= 2 ** -7, worst


LENGTHS = [([1, 33, 700, 32, 0, 257, 1025, 2000, 64], None), ([900, 5, 0, 431, 128], 300), ([160] * 7, None), ([2500] + [1] * 8, None)]


@pytest.mark.parametrize("places,rounds", [(9, 1), (9, 2), (200, 1), (40, 2)])
@pytest.mark.parametrize("seq_lens,window,run", [(*case, 0) for case in LENGTHS] + [([700, 96, 97, 1, 640], None, 96), ([1000] * 9, 64, 0)])
def test_a_list_holds_every_key_in_sight_once(ops, places, rounds, seq_lens, window, run):  # noqa: F811
    """Read back: a request's pieces follow one another from the first key that it sees to its last, cut at tiles of 32, and stand
    where and as many as each of them says, the longest requests' first."""
    step = step_of([1] * len(seq_lens), seq_lens)
    view = KVView(torch.zeros(1, 2, 8, 16, 128, dtype=torch.bfloat16, device="cuda"), torch.zeros(1, 1, dtype=torch.int32, device="cuda"),
                  torch.zeros(1, dtype=torch.int64, device="cuda"), 16, window)
    ops.begin_pass(step)
    rows, made = ops._decode_list(step, view, run, 8, 128, places, rounds, torch.device("cuda"))
    assert made and not ops._decode_list(step, view, run, 8, 128, places, rounds, torch.device("cuda"))[1]
    pieces = rows.view(-1, 8).tolist()
    used = [p for p in pieces if p[0] >= 0]
    assert pieces[: len(used)] == used and len(pieces) == places * rounds
    tiles = lambda p: p[3] // 32 - p[2] // 32 + 1  # noqa: E731
    for r, n in enumerate(seq_lens):
        mine = [(at, p) for at, p in enumerate(used) if p[0] == r]
        if n == 0:
            assert not mine
            continue
        first = max(0, n - window if window else 0, n - 1 - (n - 1) % run if run else 0)
        assert [at for at, _ in mine] == list(range(mine[0][1][6], mine[0][1][6] + mine[0][1][5]))
        assert all(p[1] == n - 1 and p[4] == i and p[5] == len(mine) and p[6] == mine[0][0] for i, (_, p) in enumerate(mine))
        assert mine[0][1][2] == first and mine[-1][1][3] == n - 1
        assert all(p[2] == q[3] + 1 and p[2] % 32 == 0 for (_, q), (_, p) in zip(mine, mine[1:]))
        assert max(tiles(p) for _, p in mine) - min(tiles(p) for _, p in mine) <= 1
    longest = [max(tiles(q) for q in used if q[0] == p[0]) for p in used]
    assert longest == sorted(longest, reverse=True)
    ops.end_pass(step)


@pytest.mark.parametrize("d,least", [(64, 2), (128, 2)])
def test_requests_of_one_place_each_are_cut_all_the_same(ops, d, least):  # noqa: F811
    """64 requests of 1,000 positions: as many pieces as requests would leave the GPU a third empty behind chains of 32 tiles."""
    step = step_of([1] * 64, [1000] * 64)
    view = KVView(torch.zeros(1, 2, 8, 16, d, dtype=torch.bfloat16, device="cuda"), torch.zeros(1, 1, dtype=torch.int32, device="cuda"),
                  torch.zeros(1, dtype=torch.int64, device="cuda"), 16, None)
    ops.begin_pass(step)
    rows, _ = ops._decode_list(step, view, 0, 8, d, 111, 2, torch.device("cuda"))
    assert min(p[5] for p in rows.view(-1, 8).tolist() if p[0] >= 0) >= least
    ops.end_pass(step)


FORMS = {  # query heads, key/value heads, head size, window, what else the call is given
    "plain": (6, 3, 128, None, {}), "gated": (6, 3, 128, None, {"gated": True}), "wide heads": (4, 2, 256, None, {"gated": True}),
    "window, kept, sink": (4, 2, 64, 300, {"sink": True, "keep_first": 70}), "runs, cap": (8, 2, 128, None, {"chunk": 200, "softcap": 20.0}),
    "two maps": (4, 2, 64, None, {"maps": True}), "two wide maps": (2, 1, 256, 500, {"maps": True})}


@pytest.mark.parametrize("places,rounds", [(9, 1), (9, 2), (200, 1), (40, 2)])
@pytest.mark.parametrize("seq_lens", [[1, 33, 700, 32, 257, 1025, 2000, 64, 900], [160] * 7, [2500] + [1] * 8])
@pytest.mark.parametrize("form", FORMS)
def test_decode_attention_by_pieces(ops, monkeypatch, form, places, rounds, seq_lens):  # noqa: F811
    """Every split that the list may make, against the plain reference, each request by itself. The keys at the tiles' borders carry
    values eight times as large as others: one left out or counted twice is two bounds off."""
    nq, nkv, d, window, extra = FORMS[form]
    extra, page = dict(extra), 16
    step = step_of([1] * len(seq_lens), seq_lens)
    pages, table = _cache(seq_lens, nkv, d, page, 21)
    pages[:, 1].mul_(torch.where(torch.arange(page, device="cuda") % 16 == 15, 4.0, 1.0)[None, None, :, None])
    pages[:, 1].mul_(torch.where(torch.arange(page, device="cuda") % 16 == 0, 4.0, 1.0)[None, None, :, None])
    q = rand(len(seq_lens), nq, d, dtype=torch.bfloat16, seed=22)
    view = KVView(pages, table, torch.zeros(len(seq_lens), dtype=torch.int64, device="cuda"), page, window)
    gate = rand(len(seq_lens), nq * d, dtype=torch.bfloat16, seed=23) if extra.pop("gated", False) else None
    if extra.pop("sink", False):
        extra["sink"] = rand(nq, seed=24)
    if extra.pop("maps", False):
        extra["difference"] = ops.MapDifference(lam=0.3, eps=1e-5, factor=0.7, dv=d)
    scale = 0.9 * d ** -0.5
    want = _reference(q, view, step, scale, gate, extra.get("sink"), extra.get("chunk", 0), extra.get("softcap", 0.0),
                      extra.get("difference"), extra.get("keep_first", 0))
    monkeypatch.setattr(ops, "decode_plan", lambda *a: (128, 1))
    monkeypatch.setattr(ops, "decode_places", lambda *a: (places, rounds))
    ops.begin_pass(step)
    for _ in range(2):  # a second layer reads the first one's list, and the tickets are back at zero
        _near(ops.paged_attention(q, view, step, scale, gate=gate, **extra), want)
    assert any(key[0] == "decode_list" for key in step.workspace["pass"] if isinstance(key, tuple))
    ops.end_pass(step)
    ops.raise_on_error(q.device)


@pytest.mark.parametrize("nq,nkv,d", [(6, 3, 128), (4, 2, 64), (4, 2, 256)])
@pytest.mark.parametrize("places,rounds", [(9, 1), (12, 2)])
def test_layers_that_share_a_list_in_a_replayed_step(ops, monkeypatch, nq, nkv, d, places, rounds):  # noqa: F811
    """Two layers of a captured pass, each behind the product that makes its projected rows; the second reads the list ahead of its
    wait. Replayed on other inputs and on lengths that go over tiles' borders, beside the form by chunks on caches of its own: the
    same new keys and values, and results that are a rounding apart. (A replay that found what the one before left, lists, rows or
    gates, would show here.)"""
    page, seq_lens, layers = 16, [1, 31, 700, 32, 257, 1023, 64, 95, 1500], 2
    table = _cache([n + 4 for n in seq_lens], nkv, d, page, 61)[1]
    step = step_of([1] * len(seq_lens), seq_lens)
    step.workspace, step.max_seq_len = {"private": True}, 1504
    plain = dataclasses.replace(step, workspace=None)
    slots = torch.zeros(len(seq_lens), dtype=torch.int64, device="cuda")
    inputs = [rand(len(seq_lens), 256, dtype=torch.bfloat16, seed=62 + i) for i in range(layers)]
    weights = [rand((2 * nq + 2 * nkv) * d, 256, dtype=torch.bfloat16, scale=1 / 16, seed=65 + i) for i in range(layers)]
    caches = [rand(int(table.max()) + 1, 2, nkv, page, d, dtype=torch.bfloat16, seed=70 + i) for i in range(layers)]
    by_list, by_chunk = ([KVView(c.clone(), table, slots, page, None) for c in caches] for _ in range(2))
    inv_freq = (10000.0 ** (-torch.arange(d // 2, dtype=torch.float64) * 2 / d)).float().cuda()
    monkeypatch.setattr(ops, "decode_plan", lambda *a: (128, 1))
    monkeypatch.setattr(ops, "decode_places", lambda *a: (places, rounds))

    def layer(views, i, step):
        rows = ops.linear(inputs[i], weights[i])
        p = ops.Projection(rows, 0, 2 * nq * d, (2 * nq + nkv) * d, nq, d, 1e-6, inv_freq)
        return ops.paged_attention(None, views[i], step, 0.9 * d ** -0.5, gate=rows, gate_col=nq * d, projection=p)

    def one_pass():
        ops.begin_pass(step)
        out = [layer(by_list, i, step) for i in range(layers)]
        ops.end_pass(step)
        return out

    def lengths(more):
        held = [n + more for n in seq_lens]
        step.seq_lens.copy_(torch.tensor(held, dtype=torch.int32))
        slots.copy_(torch.tensor([int(table[s, (n - 1) // page]) * page + (n - 1) % page for s, n in enumerate(held)]))

    lengths(0)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        one_pass()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = one_pass()
    for more in range(4):
        lengths(more)
        for i, x in enumerate(inputs):
            x.copy_(rand(*x.shape, dtype=torch.bfloat16, seed=80 + 10 * more + i))
        want = [layer(by_chunk, i, plain) for i in range(layers)]  # outside of a pass: by chunks
        graph.replay()
        for i in range(layers):
            assert torch.equal(by_list[i].pages, by_chunk[i].pages)
            _near(got[i], want[i].double())
    ops.raise_on_error(inputs[0].device)


@pytest.mark.parametrize("warps", [1, 4])
@pytest.mark.parametrize("nq,nkv,d", [(4, 2, 128), (3, 1, 64), (5, 1, 40), (2, 1, 256)])
@pytest.mark.parametrize("length", [128 * 15, 128 * 16 + 1, 128 * 37 + 5])
def test_merge_of_many_chunks(ops, monkeypatch, warps, nq, nkv, d, length):  # noqa: F811
    """Chunks of 128 keys around the sixteen that a round of the merge takes, against the plain reference."""
    seq_lens, page = [length, 130, 1], 16
    step = step_of([1] * 3, seq_lens)
    pages, table = _cache(seq_lens, nkv, d, page, 31)
    q, gate = rand(3, nq, d, dtype=torch.bfloat16, seed=32), rand(3, nq * d, dtype=torch.bfloat16, seed=33)
    view = KVView(pages, table, torch.zeros(3, dtype=torch.int64, device="cuda"), page, None)
    monkeypatch.setattr(ops, "decode_plan", lambda *a: (128, warps))
    got = ops.paged_attention(q, view, step, 0.9 * d ** -0.5, gate=gate)
    close(got, kernel_refs.paged_attention(q, view, step, 0.9 * d ** -0.5, gate=gate), torch.bfloat16)
    ops.raise_on_error(q.device)


@pytest.mark.parametrize("warps", [1, 4])
@pytest.mark.parametrize("nq,nkv,d,dv", [(2, 1, 256, 250), (16, 2, 128, 128), (2, 1, 64, 64)])
@pytest.mark.parametrize("length", [128 * 8, 128 * 16 + 1, 128 * 37 + 5])
def test_merge_of_many_chunks_of_two_maps(ops, monkeypatch, warps, nq, nkv, d, dv, length):  # noqa: F811
    """Around the eight (rows of more than 128 dims, one warp) and the sixteen chunks that a round takes."""
    seq_lens, page = [length, 130, 1], 16
    step = step_of([1] * 3, seq_lens)
    pages, table = _cache(seq_lens, nkv, d, page, 51)
    pages[:, 1, ..., dv:] = 0  # as the cache keeps values narrower than keys
    q = rand(3, nq, d, dtype=torch.bfloat16, seed=52)
    view = KVView(pages, table, torch.zeros(3, dtype=torch.int64, device="cuda"), page, None)
    difference = ops.MapDifference(lam=0.3, eps=1e-5, factor=0.7, dv=dv)
    monkeypatch.setattr(ops, "decode_plan", lambda *a: (128, warps))
    got = ops.paged_attention(q, view, step, 0.9 * d ** -0.5, difference=difference)
    want = _reference(q, view, step, 0.9 * d ** -0.5, difference=difference)
    _near(got, want)
    ops.raise_on_error(q.device)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,nkv,d,rot,whole,interleaved,biased,mixed", [
    (16, 4, 128, 64, True, True, False, False), (4, 2, 64, 64, False, False, True, False), (30, 1, 128, 32, False, False, False, False),
    (8, 4, 256, 256, False, False, False, True), (3, 1, 64, 0, True, False, True, False), (6, 5, 128, 8, True, False, False, True),
    (1, 0, 256, 128, True, True, False, False), (14, 9, 128, 12, False, True, True, False)])
def test_heads_prepared_side_by_side(ops, dtype, nq, nkv, d, rot, whole, interleaved, biased, mixed):  # noqa: F811
    """The kernel that takes a token's heads side by side against the general one, which a projection that starts off 16 bytes
    still takes. Both round float32 results once; their sums of squares are added in another order."""
    tokens, page = 700, 16  # more than the blocks that stay: some take several tokens
    heads, store = nq + 2 * max(nkv, 1), nkv > 0
    g = max(nkv, 1)
    cols = heads * d
    wide = rand(tokens, cols + 8, dtype=dtype, seed=41)
    odd = torch.empty(tokens * (cols + 8) + 1, dtype=dtype, device="cuda")[1:].view(tokens, cols + 8)
    odd.copy_(wide)
    assert odd.data_ptr() % 16
    bias = rand(cols + 8, dtype=dtype, seed=42) if biased else None
    wq, wk = (1 + rand((n if whole else 1) * d, scale=0.1, seed=43 + n) for n in (nq, g))
    inv = (10000.0 ** (-torch.arange(rot // 2, dtype=torch.float64) * 2 / rot)).float().cuda() if rot else None
    positions = torch.randint(0, 5000, (tokens,), device="cuda", dtype=torch.int32)
    slots = torch.randperm(tokens + 20, device="cuda")[:tokens].to(torch.int64)
    slots[3] = -1
    other = (rand(tokens, g * d + 8, dtype=dtype, seed=45), 8, 0.3) if mixed and store else None
    out = []
    for rows in (wide, odd):
        pages = torch.zeros(-(-(tokens + 20) // page), 2, g, page, d, dtype=dtype, device="cuda")
        kv = KVView(pages, torch.zeros(1, 1, dtype=torch.int32, device="cuda"), slots, page, None, spec=KVSpec(((g, d), (g, d)), None))
        q = ops.qkv_prepare(rows, 0, nq * d, (nq + g) * d, nq, d, bias if other is None else None, wq, wk, 1e-5, inv, positions, kv, store,
                            whole=whole, interleaved=interleaved, mix=other)
        out.append((q, pages))
    bound = 1e-5 if dtype == torch.float32 else 2 ** -7  # bfloat16: neighbours, half a unit either side
    for a, b in zip(*out):
        scale = b.float().abs().clamp(min=1.0)
        assert float(((a.float() - b.float()).abs() / scale).max()) <= bound
    ops.raise_on_error(wide.device)


@pytest.mark.parametrize("tokens", [9, 300])
@pytest.mark.parametrize("nq,nkv,d,whole", [(16, 4, 128, True), (6, 2, 64, False), (2, 1, 256, False)])
def test_heads_prepared_behind_a_product_in_a_replayed_step(ops, nq, nkv, d, whole, tokens):  # noqa: F811
    """The product and the preparation in a captured chain, replayed on other inputs and positions: bit for bit what the two give
    with a pause between them. (The preparation begins beside the product, and may read nothing of it before its wait.)"""
    page, width = 16, 256
    x, weight = rand(tokens, width, dtype=torch.bfloat16, seed=91), rand((nq + 2 * nkv) * d, width, dtype=torch.bfloat16, scale=1 / 16, seed=92)
    wq, wk = (1 + rand((n if whole else 1) * d, scale=0.1, seed=93 + n) for n in (nq, nkv))
    inv = (10000.0 ** (-torch.arange(d // 2, dtype=torch.float64) * 2 / d)).float().cuda()
    positions = torch.zeros(tokens, device="cuda", dtype=torch.int32)
    slots = torch.zeros(tokens, device="cuda", dtype=torch.int64)
    caches = [torch.zeros(-(-tokens // page) + 2, 2, nkv, page, d, dtype=torch.bfloat16, device="cuda") for _ in range(2)]

    def product():
        out = torch.empty(tokens, weight.shape[0], dtype=torch.bfloat16, device="cuda")
        return ops.linear(x, weight) if tokens <= 16 else ops._gemm_tcgen05(x, weight, out, 0, pair=False)

    def prepare(rows, pages):
        kv = KVView(pages, torch.zeros(1, 1, dtype=torch.int32, device="cuda"), slots, page, None, spec=KVSpec(((nkv, d), (nkv, d)), None))
        return ops.qkv_prepare(rows, 0, nq * d, (nq + nkv) * d, nq, d, None, wq, wk, 1e-5, inv, positions, kv, True, whole=whole)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        prepare(product(), caches[0])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = prepare(product(), caches[0])
    for again in range(4):
        x.copy_(rand(*x.shape, dtype=torch.bfloat16, seed=95 + again))
        positions.copy_(torch.randint(0, 5000, (tokens,), dtype=torch.int32))
        slots.copy_(torch.randperm(tokens + page)[:tokens])
        for pages in caches:
            pages.zero_()
        graph.replay()
        rows = product()
        torch.cuda.synchronize()
        want = prepare(rows, caches[1])
        assert torch.equal(got, want) and torch.equal(*caches)
    ops.raise_on_error(x.device)
