"""Host-side choices of the kernel dispatcher that need no GPU."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from mlx_omnia_b200.kernels import ops
from mlx_omnia_b200.parts.base import KVView


def test_width_bucket_keeps_three_bits_and_is_its_own_fixed_point():
    assert [ops.width_bucket(n) for n in (0, 1, 8, 9, 16, 17, 100, 256, 257, 5000)] == \
        [8, 8, 8, 10, 16, 20, 112, 256, 320, 5120]
    for n in range(1, 3000, 7):
        b = ops.width_bucket(n)
        assert n <= b <= max(8, n + n // 4) and ops.width_bucket(b) == b


def test_decode_plan_is_a_tile_multiple_within_bounds_and_the_same_for_a_bucket():
    for requests in (1, 3, 8, 17, 64, 100, 512):
        for nkv in (1, 3, 8):
            for longest in (1, 90, 128, 1000, 4096, 5000, 100000):
                chunk, warps = ops.decode_plan(requests, nkv, longest, 148)
                assert 128 <= chunk <= 1024 and chunk % 64 == 0 and warps in (1, 4)
                # A captured graph's batch is a power of two: same plan.
                assert (chunk, warps) == ops.decode_plan(1 << (requests - 1).bit_length(), nkv, longest, 148)


def test_decode_plan_grows_with_the_work():
    """Few pairs: short chunks and four warps a block, so that enough warps run; more pairs: one
    warp a block and the shortest chunk whose blocks the GPU holds at a time."""
    assert ops.decode_plan(1, 8, 4096, 148) == (256, 4)
    assert ops.decode_plan(2, 8, 4096, 148) == (256, 4)
    assert ops.decode_plan(4, 8, 4096, 148) == (192, 1)
    assert ops.decode_plan(8, 8, 4096, 148) == (320, 1)
    assert ops.decode_plan(8, 8, 5120, 148) == (448, 1)
    assert ops.decode_plan(16, 8, 4096, 148) == (704, 1)
    assert ops.decode_plan(64, 8, 8192, 148) == (1024, 1)
    # One long request: four warps a block, chunks so long that two blocks an SM hold them all.
    chunk, warps = ops.decode_plan(1, 8, 32768, 148)
    assert warps == 4 and 8 * -(-32768 // chunk) <= 2 * 148


def test_timeline_groups_a_step_s_kernels_by_their_place_in_a_layer():
    from mlx_omnia_b200.kernels import timeline

    layer = [("gemv", 7, 10.0), ("attention", 9, 27.0), ("gemv", 7, 3.0), ("gemv", 7, 12.0), ("gemv", 7, 6.0)]
    kernels = [("elementwise", 1, 5.0), ("elementwise", 2, 6.0)] + layer * 4 + [("elementwise", 3, 2.0)]
    lines = timeline.by_layer(kernels, "attention")
    assert len(lines) == 2 + 5 + 1 + 1
    assert lines[0].startswith("before the layers") and lines[-1].startswith("after the layers")
    assert "attention:9" in lines[3] and "27.00 us" in lines[3] and "4 layers" in lines[3]
    assert lines[7].split()[2] == "58.00"
    assert timeline.by_layer(layer, "attention") == [f"{lib}:{line} {us:8.2f} us" for lib, line, us in layer]


def test_a_pending_residual_step_is_settled_once_and_says_when_it_was_consumed(cpu_ops):
    """Without a GPU no product runs a pending step itself (the blocks then make none): settling one
    runs the residual kernel (here its plain reference) in place; asking again gives the same
    activations; a step that a product consumed keeps no activations and says so."""
    import pytest
    import torch

    import kernel_refs

    ops = cpu_ops
    x, branch = torch.randn(3, 16), torch.randn(3, 16).bfloat16()
    wb, wo = torch.rand(16) + 0.5, torch.rand(16) + 0.5
    expect_x = x.clone()
    expect_h = kernel_refs.add_rmsnorm(expect_x, branch, wb, 1e-6, wo, 1e-5)
    step = ops.PendingStep(x, branch, wb, 1e-6, wo, 1e-5)
    assert not ops.pending_supported(x, branch)
    assert torch.equal(ops.settle(step), expect_h)
    assert step.x_new is x and torch.equal(x, expect_x) and ops.residual_after(step, torch.zeros(1)) is x
    assert torch.equal(ops.settle(step), expect_h) and ops.settle(expect_h) is expect_h
    assert ops.residual_after(expect_h, x) is x
    consumed = ops.PendingStep(x, branch, wb, 1e-6, wo, 1e-5, x_new=torch.zeros_like(x))
    with pytest.raises(RuntimeError, match="already consumed"):
        ops.settle(consumed)


def test_prefill_blocks_are_listed_longest_first_and_cut_into_parts(monkeypatch):
    """The tcgen05 prefill kernel's list: every block of tokens of every multi-token request once per
    key/value head (requests that bring one token are left to the decode kernel); a block that alone
    would run longer than the device's share of all key tiles is listed as parts whose runs of tiles
    cover the block's tiles once and in order; the items with the most tiles come first; parts of one
    block share a place in the workspace and a ticket that no other block has."""
    from types import SimpleNamespace
    import numpy as np

    def blocks_of(q_lens, seq_lens, tokens_per_block, tile, nkv, window):
        items = {}
        for s, n in enumerate(q_lens):
            if n <= 1:
                continue
            for t0 in range(0, n, tokens_per_block):
                pos0 = seq_lens[s] - n + t0
                last = pos0 + min(tokens_per_block, n - t0) - 1
                first = max(0, pos0 - window + 1) if window else 0
                for h in range(nkv):
                    items[(s, t0, h)] = last // tile - first // tile + 1
        return items

    slots = 222  # one and a half places per SM of a 148-SM device
    cases = [([2048], [2048], 64, 64, 8, 0), ([7, 1, 300, 40], [7, 90, 1000, 45], 64, 64, 3, 0),
             ([500, 33], [900, 33], 32, 64, 2, 130), ([1, 1], [5, 9], 64, 64, 2, 0),
             ([256] + [1] * 8, [8000] + [4096] * 8, 64, 64, 8, 0), ([512], [40000], 64, 64, 8, 0),
             ([64], [40000], 64, 64, 8, 0)]
    for q_lens, seq_lens, per_block, tile, nkv, window in cases:
        table = ops.prefill_work_table(q_lens, seq_lens, per_block, tile, nkv, window, slots)
        want = blocks_of(q_lens, seq_lens, per_block, tile, nkv, window)
        assert table.shape == (table.shape[0], 8) and table.dtype == np.int32
        assert table.shape[0] <= len(want) + slots
        seen, places, tickets, lengths = {}, {}, {}, []
        for s, t0, h, lo, count, packed, slot0, unit in table.tolist():
            parts, part = packed & 255, packed >> 8
            tiles = want[(s, t0, h)]
            if parts == 1:
                assert (lo, count, part) == (0, -1, 0)
                count = tiles
            else:
                assert 1 < parts <= ops.PREFILL_MAX_PARTS and 0 <= part < parts and count >= 1
                places.setdefault((slot0, parts), set()).add((s, t0, h))
                tickets.setdefault(unit, set()).add((s, t0, h))
            seen.setdefault((s, t0, h), []).append((part, lo, count, parts))
            lengths.append(count)
        assert lengths == sorted(lengths, reverse=True)
        assert set(seen) == set(want)
        for key, runs in seen.items():
            runs.sort()
            assert [r[0] for r in runs] == list(range(runs[0][3]))  # every part once
            assert runs[0][1] == 0 and all(a[1] + a[2] == b[1] for a, b in zip(runs, runs[1:]))  # in order, no gap
            assert runs[-1][1] + runs[-1][2] == want[key]
        assert all(len(v) == 1 for v in places.values()) and all(len(v) == 1 for v in tickets.values())
        spans = sorted((slot0, slot0 + parts) for slot0, parts in places)
        assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))  # no two blocks share a place
        assert sorted(tickets) == list(range(len(tickets)))
        # A long block over few blocks is cut; a step with many blocks of its own is cut less or not at all.
        if q_lens == [512]:  # 64 blocks of 618 to 625 tiles on 222 places: four parts each
            assert {r[3] for runs in seen.values() for r in runs} == {4}
        if q_lens == [64]:
            assert {r[3] for runs in seen.values() for r in runs} == {ops.PREFILL_MAX_PARTS}
        if q_lens == [2048]:  # a whole prompt has blocks enough of its own: none is cut
            assert {r[3] for runs in seen.values() for r in runs} == {1}
        if q_lens == [1, 1]:
            assert table.shape[0] == 0
        padded = ops.prefill_work_table(q_lens, seq_lens, per_block, tile, nkv, window, slots, capacity=len(want) + slots)
        assert padded.shape[0] == len(want) + slots and (padded[: table.shape[0]] == table).all()
        assert (padded[table.shape[0]:, 0] == -1).all()

    monkeypatch.setattr(ops, "_ints_to_device", lambda values, device: values)
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    step = SimpleNamespace(workspace=None, q_lens=[300, 1], seq_lens_host=[5000, 77])
    work = ops._prefill_work_flat(step, 64, 64, 8, 0, None, 222)
    assert (work == ops.prefill_work_table([300, 1], [5000, 77], 64, 64, 8, 0, 222)).all()
    assert ops._prefill_work_flat(step, 64, 64, 8, 0, None, 222) is work  # built once per step


def test_which_prefill_kernel_a_step_takes():
    """One block to an SM pays for prompts from their first token, each at least 512 tokens long, that
    make at most two blocks to an SM; every other step takes the kernel with two blocks to an SM."""
    pays = lambda q, held, window=0: ops.wide_prefill_pays(q, held, 64, 8, window, 148)
    assert pays([512], [512]) and pays([1024], [1024]) and pays([2048], [2048]) and pays([2304], [2304])
    assert pays([512] * 4, [512] * 4) and pays([1024, 1024], [1024, 1024])
    assert pays([1, 2048, 1], [300, 2048, 77])                # requests that decode beside the prompt do not matter
    assert not pays([2432], [2432]) and not pays([4096], [4096]) and not pays([1536, 1536], [1536, 1536])  # too many blocks
    assert not pays([1024], [4096]) and not pays([512], [8192])  # portions of prompts under way
    assert not pays([256] * 8, [256] * 8) and not pays([2048, 300], [2048, 300])  # short prompts: short chains of tiles
    assert not pays([2048], [2048], window=600) and pays([2048], [2048], window=1024)
    assert not pays([1, 1], [50, 60]) and not pays([2048], None)
    assert ops.wide_prefill_pays([2048], [2048], 32, 8, 0, 148) is False  # groups of four: 512 blocks


def test_which_tcgen05_kernel_takes_gate_up_with_swiglu():
    """One SM to a 128-row tile or two SMs to a 256-row tile: the one that runs fewer waves of tiles
    (12,288 weight rows: 48 tiles of 128 output columns per tile of rows, 148 SMs or 74 pairs)."""
    pair = lambda rows, n=12288: ops._pair_pays(rows, n, 2048, 1, 148)
    assert not pair(264) and not pair(384)          # 144 tiles: one wave of SMs against two of pairs
    assert pair(385) and pair(512) and pair(768)    # two waves either way, and a pair's wave is the shorter
    assert pair(896) and pair(2048) and pair(8192)
    assert not pair(200)                            # under a pair's 256 rows
    assert not pair(896, 24576)                     # twice the columns: five waves of SMs against six of pairs
    assert ops.FUSED_GATE_ROWS <= 384


def test_prefill_work_table_counts_a_block_from_the_run_of_its_first_row():
    """With runs, a block's key tiles begin at the run that holds its first token (rows of a later
    run mask the rest), so the parts of a cut block cover exactly those tiles."""
    run, tile, per_block, nkv = 1024, 64, 32, 2
    table = ops.prefill_work_table([90], [2100], per_block, tile, nkv, 0, 222, run=run)
    covered = {}
    for s, t0, h, lo, count, packed, slot0, unit in table.tolist():
        parts, part = packed & 255, packed >> 8
        pos0 = 2100 - 90 + t0
        last = pos0 + min(per_block, 90 - t0) - 1
        first = pos0 - pos0 % run
        tiles = last // tile - first // tile + 1
        covered.setdefault((t0, h), []).append((lo, tiles if count < 0 else count, parts, part))
        assert count < 0 or 0 < count <= tiles
    assert len(covered) == 3 * nkv
    for (t0, h), pieces in covered.items():
        pos0 = 2100 - 90 + t0
        tiles = (pos0 + min(per_block, 90 - t0) - 1) // tile - (pos0 - pos0 % run) // tile + 1
        pieces.sort()
        assert [p[3] for p in pieces] == list(range(pieces[0][2]))
        assert pieces[0][0] == 0 and sum(p[1] for p in pieces) == tiles
        assert all(a[0] + a[1] == b[0] for a, b in zip(pieces, pieces[1:]))
    # The block that starts in the earlier run walks its tiles too; the one inside the last run only its own.
    assert sum(p[1] for p in covered[(0, 0)]) == 2099 // tile - 1024 // tile + 1 - (2099 // tile - 2041 // tile)
    assert sum(p[1] for p in covered[(64, 0)]) == 2099 // tile - 2048 // tile + 1
    # A window and a run together: the later of the two starts.
    both = ops.prefill_work_table([40], [3000], 64, tile, 1, 100, 0, run=2048)
    assert both.tolist()[0][4] == -1 and both.shape[0] == 1


def test_lightning_parts_divide_the_columns_and_fit_a_block():
    for requests in (1, 2, 8, 64):
        for heads in (1, 3, 16, 32):
            for dv in (7, 8, 16, 20, 24, 64, 96, 128, 192, 256):
                parts = ops.lightning_parts(requests, heads, dv, 148)
                cols = dv // parts
                assert dv % parts == 0 and 1 <= cols <= 384
                assert cols >= 8 or parts == 1 or dv // 8 == 0
    # One prompt of 16 heads: blocks for three quarters of the SMs, not two blocks an SM for the rest.
    assert ops.lightning_parts(1, 16, 128, 148) == 8
    assert ops.lightning_parts(64, 16, 128, 148) == 2


@pytest.mark.parametrize("d,page", [(64, 16), (16, 4)])  # prompts on tcgen05 and on mma.sync
@pytest.mark.parametrize("q_lens,beside", [([1, 4, 1], 1), ([1, 0, 1], 0), ([0, 1], 0), ([0, 1, 2], 1), ([1, 1], 0)])
def test_single_tokens_run_beside_a_prompts_kernel_only_where_there_is_one(monkeypatch, d, page, q_lens, beside):
    """The single tokens' attention leaves its wait to the prompts' kernel in front of it, so it may do that only
    behind a launch that has blocks: an entry of no tokens gives that kernel none."""
    calls = []

    def function(library, name, argtypes, defines=None):
        def call(*args):
            assert len(args) == len(argtypes)
            calls.append((name, args))
            return 0
        return call

    monkeypatch.setattr(ops, "_function", function)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    monkeypatch.setattr(ops, "_ints_to_device", lambda values, device: torch.from_numpy(np.ascontiguousarray(values)))
    monkeypatch.setattr(ops, "error_word", lambda device: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(ops, "_step_buffers", lambda step, device, wanted: [torch.zeros(1)] * len(wanted))
    held = [300 + n for n in q_lens]
    step = SimpleNamespace(num_seqs=len(q_lens), q_lens=q_lens, seq_lens_host=held, max_seq_len=max(held), decode_only=False,
                           workspace=None, cu_seqlens=torch.zeros(4), seq_lens=torch.zeros(3), positions=torch.zeros(9))
    kv = KVView(torch.zeros(2, 2, 2, page, d, dtype=torch.bfloat16), torch.zeros(len(q_lens), 100, dtype=torch.int32), None, page, None)
    ops.paged_attention(torch.zeros(sum(q_lens), 4, d, dtype=torch.bfloat16), kv, step, 1.0)
    launched = [name for name, _ in calls if "part_floats" not in name]
    assert launched[-1] == "omnia_attention_decode_tc" and len(launched) == 1 + beside
    assert calls[-1][1][-3] == beside and (not beside or "prefill" in launched[0])


def test_a_replayed_mixed_step_refuses_an_entry_without_tokens():
    """As an uncaptured step does, and before any page is taken."""
    from mlx_omnia_b200.engine.decode_graph import MixedGraphs
    from mlx_omnia_b200.engine.step import StepEntry

    graphs = MixedGraphs(SimpleNamespace(cache=SimpleNamespace(groups=[], page_size=16, capacity_tokens=lambda: 0)))
    entries = [StepEntry(SimpleNamespace(request_id=name), tokens, []) for name, tokens in (("a", [1, 2]), ("b", []))]
    with pytest.raises(ValueError, match="'b' brings no tokens"):
        graphs.run(("a shape",), entries)


@pytest.mark.parametrize("rows", [1, 16, 17, 600])
def test_experts_on_the_tensor_cores_take_bfloat16_only(monkeypatch, rows):
    """Every kernel that a step of so many rows would choose reads its operands as bfloat16."""
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    monkeypatch.setattr(ops, "_function", lambda *a: lambda *args: 0)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "error_word", lambda device: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(ops, "_step_buffers", lambda step, device, wanted: [torch.zeros(1, dtype=torch.int32)] * len(wanted))

    def experts(dtype):
        return ops.moe_experts(torch.zeros(rows, 16, dtype=dtype), None, None, torch.zeros(3, 16, 16, dtype=dtype),
                               torch.zeros(3, 16, 8, dtype=dtype), 2, None, tensor_cores=True, token_ids=torch.zeros(rows, dtype=torch.int32),
                               table=torch.zeros(5, 2, dtype=torch.int32))

    assert experts(torch.bfloat16).shape == (rows, 16)
    with pytest.raises(ops.KernelError, match="bfloat16"):
        experts(torch.float32)


@pytest.mark.parametrize("q_lens,short,long", [([1] * 31 + [32], list(range(31)), [31]), ([64, 1, 31, 40], [1, 2], [0, 3]),
                                               ([32, 100], None, "all"), ([1, 5, 31], "all", None), ([0, 32, 1], [0, 2], [1])])
def test_chunked_recurrence_takes_the_requests_that_bring_a_chunk(monkeypatch, q_lens, short, long):
    """Single tokens and short portions stay with the token kernel whoever shares their step."""
    calls = {}
    monkeypatch.setattr(ops, "_function", lambda library, name, argtypes, defines=None:
                        lambda *args: calls.update({name: args}) or 0)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    lists = {}
    monkeypatch.setattr(ops, "_ints_to_device", lambda values, device: lists.setdefault(len(lists), torch.from_numpy(values)))
    step = SimpleNamespace(num_seqs=len(q_lens), q_lens=q_lens, max_q_len=max(q_lens), workspace=None,
                           cu_seqlens=torch.zeros(9), state_slots=torch.zeros(9))
    ops.lightning_attention(torch.zeros(sum(q_lens), 320, dtype=torch.bfloat16), 0, 64, 128, 192, 4, 16, 16, torch.ones(4),
                            torch.ones(64), 1e-5, torch.zeros(4, 4, 16, 16), step)
    held = {t.data_ptr(): t.tolist() for t in lists.values()}
    for name, at, want in (("omnia_lightning_recurrence", 12, short), ("omnia_lightning_chunk", 13, long)):
        if want is None:
            assert name not in calls
            continue
        entries, count = calls[name][at: at + 2]
        assert count == (len(q_lens) if want == "all" else len(want))
        assert entries is None if want == "all" else held[entries] == want


def test_which_tcgen05_kernel_takes_the_experts():
    """Tiles of 256 rows where an expert's rows fill one, and from 384 rows on by the waves either kernel runs."""
    pair = lambda rows, experts=32, columns=768: ops._moe_pair_pays(rows * experts, experts, columns, 148)
    assert [rows for rows in range(64, 384) if pair(rows)] == list(range(136, 257))
    assert all(pair(rows) for rows in (400, 512, 700, 1024)) and pair(512, 128) and pair(400, 64, 512) and pair(512, 16, 1536)
    assert not pair(512, 8, 1024) and pair(400, 8, 1024) and pair(1024, 8, 1024)
    assert pair(1, 1, 8) is False and ops._moe_pair_pays(200, 1, 136, 148)


def test_which_experts_stream_their_weights():
    """Entries of eight rows up to six pairs an expert, of sixteen just above, tiles beyond, and for small matrices sooner."""
    entry = lambda rows, top, experts, hidden, inner: ops._moe_stream_rows(rows, rows * top, experts, hidden, inner)
    assert [entry(rows, 4, 32, 2048, 768) for rows in (1, 8, 9, 48, 49, 64, 65)] == [8, 8, 8, 8, 16, 16, 0]
    assert [entry(rows, 6, 64, 512, 512) for rows in (8, 16, 64, 65, 85)] == [8, 8, 8, 0, 0]
    assert [entry(rows, 8, 256, 1024, 256) for rows in (1, 8, 9, 64)] == [8, 8, 0, 0]
    assert [entry(rows, 6, 64, 2048, 384) for rows in (8, 16, 17)] == [8, 8, 0]
    assert [entry(rows, 8, 8, 2048, 1024) for rows in (8, 9, 16, 17)] == [8, 16, 16, 0]
    assert [entry(rows, 1, 2, 264, 24) for rows in (6, 7, 16)] == [8, 0, 0]


def test_decode_lists_of_pieces_where_there_is_work_for_every_block():
    """The same answer for all batches of a bucket, one round of blocks while a head has two places a request, and chunks at fixed
    positions for one or two requests, for short ones and for more requests than a list is made for."""
    assert ops.decode_places(1, 8, 100000, 148) == ops.decode_places(2, 8, 4096, 148) == (0, 0)
    assert ops.decode_places(8, 8, 4096, 148) == ops.decode_places(5, 8, 4096, 148) == (111, 1)
    assert ops.decode_places(8, 8, 2000, 148) == (0, 0) and ops.decode_places(256, 8, 4096, 148) == (0, 0)
    assert ops.decode_places(64, 8, 2304, 148) == (111, 2)
    # More requests than places, and few with heads of which an SM holds three blocks, were slower by a list.
    assert ops.decode_places(100, 8, 700, 148) == ops.decode_places(128, 8, 4096, 148) == (0, 0)
    assert ops.decode_places(16, 4, 3000, 148, 256) == (0, 0) and ops.decode_places(16, 4, 3000, 148, 128) == (222, 1)
    assert ops.decode_places(24, 4, 2304, 148, 256) == (222, 1)


def _calls_of_decode_attention(monkeypatch):
    """What is launched, (name, arguments), where decode attention runs on this machine's memory without a kernel behind it."""
    calls = []
    monkeypatch.setattr(ops, "_scratch", {})  # (what this machine's memory stands in for is not left to the tests of a GPU)
    monkeypatch.setattr(ops, "_zeroed", set())
    monkeypatch.setattr(ops, "_function", lambda library, name, argtypes, defines=None: lambda *args: calls.append((name, args)) or 0)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    monkeypatch.setattr(ops, "error_word", lambda device: torch.zeros(1, dtype=torch.int32))
    return calls


def _decode_step(lengths):
    step = SimpleNamespace(num_seqs=len(lengths), q_lens=[1] * len(lengths), seq_lens_host=lengths, max_seq_len=max(lengths),
                           decode_only=True, workspace=None, cu_seqlens=torch.zeros(len(lengths) + 1), seq_lens=torch.tensor(lengths))
    kv = KVView(torch.zeros(2, 2, 8, 16, 128, dtype=torch.bfloat16), torch.zeros(len(lengths), 300, dtype=torch.int32), None, 16, None)
    return step, lambda: ops.paged_attention(torch.zeros(len(lengths), 16, 128, dtype=torch.bfloat16), kv, step, 1.0)


LIST_ARGUMENT = 32  # of omnia_attention_decode_tc


def test_a_list_of_pieces_is_the_passes_own(monkeypatch):
    """Two steps whose layers run in turn have a list each, made once a pass; and there is none for a layer that is run by
    itself, whose caller may have moved the lengths on since the last call."""
    calls = _calls_of_decode_attention(monkeypatch)
    lists = lambda: [args[LIST_ARGUMENT] for name, args in calls if name == "omnia_attention_decode_tc"]  # noqa: E731
    made = lambda: [args[9] for name, args in calls if name == "omnia_decode_pieces"]  # noqa: E731
    (first, a), (second, b) = _decode_step([3000, 70] * 8), _decode_step([1500] * 16)
    a(), a()
    assert lists() == [None, None] and not made()
    ops.begin_pass(first), ops.begin_pass(second)
    calls.clear()
    a(), b(), a(), b()
    assert len(made()) == 2 and lists() == made() * 2 and made()[0] != made()[1] and None not in lists()
    ops.end_pass(first)
    calls.clear()
    a(), b()
    assert lists()[0] is None and lists()[1] is not None and not made()


def test_a_table_of_angles_is_the_passes_own(monkeypatch):
    """As the lists: one a pass, whichever steps' layers run between, and none kept outside of one."""
    calls = []
    monkeypatch.setattr(ops, "_function", lambda *a, **b: lambda *args: calls.append(args) or 0)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    a, b = (SimpleNamespace(num_tokens=9, positions=torch.arange(9), workspace=None) for _ in range(2))
    inv = torch.ones(4)
    ops.rope_angles(a, inv), ops.rope_angles(a, inv)
    assert len(calls) == 2
    ops.begin_pass(a), ops.begin_pass(b)
    tables = [ops.rope_angles(step, inv) for step in (a, b, a, b)]
    assert len(calls) == 4 and tables[0] is tables[2] and tables[1] is tables[3]
    assert tables[0].data_ptr() != tables[1].data_ptr() and tables[0].numel() == 4 * 9 * 2
    ops.end_pass(a)
    ops.rope_angles(a, inv)
    assert len(calls) == 5


def test_a_captured_step_keeps_what_a_pass_makes_where_the_pass_before_made_it(monkeypatch):
    """Nothing that a graph's kernels share between layers is allocated by the capture."""
    monkeypatch.setattr(ops, "_function", lambda *a, **b: lambda *args: 0)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "sm_count", lambda device=None: 148)
    step = SimpleNamespace(num_tokens=9, num_seqs=9, positions=torch.arange(9), seq_lens=torch.arange(9), workspace={"private": True})
    kv, inv, made = KVView(torch.zeros(1, 2, 8, 16, 128), None, None, 16, None), torch.ones(4), []
    for _ in range(2):
        ops.begin_pass(step)
        made.append((ops.rope_angles(step, inv), ops._decode_list(step, kv, 0, 8, 128, 111, 1, torch.device("cpu"))[0]))
        ops.end_pass(step)
    assert all(a is b for a, b in zip(*made))
