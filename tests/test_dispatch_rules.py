"""Host-side rules that pick kernels and orders: no GPU needed."""
from qorvix_b200 import StepEntry
from qorvix_b200.csrc import ops
from qorvix_b200.engine.runner import single_token_entries_first


def test_single_token_entries_run_first_and_rows_map_back():
    e = [StepEntry("p1", [1, 2, 3], [0, 2]), StepEntry("d1", [4], [0]), StepEntry("p2", [5, 6], []),
         StepEntry("d2", [7], [0]), StepEntry("d3", [8], [])]
    order, back = single_token_entries_first(e)
    assert order == [1, 3, 4, 0, 2]                      # decoded tokens first, each kind in the caller's order
    # the step's output rows are d1, d2, p1[0], p1[2]; the caller wants p1[0], p1[2], d1, d2
    assert back == [2, 3, 0, 1]
    # nothing to undo when the caller's order is already that
    assert single_token_entries_first([e[1], e[3], e[0]]) == ([0, 1, 2], None)
    assert single_token_entries_first([]) == ([], None)


def test_decode_attention_slices():
    # few (token, kv head) pairs: the slices fill one wave of 296 CTAs, at least 256 keys each
    assert ops.decode_variant(8, 8) == 0 and ops.decode_splits(8, 8, 1024) == 4
    assert ops.decode_splits(8, 8, 8192) == 4
    assert ops.decode_splits(8, 8, 300) == 1
    # more pairs than one wave holds: the count whose waves take the least time ...
    assert ops.decode_splits(8, 40, 2048) == 3
    assert ops.decode_splits(64, 8, 8192) == 4
    assert ops.decode_splits(64, 8, 1024) == 1
    # ... but only where the context is known; a captured step keeps one wave
    assert ops.decode_splits(64, 8, 8192, known=False) == 1
    assert ops.decode_splits(8, 8, 8192, known=False) == 4
    # very few pairs take the per-thread-load kernel with about three CTAs per SM
    assert ops.decode_variant(1, 8) == 1 and 1 <= ops.decode_splits(1, 8, 1024) <= 16
    for T in (1, 3, 8, 17, 64):
        for hkv in (1, 2, 8, 40):
            for ctx in (1, 63, 64, 1000, 8192, 100000):
                for known in (True, False):
                    assert 1 <= ops.decode_splits(T, hkv, ctx, known=known) <= 16


def test_switches(monkeypatch):
    monkeypatch.delenv("QORVIX_FOLDED_NORM", raising=False)
    monkeypatch.delenv("QORVIX_FUSED_ROPE", raising=False)
    assert ops.folded_norm_enabled(1) and ops.folded_norm_enabled(16) and not ops.folded_norm_enabled(17)
    assert ops.fused_rope_enabled(65) and not ops.fused_rope_enabled(64)
    monkeypatch.setenv("QORVIX_FOLDED_NORM", "0")
    assert not ops.folded_norm_enabled(8)
    monkeypatch.setenv("QORVIX_FOLDED_NORM", "64")
    assert ops.folded_norm_enabled(64) and not ops.folded_norm_enabled(65)
    monkeypatch.setenv("QORVIX_FUSED_ROPE", "0")
    assert not ops.fused_rope_enabled(2048)


def _stub_rmsnorm(calls, name):
    """An RMSNorm object without a device: add_norm only records what it is given."""
    import torch
    from qorvix_b200.parts.rmsnorm import RMSNorm
    n = object.__new__(RMSNorm)
    n.size, n.eps, n.weight = 8, 1e-5, torch.ones(8)

    def add_norm(residual, delta, rows=None):
        calls.append((name, "add_norm", type(delta).__name__))
        return torch.zeros(residual.shape[0], 8)
    n.add_norm = add_norm
    return n


def test_pre_norm_block_hands_a_prepared_norm_input_only_to_parts_that_take_it(monkeypatch):
    """The routing of PreNormed between the parts of a block, with stub parts (no kernels run)."""
    import torch
    from qorvix_b200.parts.base import PreNormed
    from qorvix_b200.parts.block import PreNormBlock
    monkeypatch.delenv("QORVIX_FOLDED_NORM", raising=False)
    calls = []
    n1, n2, n_after = _stub_rmsnorm(calls, "n1"), _stub_rmsnorm(calls, "n2"), _stub_rmsnorm(calls, "after")

    class FoldingMixer:
        folds_norms = True

        def forward(self, x, ctx, cache, residual=None, next_norm=None):
            calls.append(("mixer", type(x).__name__, next_norm))
            return PreNormed(scaled=torch.zeros(2, 8), stats=torch.zeros(1, 64), norm=next_norm, residual=residual)

    class FoldingFfn:
        folds_norms = True

        def forward(self, x, ctx, residual=None, next_norm=None):
            calls.append(("ffn", type(x).__name__, next_norm))
            return PreNormed(scaled=torch.zeros(2, 8), stats=torch.zeros(1, 64), norm=next_norm, residual=residual)

    class PlainFfn:
        def forward(self, x, ctx):
            calls.append(("plain_ffn", type(x).__name__, None))
            return torch.zeros(2, 8)

    class Ctx:
        next_norm = None

    def block(mixer, ffn):
        b = object.__new__(PreNormBlock)
        b.mixer_norm, b.mixer, b.ffn_norm, b.feed_forward = n1, mixer, n2, ffn
        return b

    residual = torch.zeros(2, 8)
    ctx = Ctx()
    ctx.next_norm = n_after
    # both parts fold: the mixer prepares the ffn norm's input, the ffn takes it as it is and prepares the next block's
    _, pending = block(FoldingMixer(), FoldingFfn()).forward(residual, None, ctx, None)
    assert calls == [("n1", "add_norm", "NoneType"), ("mixer", "Tensor", n2), ("ffn", "PreNormed", n_after)]
    assert isinstance(pending, PreNormed) and pending.norm is n_after
    # a block that gets a PreNormed made for its first norm hands it to a folding mixer without running the norm
    calls.clear()
    block(FoldingMixer(), FoldingFfn()).forward(residual, PreNormed(torch.zeros(2, 8), torch.zeros(1, 64), n1, residual), ctx, None)
    assert calls[0] == ("mixer", "PreNormed", n2)
    # a feed-forward that does not fold gets normed rows: its norm is run on the PreNormed (the stream is complete)
    calls.clear()
    _, pending = block(FoldingMixer(), PlainFfn()).forward(residual, None, ctx, None)
    assert calls == [("n1", "add_norm", "NoneType"), ("mixer", "Tensor", n2), ("n2", "add_norm", "PreNormed"),
                     ("plain_ffn", "Tensor", None)]
    assert isinstance(pending, torch.Tensor)
    # many tokens: nothing is folded, the parts are called the plain way (no keywords)
    calls.clear()
    big = torch.zeros(100, 8)

    class CountingMixer:
        folds_norms = True

        def forward(self, x, ctx, cache, **kw):
            calls.append(("mixer_kw", sorted(kw)))
            return torch.zeros(100, 8)

    block(CountingMixer(), PlainFfn()).forward(big, None, ctx, None)
    assert ("mixer_kw", []) in calls
    # no folding norm after the block (another kind of norm, or the final norm): the last part is told so
    calls.clear()
    ctx.next_norm = object()
    block(FoldingMixer(), FoldingFfn()).forward(residual, None, ctx, None)
    assert calls[-1] == ("ffn", "PreNormed", None)
    # a norm class the package has never seen opts in by declaring the capability, nothing else
    class ForeignNorm:
        folds_into_products = True
        size, eps = 8, 1e-6

        def scale_weight(self):
            return torch.ones(8)

    calls.clear()
    ctx.next_norm = ForeignNorm()
    block(FoldingMixer(), FoldingFfn()).forward(residual, None, ctx, None)
    assert calls[-1] == ("ffn", "PreNormed", ctx.next_norm)


def test_latent_portions_choose_by_what_either_path_costs():
    """The faster path as measured (us a layer over the latents, with keys and values formed per head), 148 SMs."""
    pays = lambda lens, pos0, H, rank: ops.latent_expand_pays(lens, pos0, H, rank, H * 256, 0, 148)
    for H, rank, new, cached, carried, expanded in (
            (16, 512, 32, 2000, 78, 85), (16, 512, 64, 2000, 115, 90), (16, 512, 128, 2000, 176, 85), (16, 512, 32, 8000, 140, 216),
            (16, 512, 64, 8000, 258, 218), (16, 512, 128, 8000, 469, 190), (16, 512, 2048, 0, 1024, 147), (8, 256, 32, 8000, 88, 175),
            (8, 256, 64, 8000, 141, 179), (8, 256, 128, 8000, 256, 142), (8, 256, 128, 2000, 112, 66), (64, 512, 32, 2000, 176, 151),
            (64, 512, 32, 8000, 465, 391)):
        assert pays([new], [cached], H, rank) == (expanded < carried), (H, rank, new, cached)
    assert not pays([1, 31], [9, 9000], 16, 512)                                # no portion
    assert not pays([1, 1, 32], [700, 900, 8000], 16, 512)                      # behind single tokens
    assert pays([512, 8], [0, 8000], 16, 512)                                   # one CTA a tile over the latents: 900 us and 278
    assert ops.latent_expand_pays([64], [8000], 8, 256, 2048, 500, 148)         # a window leaves few rows to form
    assert ops.latent_expand_pays([64], [2000], 16, 512, 4096, 0, 148, 64 * 2033) and not ops.latent_expand_pays([64], [2000], 16, 512, 4096, 0, 148, 64 * 2034)


def test_delta_rule_segments_that_go_token_by_token():
    assert ops.delta_lead([1, 1, 1], 128) == 3 and ops.delta_lead([15], 128) == 1
    assert ops.delta_lead([1, 1, 3, 16], 128) == 3                              # a portion does not take the single tokens with it
    assert ops.delta_lead([300, 2], 128) == 0 and ops.delta_lead([1, 300, 2], 256) == 1
    assert ops.delta_lead([1, 200], 64) == 2 and ops.delta_lead([200], 130) == 1  # short keys, keys that are no multiple of four
    assert ops.delta_lead([200], 128, blocks=False) == 1 and ops.delta_lead([200], 260) == 1


def test_differential_attention_segments_that_share_tiles_of_portions():
    assert ops.diff_rows_first([1, 1, 600]) == 2 and ops.diff_rows_first([20] * 8 + [600]) == 8       # short segments ahead keep their kernel
    assert ops.diff_rows_first([64]) == 0 and ops.diff_rows_first([63, 20]) == 2
    assert ops.diff_rows_first([600, 3]) == 0 and ops.diff_rows_first([300] + [20] * 8) == 9          # behind: a tile each


def test_no_room_is_an_answer(monkeypatch):
    import torch
    assert ops._room((2, 3), torch.float32, "cpu").shape == (2, 3)

    def full(*a, **k):
        raise torch.OutOfMemoryError("no room")
    monkeypatch.setattr(ops.torch, "empty", full)
    assert ops._room((2, 3), torch.float32, "cpu") is None


def test_remote_shared_memory_is_touched_behind_a_cluster_barrier_only():
    """A CTA's shared memory may be read or written by another CTA of its cluster once that CTA is known to run: in every kernel a cluster
    barrier is arrived at and waited for ahead of the first access (and, so that no CTA leaves early, behind the last one)."""
    import re
    from pathlib import Path
    seen = 0
    for path in sorted(Path(ops.__file__).parent.glob("*.cu*")):
        for kernel in re.split(r"__global__", path.read_text())[1:]:
            remote = [m.start() for m in re.finditer(r"(?:ld|st|red|atom)(?:\.\w+)*\.shared::cluster|dst_smem_cluster|map_shared_rank", kernel)]
            if not remote:
                continue
            seen += 1
            waits = [m.start() for m in re.finditer(r"barrier\.cluster\.wait|\bcl\.sync\(\)", kernel)]
            arrives = [m.start() for m in re.finditer(r"barrier\.cluster\.arrive|\bcl\.sync\(\)", kernel)]
            assert waits and waits[0] < remote[0] and arrives[0] <= waits[0], f"{path.name}: remote shared memory ahead of a cluster barrier"
            assert waits[-1] > remote[-1], f"{path.name}: a CTA may leave while its shared memory is in use"
    assert seen >= 2


def test_weights_are_read_ahead_of_the_wait_only_where_the_caller_says_they_lie_still(monkeypatch):
    """A launch may start while the one in front of it still runs; what it reads ahead of its wait must not be what that one writes.  So the
    32-bit products read w early for a model's layers alone, and the kernels have no other load there."""
    import re
    from pathlib import Path
    from types import SimpleNamespace

    import torch
    from qorvix_b200.parts.linear import Linear

    flags = []
    entry = SimpleNamespace(qv_gemm_simt=lambda *a: flags.append(a[12]) or 0)
    monkeypatch.setattr(ops, "_lib", lambda name: entry)
    monkeypatch.setattr(ops, "_need_cuda", lambda *a: None)
    monkeypatch.setattr(ops, "_stream", lambda: None)
    x, w, out = torch.zeros(2, 8), torch.zeros(4, 8), torch.zeros(2, 4)
    ops.gemm_simt(out, x, w)
    ops.gemm_simt(out, x, w, accumulate=True)
    ops.gemm(out, x, w)
    layer = object.__new__(Linear)
    layer.weight, layer.packed, layer.out_features = w, None, 4
    layer.forward(x)
    assert flags == [0, 1, 0, 0x100]

    for name, kernel, early in (("gemm_simt.cu", "gemm_simt_kernel", "if (ASYNC && settled)"), ("channel_scan.cu", "channel_gates_tile_kernel", None),
                                ("latent_attention.cu", "heads_gemm_kernel", "if (early)")):
        text = (Path(ops.__file__).parent / name).read_text()
        body = text[re.search(r"__global__[^;{]*\b%s\(" % kernel, text).end():]
        ahead = body[: body.index("pdl_wait();")]
        ahead = ahead[ahead.rindex("};") + 2:] if "};" in ahead else ahead            # behind the lambdas that are only defined there
        loads = re.findall(r"\bstage\(|\bfetch\(|w2t\[", ahead)
        assert (len(loads) == 1 and early in ahead) if early else not loads, (kernel, ahead)


def test_long_rows_of_logits_share_a_cluster_while_that_is_one_wave():
    ctas = lambda rows, V: ops._lib("sampling").qv_argmax_ctas(rows, V)
    assert ctas(1, 16384) == ctas(8, 128256) == ctas(18, 16384) == ctas(64, 65536) == 8
    assert ctas(8, 16383) == ctas(64, 16384) == ctas(64, 65535) == ctas(65, 128256) == ctas(256, 128256) == 1


def test_which_portions_the_delta_rule_takes_in_blocks():
    lead = ops.delta_lead
    assert lead([16], 128, heads=16) == 1 and lead([31], 128, heads=32) == 1 and lead([32], 128, heads=1) == 0
    assert lead([1] * 63 + [16], 128, heads=16) == 63 and lead([1] * 32 + [16], 128, heads=8) == 33
    assert lead([1] * 5 + [16] * 8, 128, heads=16) == 5 and lead([1] * 5 + [16] * 8, 128, heads=8) == 13
    assert lead([1, 32, 40], 256, heads=4) == 3 and lead([1, 32, 48], 256, heads=4) == 2 and lead([1, 32], 256, heads=16) == 1
    assert lead([255], 64, heads=8) == 1 and lead([1, 256], 64, heads=8) == 1 and lead([256] * 32, 64, heads=32) == 0
    assert lead([256] * 8, 32, heads=16) == 0 and lead([256] * 9, 32, heads=16) == 9 and lead([256], 32, heads=64) == 0
    assert lead([999], 126) == lead([999], 260) == lead([999], 128, blocks=False) == 1


def test_gates_take_tiles_where_there_are_enough_of_them():
    tiles = lambda *a: ops._lib("channel_scan").qv_channel_gates_tiles(*a)
    softplus, linear = ops.GATE_EXP_NEG_SOFTPLUS, ops.GATE_LINEAR
    assert tiles(1531, 2048, 64, softplus) and tiles(1531, 2048, 64, linear) and tiles(512, 2048, 16, linear) and tiles(300, 4096, 32, softplus)
    assert not tiles(2048, 128, 64, softplus) and not tiles(512, 2048, 32, softplus) and not tiles(512, 4096, 16, softplus) and not tiles(300, 2048, 64, linear)
    assert not tiles(255, 65536, 64, linear) and not tiles(2048, 2048, 40, linear) and not tiles(2048, 2048, 144, linear)


def test_from_where_long_segments_of_the_gated_recurrence_take_three_launches():
    least = lambda *a: ops._lib("recurrent").qv_linear_scan_parallel_from(*a)
    never = 2 ** 31 - 1
    assert least(ops.SCAN_GATED_MAX, 4, 256, 512) == least(ops.SCAN_GATED_MAX, 16, 256, 256) == 896 and least(ops.SCAN_GATED_MAX, 1, 64, 64) == 1024
    assert least(ops.SCAN_GATED_MAX, 4, 128, 256) == least(ops.SCAN_GATED_MAX, 16, 256, 64) == least(ops.SCAN_GATED_MAX, 4, 64, 64) == 1024
    assert least(ops.SCAN_GATED_MAX, 32, 128, 128) == 2048 and least(ops.SCAN_GATED_MAX, 64, 128, 64) == least(ops.SCAN_GATED_MAX, 16, 64, 64) == never
    assert least(ops.SCAN_DECAY, 4, 256, 512) == least(ops.SCAN_GATED_MAX, 1, 264, 64) == never


def test_which_portions_take_the_passes_of_several_warps_a_token():
    latent = lambda *a: ops._lib("latent_attention").qv_latent_prepare_vec(*a)
    assert latent(33, 8) and latent(149, 16) and latent(2048, 32)
    assert not latent(32, 8) and not latent(148, 16) and not latent(2048, 64)
    diff = lambda *a: ops._lib("diff_attention").qv_diff_prepare_vec(*a)
    assert diff(33, 64, 16, 64) and diff(33, 16, 4, 128) and diff(149, 32, 8, 128)
    assert not diff(32, 8, 4, 64) and not diff(148, 32, 8, 128)


def test_the_routers_rows():
    rows = lambda *a: ops._lib("moe").qv_moe_route_rows(*a)
    assert rows(2048, 65, 512) and rows(1024, 33, 512) and rows(2048, 33, 2048) and rows(300, 9, 1024)
    assert not rows(2048, 33, 512) and not rows(1025, 40, 2040) and not rows(300, 9, 512)
