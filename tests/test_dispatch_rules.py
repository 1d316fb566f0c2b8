"""Rules that choose how a kernel is launched, as far as they are plain arithmetic (no GPU)."""
import pytest

from flyweight_b200.kernels import attention

SM_COUNT = 148


@pytest.mark.parametrize("head_dim", [64, 128])
def test_the_context_slices_of_a_decode_step_cover_the_context_and_bound_a_cta(head_dim):
    """Every choice of ``decode_splits`` covers all tiles, leaves no slice empty, lets no CTA walk more
    than 128 tiles unless the context needs more than 64 slices of them, merges in a cluster only what a
    cluster can hold, and keeps all CTAs resident at once when that is possible at all."""
    resident = SM_COUNT * (5 if head_dim <= 64 else 3)
    for n_kv in (1, 4, 8):
        for n_tokens in (1, 2, 3, 8, 16, 31, 32, 48, 64, 96, 128, 200, 256, 512, 1000):
            for max_tiles in (1, 2, 7, 8, 9, 17, 64, 65, 129, 257, 513, 1000, 1985, 9000):
                splits, per, in_cluster = attention.decode_splits(n_tokens, n_kv, max_tiles, head_dim)
                what = (n_tokens, n_kv, max_tiles, splits, per, in_cluster)
                assert 1 <= splits <= 64 and per >= 1, what
                assert splits * per >= max_tiles > (splits - 1) * per, what          # covered, no empty slice
                assert per <= 128 or splits >= 32, what
                if in_cluster:
                    assert 1 < splits <= 8 and n_tokens * n_kv * splits <= attention.CLUSTER_MERGE_CTAS, what
                pairs = n_tokens * n_kv
                if pairs <= resident and max_tiles <= 128:
                    assert pairs * splits <= resident or splits == 1, what            # one round of the SMs


def test_the_measured_points_of_the_slicing_rule():
    """The choices the rule was fitted to (8 KV heads, head size 64; tiles of 64 keys)."""
    chosen = lambda batch, tiles: attention.decode_splits(batch, 8, tiles)
    assert chosen(8, 65) == (8, 9, True)            # 8 x 4,096 keys: eight slices in a cluster
    assert chosen(16, 65)[0] == 4 and chosen(32, 65)[0] == 2
    assert chosen(48, 65)[0] == 1 and chosen(64, 65)[0] == 1 and chosen(256, 9)[0] == 1
    assert chosen(128, 65)[0] == 2                  # one piece would be 1.4 rounds of the SMs
    assert chosen(8, 513) == (8, 65, True)          # 8 x 32,768 keys
    assert chosen(1, 1985)[0] >= 32 and not chosen(1, 1985)[2]      # one long request: a merge kernel


@pytest.mark.parametrize("mask,fused", [({}, True), ({"window": 64}, False), ({"chunk": 64}, False)])
def test_the_decode_kernel_that_rotates_knows_no_mask(monkeypatch, mask, fused):
    """It walks every earlier key, so a mixer with a window or with chunks goes by the kernels that take its span."""
    from types import SimpleNamespace
    import torch
    from flyweight_b200.config import PartSpec
    from flyweight_b200.kernels import ops
    from flyweight_b200.parts import build_mixer
    from flyweight_b200.parts.base import PositionEncoding
    names = {role: role for role in ("q", "k", "v", "o")}
    mixer = build_mixer(PartSpec("gqa_attention", {
        "hidden_size": 64, "num_heads": 8, "num_kv_heads": 2, "head_dim": 64,
        "position": PartSpec("rope_half_split", {"theta": 1e4, "rotary_dim": 64}), **mask}, names))
    mixer.position.prepare(16, "cpu")
    mixer.w_qkv = torch.zeros(12 * 64, 64, dtype=torch.bfloat16)
    went = []
    monkeypatch.setattr(ops, "linear", lambda h, w, dtype: torch.zeros(1, 12 * 64, dtype=dtype))
    monkeypatch.setattr(ops, "linear_into_residual", lambda out, w, residual: out)
    monkeypatch.setattr(attention, "fused_decode_attention", lambda *args: went.append("fused"))
    monkeypatch.setattr(PositionEncoding, "encode", lambda self, *args, **kw: went.append("encode"))
    monkeypatch.setattr(attention, "paged_attention", lambda ctx, q, cache, table, heads, span, *rest, **kw: went.append(span))
    cache = SimpleNamespace(k_pool=torch.zeros(1, 2, 64, 64, dtype=torch.bfloat16), v_pool=None, group=0)
    ctx = SimpleNamespace(batch=SimpleNamespace(block_tables=[torch.zeros(1, 1, dtype=torch.int32)], max_segment=1, n_tokens=1),
                          precision=SimpleNamespace(act_dtype=torch.bfloat16))
    mixer.forward(ctx, torch.zeros(1, 64, dtype=torch.bfloat16), cache)
    assert went == (["fused"] if fused else ["encode", mixer.span])


@pytest.mark.parametrize("requests,tiles,front_bytes,fused", [
    (4, 65, 4 << 20, False), (8, 65, 4 << 20, False), (8, 126, 4 << 20, False), (4, 65, 12 << 20, True),
    (2, 126, 4 << 20, True), (8, 33, 4 << 20, True), (16, 65, 4 << 20, True), (64, 17, 4 << 20, True)])
def test_many_clusters_of_eight_keep_the_small_kernel_behind_a_short_product(requests, tiles, front_bytes, fused):
    """The measured points of the rule (8 KV heads of 64, pages of 64 keys)."""
    from types import SimpleNamespace
    import torch
    cache = SimpleNamespace(k_pool=torch.zeros(1, 8, 64, 64, dtype=torch.bfloat16))
    ctx = SimpleNamespace(batch=SimpleNamespace(max_segment=1, n_tokens=requests),
                          precision=SimpleNamespace(act_dtype=torch.bfloat16))
    qkv, table = torch.zeros(1, 1, dtype=torch.bfloat16), torch.zeros(requests, tiles, dtype=torch.int32)
    assert attention.decode_fusable(ctx, qkv, cache, table, 16, 64, 0, front_bytes) == fused


def test_a_convolution_step_refuses_what_the_convolution_refuses():
    """Fewer than two taps, more than sixteen, a slot shorter than its contents: the argument checks of the C entries
    answer before anything is launched, the folded step as the convolution's own kernel."""
    from flyweight_b200.kernels import lib
    unsupported, bad = -2, -1
    here = 4096                                     # a pointer that nobody reads
    for taps, stride, want in ((1, 1024, unsupported), (17, 1 << 20, unsupported), (3, 127, bad)):
        alone = lib.library().fwb_shortconv(here, 1, here, None, here, here, here, here, here, 1, 4, 4, 64, taps, stride, None)
        folded = lib.library().fwb_linear_rows_conv(here, None, 0.0, here, here, None, here, stride, here, here, 4, 64, 256,
                                                    taps, None)
        assert alone == folded == want, (taps, stride)


@pytest.mark.parametrize("switch", ["none", "rows", "mid_size_split", "pairs", "forced_splits"])
def test_the_products_rules_are_the_same_in_both_languages(switch):
    """The native step plan states the rules of ``kernels/tensorcore.py`` again: over token counts on both sides of every
    line, ragged and even features and K, plain and gated, and with each switch turned, both choose the same."""
    import ctypes
    from flyweight_b200.kernels import lib, tensorcore as tc
    turn = {"none": lambda on: None, "rows": tc.set_rows_enabled, "mid_size_split": tc.set_mid_size_split,
            "pairs": tc.set_pairs_enabled, "forced_splits": lambda on: tc.force_splits(None if on else 2)}[switch]
    out = (ctypes.c_int * 14)()
    turn(False)
    try:
        for M in (1, 7, 8, 9, 12, 13, 16, 17, 32, 33, 48, 64, 65, 77, 96, 97, 100, 128, 129, 160, 192, 256, 300, 512, 513, 2048):
            for N in (8, 130, 384, 1000, 1024, 2048, 3072, 3840, 4608, 4864, 5120, 6144, 8192, 9216, 9600, 13312, 16384, 65536):
                for K in (8, 64, 256, 504, 512, 1024, 1032, 1912, 2048, 4096, 4608, 8192, 10752):
                    for acc in (1, 2):
                        assert lib.library().fwb_product_rules(M, N, K, acc, ctypes.addressof(out)) == 0
                        rings = tc.two_rings(M, N, K, acc) or (0, 0, 0)
                        mid = (False, 0, 0)
                        if tc.MID_FROM <= M <= tc.MID_TO:
                            kind, tile, splits = tc.mid_size_choice(M, N, K, acc, acc == 1 and M > 128 and N >= 256)
                            mid = (True, 0, 0) if kind == "pair" else (False, tile, splits)
                        splits = tc._splits_for(M, N, K, acc)
                        want = (tc._rows_takes(M, acc * N, K), tc._rows_takes_normed(M, acc * N, K), *rings,
                                tc._pairs_add(M, N), *mid, tc._decode_tile(M, N), tc.pick_splits(M, N, K), splits,
                                tc._ring_depth(M, N, splits, acc), tc._rows_takes_conv(M, N, K))
                        assert tuple(out) == tuple(int(v) for v in want), (M, N, K, acc)
    finally:
        turn(True)


def test_two_rings_of_weights_keep_their_clusters_resident():
    """A cluster of CTAs lies in one GPC: on this chip 70 clusters of four fit at two CTAs an SM, 104 at three, 33 of eight.
    A choice beyond that takes a second round, longer than the choice it replaced (9216 x 2048 at 77 tokens 15.2 -> 21.9
    us), but for the sizes where that one has a second round too."""
    from flyweight_b200.kernels import tensorcore as tc
    for M in (33, 64, 65, 96, 97, 128, 129, 160, 192, 193, 256, 300, 384, 512):
        for tiles in range(1, 160):
            for k_blocks in (16, 31, 32, 64, 128):
                for acc in (1, 2):
                    choice = tc.two_rings(M, tiles * 128, k_blocks * 64, acc)
                    if choice is None:
                        continue
                    tile, splits, stages = choice
                    an_sm = min(3, 227 * 1024 // (stages * (acc * 16384 + tile * 128) + 2560))
                    clusters, fit = tiles * -(-M // tile), {(4, 2): 70, (4, 3): 104, (8, 2): 33}[splits, an_sm]
                    two_rounds_anyway = splits == 8 and tile == 96 and (tiles >= 34 or 128 < M <= 192 and tiles >= 17)
                    assert clusters <= fit or (two_rounds_anyway and clusters <= 37), (M, tiles, k_blocks, acc, choice)


def test_the_weight_reader_leaves_what_it_is_slower_at():
    """Sizes on both sides of its lines (measured beside the rule): a head of 65,536 features over 1,024 channels, short
    K under many features, wide matrices from nine tokens on, shares that leave SMs idle under a long K."""
    from flyweight_b200.kernels import tensorcore as tc
    for M, N, K in ((1, 65536, 1024), (8, 65536, 1024), (16, 65536, 1024), (8, 32768, 512), (8, 28672, 1536), (8, 4864, 5120),
                    (16, 19456, 1024), (16, 9216, 1536), (16, 12288, 2048), (24, 9728, 1024), (32, 8192, 1024), (32, 16384, 512)):
        assert not tc._rows_takes(M, N, K), (M, N, K)
    for M, N, K in ((1, 1024, 1024), (8, 9216, 1024), (8, 32768, 1024), (8, 2048, 8192), (8, 16384, 2048), (8, 6144, 5120),
                    (16, 18432, 1024), (16, 2048, 2048), (12, 6144, 2048), (16, 16384, 2048), (24, 3072, 1024), (24, 9216, 1024), (32, 8192, 512)):
        assert tc._rows_takes(M, N, K), (M, N, K)


def test_the_slicing_rule_is_the_same_in_both_languages_and_merges_only_what_pays():
    import ctypes
    from flyweight_b200.kernels import lib
    out = (ctypes.c_int * 3)()
    for head_dim in (64, 128):
        for n_kv in (1, 2, 4, 8):
            for n_tokens in (1, 2, 4, 8, 9, 16, 18, 32, 37, 64, 74, 75, 128, 300):
                for max_tiles in (*range(1, 33), 64, 65, 129, 513, 1985, 9000):
                    chosen = attention.decode_splits(n_tokens, n_kv, max_tiles, head_dim)
                    assert lib.library().fwb_decode_attention_rule(n_tokens, n_kv, max_tiles, head_dim, ctypes.addressof(out)) == 0
                    assert tuple(out) == tuple(int(v) for v in chosen), (n_tokens, n_kv, max_tiles, head_dim)
    slices = lambda pairs, tiles, head_dim: attention.decode_splits(pairs, 1, tiles, head_dim)[0]
    assert slices(8, 5, 64) == 1 and slices(8, 6, 64) == 2 and slices(64, 8, 64) == 1 and slices(64, 10, 64) == 2
    assert slices(8, 7, 128) == 1 and slices(8, 8, 128) == 4 and slices(64, 8, 128) == 1 and slices(64, 12, 128) == 2
