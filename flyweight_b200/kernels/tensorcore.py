"""Tensor-core (tcgen05) matrix products of the bfloat16 path.

``accepts`` says whether the kernel takes a product; the dispatcher in ``ops.linear`` falls
back to the SIMT kernel otherwise, so every shape the configuration allows still runs.
"""
from __future__ import annotations

import torch

from . import lib
from .lib import KernelError, check_tensor, ptr, stream

EPI_F32, EPI_BF16, EPI_ADD_F32, EPI_SWIGLU_BF16 = 0, 1, 2, 3
# the activation on the gate rides in the bits above the epilogue code (0: silu)
GATE_ACT_SHIFT = 8


def _gated_epilogue(activation: str) -> int:
    from .ops import GATE_ACTIVATIONS
    return EPI_SWIGLU_BF16 | (GATE_ACTIVATIONS[activation] << GATE_ACT_SHIFT)


def _output_epilogue(activation) -> int:
    """A bfloat16 output with an activation of ``ops.OUTPUT_ACTIVATIONS`` applied in fp32 in front of the rounding."""
    from .ops import OUTPUT_ACTIVATIONS
    return EPI_BF16 | (OUTPUT_ACTIVATIONS[activation] << GATE_ACT_SHIFT)


SM_COUNT = 148
_enabled = True


def set_enabled(flag: bool) -> None:
    """Tests switch the tensor-core path off to compare it with the SIMT path."""
    global _enabled
    _enabled = bool(flag)
    lib.set_option("tensorcore", _enabled)


def _aligned(t: torch.Tensor) -> bool:
    return t.data_ptr() % 16 == 0


def accepts(x, w, out_dtype, addend=None) -> bool:
    if not _enabled:
        return False
    if x.dtype != torch.bfloat16 or w.dtype != torch.bfloat16:
        return False
    if out_dtype not in (torch.float32, torch.bfloat16):
        return False
    if addend is not None and out_dtype != torch.float32:
        return False
    K = x.shape[1]
    return K % 8 == 0 and K >= 8 and _aligned(x) and _aligned(w) and x.shape[0] <= 65535 * 16


_forced_splits = None
_use_pairs = True


def set_pairs_enabled(flag: bool) -> None:
    """Prompt-sized products on CTA pairs (on by default); off: the single-CTA kernel."""
    global _use_pairs
    _use_pairs = bool(flag)
    lib.set_option("pairs", _use_pairs)

# ---- decode steps of a few requests: csrc/linear_rows.cu -----------------------------------
# A few tokens' products run on a kernel that streams weights straight to mma.sync instead of through tiles of tensor
# memory: a decode step is a chain of small launches, and what counts is the time from the activations to the result.
# The lines (us on B200, tcgen05 kernel and this one; more sizes in csrc/linear_rows.cu), N being the matrix's rows:
#  * The walk over K goes 1,024 at a time, so a shorter K leaves warps idle and one a little longer than a step or two
#    pays for steps half empty: 8 tokens, 16384 x 512 8.2 and 6.9, 32768 x 512 8.4 and 11.0, 65536 x 1024 22.7 and 25.2,
#    8192 x 1536 8.9 and 7.4, 28672 x 1536 16.6 and 18.5.
#  * Every CTA reads all activations and keeps partial sums of its features: with 9 and more tokens wide matrices take
#    another round of CTAs (16 tokens, 18432 x 1024 +-0, 19456 x 1024 1.2 times, 65536 x 1024 23.6 and 35.3).
#    Up to 18,432 features over 2,048 channels they win but for the middle (12 tokens: 8192 9.6 and 8.8, 9728 x 2048 behind
#    a norm 11.5 and 11.7, 12288 12.9 and 13.5, 16384 16.4 and 14.6, where the tcgen05 kernel's CTAs make a round and a half).
#  * With a long K the tcgen05 kernel cuts K finely, and a share of features that leaves SMs idle decides: 8 tokens,
#    4864 x 5120 1.13 times its time (share 0.69), 6144 x 5120 1.02 (0.87), 4096 x 5120 0.8 (0.87).
#  * 17 to 32 tokens besides where the tcgen05 kernel's clusters would not all be resident (see ``two_rings``):
#    9216 x 1024 at 24 11.4 and 8.1, against 9728 x 1024 7.4 and 10.8.
ROWS_LONG_K, ROWS_LEAST_SHARE = 4096, 0.85
# The norm in front is folded in where K is one step of the kernel's walk: 1024 x 1024 at 8 tokens 3.3 us against 3.5 for
# the norm's kernel and the product, 9216 x 1024 5.2 against 6.2; with K = 2048 it loses (6144 x 2048: 7.6 against 6.9).
ROWS_NORMED_TO, ROWS_NORMED_K = 8, 1024
_use_rows = True


def set_rows_enabled(flag: bool) -> None:
    """Products of a few tokens on the weight reader (on by default); off: the tcgen05 kernel."""
    global _use_rows
    _use_rows = bool(flag)
    lib.set_option("rows", _use_rows)


def _rows_takes(M: int, N: int, K: int) -> bool:
    """``N``: rows of the matrix (gate and up together)."""
    if not (_enabled and _use_rows) or _forced_splits is not None or M > 32 or N * K > 1 << 26:
        return False
    if M <= 8:
        if K <= 1024:
            return N <= (24 if K < 512 else 32) * K
        if K < 2048:
            return N <= 7 * K
        return K <= ROWS_LONG_K or _rows_share(N) >= ROWS_LEAST_SHARE
    if M <= 16:
        if K <= 1024:
            return N <= (12 * K if K < 512 else min(24 * K, 18432))
        if K < 1920:
            return N <= 4096
        return K <= 2048 and (N <= 8192 or 13312 <= N <= 18432)
    if K > 1024 or N * K > 1 << 24:
        return False
    return N <= min((12 if K < 512 else 18) * K, (1 << 22) // K) or (N <= 9472 and not _all_resident(M, N, K))


def _rows_share(N: int) -> float:
    """How even the weight reader's CTAs (up to 8 tokens: two an SM, groups of eight features) lie on the SMs: the mean
    over the fullest."""
    units = -(-N // 8)
    if units <= 2 * SM_COUNT:
        return 1.0                  # one group a CTA
    per_cta = -(-units // (2 * SM_COUNT))
    ctas = -(-units // per_cta)
    return units / (SM_COUNT * per_cta * -(-ctas // SM_COUNT))


def _all_resident(M: int, N: int, K: int) -> bool:
    """Whether the clusters of the tcgen05 kernel's choice for a decode-sized product all run at once."""
    splits = _splits_for(M, N, K, 1)
    clusters = -(-N // 128) * -(-M // _decode_tile(M, N))
    an_sm = -(-clusters * splits // SM_COUNT)
    return clusters <= {1: SM_COUNT, 2: SM_COUNT // 2, 4: 35, 8: 16}[splits] * an_sm


def _rows_takes_normed(M: int, N: int, K: int) -> bool:
    return M <= ROWS_NORMED_TO and K <= ROWS_NORMED_K and _rows_takes(M, N, K)


def _rows_takes_conv(M: int, N: int, K: int) -> bool:
    """A convolution step saves the convolution's launch, 4 to 5 us, which outweighs what the product itself may lose."""
    if not (_enabled and _use_rows) or _forced_splits is not None:
        return False
    return N * K <= 1 << 26 and (M <= 8 or (M <= 16 and K <= 2048))


# Per-shape overrides found by measurement: (features, K, accumulators) -> (splits, stages);
# 0 keeps the rule's choice.  Only decode-sized token counts (<= 64) consult it.
TUNED = {}


def force_splits(splits) -> None:
    """Pin the split-K factor (None: chosen per shape).  With one fixed factor every output
    element is summed in the same order whatever the number of tokens in the step, which
    lets tests compare ways of cutting the work bit by bit."""
    global _forced_splits
    _forced_splits = splits
    lib.set_option("forced_splits", splits or 0)


def pick_splits(M: int, N: int, K: int) -> int:
    """CTAs that share one output tile's K range (a cluster, <= 8): as many as it takes to
    put work on every SM when the token tile is small (decode), 1 otherwise."""
    if _forced_splits is not None:
        return _forced_splits if M <= 64 else 1
    if M > 64:
        return 1
    return _splits_for(M, N, K, 1)


def _decode_tile(M: int, N: int) -> int:
    """Token tile of a decode-sized step.  33..64 tokens are cut into two tiles of 32 when the
    product has too few feature tiles to occupy the GPU (measured at batch 64: 6 % off the
    step); a product with many tiles keeps one token tile, so no weight is fetched twice."""
    if M <= 16:
        return 16
    if M <= 32 or -(-N // 128) < SM_COUNT:
        return 32
    return 64


_stage_cap = 8


def _ring_depth(M: int, N: int, splits: int, accumulators: int) -> int:
    """Stages of the shared-memory ring for decode-sized steps: at most four, and few enough
    that every CTA of the product is resident at once (measured: a product that needs a second
    wave of CTAs loses far more than a shallower ring does)."""
    bn = _decode_tile(M, N)
    stage = accumulators * 16384 + bn * 128
    ctas = -(-N // 128) * -(-M // bn) * splits
    per_sm = max(1, -(-ctas // SM_COUNT))
    fit = ((227 * 1024) // per_sm - 2048) // stage
    return max(2, min(3 if (accumulators == 2 and bn <= 16) else 4, fit, _stage_cap))


def _splits_for(M: int, N: int, K: int, accumulators: int) -> int:
    """Slices of K per output tile (a cluster, a power of two <= 8).  Measured inside the decode
    step of LFM2-1.2B on B200 at batch 1, 8 and 64: the step is fastest with about 400 CTAs per
    product (256 with two accumulators), as long as a slice keeps at least four 64-wide blocks."""
    bn = _decode_tile(M, N)
    tiles = -(-N // 128) * -(-M // bn)
    k_blocks = -(-K // 64)
    budget = 256 if accumulators == 2 else 400
    limit = 4 if accumulators == 2 else 8
    if accumulators == 2 and M > 32:
        return 1                    # two accumulators of two token tiles: the reduction costs more
    splits = 1
    while splits < limit and tiles * splits * 2 <= budget and k_blocks >= splits * 8:
        splits *= 2
    return splits


def two_rings(M: int, N: int, K: int, accumulators: int):
    """33 to 512 tokens, matrices that are still read like a decode step's: (token tile, slices of K, stages) with two
    CTAs, so two rings of weights, on an SM -- one leaves HBM waiting for its latency -- or None for the general rules.
    Measured on B200 (us, the general rule's choice and this one): gated 8192 x 2048 at 64 tokens 23.9 and 20.1, at 77
    23.9 and 22.1; gated 4608 x 1024 at 64 14.8 and 11.3; 2048 x 8192 at 77 17.7 and 13.8, at 160 19.5 and 15.9;
    1024 x 4608 at 256 13.2 and 10.9; 6144 x 2048 at 77 13.6 and 11.9, at 128 14.2 and 12.7.

    The lines: all clusters have to be resident at once (a cluster's CTAs lie in one GPC).  Of clusters of four 70 are with
    two CTAs an SM, 104 with three (8960 x 2048 at 77 tokens 15.2 and 13.8, 9216 x 2048 15.2 and 21.9; 6656 x 2048 at 128
    14.5 and 12.9, 6912 x 2048 14.7 and 18.7; gated 8960 x 2048 at 64 24.9 and 21.2, 9216 x 2048 24.9 and 32.3), of
    clusters of eight 33 (2048 x 4096 at 77 11.7 and 10.3, 2176 x 4096 12.2 and 15.4).  34 to 37 of eight are taken where
    the general choice needs two rounds as well (4352 x 4096 at 77 24.3 and 20.3; 2176 x 4096 at 160 22.6 and 17.7).  Below
    5,120 features with a short K the general choice is level or better (3840 x 1024 at 77 7.9 and 8.3).  csrc/plan.cu has
    the same rule."""
    if _forced_splits is not None or M <= 32 or M > MID_TO:
        return None
    tiles, k_blocks = -(-N // 128), -(-K // 64)
    if accumulators == 2:
        tile = (64 if k_blocks >= 32 else 32) if M <= 64 else 96
        if (M > 64 and k_blocks < 32) or M > 96 or k_blocks < 16 or tiles * -(-M // tile) > (74 if tile == 32 else 70):
            return None
        return tile, 4, 2
    if M <= 64 or not _mid_size_split:
        return None
    if k_blocks >= 64:
        for tile, stages in ((64, 4), (96, 3)):
            if tiles * -(-M // tile) <= (37 if tile == 96 and (M <= 96 or 128 < M <= 192) else 33):
                return tile, 8, stages
    if M <= 128 and k_blocks >= 16 and 40 <= tiles <= (70 if M <= 96 else 52):
        return (96 if M <= 96 else 64), 4, 3
    return None


# ---- 65 to 512 tokens: which tile, how many slices of K, or CTA pairs ----------------------
# Between decode-sized steps (a weight streamer on every SM) and prompt-sized ones (256-token
# tiles that fill the GPU) a product has few output tiles, and a CTA's walk over K is bound by
# latency, not by bandwidth: about 0.38 us per 64-wide block whatever the tile (0.6 us with two
# accumulators, 0.84 us for two accumulators of 256 tokens), 3 us of fixed cost, and a cluster
# reduction that costs 2.6 to 3.9 us depending on the tile and the number of slices.  The choice
# below evaluates that cost model (hundredths of a microsecond, fitted to products of LFM2-1.2B
# and LFM2-350M at 65 to 1,024 tokens on B200) for every tile and split the kernels have and takes
# the cheapest; a split is only considered when all its CTAs run at once (clusters in a second
# wave were measured far slower than the model).  The native dispatch (csrc/plan.cu) has the same
# table and the same loop.
MID_FROM, MID_TO = 65, 512
_MID_FIXED = 310
_MID_BLOCK = {1: {64: 38, 128: 38, 256: 42}, 2: {64: 63, 128: 58, 256: 84}}
_MID_PAIR_BLOCK = 36
_MID_REDUCE = {(128, 2): 360, (128, 4): 260, (64, 2): 390, (64, 4): 310}
_mid_size_split = True


def set_mid_size_split(flag: bool) -> None:
    """The cost-model choice for products of 65 to 512 tokens (on by default); off: CTA pairs
    above 128 tokens and one CTA per 128-token tile below, without a split."""
    global _mid_size_split
    _mid_size_split = bool(flag)
    lib.set_option("mid_size_split", _mid_size_split)


def mid_size_choice(M: int, N: int, K: int, accumulators: int, pair_ok: bool):
    """For ``MID_FROM <= M <= MID_TO``: ("pair", 0, 1) or ("single", token tile, slices of K)."""
    k_blocks = -(-K // 64)
    feature_tiles = -(-N // 128)
    best = None
    for tile in (64, 128, 256):
        if tile == 256 and M <= 128:
            continue
        for splits in (1, 2, 4):
            if splits > 1 and (tile > 128 or accumulators == 2 or _forced_splits is not None
                               or k_blocks < 4 * splits):
                continue
            ctas = feature_tiles * -(-M // tile) * splits
            waves = -(-ctas // SM_COUNT)
            if splits > 1 and waves > 1:
                continue
            cost = _MID_FIXED + _MID_BLOCK[accumulators][tile] * -(-k_blocks // splits) * waves
            if splits > 1:
                cost += _MID_REDUCE[(tile, splits)]
            if best is None or cost < best[0]:
                best = (cost, "single", tile, splits)
    if pair_ok:
        pairs = -(-N // 256) * -(-M // 256)
        cost = _MID_FIXED + _MID_PAIR_BLOCK * k_blocks * -(-pairs // (SM_COUNT // 2))
        if cost < best[0]:
            best = (cost, "pair", 0, 1)
    return best[1:]


def _pairs_add(M: int, N: int) -> bool:
    """Prompt-sized steps: the CTA pairs add the product into their fp32 output (2,048 x 2,048 values: 17 MB less
    written and 17 MB less read by the norm behind it)."""
    return _use_pairs and M > (MID_TO if _mid_size_split else 128) and N >= 256


def adds_in_place(x, w, residual) -> bool:
    """Whether ``gemm(x, w, fp32, addend=residual, out=residual)`` is available: up to 128 tokens on the single-CTA
    kernel and the weight reader, beyond the mid sizes on the CTA pairs (every element is read and written by the
    same thread)."""
    M = x.shape[0]
    small = M <= 128 and (M >= FUSE_FROM_TOKENS or _fuse_always or _rows_takes(M, *w.shape))
    return (_add_in_place and (small or _pairs_add(M, w.shape[0])) and accepts(x, w, torch.float32, residual)
            and residual.dtype == torch.float32 and residual.is_contiguous()
            and tuple(residual.shape) == (M, w.shape[0]))


def gemm(x, w, out_dtype, addend=None, splits=None, stages=0, tile_tokens=0, wide=-1, out=None,
         activation=None) -> torch.Tensor:
    """``x @ w.T``: x [M][K] bf16, w [N][K] bf16 -> [M][N] fp32 or bf16 (+ fp32 addend).
    ``out`` may be the addend itself (the sum in place).  ``activation`` (bf16 outputs): one of
    ``ops.OUTPUT_ACTIVATIONS``, applied on the way out."""
    check_tensor("gemm input", x, torch.bfloat16)
    check_tensor("gemm weight", w, torch.bfloat16)
    M, K = x.shape
    N = w.shape[0]
    if w.shape[1] != K:
        raise KernelError(f"gemm: input has {K} columns, weight has {w.shape[1]}")
    free_choice = splits is None and not stages and not tile_tokens and wide == -1
    if activation is not None and (out_dtype != torch.bfloat16 or addend is not None):
        raise KernelError("an activation on the way out goes with a bfloat16 output")
    pair_ok = _use_pairs and M > 128 and addend is None and out is None and N >= 256
    if free_choice and addend is not None and addend is out and out_dtype == torch.float32 and _pairs_add(M, N):
        check_tensor("gemm addend", addend, torch.float32, (M, N))
        lib.call("fwb_gemm_tcgen05_pair", ptr(x), ptr(w), ptr(out), M, N, K, N, N, EPI_ADD_F32, 0, lib.c_float(0.0),
                 stream(), tag=f"{N}x{K} added")
        return out
    rings = two_rings(M, N, K, 1) if free_choice else None
    if rings:
        tile_tokens, splits, stages = rings
    elif free_choice and _mid_size_split and MID_FROM <= M <= MID_TO:
        kind, tile_tokens, splits = mid_size_choice(M, N, K, 1, pair_ok)
        if kind == "pair":
            return gemm_pair(x, w, out_dtype, activation=activation)
    elif pair_ok and free_choice:
        return gemm_pair(x, w, out_dtype, activation=activation)       # prompt-sized: CTA pairs (cta_group::2)
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype, device=x.device)
    else:
        check_tensor("gemm output", out, out_dtype, (M, N))
    if addend is not None:
        check_tensor("gemm addend", addend, torch.float32, (M, N))
        epilogue = EPI_ADD_F32
    else:
        epilogue = EPI_F32 if out_dtype == torch.float32 else _output_epilogue(activation)
    if free_choice and _rows_takes(M, N, K):
        lib.call("fwb_linear_rows", ptr(x), ptr(w), ptr(out), ptr(addend), M, N, K, N, N, epilogue, 0,
                 lib.c_float(0.0), stream(), tag=f"{N}x{K} rows")
        return out
    if M <= 64 and (N, K, 1) in TUNED and _forced_splits is None:
        tuned = TUNED[(N, K, 1)]
        splits = splits or tuned[0] or None
        stages = stages or tuned[1]
        if len(tuned) > 2:
            tile_tokens = tile_tokens or tuned[2]
    if splits is None:
        splits = pick_splits(M, N, K)
    if M <= 64:
        stages = stages or _ring_depth(M, N, splits, 1)
        tile_tokens = tile_tokens or _decode_tile(M, N)
    lib.call("fwb_gemm_tcgen05", ptr(x), ptr(w), ptr(out), ptr(addend), M, N, K, N, N, epilogue, 0,
             splits, stages, tile_tokens, wide, lib.c_float(0.0), stream(), tag=f"{N}x{K} splits {splits}")
    return out


def conv_step_accepts(h, w_in, batch, act_dtype) -> bool:
    """A step of one token per request whose in_proj the weight reader takes does the short convolution in that
    product's epilogue (measured in the decode step: a launch of 4 to 5 us less per convolution layer)."""
    H = w_in.shape[0] // 3
    if isinstance(h, torch.Tensor) and (h.dtype != torch.bfloat16 or not _aligned(h)):
        return False                                            # (the projection on its own takes those)
    return (act_dtype == torch.bfloat16 and w_in.dtype == torch.bfloat16 and batch.max_segment == 1
            and batch.n_tokens == batch.n_segments <= 16 and w_in.shape[1] % 8 == 0 and _aligned(w_in)
            and _rows_takes_conv(batch.n_tokens, 3 * H, w_in.shape[1]))


def conv_step(h, w_in, taps, bias, state, batch) -> torch.Tensor:
    """``shortconv(linear(h, w_in))`` of a step of one token per request, in one kernel: ``h`` bf16 rows, or a norm not
    yet applied to rows of the residual."""
    K, H, L = w_in.shape[1], w_in.shape[0] // 3, taps.shape[1]
    M = batch.n_tokens
    norm_w, eps = None, 0.0
    if isinstance(h, torch.Tensor):
        x = h
    elif h.kind == "rmsnorm" and h.rows is None and _fuse_norm and M <= ROWS_NORMED_TO and K <= ROWS_NORMED_K and _norm_aligned(h):
        x, norm_w, eps = h.x, h.weight, h.eps
        check_tensor("norm weight", norm_w, torch.float32, (K,))
    else:
        x = h.materialize(torch.bfloat16)
    check_tensor("conv step input", x, torch.bfloat16 if norm_w is None else torch.float32)
    check_tensor("conv step weight", w_in, torch.bfloat16)
    check_tensor("conv taps", taps, torch.float32, (H, L))
    if bias is not None:
        check_tensor("conv bias", bias, torch.float32, (H,))
    if x.numel() != M * K:
        raise KernelError(f"conv step: {x.numel()} inputs for {M} tokens of {K}")
    if (not state.is_cuda or state.dtype != torch.float32 or tuple(state.shape[1:]) != (H, L - 1)
            or state.stride(2) != 1 or state.stride(1) != L - 1 or (state.shape[0] > 1 and state.stride(0) < H * (L - 1))):
        raise KernelError(f"conv state must be CUDA fp32 [slots][{H}][{L - 1}] with contiguous slots")
    stride = state.stride(0) if state.shape[0] > 1 else H * (L - 1)
    check_tensor("seg_slot", batch.seg_slot, torch.int32, (M,))
    out = torch.empty((M, H), dtype=torch.bfloat16, device=x.device)
    lib.call("fwb_linear_rows_conv", ptr(x), ptr(norm_w), lib.c_float(eps), ptr(w_in), ptr(taps), ptr(bias), ptr(state),
             lib.c_longlong(stride), ptr(batch.seg_slot), ptr(out), M, H, K, L, stream(), tag=f"{H}x{K} conv step")
    return out


def swiglu_accepts(x, w_gate_up) -> bool:
    return accepts(x, w_gate_up, torch.bfloat16)


def swiglu_gate_up(x, w_gate_up, splits=None, stages=0, tile_tokens=0, activation="silu", limit=0.0) -> torch.Tensor:
    """``silu(x @ gate.T) * (x @ up.T)`` as bf16, for ``w_gate_up`` = [gate rows | up rows]:
    both products accumulate side by side in tensor memory and never reach global memory.
    ``activation`` names another gated form (``ops.GATE_ACTIVATIONS``), ``limit`` its parameter."""
    check_tensor("swiglu input", x, torch.bfloat16)
    check_tensor("swiglu weight", w_gate_up, torch.bfloat16)
    M, K = x.shape
    F2 = w_gate_up.shape[0]
    F = F2 // 2
    if w_gate_up.shape[1] != K or F * 2 != F2:
        raise KernelError("swiglu: weight must be [2F][K]")
    gated = _gated_epilogue(activation)
    out = torch.empty((M, F), dtype=torch.bfloat16, device=x.device)
    if splits is None and not stages and not tile_tokens and _rows_takes(M, F2, K):
        lib.call("fwb_linear_rows", ptr(x), ptr(w_gate_up), ptr(out), ptr(None), M, F, K, F2, F, gated, F,
                 lib.c_float(limit), stream(), tag=f"swiglu {F}x{K} rows")
        return out
    if M <= 64 and (F, K, 2) in TUNED and _forced_splits is None:
        tuned = TUNED[(F, K, 2)]
        splits = splits or tuned[0] or None
        stages = stages or tuned[1]
        if len(tuned) > 2:
            tile_tokens = tile_tokens or tuned[2]
    free_choice = splits is None and not stages and not tile_tokens
    rings = two_rings(M, F, K, 2) if free_choice else None
    if rings:
        tile_tokens, splits, stages = rings
        free_choice = False
    if splits is None:
        splits = (_forced_splits if _forced_splits is not None else _splits_for(M, F, K, 2)) if M <= 64 else 1
    if M <= 64:
        stages = stages or _ring_depth(M, F, splits, 2)
        tile_tokens = tile_tokens or _decode_tile(M, F)
    pairs = free_choice and _use_pairs and M > 128 and splits == 1
    if free_choice and not pairs and _mid_size_split and MID_FROM <= M <= MID_TO:
        _, tile_tokens, splits = mid_size_choice(M, F, K, 2, False)
    if pairs:
        lib.call("fwb_gemm_tcgen05_pair", ptr(x), ptr(w_gate_up), ptr(out), M, F, K, F2, F, gated, F,
                 lib.c_float(limit), stream(), tag=f"swiglu {F}x{K}")
        return out
    lib.call("fwb_gemm_tcgen05", ptr(x), ptr(w_gate_up), ptr(out), ptr(None), M, F, K, F2, F,
             gated, F, splits, stages, tile_tokens, -1, lib.c_float(limit), stream(),
             tag=f"swiglu {F}x{K} splits {splits}")
    return out


_fuse_norm = True
_add_in_place = True
_fuse_always = False
# Residual sums go into the products' epilogues from 16 tokens on (2-3 % of the decode step of LFM2-1.2B); below that
# only where the weight reader runs the product.  Norms are not folded into the tcgen05 products any more unless
# ``fuse_always`` asks for it: with the activations of a whole row to build, the product waits longer than the norm's
# own kernel takes (us, folded and apart: 6144 x 2048 at 64 tokens 20.3 and 11.3, at 16 13.2 and 8.6; 2048 x 2048 at 64
# 8.8 and 7.7; gated 8192 x 2048 at 24 17.1 and 16.8).
FUSE_FROM_TOKENS = 16


def fuse_always(flag: bool) -> None:
    """Fold norms and residual sums at every decode-sized token count (tests of that path)."""
    global _fuse_always
    _fuse_always = bool(flag)
    lib.set_option("fuse_always", _fuse_always)



def set_norm_fusion(flag: bool) -> None:
    """Norms folded into the product that follows them (on by default).  Off: the norm kernel
    writes bf16 rows first, as prompt-sized steps always do; tests that compare cuts bit by bit
    switch it off so that every cut runs the same arithmetic."""
    global _fuse_norm, _add_in_place
    _fuse_norm = _add_in_place = bool(flag)
    lib.set_option("fuse_norm", _fuse_norm)
    lib.set_option("add_in_place", _add_in_place)


def _norm_aligned(norm) -> bool:
    return _aligned(norm.x) and _aligned(norm.weight)


def normed_accepts(M: int, K: int, w, accumulators: int, N: int, norm=None) -> bool:
    """Decode-sized token counts whose K slice per CTA is short enough that building the
    activation tiles inside the kernel stays off the critical path."""
    if not (_enabled and _fuse_norm) or w.dtype != torch.bfloat16 or M > 64 or K % 8 or not _aligned(w):
        return False
    if norm is not None and not _norm_aligned(norm):
        return False                                            # (rows or a weight off a 16-byte border: the norm's kernel)
    if _rows_takes(M, accumulators * N, K):
        return _rows_takes_normed(M, accumulators * N, K)
    if not _fuse_always:
        return False
    splits = _forced_splits if _forced_splits is not None else _splits_for(M, N, K, accumulators)
    return -(-K // 64) <= 8 * splits


def gemm_normed(x_res, norm_weight, eps, w, out_dtype, rows=None, n_rows=None, splits=None, stages=0,
                tile_tokens=0) -> torch.Tensor:
    """``rmsnorm(x_res[rows]) @ w.T`` in one kernel: fp32 residual rows in, [M][N] fp32 or bf16 out."""
    check_tensor("residual", x_res, torch.float32)
    check_tensor("norm weight", norm_weight, torch.float32)
    check_tensor("gemm weight", w, torch.bfloat16)
    K = x_res.shape[-1]
    M = x_res.numel() // K if rows is None else (rows.numel() if n_rows is None else n_rows)
    N = w.shape[0]
    if w.shape[1] != K or norm_weight.numel() != K:
        raise KernelError(f"gemm: residual has {K} columns, weight has {w.shape[1]}, norm {norm_weight.numel()}")
    out = torch.empty((M, N), dtype=out_dtype, device=x_res.device)
    if splits is None and not stages and not tile_tokens and _rows_takes_normed(M, N, K):
        lib.call("fwb_linear_rows_normed", ptr(x_res), ptr(norm_weight), ptr(rows), lib.c_float(eps), ptr(w), ptr(out),
                 M, N, K, N, N, EPI_F32 if out_dtype == torch.float32 else EPI_BF16, 0, lib.c_float(0.0), stream(),
                 tag=f"normed {N}x{K} rows")
        return out
    if splits is None:
        splits = pick_splits(M, N, K)
    stages = stages or _ring_depth(M, N, splits, 1)
    tile_tokens = tile_tokens or _decode_tile(M, N)
    lib.call("fwb_gemm_tcgen05_normed", ptr(x_res), ptr(norm_weight), ptr(rows), lib.c_float(eps), ptr(w),
             ptr(out), M, N, K, N, N, EPI_F32 if out_dtype == torch.float32 else EPI_BF16, 0, splits,
             stages, tile_tokens, lib.c_float(0.0), stream(), tag=f"normed {N}x{K} splits {splits}")
    return out


def swiglu_gate_up_normed(x_res, norm_weight, eps, w_gate_up, splits=None, stages=0, tile_tokens=0,
                          activation="silu", limit=0.0) -> torch.Tensor:
    """``silu(n @ gate.T) * (n @ up.T)`` with n = rmsnorm(x_res), in one kernel."""
    check_tensor("residual", x_res, torch.float32)
    check_tensor("norm weight", norm_weight, torch.float32)
    check_tensor("swiglu weight", w_gate_up, torch.bfloat16)
    K = x_res.shape[-1]
    M = x_res.numel() // K
    F2 = w_gate_up.shape[0]
    F = F2 // 2
    if w_gate_up.shape[1] != K or F * 2 != F2 or norm_weight.numel() != K:
        raise KernelError("swiglu: weight must be [2F][K] and the norm weight [K]")
    gated = _gated_epilogue(activation)
    out = torch.empty((M, F), dtype=torch.bfloat16, device=x_res.device)
    if splits is None and not stages and not tile_tokens and _rows_takes_normed(M, F2, K):
        lib.call("fwb_linear_rows_normed", ptr(x_res), ptr(norm_weight), ptr(None), lib.c_float(eps), ptr(w_gate_up),
                 ptr(out), M, F, K, F2, F, gated, F, lib.c_float(limit), stream(), tag=f"normed swiglu {F}x{K} rows")
        return out
    if splits is None:
        splits = _forced_splits if _forced_splits is not None else _splits_for(M, F, K, 2)
    stages = stages or _ring_depth(M, F, splits, 2)
    tile_tokens = tile_tokens or _decode_tile(M, F)
    lib.call("fwb_gemm_tcgen05_normed", ptr(x_res), ptr(norm_weight), ptr(None), lib.c_float(eps),
             ptr(w_gate_up), ptr(out), M, F, K, F2, F, gated, F, splits, stages, tile_tokens,
             lib.c_float(limit), stream(), tag=f"normed swiglu {F}x{K} splits {splits}")
    return out


def status() -> int:
    """0, or the code a wait that gave up inside the kernel left (reads and clears it;
    synchronises the device)."""
    return int(lib.library().fwb_gemm_tcgen05_status())


def gemm_pair(x, w, out_dtype, activation=None) -> torch.Tensor:
    """``x @ w.T`` on CTA pairs (tcgen05 cta_group::2), tiles of 256 features x 256 tokens, as many pairs as the GPU
    holds.  For prompt-sized steps; bf16 in, fp32 or bf16 out."""
    check_tensor("gemm input", x, torch.bfloat16)
    check_tensor("gemm weight", w, torch.bfloat16)
    M, K = x.shape
    N = w.shape[0]
    if w.shape[1] != K:
        raise KernelError(f"gemm: input has {K} columns, weight has {w.shape[1]}")
    out = torch.empty((M, N), dtype=out_dtype, device=x.device)
    epilogue = EPI_F32 if out_dtype == torch.float32 else _output_epilogue(activation)
    lib.call("fwb_gemm_tcgen05_pair", ptr(x), ptr(w), ptr(out), M, N, K, N, N, epilogue, 0, lib.c_float(0.0),
             stream(), tag=f"{N}x{K}")
    return out


def swiglu_gate_up_pair(x, w_gate_up) -> torch.Tensor:
    """The fused gate/up product with the SwiGLU epilogue on CTA pairs."""
    check_tensor("swiglu input", x, torch.bfloat16)
    check_tensor("swiglu weight", w_gate_up, torch.bfloat16)
    M, K = x.shape
    F = w_gate_up.shape[0] // 2
    out = torch.empty((M, F), dtype=torch.bfloat16, device=x.device)
    lib.call("fwb_gemm_tcgen05_pair", ptr(x), ptr(w_gate_up), ptr(out), M, F, K, 2 * F, F,
             EPI_SWIGLU_BF16, F, lib.c_float(0.0), stream())
    return out
