"""The mechanisms Diforax brought to the engine, each alone: the kernel (or the part) against the
function of ``plain_diforax`` that states the same mechanism, on hand-made batches whose segments start
at position 0, in the middle of a sequence and on single tokens, over shuffled pages and slots."""
import math

import pytest
import torch

import plain_diforax as P

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
F64 = torch.float64
BOTH = [torch.float32, torch.bfloat16]


def dev(t, dtype=None):
    return t.to(device=DEV, dtype=dtype or t.dtype).contiguous()


def close(got, want, rel, what=""):
    got, want = got.detach().cpu().to(F64), want.detach().cpu().to(F64)
    assert got.shape == want.shape, f"{what}: {tuple(got.shape)} vs {tuple(want.shape)}"
    assert torch.isfinite(got).all(), f"{what}: non-finite"
    scale = max(1.0, float(want.abs().max()))
    worst = float((got - want).abs().max())
    assert worst <= rel * scale, f"{what}: max|delta| {worst:.3e} > {rel:.1e} * {scale:.3g}"


def bf16_round(t):
    return t.to(torch.bfloat16).to(F64)


def matrix(g, rows, cols, dtype):
    m = torch.randn(rows, cols, generator=g, dtype=F64) / math.sqrt(cols)
    return bf16_round(m) if dtype == torch.bfloat16 else m.to(torch.float32).to(F64)


def precision_of(dtype):
    from flyweight_b200.parts import Precision
    return Precision("float32" if dtype == torch.float32 else "bfloat16")


class Feeder:
    """Feeds sequences to a part in steps of (sequence, new tokens) pairs: hands out pages in a shuffled
    order, keeps block tables and positions, and gives every sequence a state slot of its own."""

    def __init__(self, n_seqs, n_pages=24, seed=0, slots=None):
        self.order = torch.randperm(n_pages, generator=torch.Generator().manual_seed(seed)).tolist()
        self.pages = {s: [] for s in range(n_seqs)}
        self.done = {s: 0 for s in range(n_seqs)}
        self.slots = slots or {s: n_seqs - 1 - s for s in range(n_seqs)}

    def batch(self, step):
        from flyweight_b200.engine import Segment, StepBatch
        segments = []
        for s, m in step:
            while len(self.pages[s]) * 64 < self.done[s] + m:
                self.pages[s].append(self.order.pop())
            segments.append(Segment(f"s{s}", self.slots[s], self.done[s], [0] * m, []))
        width = max(1, max(len(self.pages[s]) for s, _ in step))
        table = [self.pages[s] + [-1] * (width - len(self.pages[s])) for s, _ in step]
        return StepBatch(segments, [table], DEV)

    def advance(self, step):
        for s, m in step:
            self.done[s] += m


def run_part(part, precision, h_seqs, steps, cache, feeder=None, feed_forward=False):
    """Outputs by sequence of a mixer (or feed-forward) over ``steps``."""
    from flyweight_b200.engine import StepContext
    feeder = feeder or Feeder(len(h_seqs))
    outs = {s: [] for s in range(len(h_seqs))}
    for step in steps:
        batch = feeder.batch(step)
        h = torch.cat([h_seqs[s][feeder.done[s]:feeder.done[s] + m] for s, m in step]).to(precision.act_dtype)
        ctx = StepContext(batch, precision, DEV)
        out = part.forward(ctx, dev(h)) if feed_forward else part.forward(ctx, dev(h), cache)
        at = 0
        for s, m in step:
            outs[s].append(out[at:at + m].float().cpu())
            at += m
        feeder.advance(step)
    return {s: torch.cat(parts) for s, parts in outs.items() if parts}


def cuts_of(lengths, sizes):
    """Steps that feed sequences of the given lengths side by side in portions of ``sizes`` (cycled)."""
    done = [0] * len(lengths)
    steps, i = [], 0
    while any(d < n for d, n in zip(done, lengths)):
        step = []
        for s, n in enumerate(lengths):
            if done[s] < n:
                m = min(sizes[(i + s) % len(sizes)], n - done[s])
                step.append((s, m))
                done[s] += m
        steps.append(step)
        i += 1
    return steps


# ------------------------------------------------------------------ x += w * unit(y), and the next norm
@pytest.mark.parametrize("W", [80, 82, 3000])
@pytest.mark.parametrize("next_dtype", [None, torch.float32, torch.bfloat16])
def test_output_norm_adds_into_the_stream(W, next_dtype):
    from flyweight_b200.kernels import ops
    g = torch.Generator().manual_seed(W)
    x = torch.randn(7, W, generator=g, dtype=torch.float32)
    y = torch.randn(7, W, generator=g, dtype=torch.float32) * 3
    w = 1 + 0.1 * torch.randn(W, generator=g, dtype=torch.float32)
    w2 = 1 + 0.1 * torch.randn(W, generator=g, dtype=torch.float32)
    want_x = x.to(F64) + P.rms_norm(y.to(F64), w.to(F64), 1e-5)
    xd = dev(x)
    h = ops.rmsnorm_add_(xd, dev(y), dev(w), 1e-5, *(() if next_dtype is None else (dev(w2), 1e-6, next_dtype)))
    close(xd, want_x, 1e-6, "the stream")
    if next_dtype is None:
        assert h is None
    else:
        assert h.dtype == next_dtype
        close(h, P.rms_norm(want_x, w2.to(F64), 1e-6), 1e-6 if next_dtype == torch.float32 else 2.0 ** -8, "the next norm")


# ------------------------------------------------------------------ the gate's activation
@pytest.mark.parametrize("T", [1, 9, 70, 300])
def test_gelu_on_the_gate(T):
    from flyweight_b200.kernels import ops, tensorcore
    g = torch.Generator().manual_seed(T)
    F, K = 192, 128
    x = bf16_round(torch.randn(T, K, generator=g, dtype=F64))
    w = bf16_round(torch.randn(2 * F, K, generator=g, dtype=F64) / math.sqrt(K) * 3)
    gu = x @ w.T
    want = P.gelu_tanh(gu[:, :F]) * gu[:, F:]
    close(ops.gate_act_mul(dev(gu, torch.float32), torch.float32, "gelu_tanh"), want, 1e-6, "unfused")
    close(ops.gate_act_mul(dev(gu, torch.float32), torch.float32, "silu"), P.silu(gu[:, :F]) * gu[:, F:], 1e-6, "silu")
    fused = tensorcore.swiglu_gate_up(dev(x, torch.bfloat16), dev(w, torch.bfloat16), activation="gelu_tanh")
    close(fused, want, 2.0 ** -7, "in the product's epilogue")
    assert tensorcore.status() == 0


# ------------------------------------------------------------------ rotation, then unit root mean square
@pytest.mark.parametrize("dtype", BOTH)
@pytest.mark.parametrize("heads,kv,dim,D,rot", [(6, 3, 32, 32, 16), (4, 1, 16, 48, 16), (2, 2, 64, 64, 32),
                                                (8, 2, 128, 128, 64), (3, 1, 24, 32, 0), (5, 5, 20, 32, 6)])
def test_rotation_then_unit_rms(dtype, heads, kv, dim, D, rot):
    """Heads of ``dim`` channels sit in rows of ``D`` (zero padding behind them): the mean of squares goes
    over ``dim``; queries, the key rows in their pages and the untouched value rows are checked."""
    from flyweight_b200.kernels import ops
    from flyweight_b200.parts.rope import Rope
    from flyweight_b200.config.spec import PartSpec
    g = torch.Generator().manual_seed(dim + rot)
    eps, T, pos0 = 1e-5, 9, 59
    raw = torch.randn(T, heads + 2 * kv, dim, generator=g, dtype=F64) * 2
    raw = bf16_round(raw) if dtype == torch.bfloat16 else raw.to(torch.float32).to(F64)
    positions = torch.arange(pos0, pos0 + T)
    want_q = P.rms_unit(P.rotate(raw[:, :heads], positions, 777.0, rot), eps)
    want_k = P.rms_unit(P.rotate(raw[:, heads:heads + kv], positions, 777.0, rot), eps)
    padded = torch.zeros(T, heads + 2 * kv, D, dtype=F64)
    padded[..., :dim] = raw
    table = Rope(PartSpec("rope", {"theta": 777.0, "rotary_dim": max(rot, 2)})).table(128, DEV) if rot else \
        torch.zeros((1, 1, 2), dtype=torch.float32, device=DEV)
    feeder = Feeder(1, n_pages=4, seed=dim)
    feeder.done[0] = pos0
    batch = feeder.batch([(0, T)])
    k_pool = torch.full((4, kv, 64, D), float("nan"), dtype=dtype, device=DEV)
    v_pool = torch.full_like(k_pool, float("nan"))
    q = ops.qk_norm_rope(dev(padded.view(T, -1), dtype), None, None, table, batch.positions, batch.tok_seg,
                         batch.block_tables[0], k_pool, v_pool, heads, kv, D, rot, eps, dtype,
                         unit_rms_after=True, norm_dim=dim)
    rel = 2e-6 if dtype == torch.float32 else 2.0 ** -8
    close(q.view(T, heads, D)[..., :dim], want_q, rel, "queries")
    assert float(q.view(T, heads, D)[..., dim:].float().abs().max() if D > dim else 0.0) == 0.0
    for i in range(T):
        page, row = feeder.pages[0][(pos0 + i) // 64], (pos0 + i) % 64
        close(k_pool[page, :, row, :dim], want_k[i], rel, f"key row of position {pos0 + i}")
        close(v_pool[page, :, row, :dim], raw[i, heads + kv:], 0.0 if dtype == torch.float32 else rel, "value row")


# ------------------------------------------------------------------ attention inside chunks: the part
def attention_spec(heads, kv, dim, vdim, chunk, rot, scale, hidden, shares=False):
    from flyweight_b200.config.spec import PartSpec
    tensors = {"q": "q", "o": "o"}
    if not shares:
        tensors.update({"k": "k", "v": "v"})
    position = PartSpec("rope", {"theta": 5000.0, "rotary_dim": rot}) if rot else PartSpec("no_position")
    return PartSpec("gqa_attention", {"hidden_size": hidden, "num_heads": heads, "num_kv_heads": kv, "head_dim": dim,
                                      "value_dim": vdim, "scale": scale, "qk_norm_eps": None, "qk_unit_rms_eps": 1e-5,
                                      "chunk": chunk, "shares_cache": shares, "position": position}, tensors)


def build_attention(spec, w, dtype, n_pages=24):
    from flyweight_b200.parts import build_mixer
    precision = precision_of(dtype)
    part = build_mixer(spec)
    part.bind(lambda n: w[n].to(dtype), precision, DEV)
    part.prepare(2048, DEV)
    cache = type("Cache", (), {})()
    kv = part.state_spec()
    cache.group, cache.state = 0, None
    if kv is not None:
        cache.k_pool = torch.full((n_pages, kv.n_kv_heads, 64, kv.head_dim), float("nan"), dtype=precision.cache_dtype, device=DEV)
        cache.v_pool = torch.full_like(cache.k_pool, float("nan"))
    return part, precision, cache


def plain_attention(h, w, heads, kv, dim, vdim, chunk, rot, scale, keys=None):
    positions = torch.arange(h.shape[0])
    if keys is None:
        keys = P.attention_keys(h, positions, w["k"], w["v"], kv, dim, vdim, 5000.0, rot, 1e-5)
    q = P.attention_queries(h, positions, w["q"], heads, dim, 5000.0, rot, 1e-5)
    return P.chunked_attention(q, positions, keys[0], keys[1], positions, scale, chunk) @ w["o"].T, keys


ATTENTION_SHAPES = [  # heads, kv, dim, vdim, chunk, rot, hidden
    (6, 3, 32, 16, 48, 16, 80), (4, 1, 16, 48, 64, 16, 96), (2, 2, 64, 64, 100, 32, 96),
    (8, 2, 128, 128, 130, 64, 128), (16, 4, 64, 64, 70, 64, 128), (3, 1, 24, 8, 5, 0, 72), (2, 1, 32, 32, 1, 32, 64),
]


@pytest.mark.parametrize("shape", ATTENTION_SHAPES)
@pytest.mark.parametrize("dtype", BOTH)
def test_chunked_attention_whole_cut_and_one_by_one(shape, dtype):
    heads, kv, dim, vdim, chunk, rot, hidden = shape
    g = torch.Generator().manual_seed(sum(shape))
    w = {"q": matrix(g, heads * dim, hidden, dtype), "k": matrix(g, kv * dim, hidden, dtype),
         "v": matrix(g, kv * vdim, hidden, dtype), "o": matrix(g, hidden, heads * vdim, dtype)}
    lengths = [300, 131, 1, 67]
    h_seqs = [torch.randn(n, hidden, generator=g, dtype=F64) for n in lengths]
    if dtype == torch.bfloat16:
        h_seqs = [bf16_round(h) for h in h_seqs]
    want = [plain_attention(h, w, heads, kv, dim, vdim, chunk, rot, 0.3)[0] for h in h_seqs]
    rel = 2e-5 if dtype == torch.float32 else 3 * 2.0 ** -7
    spec = attention_spec(heads, kv, dim, vdim, chunk, rot, 0.3, hidden)
    for name, sizes in (("whole", [1000]), ("cut", [3, 2, 64, 1, 33, 7, 128, 2]), ("one by one", [1])):
        if name == "one by one":
            lengths_now, seqs_now, want_now = lengths[1:], h_seqs[1:], want[1:]
        else:
            lengths_now, seqs_now, want_now = lengths, h_seqs, want
        part, precision, cache = build_attention(spec, w, dtype)
        got = run_part(part, precision, seqs_now, cuts_of(lengths_now, sizes), cache, Feeder(len(seqs_now), seed=len(name)))
        for s, wanted in enumerate(want_now):
            close(got[s], wanted, rel, f"{name}, sequence {s}")


@pytest.mark.parametrize("dtype", BOTH)
def test_a_layer_that_reads_another_layers_keys_under_its_own_chunk(dtype):
    heads, kv, dim, vdim, hidden = 6, 3, 32, 16, 80
    g = torch.Generator().manual_seed(5)
    w = {"q": matrix(g, heads * dim, hidden, dtype), "k": matrix(g, kv * dim, hidden, dtype),
         "v": matrix(g, kv * vdim, hidden, dtype), "o": matrix(g, hidden, heads * vdim, dtype)}
    w2 = {"q": matrix(g, heads * dim, hidden, dtype), "o": matrix(g, hidden, heads * vdim, dtype)}
    h1, h2 = (torch.randn(150, hidden, generator=g, dtype=F64) for _ in range(2))
    if dtype == torch.bfloat16:
        h1, h2 = bf16_round(h1), bf16_round(h2)
    _, keys = plain_attention(h1, w, heads, kv, dim, vdim, 48, 16, 0.2)
    want, _ = plain_attention(h2, w2, heads, kv, dim, vdim, 37, 16, 0.3, keys=keys)
    owner, precision, cache = build_attention(attention_spec(heads, kv, dim, vdim, 48, 16, 0.2, hidden), w, dtype)
    reader, _, _ = build_attention(attention_spec(heads, kv, dim, vdim, 37, 16, 0.3, hidden, shares=True), w2, dtype)
    assert reader.state_spec() is None and "k" not in reader.names
    feeder = Feeder(1)
    from flyweight_b200.engine import StepContext
    outs = []
    for m in (70, 1, 1, 50, 28):
        batch = feeder.batch([(0, m)])
        ctx = StepContext(batch, precision, DEV)
        at = feeder.done[0]
        owner.forward(ctx, dev(h1[at:at + m], precision.act_dtype), cache)
        outs.append(reader.forward(ctx, dev(h2[at:at + m], precision.act_dtype), cache).float().cpu())
        feeder.advance([(0, m)])
    close(torch.cat(outs), want, 2e-5 if dtype == torch.float32 else 3 * 2.0 ** -7, "the reading layer")


# ------------------------------------------------------------------ one key that stands out, at every edge
def edge_cases():
    cases = []
    for chunk in (50, 64, 100, 130):
        for n in (chunk * 2 + 1, chunk * 3, 257, 450):
            first = (n - 1) // chunk * chunk              # the first position the last query sees
            for far in {first, first + 1, n - 1, first - 1, first - 2, 0, 63, 64, (first // 64) * 64 - 1}:
                if 0 <= far < n:
                    cases.append((chunk, n, far))
    return sorted(set(cases))


@pytest.mark.parametrize("dtype", BOTH)
@pytest.mark.parametrize("chunk,n,far", edge_cases())
def test_one_key_that_stands_out_at_a_chunks_and_a_pages_edges(dtype, chunk, n, far):
    """Random scores hide a lost or a wrongly seen key among hundreds.  Here the last query matches the
    key at ``far`` far more than any other: if it lies inside the query's chunk the output is its value,
    if it lies just outside the output must not show it -- for a decoded token and for the last token of
    a portion, through every attention kernel."""
    from flyweight_b200.engine import StepContext
    from flyweight_b200.kernels import attention, ops
    heads, kv, hd = 12, 3, 64
    g = torch.Generator().manual_seed(chunk + n + far)
    keys = torch.randn(n, kv, hd, generator=g, dtype=F64) * 0.3
    values = torch.randn(n, kv, hd, generator=g, dtype=F64)
    query = torch.randn(heads, hd, generator=g, dtype=F64) * 0.3
    keys[far, 1] = 5.0 * query[5] / query[5].norm()          # head 5 (of key head 1) looks for `far`
    query[5] *= 6.0 / query[5].norm()
    if dtype == torch.bfloat16:
        keys, values, query = bf16_round(keys), bf16_round(values), bf16_round(query)
    seen = far >= (n - 1) // chunk * chunk
    positions = torch.arange(n)
    want = P.chunked_attention(query[None], positions[-1:], keys, values, positions, 1.0, chunk).view(heads, hd)
    if seen:
        assert float((want[5] - values[far, 1]).abs().max()) < 0.05 * float(values[far, 1].abs().max())
    else:
        assert float((want[5] - values[far, 1]).abs().max()) > 0.2
    feeder = Feeder(1, n_pages=12, seed=far)
    feeder.batch([(0, n)])                                    # hands out the pages
    k_pool = torch.full((12, kv, 64, hd), float("nan"), dtype=F64)
    v_pool = torch.full((12, kv, 64, hd), float("nan"), dtype=F64)
    for i, page in enumerate(feeder.pages[0]):
        rows = keys[i * 64:(i + 1) * 64]
        k_pool[page, :, :rows.shape[0]] = rows.transpose(0, 1)
        v_pool[page, :, :rows.shape[0]] = values[i * 64:(i + 1) * 64].transpose(0, 1)
    cache = type("Cache", (), {})()
    cache.k_pool, cache.v_pool = dev(k_pool, dtype), dev(v_pool, dtype)
    rel = 1e-5 if dtype == torch.float32 else 2.0 ** -7
    for new in sorted({1, min(40, n), min(130, n)}):
        feeder.done[0] = n - new
        batch = feeder.batch([(0, new)])
        qa = torch.zeros(new, heads, hd, dtype=F64)
        qa[-1] = query
        ctx = StepContext(batch, None, DEV)
        ways = [("tiled", True)] if dtype == torch.bfloat16 else []
        for name, tiled in [("default", False)] + ways:
            attention.force_tiled(tiled)
            try:
                out = attention.paged_attention(ctx, dev(qa, dtype).view(new, -1), cache, batch.block_tables[0],
                                                heads, -chunk, 1.0, dtype)
            finally:
                attention.force_tiled(False)
            close(out.view(new, heads, hd)[-1], want, rel, f"{name} kernel, {new} new tokens")
    assert ops is not None


# ------------------------------------------------------------------ the gated delta rule
def delta_spec(heads, kv, dim, vdim, taps, hidden):
    from flyweight_b200.config.spec import PartSpec
    names = ("q", "k", "v", "q_conv", "k_conv", "v_conv", "b", "a", "a_log", "dt_bias", "gate", "norm", "o")
    return PartSpec("gated_delta_rule", {"hidden_size": hidden, "num_heads": heads, "num_kv_heads": kv, "dim": dim,
                                         "vdim": vdim, "taps": taps, "eps": 1e-5}, {n: n for n in names})


def delta_weights(g, heads, kv, dim, vdim, taps, hidden, dtype):
    def vector(n, scale, shift=0.0):
        v = shift + scale * torch.randn(n, generator=g, dtype=F64)
        return bf16_round(v) if dtype == torch.bfloat16 else v.to(torch.float32).to(F64)
    w = {"q": matrix(g, kv * dim, hidden, dtype), "k": matrix(g, kv * dim, hidden, dtype),
         "v": matrix(g, heads * vdim, hidden, dtype), "gate": matrix(g, heads * vdim, hidden, dtype),
         "b": matrix(g, heads, hidden, dtype), "a": matrix(g, heads, hidden, dtype),
         "o": matrix(g, hidden, heads * vdim, dtype), "a_log": vector(heads, 0.5, -1.0), "dt_bias": vector(heads, 0.5),
         "norm": vector(vdim, 0.1, 1.0)}
    for name, rows in (("q_conv", kv * dim), ("k_conv", kv * dim), ("v_conv", heads * vdim)):
        w[name] = vector(rows * taps, 0.6).view(rows, taps)
    return w


def plain_delta(h, w, heads, kv, dim, vdim):
    names = {"q.conv": "q_conv", "k.conv": "k_conv", "v.conv": "v_conv", "A_log": "a_log", "g": "gate"}
    plain = {**w, **{theirs: w[ours] for theirs, ours in names.items()}}
    return P.delta_mixer(h, plain, heads, kv, dim, vdim, 1e-5)[0]


DELTA_SHAPES = [  # heads, kv, dim, vdim, taps, hidden
    (4, 2, 16, 24, 4, 80), (3, 1, 40, 20, 3, 96), (2, 2, 8, 8, 2, 64), (4, 2, 64, 128, 4, 128), (1, 1, 128, 64, 1, 72),
    (2, 1, 256, 40, 2, 64),
]


@pytest.mark.parametrize("shape", DELTA_SHAPES)
@pytest.mark.parametrize("dtype", BOTH)
def test_delta_rule_whole_cut_and_one_by_one(shape, dtype):
    """The state and the convolution's last inputs are carried through a slot: whole sequences, portions
    down to one and two tokens, four sequences side by side in slots that are not their batch places."""
    from flyweight_b200.kernels.recurrent import delta_state_size
    from flyweight_b200.parts import build_mixer
    heads, kv, dim, vdim, taps, hidden = shape
    g = torch.Generator().manual_seed(sum(shape))
    w = delta_weights(g, heads, kv, dim, vdim, taps, hidden, dtype)
    lengths = [210, 70, 1, 33]
    h_seqs = [torch.randn(n, hidden, generator=g, dtype=F64) for n in lengths]
    if dtype == torch.bfloat16:
        h_seqs = [bf16_round(h) for h in h_seqs]
    want = [plain_delta(h, w, heads, kv, dim, vdim) for h in h_seqs]
    precision = precision_of(dtype)
    part = build_mixer(delta_spec(heads, kv, dim, vdim, taps, hidden))
    part.bind(lambda n: w[n].to(dtype), precision, DEV)
    assert part.state_spec().shape == (delta_state_size(heads, kv, dim, vdim, taps),)
    rel = 2e-5 if dtype == torch.float32 else 3 * 2.0 ** -7
    cache = type("Cache", (), {})()
    for name, sizes in (("whole", [1000]), ("cut", [3, 2, 64, 1, 33, 7, 2]), ("one by one", [1])):
        cache.state = torch.zeros((6, part.state_spec().shape[0]), dtype=torch.float32, device=DEV)
        cache.state[0].fill_(float("nan"))          # nobody's slot: never read
        slots = {0: 4, 1: 2, 2: 5, 3: 1}
        got = run_part(part, precision, h_seqs, cuts_of(lengths, sizes), cache, Feeder(4, slots=slots))
        for s, wanted in enumerate(want):
            close(got[s], wanted, rel, f"{name}, sequence {s}")
        assert torch.isnan(cache.state[0]).all() and float(cache.state[3].abs().max()) == 0.0


@pytest.mark.parametrize("H,G,d,e", [(2, 1, 128, 40), (3, 3, 64, 16), (2, 2, 128, 4), (4, 2, 64, 36)])
@pytest.mark.parametrize("strong", [False, True])
def test_delta_chunks_against_the_scan_and_64_bits(H, G, d, e, strong):
    """The chunked form at the edges of its chunks of 32 and of its 16 columns, on a state that is not zero, with
    keys that repeat and with decays down to e^-60 a token: as close to 64 bits as the token-by-token scan (one rounding
    more for what differs by chance in so few tokens; both stay within 64 roundings of the largest value)."""
    from flyweight_b200.kernels import recurrent
    g = torch.Generator().manual_seed(H * d + e)
    lengths, L, C = [31, 1, 32, 33, 97, 64], 1, 2 * G * d + H * e
    T = sum(lengths)
    p = torch.randn(T, C + H * e + 2 * H, generator=g, dtype=F64).float()
    p[::3, G * d:2 * G * d] = p[0, G * d:2 * G * d]                   # the same key again and again
    if strong:
        p[:, C + H * e + H:] = 60.0 * torch.rand(T, H, generator=g).float()
    taps, zeros = torch.ones(C, 1), torch.zeros(H)
    start = torch.randn(7, recurrent.delta_state_size(H, G, d, e, L), generator=g, dtype=F64).float()
    x = p.double()
    act = x[:, :C] * torch.sigmoid(x[:, :C])
    q, k = act[:, :G * d].view(T, G, d), act[:, G * d:2 * G * d].view(T, G, d)
    q, k = (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = ((t * s).repeat_interleave(H // G, dim=1) for t, s in ((q, d ** -0.5), (k, 1.0)))
    v, beta = act[:, 2 * G * d:].view(T, H, e), torch.sigmoid(x[:, C + H * e:C + H * e + H])
    decay = torch.exp(-torch.nn.functional.softplus(x[:, C + H * e + H:]))
    want, after, at = torch.empty(T, H, e, dtype=F64), start.double().clone(), 0
    for s, n in enumerate(lengths):
        S = after[s + 1, :H * d * e].view(H, e, d)
        for t in range(at, at + n):
            S *= decay[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.einsum("hed,hd->he", S, k[t]))
            S += u[:, :, None] * k[t][:, None, :]
            want[t] = torch.einsum("hed,hd->he", S, q[t])
        at += n
    starts = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    batch = type("Batch", (), {})()
    batch.n_segments, batch.max_segment = len(lengths), max(lengths)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)
    batch.seg_start, batch.seg_slot = i32(starts), i32(list(range(1, len(lengths) + 1)))
    batch.tok_seg = i32([s for s, n in enumerate(lengths) for _ in range(n)])
    errors = []
    for chunked in (True, False):
        recurrent.CHUNKS_FROM, before = (16 if chunked else 10 ** 9), recurrent.CHUNKS_FROM
        try:
            state = dev(start, torch.float32)
            o = recurrent.delta_rule(dev(p, torch.float32), dev(taps), dev(zeros), dev(zeros), state, batch, H, G, d, e)
        finally:
            recurrent.CHUNKS_FROM = before
        errors.append((float((o.cpu().double() - want).norm() / want.norm()),
                       float((state.cpu().double() - after).norm() / after.norm())))
        close(o.cpu().view(T, H, e), want, 64 * 2.0 ** -24, f"chunked {chunked}: read out")
        close(state.cpu(), after, 64 * 2.0 ** -24, f"chunked {chunked}: state")
    assert errors[0][0] <= errors[1][0] + 2.0 ** -24 and errors[0][1] <= errors[1][1] + 2.0 ** -24, errors
    print("errors", errors)


def test_the_scan_takes_four_times_as_long_for_four_times_the_tokens():
    """128 blocks that walk a sequence token by token fit the SMs one by one.  Where some met on an SM, beside the last blocks
    of the kernel in front of them, 2,048 tokens took 5.0 times as long as 512; apart they take 3.7 times."""
    from flyweight_b200.kernels import recurrent
    H, G, d, e, L = 16, 8, 128, 128, 4
    C = 2 * G * d + H * e

    def shortest(T):
        p, zeros = torch.randn(T, C + H * e + 2 * H, device=DEV), torch.zeros(H, device=DEV)
        taps, state = torch.randn(C, L, device=DEV), torch.zeros(1, recurrent.delta_state_size(H, G, d, e, L), device=DEV)
        batch = type("Batch", (), {})()
        batch.n_segments, batch.max_segment = 1, T
        i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)
        batch.seg_start, batch.seg_slot, batch.tok_seg = i32([0, T]), i32([0]), torch.zeros(T, dtype=torch.int32, device=DEV)
        times = []
        for _ in range(8):
            first, last = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            first.record()
            for _ in range(4):
                recurrent.delta_rule(p, taps, zeros, zeros, state, batch, H, G, d, e, chunks=False)
            last.record()
            last.synchronize()
            times.append(first.elapsed_time(last))
        return min(times)

    assert shortest(2048) < 4.4 * shortest(512)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("part,bad", [("k", "nan"), ("v", "nan"), ("v", "inf"), ("q", "nan")])
def test_a_value_that_is_not_finite_reaches_no_earlier_token(d, part, bad):
    """Token 37 of 75 brings a NaN or an infinity in one head's query, key or value: the tokens before it keep the bits
    that they have without it, and what is not finite behind it is what the token-by-token scan has there."""
    from flyweight_b200.kernels import recurrent
    H = G = 2
    e, n, at = 36, 75, 37
    C = 2 * G * d + H * e
    g = torch.Generator().manual_seed(d)
    p = torch.randn(n, C + H * e + 2 * H, generator=g)
    broken = p.clone()
    broken[at, {"q": 0, "k": G * d, "v": 2 * G * d}[part] + 5] = float(bad)
    start = torch.randn(2, recurrent.delta_state_size(H, G, d, e, 1), generator=g)

    def run(p, chunks_from):
        batch = Feeder(1, slots={0: 1}).batch([(0, n)])
        recurrent.CHUNKS_FROM, before = chunks_from, recurrent.CHUNKS_FROM
        try:
            state = dev(start)
            return recurrent.delta_rule(dev(p), dev(torch.ones(C, 1)), dev(torch.zeros(H)), dev(torch.zeros(H)), state,
                                        batch, H, G, d, e).cpu()
        finally:
            recurrent.CHUNKS_FROM = before

    whole, scanned, chunked = run(p, 16), run(broken, 10 ** 9), run(broken, 16)
    assert torch.equal(chunked[:at], whole[:at])
    assert torch.equal(chunked.isfinite(), scanned.isfinite())
    assert not bool(chunked[at].isfinite().all())


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("told", [True, False])
def test_a_segment_of_the_delta_rule_does_not_see_its_company(d, told):
    """Decoding requests, short portions and long ones in one step, on both sides of the line between scan and chunks
    and in any order: outputs and states have the bits that each segment leaves in a step of its own, whether or not
    the batch says where the long ones are."""
    from flyweight_b200.kernels import recurrent
    H, G, e, L = 4, 2, 20, 4
    C, line = 2 * G * d + H * e, recurrent.CHUNKS_FROM
    g = torch.Generator().manual_seed(d)
    taps, a_log, bias = dev(torch.randn(C, L, generator=g)), dev(torch.randn(H, generator=g)), dev(torch.randn(H, generator=g))
    for lengths in ([1] * 6 + [line + 33], [line, 1, line - 1, 2 * line + 1, 5, 1], [1, 1, line - 1], [line + 7, 2 * line]):
        T = sum(lengths)
        p = dev(torch.randn(T, C + H * e + 2 * H, generator=g))
        start = dev(torch.randn(len(lengths), recurrent.delta_state_size(H, G, d, e, L), generator=g))

        def run(p, members, state):
            feeder = Feeder(len(lengths), n_pages=400, slots={s: s for s in range(len(lengths))})
            batch = feeder.batch([(s, lengths[s]) for s in members])
            if not told:
                plain = type("Batch", (), {})()
                for name in ("n_segments", "max_segment", "seg_start", "seg_slot", "tok_seg"):
                    setattr(plain, name, getattr(batch, name))
                batch = plain
            return recurrent.delta_rule(p, taps, a_log, bias, state, batch, H, G, d, e)

        together, apart = start.clone(), start.clone()
        out = run(p, range(len(lengths)), together)
        at = 0
        for s, n in enumerate(lengths):
            assert torch.equal(run(p[at:at + n].contiguous(), [s], apart), out[at:at + n]), (lengths, s)
            at += n
        assert torch.equal(together, apart), lengths


def test_delta_rule_in_32_bits_has_the_same_bits_however_it_is_cut():
    """A whole sequence, portions of many sizes and single tokens, in float32 at a head size that has a chunked form:
    outputs and the state's slot agree bit for bit."""
    from flyweight_b200.kernels.recurrent import delta_state_size
    from flyweight_b200.parts import build_mixer
    heads, kv, dim, vdim, taps, hidden = 4, 2, 64, 128, 4, 128
    g = torch.Generator().manual_seed(1)
    w = delta_weights(g, heads, kv, dim, vdim, taps, hidden, torch.float32)
    h = [torch.randn(n, hidden, generator=g) for n in (333, 150)]
    part = build_mixer(delta_spec(heads, kv, dim, vdim, taps, hidden))
    part.bind(lambda n: w[n].to(torch.float32), precision_of(torch.float32), DEV)
    results = []
    for sizes in ([1000], [257, 40, 3], [64, 1, 129], [1]):
        cache = type("Cache", (), {})()
        cache.state = torch.zeros((3, delta_state_size(heads, kv, dim, vdim, taps)), device=DEV)
        got = run_part(part, precision_of(torch.float32), h, cuts_of([333, 150], sizes), cache, Feeder(2, slots={0: 2, 1: 0}))
        results.append((got, cache.state))
    for got, state in results[1:]:
        assert all(torch.equal(got[s], results[0][0][s]) for s in got) and torch.equal(state, results[0][1])


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("keys,decay", [("silu", "weak"), ("silu", "strong"), ("repeated", "moderate"), ("aligned", "none"),
                                        ("signed", "weak")])
def test_delta_chunks_are_no_further_from_64_bits_than_the_scan(keys, decay, d):
    """600 tokens of the inputs that the recurrence meets (keys behind silu, keys that come again, keys that nearly
    coincide, keys of both signs; decays from none to e^-60 a token): the error of the chunked form in the read-out and
    in the state is at most the token-by-token scan's (2 % for chance, where it is that of the rounded inputs)."""
    from flyweight_b200.kernels import recurrent
    H, G, e, n = 4, 4, 32, 600
    C = 2 * G * d + H * e
    g = torch.Generator().manual_seed(7)
    p = torch.randn(n, C + H * e + 2 * H, generator=g)
    key = slice(G * d, 2 * G * d)
    if keys == "repeated":
        p[::3, key] = p[0, key]
    elif keys == "aligned":
        p[:, key] = 2.0 + p[0, key].abs() + 0.01 * p[:, key]
        p[:, C + H * e:C + H * e + H] = 4.0                            # beta = 0.98
    elif keys == "signed":
        p[:, :2 * G * d] = 8.0 + p[:, :2 * G * d]                      # silu is close to the identity; taps make it signed
    a = p[:, C + H * e + H:]
    a_log = torch.zeros(H)
    if decay == "none":
        a[:] = -60.0
    elif decay == "weak":
        a_log[:] = -3.0
    elif decay == "strong":
        a[:] = 60.0 * torch.rand(n, H, generator=g)
    taps, zeros = torch.ones(C, 1), torch.zeros(H)
    if keys == "signed":
        taps = torch.where(torch.rand(C, 1, generator=g) < 0.5, -0.25, 1.0)
    start = 0.1 * torch.randn(2, recurrent.delta_state_size(H, G, d, e, 1), generator=g)
    x = p.double()
    act = x[:, :C] * taps[:, 0].double()
    act = act * torch.sigmoid(act)
    unit = lambda t: t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    q, k = unit(act[:, :G * d].view(n, G, d)) * d ** -0.5, unit(act[:, key].view(n, G, d))
    v, beta = act[:, 2 * G * d:].view(n, H, e), torch.sigmoid(x[:, C + H * e:C + H * e + H])
    fade = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(x[:, C + H * e + H:]))
    S, want = start[1].double()[:H * d * e].view(H, e, d).clone(), torch.empty(n, H, e, dtype=F64)
    for t in range(n):
        S *= fade[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hed,hd->he", S, k[t]))
        S += u[:, :, None] * k[t][:, None, :]
        want[t] = torch.einsum("hed,hd->he", S, q[t])
    errors = []
    for chunks in (True, False):
        batch = Feeder(1, slots={0: 1}).batch([(0, n)])
        state = dev(start)
        o = recurrent.delta_rule(dev(p), dev(taps), dev(a_log), dev(zeros), state, batch, H, G, d, e, chunks=chunks)
        after = state[1, :H * d * e].cpu().double().view(H, e, d)
        errors.append((float((o.cpu().double() - want).norm() / want.norm()), float((after - S).norm() / S.norm())))
    print("errors", errors)
    assert n >= recurrent.CHUNKS_FROM
    assert errors[0][0] <= 1.02 * errors[1][0] and errors[0][1] <= 1.02 * errors[1][1], errors


def test_delta_inputs_of_many_short_segments():
    """The convolution in front of the recurrence reads a window of rows that crosses requests: 60 requests of one to
    five tokens in one step leave the bits and the states that each leaves in a step of its own."""
    from flyweight_b200.kernels import recurrent
    H, G, d, e, L = 4, 2, 16, 24, 4
    C = 2 * G * d + H * e
    g = torch.Generator().manual_seed(3)
    lengths = [1 + (7 * i) % 5 for i in range(60)]
    T = sum(lengths)
    p = dev(torch.randn(T, C + H * e + 2 * H, generator=g))
    taps, a_log, bias = dev(torch.randn(C, L, generator=g)), dev(torch.randn(H, generator=g)), dev(torch.randn(H, generator=g))
    start = dev(torch.randn(61, recurrent.delta_state_size(H, G, d, e, L), generator=g))
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)

    def run(p, lengths, slots, state):
        batch = type("Batch", (), {})()
        batch.n_segments, batch.max_segment = len(lengths), max(lengths)
        batch.seg_start, batch.seg_slot = i32([sum(lengths[:i]) for i in range(len(lengths) + 1)]), i32(slots)
        batch.tok_seg = i32([s for s, n in enumerate(lengths) for _ in range(n)])
        return recurrent.delta_rule(p, taps, a_log, bias, state, batch, H, G, d, e)

    assert T >= 128
    together, apart = start.clone(), start.clone()
    out = run(p, lengths, list(range(1, 61)), together)
    at = 0
    for s, n in enumerate(lengths):
        assert torch.equal(run(p[at:at + n].contiguous(), [n], [s + 1], apart), out[at:at + n]), s
        at += n
    assert torch.equal(together, apart)


def test_the_delta_state_remembers_a_write_from_hundreds_of_tokens_ago():
    """One early token writes a value under a key that no later token touches (later keys are orthogonal
    to it and decay is switched off): a query for that key, 400 tokens and several steps later, reads the
    value back.  A state that was dropped, reset or shifted between steps would not."""
    from flyweight_b200.kernels import recurrent
    H, G, d, e, L, n = 2, 1, 16, 8, 1, 400
    C = 2 * G * d + H * e
    p = torch.zeros(n, C + H * e + 2 * H, dtype=F64)
    g = torch.Generator().manual_seed(9)
    big = 20.0                                          # silu(20) ~ 20; unit vectors forget the length
    p[:, G * d + 1] = big                               # every key: axis 1
    p[:, 0 * d + 2] = big                               # every query: axis 2 (reads nothing)
    p[7, G * d:2 * G * d] = 0
    p[7, G * d + 0] = big                               # token 7 writes under axis 0
    v7 = torch.randn(H * e, generator=g, dtype=F64).abs() + 1.0
    p[:, 2 * G * d:C] = torch.randn(n, H * e, generator=g, dtype=F64)
    p[7, 2 * G * d:C] = v7
    p[:, C + H * e:C + H * e + H] = 30.0                # beta = 1
    p[:, C + H * e + H:] = -30.0                        # softplus -> 0: decay 1
    p[n - 1, 0:G * d] = 0
    p[n - 1, 0] = big                                   # the last query asks for axis 0
    taps = torch.ones(C, 1, dtype=torch.float32)
    zeros = torch.zeros(H, dtype=torch.float32)
    state = torch.zeros((2, recurrent.delta_state_size(H, G, d, e, L)), dtype=torch.float32, device=DEV)
    feeder = Feeder(1, slots={0: 1})
    outs = []
    for step in cuts_of([n], [5, 64, 1, 1, 130, 2]):
        batch = feeder.batch(step)
        at, m = feeder.done[0], step[0][1]
        outs.append(recurrent.delta_rule(dev(p[at:at + m], torch.float32), dev(taps), dev(zeros), dev(zeros), state,
                                         batch, H, G, d, e).cpu())
        feeder.advance(step)
    out = torch.cat(outs).view(n, H * e)
    want = P.silu(v7) * d ** -0.5
    close(out[n - 1], want, 1e-4, "the value written 392 tokens before")
    assert float(out[n - 2].abs().max()) < 1e-3 * float(want.abs().max())


def test_gated_head_norm():
    from flyweight_b200.kernels import recurrent
    g = torch.Generator().manual_seed(4)
    T, H, e = 9, 3, 20
    o = torch.randn(T, H, e, generator=g, dtype=torch.float32) * 4
    wide = torch.randn(T, 100 + H * e, generator=g, dtype=torch.float32)
    weight = 1 + 0.1 * torch.randn(e, generator=g, dtype=torch.float32)
    gate = wide[:, 40:40 + H * e]
    want = (P.rms_unit(o.to(F64), 1e-5) * weight.to(F64) * P.silu(gate.to(F64)).view(T, H, e)).view(T, H * e)
    for dtype in BOTH:
        out = recurrent.gated_head_norm(dev(o), dev(wide)[:, 40:40 + H * e], dev(weight), 1e-5, dtype)
        close(out, want, 1e-6 if dtype == torch.float32 else 2.0 ** -8, str(dtype))


# ------------------------------------------------------------------ the router and the experts
ROUTERS = [  # outputs, groups, keep, top
    (8, 4, 2, 3), (5, 1, 1, 1), (6, 3, 2, 4), (8, 2, 1, 2), (20, 5, 2, 6), (64, 8, 3, 8), (7, 7, 7, 7), (33, 1, 1, 5),
]


@pytest.mark.parametrize("W", [512, 520, 2112])
@pytest.mark.parametrize("N,groups,keep,top", [(8, 4, 2, 3), (33, 1, 1, 5), (20, 5, 2, 6)])
@pytest.mark.parametrize("dtype", BOTH)
def test_router_over_wide_rows(W, N, groups, keep, top, dtype):
    """Few tokens with rows of 512 entries and more take the kernel's other way through the products (K cut
    over the warps): whole turns of all warps, a last turn that only some warps take part in, a last piece."""
    from flyweight_b200.kernels import experts
    g = torch.Generator().manual_seed(N + W)
    T = 40
    h = torch.randn(T, W, generator=g, dtype=F64)
    h = bf16_round(h) if dtype == torch.bfloat16 else h.to(torch.float32).to(F64)
    router = (torch.randn(N, W, generator=g, dtype=F64) / math.sqrt(W) * 2).to(torch.float32)
    correction = (torch.randn(N, generator=g, dtype=F64) * 0.15).to(torch.float32)
    ids, weights = experts.route(dev(h, dtype), dev(router), dev(correction), groups, keep, top)
    want_ids, want_w = P.route(h, router.to(F64), correction.to(F64), groups, keep, top)
    same = (ids.cpu().long() == want_ids).all(dim=1)
    assert same.float().mean() > 0.95, f"{int((~same).sum())} of {T} tokens choose differently"
    close(weights.cpu()[same], want_w[same], 1e-5, "weights")


@pytest.mark.parametrize("N,groups,keep,top", ROUTERS)
@pytest.mark.parametrize("dtype", BOTH)
def test_router(N, groups, keep, top, dtype):
    """Chosen outputs and weights against the plain router on the same inputs.  Corrections are large
    enough to change the choice (so that a choice made on the plain scores would show) and negative for
    some outputs (so that a group counted as 0 instead of minus infinity would show)."""
    from flyweight_b200.kernels import experts
    g = torch.Generator().manual_seed(N * top)
    T, W = 300, 72
    h = torch.randn(T, W, generator=g, dtype=F64)
    h = bf16_round(h) if dtype == torch.bfloat16 else h.to(torch.float32).to(F64)
    router = (torch.randn(N, W, generator=g, dtype=F64) / math.sqrt(W) * 2).to(torch.float32)
    correction = (torch.randn(N, generator=g, dtype=F64) * 0.15 - 0.3).to(torch.float32)
    ids, weights = experts.route(dev(h, dtype), dev(router), dev(correction), groups, keep, top)
    want_ids, want_w = P.route(h, router.to(F64), correction.to(F64), groups, keep, top)
    same = (ids.cpu().long() == want_ids).all(dim=1)
    assert same.float().mean() > 0.99, f"{int((~same).sum())} of {T} tokens choose differently"
    close(weights.cpu()[same], want_w[same], 1e-5, "weights")
    plain_choice = torch.topk(torch.softmax(h @ router.to(F64).T, dim=-1), top, dim=-1).indices
    if N > top and (groups > keep or N > 8):
        assert not (plain_choice == want_ids).all(), "this case does not tell a choice without correction apart"


def experts_spec(hidden, ff, n_experts, identity, top, groups, keep):
    from flyweight_b200.config.spec import PartSpec
    tensors = {"router": "router", "correction": "correction"}
    for j in range(n_experts):
        tensors.update({f"gate{j}": f"e{j}.gate", f"up{j}": f"e{j}.up", f"down{j}": f"e{j}.down"})
    return PartSpec("routed_experts", {"hidden_size": hidden, "ffn_dim": ff, "experts": n_experts, "identity": identity,
                                       "top": top, "groups": groups, "keep_groups": keep}, tensors)


@pytest.mark.parametrize("dtype", BOTH)
@pytest.mark.parametrize("hidden,ff,n_experts,identity,top,groups,keep",
                         [(80, 48, 6, 2, 3, 4, 2), (96, 40, 5, 0, 1, 1, 1), (96, 24, 3, 3, 4, 3, 2),
                          (128, 64, 8, 0, 2, 2, 1), (64, 70, 1, 1, 2, 1, 1), (72, 16, 0, 4, 2, 2, 2)])
@pytest.mark.parametrize("T", [1, 5, 300])
def test_routed_experts(dtype, hidden, ff, n_experts, identity, top, groups, keep, T):
    """The feed-forward part against the plain one: experts that get no token, experts that get more
    than a tile of them, identity experts, a router with identity experts only.  In bfloat16 the
    corrections are far apart, so that the choice does not hang on the rounding of the scores."""
    from flyweight_b200.parts import build_feed_forward
    g = torch.Generator().manual_seed(hidden + ff + T)
    N = n_experts + identity
    w = {"router": matrix(g, N, hidden, dtype) * 3, "correction": torch.randn(N, generator=g, dtype=F64) * 0.1}
    if dtype == torch.bfloat16:
        w["correction"] = torch.randperm(N, generator=g).to(F64) * 4.0
    for j in range(n_experts):
        w[f"e{j}.gate"], w[f"e{j}.up"] = matrix(g, ff, hidden, dtype), matrix(g, ff, hidden, dtype)
        w[f"e{j}.down"] = matrix(g, hidden, ff, dtype)
    h = torch.randn(T, hidden, generator=g, dtype=F64)
    h = bf16_round(h) if dtype == torch.bfloat16 else h.to(torch.float32).to(F64)
    precision = precision_of(dtype)
    part = build_feed_forward(experts_spec(hidden, ff, n_experts, identity, top, groups, keep))
    part.bind(lambda n: w[n].to(dtype), precision, DEV)
    got = run_part(part, precision, [h], [[(0, T)]], None, feed_forward=True)[0]
    if dtype == torch.bfloat16:
        # the grouped tensor-core product (the default where the sizes allow it) beside the fp32-FMA kernel
        from flyweight_b200.kernels import experts as expert_kernels, tensorcore
        expert_kernels.set_tensor_cores(False)
        try:
            plain_way = run_part(part, precision, [h], [[(0, T)]], None, feed_forward=True)[0]
        finally:
            expert_kernels.set_tensor_cores(True)
        close(plain_way, got, 2.0 ** -7, "the two kernels of the experts' products")
        assert tensorcore.status() == 0
    plain_experts = [(w[f"e{j}.gate"], w[f"e{j}.up"], w[f"e{j}.down"]) for j in range(n_experts)]
    want = P.moe(h, w["router"], w["correction"], plain_experts, identity, groups, keep, top)
    close(got, want, 2e-5 if dtype == torch.float32 else 3 * 2.0 ** -7, "experts")
    # the same with the output norm and the residual sum in the part's last kernel
    from flyweight_b200.engine import StepContext
    x = torch.randn(T, hidden, generator=g, dtype=torch.float32)
    w_norm = 1 + 0.1 * torch.randn(hidden, generator=g, dtype=torch.float32)
    xd = dev(x)
    part.forward_add_normed(StepContext(Feeder(1).batch([(0, T)]), precision, DEV), dev(h, precision.act_dtype), xd,
                            dev(w_norm), 1e-5)
    close(xd, x.to(F64) + P.rms_norm(want, w_norm.to(F64), 1e-5), 2e-5 if dtype == torch.float32 else 3 * 2.0 ** -7,
          "normed and added")
    # a token's result does not depend on what else is in the step
    if T > 5:
        alone = run_part(part, precision, [h[:3]], [[(0, 3)]], None, feed_forward=True)[0]
        close(alone, got[:3], 0.0 if dtype == torch.float32 else 2.0 ** -8, "three tokens alone")
