"""Wide-head attention (one head, head_dim 512: the VAE mid-block shape, src/metal/mvattn_owned.zig)
against the oracle's CPU attention (src/runtime/attention.zig:21-98) through the C ABI."""
import numpy as np
import pytest
import torch

from zdraw_b200 import mattn

pytestmark = pytest.mark.gpu

# fp16 operands with f32 accumulation and half probabilities against the f32 oracle, N(0,1) inputs:
# the bounds the attention tests use for fp16 I/O.
MAX_ABS, MEAN_ABS = 1e-2, 1e-3


@pytest.fixture(scope="module")
def ctx():
    c = mattn.Context(0)
    yield c
    c.deinit()


def make(tokens, dim, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return tuple(torch.randn((tokens, dim), generator=g, device="cuda") * scale for _ in range(3))


@pytest.mark.parametrize("tokens,dim", [(256, 256), (768, 512), (1024, 512), (64, 256), (320, 512), (1600, 512), (96, 64), (160, 320), (32, 32)])
def test_small_shapes_match_cpu_attention(ctx, oracle, tokens, dim):
    q, k, v = make(tokens, dim, tokens + dim)
    out = torch.full((tokens, dim), float("nan"), device="cuda")
    ctx.wide_attention(q, k, v, out, mattn.Config(tokens, 1, 1, dim))
    torch.cuda.synchronize()
    assert ctx.last_status() == 0
    want = oracle.sdpa(q.cpu().numpy(), k.cpu().numpy(), v.cpu().numpy(), heads=1)
    err = np.abs(out.cpu().numpy() - want.reshape(tokens, dim))
    assert err.max() <= MAX_ABS and err.mean() <= MEAN_ABS
    if dim >= 256:
        assert ctx.wide_attention_route() == 0  # N(0,1) operands: norms that call for no more than a sample of the keys


@pytest.mark.parametrize("gain,route", [(1.0, 0), (1.25, 0), (3.0, 1), (6.0, 1), (10.0, 1)])
def test_peaked_rows_survive_the_estimated_row_maximum(ctx, oracle, gain, route):
    """Scores with a standard deviation of 1, 1.6, 9, 36 and 100 (row maxima near 4, 6, 30, 120 and 330): the row
    maximum that is subtracted may come from a sample of the keys (every 2nd one here), but only while the operands' norms
    keep every score below 80 in exp2 units; beyond that the exact maximum of the half products is taken, as the reference
    does (krow_softmax_h). Either way nothing overflows, nothing is clamped and accuracy holds. The tolerance is the
    fp16 one times two: a peaked softmax amplifies the rounding of P."""
    tokens, dim = 1024, 512
    q, k, v = make(tokens, dim, 5)
    q, k = q * gain, k * gain
    out = torch.full((tokens, dim), float("nan"), device="cuda")
    ctx.wide_attention(q, k, v, out, mattn.Config(tokens, 1, 1, dim))
    torch.cuda.synchronize()
    assert ctx.wide_attention_route() == route
    assert ctx.last_status() == 0
    got = out.cpu().numpy()
    assert np.isfinite(got).all()
    # the oracle sees the operands the kernel multiplies: half q and k (a peaked softmax amplifies
    # the operand rounding, which is not what this test is about)
    qh, kh = q.half().float().cpu().numpy(), k.half().float().cpu().numpy()
    want = oracle.sdpa(qh, kh, v.cpu().numpy(), heads=1).reshape(tokens, dim)
    err = np.abs(got - want)
    assert err.max() <= 2e-2 and err.mean() <= 2e-3


def test_vae_mid_block_shape_sampled_rows_and_repeat(ctx, oracle):
    """16384 tokens x 512 channels (1024 px): sampled query rows against the oracle, every output
    element written, and a second run bit-identical."""
    tokens, dim = 16384, 512
    q, k, v = make(tokens, dim, 7)
    out = torch.full((tokens, dim), float("nan"), device="cuda")
    cfg = mattn.Config(tokens, 1, 1, dim)
    ctx.wide_attention(q, k, v, out, cfg)
    again = torch.empty_like(out)
    ctx.wide_attention(q, k, v, again, cfg)
    torch.cuda.synchronize()
    assert ctx.last_status() == 0
    assert torch.equal(out, again)
    assert torch.isfinite(out).all()
    qh, kh, vh = q.cpu().numpy(), k.cpu().numpy(), v.cpu().numpy()
    got = out.cpu().numpy()
    for r in (0, 255, 256, 8191, 16383):
        want = oracle.sdpa(qh, kh, vh, heads=1, rows=(r, r + 1)).reshape(tokens, dim)[r]
        err = np.abs(got[r] - want)
        assert err.max() <= MAX_ABS and err.mean() <= MEAN_ABS, f"row {r}: {err.max()}"


@pytest.mark.parametrize("tokens", [512, 2080])
def test_large_values_and_a_dominant_key(ctx, oracle, tokens):
    """Scores near 440 from single large values, the dominant key 26 above the runner-up: norms that call for the maxima of
    all keys. At 2080 tokens (rows and keys ragged, a sample would be every 4th key) both keys lie outside the sample;
    at 512 every key is in it, and the norms are only reported."""
    dim = 512
    q, k, v = make(tokens, dim, 11, scale=0.05)
    k[7] = 0.0
    k[9] = 0.0
    k[7, 0], k[9, 0] = 500.0, 470.0   # key 7 wins by 30 * q[:, 0] / sqrt(512)
    q[:, 0] = 20.0
    out = torch.full((tokens, dim), float("nan"), device="cuda")
    ctx.wide_attention(q, k, v, out, mattn.Config(tokens, 1, 1, dim))
    torch.cuda.synchronize()
    assert ctx.wide_attention_route() == 1 and ctx.last_status() == 0
    got = out.cpu().numpy()
    assert np.isfinite(got).all()
    want = oracle.sdpa(q.half().float().cpu().numpy(), k.half().float().cpu().numpy(), v.cpu().numpy(), heads=1)
    err = np.abs(got - want.reshape(tokens, dim))
    assert err.max() <= 2e-2 and err.mean() <= 2e-3
    assert np.allclose(got, v[7].half().float().cpu().numpy()[None, :], atol=2e-3)  # key 7 takes everything


def test_constant_values_and_peaked_scores(ctx):
    """Properties that need no oracle: constant V rows come back as that constant; a query that
    matches one key far better than the rest returns that key's value."""
    tokens, dim = 512, 512
    q, k, _ = make(tokens, dim, 3)
    v = torch.full((tokens, dim), 0.75, device="cuda")
    out = torch.empty((tokens, dim), device="cuda")
    ctx.wide_attention(q, k, v, out, mattn.Config(tokens, 1, 1, dim))
    assert torch.allclose(out, v, atol=2e-3)
    k2 = torch.randn((tokens, dim), device="cuda") * 0.01
    q2 = torch.zeros((tokens, dim), device="cuda")
    k2[5] = 1.0
    q2[:] = 4.0  # score with key 5 = 4 * 512 / sqrt(512) = 90 above the rest
    v2 = torch.randn((tokens, dim), device="cuda")
    ctx.wide_attention(q2, k2, v2, out, mattn.Config(tokens, 1, 1, dim))
    torch.cuda.synchronize()
    assert torch.allclose(out, v2[5].half().float().expand_as(out), atol=2e-3)


def test_shapes_outside_the_kernels_are_declined(ctx):
    x = torch.zeros((280, 512), device="cuda")
    o = torch.empty_like(x)
    with pytest.raises(mattn.UnsupportedShape):
        ctx.wide_attention(x, x, x, o, mattn.Config(280, 1, 1, 512))  # tokens % 32 != 0
    y = torch.zeros((256, 120), device="cuda")
    with pytest.raises(mattn.UnsupportedShape):
        ctx.wide_attention(y, y, y, torch.empty_like(y), mattn.Config(256, 1, 1, 120))  # head_dim % 32 != 0
    x = torch.zeros((256, 512), device="cuda")
    o = torch.empty_like(x)
    with pytest.raises(mattn.UnsupportedShape):
        ctx.wide_attention(x, x, x, o, mattn.Config(256, 2, 2, 512))  # more than one head
    with pytest.raises(mattn.UnsupportedShape):
        ctx.wide_attention(x, x, x, o, mattn.Config(256, 1, 1, 512, causal=True))
    assert ctx.last_status() == 0


@pytest.mark.parametrize("tokens", [1024, 1056, 2080, 4096])
def test_keys_outside_the_sample_are_noticed(ctx, oracle, tokens):
    """Row maxima come from every (tokens // 512)-th key; a key outside that sample that equals a query of usual norm
    lies e^15 above the rest (512 / sqrt(512) = 22.6), beyond what the half range holds: that row (and one of the last,
    ragged block) is rescaled, the others are not, and every row matches the oracle."""
    dim = 512
    q, k, v = make(tokens, dim, tokens)
    hits = {301: 7, tokens - 1: tokens - 3}  # row -> key, no multiple of the stride (2, 2, 4, 8)
    for r, j in hits.items():
        k[j] = q[r]
    cfg = mattn.Config(tokens, 1, 1, dim)
    out = torch.full((tokens, dim), float("nan"), device="cuda")
    ctx.wide_attention(q, k, v, out, cfg)
    again = torch.full_like(out, float("nan"))
    ctx.wide_attention(q, k, v, again, cfg)
    in_place = q.clone()  # the result may take an operand's place
    ctx.wide_attention(in_place, k, v, in_place, cfg)
    torch.cuda.synchronize()
    assert ctx.wide_attention_route() == 1 and ctx.last_status() == 0
    assert torch.equal(out, again)
    assert torch.equal(out, in_place)
    got = out.cpu().numpy()
    qh, kh, vh = q.cpu().numpy(), k.cpu().numpy(), v.cpu().numpy()
    for r in (0, 255, 256, 301, 511, 512, tokens - 1):
        want = oracle.sdpa(qh, kh, vh, heads=1, rows=(r, r + 1)).reshape(tokens, dim)[r]
        err = np.abs(got[r] - want)
        assert err.max() <= MAX_ABS and err.mean() <= MEAN_ABS, f"row {r}: {err.max()}"
    assert np.allclose(got[301], vh[7], atol=4e-3)
    q2, k2, v2 = make(tokens, dim, tokens + 1)
    ctx.wide_attention(q2, k2, v2, out, cfg)
    assert ctx.wide_attention_route() == 0  # the next call starts afresh


@pytest.mark.parametrize("tokens", [1056, 2080])
def test_norms_decide_how_row_maxima_are_taken(ctx, oracle, tokens):
    """Above 1024 tokens, last row block ragged: a dominant key outside the sample (every 2nd, every 4th key) with a value
    of 500, under norms that allow scores of 600, takes the maxima of all keys; the same value with norms that keep every
    score below 80 does not; a NaN does, and the rows it is not in come out right. None of it reaches the next call."""
    dim = 512
    cfg = mattn.Config(tokens, 1, 1, dim)
    q, k, v = make(tokens, dim, 11, scale=0.05)
    out = torch.full((tokens, dim), float("nan"), device="cuda")

    def check(rows, route):
        ctx.wide_attention(q, k, v, out, cfg)
        torch.cuda.synchronize()
        assert ctx.wide_attention_route() == route and ctx.last_status() == 0
        qh, kh = q.half().float().cpu().numpy(), k.half().float().cpu().numpy()
        for r in rows:
            want = oracle.sdpa(qh, kh, v.cpu().numpy(), heads=1, rows=(r, r + 1)).reshape(tokens, dim)[r]
            err = np.abs(out[r].cpu().numpy() - want)
            assert err.max() <= 2e-2 and err.mean() <= 2e-3, f"row {r}: {err.max()}"

    k[7], k[9] = 0.0, 0.0
    k[7, 0], k[9, 0] = 500.0, 470.0  # key 7 wins by 30 * 20 / sqrt(512) = 26
    q[:, 0] = 20.0
    check((0, 255, 256, 1030, tokens - 1), 1)
    assert np.allclose(out.cpu().numpy(), v[7].half().float().cpu().numpy()[None, :], atol=2e-3)
    q[:, 0] = 0.0  # |q| = 1.2, |k| = 500
    check((0, 256, tokens - 1), 0)
    k[7], k[9] = k[8], k[8]
    q[40, 3] = float("nan")
    check((0, 39, 41, tokens - 1), 1)
    q[40, 3] = 0.0
    check((0, 40, tokens - 1), 0)


def missed(tokens, dim, seed, rows):
    """N(0, 1) operands; keys outside the sample hold multiples of the given rows' queries, three to a row in different
    blocks of 128 keys: scores of about 14, 18 and 22 (20, 26 and 32 in the exponent of 2), above some 3 of the sample."""
    q, k, v = make(tokens, dim, seed)
    stride = tokens // 512
    free = [j for j in range(tokens) if j % stride]
    for n, r in enumerate(rows):
        for i, f in enumerate((0.62, 0.8, 0.97)):
            k[free[(5 * n + 11 + i * (len(free) // 3)) % len(free)]] = q[r] * f
    return q, k, v


@pytest.mark.parametrize("tokens,n_rows", [(1024, 1), (1056, 60), (2080, 40), (3008, 100), (4096, 100)])
def test_rows_the_sample_missed(ctx, tokens, n_rows):
    """Rows with pieces at up to four scales (and their neighbours that have none), the last row block and the last block
    of keys ragged, against float64 on the half operands."""
    dim = 512
    rows = sorted({(i * 7919 + 3) % tokens for i in range(n_rows)} | {tokens - 1})
    q, k, v = missed(tokens, dim, tokens, rows)
    cfg = mattn.Config(tokens, 1, 1, dim)
    out, again = (torch.full((tokens, dim), float("nan"), device="cuda") for _ in range(2))
    ctx.wide_attention(q, k, v, out, cfg)
    ctx.wide_attention(q, k, v, again, cfg)
    torch.cuda.synchronize()
    assert ctx.wide_attention_route() == 1 and ctx.last_status() == 0
    assert torch.equal(out, again)
    scores = q.half().double() @ k.half().double().T / dim ** 0.5
    want = torch.softmax(scores, -1) @ v.double()
    # P is rounded to half by 2^-11 of its value, twice where a piece falls below the normal range; V by 2^-11; the weights
    # that are summed, rounded or not, differ by another 2^-11
    assert (out - want).abs().max() <= 4 * 2.0 ** -11 * v.abs().max()


def test_a_graph_replays_with_and_without_missed_rows(ctx):
    """One captured call, replayed on operands that the sample misses and on others: the same bytes as calls of their own."""
    tokens, dim = 2080, 512
    cfg = mattn.Config(tokens, 1, 1, dim)
    sets = [missed(tokens, dim, 3, (5, 700, 2079)), make(tokens, dim, 4), missed(tokens, dim, 5, (1, 256))]
    want = []
    for x in sets:
        o = torch.empty((tokens, dim), device="cuda")
        ctx.wide_attention(*x, o, cfg)
        want.append((o, ctx.wide_attention_route()))
    assert [r for _, r in want] == [1, 0, 1]
    q, k, v = (torch.zeros((tokens, dim), device="cuda") for _ in range(3))
    out = torch.empty((tokens, dim), device="cuda")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        ctx.wide_attention(q, k, v, out, cfg)
    for x, (o, route) in zip(sets, want):
        for dst, src in zip((q, k, v), x):
            dst.copy_(src)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, o) and ctx.wide_attention_route() == route
    assert ctx.last_status() == 0


@pytest.mark.parametrize("every", [256, 1])
def test_missed_rows_do_not_cost_a_second_product(ctx, every):
    """4096 x 512: one row in 256, or all of them, that the sample misses. Multiplying their blocks again took 1.63 times as
    long as a call with none; rescaling the rows takes 1.02 and 1.09 times."""
    tokens, dim = 4096, 512
    cfg = mattn.Config(tokens, 1, 1, dim)
    plain = make(tokens, dim, 5)
    q, k, v = (x.clone() for x in plain)
    if every == 1:
        k.copy_(q)  # every query meets itself: 22.6 above the rest
    else:
        k[9::every] = q[3::every]  # no key of the sample (every 8th)
    out = torch.empty_like(q)

    def timed(x):
        best = []
        for _ in range(9):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record()
            for _ in range(20):
                ctx.wide_attention(*x, out, cfg)
            e1.record()
            torch.cuda.synchronize()
            best.append(e0.elapsed_time(e1))
        return min(best)

    timed(plain)
    base = timed(plain)
    assert ctx.wide_attention_route() == 0
    assert timed((q, k, v)) <= 1.3 * base
    assert ctx.wide_attention_route() == 1


@pytest.mark.parametrize("tokens,dim", [(32, 32), (320, 512), (2080, 512), (4096, 512)])
def test_result_in_an_operands_place(ctx, tokens, dim):
    """The same bytes wherever the result goes: in the place of q, k or v, or overlapping two of them, also where P V is
    split over the keys (tiles of 256 x 256 that leave half of the pairs of SMs without one)."""
    x = torch.stack(make(tokens, dim, tokens))
    cfg = mattn.Config(tokens, 1, 1, dim)
    want = torch.empty((tokens, dim), device="cuda")
    ctx.wide_attention(x[0], x[1], x[2], want, cfg)
    for at in (0, tokens // 2, tokens, 2 * tokens):  # rows of the stacked q, k, v
        y = x.clone()
        out = y.view(3 * tokens, dim)[at:at + tokens]
        ctx.wide_attention(y[0], y[1], y[2], out, cfg)
        assert torch.equal(out, want)
    assert ctx.last_status() == 0
