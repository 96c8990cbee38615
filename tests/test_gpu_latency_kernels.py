"""The kernels of a decode step that keep a row in registers, at the edges of their forms."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(*shape, seed=0):
    return torch.randn(*shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed + sum(shape)))


def _close(got, want, terms):
    """32-bit results of a mean over ``terms`` squares (a chain of at most 16 a thread, then a tree) times a few factors with errors of
    an ulp or two each, expf's among them: 64 ulp of the value, and of a tenth of the largest where a sum or a product is nearly zero."""
    want = want.to(torch.float64)
    bound = 64 * 2.0 ** -24 * (want.abs() + 0.1 * want.abs().max())
    assert ((got.to(torch.float64) - want).abs() <= bound).all(), (terms, ((got - want).abs() - bound).max())


# the first and last width of every form, the loop over memory beyond them, rows of odd lengths
@pytest.mark.parametrize("per", [1, 63, 256, 257, 512, 1023, 1024, 1025, 2048, 4095, 4096, 4097, 9000])
@pytest.mark.parametrize("tokens,groups", [(1, 1), (3, 2)])
def test_gated_group_norm(per, tokens, groups):
    from xeno_rt_b200.csrc import ops
    width = per * groups
    y, z, w = _rand(tokens, width), _rand(tokens, width + 7, seed=1), _rand(width, seed=2)
    out = torch.empty_like(y)
    ops.gated_group_norm(out, y, z, w, groups, 1e-5)
    v = (y.double() * torch.nn.functional.silu(z[:, :width].double())).view(tokens, groups, per)
    want = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)).flatten(1) * w.double()
    _close(out, want, per)


@pytest.mark.parametrize("vdim", [1, 32, 33, 64, 65, 128, 129, 256, 257, 511, 512])
@pytest.mark.parametrize("per_head", [False, True])
def test_head_norm_gate(vdim, per_head):
    from xeno_rt_b200.csrc import ops
    for tokens, heads in ((1, 1), (5, 3), (2, 16)):
        o, gate = _rand(tokens, heads * vdim), _rand(tokens, heads * vdim + 5, seed=1)
        w = _rand(heads * vdim if per_head else vdim, seed=2)
        y = torch.empty_like(o)
        ops.head_norm_gate(y, o, w, gate, heads, vdim, 1e-5, "silu")
        v = o.double().view(tokens, heads, vdim)
        weight = w.double().view(-1, vdim) if w.numel() == heads * vdim and heads > 1 else w.double()
        want = v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5) * weight
        want = want.flatten(1) * torch.nn.functional.silu(gate[:, :heads * vdim].double())
        _close(y, want, vdim)


# one choice a lane: scores that are equal, of both zeros, of infinities and NaN (these take the search one choice at a time)
@pytest.mark.parametrize("experts,groups,keep,top", [(16, 4, 2, 2), (32, 8, 3, 6), (12, 3, 2, 4), (5, 1, 1, 5), (8, 8, 3, 3), (1, 1, 1, 1), (33, 3, 2, 7)])
@pytest.mark.parametrize("scores", ["softmax", "sigmoid"])
@pytest.mark.parametrize("normalize", [False, True])
def test_route_scores(experts, groups, keep, top, scores, normalize):
    """The chosen experts by the rule restated one choice at a time; ties to the lower number.  Weights: a few roundings of 32 bits."""
    from xeno_rt_b200.csrc import ops
    rng = np.random.default_rng(experts + top)
    n = 64
    logits = rng.normal(size=(n, experts)).astype(np.float32)
    logits[::3] = np.round(logits[::3])          # equal scores
    logits[1] = 0.0
    correction = (np.round(rng.normal(size=experts)) * 0.25).astype(np.float32)
    for fix in (None, correction):
        ids = torch.empty(n, top, dtype=torch.int32, device=DEV)
        weights = torch.empty(n, top, dtype=torch.float32, device=DEV)
        ops.moe_route_scores(ids, weights, torch.from_numpy(logits).to(DEV), top, groups, keep, scores=scores,
                             correction=None if fix is None else torch.from_numpy(fix).to(DEV), normalize=normalize, sum_eps=1e-9,
                             scale=2.5)
        z = torch.from_numpy(logits).to(DEV)
        if scores == "softmax":
            s = torch.softmax(z.double(), -1)
        else:
            s = torch.sigmoid(z.double())
        # choices are compared by the scores of the logits they stand for: equal logits have equal scores
        choice = s + (torch.from_numpy(fix).to(DEV).double() if fix is not None else 0.0)
        grouped = choice.view(n, groups, -1).max(-1).values
        for t in range(n):
            order = sorted(range(groups), key=lambda g: (-round(float(grouped[t, g]), 12), g))[:keep]
            allowed = [e for e in range(experts) if e // (experts // groups) in order]
            want = sorted(allowed, key=lambda e: (-round(float(choice[t, e]), 12), e))[:top]
            got = ids[t].tolist()
            # a difference below the rounding of 32 bits may decide otherwise, but equal logits (and corrections) are a tie: the lower number
            stands_for = lambda e: (logits[t, e], 0.0 if fix is None else fix[e])
            assert len(set(got)) == top, (t, got)
            assert all(a == b or (abs(float(choice[t, a] - choice[t, b])) < 1e-6 and stands_for(a) != stands_for(b))
                       for a, b in zip(got, want)), (t, got, want)
            w = s[t, ids[t].long()]
            w = w / (w.sum() + 1e-9) if normalize else w
            assert torch.allclose(weights[t].double(), 2.5 * w, rtol=2e-6, atol=1e-12)
    bad = torch.from_numpy(logits).to(DEV)
    bad[0] = float("nan")
    bad[2, 0] = float("inf")
    bad[4] = float("-inf")
    ops.moe_route_scores(ids, weights, bad, top, groups, keep, scores=scores, normalize=normalize)
    assert ((ids >= 0) & (ids < experts)).all()
    assert all(len(set(row)) == top for row in ids.tolist())  # (rows that are no numbers too)
    good = torch.tensor([i for i in range(n) if i not in (0, 2, 4)], device=DEV)
    again, _ = torch.empty_like(ids), None
    ops.moe_route_scores(again, torch.empty_like(weights), torch.from_numpy(logits).to(DEV), top, groups, keep, scores=scores, normalize=normalize)
    assert torch.equal(ids[good], again[good])


@pytest.mark.parametrize("rank,rot,heads", [(192, 64, 16), (256, 32, 5), (320, 64, 3), (40, 8, 1)])
@pytest.mark.parametrize("pairing", ["interleaved", "split_half"])
def test_latent_prepare_by_several_blocks_a_token(rank, rot, heads, pairing):
    """A token's rows are the same bits in a launch of few tokens (several blocks a token) and of many (one)."""
    from xeno_rt_b200.csrc import ops
    dim, n = 32, 300
    head_size = -(-(rank + rot) // 16) * 16
    down = heads * (dim + rot)
    qd, w = _rand(n, down + rank + rot), _rand(rank, seed=3)
    cs = _rand(n, rot // 2, 2, seed=4)
    blocks = -(-n // 64)
    table = torch.arange(blocks, dtype=torch.int32, device=DEV).view(1, -1).contiguous()
    slot = torch.zeros(n, dtype=torch.int32, device=DEV)
    slot[7] = -1
    pos = torch.arange(n, dtype=torch.int32, device=DEV)
    results = []
    for step in (n, 3):
        q = torch.full((n, heads * head_size), 9.0, dtype=torch.bfloat16, device=DEV)
        pool = torch.zeros(blocks, 1, 64, head_size, dtype=torch.bfloat16, device=DEV)
        for a in range(0, n, step):
            b = min(n, a + step)
            ops.latent_prepare(q[a:b], pool, qd[a:b], down, w, 1e-6, cs[a:b], slot[a:b], pos[a:b], table, heads, dim, rot, rank,
                               head_size, write_cache=True, pairing=pairing)
        results.append((q, pool))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


def test_padding_rows_are_cleared():
    """Convolution and scans of single tokens: rows beyond the step's tokens are zeros where that is asked for, and others as without."""
    from xeno_rt_b200.csrc import ops
    n, live = 8, 5
    cu = torch.tensor([min(i, live) for i in range(n + 1)], dtype=torch.int32, device=DEV)
    slots = torch.tensor([i if i < live else -1 for i in range(n)], dtype=torch.int32, device=DEV)
    channels, taps = 200, 4
    x, w = _rand(n, channels), _rand(channels, taps, seed=1)
    outs = []
    for clear in (False, True):
        out, state = torch.full((n, channels), float("nan"), device=DEV), _rand(n, taps - 1, channels, seed=2)
        ops.short_conv(out, x, w, state, cu, slots, 1, "silu", zero_padding=clear)
        outs.append((out, state))
    assert torch.equal(outs[0][0][:live], outs[1][0][:live]) and torch.equal(outs[0][1], outs[1][1])
    assert outs[0][0][live:].isnan().all() and (outs[1][0][live:] == 0).all()
    for heads, dim, vdim, delta in ((4, 128, 40, True), (2, 64, 256, False), (3, 48, 20, True)):
        q, k, v = _rand(n, heads * dim), _rand(n, heads * dim, seed=1), _rand(n, heads * vdim, seed=2)
        decay, beta = torch.rand(n, heads * dim, device=DEV), _rand(n, heads, seed=3)
        outs = []
        for clear in (False, True):
            out, state = torch.full((n, heads * vdim), float("nan"), device=DEV), _rand(n, heads, vdim, dim, seed=4)
            ops.state_scan(out, q, k, v, decay, beta if delta else None, state, cu, slots, heads, heads, dim, vdim, delta=delta,
                           max_new=1, zero_padding=clear)
            outs.append((out, state))
        assert torch.equal(outs[0][0][:live], outs[1][0][:live]) and torch.equal(outs[0][1], outs[1][1])
        assert outs[0][0][live:].isnan().all() and (outs[1][0][live:] == 0).all()
    heads, vdim, size = 4, 24, 128
    x, b, c, dt = _rand(n, heads * vdim), _rand(n, size, seed=1), _rand(n, size, seed=2), _rand(n, heads, seed=3)
    args = (_rand(heads, seed=5), _rand(heads, seed=6), _rand(heads, seed=7))
    outs = []
    for clear in (False, True):
        out, state = torch.full((n, heads * vdim), float("nan"), device=DEV), _rand(n, heads, vdim, size, seed=4)
        ops.ssd_scan(out, x, b, c, dt, *args, state, cu, slots, heads, 1, size, vdim, max_new=1, zero_padding=clear)
        outs.append((out, state))
    assert torch.equal(outs[0][0][:live], outs[1][0][:live]) and torch.equal(outs[0][1], outs[1][1])
    assert outs[0][0][live:].isnan().all() and (outs[1][0][live:] == 0).all()


@pytest.mark.parametrize("width", [33, 1024, 1500, 2048, 2049, 4096])
@pytest.mark.parametrize("top", [1, 2, 5])
def test_norms_of_gathered_parts(width, top):
    """The same bits as from parts written out by moe_combine; more rows than blocks run at once give what a few at a time give."""
    from xeno_rt_b200.csrc import ops
    n = 1000
    y, x0 = _rand(n * top, width), _rand(n, width, seed=1)
    rows = torch.randperm(n * top, device=DEV).to(torch.int32)
    scales = torch.rand(n, top, device=DEV)
    w, b, w2, b2 = (_rand(width, seed=s) for s in (2, 3, 4, 5))
    parts = torch.empty(top, n, width, device=DEV)
    ops.moe_combine(parts, y, rows, scales)
    plain = parts if top > 1 else parts[0]
    results = []
    for form in ("parts", "gathered", "a few at a time"):
        x, out = x0.clone(), torch.empty(n, width, dtype=torch.bfloat16, device=DEV)
        r, copy = x0.clone(), torch.empty(n, width, dtype=torch.bfloat16, device=DEV)
        if form == "parts":
            ops.layernorm_affine(plain, w, b, 1e-5, out=out, residual=x, n_parts=top, then=(w2, b2))
            ops.rmsnorm_add(r, plain, w, 1e-6, copy=copy)
        elif form == "gathered":
            ops.layernorm_affine(y, w, b, 1e-5, out=out, residual=x, then=(w2, b2), gather=(rows, scales))
            ops.rmsnorm_add(r, y, w, 1e-6, copy=copy, gather=(rows, scales))
        else:
            for a in range(0, n, 100):
                some = parts[:, a:a + 100].contiguous()
                ops.layernorm_affine(some if top > 1 else some[0], w, b, 1e-5, out=out[a:a + 100], residual=x[a:a + 100],
                                     n_parts=top, then=(w2, b2))
            ops.rmsnorm_add(r, plain, w, 1e-6, copy=copy)
        results.append((x, out, r, copy))
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))
    v = parts.double().sum(0)
    v = (v - v.mean(-1, keepdim=True)) / torch.sqrt(v.var(-1, unbiased=False, keepdim=True) + 1e-5) * w.double() + b.double()
    _close(results[0][0], x0.double() + v, width)


# the edges of the rules on 148 multiprocessors: rows of one part and of two in one round, in two, and several a block
@pytest.mark.parametrize("rows", [296, 297, 444, 445, 592, 593, 1500])
@pytest.mark.parametrize("width", [1000, 1024, 1025, 2048, 2049])
def test_layer_norm_of_many_rows_gives_the_bits_of_few(rows, width):
    from xeno_rt_b200.csrc import ops
    x, x2, r0 = _rand(rows, width), _rand(2, rows, width, seed=1), _rand(rows, width, seed=2)
    w, b, w2, b2 = (_rand(width, seed=s) for s in (3, 4, 5, 6))

    def all_forms(a, e):
        n, residuals = e - a, [r0[a:e].clone() for _ in range(3)]
        outs = [torch.empty(n, width, dtype=torch.bfloat16, device=DEV) for _ in range(3)]
        ops.layernorm_affine(x[a:e], w, b, 1e-5, out=outs[0])
        ops.layernorm_affine(x[a:e], w, b, 1e-5, residual=residuals[0])
        ops.layernorm_affine(x[a:e], w, b, 1e-5, out=outs[1], residual=residuals[1], then=(w2, b2))
        ops.layernorm_affine(x2[:, a:e].contiguous(), w, b, 1e-5, out=outs[2], residual=residuals[2], n_parts=2, then=(w2, b2))
        return outs + residuals

    some = [all_forms(a, min(rows, a + 100)) for a in range(0, rows, 100)]
    for whole, parts in zip(all_forms(0, rows), zip(*some)):
        assert torch.equal(whole, torch.cat(parts))


@pytest.mark.parametrize("width", [4097, 8192, 8193, 16384])
def test_norm_after_a_sublayer_of_wide_rows(width):
    """The last width of every form beyond 4,096 and the widest: gathered parts give the bits of parts written out, and both the norm."""
    from xeno_rt_b200.csrc import ops
    n, top = 20, 2
    y, x0, w = _rand(n * top, width), _rand(n, width, seed=1), _rand(width, seed=2)
    rows, scales = torch.randperm(n * top, device=DEV).to(torch.int32), torch.rand(n, top, device=DEV)
    parts = torch.empty(top, n, width, device=DEV)
    ops.moe_combine(parts, y, rows, scales)
    plain, gathered = x0.clone(), x0.clone()
    ops.rmsnorm_add(plain, parts, w, 1e-6)
    ops.rmsnorm_add(gathered, y, w, 1e-6, gather=(rows, scales))
    assert torch.equal(plain, gathered)
    v = parts.double().sum(0)
    v = x0.double() + v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-6) * w.double()
    _close(plain, v, width)
