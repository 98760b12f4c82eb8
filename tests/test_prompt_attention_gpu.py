"""The tensor-core prompt attention kernel through its entry points: edges of the 64-key blocks and 128-row tiles, one and two tiles, key slices, windows that
start inside a block, head sizes that end inside a 64-column chunk, groups that do not fill a tile, and rows nobody may see."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# results are bf16 (2^-9 / sqrt(3) = 1.1e-3 in the 2-norm, at most 2^-8 of a value); probabilities enter as two bf16 terms, 2^-17 of them left out
EXACT_P = 2e-3
BF16_P = 1e-2           # D = 128 without a window: probabilities in bf16


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm().clamp_min(1e-30)).item()


def _attend(q, k, v, scale, first, window, causal=True):
    """One sequence in 64 bits: q [n, Hq, D] at positions first.., k, v [m, Hkv, D]."""
    rep = q.shape[1] // k.shape[1]
    k, v = k.double().repeat_interleave(rep, 1), v.double().repeat_interleave(rep, 1)
    s = torch.einsum("qhd,khd->hqk", q.double(), k) * scale
    at, key = torch.arange(q.shape[0], device=q.device)[:, None] + first, torch.arange(k.shape[0], device=q.device)[None, :]
    hide = (key > at) if causal else torch.zeros_like(key > at)
    if window > 0:
        hide = hide | (key <= at - window)
    s = s.masked_fill(hide[None], float("-inf"))
    p = torch.softmax(s, -1).nan_to_num(0.0)
    return torch.einsum("hqk,khd->qhd", p, v)


@pytest.mark.parametrize("hq,hkv,dim,window", [(16, 2, 256, 0), (16, 4, 256, 100), (8, 2, 128, 64), (64, 4, 128, 0), (12, 1, 72, 0), (4, 4, 8, 33), (16, 1, 192, 1000),
                                               (128, 1, 64, 1)])
@pytest.mark.parametrize("new,total", [([1], [1]), ([127, 1, 128], [127, 128, 128]), ([129, 257], [129, 300]), ([1, 1, 1], [1, 64, 900]), ([40, 2], [1040, 66]), ([5], [2000])])
def test_paged(hq, hkv, dim, window, new, total):
    from nanoengine_b200.ops import sm100, sm100_attn
    sm100.clear_kernel_status()
    g = torch.Generator(device="cuda").manual_seed(3)
    nb = [-(-n // 64) for n in total]
    bt = torch.full((len(new), max(nb) + 1), -1, dtype=torch.int32, device="cuda")           # a table entry behind the context is no page
    perm = torch.randperm(sum(nb), generator=g, device="cuda", dtype=torch.int32) + 1
    kc = torch.full((sum(nb) + 2, 64, hkv, dim), float("nan"), dtype=torch.bfloat16, device="cuda")      # and a row behind it no number
    vc = kc.clone()
    q = torch.randn(sum(new), hq, dim, generator=g, device="cuda").to(torch.bfloat16)
    want, at, o = [], 0, 0
    for i, (n, m) in enumerate(zip(new, total)):
        pages = perm[at: at + nb[i]]
        at += nb[i]
        bt[i, : nb[i]] = pages
        k, v = (torch.randn(m, hkv, dim, generator=g, device="cuda").to(torch.bfloat16) for _ in "kv")
        slots = (pages.long()[:, None] * 64 + torch.arange(64, device="cuda")[None]).flatten()[:m]
        kc.view(-1, hkv, dim)[slots], vc.view(-1, hkv, dim)[slots] = k, v
        want.append(_attend(q[o: o + n], k, v, dim ** -0.5, m - n, window))
        if window > 0 and m - n - window >= 64:            # pages wholly in front of the window may have been given away
            gone = (m - n - window + 1) // 64
            vc[pages[:gone].long()] = float("inf")
        o += n
    cu = torch.tensor([0] + torch.tensor(new).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    calls = sm100_attn.PROMPT_TC_CALLS[0]
    tq, t = 128 // (hq // hkv), sum(new)
    plain = dim == 128 and window == 0
    prompt = not plain or (t >= len(new) * tq and min(t, t // tq + len(new)) * hkv > sm100_attn._sms())
    if not prompt:
        vc, kc = vc.nan_to_num(0.0), kc.nan_to_num(0.0)    # the decode kernel multiplies whole pages
    got = sm100_attn.gqa_attention_paged(q, kc, vc, bt, cu, torch.tensor(total, dtype=torch.int32, device="cuda"), dim ** -0.5, window)
    assert sm100.kernel_status()[0] == 0
    assert (sm100_attn.PROMPT_TC_CALLS[0] > calls) == prompt
    assert _rel(got, torch.cat(want)) < (BF16_P if plain else EXACT_P)


@pytest.mark.parametrize("heads,dim", [(16, 72), (3, 80), (2, 256), (1, 64), (5, 136)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("lens", [[1], [128, 0, 1, 127], [129, 300, 64], [700]])
def test_ragged(heads, dim, causal, lens):
    from nanoengine_b200.ops import sm100, sm100_attn
    sm100.clear_kernel_status()
    g = torch.Generator(device="cuda").manual_seed(4)
    t = sum(lens)
    qkv = torch.randn(t, 3, heads, dim, generator=g, device="cuda").to(torch.bfloat16)         # strided views, as a fused projection leaves them
    q, k, v = qkv.unbind(1)
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()
    want = torch.cat([_attend(q[a:b], k[a:b], v[a:b], dim ** -0.5, 0, 0, causal) for a, b in zip(cu, cu[1:])])
    calls = sm100_attn.PROMPT_TC_CALLS[0]
    got = sm100.attention_varlen(q, k, v, torch.tensor(cu, dtype=torch.int32, device="cuda"), dim ** -0.5, causal)
    assert sm100.kernel_status()[0] == 0 and sm100_attn.PROMPT_TC_CALLS[0] == calls + 1
    assert _rel(got, want) < EXACT_P


# more than 32 blocks of 64 keys a CTA, so that every barrier of the ring is used again: (heads, size, lengths, prefix of the first, window, tiles a CTA takes)
@pytest.mark.parametrize("hq,hkv,dim,new,before,window,tiles", [(32, 8, 128, [1500, 333], 900, 512, 2), (32, 8, 128, [1300, 1000], 0, 2000, 2), (16, 2, 256, [1100, 300], 1500, 0, 1),
                                                                (16, 4, 256, [900, 500], 2500, 1900, 1), (32, 4, 64, [400, 70], 2700, 0, 1), (32, 4, 64, [2100, 800], 300, 0, 2)])
def test_long_paged(hq, hkv, dim, new, before, window, tiles):
    from nanoengine_b200.ops import sm100, sm100_attn
    sm100.clear_kernel_status()
    g = torch.Generator(device="cuda").manual_seed(5)
    total = [new[0] + before, *new[1:]]
    nb = [-(-n // 64) for n in total]
    bt = torch.zeros(len(new), max(nb), dtype=torch.int32, device="cuda")
    kc, vc = (torch.randn(sum(nb), 64, hkv, dim, generator=g, device="cuda").to(torch.bfloat16) for _ in "kv")
    q = torch.randn(sum(new), hq, dim, generator=g, device="cuda").to(torch.bfloat16) * 3
    want, at, o = [], 0, 0
    for i, (n, m) in enumerate(zip(new, total)):
        bt[i, : nb[i]] = torch.arange(at, at + nb[i], device="cuda")
        k, v = (x[at: at + nb[i]].reshape(-1, hkv, dim)[:m] for x in (kc, vc))
        want.append(_attend(q[o: o + n], k, v, dim ** -0.5, m - n, window))
        at, o = at + nb[i], o + n
    cu, cl = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0] + torch.tensor(new).cumsum(0).tolist(), total))
    assert sm100_attn._fmha_tiles(sum(new), len(new), hq, hkv, dim, dim) == tiles
    got = sm100_attn.gqa_attention_paged(q, kc, vc, bt, cu, cl, dim ** -0.5, window)
    assert sm100.kernel_status()[0] == 0 and _rel(got, torch.cat(want)) < EXACT_P
    assert torch.equal(got, sm100_attn.gqa_attention_paged(q, kc, vc, bt, cu, cl, dim ** -0.5, window))


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("heads,dim,lens,tiles", [(16, 72, [1300, 1201, 77], 2), (8, 72, [2200], 1), (3, 136, [2300, 40], 1), (16, 128, [2500, 130], 2)])
def test_long_ragged(heads, dim, lens, tiles, causal):
    from nanoengine_b200.ops import sm100, sm100_attn
    sm100.clear_kernel_status()
    g = torch.Generator(device="cuda").manual_seed(6)
    q, k, v = torch.randn(sum(lens), 3, heads, dim, generator=g, device="cuda").to(torch.bfloat16).unbind(1)
    at = [0] + torch.tensor(lens).cumsum(0).tolist()
    cu = torch.tensor(at, dtype=torch.int32, device="cuda")
    want = torch.cat([_attend(3 * q[a:b], k[a:b], v[a:b], dim ** -0.5, 0, 0, causal) for a, b in zip(at, at[1:])])
    assert sm100_attn._fmha_tiles(sum(lens), len(lens), heads, heads, dim, dim) == tiles
    got = sm100.attention_varlen(3 * q, k, v, cu, dim ** -0.5, causal)
    assert sm100.kernel_status()[0] == 0 and _rel(got, want) < EXACT_P
    assert torch.equal(got, sm100.attention_varlen(3 * q, k, v, cu, dim ** -0.5, causal))


def test_a_sequence_does_not_see_its_neighbour_s_infinities():
    from nanoengine_b200.ops import sm100
    x = torch.randn(3, 200, 4, 72, device="cuda").to(torch.bfloat16)
    cu = torch.tensor([0, 100, 200], dtype=torch.int32, device="cuda")
    clean = sm100.attention_varlen(*x, cu, 0.1)
    x[:, 100:] = float("inf")
    assert torch.equal(sm100.attention_varlen(*x, cu, 0.1)[:100], clean[:100])


def _plain(q, k, v, scale, first, window):
    """In 64 bits, a key at a time: values of keys that a token may not see do not take part, whatever they are."""
    s = torch.einsum("qhd,khd->hqk", q.double(), k.double()) * scale
    at, key = torch.arange(q.shape[0], device=q.device)[:, None] + first, torch.arange(k.shape[0], device=q.device)[None, :]
    hide = (key > at) | (key <= at - window if window else torch.zeros_like(key > at))
    p, out = torch.softmax(s.masked_fill(hide[None], float("-inf")), -1), torch.zeros(*q.shape[:2], v.shape[2], dtype=torch.float64, device=q.device)
    for i in range(k.shape[0]):
        out += torch.where(hide[:, i, None, None], 0.0, p[:, :, i].t()[..., None] * v[i].double()[None])
    return out


# one key in the middle of a tile, of a block and of the first tile of a pair; infinities of both signs and no numbers in a few of its columns
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("kind,heads,dim,n,before,window", [("varlen", 4, 72, 300, 0, 0), ("varlen", 16, 64, 1300, 0, 0), ("paged", 4, 128, 300, 70, 100), ("paged", 4, 256, 90, 500, 130),
                                                            ("paged", 64, 128, 400, 0, 0), ("mla", 128, 192, 300, 0, 0), ("mla", 2, 192, 200, 0, 0)])
def test_a_value_reaches_only_the_tokens_that_see_it(kind, heads, dim, n, before, window, bad):
    from nanoengine_b200.ops import sm100, sm100_attn
    sm100.clear_kernel_status()
    g = torch.Generator(device="cuda").manual_seed(7)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)             # noqa: E731
    m, kv = n + before, 4 if heads == 64 else heads
    q, k, v, kr = r(n, heads, dim), r(m, kv, dim), r(m, kv, 128 if kind == "mla" else dim), r(m, 64)
    at = m - n + n // 3 + 7
    v[at, :, 3] = bad
    v[at + 1, :, 20] = -bad
    cu = torch.tensor([0, n], dtype=torch.int32, device="cuda")
    calls = sm100_attn.PROMPT_TC_CALLS[0]
    if kind == "varlen":
        got = sm100.attention_varlen(q, k, v, cu, dim ** -0.5, True)
    elif kind == "mla":
        k[:, :, 128:] = kr[:, None]
        got = sm100.mla_prefill_ragged(q, k[:, :, :128].contiguous(), kr, v, cu, dim ** -0.5)
    else:
        nb = -(-m // 64)
        kc, vc = (torch.zeros(nb + 1, 64, kv, dim, dtype=torch.bfloat16, device="cuda") for _ in "kv")
        kc.view(-1, kv, dim)[64: 64 + m], vc.view(-1, kv, dim)[64: 64 + m] = k, v
        bt = torch.arange(1, nb + 1, dtype=torch.int32, device="cuda")[None]
        got = sm100_attn.gqa_attention_paged(q, kc, vc, bt, cu, torch.tensor([m], dtype=torch.int32, device="cuda"), dim ** -0.5, window)
    assert sm100.kernel_status()[0] == 0
    assert sm100_attn.PROMPT_TC_CALLS[0] == calls + 1
    rep = heads // kv
    want = _plain(q, k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1), dim ** -0.5, m - n, window)
    fin = want.isfinite()
    assert torch.equal(got.isfinite(), fin) and not fin.all()
    assert torch.equal(got[~fin].nan_to_num(nan=7.0).double(), want[~fin].nan_to_num(nan=7.0, posinf=torch.finfo(torch.bfloat16).max, neginf=torch.finfo(torch.bfloat16).min))
    assert _rel(got[fin], want[fin]) < (EXACT_P if window or dim not in (128, 192) else BF16_P)


@pytest.mark.parametrize("dim,window,m,n", [(72, 0, 40, 40), (128, 70, 300, 90), (256, 0, 500, 130)])
def test_probabilities_keep_17_bits(dim, window, m, n):
    """The kernel's 32-bit slices: a probability is off by 2^-17 of itself at most, the rest is 32-bit sums and an exponential (2^-20 is a bound for both)."""
    from nanoengine_b200.ops import sm100_attn
    g = torch.Generator(device="cuda").manual_seed(8)
    hq, hkv, nb = 8, 2, -(-m // 64)
    k, v = (torch.randn(nb, 64, hkv, dim, generator=g, device="cuda").to(torch.bfloat16) for _ in "kv")
    q = (2 * torch.randn(n, hq, dim, generator=g, device="cuda")).to(torch.bfloat16)
    bt, cu, cl = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([list(range(nb))], [0, n], [m]))
    part, lse = torch.empty(2, n, hq, dim, device="cuda"), torch.empty(2, n, hq, device="cuda")
    p = lambda t: t.data_ptr()             # noqa: E731
    assert sm100_attn._fmha_call()(p(q), q.stride(0), p(k), k.stride(0), dim, 0, 0, p(v), v.stride(0), nb, p(bt), nb, p(cu), p(cl), 1, n, hq, hkv, dim, dim, 1, n // 32 + 1, 2, window, 1,
                                   dim ** -0.5, 1, 0, p(part), p(lse), torch.cuda.current_stream().cuda_stream) == 0
    w = torch.exp2(lse.double() - lse.double().amax(0))
    got = (w / w.sum(0))[..., None] * part.double()
    kk, vv = (x.reshape(-1, hkv, dim)[:m] for x in (k, v))
    want, size = _attend(q, kk, vv, dim ** -0.5, m - n, window), _attend(q, kk, vv.abs(), dim ** -0.5, m - n, window)
    assert ((got.sum(0) - want).abs() / size).max().item() < 2 ** -17 + 2 ** -20


@pytest.mark.parametrize("dim,window,n", [(256, 0, 3), (128, 900, 40), (72, 0, 1)])
def test_a_score_that_is_no_number_shows_through_slices(dim, window, n):
    from nanoengine_b200.ops import sm100_attn
    hq, hkv, m = 8, 2, 2000
    kc, vc = (torch.randn(32, 64, hkv, dim, device="cuda").to(torch.bfloat16) for _ in "kv")
    q = torch.randn(n, hq, dim, device="cuda").to(torch.bfloat16)
    kc[(m - n // 2 - 500) // 64, (m - n // 2 - 500) % 64, 1] = float("nan")                # of one key, in one of the slices, for the second half of the heads
    bt, cu, cl = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([list(range(32))], [0, n], [m]))
    got = sm100_attn.gqa_attention_paged(q, kc, vc, bt, cu, cl, dim ** -0.5, window)
    assert got[:, : hq // 2].isfinite().all() and got[:, hq // 2:].isnan().all()


def test_boundaries_past_the_tensors_end_write_nothing_there():
    """Rows and keys end with the tensors, whatever the boundaries say (the buffers of this test are longer, so that nothing can fault); those on the host are refused."""
    from nanoengine_b200.ops import sm100, sm100_attn
    t, more, h, dim = 150, 300, 4, 72
    q, k, v = (torch.randn(more, h, dim, device="cuda").to(torch.bfloat16) for _ in "qkv")
    p = lambda x: x.data_ptr()             # noqa: E731
    for causal in (0, 1):
        out = torch.full((more, h, dim), 5.0, dtype=torch.bfloat16, device="cuda")
        cu = torch.tensor([0, 100, 290], dtype=torch.int32, device="cuda")
        assert sm100_attn._fmha_call()(p(q), q.stride(0), p(k), k.stride(0), dim, 0, 0, p(v), v.stride(0), t, 0, 0, p(cu), 0, 2, t, h, h, dim, dim, 1, 4, 1, 0, causal, 0.1, 1, p(out), 0, 0,
                                       torch.cuda.current_stream().cuda_stream) == 0
        assert (out[t:] == 5.0).all()
        cu[2] = t
        assert torch.equal(out[:t], sm100.attention_varlen(q[:t], k[:t], v[:t], cu, 0.1, bool(causal)))
    for cu in (torch.tensor([0, t], dtype=torch.int32), torch.tensor([0], dtype=torch.int32, device="cuda")):
        with pytest.raises(AssertionError):
            sm100.attention_varlen(q[:t], k[:t], v[:t], cu, 0.1)


def test_a_prompt_alone_and_in_a_batch():
    """Alone its tiles do not fill the SMs and the decode steps' kernel takes it, in a batch the prompt kernel does.  Both round the same probabilities to bf16 and sum
    them in 32 bits, in another order: a few 2^-24 apart before the results are rounded to bf16, so some of them one step (2^-7 of a value at most) apart, few."""
    from nanoengine_b200.ops import sm100_attn
    g = torch.Generator(device="cuda").manual_seed(14)
    n, hq, hkv = sm100_attn._sms() * 8 // 6, 64, 4             # 8 tokens a tile: two thirds of a wave, twice that in the batch
    nb = -(-n // 64)
    kc, vc = (torch.randn(2 * nb, 64, hkv, 128, generator=g, device="cuda").to(torch.bfloat16) for _ in "kv")
    q = torch.randn(2 * n, hq, 128, generator=g, device="cuda").to(torch.bfloat16)
    bt = torch.arange(2 * nb, dtype=torch.int32, device="cuda").view(2, nb)
    cu, cl = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0, n, 2 * n], [n, n]))
    calls = sm100_attn.PROMPT_TC_CALLS[0]
    alone = sm100_attn.gqa_attention_paged(q[:n], kc, vc, bt[:1], cu[:2], cl[:1], 128 ** -0.5)
    assert sm100_attn.PROMPT_TC_CALLS[0] == calls
    both = sm100_attn.gqa_attention_paged(q, kc, vc, bt, cu, cl, 128 ** -0.5)[:n]
    assert sm100_attn.PROMPT_TC_CALLS[0] == calls + 1
    diff = (alone.double() - both.double()).abs()
    assert (diff <= 2 ** -7 * torch.maximum(alone.abs(), both.abs()).double()).all() and (diff > 0).double().mean() < 0.01
