"""The delta rule over prompts, chunked or in groups of four tokens, in 32-bit, against the recurrence in 64 bits: chunk edges, portions of every length beside short ones, carried and fresh states,
decays from none to complete, strided rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu

D = 128
# an operand of a product is kept to 2^-25 and sums are 32-bit: a few 2^-24 (6e-8) of the state's size; a log decay g is 32-bit, which moves its factor by
# |g| 2^-23 at most, and a factor counts where |g| is a few.  Results are bf16, with roundings between norm and gate.
STATE, OUT = 2e-6, 5e-3


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm().clamp_min(1e-30)).item()


def _oracle(q, k, v, g, beta, state, fresh, lens, slots):
    """q, k [T, H, D] unit vectors; g [T, H] or [T, H, D] log decays; all in 64 bits.  Returns outputs and final states."""
    outs, at = [], 0
    state = state.double().clone()
    for i, n in enumerate(lens):
        s = torch.zeros_like(state[0]) if fresh[i] else state[slots[i]].clone()
        for t in range(at, at + n):
            d = g[t].exp()
            s = s * (d[:, None, :] if d.dim() == 2 else d[:, None, None])
            u = beta[t][:, None] * (v[t] - torch.einsum("hvk,hk->hv", s, k[t]))
            s = s + u[:, :, None] * k[t][:, None, :]
            outs.append(torch.einsum("hvk,hk->hv", s, q[t]))
        if n:
            state[slots[i]] = s
        at += n
    return torch.stack(outs), state


def _inputs(lens, hk, hv, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    t = sum(lens)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")             # noqa: E731
    y = r(t, (2 * hk + hv) * D).to(torch.bfloat16)
    q, k, v = y[:, : hk * D].view(t, hk, D), y[:, hk * D: 2 * hk * D].view(t, hk, D), y[:, 2 * hk * D:].view(t, hv, D)
    state = r(len(lens) + 1, hv, D, D) * 0.2
    slots = torch.randperm(len(lens) + 1, generator=gen, device="cuda")[: len(lens)].int()
    fresh = (torch.arange(len(lens), device="cuda") % 2 == 1).int()
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()
    z, w = r(t, hv, D).to(torch.bfloat16), (1 + 0.1 * r(D)).to(torch.bfloat16)
    return gen, r, q, k, v, state, slots, fresh, cu, z, w


def _unit(x, rep, scale=1.0):
    x = x.double()
    return (x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6)).repeat_interleave(rep, 1) * scale


@pytest.mark.parametrize("hk,hv", [(1, 1), (2, 4), (3, 3)])
@pytest.mark.parametrize("lens", [[64], [65, 3, 128], [127, 1, 0, 64, 200], [16, 700], [63, 5, 17, 16]])
@pytest.mark.parametrize("decay", [0.001, 0.3, 40.0])
def test_decay_per_head(hk, hv, lens, decay):
    from nanoengine_b200.ops import sm100
    gen, r, q, k, v, state, slots, fresh, cu, z, w = _inputs(lens, hk, hv, 5)
    t = sum(lens)
    ab = r(t, 2 * hv).to(torch.bfloat16)
    a, b = ab[:, :hv], ab[:, hv:]
    A, bias = torch.full((hv,), decay, device="cuda").log(), torch.zeros(hv, device="cuda")
    g = -A.double().exp() * torch.nn.functional.softplus(a.double() + bias.double())
    want, want_state = _oracle(_unit(q, hv // hk, D ** -0.5), _unit(k, hv // hk), v.double(), g, torch.sigmoid(b.double()), state, fresh.tolist(), lens, slots.tolist())
    sm100.clear_kernel_status()
    got = sm100.gdn_recurrent(q, k, v, a, b, A, bias, state, slots, torch.tensor(cu, dtype=torch.int32, device="cuda"), fresh, z, w, 1e-6, max(lens), cu)
    zd = z.double()
    want = want * torch.rsqrt(want.square().mean(-1, keepdim=True) + 1e-6) * w.double() * zd * torch.sigmoid(zd)
    assert sm100.kernel_status()[0] == 0
    assert _rel(got.view(t, hv, D), want) < OUT
    long = [s for s, n in zip(slots.tolist(), lens) if n >= 64 or min(lens) > 4]         # the others one token at a time
    assert _rel(state[long], want_state[long]) < STATE
    rest = [s for s in range(state.shape[0]) if s not in long]
    assert _rel(state[rest], want_state[rest]) < 1e-5


@pytest.mark.parametrize("heads", [1, 3])
@pytest.mark.parametrize("lens", [[5], [16, 17, 1, 0, 33], [1, 300], [15, 48] * 40])
@pytest.mark.parametrize("bound,scale", [(-5.0, 0.5), (None, 0.05), (-0.01, 1.0), (None, 30.0)])
def test_decay_per_channel(heads, lens, bound, scale):
    from nanoengine_b200.ops import sm100
    gen, r, q, k, v, state, slots, fresh, cu, z, w = _inputs(lens, heads, heads, 6)
    t = sum(lens)
    a, b = r(t, heads * D).to(torch.bfloat16), r(t, heads).to(torch.bfloat16)
    A, bias = torch.full((heads,), scale, device="cuda").log(), r(heads * D)
    x = a.double().view(t, heads, D) + bias.double().view(1, heads, D)
    e = A.double().exp()[None, :, None]
    g = bound * torch.sigmoid(e * x) if bound is not None else -e * torch.nn.functional.softplus(x)
    want, want_state = _oracle(_unit(q, 1, D ** -0.5), _unit(k, 1), v.double(), g, torch.sigmoid(b.double()), state, fresh.tolist(), lens, slots.tolist())
    sm100.clear_kernel_status()
    got = sm100.kda_recurrent(q, k, v, a, b, A, bias, bound, state, slots, torch.tensor(cu, dtype=torch.int32, device="cuda"), fresh, z, w, 1e-6)
    want = want * torch.rsqrt(want.square().mean(-1, keepdim=True) + 1e-6) * w.double() * torch.sigmoid(z.double())
    assert sm100.kernel_status()[0] == 0
    assert _rel(got.view(t, heads, D), want) < OUT and _rel(state, want_state) < STATE


@pytest.mark.parametrize("lens", [[64], [200, 64, 5, 129]])
@pytest.mark.parametrize("alike", [0.0, 0.99])
def test_outputs_in_front_of_the_norm_are_32_bit(lens, alike, monkeypatch):
    """`alike`: every key is mostly the same vector, where the inverse of a chunk's system has the largest entries (its products of two rows are 0.98, its decay 0.999)."""
    from nanoengine_b200.ops import sm100
    hk, hv = 2, 4
    gen, r, q, k, v, state, slots, fresh, cu, z, w = _inputs(lens, hk, hv, 9)
    t = sum(lens)
    k.copy_((alike * r(1, hk, D) + (1 - alike ** 2) ** 0.5 * r(t, hk, D)).to(torch.bfloat16))
    a, b = r(t, 2 * hv).to(torch.bfloat16).split(hv, 1)
    A, bias = torch.full((hv,), 0.001, device="cuda").log(), torch.zeros(hv, device="cuda")
    g = -A.double().exp() * torch.nn.functional.softplus(a.double() + bias.double())
    want, want_state = _oracle(_unit(q, hv // hk, D ** -0.5), _unit(k, hv // hk), v.double(), g, torch.sigmoid(b.double()), state, fresh.tolist(), lens, slots.tolist())
    seen, norm = [], sm100.rmsnorm_gated
    monkeypatch.setattr(sm100, "rmsnorm_gated", lambda x, *rest: (seen.append(x.clone()), norm(x, *rest))[1])
    sm100.gdn_recurrent(q, k, v, a, b, A, bias, state, slots, torch.tensor(cu, dtype=torch.int32, device="cuda"), fresh, z, w, 1e-6, max(lens), cu)
    assert len(seen) == 1 and _rel(seen[0], want) < STATE and _rel(state, want_state) < STATE


@pytest.mark.parametrize("what", ["v", "k", "q", "gate", "beta"])
@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("at", range(8, 13))
def test_a_token_that_is_no_number_leaves_the_earlier_ones_alone(per_channel, what, at):
    from nanoengine_b200.ops import sm100
    heads, lens = 2, [at + 1 if at == 12 else 15, 9]
    gen, r, q, k, v, state, slots, fresh, cu, z, w = _inputs(lens, heads, heads, 10)
    t = sum(lens)
    a, b = r(t, heads * (D if per_channel else 1)).to(torch.bfloat16), r(t, heads).to(torch.bfloat16)
    A, bias = torch.zeros(heads, device="cuda"), torch.zeros(heads * (D if per_channel else 1), device="cuda")
    cu = torch.tensor(cu, dtype=torch.int32, device="cuda")

    def run(st):
        if per_channel:
            return sm100.kda_recurrent(q, k, v, a, b, A, bias, None, st, slots, cu, fresh, z, w, 1e-6).view(t, heads, D)
        return sm100.gdn_recurrent(q, k, v, a, b, A, bias, st, slots, cu, fresh, z, w, 1e-6, max(lens)).view(t, heads, D)

    st, clean = state.clone(), run(clean_state := state.clone())
    {"v": v, "k": k, "q": q, "gate": a.view(t, heads, -1), "beta": b.view(t, heads, 1)}[what][at, 1] = float("nan")
    got = run(st)
    hit = torch.zeros(t, heads, dtype=torch.bool, device="cuda")
    hit[at: at + 1 if what == "q" else lens[0], 1] = True                 # a query is its token's alone, the others stay in the state
    assert got[hit].isnan().all() and torch.equal(got[~hit], clean[~hit])
    assert torch.equal(st[slots[1].long()], clean_state[slots[1].long()]) and torch.equal(st[slots[0].long(), 0], clean_state[slots[0].long(), 0])


@pytest.mark.parametrize("per_channel", [False, True])
def test_an_infinite_state_row_is_not_worked_on_behind_the_end(per_channel):
    from nanoengine_b200.ops import sm100
    heads, n = 1, 9
    gen, r, q, k, v, state, slots, fresh, cu, z, w = _inputs([n], heads, heads, 11)
    a, b = r(n, heads * (D if per_channel else 1)).to(torch.bfloat16), r(n, heads).to(torch.bfloat16)
    A, bias = torch.zeros(heads, device="cuda"), torch.zeros(heads * (D if per_channel else 1), device="cuda")
    v[n - 1, 0, 5] = float("inf")                                         # the last token's write: its row of the state is infinite, of the signs of its key
    cu = torch.tensor(cu, dtype=torch.int32, device="cuda")
    if per_channel:
        sm100.kda_recurrent(q, k, v, a, b, A, bias, None, state, slots, cu, fresh, z, w, 1e-6)
    else:
        sm100.gdn_recurrent(q, k, v, a, b, A, bias, state, slots, cu, fresh, z, w, 1e-6, n)
    row = state[slots[0].long(), 0, 5]
    assert torch.equal(row, torch.where(k[n - 1, 0] > 0, float("inf"), float("-inf")))
    assert state[slots[0].long(), 0, :5].isfinite().all() and state[slots[0].long(), 0, 6:].isfinite().all()


@pytest.mark.parametrize("lens", [[2, 3], [9, 30], [70, 3, 129], [200]])
def test_strided_gates_and_tables(lens):
    from nanoengine_b200.ops import sm100
    hk, hv = 1, 2
    gen, r, q, k, v, state, slots, fresh, cu, z, w = _inputs(lens, hk, hv, 12)
    t, n = sum(lens), len(lens)
    ab = r(t, hv, 2).to(torch.bfloat16)
    A, bias, w2 = r(hv, 3) * 0.3, r(hv, 3), torch.stack([w, -w], 1)
    table = torch.stack([slots, fresh, torch.tensor(cu[1:], dtype=torch.int32, device="cuda")], 1)         # a row per sequence
    ends = torch.stack([torch.tensor(cu, dtype=torch.int32, device="cuda"), torch.zeros(n + 1, dtype=torch.int32, device="cuda")], 1)
    one, two = state.clone(), state.clone()
    want = sm100.gdn_recurrent(q, k, v, ab[..., 0].contiguous(), ab[..., 1].contiguous(), A[:, 1].contiguous(), bias[:, 2].contiguous(), one, slots, ends[:, 0].contiguous(), fresh, z, w,
                               1e-6, max(lens), cu)
    got = sm100.gdn_recurrent(q, k, v, ab[..., 0], ab[..., 1], A[:, 1], bias[:, 2], two, table[:, 0], ends[:, 0], table[:, 1], z, w2[:, 0], 1e-6, max(lens), cu)
    assert torch.equal(got, want) and torch.equal(one, two)


@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("n", [2, 4, 5, 30, 64, 130])
@pytest.mark.parametrize("others", [[1] * 40, [1] * 30 + [7] * 50, [100, 1]])
def test_a_sequence_does_not_depend_on_its_batch(per_channel, n, others):
    """Bit for bit: which form the rule takes, and in which order it sums, is a matter of the sequence's own length."""
    from nanoengine_b200.ops import sm100
    hk, hv, at = (2, 2, len(others) // 2) if per_channel else (2, 4, len(others) // 2)
    lens = others[:at] + [n] + others[at:]
    gen, r, q, k, v, state, slots, fresh, cu, z, w = _inputs(lens, hk, hv, 13)
    t, fresh = sum(lens), torch.zeros_like(fresh)
    a, b = r(t, hv * (D if per_channel else 1)).to(torch.bfloat16), r(t, hv).to(torch.bfloat16)
    A, bias = torch.zeros(hv, device="cuda"), torch.zeros(hv * (D if per_channel else 1), device="cuda")

    def run(rows, lens, st, sl, fr, host):
        ends = [0] + torch.tensor(lens).cumsum(0).tolist()
        x, c = [i[rows] for i in (q, k, v, a, b)], torch.tensor(ends, dtype=torch.int32, device="cuda")
        if per_channel:
            return sm100.kda_recurrent(*x, A, bias, -5.0, st, sl, c, fr, z[rows], w, 1e-6)
        return sm100.gdn_recurrent(*x, A, bias, st, sl, c, fr, z[rows], w, 1e-6, max(lens), ends if host or max(lens) >= 64 else None)

    for host in (False, True):
        one, all_ = state.clone(), state.clone()
        own = slice(cu[at], cu[at + 1])
        alone = run(own, [n], one, slots[at: at + 1], fresh[at: at + 1], host)
        batch = run(slice(0, t), lens, all_, slots, fresh, host)
        assert torch.equal(batch[own], alone) and torch.equal(all_[slots[at].long()], one[slots[at].long()])


@pytest.mark.parametrize("first,then", [([7, 9, 20], [1, 3, 32]), ([2, 3, 4, 6], [1, 12, 1, 1]), ([70, 40], [75, 35]), ([100, 1, 9], [66, 40, 4])])
def test_a_captured_call_follows_the_boundaries_on_the_device(first, then):
    from nanoengine_b200.ops import sm100
    hk, hv = 1, 2
    gen, r, q, k, v, state, slots, fresh, cu, z, w = _inputs(first, hk, hv, 15)
    t, longest = sum(first), max(*first, *then)
    a, b = r(t, 2 * hv).to(torch.bfloat16).split(hv, 1)
    A, bias = torch.zeros(hv, device="cuda"), torch.zeros(hv, device="cuda")
    ends = torch.tensor(cu, dtype=torch.int32, device="cuda")
    st = state.clone()
    run = lambda st, ends, host: sm100.gdn_recurrent(q, k, v, a, b, A, bias, st, slots, ends, fresh, z, w, 1e-6, longest, host)             # noqa: E731
    run(state.clone(), ends, cu)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run(st, ends, cu)
    other = [0] + torch.tensor(then).cumsum(0).tolist()
    ends.copy_(torch.tensor(other, dtype=torch.int32))
    st.copy_(state)
    graph.replay()
    want_state = state.clone()
    want = run(want_state, torch.tensor(other, dtype=torch.int32, device="cuda"), other)
    assert torch.equal(got, want) and torch.equal(st, want_state)
