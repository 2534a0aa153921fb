"""The scan of prompt portions sixteen tokens at a time, and of single tokens with a head's state in one CTA, against the
token-by-token kernel and 64-bit arithmetic."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _reference(q, k, v, lens, state, slots, *, decay, gain, beta):
    """The recurrence in 64 bits: q, k [N, H, d], v [N, H, dv], decay [N, H, d], gain [N, H] or None, beta [N, H] or None."""

    out, end = torch.empty_like(v), state.clone()
    first = 0
    for n, slot in zip(lens, slots):
        S = end[slot]
        for t in range(first, first + n):
            S = decay[t][..., None] * S
            u = v[t] if gain is None else gain[t][:, None] * v[t]
            if beta is not None:
                u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            out[t] = torch.einsum("hdv,hd->hv", S, q[t])
        end[slot] = S
        first += n
    return out, end


MIXED = [1, 1, 1, 130, 20, 200]         # single tokens, long and short portions: a kernel for each run of them
FORMS = ["head", "head_float_qk", "channel", "row", "delta_channel", "delta_token"]


# portions around a chunk's edges, key sizes that fill 2, 4 and 8 warps and none, value columns around a block of 32; single tokens
# with value columns below, at and above the 128 that a CTA holds; as many tokens as requests, but not one each
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("heads,qk_heads,d,dv,lens", [(2, 2, 128, 128, [257]), (4, 2, 40, 33, [1, 15, 16, 17, 64]), (3, 3, 16, 8, [100, 31]),
                                                      (1, 1, 72, 64, [49, 1]),
                                                      (4, 2, 128, 128, [1] * 5), (3, 3, 40, 36, [1]), (2, 1, 17, 132, [1, 1]),
                                                      (2, 2, 128, 128, [2, 0]), (4, 2, 40, 36, [0, 3, 0]), (2, 1, 17, 132, [1, 0, 0, 3]),
                                                      (2, 2, 128, 64, MIXED), (3, 1, 40, 33, MIXED)])
def test_chunks_against_the_recurrence(form, heads, qk_heads, d, dv, lens, monkeypatch):
    from llm_runtime_study_b200.ops import sequence_state as S

    if form == "row":
        qk_heads = heads
    g = torch.Generator().manual_seed(len(form) + d)
    n, slots = sum(lens), [2 * i + 1 for i in range(len(lens))]
    delta = form.startswith("delta")
    narrow = torch.float32 if delta or form == "head_float_qk" else torch.bfloat16
    q, k = (torch.randn(n, qk_heads * d, generator=g).to(narrow) for _ in range(2))
    v = torch.randn(n, heads * dv, generator=g).to(torch.float32 if delta else torch.bfloat16)
    if delta:
        q, k = (torch.nn.functional.normalize(x.view(n, qk_heads, d), dim=-1).reshape(n, -1) for x in (q, k))
    state = 0.3 * torch.randn(2 * len(lens) + 2, heads, d, dv, generator=g)
    norm_state = 0.3 * torch.randn(2 * len(lens) + 2, heads, d, generator=g)
    options, gain, beta = {}, None, None
    if form.startswith("head"):
        decay = torch.linspace(0.7, 1.0, heads)
        options["decay"] = decay
        wide = decay[None, :, None].expand(n, heads, d)
    elif form in ("channel", "delta_channel"):
        gate = torch.sigmoid(3.0 * torch.randn(n, heads, d, generator=g) + 2.0)
        gate[n // 2] *= 1e-30                        # a decay that empties the state, as strong gates do
        options["gate"] = gate.reshape(n, -1)
        wide = gate
    else:
        token = torch.sigmoid(torch.randn(n, heads, generator=g) + 2.0)
        options["row_decay" if delta else "decay"] = token
        wide = token[..., None].expand(n, heads, d)
        if form == "row":
            gain = torch.rand(n, heads, generator=g)
            options["gain"] = gain
    if delta:
        beta = torch.sigmoid(torch.randn(n, heads, generator=g))
        options["beta"] = beta
    q_start = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
    dev = lambda x: x.to(DEV)

    def run(fixed_order):
        s, ns = dev(state), dev(norm_state)
        common = dict(heads=heads, dim=d, vdim=dv, state=s, q_start=q_start, slots=torch.tensor(slots, dtype=torch.int32, device=DEV),
                      fixed_order=fixed_order, q_scale=0.5, lens=lens, **{key: dev(x) for key, x in options.items()})
        # rows of a wider projection: strides of their own
        rows = [dev(torch.cat((x, x), dim=1))[:, : x.shape[1]] for x in (q, k, v)]
        if form == "row":
            out, norm_out = S.linear_scan_row_gates(*rows, norm_state=ns, **common)
            return out, s, norm_out, ns
        return S.linear_scan(*rows, qk_heads=qk_heads, silu=form == "head", **common), s, None, None

    act = (lambda x: x * torch.sigmoid(x)) if form == "head" else (lambda x: x)
    group = heads // qk_heads
    wq, wk = (act(x.double()).view(n, qk_heads, d).repeat_interleave(group, dim=1) for x in (q, k))
    wv = act(v.double()).view(n, heads, dv)
    wide = wide.double()
    want, end = _reference(0.5 * wq, wk, wv, lens, state.double(), slots, decay=wide, gain=None if gain is None else gain.double(),
                           beta=None if beta is None else beta.double())
    if lens != MIXED:                        # every portion in chunks, short ones too
        monkeypatch.setattr(S, "portion_in_chunks", lambda *sizes: 1)
    else:
        runs = S.scan_runs(lens, S.portion_in_chunks(lens, heads, d, dv, delta))
        assert [kind for kind, _, _ in runs] == ["single", "chunks", "chain", "chunks"]
    chunked, chained = run(False), run(True)

    def error(got, ref):
        return float((got.double().cpu() - ref).norm() / ref.norm())

    pairs = [(0, want.reshape(n, -1)), (1, end)]
    if form == "row":
        ones = torch.ones(n, heads, 1, dtype=torch.float64)
        nwant, nend = _reference(0.5 * wq, wk, ones, lens, norm_state.double()[..., None], slots, decay=wide, gain=gain.double(), beta=None)
        pairs += [(2, nwant[..., 0]), (3, nend[..., 0])]
    for i, ref in pairs:
        # products of up to 16 decays and sums of up to 16 + 128 terms, a rounding of 6e-8 each, sizes adding up like their roots; SiLU
        # of 16-bit rows takes the hardware's exponential (2 units in the last place), in either kernel
        assert error(chunked[i], ref) < 2e-6, (i, error(chunked[i], ref), error(chained[i], ref))
        assert error(chunked[i], ref) < 1.5 * error(chained[i], ref) + 1e-7


@pytest.mark.parametrize("form", ["row", "delta"])
@pytest.mark.parametrize("known", [True, False])
def test_records_in_slices_give_the_same_bits(form, known, monkeypatch):
    """Portions whose records do not fit at once, in launches that follow each other: the state goes through the request's slot as the
    same float32 numbers, so nothing changes.  Portions that end inside a slice, at its end and behind it, empty ones among them."""

    from llm_runtime_study_b200.ops import sequence_state as S

    heads, d, dv, lens = 2, 40, 33, [130, 64, 63, 65] if known else [130, 64, 0, 63, 65]
    n, entries = sum(lens), len(lens)
    g = torch.Generator().manual_seed(3)
    rand = lambda *shape: torch.rand(*shape, generator=g).to(DEV)
    q, k, v = (rand(n, heads * w) - 0.5 for w in (d, d, dv))
    token, other, state, norm_state = rand(n, heads), rand(n, heads), rand(entries, heads, d, dv), rand(entries, heads, d)
    q_start = torch.tensor([sum(lens[:i]) for i in range(entries + 1)], dtype=torch.int32, device=DEV)
    common = dict(heads=heads, dim=d, vdim=dv, q_start=q_start, slots=torch.arange(entries, dtype=torch.int32, device=DEV),
                  lens=lens if known else None)
    monkeypatch.setattr(S, "portion_in_chunks", lambda *sizes: 1)

    def run():
        s, ns = state.clone(), norm_state.clone()
        if form == "row":
            return *S.linear_scan_row_gates(*(x.bfloat16() for x in (q, k, v)), decay=token, gain=other, state=s, norm_state=ns, **common), s, ns
        return S.linear_scan(q, k, v, qk_heads=heads, row_decay=token, beta=other, state=s, **common), s

    whole = run()
    for slice_bytes in (1, 1 << 18):         # a chunk of every request a launch; about two
        monkeypatch.setattr(S, "CHUNK_SLICE_BYTES", slice_bytes)
        for a, b in zip(run(), whole):
            assert torch.equal(a, b)


def test_the_normalised_read_out_of_every_token():
    """The matrix memory's read-out over its normaliser, token by token: a token whose normaliser cancels weighs as much as any other.
    Either sum is off by at most a few float32 roundings of its terms' absolute values (16-bit q, k, v; products of up to 300 decays), and the
    chunks are no further off than the chain."""

    from llm_runtime_study_b200.ops import sequence_state as S

    n, heads, d, dv = 300, 3, 128, 64
    g = torch.Generator().manual_seed(11)
    q, k, v = (torch.randn(n, heads, w, generator=g).bfloat16() for w in (d, d, dv))
    decay, gain = torch.sigmoid(torch.randn(n, heads, generator=g) + 3.0), torch.rand(n, heads, generator=g)
    dev = lambda x: x.to(DEV).reshape(n, -1)
    q_start = torch.tensor([0, n], dtype=torch.int32, device=DEV)

    def run(fixed_order):
        return S.linear_scan_row_gates(dev(q), dev(k), dev(v), heads=heads, dim=d, vdim=dv, decay=dev(decay), gain=dev(gain),
                                       state=torch.zeros(1, heads, d, dv, device=DEV), norm_state=torch.zeros(1, heads, d, device=DEV),
                                       q_start=q_start, slots=torch.zeros(1, dtype=torch.int32, device=DEV), fixed_order=fixed_order, lens=[n])

    def reference(q, k, v):
        wide = decay.double()[..., None].expand(n, heads, d)
        ones = torch.ones(n, heads, 1, dtype=torch.float64)
        sums = [_reference(q, k, x, [n], torch.zeros(1, heads, d, x.shape[2], dtype=torch.float64), [0], decay=wide, gain=gain.double(), beta=None)[0]
                for x in (v, ones)]
        return sums[0], sums[1][..., 0]

    (out, den), (size, den_size) = (reference(*(f(x.double()) for x in (q, k, v))) for f in (lambda x: x, torch.abs))
    assert float((den.abs() / den_size).min()) < 1e-3             # some normalisers all but vanish
    worst = []
    for fixed in (False, True):
        got, got_den = (x.double().cpu() for x in run(fixed))
        off = ((got.view(n, heads, dv) - out).abs() / size).amax(), ((got_den - den).abs() / den_size).amax()
        ratio, want = got.view(n, heads, dv) / got_den[..., None], out / den[..., None]
        # the ratio's error in units of what the two sums' roundings make of it
        scale = (size + want.abs() * den_size[..., None]) / den.abs()[..., None]
        worst.append(max(*map(float, off), float(((ratio - want).abs() / scale).amax())))
    # a decay's product over 300 tokens is off by 300 roundings at most, the terms that count by those of the last few dozen tokens
    assert worst[0] < 5e-6 and worst[0] < 2 * worst[1], worst


def test_as_many_rows_as_requests_are_single_tokens_only_when_the_lengths_say_so():
    """Without lengths any cut of ``q_start`` is served, empty requests included; lengths that do not fit are refused."""

    from llm_runtime_study_b200.errors import KernelError
    from llm_runtime_study_b200.ops import sequence_state as S

    heads, d = 2, 32
    g = torch.Generator().manual_seed(3)
    q, k, v = (torch.randn(3, heads * d, generator=g).bfloat16() for _ in range(3))
    begin = 0.3 * torch.randn(3, heads, d, d, generator=g)
    decay = torch.tensor([0.9, 0.8])
    for lens in ([0, 2, 1], [3, 0, 0], [1, 1, 1]):
        state = begin.to(DEV)
        first = [sum(lens[:i]) for i in range(4)]
        args = dict(heads=heads, qk_heads=heads, dim=d, vdim=d, q_start=torch.tensor(first, dtype=torch.int32, device=DEV),
                    slots=torch.arange(3, dtype=torch.int32, device=DEV), decay=decay.to(DEV))
        out = S.linear_scan(q.to(DEV), k.to(DEV), v.to(DEV), state=state, **args)
        rows = [x.double().view(3, heads, d) for x in (q, k, v)]
        want, end = _reference(*rows, lens, begin.double(), range(3), decay=decay.double()[None, :, None].expand(3, heads, d), gain=None, beta=None)
        assert float((out.double().cpu() - want.reshape(3, -1)).norm() / want.norm()) < 1e-6       # a few float32 roundings
        assert float((state.double().cpu() - end).norm() / end.norm()) < 1e-6
        with pytest.raises(KernelError, match="lengths"):
            S.linear_scan(q.to(DEV), k.to(DEV), v.to(DEV), state=state, lens=lens[:2], **args)


def test_a_bad_row_reaches_later_tokens_only():
    from llm_runtime_study_b200.ops import sequence_state as S

    n, heads, d = 64, 2, 32
    g = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(n, heads * d, generator=g).bfloat16().to(DEV) for _ in range(3))
    v[37], k[41] = float("nan"), float("inf")
    out = S.linear_scan(q, k, v, heads=heads, qk_heads=heads, dim=d, vdim=d, state=torch.zeros(1, heads, d, d, device=DEV),
                        q_start=torch.tensor([0, n], dtype=torch.int32, device=DEV), slots=torch.zeros(1, dtype=torch.int32, device=DEV),
                        decay=torch.full((heads,), 0.9, device=DEV))
    assert bool(torch.isfinite(out[:37]).all()) and not bool(torch.isfinite(out[37:]).any())


@pytest.mark.parametrize("form", ["delta", "row"])
def test_a_bad_value_in_a_chunk_reaches_its_own_column_and_later_tokens_only(form):
    """Value columns of two warps' tiles and more; tokens of a chunk before the bad one, which share its products on the tensor cores."""

    from llm_runtime_study_b200.ops import sequence_state as S

    n, heads, d, dv, bad = 80, 2, 48, 40, 37
    g = torch.Generator().manual_seed(2)
    q, k, v = (torch.randn(n, heads * w, generator=g) for w in (d, d, dv))
    v[bad, dv + 5] = float("nan")                                    # the second head's
    common = dict(heads=heads, dim=d, vdim=dv, state=torch.zeros(1, heads, d, dv, device=DEV), lens=[n],
                  q_start=torch.tensor([0, n], dtype=torch.int32, device=DEV), slots=torch.zeros(1, dtype=torch.int32, device=DEV))
    token = torch.rand(n, heads, generator=g).to(DEV)
    if form == "delta":
        out = S.linear_scan(q.to(DEV), (k / d ** 0.5).to(DEV), v.to(DEV), qk_heads=heads, row_decay=token, beta=token, **common)
    else:
        rows = (x.bfloat16().to(DEV) for x in (q, k, v))
        out, den = S.linear_scan_row_gates(*rows, decay=token, gain=token, norm_state=torch.zeros(1, heads, d, device=DEV), **common)
        assert bool(torch.isfinite(den).all())
    fine = torch.isfinite(out).view(n, heads, dv)
    want = torch.ones(n, heads, dv, dtype=torch.bool)
    want[bad:, 1, 5] = False
    assert torch.equal(fine.cpu(), want)


def _positive_case(form, heads, d, dv, n):
    """Positive numbers throughout, so that an infinity adds up to an infinity and never to NaN: (rows q, k, v, state, norm_state, options, decay [n,
    heads, d], gain or beta [n, heads])."""

    g = torch.Generator().manual_seed(7)
    rand = lambda *shape: 0.1 + 0.8 * torch.rand(*shape, generator=g)
    delta = form.startswith("delta")
    narrow = torch.float32 if delta or form == "head_float_qk" else torch.bfloat16
    q, k = (rand(n, heads * d) for _ in range(2))
    if delta:                                # rows of length one: the recurrence does not grow
        q, k = (torch.nn.functional.normalize(x.view(n, heads, d), dim=-1).reshape(n, -1) for x in (q, k))
    q, k, v = q.to(narrow), k.to(narrow), rand(n, heads * dv).to(torch.float32 if delta else torch.bfloat16)
    head, channel, token, other = rand(heads), rand(n, heads, d), rand(n, heads), rand(n, heads)
    options, wide = {"head": ({"decay": head}, head[None, :, None].expand(n, heads, d)), "channel": ({"gate": channel.reshape(n, -1)}, channel),
                     "token": ({"row_decay": token}, token[..., None].expand(n, heads, d)), "row": ({"decay": token, "gain": other}, token[..., None].expand(n, heads, d)),
                     }[form.split("_")[1] if delta else form.split("_")[0]]
    if delta:
        options["beta"] = other
    return q, k, v, rand(1, heads, d, dv), rand(1, heads, d), options, wide, other


# an infinity, and a number beyond bfloat16's largest (which rounds to an infinity), where a chunk meets them: in a value, a key, a query, the state
# it starts from; the bad token in the first chunk and in a later one, tokens of its chunk before and behind it
@pytest.mark.parametrize("where", ["v", "k", "q", "state", "large state", "large v", "large k"])
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("d,dv,n,bad", [(48, 40, 40, 5), (128, 33, 52, 37), (24, 32, 16, 9)])
def test_infinities_and_the_largest_numbers_keep_their_value(form, where, d, dv, n, bad, monkeypatch):
    from llm_runtime_study_b200.ops import sequence_state as S

    heads, huge, delta = 2, 3.395e38, form.startswith("delta")
    q, k, v, state, norm_state, options, wide, other = _positive_case(form, heads, d, dv, n)
    if delta and where in ("k", "q", "state", "large k"):
        pytest.skip("the delta rule subtracts: no sign of its infinities is the same in every order of its sums")
    if where in ("large v", "large k") and {"large v": v, "large k": k}[where].dtype != torch.float32:
        pytest.skip("16-bit rows hold no such number")
    if delta and where == "v":
        bad = n - 1                          # (the tokens behind it would subtract infinities)
    if where in ("v", "k", "q"):
        {"v": v, "k": k, "q": q}[where][bad, 3] = float("inf")
    elif where == "state":
        state[0, 0, 7, 3] = float("inf")
    elif where == "large state":
        state[0, 0, 7, 3] = huge
        q *= 0.25                            # (the read-outs stay finite)
    else:
        {"large v": v, "large k": k}[where][bad, 3] = huge
        q, k, v = q * 0.125, (k if where == "large k" else k * 0.25), (v if where == "large v" else v * 0.25)
    monkeypatch.setattr(S, "portion_in_chunks", lambda *sizes: 1)
    monkeypatch.setattr(S, "CHUNK_MIN_TOKENS", 1)
    dev = lambda x: x.to(DEV)
    s, ns = dev(state), dev(norm_state)
    common = dict(heads=heads, dim=d, vdim=dv, state=s, q_start=torch.tensor([0, n], dtype=torch.int32, device=DEV), lens=[n],
                  slots=torch.zeros(1, dtype=torch.int32, device=DEV), **{key: dev(x) for key, x in options.items()})
    if form == "row":
        out, den = S.linear_scan_row_gates(dev(q), dev(k), dev(v), norm_state=ns, **common)
    else:
        out = S.linear_scan(dev(q), dev(k), dev(v), qk_heads=heads, **common)
    rows = [x.double().view(n, heads, -1) for x in (q, k, v)]
    more = dict(decay=wide.double(), gain=other.double() if form == "row" else None, beta=other.double() if delta else None)
    want, end = _reference(*rows, [n], state.double(), [0], **more)
    pairs = [(out.view(n, heads, dv), want), (s, end)]
    if form == "row":
        nwant, nend = _reference(rows[0], rows[1], torch.ones(n, heads, 1, dtype=torch.float64), [n], norm_state.double()[..., None], [0], **more)
        pairs += [(den, nwant[..., 0]), (ns, nend[..., 0])]
    for got, ref in pairs:
        got, ref = got.double().cpu(), ref.double()
        assert not bool(ref.isnan().any()) and torch.equal(got.isinf() * got.sign(), ref.isinf() * ref.sign())
        fine = ref.isfinite()
        assert bool(fine.any())
        # sums of up to 16 + 128 terms of one sign (the delta rule's: their largest counts), a float32 rounding each
        scale = ref[fine].abs() if not delta else ref[fine].abs() + float(ref[fine].abs().max())
        assert bool(((got[fine] - ref[fine]).abs() <= 1e-5 * scale).all())
