"""Kernels that prepare or finish rows of mixers, at the edges of what their vectors, warps and tiles of tokens hold, against
64-bit arithmetic."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ints(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def close(got, want, tol):
    """``tol`` of the largest value: roundings of sums and functions whose inputs are of that size."""

    got, want = got.double().cpu(), want.double()
    assert bool(torch.isfinite(got).all())
    assert float((got - want).abs().max()) <= tol * max(1.0, float(want.abs().max()))


# float32: sums of up to 128 squares or 4,096 and a few function calls, 6e-8 each, adding up like their roots; bfloat16 outputs: half a
# step of 2^-8
def tolerance(dtype):
    return 4e-6 if dtype == torch.float32 else 2.1e-3 + 2 ** -9


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,qk_heads,d,dv,taps,rank", [(16, 16, 128, 128, 4, 32), (16, 8, 40, 24, 3, 5), (24, 24, 16, 128, 1, 0), (16, 4, 127, 1, 2, 1)])
def test_delta_prepare_tiles_of_tokens(dtype, heads, qk_heads, d, dv, taps, rank):
    """Sixteen tokens a CTA (tiles that lie in one request, that cross a border, that begin with kept inputs) against 64 bits, and,
    bit for bit, against the same requests one by one (one token a CTA)."""

    from llm_runtime_study_b200.ops import sequence_state as S

    g = torch.Generator().manual_seed(heads + d)
    lens = [1, 2, 13, 16, 17, 1, 40, 230]
    n, qk, vw = sum(lens), qk_heads * d, heads * dv
    channels, gates = 2 * qk + vw, heads * d if rank else heads
    beta_offset, low_offset = channels, channels + heads
    proj = torch.randn(n, low_offset + (rank or heads) + 3, generator=g).to(dtype)
    conv = torch.randn(2 * len(lens), taps - 1, channels, generator=g)
    w, a_log, dt = torch.randn(channels, taps, generator=g), 0.5 * torch.randn(heads, generator=g), torch.randn(gates, generator=g)
    up = torch.randn(rank, heads * d, generator=g).to(dtype) if rank else None
    slots = [2 * i + 1 for i in range(len(lens))]
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]

    def run(rows, q_start, at, entry):
        return S.delta_prepare(rows.to(DEV), heads=heads, qk_heads=qk_heads, dim=d, vdim=dv, beta_offset=beta_offset, low_offset=low_offset,
                               rank=rank, taps=w.to(DEV), conv_state=conv.to(DEV), a_log=a_log.to(DEV), dt_bias=dt.to(DEV),
                               a_up=None if up is None else up.to(DEV), q_start=ints(q_start), slots=ints(at), token_entry=ints(entry),
                               unit_eps=1e-6, q_scale=0.25)

    together = run(proj, starts, slots, [i for i, m in enumerate(lens) for _ in range(m)])
    assert n * heads >= 16 * 2 * 148
    x = proj.double()
    parts = []
    for i, m in enumerate(lens):
        rows = x[starts[i] : starts[i + 1], :channels]
        padded = torch.cat((conv[slots[i]].double(), rows))
        y = sum(padded[j : j + m] * w[:, j].double() for j in range(taps))
        parts.append(y * torch.sigmoid(y))
        if m * heads < 16 * 2 * 148:
            alone = run(proj[starts[i] : starts[i + 1]].contiguous(), [0, m], [slots[i]], [0] * m)
            for a, b in zip(alone, together):
                assert torch.equal(a, b[starts[i] : starts[i + 1]])
    y = torch.cat(parts)
    unit = lambda a: a / torch.sqrt(a.square().sum(-1, keepdim=True) + 1e-6)
    low = x[:, low_offset : low_offset + (rank or heads)]
    logits = (low @ up.double() if rank else low) + dt.double()
    rate = torch.exp(a_log.double())
    decay = torch.exp(-torch.nn.functional.softplus(logits) * (rate.repeat_interleave(d) if rank else rate))
    want = (0.25 * unit(y[:, :qk].view(n, qk_heads, d)).reshape(n, -1), unit(y[:, qk : 2 * qk].view(n, qk_heads, d)).reshape(n, -1),
            y[:, 2 * qk :], decay, torch.sigmoid(x[:, beta_offset : beta_offset + heads]))
    for got, exact in zip(together, want):
        close(got, exact, 4e-6)         # float32 results in either type; SiLU of 16-bit rows: two units in the last place more


# groups a warp holds (whole, partly idle lanes, many and few rows), whole rows, and groups no vector divides
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("taps", [1, 2, 3, 4])
def test_delta_prepare_keeps_bad_rows_within_the_taps_reach(dtype, taps):
    """An infinite or NaN row reaches the tokens whose taps meet it and no others, wherever it lies in a tile of tokens."""

    from llm_runtime_study_b200.ops import sequence_state as S

    heads, d, n = 32, 16, 200
    g = torch.Generator().manual_seed(taps)
    channels, bad = 3 * heads * d, {0: math.inf, 35: math.nan, 64: -math.inf, 110: math.inf, 199: math.nan}
    proj = torch.randn(n, channels + 2 * heads, generator=g)
    for row, value in bad.items():
        proj[row, :channels] = value
    q, k, v, decay, beta = S.delta_prepare(
        proj.to(dtype).to(DEV), heads=heads, qk_heads=heads, dim=d, vdim=d, beta_offset=channels, low_offset=channels + heads, rank=0,
        taps=torch.randn(channels, taps, generator=g).to(DEV), conv_state=torch.zeros(1, taps - 1, channels, device=DEV),
        a_log=torch.zeros(heads, device=DEV), dt_bias=torch.zeros(heads, device=DEV), a_up=None, q_start=ints([0, n]), slots=ints([0]),
        token_entry=ints([0] * n), unit_eps=1e-6, q_scale=1.0)
    assert n * heads >= 16 * 2 * 148                # sixteen tokens a CTA
    reached = torch.zeros(n, dtype=torch.bool)
    for row in bad:
        reached[row : row + taps] = True
    for name, x in (("q", q), ("k", k), ("v", v)):
        assert torch.equal(torch.isfinite(x).all(dim=1).cpu(), ~reached), name
    assert not bool(torch.isfinite(v[reached.to(DEV)]).any()) and bool(torch.isfinite(decay).all()) and bool(torch.isfinite(beta).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,groups,group,rank", [(300, 32, 128, 32), (3, 5, 128, 7), (257, 40, 36, 0), (2, 1, 4096, 0), (5, 3, 260, 0), (4, 2, 30, 3), (1, 4, 4, 1),
                                                  (50, 32, 96, 33), (47, 32, 128, 16)])
@pytest.mark.parametrize("act,divided", [("sigmoid", False), ("silu", True)])
def test_group_norm_gate(dtype, n, groups, group, rank, act, divided):
    from llm_runtime_study_b200.ops import sequence_state as S

    g = torch.Generator().manual_seed(n + group)
    width, offset = groups * group, 8
    x, weight = torch.randn(n, width, generator=g), torch.randn(group, generator=g)
    gate = torch.randn(n, offset + (rank or width) + (-(offset + (rank or width)) % 8), generator=g).to(dtype)
    up = torch.randn(rank, width, generator=g).to(dtype) if rank else None
    den, floor = torch.randn(n, groups, generator=g), torch.rand(n, groups, generator=g)
    out = S.group_norm_gate(x.to(DEV), weight.to(DEV), 1e-5, gate.to(DEV), gate_offset=offset, gate_up=None if up is None else up.to(DEV), act=act,
                            divisor=(den.to(DEV), floor.to(DEV), 1e-3) if divided else None, out_dtype=dtype)
    y = x.double().view(n, groups, group)
    if divided:
        y = y / (torch.maximum(den.abs(), floor).double() + 1e-3)[..., None]
    y = (y / torch.sqrt(y.square().mean(-1, keepdim=True) + 1e-5) * weight.double()).reshape(n, width)
    logits = gate.double()[:, offset : offset + (rank or width)]
    if rank:
        logits = logits @ up.double()
    close(out, y * (torch.sigmoid(logits) if act == "sigmoid" else logits * torch.sigmoid(logits)), tolerance(dtype))


@pytest.mark.parametrize("rank", [0, 5, 40])
def test_group_norm_gate_in_float32_gives_a_row_the_same_bits_in_any_batch(rank):
    """One row, few rows and rows that share what is read of the map."""

    from llm_runtime_study_b200.ops import sequence_state as S

    g = torch.Generator().manual_seed(rank)
    n, groups, group = 300, 32, 64
    x, gate = torch.randn(n, groups * group, generator=g).to(DEV), torch.randn(n, rank or groups * group, generator=g).to(DEV)
    up = torch.randn(rank, groups * group, generator=g).to(DEV) if rank else None
    weight = torch.randn(group, generator=g).to(DEV)
    run = lambda k: S.group_norm_gate(x[:k].contiguous(), weight, 1e-5, gate[:k].contiguous(), gate_up=up, out_dtype=torch.float32)
    together = run(n)
    for k in (1, 40, 60):
        assert torch.equal(run(k), together[:k])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,groups,group", [(1, 3, 8), (5, 300, 16), (3, 7, 6), (2, 32, 128)])
def test_sigmoid_gate(dtype, n, groups, group):
    from llm_runtime_study_b200.ops import mixer_steps as M

    g = torch.Generator().manual_seed(n)
    x, gate = torch.randn(n, groups * group, generator=g).to(dtype), torch.randn(n, groups + 5, generator=g).to(dtype)
    out = M.sigmoid_gate(x.to(DEV), gate.to(DEV), gate_offset=3, group=group)
    close(out, x.double() * torch.sigmoid(gate.double()[:, 3 : 3 + groups]).repeat_interleave(group, dim=1), tolerance(dtype))


# rows of one vector a thread, of several with a ragged end, of more than the registers hold, heads that no vector divides; a row without pages
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,nkv,d,dv", [(32, 8, 128, 128), (3, 1, 8, 16), (5, 5, 24, 40), (2, 1, 10, 8), (80, 4, 128, 64), (16, 2, 64, 64),
                                         (9, 1, 64, 72)])
def test_qk_rownorm_write(dtype, nq, nkv, d, dv):
    from llm_runtime_study_b200.ops import functional as F

    g = torch.Generator().manual_seed(nq)
    n, page = 5, 4
    width = nq * d + nkv * (d + dv)
    rows = torch.randn(n, width + (-width % 8), generator=g).to(dtype)
    qw, kw = torch.randn(nq * d, generator=g), torch.randn(nkv * d, generator=g)
    positions, entry = [0, 3, 4, 11, 2], [0, 0, 0, 1, 2]
    table = torch.tensor([[2, 5, -1], [1, 0, 4], [-1, -1, -1]], dtype=torch.int32)
    k_pool, v_pool = torch.zeros(6, nkv, page, d, dtype=dtype, device=DEV), torch.zeros(6, nkv, page, dv, dtype=dtype, device=DEV)
    q = F.qk_rownorm_write(rows.to(DEV), num_q_heads=nq, num_kv_heads=nkv, head_dim=d, value_dim=dv, q_weight=qw.to(DEV), k_weight=kw.to(DEV),
                           eps=1e-5, temp_coef=0.3, temp_every=4, positions=ints(positions), token_entry=ints(entry), block_table=table.to(DEV),
                           page_size=page, k_pool=k_pool, v_pool=v_pool)
    x = rows.double()
    norm = lambda a, w: a / torch.sqrt(a.square().mean(-1, keepdim=True) + 1e-5) * w.double()
    temp = torch.tensor([1 + 0.3 * math.log((p + 1) // 4 + 1) for p in positions], dtype=torch.float64)
    close(q.view(n, -1), norm(x[:, : nq * d], qw) * temp[:, None], tolerance(dtype))
    keys, values = torch.zeros(6, nkv, page, d, dtype=torch.float64), torch.zeros(6, nkv, page, dv, dtype=torch.float64)
    for t in range(4):
        at = int(table[entry[t], positions[t] // page])
        keys[at, :, positions[t] % page] = norm(x[t, nq * d : (nq + nkv) * d], kw).view(nkv, d)
        values[at, :, positions[t] % page] = x[t, (nq + nkv) * d : width].view(nkv, dv)
    close(k_pool, keys, tolerance(dtype))
    assert torch.equal(v_pool.double().cpu(), values)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("q_rank,kv_rank,rot,dims", [(2048, 512, 64, 64), (8, 16, 8, 4), (1000, 40, 16, 0), (12, 6, 4, 2), (8200, 64, 0, 0), (520, 0, 0, 0),
                                                      (768, 264, 8, 8), (512, 1040, 16, 16)])
def test_latent_prepare(dtype, q_rank, kv_rank, rot, dims):
    from llm_runtime_study_b200.ops import mixer_steps as M

    g = torch.Generator().manual_seed(q_rank)
    n, page, q_off = 3, 4, 8
    kv_off = q_off + q_rank + (-q_rank % 8)
    width = kv_off + kv_rank + rot
    rows = torch.randn(n, width + (-width % 8), generator=g).to(dtype)
    qw, kw = torch.randn(q_rank, generator=g), torch.randn(max(kv_rank, 1), generator=g)
    positions, entry = [1, 6, 3], [0, 0, 1]
    table = torch.tensor([[2, 3], [-1, -1]], dtype=torch.int32)
    freq = torch.rand(max(dims // 2, 1), generator=g)
    pool = torch.zeros(4, page, max(kv_rank + rot, 1), dtype=dtype, device=DEV)
    options = dict(kv_offset=kv_off, kv_rank=kv_rank, kv_weight=kw.to(DEV), rot=rot, pool=pool, block_table=table.to(DEV), page_size=page, rot_dims=dims,
                   inv_freq=freq.to(DEV) if dims else None, interleaved=True, rot_factor=1.25) if kv_rank else {}
    cq = M.latent_prepare(rows.to(DEV), q_offset=q_off, q_rank=q_rank, q_weight=qw.to(DEV), eps=1e-5, positions=ints(positions),
                          token_entry=ints(entry), **options)
    x = rows.double()
    norm = lambda a, w: a / torch.sqrt(a.square().mean(-1, keepdim=True) + 1e-5) * w.double()
    close(cq, norm(x[:, q_off : q_off + q_rank], qw), tolerance(dtype))
    if not kv_rank:
        return
    want = torch.zeros(4, page, kv_rank + rot, dtype=torch.float64)
    for t in range(2):
        turned = x[t, kv_off + kv_rank : kv_off + kv_rank + rot].clone()
        for i in range(dims // 2):
            a = positions[t] * float(freq[i])
            u, v = float(turned[2 * i]), float(turned[2 * i + 1])
            turned[2 * i], turned[2 * i + 1] = 1.25 * (u * math.cos(a) - v * math.sin(a)), 1.25 * (v * math.cos(a) + u * math.sin(a))
        want[int(table[0, positions[t] // page]), positions[t] % page] = torch.cat((norm(x[t, kv_off : kv_off + kv_rank], kw), turned))
    close(pool, want, tolerance(dtype))
