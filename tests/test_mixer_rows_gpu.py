"""Kernels that prepare or finish rows of mixers, at the edges of what their vectors, warps and tiles of tokens hold, against
64-bit arithmetic."""

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
@pytest.mark.parametrize("n,groups,group,rank", [(300, 32, 128, 32), (3, 5, 128, 7), (257, 40, 36, 0), (2, 1, 4096, 0), (5, 3, 260, 0), (4, 2, 30, 3), (1, 4, 4, 1)])
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
