"""bfloat16 projections on the 5th-generation tensor cores (tcgen05, TMEM, TMA)."""

from __future__ import annotations

import os

import torch

from ..errors import KernelError
from . import native
from .functional import GATE_ACTS
from .native import c_int, c_void_p

native.register_library(
    "b200_gemm_tcgen05", ("gemm_tcgen05.cu",),
    {
        "b200_gemm_tcgen05": [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_int,
                              c_int, c_int, c_int, c_void_p, c_void_p, c_int, c_void_p],
        "b200_gemm_tcgen05_grouped": [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p, c_int, c_int,
                                      c_void_p],
        "b200_gemm_tcgen05_error": [],
        "b200_gemm_tcgen05_pair_width": [c_int, c_int, c_int, c_int],
        "b200_gemm_tcgen05_accumulator_reused": [c_int, c_int, c_int, c_int],
        "b200_gemm_tcgen05_splitk_shape": [c_int, c_int, c_int, c_int, c_void_p, c_void_p],
        "b200_gemm_tcgen05_streamk_partial_floats": [],
        "b200_gemm_tcgen05_streamk_flags": [],
    },
)

native.register_library(
    "b200_gemm_skinny", ("gemm_skinny.cu",),
    {
        "b200_gemm_skinny": [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_void_p],
        "b200_gemm_skinny_variant": [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_int,
                                     c_void_p, c_void_p],
        "b200_gemm_skinny_residual": [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_void_p,
                                      native.c_float, c_void_p, c_void_p, c_void_p, c_void_p],
        "b200_gemm_skinny_summed": [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p, c_int, c_int,
                                    native.c_float, c_void_p],
        "b200_gemm_skinny_partial_floats": [c_int],
    },
)

native.register_library(
    "b200_gemm_features", ("gemm_features.cu",),
    {
        "b200_gemm_features": [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_int,
                               c_int, c_void_p],
        "b200_gemm_features_error": [],
        "b200_gemm_features_shape": [c_int, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p],
    },
)

PAIR_MIN_ROWS = 256   # from here on pairs of SMs work on 256 x 256 tiles (tcgen05 cta_group::2)
PAIR_WIDTHS = (128, 192, 224, 256)
PAIR_ENABLED = os.environ.get("LLM_RUNTIME_STUDY_B200_GEMM_PAIR", "1") != "0"
SKINNY_M = 16         # up to here weights are streamed straight into mma.sync fragments
KERNELS = {"persistent": 0, "pair": 1, "streamk": 2, "splitk": 3}

_STREAMK_WORKSPACE: dict[tuple, tuple[torch.Tensor, torch.Tensor]] = {}


def _streamk_workspace(device: torch.device) -> tuple[torch.Tensor, torch.Tensor]:
    """Partial accumulators and flags of the stream-K kernel, one set per device, made on first
    use and kept.  The flags are zero between launches; launches on one device share the set and
    therefore must follow each other on one stream, which is how the engine runs."""

    key = (device.type, device.index)
    have = _STREAMK_WORKSPACE.get(key)
    if have is None:
        floats = native.query("b200_gemm_tcgen05_streamk_partial_floats")
        flags = native.query("b200_gemm_tcgen05_streamk_flags")
        have = (torch.empty(floats, dtype=torch.float32, device=device), torch.zeros(flags, dtype=torch.int32, device=device))
        _STREAMK_WORKSPACE[key] = have
    return have


def supported(m: int, n: int, k: int) -> bool:
    """TMA needs rows that start on 16-byte boundaries: K a multiple of 8."""

    return k % 8 == 0 and m > 0 and n > 0


def pick_kernel(m: int, n: int, k: int) -> tuple[str, int]:
    """Which kernel and which tile width take a product of this shape (chosen from timings at the
    Qwen3-8B layer widths with 128 to 4,096 rows).  Pairs of SMs when 256 x 256 tiles fill
    most of the 74 pairs, or 128 x 256 tiles half the SMs (their tiles are narrower where that fills the pairs better; with fewer
    than 256 rows or K below 1,024 one CTA per 128 x 256 tile; 405 x 6,144 x 4,096: 22.8 us against 29.8, 700 x 4,096 x 4,096: 28.6 against 37.1), and
    for a long K range that no kernel below shares (405 x 4,096 x 12,288: 52.2 us against 58.4 with 128-column tiles); up to
    256 rows and a third of the SMs: clusters that share a tile's K range (split-K, which chooses
    its own width); stream-K when a third of the SMs or fewer would have a tile and the K range is
    long enough to share; else one CTA per 128 x 128 tile.  A product with few tiles is as slow as
    the SM that has most to pull in, so it pays to spread the bytes over more SMs.  Up to 1,024 columns that
    holds up to 512 rows: 405 x 1024 x 3072 takes 12.9 us with split-K, 20.1 with 128-column tiles and 27.0 with
    stream-K; 405 x 1024 x 2048 12.5 against 17.4.  With more rows split-K's clusters no longer fit at once (600 x 1024 x
    3072: 23.8 us) and 128-column tiles (20.2) stay ahead of stream-K (27.3).  Up to 96 columns its tiles are narrow
    and a short K range is not worth sharing (300 x 64 x 2048: 12.9 us against 11.8; x 2560: 13.5 against 13.6).
    ("pair", 256) names the kernel's rows of tiles; their width is the kernel's own choice (``b200_gemm_tcgen05_pair_width``).  Against the
    rules before the pairs' narrower tiles (256 columns only, 128 x 256 tiles one CTA each, long K ranges in 128-column tiles) the choice
    differs for 1,093 of the products of 130 to 4,096 rows, 128 to 24,576 columns and K of 1,024 to 12,288 that were timed both ways; it takes 0.86 of their
    time in the mean (405 x 6,144 x 1,024 from cold caches 16.4 us, 18.4 with one CTA a tile).  Two of them are slower, 450 and 1,024 x 8,192 x 4,104 by 5
    and 7 %: their rows are not whole 128-byte lines.  Up to 384 rows a K range of 8,192 and more keeps the kernels it had."""

    sms = native.sm_count()
    if n <= 1024 and 256 < m <= 2048 and 2048 <= k <= 4096:
        return ("splitk", 0) if m <= 512 and (n > 96 or k >= 2560) else ("persistent", 128)
    if m >= PAIR_MIN_ROWS and PAIR_ENABLED and 5 * -(-m // 256) * -(-n // 256) >= 2 * sms:   # 60 of a B200's 74 pairs
        return "pair", 256
    tiles = -(-m // 128) * -(-n // 256)
    if 2 * tiles >= sms:
        return ("pair" if m >= PAIR_MIN_ROWS and k >= 1024 and PAIR_ENABLED else "persistent"), 256
    if m <= 256 and 3 * tiles <= sms:
        return "splitk", 0
    if 3 * tiles <= sms + 2 and k >= 48 * 64:
        return "streamk", 256
    if m > 384 and k >= 8192 and PAIR_ENABLED:
        return "pair", 256
    return "persistent", 128


def by_features(m: int, n: int, k: int, out_float32: bool) -> bool:
    """Whether a product of this shape goes to the kernel that has the weight as its row operand (``linear_features``) and not to the one that
    ``pick_kernel`` names.  Timed both ways at 18 numbers of rows (17 to 2,048), 11 of columns (256 to 12,288) and 8 of K (512 to
    12,288), float32 sums and bfloat16 results, and at 22 numbers of rows (129 to 2,048) for 20 larger products, up to 151,936 columns and K of 28,672.
    Float32 rows are what it writes best: it is ahead from 129 rows on (0.40 to 0.97 of the time, 0.75
    in the mean; of the larger products 0.47 to 1.10, 0.87) but where other kernels fill the GPU better: around 2,048 columns up to 256 rows (1.05 to
    1.26), 8,192 and more columns beyond 1,024 rows (0.97 to 1.12; with a long K or as an output head from 897 on: 1.03 to 1.11), short K with many rows
    (1.06 to 1.17), 225 to 256 rows of 12,288 to 28,672 columns, which are one full round of pairs (0.93 to 1.15).  Of the bfloat16 results those with few tiles
    and a long K range (257 to 512 rows up to 4,096 columns 0.48 to 1.07, mean 0.73; to 1,024 rows up to 2,048 columns 0.51 to 0.99), 129
    to 256 rows whose 128-row tiles are half empty (3,072 to 6,144 columns: 0.65 to 1.04; with 4,096 columns and K beyond 16,384 1.08 to 1.11), and 513 to
    896 rows of wide products, whose 256-row tiles are (0.71 to 1.05, mean 0.90), but not 641 to 768 and more than 832 rows of some 16,000 to 20,000 columns
    (1.02 to 1.09) and 641 to 768 of some 5,000 with a long K (1.05 to 1.07)."""

    if not (PAIR_ENABLED and 128 < m <= 2048):
        return False
    if out_float32:
        return not ((176 < m <= 256 and 1536 < n <= 2560) or (224 < m <= 256 and 12288 <= n <= 28672 and k >= 4096)
                    or (m > 896 and k >= 4096 and n * k >= 200_000_000 and (n >= 65536 or k > 16384)) or (m > 1024 and (n >= 8192 or k < 1024)))
    if m <= 256:
        return (3072 <= n <= 4096 and k <= 16384) or (m <= 208 and 4096 < n <= 6144)
    if m <= 512:
        return n <= 4096 and k >= 3072
    if n >= 5120 and m <= 896:
        return not (14336 < n <= 20480 and (640 < m <= 768 or m > 832)) and not (n < 6144 and k > 12288 and 640 < m <= 768)
    return m <= 1024 and n <= 2048 and k >= 3072


# weight elements from which 9 to 16 rows go to the tcgen05 split-K kernel
SKINNY_LARGE = int(os.environ.get("LLM_RUNTIME_STUDY_B200_SKINNY_LARGE", 52_000_000))


def splitk_shape(m: int, n: int, k: int, sm_count: int = 0) -> tuple[int, int]:
    """(tile width, CTAs per tile) the split-K kernel chooses by itself for this product."""

    import ctypes

    width, splits = ctypes.c_int(0), ctypes.c_int(0)
    native.call("b200_gemm_tcgen05_splitk_shape", m, n, k, sm_count or native.sm_count(), ctypes.addressof(width), ctypes.addressof(splits), launches=0)
    return width.value, splits.value


def few_rows_kernel(m: int, n: int, k: int) -> str:
    """"skinny" or "splitk" for at most ``SKINNY_M`` rows.  The weight-streaming kernel handles 9 to 16
    rows as two token tiles per weight fragment and then reaches about 5 TB/s; the split-K kernel
    streams at 6 TB/s but costs about 4 us more per launch, so it takes the products whose weights
    are larger than about 100 MB (Qwen3-32B at 16 rows: 178 against 205 us per layer; Qwen3-8B
    gate/up: 37 against 43 us), and the weight-streaming kernel the rest.  Up to 8 rows the
    weight-streaming kernel is as fast or faster except where few output rows meet a very long K
    (the down projections of Qwen3-14B and 32B: 33.6 against 36.9 us, 47.0 against 52.9 us)."""

    if m > 8:
        return "splitk" if n * k >= SKINNY_LARGE else "skinny"
    return "splitk" if k >= 16384 and n * k >= SKINNY_LARGE else "skinny"


def gated_in_one(n: int, k: int) -> bool:
    """Whether a gated unit's projection of 17 to 127 rows goes to the split-K kernel, whose epilogue applies the gate, and not to the library and
    a kernel for the gate behind it: where the weights are 160 MB and more with 20,000 rows of 3,072 columns or more, and streaming them is all that
    counts (24,576 x 4,096 with 17, 64
    and 96 rows 38.0, 39.5, 40.0 us, 38.7, 41.7, 43.2 with the library; a decode step of nine such layers 1,263 -> 1,232 with 24
    requests, 1,553 -> 1,515 with 64).  Smaller ones are the library's (16,384 x 2,048 with 64 rows 18.6, 15.4; steps with them 1 % longer), and
    so are short columns, whose products are over before the next tile's begin (98,304 x 640 1.03 to 1.32 of the library's time, 49,152 x 2,048
    0.95 to 1.05), and fewer rows, which are too few tiles (8,192 x 8,192 and 8,192 x 12,288 1.37 to 1.71, 14,336 x 5,120 1.06 to 1.14, 16,384 x 4,096
    1.02 to 1.07; 24,576 x 4,096 0.85 to 0.99, 28,672 x 8,192 0.87 to 1.01)."""

    return n >= 20_000 and k >= 3072 and n * k >= 80_000_000


def gated_unit(swiglu: "bool | str") -> int:
    """The kernels' number of a gated unit: 0 for none, else its gate (``True``: SiLU)."""

    return 0 if not swiglu else GATE_ACTS["silu" if swiglu is True else swiglu]


def linear(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None = None,
           out_dtype: torch.dtype = torch.bfloat16, *, swiglu: "bool | str" = False, add_to: torch.Tensor | None = None,
           kernel: str | None = None, tile_n: int | None = None, splits: int = 0, stages: int = 0, pair_width: int = 0,
           weight_at_rest: bool = False) -> torch.Tensor:
    """``x @ weight.T (+ bias)`` on the tcgen05 tensor cores; float32 accumulation; bfloat16 or
    float32 output.

    ``swiglu``: the weight holds gate and up rows interleaved in blocks of eight and the result is
    ``silu(gate) * up``, half as wide (``"gelu_tanh"``: with that gate).  ``add_to`` (float32 ``[M, N]``): the product is added to it
    in place and it is returned.  ``kernel``: "persistent" (one CTA per tile of 128 rows and
    ``tile_n`` = 128 or 256 columns), "pair" (two CTAs per tile of 256 rows and
    ``pair_width`` = 128, 192, 224 or 256 columns, or ``tile_n`` = 256; neither lets the kernel choose so that its rounds of tiles are full), "streamk" (few
    tiles: up to three SMs share a tile's K range) or "splitk" (few rows: a cluster of ``splits``
    <= 8 CTAs shares the K range of every 128 x ``tile_n`` tile, ``tile_n`` a multiple of 32; 0 for either
    lets the kernel choose so that the SMs are filled once; ``stages``: depth of its operand ring, 0 = as
    deep as shared memory allows); chosen by shape when not given, the kernel of ``linear_features`` among them.
    ``weight_at_rest``: no kernel that may still be running on the stream writes ``weight``, as with a model's weights; some kernels then
    read it ahead of the wait for the kernel before."""

    native.require(x, "x", dtype=torch.bfloat16, dims=2)
    native.require(weight, "weight", dtype=torch.bfloat16, dims=2)
    m, k = x.shape
    n = weight.shape[0]
    if weight.shape[1] != k:
        raise KernelError(f"linear: x has width {k}, weight expects {weight.shape[1]}")
    if not supported(m, n, k):
        raise KernelError(f"tcgen05 projection needs K to be a multiple of 8, got {k}")
    if bias is not None:
        native.require(bias, "bias", dtype=torch.float32, shape=(n,))
    if swiglu and (n % 16 or add_to is not None):
        raise KernelError("the SwiGLU epilogue needs an even number of 8-feature blocks and excludes add_to")
    if add_to is not None:
        native.require(add_to, "add_to", dtype=torch.float32, shape=(m, n))
        out, out_dtype = add_to, torch.float32
    else:
        if out_dtype not in (torch.bfloat16, torch.float32):
            raise KernelError(f"unsupported output type {out_dtype}")
        out = torch.empty((m, n // 2 if swiglu else n), dtype=out_dtype, device=x.device)
    if not (kernel or tile_n or splits or stages or pair_width or swiglu) and by_features(m, n, k, out_dtype == torch.float32):
        _by_features(x, weight, bias, out, add_to is not None, (0, 0), 0, weight_at_rest)
        return out
    picked_kernel, picked_width = pick_kernel(m, n, k)
    kernel = kernel or picked_kernel
    if pair_width and (kernel != "pair" or pair_width not in PAIR_WIDTHS):
        raise KernelError(f"pair_width {pair_width} is for the pair kernel, and one of {PAIR_WIDTHS}")
    asked = tile_n
    if kernel == "splitk":
        tile_n = tile_n or 0                        # 0: the kernel chooses
        if tile_n % 32 or not 0 <= tile_n <= 256 or not 0 <= splits <= 8:
            raise KernelError(f"split-K takes tiles of 32 to 256 columns in steps of 32 and up to 8 CTAs per tile, got {tile_n}, {splits}")
    else:
        tile_n = tile_n or (picked_width if kernel == picked_kernel else 256)
        if kernel not in KERNELS or tile_n not in (128, 256) or (tile_n == 128 and kernel != "persistent"):
            raise KernelError(f"unknown projection kernel {kernel!r} or tile width {tile_n}: expected one of {sorted(KERNELS)}, "
                              "256 columns, or 128 with the persistent kernel")
    if kernel == "pair":
        tile_n = pair_width or asked or 0               # 0: the kernel chooses
    partials, flags = _streamk_workspace(x.device) if kernel == "streamk" else (None, None)
    native.call("b200_gemm_tcgen05", x.data_ptr(), weight.data_ptr(), native.ptr(bias), out.data_ptr(), m, n, k,
                out.shape[1], 1 if out_dtype == torch.float32 else 0, gated_unit(swiglu), 0 if add_to is None else 1,
                KERNELS[kernel], tile_n, splits, stages, native.ptr(partials), native.ptr(flags), 1 if weight_at_rest else 0, native.stream_ptr())
    return out


def _by_features(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None, out: torch.Tensor, add: bool, tokens: tuple[int, int],
                 splits: int, weight_at_rest: bool) -> None:
    (m, k), n = x.shape, weight.shape[0]
    native.call("b200_gemm_features", x.data_ptr(), weight.data_ptr(), native.ptr(bias), out.data_ptr(), m, n, k, n,
                1 if out.dtype == torch.float32 else 0, 1 if add else 0, tokens[0], tokens[1], splits, 1 if weight_at_rest else 0,
                native.stream_ptr())


def linear_features(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None = None, out_dtype: torch.dtype = torch.bfloat16, *,
                    add_to: torch.Tensor | None = None, tokens: tuple[int, int] = (0, 0), splits: int = 0,
                    weight_at_rest: bool = False) -> torch.Tensor:
    """As ``linear``, with the weight as the tensor cores' row operand: pairs of SMs on tiles of 256 features and ``tokens`` rows of
    ``x`` (the two numbers' sum, each a multiple of 32 up to 256, the second may be 0), ``splits`` (1, 2 or 4) pairs to a tile's K range;
    chosen by shape when not given."""

    native.require(x, "x", dtype=torch.bfloat16, dims=2)
    native.require(weight, "weight", dtype=torch.bfloat16, dims=2)
    m, k = x.shape
    n = weight.shape[0]
    if weight.shape[1] != k:
        raise KernelError(f"linear: x has width {k}, weight expects {weight.shape[1]}")
    if not supported(m, n, k):
        raise KernelError(f"tcgen05 projection needs K to be a multiple of 8, got {k}")
    if bias is not None:
        native.require(bias, "bias", dtype=torch.float32, shape=(n,))
    if add_to is not None:
        native.require(add_to, "add_to", dtype=torch.float32, shape=(m, n))
        out, out_dtype = add_to, torch.float32
    else:
        if out_dtype not in (torch.bfloat16, torch.float32):
            raise KernelError(f"unsupported output type {out_dtype}")
        out = torch.empty((m, n), dtype=out_dtype, device=x.device)
    _by_features(x, weight, bias, out, add_to is not None, tokens, splits, weight_at_rest)
    return out


def linear_with_bias(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor, *, weight_at_rest: bool = False) -> torch.Tensor:
    """``x @ weight.T + bias`` in bfloat16 for 17 to 127 rows.  Without a bias such products are the library's; behind one of those
    the sum is two launches more (the bias in bfloat16, the addition) and rounds twice.  With a K range or a number of columns up to 2,048 by
    features, else split-K, microseconds with 17, 64 and 127 rows against the library and the sum: 16,384 x 2,048 16.2, 17.1, 17.8
    (17.6, 19.9, 23.2), 2,048 x 8,192 14.3, 14.4, 15.6 (18.0, 18.4, 18.9), 24,576 x 4,096 40.5, 42.4, 46.4 (42.7, 47.3, 49.9), 4,096 x 12,288
    23.4, 25.2, 26.8 (27.6, 28.3, 28.6), 1,024 x 1,024 6.5, 6.5, 6.7 (8.1, 7.9, 8.0).  (A float32 sum is one launch and
    added in place: as fast as these, so it stays.)"""

    if PAIR_ENABLED and (x.shape[1] <= 2048 or weight.shape[0] <= 2048):
        return linear_features(x, weight, bias, torch.bfloat16, weight_at_rest=weight_at_rest)
    return linear(x, weight, bias, torch.bfloat16, kernel="splitk", weight_at_rest=weight_at_rest)


def features_shape(m: int, n: int, k: int, sm_count: int = 0) -> tuple[int, int, int]:
    """(tokens of a tile's first and second product, pairs to a tile's K range) that are chosen for this product."""

    import ctypes

    got = (ctypes.c_int * 3)()
    at = ctypes.addressof(got)
    native.call("b200_gemm_features_shape", m, n, k, sm_count or native.sm_count(), at, at + 4, at + 8, launches=0)
    return got[0], got[1], got[2]


native.register_error_probe("b200_gemm_tcgen05", "b200_gemm_tcgen05_error", "tcgen05 projection")
native.register_error_probe("b200_gemm_features", "b200_gemm_features_error", "tcgen05 projection by features")


def check_error() -> None:
    """Synchronise and raise if a bounded wait inside one of the tcgen05 kernels of this module ran out."""

    where = {1: "producer", 2: "tensor-core issue", 3: "epilogue", 4: "accumulator buffer", 5: "flag or exchange of a shared tile", -1: "device error"}
    codes = [(what, native.query(probe)) for what, probe in (("tcgen05 projection", "b200_gemm_tcgen05_error"),
                                                             ("tcgen05 projection by features", "b200_gemm_features_error"))]
    if codes[0][1]:
        for _, flags in _STREAMK_WORKSPACE.values():     # a wait that ran out may have left flags behind
            flags.zero_()
    for what, code in codes:
        if code:
            raise KernelError(f"{what}: a bounded wait ran out ({where.get(code, str(code))})")


def linear_skinny(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None = None,
                  out_dtype: torch.dtype = torch.bfloat16, *, variant: int = 0, swiglu: "bool | str" = False,
                  row_scale: torch.Tensor | None = None, sums: torch.Tensor | None = None, eps: float = 0.0) -> torch.Tensor:
    """``x @ weight.T (+ bias)`` for at most 16 rows of ``x``: the weight-streaming kernel.
    ``swiglu``: see ``linear``.  ``row_scale`` (float32 ``[16]``): the rows of ``x`` still lack these factors
    (an RMS norm left half done, see ``linear_skinny_residual``); they are applied to the product, before the bias.
    ``sums`` (float32 ``[parts, 16]``, with the norm's ``eps``) instead of it: the shares of the rows' sums of squares that make the factors, for at
    most eight rows.  ``weight`` is read ahead of the wait for the kernel before: that kernel must not write it."""

    native.require(x, "x", dtype=torch.bfloat16, dims=2)
    native.require(weight, "weight", dtype=torch.bfloat16, dims=2)
    m, k = x.shape
    n = weight.shape[0]
    if weight.shape[1] != k:
        raise KernelError(f"linear: x has width {k}, weight expects {weight.shape[1]}")
    if m > SKINNY_M or k % 8:
        raise KernelError(f"the weight-streaming kernel takes at most {SKINNY_M} rows and K a multiple of 8; got {m}, {k}")
    if bias is not None:
        native.require(bias, "bias", dtype=torch.float32, shape=(n,))
    if swiglu and n % 16:
        raise KernelError("the SwiGLU epilogue needs an even number of 8-feature blocks")
    if row_scale is not None:
        native.require(row_scale, "row_scale", dtype=torch.float32, shape=(16,))
    width = n // 2 if swiglu else n
    out = torch.empty((m, width), dtype=out_dtype, device=x.device)
    if sums is not None:
        native.require(sums, "sums", dtype=torch.float32, dims=2)
        if sums.shape[1] != 16 or row_scale is not None:
            raise KernelError("a row's factor comes as itself or as 16 columns of shares")
        native.call("b200_gemm_skinny_summed", x.data_ptr(), weight.data_ptr(), native.ptr(bias), out.data_ptr(), m, n, k, width,
                    1 if out_dtype == torch.float32 else 0, gated_unit(swiglu), sums.data_ptr(), sums.shape[0], k, float(eps), native.stream_ptr())
        return out
    native.call("b200_gemm_skinny_variant", x.data_ptr(), weight.data_ptr(), native.ptr(bias), out.data_ptr(), m, n, k, width,
                1 if out_dtype == torch.float32 else 0, variant, gated_unit(swiglu), native.ptr(row_scale), native.stream_ptr())
    return out


SUMMED_ROWS, SUMMED_WIDTH = 8, 2048      # rows, and their columns, up to which the consuming kernel forms the rows' factors itself


def linear_skinny_residual(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None, resid: torch.Tensor,
                           next_weight: torch.Tensor, eps: float, *, finish: bool = True) -> tuple[torch.Tensor, torch.Tensor]:
    """``resid += x @ weight.T (+ bias)`` in place (float32 ``[M, N]``, at most 16 rows), and on the way out
    what the RMS norm after it needs: ``resid * next_weight`` rounded to bfloat16, and every row's factor
    ``rsqrt(mean of squares + eps)`` (``[16]`` floats; rows from ``M`` on hold 0).  Returns (weighted, row_scale), or, not to
    ``finish``, (weighted, sums): the shares ``[N / 16, 16]`` of the rows' sums of squares, which ``linear_skinny`` takes."""

    native.require(x, "x", dtype=torch.bfloat16, dims=2)
    native.require(weight, "weight", dtype=torch.bfloat16, dims=2)
    m, k = x.shape
    n = weight.shape[0]
    if weight.shape[1] != k or m > SKINNY_M or k % 8:
        raise KernelError(f"the weight-streaming kernel takes at most {SKINNY_M} rows and K a multiple of 8; got {m}, {k}")
    native.require(resid, "resid", dtype=torch.float32, shape=(m, n))
    native.require(next_weight, "next_weight", dtype=torch.float32, shape=(n,))
    if bias is not None:
        native.require(bias, "bias", dtype=torch.float32, shape=(n,))
    weighted = torch.empty((m, n), dtype=torch.bfloat16, device=x.device)
    row_scale = torch.empty(16, dtype=torch.float32, device=x.device) if finish else None
    partials = torch.empty((native.query("b200_gemm_skinny_partial_floats", n) // 16, 16), dtype=torch.float32, device=x.device)
    native.call("b200_gemm_skinny_residual", x.data_ptr(), weight.data_ptr(), native.ptr(bias), resid.data_ptr(), m, n, k, n,
                next_weight.data_ptr(), float(eps), weighted.data_ptr(), native.ptr(row_scale), partials.data_ptr(),
                native.stream_ptr(), launches=2 if finish else 1)
    return weighted, (row_scale if finish else partials)
