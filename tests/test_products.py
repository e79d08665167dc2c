"""The prefill's matrix products alone, in every kind of tile, against 64-bit sums."""

import pytest
import torch

from megakernels_b200.mk import get_mk_module

# tokens: one, part of a tile, its edge, pairs of tiles and their remainders; features and inner size: edges of
# tiles and of the inner dimension's steps; the larger ones take the wide tiles
SHAPES = [
    (1, 4096, 2048), (2, 515, 130), (3, 250, 72), (17, 130, 264), (33, 2048, 1024), (61, 2048, 2048), (61, 3072, 520), (128, 512, 64), (129, 3072, 2048),
    (256, 16384, 256), (257, 1000, 328), (300, 10304, 512), (501, 2048, 8192), (2048, 4096, 512), (1100, 4100, 1096),
]


def product(result, dtype, T, N, K, seed=0):
    mk = get_mk_module(name="mk_hybrid")
    gen = torch.Generator(device="cuda").manual_seed(seed)
    pad = (K + 7) // 8 * 8
    make = lambda rows: torch.randn(rows, pad, generator=gen, device="cuda").to(dtype)  # noqa: E731
    a, w = make(T), make(N)
    a[:, K:], w[:, K:] = float("nan"), float("nan")  # (bf16: outside the tensor maps; float: read, dropped)
    w /= K**0.5
    status = torch.zeros(16, dtype=torch.int32, device="cuda")
    sums = a[:, :K].double() @ w[:, :K].double().T
    size = (a[:, :K].double().abs() @ w[:, :K].double().abs().T)
    exact = K / 16 * 2.0**-22 if dtype == torch.bfloat16 else K * 2.0**-24  # of the sum of magnitudes (see the tests)
    wrong = exact * size  # most that an element may be off before it is rounded to its type
    kw = {}
    if result == "store":
        kw["bias"] = torch.randn(N, generator=gen, device="cuda")
        out, want = torch.full((T, N), float("nan"), device="cuda"), sums + kw["bias"].double()
        wrong = wrong + 2.0**-24 * want.abs()
    elif result == "add":
        kw["scale"] = torch.randn(N, generator=gen, device="cuda")
        out = torch.randn(T, N, generator=gen, device="cuda")
        want = out.double() + sums * kw["scale"].double()
        wrong = (wrong + 2.0**-24 * sums.abs()) * kw["scale"].double().abs() + 2.0**-24 * want.abs()
    elif result == "cast":
        out, want = torch.full((T, (N + 7) // 8 * 8), float("nan"), device="cuda", dtype=dtype), sums
    elif result == "glu":
        kw.update(limit=1.5, alpha=1.7)
        g, u = sums[:, ::2].clamp(max=1.5), sums[:, 1::2].clamp(-1.5, 1.5)
        out, want = torch.full((T, N // 2), float("nan"), device="cuda", dtype=dtype), g * torch.sigmoid(1.7 * g) * (u + 1)
        wrong = 1.1 * wrong[:, ::2] * (u + 1).abs() + (g * torch.sigmoid(1.7 * g)).abs() * wrong[:, 1::2] + 2.0**-20 * (1 + want.abs())
    else:
        kw["w2"] = make(N) / K**0.5
        kw["w2"][:, K:] = float("nan")
        out = torch.full((T, (N + 7) // 8 * 8), float("nan"), device="cuda", dtype=dtype)
        up = a[:, :K].double() @ kw["w2"][:, :K].double().T
        want = sums * torch.sigmoid(sums) * up
        wrong = 1.1 * wrong * up.abs() + (sums * torch.sigmoid(sums)).abs() * exact * (a[:, :K].double().abs() @ kw["w2"][:, :K].double().abs().T)
        wrong = wrong + 2.0**-20 * want.abs()
    mk.product(result, a, w, out, status, K, **kw)
    again = out.clone() if result != "add" else None
    if again is not None:  # the same bits whatever the order of arrival
        mk.product(result, a, w, out, status, K, **kw)
        assert torch.equal(out[:, : want.shape[1]], again[:, : want.shape[1]])
    assert int(status[0]) == 0
    if result in ("cast", "silu"):
        assert torch.isnan(out[:, N:]).all()  # nothing beyond the features is written
    return out[:, : want.shape[1]].double(), want, wrong


@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K", SHAPES)
@pytest.mark.parametrize("result", ["store", "add", "cast", "glu", "silu"])
def test_bf16_products(result, T, N, K):
    """32-bit sums of exact products: an instruction adds 16 of them to the accumulator and may cut what lies below 2^-23 of
    the largest term, twice that for the sums of a cluster's parts and the alignment; K / 16 of these, none above the sum of
    magnitudes.  Their mean square is held to a quarter of that of the results (cuts have one sign), where accumulators or
    parts rounded to bf16 would be off by 1e-3.  Where the result is bf16, one rounding: an element is off by what that
    takes off the exact value, or by as much on the other side if the sum's own error reaches the middle."""
    if result == "glu" and N % 2:
        N += 1
    out, want, wrong = product(result, torch.bfloat16, T, N, K)
    error = (out - want).abs()
    once = (want.float().bfloat16().double() - want).abs() if result in ("cast", "glu", "silu") else torch.zeros_like(want)
    assert (error <= once + 2 * wrong + 2.0**-23 * want.abs()).all(), float((error - once - 2 * wrong).max())
    assert float(error.norm()) < 1.001 * float(once.norm()) + max(K / 16 * 2.0**-24, 1e-6) * float(want.norm())


@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K", SHAPES)
@pytest.mark.parametrize("result", ["store", "add", "cast", "glu"])
def test_float32_products(result, T, N, K):
    """Products are exact but for 2^-24 of them, a step of 32 of the inner dimension is cut by at most 2^-23 of its sum and added up with an error of
    2^-24 of the sum so far; one or two tokens and an inner dimension below 16 are FMA.  Far below what bf16 or tf32 operands would give
    (2^-9, 2^-11), and in the mean square below what two tf32 parts give (2e-7 at any length; units and their exponentials aside)."""
    if result == "glu" and N % 2:
        N += 1
    out, want, wrong = product(result, torch.float32, T, N, K)
    assert ((out - want).abs() <= wrong + 2.0**-24 * want.abs()).all()
    assert float((out - want).norm() / want.norm()) < (2e-6 if result == "glu" else most_wrong(K))


def most_wrong(K):
    """Largest 2-norm of the relative error of sums that stay within the size of the result: steps of 32 cut by 0 .. 2^-23 (mean square 2^-23 /
    sqrt 3) and as many roundings of 2^-24 / sqrt 3 to sums that grow to it.  Below 16, the roundings of FMA."""
    adds = K if K < 16 else (K + 31) // 32
    return 2.0**-23 * (3**-0.5 + 0.29 * (adds / 2) ** 0.5)


@pytest.mark.gpu
@pytest.mark.parametrize("K", [1, 2, 5, 8, 15, 16, 17, 31, 33, 64, 200, 1024])
@pytest.mark.parametrize("kind", ["normal", "one sign", "remainders", "dominated"])
def test_float32_products_keep_all_bits_of_their_operands(kind, K):
    """Short and long inner dimensions, where an operand's last bits show: sums of one sign, operands whose remainders are as large as they
    get at 11 and at 8 bits (their products' exact sums), one column a thousand times the others (not further off than FMA in order,
    which rounds every later sum)."""
    mk = get_mk_module(name="mk_hybrid")
    gen = torch.Generator(device="cuda").manual_seed(K)
    T, N, pad = 48, 512, (K + 7) // 8 * 8
    a, w = torch.zeros(T, pad, device="cuda"), torch.zeros(N, pad, device="cuda")
    for m in (a, w):
        if kind == "one sign":
            m[:, :K] = 1 + torch.rand(len(m), K, generator=gen, device="cuda")
        elif kind == "remainders":
            m[:, :K] = 1 + 2.0**-11 - 2.0**-23
        else:
            m[:, :K] = torch.randn(len(m), K, generator=gen, device="cuda")
    if kind == "dominated":
        a[:, K // 2] *= 1000
    out, status = torch.zeros(T, N, device="cuda"), torch.zeros(16, dtype=torch.int32, device="cuda")
    mk.product("store", a, w, out, status, K)
    want = a.double() @ w.double().T
    error = out.double() - want
    assert int(status[0]) == 0
    if kind == "remainders":
        assert (error.abs() <= 2.0**-23 * want).all()
    elif kind == "dominated":
        fma = torch.zeros(T, N, device="cuda")  # (64-bit sums of a 48-bit product and a float, rounded once)
        for k in range(K):
            fma = (fma.double() + a[:, k, None].double() * w[None, :, k].double()).float()
        assert float(error.norm()) <= 1.02 * float((fma.double() - want).norm())
    else:
        assert float(error.norm() / want.norm()) < most_wrong(K)


@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K", [(3, 260, 40), (16, 256, 8), (17, 1000, 2048), (96, 384, 520), (97, 300, 64), (160, 512, 2048), (161, 2048, 328), (320, 257, 1000)])
def test_float32_products_of_odd_operands(T, N, K):
    """Infinite operands, one that rounds to infinity where it is split, and no numbers: results are infinite or no numbers where
    64-bit sums are, the others within the bound of fp32 sums."""
    mk = get_mk_module(name="mk_hybrid")
    gen = torch.Generator(device="cuda").manual_seed(T)
    a = torch.randn(T, K, generator=gen, device="cuda")
    w = (torch.randn(N, K, generator=gen, device="cuda") / K**0.5).bfloat16().float()  # (no remainders)
    a[0, 5], a[1, 7], a[2, 3] = float("inf"), torch.finfo(torch.float32).max, float("nan")
    w[3, 1], w[200, 4] = float("-inf"), float("nan")
    out, status = torch.full((T, N), 7.0, device="cuda"), torch.zeros(16, dtype=torch.int32, device="cuda")
    mk.product("store", a, w, out, status, K)
    want = a.double() @ w.double().T
    assert int(status[0]) == 0
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isinf(), want.float().isinf())
    finite = out.isfinite()
    size = a.abs().double().nan_to_num(0, 0) @ w.abs().double().nan_to_num(0, 0).T
    assert ((out.double() - want).abs() <= (K + 1) * 2.0**-24 * size)[finite].all()


@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K", [(61, 300, 1000), (161, 2048, 8192), (300, 260, 2048)])
def test_infinite_operands_at_the_edges(T, N, K):
    """One infinite operand in the last token and one in the last feature, at either end of the inner dimension (another CTA's part
    of it): their sums are infinite, all others as before; in a bounded time (a tile is done over by all of its warps)."""
    mk = get_mk_module(name="mk_hybrid")
    gen = torch.Generator(device="cuda").manual_seed(T)
    a, w = torch.randn(T, K, generator=gen, device="cuda"), torch.randn(N, K, generator=gen, device="cuda") / K**0.5
    a[T - 1, K - 1], w[N - 1, 0] = float("inf"), float("-inf")
    out, status = torch.full((T, N), 7.0, device="cuda"), torch.zeros(16, dtype=torch.int32, device="cuda")
    mk.product("store", a, w, out, status, K)  # (the first launch loads the kernel)
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    begin.record()
    mk.product("store", a, w, out, status, K)
    end.record()
    torch.cuda.synchronize()
    want = a.double() @ w.double().T
    assert int(status[0]) == 0 and begin.elapsed_time(end) < 10
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isinf(), want.isinf())
    size = a.abs().double().nan_to_num(0, 0, 0) @ w.abs().double().nan_to_num(0, 0, 0).T
    assert ((out.double() - want).abs() <= (K + 1) * 2.0**-24 * size)[out.isfinite()].all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,T,N,K", [(torch.bfloat16, 61, 2048, 8192), (torch.bfloat16, 20, 2045, 4096), (torch.float32, 1, 300, 64),
                                         (torch.float32, 3, 260, 40), (torch.float32, 61, 2047, 1024), (torch.float32, 300, 512, 256)])
def test_scaled_sums_are_added_with_one_rounding(dtype, T, N, K):
    """Sums of products of -1, 0 and 1 are exact: what is left is the rounding of out + scale * sum (64 bits hold it but for about 2^-29 of
    the elements), one and not two.  In bf16 where CTAs share a tile's inner dimension."""
    mk = get_mk_module(name="mk_hybrid")
    gen = torch.Generator(device="cuda").manual_seed(T)
    pad = (K + 7) // 8 * 8
    a, w = (torch.randint(-1, 2, (rows, pad), generator=gen, device="cuda").to(dtype) for rows in (T, N))
    scale, out = torch.randn(N, generator=gen, device="cuda"), torch.randn(T, N, generator=gen, device="cuda")
    want = (out.double() + (a[:, :K].double() @ w[:, :K].double().T) * scale.double()).float()
    status = torch.zeros(16, dtype=torch.int32, device="cuda")
    mk.product("add", a, w, out, status, K, scale=scale)
    assert int(status[0]) == 0
    assert int((out != want).sum()) <= out.numel() * 1e-6
