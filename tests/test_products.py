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
    a[:, K:], w[:, K:] = (0, 0) if dtype == torch.bfloat16 else (float("nan"), float("nan"))  # (float rows: read, dropped)
    w /= K**0.5
    status = torch.zeros(16, dtype=torch.int32, device="cuda")
    sums = a[:, :K].double() @ w[:, :K].double().T
    size = (a[:, :K].double().abs() @ w[:, :K].double().abs().T)
    kw = {}
    if result == "store":
        kw["bias"] = torch.randn(N, generator=gen, device="cuda")
        out, want = torch.full((T, N), float("nan"), device="cuda"), sums + kw["bias"].double()
    elif result == "add":
        kw["scale"] = torch.randn(N, generator=gen, device="cuda")
        out = torch.randn(T, N, generator=gen, device="cuda")
        want = out.double() + sums * kw["scale"].double()
    elif result == "cast":
        out, want = torch.full((T, (N + 7) // 8 * 8), float("nan"), device="cuda", dtype=dtype), sums
    elif result == "glu":
        kw.update(limit=1.5, alpha=1.7)
        g, u = sums[:, ::2].clamp(max=1.5), sums[:, 1::2].clamp(-1.5, 1.5)
        out, want = torch.full((T, N // 2), float("nan"), device="cuda", dtype=dtype), g * torch.sigmoid(1.7 * g) * (u + 1)
    else:
        kw["w2"] = make(N) / K**0.5
        out = torch.full((T, (N + 7) // 8 * 8), float("nan"), device="cuda", dtype=dtype)
        want = sums * torch.sigmoid(sums) * (a[:, :K].double() @ kw["w2"][:, :K].double().T)
    mk.product(result, a, w, out, status, K, **kw)
    again = out.clone() if result != "add" else None
    if again is not None:  # the same bits whatever the order of arrival
        mk.product(result, a, w, out, status, K, **kw)
        assert torch.equal(out[:, : want.shape[1]], again[:, : want.shape[1]])
    assert int(status[0]) == 0
    if result in ("cast", "silu"):
        assert torch.isnan(out[:, N:]).all()  # nothing beyond the features is written
    return out[:, : want.shape[1]].double(), want, size


@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K", SHAPES)
@pytest.mark.parametrize("result", ["store", "add", "cast", "glu", "silu"])
def test_bf16_products(result, T, N, K):
    """32-bit sums of exact products (K 2^-24 of the sum of magnitudes at the very most), then one rounding
    to bf16 (2^-9) where that is the result; the gated units' slopes are below 4 here."""
    if result == "glu" and N % 2:
        N += 1
    out, want, size = product(result, torch.bfloat16, T, N, K)
    bound = 4 * K * 2.0**-24 * (size[:, : want.shape[1]].max() + 1) * (1 + (want.abs().max() if result == "silu" else 0))
    if result in ("cast", "glu", "silu"):
        bound = bound + want.abs() * 2.0**-8
    assert ((out - want).abs() <= bound).all(), float((out - want).abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K", SHAPES)
@pytest.mark.parametrize("result", ["store", "add", "cast", "glu"])
def test_float32_products(result, T, N, K):
    """fp32 FMA throughout: far below what bf16 or tf32 operands would give (2^-9, 2^-11)."""
    if result == "glu" and N % 2:
        N += 1
    out, want, size = product(result, torch.float32, T, N, K)
    assert ((out - want).abs() <= 4 * K * 2.0**-24 * (size.max() + 1)).all()
    assert float((out - want).norm() / want.norm()) < 2e-6
