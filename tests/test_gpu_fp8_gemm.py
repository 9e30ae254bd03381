"""The tiled FP8 GEMM (more than eight tokens) against the streaming GEMV (one token at a time, itself checked against the oracle):
the same products summed in fp32 in another order, at sizes that end inside a tile, a K step and a scale block row; weights
that hold the two NaN codes, which read as zero."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,rule", [(16, 32, "e8m0"), (200, 96, "e8m0"), (129, 416, "e8m0"), (384, 1184, "e8m0"), (130, 128, "f32"), (300, 640, "f32")])
@pytest.mark.parametrize("rows", [9, 32, 33, 64, 65, 300])
@pytest.mark.parametrize("nan", [False, True])
def test_rows_match_single_tokens(n, k, rule, rows, nan):
    import torch

    import cachalot_b200 as cb

    g = torch.Generator(device="cuda").manual_seed(n + k + rows)
    w = (torch.randn((n, k), device="cuda", generator=g) * 64).to(torch.float8_e4m3fn).view(torch.uint8)
    if nan:
        w[n // 2, k // 3], w[0, 0] = 0x7F, 0xFF
    if rule == "e8m0":
        s = torch.randint(112, 118, (-(-n // 32), k // 32), device="cuda", generator=g).to(torch.uint8)
    else:
        s = (torch.rand((-(-n // 128), k // 128), device="cuda", generator=g) + 0.1) * 1e-3
    x = (torch.randn((rows, k), device="cuda", generator=g) * torch.rand((rows, 1), device="cuda", generator=g).mul(8).exp()).to(torch.bfloat16)
    got = cb.fp8_linear(x, w, s, out_dtype=torch.float32)
    want = torch.cat([cb.fp8_linear(x[i:i + 1], w, s, out_dtype=torch.float32) for i in range(rows)])
    assert bool(torch.isfinite(got).all())
    # k products summed in fp32: k * 2**-24 of the sum of magnitudes, itself at most sqrt(k) times a row's largest output here
    bound = 4 * k * 2.0 ** -24 * want.abs().amax(1, keepdim=True)
    assert bool(((got - want).abs() <= bound).all())
    # bf16 results: the fp32 ones rounded, one step apart where the sum order moved a value over a boundary
    b = cb.fp8_linear(x, w, s).float()
    assert bool(((b - got).abs() <= got.abs() * 2.0 ** -8 + 1e-30).all())
