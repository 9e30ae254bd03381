"""FP8 linears of more than eight tokens against the streaming GEMV (one token at a time, itself checked against the oracle):
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


@pytest.mark.parametrize("rule", ["e8m0", "f32"])
@pytest.mark.parametrize("k", [1536, 8192])
@pytest.mark.parametrize("rows", [32, 64, 300])
def test_fp32_sums_as_accurate_as_few_tokens(rule, k, rows):
    """The error of the fp32 results against float64 over 2**13 outputs and more is no larger than that of the streaming GEMV
    (eight tokens at a time), which adds K in slices; a single running sum over K = 8192 has twice its error."""
    import torch

    import cachalot_b200 as cb

    n, block = 256, 32 if rule == "e8m0" else 128
    g = torch.Generator(device="cuda").manual_seed(k + rows)
    w = (torch.randn((n, k), device="cuda", generator=g) * 64).to(torch.float8_e4m3fn).view(torch.uint8)
    if rule == "e8m0":
        s = torch.randint(112, 118, (n // 32, k // 32), device="cuda", generator=g).to(torch.uint8)
        s64 = torch.ldexp(torch.ones(s.shape, device="cuda", dtype=torch.float64), s.double() - 127)
    else:
        s = (torch.rand((n // 128, k // 128), device="cuda", generator=g) + 0.5) * 1e-3
        s64 = s.double()
    x = torch.randn((rows, k), device="cuda", generator=g).to(torch.bfloat16)
    q = cb.quantize_fp8_activation(x, block, rule)
    x64 = q.values.view(torch.float8_e4m3fn).double() * q.scales.double().repeat_interleave(block, 1)
    want = x64 @ (w.view(torch.float8_e4m3fn).double() * s64.repeat_interleave(block, 0).repeat_interleave(block, 1)).T
    err = lambda y: float((y.double() - want).norm() / want.norm())  # noqa: E731
    many = err(cb.fp8_linear(x, w, s, out_dtype=torch.float32))
    few = err(torch.cat([cb.fp8_linear(x[i:i + 8], w, s, out_dtype=torch.float32) for i in range(0, rows, 8)]))
    assert many <= 1.05 * few, f"{many:.3e} against {few:.3e}"  # the figure itself spreads by about 1 % over 8192 outputs


@pytest.mark.parametrize("rows", [17, 300])
def test_infinite_activations(rows):
    """An infinite activation makes its row's results infinite or NaN exactly where one token at a time makes them so."""
    import torch

    import cachalot_b200 as cb

    g = torch.Generator(device="cuda").manual_seed(rows)
    w = (torch.randn((200, 1024), device="cuda", generator=g) * 64).to(torch.float8_e4m3fn).view(torch.uint8)
    s = torch.rand((2, 8), device="cuda", generator=g) * 1e-3 + 1e-4
    x = torch.randn((rows, 1024), device="cuda", generator=g).to(torch.bfloat16)
    x[1, 3], x[rows - 1, 1000] = float("inf"), float("-inf")
    got = cb.fp8_linear(x, w, s, out_dtype=torch.float32)
    want = torch.cat([cb.fp8_linear(x[i:i + 1], w, s, out_dtype=torch.float32) for i in range(rows)])
    assert bool((torch.isinf(want[1]) | torch.isnan(want[1])).any())
    bad = ~torch.isfinite(want)
    assert torch.equal(~torch.isfinite(got), bad)
    assert torch.equal(torch.nan_to_num(got[bad], nan=7.0), torch.nan_to_num(want[bad], nan=7.0))


@pytest.mark.parametrize("rows,n,k,per_lane", [(9, 4096, 1024, True), (16, 4096, 1024, True), (32, 1024, 1024, True), (32, 4736, 512, True),
                                               (17, 4800, 512, False), (33, 200, 416, False), (80, 200, 416, False), (300, 130, 1024, False)])
@pytest.mark.parametrize("rule", ["e8m0", "f32"])
def test_weights_off_sixteen_bytes(rows, n, k, per_lane, rule):
    """Rows that are not 16-byte aligned always take the kernel that splits K over warps.  Up to 16 tokens, and up to 32 of a
    matrix whose 32-row CTAs fit on the SMs at once, aligned rows take it too (the GEMM needs up to three times as long
    there): the same bits.  Other calls differ by the order of the fp32 sums."""
    import torch

    import cachalot_b200 as cb

    if rule == "f32" and k % 128:
        pytest.skip("blocks of 128")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert per_lane == (rows <= 16 or (rows <= 32 and -(-n // 32) <= sms)), "the sizes are chosen for 148 SMs"
    g = torch.Generator(device="cuda").manual_seed(n + k + rows)
    w = (torch.randn((n, k), device="cuda", generator=g) * 64).to(torch.float8_e4m3fn).view(torch.uint8)
    off = torch.empty(n * k + 8, dtype=torch.uint8, device="cuda")[8:].view(n, k)
    off.copy_(w)
    assert w.data_ptr() % 16 == 0 and off.data_ptr() % 16 == 8
    if rule == "e8m0":
        s = torch.randint(112, 118, (-(-n // 32), k // 32), device="cuda", generator=g).to(torch.uint8)
    else:
        s = (torch.rand((-(-n // 128), k // 128), device="cuda", generator=g) + 0.1) * 1e-3
    x = torch.randn((rows, k), device="cuda", generator=g).to(torch.bfloat16)
    a, b = cb.fp8_linear(x, w, s, out_dtype=torch.float32), cb.fp8_linear(x, off, s, out_dtype=torch.float32)
    if per_lane:
        assert torch.equal(a, b)
    else:  # as in test_rows_match_single_tokens
        assert bool(((a - b).abs() <= 4 * k * 2.0 ** -24 * b.abs().amax(1, keepdim=True)).all())
