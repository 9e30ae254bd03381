"""The native call path of the operators gives what their general form gives: the same kernels on the same bytes, so the
same bits.  A float32 or strided activation (bf16 values either way) is what the native path hands over to the general one;
a spy on the module says which of the two a call took."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["fp4", "affine"])
def bank(request):
    import cachalot_b200 as cb

    fmt = cb.FP4_FORMAT if request.param == "fp4" else cb.affine_format(512, 384)
    b = cb.SlabBank(fmt, 512, 384, 16, layers=2, n_experts=8)
    b.fill_random(torch.Generator(device="cuda").manual_seed(1))
    return b


class Spy:
    """The native module with a note of every call: did it take it?"""

    def __init__(self, module):
        self.module, self.took = module, []

    def __getattr__(self, name):
        def call(*args):
            y = getattr(self.module, name)(*args)
            self.took.append(y is not None)
            return y
        return call


@pytest.fixture
def spy(monkeypatch):
    from cachalot_b200 import ops

    s = Spy(ops._host)
    monkeypatch.setattr(ops, "_host", s)
    return s


def _fp8(n, k, rule, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = (torch.randn((n, k), device="cuda", generator=g) * 64).to(torch.float8_e4m3fn).view(torch.uint8)
    if rule == "e8m0":
        return w, torch.randint(112, 116, (-(-n // 32), k // 32), device="cuda", generator=g).to(torch.uint8)
    return w, torch.rand((-(-n // 128), k // 128), device="cuda", generator=g) * 1e-3


def _x(*shape):
    return torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)).to(torch.bfloat16)


@pytest.mark.parametrize("rule", ["e8m0", "f32"])
@pytest.mark.parametrize("rows", [None, 1, 3])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_fp8_linear(spy, rule, rows, dtype):
    import cachalot_b200 as cb

    x = _x(384) if rows is None else _x(rows, 384)
    w, s = _fp8(200, 384, rule, 3)
    assert torch.equal(cb.fp8_linear(x, w, s, out_dtype=dtype), cb.fp8_linear(x.float(), w, s, out_dtype=dtype))
    assert spy.took == [True, False]


@pytest.mark.parametrize("rows", [None, 1, 9])
def test_bf16_gemv(spy, rows):
    import cachalot_b200 as cb

    x = _x(320) if rows is None else _x(rows, 320)
    w = _x(77, 320)
    assert torch.equal(cb.bf16_gemv_f32(x.float(), w), cb.bf16_gemv_f32(x, w))
    assert spy.took == [True, False]


@pytest.mark.parametrize("rows", [1, 3, 9])
def test_moe_forward(bank, spy, rows):
    import cachalot_b200 as cb

    x = _x(rows, bank.hidden)
    slots = torch.arange(rows * 4, device="cuda", dtype=torch.int32).reshape(rows, 4) % 16
    w = torch.rand((rows, 4), device="cuda")
    assert torch.equal(cb.moe_forward(x, slots, w, bank), cb.moe_forward(x.float(), slots.long(), w, bank))
    assert spy.took == [True, False]


@pytest.mark.parametrize("want", [False, True])
def test_layer_decode(bank, spy, want):
    import cachalot_b200 as cb

    x, logits, bias = _x(bank.hidden), torch.randn(8, device="cuda"), torch.randn(8, device="cuda")
    a = cb.moe_layer_decode(x, logits, bank, layer=1, topk=3, bias=bias, want_routing=want)
    b = cb.moe_layer_decode(x.float(), logits, bank, layer=1, topk=3, bias=bias, want_routing=want)
    for u, v in zip(a if want else [a], b if want else [b]):
        assert torch.equal(u, v)
    assert spy.took == [True, False]


@pytest.mark.parametrize("mx", [0, 1])
def test_prefill(bank, spy, mx):
    import cachalot_b200 as cb

    x, ids = _x(37, bank.hidden), torch.randint(0, 8, (37, 2), device="cuda", dtype=torch.int32)
    w = torch.rand((37, 2), device="cuda")
    a = cb.moe_prefill_grouped(x, ids, w, bank, layer=1, mxfp4_act=mx)
    assert torch.equal(a, cb.moe_prefill_grouped(x.float(), ids, w, bank, layer=1, mxfp4_act=mx))
    assert spy.took == [True, False]


@pytest.mark.parametrize("rule", ["e8m0", "f32"])
@pytest.mark.parametrize("fused13", [False, True])
def test_block(bank, spy, rule, fused13):
    import cachalot_b200 as cb

    h, i = bank.hidden, 256
    (w1, s1), (w3, s3), (w2, s2) = _fp8(i, h, rule, 4), _fp8(i, h, rule, 5), _fp8(h, i, rule, 6)
    if fused13:
        w1, s1, w3, s3 = torch.cat([w1, w3]), torch.cat([s1, s3]), None, None
    x, gate, bias = _x(h), _x(8, h), torch.randn(8, device="cuda")
    kw = dict(layer_id=1, gate_weight=gate, gate_bias=bias, expert_store=bank, shared_w1=w1, shared_w1_scales=s1, shared_w2=w2,
              shared_w2_scales=s2, shared_w3=w3, shared_w3_scales=s3, topk=3)
    (a, ra), (b, rb) = cb.moe_layer_forward(x, **kw), cb.moe_layer_forward(x.float(), **kw)
    assert spy.took == [True, False, False]  # the general form hands x to the layer's operator as it is
    spy.took.clear()
    assert torch.equal(a, b) and torch.equal(ra.indices, rb.indices) and torch.equal(ra.weights, rb.weights) and torch.equal(ra.scores, rb.scores)
    y = cb.shared_expert_forward_batched(_x(5, h), w1=w1, w1_scales=s1, w3=w3, w3_scales=s3, w2=w2, w2_scales=s2)
    assert torch.equal(y, cb.shared_expert_forward_batched(_x(5, h).float(), w1=w1, w1_scales=s1, w3=w3, w3_scales=s3, w2=w2, w2_scales=s2))
    assert spy.took == [True, False]


def test_refused_arguments(bank, spy):
    """What the kernels do not take gets the general form's exception."""
    import cachalot_b200 as cb

    x, slots, w = _x(3, bank.hidden), torch.zeros((3, 2), device="cuda", dtype=torch.int32), torch.rand((3, 2), device="cuda")
    for bad in ((x[:, :-1], slots, w), (x, slots[:2], w), (x, slots, w[:, :1]), (x.cpu(), slots, w)):
        with pytest.raises(ValueError):
            cb.moe_forward(*bad, bank)
    with pytest.raises(KeyError):
        cb.moe_forward(x, slots, w, bank, out_dtype=torch.float16)
    logits = torch.randn(8, device="cuda")
    for kw in (dict(topk=0), dict(topk=9), dict(bias=torch.zeros(7, device="cuda"))):
        with pytest.raises(ValueError):
            cb.moe_layer_decode(x[0], logits, bank, **kw)
    m, s = _fp8(200, 384, "e8m0", 3)
    for bad in ((_x(3, 352), m, s), (_x(3, 384), m, s[:6]), (_x(2, 3, 384), m, s)):
        with pytest.raises(ValueError):
            cb.fp8_linear(*bad)
    assert spy.took and not any(spy.took)


def test_numbers_beyond_32_bits_are_refused(bank):
    """Not cut to their low bits on the way to the C ABI."""
    import cachalot_b200 as cb

    x, logits = _x(bank.hidden), torch.randn(8, device="cuda")
    with pytest.raises(ValueError, match="Invalid topk"):
        cb.moe_layer_decode(x, logits, bank, topk=2 ** 32 + 3)
    ids, w = torch.zeros((4, 2), device="cuda", dtype=torch.int32), torch.rand((4, 2), device="cuda")
    with pytest.raises(IndexError):
        cb.moe_prefill_grouped(_x(4, bank.hidden), ids, w, bank, layer=2 ** 32)


def test_other_threads_run_while_a_call_waits_for_the_gpu():
    """A 2-bit batch with bf16 scales is one launch per token: thousands of them fill the launch queue, and the call waits
    there.  The interpreter's lock is not held meanwhile."""
    import threading
    import time

    import cachalot_b200 as cb

    bank = cb.SlabBank(cb.affine_format(2048, 768, 2, 128, "bfloat16"), 2048, 768, 4)
    bank.fill_random(torch.Generator(device="cuda").manual_seed(1))
    rows = 6000
    x, slots, w = _x(rows, 2048), torch.zeros((rows, 2), dtype=torch.int32, device="cuda"), torch.rand((rows, 2), device="cuda")
    cb.moe_forward(x[:4], slots[:4], w[:4], bank)
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.0005)

    th = threading.Thread(target=tick)
    th.start()
    try:
        t0 = time.perf_counter()
        out = cb.ops._host.moe_forward(x, slots, w, bank.slab, cb.ops.addressof(bank.desc), 10.0, bank.default_numerics, cb.ops._ODT[torch.float32], None)
        t1 = time.perf_counter()
    finally:
        stop.set()
        th.join()
    torch.cuda.synchronize()
    assert out is not None and t1 - t0 > 0.02, f"the call returned after {t1 - t0:.4f} s: too short to say anything"
    assert sum(t0 + 0.005 < t < t1 - 0.005 for t in ticks) >= 3
