"""GPU parity of the grouped f16 tensor-core kernels (several tokens over a 2-bit bank) against the float64 oracle: rows of w2
that start in mid-group, tiles and stages that end early, units of 1 to 64 rows and experts of 65 and more, absent experts,
more routed rows than one plan takes; and which calls go there instead of token by token.  Groups of 64 and hidden sizes off
128 run on the one-warp kernels; a few of them are here too.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle import affine, configs  # noqa: E402
from tests.helpers import bf16_tensor, make_bank, within_bf16_flips  # noqa: E402


def _bank(rng, hidden, inter, n_exp, group):
    import cachalot_b200 as cb

    experts = []
    for _ in range(n_exp):
        e = {}
        for p, (n, k) in (("w1", (inter, hidden)), ("w2", (hidden, inter)), ("w3", (inter, hidden))):
            groups = n * k // group
            s = (rng.uniform(0.5, 1.5, groups) / np.sqrt(k)).astype(np.float16)
            e[f"{p}.weight"] = affine.pack_bits(rng.integers(0, 4, (n, k), dtype=np.uint8), 2)
            e[f"{p}.scales"] = s
            e[f"{p}.biases"] = (-1.5 * s.astype(np.float32) + rng.normal(0, 0.2, groups) / np.sqrt(k)).astype(np.float16)
        experts.append(e)
    return experts, make_bank(experts, cb.affine_format(hidden, inter, 2, group), hidden, inter)


def _want(x, slots, w, experts, group):
    out = np.zeros(x.shape, np.float32)
    for t in range(x.shape[0]):
        for j in range(slots.shape[1]):
            if slots[t, j] >= 0:
                out[t] += affine.affine_expert_forward(x[t], experts[slots[t, j]], bits=2, group_size=group, weight=w[t, j], swiglu_limit=10.0,
                                                       acc=np.float64)
    return out


@pytest.mark.parametrize("hidden,inter,group", [(128, 64, 64), (256, 192, 128), (512, 320, 64), (1088, 448, 128), (640, 2880, 128),
                                               (384, 64, 128), (512, 320, 128), (1152, 448, 128)])
@pytest.mark.parametrize("tokens", [6, 17, 66])  # six: the fewest that go to these kernels at all shapes that they take
def test_batch(hidden, inter, group, tokens):
    import torch

    import cachalot_b200 as cb

    rng = np.random.default_rng(hidden + inter + tokens)
    experts, bank = _bank(rng, hidden, inter, 5, group)
    x = configs.round_bf16((rng.standard_normal((tokens, hidden)) * np.exp(rng.uniform(-6, 6, (tokens, 1)))).astype(np.float32))
    # expert 0 takes every token (66: a unit of 64 and one of 2), the others some, one route slot in seven is absent
    slots = np.stack([np.zeros(tokens, np.int32), rng.integers(1, 5, tokens, dtype=np.int32)], 1)
    slots[::7, 1] = -1
    w = rng.uniform(0.1, 1.0, slots.shape).astype(np.float32)
    want = _want(x, slots, w, experts, group)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    args = (bf16_tensor(x), torch.from_numpy(slots).cuda(), torch.from_numpy(w).cuda(), bank)
    got = cb.moe_forward(*args, status=status)
    assert int(status.item()) == 0
    for t in range(tokens):  # rows differ in size: each against its own largest value
        assert within_bf16_flips(got[t].cpu().numpy(), want[t]), f"token {t}"
    assert torch.equal(cb.moe_forward(*args, out_dtype=torch.bfloat16), got.to(torch.bfloat16))


@pytest.mark.parametrize("hidden,inter,group", [(640, 2880, 128), (1152, 320, 128), (4096, 2880, 128), (5120, 2304, 128), (384, 576, 128)])
def test_stages_with_one_operand_slot(hidden, inter, group):
    """Inter of 4i+1 steps of 64 codes, one group-sum stage or two, and the sizes of whole banks, three to five shared-memory
    stages, several units per CTA: no warp may come late to a stage that only the other half of the unpacking warps works on."""
    import torch

    import cachalot_b200 as cb

    rng = np.random.default_rng(hidden + group)
    experts, bank = _bank(rng, hidden, inter, 3, group)
    tokens = 500
    x = configs.round_bf16(rng.standard_normal((tokens, hidden)).astype(np.float32))
    slots = np.stack([rng.permutation(3)[:2] for _ in range(tokens)]).astype(np.int32)
    w = rng.uniform(0.1, 1.0, slots.shape).astype(np.float32)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    args = (bf16_tensor(x), torch.from_numpy(slots).cuda(), torch.from_numpy(w).cuda(), bank)
    got = cb.moe_forward(*args, status=status)
    for _ in range(20):
        assert torch.equal(cb.moe_forward(*args, status=status), got)
    assert int(status.item()) == 0
    some = [0, 255, tokens - 1]
    assert within_bf16_flips(got[some].cpu().numpy(), _want(x[some], slots[some], w[some], experts, group))


@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("tokens,experts,grouped", [(32, 128, False), (512, 128, True)])
def test_prefill_scratch(tokens, experts, grouped, general):
    """A chunk that goes token by token takes the scratch of that route only; a grouped one two buffers of 16-bit rows."""
    import torch

    import cachalot_b200 as cb

    hidden, inter, k = 4096, 2880, 6
    bank = cb.SlabBank(cb.affine_format(hidden, inter), hidden, inter, experts, layers=1, n_experts=experts)
    bank.fill_random(torch.Generator(device="cuda").manual_seed(1))
    x = torch.randn((tokens, hidden), device="cuda").to(torch.bfloat16)
    ids = torch.rand((tokens, experts), device="cuda").topk(k, 1).indices.to(torch.int32)
    w = torch.rand((tokens, k), device="cuda")
    args = (x.float() if general else x, ids, w, bank)
    cb.ops._workspaces.clear()
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    # bytes asked for: a block that the allocator hands out again may be up to 1 MiB larger than the request
    before = torch.cuda.memory_stats()["requested_bytes.all.current"]
    out = cb.moe_prefill_grouped(*args)
    used = torch.cuda.memory_stats()["requested_bytes.all.peak"] - before - out.numel() * 4 - (x.numel() * 2 if general else 0)
    rows = tokens * k
    need = rows * 2 * (hidden + 128 + hidden) if grouped else rows * inter * 4
    assert used <= need + rows * 64 + (1 << 18), f"{used} bytes for {rows} rows"  # + per-row plans, per-expert counts


def test_infinite_and_nan_activations():
    """An infinite or NaN activation does to its row, and to no other, what it does in the one-token kernel.  All biases of
    these banks are negative: -inf drives gate and up to +inf, which the clamp makes finite again, as it does NaN; +inf ends
    as NaN."""
    import torch

    import cachalot_b200 as cb

    rng = np.random.default_rng(11)
    experts, bank = _bank(rng, 512, 320, 3, 128)
    assert all((e[f"{p}.biases"] < 0).all() for e in experts for p in ("w1", "w3"))
    x = rng.standard_normal((24, 512)).astype(np.float32)
    x[1, 70], x[2, 511], x[3, 0], x[4, [3, 300]], x[5] = -np.inf, np.inf, np.nan, -np.inf, x[5] * 1e30
    xt = bf16_tensor(x)
    slots = torch.from_numpy(np.stack([rng.permutation(3)[:2] for _ in range(24)]).astype(np.int32)).cuda()
    w = torch.rand((24, 2), device="cuda") + 0.1
    got = cb.moe_forward(xt, slots, w, bank).cpu().numpy()
    want = torch.cat([cb.moe_forward(xt[i:i + 1], slots[i:i + 1], w[i:i + 1], bank) for i in range(24)]).cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.isnan(want[2]).all() and np.isfinite(want[[0, 1, 3, 4, 5]]).all()
    for t in (1, 3, 4, 5):  # every expert's output is one bf16 rounding away from the other kernel's, at most one step
        assert np.abs(got[t] - want[t]).max() < 2.0 ** -7 * np.abs(want[t]).max(), f"token {t}"
    xt[1:6] = 1.0
    assert np.array_equal(cb.moe_forward(xt, slots, w, bank).cpu().numpy()[6:], got[6:])


@pytest.mark.parametrize("hidden,inter,tokens,k,n_slots,grouped", [
    (4096, 2880, 192, 6, 384, False),  # two runs of 576 rows, over up to 384 experts each: 2.5 ms a run against 2.2 token by token
    (1024, 512, 192, 6, 64, True), (1024, 512, 3, 1, 1, False), (1024, 512, 6, 1, 1, True), (2048, 768, 4, 4, 16, False)])
def test_route_of_a_batch(hidden, inter, tokens, k, n_slots, grouped):
    """Where one run of the grouped kernels (at most 1024 routed rows) does not pay for the experts it may touch, a batch goes
    token by token: the same bits as one call per token, which the grouped kernels' sums do not have."""
    import torch

    import cachalot_b200 as cb

    g = torch.Generator(device="cuda").manual_seed(tokens)
    bank = cb.SlabBank(cb.affine_format(hidden, inter), hidden, inter, n_slots)
    bank.fill_random(g)
    x = torch.randn((tokens, hidden), device="cuda", generator=g).to(torch.bfloat16)
    slots = torch.rand((tokens, n_slots), device="cuda", generator=g).topk(k, 1).indices.to(torch.int32)
    w = torch.rand((tokens, k), device="cuda", generator=g) + 0.1
    got = cb.moe_forward(x, slots, w, bank)
    one = torch.cat([cb.moe_forward(x[i:i + 1], slots[i:i + 1], w[i:i + 1], bank) for i in range(tokens)])
    assert torch.equal(got, one) != grouped


def test_more_rows_than_one_plan():
    import torch

    import cachalot_b200 as cb

    rng = np.random.default_rng(7)
    experts, bank = _bank(rng, 256, 128, 3, 128)
    x = configs.round_bf16(rng.standard_normal((1100, 256)).astype(np.float32))
    slots = rng.integers(0, 3, (1100, 1), dtype=np.int32)
    w = rng.uniform(0.1, 1.0, slots.shape).astype(np.float32)
    got = cb.moe_forward(bf16_tensor(x), torch.from_numpy(slots).cuda(), torch.from_numpy(w).cuda(), bank).cpu().numpy()
    assert within_bf16_flips(got, _want(x, slots, w, experts, 128))


@pytest.mark.parametrize("hidden,inter,group", [(256, 192, 128), (1152, 448, 128)])
def test_units(hidden, inter, group):
    """Experts of 1, 16, 17, 63, 64, 65 and 129 rows: units that end at, before and behind the sixteens of a tile's loads, and
    one, two and three units of an expert."""
    import torch

    import cachalot_b200 as cb

    rng = np.random.default_rng(group)
    counts = [1, 16, 17, 63, 64, 65, 129]
    experts, bank = _bank(rng, hidden, inter, len(counts), group)
    slots = rng.permutation(np.repeat(np.arange(len(counts), dtype=np.int32), counts))[:, None]
    x = configs.round_bf16(rng.standard_normal((len(slots), hidden)).astype(np.float32))
    w = rng.uniform(0.1, 1.0, slots.shape).astype(np.float32)
    got = cb.moe_forward(bf16_tensor(x), torch.from_numpy(slots).cuda(), torch.from_numpy(w).cuda(), bank).cpu().numpy()
    want = _want(x, slots, w, experts, group)
    for e in range(len(counts)):
        mine = slots[:, 0] == e
        assert within_bf16_flips(got[mine], want[mine]), f"expert of {counts[e]} rows"


@pytest.mark.parametrize("scale_dtype,group,hidden,k,small", [("bfloat16", 128, 1024, 3, False), ("float16", 64, 1024, 3, False),
                                                               ("float16", 128, 1088, 3, False), ("float16", 128, 1024, 9, False),
                                                               ("float16", 128, 1024, 3, True)])
def test_where_the_kernels_do_not_apply(scale_dtype, group, hidden, k, small):
    """A bank with bf16 scales, and a chunk that gets only the scratch of the token-by-token route (what a caller that sized it
    before the grouped kernels came hands over): the bits of one call per token.  Groups of 64, hidden sizes off 128 and more
    than eight experts per token, where the one-token kernel does not run either: the accuracy of the one-warp kernels."""
    import ctypes

    import torch

    import cachalot_b200 as cb
    from cachalot_b200 import _lib

    inter, tokens, n = 512, 40, 12
    g = torch.Generator(device="cuda").manual_seed(5)
    bank = cb.SlabBank(cb.affine_format(hidden, inter, 2, group, scale_dtype), hidden, inter, n, layers=1, n_experts=n)
    bank.fill_random(g)
    x = torch.randn((tokens, hidden), device="cuda", generator=g).to(torch.bfloat16)
    ids = torch.rand((tokens, n), device="cuda", generator=g).topk(k, 1).indices.to(torch.int32)
    w = torch.rand((tokens, k), device="cuda", generator=g) + 0.1
    one = torch.cat([cb.moe_forward(x[i:i + 1], ids[i:i + 1], w[i:i + 1], bank) for i in range(tokens)])
    if not small:
        batch, chunk = cb.moe_forward(x, ids, w, bank), cb.moe_prefill_grouped(x, ids, w, bank)
        if scale_dtype == "bfloat16":
            assert torch.equal(batch, one) and torch.equal(chunk, one)
        else:
            assert torch.equal(chunk, cb.moe_forward(x, ids, w, bank, simple=True))
            if group == 64:
                assert torch.equal(batch, chunk)
        return
    assert not torch.equal(cb.moe_prefill_grouped(x, ids, w, bank), one)  # with room it takes the grouped kernels
    up = lambda v: -(-v // 256) * 256  # noqa: E731
    need = up(tokens * k * inter * 4) + up(tokens * k * 4)
    perm, offsets = cb.group_rows(ids, n)
    out, status = torch.zeros((tokens, hidden), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ws = torch.empty(need + 256, dtype=torch.uint8, device="cuda")
    call = lambda size: _lib.lib.cachalot_moe_prefill(  # noqa: E731
        bank.slab.data_ptr(), ctypes.byref(bank.desc), x.data_ptr(), perm.data_ptr(), offsets.data_ptr(), bank.slot_table[0].data_ptr(),
        w.data_ptr(), tokens, k, n, 10.0, 0, up(ws.data_ptr()), size, out.data_ptr(), status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert call(need - 1) == _lib.ESCRATCH
    assert call(need) == _lib.OK
    assert torch.equal(out, one) and int(status.item()) == 0


@pytest.mark.parametrize("tokens", [5, 200])
def test_prefill(tokens):
    import torch

    import cachalot_b200 as cb

    rng = np.random.default_rng(tokens)
    experts, bank = _bank(rng, 384, 320, 8, 128)
    bank.slot_table[0, 3] = -1
    x = configs.round_bf16(rng.standard_normal((tokens, 384)).astype(np.float32))
    ids = np.stack([rng.permutation(8)[:3] for _ in range(tokens)]).astype(np.int32)
    w = rng.uniform(0.1, 1.0, ids.shape).astype(np.float32)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = cb.moe_prefill_grouped(bf16_tensor(x), torch.from_numpy(ids).cuda(), torch.from_numpy(w).cuda(), bank, status=status).cpu().numpy()
    assert int(status.item()) == 0
    assert within_bf16_flips(got, _want(x, np.where(ids == 3, -1, ids), w, experts, 128))


def test_accumulation_is_exact_on_integers():
    """Weights -1, 0, 1, 2 and small integer activations: every sum is a whole number below 2**24, so gate and up come out
    exactly and an identity-like down projection shows them to the last bit."""
    import torch

    import cachalot_b200 as cb

    rng = np.random.default_rng(3)
    hidden, inter = 256, 128
    e = {}
    lev = {"w1": np.zeros((inter, hidden), np.uint8), "w3": rng.integers(0, 4, (inter, hidden), dtype=np.uint8),
           "w2": np.where(np.eye(hidden, inter, dtype=np.uint8) > 0, 2, 1).astype(np.uint8)}
    lev["w1"][:] = 1
    lev["w1"][:, 0] = 3  # gate = 2 x[0] = 64 for every unit
    for p, n in (("w1", inter * hidden), ("w2", inter * hidden), ("w3", inter * hidden)):
        e[f"{p}.weight"] = affine.pack_bits(lev[p], 2)
        e[f"{p}.scales"], e[f"{p}.biases"] = np.ones(n // 128, np.float16), -np.ones(n // 128, np.float16)
    bank = make_bank([e], cb.affine_format(hidden, inter), hidden, inter)
    x = rng.integers(-3, 4, (9, hidden)).astype(np.float32)
    x[:, 0] = 32
    u = configs.round_bf16(x @ (lev["w3"].astype(np.float32) - 1).T)
    want = np.zeros((9, hidden), np.float32)
    want[:, :inter] = configs.round_bf16(np.float32(64) * u)
    got = cb.moe_forward(bf16_tensor(x), torch.zeros((9, 1), dtype=torch.int32, device="cuda"), torch.ones((9, 1), device="cuda"), bank,
                         swiglu_limit=0.0).cpu().numpy()
    assert np.array_equal(got, want)
