"""Each kernel alone against a plain 32-bit torch reference of the same operation, at sizes
other than the engine's tiny configurations: odd widths, tails of tiles, head sizes in steps
of 16, grouped heads, windows, page edges."""

from __future__ import annotations

import math
from types import SimpleNamespace

import pytest
import torch
import torch.nn.functional as F

import plain_gpt

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]


@pytest.fixture(scope="module")
def ops():
    from mini_gpt_inference_b200.kernels.ops import default_ops

    return default_ops("cuda:0")


def _tol(dtype, scale=1.0):
    return (2e-5 if dtype == torch.float32 else 1.6e-2) * scale


def randn(*shape, dtype=torch.float32, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(dtype).cuda()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width,vocab", [(96, 509), (520, 1000), (33, 77)])
def test_embed(ops, dtype, width, vocab):
    tok, pos = randn(vocab, width, dtype=dtype, seed=1), randn(300, width, dtype=dtype, seed=2)
    ids = torch.randint(0, vocab, (45,), dtype=torch.int32).cuda()
    positions = torch.randint(0, 300, (45,), dtype=torch.int32).cuda()
    got = ops.embed(ids, positions, tok, pos)
    want = tok.float()[ids.long()] + pos.float()[positions.long()]
    assert got.dtype == torch.float32 and torch.equal(got, want)
    assert torch.equal(ops.embed(ids, positions, tok, None), tok.float()[ids.long()])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows,width,eps,bias", [(7, 96, 3e-4, False), (130, 520, 1e-5, True),
                                                 (1, 33, 1e-2, True), (64, 2048, 1e-5, True)])
def test_layernorm(ops, dtype, rows, width, eps, bias):
    x = randn(rows, width, seed=3, scale=3.0) + 1.5          # a mean far from zero
    gain = randn(width, seed=4) + 1.0
    shift = randn(width, seed=5) if bias else None
    got = ops.layernorm(x, gain, shift, eps, dtype)
    want = F.layer_norm(x.double(), (width,), gain.double(), None if shift is None else shift.double(), eps)
    assert got.dtype == dtype
    assert (got.double() - want).abs().max() <= _tol(dtype, 4.0)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("m,n,k", [(1, 509, 96), (45, 200, 96), (130, 96, 200), (64, 1536, 512),
                                   (3, 77, 33), (257, 65, 129), (8, 50304, 512), (300, 2048, 512),
                                   (2048, 512, 2048), (17, 1536, 512), (33, 512, 2048),
                                   (65, 1536, 512), (128, 128, 64), (129, 130, 72), (16, 16, 8)])
def test_linear_and_epilogues(ops, dtype, m, n, k):
    x = randn(m, k, dtype=dtype, seed=6)
    w = randn(n, k, dtype=dtype, seed=7, scale=1 / math.sqrt(k))
    b = randn(n, seed=8)
    ref = x.double() @ w.double().T
    assert (ops.linear(x, w, None, "none", dtype).double() - ref).abs().max() <= _tol(dtype, 3)
    assert (ops.linear(x, w, b, "none", dtype).double() - (ref + b.double())).abs().max() <= _tol(dtype, 3)
    gelu = plain_gpt.gelu_tanh(ref + b.double())
    assert (ops.linear(x, w, b, "gelu_tanh", dtype).double() - gelu).abs().max() <= _tol(dtype, 3)
    logits = ops.logits(x, w)
    assert logits.dtype == torch.float32
    assert (logits.double() - ref).abs().max() <= 2e-5        # inputs exact, 32-bit sums and output
    res = randn(m, n, seed=9)
    before = res.clone()
    ops.linear_residual(x, w, b, res)
    assert (res.double() - (before.double() + ref + b.double())).abs().max() <= 3e-5
    ops.check_status()


def test_tensor_core_and_cuda_core_products_agree(ops):
    """The tcgen05 path and the plain FMA path compute the same sums from the same bfloat16
    inputs; with 32-bit output they differ only by the order of the additions."""
    # (the last shape has enough tiles for the 128 x 256 variant of the tensor-core kernel)
    for m, n, k in [(5, 300, 512), (200, 136, 200), (64, 50304, 512), (1000, 1536, 512), (4200, 4800, 328)]:
        x = randn(m, k, dtype=torch.bfloat16, seed=11)
        w = randn(n, k, dtype=torch.bfloat16, seed=12, scale=1 / math.sqrt(k))
        ops.use_tensor_cores = True
        before = ops.launches
        fast = ops.logits(x, w)
        ops.use_tensor_cores = False
        slow = ops.logits(x, w)
        ops.use_tensor_cores = True
        assert ops.launches == before + 2
        assert (fast - slow).abs().max() <= 1e-5, (m, n, k)
    ops.check_status()


def test_tensor_core_tiles_of_256_columns_with_every_epilogue(ops):
    """Steps of thousands of tokens on a large matrix take tiles of 128 x 256: bias, GELU with a
    bfloat16 store, the residual add and the QKV projection's page write must come out as from the
    plain FMA kernel (the same bfloat16 inputs, sums in another order)."""
    m, k = 4300, 200
    n_head, n_kv, d, pt = 40, 20, 64, 16                    # 5120 columns: 34 x 20 tiles of 256
    n = (n_head + 2 * n_kv) * d
    x = randn(m, k, dtype=torch.bfloat16, seed=41)
    w = randn(n, k, dtype=torch.bfloat16, seed=42, scale=1 / math.sqrt(k))
    b = randn(n, seed=43)
    res = randn(m, n, seed=44)
    pages = -(-m // pt) + 2
    slots = torch.randperm(pages * pt)[:m].to(torch.int32)
    slots[7] = -1
    slots = slots.cuda()

    def run():
        cache = SimpleNamespace(k_pages=torch.zeros(pages, n_kv, pt, d, dtype=torch.bfloat16).cuda(),
                                v_pages=torch.zeros(pages, n_kv, pt, d, dtype=torch.bfloat16).cuda(),
                                page_tokens=pt, writes=True)
        r = res.clone()
        ops.linear_residual(x, w, b, r)
        return (ops.linear(x, w, b, "gelu_tanh", torch.bfloat16).float(), r,
                ops.linear_qkv(x, w, b, n_head, n_kv, d, cache, slots, torch.bfloat16).float(), cache)

    before = ops.launches
    fast = run()
    assert ops.launches == before + 3, "each call was expected to be one tensor-core launch"
    ops.use_tensor_cores = False
    try:
        slow = run()
    finally:
        ops.use_tensor_cores = True
    def one_bf16_step(a, c):
        # results rounded to bfloat16 may land on neighbouring values where a sum lies at a rounding
        # edge (a step is 2^-7 of the value's power of two), never further apart
        return bool(((a - c).abs() <= 2.0 ** -7 * c.abs().clamp(min=2.0 ** -6)).all())

    assert one_bf16_step(fast[0], slow[0])
    assert (fast[1] - slow[1]).abs().max() <= 1e-5          # 32-bit sums in another order
    assert one_bf16_step(fast[2], slow[2])
    for a, c in ((fast[3].k_pages, slow[3].k_pages), (fast[3].v_pages, slow[3].v_pages)):
        assert one_bf16_step(a.float(), c.float())
    # keys of token i lie where its slot says, bit for bit what the projection returned
    qkv = ops.linear_qkv(x, w, b, n_head, n_kv, d, fast[3], slots, torch.bfloat16)
    tok = 100
    s_ = int(slots[tok])
    assert torch.equal(fast[3].k_pages[s_ // pt, :, s_ % pt].reshape(-1), qkv[tok, n_head * d: (n_head + n_kv) * d])
    ops.check_status()


def _sum_bound(x, w):
    """How far 32-bit sums of x @ w.T in steps of 16 terms can be off: a rounding (of up to 2^-23) of what is there per step."""
    return 2.0 ** -23 * math.ceil(x.shape[1] / 16) * (x.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("m,n,k,pairs,blocks", [
    (129, 8200, 64, 1, 1), (2049, 4804, 200, 1, 1), (1100, 8192, 1032, 1, 1), (700, 8203, 72, 1, 1), (5000, 2056, 136, 1, 1),
    (257, 9, 8, 1, 1), (130, 519, 200, 1, 2),
    (129, 4800, 3072, 2, 2), (129, 4801, 3080, 2, 2), (777, 6144, 2048, 2, 1), (777, 6147, 2056, 2, 1), (500, 6148, 2048, 2, 1)])
def test_tensor_core_tiles_by_one_cta_and_by_pairs(ops, m, n, k, pairs, blocks):
    """Sizes on both sides of the rule that cuts a product into tiles (CTAs a tile, k blocks a stage): one tile a CTA and several
    (two accumulators in turn), a last tile of few columns, a pair whose second CTA has one row, rows that TMA cannot store (n no
    multiple of 4 or 8)."""
    import ctypes

    cut = [ctypes.c_int() for _ in range(3)]
    for out_bf16 in (0, 1):
        ops.lib.mg_linear_tc_cut(m, n, k, out_bf16, *[ctypes.byref(c) for c in cut])
        assert (cut[0].value, cut[2].value) == (pairs, blocks)
    x = randn(m, k, dtype=torch.bfloat16, seed=21)
    w = randn(n, k, dtype=torch.bfloat16, seed=22, scale=1 / math.sqrt(k))
    b = randn(n, seed=23)
    ref = x.double() @ w.double().T + b.double()
    off = _sum_bound(x, w) + 2.0 ** -23 * (ref.abs() + b.double().abs())
    for act, fn, slope in (("none", lambda t: t, 1.0), ("gelu_tanh", plain_gpt.gelu_tanh, 1.13),
                           ("relu_sq", lambda t: t.clamp_min(0) ** 2, 2 * ref.abs() + 1.0)):
        want = fn(ref)
        got = ops.linear(x, w, b, act, torch.bfloat16).double()
        # half a unit in the last place, 2^-8, and the hardware's tanh in whole columns of prompts, 2^-10.9 of one
        tanh_off = 2.0 ** -11.9 * ref.abs() if act == "gelu_tanh" and m > 128 and n % 8 == 0 else 0.0
        assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1.01 * (slope * off + tanh_off)).all(), act
        got = ops.linear(x, w, b, act, torch.float32).double()
        assert ((got - want).abs() <= 2.0 ** -22 * (want.abs() + ref.abs()) + slope * off).all(), act
    res = randn(m, n, seed=24)
    got = res.clone()
    ops.linear_residual(x, w, b, got)
    assert ((got.double() - res.double() - ref).abs() <= off + 2.0 ** -23 * (res.double().abs() + ref.abs())).all()
    ops.check_status()


def test_pairs_copy_keys_and_values_to_their_pages(ops):
    """777 tokens of 64 query and 16 key/value heads of 64 (pairs of CTAs, two rounds): every page row is what the projection
    returned, bit for bit; a token without a slot leaves the pages alone."""
    m, n_head, n_kv, d, pt, k = 777, 64, 16, 64, 32, 2048
    x = randn(m, k, dtype=torch.bfloat16, seed=1)
    w = randn((n_head + 2 * n_kv) * d, k, dtype=torch.bfloat16, seed=2, scale=1 / math.sqrt(k))
    b = randn((n_head + 2 * n_kv) * d, seed=3)
    pages = -(-m // pt) + 1
    slots = torch.randperm(pages * pt, generator=torch.Generator().manual_seed(4))[:m].to(torch.int32).cuda()
    slots[5] = slots[700] = -1
    cache = SimpleNamespace(k_pages=torch.zeros(pages, n_kv, pt, d, dtype=torch.bfloat16, device="cuda"),
                            v_pages=torch.zeros(pages, n_kv, pt, d, dtype=torch.bfloat16, device="cuda"), page_tokens=pt, writes=True)
    qkv = ops.linear_qkv(x, w, b, n_head, n_kv, d, cache, slots, torch.bfloat16)
    want = x.double() @ w.double().T + b.double()
    assert ((qkv.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1.01 * _sum_bound(x, w) + 1e-6).all()
    live = slots >= 0
    at = slots[live].long()
    for part, held in ((qkv[:, n_head * d: (n_head + n_kv) * d], cache.k_pages), (qkv[:, (n_head + n_kv) * d:], cache.v_pages)):
        assert torch.equal(held[at // pt, :, at % pt].reshape(len(at), -1), part[live])
        rest = torch.ones(pages * pt, dtype=torch.bool, device="cuda")
        rest[at] = False
        assert (held.transpose(1, 2).reshape(pages * pt, -1)[rest] == 0).all()
    ops.check_status()


@pytest.mark.parametrize("m", [8, 17, 64, 65, 128, 129, 700])
@pytest.mark.parametrize("n", [520, 2048, 2052])
def test_gelu_of_bfloat16_results_is_right_to_its_last_place(ops, m, n):
    """Also where it is nearly zero: the products are exact here (one term each), so a result is the rounding of GELU(u).
    Only the whole columns of prompts take the hardware's tanh."""
    x, w = torch.zeros(m, 64), torch.zeros(n, 64)
    x[:, 0], w[:, 0] = 1.0 + torch.arange(m) / 128.0, torch.linspace(-4.0, 4.0, n)
    x, w = x.to(torch.bfloat16).cuda(), w.to(torch.bfloat16).cuda()
    u = x.double() @ w.double().T
    # 2^-8 from rounding (and 2^-15 before it); the kernels of few tokens use tanhf, which is off by up to two units in the last
    # place: below one 2^-24 each, halved by the formula, so |u| 2^-24, and as much again for what its argument (2^-22 of it)
    # and 1 + tanh are off; the hardware's tanh is off by up to 2^-10.98 of one
    want = 0.5 * u * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (u + 0.044715 * u ** 3)))
    tanh_off = 2.0 ** -10.9 if m > 128 and n % 8 == 0 else 2.0 ** -22
    got = ops.linear(x, w, None, "gelu_tanh", torch.bfloat16).double()
    assert ((got - want).abs() <= 2.0 ** -7.99 * want.abs() + 0.5 * tanh_off * u.abs()).all()
    ops.check_status()


@pytest.mark.parametrize("m", [1, 2, 3, 5, 8, 11, 16])
@pytest.mark.parametrize("n,k", [(1536, 512), (512, 2048), (509, 96), (50304, 512), (200, 200), (77, 40)])
def test_small_batch_projection_with_fused_norm(ops, m, n, k):
    """Up to 16 tokens take the weight-streaming kernel; with a deferred LayerNorm (and a row
    gather) fused into its prologue it must agree with the separate kernels."""
    x32 = randn(m + 3, k, seed=21, scale=2.0) + 0.5
    rows = torch.tensor([(3 * i + 1) % (m + 3) for i in range(m)], dtype=torch.int32).cuda()
    gain, shift = randn(k, seed=22) + 1.0, randn(k, seed=23)
    w = randn(n, k, dtype=torch.bfloat16, seed=24, scale=1 / math.sqrt(k))
    b = randn(n, seed=25)
    want = torch.nn.functional.layer_norm(x32[rows.long()].double(), (k,), gain.double(), shift.double(), 1e-5)
    want = want.to(torch.bfloat16).double() @ w.double().T + b.double()
    before = ops.launches
    fused = ops.linear(ops.defer_layernorm(x32, gain, shift, 1e-5, torch.bfloat16, rows), w, b, "none",
                       torch.float32)
    assert ops.launches == before + 1, "norm, gather and projection were expected in one kernel"
    assert (fused.double() - want).abs().max() <= 2e-2       # bf16 rounding of the normalised rows
    ops.use_skinny = False
    try:
        apart = ops.linear(ops.defer_layernorm(x32, gain, shift, 1e-5, torch.bfloat16, rows), w, b, "none",
                           torch.float32)
    finally:
        ops.use_skinny = True
    assert (fused - apart).abs().max() <= 2e-5               # same bf16 inputs, 32-bit sums
    res = randn(m, n, seed=26)
    keep = res.clone()
    y = ops.layernorm(ops.gather_rows(x32, rows), gain, shift, 1e-5, torch.bfloat16)
    ops.linear_residual(y, w, b, res)
    assert (res.double() - (keep.double() + want)).abs().max() <= 2e-2
    g = ops.linear(y, w, b, "gelu_tanh", torch.bfloat16)
    assert (g.double() - plain_gpt.gelu_tanh(want)).abs().max() <= 5e-2
    ops.check_status()


@pytest.mark.parametrize("m,c,f,bias", [(1, 512, 2048, True), (8, 512, 2048, True), (16, 512, 2048, True),
                                        (9, 512, 2048, False), (5, 96, 200, False), (3, 64, 256, True),
                                        (11, 768, 3072, True), (8, 1600, 6400, True), (2, 192, 520, True),
                                        (7, 40, 24, True), (16, 1024, 72, False)])
def test_whole_feed_forward_in_one_kernel(ops, m, c, f, bias):
    """LayerNorm, fc, tanh-GELU and proj of up to 16 tokens as one kernel that adds partial products
    of slices of the inner dimension into a zeroed buffer: against the formula (with the same
    roundings to bfloat16 as the two-kernel path) and against that path; three times in a row, so
    that the three buffers have taken every role."""
    x = randn(m, c, seed=41, scale=2.0) + 0.3
    gain, shift = randn(c, seed=42) + 1.0, (randn(c, seed=43) if bias else None)
    w1 = randn(f, c, dtype=torch.bfloat16, seed=44, scale=1 / math.sqrt(c))
    w2 = randn(c, f, dtype=torch.bfloat16, seed=45, scale=1 / math.sqrt(f))
    b1, b2 = (randn(f, seed=46), randn(c, seed=47)) if bias else (None, None)

    def formula(xin):
        y = F.layer_norm(xin.double(), (c,), gain.double(), None if shift is None else shift.double(), 1e-5)
        h = y.to(torch.bfloat16).double() @ w1.double().T + (b1.double() if bias else 0)
        h = plain_gpt.gelu_tanh(h).to(torch.bfloat16).double()
        return xin.double() + h @ w2.double().T + (b2.double() if bias else 0)

    before = ops.launches
    if c > 512:
        # wider than the fused kernel takes: the two projections run, in place
        keep = x.clone()
        same = ops.mlp_residual(ops.defer_layernorm(x, gain, shift, 1e-5, torch.bfloat16), w1, b1, w2, b2,
                                "gelu_tanh", x, torch.bfloat16)
        assert same is x and ops.launches == before + 2
        want = formula(keep)
        assert (same.double() - want).abs().max() <= 2e-2 * max(1.0, float(want.abs().max()))
        return
    first = ops.mlp_residual(ops.defer_layernorm(x, gain, shift, 1e-5, torch.bfloat16), w1, b1, w2, b2,
                             "gelu_tanh", x, torch.bfloat16)
    assert first is not x, "the fused kernel was expected to run and hand back another buffer"
    assert ops.launches == before + 2                      # the zero fill of the first call, and the kernel
    want = formula(x)
    scale = max(1.0, float(want.abs().max()))
    assert (first.double() - want).abs().max() <= 2e-2 * scale   # a hidden value at a bfloat16 rounding edge
    second = ops.mlp_residual(ops.defer_layernorm(first, gain, shift, 1e-5, torch.bfloat16), w1, b1, w2, b2,
                              "gelu_tanh", first, torch.bfloat16)
    assert ops.launches == before + 3 and second is not first and second is not x
    assert (second.double() - formula(first)).abs().max() <= 2e-2 * scale
    third = ops.mlp_residual(ops.defer_layernorm(second, gain, shift, 1e-5, torch.bfloat16), w1, b1, w2, b2,
                             "gelu_tanh", second, torch.bfloat16)
    assert third is x and ops.launches == before + 4         # the first buffer's turn again
    assert (third.double() - formula(second)).abs().max() <= 2e-2 * scale
    # the two-kernel path from the same input
    x2 = second.clone()
    ops.use_fused_mlp = False
    try:
        apart = ops.mlp_residual(ops.defer_layernorm(x2, gain, shift, 1e-5, torch.bfloat16), w1, b1, w2, b2,
                                 "gelu_tanh", x2, torch.bfloat16)
    finally:
        ops.use_fused_mlp = True
    assert apart is x2
    assert (apart - third).abs().max() <= 1e-2 * scale
    ops.check_status()


@pytest.mark.parametrize("m", [17, 24, 32, 33, 50, 64, 65, 96, 100, 128])
@pytest.mark.parametrize("n,k", [(1536, 512), (512, 2048), (509, 96), (200, 200), (77, 40), (2048, 4096),
                                 (6400, 1600), (4800, 1600), (5003, 520)])
def test_mid_batch_projection_over_a_cluster(ops, monkeypatch, m, n, k):
    """17 to 128 tokens: every epilogue of whichever kernel the rule gives the size to, against the formula; and up to 64
    tokens the kernel that cuts K over the CTAs of a cluster (partial sums met through distributed shared memory) beside
    the tensor-core GEMM."""
    x = randn(m, k, dtype=torch.bfloat16, seed=31)
    w = randn(n, k, dtype=torch.bfloat16, seed=32, scale=1 / math.sqrt(k))
    b = randn(n, seed=33)
    want = x.double() @ w.double().T + b.double()
    before = ops.launches
    got = ops.linear(x, w, b, "none", torch.float32)
    assert ops.launches == before + 1
    assert (got.double() - want).abs().max() <= 2e-4
    if m <= 64:
        rule, sums = type(ops)._cluster_pays, []
        for pays in (True, False):
            monkeypatch.setattr(type(ops), "_cluster_pays", staticmethod(lambda m, n, k, pays=pays: pays))
            sums.append(ops.linear(x, w, b, "none", torch.float32))
        monkeypatch.setattr(type(ops), "_cluster_pays", staticmethod(rule))
        assert torch.equal(got, sums[0 if rule(m, n, k) else 1])
        assert (sums[0] - sums[1]).abs().max() <= 1e-4        # same bf16 inputs, 32-bit sums
        if n > 200 and k > 200:                               # (two kernels: where sums are long, some differ in their last bit)
            assert not torch.equal(sums[0], sums[1])
    res = randn(m, n, seed=34)
    keep = res.clone()
    ops.linear_residual(x, w, b, res)
    assert (res.double() - (keep.double() + want)).abs().max() <= 2e-4
    gl = ops.linear(x, w, None, "gelu_tanh", torch.bfloat16)
    assert (gl.double() - plain_gpt.gelu_tanh(want - b.double())).abs().max() <= 3e-2
    ops.check_status()


@pytest.mark.parametrize("m,n,k", [(64, 2048, 512), (40, 6400, 1600), (33, 8192, 256)])
def test_mid_batch_projection_without_the_tensor_core_gemm(ops, monkeypatch, m, n, k):
    """With the tensor-core GEMM switched off, sizes that the rule gives to it go to the cluster kernel, not to the plain one."""
    x, w = randn(m, k, dtype=torch.bfloat16, seed=35), randn(n, k, dtype=torch.bfloat16, seed=36, scale=1 / math.sqrt(k))
    assert not ops._cluster_pays(m, n, k)
    monkeypatch.setattr(ops, "use_tensor_cores", False)
    got = ops.linear(x, w, None, "none", torch.float32)
    out = torch.empty(m, n, device="cuda")
    code = ops.lib.mg_linear_cluster(x.data_ptr(), w.data_ptr(), None, out.data_ptr(), None, m, n, k, 0, 0, None, None, None, 0, 0, 0,
                                     0, 0, torch.cuda.current_stream().cuda_stream)
    assert code == 0 and torch.equal(got, out)
    assert (got.double() - x.double() @ w.double().T).abs().max() <= 2e-4


@pytest.mark.parametrize("m", [1, 5, 8, 16, 24, 33, 64])
@pytest.mark.parametrize("vocab,k,limit", [(50304, 512, None), (50304, 512, 50257), (509, 96, 300), (77, 40, None),
                                           (9001, 200, 9000)])
def test_greedy_choice_on_the_way_of_the_head_projection(ops, m, vocab, k, limit):
    """The head's projection may leave the argmax of every row while it writes the logits: it
    must be the argmax of exactly those logits (lowest index among equals, ids at or above the
    limit never), whichever kernel runs."""
    x32 = randn(m + 2, k, seed=61, scale=1.5)
    rows = torch.tensor([(3 * i + 1) % (m + 2) for i in range(m)], dtype=torch.int32).cuda()
    gain, shift = randn(k, seed=62) + 1.0, randn(k, seed=63)
    w = randn(vocab, k, dtype=torch.bfloat16, seed=64, scale=1 / math.sqrt(k))
    w[vocab // 2] = w[3]                                        # equal logits: the lower index must win
    w[vocab - 1] = w[3]
    ids = torch.full((m,), -1, dtype=torch.int32, device="cuda")
    y = ops.defer_layernorm(x32, gain, shift, 1e-5, torch.bfloat16, rows)
    logits, taken = ops.logits(y, w, ids, limit)
    if not taken:
        ids = ops.argmax(logits, limit)
    assert taken == (m <= 16), "up to 16 rows the projection takes the choice on its way"
    masked = logits.clone()
    if limit is not None:
        masked[:, limit:] = -float("inf")
    want = masked.argmax(-1)
    best = masked.max(-1).values
    first = (masked == best[:, None]).float().argmax(-1)      # lowest index among equal maxima
    assert torch.equal(ids.long(), first), (ids, want)
    plain = ops.logits(y, w)
    assert torch.equal(plain, logits), "the logits themselves must not change"
    ops.check_status()


@pytest.mark.parametrize("m", [3, 16, 24, 64])
def test_streaming_projection_of_a_wide_matrix_takes_up_to_64_rows(ops, m):
    """The kernel that streams a wide matrix through shared memory is used for up to 16 rows; it
    takes 64, checked here by raising the limit."""
    from mini_gpt_inference_b200.kernels import ops as ops_module

    n, k = 9001, 200
    x = randn(m, k, dtype=torch.bfloat16, seed=71)
    w = randn(n, k, dtype=torch.bfloat16, seed=72, scale=1 / math.sqrt(k))
    b = randn(n, seed=73)
    want = x.double() @ w.double().T + b.double()
    was = ops_module.STREAM_ROWS
    ops_module.STREAM_ROWS = 64
    ops.use_wide = False                                     # (the kernel of tiled copies takes 16 rows; this one is meant)
    try:
        ids = torch.full((m,), -1, dtype=torch.int32, device="cuda")
        got = ops.linear(x, w, b, "none", torch.float32)
        logits, taken = ops.logits(x, w, ids, 9000)
    finally:
        ops_module.STREAM_ROWS = was
        ops.use_wide = True
    assert taken
    assert (got.double() - want).abs().max() <= 2e-4
    masked = logits.clone()
    masked[:, 9000:] = -float("inf")
    assert torch.equal(ids.long(), masked.argmax(-1))
    ops.check_status()


@pytest.mark.parametrize("wide", [True, False], ids=["tiles", "rows"])
@pytest.mark.parametrize("m", [1, 5, 8, 13, 16])
@pytest.mark.parametrize("n,k", [(640, 1600), (203, 6400), (9001, 1608), (77, 3080), (4800, 1600), (1600, 6400)])
def test_streamed_projection_of_long_rows(ops, m, n, k, wide):
    """Large matrices are streamed: as boxes of whole rows by TMA through a ring (rows of a multiple
    of 64 and up to 2048 values; longer ones only for the residual epilogue, K cut over CTAs whose
    partial sums are added in L2), or, where that kernel refuses, row by row in K chunks (a tile's
    sums stay in registers from chunk to chunk); with the LayerNorm prologue: one launch, and the
    same numbers as the separate kernels."""
    x32 = randn(m + 3, k, seed=81, scale=2.0) + 0.5
    rows = torch.tensor([(3 * i + 1) % (m + 3) for i in range(m)], dtype=torch.int32).cuda()
    gain, shift = randn(k, seed=82) + 1.0, randn(k, seed=83)
    w = randn(n, k, dtype=torch.bfloat16, seed=84, scale=1 / math.sqrt(k))
    b = randn(n, seed=85)
    want = torch.nn.functional.layer_norm(x32[rows.long()].double(), (k,), gain.double(), shift.double(), 1e-5)
    want = want.to(torch.bfloat16).double() @ w.double().T + b.double()
    flags = (ops.stream_min_bytes, ops.stream_max_chunks, ops.use_skinny, ops.use_cluster, ops.use_wide)
    ops.stream_min_bytes, ops.stream_max_chunks, ops.use_skinny, ops.use_cluster = 0, 1 << 20, False, False
    ops.use_wide = wide
    # 16 rows of 6400 values leave no room for stages beside them: refused, other kernels take it
    fits = (8 if m <= 8 else 16) * (2 * k + 64) + 8 * k + 8 * 4 * 8 * (2 * 64 + 64) <= 226 * 1024
    if wide:
        fits = fits or k <= 2048                              # the tiled kernel stages rows of up to 2048 values
    try:
        before = ops.launches
        fused = ops.linear(ops.defer_layernorm(x32, gain, shift, 1e-5, torch.bfloat16, rows), w, b, "none",
                           torch.float32)
        assert (ops.launches == before + 1) == fits, "norm, gather and projection in one streaming kernel"
        y = ops.layernorm(ops.gather_rows(x32, rows), gain, shift, 1e-5, torch.bfloat16)
        streamed = ops.linear(y, w, b, "none", torch.float32)
        g = ops.linear(y, w, b, "gelu_tanh", torch.bfloat16)
        res = randn(m, n, seed=86)
        keep = res.clone()
        ops.linear_residual(y, w, b, res)
        ops.use_stream = ops.use_wide = False
        apart = ops.linear(y, w, b, "none", torch.float32)
    finally:
        ops.stream_min_bytes, ops.stream_max_chunks, ops.use_skinny, ops.use_cluster, ops.use_wide = flags
        ops.use_stream = True
    assert (fused.double() - want).abs().max() <= 2e-2       # bf16 rounding of the normalised rows
    assert (fused - streamed).abs().max() <= 2e-5             # the fused norm rounds as the stand-alone kernel
    assert (streamed - apart).abs().max() <= 2e-5             # same bf16 inputs, 32-bit sums
    assert (res.double() - (keep.double() + want)).abs().max() <= 2e-2
    assert (g.double() - plain_gpt.gelu_tanh(want)).abs().max() <= 5e-2
    ops.check_status()


@pytest.mark.parametrize("m,vocab,k,limit", [(1, 50304, 512, None), (8, 50257, 1600, 50000), (16, 9001, 192, 9000),
                                             (3, 777, 64, None), (13, 50257, 1024, None)])
def test_large_matrix_kernel_takes_the_greedy_choice_on_its_way(ops, m, vocab, k, limit):
    """The head through the kernel of tiled copies: 32-bit logits, and the first stage of the greedy
    argmax in its epilogue (lowest index among equal maxima, ids at or above the limit excluded)."""
    x = randn(m, k, dtype=torch.bfloat16, seed=75)
    w = randn(vocab, k, dtype=torch.bfloat16, seed=76, scale=1 / math.sqrt(k))
    w[vocab // 2] = w[7]                                     # a tie between two rows
    flags = (ops.stream_min_bytes, ops.use_stream, ops.use_skinny)
    ops.stream_min_bytes, ops.use_stream, ops.use_skinny = 0, False, False
    try:
        ids = torch.full((m,), -1, dtype=torch.int32, device="cuda")
        before = ops.launches
        logits, taken = ops.logits(x, w, ids, limit)
        assert taken and ops.launches == before + 2          # the projection and the merge of its candidates
    finally:
        ops.stream_min_bytes, ops.use_stream, ops.use_skinny = flags
    want = x.double() @ w.double().T
    assert (logits.double() - want).abs().max() <= 2e-5
    masked = logits.clone()
    if limit is not None:
        masked[:, limit:] = -float("inf")
    best = masked.max(-1).values
    first = (masked == best[:, None]).float().argmax(-1)     # lowest index among equal maxima
    assert torch.equal(ids.long(), first)
    ops.check_status()


def test_large_matrix_kernel_at_random_shapes(ops):
    """Shapes drawn at random (1 to 16 tokens, rows in multiples of 64 up to 4096, any number of
    weight rows, each epilogue, with and without bias and LayerNorm prologue): the cuts of the
    kernel of tiled copies (rows per box, slices of K, warps that own or share a box, bias kept in
    shared memory or not) against a 64-bit product."""
    import random

    rng = random.Random(5)
    flags = (ops.stream_min_bytes, ops.use_stream, ops.use_skinny, ops.use_cluster)
    ops.stream_min_bytes, ops.use_stream, ops.use_skinny, ops.use_cluster = 0, False, False, False
    taken = 0
    try:
        for case in range(40):
            m = rng.choice([1, 2, 3, 5, 8, 9, 13, 16])
            k = 64 * rng.choice([1, 2, 3, 5, 8, 12, 16, 17, 25, 32, 40, 64])
            n = rng.choice([8, 17, 64, 100, 333, 1024, 1601, 4099, 20011, 70001])
            epilogue = rng.choice(["none", "gelu_tanh", "residual"])
            prologue = rng.random() < 0.5 and k <= 2048
            with_bias = rng.random() < 0.7
            x32 = randn(m, k, seed=200 + case, scale=1.5) + 0.25
            gain, shift = randn(k, seed=300 + case) + 1.0, randn(k, seed=400 + case)
            w = randn(n, k, dtype=torch.bfloat16, seed=500 + case, scale=1 / math.sqrt(k))
            b = randn(n, seed=600 + case) if with_bias else None
            if prologue:
                xin = ops.defer_layernorm(x32, gain, shift, 1e-5, torch.bfloat16)
                xr = torch.nn.functional.layer_norm(x32.double(), (k,), gain.double(), shift.double(), 1e-5)
                xr = xr.to(torch.bfloat16).double()
            else:
                xin = x32.to(torch.bfloat16)
                xr = xin.double()
            want = xr @ w.double().T + (b.double() if with_bias else 0.0)
            before = ops.launches
            if epilogue == "residual":
                res = randn(m, n, seed=700 + case)
                keep = res.clone()
                if prologue:
                    xin = xin.materialize()
                ops.linear_residual(xin, w, b, res)
                got, want = res.double(), keep.double() + want
                tol = 2e-2 if prologue else 2e-4
            else:
                got = ops.linear(xin, w, b, epilogue, torch.float32).double()
                if epilogue == "gelu_tanh":
                    want = plain_gpt.gelu_tanh(want)
                tol = 2e-2 if prologue else 2e-4
            taken += int(ops.launches == before + 1)
            assert (got - want).abs().max() <= tol, (case, m, n, k, epilogue, prologue, with_bias)
    finally:
        ops.stream_min_bytes, ops.use_stream, ops.use_skinny, ops.use_cluster = flags
    assert taken >= 25, "most of these shapes are the kernel's own (the others it refuses: other kernels run)"
    ops.check_status()


def test_large_matrix_kernel_asks_for_the_matrix_that_followed_it_last_time(ops):
    """The kernel for large matrices asks the weights of the projection that came next the last
    time into L2 (a hint learned from the order of the calls): results do not change with it, and
    a matrix that is gone is not asked for."""
    import gc

    m, n, k = 8, 4800, 1600
    x = randn(m, k, dtype=torch.bfloat16, seed=95)
    w1 = randn(n, k, dtype=torch.bfloat16, seed=96, scale=1 / math.sqrt(k))
    w2 = randn(n, k, dtype=torch.bfloat16, seed=97, scale=1 / math.sqrt(k))
    want1 = x.double() @ w1.double().T
    first = ops.linear(x, w1, None, "none", torch.float32)                # nothing is known to follow w1 yet
    ops.linear(x, w2, None, "none", torch.float32)
    assert ops._next_weight[w1.data_ptr()]() is w2
    again = ops.linear(x, w1, None, "none", torch.float32)                # asks for w2 on its way
    assert torch.equal(first, again) and (first.double() - want1).abs().max() <= 2e-5
    del w2
    gc.collect()
    assert ops._next_weight[w1.data_ptr()]() is None
    once_more = ops.linear(x, w1, None, "none", torch.float32)            # the follower is gone: no hint
    assert torch.equal(first, once_more)
    ops.check_status()


@pytest.mark.parametrize("wide", [True, False], ids=["tiles", "rows"])
@pytest.mark.parametrize("m", [1, 8, 16])
def test_streamed_qkv_projection_writes_keys_and_values(ops, m, wide):
    """A QKV matrix of many megabytes is streamed as well; the epilogue of the streaming kernel
    copies key and value features to their cache rows like the other projection kernels."""
    n_head, n_kv, d, pt, k = 5, 5, 64, 16, 1600
    width = (n_head + 2 * n_kv) * d
    x = randn(m, k, dtype=torch.bfloat16, seed=91)
    w = randn(width, k, dtype=torch.bfloat16, seed=92, scale=1 / math.sqrt(k))
    b = randn(width, seed=93)
    pages = 6
    slots = torch.randperm(pages * pt)[:m].to(torch.int32)
    if m > 1:
        slots[0] = -1                                        # a padding row writes nothing
    slots = slots.cuda()
    cache = SimpleNamespace(k_pages=torch.zeros(pages, n_kv, pt, d, dtype=torch.bfloat16).cuda(),
                            v_pages=torch.zeros(pages, n_kv, pt, d, dtype=torch.bfloat16).cuda(),
                            page_tokens=pt, writes=True)
    flags = (ops.stream_min_bytes, ops.stream_max_chunks, ops.use_skinny, ops.use_cluster, ops.use_wide)
    ops.stream_min_bytes, ops.stream_max_chunks, ops.use_skinny, ops.use_cluster, ops.use_wide = 0, 1 << 20, False, False, wide
    try:
        before = ops.launches
        qkv = ops.linear_qkv(x, w, b, n_head, n_kv, d, cache, slots, torch.bfloat16)
        assert ops.launches == before + 1, "projection and page write were expected in one streaming kernel"
    finally:
        ops.stream_min_bytes, ops.stream_max_chunks, ops.use_skinny, ops.use_cluster, ops.use_wide = flags
    kk = qkv[:, n_head * d: (n_head + n_kv) * d].reshape(m, n_kv, d)
    vv = qkv[:, (n_head + n_kv) * d:].reshape(m, n_kv, d)
    want_k, want_v = torch.zeros_like(cache.k_pages), torch.zeros_like(cache.v_pages)
    for i, s_ in enumerate(slots.tolist()):
        if s_ >= 0:
            want_k[s_ // pt, :, s_ % pt] = kk[i]
            want_v[s_ // pt, :, s_ % pt] = vv[i]
    assert torch.equal(cache.k_pages, want_k) and torch.equal(cache.v_pages, want_v)
    ref = x.double() @ w.double().T + b.double()
    assert (qkv.double() - ref).abs().max() <= 5e-2
    ops.check_status()


@pytest.mark.parametrize("heads", [(6, 2, 32), (3, 1, 48)])
@pytest.mark.parametrize("m", [1, 4, 8, 9, 40, 70, 200, 333])
def test_qkv_projection_writes_keys_and_values_to_their_pages(ops, m, heads):
    # every projection kernel (small batch, mid batch, tensor cores) has the copy in its epilogue
    n_head, n_kv, d = heads
    pt, k = 8, 96
    pages = max(12, m // pt + 3)
    width = (n_head + 2 * n_kv) * d
    x = randn(m, k, dtype=torch.bfloat16, seed=31)
    w = randn(width, k, dtype=torch.bfloat16, seed=32, scale=0.1)
    b = randn(width, seed=33)
    slots = torch.randperm(pages * pt)[:m].to(torch.int32)
    slots[0] = -1                                            # a padding row writes nothing
    slots = slots.cuda()
    cache = SimpleNamespace(k_pages=torch.zeros(pages, n_kv, pt, d, dtype=torch.bfloat16).cuda(),
                            v_pages=torch.zeros(pages, n_kv, pt, d, dtype=torch.bfloat16).cuda(),
                            page_tokens=pt, writes=True)
    qkv = ops.linear_qkv(x, w, b, n_head, n_kv, d, cache, slots, torch.bfloat16)
    kk = qkv[:, n_head * d: (n_head + n_kv) * d].reshape(m, n_kv, d)
    vv = qkv[:, (n_head + n_kv) * d:].reshape(m, n_kv, d)
    want_k, want_v = torch.zeros_like(cache.k_pages), torch.zeros_like(cache.v_pages)
    for i, s_ in enumerate(slots.tolist()):
        if s_ >= 0:
            want_k[s_ // pt, :, s_ % pt] = kk[i]
            want_v[s_ // pt, :, s_ % pt] = vv[i]
    assert torch.equal(cache.k_pages, want_k) and torch.equal(cache.v_pages, want_v)
    ref = x.double() @ w.double().T + b.double()
    assert (qkv.double() - ref).abs().max() <= 5e-2


@pytest.mark.parametrize("n_head,d,dv,window,softcap", [(16, 576, 512, 200, 0.0), (24, 328, 264, 0, 20.0), (16, 704, 512, 0, 0.0)])
def test_wide_rows_of_long_prompts(ops, n_head, d, dv, window, softcap):
    """Key rows that hold their values, steps of so many rows that a CTA takes 64 (32 where 64 do not fit): as the general
    kernel has it, within the rounding of weights and outputs to bfloat16."""
    g = torch.Generator().manual_seed(d)
    lens, befores, pt = [901, 330], [0, 77], 16
    ends = [b + n for b, n in zip(befores, lens)]
    pages = sum(-(-e // pt) for e in ends) + 1
    order, tables = torch.randperm(pages, generator=g).tolist(), torch.full((2, 64), -1, dtype=torch.int32)
    rows = torch.full((pages, 1, pt, d), float("nan"))
    for r, e in enumerate(ends):
        for i in range(-(-e // pt)):
            tables[r, i] = page = order.pop()
            have = min(e - i * pt, pt)                # behind a request's last token: no numbers
            rows[page, 0, :have] = torch.randn(have, d, generator=g)
    pages_cuda = rows.to(torch.bfloat16).cuda()
    cache = SimpleNamespace(k_pages=pages_cuda, v_pages=pages_cuda, group=0, page_tokens=pt, window=window or None, writes=False,
                            values_in_keys=True)
    i32 = lambda v: torch.as_tensor(v, dtype=torch.int32).cuda()
    ctx = SimpleNamespace(block_tables=[tables.cuda()], positions=i32([b + i for b, n in zip(befores, lens) for i in range(n)]),
                          token_request=i32([r for r, n in enumerate(lens) for _ in range(n)]), decode_only=False,
                          max_ctx_after=max(ends), host_q_len=lens, req_q_len=i32(lens), req_q_start=i32([0, lens[0]]))
    q = (torch.randn(sum(lens), n_head * d, generator=g) * 1.5).to(torch.bfloat16).cuda()
    sink = torch.randn(n_head, generator=g).cuda()
    run = lambda: ops.paged_attention_general(q, n_head, 1, d, dv, d ** -0.5, cache, ctx, softcap=softcap, sinks=sink).float()
    before = ops.launches
    got = run()
    assert ops.launches == before + 1 and not torch.isnan(got).any()
    ops.use_mma_attention = False
    try:
        want = run()
    finally:
        ops.use_mma_attention = True
    assert (got - want).abs().max() <= _tol(torch.bfloat16, 1.5)
    assert (got - want).norm() <= 6e-3 * want.norm()      # two roundings of 2^-9 and one of the weights


@pytest.mark.parametrize("rows_are_inputs", [True, False])
@pytest.mark.parametrize("n,heads,n_in,n_out,gap", [(65, 3, 128, 512, 64), (300, 2, 64, 192, 8), (129, 16, 512, 128, 0)])
def test_heads_small_products_of_many_tokens(ops, n, heads, n_in, n_out, gap, rows_are_inputs):
    """Inputs and outputs of a head among other columns, which stay as they are; against 64 bits."""
    x = randn(n, heads * (n_in + gap) + 8, dtype=torch.bfloat16, seed=51)
    w = randn(heads * (n_in if rows_are_inputs else n_out), n_out if rows_are_inputs else n_in, dtype=torch.bfloat16, seed=52,
              scale=1 / math.sqrt(n_in))
    out = randn(n, heads * (n_out + gap) + 8, dtype=torch.bfloat16, seed=53)
    before, kept = ops.launches, out.clone()
    ops.head_linear(x, 8, n_in + gap, w, rows_are_inputs, heads, n_in, n_out, out=out, out_off=8, out_head=n_out + gap)
    assert ops.launches == before + 1
    mats = w.double().view(heads, n_in, n_out) if rows_are_inputs else w.double().view(heads, n_out, n_in).transpose(1, 2)
    ins = x[:, 8:].double().reshape(n, heads, n_in + gap)[..., :n_in]
    want = torch.einsum("nhi,hij->nhj", ins, mats)
    got = out[:, 8:].reshape(n, heads, n_out + gap)
    # half a unit in the last place of bfloat16, and 32-bit sums of up to 512 products
    assert ((got[..., :n_out].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()
    rest = kept[:, 8:].reshape(n, heads, n_out + gap)[..., n_out:]
    assert torch.equal(got[..., n_out:], rest) and torch.equal(out[:, :8], kept[:, :8])
    # the matrices are read as they are at the call: nothing of them is kept from one call for the next
    w.mul_(-2.0)
    again = ops.head_linear(x, 8, n_in + gap, w, rows_are_inputs, heads, n_in, n_out).view(n, heads, n_out)
    assert torch.equal(again, -2.0 * got[..., :n_out])
    ops.check_status()


@pytest.mark.parametrize("gated,activation,weigh_input", [(True, "silu", False), (False, "relu_sq", True)])
@pytest.mark.parametrize("n,width,inner,experts,top", [(65, 136, 200, 5, 2), (300, 264, 68 * 4, 3, 3), (700, 512, 384, 17, 2), (130, 72, 520, 200, 1)])
def test_experts_of_many_tokens(ops, monkeypatch, n, width, inner, experts, top, gated, activation, weigh_input):
    """Tiles over each expert's rows: experts without rows, rows that end inside a tile and inside a box of 32, widths that end
    inside a tile; against the products in 64 bits, hidden features rounded to bfloat16."""
    g = torch.Generator().manual_seed(n)
    y = randn(n, width, dtype=torch.bfloat16, seed=44)
    w_in = randn(experts, (2 if gated else 1) * inner, width, dtype=torch.bfloat16, seed=45, scale=1 / math.sqrt(width))
    w_out = randn(experts, width, inner, dtype=torch.bfloat16, seed=46, scale=1 / math.sqrt(inner))
    ids = torch.stack([torch.randperm(experts, generator=g)[:top] for _ in range(n)]).to(torch.int32)
    if experts > 3:
        ids[ids == 2] = 1                            # an expert without rows (a token may then have one expert twice)
    ids[7] = -1                                      # a padding row
    weights = torch.rand(n, top, generator=g).cuda()
    residual = randn(n, width, seed=47)
    want = residual.double()
    for e in range(experts):
        for t, k in (ids == e).nonzero().tolist():
            w = weights[t, k].double()
            z = w_in[e].double() @ y[t].double() * (w if weigh_input else 1.0)
            h = z[:inner] * torch.sigmoid(z[:inner]) * z[inner:] if gated else z.clamp_min(0) ** 2
            want[t] += w_out[e].double() @ h.to(torch.bfloat16).double() * (1.0 if weigh_input else w)
    monkeypatch.setattr(type(ops), "_moe_tc_pays", staticmethod(lambda *sizes: True))
    before = ops.launches
    ops.moe_experts_residual(y, ids.cuda(), weights, w_in, w_out, residual, activation, 0.0, gated, weigh_input)
    assert ops.launches == before + 5
    # here and there a hidden feature is rounded to the other neighbour: 2^-8 of it, times a weight of 1 / sqrt(inner)
    assert (residual.double() - want).abs().max() <= 2e-2
    assert (residual.double() - want).norm() <= 1e-3 * want.norm()
    ops.check_status()


@pytest.mark.parametrize("gated,activation,weigh_input", [(True, "silu", False), (True, "clamped_swish", False),
                                                          (False, "relu_sq", True), (False, "gelu_tanh", False)])
@pytest.mark.parametrize("n,width,inner,experts,top", [(1, 1024, 1024, 9, 3), (8, 136, 200, 5, 2), (9, 264, 72, 3, 3), (16, 1160, 24, 4, 4),
                                                       (16, 8, 8, 70, 5)])
@pytest.mark.parametrize("repeats", [False, True])
def test_experts_of_few_tokens(ops, monkeypatch, n, width, inner, experts, top, gated, activation, weigh_input, repeats):
    """Steps of up to 16 tokens: no further from the 64-bit result than the kernels of larger steps, at widths that end inside
    a warp's share of K and inside a CTA's rows, with up to 16 tokens an expert and padding rows; with tokens that name one
    expert several times (as a router's choice for a row of scores that are not numbers), up to 64 entries an expert."""
    g = torch.Generator().manual_seed(n * 31 + inner)
    y = randn(n, width, dtype=torch.bfloat16, seed=41)
    w_in = randn(experts, (2 if gated else 1) * inner, width, dtype=torch.bfloat16, seed=42, scale=1 / math.sqrt(width))
    w_out = randn(experts, width, inner, dtype=torch.bfloat16, seed=43, scale=1 / math.sqrt(inner))
    ids = torch.stack([torch.randperm(experts, generator=g)[:top] for _ in range(n)]).to(torch.int32)
    if n > 8:
        ids[5] = -1                                  # a padding row
    if repeats:
        ids[::2] = 0                                 # expert 0 alone, `top` times
        ids[1:4, 0] = 0
    weights = torch.rand(n, top, generator=g).cuda()
    ids = ids.cuda()

    def run():
        residual = torch.zeros(n, width, device="cuda")
        ops.moe_experts_residual(y, ids, weights, w_in, w_out, residual, activation, 7.0, gated, weigh_input)
        return residual.double()

    want = torch.zeros(n, width, dtype=torch.float64, device="cuda")
    for t in range(n):
        for k in range(top):
            e = int(ids[t, k])
            if e < 0:
                continue
            w = weights[t, k].double()
            z = w_in[e].double() @ y[t].double() * (w if weigh_input else 1.0)
            a, u = (z[:inner], z[inner:]) if gated else (z, None)
            if activation == "silu":
                h = a * torch.sigmoid(a) * u
            elif activation == "clamped_swish":
                a, u = a.clamp(max=7.0), u.clamp(-7.0, 7.0)
                h = a * torch.sigmoid(1.702 * a) * (u + 1.0)
            else:
                h = a.clamp_min(0) ** 2 if activation == "relu_sq" else plain_gpt.gelu_tanh(a)
            want[t] += w_out[e].double() @ h.to(torch.bfloat16).double() * (1.0 if weigh_input else w)
    monkeypatch.setattr(type(ops), "_moe_few_pays", staticmethod(lambda *sizes: True))
    before = ops.launches
    few = run()
    assert ops.launches == before + 3
    ops.use_moe_few = False
    try:
        tiles = run()
    finally:
        ops.use_moe_few = True
    # the hidden features are rounded to bfloat16 on both sides, here and there to the other neighbour
    assert (few - want).norm() <= 1.05 * (tiles - want).norm() + 1e-6 * want.norm()
    assert (few - want).abs().max() <= 2e-2


@pytest.mark.parametrize("n,width,inner,experts,top", [(4, 1024, 1024, 9, 3), (16, 264, 72, 3, 3), (1, 2048, 136, 8, 2)])
def test_experts_of_few_tokens_started_ahead(ops, monkeypatch, n, width, inner, experts, top):
    """In a captured step the second product's kernel starts, and reads the ids, before the first has ended.  Layer after layer, with ids
    that change from replay to replay (padding, experts without a token, all tokens at one expert): the bits of kernels that
    run one after the other."""
    g = torch.Generator().manual_seed(n + width)
    layers = 3
    y = randn(n, width, dtype=torch.bfloat16, seed=44)
    w_in = [randn(experts, 2 * inner, width, dtype=torch.bfloat16, seed=45 + i, scale=1 / math.sqrt(width)) for i in range(layers)]
    w_out = [randn(experts, width, inner, dtype=torch.bfloat16, seed=55 + i, scale=1 / math.sqrt(inner)) for i in range(layers)]
    ids = [torch.zeros(n, top, dtype=torch.int32, device="cuda") for _ in range(layers)]
    weights, residual = torch.rand(n, top, generator=g).cuda(), torch.zeros(n, width, device="cuda")
    monkeypatch.setattr(type(ops), "_moe_few_pays", staticmethod(lambda *sizes: True))

    def run():
        ops.scale_(residual, 0.0)
        for i in range(layers):
            ops.moe_experts_residual(y, ids[i], weights, w_in[i], w_out[i], residual, "silu", 7.0, True, False)

    run()
    torch.cuda.synchronize()
    graph, launches = torch.cuda.CUDAGraph(), ops.launches
    ops.set_dependent_launch(True)
    try:
        with torch.cuda.graph(graph):
            run()
    finally:
        ops.set_dependent_launch(False)
    assert ops.launches == launches + 1 + 3 * layers
    for turn in range(6):
        for i in range(layers):
            chosen = torch.stack([torch.randperm(experts, generator=g)[:top] for _ in range(n)]).to(torch.int32)
            if turn % 3 == 1:
                chosen[-1] = -1
            if turn % 3 == 2:
                chosen[:] = (turn + i) % experts
            ids[i].copy_(chosen)
        run()
        want = residual.clone()
        for _ in range(3):
            graph.replay()
            assert torch.equal(residual, want), turn


def _attention_case(ops, dtype, n_head, n_kv_head, head_dim, page_tokens, window, lengths, q_lens,
                    seed=0, spike=None, portions=False):
    """Requests with `lengths[i]` tokens in total, of which the last `q_lens[i]` are new.
    spike = (request, key position, gain): that key is `gain` in every feature and the request's
    queries of head 0 are all ones, so that its score stands far above every other."""
    g = torch.Generator().manual_seed(seed)
    R = len(lengths)
    max_pages = max(-(-n // page_tokens) for n in lengths) + 1
    num_pages = sum(-(-n // page_tokens) for n in lengths) + 3
    perm = torch.randperm(num_pages, generator=g).tolist()       # pages in scattered order
    tables = torch.full((R, max_pages), -1, dtype=torch.int32)
    k_all, v_all = [], []
    k_pages = torch.full((num_pages, n_kv_head, page_tokens, head_dim), float("nan"))
    v_pages = torch.full((num_pages, n_kv_head, page_tokens, head_dim), float("nan"))
    for r, n in enumerate(lengths):
        k = torch.randn(n, n_kv_head, head_dim, generator=g).to(dtype).float()
        v = torch.randn(n, n_kv_head, head_dim, generator=g).to(dtype).float()
        if spike is not None and spike[0] == r:
            k[spike[1]] = spike[2]
        k_all.append(k)
        v_all.append(v)
        for i in range(-(-n // page_tokens)):
            page = perm.pop()
            tables[r, i] = page
            chunk = slice(i * page_tokens, min(n, (i + 1) * page_tokens))
            k_pages[page, :, : chunk.stop - chunk.start] = k[chunk].transpose(0, 1)
            v_pages[page, :, : chunk.stop - chunk.start] = v[chunk].transpose(0, 1)
    # unused rows of pages hold NaN: reading past a request's length would poison the output
    qkv_rows, token_request, positions, want = [], [], [], []
    scale = 1.0 / math.sqrt(head_dim)
    for r, (n, ql) in enumerate(zip(lengths, q_lens)):
        q = torch.randn(ql, n_head, head_dim, generator=g).to(dtype).float() * 2.0
        if spike is not None and spike[0] == r:
            q[:, 0] = 1.0
        for i in range(ql):
            p = n - ql + i
            lo = 0 if not window else max(0, p - window + 1)
            row = torch.zeros(n_head, head_dim, dtype=torch.float64)
            for h in range(n_head):
                kh = h // (n_head // n_kv_head)
                s = (k_all[r][lo: p + 1, kh].double() @ q[i, h].double()) * scale
                row[h] = torch.softmax(s, 0) @ v_all[r][lo: p + 1, kh].double()
            want.append(row.reshape(-1))
            filler = torch.zeros(2 * n_kv_head * head_dim)
            qkv_rows.append(torch.cat([q[i].reshape(-1), filler]))
            token_request.append(r)
            positions.append(p)
    cache = SimpleNamespace(k_pages=k_pages.to(dtype).cuda(), v_pages=v_pages.to(dtype).cuda(),
                            group=0, page_tokens=page_tokens, window=window or None, writes=False)
    from mini_gpt_inference_b200.parts.context import HostBatch, StepPlan

    # the host half of the tiled prompt attention, as the attention mixer asks for it
    plan = StepPlan()
    ops.plan_prompt_attention(HostBatch(q_lens, [n - ql for n, ql in zip(lengths, q_lens)], [0] * len(q_lens),
                                        dtype), plan, n_head, n_kv_head, head_dim)
    ctx = SimpleNamespace(block_tables=[tables.cuda()],
                          token_request=torch.tensor(token_request, dtype=torch.int32).cuda(),
                          positions=torch.tensor(positions, dtype=torch.int32).cuda(),
                          decode_only=all(q == 1 for q in q_lens), max_ctx_after=max(lengths),
                          extra={k: torch.from_numpy(v).cuda() for k, v in plan.arrays.items()})
    if portions:                                   # what a step of the runner has besides: each request's rows
        ctx.host_q_len, starts = list(q_lens), [sum(q_lens[:i]) for i in range(R)]
        ctx.req_q_start = torch.tensor(starts, dtype=torch.int32).cuda()
        ctx.req_q_len = torch.tensor(q_lens, dtype=torch.int32).cuda()
        ctx.host_ctx_before = [n - ql for n, ql in zip(lengths, q_lens)]
        ctx.req_ctx_before = torch.tensor(ctx.host_ctx_before, dtype=torch.int32).cuda()
    qkv = torch.stack(qkv_rows).to(dtype).cuda()
    before = ops.launches
    got = ops.paged_attention(qkv, n_head, n_kv_head, head_dim, scale, cache, ctx)
    _attention_case.kernels = ops.launches - before
    return got.double().cpu(), torch.stack(want)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n_head,n_kv_head,head_dim,page_tokens,window", [
    (8, 8, 64, 16, 0), (3, 3, 32, 8, 0), (5, 1, 48, 4, 0), (6, 2, 16, 16, 0), (4, 4, 80, 32, 0),
    (2, 2, 128, 16, 0), (4, 2, 256, 64, 0), (4, 4, 32, 8, 5), (6, 3, 64, 16, 33)])
def test_paged_attention_general(ops, dtype, n_head, n_kv_head, head_dim, page_tokens, window):
    pt = page_tokens
    lengths = [1, 2, pt - 1, pt, pt + 1, 2 * pt, 3 * pt + 1, 150]
    q_lens = [1, 2, 1, pt, 3, 1, 2 * pt + 1, 31]
    got, want = _attention_case(ops, dtype, n_head, n_kv_head, head_dim, pt, window, lengths, q_lens)
    assert not torch.isnan(got).any(), "attention read a cache row beyond a request's length"
    assert (got - want).abs().max() <= _tol(dtype, 1.0)


@pytest.mark.parametrize("n_head,n_kv_head,head_dim,page_tokens,window,sinks,gated,copies", [
    (4, 4, 64, 16, 0, False, False, 1), (8, 2, 64, 24, 70, True, True, 1), (3, 3, 32, 8, 1, False, False, 1),
    (4, 1, 128, 64, 129, True, False, 1), (16, 16, 32, 16, 0, False, True, 20)])
def test_32_bit_attention_of_portions_and_single_tokens_agrees_bit_for_bit(ops, n_head, n_kv_head, head_dim, page_tokens,
                                                                         window, sinks, gated, copies):
    """330 tokens of one request as a whole, as portions, and one by one (with ``copies``: so often that the key blocks are
    done in several passes): the same numbers, and those of the general kernel within rounding."""
    n, g = 330, torch.Generator().manual_seed(5)
    pages = -(-n // page_tokens)
    order = torch.randperm(pages, generator=g)
    kv = [torch.randn(pages, n_kv_head, page_tokens, head_dim, generator=g) for _ in range(2)]
    for t in kv:                                     # behind the request's last token: no numbers
        t[order[-1], :, (n - 1) % page_tokens + 1:] = float("nan")
    cache = SimpleNamespace(k_pages=kv[0].cuda(), v_pages=kv[1].cuda(), group=0, page_tokens=page_tokens,
                            window=window or None, writes=False)
    q = torch.randn(n, n_head * head_dim, generator=g).cuda() * 2.0
    gate = torch.randn(n, n_head * head_dim, generator=g).cuda() if gated else None
    sink = torch.randn(n_head, generator=g).cuda() if sinks else None

    def step(rows, lens, single=False):
        rows, requests = torch.as_tensor(rows), len(lens)
        i32 = lambda v: torch.as_tensor(v, dtype=torch.int32).cuda()
        ctx = SimpleNamespace(block_tables=[i32(order).repeat(requests, 1)], positions=i32(rows),
                              token_request=i32([r for r, m in enumerate(lens) for _ in range(m)]), decode_only=single,
                              max_ctx_after=int(rows.max()) + 1, host_q_len=lens, req_q_len=i32(lens),
                              req_q_start=i32([sum(lens[:r]) for r in range(requests)]))
        return ops.paged_attention_general(q[rows.cuda()], n_head, n_kv_head, head_dim, head_dim, head_dim ** -0.5, cache, ctx,
                                           gate=None if gate is None else gate[rows.cuda()], sinks=sink)

    whole = step(list(range(n)), [n])
    assert not torch.isnan(whole).any()
    assert torch.equal(step(list(range(100, n)), [1, 63, 66, 100]), whole[100:])
    before = ops.launches
    ones = step(list(range(n)) * copies, [1] * n * copies, single=True)
    assert (ops.launches - before > 2) == (copies > 1)
    assert torch.equal(ones, whole.repeat(copies, 1))
    ops.use_fp32_attention = False
    try:
        general = step(list(range(n)), [n])
    finally:
        ops.use_fp32_attention = True
    # sums of up to 330 numbers of size 1, in another order
    assert (whole - general).abs().max() <= 2e-5


@pytest.mark.parametrize("what", ["query", "key", "block", "low query"])
@pytest.mark.parametrize("single", [False, True], ids=["portions", "single"])
def test_32_bit_attention_keeps_what_is_no_number(ops, what, single):
    """Results are no numbers exactly where the general kernel's are: a token whose query is none, tokens that see a key (or a
    whole block of 64) that is none, a token all of whose scores are -inf."""
    n, n_head, head_dim, page_tokens, g = 150, 2, 64, 16, torch.Generator().manual_seed(9)
    pages = -(-n // page_tokens)
    kv = [torch.randn(pages, n_head, page_tokens, head_dim, generator=g) for _ in range(2)]
    q = torch.randn(n, n_head * head_dim, generator=g)
    if what == "query":
        q[140, 3] = float("nan")
    elif what == "key":
        kv[0][90 // page_tokens, 1, 90 % page_tokens, 5] = float("nan")
    elif what == "block":
        kv[0][:4, 0, :, 7] = float("nan")                    # keys 0 to 63 of one head
    else:
        q[140, 0] = -float("inf")
        kv[0][:, 0, :, 0].abs_().add_(1.0)
    i32 = lambda v: torch.as_tensor(v, dtype=torch.int32).cuda()
    lens = [1] * n if single else [n]
    cache = SimpleNamespace(k_pages=kv[0].cuda(), v_pages=kv[1].cuda(), group=0, page_tokens=page_tokens, window=None, writes=False)
    ctx = SimpleNamespace(block_tables=[torch.arange(pages, dtype=torch.int32).repeat(len(lens), 1).cuda()], positions=i32(range(n)),
                          token_request=i32([r for r, m in enumerate(lens) for _ in range(m)]), decode_only=single,
                          max_ctx_after=n, host_q_len=lens, req_q_len=i32(lens), req_q_start=i32(range(len(lens))))

    def run():
        return ops.paged_attention_general(q.cuda(), n_head, n_head, head_dim, head_dim, 0.125, cache, ctx)

    got = run()
    ops.use_fp32_attention = False
    try:
        general = run()
    finally:
        ops.use_fp32_attention = True
    assert torch.isnan(general).any() and not torch.isnan(general).all()
    assert torch.equal(torch.isnan(got), torch.isnan(general))
    assert torch.allclose(got, general, rtol=0, atol=2e-5, equal_nan=True)


@pytest.mark.parametrize("n,k", [(512, 2048), (2048, 512), (50304, 64), (130, 100), (65, 129), (9, 4)])
def test_32_bit_products_do_not_hang_on_the_rows_beside_them(ops, n, k):
    """Tiles of every size and the kernel of a few rows: bit for bit the same, with every epilogue."""
    m = 2304 if n <= 2048 else 300
    x, w, b = randn(m, k, seed=31), randn(n, k, seed=32, scale=1 / math.sqrt(k)), randn(n, seed=33)
    ref = x.double() @ w.double().T + b.double()
    for act in ("none", "gelu_tanh", "relu_sq"):
        whole = ops.linear(x, w, b, act, torch.float32)
        for rows in (1, 8, 9, 16, 17, 64, 65, 129, 257):
            assert torch.equal(ops.linear(x[:rows], w, b, act, torch.float32), whole[:rows]), (act, rows)
        if act == "none":
            assert (whole.double() - ref).abs().max() <= 2e-5
    res = randn(m, n, seed=34)
    whole = res.clone()
    ops.linear_residual(x, w, b, whole)
    assert (whole.double() - res.double() - ref).abs().max() <= 3e-5
    few = res[:5].clone()
    ops.linear_residual(x[:5], w, b, few)
    assert torch.equal(few, whole[:5])


@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 130])
@pytest.mark.parametrize("n,k", [(130, 260), (33, 64), (64, 68), (1540, 1032), (5, 4)])
def test_32_bit_products_by_bfloat16_pieces(ops, m, n, k):
    """Tiles of 128 x 64 and the kernel of a few rows at their edges: no further from the 64-bit result than what a
    32-bit sum of k terms may be off, as far as the FMA tiles with what is no number, infinite, huge or tiny, and by the
    same sums as those where a row holds such numbers."""
    x, w, b = randn(m, k, seed=41), randn(n, k, seed=42), randn(n, seed=43)
    ref, size = x.double() @ w.double().T + b.double(), x.double().abs() @ w.double().abs().T + b.double().abs()
    # three pieces hold all 24 bits; a slice of 64 terms is rounded (or cut) ten times at its full size, slices and bias once each
    bound = (10 + -(-k // 64) + 2) * 2.0 ** -23 * size
    assert ((ops.linear(x, w, b, "none", torch.float32).double() - ref).abs() <= bound).all()
    x[0, k - 1], w[n - 1, 0] = float("inf"), float("nan")
    if m > 7:
        x[3], x[4], x[5, 1], x[6, k // 2] = 1e-36, 1e36, 2e38, float("nan")
    w[1], w[2] = 0.0, 1e-38
    w[3, k // 2] = -float("inf")
    got = ops.linear(x, w, b, "none", torch.float32)
    ops.use_split = False
    try:
        want = ops.linear(x, w, b, "none", torch.float32)
    finally:
        ops.use_split = True
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    assert torch.equal(got[0].nan_to_num(), want[0].nan_to_num()) and torch.equal(got[:, 2].nan_to_num(), want[:, 2].nan_to_num())
    finite = torch.isfinite(want)
    size = x.double().abs() @ w.double().abs().T + b.double().abs()
    assert ((got.double() - want.double()).abs() <= 2 * (k + 2) * 2.0 ** -24 * size)[finite].all()


@pytest.mark.parametrize("m", [8, 16, 130])
@pytest.mark.parametrize("n,k", [(70, 260), (33, 64)])
def test_32_bit_products_near_the_ends_of_the_range(ops, m, n, k):
    """Rows whose products pass the end of the range (and those that end just inside it) give what the FMA tiles give, infinities of
    the same sign and no numbers in the same places; numbers so small that bfloat16 pieces do not hold them keep their bits beside large ones."""
    x, w = randn(m, k, seed=51), randn(n, k, seed=52)
    x[0], w[0] = 3e25, 1e25
    x[1], w[1] = x[1].abs() * 1e20, -w[1].abs() * 1e30
    x[2], w[2] = 0.0, 0.0
    x[2, :4], w[2, :4] = 1.9999 * 2.0 ** 63, 1.9999 * 2.0 ** 61              # four products that just stay inside
    x[3], w[3] = x[3] * 2.0 ** 60, w[3] * 2.0 ** 62
    x[4, k // 2:], w[4, : k // 2] = x[4, k // 2:] * 2.0 ** -114, 0.0            # large numbers meet zeros, and small ones large ones
    w[4, k // 2:] = w[4, k // 2:] * 2.0 ** 40
    x[5], w[5] = x[5] * 2.0 ** -70, w[5] * 2.0 ** -70                        # results below the least normal number
    w[6] = w[6] * 2.0 ** -130
    x[7] = x[7] * 2.0 ** 124
    got = ops.linear(x, w, None, "none", torch.float32)
    ops.use_split = False
    try:
        want = ops.linear(x, w, None, "none", torch.float32)
    finally:
        ops.use_split = True
    ops.check_status()
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    assert torch.equal(got[torch.isinf(want)], want[torch.isinf(want)]) and torch.isfinite(got[2, 2])
    assert torch.isinf(want).any() and torch.isfinite(want[4]).any()
    ref, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    finite = torch.isfinite(want)
    # the bound of the test above; below the normal numbers every addition is cut at 2^-149 instead
    steps = 10 + -(-k // 64) + 2
    bound = (steps * 2.0 ** -23 * size).clamp(min=steps * -(-k // 64) * 2.0 ** -149)
    by_fma = ((k + 2) * 2.0 ** -24 * size).clamp(min=(k + 2) * 2.0 ** -149)
    assert ((got.double() - ref).abs() <= torch.maximum(bound, by_fma))[finite].all()


@pytest.mark.parametrize("m", [16, 256])
def test_32_bit_products_hold_all_bits_of_their_inputs(ops, m):
    """A result of one product is that product, rounded once: h h' is exact in its accumulator, and what lies below (the cut of
    the rest, 2^-31 of the product at most, and l l') moves the rounding by less than a thirtieth of its half place."""
    n, k = 96, 132
    g = torch.Generator(device="cuda").manual_seed(81)
    w = 1.0 + 2.0 ** -8 + 2.0 ** -14 * torch.randn(n, k, generator=g, device="cuda")       # (where m m' and m l' are largest)
    w[n // 2:] = randn(n - n // 2, k, seed=82)
    x = torch.zeros(m, k, device="cuda")
    at = torch.arange(m, device="cuda") % k
    x[torch.arange(m, device="cuda"), at] = 1.0 + 2.0 ** -8 + 2.0 ** -14 * torch.randn(m, generator=g, device="cuda")
    want = x.double() @ w.double().T
    got = ops.linear(x, w, None, "none", torch.float32)
    assert ((got.double() - want).abs() <= 2.0 ** -24 * (1 + 1 / 30) * want.abs()).all()


@pytest.mark.parametrize("k", [64, 512])
def test_32_bit_sums_of_one_sign_are_no_further_off_than_multiply_adds(ops, k):
    """The tensor cores cut where an addition rounds, so sums of numbers of one sign come out too small, by as much in every slice: few
    such additions may follow each other among a slice's largest products."""
    x, w = randn(512, k, seed=91).abs(), randn(256, k, seed=92).abs()
    want = x.double() @ w.double().T

    def error():
        return float((ops.linear(x, w, None, "none", torch.float32).double() - want).norm() / want.norm())

    here = error()
    ops.use_split = False
    try:
        by_fma = error()
    finally:
        ops.use_split = True
    assert here <= 1.05 * by_fma


@pytest.mark.parametrize("n,k", [(4100, 68), (4101, 260)])
def test_32_bit_products_of_many_tiles_with_rows_that_do_not_split(ops, n, k):
    """Four tiles of 128 x 64 a CTA, so that the sets of marks are used again, with such rows in several of them: those results are the
    FMA tiles' to the bit, added into a residual stream once, and all others what they are without such rows."""
    m = 1030
    x, w, b = randn(m, k, seed=61), randn(n, k, seed=62), randn(n, seed=63)
    clean = ops.linear(x, w, b, "none", torch.float32)
    xs, ws = [0, 127, 300, 640, 1029], [5, 1000, 2047, 4099]
    for i, r in enumerate(xs):
        x[r, (37 * i) % k] = (float("nan"), float("inf"), 1e-37, 3e38, -float("inf"))[i]
    for i, r in enumerate(ws):
        w[r, (11 * i) % k] = (float("nan"), 2e-38, 1.7e38, -float("inf"))[i]
    res = randn(m, n, seed=64)
    got, added = ops.linear(x, w, b, "none", torch.float32), res.clone()
    ops.linear_residual(x, w, b, added)
    ops.use_split = False
    try:
        want = ops.linear(x, w, b, "none", torch.float32)
    finally:
        ops.use_split = True
    ops.check_status()
    odd = torch.zeros(m, n, dtype=torch.bool, device="cuda")
    odd[xs], odd[:, ws] = True, True
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.isnan(want).any()
    assert torch.equal(got[odd].nan_to_num(7.0), want[odd].nan_to_num(7.0)) and torch.equal(got[~odd], clean[~odd])
    assert torch.equal(added.nan_to_num(7.0), (res + got).nan_to_num(7.0))


@pytest.mark.parametrize("m", [8, 128])
def test_32_bit_products_of_rows_that_do_not_split_take_no_age(ops, m):
    """Inputs that hold what is no number take a second walk over the operands, not a chain of dependent loads for each result
    (2 to 5 times the usual time; 14 and 69 times it so)."""
    n, k = 512, 2048
    x, w, out = randn(m, k, seed=71), randn(n, k, seed=72), torch.empty(m, n, device="cuda")

    def microseconds():
        best = float("inf")
        for _ in range(8):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            start.record()
            for _ in range(20):
                ops.linear(x, w, None, "none", torch.float32, out=out)
            end.record()
            torch.cuda.synchronize()
            best = min(best, start.elapsed_time(end) * 1e3 / 20)
        return best

    usual = microseconds()
    x[:, 3] = float("nan")
    assert microseconds() < 10 * max(usual, 5.0) and torch.isnan(out).all()


@pytest.mark.parametrize("single", [False, True], ids=["portions", "single"])
@pytest.mark.parametrize("n_head,n_kv_head,head_dim,page_tokens,window", [
    (4, 4, 128, 64, 0), (6, 2, 104, 16, 0), (5, 1, 48, 4, 0), (4, 4, 80, 24, 70), (2, 2, 96, 16, 0), (64, 1, 8, 8, 0),
    (2, 1, 128, 16, 64)])
def test_heads_of_other_sizes_on_the_warp_level_tensor_cores(ops, n_head, n_kv_head, head_dim, page_tokens, window, single):
    """bfloat16 heads that the tcgen05 and the single-token kernels do not take: no further from the 64-bit result than the
    kernel of a warp per token and head, whose softmax weights are 32-bit numbers."""
    lengths = [1, 63, 64, 65, 127, 128, 129, 300, 17]
    q_lens = [1] * len(lengths) if single else [1, 63, 1, 65, 64, 63, 2, 257, 17]
    args = (ops, torch.bfloat16, n_head, n_kv_head, head_dim, page_tokens, window, lengths, q_lens)
    ops.use_split_attention = False
    try:
        got, want = _attention_case(*args, seed=8, portions=True)
        ops.use_mma_attention = False
        general, _ = _attention_case(*args, seed=8, portions=True)
    finally:
        ops.use_split_attention = ops.use_mma_attention = True
    ops.check_status()
    assert not torch.isnan(got).any()
    assert (got - want).abs().max() <= _tol(torch.bfloat16, 1.0)
    # both round their outputs to bfloat16, which is nearly all of either error; one rounding that falls the other way may
    # move the sum of squares of some thousand outputs by a few per cent
    assert (got - want).norm() <= 1.03 * (general - want).norm()


@pytest.mark.parametrize("n_head,n_kv_head,page_tokens,window", [(4, 4, 64, 0), (6, 2, 16, 0), (3, 1, 128, 200), (2, 2, 8, 33)])
def test_prompt_portions_of_heads_of_128_on_the_tensor_cores(ops, n_head, n_kv_head, page_tokens, window):
    """Whole prompts, later portions, single tokens among them, tiles cut along the keys: no further from the 64-bit result
    than the kernel of a warp per token and head, whose softmax weights are 32-bit numbers."""
    lengths = [1, 64, 129, 300, 1100, 700]
    q_lens = [1, 64, 129, 150, 130, 1]
    args = (ops, torch.bfloat16, n_head, n_kv_head, 128, page_tokens, window, lengths, q_lens)
    ops.use_mma_attention = False
    try:
        got, want = _attention_case(*args, seed=9)
        ops.use_prefill_tc = False
        general, _ = _attention_case(*args, seed=9)
    finally:
        ops.use_mma_attention = ops.use_prefill_tc = True
    ops.check_status()
    assert not torch.equal(got, general), "the two kernels were expected to differ in rounding"
    assert not torch.isnan(got).any()
    assert (got - want).abs().max() <= _tol(torch.bfloat16, 1.0)
    # (nearly all of either error is the outputs' rounding to bfloat16, see above)
    assert (got - want).norm() <= 1.03 * (general - want).norm()


@pytest.mark.parametrize("window", [0, 90])
@pytest.mark.parametrize("n_head,n_kv_head,head_dim", [(4, 2, 48), (3, 3, 80), (8, 1, 128), (2, 2, 128)])
def test_a_value_that_is_no_number_leaves_the_tokens_in_front_of_it_alone(ops, n_head, n_kv_head, head_dim, window):
    """Portions of prompts of heads other than 64: results are finite exactly where the general kernel's are."""
    n, page_tokens, g = 300, 16, torch.Generator().manual_seed(head_dim)
    pages = -(-n // page_tokens)
    kv = [torch.randn(pages, n_kv_head, page_tokens, head_dim, generator=g) for _ in range(2)]
    for t, f, value in ((100, 5, "nan"), (101, 5, "inf"), (130, 6, "inf"), (131, 7, "-inf"), (256, 40, "nan"), (299, 0, "nan")):
        kv[1][t // page_tokens, 0, t % page_tokens, f] = float(value)
    qkv = torch.randn(n, (n_head + 2 * n_kv_head) * head_dim, generator=g).to(torch.bfloat16).cuda()
    i32 = lambda v: torch.as_tensor(v, dtype=torch.int32).cuda()
    from mini_gpt_inference_b200.parts.context import HostBatch, StepPlan

    def run(begin):
        plan = StepPlan()
        ops.plan_prompt_attention(HostBatch([n - begin], [begin], [0], torch.bfloat16), plan, n_head, n_kv_head, head_dim)
        ctx = SimpleNamespace(block_tables=[torch.arange(pages, dtype=torch.int32)[None].cuda()], positions=i32(range(begin, n)),
                              token_request=i32([0] * (n - begin)), decode_only=False, max_ctx_after=n, host_q_len=[n - begin],
                              req_q_len=i32([n - begin]), req_q_start=i32([0]),
                              extra={k: torch.from_numpy(v).cuda() for k, v in plan.arrays.items()})
        cache = SimpleNamespace(k_pages=kv[0].to(torch.bfloat16).cuda(), v_pages=kv[1].to(torch.bfloat16).cuda(), group=0,
                                page_tokens=page_tokens, window=window or None, writes=False)
        return ops.paged_attention(qkv[begin:], n_head, n_kv_head, head_dim, head_dim ** -0.5, cache, ctx).float()

    for begin in (0, 37):
        got = run(begin)
        ops.use_mma_attention = ops.use_prefill_tc = False
        try:
            general = run(begin)
        finally:
            ops.use_mma_attention = ops.use_prefill_tc = True
        finite = torch.isfinite(general)
        assert finite.any() and not finite.all()
        assert torch.equal(torch.isfinite(got), finite)
        assert (got - general)[finite].abs().max() <= 1.6e-2
    ops.check_status()


@pytest.mark.parametrize("n,context", [(3, 200), (3, 500), (3, 1990), (700, 500), (700, 1990)])
def test_ranges_of_single_tokens_are_merged(ops, n, context):
    """Few ranges and many, of few tokens and of more than the GPU holds at once (other numbers of ranges asked for ahead):
    the same results as the general kernel, for tokens at all places of the context."""
    n_head, n_kv_head, head_dim, page_tokens, g = 16, 4, 48, 16, torch.Generator().manual_seed(n + context)
    pages = -(-context // page_tokens)
    kv = [torch.randn(pages, n_kv_head, page_tokens, head_dim, generator=g).to(torch.bfloat16).cuda() for _ in range(2)]
    qkv = torch.randn(n, (n_head + 2 * n_kv_head) * head_dim, generator=g).to(torch.bfloat16).cuda()
    cache = SimpleNamespace(k_pages=kv[0], v_pages=kv[1], group=0, page_tokens=page_tokens, window=None, writes=False)
    positions = torch.linspace(0, context - 1, n).to(torch.int32)
    ctx = SimpleNamespace(block_tables=[torch.arange(pages, dtype=torch.int32).repeat(n, 1).cuda()], positions=positions.cuda(),
                          token_request=torch.arange(n, dtype=torch.int32).cuda(), decode_only=True, max_ctx_after=context, extra={})
    got = ops.paged_attention(qkv, n_head, n_kv_head, head_dim, head_dim ** -0.5, cache, ctx).float()
    ops.use_mma_attention = False
    try:
        general = ops.paged_attention(qkv, n_head, n_kv_head, head_dim, head_dim ** -0.5, cache, ctx).float()
    finally:
        ops.use_mma_attention = True
    assert (got - general).abs().max() <= 2.0 ** -7 * general.abs().max()      # the last place of the largest
    assert not torch.equal(got, torch.zeros_like(got))


@pytest.mark.parametrize("gain", [4.0, 9.0, 24.0])
def test_prompt_attention_with_a_key_far_above_the_others(ops, gain):
    """One key, hundreds of positions into the prompt, scores 8 * gain above the rest (head 0; other
    heads see it at random heights, above and below).  The tensor-core kernel takes each row's
    reference exponent from the first block and must move it when this key comes: at 9 the
    weights leave the range it allows, at 24 they leave the range of 32-bit floats.  Queries
    before the key must not see it; the tile is cut along the keys, so parts with references far
    apart are merged."""
    lengths, q_lens = [1000, 300], [700, 300]
    got, want = _attention_case(ops, torch.bfloat16, 4, 2, 64, 16, 0, lengths, q_lens, seed=5,
                                spike=(0, 611, gain))
    ops.check_status()
    assert not torch.isnan(got).any()
    # rows that see the key return its value row, not an average of many: the results are as
    # large as single values are (up to 4), and a bfloat16 result is that much coarser
    assert (got - want).abs().max() <= _tol(torch.bfloat16, max(1.0, float(want.abs().max())))
    assert float(want.abs().max()) > 2.0


@pytest.mark.parametrize("n_head,n_kv_head,page_tokens,window", [
    (8, 8, 16, 0), (2, 2, 8, 0), (4, 1, 64, 0), (2, 2, 128, 0), (2, 1, 256, 0), (3, 3, 32, 0),
    (4, 2, 16, 33), (2, 2, 64, 200)])
def test_prompt_portions_on_the_tensor_cores(ops, n_head, n_kv_head, page_tokens, window):
    """Portions of prompts with head size 64 in bfloat16 take the tcgen05 kernel: query tiles of
    128 rows over key blocks of 64 from the pages; tiles that start anywhere in a request,
    tiles of one row, contexts that end at any place inside a block or a page."""
    lengths = [300, 129, 128, 1000, 1, 77, 513, 1300, 2048]
    q_lens = [300, 129, 5, 700, 1, 2, 257, 3, 130]
    got, want = _attention_case(ops, torch.bfloat16, n_head, n_kv_head, 64, page_tokens, window,
                                lengths, q_lens, seed=3)
    ops.check_status()
    assert not torch.isnan(got).any()
    assert (got - want).abs().max() <= _tol(torch.bfloat16, 1.0)
    ops.use_prefill_tc = False
    try:
        general, _ = _attention_case(ops, torch.bfloat16, n_head, n_kv_head, 64, page_tokens, window,
                                     lengths, q_lens, seed=3)
    finally:
        ops.use_prefill_tc = True
    assert (general - got).abs().max() <= _tol(torch.bfloat16, 1.0)
    assert not torch.equal(general, got), "the two kernels were expected to differ in rounding"


@pytest.mark.parametrize("n_head,n_kv_head,head_dim,page_tokens,window", [
    (8, 8, 64, 16, 0), (8, 8, 64, 64, 0), (3, 3, 32, 8, 0), (6, 2, 16, 16, 0), (2, 2, 128, 16, 0),
    (4, 2, 256, 64, 0), (4, 4, 32, 8, 5), (6, 3, 64, 16, 300)])
def test_paged_attention_split_over_keys(ops, n_head, n_kv_head, head_dim, page_tokens, window):
    """Single query tokens in bfloat16 take the kernel that splits the keys into blocks of 256
    and merges: lengths around the block edges (blocks of 32 to 256 keys by head size), one token, long contexts."""
    lengths = [1, 2, 63, 64, 65, 127, 129, 255, 256, 257, 511, 513, 700, 1025, page_tokens, page_tokens + 1]
    got, want = _attention_case(ops, torch.bfloat16, n_head, n_kv_head, head_dim, page_tokens, window,
                                lengths, [1] * len(lengths))
    assert _attention_case.kernels == 1, "the split kernel (with its own merge) was expected to run"
    ops.check_status()
    assert not torch.isnan(got).any()
    assert (got - want).abs().max() <= _tol(torch.bfloat16, 1.0)
    # the general kernel gives the same within rounding
    ops.use_split_attention = False
    try:
        general, _ = _attention_case(ops, torch.bfloat16, n_head, n_kv_head, head_dim, page_tokens, window,
                                     lengths, [1] * len(lengths))
    finally:
        ops.use_split_attention = True
    assert (general - got).abs().max() <= _tol(torch.bfloat16, 1.0)


@pytest.mark.parametrize("n_head,n_kv_head,head_dim,page_tokens,rows", [
    (8, 8, 64, 64, 64),        # the 50M model's batch of 64: 64 x 8 x 9 blocks
    (24, 2, 64, 16, 170),      # 12 query heads per kv head: two tiles of eight heads per CTA
    (40, 2, 32, 8, 200),       # 20 heads per kv head: two CTAs per kv head, the second not full
    (4, 4, 128, 32, 70)])
def test_split_attention_of_many_rows_merges_in_a_second_kernel(ops, n_head, n_kv_head, head_dim,
                                                                  page_tokens, rows):
    """A grid of several waves leaves its partial rows in scratch and a second kernel merges them.
    Every row's context is long enough for three or more key blocks that all hold keys, and the
    lengths differ from row to row, so that a block merged twice, dropped, or taken from the
    neighbour's scratch shows."""
    block = ops.lib.mg_attention_split_keys(head_dim)
    lengths = [2 * block + 37 + (11 * i) % (2 * block + 150) for i in range(rows)]
    assert min(lengths) > 2 * block
    got, want = _attention_case(ops, torch.bfloat16, n_head, n_kv_head, head_dim, page_tokens, 0,
                                lengths, [1] * rows, seed=11)
    assert _attention_case.kernels == 2, "the merge was expected to run as a kernel of its own"
    ops.check_status()
    assert not torch.isnan(got).any()
    assert (got - want).abs().max() <= _tol(torch.bfloat16, 1.0)
    # the counters stay zero for the next launch, whichever kernel merged
    assert int(ops._counters(1).abs().sum()) == 0


@pytest.mark.parametrize("n_head,n_kv_head,head_dim,page_tokens,lengths,launches", [
    (2, 2, 64, 64, [2049, 2200, 4097, 6000, 8191, 2176], 1),     # 17 to 64 blocks of 128 keys, merged by the last CTA
    (4, 1, 64, 16, [9000, 3333], 1),                             # grouped heads, 71 and 27 blocks
    (2, 2, 32, 64, [4400, 5000, 7000], 1),                       # blocks of 256 keys: 18 to 28
    (2, 2, 128, 32, [1100, 1500, 2300], 1),                      # blocks of 64 keys: 18 to 36
    (8, 8, 64, 64, [2100 + 37 * i for i in range(12)], 2)])      # 12 x 8 x 20 blocks: the second kernel merges
def test_split_attention_with_many_key_blocks(ops, n_head, n_kv_head, head_dim, page_tokens, lengths, launches):
    """Contexts of more than sixteen key blocks: the merge then shares a row's blocks among the four
    warps of a CTA (quarters, added in warp order), inside the attention kernel or in the second one.
    A spike far back in the longest request must still decide its row."""
    block = ops.lib.mg_attention_split_keys(head_dim)
    assert min(lengths) > 16 * block
    longest = max(range(len(lengths)), key=lambda i: lengths[i])
    for spike in (None, (longest, 5, 3.0)):
        got, want = _attention_case(ops, torch.bfloat16, n_head, n_kv_head, head_dim, page_tokens, 0,
                                    lengths, [1] * len(lengths), seed=21, spike=spike)
        assert _attention_case.kernels == launches
        ops.check_status()
        assert not torch.isnan(got).any()
        assert (got - want).abs().max() <= _tol(torch.bfloat16, 1.0)
    assert int(ops._counters(1).abs().sum()) == 0


@pytest.mark.parametrize("dtype", DTYPES)
def test_far_key_among_hundreds_decides(ops, dtype):
    """One key far back gets a score that dominates: the output must be that key's value."""
    n_head, head_dim, pt, n = 2, 64, 16, 700
    g = torch.Generator().manual_seed(5)
    k = torch.randn(n, n_head, head_dim, generator=g) * 0.1
    v = torch.randn(n, n_head, head_dim, generator=g)
    q = torch.randn(1, n_head, head_dim, generator=g)
    far = 3                                                      # in the first page
    k[far] = q[0] * 4.0                                          # score ~ 4 |q|^2 / 8 >> the rest
    pages = -(-n // pt)
    kp = torch.zeros(pages, n_head, pt, head_dim)
    vp = torch.zeros(pages, n_head, pt, head_dim)
    for i in range(pages):
        sl = slice(i * pt, min(n, (i + 1) * pt))
        kp[i, :, : sl.stop - sl.start] = k[sl].transpose(0, 1)
        vp[i, :, : sl.stop - sl.start] = v[sl].transpose(0, 1)
    cache = SimpleNamespace(k_pages=kp.to(dtype).cuda(), v_pages=vp.to(dtype).cuda(), group=0,
                            page_tokens=pt, window=None, writes=False)
    ctx = SimpleNamespace(block_tables=[torch.arange(pages, dtype=torch.int32)[None].cuda()],
                          token_request=torch.zeros(1, dtype=torch.int32).cuda(),
                          positions=torch.tensor([n - 1], dtype=torch.int32).cuda(),
                          decode_only=True, max_ctx_after=n)
    qkv = torch.cat([q.reshape(1, -1), torch.zeros(1, 2 * n_head * head_dim)], 1).to(dtype).cuda()
    got = ops.paged_attention(qkv, n_head, n_head, head_dim, 1 / math.sqrt(head_dim), cache, ctx)
    want = v[far].to(dtype).float().reshape(-1)
    assert (got.float().cpu()[0] - want).abs().max() < 2e-2


@pytest.mark.parametrize("dtype", DTYPES)
def test_kv_store_places_rows(ops, dtype):
    n_head, n_kv, d, pt, pages = 6, 2, 48, 8, 9
    qkv = randn(11, (n_head + 2 * n_kv) * d, dtype=dtype, seed=3)
    slots = torch.tensor([5, 70, 8, 9, 63, 0, 33, 34, 35, 71, -1], dtype=torch.int32).cuda()
    cache = SimpleNamespace(k_pages=torch.zeros(pages, n_kv, pt, d, dtype=dtype).cuda(),
                            v_pages=torch.zeros(pages, n_kv, pt, d, dtype=dtype).cuda(),
                            page_tokens=pt)
    ops.kv_store(qkv, n_head, n_kv, d, cache, slots)
    k = qkv[:, n_head * d: (n_head + n_kv) * d].reshape(11, n_kv, d)
    v = qkv[:, (n_head + n_kv) * d:].reshape(11, n_kv, d)
    want_k = torch.zeros_like(cache.k_pages)
    want_v = torch.zeros_like(cache.v_pages)
    for i, s in enumerate(slots.tolist()):
        if s >= 0:
            want_k[s // pt, :, s % pt] = k[i]
            want_v[s // pt, :, s % pt] = v[i]
    assert torch.equal(cache.k_pages, want_k) and torch.equal(cache.v_pages, want_v)


def test_gather_rows_and_argmax(ops):
    x = randn(40, 77, seed=1)
    rows = torch.tensor([3, 3, 39, 0], dtype=torch.int32).cuda()
    assert torch.equal(ops.gather_rows(x, rows), x[rows.long()])
    logits = randn(9, 50304, seed=2)
    logits[4, 50300] = 99.0
    logits[5, 17] = logits[5, 4000] = 50.0                     # a tie: the lower index wins
    got = ops.argmax(logits)
    assert got.tolist() == logits.argmax(-1).tolist() or got[5] == 17
    assert got[4] == 50300 and got[5] == 17
    limited = ops.argmax(logits, 50257)
    assert limited[4] == logits[4, :50257].argmax()


def _draws(ops, logits_row, temperature, top_k, top_p, n, seed=1234):
    rows = logits_row[None].expand(n, -1).contiguous()
    i32 = lambda v: torch.full((n,), v, dtype=torch.int32).cuda()          # noqa: E731
    f32 = lambda v: torch.full((n,), v, dtype=torch.float32).cuda()        # noqa: E731
    counter = torch.arange(n, dtype=torch.int32).cuda()
    return ops.sample(rows, f32(temperature), None if top_k is None else i32(top_k),
                      None if top_p is None else f32(top_p), i32(seed & 0xFFFF), i32(seed >> 16),
                      counter)


@pytest.mark.parametrize("vocab", [509, 50304])
@pytest.mark.parametrize("temperature,top_k,top_p", [(1.0, None, None), (0.7, 5, None),
                                                     (1.3, None, 0.6), (0.9, 40, 0.8)])
def test_sampler_draws_from_the_reference_distribution(ops, vocab, temperature, top_k, top_p):
    g = torch.Generator().manual_seed(3)
    logits = (torch.randn(vocab, generator=g) * 2.5).cuda()
    want = plain_gpt.sampling_distribution(logits.cpu(), temperature, top_k, top_p)
    n = 40000
    ids = _draws(ops, logits, temperature, top_k, top_p, n).long().cpu()
    counts = torch.bincount(ids, minlength=vocab).double()
    # nothing outside the support (allowing the one token at the top-p edge to differ by rounding)
    outside = counts[want == 0].sum().item()
    assert outside <= (0 if top_p is None else 0.002 * n), outside
    # frequencies follow the probabilities: compare on the 20 likeliest tokens
    top = want.topk(20).indices
    freq = counts[top] / n
    sigma = (want[top] * (1 - want[top]) / n).sqrt()
    assert ((freq - want[top]).abs() <= 5 * sigma + 2e-3).all(), (freq, want[top])


@pytest.mark.parametrize("vocab", [1, 7, 512, 8192, 8193, 16385, 32769, 65536, 65537, 131072, 131073])
def test_sampler_at_the_edges_of_its_cuts(ops, vocab):
    """One CTA a row up to 8,192 ids, clusters of 2, 4 and 8 beyond, twice the values a thread beyond 65,536, one CTA again
    beyond 131,072: drawn ids lie in the support the oracle gives them, also where it is one id at an end of the row, on a
    limit in front of the row's largest value, in a row with infinities and in a greedy row between drawn ones."""
    g = torch.Generator().manual_seed(vocab)
    logits = torch.randn(6, vocab, generator=g) * 3.0
    logits[1, vocab - 1], logits[2, 0] = 60.0, 60.0
    limit = max(1, vocab - 1)
    if vocab > 2:
        logits[3, 1: vocab // 2] = float("-inf")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32).cuda()              # noqa: E731
    temperature, k, p = [0.9, 0.7, 0.7, 1.1, 0.0, 1.0], [9, 0, 0, 5, 3, 0], [0.8, 0.5, 1.0, 1.0, 0.5, 0.6]
    for n in range(4):
        got = ops.sample(logits.cuda(), torch.tensor(temperature).cuda(), i32(k), torch.tensor(p).cuda(), i32([n] * 6),
                         i32(list(range(6))), i32([5 + n] * 6), limit).tolist()
        assert got[4] == int(logits[4, :limit].argmax())
        for r in (0, 1, 2, 3, 5):
            # (a mass within 32-bit rounding of top-p may fall either way)
            want = plain_gpt.sampling_distribution(logits[r, :limit], temperature[r], k[r] or None,
                                                   min(1.0, p[r] + 1e-5) if p[r] < 1 else None)
            assert 0 <= got[r] < limit and want[got[r]] > 0, (r, got[r])


@pytest.mark.parametrize("vocab", [700, 8193, 40001, 70000])
def test_sampler_with_few_left_by_top_k(ops, vocab):
    """Up to 512 values that top-k can keep go to one CTA; more (ties, a large k), infinite values
    take the passes over the whole row.  Every drawn id is in the oracle's support, and greedy rows have the lowest index among equals."""
    g = torch.Generator().manual_seed(vocab)
    logits = torch.randn(10, vocab, generator=g) * 2.0
    logits[1] = logits[1].round()                                          # thousands of ties
    logits[2, 5:] = -float("inf")                                          # fewer numbers than k
    logits[3] = 0.0
    logits[4] = logits[4] * 1e-4
    logits[5, vocab // 2] = float("inf")
    logits[6, 3] = logits[6, vocab - 1] = 30.0
    logits[7, 11], logits[7, 12], logits[7, vocab - 2] = 25.0, float("nan"), 25.0
    logits[8] = -float("inf")
    logits[9] -= 1e4
    i32 = lambda v: torch.tensor(v, dtype=torch.int32).cuda()              # noqa: E731
    f32 = lambda v: torch.tensor(v, dtype=torch.float32).cuda()            # noqa: E731
    k, p = [512, 3, 50, 40, 513, 7, 1, 9, 4, 64], [0.95, 1.0, 0.7, 1.0, 0.9, 1.0, 0.3, 1.0, 1.0, 0.6]
    temperature = [1.3, 1.0, 0.8, 1.0, 1.0, 0.9, 1.0, 0.0, 0.0, 1.0]
    for n in range(4):
        got = ops.sample(logits.cuda(), f32(temperature), i32(k), f32(p), i32([n] * 10), i32(list(range(10))), i32([n] * 10)).tolist()
        assert 0 <= got[5] < vocab and got[6] in (3, vocab - 1) and got[7] == 11 and got[8] == 0
        for r in (0, 1, 2, 3, 4, 9):
            want = plain_gpt.sampling_distribution(logits[r], temperature[r], k[r], min(1.0, p[r] + 1e-5) if p[r] < 1 else None)
            assert want[got[r]] > 0, (r, got[r])


def test_sampler_is_greedy_at_zero_and_repeatable_by_seed(ops):
    g = torch.Generator().manual_seed(4)
    logits = torch.randn(6, 1000, generator=g).cuda()
    zeros = torch.zeros(6).cuda()
    i32 = lambda v: torch.full((6,), v, dtype=torch.int32).cuda()          # noqa: E731
    got = ops.sample(logits, zeros, None, None, i32(1), i32(2), i32(3))
    assert got.tolist() == logits.argmax(-1).tolist()
    # mixed rows: greedy and stochastic side by side (tests/test_sampling.py:63-78)
    temps = torch.tensor([0.0, 1.0, 0.0, 1.0, 1.0, 0.0]).cuda()
    a = ops.sample(logits, temps, None, None, i32(7), i32(0), i32(5))
    b = ops.sample(logits, temps, None, None, i32(7), i32(0), i32(5))
    c = ops.sample(logits, temps, None, None, i32(8), i32(0), i32(5))
    assert a.tolist() == b.tolist()
    assert [a[i].item() for i in (0, 2, 5)] == [logits[i].argmax().item() for i in (0, 2, 5)]
    assert a.tolist() != c.tolist()
    # a row's draw does not depend on the rows beside it
    alone = ops.sample(logits[3:4].contiguous(), temps[3:4].contiguous(), None, None,
                       i32(7)[:1], i32(0)[:1], i32(5)[:1])
    assert alone[0] == a[3]
    # top_k = 1 is greedy whatever the temperature
    k1 = ops.sample(logits, torch.full((6,), 5.0).cuda(), i32(1), None, i32(7), i32(0), i32(5))
    assert k1.tolist() == logits.argmax(-1).tolist()


def test_refusals_are_clear(ops):
    from mini_gpt_inference_b200.kernels.library import KernelLibraryError

    with pytest.raises(KernelLibraryError, match="contiguous"):
        ops.layernorm(randn(4, 8).T, randn(4), None, 1e-5, torch.float32)
    with pytest.raises(KernelLibraryError, match="dtype"):
        ops.linear(randn(4, 8), randn(3, 8, dtype=torch.bfloat16), None, "none", torch.float32)
    with pytest.raises(KernelLibraryError, match="head_dim"):
        cache = SimpleNamespace(k_pages=torch.zeros(2, 1, 4, 2048).cuda(), v_pages=torch.zeros(2, 1, 4, 2048).cuda(),
                                group=0, page_tokens=4, window=None)
        ctx = SimpleNamespace(block_tables=[torch.zeros(1, 2, dtype=torch.int32).cuda()],
                              token_request=torch.zeros(1, dtype=torch.int32).cuda(),
                              positions=torch.zeros(1, dtype=torch.int32).cuda())
        ops.paged_attention(torch.zeros(1, 3 * 2048).cuda(), 1, 1, 2048, 1.0, cache, ctx)
