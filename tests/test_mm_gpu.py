"""The grouped tensor-core GEMM (`mul_mm_id`) and the prefill block against the CPU oracle.
Cases follow src/ops/mm_id.rs:94-166, 379-437 of the reference; bound rel-L2 < 1e-3 for the
f16-tile path (the reference measures ~2.6e-4 for its own f16 tiles)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DTYPES = [(12, "Q4K"), (14, "Q6K")]


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available()
    return torch.device("cuda:0")


def _case(orc, dev, dt, n_expert, n_out, k, t, top_k, xpr, ids, seed, shared_map=False):
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    raw = orc.quantize(dt, orc.pseudo_random(n_expert * n_out * k, seed, -1.0, 1.0))
    stack = ExpertStack.from_bytes(raw, dt, n_expert, n_out, k, device=dev)
    x = orc.pseudo_random(t * xpr * k, seed ^ 0xABCD, -1.0, 1.0).reshape(t, xpr, k)
    xd, idd = torch.from_numpy(x).to(dev), torch.from_numpy(ids.astype(np.int32)).to(dev)
    if shared_map:
        got = ops.mul_mm_id_shared(stack, xd, idd, ops.prepare_map0(n_expert, idd))
    else:
        got = ops.mul_mm_id(stack, xd, idd)
    torch.cuda.synchronize()
    assert tuple(got.shape) == (t, top_k, n_out)
    return got.cpu().numpy(), orc.mul_id(dt, raw, n_expert, n_out, k, x, ids)


@pytest.mark.parametrize("dt,name", DTYPES)
@pytest.mark.parametrize("t,top_k,ne,xpr,seed,iseed", [(16, 2, 4, 1, 0x1600, 0x41), (64, 2, 4, 1, 0x6400, 0x42),
                                                      (40, 4, 6, 4, 0x1601, 0x43)])
def test_mm_small(orc, dev, dt, name, t, top_k, ne, xpr, seed, iseed):
    ids = orc.distinct_ids(t, top_k, ne, iseed)
    got, want = _case(orc, dev, dt, ne, 8, 256, t, top_k, xpr, ids, seed)
    assert orc.rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("dt,name", DTYPES)
def test_mm_production_scale(orc, dev, dt, name):
    # 256 experts, top-10, a 512-token chunk; both activation layouts (src/ops/mm_id.rs:121-166)
    ids = orc.distinct_ids(512, 10, 256, 0x52)
    for xpr, seed in ((1, 0x53), (10, 0x54)):
        got, want = _case(orc, dev, dt, 256, 64, 256, 512, 10, xpr, ids, seed)
        assert orc.rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("dt,name", DTYPES)
def test_mm_ragged_rows_multi_block_k_and_big_expert(orc, dev, dt, name):
    # n_out = 200 (two weight tiles, ragged), k = 768, one expert taking > 256 rows (two row tiles)
    t, top_k, ne = 300, 2, 3
    ids = np.stack([np.zeros(t, np.uint32), 1 + (np.arange(t) % 2).astype(np.uint32)], axis=1)
    got, want = _case(orc, dev, dt, ne, 200, 768, t, top_k, 1, ids, 0x77)
    assert orc.rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("dt,name", DTYPES)
@pytest.mark.parametrize("t,n_out,k", [(80, 128, 256), (82, 130, 1280), (257, 124, 512), (81, 131, 768)])
def test_mm_tile_shapes(orc, dev, dt, name, t, n_out, k):
    """40 and 41 rows an expert and a row past a tile, row counts of the matrix
    that are no multiple of the copy's eight rows or of four, more than four super-blocks.  Both operands are rounded to f16
    (2^-11 each), sums are f32: well under 1e-3."""
    ids = (np.arange(t, dtype=np.uint32) % 2)[:, None]
    got, want = _case(orc, dev, dt, 2, n_out, k, t, 1, 1, ids, 0x90 + t)
    assert orc.rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("dt,name", DTYPES)
@pytest.mark.parametrize("per_expert", [20, 21, 50, 51])
@pytest.mark.parametrize("n_out,k", [(128, 256), (256, 768), (384, 512)])
def test_mm_tile_heights(orc, dev, dt, name, per_expert, n_out, k):
    """Row tiles of 64, 128 and 192 rows on either side of their rule, in single CTAs (odd numbers of 128 weight rows) and in pairs, rows
    of one, two and three blocks (which the groups of a wide stage take in turn), lists that just fit a tile and that just do not.  Bound as in
    test_mm_tile_shapes."""
    counts = [63, 64, 65, 1, 0, 16, 17, 129]
    counts += [0] * 4
    counts[-1] = per_expert * len(counts) - sum(counts) if per_expert * len(counts) >= sum(counts) else 0
    counts += [0] * (-(-sum(counts) // per_expert) - len(counts))
    ids = np.repeat(np.arange(len(counts), dtype=np.uint32), counts)[np.random.default_rng(per_expert).permutation(sum(counts))][:, None]
    got, want = _case(orc, dev, dt, len(counts), n_out, k, sum(counts), 1, 1, ids, 0xC0)
    assert orc.rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("ne", [16, 8, 2])
@pytest.mark.parametrize("dt,name", DTYPES)
def test_mm_operand_bits(dev, dt, name, ne):
    """One-hot activations give the f16 operands themselves.  Both forms of the conversion: a warp's 32 rows all with a small d, all but
    one (at the line itself), all just below the line, all large and of either sign.  Scale and offset are rounded to f16 once and the
    weight once, so the bits are known.  Tiles of 64, 128 and 192 rows."""
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    rng = np.random.default_rng(dt)
    line = 2.0 ** -10 if dt == 12 else 2.0 ** -13
    below = np.nextafter(np.float16(line), np.float16(0))
    d = np.concatenate([rng.uniform(0.55, 0.95, 32) * line, rng.uniform(0.55, 0.95, 32) * line, np.full(32, below),
                        rng.uniform(1.0, 64.0, 32) * line * rng.choice([-1.0, 1.0], 32)]).astype(np.float16)
    d[40] = line
    b = rng.integers(0, 256, (128, 144 if dt == 12 else 210), dtype=np.uint8)
    w = np.zeros((128, 256))
    if dt == 12:
        b[:, 0:2] = d[:, None].view(np.uint8)
        dmin = (rng.uniform(-1.0, 1.0, 128) * 0.01).astype(np.float16)
        b[:, 2:4] = dmin[:, None].view(np.uint8)
        q = b[:, 4:16].astype(np.int32)
        for j in range(8):
            sc, mn = (q[:, j] & 63, q[:, j + 4] & 63) if j < 4 else ((q[:, j + 4] & 15) | (q[:, j - 4] >> 6) << 4, (q[:, j + 4] >> 4) | (q[:, j] >> 6) << 4)
            s, m = (d.astype(np.float64) * sc).astype(np.float16), (-dmin.astype(np.float64) * mn).astype(np.float16)
            n = (b[:, 16 + 32 * (j // 2):48 + 32 * (j // 2)] >> (4 * (j & 1))) & 15
            w[:, 32 * j:32 * j + 32] = n * s.astype(np.float64)[:, None] + m.astype(np.float64)[:, None]
    else:
        b[:, 208:210] = d[:, None].view(np.uint8)
        for n in range(2):
            for g in range(4):
                lo = (b[:, 64 * n + 32 * (g & 1):64 * n + 32 * (g & 1) + 32] >> (4 * (g >> 1))) & 15
                hi = (b[:, 128 + 32 * n:160 + 32 * n] >> (2 * g)) & 3
                sc = np.repeat(b[:, 192 + 8 * n + 2 * g:194 + 8 * n + 2 * g].view(np.int8).astype(np.float64), 16, axis=1)
                s = (d.astype(np.float64)[:, None] * sc).astype(np.float16).astype(np.float64)
                w[:, 128 * n + 32 * g:128 * n + 32 * g + 32] = ((lo | hi << 4).astype(np.float64) - 32.0) * s
    want = w.astype(np.float16).astype(np.float32)
    st = ExpertStack.from_bytes(np.concatenate([b.reshape(-1)] * ne), dt, ne, 128, 256, device=dev)
    got = ops.mul_mm_id(st, torch.eye(256, device=dev).view(256, 1, 256), torch.zeros(256, 1, dtype=torch.int32, device=dev))
    assert np.array_equal(got.cpu().numpy()[:, 0].T, want)


@pytest.mark.parametrize("n_out,k", [(6, 256), (130, 512), (128, 512), (131, 1024), (198, 1024), (129, 2048), (256, 2048), (64, 3072)])
def test_mm_q6k_row_groups(orc, dev, n_out, k):
    """Q6_K rows of one to twelve blocks: lines of one, two, four and eight rows, row counts that they divide and that they do
    not.  The first expert's list is a row longer than a row tile (rows 129 of 5 experts, then 193 of 2).  f16 operands, f32 sums."""
    for ne, t in ((5, 129), (2, 193)):
        got, want = _case(orc, dev, 14, ne, n_out, k, t, 1, 1, np.zeros((t, 1), np.uint32) + (ne == 5), 0xA0 + k)
        assert orc.rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("counts", [(193, 385, 577, 0, 1), (192, 384, 208, 16, 17), (129, 0, 0, 31, 0, 257, 1, 0, 16, 33, 0, 0, 47, 0, 0)])
def test_mm_even_row_tiles(orc, dev, counts):
    """Lists of zero to four row tiles, of heights that do and do not divide, of 192 rows a tile (the first two) and 128.  Bound as in
    test_mm_tile_shapes."""
    ids = np.repeat(np.arange(len(counts), dtype=np.uint32), counts)[np.random.default_rng(len(counts)).permutation(sum(counts))][:, None]
    got, want = _case(orc, dev, 12, len(counts), 64, 256, sum(counts), 1, 1, ids, 0xB0)
    assert orc.rel_l2(got, want) < 1e-3


def test_mm_shared_map0_bitwise_equals_self_contained(orc, dev):
    ids = orc.distinct_ids(96, 4, 8, 0x61)
    a, _ = _case(orc, dev, 12, 8, 64, 512, 96, 4, 1, ids, 0x62, shared_map=False)
    b, _ = _case(orc, dev, 12, 8, 64, 512, 96, 4, 1, ids, 0x62, shared_map=True)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_mm_errors_not_faults(orc, dev):
    from maxuna_b200 import LmoeError, ops
    from maxuna_b200.gguf import ExpertStack

    raw = orc.quantize(12, orc.pseudo_random(4 * 8 * 256, 1, -1.0, 1.0))
    stack = ExpertStack.from_bytes(raw, 12, 4, 8, 256, device=dev)
    ids = torch.zeros(2, 2, dtype=torch.int32, device=dev)
    with pytest.raises(LmoeError):
        ops.mul_mm_id(stack, torch.zeros(2, 1, 128, device=dev), ids)
    scratch = ops.prepare_map0(4, ids)
    with pytest.raises(LmoeError):  # scratch laid out for another geometry
        ops.mul_mm_id_shared(stack, torch.zeros(3, 1, 256, device=dev), torch.zeros(3, 2, dtype=torch.int32, device=dev), scratch)
    assert ops.supported(12, 10) and ops.supported(14, 10) and not ops.supported(8, 10)
    torch.cuda.synchronize()


def _check_block(orc, blk, host, x, tol):
    xd = torch.from_numpy(x).to(blk.router.device)
    out, ids, w = blk.forward(xd, return_routing=True, path="prefill")
    torch.cuda.synchronize()
    blk.check_device_flag()
    want, ids_o, w_o = host.forward(x)
    assert np.array_equal(ids.cpu().numpy().astype(np.uint32), ids_o)
    assert np.array_equal(w.cpu().numpy().view(np.uint32), w_o.view(np.uint32))
    err = orc.rel_l2(out.cpu().numpy(), want)
    assert err < tol, err
    return err


def test_prefill_block_tiny(orc, dev):
    from maxuna_b200.moe import MoeBlock

    blk = MoeBlock.random(256, 256, 8, 3, seed=21, device=dev, weight_std=0.25)
    host = blk.host_layer(orc)
    rng = np.random.default_rng(22)
    for t in (32, 33, 100, 300):
        _check_block(orc, blk, host, rng.standard_normal((t, 256)).astype(np.float32), 2e-3)
    # the op-by-op sequence of the reference (mm_id + rescale + combine) agrees too
    x = rng.standard_normal((64, 256)).astype(np.float32)
    want, _, _ = host.forward(x)
    got = blk.forward_unfused(torch.from_numpy(x).to(dev), use_mm=True).cpu().numpy()
    assert orc.rel_l2(got, want) < 2e-3


@pytest.mark.parametrize("hidden,ff", [(256, 256), (512, 768), (768, 256)])
@pytest.mark.parametrize("t", [80, 81, 200, 201])
def test_prefill_block_tile_heights(orc, dev, hidden, ff, t):
    """The fused gate/up product on either side of the rule for row tiles (20 and 50 rows an expert), with rows of one, two and three
    blocks in both products.  Bound as above."""
    from maxuna_b200.moe import MoeBlock

    blk = MoeBlock.random(hidden, ff, 8, 2, seed=hidden + ff, device=dev, weight_std=0.1)
    _check_block(orc, blk, blk.host_layer(orc), np.random.default_rng(t).standard_normal((t, hidden)).astype(np.float32), 2e-3)


@pytest.mark.parametrize("hidden,ne,top_k,t,bias", [(3072, 256, 10, 641, False), (3072, 256, 10, 771, False), (3072, 256, 10, 2501, True), (4096, 96, 12, 1531, True),
                                                    (1024, 256, 32, 2401, False), (512, 96, 8, 18313, True), (768, 128, 1, 5089, False),
                                                    (1280, 64, 8, 5001, True)])
def test_prefill_routing_through_the_filter(dev, hidden, ne, top_k, t, bias):
    """Long prompts take the tensor core's bounds first: ids and weights are those of the stand-alone routing, which are the oracle's, to
    the bit.  Both token tiles of either kernel, ragged counts; tokens that keep all experts (an infinity, NaN, values beyond the f16
    range, zeros: every score ties), tiny and large ones, router rows that are equal and a bias that excludes an expert."""
    from maxuna_b200.moe import MoeBlock

    gen = torch.Generator(device=dev)
    gen.manual_seed(t)
    b = 0.2 * torch.rand(ne, generator=gen, device=dev) - 0.1 if bias else None
    if bias:
        b[3], b[5], b[7] = float("-inf"), b[6], 40.0
    blk = MoeBlock.random(hidden, 256, ne, top_k, seed=hidden + ne, device=dev, bias=b)
    blk.router[6] = blk.router[5]
    blk.router[ne - 1] = blk.router[0]
    x = torch.randn(t, hidden, generator=gen, device=dev)
    x[2] = 0.0
    x[3] *= 1e-6
    x[5] *= 300.0
    x[7, 11] = 1e6
    x[t // 2, 4] = float("inf")
    x[t // 2 + 1, 9] = float("nan")
    x[t - 1, 0] = 7e4
    left = _check_routing(blk, x)
    # ordinary tokens keep little more than top_k; about a dozen here keep them all
    assert t * top_k <= left <= t * (1.5 * top_k + 3) + 12 * ne


def _check_routing(blk, x, with_handed=False):
    """Ids and weights of a prompt against the stand-alone routing, to the bit; returns the count of experts that the filter left
    (0: the filter did not run), and that of the tokens that got all their logits."""
    blk.workspace(x.shape[0])[:32].zero_()
    _, ids, w = blk.forward(x, return_routing=True, path="prefill")
    ids2, w2 = blk.route(x)
    torch.cuda.synchronize()
    left, handed = blk.workspace(x.shape[0])[16:24].view(torch.int32).tolist()
    blk.check_device_flag()
    assert torch.equal(ids, ids2) and torch.equal(w.view(torch.int32), w2.view(torch.int32))
    return (left, handed) if with_handed else left


@pytest.mark.parametrize("value", [float("-inf"), torch.finfo(torch.float32).min, -1e9, float("inf"), float("nan")])
@pytest.mark.parametrize("hidden,ne,top_k,t", [(3072, 256, 10, 2048), (4096, 96, 8, 2500)])
def test_prefill_routing_filter_with_any_bias(dev, hidden, ne, top_k, t, value):
    """An expert that its bias excludes or fixes, by an infinity, the type's lowest value or NaN, leaves the other experts' bounds as they
    are."""
    from maxuna_b200.moe import MoeBlock

    gen = torch.Generator(device=dev)
    gen.manual_seed(t)
    b = 0.2 * torch.rand(ne, generator=gen, device=dev) - 0.1
    b[3] = value
    blk = MoeBlock.random(hidden, 256, ne, top_k, seed=hidden + ne, device=dev, bias=b)
    left = _check_routing(blk, torch.randn(t, hidden, generator=gen, device=dev))
    assert t * top_k <= left <= t * (1.5 * top_k + 3)


def test_prefill_routing_filter_with_small_scores(dev):
    """Scores near 1e-6 are told apart as well as others: the bounds are relative."""
    from maxuna_b200.moe import MoeBlock

    gen = torch.Generator(device=dev)
    gen.manual_seed(14)
    blk = MoeBlock.random(3072, 256, 256, 10, seed=14, device=dev, bias=torch.zeros(256, device=dev))
    x = torch.randn(2048, 3072, generator=gen, device=dev)
    x[:, 0] = 10.0
    blk.router[:, 0] = -1.4
    left = _check_routing(blk, x)
    assert 2048 * 10 <= left <= 2048 * 30


@pytest.mark.parametrize("hidden,ne,top_k,t,hands", [(3072, 256, 10, 2501, True), (3072, 256, 10, 801, True), (1024, 256, 32, 20001, True), (4096, 96, 12, 1531, True),
                                                     (512, 96, 8, 18313, True), (768, 128, 1, 5089, False)])
@pytest.mark.parametrize("case", ["all", "runs", "few"])
def test_prefill_routing_where_bounds_do_not_tell(dev, hidden, ne, top_k, t, hands, case):
    """Tokens whose scores all tie, or whose bounds are wider than the scores' differences, get all their logits from the tiled product: every token, runs of
    them between ordinary ones, or one in fifty, which most blocks compute themselves.  Tile heights of 16 and 8, ragged last tiles, more and fewer tiles than SMs; a hidden
    size that the tiled product does not take."""
    from maxuna_b200.moe import MoeBlock

    gen = torch.Generator(device=dev)
    gen.manual_seed(t)
    blk = MoeBlock.random(hidden, 256, ne, top_k, seed=hidden + ne, device=dev, bias=torch.zeros(ne, device=dev))
    x = torch.randn(t, hidden, generator=gen, device=dev)
    blk.router[:, 7] = blk.router[0, 7]  # a channel that no expert prefers: a large value in it widens the bounds only
    at = torch.arange(t, device=dev)
    tie = {"all": at >= 0, "runs": at // 37 % 2 == 0, "few": at % 50 == 13}[case]
    x[tie, 7] = 3e4 * (1 - 2 * (at[tie] % 2).float())
    left, handed = _check_routing(blk, x, with_handed=True)
    ties = int(tie.sum())
    assert left >= ties * ne // 2 + (t - ties) * top_k
    assert (ties // 2 if hands and case != "few" else 0) <= handed <= (t if hands else 0)


@pytest.mark.parametrize("hidden,ne,top_k,t", [(3072, 256, 10, 2501), (3072, 256, 10, 801), (4096, 96, 12, 1531), (768, 128, 1, 5089)])
@pytest.mark.parametrize("bias", [False, True])
def test_prefill_routing_of_rows_of_zeros(dev, hidden, ne, top_k, t, bias):
    """A padded prompt: rows of zeros, of values too small for their squares and of values whose logits just reach 2^-27 get their ids without a
    logit, larger ones not; a router of zeros."""
    from maxuna_b200.moe import MoeBlock

    gen = torch.Generator(device=dev)
    gen.manual_seed(t)
    b = 0.2 * torch.rand(ne, generator=gen, device=dev) - 0.1 if bias else torch.zeros(ne, device=dev)
    blk = MoeBlock.random(hidden, 256, ne, top_k, seed=hidden + ne, device=dev, bias=b)
    x = torch.randn(t, hidden, generator=gen, device=dev)
    at = torch.arange(t, device=dev)
    small = torch.tensor([0.0, 1e-25, 1e-20, 2.0 ** -40, 2.0 ** -33, 2.0 ** -30, 2.0 ** -24], device=dev)
    pad = at % 16 >= 9
    x[pad] *= small[at[pad] % 16 - 9][:, None]
    left = _check_routing(blk, x)
    ordinary = int((~pad).sum())
    # of the seven kinds of small rows the last three may count as others do
    assert ordinary * top_k <= left <= ordinary * (1.5 * top_k + 3) + 3 * t // 16 * ne
    blk.router.zero_()
    assert _check_routing(blk, x) == 0


def test_prefill_block_wide_ff(orc, dev):
    # expert_ff = 512: two Q6_K super-blocks per down row (the 256-row down kernel), ragged row tiles
    from maxuna_b200.moe import MoeBlock

    blk = MoeBlock.random(256, 512, 6, 2, seed=31, device=dev, weight_std=0.25)
    host = blk.host_layer(orc)
    rng = np.random.default_rng(32)
    for t in (40, 700):
        _check_block(orc, blk, host, rng.standard_normal((t, 256)).astype(np.float32), 2e-3)


def test_prefill_block_production_shape(orc, dev):
    from maxuna_b200.moe import MoeBlock

    blk = MoeBlock.random(3072, 1024, 256, 10, seed=2, device=dev)
    host = blk.host_layer(orc)
    x = np.random.default_rng(23).standard_normal((48, 3072)).astype(np.float32)
    _check_block(orc, blk, host, x, 2e-3)


@pytest.mark.parametrize("hidden,ff,ne,top_k,up_dt,t", [(256, 256, 4, 2, 12, 7), (512, 1536, 8, 3, 12, 100), (1024, 768, 16, 4, 14, 333),
                                                        (256, 2048, 3, 2, 12, 300)])
def test_ffn_mm_equals_the_ops(dev, hidden, ff, ne, top_k, up_dt, t):
    """One call for the grouped-GEMM chain gives the bits of its ops one by one: both tile widths, rows of one to eight blocks,
    several widths, and an id that names no expert (which counts nothing here)."""
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    mk = lambda dt, o, k, s: ExpertStack.random(dt, ne, o, k, seed=s, device=dev)
    e = (mk(12, ff, hidden, 1), mk(up_dt, ff, hidden, 2), mk(14, hidden, ff, 3))
    gen = torch.Generator(device=dev)
    gen.manual_seed(t)
    x = torch.randn(t, hidden, generator=gen, device=dev)
    x[t // 2] *= 1e4
    ids = torch.stack([torch.randperm(ne, generator=gen, device=dev)[:top_k] for _ in range(t)]).to(torch.int32)
    w = torch.rand(t, top_k, generator=gen, device=dev)
    m, xg = ops.prepare_map0(ne, ids), x.view(t, 1, hidden)
    act, l2 = ops.l2_rescale(ops.silu_mul(ops.mul_mm_id_shared(e[0], xg, ids, m), ops.mul_mm_id_shared(e[1], xg, ids, m)))
    want = ops.combine(ops.mul_mm_id_shared(e[2], act, ids, m), l2, w)
    assert torch.equal(ops.ffn_mm(e, ids, w, x).view(torch.int32), want.view(torch.int32))
    ids[0, 0] = ne + 1
    got = ops.ffn_mm(e, ids, w, x)
    assert torch.isfinite(got).all() and torch.equal(got[1:], want[1:])


@pytest.mark.parametrize("ff", [256, 768, 1024, 1792, 4096, 12288])
def test_ffn_mm_wide_rows(dev, ff):
    """Activation rows from one warp pair a block to the widest that fits, whole and broken turns of its threads: the bits of the
    ops one by one, and a slot whose id names no expert is a zero row."""
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    ne, t, top_k, hidden = 3, 70, 2, 256
    mk = lambda dt, o, k, s: ExpertStack.random(dt, ne, o, k, seed=s, device=dev)
    e = (mk(12, ff, hidden, 1), mk(12, ff, hidden, 2), mk(14, hidden, ff, 3))
    gen = torch.Generator(device=dev)
    gen.manual_seed(ff)
    x = torch.randn(t, hidden, generator=gen, device=dev)
    ids = torch.stack([torch.randperm(ne, generator=gen, device=dev)[:top_k] for _ in range(t)]).to(torch.int32)
    ids[5, 1] = ne
    w = torch.rand(t, top_k, generator=gen, device=dev)
    m, xg = ops.prepare_map0(ne, ids), x.view(t, 1, hidden)
    act, l2 = ops.l2_rescale(ops.silu_mul(ops.mul_mm_id_shared(e[0], xg, ids, m), ops.mul_mm_id_shared(e[1], xg, ids, m)))
    down = ops.mul_mm_id_shared(e[2], act, ids, m)
    down[5, 1], l2[5, 1] = 0.0, 1.0
    want = ops.combine(down, l2, w)
    assert torch.equal(ops.ffn_mm(e, ids, w, x).view(torch.int32), want.view(torch.int32))


def test_combine_after_a_wait_that_ran_out(dev):
    """The sum that ends `lmoe_ffn_mm` on products whose device flag is set: NaN, not a wrong finite row; on a clean flag the sum."""
    import ctypes as C

    from maxuna_b200 import ops
    from maxuna_b200._native import lib
    from maxuna_b200.gguf import stream_ptr

    # launch_combine(down, col_l2, w, seq, top_k, n_out, out, stream, flag) of csrc/glue.cu
    f = lib()._Z14launch_combinePKfS0_S0_iiiPfP11CUstream_stPKj
    f.argtypes = [C.c_void_p] * 3 + [C.c_int] * 3 + [C.c_void_p] * 3
    for n_out in (64, 65):  # four columns a thread, and one
        down, w = torch.randn(5, 3, n_out, device=dev), torch.rand(5, 3, device=dev)
        for flag in (0, 2):
            word, out = torch.tensor([flag, 0, 0, 0], dtype=torch.int32, device=dev), torch.zeros(5, n_out, device=dev)
            assert f(down.data_ptr(), None, w.data_ptr(), 5, 3, n_out, out.data_ptr(), stream_ptr(), word.data_ptr()) == 0
            assert torch.isnan(out).all() if flag else torch.equal(out, ops.combine(down, None, w))


@pytest.mark.parametrize("dt,name", DTYPES)
@pytest.mark.parametrize("n_out", [1, 128, 129, 257, 640, 1664, 1665, 1800, 1921])
def test_mm_single_and_paired_ctas(orc, dev, dt, name, n_out):
    """Odd numbers of blocks of 128 weight rows go to single CTAs up to 13, the others to pairs: either side of the rule, last blocks of
    one row and full ones, a pair whose second CTA has no row, both row-tile heights.  Bound as in test_mm_tile_shapes."""
    for t, k in ((70, 512), (200, 256)):
        ids = (np.arange(t, dtype=np.uint32) % 2)[:, None]
        got, want = _case(orc, dev, dt, 2, n_out, k, t, 1, 1, ids, 0xC0 + n_out)
        assert orc.rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("dt,name", DTYPES)
@pytest.mark.parametrize("n_out,k,t", [(384, 256, 100), (384, 512, 700), (512, 256, 700), (512, 512, 100)])
def test_mm_repeated_calls_are_bitwise_equal(dev, dt, name, n_out, k, t):
    """Many tiles of few stages, so that every hand-over between the warps and the CTAs of a pair comes round often: a stale operand
    would show as a difference between calls on the same inputs."""
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    ne, top_k = 48, 8
    st = ExpertStack.random(dt, ne, n_out, k, seed=7, device=dev)
    gen = torch.Generator(device=dev)
    gen.manual_seed(t)
    x = torch.randn(t, 1, k, generator=gen, device=dev)
    ids = torch.rand(t, ne, generator=gen, device=dev).argsort(1)[:, :top_k].to(torch.int32).contiguous()
    m = ops.prepare_map0(ne, ids)
    want = ops.mul_mm_id_shared(st, x, ids, m).view(torch.int32)
    for _ in range(50):
        assert torch.equal(ops.mul_mm_id_shared(st, x, ids, m).view(torch.int32), want)


def test_ffn_mm_id_without_expert_in_a_stale_workspace(dev):
    """A slot whose id names no expert is a zero row of the sum, whatever the workspace held: all bytes 0xFF (NaN, and positions that
    the lists would have to overwrite) and all zero (positions of the first row)."""
    from maxuna_b200 import ops
    from maxuna_b200._native import check, lib
    from maxuna_b200.gguf import ExpertStack, stream_ptr

    ne, t, top_k, hidden, ff = 4, 40, 2, 256, 512
    mk = lambda dt, o, k, s: ExpertStack.random(dt, ne, o, k, seed=s, device=dev)
    g, u, d = mk(12, ff, hidden, 1), mk(12, ff, hidden, 2), mk(14, hidden, ff, 3)
    x, w = torch.randn(t, hidden, device=dev), torch.rand(t, top_k, device=dev)
    ids = torch.stack([torch.randperm(ne, device=dev)[:top_k] for _ in range(t)]).to(torch.int32)
    ids[0, 0], ids[7, 1], ids[9] = ne, -1, ne + 3
    m, xg = ops.prepare_map0(ne, ids), x.view(t, 1, hidden)
    act, l2 = ops.l2_rescale(ops.silu_mul(ops.mul_mm_id_shared(g, xg, ids, m), ops.mul_mm_id_shared(u, xg, ids, m)))
    down = ops.mul_mm_id_shared(d, act, ids, m)
    gone = (ids < 0) | (ids >= ne)
    down[gone], l2[gone] = 0.0, 1.0
    want = ops.combine(down, l2, w)
    n = lib().lmoe_ffn_mm_workspace_bytes(g.handle, d.handle, t, top_k)
    for fill in (0xFF, 0):
        ws, out = torch.full((n,), fill, dtype=torch.uint8, device=dev), torch.empty(t, hidden, device=dev)
        check(lib().lmoe_ffn_mm(g.handle, u.handle, d.handle, ids.data_ptr(), t, top_k, w.data_ptr(), x.data_ptr(), t, hidden, out.data_ptr(),
                                ws.data_ptr(), n, stream_ptr()))
        assert torch.equal(out.view(torch.int32), want.view(torch.int32))
        check(lib().lmoe_check_device_flag(ws.data_ptr(), stream_ptr()))


def test_fused_experts_wider_than_the_one_call(dev, monkeypatch):
    """`FusedExperts.forward` calls the ops one by one for experts wider than `lmoe_ffn_mm` takes: the same bits."""
    from maxuna_b200 import ops
    from maxuna_b200.moe import MoeBlock

    blk = MoeBlock.random(512, 768, 8, 3, seed=4, device=dev)
    x = torch.randn(90, 512, device=dev)
    want = blk.forward_unfused(x, use_mm=True)
    monkeypatch.setattr(ops, "FFN_MM_MAX_FF", 512)
    monkeypatch.setattr(ops, "ffn_mm", None)
    assert torch.equal(blk.forward_unfused(x, use_mm=True).view(torch.int32), want.view(torch.int32))
