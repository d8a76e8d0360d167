"""Op-level parity on the GPU, through the C ABI, against the CPU oracle.

The cases follow the reference's on-device kernel tests: mul_mv_id
(src/ops/mv_id.rs:100-203), combine / silu_mul (src/ops/combine.rs:76-124,
src/ops/silu_mul.rs:58-99), routing (src/moe.rs:405-500), with the reference's
bound of rel-L2 < 1e-3 against the dequantize-then-dot oracle and bit-exact
expert ids.
"""
import json
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

GOLD = os.path.join(os.path.dirname(__file__), "golden")
DTYPES = [(12, "Q4K"), (14, "Q6K")]


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    return torch.device("cuda:0")


def _stack(orc, dev, dt, n_expert, n_out, k, seed):
    from maxuna_b200.gguf import ExpertStack

    w = orc.pseudo_random(n_expert * n_out * k, seed, -1.0, 1.0)
    raw = orc.quantize(dt, w)
    return ExpertStack.from_bytes(raw, dt, n_expert, n_out, k, device=dev), raw


def _run_mv(orc, dev, dt, n_expert, n_out, k, t, top_k, xpr, ids, seed, base_off=0):
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    w = orc.pseudo_random(n_expert * n_out * k, seed, -1.0, 1.0)
    raw = orc.quantize(dt, w)
    stack = ExpertStack.from_bytes(raw, dt, n_expert, n_out, k, device=dev, base_off=base_off)
    x = orc.pseudo_random(t * xpr * k, seed ^ 0xABCD, -1.0, 1.0).reshape(t, xpr, k)
    got = ops.mul_mv_id(stack, torch.from_numpy(x).to(dev), torch.from_numpy(ids.astype(np.int32)).to(dev))
    assert tuple(got.shape) == (t, top_k, n_out)
    want = orc.mul_id(dt, raw, n_expert, n_out, k, x, ids)
    return got.cpu().numpy(), want


@pytest.mark.parametrize("dt,name", DTYPES)
def test_mv_shared_row_gate_up(orc, dev, dt, name):
    ids = orc.random_ids(3, 2, 4, 0x11)
    got, want = _run_mv(orc, dev, dt, 4, 8, 256, 3, 2, 1, ids, 0x100)
    assert orc.rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("dt,name", DTYPES)
def test_mv_per_slot_row_down(orc, dev, dt, name):
    ids = orc.random_ids(5, 4, 4, 0x22)
    got, want = _run_mv(orc, dev, dt, 4, 8, 256, 5, 4, 4, ids, 0x200)
    assert orc.rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("dt,name", DTYPES)
def test_mv_repeated_expert_ids(orc, dev, dt, name):
    ids = np.ones((4, 3), np.uint32)
    got, want = _run_mv(orc, dev, dt, 4, 8, 256, 4, 3, 1, ids, 0x300)
    assert orc.rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("dt,name", DTYPES)
def test_mv_ragged_n_out_and_two_blocks(orc, dev, dt, name):
    # n_out = 100 (ragged last row group), k = 512 = two super-blocks per row
    for xpr, seed, iseed in ((1, 0x100, 0x11), (4, 0x200, 0x22)):
        ids = orc.random_ids(5, 4, 8, iseed)
        got, want = _run_mv(orc, dev, dt, 8, 100, 512, 5, 4, xpr, ids, seed)
        assert orc.rel_l2(got, want) < 1e-3


def test_mv_base_off_bitwise(orc, dev):
    ids = orc.random_ids(3, 2, 4, 0x44)
    a, _ = _run_mv(orc, dev, 12, 4, 8, 256, 3, 2, 1, ids, 0x0FF5E7, base_off=0)
    b, _ = _run_mv(orc, dev, 12, 4, 8, 256, 3, 2, 1, ids, 0x0FF5E7, base_off=96)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_mv_shape_mismatch_errors(orc, dev):
    from maxuna_b200 import LmoeError, ops

    stack, _ = _stack(orc, dev, 12, 4, 8, 256, 1)
    x = torch.zeros(1, 1, 128, device=dev)
    ids = torch.zeros(1, 2, dtype=torch.int32, device=dev)
    with pytest.raises(LmoeError):
        ops.mul_mv_id(stack, x, ids)
    with pytest.raises(LmoeError):
        ops.mul_mv_id(stack, torch.zeros(2, 1, 256, device=dev), ids)  # ids t != x t
    with pytest.raises(LmoeError):
        ops.mul_mv_id(stack, torch.zeros(1, 1, 256, device=dev, dtype=torch.float16), ids)
    torch.cuda.synchronize()  # the context must still be healthy


@pytest.mark.parametrize("dt,name", DTYPES)
@pytest.mark.parametrize("n_expert,n_out,k,t,top_k,xpr", [
    (1, 64, 256, 3, 1, 1), (1, 65, 512, 4, 1, 1), (1, 63, 1280, 33, 1, 1), (1, 130, 3072, 5, 13, 13),  # one matrix: 3 / 4 / 33 / 65 pairs
    (3, 127, 768, 2, 3, 3), (2, 16, 8192 + 256, 1, 2, 1)])                                            # odd block counts, two staged chunks
def test_mv_tile_edges(orc, dev, dt, name, n_expert, n_out, k, t, top_k, xpr):
    """Row, pair and K edges of little work, an empty slot and an outlier channel.  Bound: activations and sums are f32 or better
    and the oracle's own f32 sums err by about sqrt(k) * 2^-24 (5e-6 at 8448)."""
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    raw = orc.quantize(dt, orc.pseudo_random(n_expert * n_out * k, 0x900 + k, -1.0, 1.0))
    stack = ExpertStack.from_bytes(raw, dt, n_expert, n_out, k, device=dev)
    x = orc.pseudo_random(t * xpr * k, 0x33, -1.0, 1.0).reshape(t, xpr, k)
    x[0, 0, 7] = 50.0
    ids = (np.arange(t * top_k, dtype=np.uint32) % n_expert).reshape(t, top_k)
    got = ops.mul_mv_id(stack, torch.from_numpy(x).to(dev), torch.from_numpy(ids.astype(np.int32)).to(dev)).cpu().numpy()
    assert orc.rel_l2(got, orc.mul_id(dt, raw, n_expert, n_out, k, x, ids)) < 1e-5
    ids[t - 1, top_k - 1] = n_expert
    hole = ops.mul_mv_id(stack, torch.from_numpy(x).to(dev), torch.from_numpy(ids.astype(np.int32)).to(dev)).cpu().numpy()
    assert not hole[t - 1, top_k - 1].any()
    hole[t - 1, top_k - 1] = got[t - 1, top_k - 1]
    assert np.array_equal(hole, got)


@pytest.mark.parametrize("n_expert,n_out,k,t,top_k", [
    (3, 8, 256, 2, 2),       # one super-block per row, one unit shorter than a row tile
    (5, 72, 512, 7, 3),      # two; three to five pairs of an expert
    (4, 200, 768, 9, 2),     # three: rows of odd word alignment (Q6_K), a tail unit
    (2, 136, 1280, 6, 1),    # five: a second turn of the K split for one warp only
    (7, 40, 256, 700, 3),    # more pairs than an expert's are looked for among, many blocks of each expert
    (3, 1032, 4096, 3, 3),   # more shared memory than two blocks of an SM have
    # the same edges with as many rows as the form needs in order to be taken
    (3, 64, 256, 130, 2), (5, 72, 512, 80, 3), (4, 200, 768, 41, 2), (2, 136, 1280, 61, 1), (7, 72, 256, 700, 3),
    (3, 520, 3584, 3, 3), (3, 520, 5120, 3, 3),  # one block an SM: Q6_K, Q4_K
])
@pytest.mark.parametrize("dt,name", DTYPES)
def test_mv_pairs_by_expert(orc, dev, dt, name, n_expert, n_out, k, t, top_k):
    """Pairs grouped by expert, and the same by rows where that is the faster form: group, unit and K edges, repeated experts in
    any order, empty slots.  Bound as above."""
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    raw = orc.quantize(dt, orc.pseudo_random(n_expert * n_out * k, 0x700 + k, -1.0, 1.0))
    stack = ExpertStack.from_bytes(raw, dt, n_expert, n_out, k, device=dev)
    x = orc.pseudo_random(t * k, 0x35, -1.0, 1.0).reshape(t, 1, k)
    ids = np.random.default_rng(t).integers(0, n_expert + 1, (t, top_k)).astype(np.uint32)  # n_expert: an empty slot
    got = ops.mul_mv_id(stack, torch.from_numpy(x).to(dev), torch.from_numpy(ids.astype(np.int32)).to(dev)).cpu().numpy()
    assert not got[ids == n_expert].any()
    want = orc.mul_id(dt, raw, n_expert, n_out, k, x, np.minimum(ids, n_expert - 1))
    want[ids == n_expert] = 0
    assert orc.rel_l2(got, want) < 1e-5


@pytest.mark.parametrize("n_out,k,pairs", [
    (72, 256, 2369),    # row blocks by themselves, one pair in the last group
    (256, 1280, 1185),  # one whole cluster of row blocks, a second staged run of k
    (1100, 512, 285),   # the last cluster has blocks without rows
])
@pytest.mark.parametrize("dt,name", DTYPES)
def test_mv_many_pairs_of_one_matrix(orc, dev, dt, name, n_out, k, pairs):
    """The many-pair form at the edges of its row blocks, clusters and pair groups, and empty slots.  Bound as above."""
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    raw = orc.quantize(dt, orc.pseudo_random(n_out * k, 0x500 + k, -1.0, 1.0))
    stack = ExpertStack.from_bytes(raw, dt, 1, n_out, k, device=dev)
    x = orc.pseudo_random(pairs * k, 0x36, -1.0, 1.0).reshape(pairs, 1, k)
    ids = (np.arange(pairs, dtype=np.uint32) % 7 == 3).astype(np.uint32)[:, None]  # 1: an empty slot
    got = ops.mul_mv_id(stack, torch.from_numpy(x).to(dev), torch.from_numpy(ids.astype(np.int32)).to(dev)).cpu().numpy()
    want = orc.mul_id(dt, raw, 1, n_out, k, x, np.zeros_like(ids))
    want[ids == 1] = 0
    assert not got[ids == 1].any() and orc.rel_l2(got, want) < 1e-5


@pytest.mark.parametrize("n_out,k,t,top_k,xpr", [
    (130, 256, 2001, 1, 1),   # one super-block, two rows in the last block, one token in the last group
    (1000, 1280, 167, 2, 2),  # an odd number of super-blocks; a row of x for every slot
    (390, 768, 513, 2, 1),    # slots that share a row of x
    (128, 512, 8200, 1, 1),   # several rounds over the device
    (131, 768, 1201, 1, 1),   # an odd number of blocks in all: the last Q6_K one ends in the middle of a word
])
@pytest.mark.parametrize("dt,name", DTYPES)
def test_mv_dense(orc, dev, dt, name, n_out, k, t, top_k, xpr):
    """One matrix and many pairs on the tensor cores: ragged rows and pairs, empty slots, values that span the range of f32, an infinity
    and NaN that stay in their rows.  Exact products and sums but for the f32 roundings once a super-block: bound as in
    test_mv_range_and_resolution, against 64-bit sums."""
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    raw = orc.quantize(dt, orc.pseudo_random(n_out * k, 0xD00 + k, -1.0, 1.0))
    stack = ExpertStack.from_bytes(raw, dt, 1, n_out, k, device=dev)
    rng = np.random.default_rng(t)
    ids = (np.arange(t * top_k, dtype=np.uint32) % 11 == 4).astype(np.uint32).reshape(t, top_k)  # 1: an empty slot
    run = lambda v: ops.mul_mv_id(stack, torch.from_numpy(v).to(dev), torch.from_numpy(ids.astype(np.int32)).to(dev)).cpu().numpy()
    x = rng.standard_normal((t, xpr, k)).astype(np.float32)
    x[0::3, :, 7::256] *= 1e4
    x[2::3] *= (2.0 ** rng.integers(-60, 60, (len(x[2::3]), 1, 1))).astype(np.float32)
    got = run(x)
    w = stack.dequantize()[0].double()
    want = torch.from_numpy(x).to(dev).double() @ w.T  # [t, xpr, n_out]
    want = want.expand(t, top_k, n_out).cpu().numpy() if xpr == 1 else want.cpu().numpy()
    assert not got[ids == 1].any()
    err = np.linalg.norm(got - want, axis=2) / np.linalg.norm(want, axis=2)
    assert err[ids == 0].max() < 8 * 2.0 ** -24
    x[3, 0, 40], x[5, 0, 11] = np.inf, np.nan
    bad, keep = run(x), [r for r in range(t) if r not in (3, 5)]
    assert not np.isfinite(bad[3, 0]).any() and np.isnan(bad[5, 0]).all() and np.array_equal(bad[keep], got[keep])


@pytest.mark.parametrize("case", ["top", "low", "negative"])
@pytest.mark.parametrize("dt,name", DTYPES)
def test_mv_dense_large_sums(dev, dt, name, case):
    """A super-block's sums at their largest: weights of one sign and near the largest integers, activations of one sign whose leading
    (`top`) or lower (`low`) bits are nearly all set, an odd number of weight rows and of super-blocks.  The sums of a super-block are exact, d and the
    scale of the activations are powers of two and the mins are zero, so what rounds, by 2^-24 of its own size, are the additions of the digits' sums: two at up to the size of the
    result, the lower ones a hundredth of that; for Q6_K these two in the part that comes in eight times (at most 1 + 4 / 121 of the result), and then the
    addition of the other part."""
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    n_out, k, t = 131, 256, 2001
    rng = np.random.default_rng(dt)
    b = np.zeros((n_out, 144 if dt == 12 else 210), dtype=np.uint8)
    if dt == 12:
        b[:, 0:2] = np.float16(2.0 ** -7).reshape(1).view(np.uint8)
        sc = rng.integers(58, 64, (n_out, 8))  # scales; the mins are zero
        b[:, 4:8] = sc[:, :4] | (sc[:, 4:] >> 4) << 6
        b[:, 12:16] = sc[:, 4:] & 15
        q = rng.integers(13, 16, (n_out, 8, 32))
        b[:, 16:144] = (q[:, 0::2] | q[:, 1::2] << 4).reshape(n_out, 128)
    else:
        b[:, 208:210] = np.float16(2.0 ** -7).reshape(1).view(np.uint8)
        b[:, 192:208] = rng.integers(-128, -120, (n_out, 16)).astype(np.int8).view(np.uint8)  # times values of -32 to -29
        b[:, 0:128] = rng.integers(0, 4, (n_out, 128)) * 0x11
    stack = ExpertStack.from_bytes(b.reshape(-1), dt, 1, n_out, k, device=dev)
    bits = rng.integers(0, 1 << 5, (t, k)) * 0x010101  # five low bits of every byte at random, the others set
    x = (0x7F0000 | 0x6060 | bits & 0x1F1F1F if case == "low" else 0xE06060 | bits).astype(np.int64)
    x = (x if case == "low" else x << 6).astype(np.float64) * 2.0 ** -29
    x[:, 17] = 1.0 if case == "low" else 1.96875  # the block's scale: 2^29 integers to 1
    x = (-x if case == "negative" else x).astype(np.float32).reshape(t, 1, k)
    got = ops.mul_mv_id(stack, torch.from_numpy(x).to(dev), torch.zeros(t, 1, dtype=torch.int32, device=dev)).cpu().numpy()[:, 0]
    want = (torch.from_numpy(x).to(dev).double()[:, 0] @ stack.dequantize()[0].double().T).cpu().numpy()
    assert np.abs(got / want - 1).max() < (2.1 if dt == 12 else 3.2) * 2.0 ** -24


@pytest.mark.parametrize("n_expert,n_out,k,t,top_k", [(4, 512, 768, 17, 2), (1, 1100, 512, 285, 1), (1, 64, 8192, 40, 1)])
@pytest.mark.parametrize("dt,name", DTYPES)
def test_mv_range_and_resolution(orc, dev, dt, name, n_expert, n_out, k, t, top_k):
    """The forms for pairs by expert, for one matrix and for long rows, with activations that have one value of a block 10^4
    times the others, that are products (as SwiGLU's are), and that span the range of f32.  Bound against 64-bit sums: values
    are held to 2^-30 of their block's largest, and a result is some eight f32 roundings away from exact sums of up to twice
    its size; blocks below 2^-97 are held to 2^-126.  Infinities and NaN stay in their rows."""
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    raw = orc.quantize(dt, orc.pseudo_random(n_expert * n_out * k, 0xA00 + k, -1.0, 1.0))
    stack = ExpertStack.from_bytes(raw, dt, n_expert, n_out, k, device=dev)
    rng = np.random.default_rng(k)
    ids = (np.arange(t * top_k, dtype=np.uint32) % n_expert).reshape(t, top_k)
    run = lambda v: ops.mul_mv_id(stack, torch.from_numpy(v).to(dev), torch.from_numpy(ids.astype(np.int32)).to(dev)).cpu().numpy()
    x = rng.standard_normal((t, 1, k)).astype(np.float32)
    x[0::3, 0, 7::256] *= 1e4
    x[1::3] *= rng.standard_normal(x[1::3].shape).astype(np.float32)
    x[2::3] *= (2.0 ** rng.integers(-60, 60, (len(x[2::3]), 1, 1))).astype(np.float32)
    got, want = run(x), orc.mul_id(dt, raw, n_expert, n_out, k, x, ids, accum64=True)
    for r in range(t):
        scale = 1.0 / np.abs(want[r]).max()
        assert orc.rel_l2(got[r] * scale, want[r] * scale) < 8 * 2.0 ** -24
    tiny = np.zeros_like(x)
    tiny[:, 0, 5], tiny[0, 0, 300], tiny[1, 0, 9] = 1e-33, 1e-42, 3e-34
    got, want = run(tiny), orc.mul_id(dt, raw, n_expert, n_out, k, tiny, ids, accum64=True)
    assert np.isfinite(got).all() and orc.rel_l2(got * np.float64(1e30), want * np.float64(1e30)) < 1e-4
    base = run(x)
    x[3, 0, 40], x[5, 0, 11] = np.inf, np.nan
    got, keep = run(x), [r for r in range(t) if r not in (3, 5)]
    assert not np.isfinite(got[3]).any() and np.isnan(got[5]).all() and np.array_equal(got[keep], base[keep])


@pytest.mark.parametrize("n_expert,n_out,k,pairs", [
    (3, 1024, 256, (7, 8, 15, 16)), (2, 1024, 1024, (3, 4, 8, 9)), (2, 512, 2048, (4, 5)), (2, 512, 3072, (3, 4)),  # rows by length
    (1, 31, 512, (600,)), (1, 32, 512, (600,)), (1, 63, 768, (300,)), (1, 64, 768, (300,)), (2, 15, 2048, (300,)), (2, 16, 2048, (300,)),
    (3, 100, 768, (200,)), (2, 64, 8192, (31, 32, 40)), (1, 7, 32768 + 256, (2,))])                              # ring misses
@pytest.mark.parametrize("dt,name", DTYPES)
def test_mv_forms_agree(orc, dev, dt, name, n_expert, n_out, k, pairs):
    """Both sides of every line between the mat-vec forms: the same product, to the roundings of the two evaluations."""
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    raw = orc.quantize(dt, orc.pseudo_random(n_expert * n_out * k, 0xB00 + k, -1.0, 1.0))
    stack = ExpertStack.from_bytes(raw, dt, n_expert, n_out, k, device=dev)
    for t in pairs:
        x = orc.pseudo_random(t * k, 0x38, -1.0, 1.0).reshape(t, 1, k)
        ids = (np.arange(t, dtype=np.uint32) * 7 % (n_expert + 1))[:, None]
        got = ops.mul_mv_id(stack, torch.from_numpy(x).to(dev), torch.from_numpy(ids.astype(np.int32)).to(dev)).cpu().numpy()
        want = orc.mul_id(dt, raw, n_expert, n_out, k, x, np.minimum(ids, n_expert - 1), accum64=True)
        want[ids == n_expert] = 0
        assert not got[ids == n_expert].any() and orc.rel_l2(got, want) < 8 * 2.0 ** -24


@pytest.mark.parametrize("dt,name", DTYPES)
def test_plain_mv(orc, dev, dt, name):
    from maxuna_b200 import ops

    n_out, k, t = 100, 768, 3
    raw = orc.quantize(dt, orc.pseudo_random(n_out * k, 7, -1.0, 1.0))
    x = orc.pseudo_random(t * k, 8, -1.0, 1.0).reshape(t, k)
    buf = torch.zeros(raw.size + 128, dtype=torch.uint8, device=dev)
    buf[: raw.size] = torch.from_numpy(raw).to(dev)
    got = ops.mul_mv(buf, dt, n_out, k, torch.from_numpy(x).to(dev)).cpu().numpy()
    assert orc.rel_l2(got, orc.mul_mv(dt, raw, n_out, k, x)) < 1e-3


@pytest.mark.parametrize("n_out,k,t", [(4096, 256, 1), (4104, 512, 3), (4112, 768, 2), (4096 + 16 * 150, 3072, 1)])
def test_plain_mv_q6k_streamed(orc, dev, n_out, k, t):
    """The streamed Q6_K kernel behind `lmoe_mul_mv` (rows in 16-row chunks through shared memory, integer tensor
    cores; one token) and the forms behind it for more tokens: odd and even super-block counts per row (the 210-byte
    blocks change word alignment), more than one chunk per CTA, and an outlier channel.  Same oracle and a tighter
    bound than the reference's 1e-3 (src/ops/mv_id.rs:300-330): the activations carry 21 bits."""
    from maxuna_b200 import ops

    raw = orc.quantize(14, orc.pseudo_random(n_out * k, 70 + k, -1.0, 1.0))
    x = orc.pseudo_random(t * k, 8, -1.0, 1.0).reshape(t, k)
    x[0, 5] = 300.0
    buf = torch.zeros(raw.size + 128, dtype=torch.uint8, device=dev)
    buf[: raw.size] = torch.from_numpy(raw).to(dev)
    got = ops.mul_mv(buf, 14, n_out, k, torch.from_numpy(x).to(dev)).cpu().numpy()
    want = orc.mul_mv(14, raw, n_out, k, x)
    assert np.isfinite(got).all()
    assert orc.rel_l2(got, want) < 1e-5
    assert np.abs(got - want).max() < 1e-5 * np.abs(want).max() * 10


@pytest.mark.parametrize("n_out,k", [(4097, 512), (4104, 256), (4111, 768), (4100, 1280), (4096 + 16 * 150 + 7, 2816)])
def test_plain_mv_q6k_streamed_ragged(orc, dev, n_out, k):
    """The streamed kernel, one token, with a last chunk of fewer than sixteen rows (all remainders of its bytes by 16) and odd
    block counts of several blocks; then blocks near the end of the f32 range, as exact as 21 bits above 2^-126 are."""
    from maxuna_b200 import ops

    raw = orc.quantize(14, orc.pseudo_random(n_out * k, 71 + k, -1.0, 1.0))
    buf = torch.zeros(raw.size + 128, dtype=torch.uint8, device=dev)
    buf[: raw.size] = torch.from_numpy(raw).to(dev)
    x = orc.pseudo_random(k, 9, -1.0, 1.0).reshape(1, k)
    tiny = np.zeros_like(x)
    tiny[0, 5], tiny[0, k - 1] = 1e-33, -3e-33
    for v, tol in ((x, 1e-5), (tiny, 1e-4)):
        got = ops.mul_mv(buf, 14, n_out, k, torch.from_numpy(v).to(dev)).cpu().numpy()
        want = orc.mul_mv(14, raw, n_out, k, v)
        scale = np.float64(1e30) if tol == 1e-4 else 1.0
        assert np.isfinite(got).all() and orc.rel_l2(got * scale, want * scale) < tol


@pytest.mark.parametrize("dt,name", DTYPES)
def test_device_codec_matches_oracle(orc, dev, dt, name):
    from maxuna_b200.gguf import ExpertStack

    rng = np.random.default_rng(5)
    w = (rng.standard_normal((3, 4, 512)) * 0.02).astype(np.float32)
    st = ExpertStack.quantize(torch.from_numpy(w).to(dev), dt)
    raw = st.raw()
    # device decode == oracle decode of the same bytes, bit for bit
    deq_dev = st.dequantize().cpu().numpy().ravel()
    deq_cpu = orc.dequantize(dt, raw)
    np.testing.assert_allclose(deq_dev, deq_cpu, rtol=1e-6, atol=1e-9)
    # and the device encoder produces valid blocks close to the input
    assert orc.rel_l2(deq_cpu, w) < (0.08 if dt == 12 else 0.02)
    # golden blocks (gguf-py decode) through the device decoder
    z = np.load(os.path.join(GOLD, "kquant_decode.npz"))
    key = "q4k" if dt == 12 else "q6k"
    blocks = z[key + "_blocks"]
    g = ExpertStack.from_bytes(blocks.reshape(-1), dt, 1, blocks.shape[0], 256, device=dev)
    np.testing.assert_allclose(g.dequantize().cpu().numpy().reshape(-1, 256), z[key + "_decoded"], rtol=2e-6, atol=1e-9)


def test_routing_known_answers(orc, dev):
    from maxuna_b200 import ops

    for c in json.load(open(os.path.join(GOLD, "routing_kat.json"))):
        logits = torch.tensor([c["logits"]], dtype=torch.float32, device=dev)
        bias = torch.tensor(c["bias"], dtype=torch.float32, device=dev)
        ids, w = ops.route_from_logits(logits, bias, c["top_k"], c["scale"], c["norm"])
        assert ids[0].tolist() == c["ids"], c["name"]
        want = np.array(c["weights"])
        assert np.all(np.abs(w[0].cpu().numpy() - want) <= c["atol"] + c["rtol"] * np.abs(want)), c["name"]
    # router matmul == direct logits with an identity router (src/moe.rs:486-500)
    x = torch.tensor([[2.0, -2.0, 0.0, 1.0, -1.0, 3.0, 0.5, -0.5]], device=dev)
    ids, w = ops.route(torch.eye(8, device=dev), None, x, 3)
    ids2, w2 = ops.route_from_logits(x, None, 3)
    assert torch.equal(ids, ids2) and torch.equal(w, w2)


@pytest.mark.parametrize("t", [1, 2, 3, 16, 33, 257, 2100, 2400])   # the last two: tokens per block sized to whole waves
def test_routing_bit_exact_vs_oracle(orc, dev, t):
    from maxuna_b200 import ops

    rng = np.random.default_rng(100 + t)
    router = (rng.standard_normal((256, 3072)) * 0.02).astype(np.float32)
    bias = rng.uniform(-0.1, 0.1, 256).astype(np.float32)
    x = rng.standard_normal((t, 3072)).astype(np.float32)
    ids, w = ops.route(torch.from_numpy(router).to(dev), torch.from_numpy(bias).to(dev), torch.from_numpy(x).to(dev), 10)
    ids_o, w_o = orc.route(router, bias, x, 10)
    assert np.array_equal(ids.cpu().numpy().astype(np.uint32), ids_o)
    assert np.array_equal(w.cpu().numpy().view(np.uint32), w_o.view(np.uint32))  # weights bit-exact too


@pytest.mark.parametrize("t,hidden,ne", [(301, 512, 20), (81, 2048, 130), (335, 3072, 17), (90, 4096, 70), (23, 3072, 256), (179, 6144, 33)])
def test_routing_tiles_bit_exact(orc, dev, t, hidden, ne):
    """The register-tiled router product at the edges of its token and expert tiles, in both tile shapes: same fixed summation
    order, so ids and weights are bitwise the oracle's."""
    from maxuna_b200 import ops

    rng = np.random.default_rng(hidden)
    router = (rng.standard_normal((ne, hidden)) * 0.02).astype(np.float32)
    x = rng.standard_normal((t, hidden)).astype(np.float32)
    ids, w = ops.route(torch.from_numpy(router).to(dev), None, torch.from_numpy(x).to(dev), 16)
    ids_o, w_o = orc.route(router, None, x, 16)
    assert np.array_equal(ids.cpu().numpy().astype(np.uint32), ids_o)
    assert np.array_equal(w.cpu().numpy().view(np.uint32), w_o.view(np.uint32))


@pytest.mark.parametrize("t,hidden,ne", [(2048, 256, 64), (2051, 384, 61), (2600, 3072, 8), (4099, 512, 7)])
def test_routing_many_tokens_bit_exact(orc, dev, t, hidden, ne):
    """Short router rows in large numbers, and few experts on either side of the tiled form: bitwise the oracle's."""
    from maxuna_b200 import ops

    rng = np.random.default_rng(t)
    router = (rng.standard_normal((ne, hidden)) * 0.02).astype(np.float32)
    x = rng.standard_normal((t, hidden)).astype(np.float32)
    ids, w = ops.route(torch.from_numpy(router).to(dev), None, torch.from_numpy(x).to(dev), 4)
    ids_o, w_o = orc.route(router, None, x, 4)
    assert np.array_equal(ids.cpu().numpy().astype(np.uint32), ids_o)
    assert np.array_equal(w.cpu().numpy().view(np.uint32), w_o.view(np.uint32))


@pytest.mark.parametrize("hidden", [256, 260])
def test_routing_beyond_one_grid(dev, hidden):
    """More tokens than the rows of one grid serve: the same bits as in two calls."""
    from maxuna_b200 import ops

    t, cut = 65535 * 4 + 7, 131072
    router, x = torch.randn(5, hidden, device=dev) * 0.02, torch.randn(t, hidden, device=dev)
    ids, w = ops.route(router, None, x, 2)
    for part in (slice(0, cut), slice(cut, t)):
        i, v = ops.route(router, None, x[part], 2)
        assert torch.equal(ids[part], i) and torch.equal(w[part], v)


@pytest.mark.parametrize("ne,top_k", [(1, 1), (31, 31), (128, 8), (129, 32), (257, 10), (512, 32)])
def test_routing_selection_widths(orc, dev, ne, top_k):
    """Selection at the edges of the scores a lane holds, with ties, infinities and signed zeros: bitwise the oracle's."""
    from maxuna_b200 import ops

    rng = np.random.default_rng(ne)
    logits = rng.integers(-3, 4, (11, ne)).astype(np.float32)
    logits[1] = -logits[1] * 0.0
    logits[2, : ne // 2] = -np.inf
    logits[3, ne // 3] = np.inf
    bias = np.where(rng.random(ne) < 0.3, -0.5, 0.0).astype(np.float32)
    ids, w = ops.route_from_logits(torch.from_numpy(logits).to(dev), torch.from_numpy(bias).to(dev), top_k)
    ids_o, w_o = orc.route_from_logits(logits, bias, top_k)
    assert np.array_equal(ids.cpu().numpy().astype(np.uint32), ids_o)
    assert np.array_equal(w.cpu().numpy().view(np.uint32), w_o.view(np.uint32))


@pytest.mark.parametrize("ne,top_k", [(5, 5), (64, 8), (200, 10), (512, 32)])
def test_routing_ids_are_distinct(orc, dev, ne, top_k):
    """A token's ids are distinct and in range whatever its scores are: all or some NaN, and a bias that leaves fewer finite
    scores than slots (the row lists and sums behind them take distinct ids for granted).  Where no score is NaN, and where
    all are, ids are the oracle's."""
    from maxuna_b200 import ops

    rng = np.random.default_rng(ne)
    logits = rng.standard_normal((9, ne)).astype(np.float32)
    logits[0] = np.nan
    logits[1, 1:] = np.nan
    logits[2, rng.random(ne) < 0.7] = np.nan
    bias = np.zeros(ne, dtype=np.float32)
    bias[top_k // 2:] = -np.inf
    for b in (None, bias):
        ids, _ = ops.route_from_logits(torch.from_numpy(logits).to(dev), None if b is None else torch.from_numpy(b).to(dev), top_k)
        ids = ids.cpu().numpy().astype(np.uint32)
        assert ids.max() < ne and all(len(set(r)) == top_k for r in ids.tolist())
        want, _ = orc.route_from_logits(logits, b, top_k)
        assert np.array_equal(ids[[0, *range(3, 9)]], want[[0, *range(3, 9)]])


def test_routing_odd_hidden_and_ties(orc, dev):
    from maxuna_b200 import ops

    rng = np.random.default_rng(9)
    for hidden, ne in ((200, 16), (7, 8)):
        router = rng.standard_normal((ne, hidden)).astype(np.float32)
        x = rng.standard_normal((5, hidden)).astype(np.float32)
        ids, w = ops.route(torch.from_numpy(router).to(dev), None, torch.from_numpy(x).to(dev), 3)
        ids_o, w_o = orc.route(router, None, x, 3)
        assert np.array_equal(ids.cpu().numpy().astype(np.uint32), ids_o)
    # all-equal scores: lowest indices first, in order
    ids, _ = ops.route_from_logits(torch.zeros(4, 256, device=dev), None, 10)
    assert ids.cpu().numpy().tolist() == [list(range(10))] * 4


@pytest.mark.parametrize("seq", [1, 8, 512])
def test_combine_and_silu_mul(orc, dev, seq):
    from maxuna_b200 import ops

    rng = np.random.default_rng(seq)
    top_k, n_out = 10, 96
    mag = lambda shape: (10.0 ** rng.uniform(-6, 4, shape) * rng.choice([-1.0, 1.0], shape)).astype(np.float32)
    down, w = mag((seq, top_k, n_out)), rng.uniform(0, 1, (seq, top_k)).astype(np.float32)
    l2 = (10.0 ** rng.uniform(-6, 4, (seq, top_k, 1))).astype(np.float32)
    td = lambda a: torch.from_numpy(a).to(dev)
    # fixed summation order => bitwise equal to the oracle's restatement of that order
    assert np.array_equal(ops.combine(td(down), None, td(w)).cpu().numpy().view(np.uint32),
                          orc.combine(down, None, w).view(np.uint32))
    assert np.array_equal(ops.combine(td(down), td(l2), td(w)).cpu().numpy().view(np.uint32),
                          orc.combine(down, l2, w).view(np.uint32))
    g = rng.standard_normal((seq, top_k, 64)).astype(np.float32) * 4
    u = rng.standard_normal((seq, top_k, 64)).astype(np.float32)
    np.testing.assert_allclose(ops.silu_mul(td(g), td(u)).cpu().numpy(), orc.silu_mul(g, u), rtol=2e-6, atol=1e-7)


@pytest.mark.parametrize("n", [1, 3, 1025, (1 << 18) - 1, 1 << 18, (1 << 18) + 3])
def test_silu_mul_counts_and_alignment(orc, dev, n):
    """Counts off a multiple of four and rows off a 16-byte boundary: the same values, and nothing written past the last one."""
    from maxuna_b200._native import check, lib
    from maxuna_b200.gguf import stream_ptr

    rng = np.random.default_rng(n)
    g, u = (rng.standard_normal(n).astype(np.float32) * 3 for _ in range(2))
    want = orc.silu_mul(g, u)
    for off in (0, 1):
        bg, bu = (torch.from_numpy(np.concatenate([np.zeros(off, np.float32), v])).to(dev) for v in (g, u))
        out = torch.full((n + off + 4,), 7.0, device=dev)
        check(lib().lmoe_silu_mul(bg.data_ptr() + 4 * off, bu.data_ptr() + 4 * off, n, out.data_ptr() + 4 * off, stream_ptr()))
        np.testing.assert_allclose(out[off:off + n].cpu().numpy(), want, rtol=2e-6, atol=1e-7)
        assert (out[off + n:] == 7).all() and (out[:off] == 7).all()


@pytest.mark.parametrize("rows,top_k,n", [(3, 1, 97), (5, 6, 33), (2, 22, 132), (1, 64, 4)])
def test_glue_edges(orc, dev, rows, top_k, n):
    """Scalar and four-wide forms of combine and silu_mul, a row count off the block size, and the range guard: a zero row, and
    both outputs within three roundings plus n/2 ulp of the sum of squares."""
    from maxuna_b200 import ops

    rng = np.random.default_rng(n)
    a = rng.standard_normal((rows, top_k, n)).astype(np.float32)
    a[0, 0] = 0
    b, w = rng.standard_normal(a.shape).astype(np.float32), rng.uniform(0, 1, (rows, top_k)).astype(np.float32)
    td = lambda v: torch.from_numpy(v).to(dev)
    assert np.array_equal(ops.combine(td(a), None, td(w)).cpu().numpy(), orc.combine(a, None, w))
    np.testing.assert_allclose(ops.silu_mul(td(a), td(b)).cpu().numpy(), orc.silu_mul(a, b), rtol=2e-6, atol=1e-7)
    got, l2 = (v.cpu().numpy() for v in ops.l2_rescale(td(a)))
    want = np.clip(np.sqrt((a.astype(np.float64) ** 2).sum(2, keepdims=True)), 1e-8, 1e30)
    tol = (3 + n / 2) * 2.0 ** -24
    np.testing.assert_allclose(l2, want, rtol=tol)
    np.testing.assert_allclose(got, a * 32768.0 / want, rtol=tol)


def test_map0_matches_oracle(orc, dev):
    from maxuna_b200 import ops

    for t, top_k, ne, seed in ((40, 4, 6, 0x43), (512, 10, 256, 0x52), (1000, 10, 256, 0x53), (1, 2, 4, 1)):
        ids = orc.distinct_ids(t, top_k, ne, seed)
        s = ops.prepare_map0(ne, torch.from_numpy(ids.astype(np.int32)).to(dev))
        tpe, m = orc.map0(ids, ne)
        assert np.array_equal(s.tpe().cpu().numpy().astype(np.uint32), tpe)
        got = s.ids_map().cpu().numpy()
        for e in range(ne):
            assert np.array_equal(got[e, : tpe[e]], m[e, : tpe[e]])


@pytest.mark.parametrize("t", [1024, 1025, 1028, 4096, 4097, 8196])
def test_map0_chunk_edges(orc, dev, t):
    """Block sizes, chunks and the vector and scalar loads of the token lists, with empty slots: bytes equal the oracle's."""
    from maxuna_b200 import ops

    ids = orc.distinct_ids(t, 3, 9, t)
    ids[t - 1, 2] = 9
    s = ops.prepare_map0(8, torch.from_numpy(ids.astype(np.int32)).to(dev))
    for e in range(8):
        want = np.flatnonzero(ids.reshape(-1) == e)
        assert s.tpe()[e].item() == want.size
        assert np.array_equal(s.ids_map()[e, : want.size].cpu().numpy(), want)


def test_prefill_with_a_nan_token(orc, dev):
    """A token with a NaN in its hidden state goes through the grouped products beside others: its own row is NaN, the other
    rows are what they are without it."""
    blk = _tiny_block(dev)
    x = torch.from_numpy(orc.pseudo_random(96 * 256, 5, -1.0, 1.0).reshape(96, 256)).to(dev)
    want = blk.forward(x, path="prefill")
    x[40, 7] = float("nan")
    got, ids, _ = blk.forward(x, return_routing=True, path="prefill")
    torch.cuda.synchronize()
    blk.check_device_flag()
    assert sorted(set(ids[40].tolist())) == sorted(ids[40].tolist())
    keep = [i for i in range(96) if i != 40]
    assert torch.isnan(got[40]).all() and torch.isfinite(got[keep]).all()
    assert orc.rel_l2(got[keep].cpu().numpy(), want[keep].cpu().numpy()) < 1e-6  # the same products, other row tiles


def _tiny_block(dev, seed=3, hidden=256, ff=256, ne=8, top_k=3, shared=True):
    from maxuna_b200.moe import MoeBlock

    return MoeBlock.random(hidden, ff, ne, top_k, seed=seed, device=dev, shared=shared, weight_std=0.25)


def test_unfused_block_vs_oracle(orc, dev):
    blk = _tiny_block(dev)
    host = blk.host_layer(orc)
    x = np.random.default_rng(4).uniform(-1, 1, (5, blk.hidden)).astype(np.float32)
    want, ids_o, w_o = host.forward(x)
    xd = torch.from_numpy(x).to(dev)
    ids, w = blk.route(xd)
    assert np.array_equal(ids.cpu().numpy().astype(np.uint32), ids_o)
    got = blk.forward_unfused(xd).cpu().numpy()
    assert orc.rel_l2(got, want) < 1e-3


@pytest.mark.parametrize("hidden,ff,sh_ff,ne,top_k,up_dt", [(256, 256, 256, 4, 2, 12), (2048, 768, 768, 16, 4, 12), (3072, 1024, 512, 24, 10, 12),
                                                            (1024, 2048, 2048, 3, 3, 14)])
def test_ffn_mv_equals_the_ops(dev, hidden, ff, sh_ff, ne, top_k, up_dt):
    """One call for the mat-vec chain gives the bits of its ops one by one: products that share a launch and that do not (few
    rows; another type; a shared expert of another width; many pairs of one matrix), an id that names no expert, no shared or
    no routed experts."""
    from maxuna_b200 import ops
    from maxuna_b200.gguf import ExpertStack

    mk = lambda dt, n, o, k, s: ExpertStack.random(dt, n, o, k, seed=s, device=dev)
    e = (mk(12, ne, ff, hidden, 1), mk(up_dt, ne, ff, hidden, 2), mk(14, ne, hidden, ff, 3))
    sh = (mk(12, 1, sh_ff, hidden, 4), mk(12, 1, sh_ff, hidden, 5), mk(14, 1, hidden, sh_ff, 6))
    gen = torch.Generator(device=dev)
    gen.manual_seed(7)
    for t in (1, 2, 3, 9, 64, 130):
        x = torch.randn(t, hidden, generator=gen, device=dev)
        ids = torch.stack([torch.randperm(ne, generator=gen, device=dev)[:top_k] for _ in range(t)]).to(torch.int32)
        ids[t // 2, 0] = ne + 5
        w = torch.rand(t, top_k, generator=gen, device=dev)

        def chain(stacks, idx):
            xg = x.view(t, 1, hidden)
            return ops.mul_mv_id(stacks[2], ops.silu_mul(ops.mul_mv_id(stacks[0], xg, idx), ops.mul_mv_id(stacks[1], xg, idx)), idx)

        routed = ops.combine(chain(e, ids), None, w)
        shared = chain(sh, torch.zeros(t, 1, dtype=torch.int32, device=dev)).view(t, hidden)
        for got, want in ((ops.ffn_mv(e, ids, w, sh, x), routed + shared), (ops.ffn_mv(e, ids, w, None, x), routed),
                          (ops.ffn_mv(None, None, None, sh, x), shared)):
            assert torch.equal(got.view(torch.int32), want.view(torch.int32)), t


def test_ffn_mv_errors(dev):
    from maxuna_b200 import LmoeError, ops
    from maxuna_b200.gguf import ExpertStack

    mk = lambda dt, n, o, k: ExpertStack.random(dt, n, o, k, device=dev)
    e = (mk(12, 4, 256, 512), mk(12, 4, 256, 512), mk(14, 4, 512, 256))
    x, ids, w = torch.zeros(2, 512, device=dev), torch.zeros(2, 2, dtype=torch.int32, device=dev), torch.zeros(2, 2, device=dev)
    for bad in ((e, ids, w, None, torch.zeros(2, 256, device=dev)), (e, ids, w[:1], None, x), (e, ids[:1], w, None, x),
                ((e[0], mk(12, 4, 128, 512), e[2]), ids, w, None, x), ((e[0], e[1], mk(14, 4, 512, 512)), ids, w, None, x),
                (e, ids, w, (e[0], e[1], mk(14, 1, 256, 256)), x), (e, ids, w.double(), None, x)):
        with pytest.raises(LmoeError):
            ops.ffn_mv(*bad)


@pytest.mark.parametrize("t,hidden", [(1023, 2048), (1535, 2048), (1536, 2048), (1024, 3076), (2047, 2052), (2048, 2052), (1100, 2044), (2, 4), (333, 1540)])
@pytest.mark.parametrize("top_k,shared", [(1, False), (3, True), (11, True), (12, False), (12, True), (25, False)])
def test_sum_of_sorted_rows(dev, t, hidden, top_k, shared):
    """The slot sum by token and by columns, on either side of the line between them and of twelve rows: the additions in slot order, empty
    slots left out, the shared row last.  f32 additions in the same order, so the bits."""
    from maxuna_b200._native import check, lib
    from maxuna_b200.gguf import stream_ptr

    gen = torch.Generator(device=dev)
    gen.manual_seed(t + hidden + top_k)
    rows = torch.randn(t * top_k, hidden, generator=gen, device=dev)
    pos = torch.randperm(t * top_k, generator=gen, device=dev).to(torch.int32).view(t, top_k)
    pos[torch.rand(t, top_k, generator=gen, device=dev) < 0.1] = -1
    sh = torch.randn(t, hidden, generator=gen, device=dev) if shared else None
    out = torch.empty(t, hidden, device=dev)
    check(lib().lmoe_ep_combine(rows.data_ptr(), pos.data_ptr(), sh.data_ptr() if shared else None, t, top_k, hidden, out.data_ptr(), stream_ptr()))
    want = torch.zeros(t, hidden, device=dev)
    for k in range(top_k):
        want = torch.where((pos[:, k] >= 0)[:, None], want + rows[pos[:, k].clamp(min=0).long()], want)
    assert torch.equal(out, want + sh if shared else want)
