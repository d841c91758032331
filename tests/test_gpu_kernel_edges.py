"""Kernels whose way of working depends on the size of the input, at the sizes where it changes and around the edges of
their tiles: against the oracle (or numpy's sort), bit for bit."""
import numpy as np
import pytest
import torch

from oracle import port
from tests.test_gpu_tbe import _t, make_case

pytestmark = pytest.mark.gpu

DEV = "cuda"


# bags per group 1 .. G, the last group short; widths that leave rows or output columns off 16 bytes
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("rows,dims,B,max_len", [
    ([50, 30], [128, 20], 19, 9),             # one bag per group
    ([700], [8], 70_001, 2),                  # two-lane groups, whole groups
    ([300, 200], [128, 64], 9_601, 3),        # a few bags per group
    ([90, 60, 40], [8, 18, 64], 4_003, 5),    # rows and columns off 16 bytes
    ([200], [512], 401, 30),                  # several vectors per lane, long bags
    ([400, 90], [64, 64], 12_001, 40),        # long bags, several per group
])
def test_forward_bags_per_group(rows, dims, B, max_len, mode):
    from recsdk_b200 import ops

    c = make_case(np.random.default_rng(B), rows, dims, B, max_len, empty_frac=0.2)
    exp = port.tbe_forward(c["w"], c["wo"], c["do"], c["indices"], c["offsets"], c["T"], B, c["total_D"], c["max_D"], mode)
    out = ops.tbe_forward(_t(c["w"]), _t(c["wo"]), _t(c["do"]), _t(c["indices"]), _t(c["offsets"]), c["total_D"],
                          c["max_D"], mode)
    np.testing.assert_array_equal(out.cpu().numpy(), exp)


def _backward_equals_oracle(indices, rows, dim, B, bits, opt=1, mode=0):
    """One table; `indices` over B bags of equal length."""
    from recsdk_b200 import ops

    rng = np.random.default_rng(indices.size)
    offsets = np.linspace(0, indices.size, B + 1).astype(np.int64)
    grad = rng.standard_normal((B, dim)).astype(np.float32)
    w = rng.uniform(-0.05, 0.05, rows * dim).astype(np.float32)
    m1 = np.full_like(w, 0.1)
    dw, dm1 = _t(w), _t(m1)
    wo, do, hs = np.zeros(1, np.int64), np.array([0, dim], np.int32), np.array([0, rows], np.int64)
    port.tbe_backward(grad, w, m1, None, wo, do, hs, indices, offsets, 1, B, dim, dim, mode, opt, 0.05, 1e-8, 0.9, 0.999, 1,
                      reduce_chunk=64)
    ops.tbe_backward(_t(grad), dw, dm1, None, _t(wo), _t(do), _t(hs), _t(indices), _t(offsets), dim, dim, mode, opt, 0.05,
                     1e-8, 0.9, 0.999, 1, total_hash_size_bits=bits, reduce_chunk=64)
    np.testing.assert_array_equal(dw.cpu().numpy(), w)
    np.testing.assert_array_equal(dm1.cpu().numpy(), m1)


# the one-block plan (up to 8192 positions), the sort of mid-size and the sort of large batches; 32- and 64-bit keys
@pytest.mark.parametrize("bits", [20, 27, 40])
@pytest.mark.parametrize("n", [1, 1023, 1025, 8191, 8192, 8193, (1 << 20) - 1, (1 << 20) + 4097])
def test_backward_plan_sizes(n, bits):
    rng = np.random.default_rng(n)
    _backward_equals_oracle(rng.integers(0, 60_000, n), 60_000, 4, min(n, 5_000), bits)


# runs around the direct / chunked borders (8, 16, 64 by the size of the batch), a chunk, the borders above which the sum of
# a run's chunk sums gets its own kernel (112 chunks, if the longest run has more than 224), and that kernel's ring of 256
# chunk sums taken around more than once
RUNS = [1, 2, 7, 8, 9, 15, 16, 17, 63, 64, 65, 128, 129, 4095, 4096, 4097, 4161, 14_000, 16 * 64, 17 * 64 + 1]
LONG_RUNS = [112 * 64, 112 * 64 + 1, 224 * 64, 224 * 64 + 1, 256 * 64, 256 * 64 + 1, 40_000]


@pytest.mark.parametrize("dim", [4, 8, 16, 32, 36, 64, 128, 18])
def test_backward_run_lengths(dim):
    rng = np.random.default_rng(dim)

    def check(lengths, bags, mode):
        ids = rng.permutation(np.repeat(np.arange(len(lengths)), lengths))
        _backward_equals_oracle(ids, len(lengths), dim, bags, 8, mode=mode)
        return ids.size

    assert check(RUNS[:12], 301, 1) < 8192
    assert 32_768 < check(RUNS, 3_001, 0) < 1 << 17
    assert 65_536 < check(RUNS + LONG_RUNS[:3] + [9_000, 10_000], 3_001, 0) < 1 << 17  # 224 chunks: the kernel stays idle
    assert 1 << 17 < check(RUNS + LONG_RUNS, 3_001, 0) < 3 << 17


# the same kernel on rows narrower than the widest, their widths no multiple of its 32 columns
@pytest.mark.parametrize("opt", [1, 2])
@pytest.mark.parametrize("dims", [[20, 72], [100, 36], [7, 33]])
def test_backward_long_runs_of_mixed_widths(dims, opt):
    from recsdk_b200 import ops

    rng = np.random.default_rng(sum(dims))
    B, per_bag = 2_000, 17
    n, total = 2 * B * per_bag, sum(dims)
    assert n > 65_536  # from there on that kernel is launched
    indices = np.where(rng.random(n) < 0.9, 1, rng.integers(0, 3, n))
    offsets = np.arange(2 * B + 1, dtype=np.int64) * per_bag
    wo, do, hs = np.array([0, 3 * dims[0]], np.int64), np.array([0, dims[0], total], np.int32), np.array([0, 3, 6], np.int64)
    grad = rng.standard_normal((B, total)).astype(np.float32)
    w = rng.uniform(-0.05, 0.05, 3 * total).astype(np.float32)
    m1, m2 = np.full_like(w, 0.1), np.full_like(w, 0.2)
    dw, dm1, dm2 = _t(w), _t(m1), _t(m2)
    port.tbe_backward(grad, w, m1, m2, wo, do, hs, indices, offsets, 2, B, total, max(dims), 0, opt, 0.05, 1e-8, 0.9, 0.999, 1,
                      reduce_chunk=64)
    ops.tbe_backward(_t(grad), dw, dm1, dm2, _t(wo), _t(do), _t(hs), _t(indices), _t(offsets), total, max(dims), 0, opt, 0.05,
                     1e-8, 0.9, 0.999, 1, total_hash_size_bits=8, reduce_chunk=64)
    for got, exp in ((dw, w), (dm1, m1), (dm2, m2)):
        np.testing.assert_array_equal(got.cpu().numpy(), exp)


@pytest.mark.parametrize("world", [1, 3, 64])
@pytest.mark.parametrize("features,batch,max_len,vocab", [(1, 1, 1, 5), (3, 129, 9, 40), (5, 4_097, 6, 100_000)])
def test_bucketize_dedup(features, batch, max_len, vocab, world):
    from recsdk_b200 import ops

    rng = np.random.default_rng(world * batch)
    lengths = rng.integers(0, max_len + 1, features * batch)
    lengths[0] = 1
    ids = rng.integers(0, vocab, int(lengths.sum())) * 0x1E3779B97F4A7C15 & ((1 << 63) - 1)
    for count in (False, True):
        el, ei, ep, ec = port.bucketize(lengths, ids, features, world, True, True, count)
        nl, ni, perm, cnt, k = ops.bucketize(_t(lengths), _t(ids), features, world, True, count)
        k = int(k.item())
        assert k == ei.size
        np.testing.assert_array_equal(nl.cpu().numpy(), el)
        np.testing.assert_array_equal(ni.cpu().numpy()[:k], ei)
        np.testing.assert_array_equal(perm.cpu().numpy(), ep)
        if count:
            np.testing.assert_array_equal(cnt.cpu().numpy()[:k], ec)


# tiles of 2048, rounds of four runs, the size limits of the merge sort (65536 for 21 bits, 98304 for 33, 196608 for 64)
# and where the sort for large inputs begins; the widths on either side of its rule
@pytest.mark.parametrize("bits", [20, 21, 33, 64])
@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 8193, 40_000, 65_536, 65_537, 98_304, 98_305, 131_073, 196_608, 196_609,
                               (1 << 20) - 1, 1 << 20, (1 << 20) + 1])
def test_unique_sizes(n, bits):
    from recsdk_b200 import ops

    rng = np.random.default_rng(n + bits)
    top = (1 << min(bits, 63)) - 1
    ids = np.where(rng.random(n) < 0.5, rng.integers(0, top, n, endpoint=True), rng.integers(0, 50, n))
    ids[-1] = top
    exp, inv = np.unique(ids, return_inverse=True)
    uq, got, cnt = ops.unique_sorted(_t(ids), bits)
    assert int(cnt.item()) == exp.size
    np.testing.assert_array_equal(uq.cpu().numpy()[:exp.size], exp)
    np.testing.assert_array_equal(got.cpu().numpy(), inv)


# ids wider than key_bits: every sort orders them by the same low bits, and the inverse names a place in the buffer
@pytest.mark.parametrize("bits,wide", [(21, 31), (33, 44), (47, 63)])
@pytest.mark.parametrize("n", [2_300, 70_001, (1 << 20) + 1])
def test_unique_ids_wider_than_the_key(n, bits, wide):
    from recsdk_b200 import ops

    rng = np.random.default_rng(n + bits)
    ids = np.where(rng.random(n) < 0.7, rng.integers(0, 1 << wide, n), rng.integers(0, 40, n))
    uq, got, cnt = ops.unique_sorted(_t(ids), bits)
    u, inv = int(cnt.item()), got.cpu().numpy()
    assert inv.min() >= 0 and inv.max() == u - 1 < n
    np.testing.assert_array_equal(uq.cpu().numpy()[:u][inv], ids)


# more tables than a group holds, empty segments, one mapper for two tables: as table after table
@pytest.mark.parametrize("per_table", [[5], [0, 0], [0, 3000, 0, 1, 2049], [700] * 19 + [0, 4097]])
@pytest.mark.parametrize("shared", [False, True])
def test_mappers_together_equal_one_by_one(per_table, shared):
    from recsdk_b200 import IdsMapper

    T, n = len(per_table), sum(per_table)
    rng = np.random.default_rng(n + T)
    offs = np.concatenate([[0], np.cumsum(per_table)]).astype(np.int64)

    def mappers():
        ms = [IdsMapper(8192) for _ in range(T)]
        if shared and T > 1:
            ms[-1] = ms[0]
        return ms

    together, single = mappers(), mappers()
    for _ in range(2):
        ids = _t(rng.integers(0, 3000, n))
        outs = []
        for way in (0, 1):
            hi, uq, uid, inv = (torch.zeros(max(n, 1), dtype=torch.int64, device=DEV) for _ in range(4))
            uo = torch.zeros(T + 1, dtype=torch.int64, device=DEV)
            if way == 0:
                IdsMapper.parallel_ids2indices_unique_out(together, ids, hi, offs, uq, uid, inv, uo)
            else:
                for t in range(T):
                    single[t].ids2indices_unique_out(ids, hi, torch.from_numpy(offs), uq, uid, inv, uo, t)
            outs.append([x.cpu().numpy() for x in (hi, uq, uid, inv, uo)])
        for a, b in zip(*outs):
            np.testing.assert_array_equal(a, b)
    assert [m.size() for m in together] == [m.size() for m in single]


# segments on either side of the number of scan tiles (1024 of 2048 ids) up to which the offsets are added up tile by tile
@pytest.mark.parametrize("long", [1024 * 2048, 1024 * 2048 + 1, 5_000_000])
def test_mapper_segments_of_many_tiles(long):
    from recsdk_b200 import IdsMapper

    per_table = [3_000, long, 0, 2_049]
    offs = np.concatenate([[0], np.cumsum(per_table)]).astype(np.int64)
    n, T = int(offs[-1]), len(per_table)
    ids = np.random.default_rng(long).integers(0, long // 3, n)
    hi, uq, uid, inv = (torch.zeros(n, dtype=torch.int64, device=DEV) for _ in range(4))
    uo = torch.zeros(T + 1, dtype=torch.int64, device=DEV)
    IdsMapper.parallel_ids2indices_unique_out([IdsMapper(max(k, 16)) for k in per_table], _t(ids), hi, offs, uq, uid, inv, uo)
    hi, uid, inv, uo = (x.cpu().numpy() for x in (hi, uid, inv, uo))
    for t in range(T):
        seg = ids[offs[t]:offs[t + 1]]
        keys, first, which = np.unique(seg, return_index=True, return_inverse=True)
        come = np.argsort(first)  # keys get slots, and stand in the unique list, in the order they come
        slot = np.empty(keys.size, np.int64)
        slot[come] = np.arange(keys.size)
        assert uo[t + 1] - uo[t] == keys.size
        np.testing.assert_array_equal(uid[uo[t]:uo[t + 1]], keys[come])
        np.testing.assert_array_equal(hi[offs[t]:offs[t + 1]], slot[which])
        np.testing.assert_array_equal(inv[offs[t]:offs[t + 1]], slot[which])


def test_mappers_together_report_the_table_that_failed():
    from recsdk_b200 import IdsMapper

    ms = [IdsMapper(64) for _ in range(3)]
    ids = _t(np.array([1, 2, 3, -5, 4, 5], np.int64))
    hi, uq, uid, inv = (torch.zeros(6, dtype=torch.int64, device=DEV) for _ in range(4))
    with pytest.raises(RuntimeError, match="-5"):
        IdsMapper.parallel_ids2indices_unique_out(ms, ids, hi, [0, 2, 4, 6], uq, uid, inv,
                                                  torch.zeros(4, dtype=torch.int64, device=DEV))


# one mapper for several segments, each longer than the one before, so that its workspace grows while the call collects
# the tables; the workspaces of the earlier segments have to outlive their kernels
def test_registered_mapper_whose_workspace_grows_within_a_call():
    from recsdk_b200 import IdsMapper, torch_ops

    if not torch_ops.available():
        pytest.skip("torch op library not built")
    torch_ops.load()
    per_table = [30, 700, 3_000, 9_000, 9_000, 40_000]
    T, n = len(per_table), sum(per_table)
    offs = torch.from_numpy(np.concatenate([[0], np.cumsum(per_table)]).astype(np.int64))
    ids = _t(np.random.default_rng(5).integers(0, 30_000, n))
    registered, other = torch.classes.recsdk.IdsMapper(65_536, True), torch.classes.recsdk.IdsMapper(65_536, True)
    single, single_other = IdsMapper(65_536), IdsMapper(65_536)
    outs = []
    for way in (0, 1):
        hi, uq, uid, inv = (torch.zeros(n, dtype=torch.int64, device=DEV) for _ in range(4))
        uo = torch.zeros(T + 1, dtype=torch.int64, device=DEV)
        if way == 0:
            ms = [registered] * T
            ms[4] = other
            torch.classes.recsdk.IdsMapper.parallel_ids2indices_unique_out(ms, ids, hi, offs, uq, uid, inv, uo)
        else:
            for t in range(T):
                (single_other if t == 4 else single).ids2indices_unique_out(ids, hi, offs, uq, uid, inv, uo, t)
        outs.append([x.cpu().numpy() for x in (hi, uq, uid, inv, uo)])
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
    assert registered.size() == single.size() and other.size() == single_other.size()


@pytest.mark.parametrize("D", [1, 6, 64, 132])
@pytest.mark.parametrize("B,L", [(1, 1), (37, 7), (1_500, 33)])
def test_jagged_dense_row_groups(B, L, D):
    from recsdk_b200 import ops

    rng = np.random.default_rng(B + D)
    lengths = rng.integers(0, L + 3, B)
    lengths[0] = max(1, lengths[0])
    offs = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    values = rng.standard_normal((int(offs[-1]), D)).astype(np.float32)
    dense = ops.jagged_to_padded_dense(_t(values), [_t(offs)], L, 0.5)
    exp = port.jagged_to_padded_dense(values, offs, L, 0.5)
    np.testing.assert_array_equal(dense.cpu().numpy(), exp)
    back, _ = ops.dense_to_jagged(dense, [_t(offs)], int(offs[-1]))
    np.testing.assert_array_equal(back.cpu().numpy()[:int(offs[-1])], port.dense_to_jagged(exp, offs))
