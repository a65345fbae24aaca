"""GPU parity: quantised-inference TBE forward through the C ABI vs the CPU oracle."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from tests import helpers
from tests.test_tbe_forward_gpu import non_finite_weights
from torchlib_xpu_b200 import cabi, workloads

pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-3, 1e-3   # int8 / int4 pooling, fp16 output


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _run(W, wo, tys, Do, rows, B, indices, offsets, psw, pooling, out_dtype, row_alignment,
         tell_types=True):
    """tell_types: pass the set of table types along (the call may then skip the kernel of the types
    that are absent); the result must not depend on it."""
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = cabi.nbit_forward(_dev(W), _dev(wo), _dev(tys), _dev(Do), int(Do[-1]),
                            int(np.max(np.diff(Do))), _dev(indices), _dev(offsets), B, pooling,
                            None if psw is None else _dev(psw), out_dtype, row_alignment,
                            _dev(np.asarray(rows, dtype=np.int64)), status,
                            table_types=set(int(t) for t in tys) if tell_types else None)
    torch.cuda.synchronize()
    return out, int(status.item())


@pytest.mark.parametrize("row_alignment", [16, 1])
@pytest.mark.parametrize("out_dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("pooling", [oracle.SUM, oracle.MEAN])
@pytest.mark.parametrize("weighted", [False, True])
def test_nbit_mixed_tables(row_alignment, out_dtype, pooling, weighted):
    rng = workloads.rng_for(300)
    tys = [oracle.INT8, oracle.INT4, oracle.INT8, oracle.INT4, oracle.INT2, oracle.FP16,
           oracle.FP32, oracle.INT8, oracle.INT4, oracle.INT4]
    Ds = [128, 128, 64, 256, 64, 128, 32, 20, 36, 1024]
    rows = [90, 80, 70, 60, 50, 40, 30, 20, 25, 12]
    T, B = len(tys), 41
    W, wo, Do, tys_a = helpers.quantised_tables(rng, rows, Ds, tys, row_alignment)
    _, offsets, indices = helpers.ragged_bags(rng, T, B, rows, 0, 50, empty_fraction=0.1)
    psw = rng.random(indices.size).astype(np.float32) if weighted else None
    want = oracle.nbit_forward(W, wo, tys_a, Do, row_alignment, B, indices, offsets, psw, pooling)
    got, status = _run(W, wo, tys_a, Do, rows, B, indices, offsets, psw, pooling, out_dtype,
                       row_alignment)
    assert status == 0
    np.testing.assert_allclose(got.float().cpu().numpy(), want, rtol=RTOL, atol=ATOL)


def test_nbit_single_row_bags_are_plain_dequantisation():
    """One row per bag, fp32 out: q*scale + bias per element, to fp32 rounding."""
    rng = workloads.rng_for(301)
    for ty, D in ((oracle.INT8, 128), (oracle.INT4, 128), (oracle.INT4, 64), (oracle.INT8, 256)):
        rows = 64
        W, wo, Do, tys_a = helpers.quantised_tables(rng, [rows], [D], [ty], 16)
        indices, offsets = rng.permutation(rows).astype(np.int64), np.arange(rows + 1, dtype=np.int64)
        want = oracle.nbit_forward(W, wo, tys_a, Do, 16, rows, indices, offsets)
        got, status = _run(W, wo, tys_a, Do, [rows], rows, indices, offsets, None, oracle.SUM,
                           torch.float32, 16)
        assert status == 0
        np.testing.assert_allclose(got.cpu().numpy(), want, rtol=1e-6, atol=1e-6)


def test_nbit_flags_out_of_range_indices():
    rng = workloads.rng_for(302)
    W, wo, Do, tys_a = helpers.quantised_tables(rng, [30], [128], [oracle.INT4], 16)
    _, offsets, indices = helpers.ragged_bags(rng, 1, 6, [30], 2, 5)
    bad = indices.copy()
    bad[1] = 30
    got, status = _run(W, wo, tys_a, Do, [30], 6, bad, offsets, None, oracle.SUM, torch.float32, 16)
    assert status & cabi.DEV_INDEX_OUT_OF_RANGE
    keep = np.ones(indices.size, dtype=np.float32)
    keep[1] = 0
    want = oracle.nbit_forward(W, wo, tys_a, Do, 16, 6, np.where(keep > 0, indices, 0), offsets, keep)
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=1e-5, atol=1e-5)


def test_nbit_named_config_scaled_down_against_oracle():
    """The quantised configuration's shape (half INT8, half INT4, D=128, L~U{1..100}, Zipf 1.1,
    fp16 out) with fewer tables and rows, against the oracle."""
    T, E, D, B = 8, 50_000, 128, 1024
    inp = workloads.tbe_inputs(T, B, E, D, 1, 100, 3, "zipf", 1.1)
    rng = workloads.rng_for(3000)
    tys = [oracle.INT8 if t < T // 2 else oracle.INT4 for t in range(T)]
    W, wo, Do, tys_a = helpers.quantised_tables(rng, [E] * T, [D] * T, tys, 16)
    want = oracle.nbit_forward(W, wo, tys_a, Do, 16, B, inp.indices, inp.offsets)
    got, status = _run(W, wo, tys_a, Do, [E] * T, B, inp.indices, inp.offsets, None, oracle.SUM,
                       torch.float16, 16)
    assert status == 0
    np.testing.assert_allclose(got.float().cpu().numpy(), want, rtol=RTOL, atol=ATOL)
    blind, status = _run(W, wo, tys_a, Do, [E] * T, B, inp.indices, inp.offsets, None, oracle.SUM,
                         torch.float16, 16, tell_types=False)
    assert status == 0 and torch.equal(blind, got)


@pytest.mark.parametrize("ty,D", [(oracle.INT8, 128), (oracle.INT8, 4), (oracle.INT8, 68), (oracle.INT4, 128),
                                  (oracle.INT4, 8), (oracle.INT4, 72)])
@pytest.mark.parametrize("weighted", [False, True])
def test_nbit_register_gather_shapes(ty, D, weighted):
    """INT8 / INT4 rows of 4 ... 128 elements (the register-gather kernel, one or two code words per
    lane, some lanes idle), bags of 0 ... 70 rows with ids out of range mixed in, MEAN pooling."""
    rng = workloads.rng_for(310 + D)
    rows, B = [500, 37], 97
    W, wo, Do, tys_a = helpers.quantised_tables(rng, rows, [D, D], [ty, ty], 16)
    _, offsets, indices = helpers.ragged_bags(rng, 2, B, rows, 0, 70, empty_fraction=0.1)
    psw = rng.random(indices.size).astype(np.float32) if weighted else None
    want = oracle.nbit_forward(W, wo, tys_a, Do, 16, B, indices, offsets, psw, oracle.MEAN)
    got, status = _run(W, wo, tys_a, Do, rows, B, indices, offsets, psw, oracle.MEAN, torch.float32, 16)
    assert status == 0
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("weighted,pooling,idx_dtype,B", [
    (False, oracle.SUM, np.int64, 16001),      # groups of 3 bags, the last group short
    (True, oracle.MEAN, np.int32, 40000),      # groups of 8 (the most a warp takes)
    (False, oracle.MEAN, np.int32, 25013),
])
def test_nbit_groups_of_bags(weighted, pooling, idx_dtype, B):
    """A grid of more than about 47 k bags gives every warp a GROUP of consecutive bags to pool as one
    stream of lookups. INT8 and INT4 rows of 128, 64 and 20 / 40 elements (and a table of a type the
    register kernel leaves to the ring engine), bags of 0 to 40 lookups, runs of empty bags -- the tail
    of a table and whole groups included -- and ids out of range."""
    rng = workloads.rng_for(320 + B)
    tys = [oracle.INT8, oracle.INT4, oracle.INT8, oracle.INT4, oracle.INT2, oracle.INT8]
    Ds = [128, 128, 64, 40, 64, 20]
    rows = [3000, 2000, 1000, 500, 300, 600]
    T = len(Ds)
    W, wo, Do, tys_a = helpers.quantised_tables(rng, rows, Ds, tys, 16)
    lengths, _, _ = helpers.ragged_bags(rng, T, B, rows, 0, 40, empty_fraction=0.33)
    lengths[B - 40:B] = 0
    lengths[2 * B:2 * B + 64] = 0
    lengths[-5:] = 0
    offsets = np.zeros(T * B + 1, dtype=np.int64)
    np.cumsum(lengths, out=offsets[1:])
    indices = np.zeros(int(offsets[-1]), dtype=np.int64)
    for t in range(T):
        a, b = int(offsets[t * B]), int(offsets[(t + 1) * B])
        indices[a:b] = rng.integers(0, rows[t], size=b - a, dtype=np.int64)
    bad_at = rng.choice(indices.size, size=200, replace=False)
    bad = indices.copy()
    bad[bad_at[:100]] = 5000               # past every table
    bad[bad_at[100:]] = -1
    psw = rng.random(indices.size).astype(np.float32) if weighted else None
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = cabi.nbit_forward(_dev(W), _dev(wo), _dev(tys_a), _dev(Do), int(Do[-1]), int(np.max(np.diff(Do))),
                            _dev(bad.astype(idx_dtype)), _dev(offsets.astype(idx_dtype)), B, pooling,
                            None if psw is None else _dev(psw), torch.float32, 16,
                            _dev(np.asarray(rows, dtype=np.int64)), status)
    torch.cuda.synchronize()
    assert int(status.item()) & cabi.DEV_INDEX_OUT_OF_RANGE
    # flagged lookups contribute nothing (MEAN still divides by the bag's length)
    keep = np.ones(indices.size, dtype=np.float32)
    keep[bad_at] = 0.0
    want = oracle.nbit_forward(W, wo, tys_a, Do, 16, B, np.where(keep > 0, indices, 0), offsets,
                               keep if psw is None else psw * keep, pooling)
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=RTOL, atol=ATOL)


@pytest.mark.parametrize("D", [16, 32, 48, 64, 96, 112, 128, 144, 256, 272, 512])
@pytest.mark.parametrize("weighted,pooling,out_dtype,align,B", [
    (False, oracle.SUM, torch.float32, 16, 29),      # vectors, one bag per warp
    (True, oracle.MEAN, torch.float16, 16, 12011),   # vectors, groups of two bags, the last group short
    (False, oracle.MEAN, torch.float32, 8, 29),      # INT4 by vectors, INT8 by words (or the ring engine)
    (True, oracle.SUM, torch.float32, 4, 29),        # words (or the ring engine)
])
def test_nbit_rows_in_vectors_of_sixteen_codes(D, weighted, pooling, out_dtype, align, B):
    """Rows of 1 to 32 vectors (groups of 2 to 32 lanes, full and with idle lanes), next to rows that are not
    whole vectors; empty bags (the last ones too), ids out of range, one with an infinite weight."""
    rng = workloads.rng_for(330 + D)
    tys, Ds, rows = [oracle.INT8, oracle.INT4, oracle.INT8, oracle.INT4], [D, D, 20, 24], [90, 210, 30, 40]
    T = len(tys)
    W, wo, Do, tys_a = helpers.quantised_tables(rng, rows, Ds, tys, align)
    lengths, _, _ = helpers.ragged_bags(rng, T, B, rows, 0, 9 if B > 100 else 80, empty_fraction=0.2)
    lengths[B - 3:B] = 0
    lengths[-2:] = 0
    offsets = np.zeros(T * B + 1, dtype=np.int64)
    np.cumsum(lengths, out=offsets[1:])
    indices = np.concatenate([rng.integers(0, rows[t], size=int(offsets[(t + 1) * B] - offsets[t * B]))
                              for t in range(T)]).astype(np.int64)
    bad_at = rng.choice(int(offsets[2 * B]), size=20, replace=False)
    bad, keep = indices.copy(), np.ones(indices.size, dtype=np.float32)
    bad[bad_at[:10]], bad[bad_at[10:]], keep[bad_at] = 210, -1, 0.0
    psw = rng.random(indices.size).astype(np.float32) if weighted else None
    given = None if psw is None else psw.copy()
    if weighted and align == 16:
        given[bad_at[0]] = np.inf
    got, status = _run(W, wo, tys_a, Do, rows, B, bad, offsets, given, pooling, out_dtype, align, tell_types=B > 100)
    assert status & cabi.DEV_INDEX_OUT_OF_RANGE
    want = oracle.nbit_forward(W, wo, tys_a, Do, align, B, np.where(keep > 0, indices, 0), offsets,
                               keep if psw is None else psw * keep, pooling)
    got = got.float().cpu().numpy()
    assert np.isfinite(got).all()
    if out_dtype == torch.float16:
        np.testing.assert_allclose(got, want, rtol=RTOL, atol=ATOL)
    else:   # sums of at most 80 dequantised terms of magnitude about 1, in another order
        np.testing.assert_allclose(got, want, rtol=1e-5, atol=2e-5)


@pytest.mark.parametrize("D,align", [(128, 4), (64, 4), (24, 16), (128, 16), (32, 16), (256, 16)])
@pytest.mark.parametrize("B", [40, 12000])   # one bag per warp, groups of bags
def test_nbit_weights_that_are_not_finite_stay_in_their_bags(D, align, B):
    """A lookup that is skipped adds nothing whatever its weight, and the weight of a good lookup reaches its own bag
    only: rows fetched as words and as vectors."""
    rng = workloads.rng_for(360 + D)
    tys, rows = [oracle.INT8, oracle.INT4, oracle.INT8], [300, 70, 500]
    T = len(tys)
    W, wo, Do, tys_a = helpers.quantised_tables(rng, rows, [D] * T, tys, align)
    _, offsets, indices = helpers.ragged_bags(rng, T, B, rows, 0, 70 if B < 100 else 9, empty_fraction=0.1)
    bad, psw, kept, touched = non_finite_weights(rng, offsets, indices, rows, T, B)
    got, status = _run(W, wo, tys_a, Do, rows, B, bad, offsets, psw, oracle.SUM, torch.float32, align)
    assert status & cabi.DEV_INDEX_OUT_OF_RANGE
    want = oracle.nbit_forward(W, wo, tys_a, Do, align, B, indices, offsets, np.where(np.isfinite(kept), kept, 0), oracle.SUM)
    got = got.cpu().numpy()
    for t in range(T):
        clean = ~touched[t * B:(t + 1) * B]
        # sums of at most 70 dequantised terms of magnitude <= 1.5, in another order
        np.testing.assert_allclose(got[clean, t * D:(t + 1) * D], want[clean, t * D:(t + 1) * D], rtol=1e-5, atol=3e-5)


@pytest.mark.parametrize("T", [2, 31, 33, 64, 129, 1023, 1024, 1025, 2100])
@pytest.mark.parametrize("types", ["alternating", "one_int8", "one_int4", "random"])
def test_nbit_tables_of_both_types_at_every_count(T, types):
    """Grids of more than one wave take INT8 tables before the others: every table is pooled once, wherever its type
    puts it."""
    rng = workloads.rng_for(370 + T)
    ty = {"alternating": np.arange(T) % 2, "one_int8": (np.arange(T) != T - 1).astype(int),
          "one_int4": (np.arange(T) == T // 2).astype(int), "random": rng.integers(0, 2, size=T)}[types]
    tys = [oracle.INT4 if x else oracle.INT8 for x in ty]
    rows, D = 7, 16
    B = 10_000 // T + 3       # one bag per CTA, more CTAs than run at a time
    W, wo, Do, tys_a = helpers.quantised_tables(rng, [rows] * T, [D] * T, tys, 16)
    _, offsets, indices = helpers.ragged_bags(rng, T, B, [rows] * T, 0, 3)
    want = oracle.nbit_forward(W, wo, tys_a, Do, 16, B, indices, offsets)
    for tell in (True, False):
        got, status = _run(W, wo, tys_a, Do, [rows] * T, B, indices, offsets, None, oracle.SUM, torch.float32, 16, tell)
        assert status == 0
        np.testing.assert_allclose(got.cpu().numpy(), want, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("Ds,align", [((128, 64, 32), 16), ((512, 256, 16), 16), ((128, 40, 64), 4)])
@pytest.mark.parametrize("B,rpd", [(40, 14), (16_003, 5_335)])      # one bag per warp, groups of bags
@pytest.mark.parametrize("out_dtype,col0,extra", [(torch.float16, 8, 8), (torch.float16, 3, 2), (torch.float32, 1, 2)])
def test_nbit_across_destinations(Ds, align, B, rpd, out_dtype, col0, extra):
    """num_dests > 1, rows fetched as vectors and as words: a destination's last row falls inside a group of bags;
    aligned and unaligned output rows."""
    rng = workloads.rng_for(380 + sum(Ds))
    tys, rows, T, G = [oracle.INT8, oracle.INT4, oracle.INT4], [60, 300, 20], 3, 3
    if Ds[1] == 40:
        tys = [oracle.INT8, oracle.INT4, oracle.INT8]
    W, wo, Do, tys_a = helpers.quantised_tables(rng, rows, Ds, tys, align)
    _, offsets, indices = helpers.ragged_bags(rng, T, B, rows, 0, 5, empty_fraction=0.2)
    want = oracle.nbit_forward(W, wo, tys_a, Do, align, B, indices, offsets)
    total_D = int(Do[-1])
    stride = col0 + total_D + extra
    bufs = [torch.full((rpd, stride), -7.0, dtype=out_dtype, device="cuda") for _ in range(G)]
    held = [_dev(a) for a in (W, wo, tys_a, Do, indices, offsets)]
    p = cabi.NbitForwardParams()
    p.dev_weights, p.weights_offsets, p.weights_tys, p.D_offsets, p.indices, p.offsets = (a.data_ptr() for a in held)
    for g in range(G):
        p.outputs[g] = bufs[g].data_ptr()
    p.output_stride, p.output_col_offset, p.rows_per_dest, p.num_dests = stride, col0, rpd, G
    p.T, p.B, p.max_D, p.row_alignment, p.index_bytes = T, B, max(Ds), align, 8
    p.output_dtype, p.pooling_mode = cabi.FP16 if out_dtype == torch.float16 else cabi.FP32, oracle.SUM
    assert cabi.lib().b200tbe_nbit_forward(ctypes.byref(p), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    for g, buf in enumerate(bufs):
        blk = buf.float().cpu().numpy()
        n = min(rpd, B - g * rpd)
        np.testing.assert_allclose(blk[:n, col0:col0 + total_D], want[g * rpd:g * rpd + n], rtol=RTOL, atol=ATOL)
        assert np.all(blk[:, :col0] == -7.0) and np.all(blk[:, col0 + total_D:] == -7.0) and np.all(blk[n:] == -7.0)
