"""GPU parity of the module facades (the callers one step above the operator boundary)."""
import numpy as np
import pytest
import torch

import oracle
from tests import helpers
from torchlib_xpu_b200 import workloads
from torchlib_xpu_b200.tbe_modules import (IntNBitTableBatchedEmbeddingBagsCodegen, OptimType, PoolingMode,
                                           SparseType, SplitTableBatchedEmbeddingBagsCodegen)

pytestmark = pytest.mark.gpu


def test_training_module_steps_match_the_oracle():
    rng = workloads.rng_for(700)
    specs, B = [(500, 128), (300, 64), (80, 32)], 64
    mod = SplitTableBatchedEmbeddingBagsCodegen(specs, OptimType.EXACT_ROWWISE_ADAGRAD, 0.05, 1e-8,
                                                PoolingMode.MEAN, SparseType.FP16)
    W = mod.weights_dev.detach().cpu().numpy().copy()
    mom = np.zeros(sum(r for r, _ in specs), dtype=np.float32)
    wo = mod.weights_offsets.cpu().numpy()
    Do = mod.D_offsets.cpu().numpy()
    hs = mod.hash_size_cumsum.cpu().numpy()
    for step in range(2):
        _, offsets, indices = helpers.ragged_bags(rng, len(specs), B, [r for r, _ in specs], 0, 12, 0.1)
        grad = rng.standard_normal((B, int(Do[-1]))).astype(np.float32)
        out = mod(torch.from_numpy(indices).cuda(), torch.from_numpy(offsets).cuda())
        want = oracle.tbe_forward(W, oracle.FP16, wo, Do, B, indices, offsets, None, oracle.MEAN)
        np.testing.assert_allclose(out.detach().cpu().numpy(), want, rtol=1e-3, atol=1e-3)
        out.backward(torch.from_numpy(grad).cuda())
        oracle.tbe_backward(W, oracle.FP16, wo, Do, hs, B, indices, offsets, grad, mom, hs[:-1],
                            oracle.ROWWISE_ADAGRAD, 0.05, 1e-8, None, oracle.MEAN)
        torch.cuda.synchronize()
        np.testing.assert_allclose(mod.weights_dev.detach().float().cpu().numpy(), W.astype(np.float32),
                                   rtol=1e-3, atol=1e-3)
        np.testing.assert_allclose(mod.momentum1_dev.cpu().numpy(), mom, rtol=1e-4, atol=1e-6)
        W = mod.weights_dev.detach().cpu().numpy().copy()   # keep the two in lock step
        mom = mod.momentum1_dev.cpu().numpy().copy()
    views = mod.split_embedding_weights()
    assert [tuple(v.shape) for v in views] == specs


def test_inference_module_quantises_and_pools():
    rng = workloads.rng_for(701)
    specs = [(200, 128, SparseType.INT8), (150, 128, SparseType.INT4), (60, 64, SparseType.FP16),
             (40, 32, SparseType.INT2)]
    mod = IntNBitTableBatchedEmbeddingBagsCodegen(specs)
    tables = [rng.uniform(-1, 1, size=(r, d)).astype(np.float32) for r, d, _ in specs]
    for t, tab in enumerate(tables):
        mod.assign_table(t, torch.from_numpy(tab))
    B = 48
    _, offsets, indices = helpers.ragged_bags(rng, len(specs), B, [r for r, _, _ in specs], 0, 25, 0.1)
    out = mod(torch.from_numpy(indices).cuda(), torch.from_numpy(offsets).cuda())
    assert out.dtype == torch.float16 and out.shape == (B, 128 + 128 + 64 + 32)
    W = mod.weights_dev.cpu().numpy()
    want = oracle.nbit_forward(W, mod.weights_offsets.cpu().numpy(), mod.weights_tys.cpu().numpy(),
                               mod.D_offsets.cpu().numpy(), 16, B, indices, offsets)
    np.testing.assert_allclose(out.float().cpu().numpy(), want, rtol=1e-3, atol=1e-3)
    # and the quantised tables are what the oracle's quantiser makes of the same floats
    for t, (r, d, ty) in enumerate(specs):
        if ty in (SparseType.INT8, SparseType.INT4, SparseType.INT2):
            start, stride = int(mod.weights_offsets[t]), mod.row_strides[t]
            got = W[start:start + r * stride].reshape(r, stride)
            assert np.array_equal(got, oracle.quantize_rows(tables[t], int(ty), 16))


def _table_at(place, values):
    """A new int64 index table in the memory that a freed one had."""
    others = []
    while len(others) < 8192:
        others.append(torch.tensor(values, device="cuda"))
        if others[-1].data_ptr() == place:
            return others[-1]
    raise AssertionError("the allocator did not hand out the freed table's memory")


def test_row_counts_of_one_table_are_never_those_of_an_earlier_one():
    """Row counts are remembered between calls. An index table built after another one was freed lies where that
    one lay, with as many entries: its own counts apply, in the range check of the forward and in the key bits of
    the backward's sort."""
    lookup = torch.ops.fbgemm.split_embedding_codegen_lookup_sgd_function
    large, D = 70000, 16
    ids = torch.tensor([0, large - 1, 2, large - 1], device="cuda")
    offsets = torch.arange(ids.numel() + 1, device="cuda")
    wo, Do = torch.zeros(1, dtype=torch.int64, device="cuda"), torch.tensor([0, D], dtype=torch.int32, device="cuda")
    e, ei = torch.empty(0, device="cuda"), torch.empty(0, dtype=torch.int32, device="cuda")
    torch.ops.fbgemm.b200tbe_pop_device_status(e)

    def step(rows, table):
        w = torch.ones(large * D, device="cuda")
        placeholder = torch.zeros(1, device="cuda", requires_grad=True)
        out = lookup(placeholder, w, e, e, ei, wo, Do, D, D, table, 17, ids.clamp(max=rows - 1), offsets, 0, None, None, ei,
                     False, 0.0, False, 0.5, 0)
        out.backward(torch.ones_like(out))
        return out.detach()[:, 0].tolist(), w[::D]

    first = torch.tensor([0, 3], device="cuda")
    place = first.data_ptr()
    assert step(3, first)[0] == [1.0] * 4
    del first
    out, w = step(large, _table_at(place, [0, large]))
    assert out == [1.0] * 4
    want = torch.ones(large)
    want[0], want[2], want[large - 1] = 0.5, 0.5, 0.0
    assert torch.equal(w.cpu(), want)
    assert torch.ops.fbgemm.b200tbe_pop_device_status(e) == 0


def test_row_counts_follow_a_write_to_the_index_table():
    mod = SplitTableBatchedEmbeddingBagsCodegen([(64, 16)], OptimType.EXACT_SGD, 0.5)
    mod.weights_dev.data.fill_(1.0)
    ids, offsets = torch.tensor([0, 40], device="cuda"), torch.arange(3, device="cuda")
    with torch.no_grad():
        for rows in (64, 40, 41):
            mod.hash_size_cumsum.copy_(torch.tensor([0, rows], device="cuda"))
            assert mod(ids, offsets)[:, 0].tolist() == [1.0, 1.0 if rows > 40 else 0.0]
    torch.ops.fbgemm.b200tbe_pop_device_status(ids)


def test_quantised_row_counts_belong_to_all_that_they_depend_on():
    """Two modules' tables behind one and the same weights_offsets tensor: the row counts come from the buffer's
    size, the rows' type and width and their alignment too."""
    rng = workloads.rng_for(702)
    specs = [(4, 32, SparseType.INT8), (300, 32, SparseType.INT8), (300, 32, SparseType.INT4), (300, 64, SparseType.INT8)]
    offsets = torch.arange(2, device="cuda")
    shared = None
    torch.ops.fbgemm.b200tbe_pop_device_status(offsets)
    for rows, dim, ty in specs:
        mod = IntNBitTableBatchedEmbeddingBagsCodegen([(rows, dim, ty)], output_dtype=SparseType.FP32)
        tab = rng.uniform(-1, 1, size=(rows, dim)).astype(np.float32)
        mod.assign_table(0, torch.from_numpy(tab))
        shared = mod.weights_offsets if shared is None else shared
        mod.weights_offsets = shared
        out = mod(torch.tensor([rows - 1], device="cuda"), offsets)
        want = oracle.nbit_forward(mod.weights_dev.cpu().numpy(), np.zeros(1, np.int64), np.array([int(ty)], np.uint8),
                                   np.array([0, dim], np.int32), 16, 1, np.array([rows - 1]), np.array([0, 1]))
        np.testing.assert_allclose(out.cpu().numpy(), want, rtol=1e-6, atol=1e-6)
    assert torch.ops.fbgemm.b200tbe_pop_device_status(offsets) == 0
