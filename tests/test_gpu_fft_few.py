"""Transforms of few columns, whose tiles all run at once: 2^11..2^13 points in tiles of 2^12
and 2^13 elements, 2^14 and longer with more threads a tile. One column, column counts that
leave a tile half empty, and counts on both sides of the lines (a device of 148 SMs: 296
tiles, 148 tiles), against the oracle. Every value is exact."""
import numpy as np
import pytest

from helpers import m31, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_size,ncols,blowup", [
    (11, 1, 1), (11, 3, 3), (11, 592, 1), (11, 593, 1),
    (12, 1, 2), (12, 5, 1), (12, 148, 1), (12, 296, 1), (12, 297, 1),
    (13, 1, 1), (13, 7, 2), (13, 149, 1), (13, 296, 1),
    (14, 1, 1), (14, 74, 1), (14, 149, 1), (15, 2, 1), (16, 37, 1), (17, 19, 1),
])
def test_few_columns_match_oracle(stwo, oracle, log_size, ncols, blowup):
    L = stwo._lib
    lib = L.lib()
    B = stwo.CudaBackend
    r = rng(5200 + log_size * 1000 + ncols)
    n = 1 << log_size
    tree = B.precompute_twiddles(stwo.CanonicCoset(log_size + blowup).half_coset())
    tw, itw = tree.twiddles.to_numpy(), tree.itwiddles.to_numpy()
    vals = m31(r, ncols * n).reshape(ncols, n)
    bufs = [stwo.BaseFieldVec.from_numpy(v) for v in vals]
    outs = [stwo.BaseFieldVec.new_uninitialized(n << blowup) for _ in range(ncols)]
    src, dst = L.ptr_array([b.device_ptr for b in bufs]), L.ptr_array([o.device_ptr for o in outs])
    logs = L.u32_array([log_size] * ncols)
    L.check(lib.stwo_interpolate_columns(src, logs, ncols, tree.itwiddles.device_ptr, len(tree.itwiddles), None))
    L.check(lib.stwo_extend_evaluate_columns(src, logs, dst, blowup, ncols, tree.twiddles.device_ptr,
                                             len(tree.twiddles), None))
    L.check(lib.stwo_stream_synchronize(None))

    def oc(log):
        c = stwo.CanonicCoset(log).half_coset()
        return oracle.coset(c.initial_index, c.step_size, c.log_size)
    for k in sorted({0, 1, ncols // 2, ncols - 1} & set(range(ncols))):
        coeffs = oracle.interpolate(oc(log_size), vals[k], itw)
        assert (bufs[k].to_numpy() == coeffs).all(), k
        assert (outs[k].to_numpy() == oracle.evaluate(oc(log_size + blowup), coeffs, tw)).all(), k
    # the other columns through the round trip
    L.check(lib.stwo_evaluate_columns(src, logs, ncols, tree.twiddles.device_ptr, len(tree.twiddles), None))
    L.check(lib.stwo_stream_synchronize(None))
    assert all((b.to_numpy() == v).all() for b, v in zip(bufs, vals))
