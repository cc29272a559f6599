"""Batch inverse at the edges of a thread's, a warp's and a CTA's share, and on QM31 values
with coordinates at the ends of the field (zero norm parts, P - 1). Every value is exact."""
import itertools

import numpy as np
import pytest

from helpers import P, m31, m31_nonzero, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 33, 481, 511, 513, 2047, 2049, 4097])
def test_sizes(stwo, oracle, n):
    L = stwo._lib
    v = m31_nonzero(rng(n), n)
    guard = np.concatenate([v, np.full(64, 7, np.uint32)])
    src, dst = stwo.BaseFieldVec.from_numpy(guard), stwo.BaseFieldVec.from_numpy(guard)
    L.check(L.lib().stwo_batch_inverse_m31(src.device_ptr, dst.device_ptr, n, None))
    L.check(L.lib().stwo_stream_synchronize(None))
    got = dst.to_numpy()
    assert (got[:n] == oracle.batch_inverse_m31(v)).all() and (got[n:] == 7).all()
    q = m31(rng(50 + n), 4 * n).reshape(n, 4)
    q[:, 3] |= 1
    guard = np.concatenate([q, np.full((64, 4), 7, np.uint32)])
    src, dst = stwo.SecureFieldVec.from_numpy(guard), stwo.SecureFieldVec.from_numpy(guard)
    L.check(L.lib().stwo_batch_inverse_qm31(src.device_ptr, dst.device_ptr, n, None))
    L.check(L.lib().stwo_stream_synchronize(None))
    got = dst.to_numpy()
    assert (got[:n] == oracle.batch_inverse_qm31(q)).all() and (got[n:] == 7).all()


def test_end_values(stwo, oracle):
    ends = [0, 1, 2, 1 << 30, P - 2, P - 1]
    q = np.array([c for c in itertools.product(ends, repeat=4) if any(c)], np.uint32)
    src, dst = stwo.SecureFieldVec.from_numpy(q), stwo.SecureFieldVec.new_uninitialized(len(q))
    stwo.CudaBackend.batch_inverse(src, dst)
    assert (dst.to_numpy() == oracle.batch_inverse_qm31(q)).all()
