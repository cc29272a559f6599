"""Launches of many short columns: a 2^14-element tile covers several columns, its last tile
fewer than it could hold. Columns at equal distances (a matrix's rows, with and without a
gap between them) travel as a base and a step, others through a table. Compared with the
oracle on columns at both ends and at tile boundaries; what lies behind and between the
columns stays as it was. Every value is exact."""
import numpy as np
import pytest

from helpers import m31, rng

pytestmark = pytest.mark.gpu

GUARD = 0x5A5A5A5A


def _matrix(stwo, values, stride):
    """values' rows at multiples of stride words in one buffer, guard words elsewhere."""
    n, size = values.shape
    host = np.full((n + 1, stride), GUARD, np.uint32)
    host[:n, :size] = values
    return host, stwo.BaseFieldVec.from_numpy(host)


@pytest.mark.parametrize("log_size,ncols,blowup,gap,shuffle", [
    (4, 16400, 1, 0, False),   # one layer group per thread pair, columns far shorter than a warp's part
    (5, 9001, 2, 0, True),
    (6, 16389, 1, 4, False),
    (7, 8195, 1, 0, False),
    (8, 4099, 2, 8, False),
    (9, 2051, 1, 0, True),
    (10, 1025, 2, 0, False),
    (11, 515, 1, 4, False),
    (12, 259, 2, 0, True),
    (13, 131, 1, 0, False),    # the extension's tile is one column
    (14, 67, 1, 4, False),
])
def test_short_columns_match_oracle(stwo, oracle, log_size, ncols, blowup, gap, shuffle):
    L = stwo._lib
    lib = L.lib()
    B = stwo.CudaBackend
    r = rng(7100 + log_size)
    n, m = 1 << log_size, 1 << (log_size + blowup)
    tree = B.precompute_twiddles(stwo.CanonicCoset(log_size + blowup).half_coset())
    tw, itw = tree.twiddles.to_numpy(), tree.itwiddles.to_numpy()
    vals = m31(r, ncols * n).reshape(ncols, n)
    _, buf = _matrix(stwo, vals, n + gap)
    _, out = _matrix(stwo, np.full((ncols, m), GUARD, np.uint32), m + gap)
    order = r.permutation(ncols) if shuffle else np.arange(ncols)
    src = L.ptr_array([buf.device_ptr + 4 * (n + gap) * int(k) for k in order])
    dst = L.ptr_array([out.device_ptr + 4 * (m + gap) * int(k) for k in order])
    logs = L.u32_array([log_size] * ncols)
    L.check(lib.stwo_interpolate_columns(src, logs, ncols, tree.itwiddles.device_ptr, len(tree.itwiddles), None))
    L.check(lib.stwo_extend_evaluate_columns(src, logs, dst, blowup, ncols, tree.twiddles.device_ptr,
                                             len(tree.twiddles), None))
    L.check(lib.stwo_stream_synchronize(None))
    got, ext = buf.to_numpy().reshape(ncols + 1, n + gap), out.to_numpy().reshape(ncols + 1, m + gap)
    assert (got[ncols] == GUARD).all() and (ext[ncols] == GUARD).all()
    assert (got[:, n:] == GUARD).all() and (ext[:, m:] == GUARD).all()

    def oc(c):
        return oracle.coset(c.initial_index, c.step_size, c.log_size)
    hc, ehc = oc(stwo.CanonicCoset(log_size).half_coset()), oc(stwo.CanonicCoset(log_size + blowup).half_coset())
    per_tile = max(1, 1 << (14 - log_size))
    for k in sorted({0, 1, per_tile - 1, per_tile, ncols // 2, ncols - 2, ncols - 1}):
        coeffs = oracle.interpolate(hc, vals[k], itw)
        assert (got[k, :n] == coeffs).all(), k
        assert (ext[k, :m] == oracle.evaluate(ehc, coeffs, tw)).all(), k
    # every other column, through the transforms' own round trip
    L.check(lib.stwo_evaluate_columns(src, logs, ncols, tree.twiddles.device_ptr, len(tree.twiddles), None))
    L.check(lib.stwo_stream_synchronize(None))
    assert (buf.to_numpy().reshape(ncols + 1, n + gap)[:ncols, :n] == vals).all()
