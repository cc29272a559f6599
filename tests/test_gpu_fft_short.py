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


def _check(stwo, oracle, log_size, ncols, blowup, seed):
    """Interpolate and extend a matrix's rows with guard words behind and between them; rows at
    both ends and at tile boundaries against the oracle, the others by the round trip."""
    L = stwo._lib
    lib = L.lib()
    r = rng(seed)
    n, m, gap = 1 << log_size, 1 << (log_size + blowup), 4
    tree = stwo.CudaBackend.precompute_twiddles(stwo.CanonicCoset(log_size + blowup).half_coset())
    tw, itw = tree.twiddles.to_numpy(), tree.itwiddles.to_numpy()
    vals = m31(r, ncols * n).reshape(ncols, n)
    _, buf = _matrix(stwo, vals, n + gap)
    _, out = _matrix(stwo, np.full((ncols, m), GUARD, np.uint32), m + gap)
    src = L.ptr_array([buf.device_ptr + 4 * (n + gap) * k for k in range(ncols)])
    dst = L.ptr_array([out.device_ptr + 4 * (m + gap) * k for k in range(ncols)])
    logs = L.u32_array([log_size] * ncols)
    L.check(lib.stwo_interpolate_columns(src, logs, ncols, tree.itwiddles.device_ptr, len(tree.itwiddles), None))
    L.check(lib.stwo_extend_evaluate_columns(src, logs, dst, blowup, ncols, tree.twiddles.device_ptr,
                                             len(tree.twiddles), None))
    L.check(lib.stwo_stream_synchronize(None))
    got, ext = buf.to_numpy().reshape(ncols + 1, n + gap), out.to_numpy().reshape(ncols + 1, m + gap)
    assert (got[ncols] == GUARD).all() and (ext[ncols] == GUARD).all()
    assert (got[:, n:] == GUARD).all() and (ext[:, m:] == GUARD).all()

    def oc(log):
        c = stwo.CanonicCoset(log).half_coset()
        return oracle.coset(c.initial_index, c.step_size, c.log_size)
    per_tile = max(1, 1 << (14 - log_size))
    for k in sorted({0, 1, per_tile - 1, per_tile, ncols // 2, ncols - 1} & set(range(ncols))):
        coeffs = oracle.interpolate(oc(log_size), vals[k], itw)
        assert (got[k, :n] == coeffs).all(), k
        assert (ext[k, :m] == oracle.evaluate(oc(log_size + blowup), coeffs, tw)).all(), k
    L.check(lib.stwo_evaluate_columns(src, logs, ncols, tree.twiddles.device_ptr, len(tree.twiddles), None))
    L.check(lib.stwo_stream_synchronize(None))
    assert (buf.to_numpy().reshape(ncols + 1, n + gap)[:ncols, :n] == vals).all()


@pytest.mark.parametrize("log_size,ncols,blowup", [(11, 593, 1), (12, 297, 1), (13, 299, 1), (13, 297, 2)])
def test_partial_last_tile_with_32_elements_a_thread(stwo, oracle, log_size, ncols, blowup):
    """A 2^14 tile over 8, 4 or 2 columns by 512 threads, its last tile not full."""
    L = stwo._lib
    try:
        L.check(L.lib().stwo_set_tunable(b"fft_ept_contig_small", 5))
        _check(stwo, oracle, log_size, ncols, blowup, 7200 + log_size)
    finally:
        L.check(L.lib().stwo_set_tunable(b"fft_ept_contig_small", 6))


@pytest.mark.parametrize("log_size,ncols,blowup", [
    (4, 66, 10), (4, 70, 11), (5, 65, 9), (7, 67, 8), (8, 33, 7),
    (10, 64, 4), (10, 65, 5), (10, 70, 4), (9, 3, 12),
])
def test_short_columns_extended_beyond_a_tile(stwo, oracle, log_size, ncols, blowup):
    """Few coefficients evaluated on 2^14 points and more: the pass has 4..10 layers, its tile
    lies within one column, and reads of the coefficients wrap within the tile."""
    _check(stwo, oracle, log_size, ncols, blowup, 7300 + 20 * log_size + ncols)
