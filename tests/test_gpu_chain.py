"""Chains of dependent calls on one stream with no wait between them: each kernel's CTAs may
be placed while the one before drains, so every kernel has to wait for it before it reads.
The chain's result equals the same calls waited for one by one (all values are exact)."""
import numpy as np
import pytest

from helpers import P, m31, random_qm31, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 1000, 1 << 16])
def test_accumulate_chain(stwo, n):
    L = stwo._lib
    r = rng(n)
    a, b = [m31(r, n) for _ in range(4)], [m31(r, n) for _ in range(4)]
    x, y = stwo.SecureColumnByCoords.from_numpy(a), stwo.SecureColumnByCoords.from_numpy(b)
    for _ in range(40):
        L.check(L.lib().stwo_accumulate(x.ptrs(), y.ptrs(), n, None))
        L.check(L.lib().stwo_accumulate(y.ptrs(), x.ptrs(), n, None))
    L.check(L.lib().stwo_stream_synchronize(None))
    a, b = [c.astype(np.uint64) for c in a], [c.astype(np.uint64) for c in b]
    for _ in range(40):
        a = [(u + v) % P for u, v in zip(a, b)]
        b = [(u + v) % P for u, v in zip(b, a)]
    assert all((g == e).all() for g, e in zip(x.to_numpy(), a))
    assert all((g == e).all() for g, e in zip(y.to_numpy(), b))


@pytest.mark.parametrize("log_size", [6, 13, 18])
def test_mixed_chain_equals_waited_calls(stwo, log_size):
    """interpolate -> extend -> fold -> fold -> accumulate -> tree -> inverse, three rounds."""
    L = stwo._lib
    lib = L.lib()
    B = stwo.CudaBackend
    r = rng(90 + log_size)
    n, m = 1 << log_size, 2 << log_size
    tree = B.precompute_twiddles(stwo.CanonicCoset(log_size + 1).half_coset())
    tw, itw, size = tree.twiddles.device_ptr, tree.itwiddles.device_ptr, len(tree.twiddles)
    start = [m31(r, n) for _ in range(4)]
    alphas = [L.QM31(*random_qm31(r)) for _ in range(6)]
    logs = L.u32_array([log_size] * 4)

    def run(wait):
        def done(rc):
            L.check(rc)
            if wait:
                L.check(lib.stwo_stream_synchronize(None))
        cols = stwo.SecureColumnByCoords.from_numpy(start)
        ext = stwo.SecureColumnByCoords.zeros(m)
        line, half = stwo.SecureColumnByCoords.zeros(n), stwo.SecureColumnByCoords.zeros(n // 2)
        layers = [stwo.Blake2sHashVec.new_uninitialized(1 << k) for k in range(log_size + 1)]
        inv = stwo.BaseFieldVec.new_uninitialized(n)
        for k in range(3):
            done(lib.stwo_interpolate_columns(cols.ptrs(), logs, 4, itw, size, None))
            done(lib.stwo_extend_evaluate_columns(cols.ptrs(), logs, ext.ptrs(), 1, 4, tw, size, None))
            done(lib.stwo_fold_circle_into_line(ext.ptrs(), m, alphas[2 * k], itw, size - n, line.ptrs(), None))
            done(lib.stwo_fold_line(line.ptrs(), n, alphas[2 * k + 1], itw, size - n, half.ptrs(), None))
            done(lib.stwo_accumulate(cols.ptrs(), line.ptrs(), n, None))
            for lg in range(log_size, -1, -1):
                done(lib.stwo_merkle_commit_layer(
                    lg, layers[lg + 1].device_ptr if lg < log_size else None, line.ptrs(), 4 if lg == log_size else 0,
                    layers[lg].device_ptr, None))
            done(lib.stwo_batch_inverse_m31(line.columns[0].device_ptr, inv.device_ptr, n, None))
        L.check(lib.stwo_stream_synchronize(None))
        return cols.to_numpy() + line.to_numpy() + half.to_numpy() + [layers[0].to_numpy(), inv.to_numpy()]

    for got, expect in zip(run(False), run(True)):
        assert (got == expect).all()
