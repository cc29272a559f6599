"""The device-memory bound of a proof (what the server admits jobs by, and the slab that a
proof reserves) covers what the proof allocates on the device, and little more. The
decommitment's reads go through pinned host memory, so the query count does not enter."""
import pytest

from conftest import load_package

SHAPES = [(2, 3, 1), (6, 100, 2), (8, 40, 1), (10, 256, 1), (12, 64, 4), (14, 1024, 1)]


@pytest.mark.parametrize("own", [True, False])
@pytest.mark.parametrize("shape", SHAPES)
def test_bound_is_the_same_for_every_query_count(shape, own):
    stwo = load_package()
    bounds = {stwo.WideFibJob(*shape, q, 5).device_bytes(own_twiddles=own) for q in (1, 3, 70, 1024)}
    assert len(bounds) == 1 and bounds.pop() > 0


@pytest.mark.gpu
@pytest.mark.parametrize("queries", [1, 1024])
@pytest.mark.parametrize("shape", SHAPES)
def test_bound_covers_the_proof_and_little_more(shape, queries):
    """At most 64 KiB above: up to 256 bytes for each of at most 29 tables that a shape may do
    without, one tree of at most 2^4 leaves, a third transform table of 16 bytes a column
    (the evaluation partials are exact up to 2^15 rows)."""
    stwo = load_package()
    job = stwo.WideFibJob(*shape, queries, 0)
    a0, a1 = stwo.wide_fib_inputs(shape[0], 41)
    tree = stwo.CudaBackend.precompute_twiddles(stwo.CanonicCoset(shape[0] + 1 + shape[2]).half_coset())
    for twiddles in (None, tree):
        _, stats = stwo.prove_wide_fib(job, a0, a1, twiddles=twiddles)
        bound = job.device_bytes(own_twiddles=twiddles is None)
        assert bound - (64 << 10) <= stats["device_bytes"] <= bound
