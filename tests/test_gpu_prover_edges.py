"""Proof bytes against the oracle prover where the FRI tail and the decommitment plan change
form: the largest inner layer at each side of the tail's split and of its first layer, the
last layer of every blowup, and query counts from one to more than the domain has points
(every node opened, no witness left)."""
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [
    (6, 3, 1, 2, 0),       # largest inner layer 2^7: the tail is one CTA's alone
    (7, 3, 1, 2, 0),       # 2^8
    (8, 5, 1, 3, 0),       # 2^9: the first split layer
    (9, 4, 4, 3, 0),       # 2^13: the tail's largest layer, last layer of 16 values
    (12, 4, 2, 4, 0),      # 2^14: one layer before the tail
    (5, 3, 3, 1, 0),
    (2, 3, 1, 1024, 0),    # every position queried
    (3, 7, 2, 200, 1),
    (8, 40, 1, 1024, 2),
], ids=lambda j: "L%d_N%d_B%d_q%d_pow%d" % j)
def test_proof_equals_oracle_proof(oracle, t):
    stwo = load_package()
    a0, a1 = stwo.wide_fib_inputs(t[0], 9000 + t[0] * 31 + t[3])
    proof, _ = stwo.prove_wide_fib(stwo.WideFibJob(*t), a0, a1)
    want, rc = oracle.wide_fib_prove(t[0], t[1], a0, a1, t[2], t[3], t[4])
    assert rc == 0
    assert proof == want


def test_batch_equals_single_proofs_across_the_split():
    """Several clusters in one launch, each with its own job's memory."""
    stwo = load_package()
    job = stwo.WideFibJob(10, 5, 1, 6, 2)
    tree = stwo.CudaBackend.precompute_twiddles(stwo.CanonicCoset(12).half_coset())
    inputs = [stwo.wide_fib_inputs(10, 70 + k) for k in range(5)]
    proofs, status, _ = stwo.prove_wide_fib_batch(job, inputs, tree)
    assert status == [0] * 5
    for (a0, a1), proof in zip(inputs, proofs):
        assert proof == stwo.prove_wide_fib(job, a0, a1, twiddles=tree)[0]
