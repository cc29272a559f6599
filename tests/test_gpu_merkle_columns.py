"""The tree kernel at every kind of column count: four columns take their own compression
(twelve zero message words), other counts full and zero-padded chunks in one loop. Each
count at the leaves and, with children, at a dense and a thin inner layer; every layer
equals the oracle's."""
import pytest

from helpers import m31, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [1, 3, 4, 5, 8, 15, 16, 17, 20, 32, 36])
def test_tree_layers_match_oracle(stwo, oracle, nc):
    L = stwo._lib
    r = rng(3100 + nc)
    logs = [11] * nc + [10] * nc + [3] * nc + [0] * nc
    cols = [m31(r, 1 << lg) for lg in logs]
    bufs = [stwo.BaseFieldVec.from_numpy(c) for c in cols]
    layers = [stwo.BaseFieldVec.new_uninitialized(8 << l) for l in range(12)]
    L.check(L.lib().stwo_merkle_commit_tree(L.ptr_array([b.device_ptr for b in bufs]), L.u32_array(logs), len(logs),
                                            11, L.ptr_array([x.device_ptr for x in layers]), None))
    L.check(L.lib().stwo_stream_synchronize(None))
    want = oracle.merkle_commit(cols)
    for l in range(12):
        assert (layers[l].to_numpy().reshape(-1, 8) == want[l]).all(), l


@pytest.mark.parametrize("per", [(15, 1, 1, 1), (15, 16, 1, 1), (4, 3, 0, 2), (1, 4, 4, 5)])
@pytest.mark.parametrize("top", [2, 16, 17])
def test_small_trees_of_several_sizes_match_oracle(stwo, oracle, top, per):
    """Both sides of the rule for small trees: 16 and 17 as the largest log size, 15 and 16
    columns, one and two inner layers with other than four."""
    L = stwo._lib
    r = rng(3200 + top)
    logs = [lg for n, lg in zip(per, (top, top - 1, top // 2, 0)) for _ in range(n)]
    cols = [m31(r, 1 << lg) for lg in logs]
    bufs = [stwo.BaseFieldVec.from_numpy(c) for c in cols]
    layers = [stwo.BaseFieldVec.new_uninitialized(8 << l) for l in range(top + 1)]
    L.check(L.lib().stwo_merkle_commit_tree(L.ptr_array([b.device_ptr for b in bufs]), L.u32_array(logs), len(logs),
                                            top, L.ptr_array([x.device_ptr for x in layers]), None))
    L.check(L.lib().stwo_stream_synchronize(None))
    want = oracle.merkle_commit(cols)
    for l in range(top + 1):
        assert (layers[l].to_numpy().reshape(-1, 8) == want[l]).all(), l


@pytest.mark.parametrize("top,inner", [(4, 1), (14, 1), (15, 1), (15, 2), (16, 2), (16, 3), (17, 3), (17, 4), (18, 4),
                                       (18, 5), (19, 5), (19, 6), (20, 7)])
def test_trees_of_many_sizes_match_oracle(stwo, oracle, top, inner):
    """The rule's line over the tree's size: the inner layers it asks for up to 2^14 leaves, at
    2^15..2^19, and none above. Columns of the given number of inner sizes, the first of them
    with three, and four at one size more, whose layer the rule does not count."""
    L = stwo._lib
    r = rng(3300 + 10 * top + inner)
    logs = [top, top] + [top - 1] * 3 + [top - 1 - k for k in range(1, inner)] + [top - 1 - inner] * 4
    cols = [m31(r, 1 << lg) for lg in logs]
    bufs = [stwo.BaseFieldVec.from_numpy(c) for c in cols]
    layers = [stwo.BaseFieldVec.new_uninitialized(8 << l) for l in range(top + 1)]
    L.check(L.lib().stwo_merkle_commit_tree(L.ptr_array([b.device_ptr for b in bufs]), L.u32_array(logs), len(logs),
                                            top, L.ptr_array([x.device_ptr for x in layers]), None))
    L.check(L.lib().stwo_stream_synchronize(None))
    want = oracle.merkle_commit(cols)
    for l in range(top + 1):
        assert (layers[l].to_numpy().reshape(-1, 8) == want[l]).all(), l
