"""The public calls on streams of the caller's: non-blocking streams, work of others (torch)
between the calls, two streams joined by events, and capture into a CUDA graph. Results
equal those of the same calls waited for one by one (all values are exact)."""
import numpy as np
import pytest

from helpers import m31, random_qm31, rng

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


class Calls:
    """Buffers of one chain over `ncols` matrix rows of 2^log_size, and its calls."""

    def __init__(self, stwo, log_size, ncols, seed):
        assert ncols >= 4  # (the fold takes the first four rows as coordinates)
        self.L, self.lib, self.log, self.n = stwo._lib, stwo._lib.lib(), log_size, ncols
        self.tree = stwo.CudaBackend.precompute_twiddles(stwo.CanonicCoset(log_size + 1).half_coset())
        r = rng(seed)
        size = 1 << log_size

        def dev(a):
            return torch.from_numpy(a.astype(np.int32)).cuda()
        self.cols = dev(m31(r, ncols * size).reshape(ncols, size))
        self.ext = torch.zeros((ncols, 2 * size), dtype=torch.int32, device="cuda")
        self.mirror = torch.zeros_like(self.ext)
        self.line = dev(m31(r, 4 * size).reshape(4, size))
        self.layer = torch.zeros((2 * size, 8), dtype=torch.int32, device="cuda")
        self.inv = torch.zeros(2 * size, dtype=torch.int32, device="cuda")
        self.alpha = self.L.QM31(*random_qm31(r))
        self.logs = self.L.u32_array([log_size] * ncols)
        torch.cuda.synchronize()

    def ptrs(self, t):
        return self.L.ptr_array([row.data_ptr() for row in t])

    def interpolate(self, st):
        return self.lib.stwo_interpolate_columns(self.ptrs(self.cols), self.logs, self.n,
                                                 self.tree.itwiddles.device_ptr, len(self.tree.itwiddles), st)

    def extend(self, st):
        return self.lib.stwo_extend_evaluate_columns(self.ptrs(self.cols), self.logs, self.ptrs(self.ext), 1, self.n,
                                                     self.tree.twiddles.device_ptr, len(self.tree.twiddles), st)

    def fold(self, st):
        return self.lib.stwo_fold_circle_into_line(self.ptrs(self.mirror[:4]), 2 << self.log, self.alpha,
                                                   self.tree.itwiddles.device_ptr,
                                                   len(self.tree.itwiddles) - (1 << self.log), self.ptrs(self.line),
                                                   st)

    def hash(self, st):
        return self.lib.stwo_merkle_commit_layer(self.log + 1, None, self.ptrs(self.mirror), self.n,
                                                 self.layer.data_ptr(), st)

    def inverse(self, st):
        return self.lib.stwo_batch_inverse_m31(self.mirror[0].data_ptr(), self.inv.data_ptr(), 2 << self.log, st)

    def round(self, stream, wait=False):
        """interpolate -> extend -> torch: rows reversed into the mirror -> fold, layer, inverse ->
        torch: the next round's columns."""
        def done(rc):
            self.L.check(rc)
            if wait:
                torch.cuda.synchronize()
        st = stream.cuda_stream
        with torch.cuda.stream(stream):
            done(self.interpolate(st))
            done(self.extend(st))
            self.mirror.copy_(self.ext.flip(1))
            done(0)
            done(self.fold(st))
            done(self.hash(st))
            done(self.inverse(st))
            self.cols.copy_(self.ext[:, : 1 << self.log])
            done(0)

    def results(self):
        torch.cuda.synchronize()
        return [t.clone() for t in (self.cols, self.ext, self.line, self.layer, self.inv)]


def _equal(a, b):
    return all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("log_size,ncols", [(6, 5), (11, 70), (13, 8), (16, 4)])
def test_chain_on_a_non_blocking_stream(stwo, log_size, ncols):
    runs = []
    for wait in (False, True):
        c, s = Calls(stwo, log_size, ncols, 400 + log_size), torch.cuda.Stream()
        for _ in range(6):
            c.round(s, wait)
        runs.append(c.results())
    assert _equal(*runs)


@pytest.mark.parametrize("log_size", [8, 14])
def test_two_streams_joined_by_events(stwo, log_size):
    """Each round's transforms on one stream and what reads them on another, ordered both ways
    by events only."""
    runs = []
    for wait in (False, True):
        c = Calls(stwo, log_size, 6, 500 + log_size)
        a, b = torch.cuda.Stream(), torch.cuda.Stream()
        for _ in range(6):
            stwo._lib.check(c.interpolate(a.cuda_stream))
            stwo._lib.check(c.extend(a.cuda_stream))
            b.wait_event(a.record_event())
            if wait:
                torch.cuda.synchronize()
            with torch.cuda.stream(b):
                c.mirror.copy_(c.ext)
            stwo._lib.check(c.fold(b.cuda_stream))
            stwo._lib.check(c.hash(b.cuda_stream))
            stwo._lib.check(c.inverse(b.cuda_stream))
            with torch.cuda.stream(b):
                c.cols.copy_(c.ext[:, : 1 << log_size])
            a.wait_event(b.record_event())
            if wait:
                torch.cuda.synchronize()
        runs.append(c.results())
    assert _equal(*runs)


@pytest.mark.parametrize("log_size,ncols", [(4, 100), (10, 65), (12, 100), (15, 70), (13, 4)])
def test_captured_rows_replay_on_new_inputs(stwo, log_size, ncols):
    """A round over matrix rows (above 64 columns: as base and step) recorded into a graph and
    replayed on changed inputs."""
    c, d = Calls(stwo, log_size, ncols, 600), Calls(stwo, log_size, ncols, 600)
    s = torch.cuda.Stream()
    d.round(s)  # (first launches of every kernel outside the capture)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        c.round(s)
    for seed in (601, 602):
        fresh = torch.from_numpy(m31(rng(seed), ncols << log_size).astype(np.int32)).cuda().reshape(ncols, -1)
        for x in (c, d):
            x.cols.copy_(fresh)
            x.line.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            graph.replay()
        d.round(s, wait=True)
        assert _equal(c.results(), d.results())


@pytest.mark.parametrize("order", ["descending", "mixed"])
def test_staged_tables_are_refused_under_capture(stwo, order):
    """More than 64 columns not at equal distances, and whole trees, copy a table from the
    call's own memory: refused while the stream is captured, computed otherwise."""
    L, lib = stwo._lib, stwo._lib.lib()
    c = Calls(stwo, 5, 100, 700)
    want = Calls(stwo, 5, 100, 700)
    rows = np.arange(100)[::-1] if order == "descending" else rng(701).permutation(100)
    ptrs = L.ptr_array([c.cols[int(k)].data_ptr() for k in rows])
    layers = [torch.zeros((1 << l, 8), dtype=torch.int32, device="cuda") for l in range(6)]
    layer_ptrs = L.ptr_array([t.data_ptr() for t in layers])
    tw, size = c.tree.itwiddles.device_ptr, len(c.tree.itwiddles)
    s = torch.cuda.Stream()
    x = torch.zeros(4, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        x.add_(1)
        status = [lib.stwo_interpolate_columns(ptrs, c.logs, 100, tw, size, s.cuda_stream),
                  lib.stwo_merkle_commit_tree(ptrs, c.logs, 100, 5, layer_ptrs, s.cuda_stream)]
    L.clear_error()
    assert status == [L.ERR_INVALID_ARGUMENT] * 2
    graph.replay()
    L.check(lib.stwo_interpolate_columns(ptrs, c.logs, 100, tw, size, s.cuda_stream))
    L.check(want.interpolate(None))
    torch.cuda.synchronize()
    assert torch.equal(c.cols, want.cols) and x.tolist() == [1] * 4
