"""The settings of the transforms' elements per thread reach the launches they name. Each
setting runs in a process of its own, which lists the pass kernels it launched (their
template arguments: layers, column bits, inverse, log2 elements a thread, compiled lowest
layer, log2 tile) and a digest of its results; every setting computes the same values."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import ctypes as C, hashlib, json, os, re, sys, tempfile
sys.path.insert(0, os.getcwd())
import torch
import stwo_gpu_b200 as stwo
L = stwo._lib
lib = L.lib()
spec = json.loads(sys.argv[1])
for name, value in spec["tunables"]:
    L.check(lib.stwo_set_tunable(name.encode(), value))
top = max(log + blowup for _, log, blowup in spec["shapes"])
tree = stwo.CudaBackend.precompute_twiddles(stwo.CanonicCoset(top).half_coset())
gen = torch.Generator("cuda").manual_seed(5)
digest = hashlib.sha256()
def transforms():
    for ncols, log, blowup in spec["shapes"]:
        cols = torch.randint(0, 2**31 - 1, (ncols, 1 << log), dtype=torch.int32, device="cuda", generator=gen)
        out = torch.zeros((ncols, 1 << (log + blowup)), dtype=torch.int32, device="cuda")
        src, dst = L.ptr_array([c.data_ptr() for c in cols]), L.ptr_array([o.data_ptr() for o in out])
        logs = L.u32_array([log] * ncols)
        torch.cuda.synchronize()
        L.check(lib.stwo_interpolate_columns(src, logs, ncols, tree.itwiddles.device_ptr, len(tree.itwiddles), None))
        L.check(lib.stwo_extend_evaluate_columns(src, logs, dst, blowup, ncols, tree.twiddles.device_ptr,
                                                 len(tree.twiddles), None))
        torch.cuda.synchronize()
        digest.update(cols.cpu().numpy().tobytes())
        digest.update(out.cpu().numpy().tobytes())
with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
    transforms()
    if spec["autotune"]:
        buf = C.create_string_buffer(4096)
        L.check(lib.stwo_autotune(buf, 4096))
    torch.cuda.synchronize()
path = os.path.join(tempfile.mkdtemp(), "trace.json")
prof.export_chrome_trace(path)
passes = []
for e in json.load(open(path))["traceEvents"]:
    m = re.search(r"fftT_kernel<(\d+), (\d+), (\w+), (\d+), (\d+), (\d+)>", e.get("name", ""))
    if m and e.get("cat") == "kernel":
        inv = m[3] in ("true", "1")
        passes.append([int(m[1]), int(m[2]), inv, int(m[4]), int(m[5]), int(m[6]), e["args"]["grid"][0]])
print(json.dumps({"passes": passes, "digest": digest.hexdigest()}))
"""


def run(shapes, tunables=(), env=None, autotune=False):
    spec = json.dumps({"shapes": shapes, "tunables": list(tunables), "autotune": autotune})
    e = {k: v for k, v in os.environ.items() if k != "STWO_FFT_EPT_LOG"}
    e.update(env or {})
    r = subprocess.run([sys.executable, "-c", PROGRAM, spec], cwd=ROOT, env=e, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    got = json.loads(r.stdout.strip().splitlines()[-1])
    if not got["passes"]:
        pytest.skip("the profiler lists no kernels here")
    return got


def test_forced_elements_per_thread_reach_every_pass():
    """Small launches, which spread over more threads by themselves, and large ones."""
    shapes = [[1, 11, 1], [64, 12, 1], [3, 13, 2], [1, 14, 1], [4, 16, 1], [700, 12, 1]]
    base = run(shapes)
    small = {(11, 4, 12), (12, 4, 12), (13, 5, 13), (14, 5, 14)}
    assert {(g, ept, t) for g, c, _, ept, _, t, _ in base["passes"] if c == 0} >= small
    for value in (5, 6):
        got = run(shapes, env={"STWO_FFT_EPT_LOG": str(value)})
        assert {(ept, t) for *_, ept, _, t, _ in got["passes"]} == {(value, 14)}
        assert got["digest"] == base["digest"]


def test_autotune_times_both_candidates_of_every_launch():
    """Every contiguous 14-layer launch shape that autotune times runs with 2^5 and with 2^6
    elements a thread; one that the library chooses by itself would run with the same twice."""
    got = run([[300, 4, 1]], autotune=True)
    shapes = {}
    for g, c, inv, ept, _, _, grid in got["passes"]:
        if g == 14 and c == 0:
            shapes.setdefault((inv, grid), set()).add(ept)
    assert len(shapes) >= 4 and all(v == {5, 6} for v in shapes.values()), shapes


def test_strided_passes_of_both_settings_are_compiled_for_their_row_distance():
    """The strided pass right above the bottom one (lowest layer 14, 6 layers and more), with 32
    as with 64 elements a thread, so that the setting compares like with like."""
    shapes = [[2, 20, 1], [1, 22, 1], [1, 23, 1]]
    found = []
    for value in (6, 5):
        got = run(shapes, tunables=[["fft_ept_strided", value]])
        strided = sorted({(g, c, inv, lowest, ept) for g, c, inv, ept, lowest, _, _ in got["passes"] if c})
        assert strided and all(lowest == 14 and ept == value for *_, lowest, ept in strided), strided
        found.append(([s[:3] for s in strided], got["digest"]))
    assert found[0] == found[1]
