"""What is timed: the work that programs have this library do, through its public entry points.

Programs come in three kinds, and the cases follow them:

* a prover written elsewhere (the reference's Rust backend, or any other) that calls the C ABI's
  asynchronous tier on its own device buffers: transforms, trees, quotients, folds, inverses,
  out-of-domain evaluations;
* a program on the Python mirror of the backend traits (`CudaBackend`), one call per trait method;
* a program that wants proofs: one at a time (`prove_wide_fib`), or many jobs of uneven sizes at
  once (`ProofServer`).

All values are M31 elements, uniform in [0, 2^31 - 1): trace columns, evaluations and quotients of
a proof are indistinguishable from uniform ones, and no path depends on the values. Everything
that comes back is a whole number of the field, a hash or a proof byte.
"""
import numpy as np
import torch

from stwo_gpu_b200 import (BaseFieldVec, CanonicCoset, CircleEvaluation, CudaBackend, ProofServer, ProveCache,
                           WideFibJob, prove_wide_fib, wide_fib_inputs)
from stwo_gpu_b200 import _lib as L

P = (1 << 31) - 1


def listed():
    return [
        # The smallest calls: a short table committed through the trait methods, one synchronous call
        # each (interpolate_columns, evaluate_polynomials, commit_on_layer per layer). Latency only.
        {"name": "trait_commit_3x2^10", "op": "trait_commit", "columns": 3, "log": 10, "blowup": 1},
        # An ordinary trace commit's transforms: an odd number of columns of a middle size.
        {"name": "lde_101x2^16", "op": "lde", "columns": 101, "log": 16, "blowup": 1},
        # The largest transforms: a few very long columns, interpolated and extended fourfold.
        {"name": "lde_8x2^24", "op": "lde", "columns": 8, "log": 24, "blowup": 2},
        # Very many short columns (2^16 polynomials of 2^10 coefficients, extended fourfold).
        {"name": "lde_65536x2^10", "op": "lde", "columns": 65536, "log": 10, "blowup": 2},
        # The commitment of a proof with tables of many heights: four columns at each log size.
        {"name": "tree_4_at_12..22", "op": "tree", "per_size": 4, "min_log": 12, "max_log": 22},
        # DEEP quotients of a long trace that is sampled at four points.
        {"name": "quotients_32x2^22x4", "op": "quotients", "columns": 32, "log": 22, "points": 4},
        # The FRI folds of a long quotient: circle to line, then to the last layer.
        {"name": "folds_2^24", "op": "folds", "log": 24},
        # Denominators of a lookup argument inverted at once; their number is no power of two.
        {"name": "inverse_qm31_9999991", "op": "inverse", "field": "qm31", "n": 9999991},
        # Out-of-domain values of a trace with columns of two heights.
        {"name": "oods_32x2^21..22", "op": "oods", "columns": 32, "min_log": 21, "max_log": 22},
        # One small proof after another, the same shape every time (the cache and its graph).
        {"name": "proof_64x2^12", "op": "proof", "log": 12, "columns": 64, "blowup": 1, "queries": 3, "pow_bits": 5,
         "cache": True},
        # One large proof.
        {"name": "proof_256x2^20", "op": "proof", "log": 20, "columns": 256, "blowup": 1, "queries": 3,
         "pow_bits": 10, "cache": False},
        # A burst of jobs of uneven sizes through the proof server, inputs on the host.
        {"name": "serve_24_jobs", "op": "serve", "jobs": 24, "min_log": 10, "max_log": 20, "workers": 8},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    op = rng.choice(["trait_commit", "lde", "lde", "lde", "tree", "tree", "quotients", "quotients", "folds", "inverse",
                     "oods", "proof", "proof", "proof", "serve"])
    if op == "trait_commit":
        return {"op": op, "columns": rng.randint(1, 12), "log": rng.randint(6, 13), "blowup": rng.randint(1, 2)}
    if op == "lde":
        log, blowup = rng.randint(5, 23), rng.randint(1, 3)
        most = max(1, min(65536, 1 << (28 - log - blowup)))
        return {"op": op, "columns": _log_uniform(rng, 1, most), "log": log, "blowup": blowup}
    if op == "tree":
        top = rng.randint(8, 21)
        return {"op": op, "per_size": _log_uniform(rng, 1, 40), "min_log": rng.randint(4, top), "max_log": top}
    if op == "quotients":
        log = rng.randint(8, 21)
        return {"op": op, "columns": _log_uniform(rng, 1, min(300, 1 << (28 - log))), "log": log,
                "points": rng.randint(1, 4)}
    if op == "folds":
        return {"op": op, "log": rng.randint(8, 24)}
    if op == "inverse":
        return {"op": op, "field": rng.choice(["m31", "qm31"]), "n": _log_uniform(rng, 100, 16000000)}
    if op == "oods":
        top = rng.randint(8, 22)
        return {"op": op, "columns": _log_uniform(rng, 1, min(300, 1 << (28 - top))), "min_log": rng.randint(6, top),
                "max_log": top}
    if op == "proof":
        log, blowup = rng.randint(4, 18), rng.randint(1, 2)
        return {"op": op, "log": log, "columns": _log_uniform(rng, 3, min(1024, 1 << (27 - log - blowup))),
                "blowup": blowup, "queries": rng.randint(1, 30), "pow_bits": rng.randint(0, 10),
                "cache": rng.random() < 0.5}
    top = rng.randint(12, 18)
    return {"op": op, "jobs": rng.randint(4, 24), "min_log": rng.randint(8, top), "max_log": top,
            "workers": rng.choice([1, 4, 8])}


# ----------------------------------------------------------------------------- helpers
def _uniform(gen, *shape):
    return torch.randint(0, P, shape, dtype=torch.int32, device="cuda", generator=gen)


def _ptrs(tensors):
    return L.ptr_array([t.data_ptr() for t in tensors])


def _stream():
    return torch.cuda.current_stream().cuda_stream or None


def _qm31(rng):
    return tuple(int(v) for v in rng.integers(0, P, 4))


def _cm_mul(x, y):
    return ((x[0] * y[0] - x[1] * y[1]) % P, (x[0] * y[1] + x[1] * y[0]) % P)


def _q_mul(x, y):
    ac, bd = _cm_mul(x[:2], y[:2]), _cm_mul(x[2:], y[2:])
    rbd = _cm_mul((2, 1), bd)
    ad, bc = _cm_mul(x[:2], y[2:]), _cm_mul(x[2:], y[:2])
    return ((ac[0] + rbd[0]) % P, (ac[1] + rbd[1]) % P, (ad[0] + bc[0]) % P, (ad[1] + bc[1]) % P)


def _q_inv(x):
    a, b = x[:2], x[2:]
    aa, rbb = _cm_mul(a, a), _cm_mul((2, 1), _cm_mul(b, b))
    d = ((aa[0] - rbb[0]) % P, (aa[1] - rbb[1]) % P)
    n = pow((d[0] * d[0] + d[1] * d[1]) % P, P - 2, P)
    di = (d[0] * n % P, -d[1] * n % P)
    ra, rb = _cm_mul(a, di), _cm_mul(b, di)
    return (ra[0], ra[1], -rb[0] % P, -rb[1] % P)


def _circle_point(rng):
    """A point of the circle over QM31, as a channel draws it: ((1 - t^2) / (1 + t^2), 2t / (1 + t^2))."""
    t = _qm31(rng)
    t2 = _q_mul(t, t)
    inv = _q_inv(((1 + t2[0]) % P, t2[1], t2[2], t2[3]))
    x = _q_mul(((1 - t2[0]) % P, -t2[1] % P, -t2[2] % P, -t2[3] % P), inv)
    return x, _q_mul(tuple(2 * v % P for v in t), inv)


class _DeviceArray:
    """A library buffer as torch sees it (no copy; the buffer lives as long as the tensor)."""

    def __init__(self, vec):
        self.vec = vec
        self.__cuda_array_interface__ = {"shape": (len(vec) * vec.words_per_elem,), "typestr": "<i4",
                                         "data": (vec.device_ptr, False), "version": 3}


def _tensor(vec):
    return torch.as_tensor(_DeviceArray(vec), device="cuda")


def _twiddles(log):
    return CudaBackend.precompute_twiddles(CanonicCoset(max(log, 4)).half_coset())


def _served_jobs(case, rng):
    return [WideFibJob(int(rng.integers(case["min_log"], case["max_log"] + 1)), int(rng.choice([16, 32, 64, 128])))
            for _ in range(case["jobs"])]


def _shapes_rng(case):
    # The shapes of a burst (and the sizes of mixed columns) are the case's own; the seed draws the values.
    return np.random.default_rng([case.get("jobs", 0), case.get("columns", 0), case["min_log"], case["max_log"]])


def _mixed_logs(case):
    return [int(v) for v in _shapes_rng(case).integers(case["min_log"], case["max_log"] + 1, case["columns"])]


def _tree_logs(case):
    return [lg for lg in range(case["max_log"], case["min_log"] - 1, -1) for _ in range(case["per_size"])]


# ----------------------------------------------------------------------------- prepare
def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    s = {"case": dict(case), "op": case["op"]}
    op = case["op"]
    if op == "trait_commit":
        s["domain"] = CanonicCoset(case["log"])
        s["values"] = [BaseFieldVec.from_numpy(rng.integers(0, P, 1 << case["log"], dtype=np.uint32))
                       for _ in range(case["columns"])]
        s["twiddles"] = _twiddles(case["log"] + case["blowup"])
    elif op == "lde":
        n, log, blowup = case["columns"], case["log"], case["blowup"]
        s["values"] = _uniform(gen, n, 1 << log)
        s["out"] = torch.empty((n, 1 << (log + blowup)), dtype=torch.int32, device="cuda")
        s["twiddles"] = _twiddles(log + blowup)
        s["value_ptrs"], s["out_ptrs"] = _ptrs(s["values"]), _ptrs(s["out"])
        s["logs"] = L.u32_array([log] * n)
    elif op == "tree":
        logs = _tree_logs(case)
        s["columns"] = [_uniform(gen, 1 << lg) for lg in logs]
        s["layers"] = [torch.empty((1 << lg, 8), dtype=torch.int32, device="cuda")
                       for lg in range(case["max_log"] + 1)]
        s["column_ptrs"], s["layer_ptrs"] = _ptrs(s["columns"]), _ptrs(s["layers"])
        s["logs"] = L.u32_array(logs)
    elif op == "quotients":
        n, log, points = case["columns"], case["log"], case["points"]
        s["columns"] = _uniform(gen, n, 1 << log)
        s["out"] = torch.empty((4, 1 << log), dtype=torch.int32, device="cuda")
        s["column_ptrs"], s["out_ptrs"] = _ptrs(s["columns"]), _ptrs(s["out"])
        s["domain"] = CanonicCoset(log).half_coset()
        pts = [_circle_point(rng) for _ in range(points)]
        s["points"] = (L.SPoint * points)(*[L.SPoint(L.QM31(*x), L.QM31(*y)) for x, y in pts])
        s["sizes"] = L.u32_array([n] * points)
        s["indices"] = L.u32_array(list(range(n)) * points)
        s["sampled"] = (L.QM31 * (n * points))(*[L.QM31(*_qm31(rng)) for _ in range(n * points)])
        s["coeff"] = L.QM31(*_qm31(rng))
    elif op == "folds":
        log = case["log"]
        s["layers"] = [_uniform(gen, 4, 1 << log)]
        s["layers"] += [torch.zeros((4, 1 << lg), dtype=torch.int32, device="cuda") for lg in range(log - 1, 3, -1)]
        s["ptrs"] = [_ptrs(v) for v in s["layers"]]
        s["alphas"] = [L.QM31(*_qm31(rng)) for _ in s["layers"]]
        s["twiddles"] = _twiddles(log)
    elif op == "inverse":
        n = case["n"]
        v = _uniform(gen, n) if case["field"] == "m31" else _uniform(gen, n, 4)
        s["values"] = torch.where(v == 0, torch.ones_like(v), v)
        s["out"] = torch.empty_like(v)
    elif op == "oods":
        logs = _mixed_logs(case)
        s["columns"] = [_uniform(gen, 1 << lg) for lg in logs]
        s["column_ptrs"], s["logs"] = _ptrs(s["columns"]), L.u32_array(logs)
        x, y = _circle_point(rng)
        s["points"] = (L.SPoint * len(logs))(*[L.SPoint(L.QM31(*x), L.QM31(*y)) for _ in logs])
        s["out"] = torch.empty((len(logs), 4), dtype=torch.int32, device="cuda")
        s["scratch_bytes"] = int(L.lib().stwo_eval_at_points_scratch_bytes(s["logs"], len(logs)))
        s["scratch"] = torch.empty(s["scratch_bytes"] // 4 + 4, dtype=torch.int32, device="cuda")
    elif op == "proof":
        s["job"] = WideFibJob(case["log"], case["columns"], case["blowup"], case["queries"], case["pow_bits"])
        s["inputs"] = wide_fib_inputs(case["log"], int(seed))
        s["twiddles"] = _twiddles(case["log"] + 1 + case["blowup"])
        s["cache"] = ProveCache() if case["cache"] else None
        s["stream"] = torch.cuda.Stream()
    elif op == "serve":
        s["jobs"] = _served_jobs(case, _shapes_rng(case))
        s["inputs"] = [wide_fib_inputs(j.log_n_rows, int(seed) * 1000 + k) for k, j in enumerate(s["jobs"])]
        s["server"] = ProofServer(n_workers=case["workers"], device_budget_bytes=24 << 30,
                                  max_domain_log=case["max_log"] + 2)
    else:
        raise ValueError(f"unknown op {op}")
    return s


# ----------------------------------------------------------------------------- run
def _run_trait_commit(s):
    # The polynomials' coefficients stay in the value columns, as interpolate leaves them.
    domain = s["domain"].circle_domain()
    polys = CudaBackend.interpolate_columns([CircleEvaluation(domain, v) for v in s["values"]], s["twiddles"])
    evals = CudaBackend.evaluate_polynomials(polys, s["case"]["blowup"], s["twiddles"])
    layer, layers = None, []
    for lg in range(s["case"]["log"] + s["case"]["blowup"], -1, -1):
        layer = CudaBackend.commit_on_layer(lg, layer, [] if layers else [e.values for e in evals])
        layers.append(layer)
    return {"evaluations": [_tensor(e.values) for e in evals], "layers": [_tensor(v) for v in layers]}


def _run_lde(s):
    lib, n, tw, st = L.lib(), s["case"]["columns"], s["twiddles"], _stream()
    L.check(lib.stwo_interpolate_columns(s["value_ptrs"], s["logs"], n, tw.itwiddles.device_ptr, len(tw.itwiddles),
                                         st))
    L.check(lib.stwo_extend_evaluate_columns(s["value_ptrs"], s["logs"], s["out_ptrs"], s["case"]["blowup"], n,
                                             tw.twiddles.device_ptr, len(tw.twiddles), st))
    return {"coefficients": s["values"], "evaluations": s["out"]}


def _run_tree(s):
    L.check(L.lib().stwo_merkle_commit_tree(s["column_ptrs"], s["logs"], len(s["columns"]), s["case"]["max_log"],
                                            s["layer_ptrs"], _stream()))
    return s["layers"]


def _run_quotients(s):
    d = s["domain"]
    L.check(L.lib().stwo_accumulate_quotients(
        d.initial_index, d.step_size, s["case"]["log"], s["column_ptrs"], s["case"]["columns"], s["coeff"],
        s["points"], s["sizes"], s["indices"], s["sampled"], s["case"]["points"], s["out_ptrs"], _stream()))
    return s["out"]


def _run_folds(s):
    lib, tw, st = L.lib(), s["twiddles"], _stream()
    size = len(tw.itwiddles)
    for k in range(len(s["layers"]) - 1):
        n = 1 << (s["case"]["log"] - k)
        fold = lib.stwo_fold_line if k else lib.stwo_fold_circle_into_line
        L.check(fold(s["ptrs"][k], n, s["alphas"][k], tw.itwiddles.device_ptr, size - (n if k else n >> 1),
                     s["ptrs"][k + 1], st))
    return s["layers"][1:]


def _run_inverse(s):
    lib = L.lib()
    f = lib.stwo_batch_inverse_m31 if s["case"]["field"] == "m31" else lib.stwo_batch_inverse_qm31
    L.check(f(s["values"].data_ptr(), s["out"].data_ptr(), s["case"]["n"], _stream()))
    return s["out"]


def _run_oods(s):
    L.check(L.lib().stwo_eval_at_points(s["column_ptrs"], s["logs"], len(s["columns"]), s["points"],
                                        s["out"].data_ptr(), s["scratch"].data_ptr(), s["scratch_bytes"], _stream()))
    return s["out"]


def _proof_bytes(job, proof):
    """The proof and its length, zero-padded to a size that the job's shape sets (queries that coincide make a
    proof shorter, and which do depends on the inputs)."""
    most = (job.n_columns + 8) * (64 + 16 * job.n_queries) + (job.n_queries + 1) * (job.log_n_rows + 8) ** 2 * 64
    out = np.zeros(most, np.uint8)
    out[:len(proof)] = np.frombuffer(proof, np.uint8)
    return [out, len(proof)]


def _run_proof(s):
    proof, _ = prove_wide_fib(s["job"], *s["inputs"], twiddles=s["twiddles"], stream=s["stream"].cuda_stream,
                              cache=s["cache"])
    return _proof_bytes(s["job"], proof)


def _run_serve(s):
    for k, (job, (a0, a1)) in enumerate(zip(s["jobs"], s["inputs"])):
        s["server"].submit(k, job, a0, a1)
    done = {}
    while len(done) < len(s["jobs"]):
        for r in s["server"].poll():
            if r["status"]:
                raise RuntimeError(f"job {r['job_id']}: {r['error']}")
            done[r["job_id"]] = _proof_bytes(s["jobs"][r["job_id"]], r["proof"])
    return [done[k] for k in range(len(s["jobs"]))]


_RUN = {"trait_commit": _run_trait_commit, "lde": _run_lde, "tree": _run_tree, "quotients": _run_quotients,
        "folds": _run_folds, "inverse": _run_inverse, "oods": _run_oods, "proof": _run_proof, "serve": _run_serve}


def run(state):
    return _RUN[state["op"]](state)


# ----------------------------------------------------------------------------- work
# Operations are counted in the field: a butterfly is a product, a sum and a difference; a product of a base
# value and a QM31 one is four products. A Blake2s compression is 80 G functions of 14 word operations.
_COMPRESSION = 80 * 14


def _lde_work(columns, log, blowup):
    n, m = 1 << log, 1 << (log + blowup)
    return {"bytes": 4 * columns * (2 * n + m), "flops": 3 * columns * (log * n // 2 + log * m // 2)}


def _tree_work(sizes):
    """sizes: {log: columns}. The columns read, every node written; a node hashes its children and its columns."""
    top, nbytes, ops = max(sizes), 0, 0
    for lg in range(top, -1, -1):
        words = sizes.get(lg, 0)
        nbytes += (1 << lg) * (4 * words + 32)
        ops += (1 << lg) * ((lg < top) + -(-words // 16)) * _COMPRESSION
    return {"bytes": nbytes, "flops": ops}


def _proof_work(log, columns, blowup):
    """Inputs, and what has to be in memory for the decommitment: the extended trace and composition columns,
    the quotient column and its folds, and the nodes of their trees."""
    ext, comp = log + blowup, log + 1 + blowup
    parts = [_lde_work(columns, log, blowup), _tree_work({ext: columns}), _lde_work(4, log + 1, blowup),
             _tree_work({comp: 4})]
    parts += [_tree_work({lg: 4}) for lg in range(1, comp + 1)]
    nbytes = 8 * (1 << log) + 4 * columns * (1 << ext) + 16 * (1 << comp) + 32 * (2 << ext) + 96 * (2 << comp)
    return {"bytes": nbytes, "flops": sum(p["flops"] for p in parts)}


def work(case):
    op = case["op"]
    if op == "trait_commit":
        a = _lde_work(case["columns"], case["log"], case["blowup"])
        b = _tree_work({case["log"] + case["blowup"]: case["columns"]})
        return {"bytes": a["bytes"] + 32 * (2 << (case["log"] + case["blowup"])), "flops": a["flops"] + b["flops"]}
    if op == "lde":
        return _lde_work(case["columns"], case["log"], case["blowup"])
    if op == "tree":
        return _tree_work({lg: case["per_size"] for lg in range(case["min_log"], case["max_log"] + 1)})
    if op == "quotients":
        n = 1 << case["log"]
        return {"bytes": n * (4 * case["columns"] + 16), "flops": n * 8 * case["columns"] * case["points"]}
    if op == "folds":
        # every layer read once (sixteen bytes a value) with its inverse twiddles, every folded one written
        n = 1 << case["log"]
        return {"bytes": 16 * (2 * n) + 16 * n + 4 * n, "flops": 40 * n}
    if op == "inverse":
        return {"bytes": case["n"] * (8 if case["field"] == "m31" else 32),
                "flops": case["n"] * (3 if case["field"] == "m31" else 50)}
    if op == "oods":
        n = sum(1 << lg for lg in _mixed_logs(case))
        return {"bytes": 4 * n + 16 * case["columns"], "flops": 8 * n}
    if op == "proof":
        return _proof_work(case["log"], case["columns"], case["blowup"])
    parts = [_proof_work(j.log_n_rows, j.n_columns, j.log_blowup) for j in _served_jobs(case, _shapes_rng(case))]
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


def exact(case, seed):
    """Every output is a whole number of the field, a hash or a proof byte: there is nothing to round."""
    return None
