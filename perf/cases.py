"""The work a user has this framework do, as cases to be timed.

A case goes through the public entry points only: `pixgpu.Chain` (batches
submitted from host records, or from events resident in the device pool), the
standalone fits and the vertex finder of the C ABI.  The events come from the
synthetic detector's calibrated model (ttbar-like: PU50 has about 57k digis,
18k hits and 1.6k loose tracks) or its dense model.
"""
import ctypes
import math
import os
import random
import struct
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "pixeltrack-standalone_b200"))
import pixgpu  # noqa: E402

# fields of a result view after its eight counts: name, type, values per track or per vertex
_TRACK = [("tuple_index", np.uint32, 1), ("track_n_hits", np.uint8, 1), ("quality", np.uint8, 1),
          ("state", np.float32, 5), ("cov", np.float32, 15), ("pt", np.float32, 1), ("eta", np.float32, 1),
          ("chi2", np.float32, 1), ("hits", np.uint32, 5), ("vertex", np.int16, 1)]
_VERTEX = [("zv", np.float32, 1), ("wv", np.float32, 1), ("vchi2", np.float32, 1), ("ptv2", np.float32, 1),
           ("ndof", np.int32, 1), ("sort_ind", np.uint16, 1)]
_FIELDS = [(n, np.dtype(d), k, i < len(_TRACK)) for i, (n, d, k) in enumerate(_TRACK + _VERTEX)]
_VIEW = struct.Struct("8I16Q")
_DETECTOR = []


def _detector():
    """The detector's conditions: the same for every case and seed."""
    if not _DETECTOR:
        _DETECTOR.append(pixgpu.Detector())
    return _DETECTOR[0]


def _chain_case(name, how, events, pu, **more):
    return dict({"name": name, "kind": "chain", "how": how, "events": events, "batch": events, "slots": 1, "pu": pu,
                 "pu_max": pu, "model": "calibrated", "wide": False, "fed_scan": "host", "riemann": False,
                 "mixed": False, "vertex_algo": 0}, **more)


def listed():
    return [
        # one event from its raw record to its tracks: what a trigger node's user waits for
        _chain_case("event_pu50", "submit", 1, 50),
        # a small batch, as continuous batching forms them under load
        _chain_case("batch8_pu50", "submit", 8, 50),
        # the low-pileup sample (PU20) from host records, batches in flight together, FED scan on the device
        _chain_case("stream_pu20", "submit", 93, 20, batch=31, slots=3, fed_scan="device"),
        # the throughput batch on events already on the device, alone
        _chain_case("batch64_pu50", "pool", 64, 50),
        # the same batches in flight together: sustained throughput
        _chain_case("stream_pu50", "pool", 192, 50, batch=64, slots=3),
        # uneven pileup with the wide containers (high-luminosity running)
        _chain_case("uneven_pu20_200", "pool", 12, 20, pu_max=200, wide=True),
        # the dense model (every track prompt) through the Riemann fit and the DBSCAN vertices
        _chain_case("dense_riemann", "pool", 24, 40, model="dense", riemann=True, vertex_algo=1),
        # standalone fits of tuples on the device: a large sample, an event's worth, the precision variant, Riemann
        {"name": "fit_4hit", "kind": "fit", "algo": "broken_line", "hits": 4, "n": 1000000},
        {"name": "fit_3hit_event", "kind": "fit", "algo": "broken_line", "hits": 3, "n": 6007},
        {"name": "fit_3hit_mixed", "kind": "fit", "algo": "broken_line_mixed", "hits": 3, "n": 250000},
        {"name": "fit_4hit_riemann", "kind": "fit", "algo": "riemann", "hits": 4, "n": 200003},
        # the vertex finder alone on one event's tracks, for callers that may not allocate
        {"name": "vertices_pu50", "kind": "vertices", "pu": 50},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what = rng.choice(["submit", "submit", "pool", "pool", "stream", "uneven", "options", "fit", "fit", "vertices"])
    if what == "submit":
        return _unnamed(_chain_case("", "submit", _log_int(rng, 1, 32), rng.randint(10, 60),
                                    fed_scan=rng.choice(["host", "device"])))
    if what == "pool":
        return _unnamed(_chain_case("", "pool", rng.randint(17, 64), rng.randint(20, 55)))
    if what == "stream":
        slots, batch = rng.randint(2, 3), rng.randint(9, 60)
        return _unnamed(_chain_case("", rng.choice(["submit", "pool"]), slots * batch, rng.randint(20, 50),
                                    batch=batch, slots=slots))
    if what == "uneven":
        lo = rng.randint(20, 60)
        return _unnamed(_chain_case("", "pool", rng.randint(2, 12), lo, pu_max=rng.randint(100, 200), wide=True))
    if what == "options":
        return _unnamed(_chain_case("", "pool", rng.randint(4, 24), rng.randint(20, 40), model="dense",
                                    riemann=rng.random() < 0.5, mixed=rng.random() < 0.3,
                                    vertex_algo=rng.randint(0, 2)))
    if what == "fit":
        algo = rng.choice(["broken_line", "broken_line", "broken_line_mixed", "riemann", "riemann_mixed"])
        return {"kind": "fit", "algo": algo, "hits": rng.choice([3, 4]),
                "n": _log_int(rng, 1000, 300000 if algo.startswith("riemann") else 1000000)}
    return {"kind": "vertices", "pu": rng.randint(10, 60)}


def _unnamed(case):
    del case["name"]
    return case


# ------------------------------------------------------------------ inputs
def _events(case, seed, n):
    """n raw records; the pileup of event k is uniform between pu and pu_max."""
    det, rng = _detector(), random.Random(seed)
    pus = [rng.uniform(case["pu"], case.get("pu_max", case["pu"])) for _ in range(n)]
    base = pixgpu.BENCH_SEED_BASE + 1000003 * (seed + 1)
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as ex:
        return list(ex.map(lambda k: det.event(base + k, pus[k], model=case.get("model", "calibrated")), range(n)))


def _prepare_chain(case, seed):
    n, batch = case["events"], case["batch"]
    raws = _events(case, seed, min(n, 64))  # the batches of a longer stream hold the same events in other orders
    order = random.Random(seed + 1)
    words = 400000 if case["wide"] else 160000
    chain = pixgpu.Chain(_detector().es, max_events=batch, max_words_per_batch=batch * words, slots=case["slots"],
                         pool_words=len(raws) * words + 400000 if case["how"] == "pool" else 0,
                         riemann_fit=case["riemann"], mixed_fit=case["mixed"], vertex_algo=case["vertex_algo"],
                         fed_scan=case["fed_scan"], caps=pixgpu.WIDE_CAPS if case["wide"] else None)
    chain.tune_load(os.path.join(pixgpu.PKG, "tuning", "launch_tuning.txt"))
    source = raws
    if case["how"] == "pool":
        source = []
        for r in raws:
            while (h := chain.pool_put(r)) is None:
                pass
            source.append(h)
    batches = []
    for _ in range(case["slots"]):
        batches.append([source[k] for k in (order.sample(range(len(raws)), batch))])
    # places of a view that stay unwritten, because an event has fewer tracks, are zero
    per_pu = 140 if case["model"] == "dense" else 64
    most = (min(16384, per_pu * case["pu_max"] + 256), min(1024, 4 * case["pu_max"] + 64))
    state = {"case": case, "chain": chain, "batches": batches, "held": [], "most": most}
    for slot, (bases, stride) in enumerate(_run_chain(state, _places)):
        for at, (_, d, k, t) in zip(bases, _FIELDS):
            for e in range(batch):
                ctypes.memset(at + e * stride, 0, (16384 if t else 1024) * k * d.itemsize)
    return state


def _prepare_fit(case, seed):
    n, N = case["n"], case["hits"]
    parts = 16 if n >= 16000 else 1
    sizes = [n // parts + (k < n % parts) for k in range(parts)]
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as ex:
        got = list(ex.map(lambda k: pixgpu.fit_tuples(1000003 * (seed + 1) + k, sizes[k], N)[:2], range(parts)))
    hits = torch.from_numpy(np.concatenate([h for h, _ in got])).cuda()
    ge = torch.from_numpy(np.concatenate([g for _, g in got])).cuda()
    out = {"state": (n, 5), "cov": (n, 15), "pt": (n,), "eta": (n,), "chi2": (n,)}
    out = {k: torch.empty(s, dtype=torch.float32, device="cuda") for k, s in out.items()}
    chain = pixgpu.Chain(_detector().es, max_events=1, max_words_per_batch=300000)
    return {"case": case, "chain": chain, "hits": hits, "ge": ge, "out": out}


def _prepare_vertices(case, seed):
    """One event's track SoA, as the chain makes it."""
    chain = pixgpu.Chain(_detector().es, max_events=1, max_words_per_batch=300000)
    chain.process(_events(case, seed, 1))
    got = {k: chain.product(0, k) for k in ("nTuples", "tupleOff", "quality", "pt", "state", "cov")}
    chain.close()
    n = got["nTuples"]

    def up(name, k, dtype):
        return torch.from_numpy(np.ascontiguousarray(got[name].reshape(-1)[:k]).view(dtype)).cuda()

    v = pixgpu.NOALLOC_VERTEX_SLOTS
    ins = [up("tupleOff", n + 1, np.int32), up("quality", n, np.uint8), up("pt", n, np.float32),
           up("state", 5 * n, np.float32), up("cov", 15 * n, np.float32)]
    outs = [torch.zeros(pixgpu.NOALLOC_MAX_TUPLES, dtype=torch.int16, device="cuda")] + \
        [torch.zeros(v, dtype=torch.float32, device="cuda") for _ in range(4)] + \
        [torch.zeros(v, dtype=torch.int32, device="cuda"), torch.zeros(v, dtype=torch.int16, device="cuda")]
    return {"case": case, "ins": ins, "outs": outs}


def prepare(case, seed):
    return {"chain": _prepare_chain, "fit": _prepare_fit, "vertices": _prepare_vertices}[case["kind"]](case, seed)


# ------------------------------------------------------------------ one pass
def _places(state, slot, n):
    """Where the results of the finished batch on `slot` lie: the fields' addresses for event 0, and the distance
    from an event to the next."""
    view = pixgpu.ResultView()
    got = []
    for k in (0, n - 1):
        state["chain"]._check(pixgpu.gpu_lib().pg_result(state["chain"]._h, slot, k, ctypes.byref(view)), "pg_result")
        got.append(_VIEW.unpack(bytes(view))[8:])
    stride = (got[1][0] - got[0][0]) // max(1, n - 1)
    if any(b - a != stride * (n - 1) for a, b in zip(*got)):
        raise RuntimeError("the events' results are not evenly spaced")
    return got[0], stride


def _results(state, slot, n):
    """The results of the finished batch on `slot`, read in place: arrays over [event][track or vertex]."""
    lib, chain, view = pixgpu.gpu_lib(), state["chain"], pixgpu.ResultView()
    counts = np.empty((n, 8), np.uint32)
    for k in range(n):
        chain._check(lib.pg_result(chain._h, slot, k, ctypes.byref(view)), "pg_result")
        counts[k] = _VIEW.unpack_from(view)[:8]
    out = {"counts": counts}
    bases, stride = _places(state, slot, n)
    if counts[:, 0].max() > state["most"][0] or counts[:, 2].max() > state["most"][1]:
        raise RuntimeError("more tracks or vertices than the views show")
    for at, (name, d, k, tracks) in zip(bases, _FIELDS):
        rows = state["most"][0 if tracks else 1]
        whole = (ctypes.c_char * (stride * (n - 1) + rows * k * d.itemsize)).from_address(at)
        whole.chain = chain  # whose memory it is: kept for as long as the arrays are
        out[name] = np.ndarray((n, rows * k), d, whole, strides=(stride, d.itemsize))
    return out


def _run_chain(state, read=_results):
    """Every batch on a slot of its own, in flight together; a batch's results stay in place until the next pass."""
    chain, pooled = state["chain"], state["case"]["how"] == "pool"
    for slot in state["held"]:
        chain.release(slot)
    state["held"] = []
    for b in state["batches"]:
        state["held"].append(chain.submit_pooled(b, keep=True) if pooled else chain.submit(b))
    out = []
    for slot, b in zip(state["held"], state["batches"]):
        chain.wait(slot)
        out.append(read(state, slot, len(b)))
    return out


def _run_fit(state):
    c, o = state["case"], state["out"]
    chain = state["chain"]
    fn = getattr(pixgpu.gpu_lib(), "pg_fit_" + c["algo"])
    chain._check(fn(chain._h, c["hits"], c["n"], state["hits"].data_ptr(), state["ge"].data_ptr(), pixgpu.B_FIELD,
                    o["state"].data_ptr(), o["cov"].data_ptr(), o["pt"].data_ptr(), o["eta"].data_ptr(),
                    o["chi2"].data_ptr(), torch.cuda.current_stream().cuda_stream), "pg_fit_" + c["algo"])
    return o


def _run_vertices(state):
    n, flags = pixgpu.vertices_noalloc(*state["ins"], *state["outs"])
    names = ("zv", "wv", "chi2", "ptv2", "ndof", "sort_ind")
    return dict(zip(names, state["outs"][1:]), idv=state["outs"][0], n=n, flags=flags)


def run(state):
    return {"chain": _run_chain, "fit": _run_fit, "vertices": _run_vertices}[state["case"]["kind"]](state)


def work(case):
    """Inputs read once and outputs written once: FED words with their FED bytes, and the stored tracks."""
    if case["kind"] == "fit":
        n, N = case["n"], case["hits"]
        # counted from the algorithm: the fast fit, two band matrices and their inverses, the covariances
        return {"bytes": n * (48 * N + 92), "flops": n * (1900 if N == 4 else 1200)}
    pu = (case["pu"] + case.get("pu_max", case["pu"])) / 2
    if case["kind"] == "vertices":
        return {"bytes": 212 * pu * (8 + 4 + 1 + 12 + 2), "flops": 0}
    dense = case["model"] == "dense"
    return {"bytes": case["events"] * pu * ((1220 if dense else 1140) * 4.5 + (70 if dense else 32) * 120), "flops": 0}


# ------------------------------------------------------------------ the fits in 64 bits
def exact(case, seed):
    """The broken-line fit in plain double precision (fits: its mixed variant too); the chain's cuts, graph search
    and vertexing, and the Riemann fit with its single-precision eigenvectors, have no such value here."""
    if case["kind"] != "fit" or not case["algo"].startswith("broken_line"):
        return None
    s = _prepare_fit(case, seed)
    parts = [_broken_line(s["hits"][k:k + 125000], s["ge"][k:k + 125000].double())
             for k in range(0, case["n"], 125000)]
    return {k: torch.cat([p[k] for p in parts]) for k in parts[0]}


def _broken_line(x, ge):
    """x[n, N, 3], ge[n, N, 6]: the two-step broken-line fit (reference circle, s-z line, circle) in float64."""
    B, N = pixgpu.B_FIELD, x.shape[1]
    X, Y, Zh = x[..., 0], x[..., 1], x[..., 2]
    cross = lambda ax, ay, bx, by: ax * by - ay * bx  # noqa: E731
    m = N // 2
    ax, ay, bx, by = X[:, m] - X[:, 0], Y[:, m] - Y[:, 0], X[:, -1] - X[:, m], Y[:, -1] - Y[:, m]
    cx, cy = X[:, 0] - X[:, -1], Y[:, 0] - Y[:, -1]
    half, a2, c2 = 0.5 / cross(cx, cy, ax, ay), ax * ax + ay * ay, cx * cx + cy * cy
    x0, y0 = X[:, 0] - (ay * c2 + cy * a2) * half, Y[:, 0] + (ax * c2 + cx * a2) * half
    rho = torch.sqrt(a2 * (bx * bx + by * by) * c2) / (2 * cross(bx, by, ax, ay).abs())
    rx, ry = X - x0[:, None], Y - y0[:, None]
    turn = torch.atan2(cross(rx[:, 0], ry[:, 0], rx[:, -1], ry[:, -1]), rx[:, 0] * rx[:, -1] + ry[:, 0] * ry[:, -1])
    q = torch.where(cross(X[:, 1] - X[:, 0], Y[:, 1] - Y[:, 0], X[:, -1] - X[:, -2], Y[:, -1] - Y[:, -2]) > 0, -1., 1.)
    q = q.double()
    slope = -q * (Zh[:, -1] - Zh[:, 0]) / (rho * turn)
    cs = 1 / torch.sqrt(1 + slope ** 2)
    sn = slope * cs
    centre = torch.sqrt(x0 * x0 + y0 * y0)
    px, py = (-rho * x0 / centre)[:, None], (-rho * y0 / centre)[:, None]
    s = (q * rho)[:, None] * torch.atan2(cross(rx, ry, px, py), rx * px + ry * py)
    S, Z = cs[:, None] * s + sn[:, None] * Zh, -sn[:, None] * s + cs[:, None] * Zh

    def scatter(length):  # variance of the multiple-scattering angle over `length` of detector
        t = length.abs() * (0.06 / 16)
        return 0.7 * (13.6e-3) ** 2 / ((B * rho).clamp(max=20) ** 2 * (1 + slope ** 2)) * t * (1 + 0.038 * t.log()) ** 2

    var = [scatter(S[:, i + 1] - S[:, i]) + scatter(S[:, i] - S[:, i - 1]) for i in range(1, N - 1)]

    def kinks(t, w, v, bend):
        """Normal matrix of hits (weights w) and kinks (variances v): the kink at i is row @ u, u the offsets
        (and, with bend, the curvature correction)."""
        A = torch.diag_embed(torch.cat([w, torch.zeros_like(w[:, :1])], 1) if bend else w)
        rows = []
        for i in range(1, N - 1):
            d0, d1 = t[:, i] - t[:, i - 1], t[:, i + 1] - t[:, i]
            row = torch.zeros_like(A[:, 0])
            row[:, i - 1], row[:, i], row[:, i + 1] = 1 / d0, -(1 / d0 + 1 / d1), 1 / d1
            if bend:
                row[:, N] = (d0 + d1) / 2
            A = A + row[:, :, None] * row[:, None, :] / v[i - 1][:, None, None]
            rows.append(row)
        return A, rows

    def solve(t, w, v, meas, bend):
        A, rows = kinks(t, w, v, bend)
        scale = A.diagonal(dim1=1, dim2=2).sqrt()  # equilibrated: the offsets' and the curvature's units differ
        inv = torch.linalg.inv(A / (scale[:, :, None] * scale[:, None, :])) / (scale[:, :, None] * scale[:, None, :])
        rhs = w * meas
        u = (inv[:, :, :N] * rhs[:, None, :]).sum(2)
        chi2 = (w * (meas - u[:, :N]) ** 2).sum(1)
        for row, vi in zip(rows, v):
            chi2 = chi2 + (row * u).sum(1) ** 2 / vi
        return inv, u, chi2

    # s-z line
    r = torch.sqrt(rx * rx + ry * ry)
    jx, jy = ry / r, -rx / r
    vtt = jx * jx * ge[..., 0] + 2 * jx * jy * ge[..., 1] + jy * jy * ge[..., 2]
    vtz = jx * ge[..., 3] + jy * ge[..., 4]
    c_, s_ = cs[:, None], sn[:, None]
    w = 1 / (s_ * s_ * vtt - 2 * s_ * c_ * vtz + c_ * c_ * ge[..., 5])
    I, u, lchi2 = solve(S, w, var, Z, False)
    d = 1 / (S[:, 1] - S[:, 0])
    l0, l1 = (u[:, 1] - u[:, 0]) * d, u[:, 0]
    L = torch.stack([(I[:, 0, 0] - 2 * I[:, 0, 1] + I[:, 1, 1]) * d * d + scatter(S[:, 1] - S[:, 0]),
                     (I[:, 0, 1] - I[:, 0, 0]) * d, (I[:, 0, 1] - I[:, 0, 0]) * d, I[:, 0, 0]], 1).reshape(-1, 2, 2)
    zero, one = torch.zeros_like(l0), torch.ones_like(l0)

    def carried(J, C):
        J = torch.stack([torch.stack(row, 1) for row in J], 1)
        return J @ C @ J.transpose(1, 2)

    L = carried([[one, zero], [-S[:, 0], one]], L)
    l1 = l1 - l0 * S[:, 0]
    k = 1 / (cs - l0 * sn)
    L = carried([[k * k, zero], [l1 * sn * k * k, k]], L)
    l1, l0 = l1 * k, (sn + l0 * cs) * k
    # circle
    var = [v * (1 + slope ** 2) for v in var]
    meas = r - rho[:, None]
    ux, uy = rx / r, ry / r
    w = 1 / (ux * ux * ge[..., 0] + 2 * ux * uy * ge[..., 1] + uy * uy * ge[..., 2])
    I, u, cchi2 = solve(s, w, var, meas, True)
    dx, dy = X[:, 0] + (u[:, 0] - meas[:, 0]) * ux[:, 0], Y[:, 0] + (u[:, 0] - meas[:, 0]) * uy[:, 0]
    ex, ey = X[:, 1] + (u[:, 1] - meas[:, 1]) * ux[:, 1], Y[:, 1] + (u[:, 1] - meas[:, 1]) * uy[:, 1]
    fx, fy = ex - dx, ey - dy
    f2 = fx * fx + fy * fy
    par = [torch.atan2(fy, fx), -q * (0.25 * f2) / (rho + torch.sqrt(rho ** 2 - 0.25 * f2)), q * (1 / rho + u[:, N])]
    side = torch.sqrt((2 * rho) ** 2 - f2)
    J = [[(uy[:, 0] * fx - fy * ux[:, 0]) / f2, (uy[:, 1] * fx - fy * ux[:, 1]) / f2, zero],
         [q / 2 * (fx * ux[:, 0] + fy * uy[:, 0]) / side, q / 2 * (fx * ux[:, 1] + fy * uy[:, 1]) / side, zero],
         [zero, zero, q]]
    pick = torch.tensor([0, 1, N], device=x.device)
    C = carried(J, I[:, pick][:, :, pick])

    def moved(par, C, tx, ty):  # the circle's parameters about another point
        phi, dca, kap = par
        s0, c0 = torch.sin(phi), torch.cos(phi)
        dp, do, uu = tx * c0 + ty * s0, tx * s0 - ty * c0 + dca, 1 + kap * dca
        cc, bb = -kap * ty + uu * c0, kap * tx + uu * s0
        A = 2 * do + kap * (do ** 2 + dp ** 2)
        U = torch.sqrt(1 + kap * A)
        xi, v, lam = 1 / (bb ** 2 + cc ** 2), 1 + kap * do, 0.5 * A / (U * (1 + U) ** 2)
        mu, zeta = 1 / (U * (1 + U)) + kap * lam, do ** 2 + dp ** 2
        J = [[xi * uu * v, -xi * kap ** 2 * dp, xi * dp], [2 * mu * uu * dp, 2 * mu * v, mu * zeta - lam * A],
             [zero, zero, one]]
        return [torch.atan2(bb, cc), A / (1 + U), kap], carried(J, C)

    par, C = moved(par, C, 0.5 * fx, 0.5 * fy)
    C[:, 0, 0] += (1 + slope ** 2) * scatter(S[:, 1] - S[:, 0])
    par, C = moved(par, C, dx, dy)
    cov = torch.zeros(len(x), 15, dtype=torch.float64, device=x.device)
    for at, v in ((0, C[:, 0, 0]), (1, C[:, 0, 1]), (2, C[:, 0, 2] / B), (5, C[:, 1, 1]), (6, C[:, 1, 2] / B),
                  (9, C[:, 2, 2] / B ** 2), (12, L[:, 0, 0]), (13, L[:, 0, 1]), (14, L[:, 1, 1])):
        cov[:, at] = v
    return {"state": torch.stack([par[0], par[1], par[2] / B, l0, l1], 1), "cov": cov, "pt": B / par[2].abs(),
            "eta": torch.asinh(l0), "chi2": (cchi2 + lchi2) / (2 * N - 5)}
