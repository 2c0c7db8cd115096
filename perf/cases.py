"""The work users have this library do, as measured cases.

Every case goes through the public entry points of ``lpgpu`` (the ctypes
binding of ``include/lpgpu.h``) on hypergraphs of the shapes this repository's
generators, tests and benchmark use (``mt-kahypar_gb300/lpgpu/gen.py``), drawn
on the GPU so that new inputs are quick to make. A case is one of these calls:

* ``refine``    restore the start partition of a resident hypergraph, refine it,
                download the partition (a refiner called on a session it keeps)
* ``level``     upload + set_partition + refine + download from page-locked host
                buffers (one level of a multilevel partitioner, one request of
                a server, the benchmark's end-to-end step)
* ``oneshot``   ``lpgpu_refine_km1`` on ordinary host arrays
* ``batch``     many small hypergraphs: upload_instances +
                set_partition_instances + refine + download
* ``stepped``   a server's running set: set_partition + begin_rounds of every
                session, one stepper round at a time until all are done,
                end_rounds + download
* ``rebalance`` set_partition of an overloaded partition + rebalance + download
* ``query``     set_partition + best_moves + block weights + km1 / cut / imbalance

Shapes: ``geom`` (geometric net sizes, pins in a +-512 window, unit weights),
``zipf`` (Zipf 2.2 net sizes up to 4,096, 80 % of pins in a +-4,096 window and
20 % uniform, weighted) and ``rownet`` (power-law nets up to 8,192, half of the
pins in a +-16,384 band, unit weights, contiguous blocks with 10 % of the
vertices reassigned).
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (ROOT, os.path.join(ROOT, "mt-kahypar_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

EPS = 0.03
WINDOW = {"geom": 512, "zipf": 4096, "rownet": 16384}
UNIFORM = {"geom": 0.0, "zipf": 0.2, "rownet": 0.5}
NETS_PER_VERTEX = {"geom": 1.1, "zipf": 1.2, "rownet": 1.0}


# ------------------------------------------------------------------- cases

def _case(name, call, shape, n, k, rounds, **more):
    c = {"call": call, "shape": shape, "n": n, "k": k, "rounds": rounds, "rebalancing": 1, "revert": 1,
         "threshold": 100, "instances": 1}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest request the batched and served workloads draw: launches and latency
        _case("refine_1k", "refine", "geom", 1024, 2, 5),
        # the small plain workload (16,384 vertices, k = 2)
        _case("refine_16k", "refine", "geom", 16384, 2, 5),
        # an ordinary served request, odd size, most blocks the persistent form takes
        _case("refine_zipf_131k", "refine", "zipf", 131071, 64, 8),
        # the large plain workload (1M vertices, weighted, k = 32)
        _case("refine_zipf_1m", "refine", "zipf", 1048576, 32, 10),
        # the row-net workload (4.2M vertices, 33.5M pins, k = 128): the benchmark's headline
        _case("refine_rownet_4m", "refine", "rownet", 4194304, 128, 10),
        # many blocks (k above 128 takes the warp-window sweep), border vertices only
        _case("refine_geom_250k_k300", "refine", "geom", 250007, 300, 5, rebalancing=0),
        # one level of a multilevel run, host buffers to host buffers
        _case("level_zipf_400k", "level", "zipf", 399989, 16, 8),
        # one-shot call on ordinary arrays, as an FFI user makes it
        _case("oneshot_geom_10k", "oneshot", "geom", 10007, 8, 5),
        # the batched workload (1,024 to 65,536 vertices, k in {2, 4, 8, 16}), end to end
        _case("batch_1280", "batch", "geom", 65536, 16, 5, instances=1280),
        # a server's running set of small requests, round by round
        _case("stepped_24", "stepped", "zipf", 32768, 64, 8, instances=24),
        # an overloaded partition made feasible again
        _case("rebalance_zipf_200k", "rebalance", "zipf", 200003, 32, 16),
        # gains and metrics of a partition, as a driver or a test asks for them
        _case("query_zipf_500k", "query", "zipf", 500009, 32, 0),
    ]


def _log_int(rng, lo, hi):
    x = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, x))


def draw(rng):
    call = rng.choice(["refine", "refine", "refine", "refine", "level", "level", "oneshot", "batch", "stepped",
                       "rebalance", "query"])
    shape = rng.choice(["geom", "zipf", "zipf", "rownet"])
    if call == "batch":
        inst = _log_int(rng, 16, 1280)
        return _case(None, call, "geom", _log_int(rng, 4096, 65536), rng.choice([2, 4, 8, 16]), 5, instances=inst)
    if call == "stepped":
        return _case(None, call, rng.choice(["geom", "zipf"]), _log_int(rng, 4096, 65536),
                     rng.choice([2, 4, 8, 16, 32, 64]), rng.randint(5, 8), instances=_log_int(rng, 4, 48))
    if call == "oneshot":
        n, k = _log_int(rng, 1024, 131072), rng.choice([2, 4, 8, 16, 32, 64])
    elif call == "rebalance":
        n, k = _log_int(rng, 4096, 1048576), rng.choice([2, 4, 8, 16, 32, 64])
    else:
        n, k = _log_int(rng, 1024, 2097152), rng.choice([2, 3, 8, 16, 32, 61, 64, 128])
        if call == "refine" and n >= 16384 and rng.random() < 0.2:
            k, n = rng.randint(129, 600), min(n, 524288)
    k = min(k, max(2, n // 16))
    if call == "refine":
        return _case(None, call, shape, n, k, rng.randint(5, 10), rebalancing=rng.choice([1, 1, 0]),
                     revert=rng.choice([1, 1, 1, 0]), threshold=rng.choice([100, 100, 0]))
    rounds = {"rebalance": 16, "query": 0}.get(call, rng.randint(5, 8))
    return _case(None, call, shape, n, k, rounds)


# --------------------------------------------------------- inputs from the seed

def _table(shape, m, lo_hi=None):
    """Net-size distribution (sizes, probabilities)."""
    if shape == "geom":
        lo, hi = 2, 256
        d = np.arange(1, hi + 1, dtype=np.float64)
        p = 0.75 ** (d - 1) * 0.25      # geometric of mean 4 ...
        p[-1] = 0.75 ** (hi - 1)
        p[lo - 1] += p[:lo - 1].sum()   # ... clipped to [2, 256]
        return d[lo - 1:], p[lo - 1:]
    lo, hi, alpha = (2, 4096, 2.2) if shape == "zipf" else (1, 8192, 1.919)
    d = np.arange(lo, hi + 1, dtype=np.float64)
    p = d ** -alpha
    return d, p / p.sum()


def _mean_size(shape):
    d, p = _table(shape, 0)
    return float((d * p).sum() / p.sum())


def _sizes(case):
    """Vertex counts of the case's instances (the same for every seed) and their k."""
    if case["instances"] == 1:
        return [case["n"]], [case["k"]]
    rng = np.random.default_rng(case["instances"] * 1000003 + case["n"])
    ns = np.exp(rng.uniform(math.log(1024), math.log(max(1025, case["n"])), case["instances"])).round().astype(int)
    ks = [k for k in (2, 4, 8, 16, 32, 64) if k <= case["k"]]
    return ns.tolist(), rng.choice(ks, case["instances"]).tolist()


def _generate(case, seed, device="cuda"):
    """CSR arrays of the case's instances side by side (vertex ids local to
    each instance), weights and start partitions, as CUDA tensors."""
    g = torch.Generator(device=device)
    g.manual_seed(1 + 7919 * int(seed))
    shape = case["shape"]
    ns, ks = _sizes(case)
    ms = [max(1, int(round(NETS_PER_VERTEX[shape] * x))) for x in ns]
    n_t = torch.tensor(ns, device=device)
    m_t = torch.tensor(ms, device=device)
    M = sum(ms)
    d, p = _table(shape, M)
    cdf = torch.from_numpy(np.cumsum(p) / p.sum()).to(device)
    inst = torch.repeat_interleave(torch.arange(len(ns), device=device), m_t)
    n_of = n_t[inst]
    size = int(d[0]) + torch.searchsorted(cdf, torch.rand(M, generator=g, device=device, dtype=torch.float64))
    size = torch.minimum(size.clamp_(max=int(d[-1])), n_of)
    net = torch.repeat_interleave(torch.arange(M, device=device), size)
    if shape == "rownet":  # row r sits on the diagonal
        first = torch.cumsum(m_t, 0) - m_t
        anchor = (torch.arange(M, device=device) - first[inst]) * n_of // m_t[inst]
    else:
        anchor = (torch.rand(M, generator=g, device=device, dtype=torch.float64) * n_of).long()
    n_pin = n_of[net]
    w = (n_pin // 2).clamp_(max=WINDOW[shape])
    pin = anchor[net] - w + (torch.rand(net.shape, generator=g, device=device, dtype=torch.float64) * (2 * w + 1)).long()
    if UNIFORM[shape] > 0:
        far = torch.rand(net.shape, generator=g, device=device) < UNIFORM[shape]
        pin = torch.where(far, (torch.rand(net.shape, generator=g, device=device, dtype=torch.float64) * n_pin).long(),
                          pin)
        del far
    pin = torch.minimum(pin.clamp_(min=0), n_pin - 1)
    stride = max(ns)
    key = torch.unique(net * stride + pin)  # sorted, duplicate pins of a net removed
    del net, pin, n_pin, w
    if shape != "rownet":  # a net that lost all but one pin gets a neighbour
        cnt = torch.bincount(key // stride, minlength=M)
        lone = key[cnt[key // stride] == 1]
        e, v = lone // stride, lone % stride
        key = torch.sort(torch.cat([key, e * stride + (v + 1) % n_of[e]]))[0]
    cnt = torch.bincount(key // stride, minlength=M)
    pins = (key % stride).int()
    off = torch.zeros(M + 1, dtype=torch.int64, device=device)
    torch.cumsum(cnt, 0, out=off[1:])
    N = sum(ns)
    if shape == "zipf":
        w_v = torch.randint(1, 5, (N,), generator=g, device=device, dtype=torch.int32)
        w_e = torch.randint(1, 9, (M,), generator=g, device=device, dtype=torch.int32)
    else:
        w_v = torch.ones(N, dtype=torch.int32, device=device)
        w_e = torch.ones(M, dtype=torch.int32, device=device)
    parts = []
    for x, k in zip(ns, ks):
        if case["call"] == "rebalance":  # a quarter of the vertices crowd into every fourth block
            b = torch.randperm(x, generator=g, device=device) % k
            crowd = torch.rand(x, generator=g, device=device) < 0.25
            b = torch.where(crowd, b // 4 * 4, b)
        elif shape == "rownet":
            b = torch.arange(x, device=device) * k // x
            moved = torch.rand(x, generator=g, device=device) < 0.1
            b = torch.where(moved, torch.randint(0, k, (x,), generator=g, device=device), b)
        else:
            b = torch.randperm(x, generator=g, device=device) % k
        parts.append(b.int())
    return {"ns": ns, "ms": ms, "ks": ks, "off": off, "pins": pins, "w_v": w_v, "w_e": w_e, "part": torch.cat(parts)}


def _pinned(t):
    """Page-locked host copy; the array keeps its memory alive."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def prepare(case, seed):
    import lpgpu
    from lpgpu.gen import Hypergraph

    g = _generate(case, seed)
    call = case["call"]
    keep = (lambda t: t.cpu().numpy()) if call == "oneshot" else _pinned
    off, pins, w_v, w_e, part = (keep(g[x]) for x in ("off", "pins", "w_v", "w_e", "part"))
    out = _pinned(torch.zeros_like(g["part"]))
    hgs, parts, outs = [], [], []
    v0 = e0 = 0
    local = off
    if len(g["ns"]) > 1:  # every instance's offsets from 0, with the closing entry
        first = torch.cumsum(torch.tensor([0] + g["ms"]), 0)
        inst = torch.repeat_interleave(torch.arange(len(g["ms"])), torch.tensor(g["ms"]) + 1)
        at = torch.arange(len(inst)) - inst
        o = torch.from_numpy(off)
        local = _pinned(o[at] - o[first[inst]])
    for i, (n, m) in enumerate(zip(g["ns"], g["ms"])):
        o = local[e0 + i:e0 + i + m + 1]
        hgs.append(Hypergraph(n, m, o, pins[off[e0]:off[e0 + m]], w_v[v0:v0 + n], w_e[e0:e0 + m]))
        parts.append(part[v0:v0 + n])
        outs.append(out[v0:v0 + n])
        v0, e0 = v0 + n, e0 + m
    cfg = lpgpu.default_config(rounds=case["rounds"], rebalancing=case["rebalancing"], revert=case["revert"],
                               activation_threshold=case["threshold"])
    st = {"case": case, "cfg": cfg, "hgs": hgs, "parts": parts, "outs": outs, "out": out, "ks": g["ks"]}
    if call in ("refine", "query", "rebalance"):
        s = lpgpu.Session()
        s.upload(hgs[0])
        s.set_partition(case["k"], parts[0], eps=EPS)
        if call == "refine":
            s.save_partition()
        st["s"] = s
    elif call in ("level", "batch"):
        st["s"] = lpgpu.Session()
    elif call == "stepped":
        st["sessions"] = [lpgpu.Session().upload(h) for h in hgs]
        st["stepper"] = lpgpu.Stepper()
    return st


# ---------------------------------------------------------------- one pass

def _download(s, out):
    """lpgpu_session_get_partition into the caller's buffer."""
    import lpgpu
    status = lpgpu.lib().lpgpu_session_get_partition(s._h, out.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)))
    if status != lpgpu.OK:
        raise RuntimeError("get_partition failed with status %d" % status)
    return out


def _result(r):
    d = r.as_dict()
    return {x: d[x] for x in ("km1_before", "km1_after", "delta", "moves", "pins_processed", "rounds", "imbalance")}


def run(state):
    import lpgpu

    case, cfg = state["case"], state["cfg"]
    call, k = case["call"], case["k"]
    if call == "refine":
        s = state["s"]
        s.restore_partition()
        r = _result(s.refine(cfg))
        return {"partition": _download(s, state["out"]), **r}
    if call == "level":
        s = state["s"]
        s.upload(state["hgs"][0])
        s.set_partition(k, state["parts"][0], eps=EPS)
        r = _result(s.refine(cfg))
        return {"partition": _download(s, state["out"]), **r}
    if call == "oneshot":
        part, r = lpgpu.refine_km1(state["hgs"][0], k, state["parts"][0], eps=EPS, cfg=cfg)
        return {"partition": part, **_result(r)}
    if call == "batch":
        s = state["s"]
        s.upload_instances(state["hgs"])
        s.set_partition_instances(state["ks"], state["parts"], eps=EPS)
        r = _result(s.refine(cfg))
        s.partition_instances(state["outs"])
        return {"partition": state["out"], "instance_km1": s.instance_km1(), **r}
    if call == "stepped":
        sessions = state["sessions"]
        for s, kk, p in zip(sessions, state["ks"], state["parts"]):
            s.set_partition(kk, p, eps=EPS)
            s.begin_rounds(cfg)
        running = list(range(len(sessions)))
        while running:
            done = state["stepper"].round([sessions[i] for i in running])
            running = [i for i, d in zip(running, done) if not d]
        km1 = np.zeros(len(sessions), np.int64)
        for i, s in enumerate(sessions):
            km1[i] = s.end_rounds().km1_after
            _download(s, state["outs"][i])
        return {"partition": state["out"], "km1_after": km1}
    if call == "rebalance":
        s = state["s"]
        s.set_partition(k, state["parts"][0], eps=EPS)
        r = _result(s.rebalance(case["rounds"]))
        return {"partition": _download(s, state["out"]), **r}
    s = state["s"]  # query
    s.set_partition(k, state["parts"][0], eps=EPS)
    to, gain, border = s.best_moves()
    km1, cut, imbalance = s.metrics()
    return {"to": to, "gain": gain, "border": border, "block_weights": s.block_weights(), "km1": km1, "cut": cut,
            "imbalance": imbalance}


def work(case):
    """Bytes: net offsets, pins, weights and the partition read once, the
    outputs written once. The arithmetic is integer: no flops."""
    ns, _ = _sizes(case)
    n = sum(ns)
    m = sum(max(1, int(round(NETS_PER_VERTEX[case["shape"]] * x))) for x in ns)
    pins = m * _mean_size(case["shape"])
    read = 8 * (m + 1) + 4 * pins + 4 * m + 4 * n + 4 * n
    written = 9 * n if case["call"] == "query" else 4 * n
    return {"bytes": float(read + written), "flops": 0.0}


# ------------------------------------------------- 64-bit values of the outputs

def _km1_cut(off, pins, part, w_e, k):
    m = len(off) - 1
    net = torch.repeat_interleave(torch.arange(m, device=off.device), off[1:] - off[:-1])
    lam = torch.bincount(torch.unique(net * k + part[pins.long()].long()) // k, minlength=m)
    return int(((lam - 1).clamp(min=0) * w_e.long()).sum()), int(((lam > 1) * w_e.long()).sum())


def exact(case, seed):
    if case["instances"] > 1:
        return None
    g = _generate(case, seed)
    n, k = case["n"], case["k"]
    off, pins, part, w_e, w_v = g["off"], g["pins"], g["part"], g["w_e"], g["w_v"]
    km1, cut = _km1_cut(off, pins, part, w_e, k)
    if case["call"] != "query":  # the start's objective; the refined state follows the library's own rules
        return {"partition": None, "km1_before": km1, "km1_after": None, "delta": None, "moves": None,
                "pins_processed": None, "rounds": None, "imbalance": None}
    # best move of every vertex from dense pin counts, in slices of vertices
    m = len(off) - 1
    net = torch.repeat_interleave(torch.arange(m, device=off.device), off[1:] - off[:-1])
    v = pins.long()
    bw = torch.bincount(part.long(), weights=w_v.double(), minlength=k).long()
    perfect = math.ceil(int(w_v.long().sum()) / float(k))
    lmax = int((1.0 + EPS) * float(perfect))
    phi = torch.bincount(net * k + part[v].long(), minlength=m * k).view(m, k)
    internal = torch.zeros(n, dtype=torch.int64, device=off.device)
    many = phi[net, part[v].long()] > 1
    internal.index_add_(0, v, w_e.long()[net] * many)
    border = torch.zeros(n, dtype=torch.int64, device=off.device)
    border.index_add_(0, v, ((phi > 0).sum(1) > 1).long()[net])
    pen = torch.zeros(n, k, dtype=torch.int64, device=off.device)
    for a in range(0, len(v), 1 << 22):
        s = slice(a, a + (1 << 22))
        pen.index_add_(0, v[s], (phi[net[s]] > 0) * w_e.long()[net[s]][:, None])
    blocked = (bw[None, :] + w_v.long()[:, None] > lmax)
    blocked[torch.arange(n, device=off.device), part.long()] = True
    pen[blocked] = -1
    best = pen.max(1)[0]
    to = (pen == best[:, None]).int().argmax(1)  # lowest block of the largest penalty
    # vertices above 100,000 incident nets are never border vertices
    border = (border > 0) & (torch.bincount(v, minlength=n) <= 100000)
    move = border & (best > internal)
    to = torch.where(move, to, part.long())
    gain = torch.where(move, internal - best, torch.zeros_like(best))
    return {"to": to.cpu().numpy(), "gain": gain.cpu().numpy(), "border": border.cpu().numpy(),
            "block_weights": bw.cpu().numpy(), "km1": km1, "cut": cut,
            "imbalance": float(bw.max()) / perfect - 1.0}
