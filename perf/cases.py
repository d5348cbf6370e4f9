"""The framework's work as a set of timed cases.

A case is a dict of plain values; ``kind`` names the call and the rest its sizes.
:func:`listed` are the cases to watch, :func:`draw` gives more of the same ranges,
:func:`prepare` makes what a program has in hand before the call (its kept code object
and new inputs), :func:`run` is one call through the public entry points, :func:`work` the
bytes and operations the call cannot do without, and :func:`exact` the same outputs in 64
bits from plain torch, where the outputs are computed numbers that such a restatement
reaches in reasonable time.
"""

import ctypes as C
import functools
import importlib
import math
import os

import numpy as np
import torch

cb = importlib.import_module("com-rs_gb300")

HERE = os.path.dirname(os.path.abspath(__file__))
WEIGHTS = os.path.join(os.path.dirname(HERE), "com-rs_gb300", "weights")

# (base graph, Z) of the f32 codes: the benchmark codes and liftings of the uneven mix
F32_LIFTINGS = ((1, 384), (2, 52), (1, 208), (2, 128))
RATES = ((1, 3), (1, 2), (2, 3), (5, 6))
# the Eb/N0 above which frames of a modulation and rate begin to decode, roughly
WATERFALL = {4: 1.5, 16: 4.0, 64: 7.0, 256: 10.5}
RATE_DB = {(1, 3): -1.0, (1, 2): 0.0, (2, 3): 1.2, (5, 6): 2.8}


def listed():
    return [
        # a receiver's latency: one large codeword in device memory, soft output wanted
        dict(name="decode_one", kind="decode", bg=1, z=384, k=8448, e=25344, n=1, margin=0.6, rate="1/3"),
        # the headline Monte Carlo trial: BG1 Z = 384, 16-QAM, one launch's batch in f32
        dict(name="trial_bg1_f32", kind="trial", precision="f32", bg=1, z=384, k=8448, e=25344, m=16, n=8192, ebn0=2.7),
        # the small reference-exact trial: BG2 Z = 52, QPSK, f64 (the default precision)
        dict(name="trial_bg2_f64", kind="trial", precision="f64", bg=2, z=52, k=520, e=1040, m=4, n=4096, ebn0=1.5),
        # the f64 drop-in decoder on host arrays, an odd block size with a redundancy
        # version and the bit interleaver (a retransmission of a transport block)
        dict(name="decode_host_f64", kind="decode_host", k=3001, e=6004, rv=3, qm=4, n=96, sigma=0.66),
        # the transmitter's side: blocks of the large code encoded from host bits
        dict(name="encode_bg1", kind="encode", bg=1, z=384, k=8448, e=25344, rv=0, qm=1, n=128),
        # the uneven batch: 16384 codewords of both base graphs, six liftings, four rates
        # and modulations in one replayed graph
        dict(name="mix", kind="mix", n=16384, draw=2024),
        # the learned decoder at its operating point: BG1 Z = 384, 64-QAM, 8 iterations
        dict(name="learned_bg1", kind="learned", protocol="c5", n=4096, ebn0=6.97),
        # gradients of a network on BG2 Z = 52 from a program's own frames (host arrays)
        dict(name="gradients_bg2", kind="gradients", bg=2, z=52, k=520, e=1040, n=1024, iterations=10, shared=True,
             multi=1, sigma=0.85),
        # one training step of the network at scale: BG1 Z = 384, 64-QAM, 8 iterations
        dict(name="train_bg1", kind="train", protocol="c5", n=512),
        # a generic code with its default decoder: PEG(576, 288), f64 layered sum-product
        dict(name="peg_f64", kind="sparse", code="peg", size=576, info=288, precision="f64", rule="sum_product",
             layered=True, iterations=50, n=2000, sigma=0.72),
        # a long standard code, f32: DVB-S2 short frames, rate 1/2, layered sum-product
        dict(name="dvbs2_f32", kind="sparse", code="dvbs2", size=16200, info=7200, precision="f32", rule="sum_product",
             layered=True, iterations=50, n=152, sigma=0.80),
        # trials of a specification's link: 8 blocks of PEG(1024, 512), 16-QAM, interleaved
        dict(name="link", kind="link", size=1024, info=512, blocks=8, m=16, n=512, ebn0=4.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _f32_code(rng):
    bg, z = rng.choice(F32_LIFTINGS)
    k = (22 if bg == 1 else 10) * z
    rate = rng.choice(RATES)
    # an odd number of sent bits now and then, within the circular buffer
    e = min(-(-k * rate[1] // rate[0]) + rng.choice((0, 0, 1, 3)), (66 if bg == 1 else 50) * z)
    return bg, z, k, e, rate


def draw(rng):
    kind = rng.choice(("decode", "trial", "trial64", "decode_host", "encode", "mix", "learned", "gradients", "train",
                       "sparse", "dvbs2", "link"))
    if kind == "decode":
        bg, z, k, e, rate = _f32_code(rng)
        return dict(kind="decode", bg=bg, z=z, k=k, e=e, n=_log_int(rng, 1, 600), margin=round(rng.uniform(0.2, 1.5), 2),
                    rate=f"{rate[0]}/{rate[1]}")
    if kind == "trial":
        bg, z, k, e, rate = _f32_code(rng)
        m = rng.choice((4, 16, 64, 256))
        return dict(kind="trial", precision="f32", bg=bg, z=z, k=k, e=e, m=m, n=_log_int(rng, 32, 8000),
                    ebn0=round(WATERFALL[m] + RATE_DB[rate] + rng.uniform(-0.5, 1.5), 2))
    if kind == "trial64":
        z = rng.choice((20, 36, 52, 104, 176))
        k = 10 * z - rng.choice((0, 0, 7))
        rate = rng.choice(RATES)
        m = rng.choice((4, 16, 64))
        return dict(kind="trial", precision="f64", bg=2, z=z, k=k, e=min(k * rate[1] // rate[0], 50 * z), m=m,
                    n=_log_int(rng, 32, 4096 * 52 // max(z, 52)),
                    ebn0=round(WATERFALL[m] + RATE_DB[rate] + rng.uniform(-0.5, 1.5), 2))
    if kind == "decode_host":
        k = _log_int(rng, 100, 8448)
        qm = rng.choice((1, 2, 4, 6))
        e = -(-int(k * rng.uniform(1.6, 3.2)) // qm) * qm
        return dict(kind="decode_host", k=k, e=e, rv=rng.choice((0, 0, 3)), qm=qm,
                    n=_log_int(rng, 1, max(2, 96 * 3001 // k)), sigma=round(rng.uniform(0.55, 0.75), 3))
    if kind == "encode":
        bg, z, k, e, _ = _f32_code(rng)
        if rng.random() < 0.5:
            k -= rng.randrange(1, z)
        return dict(kind="encode", bg=bg, z=z, k=k, e=e, rv=0, qm=1, n=_log_int(rng, 1, 128))
    if kind == "mix":
        return dict(kind="mix", n=_log_int(rng, 200, 16000), draw=rng.randrange(1, 10000))
    if kind == "learned":
        p = rng.choice(("c4", "c5"))
        return dict(kind="learned", protocol=p, n=_log_int(rng, 64, 4096 if p == "c5" else 16000),
                    ebn0=round(rng.uniform(6.8, 7.4) if p == "c5" else rng.uniform(1.8, 3.0), 2))
    if kind == "gradients":
        z = rng.choice((52, 52, 20, 128))
        return dict(kind="gradients", bg=2, z=z, k=10 * z, e=20 * z, n=_log_int(rng, 32, 1024 * 52 // max(z, 52)),
                    iterations=rng.randrange(5, 11), shared=rng.random() < 0.7, multi=rng.choice((0, 1, 2)),
                    sigma=round(rng.uniform(0.7, 0.9), 3))
    if kind == "train":
        p = rng.choice(("c4", "c5"))
        return dict(kind="train", protocol=p, n=_log_int(rng, 64, 500 if p == "c5" else 4000))
    if kind == "sparse":
        size, info = rng.choice(((576, 288), (648, 540), (1024, 512), (301, 150), (2000, 1000)))
        rule = rng.choice(("sum_product", "normalized_min_sum", "offset_min_sum"))
        layered = rng.random() < 0.7
        return dict(kind="sparse", code="peg", size=size, info=info, precision=rng.choice(("f64", "f32")), rule=rule,
                    layered=layered, iterations=20 if layered else 40, n=_log_int(rng, 1, 2000 * 576 // max(size, 576)),
                    sigma=0.45 if info > size // 2 else round(rng.uniform(0.6, 0.72), 3))
    if kind == "dvbs2":
        rate, info = rng.choice((("1/2", 7200), ("2/3", 10800), ("3/4", 11880), ("5/6", 13320)))
        sigma = {"1/2": 0.80, "2/3": 0.64, "3/4": 0.58, "5/6": 0.52}[rate]
        return dict(kind="sparse", code="dvbs2", size=16200, info=info, precision="f32",
                    rule=rng.choice(("sum_product", "normalized_min_sum")), layered=rng.random() < 0.5, iterations=30,
                    n=_log_int(rng, 1, 150), sigma=sigma)
    return dict(kind="link", size=1024, info=512, blocks=rng.choice((1, 3, 8)), m=rng.choice((4, 16, 64)),
                n=_log_int(rng, 16, 512), ebn0=round(rng.uniform(3.0, 7.0), 2))


# ---------------------------------------------------------------- what a program keeps
# Code objects, networks and links are made once and used for many inputs.


@functools.lru_cache(maxsize=None)
def _nr(precision, **kw):
    code = cb.NrLdpc(kw.pop("k"), kw.pop("e"), precision=precision, **dict(kw))
    if precision == "f32":
        code.prepare()
    return code


@functools.lru_cache(maxsize=None)
def _sparse(code, size, info, precision, rule, layered, iterations):
    kw = dict(rule=rule, layered=layered, max_iterations=iterations, precision=precision)
    if code == "dvbs2":
        rate = {7200: "1/2", 10800: "2/3", 11880: "3/4", 13320: "5/6"}[info]
        return cb.Dvbs2Ldpc("short", rate, **kw)
    return cb.Ldpc.peg(size, info, **kw)


@functools.lru_cache(maxsize=None)
def _link(size, info, blocks, m):
    return cb.Link(_sparse("peg", size, info, "f64", "sum_product", True, 50), blocks, m, True, 1, "exact")


@functools.lru_cache(maxsize=2)
def _mix(n, draw):
    return cb.MixBatch(cb.draw_mixed_batch(n, seed=draw), name="bicm_ldpc_mix")


@functools.lru_cache(maxsize=None)
def _protocol(name):
    """(code, network with its trained weights, the weights, the protocol's settings)."""
    learned = importlib.import_module("com-rs_gb300.learned")
    p = learned.PROTOCOLS[name]
    code = _nr("f32", k=p["k"], e=p["e"], base_graph=p["bg"], lifting_size=p["z"], max_iterations=p["T"])
    net = cb.LearnedNms(code, p["T"], shared=p["shared"])
    learned.load(net, os.path.join(WEIGHTS, f"learned_{name}.npz"))
    return code, net, net.weights(), p


@functools.lru_cache(maxsize=None)
def _net(bg, z, k, e, iterations, shared):
    code = _nr("f32", k=k, e=e, base_graph=bg, lifting_size=z, max_iterations=iterations)
    return code, cb.LearnedNms(code, iterations, shared=shared)


# ---------------------------------------------------------------- inputs
def _bpsk_llr(coded, sigma, seed, dtype):
    """Channel LLRs 2 y / sigma^2 of antipodal bits in Gaussian noise (one dimension of
    Gray QPSK), on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = torch.as_tensor(coded, device="cuda")
    y = 1.0 - 2.0 * c.double() + sigma * torch.randn(c.shape, generator=g, device="cuda", dtype=torch.float64)
    return (y * (2.0 / sigma ** 2)).to(dtype)


def _bits(seed, *shape):
    return np.random.default_rng(seed).integers(0, 2, shape, dtype=np.uint8)


def _decode_sigma(case):
    """The noise `margin` dB above the rate's waterfall, as Eb/N0 of antipodal bits."""
    num, den = (int(x) for x in case["rate"].split("/"))
    ebn0 = WATERFALL[4] + RATE_DB[(num, den)] + case["margin"]
    return math.sqrt(1.0 / (2.0 * (case["k"] / case["e"]) * 10 ** (ebn0 / 10)))


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, case=case, seed=seed)
    if kind == "decode":
        code = _nr("f32", k=case["k"], e=case["e"], base_graph=case["bg"], lifting_size=case["z"])
        n, k = case["n"], case["k"]
        s["code"] = code
        s["llr"] = _bpsk_llr(code.encode(_bits(seed, n, k)), _decode_sigma(case), seed, torch.float32).contiguous()
        s["bits"] = torch.zeros(n, (k + 31) // 32, dtype=torch.int32, device="cuda")
        s["app"] = torch.zeros(n, k, dtype=torch.float32, device="cuda")
        s["its"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    elif kind == "trial":
        s["code"] = _nr(case["precision"], k=case["k"], e=case["e"], base_graph=case["bg"], lifting_size=case["z"])
    elif kind == "decode_host":
        code = _nr("f64", k=case["k"], e=case["e"], rv=case["rv"], qm=case["qm"])
        s["code"] = code
        s["llr"] = _bpsk_llr(code.encode(_bits(seed, case["n"], case["k"])), case["sigma"], seed,
                             torch.float64).cpu().numpy()
    elif kind == "encode":
        s["code"] = _nr("f32", k=case["k"], e=case["e"], base_graph=case["bg"], lifting_size=case["z"], rv=case["rv"],
                        qm=case["qm"])
        s["info"] = _bits(seed, case["n"], case["k"])
    elif kind == "mix":
        s["batch"] = _mix(case["n"], case["draw"])
    elif kind in ("learned", "train"):
        s["code"], s["net"], s["weights"], s["protocol"] = _protocol(case["protocol"])
    elif kind == "gradients":
        code, net = _net(case["bg"], case["z"], case["k"], case["e"], case["iterations"], case["shared"])
        s["code"], s["net"] = code, net
        full = cb.NrLdpc(case["k"], 50 * case["z"], base_graph=case["bg"], lifting_size=case["z"], precision="f32")
        u = _bits(seed, case["n"], case["k"])
        sent = full.encode(u)  # every bit but the first 2Z systematic ones, which are u's
        s["cw"] = np.concatenate([u[:, :2 * case["z"]], sent], axis=1)
        s["llr"] = _bpsk_llr(sent[:, :case["e"]], case["sigma"], seed, torch.float32).cpu().numpy()
    elif kind == "sparse":
        code = _sparse(case["code"], case["size"], case["info"], case["precision"], case["rule"], case["layered"],
                       case["iterations"])
        s["code"] = code
        dtype = torch.float64 if case["precision"] == "f64" else torch.float32
        s["llr"] = _bpsk_llr(code.encode(_bits(seed, case["n"], code.k)), case["sigma"], seed, dtype).cpu().numpy()
    else:
        s["link"] = _link(case["size"], case["info"], case["blocks"], case["m"])
    return s


def _records(r):
    return {name: np.ascontiguousarray(r[name]) for name in r.dtype.names if name != "reserved"}


def run(s):
    kind, case, seed = s["kind"], s["case"], s["seed"]
    if kind == "decode":
        lib, code = cb.lib(), s["code"]
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        st = lib.cb_decode_device(code._h, C.c_void_p(s["llr"].data_ptr()), case["n"], C.c_void_p(s["bits"].data_ptr()),
                                  C.c_void_p(s["app"].data_ptr()), C.c_void_p(s["its"].data_ptr()), stream)
        if st:
            raise cb.ComrsError(st, lib.cb_last_error(code._h).decode())
        return {"bits": s["bits"], "app": s["app"], "iterations": s["its"]}
    if kind == "trial":
        return _records(s["code"].run_frames(seed, "bicm_ldpc", 0, 0, case["n"], case["ebn0"], case["m"]))
    if kind == "decode_host":
        bits, app, its = s["code"].decode_full(s["llr"])
        return {"bits": bits, "app": app, "iterations": its}
    if kind == "encode":
        return {"coded": s["code"].encode(s["info"])}
    if kind == "mix":
        return _records(s["batch"].run(seed))
    if kind == "learned":
        return _records(s["net"].run_frames(seed, "learned_eval", 0, 0, case["n"], case["ebn0"], s["protocol"]["m"]))
    if kind == "gradients":
        loss, ga, gb = s["net"].gradients(s["llr"], s["cw"], case["multi"])
        return {"loss": loss, "g_alpha": ga, "g_beta": gb}
    if kind == "train":
        # the step from the trained weights, with a fresh optimiser: the call can be repeated
        net, p = s["net"], s["protocol"]
        net.set_weights(*s["weights"])
        loss = net.train_step(seed, "learned_train", case["n"], p["lo"], p["hi"], 1e-3, p["m"])
        alpha, beta = net.weights()
        net.set_weights(*s["weights"])
        return {"loss": loss, "alpha": alpha, "beta": beta}
    if kind == "sparse":
        post, its = s["code"].decode_llr(s["llr"])
        return {"post": post, "iterations": its}
    return _records(s["link"].run_trials(seed, "bicm", 0, 0, case["n"], case["ebn0"]))


# ---------------------------------------------------------------- work
def _nr_edges(bg, z):
    return (316 if bg == 1 else 197) * z


def _n_full(bg, z):
    return (68 if bg == 1 else 52) * z


def _nr_shape(k):
    """(base graph, Z) of k information bits by the standard's size rule (rates up to 2/3)."""
    bg = 2 if k <= 640 else 1
    kb = 22 if bg == 1 else (10 if k > 640 else 9 if k > 560 else 8 if k > 192 else 6)
    z = min(a * 2 ** j for a in (2, 3, 5, 7, 9, 11, 13, 15) for j in range(8) if a * 2 ** j <= 384 and kb * a * 2 ** j >= k)
    return bg, z


def work(case):
    """10 operations per edge and iteration (the min-sum row; 40 for the sum-product row's
    tanh and atanh), 50 per drawn dimension of the noise and its demapping, 30 per edge and
    iteration of a network's forward and backward passes."""
    kind, n = case["kind"], case["n"]
    if kind == "decode":
        return {"bytes": n * (4 * case["e"] + case["k"] / 8 + 4 * case["k"] + 4),
                "flops": n * 8 * 10 * _nr_edges(case["bg"], case["z"])}
    if kind == "trial":
        its = 14 if case["bg"] == 1 else 9
        return {"bytes": 8 * n, "flops": n * (its * 10 * _nr_edges(case["bg"], case["z"]) + 50 * case["e"])}
    if kind == "decode_host":
        return {"bytes": n * (8 * case["e"] + 9 * case["k"] + 4), "flops": n * 8 * 10 * _nr_edges(*_nr_shape(case["k"]))}
    if kind == "encode":
        return {"bytes": n * (case["k"] + case["e"]), "flops": n * _nr_edges(case["bg"], case["z"]) / 32}
    if kind == "mix":
        # the mean of the drawn items: about 20 iterations of 256 Z = 139 average edges
        return {"bytes": 8 * n, "flops": n * (20 * 10 * 256.5 * 139 + 50 * 4300)}
    if kind == "learned":
        bg, z, e = (1, 384, 16896) if case["protocol"] == "c5" else (2, 52, 1040)
        return {"bytes": 8 * n, "flops": n * (6 * 12 * _nr_edges(bg, z) + 50 * e)}
    if kind == "gradients":
        w = case["iterations"] * _nr_edges(case["bg"], case["z"])
        nw = w if not case["shared"] else w // case["z"]
        return {"bytes": n * (4 * case["e"] + _n_full(case["bg"], case["z"])) + 16 * nw, "flops": 30 * n * w}
    if kind == "train":
        bg, z, t = (1, 384, 8) if case["protocol"] == "c5" else (2, 52, 10)
        return {"bytes": 32 * t * _nr_edges(bg, z) // z, "flops": 30 * n * t * _nr_edges(bg, z)}
    if kind == "sparse":
        size = 8 if case["precision"] == "f64" else 4
        # three ones a column in a PEG code, about 3.1 in the DVB-S2 codes
        edges = 3 * case["size"] if case["code"] == "peg" else 3.1 * case["size"]
        per = 40 if case["rule"] == "sum_product" else 10
        return {"bytes": n * (2 * size * case["size"] + 4), "flops": n * 10 * per * edges}
    return {"bytes": 16 * n, "flops": n * case["blocks"] * (10 * 40 * 3 + 50) * case["size"]}


# ---------------------------------------------------------------- in 64 bits
def _full_llr(case, bit_map, llr, n_full, k, k_info):
    """The sent LLRs at their positions of the whole word, known (filler) bits at 30."""
    post = torch.zeros(llr.shape[0], n_full, dtype=torch.float64, device="cuda")
    post.index_add_(1, torch.as_tensor(bit_map, device="cuda", dtype=torch.int64), llr.double())
    post[:, k_info:k] = 30.0
    return post


def _layers(entries, z):
    """Per base row: the variables [Z x degree] of its lifted rows."""
    r = torch.arange(z, device="cuda")[:, None]
    out = []
    for layer in range(int(entries[:, 0].max()) + 1):
        e = torch.as_tensor(entries[entries[:, 0] == layer], device="cuda", dtype=torch.int64)
        out.append(e[None, :, 1] * z + (r + e[None, :, 2]) % z)
    return out


def _min_sum(x, mag):
    """The messages of rows x [..., degree]: the product of the other signs times
    ``mag(i, the smallest other magnitude)`` of edge i."""
    sign = torch.where(x < 0, -1.0, 1.0).double()
    a = x * sign
    m1, m2 = torch.full_like(a[..., 0], math.inf), torch.full_like(a[..., 0], math.inf)
    i1 = torch.zeros_like(m1, dtype=torch.int64)
    for i in range(x.shape[-1]):
        v = a[..., i]
        first = v < m1
        m2 = torch.where(first, m1, torch.where(v < m2, v, m2))
        m1 = torch.where(first, v, m1)
        i1 = torch.where(first, torch.full_like(i1, i), i1)
    total = sign.prod(-1)
    return torch.stack([total * sign[..., i] * mag(i, torch.where(i1 == i, m2, m1)) for i in range(x.shape[-1])], -1)


def _failing(post, layers):
    bad = torch.zeros(post.shape[0], dtype=torch.bool, device="cuda")
    for v in layers:
        bad |= ((post[:, v] < 0).sum(-1) & 1).bool().any(-1)
    return bad


def _nr_decode(post, layers, iterations=20, alpha=0.75):
    msgs = [torch.zeros(post.shape[0], *v.shape, dtype=torch.float64, device="cuda") for v in layers]
    its = torch.zeros(post.shape[0], dtype=torch.int64, device="cuda")
    live = _failing(post, layers)
    its[live] = iterations
    for t in range(1, iterations + 1):
        rows = live.nonzero()[:, 0]
        if not rows.numel():
            break
        p = post[rows]
        for i, v in enumerate(layers):
            x = p[:, v] - msgs[i][rows]
            y = _min_sum(x, lambda _, m: alpha * m)
            msgs[i][rows] = y
            p[:, v.reshape(-1)] = (x + y).reshape(len(rows), -1)
        post[rows] = p
        bad = _failing(p, layers)
        its[rows[~bad]] = t
        live[rows[~bad]] = False
    return post, its


def _sparse_layered(llr, rows, iterations):
    """Layered sum-product, the rows one after the other, each word until its syndrome is zero."""
    rows = [torch.as_tensor(r, device="cuda", dtype=torch.int64) for r in rows]
    by_degree = {}
    for r in rows:
        by_degree.setdefault(len(r), []).append(r)
    tests = [torch.stack(v)[None] for v in by_degree.values()]
    post = llr.clone()
    live = torch.zeros(len(post), dtype=torch.bool, device="cuda")
    for v in tests:
        live |= ((post[:, v[0]] < 0).sum(-1) & 1).bool().any(-1)
    its = torch.where(live, iterations, 0)
    msgs = [torch.zeros(len(post), len(r), dtype=torch.float64, device="cuda") for r in rows]
    bound = 0.999999999999
    for t in range(1, iterations + 1):
        if not bool(live.any()):
            break
        keep = live[:, None]
        for i, r in enumerate(rows):
            old = post[:, r]
            x = old - msgs[i]
            th = torch.tanh(x * 0.5)
            y = torch.stack([2 * torch.atanh(torch.cat([th[:, :j], th[:, j + 1:]], 1).prod(1).clamp(-bound, bound))
                             for j in range(len(r))], 1)
            msgs[i] = torch.where(keep, y, msgs[i])
            post[:, r] = torch.where(keep, x + y, old)
        bad = torch.zeros_like(live)
        for v in tests:
            bad |= ((post[:, v[0]] < 0).sum(-1) & 1).bool().any(-1)
        its = torch.where(live & ~bad, t, its)
        live = live & bad
    return post, its


def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode", "decode_host"):
        s = prepare(case, seed)
        code = s["code"]
        ent, bit_map = code.tables()  # the code's definition: the lifted entries and the sent positions
        llr = torch.as_tensor(s["llr"], device="cuda")
        post = _full_llr(case, bit_map, llr, code.n_full, code.k_sys, code.k_info)
        post, _ = _nr_decode(post, _layers(ent, code.z))
        return {"bits": None, "app": post[:, :code.k_info].cpu(), "iterations": None}
    if kind == "gradients":
        s = prepare(case, seed)
        code, n, T = s["code"], case["n"], case["iterations"]
        if n * T * code.edges > 110_000_000:
            return None
        ent, bit_map = code.tables()
        layers = _layers(ent, code.z)
        shape = (T, code.n_entries) if case["shared"] else (T, code.n_entries, code.z)
        al = torch.full(shape, 0.75, dtype=torch.float64, device="cuda", requires_grad=True)
        be = torch.zeros(shape, dtype=torch.float64, device="cuda", requires_grad=True)
        start = np.searchsorted(ent[:, 0], np.arange(len(layers)))
        sgn = 1.0 - 2.0 * torch.as_tensor(s["cw"], device="cuda").double()
        post = _full_llr(case, bit_map, torch.as_tensor(s["llr"], device="cuda"), code.n_full, code.k_sys, code.k_info)
        msgs = [torch.zeros(n, *v.shape, dtype=torch.float64, device="cuda") for v in layers]
        loss = 0.0
        for t in range(T):
            for i, v in enumerate(layers):
                x = post[:, v] - msgs[i]
                y = _min_sum(x, lambda j, m: torch.relu(al[t, start[i] + j] * m - be[t, start[i] + j]))
                msgs[i] = y
                post = post.index_copy(1, v.reshape(-1), (x + y).reshape(n, -1))
            w = {0: float(t == T - 1), 1: 1.0 / T, 2: 2.0 * (t + 1) / (T * (T + 1))}[case["multi"]]
            if w:
                loss = loss + w * torch.nn.functional.softplus(-sgn * post).mean()
        ga, gb = torch.autograd.grad(loss, (al, be))
        return {"loss": float(loss), "g_alpha": ga.reshape(-1).cpu(), "g_beta": gb.reshape(-1).cpu()}
    if kind == "sparse" and case["code"] == "peg" and case["layered"] and case["rule"] == "sum_product":
        if case["size"] > 700:
            return None
        s = prepare(case, seed)
        llr = torch.as_tensor(s["llr"], device="cuda").double()
        post, _ = _sparse_layered(llr, s["code"].rows, case["iterations"])
        return {"post": post.cpu(), "iterations": None}
    # counts and codewords are whole numbers; a training step draws its frames inside the call
    return None
