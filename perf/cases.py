"""Performance cases of the classifier: the calls a user's program makes, through the public entry points.

A case is a dict of plain values.  `kind` names the call:
  classify   Classifier.classify / classify_i16: raw reads on the host in, result records on the host out
  device     Classifier.classify_device: raw reads on the GPU in, result records on the GPU out
  serve      Read Until: three 1,600-sample chunks of every channel's read, resumed from the row state on the GPU
  normalize  Classifier.normalize: window and z-score of raw reads on the GPU
  static     dtwx_distances_static: z-scored reads on the GPU, no allocation by the library
  create     a Classifier for a new target genome, with its squiggle read back
Inputs follow the repository's simulator: uniform random genomes, 4,096 6-mer levels of N(90, 12) pA, one k-mer
held for a geometric dwell of mean 9 samples, 1.8 pA of noise, half the reads from the target genome, any strand.
"""
import ctypes

import numpy as np
import torch

import dtwax_gb300 as d

CHUNK = 1600           # samples of a Read Until chunk (0.4 s at 4 kHz)
OFFSET, RANGE, DIGITISATION = 12.0, 1400.0, 8192.0   # a flow cell's ADC scaling
ADAPTER, QUERY = 1952, 2048                          # the command line's window
PRECISION = {"fp16": d.FP16, "fp32": d.FP32, "mixed": d.MIXED}
MOST_CELLS = 2.0e12    # drawn cases stay below the largest listed one (8.2e12 cells)
EXACT_CELLS = 1.1e12   # above this the 64-bit answer takes too long
EXACT_REF_DEL = 2.2e11


def _case(name, kind, **kw):
    c = dict(kind=kind, genome=48_502, reads=1, lo=2000, hi=2000, precision="fp16", ref_del=False, concat=False,
             i16=False, window=False, state="fp32")
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one FIFO batch of the command line: 10 reads, 2,048 samples after the adapter, lambda phage
        _case("cli_10x2048_lambda", "classify", reads=10, lo=3700, hi=6500, window=True),
        # a small study: 512 reads of raw ADC samples against lambda
        _case("lambda_512x2000_i16", "classify", reads=512, i16=True),
        # the benchmark's precision-study shape, reads resident on the GPU; the largest case
        _case("mb1_2048x2000", "device", genome=1_000_000, reads=2048),
        # bacterial genome, reads of 1,000 to 8,000 samples in one batch
        _case("mb5_96_uneven", "device", genome=5_000_000, reads=96, lo=1000, hi=8000),
        # FP32 cells: the reference's plain precision, both strands
        _case("fp32_mb1_192x2000", "device", genome=1_000_000, reads=192, precision="fp32"),
        # FP16 differences with an FP32 path cost
        _case("mixed_mb1_192x2000", "device", genome=1_000_000, reads=192, precision="mixed"),
        # the recurrence with the left predecessor, in both cell types it is built for
        _case("refdel_fp16_lambda_2048x1000", "device", reads=2048, lo=1000, hi=1000, ref_del=True),
        _case("refdel_fp32_lambda_512x2000", "classify", reads=512, precision="fp32", ref_del=True),
        # Read Until on a bacterial genome: the few reads that wait for a batch at one time
        _case("serve_4_mb5", "serve", genome=5_000_000, reads=4, lo=CHUNK * 3, hi=CHUNK * 3),
        # the normaliser alone, before a user's own use of the z-scored reads
        _case("normalize_2048_uneven", "normalize", reads=2048, lo=1000, hi=8000),
        # next to a basecaller that owns the GPU's memory: FP32, the library's fixed scratch
        _case("static_64_lambda", "static", reads=64, lo=500, hi=2048, precision="fp32"),
        # a new target: genome in, squiggle of both strands built, z-scored and read back
        _case("create_mb5", "create", genome=5_000_000),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["classify", "classify", "device", "device", "device", "serve", "normalize", "static", "create"])
    c = _case(None, kind, genome=_log(rng, 5_000, 5_000_000))
    if kind in ("classify", "device"):
        c["precision"] = rng.choice(["fp16", "fp16", "fp16", "fp32", "mixed"])
        c["ref_del"] = c["precision"] != "mixed" and rng.random() < 0.25
        c["concat"] = c["precision"] == "fp32" and rng.random() < 0.25
        c["i16"] = kind == "classify" and rng.random() < 0.4
        c["window"] = kind == "classify" and rng.random() < 0.3
        c["reads"] = _log(rng, 1, 2048)
        c["lo"] = _log(rng, 200, 4000)
        c["hi"] = rng.choice([c["lo"], min(8000, c["lo"] * rng.randint(2, 8))])
        if c["window"]:
            c["lo"], c["hi"] = 3700, rng.randint(4001, 7000)
    elif kind == "serve":
        c.update(genome=_log(rng, 50_000, 5_000_000), precision=rng.choice(["fp16", "fp16", "fp32", "mixed"]),
                 reads=_log(rng, 1, 16), lo=CHUNK * 3, hi=CHUNK * 3)
        if c["precision"] == "fp16" and rng.random() < 0.5:
            c["state"] = "fp16"
    elif kind == "normalize":
        c.update(genome=5_000, reads=_log(rng, 1, 4096), lo=_log(rng, 200, 4000))
        c["hi"] = min(8000, c["lo"] * rng.randint(1, 8))
    elif kind == "static":
        c.update(genome=_log(rng, 5_000, 200_000), reads=_log(rng, 1, 512), lo=_log(rng, 100, 2048), hi=2048,
                 precision="fp32")
    else:
        c["precision"] = rng.choice(["fp16", "fp32"])
    # a pass stays well below the largest listed case; one read of the REF_DEL recurrence is one warp's work
    most = MOST_CELLS / (20 if c["ref_del"] or kind == "static" else 1)
    rows = c["hi"] if not c["window"] else QUERY
    while kind in ("classify", "device", "static", "serve") and (
            _cells(c) > most or (c["ref_del"] and rows * c["genome"] > 2.0e8)):
        if c["reads"] > 64 and not (c["ref_del"] and rows * c["genome"] > 2.0e8):
            c["reads"] = c["reads"] * 2 // 3 + 1
        else:
            c["genome"] = c["genome"] * 2 // 3 + 1
    return c


def _m(c):
    return c["genome"] - 5


def _mean_rows(c):
    return QUERY if c["window"] else (c["lo"] + c["hi"]) / 2


def _cells(c):
    return 2.0 * c["reads"] * _mean_rows(c) * _m(c)


# ---------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _codes(genome):
    """6-mer codes of both strands of a genome given as 2-bit bases (A<C<G<T)."""
    out = []
    for s in (genome, 3 - genome.flip(0)):
        m = s.numel() - 5
        k = torch.zeros(m, dtype=torch.int64, device=s.device)
        for i in range(6):
            k = k * 4 + s[i:i + m]
        out.append(k)
    return torch.stack(out)


def _inputs(c, seed):
    """Genome, level table and reads of a case: everything comes from the seed."""
    g = _gen(seed)
    rnd = lambda n: torch.rand(n, generator=g, device="cuda")  # noqa: E731
    genome = torch.randint(0, 4, (c["genome"],), generator=g, device="cuda")
    table = torch.randn(4096, generator=g, device="cuda") * 12.0 + 90.0
    x = dict(genome=genome, table=table)
    if c["kind"] == "create":
        return x
    n = c["reads"]
    # lengths spread evenly over lo..hi, in an order of the seed's: every seed has the same total
    lens = c["lo"] + (c["hi"] - c["lo"]) * (2 * torch.randperm(n, generator=g, device="cuda") + 1) // (2 * n)
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = lens.cumsum(0)
    total = int(off[-1])
    # the level of each sample: a k-mer is left with probability 1/9 after each sample
    step = (rnd(total) < 1.0 / 9.0).to(torch.int64).cumsum(0)
    owner = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    at = step - step[off[:-1]][owner]
    m = _m(c)
    start = (rnd(n) * (m - (lens.to(torch.float32) / 9.0 * 1.3).clamp(max=m - 1))).to(torch.int64).clamp(0, m - 1)
    strand = torch.randint(0, 2, (n,), generator=g, device="cuda")
    target = torch.arange(n, device="cuda") % 2 == 0
    levels = table[_codes(genome)]
    other = table[_codes(torch.randint(0, 4, (c["genome"],), generator=g, device="cuda"))]
    both = torch.stack([other, levels]).reshape(-1)
    pos = (start[owner] + at).clamp(max=m - 1)
    sig = both[(target[owner].to(torch.int64) * 2 + strand[owner]) * m + pos]
    sig = sig + 1.8 * torch.randn(total, generator=g, device="cuda")
    if c["i16"]:
        x["raw16"] = (sig * (DIGITISATION / RANGE) - OFFSET).round().to(torch.int16)
    x.update(raw=sig.to(torch.float32), offsets=off.cpu().numpy(), lens=lens)
    return x


def _zscored64(x, offsets, eps=1e-4):
    """Every read of a flat batch z-scored on its own, in 64 bits."""
    off = torch.as_tensor(offsets, device="cuda")
    n = off.numel() - 1
    lens = off[1:] - off[:-1]
    owner = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    x = x.double()
    zero = torch.zeros(n, dtype=torch.float64, device="cuda")
    count = lens.double().clamp(min=1)
    mean = zero.index_add(0, owner, x) / count
    dev = x - mean[owner]
    var = zero.index_add(0, owner, dev * dev) / count
    return dev / torch.sqrt(var + eps)[owner]


def _levels64(x):
    """z-scored levels of both strands, in 64 bits."""
    lev = x["table"].double()[_codes(x["genome"])]
    return (lev - lev.mean(1, keepdim=True)) / lev.std(1, unbiased=False, keepdim=True)


def _sequence(x):
    return np.frombuffer(b"ACGT", np.uint8)[x["genome"].cpu().numpy()].tobytes()


def _config(c):
    cfg = dict(precision=PRECISION[c["precision"]], recurrence=d.REF_DEL if c["ref_del"] else d.NO_REF_DEL)
    if c["concat"]:
        cfg["strand_mode"] = d.STRANDS_CONCAT
    if c["window"]:
        cfg.update(adapter_skip=ADAPTER, query_len=QUERY, require_full=1)
    if c["kind"] == "serve":
        cfg["threshold"] = -1.0  # every read is followed for its three chunks
        if c["state"] == "fp16":
            cfg["state_precision"] = d.STATE_FP16
    return cfg


def prepare(case, seed):
    c = case
    x = _inputs(c, seed)
    table = x["table"].cpu().numpy()
    s = dict(case=c)
    if c["kind"] == "create":
        s.update(sequence=_sequence(x), table=table)
        return s
    n = c["reads"]
    s["offsets"] = x["offsets"]
    if c["kind"] == "static":
        z = _levels64(x)
        pairs = torch.zeros((-(-z.shape[1] // 512) * 512, 2), dtype=torch.float32, device="cuda")
        pairs[: z.shape[1]] = z.t().float()
        s.update(pairs=pairs, m=z.shape[1], query=_zscored64(x["raw"], x["offsets"]).float(),
                 out=torch.zeros(32 * n, dtype=torch.uint8, device="cuda"))
        return s
    s["clf"] = d.Classifier(sequence=_sequence(x), level_table=table, **_config(c))
    if c["kind"] == "classify":
        if c["i16"]:
            s["raw"] = x["raw16"].cpu().numpy()
            s["scale"] = [np.full(n, v, np.float32) for v in (OFFSET, RANGE, DIGITISATION)]
        else:
            s["raw"] = x["raw"].cpu().numpy()
    elif c["kind"] == "device":
        s.update(raw=x["raw"], out=torch.zeros(32 * n, dtype=torch.uint8, device="cuda"))
    elif c["kind"] == "normalize":
        s.update(raw=x["raw"], query=torch.zeros_like(x["raw"]))
    else:
        s["chunks"] = x["raw"].cpu().numpy().reshape(n, 3, CHUNK)
        s["next"] = 1
        s["clf"].serve_start(max_in_flight=n, chunks_per_decision=3)
    return s


# ---------------------------------------------------------------- one pass

def _records(out):
    """The fields of result records that stay on the GPU."""
    f, i, w = out.view(torch.float32).view(-1, 8), out.view(torch.int32).view(-1, 8), out.view(torch.int64).view(-1, 4)
    return dict(score=f[:, 0], score_fwd=f[:, 1], score_rev=f[:, 2], strand=i[:, 3], end_pos=w[:, 2], call=i[:, 6],
                n_samples=i[:, 7])


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "create":
        with d.Classifier(sequence=s["sequence"], level_table=s["table"], **_config(c)) as clf:
            fwd, rev = clf.reference()
        return dict(fwd=fwd, rev=rev)
    if kind == "classify":
        if c["i16"]:
            o, r, g = s["scale"]
            res = s["clf"].classify_i16(raw=s["raw"], offsets=s["offsets"], offset=o, range_=r, digitisation=g)
        else:
            res = s["clf"].classify(raw=s["raw"], offsets=s["offsets"])
        return {k: res[k] for k in d.RESULT_DTYPE.names}
    if kind == "device":
        s["clf"].classify_device(s["raw"].data_ptr(), s["offsets"], s["out"].data_ptr())
        return _records(s["out"])
    if kind == "normalize":
        s["clf"].normalize(s["raw"].data_ptr(), s["offsets"], s["query"].data_ptr())
        return s["query"]
    if kind == "static":
        lib = d.load_library()
        rc = lib.dtwx_distances_static(
            ctypes.c_void_p(s["pairs"].data_ptr()), s["m"], ctypes.c_void_p(s["query"].data_ptr()),
            s["offsets"].ctypes.data_as(ctypes.POINTER(ctypes.c_int64)), s["offsets"].size - 1, ctypes.c_float(194.0),
            ctypes.c_void_p(s["out"].data_ptr()), None)
        if rc != 0:
            raise d.DtwxError(rc, lib.dtwx_last_error(None).decode(errors="replace"))
        return _records(s["out"])
    # Read Until: each round every channel delivers its next chunk
    clf, first, n = s["clf"], s["next"], c["reads"]
    s["next"] += n
    for k in range(3):
        for r in range(n):
            clf.submit_chunk(r, first + r, s["chunks"][r, k], is_last=k == 2)
        clf.serve_step()
        clf.serve_drain()
    got = clf.poll_decisions()
    out = {k: np.array([g[k] for g in got], np.int64) for k in ("channel", "chunks", "samples", "strand", "end_pos",
                                                               "call", "decided")}
    out["read"] = np.array([g["read_number"] - first for g in got], np.int64)
    out["score"] = np.array([g["score"] for g in got], np.float32)
    return out


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    c = case
    m, total = _m(c), c["reads"] * (c["lo"] + c["hi"]) / 2
    if c["kind"] == "create":
        # genome in, two strands of FP32 levels out; a difference and a product per level
        return dict(bytes=c["genome"] + 2 * 4 * m, flops=2 * 2 * 4 * m)
    if c["kind"] == "normalize":
        return dict(bytes=8 * total, flops=6 * total)
    if c["window"]:
        total = c["reads"] * QUERY
    level = 8 if c["precision"] == "fp32" else 4  # bytes of a column's two levels
    cells = 2.0 * total * m
    state = 0
    if c["kind"] == "serve":  # the row state: written after each of three chunks, read before the last two
        state = 5 * c["reads"] * m * (4 if c["state"] == "fp16" else 8)
    # a cell: difference, minimum (two with the left predecessor), product, sum
    return dict(bytes=total * (2 if c["i16"] else 4) + level * m + 32 * c["reads"] + state,
                flops=cells * (5 if c["ref_del"] else 4))


# ---------------------------------------------------------------- the same in 64 bits

def _sweep64(ref, q, offsets, ref_del, marks=None):
    """Minimum of the last row of every read on every sequence of ref [S, m]: [n, S].
    marks: row counts after which the minimum is wanted, for reads of one length: [n, len(marks), S]."""
    S, m = ref.shape
    lens = np.diff(offsets)
    n = lens.size
    out = torch.full((n, len(marks) if marks else 1, S), float("inf"), dtype=torch.float64, device="cuda")
    order = np.argsort(-lens, kind="stable")
    block = max(1, int(64e6 // (S * m * 8)))
    for b in range(0, n, block):
        ids = order[b:b + block]
        most = int(lens[ids[0]])
        if most == 0:
            continue
        rows = torch.zeros((most, ids.size), dtype=torch.float64, device="cuda")
        ends = {}
        for k, r in enumerate(ids):
            rows[: lens[r], k] = q[int(offsets[r]): int(offsets[r + 1])]
            for w, at in enumerate(marks or [int(lens[r])]):
                ends.setdefault(at, []).append((k, int(r), w))
        D = torch.zeros((ids.size, S, m), dtype=torch.float64, device="cuda")
        low, diff = torch.empty_like(D), torch.empty_like(D)
        for i in range(most):
            torch.sub(ref, rows[i].view(-1, 1, 1), out=diff)
            torch.minimum(D[..., 1:], D[..., :-1], out=low[..., 1:])
            low[..., 0] = D[..., 0]
            if not ref_del:
                torch.addcmul(low, diff, diff, out=D)
            else:
                # D[j] = cost[j] + min(low[j], D[j-1]): a running minimum over the prefix sums of the costs
                diff.mul_(diff)
                run_ = diff.cumsum(-1)
                low.add_(diff).sub_(run_)
                D = torch.cummin(low, -1).values.add_(run_)
            for k, r, w in ends.get(i + 1, ()):
                out[r, w] = D[k].amin(-1)
    return out


def exact(case, seed):
    c = case
    if c["kind"] in ("classify", "device", "static", "serve"):
        if _cells(c) > (EXACT_REF_DEL if c["ref_del"] else EXACT_CELLS):
            return None
    x = _inputs(c, seed)
    if c["kind"] == "create":
        z = _levels64(x)
        return dict(fwd=z[0], rev=z[1])
    raw, offsets = x["raw"], x["offsets"]
    if c["i16"]:
        raw = (x["raw16"].double() + OFFSET) * (RANGE / DIGITISATION)
    if c["kind"] == "normalize":
        return _zscored64(raw, offsets)
    if c["window"]:
        lens = np.diff(offsets)
        keep = lens >= ADAPTER + QUERY
        raw = torch.cat([raw[int(o) + ADAPTER: int(o) + ADAPTER + QUERY] for o, k in zip(offsets[:-1], keep) if k]
                        or [raw[:0]])
        offsets = np.concatenate([[0], np.cumsum(np.where(keep, QUERY, 0))])
    ref = _levels64(x)
    if c["kind"] == "serve":
        n = c["reads"]
        q = _zscored64(raw, np.arange(3 * n + 1) * CHUNK)
        low = _sweep64(ref, q, offsets, c["ref_del"], [CHUNK, 2 * CHUNK, 3 * CHUNK]).amin(-1)
        none = {k: None for k in ("channel", "chunks", "samples", "strand", "end_pos", "call", "decided", "read")}
        return dict(none, score=low.t().reshape(-1))  # the decisions come round by round
    q = _zscored64(raw, offsets)
    low = _sweep64(ref.reshape(1, -1) if c["concat"] else ref, q, offsets, c["ref_del"])[:, 0]
    none = {k: None for k in ("strand", "end_pos", "call", "n_samples")}
    return dict(none, score=low.amin(-1), score_fwd=low[:, 0], score_rev=low[:, -1])
