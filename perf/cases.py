"""Performance cases: the work a user of care_b200 has it do, through its
public entry points.

Every case is one call (or one short job) on a seeded synthetic read set:
a random genome with repeat families, reads with position-dependent
substitution rates and Phred scores drawn around them. The kinds:

- "correct"   correct_range over resident reads and tables (STEP2): a whole
              read set or a sub-range of anchors, single- or paired-end,
              without qualities or with 1, 2 or 8 bits each, with the plain or
              the learned decision, with or without candidate correction
- "job"       host arrays in, corrected reads out: upload, minhash tables,
              correction
- "fastq"     a FASTQ file in, a corrected FASTQ file out, parsed on the device
- "noalloc"   the allocation-free entry point on caller-owned device buffers
- "logits"    the decision network on host rows (forward)
- "gradient"  loss and gradient of the decision network (forward, backward)

Read sets are made on the GPU, so that preparing a case stays short.
"""
import ctypes
import math
import os
import shutil
import tempfile

import numpy as np
import torch

import care_b200
from care_b200 import autotune, learned

DATA = os.path.join(os.path.dirname(os.path.abspath(care_b200.__file__)), "data")
CHUNK = 1 << 18                       # reads made at a time


def _reads(**kw):
    """A correction case: the fields every such case has, with their defaults."""
    case = {"kind": "correct", "reads": 100_000, "lmin": 150, "lmax": 150, "paired": True, "coverage": 30.0,
            "maps": 32, "k": 20, "qbits": 2, "repeats": 0.02, "indels": False, "n_rate": 0.0, "learned": False,
            "candidates": False, "first": 0, "count": 0, "mapping": "default"}
    case.update(kw)
    return case


def listed():
    return [
        # a few anchors of a resident paired-end set: what one call of the reference's batch loop hands over, where
        # launches and latency count
        _reads(name="pe150_call_128", reads=100_000, first=20_002, count=128),
        # an ordinary batch of anchors on caller-owned device buffers, reads without qualities of an odd length
        _reads(name="noalloc_se125", kind="noalloc", reads=12_001, lmin=125, lmax=125, paired=False, qbits=0,
               maps=16, first=501, count=4095),
        # single-end reads without qualities, 100 bases, 16 maps, the default launch mapping
        _reads(name="se100_noq", reads=300_000, lmin=100, lmax=100, paired=False, qbits=0, maps=16, repeats=0.0),
        # the 5 Mbp paired-end set of the benchmark, its committed mapping
        _reads(name="pe150_q2", reads=1_000_000, mapping="pe"),
        # the same model with the learned decision
        _reads(name="pe150_learned", reads=400_000, learned=True, mapping="pe"),
        # reads of 50 to 250 bases from a genome of repeat families: uneven numbers of candidates per anchor
        _reads(name="se_uneven_q2", reads=400_000, lmin=50, lmax=250, paired=False, coverage=40.0, repeats=0.08,
               mapping="uneven"),
        # the large set's model: 50x, 48 maps, indels, reads with N left out
        _reads(name="pe150_50x_h48", reads=1_300_000, coverage=50.0, maps=48, repeats=0.05, indels=True,
               n_rate=1e-3, mapping="large"),
        # candidate correction with raw qualities, reads of 70 to 120 bases, the caller ordering what it gets
        _reads(name="se_q8_candidates", reads=30_001, lmin=70, lmax=120, paired=False, qbits=8, maps=24, k=18,
               candidates=True),
        # a whole job on host arrays, 1-bit qualities
        _reads(name="job_pe100_q1", kind="job", reads=160_000, lmin=100, lmax=100, qbits=1, maps=24),
        # a whole job on files
        _reads(name="fastq_pe151_q2", kind="fastq", reads=60_000, lmin=151, lmax=151, coverage=25.0),
        # the decision network's rows of a large batch, and one training batch
        {"name": "logits_300k", "kind": "logits", "rows": 300_000},
        {"name": "gradient_64k", "kind": "gradient", "rows": 65_536},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["correct", "correct", "correct", "correct", "part", "part", "learned", "candidates", "job",
                       "fastq", "noalloc", "logits", "gradient"])
    if kind == "logits":
        return {"kind": kind, "rows": _log_int(rng, 500, 300_000)}
    if kind == "gradient":
        return {"kind": kind, "rows": _log_int(rng, 500, 131_072)}
    paired = rng.random() < 0.5
    fixed = paired or rng.random() < 0.5
    lmax = rng.randint(70, 250)
    lmin = lmax if fixed else rng.randint(50, lmax - 10)
    reads = _log_int(rng, 2_000, 400_000)
    if kind == "candidates":
        reads = min(reads, 30_000)
    if kind in ("job", "fastq"):
        reads = min(reads, 150_000)
        lmin = lmax if kind == "fastq" else lmin
    if kind == "noalloc":
        reads = min(reads, 12_000)
    reads -= reads % 2 if paired else 0
    case = _reads(kind=kind if kind in ("job", "fastq", "noalloc") else "correct", reads=reads, lmin=lmin, lmax=lmax,
                  paired=paired, coverage=float(rng.randint(20, 50)), maps=rng.choice([8, 16, 24, 31, 32, 48]),
                  k=rng.randint(17, 24), qbits=rng.choice([0, 1, 2, 2, 8]),
                  repeats=rng.choice([0.0, 0.02, 0.05, 0.08]), indels=rng.random() < 0.3)
    if kind == "learned":
        case.update(learned=True, paired=True, lmin=case["lmax"], reads=reads - reads % 2)
    if kind == "candidates":
        case.update(candidates=True)
    if kind in ("correct", "job") and rng.random() < 0.3:
        case.update(n_rate=1e-3)
    if kind in ("part", "noalloc"):
        first = rng.randint(0, reads // 2)
        count = _log_int(rng, 2, min(reads // 2, 4096))
        even = 2 if case["paired"] else 1
        case.update(first=first - first % even, count=max(even, count - count % even))
    if case["kind"] == "correct":
        case.update(mapping=rng.choice(["default", "pe" if case["lmin"] == case["lmax"] else "uneven"]))
    return case


# ---------------------------------------------------------------- read sets

def _genome(size, fraction, g, dev):
    """Random bases; `fraction` of them in families of repeats (units of 300
    to 5,000 bases, 5 to 60 copies, 0.5 to 2 % divergence)."""
    genome = torch.randint(0, 4, (size,), generator=g, device=dev, dtype=torch.uint8)
    left = int(fraction * size)
    while left > 0:
        u, c, d = (torch.rand(3, generator=g, device=dev).cpu().numpy() * [1, 1, 0.015]).tolist()
        unit = min(int(300 * (5000 / 300) ** u), max(1, size // 8))
        copies = int(5 * 12 ** c)
        seq = torch.randint(0, 4, (unit,), generator=g, device=dev, dtype=torch.uint8).repeat(copies, 1)
        hit = torch.rand((copies, unit), generator=g, device=dev) < 0.005 + d
        seq = torch.where(hit, (seq + torch.randint(1, 4, seq.shape, generator=g, device=dev, dtype=torch.uint8)) & 3, seq)
        at = torch.randint(0, size - unit + 1, (copies,), generator=g, device=dev)
        for i, p in enumerate(at.tolist()):              # later copies over earlier ones
            genome[p:p + unit] = seq[i]
        left -= unit * copies
    return genome


def _chunk(case, genome, n, g, dev):
    """n reads: codes (n, lmax), lengths, Phred scores, N flags."""
    L, G = case["lmax"], genome.numel()
    j = torch.arange(L, device=dev)
    if case["paired"]:
        m = n // 2
        frag = (400 + 40 * torch.randn(m, generator=g, device=dev)).round().clamp(L + 1, 800).long().clamp(max=G)
        start = (torch.rand(m, generator=g, device=dev, dtype=torch.float64) * (G - frag + 1).double()).long()
        flip = torch.rand(m, generator=g, device=dev) < 0.5
        begin = torch.stack([start, start + frag - L], 1)
        rc = torch.stack([flip, ~flip], 1)
        begin = torch.where(flip[:, None], begin.flip(1), begin).reshape(-1)
        rc = rc.reshape(-1)
        length = torch.full((n,), L, device=dev, dtype=torch.long)
    else:
        length = torch.randint(case["lmin"], L + 1, (n,), generator=g, device=dev)
        length[0] = L                                    # the storage is as wide as the case says
        begin = (torch.rand(n, generator=g, device=dev, dtype=torch.float64) * (G - length + 1).double()).long()
        rc = torch.rand(n, generator=g, device=dev) < 0.5
    pos = j[None, :].expand(n, L)
    if case["indels"]:                                   # one inserted or deleted base in about 1.5 % of 150 bp reads
        hit = torch.rand(n, generator=g, device=dev) < 1.0 - (1.0 - 1e-4) ** L
        at = torch.randint(1, L, (n,), generator=g, device=dev)
        step = torch.where(torch.rand(n, generator=g, device=dev) < 0.5, 1, -1) * hit
        pos = pos + step[:, None] * (pos >= at[:, None])
    src = torch.where(rc[:, None], begin[:, None] + length[:, None] - 1 - pos, begin[:, None] + pos).clamp_(0, G - 1)
    code = genome[src]
    code = torch.where(rc[:, None], 3 - code, code)
    rate = 0.002 + 0.013 * (j[None, :] / (length[:, None] - 1).clamp(min=1)).clamp(max=1.0)
    err = torch.rand((n, L), generator=g, device=dev) < rate
    code = torch.where(err, (code + torch.randint(1, 4, (n, L), generator=g, device=dev, dtype=torch.uint8)) & 3, code)
    q = (-10.0 * torch.log10(rate) + 3.0 * torch.randn((n, L), generator=g, device=dev)).round().clamp(2, 40).to(torch.uint8)
    valid = j[None, :] < length[:, None]
    isn = (torch.rand((n, L), generator=g, device=dev) < case["n_rate"]) & valid
    return torch.where(valid, code, 0), length, torch.where(valid, q, 0), isn.any(1), valid


def _words(v, bits):
    """Codes (n, L) of `bits` bits each -> uint32 rows, first code in the highest bits."""
    n, L = v.shape
    per = 32 // bits
    w = (L + per - 1) // per
    p = torch.zeros((n, w * per), device=v.device, dtype=torch.int32)
    p[:, :L] = v
    shift = 32 - bits * (1 + torch.arange(per, device=v.device, dtype=torch.int32))
    return (p.view(n, w, per) << shift).sum(2, dtype=torch.int32)


def _encode_quality(q, valid, bits):
    if bits == 8:                                        # the Phred+33 characters, four per word
        n, L = q.shape
        p = torch.zeros((n, 4 * ((L + 3) // 4)), device=q.device, dtype=torch.uint8)
        p[:, :L] = torch.where(valid, q + 33, 0)
        return p.view(torch.int32)
    bounds = torch.tensor([13] if bits == 1 else [4, 13, 20], device=q.device, dtype=torch.uint8)
    code = torch.bucketize(q, bounds)                    # first bin whose bound is not below q
    return _words(torch.where(valid, code, 0).to(torch.int32), bits)


def _read_set(case, seed):
    """The read storage of a case, as host arrays."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(seed * 1_000_003 + case["reads"])
    mean = 0.5 * (case["lmin"] + case["lmax"])
    size = max(2_000, int(case["reads"] * mean / case["coverage"]))
    genome = _genome(size, case["repeats"], g, dev)
    n = case["reads"]
    out = {"packed": [], "lengths": [], "quals": [], "ambiguous": []}
    for b in range(0, n, CHUNK):
        code, length, q, isn, valid = _chunk(case, genome, min(CHUNK, n - b), g, dev)
        out["packed"].append(_words(code.to(torch.int32), 2).cpu())
        out["lengths"].append(length.to(torch.int32).cpu())
        out["ambiguous"].append((isn.nonzero().view(-1) + b).to(torch.int32).cpu())
        if case["qbits"]:
            out["quals"].append(_encode_quality(q, valid, case["qbits"]).cpu())
    r = {k: torch.cat(v).numpy() if v else None for k, v in out.items()}
    for k in ("packed", "quals", "ambiguous"):
        if r[k] is not None:
            r[k] = r[k].view(np.uint32)
    return r


def _write_fastq(case, seed, path):
    """The read set of a case (fixed lengths) as 4-line FASTQ records."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(seed * 1_000_003 + case["reads"])
    L, n = case["lmax"], case["reads"]
    genome = _genome(max(2_000, int(n * L / case["coverage"])), case["repeats"], g, dev)
    letters = torch.tensor(list(b"ACGT"), device=dev, dtype=torch.uint8)
    with open(path, "wb") as f:
        for b in range(0, n, CHUNK):
            m = min(CHUNK, n - b)
            code, _, q, _, _ = _chunk(case, genome, m, g, dev)
            rec = torch.full((m, 14 + 2 * L), ord("\n"), device=dev, dtype=torch.uint8)
            rec[:, 0], rec[:, 1] = ord("@"), ord("r")
            ids = torch.arange(b, b + m, device=dev)
            for d in range(7):
                rec[:, 8 - d] = (ord("0") + (ids // 10 ** d) % 10).to(torch.uint8)
            rec[:, 10:10 + L] = letters[code.long()]
            rec[:, 11 + L] = ord("+")
            rec[:, 13 + L:13 + 2 * L] = q + 33
            f.write(rec.cpu().numpy().tobytes())


# ------------------------------------------------------------------- cases

def _options(case):
    return care_b200.default_options(
        kmerlength=case["k"], num_maps=case["maps"], estimated_coverage=case["coverage"],
        use_quality=int(case["qbits"] > 0), quality_bits=case["qbits"] or 8, paired_end=int(case["paired"]),
        exclude_ambiguous=int(case["n_rate"] > 0), correct_candidates=int(case["candidates"]),
        correction_type=int(case["learned"]))


def _corrector(case):
    c = care_b200.Corrector(_options(case))
    if case["mapping"] != "default":
        c.tuning = autotune.load(case["mapping"])
    if case["learned"]:
        c.set_mlp(learned.load_params(os.path.join(DATA, "mlp_pe30x.bin")))
    return c


def _network(case, seed):
    """Rows around the network's own input normalisation, labels nearly all
    1 and false-positive rows weighted, as its training sets are."""
    params = learned.load_params(os.path.join(DATA, "mlp_pe30x.bin"))
    mean, istd = params[care_b200.MLP_PARAMS:care_b200.MLP_PARAMS + 24], params[care_b200.MLP_PARAMS + 24:]
    rng = np.random.default_rng(seed)
    x = mean + rng.standard_normal((case["rows"], care_b200.MLP_FEATURES), dtype=np.float32) / istd
    y = (rng.random(case["rows"]) < 0.95).astype(np.float32)
    w = np.where((y == 0) & (rng.random(case["rows"]) < 0.3), np.float32(learned.FP_WEIGHT), np.float32(1.0))
    return params, np.ascontiguousarray(x, np.float32), y, w


class _Files:
    """A folder that goes with the state."""

    def __init__(self):
        self.path = tempfile.mkdtemp(prefix="care_b200_case_")

    def __del__(self):
        shutil.rmtree(self.path, ignore_errors=True)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("logits", "gradient"):
        params, x, y, w = _network(case, seed)
        m = care_b200.Mlp()
        m.params = params
        return {"case": case, "mlp": m, "x": x, "y": y, "w": w}
    if kind == "fastq":
        d = _Files()
        state = {"case": case, "dir": d, "in": os.path.join(d.path, "in.fq"), "out": os.path.join(d.path, "out.fq")}
        _write_fastq(case, seed, state["in"])
        state["corrector"] = _corrector(case)
        return state
    r = _read_set(case, seed)
    c = _corrector(case)
    if kind == "job":
        return {"case": case, "corrector": c, "reads": r}
    c.upload_reads(r["packed"], r["lengths"], r["quals"], r["ambiguous"])
    c.build_tables()
    if kind == "noalloc":
        return _device_buffers(case, r, c)
    return {"case": case, "corrector": c, "count": case["count"] or case["reads"] - case["first"]}


def _device_buffers(case, r, c):
    """Reads and tables in device memory of the caller."""
    dev = torch.device("cuda")

    def put(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(dev)

    flags = np.zeros(case["reads"], np.uint8)
    flags[r["ambiguous"]] = 1
    descs, slots, values = care_b200.table_device_layout([c.get_table(i) for i in range(c.num_maps)])
    q = r["quals"] if r["quals"] is not None else np.zeros((1, 1), np.uint32)
    held = [put(r["packed"].view(np.int32)), put(r["lengths"]), put(q.view(np.int32)), put(flags),
            put(np.frombuffer(descs, np.uint8).copy()), put(np.frombuffer(slots, np.uint8).copy()),
            put(values.view(np.int32))]
    s, ln, qd, am, d, sl, v = (t.data_ptr() for t in held)
    count = case["count"] or min(case["reads"] - case["first"], care_b200.NOALLOC_MAX_ANCHORS)
    outs = {"status": torch.zeros(count, dtype=torch.uint8, device=dev),
            "num_edits": torch.zeros(count, dtype=torch.int32, device=dev),
            "sequences": torch.zeros((count, c.max_length), dtype=torch.uint8, device=dev)}
    return {"case": case, "opts": _options(case), "count": count, "held": held, "outs": outs,
            "reads": care_b200.DeviceReads(s, r["packed"].shape[1], ln, qd, q.shape[1], am, case["reads"], c.max_length),
            "tables": care_b200.DeviceTables(c.num_maps, d, sl, v, c.result_threshold)}


class _Held:
    """Memory of a corrector's results, which lives as long as the corrector."""

    def __init__(self, corrector, pointer, shape, dtype):
        self.corrector = corrector
        self.__array_interface__ = {"data": (ctypes.cast(pointer, ctypes.c_void_p).value, False), "shape": shape,
                                    "typestr": np.dtype(dtype).str, "version": 3}


def _view(c, pointer, shape, dtype):
    return np.asarray(_Held(c, pointer, shape, dtype)) if math.prod(shape) else np.zeros(shape, dtype)


def _results(case, c, raw):
    n, L = raw.num_anchors, raw.max_length
    out = {"status": _view(c, raw.anchor_status, (n,), np.uint8),
           "num_edits": _view(c, raw.anchor_num_edits, (n,), np.int32),
           "sequences": _view(c, raw.anchor_sequences, (n, L), np.uint8)}
    if case["candidates"]:
        # corrections of candidates come in no order: the caller puts them in the order of read and anchor, into
        # arrays with room for one per read and unit of coverage
        m = int(raw.num_candidates)
        room = int(case["reads"] * case["coverage"])
        part = [torch.from_numpy(_view(c, p, s, t)).cuda() for p, s, t in (
            (raw.cand_read_ids, (m,), np.int32), (raw.cand_anchor_ids, (m,), np.int32),
            (raw.cand_shifts, (m,), np.int32), (raw.cand_use_edits, (m,), np.uint8),
            (raw.cand_sequences, (m, L), np.uint8))]
        order = torch.argsort((part[0].long() << 32) | part[1].long())[:room]
        for name, v in zip(("cand_read", "cand_anchor", "cand_shift", "cand_edits", "cand_sequences"), part):
            out[name] = v.new_zeros((room,) + v.shape[1:])
            torch.index_select(v, 0, order, out=out[name][:order.numel()])
        out["cand_count"] = m
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "logits":
        return state["mlp"].forward(state["x"])
    if kind == "gradient":
        loss, grad = state["mlp"].gradient(state["x"], state["y"], state["w"])
        return {"loss": loss, "gradient": grad}
    if kind == "noalloc":
        o = state["outs"]
        care_b200.correct_range_noalloc(state["opts"], state["reads"], state["tables"], case["first"], state["count"],
                                        o["status"].data_ptr(), o["num_edits"].data_ptr(), o["sequences"].data_ptr(),
                                        torch.cuda.current_stream().cuda_stream)
        return o
    c = state["corrector"]
    if kind == "fastq":
        c.load_files([state["in"]], device=True)
        c.build_tables()
        c.correct_range_raw(0, c.num_reads)
        c.write_output(state["out"])
        return np.fromfile(state["out"], np.uint8)
    if kind == "job":
        r = state["reads"]
        c.upload_reads(r["packed"], r["lengths"], r["quals"], r["ambiguous"])
        c.build_tables()
        return _results(case, c, c.correct_range_raw(0, case["reads"]))
    return _results(case, c, c.correct_range_raw(case["first"], state["count"]))


def work(case):
    """Bytes of the inputs (the anchors' and the candidates' rows, qualities,
    keys and table entries) and of the results. Correction is integer and
    byte work; the operations counted are the network's."""
    if case["kind"] == "logits":
        return {"bytes": case["rows"] * (24 + 1) * 4, "flops": case["rows"] * 12_416}
    if case["kind"] == "gradient":
        return {"bytes": case["rows"] * (24 + 2) * 4 + 4 * care_b200.MLP_PARAMS, "flops": case["rows"] * 3 * 12_416}
    n = case["reads"]
    count = case["count"] or n - case["first"]
    L = 0.5 * (case["lmin"] + case["lmax"])
    row = 4 * math.ceil(case["lmax"] / 16) + 4 * math.ceil(case["lmax"] * case["qbits"] / 32) + 4
    per_anchor = case["maps"] * (8 + 16 + 4) + case["lmax"] + 5
    rows = min(n, count * 2 * case["coverage"])                # reads of the storage that a call meets
    if case["candidates"]:
        per_anchor += 0.4 * case["coverage"] * (13 + L)
    if case["kind"] == "fastq":
        per_anchor += 4 * L
    return {"bytes": int(count * per_anchor + rows * row), "flops": 0}


def tolerance(case):
    # bf16 operands and activations, fp32 sums: measured against the same network in 64 bits, the logits are 1.3e-3 off,
    # the gradient 8e-4 and the loss 3e-4; four times that. Corrections are whole numbers and bytes.
    if case["kind"] == "logits":
        return {"rel": 5e-3, "max": 0.1}
    if case["kind"] == "gradient":
        return {"rel": 4e-3, "max": 0.1}
    return "exact"


def exact(case, seed):
    if case["kind"] not in ("logits", "gradient"):
        return None                                            # whole numbers and bytes
    params, x, y, w = _network(case, seed)
    p = torch.from_numpy(params).double().cuda().requires_grad_(True)
    xd = torch.from_numpy(x).double().cuda()
    at = np.cumsum([0, 1536, 64, 4096, 64, 64, 1, 24, 24])
    w1, b1, w2, b2, w3, b3, mean, istd = (p[a:b] for a, b in zip(at[:-1], at[1:]))
    h = torch.nn.functional.gelu(((xd - mean.detach()) * istd.detach()) @ w1.view(64, 24).T + b1)
    h = torch.nn.functional.gelu(h @ w2.view(64, 64).T + b2)
    logit = h @ w3 + b3
    if case["kind"] == "logits":
        return logit.detach()
    yd, wd = torch.from_numpy(y).double().cuda(), torch.from_numpy(w).double().cuda()
    loss = (torch.nn.functional.binary_cross_entropy_with_logits(logit, yd, reduction="none") * wd).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "gradient": p.grad[:care_b200.MLP_PARAMS]}
