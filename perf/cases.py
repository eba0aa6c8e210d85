"""Workloads of this library as its users run it, for timing and for comparing results.

Each case is one call (or one replay of a plan) through the public entry
points: the one-pair functions of parasail.h, database searches, batches of
independent pairs, all-against-all statistics, CIGARs and long global pairs.
Sizes are the repository's own benchmark configurations, cut where a pass
would take longer than a second, and the sizes between them.

  listed()            the fixed cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) inputs made from the seed, profiles, plans and output buffers
  run(state)          one pass; returns its outputs
  work(case)          bytes and lane operations a pass cannot do without
  exact(case, seed)   64-bit values where they are cheap (the one-pair calls)
"""
import functools
import math

import numpy as np
import torch

import parasail_b200 as pb

AA = "ARNDCQEGHILKMFPSTWYV"
# amino-acid background frequencies of Robinson & Robinson (1991)
AA_FREQ = (0.07805, 0.05129, 0.04487, 0.05364, 0.01925, 0.04264, 0.06295, 0.07377, 0.02199, 0.05142,
           0.09019, 0.05744, 0.02243, 0.03856, 0.05203, 0.07120, 0.05841, 0.01330, 0.03216, 0.06441)
MAX_CELLS = 1.0e11      # of a drawn case

PAIR_FUNCS = ("sw_striped_profile_16", "sw_scan_profile_sat", "nw_scan_profile_16", "sg_striped_profile_32",
              "sg_qx_stats_striped_profile_16", "nw_stats_scan_profile_32", "sw_stats_striped_profile_32")
SEARCH_FUNCS = ("sw_striped_profile_sat", "sw_striped_profile_16", "sw_scan_profile_32", "sg_qx_striped_profile_16",
                "nw_scan_profile_32")
READ_FUNCS = ("nw_stats_striped_16", "nw_stats_scan_16", "sg_qx_stats_striped_16", "sg_qx_stats_scan_16",
              "sg_striped_16", "sw_stats_striped_32")
PROTEIN_FUNCS = ("nw_striped_sat", "nw_scan_32", "sg_stats_striped_32", "sw_striped_sat", "sw_stats_scan_16")
ALL_FUNCS = ("sw_stats_striped_profile_32", "sw_striped_profile_sat", "sw_stats_striped_profile_16")
CIGAR_FUNCS = ("sg_qx_trace_striped_16", "sw_trace_striped_32", "nw_trace_scan_32")


def listed():
    return [
        # the drop-in API as a caller's loop over pairs uses it: one pair per call, score only
        {"name": "pair_sw", "kind": "pair", "func": "sw_striped_profile_16", "qlen": 300, "tlen": 350},
        # the same with statistics: a read or domain placed in a longer target
        {"name": "pair_sg_stats", "kind": "pair", "func": "sg_qx_stats_striped_profile_16", "qlen": 300, "tlen": 332},
        # one protein query against a small set, searched again and again: a recorded plan
        {"name": "plan_1x1k", "kind": "plan", "func": "sw_striped_profile_16", "nq": 1, "qlen": 300, "n": 1000,
         "open": 10, "gap": 1},
        # protein database search, five queries of 100 to 2000 residues, inputs on the device
        {"name": "search_5x200k", "kind": "search", "host": False, "func": "sw_striped_profile_sat", "nq": 5,
         "qlen": 0, "n": 200000, "open": 11, "gap": 1},
        # a query file against a small database, from host memory
        {"name": "search_40x10k", "kind": "search", "host": True, "func": "sw_striped_profile_sat", "nq": 40,
         "qlen": 270, "n": 10000, "open": 11, "gap": 1},
        # a million DNA reads against their windows, global with statistics, inputs on the device
        {"name": "reads_nw_stats_1m", "kind": "reads", "host": False, "func": "nw_stats_striped_16", "n": 1000000,
         "lo": 100, "hi": 300},
        # the same reads semi-global from host memory, a smaller batch
        {"name": "reads_sg_stats_host", "kind": "reads", "host": True, "func": "sg_qx_stats_scan_16", "n": 150000,
         "lo": 100, "hi": 300},
        # homologous protein pairs of all lengths, global score through the 8 -> 16 -> 32 chain
        {"name": "proteins_nw_100k", "kind": "proteins", "host": False, "func": "nw_striped_sat", "n": 100000,
         "median": 270},
        # all against all of a protein set with local statistics
        {"name": "all_vs_all_1k", "kind": "all", "func": "sw_stats_striped_profile_32", "n": 1024, "lo": 50, "hi": 1500},
        # traceback: CIGARs of reads in their windows
        {"name": "cigar_reads_40k", "kind": "cigar", "func": "sg_qx_trace_striped_16", "n": 40000, "lo": 100, "hi": 300},
        # long DNA pairs, full global alignment
        {"name": "long_nw_64", "kind": "long", "n": 64, "lo": 5000, "hi": 50000, "div": 0.08},
        # long DNA pairs in a fixed band
        {"name": "long_banded_256", "kind": "banded", "n": 256, "lo": 5000, "hi": 50000, "div": 0.05, "k": 500},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("pair", "plan", "search", "reads", "proteins", "all", "cigar", "long", "banded"))
    if kind == "pair":
        return {"kind": kind, "func": rng.choice(PAIR_FUNCS), "qlen": _log(rng, 30, 2000), "tlen": _log(rng, 30, 2000)}
    if kind == "plan":
        return {"kind": kind, "func": rng.choice(("sw_striped_profile_16", "sw_striped_profile_sat")),
                "nq": rng.randint(1, 4), "qlen": _log(rng, 50, 1500), "n": _log(rng, 100, 20000), "open": rng.choice((10, 11)),
                "gap": rng.choice((1, 2))}
    if kind == "search":
        case = {"kind": kind, "host": rng.random() < 0.5, "func": rng.choice(SEARCH_FUNCS), "nq": _log(rng, 1, 60),
                "qlen": _log(rng, 80, 1500), "n": _log(rng, 1000, 200000), "open": rng.choice((10, 11, 13)),
                "gap": rng.choice((1, 2))}
    elif kind == "reads":
        lo = _log(rng, 30, 300)
        case = {"kind": kind, "host": rng.random() < 0.5, "func": rng.choice(READ_FUNCS), "n": _log(rng, 2000, 600000),
                "lo": lo, "hi": lo + rng.randint(0, 200)}
    elif kind == "proteins":
        case = {"kind": kind, "host": rng.random() < 0.5, "func": rng.choice(PROTEIN_FUNCS), "n": _log(rng, 2000, 150000),
                "median": _log(rng, 100, 500)}
    elif kind == "all":
        lo = _log(rng, 30, 400)
        case = {"kind": kind, "func": rng.choice(ALL_FUNCS), "n": _log(rng, 60, 1000), "lo": lo,
                "hi": lo + rng.randint(50, 1000)}
    elif kind == "cigar":
        lo = _log(rng, 30, 300)
        case = {"kind": kind, "func": rng.choice(CIGAR_FUNCS), "n": _log(rng, 1000, 40000), "lo": lo,
                "hi": lo + rng.randint(0, 200)}
    elif kind == "long":
        case = {"kind": kind, "n": rng.randint(4, 64), "lo": 1500, "hi": _log(rng, 3000, 50000),
                "div": round(rng.uniform(0.01, 0.15), 3)}
    else:
        case = {"kind": kind, "n": _log(rng, 8, 256), "lo": 1500, "hi": _log(rng, 3000, 50000),
                "div": round(rng.uniform(0.01, 0.10), 3), "k": _log(rng, 50, 1000)}
    while _cells(case) > MAX_CELLS:
        case["n"] = max(1, case["n"] // 2)
    return case


def _mean_lengths(case):
    """Mean query and target lengths of a case."""
    kind = case["kind"]
    if kind == "pair":
        return case["qlen"], case["tlen"]
    if kind == "plan":
        return case["qlen"], 300
    if kind == "search":
        return 770 if case["qlen"] == 0 else case["qlen"], 350
    if kind == "proteins":
        return 1.2 * case["median"], 1.2 * case["median"]
    mid = (case["lo"] + case["hi"]) / 2
    return (mid, mid + 32) if kind in ("reads", "cigar") else (mid, mid)


def _pairs(case):
    kind, n = case["kind"], case.get("n", 1)
    return n * (n - 1) // 2 if kind == "all" else n * case.get("nq", 1)


def _cells(case):
    q, t = _mean_lengths(case)
    if case["kind"] == "banded":
        return case["n"] * q * (2 * case["k"] + 1)
    if case["kind"] == "long":     # uniform lengths: the mean of the square
        return case["n"] * (case["lo"] ** 2 + case["lo"] * case["hi"] + case["hi"] ** 2) / 3
    return _pairs(case) * q * t


def work(case):
    """Sequences once and results once; lane operations per cell: 6 for a
    local score, 5 for a global one, 9 more for the statistics or the path."""
    q, t = _mean_lengths(case)
    kind, n, p = case["kind"], case.get("n", 1), _pairs(case)
    func = case.get("func", "nw")
    seqs = n * q if kind == "all" else case.get("nq", 1) * q + n * t if kind in ("plan", "search") else p * (q + t)
    ops = (6 if func.startswith("sw") else 5) + (9 if "stats" in func or "trace" in func else 0)
    return {"bytes": seqs + p * (4 if kind in ("long", "banded") else 32) + (p * 4 * 20 if kind == "cigar" else 0),
            "flops": _cells(case) * ops}


# ---------------------------------------------------------------------------
# inputs

@functools.lru_cache(None)
def _matrix(name):
    if name == "blosum62":
        return pb.matrix_lookup("blosum62")
    return pb.matrix_create("ACGT", *((2, -3) if name == "dna23" else (1, -2)))


@functools.lru_cache(None)
def _mapper(name):
    return torch.from_numpy(np.ctypeslib.as_array(_matrix(name).contents.mapper, shape=(256,)).astype(np.uint8)).cuda()


class _Gen:
    """Random sequences on the device, as ASCII, from one seed."""

    def __init__(self, seed, protein):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)
        if protein:
            self.cdf = torch.cumsum(torch.tensor(AA_FREQ, device="cuda"), 0)
            self.letters = torch.tensor(list(AA.encode()), dtype=torch.uint8, device="cuda")
        else:
            self.cdf = torch.tensor([0.25, 0.5, 0.75, 1.0], device="cuda")
            self.letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")

    def rand(self, n):
        return torch.rand(n, generator=self.g, device="cuda")

    def residues(self, n):
        k = torch.searchsorted(self.cdf, self.rand(n), out_int32=True).clamp_(max=len(self.letters) - 1)
        return self.letters[k]

    def lengths(self, n, lo, hi):
        return torch.randint(lo, hi + 1, (n,), generator=self.g, device="cuda")

    def lognormal(self, n, median, lo, hi):
        z = torch.randn(n, generator=self.g, device="cuda")
        return torch.exp(math.log(median) + 0.72 * z).round().long().clamp_(lo, hi)

    def mutate(self, seq, lens, sub, indel):
        """Each residue replaced with probability `sub` and dropped or
        followed by a random one with probability indel / 2 each; the first
        residue of a sequence stays."""
        n = seq.numel()
        res = torch.where(self.rand(n) < sub, self.residues(n), seq)
        u = self.rand(n)
        counts = 1 - (u < indel / 2).int() + (u >= 1 - indel / 2).int()
        off = _offsets(lens)
        counts[off] = counts[off].clamp(min=1)
        ends = torch.cumsum(counts, 0, dtype=torch.int64)
        at = torch.repeat_interleave(torch.arange(n, dtype=torch.int32, device="cuda"), counts)
        out = res[at]
        new = torch.zeros(at.numel(), dtype=torch.bool, device="cuda")
        new[1:] = at[1:] == at[:-1]
        out = torch.where(new, self.residues(at.numel()), out)
        last = ends[off + lens - 1]
        return out, torch.diff(last, prepend=last.new_zeros(1))


def _offsets(lens):
    return torch.cumsum(lens, 0) - lens


def _prefixes(seq, lens, keep):
    """The first keep[k] residues of every sequence."""
    o, d = _offsets(lens), _offsets(keep)
    return seq[torch.repeat_interleave(o - d, keep) + torch.arange(int(keep.sum()), device="cuda")]


def _set(seq, lens, mapper, host, off=None):
    """(characters or codes, offsets, lengths), in host or device memory."""
    off = _offsets(lens) if off is None else off
    lens = lens.int()
    if host:
        return seq.cpu().numpy(), off.cpu().numpy(), lens.cpu().numpy()
    return mapper[seq.long()], off.contiguous(), lens.contiguous()


def _ptrs(s):
    return [x.ctypes.data if isinstance(x, np.ndarray) else x.data_ptr() for x in s]


def _records(n, host):
    return np.zeros((n, 8), np.int32) if host else torch.zeros((n, 8), dtype=torch.int32, device="cuda")


def _database(gen, queries, n, median=270.0):
    """Log-normal target lengths, one target in a hundred a homolog of a query
    (30% identity); the homologs stand among the others by their offsets."""
    nh = n // 100
    lens = gen.lognormal(n - nh, median, 20, 5000)
    seq = gen.residues(int(lens.sum()))
    if nh:
        pick = [queries[k % len(queries)] for k in range(nh)]
        hl = torch.tensor([len(p) for p in pick], device="cuda")
        hs, hl = gen.mutate(torch.cat(pick), hl, 0.70, 0.02)
        seq, lens = torch.cat([seq, hs]), torch.cat([lens, hl])
    mix = torch.randperm(n, generator=gen.g, device="cuda")
    return seq, lens[mix], _offsets(lens)[mix]


class _Plan:
    """A recorded database search and the buffers that it uses."""

    def __init__(self, func, profiles, target, n, open_, gap, rec):
        self.keep = (profiles, target, rec)
        arr = pb.ctypes.cast(pb.profile_array(profiles), pb.ctypes.c_void_p)
        self.ptr = pb.lib.parasail_b200_db_plan_create(func.encode(), arr, len(profiles), *_ptrs(target), n, open_,
                                                       gap, rec.data_ptr())
        if not self.ptr:
            raise RuntimeError("parasail_b200_db_plan_create failed")

    def __del__(self):
        if self.ptr and pb.lib is not None:
            pb.lib.parasail_b200_db_plan_free(self.ptr)
        self.ptr = None


def _profiles(func, queries, matrix):
    width = func.rsplit("_", 1)[1]
    creator = "parasail_profile_create_%s%s" % ("stats_" if "_stats" in func else "", width)
    return [pb.ProfileHandle(creator, bytes(q.cpu().numpy()), matrix) for q in queries]


def _one_pair(case, seed):
    """A query and a target that holds a diverged copy of it."""
    gen = _Gen(seed, True)
    q = gen.residues(case["qlen"])
    t, _ = gen.mutate(q, torch.tensor([case["qlen"]], device="cuda"), 0.4, 0.02)
    t = torch.cat([t, gen.residues(case["tlen"])])[:case["tlen"]]
    return bytes(q.cpu().numpy()), bytes(t.cpu().numpy())


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "func": case.get("func"), "n": case.get("n", 1)}
    if kind == "pair":
        q, t = _one_pair(case, seed)
        m = _matrix("blosum62")
        creator = "parasail_profile_create_%s%s" % ("stats_" if "_stats" in case["func"] else "",
                                                    case["func"].rsplit("_", 1)[1])
        state.update(profile=pb.ProfileHandle(creator, q, m), target=t)
    elif kind in ("plan", "search"):
        gen = _Gen(seed, True)
        host = bool(case.get("host"))
        if kind == "plan":
            ql = [case["qlen"]] * case["nq"]
        elif case["qlen"] == 0:
            ql = [(100, 250, 500, 1000, 2000)[k % 5] for k in range(case["nq"])]
        else:
            ql = gen.lognormal(case["nq"], case["qlen"], 20, 3000).tolist()
        queries = [gen.residues(x) for x in ql]
        if kind == "plan":
            lens = gen.lengths(case["n"], 100, 500)
            seq, off = gen.residues(int(lens.sum())), None
        else:
            seq, lens, off = _database(gen, queries, case["n"])
        target = _set(seq, lens, _mapper("blosum62"), host, off)
        profiles = _profiles(case["func"], queries, _matrix("blosum62"))
        rec = _records(len(ql) * case["n"], host)
        state.update(host=host, profiles=profiles, target=target, rec=rec, open=case["open"], gap=case["gap"])
        if kind == "plan":
            state["plan"] = _Plan(case["func"], profiles, target, case["n"], case["open"], case["gap"], rec)
        else:
            state["array"] = pb.profile_array(profiles)
    elif kind in ("reads", "cigar"):
        gen = _Gen(seed, False)
        host = kind == "cigar" or case["host"]
        rl = gen.lengths(case["n"], case["lo"], case["hi"])
        windows = gen.residues(int((rl + 32).sum()))
        reads, ql = gen.mutate(_prefixes(windows, rl + 32, rl), rl, 0.05, 0.01)
        m = _mapper("dna23")
        state.update(host=host, q=_set(reads, ql, m, host), t=_set(windows, rl + 32, m, host), matrix=_matrix("dna23"),
                     rec=_records(case["n"], host), open=5, gap=2)
        if kind == "cigar":
            # room for the longest reads (an inserted residue at most per twenty) and their windows
            state["cigars"] = np.zeros(case["n"] * (2 * case["hi"] + case["hi"] // 20 + 64), np.uint32)
            assert int((ql + rl + 32).sum()) <= len(state["cigars"])
            state["more"] = [np.zeros(case["n"], np.int32) for _ in range(3)]
    elif kind == "proteins":
        gen = _Gen(seed, True)
        lens = gen.lognormal(case["n"], case["median"], 20, 2000)
        a = gen.residues(int(lens.sum()))
        b, bl = gen.mutate(a, lens, 0.5, 0.04)
        m = _mapper("blosum62")
        state.update(host=case["host"], q=_set(a, lens, m, case["host"]), t=_set(b, bl, m, case["host"]),
                     matrix=_matrix("blosum62"), rec=_records(case["n"], case["host"]), open=11, gap=1)
    elif kind == "all":
        # one sequence in five a diverged copy (40% identity) of another
        gen = _Gen(seed, True)
        n, nf = case["n"], case["n"] // 5
        lens = gen.lengths(n - nf, case["lo"], case["hi"])
        seq = gen.residues(int(lens.sum()))
        fam = torch.randint(0, max(1, (n - nf) // 16), (nf,), generator=gen.g, device="cuda")
        off = _offsets(lens)
        src = torch.cat([seq[off[f]:off[f] + lens[f]] for f in fam.tolist()]) if nf else seq[:0]
        if nf:
            hs, hl = gen.mutate(src, lens[fam], 0.6, 0.03)
            seq, lens = torch.cat([seq, hs]), torch.cat([lens, hl])
        mix = torch.randperm(n, generator=gen.g, device="cuda")
        state.update(t=_set(seq, lens[mix], _mapper("blosum62"), False, _offsets(lens)[mix]),
                     matrix=_matrix("blosum62"), rec=_records(n * (n - 1) // 2, False), open=11, gap=1)
    else:
        gen = _Gen(seed, False)
        lens = gen.lengths(case["n"], case["lo"], case["hi"])
        a = gen.residues(int(lens.sum()))
        b, bl = gen.mutate(a, lens, 0.7 * case["div"] * 4 / 3, 0.3 * case["div"])
        m = _mapper("dna12")
        state.update(q=_set(a, lens, m, True), t=_set(b, bl, m, True), matrix=_matrix("dna12"), open=4, gap=1,
                     scores=np.zeros(case["n"], np.int32), k=case.get("k", 0))
    return state


def _check(rc):
    if rc != 0:
        raise RuntimeError("the call failed")


def run(s):
    kind, lib = s["kind"], pb.lib
    if kind == "pair":
        return pb.align_profile("parasail_" + s["func"], s["profile"], s["target"], 11, 1)
    if kind == "plan":
        _check(lib.parasail_b200_db_plan_run(s["plan"].ptr))
        return s["rec"]
    if kind == "search":
        call = lib.parasail_b200_batch_db if s["host"] else lib.parasail_b200_batch_db_device
        _check(call(s["func"].encode(), pb.ctypes.cast(s["array"], pb.ctypes.c_void_p), len(s["profiles"]),
                    *_ptrs(s["target"]), s["n"], s["open"], s["gap"], *_ptrs([s["rec"]])))
        return s["rec"]
    if kind in ("reads", "proteins"):
        call = lib.parasail_b200_batch_pairs if s["host"] else lib.parasail_b200_batch_pairs_device
        _check(call(s["func"].encode(), s["matrix"], *_ptrs(s["q"]), *_ptrs(s["t"]), s["n"], s["open"], s["gap"],
                    *_ptrs([s["rec"]])))
        return s["rec"]
    if kind == "all":
        _check(lib.parasail_b200_batch_all_device(s["func"].encode(), s["matrix"], *_ptrs(s["t"]), s["n"], s["open"],
                                                  s["gap"], *_ptrs([s["rec"]])))
        return s["rec"]
    if kind == "cigar":
        _check(lib.parasail_b200_batch_pairs_cigar(s["func"].encode(), s["matrix"], *_ptrs(s["q"]), *_ptrs(s["t"]),
                                                   s["n"], s["open"], s["gap"],
                                                   *_ptrs([s["rec"], s["cigars"]] + s["more"])))
        return [s["rec"], s["cigars"].view(np.int32)] + s["more"]
    if kind == "long":
        _check(lib.parasail_b200_nw_long(s["matrix"], *_ptrs(s["q"]), *_ptrs(s["t"]), s["n"], s["open"], s["gap"],
                                         *_ptrs([s["scores"]])))
        return s["scores"]
    _check(lib.parasail_b200_nw_banded_batch(s["matrix"], *_ptrs(s["q"]), *_ptrs(s["t"]), s["n"], s["open"], s["gap"],
                                             s["k"], *_ptrs([s["scores"]])))
    return s["scores"]


def exact(case, seed):
    """Score and end of the one-pair local and global calls by a row-wise
    64-bit dynamic program; results of whole numbers elsewhere need none."""
    if case["kind"] != "pair" or case["func"].startswith("sg") or "stats" in case["func"]:
        return None
    local = case["func"].startswith("sw")
    q, t = _one_pair(case, seed)
    m = _matrix("blosum62").contents
    table = np.ctypeslib.as_array(m.matrix, shape=(m.size * m.size,)).reshape(m.size, m.size).astype(np.int64)
    mapper = np.ctypeslib.as_array(m.mapper, shape=(256,))
    qc, tc = mapper[list(q)], mapper[list(t)]
    n, open_, gap, none = len(t), 11, 1, -(1 << 40)
    cols = np.arange(n + 1, dtype=np.int64)
    h = np.zeros(n + 1, np.int64) if local else np.where(cols > 0, -open_ - (cols - 1) * gap, 0)
    f = np.full(n + 1, none, np.int64)
    best, ends = (0, (0, 0)), {}
    for i, c in enumerate(qc):
        f = np.maximum(f - gap, h - open_)
        d = np.full(n + 1, none, np.int64)
        d[1:] = np.maximum(h[:-1] + table[tc, c], f[1:])
        d[0] = 0 if local else -open_ - i * gap
        if local:
            d = np.maximum(d, 0)
        # E(j) = max over k < j of d(k) - open - (j - k - 1) gap
        run_max = np.maximum.accumulate(d + gap * cols)
        h = d.copy()
        h[1:] = np.maximum(d[1:], run_max[:-1] - open_ - (cols[1:] - 1) * gap)
        if local:
            top = int(h.max())
            if top > 0:
                ends.setdefault(top, []).append((int(h.argmax()) - 1, i))
                best = max(best, (top, (0, 0)))
    if not local:
        return {"score": int(h[-1]), "end_query": len(q) - 1, "end_ref": n - 1, "flag": None}
    if best[0] == 0:
        return {"score": 0, "end_query": 0, "end_ref": 0, "flag": None}
    j, i = min(ends[best[0]])      # the first column with the maximum, then the first row
    return {"score": best[0], "end_query": i, "end_ref": j, "flag": None}
