"""Performance cases of the string sorter: calls that programs make through its
public entry points (pssgpu_sort_device, pssgpu_sort_batch_device,
pssgpu_merge_lcp_device, pssgpu_sort_host), with the shapes of this
repository's workloads (workloads.py, serving.py, bench.py), from the smallest
serving request to the 64 Mi-string sort.

Kinds of cases:
  sort    one device-resident arena of random strings; equal strings occur as
          they do in such data, so the permutation is applied to a column of
          64-bit codes of the strings (what a program that sorts rows by a
          string key does with it) and that column is returned
  prefix  strings behind 4096 Zipf-distributed 48-char prefixes
  dna     all suffixes of an ACGT text with copied blocks
  batch   many independent instances in one call
  merge   sorted shards with LCP arrays into one sorted sequence
  host    pinned host arena in, permutation and LCPs back in pinned memory
"""
import importlib
import math

import numpy as np
import torch

pss = importlib.import_module("parallel-string-sorting_b200")

MI = 1 << 20
PAD = 16
ALPHABETS = {4: b"ACGT", 10: b"0123456789", 26: b"abcdefghijklmnopqrstuvwxyz", 95: bytes(range(32, 127))}
CHUNK_CHARS = 256 * MI  # chars generated at once


def listed():
    return [
        # A near-minimal serving request (the stream's requests start at 1 KB;
        # this one has about 10 KB): launches and round trips are all there is.
        {"name": "request_10KB", "kind": "sort", "n": 311, "alphabet": 95, "lmin": 1, "lmax": 64, "lcp": True},
        # The stream's median request, 256 KB (sizes are log-uniform, 1 KB to 64 MB).
        {"name": "request_256KB", "kind": "sort", "n": 7801, "alphabet": 26, "lmin": 1, "lmax": 64, "lcp": False},
        # psstest's random10: 10 MiB of digit strings, plain sort.
        {"name": "digits_10MB", "kind": "sort", "n": 487463, "alphabet": 10, "lmin": 1, "lmax": 40, "lcp": False},
        # The stream's largest request, 64 MB, over its smallest alphabet, with LCPs.
        {"name": "request_64MB", "kind": "sort", "n": 1953125, "alphabet": 4, "lmin": 1, "lmax": 64, "lcp": True},
        # High-LCP strings with LCP output at an ordinary, ragged size.
        {"name": "prefix_4M_lcp", "kind": "prefix", "n": 4194301, "lcp": True},
        # The headline sort: 64 Mi strings, 4.36 GB of chars.
        {"name": "prefix_64M", "kind": "prefix", "n": 64 * MI, "lcp": False},
        # Suffix array with LCP array of a text of an odd, smaller size.
        {"name": "dna_5M_lcp", "kind": "dna", "text": 5000001, "lcp": True},
        # Suffix array of the 32 MiB text.
        {"name": "dna_32M", "kind": "dna", "text": 32 * MI, "lcp": False},
        # A server's batch: some hundred requests of mixed sizes, with LCPs.
        {"name": "batch_613", "kind": "batch", "ninst": 613, "smin": 16, "smax": 65536, "chars": 128 * MI, "lcp": True},
        # 100k instances, 1 GiB of chars.
        {"name": "batch_100k", "kind": "batch", "ninst": 100000, "smin": 16, "smax": MI, "chars": 1024 * MI, "lcp": False},
        # Merge of eight sorted shards with their LCP arrays.
        {"name": "merge_8x2M", "kind": "merge", "n": 16 * MI, "runs": 8},
        # End to end from host memory, as a psstest contestant is called.
        {"name": "host_1.5M_lcp", "kind": "host", "n": 1500007, "lcp": True},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["sort", "sort", "sort", "prefix", "dna", "batch", "merge", "host"])
    lcp = rng.random() < 0.5
    if kind == "sort":
        return {"kind": kind, "n": log(64, 4 * MI), "alphabet": rng.choice(sorted(ALPHABETS)), "lmin": 1,
                "lmax": rng.choice([24, 40, 64]), "lcp": lcp}
    if kind == "prefix":
        return {"kind": kind, "n": log(100000, 48 * MI), "lcp": lcp}
    if kind == "dna":
        return {"kind": kind, "text": log(MI, 32 * MI), "lcp": lcp}
    if kind == "batch":
        ninst = log(100, 100000)
        return {"kind": kind, "ninst": ninst, "smin": 16, "smax": log(1024, MI),
                "chars": min(1024 * MI, max(8 * MI, ninst * 32768)), "lcp": lcp}
    if kind == "merge":
        return {"kind": kind, "n": log(MI, 16 * MI), "runs": rng.randint(2, 16)}
    return {"kind": kind, "n": log(100000, 4 * MI), "lcp": lcp}


class Strings:
    """A device arena of random strings of the given lengths. Each string is a
    prefix from a table (prefix_of: its row per string; no table: none) and
    random chars of the alphabet; code[i] is a 64-bit code of string i (and of
    group[i], when given) that equal strings share."""

    def __init__(self, gen, lens, alphabet, table=None, prefix_of=None, group=None):
        self.gen, self.lens, self.table, self.prefix_of, self.group = gen, lens, table, prefix_of, group
        self.alphabet = torch.tensor(list(alphabet), dtype=torch.uint8, device="cuda")
        ends = torch.cumsum(lens + 1, 0)
        self.offs = ends - (lens + 1)
        self.nchars = int(ends[-1])
        self.chars = torch.zeros(self.nchars + PAD, dtype=torch.uint8, device="cuda")
        self.code = torch.empty_like(lens)
        weights = np.random.RandomState(7).randint(-2 ** 62, 2 ** 62, 1024, dtype=np.int64) * 2 + 1
        self.weights = torch.from_numpy(weights).cuda()
        n, step = lens.numel(), max(1, CHUNK_CHARS * lens.numel() // self.nchars)
        for i in range(0, n, step):
            self.write(torch.arange(i, min(i + step, n), device="cuda"))

    def write(self, ids):
        lens = self.lens[ids]
        ends = torch.cumsum(lens + 1, 0)
        row = torch.repeat_interleave(torch.arange(ids.numel(), device="cuda"), lens + 1)
        pos = torch.arange(row.numel(), device="cuda") - (ends - lens - 1)[row]
        ch = self.alphabet[torch.randint(self.alphabet.numel(), (row.numel(),), generator=self.gen, device="cuda",
                                         dtype=torch.int32)]
        if self.table is not None:
            width = self.table.shape[1]
            fixed = self.table.reshape(-1)[self.prefix_of[ids][row] * width + pos.clamp(max=width - 1)]
            ch = torch.where(pos < width, fixed, ch)
        ch[ends - 1] = 0
        self.chars[self.offs[ids][row] + pos] = ch
        total = torch.cumsum(ch.to(torch.int64) * self.weights[pos], 0)[ends - 1]
        code = total.clone()
        code[1:] -= total[:-1]
        self.code[ids] = code if self.group is None else code + self.group[ids] * int(self.weights[1000])

    def make_distinct(self):
        """Draws strings again until no two (of one group) are equal, so that
        one permutation alone is the sorted one."""
        while True:
            code, idx = torch.sort(self.code)
            again = idx[1:][code[1:] == code[:-1]]
            if not again.numel():
                return self
            self.write(again)


def generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def prefix_strings(n, seed):
    """Zipf (s = 1.1) choice of 4096 48-char prefixes, suffixes of length U[8, 24]."""
    gen = generator(seed)
    table = torch.randint(97, 123, (4096, 48), generator=gen, device="cuda", dtype=torch.uint8)
    cdf = torch.cumsum(torch.arange(1, 4097, device="cuda", dtype=torch.float64) ** -1.1, 0)
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * cdf[-1]
    which = torch.searchsorted(cdf, u).clamp_(max=4095)
    del u
    lens = torch.randint(56, 73, (n,), generator=gen, device="cuda")
    return Strings(gen, lens, ALPHABETS[26], table, which).make_distinct()


def dna(length, seed):
    """A uniform ACGT text, 5% of it overwritten by copies of earlier blocks of 1 to 10 KiB."""
    gen = generator(seed)
    acgt = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")
    chars = torch.zeros(length + 1 + PAD, dtype=torch.uint8, device="cuda")
    chars[:length] = acgt[torch.randint(4, (length,), generator=gen, device="cuda")]
    rng, written = np.random.RandomState(seed % (1 << 32)), 0
    while written < length // 20:
        size = 1024 + rng.randint(9 * 1024 + 1)
        dst = size + rng.randint(length - 2 * size)
        src = rng.randint(dst - size + 1)
        chars[dst:dst + size] = chars[src:src + size].clone()
        written += size
    return chars, torch.arange(length + 1, device="cuda")


def batch_sizes(case):
    """Instance sizes, log-uniform (its quantiles) and scaled to the case's
    chars (23.8 a string), in ascending order."""
    n = case["ninst"]
    u = (np.arange(n) + 0.5) / n
    raw = np.exp(np.log(case["smin"]) + u * np.log(case["smax"] / case["smin"]))
    lo, hi = 0.0, 1.0
    if np.maximum(case["smin"], raw).sum() * 23.8 > case["chars"]:
        for _ in range(40):
            mid = (lo + hi) / 2
            lo, hi = (mid, hi) if np.maximum(case["smin"], raw * mid).sum() * 23.8 <= case["chars"] else (lo, mid)
    else:
        lo = 1.0
    return np.maximum(case["smin"], np.floor(raw * lo)).astype(np.int64)


def results(n, lcp):
    """The buffers a program hands to the call: permutation and, if wanted, LCPs."""
    perm = torch.zeros(n, dtype=torch.int32, device="cuda")
    return perm, torch.zeros(n, dtype=torch.int32, device="cuda") if lcp else None


def prepare(case, seed):
    ctx = pss.default_context()
    kind = case["kind"]
    state = {"kind": kind, "ctx": ctx}
    if kind == "sort":
        gen = generator(seed)
        lens = torch.randint(case["lmin"], case["lmax"] + 1, (case["n"],), generator=gen, device="cuda")
        s = Strings(gen, lens, ALPHABETS[case["alphabet"]])
        state["code"], state["sorted_code"] = s.code, torch.empty_like(s.code)
    elif kind in ("prefix", "merge", "host"):
        s = prefix_strings(case["n"], seed)
    elif kind == "batch":
        sizes = np.random.RandomState(seed % (1 << 32)).permutation(batch_sizes(case))
        inst = np.zeros(case["ninst"] + 1, dtype=np.uint64)
        np.cumsum(sizes, out=inst[1:])
        gen = generator(seed)
        n = int(inst[-1])
        lens = torch.exp(torch.randn(n, generator=gen, device="cuda") * 0.5 + 3.0).round_().clamp_(1, 256).to(torch.int64)
        group = torch.repeat_interleave(torch.arange(case["ninst"], device="cuda"), torch.from_numpy(sizes).cuda())
        s = Strings(gen, lens, ALPHABETS[95], group=group).make_distinct()
        state["inst"] = inst
    if kind == "dna":
        state["chars"], state["offs"] = dna(case["text"], seed)
        state["nchars"] = case["text"] + 1
    else:
        state["chars"], state["offs"], state["nchars"] = s.chars, s.offs, s.nchars
    n = state["offs"].numel()
    if kind == "host":
        for name in ("chars", "offs"):
            state[name] = state[name].cpu().pin_memory().numpy()
        state["chars"] = state["chars"][:state["nchars"]]
        state["offs"] = state["offs"].view(np.uint64)
        state["perm"] = torch.zeros(n, dtype=torch.int32).pin_memory().numpy().view(np.uint32)
        state["lcp"] = torch.zeros(n, dtype=torch.int32).pin_memory().numpy().view(np.uint32) if case["lcp"] else None
        return state
    state["perm"], state["lcp"] = results(n, kind == "merge" or case["lcp"])
    if kind == "merge":
        # shards as the sorter leaves them: ids of the whole arena, in order, with LCPs
        runs = np.array([n * k // case["runs"] for k in range(case["runs"] + 1)], dtype=np.uint64)
        ids, lcps = results(n, True)
        torch.cuda.synchronize()
        for a, b in zip(runs[:-1].tolist(), runs[1:].tolist()):
            ctx.sort_device(state["chars"], state["nchars"], state["offs"][a:b], ids[a:b], lcps[a:b])
            ids[a:b] += a
        state["runs"], state["ids"], state["lcps"] = runs, ids, lcps
    return state


def run(state):
    ctx, kind = state["ctx"], state["kind"]
    if kind == "host":
        ctx.sort_host(state["chars"], state["offs"], lcp=state["lcp"] is not None, out_perm=state["perm"],
                      out_lcp=state["lcp"])
    elif kind == "batch":
        ctx.sort_batch_device(state["chars"], state["nchars"], state["offs"], state["inst"], state["perm"], state["lcp"])
    elif kind == "merge":
        ctx.merge_lcp_device(state["chars"], state["nchars"], state["offs"], state["runs"], state["ids"], state["lcps"],
                             state["perm"], state["lcp"])
    else:
        ctx.sort_device(state["chars"], state["nchars"], state["offs"], state["perm"], state["lcp"])
    out = {}
    if kind == "sort":
        out["code"] = torch.index_select(state["code"], 0, state["perm"], out=state["sorted_code"])
    else:
        out["perm"] = state["perm"].view(np.int32) if kind == "host" else state["perm"]
    if state["lcp"] is not None:
        out["lcp"] = state["lcp"].view(np.int32) if kind == "host" else state["lcp"]
    return out


def work(case):
    """Arena and offsets read once, permutation (and LCPs) written once; the
    merge reads ids, LCPs, offsets and the 8 chars at each string's LCP."""
    kind = case["kind"]
    if kind == "merge":
        return {"bytes": case["n"] * (4 + 4 + 8 + 8 + 8), "flops": 0}
    if kind == "dna":
        n = chars = case["text"] + 1
    elif kind == "batch":
        n = int(batch_sizes(case).sum())
        chars = n * 23.8
    elif kind == "sort":
        n = case["n"]
        chars = n * ((case["lmin"] + case["lmax"]) / 2 + 1)
    else:
        n = case["n"]
        chars = n * 65
    out = 4 + (4 if case["lcp"] else 0) + (16 if kind == "sort" else 0)
    return {"bytes": chars + n * (8 + out), "flops": 0}
