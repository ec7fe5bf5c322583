"""The work a user of gkc_b200 has it do, as timed cases.

Every case goes through the public Python entry points (thin calls over the
C ABI).  A state holds what a counting program keeps between calls: its
context, the reads in HBM (or in page-locked host memory for the host forms)
and result buffers of its own, larger than the results (the rest of them
stays zero).  All outputs are integers and are the same from run to run, so
there are no 64-bit values to compare them with.

Read sources (the generators of the library, seeded):
  genome  fixed-length reads of a random genome at a given coverage, 0.5%
          substitutions (sequencing data: most k-mers seen many times)
  iid     uniform random reads with 0.1% N (every k-mer distinct)
  long    lognormal read lengths (median 8 kbp, 1-50 kbp), 5% errors with
          insertions and deletions (mostly distinct k-mers, ragged reads)
"""
import ctypes
import math

import numpy as np
import torch

import gkc_b200 as G
from gkc_b200 import shard


def listed():
    return [
        # the smallest counting job a server gets (1e5 bases): launches and latency
        case("job_100k", "pipeline", "genome", 100_050, 31, 11, 256),
        # small random reads with N: every k-mer distinct, superkmers cut by N
        case("iid_n_3m", "pipeline", "iid", 3_000_000, 31, 11, 256),
        # short-read sequencing of a genome at 30x: the main use, and the largest case
        case("short_k31_900m", "pipeline", "genome", 900_000_000, 31, 11, 256),
        # long reads, homopolymer-compressed, short minimizer windows
        case("long_hpc_k25_200m", "pipeline", "long", 200_000_000, 25, 15, 256, coverage=20, hpc=True),
        # a bacterial genome in long reads with the reference's defaults (k 21, p 7, 31 bins)
        case("default_k21_135m", "pipeline", "long", 135_000_000, 21, 7, 31, coverage=29),
        # long k-mers: 16-byte keys
        case("k63_150m", "pipeline", "genome", 150_000_000, 63, 13, 256, read_len=250),
        # the merged list without k-mers seen once, copied to the host (what a database or an assembler reads)
        case("merged_min2_60m", "merged", "genome", 60_000_000, 31, 11, 256),
        # bin sharding over two ranks: partition, superkmer exchange, owned bins counted
        case("shard2_120m", "shard", "genome", 120_000_000, 31, 11, 256),
        # (minimizer, position, strand) of every window, for an index
        case("minimizers_k25_100m", "minimizers", "long", 100_000_000, 25, 15, 256, coverage=20),
        # position lists of the quarter of the k-mers that a sketch keeps
        case("subsample_k63_75m", "subsample", "genome", 75_000_000, 63, 13, 256, read_len=250),
        # one bin's superkmers from host memory: the call of a program that keeps its own superkmer store
        case("host_bin_1m", "host_bin", "genome", 20_000_000, 31, 11, 1),
        # batches streamed from page-locked host memory, results back to it
        case("stream_4x20m", "stream", "genome", 80_000_000, 31, 11, 256, batches=4),
    ]


def case(name, kind, source, bases, k, p, nbins, coverage=30, read_len=150, hpc=False, batches=1):
    return {"name": name, "kind": kind, "source": source, "bases": bases, "k": k, "p": p, "nbins": nbins,
            "coverage": coverage, "read_len": read_len, "hpc": hpc, "batches": batches}


def draw(rng):
    """Another case of the same ranges: any k and p, odd read lengths and bin
    counts, sizes spread over their logarithm."""
    kind = rng.choice(("pipeline",) * 6 + ("merged", "shard", "minimizers", "subsample", "host_bin", "stream"))
    source = rng.choice(("genome", "genome", "iid", "long"))
    k = rng.choice((rng.randint(17, 32), 21, 25, 31, rng.randint(33, 64)))
    if kind == "host_bin" or kind == "stream":
        source, k = "genome", min(k, 32)
    p = rng.randint(7, min(16, k - 4))
    most = {"pipeline": 200e6, "merged": 60e6, "shard": 120e6, "minimizers": 50e6, "subsample": 50e6,
            "host_bin": 20e6, "stream": 80e6}[kind]
    bases = int(math.exp(rng.uniform(math.log(1e5), math.log(most))))
    c = case("", kind, source, bases, k, p, rng.choice((31, 64, 100, 256, 256, 512, 1000)),
             coverage=rng.choice((5, 20, 30, 60)), read_len=rng.choice((100, 151, 250, rng.randint(80, 300))),
             hpc=kind == "pipeline" and rng.random() < 0.25, batches=rng.randint(2, 5) if kind == "stream" else 1)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs

def genome_of(case, seed):
    n = max(2000, case["bases"] // case["coverage"])
    g = torch.empty(n, dtype=torch.uint8, device="cuda")
    check(G.lib().gkc_synth_genome(1, seed, n, 0.05, 0.01, g.data_ptr()))
    return g


def check(status):
    if status != 0:
        raise G.GkcError(status, "generator")


def reads_of(case, seed):
    """(reads, offsets, number of reads) on the device."""
    L = G.lib()
    if case["source"] == "long":
        g = genome_of(case, seed)
        cap = case["bases"] // 1000 + 64
        host = np.zeros(cap + 1, np.uint64)
        longest = min(50_000, g.numel() // 2)
        n = L.gkc_synth_long_read_offsets(seed, min(8000.0, longest / 2), 0.5, min(1000, longest), longest,
                                          case["bases"], cap, host.ctypes.data)
        offs = torch.from_numpy(host[:n + 1].view(np.int64).copy()).cuda()
        reads = torch.empty(int(host[n]), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        check(L.gkc_synth_long_reads(1, seed, g.data_ptr(), g.numel(), n, offs.data_ptr(), reads.data_ptr()))
        return reads, offs, n
    n, length = max(1, case["bases"] // case["read_len"]), case["read_len"]
    reads = torch.empty(n * length, dtype=torch.uint8, device="cuda")
    offs = torch.empty(n + 1, dtype=torch.int64, device="cuda")
    if case["source"] == "iid":
        check(L.gkc_synth_iid_reads(1, seed, n, length, 0.001, reads.data_ptr(), offs.data_ptr()))
    else:
        g = genome_of(case, seed)
        check(L.gkc_synth_short_reads(1, seed, g.data_ptr(), g.numel(), 0, n, length, 0.005, reads.data_ptr(),
                                      offs.data_ptr()))
    return reads, offs, n


def host_superkmers(case, seed):
    """One bin's superkmers as a store holds them: lengths, and each one's
    bases packed four to a byte, back to back.  They are cut from a genome at
    random places on both strands, with k .. 2k - p bases each."""
    r = np.random.default_rng(seed)
    k, n = case["k"], max(1, case["bases"] // 20)
    genome = r.integers(0, 4, max(2000, case["bases"] // case["coverage"]), dtype=np.uint8)
    lens = r.integers(k, 2 * k - case["p"] + 1, n).astype(np.uint32)
    nbytes = (lens + 3) // 4
    first = np.concatenate([[0], np.cumsum(nbytes.astype(np.int64))])
    start = r.integers(0, len(genome) - 2 * k, n)
    step = np.where(r.random(n) < 0.5, 1, -1)  # backwards and complemented: the other strand
    origin = np.where(step > 0, start, start + lens - 1)
    own = np.repeat(np.arange(n), nbytes)
    q = np.arange(int(first[-1])) - first[own]
    packed = np.zeros(len(own), np.uint8)
    for t in range(4):
        j = 4 * q + t
        inside = j < lens[own]
        at = np.where(inside, origin[own] + step[own] * j, 0)
        code = np.where(step[own] > 0, genome[at], 3 - genome[at])
        packed |= np.where(inside, code << (6 - 2 * t), 0).astype(np.uint8)
    return lens, packed


def expected_distinct(case, bases):
    """(distinct k-mers, k-mers) of so many bases, from the genome size and
    the error rate."""
    k = case["k"]
    reads = bases // (8000 if case["source"] == "long" else case["read_len"])
    kmers = max(0, bases - reads * (k - 1))
    new = {"iid": 1.0, "genome": 1 - 0.995 ** k, "long": 1 - 0.95 ** k}[case["source"]]
    genome = 0 if case["source"] == "iid" else max(2000, case["bases"] // case["coverage"])
    return min(kmers, genome + new * kmers), kmers


def room_for(case, bases):
    """Entries of a result buffer: what a program expects and a quarter more."""
    if case["source"] != "genome":
        return bases + 60_000
    return int(1.25 * expected_distinct(case, bases)[0]) + 20_000


def device_result(room, nbins, words):
    return {"bin_off": torch.zeros(nbins + 1, dtype=torch.int64, device="cuda"),
            "keys": torch.zeros(room * words, dtype=torch.int64, device="cuda"),
            "counts": torch.zeros(room, dtype=torch.int32, device="cuda")}


def host_result(room, nbins, words):
    return {"bin_off": torch.zeros(nbins + 1, dtype=torch.int64).pin_memory(),
            "keys": torch.zeros(room * words, dtype=torch.int64).pin_memory(),
            "counts": torch.zeros(room, dtype=torch.int32).pin_memory()}


def prepare(case, seed):
    kind, words = case["kind"], 1 if case["k"] <= 32 else 2
    s = {"kind": kind, "prm": G.params(case["k"], case["p"], case["nbins"], case["hpc"]), "ctx": G.Context(0)}
    if kind == "host_bin":
        s["k"] = case["k"]
        s["lens"], s["packed"] = host_superkmers(case, seed)
        s["out"] = host_result(max(2000, case["bases"] // case["coverage"]), 1, 1)
        return s
    reads, offs, n = reads_of(case, seed)
    s.update(reads=reads, offs=offs, n=n)
    room = room_for(case, case["bases"])
    if kind == "pipeline":
        s["out"] = device_result(room, case["nbins"], words)
    elif kind == "merged":
        s["out"] = host_result(room, 1, words)
    elif kind == "shard":  # each rank has a context and half of the reads
        half = n // 2
        cut = int(offs[half])
        s["ranks"] = []
        for r, (part, o, m) in enumerate(((reads[:cut], offs[:half + 1], half), (reads[cut:], offs[half:] - cut, n - half))):
            ctx = G.Context(0) if r else s["ctx"]
            nbins = int(shard.owner_bounds(case["nbins"], 2)[r + 1]) - int(shard.owner_bounds(case["nbins"], 2)[r])
            s["ranks"].append((ctx, part.clone(), o.clone(), m, device_result(room * 4 // 5, nbins, words)))
    elif kind == "minimizers":
        s["out"] = {"mm": torch.zeros(case["bases"] + 60_000, dtype=torch.int32, device="cuda"),
                    "pos": torch.zeros(case["bases"] + 60_000, dtype=torch.uint8, device="cuda"),
                    "strand": torch.zeros(case["bases"] + 60_000, dtype=torch.int8, device="cuda")}
    elif kind == "subsample":
        s["out"] = {"keys": torch.zeros((case["bases"] // 2 + 30_000) * words, dtype=torch.int64, device="cuda"),
                    "pos_off": torch.zeros(case["bases"] // 2 + 30_000, dtype=torch.int64, device="cuda"),
                    "positions": torch.zeros(case["bases"] // 2 + 30_000, dtype=torch.int32, device="cuda")}
    elif kind == "stream":
        # the reads in page-locked host memory, one output set per batch
        h_reads, h_offs = reads.cpu().pin_memory(), offs.cpu()
        s["batches"] = []
        for b in range(case["batches"]):
            lo, hi = n * b // case["batches"], n * (b + 1) // case["batches"]
            o = (h_offs[lo:hi + 1] - h_offs[lo]).pin_memory()
            part = h_reads[int(h_offs[lo]):int(h_offs[hi])]
            s["batches"].append((part, o, hi - lo, host_result(room_for(case, part.numel()), case["nbins"], 1)))
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------- run

def copy_out(ctx, out):
    """The context's count result into the program's buffers (device or
    page-locked host memory)."""
    ctx._check(ctx._L.gkc_count_copy_out(ctx.h, out["bin_off"].data_ptr(), out["keys"].data_ptr(),
                                         out["counts"].data_ptr()), "count_copy_out")
    return out


def fits(n, out):
    if n > out["counts"].numel():
        raise ValueError(f"{n} k-mers do not fit the result buffers")


class Array:
    """A device array of the library, for torch.as_tensor (no copy)."""

    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": (int(n),), "typestr": typestr,
                                         "version": 3}


def take(out, ptr, n, typestr):
    out[:n].copy_(torch.as_tensor(Array(ptr, n, typestr), device="cuda"))


def run(s):
    return RUN[s["kind"]](s)


def run_pipeline(s):
    _, cv = s["ctx"].pipeline_device(s["reads"], s["reads"].numel(), s["offs"], s["n"], s["prm"])
    fits(cv.n_distinct, s["out"])
    return {"n": int(cv.n_distinct), **copy_out(s["ctx"], s["out"])}


def run_merged(s):
    ctx, out = s["ctx"], s["out"]
    ctx.pipeline_device(s["reads"], s["reads"].numel(), s["offs"], s["n"], s["prm"])
    n = ctypes.c_uint64()
    most = 0xFFFFFFFF
    ctx._check(ctx._L.gkc_count_output(ctx.h, 2, most, 1, ctypes.byref(n), None, None, None), "count_output")
    fits(n.value, out)
    ctx._check(ctx._L.gkc_count_output(ctx.h, 2, most, 1, ctypes.byref(n), out["bin_off"].data_ptr(),
                                       out["keys"].data_ptr(), out["counts"].data_ptr()), "count_output")
    return {"n": int(n.value), **out}


def run_shard(s):
    engines = []
    for ctx, reads, offs, n, _ in s["ranks"]:
        view = ctx.partition_device(reads, reads.numel(), offs, n, s["prm"])
        engines.append(shard.DeviceEngine(ctx, view))
    _, local = shard.exchange_local(engines, s["prm"])
    result = []
    for (ctx, _, _, _, out), prm in zip(s["ranks"], local):
        cv = ctx.count_device(prm)
        fits(cv.n_distinct, out)
        result.append({"n": int(cv.n_distinct), **copy_out(ctx, out)})
    return result


def run_minimizers(s):
    out = s["out"]
    s["ctx"].minimizers_device(s["reads"], s["reads"].numel(), s["offs"], s["n"], s["prm"], out["mm"], out["pos"],
                               out["strand"])
    return out


def run_subsample(s):
    out = s["out"]
    v = s["ctx"].subsample_positions_device(s["reads"], s["reads"].numel(), s["offs"], s["n"], s["prm"], 4)
    if v.n_positions >= out["positions"].numel():
        raise ValueError("the positions do not fit the result buffers")
    if v.n_positions:
        take(out["keys"], v.keys, v.n_distinct * v.key_words, "<i8")
        take(out["pos_off"], v.pos_off, v.n_distinct + 1, "<i8")
        take(out["positions"], v.positions, v.n_positions, "<i4")
    torch.cuda.current_stream().synchronize()  # the library's arrays are free for the next call
    return {"n": int(v.n_distinct), **out}


def run_host_bin(s):
    n = s["ctx"].count_superkmers_host(s["k"], s["lens"], s["packed"])
    fits(n, s["out"])
    return {"n": n, **copy_out(s["ctx"], s["out"])}


def run_stream(s):
    ctx, tickets, found = s["ctx"], [], []
    for i, (reads, offs, n, out) in enumerate(s["batches"]):
        if i >= 2:
            found.append(ctx.stream_wait(tickets[i - 2])[0])
        tickets.append(ctx.stream_submit(reads, offs, n, s["prm"], out["bin_off"], out["keys"], out["counts"],
                                         out["counts"].numel()))
    found += [ctx.stream_wait(t)[0] for t in tickets[len(found):]]
    return [{"n": d, **b[3]} for b, d in zip(s["batches"], found)]


RUN = {"pipeline": run_pipeline, "merged": run_merged, "shard": run_shard, "minimizers": run_minimizers,
       "subsample": run_subsample, "host_bin": run_host_bin, "stream": run_stream}


# -------------------------------------------------------------------- work

def work(case):
    """Bytes in and out of one pass, each once: reads and offsets (or packed
    superkmers and lengths) in, the result out.  The distinct k-mers are
    estimated from the genome and the error rate."""
    k, bases, kind = case["k"], case["bases"], case["kind"]
    width = 8 if k <= 32 else 16
    if kind == "host_bin":
        n = bases // 20
        mean = (3 * k - case["p"]) / 2
        distinct = min(n * (mean - k + 1), bases // case["coverage"])
        return {"bytes": n * (4 + mean / 4) + 12 * distinct, "flops": 0}
    distinct, kmers = expected_distinct(case, bases)
    if case["hpc"]:  # a quarter of the bases are repeats
        distinct, kmers = min(distinct, 0.75 * kmers), 0.75 * kmers
    into = bases + 8 * (bases // (8000 if case["source"] == "long" else case["read_len"]) + 1)
    if kind == "minimizers":
        return {"bytes": into + 6 * bases, "flops": 0}
    if kind == "subsample":
        return {"bytes": into + (width + 8) * distinct / 4 + 4 * kmers / 4, "flops": 0}
    if kind == "merged":
        distinct = min(distinct, bases // case["coverage"])
    return {"bytes": into + (width + 4) * distinct, "flops": 0}
