"""The calls this engine is timed on: what users of its scorers and fingerprints have it do, from one handful of short
reads to whole batches, cross products, long pairs and documents.

Every case goes through the Python callables (``engine.pairwise``, ``engine(queries, candidates)``,
``Fingerprints(...)``). Inputs are synthetic, made on the GPU from the seed alone, with the shapes of the engine's own
benchmark configurations (``stringzillas_gb300/workloads.py``, ``bench.py``) around which the drawn cases spread.
Engines are kept per cost model, as a program keeps its handles; nothing else outlives a state. Every output is a whole
number (distances, scores, hashes, counts) and is compared exactly, so there is no ``exact``.
"""
import math

import numpy as np
import torch

import stringzillas_gb300 as szs
from stringzillas_gb300 import workloads

# Cost models by name: Levenshtein (match, mismatch, open, extend); alignments are (table, open, extend).
LEVENSHTEIN_COSTS = {"unit": (0, 1, 1, 1), "affine": (0, 2, 3, 1), "linear": (0, 2, 3, 3)}
ALIGNMENT_GAPS = {"protein": (-11, -1), "dna": (-5, -2), "dna_linear": (-3, -3)}
# Operations the recurrences need per cell: the bit-parallel step's ten operations per 32 rows, else one opt per track.
OPS_PER_CELL = {"unit": 10 / 32, "linear": 4, "dna_linear": 4}
AFFINE_OPS_PER_CELL = 7
MOST_CELLS = 4.0e10  # a drawn case stays below the largest listed ones

_engines = {}


def listed():
    return [
        # A handful of reads scored from host memory: one call's latency (launches, planning, copies) counts.
        pairs("lev_few_reads", "lev", "unit", "dna", 64, 64, 256, 0.05, 0.02, host=True),
        # Read deduplication and barcode matching: a whole batch of short DNA reads (the headline configuration).
        pairs("lev_reads", "lev", "unit", "dna", 1 << 20, 100, 300, 0.03, 0.01),
        # Long-read comparison: thousands of bases a side.
        pairs("lev_long_reads", "lev", "unit", "dna", 4096, 1000, 4000, 0.03, 0.01),
        # Spell checking and record linkage: every token of one vocabulary against another.
        cross("lev_words_cross", "lev", "unit", "text", 2048, 2048, 4, 16),
        # All-against-all distances of equal-length sequences, at the reference's published methodology.
        cross("lev_cross_1k", "lev", "unit", "dna", 197, 198, 1000, 1000),
        # Weighted edit distances of lines of text.
        pairs("lev_text_costs", "lev", "affine", "text", 65536, 100, 300, 0.05, 0.02),
        # Multilingual text: UTF-8 distances, transcoding included.
        pairs("lev_utf8_cjk", "lev_utf8", "unit", "cjk", 65536, 100, 300, 0.05, 0.02),
        # Protein search: global alignment scores against homologues, lengths of real proteins.
        pairs("nw_protein", "nw", "protein", "protein", 262144, 350, 0, 0.30, 0.02),
        # Two very long sequences: one pair has to use the whole GPU.
        pairs("nw_long_pair", "nw", "protein", "protein", 1, 30000, 30000, 0.30, 0.02),
        # Short-read mapping: local scores of many short pairs.
        pairs("sw_short_reads", "sw", "dna", "dna", 1 << 20, 16, 128, 0.10, 0.02),
        # Local alignment of genomic fragments sharing a segment, lengths log-uniform over a wide range.
        pairs("sw_long_dna", "sw", "dna", "local", 1024, 1000, 30000, 0.10, 0.0),
        # Near-duplicate detection: Min-Hash fingerprints of documents.
        {"name": "minhash_docs", "form": "minhash", "count": 16384, "low": 1000, "high": 3000, "dims": 1024, "bits": 64},
    ]


def pairs(name, algo, costs, data, count, low, high, substitutions, indels, host=False, bits=64):
    """(first[i], second[i]) pairs; the second string is a mutant of the first. Protein lengths are log-normal around
    `low` when `high` is 0; `local` pairs are unrelated but for one shared segment."""
    return {"name": name, "form": "pairs", "algo": algo, "costs": costs, "data": data, "count": count, "low": low,
            "high": high, "substitutions": substitutions, "indels": indels, "host": host, "bits": bits}


def cross(name, algo, costs, data, rows, columns, low, high, bits=64):
    return {"name": name, "form": "cross", "algo": algo, "costs": costs, "data": data, "rows": rows,
            "columns": columns, "low": low, "high": high, "bits": bits}


def draw(rng):
    def spread(low, high):  # log-uniform over sizes spanning orders of magnitude
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    def capped(count, cells_each):
        return max(1, min(count, int(MOST_CELLS / cells_each)))

    bits = rng.choice([32, 64])
    # From near-identical reads to unrelated ones.
    substitutions = rng.choice([0.005, 0.03, 0.05, 0.10, 0.20, 0.75])
    indels = rng.choice([0.0, 0.01, 0.02, 0.05])
    family = rng.choice(["few", "reads", "long_reads", "words", "cross", "text", "utf8", "protein", "long", "short",
                         "local", "minhash"])
    if family == "few":
        low = rng.randint(8, 200)
        case = pairs("", "lev", rng.choice(["unit", "unit", "affine"]), rng.choice(["dna", "text"]), spread(1, 512), low,
                     low + rng.randint(0, 200), substitutions, indels, host=True, bits=bits)
    elif family == "reads":
        low = rng.randint(16, 250)
        high = low + rng.randint(0, 250)
        case = pairs("", "lev", "unit", rng.choice(["dna", "dna", "text"]), capped(spread(1 << 12, 1 << 20), high * high),
                     low, high, substitutions, indels, bits=bits)
    elif family == "long_reads":
        low = spread(520, 4000)
        high = low + spread(1, 4000)
        case = pairs("", "lev", "unit", "dna", capped(spread(16, 8192), high * high), low, high, substitutions, indels,
                     bits=bits)
    elif family == "words":
        low = rng.randint(1, 12)
        case = cross("", "lev", "unit", rng.choice(["text", "dna"]), spread(64, 2048), spread(64, 2048), low,
                     low + rng.randint(0, 36), bits=bits)
    elif family == "cross":
        algo = rng.choice(["lev", "nw", "sw"])
        low = spread(65, 1000)
        case = cross("", algo, "unit" if algo == "lev" else rng.choice(["dna", "dna_linear"]), "dna", spread(16, 256),
                     spread(16, 256), low, low + rng.choice([0, 0, rng.randint(1, 300)]), bits=bits)
    elif family == "text":
        low = rng.randint(30, 300)
        high = low + rng.randint(0, 300)
        case = pairs("", "lev", rng.choice(["affine", "linear"]), "text", capped(spread(1 << 10, 1 << 17), high * high),
                     low, high, substitutions, indels, bits=bits)
    elif family == "utf8":
        low = rng.randint(10, 200)
        high = low + rng.randint(0, 200)
        case = pairs("", "lev_utf8", rng.choice(["unit", "unit", "affine"]), rng.choice(["cjk", "latin"]),
                     capped(spread(1 << 8, 1 << 16), high * high), low, high, substitutions, indels, bits=bits)
    elif family == "protein":
        median = spread(80, 700)
        case = pairs("", "nw", "protein", "protein", capped(spread(1 << 11, 1 << 18), 2.1 * median * median), median, 0,
                     rng.choice([0.1, 0.3, 0.5]), 0.02, bits=bits)
    elif family == "long":
        length = spread(3000, 30000)
        algo, costs, data = rng.choice([("nw", "protein", "protein"), ("sw", "dna", "dna"), ("lev", "linear", "dna"),
                                        ("lev", "unit", "dna")])
        case = pairs("", algo, costs, data, capped(spread(1, 16), 4.0 * length * length), length, length + 100, 0.1, 0.02,
                     bits=bits)
    elif family == "short":
        low = rng.randint(8, 64)
        algo, costs, data = rng.choice([("sw", "dna", "dna"), ("nw", "protein", "protein"), ("lev", "affine", "dna")])
        case = pairs("", algo, costs, data, spread(1 << 13, 1 << 20), low, low + rng.randint(0, 64), 0.1, 0.02, bits=bits)
    elif family == "local":
        low = spread(600, 4000)
        case = pairs("", "sw", "dna", "local", spread(32, 768), low, min(30000, 4 * low + spread(1, 20000)), 0.1, 0.0,
                     bits=bits)
        case["count"] = capped(case["count"], _mean_product(case))
    else:
        low = spread(20, 2000)
        case = {"form": "minhash", "count": spread(64, 8192), "low": low, "high": low + spread(1, 1000),
                "dims": rng.choice([64, 100, 128, 256, 512, 1024]), "bits": bits}
    case.pop("name", None)
    return case


# ---- inputs -----------------------------------------------------------------------------------------------------------


def prepare(case, seed):
    generator = torch.Generator(device="cuda")
    generator.manual_seed(seed)
    state = {"case": case}
    count = case["count"] if case["form"] != "cross" else case["rows"]
    lengths = _lengths(case, count, generator)
    if case["form"] == "minhash":
        offsets = _offsets(lengths)
        state["texts"] = _strs(_bytes("text", _codes(95, int(offsets[-1]), generator)), offsets, case)
        state["engine"] = _engine("minhash", case["dims"])
        state["out"] = tuple(torch.zeros((count, case["dims"]), dtype=torch.int32, device="cuda") for _ in range(2))
    elif case["form"] == "cross":
        symbols = 4 if case["data"] == "dna" else 95
        for side, side_lengths in (("first", lengths), ("second", _lengths(case, case["columns"], generator))):
            offsets = _offsets(side_lengths)
            state[side] = _strs(_bytes(case["data"], _codes(symbols, int(offsets[-1]), generator)), offsets, case)
        state["engine"] = _engine(case["algo"], case["costs"])
        state["out"] = torch.zeros((case["rows"], case["columns"]), dtype=torch.int64, device="cuda")
    else:
        make = _local_pairs if case["data"] == "local" else _mutant_pairs
        (first, first_offsets), (second, second_offsets) = make(case, lengths, generator)
        state["first"] = _strs(first, first_offsets, case)
        state["second"] = _strs(second, second_offsets, case)
        state["engine"] = _engine(case["algo"], case["costs"])
        state["out"] = None if case["host"] else torch.zeros(count, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()  # the engine works on its own stream
    return state


def run(state):
    if state["case"]["form"] == "minhash":
        return state["engine"](state["texts"], out=state["out"])
    if state["case"]["form"] == "cross":
        return state["engine"](state["first"], state["second"], out=state["out"])
    return state["engine"].pairwise(state["first"], state["second"], out=state["out"])


def work(case):
    """Inputs once, results once; cells times the recurrence's operations (from the lengths' means)."""
    if case["form"] == "minhash":
        text = case["count"] * (case["low"] + case["high"]) / 2
        # A rolling hash's update modulo a 42-bit prime is sixteen 32-bit integer operations.
        return {"bytes": text + 8 * (case["count"] + 1) + 8 * case["count"] * case["dims"],
                "flops": 16 * text * case["dims"]}
    mean, square = _mean_length(case), _mean_product(case)
    width = {"cjk": 3, "latin": 1.5}.get(case["data"], 1)
    if case["form"] == "cross":
        strings, results = case["rows"] + case["columns"], case["rows"] * case["columns"]
        square = mean * mean
    else:
        strings, results = 2 * case["count"], case["count"]
    return {"bytes": strings * (mean * width + case["bits"] / 8) + 8 * results,
            "flops": results * square * OPS_PER_CELL.get(case["costs"], AFFINE_OPS_PER_CELL)}


def _mean_length(case):
    if case.get("high") == 0:
        return case["low"] * math.exp(0.18)  # log-normal, sigma 0.6
    if case["data"] == "local":
        return (case["high"] - case["low"]) / math.log(max(case["high"] / case["low"], 1 + 1e-9))
    return (case["low"] + case["high"]) / 2


def _mean_product(case):
    """Mean of len(first) * len(second): partners of mutants share their length, local pairs do not."""
    mean = _mean_length(case)
    if case.get("high") == 0:
        return case["low"] ** 2 * math.exp(2 * 0.36)
    if case["data"] == "local":
        return mean * mean
    return mean * mean + (case["high"] - case["low"]) ** 2 / 12


def _engine(algo, costs):
    """One engine per cost model, kept as a program keeps its handles."""
    if (algo, costs) not in _engines:
        if algo == "minhash":
            engine = szs.Fingerprints(costs)
        elif algo == "lev":
            engine = szs.LevenshteinDistances(*LEVENSHTEIN_COSTS[costs])
        elif algo == "lev_utf8":
            engine = szs.LevenshteinDistancesUTF8(*LEVENSHTEIN_COSTS[costs])
        else:
            table = workloads.protein_table() if costs == "protein" else workloads.dna_table()
            gap_open, gap_extend = ALIGNMENT_GAPS[costs]
            kind = szs.NeedlemanWunschScores if algo == "nw" else szs.SmithWatermanScores
            engine = kind(*table, open=gap_open, extend=gap_extend)
        _engines[algo, costs] = engine
    return _engines[algo, costs]


def _strs(data, offsets, case):
    offsets = offsets.to(torch.int32) if case["bits"] == 32 else offsets
    if case.get("host"):
        return szs.Strs.from_buffers(data.cpu().numpy(), offsets.cpu().numpy())
    return szs.Strs.from_buffers(data, offsets)


def _lengths(case, count, generator):
    low, high = case["low"], case["high"]
    if high == 0:  # proteins: log-normal, clipped
        normal = torch.randn(count, generator=generator, device="cuda", dtype=torch.float64)
        return (low * torch.exp(0.6 * normal)).round().clamp(50, 2000).to(torch.int64)
    if case.get("data") == "local":
        uniform = torch.rand(count, generator=generator, device="cuda", dtype=torch.float64)
        return torch.exp(math.log(low) + uniform * (math.log(high) - math.log(low))).to(torch.int64)
    return torch.randint(low, high + 1, (count,), generator=generator, device="cuda")


def _offsets(lengths):
    offsets = torch.zeros(lengths.shape[0] + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lengths, 0, out=offsets[1:])
    return offsets


def _codes(symbols, size, generator, frequencies=None):
    """`size` symbol codes, uniform or by `frequencies`."""
    if frequencies is None:
        kind = torch.uint8 if symbols <= 256 else torch.int16
        return torch.randint(0, symbols, (size,), generator=generator, device="cuda", dtype=kind)
    edges = torch.from_numpy(np.cumsum(frequencies / np.sum(frequencies))[:-1].astype(np.float32)).cuda()
    uniform = torch.rand(size, generator=generator, device="cuda")
    return torch.bucketize(uniform, edges, out_int32=True).to(torch.uint8)


def _bytes(data, codes):
    letters = {"dna": workloads.DNA, "local": workloads.DNA, "text": workloads.PRINTABLE,
               "protein": workloads.AMINO_ACIDS}[data]
    return torch.from_numpy(letters.copy()).cuda()[codes.to(torch.int32)]


def _utf8(data, codes, offsets):
    """UTF-8 bytes of code points: CJK ideographs (three bytes each), or Latin text (one or two bytes each)."""
    points = codes.to(torch.int32)
    if data == "cjk":
        points = points + workloads.CJK_FIRST
        parts = [0xE0 | (points >> 12), 0x80 | ((points >> 6) & 0x3F), 0x80 | (points & 0x3F)]
        return torch.stack(parts, dim=1).to(torch.uint8).reshape(-1), 3 * offsets
    points = torch.where(points < 95, points + 32, points + (0xC0 - 95))  # printable ASCII, then U+00C0 and up
    wide = points >= 0x80
    starts = _offsets(1 + wide.to(torch.int64))
    out = torch.empty(int(starts[-1]), dtype=torch.uint8, device="cuda")
    out[starts[:-1]] = torch.where(wide, 0xC0 | (points >> 6), points).to(torch.uint8)
    out[starts[:-1][wide] + 1] = (0x80 | (points[wide] & 0x3F)).to(torch.uint8)
    return out, starts[offsets]


def _mutant_pairs(case, lengths, generator):
    """Strings and their mutants: substitutions to another symbol, then single-symbol insertions and deletions."""
    data = case["data"]
    symbols = {"dna": 4, "protein": 20, "text": 95, "cjk": workloads.CJK_COUNT, "latin": 159}[data]
    frequencies = workloads.AMINO_FREQUENCIES if data == "protein" else None
    offsets = _offsets(lengths)
    size = int(offsets[-1])
    first = _codes(symbols, size, generator, frequencies)
    chance = torch.rand(size, generator=generator, device="cuda")
    other = torch.randint(1, symbols, (size,), generator=generator, device="cuda", dtype=torch.int16)
    second = torch.where(chance < case["substitutions"], (first.to(torch.int16) + other) % symbols, first.to(torch.int16))
    chance = torch.rand(size, generator=generator, device="cuda")
    delete, insert = chance < case["indels"] / 2, chance > 1 - case["indels"] / 2
    copies = 1 - delete.to(torch.int64) + insert.to(torch.int64)
    ends = _offsets(copies)
    second = torch.repeat_interleave(second, copies)
    at = (ends[1:] - 1)[insert]
    second[at] = _codes(symbols, at.shape[0], generator, frequencies).to(torch.int16)
    second_offsets = ends[offsets]
    if data in ("cjk", "latin"):
        return _utf8(data, first, offsets), _utf8(data, second, second_offsets)
    return (_bytes(data, first), offsets), (_bytes(data, second), second_offsets)


def _local_pairs(case, lengths, generator):
    """Unrelated strings that share one segment, copied with some divergence."""
    count = lengths.shape[0]
    second_lengths = _lengths(case, count, generator)
    offsets, second_offsets = _offsets(lengths), _offsets(second_lengths)
    first = _codes(4, int(offsets[-1]), generator)
    second = _codes(4, int(second_offsets[-1]), generator)
    longest = torch.minimum(lengths, second_lengths)
    segments = torch.minimum(torch.randint(500, 5001, (count,), generator=generator, device="cuda"), longest)

    def place(room):  # a start that leaves the segment inside its string
        uniform = torch.rand(count, generator=generator, device="cuda", dtype=torch.float64)
        return (uniform * (room - segments + 1)).to(torch.int64).clamp(max=room - segments)

    first_at, second_at = offsets[:-1] + place(lengths), second_offsets[:-1] + place(second_lengths)
    starts = _offsets(segments)
    within = torch.arange(int(starts[-1]), device="cuda") - torch.repeat_interleave(starts[:-1], segments)
    copied = first[torch.repeat_interleave(first_at, segments) + within]
    diverged = torch.rand(copied.shape[0], generator=generator, device="cuda") < case["substitutions"]
    copied = torch.where(diverged, _codes(4, copied.shape[0], generator), copied)
    second[torch.repeat_interleave(second_at, segments) + within] = copied
    return (_bytes("local", first), offsets), (_bytes("local", second), second_offsets)
