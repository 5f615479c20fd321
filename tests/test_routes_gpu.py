"""Which kernels a call launches, read from the engine's trace (``SZS_GB300_TRACE``) in a process of its own: parity tests
alone would pass as well with a route never taken. Every call is checked against the oracle too."""
import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import sys
sys.path.insert(0, {repo!r})
import numpy as np
import torch
import stringzillas_gb300 as szs
from oracle import oracle
DNA = np.frombuffer(b"ACGT", dtype=np.uint8)
rng = np.random.default_rng(11)
port = oracle.Port()

def tape(lengths):
    offsets = np.zeros(len(lengths) + 1, dtype=np.int64)
    offsets[1:] = np.cumsum(lengths)
    return DNA[rng.integers(0, 4, offsets[-1])], offsets

def mutant(data, rate):
    data = data.copy()
    where = rng.random(len(data)) < rate
    data[where] = DNA[rng.integers(0, 4, int(where.sum()))]
    return data

def check(engine, costs, first, second, repeat=1, where="cuda"):
    want = port.pairs(costs, *((d, o.astype(np.uint64)) for d, o in (first, second)))
    def repeated(side):
        data, offsets = side
        return np.tile(data, repeat), np.concatenate([offsets[:-1] + i * offsets[-1] for i in range(repeat)] + [[repeat * offsets[-1]]])
    place = (lambda x: torch.from_numpy(x).cuda()) if where == "cuda" else (lambda x: torch.from_numpy(x).pin_memory())
    sides = [szs.Strs.from_buffers(*map(place, repeated(side))) for side in (first, second)]
    out = place(np.zeros(len(want) * repeat, dtype=np.int64))
    engine.pairwise(*sides, out=out)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), np.tile(want, repeat))
"""


def trace(script):
    """The trace lines of one process that runs the script."""
    env = dict(os.environ, SZS_GB300_TRACE="1")
    done = subprocess.run([sys.executable, "-c", PRELUDE.format(repo=REPO) + script], env=env, capture_output=True,
                          text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    return [line for line in done.stderr.splitlines() if line.startswith("[szs_gb300]")]


def near_counts(lines):
    found = [re.search(r"near diagonal tried (\d+) failed (\d+)", line) for line in lines]
    return [(int(m.group(1)), int(m.group(2))) for m in found if m]


@pytest.mark.parametrize("unrelated,tried", [(0.0, True), (0.3, False)])
def test_near_diagonal_trial_of_a_small_batch(unrelated, tried):
    """Alike reads are tried near their diagonal; with a third of them unrelated, a batch of few goes without."""
    lines = trace(f"""
first = tape(rng.integers(150, 300, 3000))
second = mutant(first[0], 0.04), first[1]
for i in range(int({unrelated} * 3000)):
    second[0][first[1][i * 3]:first[1][i * 3 + 1]] = DNA[rng.integers(0, 4, first[1][i * 3 + 1] - first[1][i * 3])]
check(szs.LevenshteinDistances(), oracle.levenshtein_costs(), first, second)
""")
    counts = near_counts(lines)
    assert bool(counts) == tried
    if tried:
        assert counts[-1][0] == 3000 and counts[-1][1] < 30


def test_near_diagonal_trial_gives_up():
    """A batch whose sampled ends look alike while the strings between are unrelated: the first waves are tried in vain, and
    the rest is left to the full kernels untried."""
    lines = trace("""
first = tape(rng.integers(140, 180, 1000))
second = DNA[rng.integers(0, 4, first[1][-1])], first[1]
for i in range(1000):
    begin, end = first[1][i], first[1][i + 1]
    second[0][begin:begin + 24] = first[0][begin:begin + 24]
    second[0][end - 24:end] = first[0][end - 24:end]
check(szs.LevenshteinDistances(), oracle.levenshtein_costs(), first, second, repeat=400)
""")
    tried, failed = near_counts(lines)[-1]
    assert 4096 <= tried < 400000 and failed >= tried // 16 * 15


@pytest.mark.parametrize("rate,tried", [(0.04, True), (1.0, False)])
def test_near_diagonal_trial_of_pinned_chunks(rate, tried):
    """Chunks of pinned-host calls are planned before their strings land: they go by the first chunk's pairs."""
    lines = trace(f"""
first = tape(rng.integers(140, 200, 6000))
engine = szs.LevenshteinDistances()
engine.set_tuning({{"pipeline_chunk_kb": 256}})
check(engine, oracle.levenshtein_costs(), first, (mutant(first[0], {rate}), first[1]), where="pinned")
""")
    chunks = [line for line in lines if re.search(r"chunk +\d+ +pairs", line)]
    jobs = [line for line in lines if "job kind 8 " in line]
    assert len(chunks) >= 4
    assert len(jobs) >= len(chunks) if tried else not jobs


def test_largest_pairs_of_a_batch_in_groups():
    """Many 16-bit band pairs of very different sizes: the largest size classes take groups of CTAs, the others single ones,
    in one call."""
    lines = trace("""
lengths = np.concatenate([rng.integers(2050, 2400, 360), [9000, 8200, 12000]])
other = np.concatenate([rng.integers(2050, 2600, 360), [9500, 16000, 8500]])
table = np.zeros((32, 32), dtype=np.int8)
table[1:5, 1:5] = -3
np.fill_diagonal(table[1:5, 1:5], 2)
classes = np.zeros(256, dtype=np.uint8)
classes[DNA] = [1, 2, 3, 4]
engine = szs.SmithWatermanScores(classes, table, open=-5, extend=-2)
check(engine, oracle.alignment_costs(oracle.SMITH_WATERMAN, classes, table, -5, -2), tape(lengths), tape(other))
""")
    found = [re.search(r"band16 bits .*pairs +(\d+) +ctas per pair +(\d+)", line) for line in lines]
    jobs = [(int(m.group(1)), int(m.group(2))) for m in found if m]
    assert sum(pairs for pairs, _ in jobs) == 363
    assert any(group > 1 for _, group in jobs) and any(group == 1 for _, group in jobs)
