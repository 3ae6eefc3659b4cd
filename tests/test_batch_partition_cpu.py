"""How a batch's cavities are put into groups (partition.h): in order, at the least
cost of all cuts, so that several cavities share a group that the L2 does not
hold only where further groups would cost more."""
import itertools
import os
import random
import subprocess

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
L2 = 132_644_864
LAUNCH, FITS, RISE, MISS = 8e6, 0.42, 1.1, 0.46


def node_bytes(sizes, per_node):
    return [ny * ((nx + 31) // 32 * 32) * per_node for nx, ny in sizes]


def cost(b):
    return LAUNCH + b * (1 + min(RISE * max((b - FITS * L2) / (L2 - FITS * L2), 0.0) ** 2, MISS))


def cheapest(sizes):
    n = len(sizes)
    return min(sum(cost(sum(sizes[i:j])) for i, j in zip((0, *cut), (*cut, n)))
               for k in range(n) for cut in itertools.combinations(range(1, n), k))


def test_groups(tmp_path):
    exe = tmp_path / "partition_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "cfd_cavity_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "partition_check.cpp"), "-o", str(exe)], check=True)
    sweep = [((64, 256), (96, 384), (128, 512))[i % 3] for i in range(64)]
    # (sizes, the largest group of several cavities in MB, the groups)
    named = [
        ([50_000_000] * 4, 72, 4),
        (node_bytes([(256, 1024)] * 4, 148), 78, 2),
        (node_bytes([(512, 2048)], 148), 0, 1),
        (node_bytes([(180, 1024)] * 6, 148), 72, 3),
        (node_bytes(sweep, 148), 72, 6),  # 375 MB: five groups of 75 would miss more than a launch costs
        (node_bytes(sweep, 76), 74, 3),
        (node_bytes(sweep * 4, 296), 74, None),
        ([1], 0, 1),
    ]
    rng = random.Random(3)
    drawn = [[int(10 ** rng.uniform(5, 8.4)) for _ in range(rng.randrange(1, 11))] for _ in range(60)]
    cases = [n[0] for n in named] + drawn
    text = "\n".join(" ".join(map(str, [L2, *b, 0])) for b in cases)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
    assert len(out) == len(cases)
    for k, (b, line) in enumerate(zip(cases, out)):
        *first, total = line.split()
        first = [int(x) for x in first]
        assert first[0] == 0 and first[-1] == len(b) and all(i < j for i, j in zip(first, first[1:]))
        groups = [b[i:j] for i, j in zip(first, first[1:])]
        assert abs(float(total) / sum(cost(sum(g)) for g in groups) - 1) < 1e-12
        if k < len(named):
            _, largest, count = named[k]
            assert max((sum(g) for g in groups if len(g) > 1), default=0) <= largest * 1e6, (k, first)
            assert count is None or len(groups) == count, (k, first)
        elif all(len(g) == 1 or sum(g) <= 4 * L2 for g in [b]):
            assert float(total) <= cheapest(b) * (1 + 1e-12), (b, first)
