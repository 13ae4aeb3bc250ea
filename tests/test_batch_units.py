"""Batches of many sets are bounded by their units and by the device memory
their sets need (batch_units, eddy_host.cpp).  CPU only."""
import os
import random
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "eddy-gpu_gb300", "csrc")


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("batch") / "batch_units")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
                    os.path.join(HERE, "batch_units_main.cpp"), os.path.join(CSRC, "eddy_host.cpp"),
                    "-o", exe], check=True)

    def run(max_units, max_bytes, jobs):
        args = [str(x) for x in [max_units, max_bytes] + [v for j in jobs for v in j]]
        r = subprocess.run([exe] + args, capture_output=True, text=True, check=True)
        return [int(x) for x in r.stdout.split()]

    return run


def test_units_alone_bound_small_sets(cut):
    assert cut(1000, 1 << 35, [(999, 1 << 20)] * 4) == [1000, 1000, 1000, 996]
    assert cut(32768, 1 << 35, [(1, 1 << 10)] * 300) == [300]


def test_memory_bounds_many_sets(cut):
    gb = 1 << 30
    # 989 sets of 0.3 GB: 106 of them a batch
    got = cut(18791, 32 * gb, [(19, 3 * gb // 10)] * 989)
    assert max(got) == 19 * 106 and sum(got) == 19 * 989
    # a set above the bound is a batch of its own
    assert cut(100, 32 * gb, [(5, gb), (7, 91 * gb), (3, gb), (4, gb)]) == [5, 7, 7]
    assert cut(4, 32 * gb, [(9, 91 * gb), (2, gb)]) == [4, 4, 1, 2]


@pytest.mark.parametrize("seed", range(20))
def test_every_batch_within_both_bounds(seed, cut):
    rng = random.Random(seed)
    jobs = [(rng.randint(1, 50), rng.randint(0, 40)) for _ in range(rng.randint(1, 60))]
    units, room = rng.randint(1, 200), rng.randint(1, 150)
    got = cut(units, room, jobs)
    owner = [j for j, (k, _) in enumerate(jobs) for _ in range(k)]
    assert sum(got) == len(owner) and min(got) >= 1 and max(got) <= units
    at = 0
    for k in got:
        held = sorted(set(owner[at:at + k]))
        assert len(held) == 1 or sum(jobs[j][1] for j in held) <= room
        at += k
        if k < units and at < len(owner):  # the next set did not fit
            assert sum(jobs[j][1] for j in held) + jobs[owner[at]][1] > room
