"""Searches on several threads at once whose launches of one kernel need
different amounts of shared memory: neither may take the other's away."""
import threading

import pytest

import puzzlesearch_b200 as psb

pytestmark = pytest.mark.gpu


def together(*jobs):
    """Runs the jobs in a thread each, all to the end; what they raised."""
    failed = []

    def run(job):
        try:
            job()
        except Exception as e:  # handed to the test's thread
            failed.append(e)

    threads = [threading.Thread(target=run, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return failed


def test_one_launch_searches():
    """All of them run in one launch (11 disks take 128 KB a block, 9 disks 38 KB)."""
    whole = {9: [], 11: []}

    def search(disks, runs):
        def job():
            p = psb.FourPegHanoiSimple(disks)
            for _ in range(runs):
                whole[disks].append(psb.bfs(p, "two_bit", 0, max_depth=2)["stats"]["expand_launches"])
        return job

    assert not together(search(11, 2000), search(11, 2000), search(9, 2000), search(9, 2000))
    assert set(whole[9]) == set(whole[11]) == {1}

@pytest.mark.parametrize("algo", ["two_bit", "three_bit", "frontier"])
@pytest.mark.parametrize("puzzle", ["hanoi", "sliding"])
def test_level_kernels(puzzle, algo):
    """Windows of different size in the two threads: 64 KB and more of marks against 1 KB."""
    wide = 18 if algo == "frontier" else 20
    p = psb.FourPegHanoiSimple(7) if puzzle == "hanoi" else psb.SlidingTilePuzzleSimple(3, 3)
    want = psb.bfs(p, algo, 0)["counts"]
    got = []

    def search(window_bits):
        def job():
            for _ in range(60):
                got.append(psb.bfs(p, algo, 0, window_bits=window_bits, threads=256)["counts"])
        return job

    assert not together(search(wide), search(10), search(10))
    assert len(got) == 180 and all(c == want for c in got)
