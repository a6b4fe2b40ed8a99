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
