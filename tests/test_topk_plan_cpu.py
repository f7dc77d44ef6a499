"""Host arithmetic of a joint top-K selection's workspace: the counters that a call clears
are those of the buckets that it selects from, and lie inside what it asked for, whatever
is empty and whatever share is sent (no device work)."""
import ctypes
import itertools
import random

import pytest

BLOCK = 33024                                 # one bucket's counters


@pytest.fixture(scope="module")
def plan():
    from singa_b200 import _lib
    lib = _lib.lib()

    def of(sizes, share, mode):
        n = len(sizes)
        ks = [lib.sgb_topk_count(share, s) for s in sizes]
        counters = ctypes.c_size_t(-1)
        bytes_ = lib.sgb_sparse_topk_plan((ctypes.c_size_t * n)(*sizes), (ctypes.c_size_t * n)(*ks), n, mode,
                                          ctypes.byref(counters))
        return bytes_, counters.value, sum(1 for s, k in zip(sizes, ks) if s and k)
    return of


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("share", [-1.0, 0.0, 1e-9, 0.01, 0.3, 1.0])
def test_what_is_cleared_lies_inside_the_workspace(plan, share, mode):
    rng = random.Random(int(share * 1000) + mode)
    lists = [[100, 1000, 0], [1000, 1000], [4000] * 16, [12000] * 32, [0] * 31 + [5]]
    for count in range(1, 65):
        sizes = [rng.choice([0, 1, rng.randint(1, 20000)]) for _ in range(count)]
        lists += [sizes[i:i + 32] for i in range(0, count, 32)]
    lists += [list(p) for p in itertools.product((0, 1, 4097), repeat=3)]
    for sizes in lists:
        need, counters, selected = plan(sizes, share, mode)
        if not any(sizes):
            assert need == 0
            continue
        assert counters == selected * BLOCK and counters <= need, (sizes, share)


def test_more_buckets_than_one_launch_takes(plan):
    assert plan([5] * 33, 0.5, 0)[0] == 0
