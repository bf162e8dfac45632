"""CPU tests of the plan by which the attention kernel's last rounds are dealt out by key blocks (csrc/sage3_split.h, compiled with tests/split_plan.cpp): every key
block of every query tile is walked once, from the tile's last block to its first, and what a slot waits for has been drawn before it and waits for nothing."""
import ctypes as C
import os
import pathlib
import random
import subprocess

import pytest

from tests import test_shared_tiles_gpu

SLOTS = 160


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("plan") / "split_plan.so"
    cuda = pathlib.Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", f"-isystem{cuda / 'include'}",
                           str(pathlib.Path(__file__).with_name("split_plan.cpp")), "-o", str(so)])
    return C.CDLL(str(so))


def plan(lib, causal, heads, nqt, Nk, shift, D=128, sms=148):
    """(pairs ahead, blocks per slot, of slot 0, rest0, [first tile and block of slot m]); no slots: nothing is dealt out."""
    out, first = (C.c_int * 5)(), (C.c_uint32 * SLOTS)()
    lib.split_plan(int(causal), heads, nqt, Nk, shift, D, sms, out, first)
    whole, slots, blocks, rest, rest0 = out
    return whole, blocks, rest, rest0, [(f & 0xfff, f >> 12) for f in first[:slots]]


def check(lib, causal, heads, nqt, Nk, shift, D, sms):
    whole, blocks, rest, rest0, first = plan(lib, causal, heads, nqt, Nk, shift, D, sms)
    if not first:
        assert blocks == 0
        return False
    nb = [lib.split_blocks(int(causal), mt, Nk, shift) for mt in range(nqt)]
    tile = (C.c_int * 2)()
    walked = {}                            # (head, tile) -> [(first block, end, slot)] in the order of the walk
    # the pairs ahead, as the kernel's units: neighbours of a head without a mask, those with the most keys of all heads first with one
    npair = (nqt + 1) // 2 if causal else nqt // 2
    assert whole % sms == 0 and (whole == 0 or nqt % 2 == 0 or not causal)      # (the rounds ahead are even)
    for u in range(whole):
        h, mt = (u % heads, 2 * (npair - 1 - u // heads)) if causal else (u // npair, 2 * (u % npair))
        for t in (mt, mt + 1):
            assert h < heads and 0 <= t < nqt and (h, t) not in walked
            walked[h, t] = [(0, nb[t], None)]
    # the slots, in the order in which they are drawn, each as the kernel's producer walks it
    assert len(first) <= sms
    for m, (j, lo) in enumerate(first):
        left = rest if m == 0 else blocks
        assert 0 < left <= blocks
        parts = 0
        while left > 0:
            lib.split_tile(int(causal), j, nqt, heads, whole, rest0, tile)
            h, t = tile
            assert 0 <= h < heads and 0 <= t < nqt
            hi = min(nb[t], lo + left)
            assert lo < hi
            before = walked.setdefault((h, t), [])
            if hi < nb[t]:                 # goes on from the part of the slot drawn just before, where it came first and waited for nothing
                assert [b[0] for b in before] == [hi] and before[0][1:] == (nb[t], m - 1) and first[m - 1] == (j, hi)
            else:
                assert not before
            assert lo == 0 or parts == 0   # (what another slot goes on from comes first)
            before.append((lo, hi, m))
            left -= hi - lo
            j, lo, parts = j + 1, 0, parts + 1
    assert len(walked) == heads * nqt
    for (h, t), parts in walked.items():
        assert len(parts) <= 2 and parts[0][1] == nb[t] and parts[-1][0] == 0, (h, t, parts)
    return True


def test_every_block_is_in_one_slot(lib):
    r = random.Random(7)
    dealt = set()
    for _ in range(6000):
        causal, sms = r.random() < 0.5, r.choice((148, 148, 132, 160, 1, 2, 7, 31))
        nqt = int(1.6 ** r.uniform(0, 10))
        heads = max(1, int(r.uniform(0.5, 5) * sms / nqt))
        Nk = r.randint(1900, 6000)
        shift = Nk - 128 * nqt + r.randrange(128) if r.random() < 0.8 else r.randint(-3000, 6000)
        if check(lib, causal, heads, nqt, Nk, shift, r.choice((64, 128)), sms):
            whole = plan(lib, causal, heads, nqt, Nk, shift, 128, sms)[0]
            dealt.add((causal, nqt == 1, nqt % 2, whole > 0))
    # one tile per head, odd and even numbers of tiles, with and without rounds ahead (with a mask an odd number has none)
    assert dealt >= {(c, False, odd, ahead) for c in (False, True) for odd in (0, 1) for ahead in (False, True) if not (c and odd and ahead)} | {(False, True, 1, False),
                                                                                                                                 (True, True, 1, False)}


@pytest.mark.parametrize("causal", [False, True])
def test_the_largest_plans_fit_their_fields(lib, causal):
    """The most tiles that are dealt out (just under three per SM, or all of two pairs per SM) over the longest sequence."""
    for heads, nqt in ((443, 1), (222, 2), (221, 2), (147, 3), (49, 9), (1, 295), (1, 440)):
        for sms in (148, 160):
            check(lib, causal, heads, nqt, 1 << 24, (1 << 24) - 128 * nqt, 128, sms)
    assert check(lib, causal, 200, 1, 1 << 24, (1 << 24) - 128, 128, 148)
    assert not check(lib, causal, 200, 1, 1 << 24, (1 << 24) - 128, 128, SLOTS + 1)


def walk(causal, heads, nqt, sms):
    """SM by SM: what the one that ends last walks, in tiles, where each draws its next unit when it begins one, those with two tiles first."""
    npair = (nqt + 1) // 2
    pairs = [2 if nqt % 2 == 0 or (p >= heads if causal else p % npair != npair - 1) else 1 for p in range(heads * npair)]
    rest = len(pairs) % sms
    whole = len(pairs) - rest if nqt > 1 and 2 * rest <= sms else len(pairs)
    units = pairs[:whole] + [1] * sum(pairs[whole:])
    queue = iter(units[sms:])
    ends = {}                                                   # time -> units drawn by the SMs that end one then
    for u in sorted(units[:sms], reverse=True):
        ends.setdefault(u, []).append(next(queue, 0))
    t = last = 0
    while ends:
        t += 1
        for u in sorted(ends.pop(t, []), reverse=True):
            last = t
            if u:
                ends.setdefault(t + u, []).append(next(queue, 0))
    return last


def test_the_walk_without_slots(lib):
    r = random.Random(9)
    for _ in range(3000):
        sms, nqt = r.choice((148, 148, 132, 1, 2, 7, 31)), int(1.6 ** r.uniform(0, 9))
        heads, causal = max(1, int(r.uniform(0.3, 12) * sms / nqt)), r.random() < 0.5
        assert lib.split_walk(int(causal), heads, nqt, sms) == walk(causal, heads, nqt, sms), (causal, heads, nqt, sms)


@pytest.mark.parametrize("heads,N,D,shared", [(12, 2830, 64, False), (28, 3143, 64, False), (24, 3604, 128, True), (28, 3926, 128, False), (28, 3143, 128, False),      # odd numbers of tiles
                                              (5, 7547, 128, True), (6, 6245, 128, True), (3, 6272, 128, True), (6, 8997, 64, False), (5, 16384, 128, True), (24, 16384, 128, False),
                                              (64, 6979, 128, True), (24, 119056, 128, True), (32, 8192, 128, False)])
def test_slots_where_they_save_more_than_they_cost(lib, heads, N, D, shared):
    assert bool(plan(lib, False, heads, (N + 127) // 128, N, 0, D)[-1]) == shared


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("H,group,Nq,Nk,causal,rounds", test_shared_tiles_gpu.CASES)
def test_the_cases_run_on_the_gpu_are_what_they_claim(lib, D, H, group, Nq, Nk, causal, rounds):
    whole, *_, first = plan(lib, causal, H, (Nq + 127) // 128, Nk, Nk - Nq, D)
    assert (whole // 148 if first else None) == rounds


@pytest.mark.parametrize("D", [64, 128])
def test_calls_alone_share_nothing_and_both_streams_do(lib, D):
    """What the GPU tests compare with, and the problems that they run at the same time."""
    for H, group, Nq, Nk, causal, rounds in test_shared_tiles_gpu.CASES:
        assert not plan(lib, causal, 1, (Nq + 127) // 128, Nk, Nk - Nq, D)[-1]
    assert plan(lib, True, 32, 8, 6000, 5000, D)[-1] and plan(lib, False, 100, 3, 3200, 2816, D)[-1]
    assert plan(lib, True, 64, 8, 6000, 5000, D)[-1]          # two batch entries, in a workspace without room for it
    # a part of one block behind a border, some of whose rows see none of its keys
    *_, rest0, first = plan(lib, True, 48, 7, 4166, 3381, D)
    tile = (C.c_int * 2)()
    alone = 0
    for j, lo in first:
        lib.split_tile(1, j, 7, 48, 0, rest0, tile)
        alone += 0 < lo == lib.split_blocks(1, tile[1], 4166, 3381) - 1
    assert alone >= 3 and 3381 % 128 > 32
