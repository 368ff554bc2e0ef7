"""The library's host code where a device or a system runs short, on a CUDA runtime that runs nothing (fake_runtime.py): what
it launches, allocates and reports, not what the kernels compute."""
import os
import subprocess
import sys

import numpy as np
import pytest

import fake_runtime
from fake_runtime import (ATTRIBUTES, FAILED, FUSED_ONE, FUSED_SEVERAL, FUSED_WRONG, LAUNCHES, MALLOCS, NULL_TABLES, REPLAYS,
                          STALE_REPLAYS)


@pytest.fixture
def fake():
    gsb, dev = fake_runtime.load()
    dev.fake_set_capacity(1 << 40)
    dev.fake_reset()
    yield gsb, dev
    dev.fake_set_capacity(1 << 40)


def plan(n, seed=11):
    import workloads
    return workloads.matching_instance(n, n, seed, 8, 20000)["plan"]


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("n,prefix", [(16, 0), (36, 0), (36, 20)])
def test_launches_per_item(fake, n, prefix, prec):
    """Every mode's count is what a call of one item queues (beside the item index, and the least conditional of a
    'prob'): a whole item of a narrow plan is one launch, without an index."""
    gsb, dev = fake
    with gsb.Engine.from_text(plan(n), precision=prec) as eng:
        eng.set_hybrid_prefix(prefix)
        line = np.zeros((1, eng.ns), np.int8)
        index = 0 if n == 16 else 1

        def queued(call):
            before = dev.fake_count(LAUNCHES)
            call()
            return dev.fake_count(LAUNCHES) - before - index
        assert queued(lambda: eng.hybrid(line, 1)) == eng.launches_per_item(2)
        assert queued(lambda: eng.sample(1, 1)) == eng.launches_per_item(1)
        assert queued(lambda: eng.chain(line)) == eng.launches_per_item(0)
        if n == 16:
            assert [eng.launches_per_item(m) for m in range(3)] == [1, 1, 1]
        else:   # a hybrid item without a prefix: a norm and a write pass per wide step, as unfused sampling
            eng.set_hybrid_prefix(0)
            hybrid = eng.launches_per_item(2)
            eng.set_fusion(1)
            assert hybrid == eng.launches_per_item(1) == eng.launches_per_item(2)


def batch_strings(plans, K, npre=2, nsuf=2):
    ns = [int(p.split()[1]) for p in plans]
    return [K] * len(plans), [np.zeros((npre, K), np.int8)] * len(plans), \
        [np.zeros((npre, nsuf, n - K), np.int8) for n in ns]


def test_batch_without_room_for_other_strings(fake):
    """A set_strings that runs out of memory at any of its allocations leaves a batch that runs the strings it had, or says
    that it has none, never one whose launch has no pass table; and that takes new strings once there is room."""
    gsb, dev = fake
    plans = [plan(n) for n in (18, 24)]
    b = gsb.Batch(plans)
    failed = 0
    for room in (0, 1 << 8, 1 << 10, 1 << 12, 1 << 14, 1 << 15, 1 << 16, 1 << 17):
        b.set_strings(*batch_strings(plans, 8))
        b.run()
        dev.fake_set_capacity(dev.fake_used() + room if room else 0)
        try:
            b.set_strings(*batch_strings(plans, 9, npre=64, nsuf=16))
        except gsb.GsbError:
            failed += 1
        dev.fake_set_capacity(1 << 40)
        try:
            b.run()
        except gsb.GsbError as e:
            assert "no strings set" in str(e)
        assert dev.fake_count(NULL_TABLES) == 0
    assert failed > 3
    b.close()
    assert dev.fake_used() == 0


def test_batch_without_threads(fake, tmp_path):
    """Pass lists are made by several threads where the system has them, and by the caller alone where it has none."""
    lib = str(tmp_path / "no_threads.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", lib, os.path.join(fake_runtime.HERE, "fake_cuda", "no_threads.c")], check=True)
    texts = tmp_path / "plan.txt"
    texts.write_text(plan(18))
    run = """
import ctypes, sys
lib = ctypes.CDLL(sys.argv[1])
text = open(sys.argv[2], "rb").read()
n, K = 40, 8
ns = int(text.split()[1])
h = ctypes.c_void_p()
assert lib.gsb_batch_open((ctypes.c_char_p * n)(*[text] * n), (ctypes.c_size_t * n)(*[len(text)] * n), n, 64, 0, ctypes.byref(h)) == 0
zeros = (ctypes.c_int8 * (n * ns))()
assert lib.gsb_batch_set_strings(h, (ctypes.c_int * n)(*[K] * n), 1, 1, zeros, zeros) == 0
out = (ctypes.c_double * n)()
assert lib.gsb_batch_run(h, out, None) == 0
"""
    r = subprocess.run([sys.executable, "-c", run, fake_runtime.LIB, str(texts)], env=dict(os.environ, LD_PRELOAD=lib),
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


def test_batch_without_room_for_another_shape(fake):
    """A shape whose item lists or arenas find no memory leaves no graph behind that points at freed ones."""
    gsb, dev = fake
    plans = [plan(n) for n in (18, 24)]
    b = gsb.Batch(plans)
    b.set_strings(*batch_strings(plans, 8))
    small, large = (128, 12, 1), (128, 12, 4)
    b.set_shape(*large)
    b.run()
    b.set_shape(*small)          # the arenas of the larger shape serve it
    b.run()
    dev.fake_set_capacity(0)
    b.set_shape(*large)
    with pytest.raises(gsb.GsbError):
        b.run()
    b.set_shape(*small)
    try:
        b.run()
    except gsb.GsbError:
        pass
    assert dev.fake_count(STALE_REPLAYS) == 0
    dev.fake_set_capacity(1 << 40)
    for shape in (small, large):
        b.set_shape(*shape)
        b.run()
    assert dev.fake_count(STALE_REPLAYS) == dev.fake_count(NULL_TABLES) == 0
    b.close()
    assert dev.fake_used() == 0


def test_errors_that_were_reported_do_not_come_back(fake):
    """An allocation that failed is its own call's error, not that of the next call whose launches are checked."""
    gsb, dev = fake
    plans = [plan(36), plan(24)]
    with gsb.Engine.from_text(plans[0], precision=128) as eng:
        line = np.zeros((1, eng.ns), np.int8)

        def without_room(call):
            dev.fake_set_capacity(0)
            with pytest.raises(gsb.GsbError):
                call()
            dev.fake_set_capacity(1 << 40)
            eng.prob(line)
        eng.prob(line)
        b = gsb.Batch(plans)
        without_room(lambda: b.set_strings(*batch_strings(plans, 8)))
        b.set_strings(*batch_strings(plans, 8))
        without_room(b.run)
        without_room(lambda: gsb.Batch(plans))
        without_room(lambda: gsb.Engine.from_text(plans[1]))
        without_room(lambda: gsb.GradSweep(plans[1]))
        without_room(lambda: gsb.dp_extend(np.ones(1, complex), 0, 0, 0, [], [], [1, 0, 1, 0]))
        b.close()


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("room", [0, 1, 2, 5, 31, 64])
def test_slots_where_arenas_do_not_fit(fake, room, prec):
    """A call of 100 strings on a device with room for `room` arenas beside the engine's: as many slots as fit (two slots take
    one arena more, the engine's own being one of them), found once, with a call of few strings before and after it."""
    gsb, dev = fake
    text = plan(36)
    arena = (16 if prec == 128 else 8) << int(text.split()[2])
    slots = max([1] + [s for s in (2, 4, 8, 16, 32, 64) if (1 if s == 2 else s) <= room])
    with gsb.Engine.from_text(text, precision=prec) as eng:
        few, many = np.zeros((min(slots, 4), eng.ns), np.int8), np.zeros((100, eng.ns), np.int8)
        eng.chain(few)
        small = dev.fake_used()
        dev.fake_set_capacity(small + max(0, room - (0 if slots == 1 else 1 if len(few) == 2 else len(few))) * arena)
        dev.fake_reset()
        eng.chain(many)
        tried = dev.fake_count(FAILED)
        assert dev.fake_count(REPLAYS) == -(-100 // slots)
        dev.fake_reset()
        for _ in range(2):
            eng.chain(many)
            eng.chain(few)
        assert dev.fake_count(FAILED) == dev.fake_count(MALLOCS) == 0 and tried <= 7
        assert dev.fake_count(REPLAYS) == 2 * (-(-100 // slots) + 1)


@pytest.mark.parametrize("prec", [128, 64])
def test_batch_without_room_for_cluster_arenas(fake, prec):
    """Cluster teams have arenas beside those of the block teams. Without room for both, or above the tuner's bound, the wide
    instances go to block teams."""
    gsb, dev = fake
    # one instance of width 15 whose cost is above an even share of the batch, 300 of the same width below it: both kinds of
    # teams have arenas of 2^15 entries
    plans = [plan(38, 5)] * 300 + [plan(39, 3)]
    assert {p.split()[2] for p in plans} == {"15"}
    b = gsb.Batch(plans, precision=prec)
    b.set_strings(*batch_strings(plans, 8, 1, 1))
    b.run()
    both, with_clusters = dev.fake_largest(), dev.fake_used()
    b.close()
    assert dev.fake_used() == 0
    b = gsb.Batch(plans, precision=prec)
    b.set_strings(*batch_strings(plans, 8, 1, 1))
    dev.fake_reset()
    dev.fake_set_capacity(with_clusters - (1 << 20))
    b.run()
    assert dev.fake_largest() < both
    dev.fake_reset()
    b.run()
    assert dev.fake_count(MALLOCS) == 0
    b.close()


@pytest.mark.parametrize("prec", [128, 64])
def test_opens_load_no_kernel(fake, prec):
    """Asking for a kernel's attributes loads it. An open of a narrow engine, a batch or a gradient sweep leaves that to the
    first call, and an engine whose runs fit the default shared memory never asks."""
    gsb, dev = fake
    text = plan(24)
    with gsb.Engine.from_text(text, precision=prec) as eng:
        assert dev.fake_count(ATTRIBUTES) == 0
        eng.prob(np.zeros((1, eng.ns), np.int8))
        assert dev.fake_count(ATTRIBUTES) == 0
    b = gsb.Batch([text], precision=prec)
    g = gsb.GradSweep(text)
    assert dev.fake_count(ATTRIBUTES) == 0
    b.set_strings(*batch_strings([text], 8))
    b.run()
    assert dev.fake_count(ATTRIBUTES) == 1
    b.close()
    g.close()


@pytest.mark.parametrize("prec", [128, 64])
def test_runs_that_need_shared_memory_ask_for_it(fake, prec):
    """A run over 2^12 entries of complex128 needs 64 KB; of complex64, 32 KB."""
    gsb, dev = fake
    text = plan(36)
    with gsb.Engine.from_text(text, precision=prec) as eng:
        opened = dev.fake_count(ATTRIBUTES)
        line = np.zeros((1, eng.ns), np.int8)
        eng.chain(line)
        eng.chain(line)
        assert dev.fake_count(ATTRIBUTES) == opened + (1 if prec == 128 else 0)


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("count", [1, 2, 3, 100])
def test_fused_kernels_by_items(fake, count, prec):
    """Launches of one item take the kernels whose pointers are parameters, launches of several those that compute them."""
    gsb, dev = fake
    with gsb.Engine.from_text(plan(44), precision=prec) as eng:
        lines = np.zeros((count, eng.ns), np.int8)
        eng.set_hybrid_prefix(eng.ns - 4)
        for call in (lambda: eng.chain(lines), lambda: eng.sample(count, 1), lambda: eng.hybrid(lines, 1)):
            dev.fake_reset()
            call()
            one, several = dev.fake_count(FUSED_ONE), dev.fake_count(FUSED_SEVERAL)
            assert (one > 0, several > 0) == (count == 1, count > 1) and dev.fake_count(FUSED_WRONG) == 0


@pytest.mark.parametrize("prec", [128, 64])
def test_tables_take_the_place_of_slots(fake, prec):
    """A dump or a resume that finds no memory beside the slots' arenas takes theirs; a later call of several strings goes
    on with as many as fit."""
    gsb, dev = fake
    text = plan(36)
    entry = 16 if prec == 128 else 8
    with gsb.Engine.from_text(text, precision=prec) as eng:
        lines = np.zeros((64, eng.ns), np.int8)
        K = max(range(eng.ns), key=lambda k: np.ldexp(eng.dump_shape(k)[1], eng.dump_shape(k)[0]))
        nk, ntq = eng.dump_shape(K)
        table = (entry * ntq) << nk
        slices = 20
        eng.chain(lines)
        arenas = (64 * entry) << int(text.split()[2])
        assert arenas > (slices + 1) * table
        dev.fake_set_capacity(dev.fake_used() + table // 2)
        dump, ls, _ = eng.prefix(lines[0], K)
        eng.chain(lines)
        eng.resume(lines[0], K, 1, 0, [dump] * slices, [ls] * slices)
        eng.chain(lines)
        dev.fake_reset()
        eng.chain(lines)
        assert dev.fake_count(FAILED) == 0 and dev.fake_count(REPLAYS) < 64


def test_batch_without_one_of_its_buffers(fake):
    """The same, whichever allocation of a set_strings or of the run after it fails."""
    gsb, dev = fake
    plans = [plan(n) for n in (18, 24)]
    for nth in range(1, 12):
        b = gsb.Batch(plans)
        for K, npre in ((4, 1), (8, 2)):
            dev.fake_fail(nth if K == 8 else 0)
            try:
                b.set_strings(*batch_strings(plans, K, npre=npre))
                b.run()
            except gsb.GsbError as e:
                assert K == 8 and "out of memory" in str(e)
        dev.fake_fail(0)
        try:
            b.run()
        except gsb.GsbError as e:
            assert "no strings set" in str(e)
        b.set_strings(*batch_strings(plans, 8))
        b.run()
        b.close()
    assert dev.fake_count(NULL_TABLES) == dev.fake_count(STALE_REPLAYS) == 0 < dev.fake_count(FAILED)


def test_batch_with_other_prefix_lengths(fake):
    """Prefix lengths that change from call to call take no device memory once their passes and strings have had room, and
    keep the graph."""
    gsb, dev = fake
    plans = [plan(n) for n in (12, 18, 24, 36)]
    b = gsb.Batch(plans)
    for turn in range(3):
        dev.fake_reset()
        for K in range(1, 12):
            b.set_strings(*batch_strings(plans, K))
            b.run()
    assert dev.fake_count(MALLOCS) == 0 and dev.fake_count(LAUNCHES) == 0 and dev.fake_count(REPLAYS) == 11
    b.close()
    assert dev.fake_used() == 0
