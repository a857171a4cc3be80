"""The commit kernels' warp code on the CPU: the device headers themselves, compiled for the host
against tests/warp_emu (each lane a fiber, a seeded scheduler between any two accesses to memory), so
that interleavings of a few warps which the GPU meets once in millions are run on purpose."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import csmv_gb300 as cg
import oracle as orc
from oracle import p

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "csmv-gpu-stm_gb300" / "csrc"


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    d = tmp_path_factory.mktemp("warp_emu")
    src = d / "csmv-gpu-stm_gb300" / "csrc"
    src.mkdir(parents=True)
    (d / "include").mkdir()
    for f in ("csmv.h", "csmv_tx.cuh"):
        shutil.copy(ROOT / "include" / f, d / "include")
    for f in ("bank_kernel.cuh", "memcd_kernel.cuh"):
        shutil.copy(CSRC / f, src)
    here = Path(__file__).parent / "warp_emu"
    shutil.copy(here / "csmv_prims.cuh", src)
    for f in ("cooperative_groups.h", "driver.cpp"):
        shutil.copy(here / f, d)
    lib = d / "libemu.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-w", "-fPIC", "-shared", f"-I{d}", str(d / "driver.cpp"),
                    "-o", str(lib)], check=True)
    so = C.CDLL(str(lib))
    P, U = C.c_void_p, C.c_uint32
    so.emu_memcd.argtypes = [U, U, P, P, P, P, U, C.c_uint64, U, P, P, P, P, P, U, P, P]
    so.emu_complete.argtypes = [U, U, P, P, U, U, C.c_uint64, P, P]
    so.emu_short_funds.argtypes, so.emu_short_funds.restype = [U, P, P, U, P, C.c_uint64, P], U
    so.emu_write_overlap.argtypes = [P, P, U, P]
    return so


def _cache_run(emu, seed, *, warps=6, rounds=24, n_sets=1, n_keys=20, switch_log2=4):
    """Rounds of one key each (a round's SETs share a hold), every round under its own LRU tick, from
    an empty table; the commit log replayed one SET at a time."""
    rng = np.random.default_rng(seed)
    n = 32 * rounds
    req = cg.memcd_generate(cg.memcd_workload(1 << 12, n, seed=seed, get_pct=0, dist=cg.DIST_UNIFORM))
    ids = rng.integers(0, n_keys, rounds).repeat(32).astype(np.uint32)
    req.key[:] = np.stack([ids, ids * np.uint32(2654435761), ids ^ np.uint32(0x5bd1e995), ids + np.uint32(7)], 1)
    ticks = rng.permutation(rounds).astype(np.uint32) + np.uint32(1)
    tags, recs = orc.memcd_empty_table(n_sets)
    cap = 1 << 16
    found, val_out = np.zeros(n, np.uint32), np.zeros((n, 8), np.uint32)
    log, outcome, end = np.full(cap, 0xFFFFFFFF, np.uint32), np.zeros(n, np.uint32), C.c_uint32()
    kind, key, val = (np.ascontiguousarray(a, np.uint32) for a in (req.kind, req.key, req.val))
    rc = emu.emu_memcd(warps, rounds, p(kind), p(key), p(val), p(ticks), n_sets, seed,
                       switch_log2, p(tags), p(recs), p(found), p(val_out), p(log), cap, p(outcome),
                       C.byref(end))
    assert rc == 0, rc
    table = orc.memcd_empty_table(n_sets)
    sets = 0
    for ts in range(1, end.value + 1):
        r = int(log[ts - 1])
        if r == 0xFFFFFFFF:
            continue
        assert outcome[r] == ts
        sets += 1
        table = orc.memcd_serial(kind[r:r + 1], key[r:r + 1], val[r:r + 1], int(ticks[r // 32]), n_sets, table,
                                 ts - 1)[4:]
    assert sets == int(kind.sum())
    return tags, recs, table, end.value - sets


@pytest.mark.parametrize("seed", range(2))
def test_cache_versions_survive_failed_sets(emu, seed):
    """SETs of different keys in one cache set under differing ticks: a SET that fails its validation
    puts back the older version that it withdrew, whatever other SETs did to it meanwhile, and the
    table equals the replay of the commit log, both versions of every entry."""
    holes = 0
    for s in range(45):
        tags, recs, table, h = _cache_run(emu, 45 * seed + s)
        holes += h
        np.testing.assert_array_equal(tags, table[0])
        np.testing.assert_array_equal(recs, table[1])
    assert holes > 0  # validations did fail


@pytest.mark.parametrize("warps", [1, 2, 5])
@pytest.mark.parametrize("clock0", [0, 31, 4000])
def test_clock_covers_only_acquired_completions(emu, warps, clock0):
    """The warp that moves the clock has acquired, in each lane, the completion words it moves it
    over: what a snapshot at the new clock reads was written back before. The clock ends behind the
    last range."""
    rng = np.random.default_rng(clock0 + warps)
    for seed in range(5):
        end = clock0 + np.cumsum(rng.integers(1, 33, 100))
        lo = np.concatenate([[clock0], end[:-1]]) + 1
        perm = rng.permutation(100)
        lo, hi = lo[perm].astype(np.uint32), end[perm].astype(np.uint32)
        fin, bad = C.c_uint32(), C.c_uint32()
        assert emu.emu_complete(warps, 100, p(lo), p(hi), clock0, 127, seed, C.byref(fin), C.byref(bad)) == 0
        assert fin.value == end[-1]
        assert bad.value == 0


@pytest.mark.parametrize("nr", [2, 3, 8])
def test_transfers_without_funds_look_twice_behind_a_fence(emu, nr):
    """A transfer that writes nothing commits on two looks at its accounts' commit words; a fence
    of the lane lies between them."""
    rng = np.random.default_rng(nr)
    addr = rng.permuted(np.tile(np.arange(40), (32, 1)), axis=1)[:, :nr].astype(np.uint32)
    op = np.full(32, cg.KIND_TRANSFER | nr << 2 | 5 << 8 | 4095 << 20, np.uint32)
    value = np.full(40, 4, np.int32)
    addr = np.ascontiguousarray(addr)
    bad = C.c_uint32()
    assert emu.emu_short_funds(nr, p(op), p(addr), 40, p(value), 1, C.byref(bad)) == 0xFFFFFFFF
    assert bad.value == 0


def test_write_overlap_names_the_lower_lanes_with_a_common_address(emu):
    rng = np.random.default_rng(4)
    for case in range(40):
        n_acc = int(rng.choice([2, 10, 64, 1000]))
        ws, nws = rng.integers(0, n_acc, (32, 2)).astype(np.uint32), rng.integers(0, 3, 32).astype(np.uint32)
        active = int(rng.integers(0, 1 << 32))
        out = np.zeros(32, np.uint32)
        emu.emu_write_overlap(p(ws), p(nws), active, p(out))
        sets = [set(ws[l, :nws[l]].tolist()) if active >> l & 1 else set() for l in range(32)]
        for l in range(32):
            assert out[l] == sum(1 << i for i in range(l) if sets[i] & sets[l])
