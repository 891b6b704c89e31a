"""The geometry expansion's counters (emit_slot in csrc/persistent.cuh, compiled
for the host). When the levels get small, one block per side goes on alone and
the other blocks leave after reading the last level's count; one that reads
late has to find it unchanged, or it would stay at a barrier that nobody else
reaches. The levels are played through in order; CPU only, needs nvcc."""

import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "native", "emit_slots_host.cu")
OUT = os.path.join(ROOT, "tests", "_build", "emit_slots_host.so")
CSRC = os.path.join(ROOT, "dmsc_b200", "csrc")
DEPS = [SRC] + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
SLOTS = 8  # counters per side, all zero at the start


@pytest.fixture(scope="module")
def lib():
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    nvcc = cand if os.path.exists(cand) else shutil.which("nvcc")
    if not nvcc:
        pytest.skip("nvcc not available")
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in DEPS):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-Xcompiler", "-fPIC",
                               "-shared", "--expt-relaxed-constexpr", "-o", OUT + ".tmp", SRC])
        os.replace(OUT + ".tmp", OUT)
    return ctypes.CDLL(OUT)


def _play(slot, segs, first_solo, levels=30):
    """Counts of every level in turn, as the kernel reads, clears and appends
    them: True when each level reads what the level before it appended and the
    last count of the whole grid is never written again."""
    cnt = [0] * SLOTS
    tasks = [1000 + 7 * lv for lv in range(levels + 1)]  # appended for each level
    cnt[slot(0, False)] = tasks[0]  # before the first level
    ok, held = True, None
    for lv in range(levels):
        solo = lv > first_solo  # as read at the top of the level
        ok = ok and cnt[slot(lv, solo)] == tasks[lv]
        if lv == first_solo:
            held = slot(lv, False)
        solo = lv >= first_solo  # from here on
        cnt[slot(lv + 2, solo)] = 0
        cnt[slot(lv + 1, solo)] += tasks[lv + 1]
        cnt[segs] += 1
        ok = ok and (held is None or cnt[held] == tasks[first_solo])
    return ok


@pytest.mark.parametrize("first_solo", range(8))
def test_last_grid_count_is_left_alone(lib, first_solo):
    segs = lib.emit_segs_host()
    used = [lib.emit_slot_host(lv, s) for lv in range(9) for s in (0, 1)]
    assert segs not in used and all(0 <= k < SLOTS for k in [segs, *used])
    assert _play(lambda lv, solo: lib.emit_slot_host(lv, int(solo)), segs, first_solo)
    # one rotation for both kinds of levels is what must not be
    assert not _play(lambda lv, solo: lib.emit_slot_host(lv, 0), segs, first_solo)
