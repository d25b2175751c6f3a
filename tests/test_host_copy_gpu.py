"""Results copied into pageable memory (staged, several threads) against the
same results copied into pinned memory (one direct copy)."""
from __future__ import annotations

import os
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np
import pytest

import openlb_b200 as ob
from tests import cases as C

pytestmark = pytest.mark.gpu


def copy_threads():
    """The library's copy threads alive in this process."""
    names = []
    for task in os.listdir("/proc/self/task"):
        try:
            names.append(Path("/proc/self/task", task, "comm").read_text().strip())
        except FileNotFoundError:  # it ended meanwhile
            pass
    return names.count("olb-copy")


def make_staged(lat):
    """Copies of 1 MiB and more take the staged way once 32 MiB have gone directly."""
    out = lat.get_moments()
    for _ in range((32 << 20) // (3 * 4 * lat.n) + 1):
        lat.get_moments(out=out)
    assert copy_threads() > 0


def pinned(lat):
    torch = pytest.importorskip("torch")
    return lat.get_moments(out=tuple(torch.empty(k * lat.n, pin_memory=True).numpy() for k in (1, 3)))


# rho of 1 MiB less 2 KiB (a direct copy), exactly 1 MiB, a little more, and 4.2 MiB;
# u three times as much, whole 512 KiB chunks and remainders
@pytest.mark.parametrize("size", [(8, 64, 511), (4, 256, 256), (5, 229, 229), (33, 257, 131)])
def test_pageable_equals_pinned(size):
    n = size[0] * size[1] * size[2]
    case = C.periodic_case(19, size)
    rng = np.random.default_rng(n)
    with ob.Lattice(19, size, case.periodic) as lat:
        lat.set_dynamics(C.to_abi_table(case))
        lat.ini_equilibrium((1 + 0.01 * rng.standard_normal(n)).astype(np.float32),
                            (0.03 * rng.standard_normal((3, n))).astype(np.float32))
        lat.collide_and_stream(3)
        want = pinned(lat)
        make_staged(lat)
        for _ in range(3):
            got = lat.get_moments()
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1].reshape(-1), want[1].reshape(-1))
        # into the middle of a larger array, not at a page's start
        room = np.full(n + 64, np.float32(7))
        room_u = np.full(3 * n + 64, np.float32(7))
        lat.get_moments(out=(room[17:17 + n], room_u[31:31 + 3 * n]))
        assert np.array_equal(room[17:17 + n], want[0]) and np.array_equal(room_u[31:31 + 3 * n], want[1].reshape(-1))
        assert np.all(room[:17] == 7) and np.all(room[17 + n:] == 7)
        assert np.all(room_u[:31] == 7) and np.all(room_u[31 + 3 * n:] == 7)


def test_threads_with_their_own_lattices():
    """One copy holds the staging ring; the others go the direct way.  Handles
    come and go while copies run."""
    errors = []

    def work(k):
        try:
            for r in range(4):
                with ob.Lattice(19, (6, 300, 300 + k), (True,) * 3) as lat:
                    n = lat.n
                    rng = np.random.default_rng(10 * k + r)
                    lat.set_dynamics([ob.BGKdynamics(omega=1.3)])
                    rho = (1 + 0.01 * rng.standard_normal(n)).astype(np.float32)
                    lat.ini_equilibrium(rho, (0.03 * rng.standard_normal((3, n))).astype(np.float32))
                    a, b = lat.get_moments(), pinned(lat)
                    if not (np.array_equal(a[0], b[0]) and np.array_equal(a[1].reshape(-1), b[1].reshape(-1))):
                        errors.append((k, r))
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    with ob.Lattice(19, (8, 64, 511), (True,) * 3) as lat:
        make_staged(lat)
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not errors, errors


def test_small_solves_make_no_ring():
    """A handle per solve: neither pinned buffers nor threads until the handles alive
    have copied 32 MiB, and none left when the last one is closed."""
    assert copy_threads() == 0
    for _ in range(4):  # 14 MB each
        with ob.Lattice(19, (96, 96, 96), (True,) * 3) as lat:
            lat.set_dynamics([ob.BGKdynamics(omega=1.3)])
            lat.get_moments()
            assert copy_threads() == 0
    with ob.Lattice(19, (96, 96, 96), (True,) * 3) as lat:
        lat.set_dynamics([ob.BGKdynamics(omega=1.3)])
        for _ in range(3):
            lat.get_moments()
        assert copy_threads() > 0
        with ob.Lattice(19, (8, 8, 8), (True,) * 3):
            pass
        assert copy_threads() > 0
    assert copy_threads() == 0


def test_a_copy_behind_a_solve_keeps_one_core_waiting():
    """get_moments called with a third of a second of steps still queued: the copy
    threads sleep until there is something to copy."""
    with ob.Lattice(19, (256, 256, 256), (True,) * 3) as lat:
        lat.set_dynamics([ob.BGKdynamics(omega=1.3)])
        lat.ini_equilibrium(np.ones(lat.n, np.float32), np.zeros((3, lat.n), np.float32))
        out = lat.get_moments()
        for _ in range(2):
            lat.get_moments(out=out)
        steps = int(350 / (lat.time_steps(20) / 20))
        assert steps < 1000  # all of them queued at once
        cpu, wall = time.process_time(), time.perf_counter()
        lat.collide_and_stream(steps)
        lat.get_moments(out=out)
        cpu, wall = time.process_time() - cpu, time.perf_counter() - wall
        # the waiting caller is 1; seven threads for the 8 ms of the copy add under 0.2
        assert wall > 0.3 and cpu / wall < 1.5, (cpu, wall)


# a program that asks for waits that sleep (cudaDeviceScheduleBlockingSync)
SLEEPING = """
import ctypes, sys, time
assert ctypes.CDLL("libcuda.so.1").cuInit(0) == 0
assert ctypes.CDLL("libcuda.so.1").cuDevicePrimaryCtxSetFlags_v2(0, 4) == 0
import numpy as np
import openlb_b200 as ob
with ob.Lattice(27, (192, 192, 192), (True,) * 3, storage="f64") as lat:  # half a millisecond a step
    lat.set_dynamics([ob.BGKdynamics(omega=1.3)])
    lat.ini_equilibrium(np.ones(lat.n), np.zeros((3, lat.n)))
    out = lat.get_moments()
    lat.get_moments(out=out)
    lat.collide_and_stream(2, stats=True)
    steps = int(400 / (lat.time_steps(20) / 20))
    assert steps < 1000  # all of them queued at once
    cpu, wall = time.process_time(), time.perf_counter()
    if sys.argv[1] == "copy":
        lat.collide_and_stream(steps)
        lat.get_moments(out=out)
    else:
        lat.collide_and_stream(steps, stats=True)
    print(time.process_time() - cpu, time.perf_counter() - wall)
"""


def cpu_and_wall_of_a_sleeping_wait(what):
    r = subprocess.run([sys.executable, "-c", SLEEPING, what], capture_output=True, text=True, timeout=300,
                       cwd=Path(__file__).resolve().parents[1])
    assert r.returncode == 0, r.stderr[-2000:]
    return (float(v) for v in r.stdout.split())


def test_a_program_whose_waits_sleep_sleeps_behind_a_solve():
    cpu, wall = cpu_and_wall_of_a_sleeping_wait("copy")
    # 0.1 s of processor time at most for enqueueing and for seven threads' part of 226 MB
    assert wall > 0.3 and cpu < 0.5 * wall, (cpu, wall)


def test_a_program_whose_waits_sleep_sleeps_for_statistics():
    cpu, wall = cpu_and_wall_of_a_sleeping_wait("statistics")
    # under 0.1 s for enqueueing and a millisecond of polling
    assert wall > 0.3 and cpu < 0.5 * wall, (cpu, wall)
