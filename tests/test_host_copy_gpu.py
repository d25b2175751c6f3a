"""Results copied into pageable memory (staged, several threads) against the
same results copied into pinned memory (one direct copy)."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import openlb_b200 as ob
from tests import cases as C

pytestmark = pytest.mark.gpu


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
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
