"""Step-kernel tiling, the two-cell kernel of the natural 16-bit layout, the
statistics reduction and chained launches, at the sizes where they change over:
planes smaller than a block, exactly a block, one cell more; block counts on
both sides of the in-kernel reduction."""
from __future__ import annotations

import numpy as np
import pytest

import openlb_b200 as ob
from oracle import oracle as O
from tests import cases as C

pytestmark = pytest.mark.gpu

STEPS = 4
# 16-bit storage rounds every stored deviation once per step, by at most half a
# unit in the last place (2^-11 FP16, 2^-8 BF16 relative); the collision spreads
# that over the other populations with weights summing to at most |1 - omega| +
# omega < 4: errors stay below 4 * steps roundings of the largest deviation.
UNIT = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8}


def advance(case, f0, steps, storage, shape=None, variant=None):
    with ob.Lattice(case.q, case.size, case.periodic, storage=storage) as lat:
        lat.set_dynamics(C.to_abi_table(case), case.dyn_id)
        if shape:
            lat.set_launch_shape(*shape)
        if variant is not None:
            lat.set_step_variant(variant)
        lat.set_populations(f0)
        lat.collide_and_stream(steps)
        return lat.get_populations()


def check(case, f0, got, storage):
    ref = f0.copy()
    O.step(case, ref, STEPS)
    if storage in UNIT:
        valid = ~np.isnan(ref)
        bound = 4 * STEPS * UNIT[storage] * max(np.abs(f0).max(), np.abs(ref[valid]).max())
        assert np.abs(got - ref)[valid].max() <= bound
    else:
        rel, _ = C.pop_tolerance_violation(case.q, got, ref, 1e-5)
        assert rel <= 1e-5, rel


# planes (ny * nz) of 1, 63, 64, 65, 128, 129, 255, 256, 257, 513 cells
PLANES = [(1, 1), (7, 9), (4, 16), (5, 13), (8, 16), (3, 43), (5, 51), (16, 16), (257, 1), (19, 27)]


# 16-bit with odd nx: one cell per thread (variant 0) and two (1)
@pytest.mark.parametrize("storage,nx,variant", [("f32", 3, None), ("f16", 4, None), ("f16", 3, 0), ("f16", 3, 1),
                                                ("bf16", 5, 0), ("bf16", 5, 1)])
@pytest.mark.parametrize("plane", PLANES)
def test_periodic_planes_around_a_block(storage, nx, variant, plane):
    rng = np.random.default_rng(31 + plane[0])
    case = C.periodic_case(19, (nx,) + plane, kind=O.FORCED_TRT)
    f0 = C.random_state(19, case.n, np.float32, rng)
    check(case, f0, advance(case, f0, STEPS, storage, variant=variant), storage)


@pytest.mark.parametrize("storage", ["f32", "f64"])
@pytest.mark.parametrize("variant", range(4))
@pytest.mark.parametrize("plane", PLANES)
def test_planes_around_a_block_in_every_step_variant(storage, variant, plane):
    """One and two cells per thread (a second run that is empty, partial, full)."""
    dtype, rtol = (np.float32, 1e-5) if storage == "f32" else (np.float64, 1e-12)
    case = C.periodic_case(19, (3,) + plane, kind=O.FORCED_TRT)
    f0 = C.random_state(19, case.n, dtype, np.random.default_rng(37 + plane[0]))
    ref = f0.copy()
    O.step(case, ref, STEPS)
    with ob.Lattice(19, case.size, case.periodic, storage=storage) as lat:
        lat.set_dynamics(C.to_abi_table(case))
        lat.set_step_variant(variant)
        lat.set_populations(f0)
        lat.collide_and_stream(STEPS - 1)
        assert lat.collide_and_stream(1, stats=True)["n_cells"] == case.n
        rel, _ = C.pop_tolerance_violation(19, lat.get_populations(), ref, rtol)
    assert rel <= rtol, rel


@pytest.mark.parametrize("q,storage,nx,variant", [(19, "f16", 5, 0), (19, "f16", 5, 1), (27, "bf16", 5, 0),
                                                  (27, "bf16", 5, 1), (19, "f16", 6, None), (19, "f32", 5, None)])
@pytest.mark.parametrize("plane", [(7, 9), (3, 43), (16, 16), (9, 57)])
def test_cavity_planes_around_a_block(q, storage, nx, variant, plane):
    rng = np.random.default_rng(57 + plane[1])
    case = C.cavity_case(q, (nx,) + plane)
    f0 = C.random_state(q, case.n, np.float32, rng, amp_u=0.01)
    # slots fed from outside the box hold what the wrap brings; only walls read them
    check(case, f0, advance(case, f0, STEPS, storage, variant=variant), storage)


def test_flat_tiles_and_rectangles_agree():
    """The same instantiation cut either way: bit for bit."""
    rng = np.random.default_rng(3)
    for case in (C.periodic_case(19, (6, 21, 37)), C.cavity_case(19, (6, 21, 37))):
        f0 = C.random_state(19, case.n, np.float32, rng, amp_u=0.01)
        flat = advance(case, f0, 5, "f32")
        for shape in ((32, 8), (64, 4), (32, 1)):
            assert np.array_equal(flat, advance(case, f0, 5, "f32", shape), equal_nan=True)


# one block per plane: 1024 blocks reduce in the step kernel, 1025 and 4099 in a
# kernel of their own (2 and 5 blocks)
@pytest.mark.parametrize("nx", [7, 1024, 1025, 4099])
def test_statistics_around_the_in_kernel_reduction(nx):
    rng = np.random.default_rng(nx)
    case = C.periodic_case(19, (nx, 16, 16))
    f0 = C.random_state(19, case.n, np.float32, rng)
    with ob.Lattice(19, case.size, case.periodic) as lat:
        lat.set_dynamics(C.to_abi_table(case))
        lat.set_step_variant(1)  # one cell per thread
        lat.set_populations(f0)
        for _ in range(3):  # again: the reduction leaves its counters as it found them
            rho, u = (a.astype(np.float64) for a in lat.get_moments())
            st = lat.collide_and_stream(1, stats=True)
            u2 = (u * u).sum(0)
            assert st["n_cells"] == case.n and st["n_nonfinite"] == 0
            # per-cell values are FP32 (2^-24 relative, a few operations each), their sums FP64
            np.testing.assert_allclose(st["sum_rho"], rho.sum(), rtol=1e-6)
            np.testing.assert_allclose(st["sum_usqr"], u2.sum(), rtol=1e-5)
            np.testing.assert_allclose(st["max_usqr"], u2.max(), rtol=1e-5)


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("boundary", [False, True])
def test_chained_steps_equal_separate_steps(storage, boundary):
    """Launches that overlap their predecessor's end give what launches with a
    synchronisation between them give, bit for bit."""
    rng = np.random.default_rng(12)
    case = (C.interpolated_channel_case(19, (14, 12, 10)) if boundary else C.cavity_case(19, (14, 12, 10)))
    f0 = C.random_state(19, case.n, np.float32, rng, amp_u=0.01)
    out = []
    for together in (True, False):
        with ob.Lattice(19, case.size, case.periodic, storage=storage) as lat:
            lat.set_dynamics(C.to_abi_table(case), case.dyn_id)
            if boundary:
                lat.set_boundary_values(*C.boundary_cells_and_values(case))
                lat.set_boundary_noise(0.02, 5)
            lat.set_populations(f0)
            if together:
                lat.collide_and_stream(60)
            else:
                for _ in range(60):
                    lat.collide_and_stream(1)
                    lat.synchronize()
            out.append(lat.get_populations())
    assert np.array_equal(out[0], out[1], equal_nan=True)


@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_caller_owned_steps_under_graph_capture(storage):
    """Chained launches captured into a CUDA graph: a replay gives what the calls give."""
    import ctypes

    torch = pytest.importorskip("torch")
    from openlb_b200 import _abi

    size, steps = (9, 20, 33), 6
    n = size[0] * size[1] * size[2]
    dtype = torch.float32 if storage == "f32" else torch.bfloat16
    start = (1e-3 * torch.randn(19, (n + 63) // 64 * 64, generator=torch.Generator().manual_seed(1))).to(dtype).cuda()
    lib = _abi.load()
    desc = _abi.Desc()
    desc.q, desc.nx, desc.ny, desc.nz = (19,) + size
    for e in range(3):
        desc.periodic[e] = 1
    desc.storage = _abi.STORAGE[storage]
    bulk = ob.BGKdynamics(omega=1.4).params()

    def call(buf, stream):
        _abi.check(lib, lib.olb_b200_collide_and_stream_noalloc(
            ctypes.byref(desc), ctypes.c_void_p(buf.data_ptr()), 0, ctypes.byref(bulk), steps, None,
            ctypes.c_void_p(stream)))

    want, got = start.clone(), start.clone()
    call(want, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(got, torch.cuda.current_stream().cuda_stream)
    assert torch.equal(got, start)  # captured, not run
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)


def test_force_field_outlives_set_dynamics():
    """The FORCE field stays the lattice's until it is removed: setting the dynamics
    again neither frees nor forgets it."""
    rng = np.random.default_rng(6)
    case = C.with_force_field(C.periodic_case(19, (8, 9, 10), kind=O.FORCED_BGK), np.float32, rng)
    f0 = C.random_state(19, case.n, np.float32, rng)
    out = []
    for again in (False, True):
        with ob.Lattice(19, case.size, case.periodic) as lat:
            lat.set_dynamics(C.to_abi_table(case))
            lat.set_force_field(case.force_field)
            if again:
                lat.set_dynamics(C.to_abi_table(case))
            lat.set_populations(f0)
            lat.collide_and_stream(4)
            out.append(lat.get_populations())
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("q,storage", [(19, "f16"), (19, "bf16"), (27, "f16")])
@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("kind", [ob.BGKdynamics(omega=1.2), ob.ForcedBGKdynamics(omega=1.2, force=(1e-4, 0, 0))],
                         ids=["bgk", "forced"])
def test_cells_that_pass_through_keep_their_bits(q, storage, kind, variant):
    """NoDynamics cells among fluid, walls and moving walls in 16-bit storage, odd nx (one
    cell per thread and two): what streams out of them is what was stored, bit for bit, with pairs of populations of
    very different size and with an infinity or NaN in one population of a cell."""
    rng = np.random.default_rng(5)
    size = (5, 9, 29)
    n = 5 * 9 * 29
    ids = rng.choice(4, n, p=[0.5, 0.3, 0.1, 0.1]).astype(np.uint8)
    f0 = (rng.choice([-1, 1], (q, n)) * np.exp2(rng.uniform(-18, -2, (q, n)))).astype(np.float32)
    passing = np.flatnonzero(ids == 1)
    for value, cells in ((np.inf, passing[::7]), (np.nan, passing[3::7])):
        f0[rng.integers(0, q, len(cells)), cells] = value
    source = (ids == 1).reshape(size)
    with ob.Lattice(q, size, (True,) * 3, storage=storage) as lat:
        lat.set_dynamics([kind, ob.NoDynamics(), ob.BounceBack(), ob.BounceBackVelocity((0.03, 0, 0))], ids)
        lat.set_step_variant(variant)
        lat.set_populations(f0.reshape(-1))
        before = lat.get_populations().reshape((q,) + size)
        for _ in range(3):  # both parities
            lat.collide_and_stream(1)
            after = lat.get_populations().reshape((q,) + size)
            for i, c in enumerate(ob.descriptor(q).c):
                came = np.roll(source, c, axis=(0, 1, 2))
                assert np.array_equal(after[i][came], np.roll(before[i], c, axis=(0, 1, 2))[came], equal_nan=True)
            before = after


@pytest.mark.parametrize("storage,nx", [("f16", 5), ("bf16", 5), ("f16", 6), ("f32", 5)])
def test_a_launch_shape_is_what_runs(storage, nx):
    """A shape set by the caller cuts the step's blocks: the populations are the same bit
    for bit, the sums of the statistics are added in another order.  The velocities
    range over five decades, so that the order shows in some of the FP64 sums."""
    rng = np.random.default_rng(8)
    size = (nx, 61, 75)
    n = nx * 61 * 75
    fields = [(rng.choice([-1, 1], (3, n)) * 10 ** rng.uniform(-6, -1, (1, n))).astype(np.float32) for _ in range(24)]
    out, sums = [], set()
    with ob.Lattice(19, size, (True,) * 3, storage=storage) as lat:
        lat.set_dynamics([ob.BGKdynamics(omega=1.3)])
        for shape in ((0, 0), (64, 2), (32, 1)):
            lat.set_launch_shape(*shape)
            seen = []
            for u in fields:
                lat.ini_equilibrium(np.ones(n, np.float32), u)
                seen.append(lat.collide_and_stream(1, stats=True)["sum_usqr"])
            sums.add(tuple(seen))
            lat.collide_and_stream(2)
            out.append(lat.get_populations())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    assert len(sums) == 3


# launch shapes timed at nz = 75: 64x4, 32x8 and flat tiles
@pytest.mark.parametrize("storage,nx,kernels", [
    ("f16", 5, [(1, 3), (2, 3), (1, 3), (2, 3)]),          # natural layout: one or two cells
    ("f16", 6, [(1, 3), (1, 4), (1, 3), (1, 4)]),          # one element per thread
    ("f32", 5, [(1, 3), (1, 4), (2, 2), (2, 3)]),
])
def test_tuning_reports_the_kernel_that_runs(storage, nx, kernels):
    with ob.Lattice(19, (nx, 20, 75), (True,) * 3, storage=storage) as lat:
        lat.set_dynamics([ob.BGKdynamics(omega=1.3)])
        for variant, kernel in enumerate(kernels):
            lat.set_step_variant(variant)
            t = lat.tuning()
            assert (t["variant"], t["cells_per_thread"], t["min_blocks_per_sm"]) == (variant,) + kernel
        assert lat.autotune(2)["candidates"] == 3 * len(set(kernels))


# the default of each lattice class on both sides of its changes: one wave (148 * 3
# blocks of 256 threads: 48 x 48 x 49 cells fit, 49 x 51 x 47 do not), 2^21 cells
@pytest.mark.parametrize("q,storage,size,open_,walls,open_forced,walls_forced", [
    (19, "f32", (48, 48, 49), 0, 0, 0, 0), (19, "f32", (49, 51, 47), 1, 1, 1, 1), (19, "f32", (128, 128, 128), 3, 1, 1, 3),
    (27, "f32", (49, 51, 47), 1, 1, 1, 1), (27, "f32", (128, 128, 128), 3, 1, 1, 1),
    (19, "f64", (49, 51, 47), 0, 0, 0, 0), (27, "f64", (48, 48, 49), 0, 0, 0, 0), (27, "f64", (49, 51, 47), 0, 0, 2, 2),
    (19, "f16", (48, 64, 64), 0, 0, 0, 0), (19, "f16", (80, 80, 80), 1, 1, 1, 1), (27, "bf16", (80, 80, 80), 0, 0, 0, 0),
    # natural 16-bit layout: two blocks per SM (75 776 cells) in D3Q19, three in D3Q27
    # (not open BGK in D3Q19)
    (19, "f16", (37, 64, 32), 1, 0, 0, 0), (19, "bf16", (37, 64, 33), 1, 1, 1, 1),
    (27, "bf16", (37, 64, 48), 0, 0, 0, 0), (27, "f16", (49, 51, 47), 1, 1, 1, 1),
])
def test_default_step_variants(q, storage, size, open_, walls, open_forced, walls_forced):
    n = size[0] * size[1] * size[2]
    ids = (np.arange(n) % 7 == 0).astype(np.uint8)
    got = []
    with ob.Lattice(q, size, (True,) * 3, storage=storage) as lat:
        for bulk in (ob.BGKdynamics(omega=1.3), ob.ForcedTRTdynamics(omega=1.3, force=(1e-5, 0, 0))):
            for table, cells in (([bulk], None), ([bulk, ob.BounceBack()], ids)):
                lat.set_dynamics(table, cells)
                got.append(lat.tuning()["variant"])
    assert got == [open_, walls, open_forced, walls_forced]


@pytest.mark.parametrize("drop", ["set_dynamics", "set_step_variant"])
def test_a_dropped_tuning_takes_its_launch_shape_along(drop):
    """What the autotuner chose for one kernel class is not left to another: the lattice
    is as one that was never tuned.  (Several sizes: the tuner may choose the default.)"""
    walls = [ob.BGKdynamics(omega=1.3), ob.BounceBack()]
    for nz in (64, 100, 128, 192, 250, 256, 300, 384):
        size = (16, 24, nz)
        ids = (np.arange(16 * 24 * nz) % 5 == 0).astype(np.uint8)
        seen = []
        for tune in (False, True):
            with ob.Lattice(19, size, (True,) * 3) as lat:
                lat.set_dynamics([walls[0]])
                if tune:
                    assert lat.autotune(2)["tuned"]
                if drop == "set_dynamics":
                    lat.set_dynamics(walls, ids)
                else:
                    lat.set_step_variant(1)
                seen.append(lat.tuning())
        assert not seen[1]["tuned"] and seen[0] == seen[1], (nz, seen)


@pytest.mark.parametrize("storage,nx,threads", [("f32", 5, 256), ("f64", 6, 256), ("f16", 5, 64), ("bf16", 6, 64)])
@pytest.mark.parametrize("nz", [9, 75, 300])
def test_the_reported_block_is_the_one_launched(storage, nx, threads, nz):
    with ob.Lattice(19, (nx, 20, nz), (True,) * 3, storage=storage) as lat:
        lat.set_dynamics([ob.BGKdynamics(omega=1.3)])

        def reported():
            info, tuning = lat.info(), lat.tuning()
            assert (info["block_z"], info["block_y"]) == (tuning["block_z"], tuning["block_y"])
            return info["block_z"], info["block_y"]

        assert reported() == (threads, 1)  # flat tiles
        lat.set_launch_shape(32, 4)
        assert reported() == (32, 4)
        lat.set_launch_shape(0, 0)
        assert reported() == (threads, 1)
