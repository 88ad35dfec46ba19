"""GPU parity at the edges of the update's fast paths: the shared-reciprocal
quotients of the Vay push at the limits of their range, work items of tile
lists (crowded, single and empty tiles, lists around a chunk's length), the 1D
kernel's chunk lengths, the one-launch field update at its size limit and the
smoothing passes of mixed boundaries. Particles, fields and smoothed currents
bit for bit against the oracle, J and Rho within 1e-6 of their maximum of the
FP64-accumulated deposit (one FP32 rounding of an exact sum of FP32
contributions, 6e-8 each)."""
import numpy as np
import pytest

import oracle
from _cases import random_fields, random_particles
from _gpu_helpers import Pair, assert_bits, make_params

pytestmark = pytest.mark.gpu

J_TOL = 1e-6


def _state(N, n, seed, amp=0.3, periodic=(True, True), smoothing=0, tile=(0, 0)):
    params = make_params(N, periodic=periodic, capacity=max(n, 1), tile=tile,
                         smoothing=smoothing)
    m = oracle.make_mesh(params.N, params.guard, size=params.size)
    rng = np.random.default_rng(seed)
    f = random_fields(m, rng, amp=amp)
    for key in ("E", "B", "Ebg", "Bbg"):
        for c in range(3):
            oracle.send_guard_cells(m, f[key][c], (1, 1, 0))
    return params, m, rng, f


@pytest.mark.parametrize("N", [(64, 48), (512,)])
@pytest.mark.parametrize("amp", [0.0, 1e-34, 0.3, 3e4, 1e7])
def test_push_quotients_at_their_range(N, amp):
    """Zero, denormal, tiny, large and huge momentum components (gamma past
    2^24 too) in zero, tiny, ordinary and huge fields: the quotients by gamma
    equal the plain divisions on both sides of every bound."""
    params, m, rng, f = _state(N, 6000, 3, amp=amp)
    p = random_particles(m, 6000, rng)
    sizes = np.array([0.0, 1e-42, 3e-39, 7e-31, 8e-31, 1e-20, 1.0, 1e3, 1.6e7, 1.7e7, 1e9],
                     np.float32)
    for k in ("p1", "p2", "p3"):
        sgn = np.where(rng.random(6000) < 0.5, -1, 1).astype(np.float32)
        p[k][:] = sgn * sizes[rng.integers(0, len(sizes), 6000)] * (
            1 + rng.random(6000, dtype=np.float32))
    pr = Pair(params, f, p)
    pr.both_update_particles(0)
    pr.check_particles()


@pytest.mark.parametrize("tile", [(16, 16), (4, 4)])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 40000])
@pytest.mark.parametrize("crowd", [False, True])
def test_2d_work_items(tile, n, crowd):
    """Tile lists cut into work items of whole chunks: all particles in one
    tile (the others empty), or spread; lists of a chunk's length and one
    around it. Three steps keep the tile order that the items index."""
    params, m, rng, f = _state((64, 48), n, 11, tile=tile)
    p = random_particles(m, n, rng, gamma_max=5.0)
    if crowd:
        c1 = rng.integers(18, 20, n)
        c2 = rng.integers(18, 20, n)
        p["cell"][:] = (c1 + c2 * m.dims[0]).astype(np.uint32)
    pr = Pair(params, f, p)
    for step in range(3):
        pr.both_update_particles(step)
        pr.check_particles()
        pr.check_current(J_TOL, rho=True)


@pytest.mark.parametrize("n", [1, 257, 20000, 148 * 1024, 148 * 1024 * 2 + 3])
def test_1d_chunk_lengths(n):
    params, m, rng, f = _state((512,), n, 5)
    p = random_particles(m, n, rng, gamma_max=5.0)
    pr = Pair(params, f, p)
    pr.both_update_particles(0)
    pr.check_particles()
    pr.check_current(J_TOL, rho=True)


@pytest.mark.parametrize("N", [(64, 64), (64, 65), (4096,), (4097,), (5, 7)])
def test_update_fields_at_the_small_grid_limit(N):
    params, m, rng, f = _state(N, 1, 4)
    for c in range(3):
        f["J"][c][:] = (0.1 * rng.standard_normal(f["J"][c].shape)).astype(np.float32)
    pr = Pair(params, f, random_particles(m, 0, rng))
    g0, g1 = m.guard[0], m.guard[1]
    sl = ((slice(g1, m.dims[1] - g1) if m.dimension > 1 else slice(0, 1)),
          slice(g0, m.dims[0] - g0))
    for step in range(2):
        pr.both_update_fields(step)
        g = pr.data.fields_host()
        for key in ("E", "B"):
            for c in range(3):
                assert_bits(g[key][c], pr.f[key][c], f"{key}{c + 1} step {step}")
        for key in ("divE", "divB"):
            assert_bits(g[key][sl], pr.f[key][sl], key)


@pytest.mark.parametrize("N,periodic", [((33, 21), (True, True)), ((33, 21), (True, False)),
                                        ((33, 21), (False, True)), ((33, 21), (False, False)),
                                        ((300,), (True, True)), ((300,), (False, True))])
def test_smooth_current_bitexact(N, periodic):
    """J and Rho given as arrays: two smoothing passes with the guards of the
    periodic dims refreshed after each, in dim order, guard rows of the other
    dim included."""
    params, m, rng, f = _state(N, 1, 9, periodic=periodic, smoothing=2)
    pr = Pair(params, f, random_particles(m, 0, rng))
    per = pr.periodic
    bnd = [int(not per[0]), int(not per[0]), int(not per[1]), int(not per[1])]
    arrs = [rng.standard_normal(pr.f["J"][0].shape).astype(np.float32) for _ in range(5)]
    pr.data.set_fields({"J": arrs[:3], "Rho": arrs[3:]})
    pr.pusher.smooth_current(pr.data, 0)
    g = pr.data.fields_host()
    for k, a in enumerate(arrs):
        ref = a.copy()
        for _ in range(2):
            oracle.filter_current(m, ref, ref.copy(), bnd)
            oracle.send_guard_cells(m, ref, per)
        assert_bits((g["J"] + g["Rho"])[k], ref, f"array {k}")


@pytest.mark.parametrize("n,order", [(1, "random"), (3, "random"), (4095, "random"),
                                     (4097, "cells"), (70001, "random"), (70002, "cells"),
                                     (70003, "reverse")])
@pytest.mark.parametrize("half", [False, True])
def test_sort_by_cell_around_its_tiles(n, order, half):
    """sort_by_cell of random, cell-ordered and reversed stores with empty
    slots, in place and into the other half of the capacity (whose start is
    not 16-byte aligned for odd n): every member equals the stable sort."""
    params, m, rng, _ = _state((40, 24), n, 21)
    p = random_particles(m, n, rng)
    if order != "random":
        perm = np.argsort(p["cell"], kind="stable")
        for k in p:
            p[k][:] = p[k][perm if order == "cells" else perm[::-1]]
    p["cell"][rng.random(n) < 0.05] = oracle.MAX_CELL
    pr = Pair(params, {}, p, capacity=2 * n if half else n)
    if half:
        pr.env.set_compaction(2)
    pr.data.sort_particles()
    n_ref = oracle.sort_by_cell(m, pr.p, n)
    first, end = pr.data.slot_range()
    assert (first, end) == ((n, n + n_ref) if half else (0, n_ref))
    got = {k: v[first:end] for k, v in pr.data.particles_host().items()}
    for k, _ in oracle.PTC_FIELDS:
        assert_bits(got[k], pr.p[k][:n_ref], f"sorted {k}")


def test_update_waits_for_the_state_it_was_given():
    """The state's tensors are still being written on the caller's stream when
    the first update is called (a 0.1 s kernel in front of them): the update
    sees all of them."""
    import torch
    from aperture3_b200 import SimData, SimEnvironment, ic, ptc_updater
    params, fields, ptc = ic.box2d(seed=3, N=64, ppc=8, device=torch.device("cuda", 0))
    n = ptc["x1"].numel()
    got = []
    for cycles in (0, int(2e8)):
        env = SimEnvironment(params)
        data = SimData(env, capacity=2 * n)
        env.set_compaction(2)
        torch.cuda.synchronize()
        if cycles:
            torch.cuda._sleep(cycles)
        data.set_fields_device(fields)
        data.set_particles_device({k: v.clone() for k, v in ptc.items()})
        for step in range(2):
            ptc_updater(env).update_particles(data, params.delta_t, step)
        torch.cuda.synchronize()
        a, b = data.slot_range()
        got.append({k: v[a:b].clone() for k, v in data.particles.items()})
        env.close()
    assert int((got[1]["cell"] != -1).sum()) == n
    for k in got[0]:
        assert torch.equal(got[0][k], got[1][k]), k


@pytest.mark.parametrize("N,tile", [((63, 48), (16, 16)), ((37, 29), (8, 8)), ((97, 50), (32, 16))])
@pytest.mark.parametrize("field_load", ["tma", "plain"])
def test_2d_deposit_of_offsets_outside_the_cell(N, tile, field_load):
    """Particles that their caller placed up to half a cell outside their cell
    (and at -0.0, 1 and next to both) deposit the clamped weights of any
    offset, at every node and face of their range. Free streaming, so that the
    deposit alone is compared; the second step starts from moved offsets."""
    n = 5000
    params, m, rng, f = _state(N, n, 17, amp=0.0, tile=tile)
    p = random_particles(m, n, rng, gamma_max=50.0)
    one = np.float32(1)
    sides = np.array([-0.45, -0.2, -1e-3, -1e-8, -0.0, 0.0, 0.5, 0.9, 1.0,
                      np.nextafter(one, one * 2), 1.001, 1.3, 1.45], np.float32)
    for k in ("x1", "x2"):
        p[k][:] = sides[rng.integers(0, len(sides), n)]
    pr = Pair(params, f, p, row_align=4 if field_load == "tma" else 1)
    for step in range(2):
        pr.both_update_particles(step)
        pr.check_particles()
        pr.check_current(J_TOL, rho=True)


@pytest.mark.parametrize("kind", ["box", "logsph"])
def test_contexts_of_different_species_counts_take_turns(kind):
    """Contexts with three and with two charge densities share their kernel
    but not the shared memory of a launch: each runs again after the other."""
    import torch
    from aperture3_b200 import SimData, SimEnvironment, ic, ptc_updater
    from aperture3_b200.sim import ptc_updater_logsph
    dev = torch.device("cuda", 0)
    runs = []
    for species in (3, 2):
        if kind == "logsph":
            params, fields, ptc = ic.logsph(seed=3, N=64, ppc=8, device=dev)
        else:
            params, fields, ptc = ic.box2d(seed=3, N=64, ppc=8, device=dev)
        params.num_species, params.data_interval, params.tile_size = species, 1, (16, 16, 0)
        env = SimEnvironment(params)
        data = SimData(env, capacity=ptc["x1"].numel())
        data.set_fields_device(fields)
        data.set_particles_device(ptc)
        runs.append((env, data))
    cls = ptc_updater_logsph if kind == "logsph" else ptc_updater
    for step in range(3):
        for env, data in runs:
            cls(env).update_particles(data, env.params.delta_t, step)
    (_, a), (_, b) = runs
    for k in a.particles:
        assert torch.equal(a.particles[k], b.particles[k]), k
    for s in range(2):
        assert torch.equal(a.Rho[s], b.Rho[s])
    assert not a.Rho[2].any()
    for env, _ in runs:
        env.close()


def test_smoothing_of_rows_of_different_lengths_from_two_threads():
    """The 1D gap lab's rows in shared memory: two threads with rows of
    different lengths smooth at the same time, and get what they get alone."""
    import threading
    import torch
    from aperture3_b200 import SimData, SimEnvironment, SimParams
    from aperture3_b200.sim import ptc_updater_1dgap

    def make(N):
        p = SimParams(N=(N, 1, 1), guard=(2, 0, 0), lower=(0.0, 0.0, 0.0), size=(1.0, 1.0, 1.0),
                      delta_t=0.5 / N, q_e=1.0, num_species=2, current_smoothing=2,
                      periodic_boundary=(False, False, False), max_ptc_number=1, B0=0.7,
                      coord_system="1dgap")
        env = SimEnvironment(p)
        data = SimData(env, capacity=1)
        g = torch.Generator().manual_seed(N)
        data.E[0].copy_(torch.randn(data.E[0].shape, generator=g))
        torch.cuda.synchronize()
        return env, data

    def smooth(env, data, times):
        for _ in range(times):
            ptc_updater_1dgap(env).update_particles(data, env.params.delta_t, 0)

    sizes = (7000, 25000)
    want = []
    for N in sizes:
        env, data = make(N)
        smooth(env, data, 1)
        want.append(data.E[2].clone())
        env.close()
    runs, failed = [make(N) for N in sizes], []

    def body(env, data):
        try:
            smooth(env, data, 200)
        except Exception as e:  # noqa: BLE001 (reported below)
            failed.append(e)

    threads = [threading.Thread(target=body, args=r) for r in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for (env, data), w in zip(runs, want):
        assert torch.equal(data.E[2], w)
        env.close()


@pytest.mark.parametrize("from_host", [False, True])
def test_setters_wait_for_queued_updates(from_host):
    """Particles and fields are replaced while pipelined updates of the old
    ones are still queued: the new state is as in a context that had none."""
    import torch
    from aperture3_b200 import SimData, SimEnvironment, ic, ptc_updater
    dev = torch.device("cuda", 0)
    params, fields, ptc = ic.box2d(seed=3, N=256, ppc=32, device=dev)
    _, fields2, ptc2 = ic.box2d(seed=4, N=256, ppc=32, device=dev)
    n = ptc["x1"].numel()
    got = []
    for queued in (0, 30):
        env = SimEnvironment(params)
        data = SimData(env, capacity=n)
        data.set_fields_device(fields)
        data.set_particles_device(ptc)
        env.set_sync(False)
        pusher = ptc_updater(env)
        for step in range(queued):
            pusher.update_particles(data, params.delta_t, step)
        if from_host:
            host = ic.to_numpy_ptc(ptc2)
            data.set_fields({k: [f.cpu().numpy() for f in v] for k, v in fields2.items()})
            data.set_particles(host)
        else:
            data.set_fields_device(fields2)
            data.set_particles_device(ptc2)
        pusher.update_particles(data, params.delta_t, 0)
        env.sync()
        got.append([t.clone() for t in (*data.particles.values(), *data.J, *data.E, *data.B)])
        env.close()
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_a_new_tile_shape_is_ordered_with_the_updates():
    """The buffers of a new tile shape are cleared in the updates' order, not
    in that of the default stream, whose earlier work (a kernel of some 10 ms
    here) ends while the updates run."""
    import torch
    from aperture3_b200 import SimData, SimEnvironment, ic, ptc_updater
    dev = torch.device("cuda", 0)
    params, fields, ptc = ic.box2d(seed=3, N=128, ppc=16, device=dev)
    got = []
    for cycles in (0, int(2e7)):
        env = SimEnvironment(params)
        data = SimData(env, capacity=ptc["x1"].numel())
        data.set_fields_device(fields)
        data.set_particles_device(ptc)
        env.set_sync(False)
        torch.cuda.synchronize()
        if cycles:
            torch.cuda._sleep(cycles)
        env.set_tile_shape(8, 8)
        for step in range(400):
            ptc_updater(env).update_particles(data, params.delta_t, step)
        env.sync()
        torch.cuda.synchronize()
        got.append([t.clone() for t in (*data.particles.values(), *data.J)])
        env.close()
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("tile,chunk,species", [((16, 16), 2048, 1), ((16, 16), 2048, 2),
                                                ((16, 8), 2048, 8), ((8, 8), 2048, 2),
                                                ((4, 4), 2048, 3), ((32, 16), 0, 2),
                                                ((32, 16), 0, 8), ((32, 16), 1024, 6),
                                                ((32, 16), 2048, 2), ((16, 16), 1024, 4)])
def test_2d_chunks_and_species_on_both_sides_of_the_shared_memory_rule(tile, chunk, species):
    """Tiles, chunks and species counts whose CTA leaves room for a second one
    on the SM, and some that take a shorter chunk instead; tiles of one to
    several work items."""
    n = 60000
    params, m, rng, f = _state((97, 50), n, 23, tile=tile)
    params.chunk, params.num_species = chunk, species
    p = random_particles(m, n, rng, gamma_max=5.0, species=range(species))
    pr = Pair(params, f, p)
    for step in range(2):
        pr.both_update_particles(step)
        pr.check_particles()
        pr.check_current(J_TOL, rho=True)


@pytest.mark.parametrize("N", [(63, 48), (512,)])
def test_fields_at_offsets_outside_the_cell(N):
    """Particles placed up to half a cell outside their cell are pushed by the
    fields there, bit for bit: above 1 the third node of a component counts."""
    n = 5000
    params, m, rng, f = _state(N, n, 19, amp=0.05)
    p = random_particles(m, n, rng, gamma_max=2.0)
    one = np.float32(1)
    sides = np.array([-0.45, -0.2, -1e-3, -1e-8, -0.0, 0.0, 0.5, 0.9, 1.0,
                      np.nextafter(one, one * 2), 1.001, 1.3, 1.45], np.float32)
    for k in ("x1", "x2")[:m.dimension]:
        p[k][:] = sides[rng.integers(0, len(sides), n)]
    pr = Pair(params, f, p)
    for step in range(2):
        pr.both_update_particles(step)
        pr.check_particles()
        pr.check_current(J_TOL, rho=True)


def test_logsph_push_at_offsets_outside_the_cell():
    """Log-spherical particles placed up to 0.4 cells outside their cell (away
    from the axis): pushed as near the FP64 oracle as the FP32 oracle is, with
    the bounds of the ordinary step."""
    from oracle import logsph as ls
    from test_gpu_logsph import LsCase, _check_against_f64
    case = LsCase((128, 64), 40000, 3)
    rng = np.random.default_rng(29)
    row = case.p["cell"].astype(np.int64) // case.m.dims[0] - case.m.guard[1]
    far = (row >= 3) & (row < 64 - 3)
    sides = np.array([-0.4, -0.2, -1e-3, 0.0, 0.5, 1.0, 1.001, 1.2, 1.4], np.float32)
    for k in ("x1", "x2"):
        case.p[k][far] = sides[rng.integers(0, len(sides), case.n)][far]
    case.p64 = ls.to_f64(case.p)
    case.data.set_particles(case.p)
    case.step_particles(0)
    _check_against_f64(case, "offsets outside the cell")
    case.close()
