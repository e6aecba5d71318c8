"""Near lists against the full cell walk (PBD_FLAG_FULL_WALK).

A walking pass (lambda, omega) records the entries within the cut for the pass after it at the
same positions (delta, viscosity); the entries left out add exact zeros there, so a step with
near lists must be bit-identical to a step that walks the cells in every pass, over many frames,
for every pass mix (density solve, contacts, vorticity, viscosity, solids, batches, the
cell-end quirk's long ranges, fast motion)."""
import numpy as np
import pytest

from helpers import device_events

pytestmark = pytest.mark.gpu


def _run(pbd, params, pos, vel, frames, inv_mass=None, full_walk=False):
    p = params.copy()
    if full_walk:
        p.flags |= pbd.FLAG_FULL_WALK
    sim = pbd.Sim(p, len(pos))
    if inv_mass is None:
        sim.add_particles(pos, vel)
    else:
        sim.add_particles_mass(pos, vel, inv_mass)
    sim.step(frames)
    sim.sync()
    st = sim.state()
    sim.close()
    return st


def _same(a, b):
    for k in ("x", "v", "p", "ids"):
        assert np.array_equal(a[k], b[k]), k


CASES = [
    # shape, box, vorticity, viscosity, quirk, velocity sigma
    ((20, 20, 20), 32, 0.0, 0.0, True, 0.0),
    ((20, 20, 20), 32, 0.0005, 0.01, True, 0.0),
    ((16, 24, 16), 32, 0.0, 0.01, False, 0.0),
    ((13, 7, 11), 24, 0.0, 0.0, True, 3.0),
]


@pytest.mark.parametrize("shape,box,vort,visc,quirk,sigma", CASES)
def test_lists_bit_identical_to_full_walk(need_gpu, pbd, scenes, shape, box, vort, visc, quirk, sigma):
    params = scenes.workload_params(pbd, box, 1000.0, vorticity=vort, viscosity=visc)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    if not quirk:
        params.flags &= ~pbd.FLAG_CELL_END_QUIRK
    pos, vel = scenes.lattice(*shape, seed=3)
    if sigma:
        vel[:, :3] = np.random.default_rng(3).normal(0, sigma, size=(len(vel), 3)).astype(np.float32)
    a = _run(pbd, params, pos, vel, 40)
    b = _run(pbd, params, pos, vel, 40, full_walk=True)
    _same(a, b)


def test_lists_fast_motion(need_gpu, pbd, scenes):
    # fast random motion: particles move up to a few cells per frame
    params = scenes.workload_params(pbd, 24, 1000.0)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(12, 12, 12, spacing=0.8, seed=4)
    vel[:, :3] = np.random.default_rng(4).normal(0, 40, size=(len(vel), 3)).astype(np.float32)
    a = _run(pbd, params, pos, vel, 12)
    b = _run(pbd, params, pos, vel, 12, full_walk=True)
    _same(a, b)


def test_lists_with_solids(need_gpu, pbd, scenes):
    pos, vel, w = scenes.solids_scene(fluid_shape=(16, 16, 16), n_boxes=2, box_shape=(6, 6, 8), box=48, seed=5)
    params = scenes.workload_params(pbd, 48, 1000.0)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    a = _run(pbd, params, pos, vel, 30, inv_mass=w)
    b = _run(pbd, params, pos, vel, 30, inv_mass=w, full_walk=True)
    _same(a, b)


def test_lists_in_batches(need_gpu, pbd, scenes):
    sl = scenes.batched_scenes(nscenes=4, n_range=(500, 3000), box_range=(20, 32), seed=9)
    shared = scenes.workload_params(pbd, 32, 1000.0)
    shared.lambda_epsilon = 0.1
    out = []
    for fw in (False, True):
        p = shared.copy()
        if fw:
            p.flags |= pbd.FLAG_FULL_WALK
        descs = [pbd.scene_desc(sc["n"], sc["rest_density"], sc["gravity"], sc["box"]) for sc in sl]
        b = pbd.Batch(p, descs)
        for k, sc in enumerate(sl):
            b.add_particles(k, sc["pos"], sc["vel"])
        b.step(25)
        b.sync()
        out.append([b.state(k) for k in range(len(sl))])
        b.close()
    for s1, s2 in zip(*out):
        assert np.array_equal(s1["x"], s2["x"]) and np.array_equal(s1["v"], s2["v"])


@pytest.mark.parametrize("vort,visc", [(0.0, 0.0), (0.0005, 0.01), (0.0, 0.01)])
def test_lists_dense_blob_without_lists(need_gpu, pbd, scenes, vort, visc):
    """a blob at spacing 0.35 inside a lattice at spacing 1: the blob's particles have more than
    128 entries (no full list) and up to ~100 within the cut (no near list), so every pass hands
    them to its cooperative blocks through the noted sets; the rest walk stored lists"""
    params = scenes.workload_params(pbd, 32, 1000.0, vorticity=vort, viscosity=visc)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    params.flags &= ~pbd.FLAG_CELL_END_QUIRK
    pos, vel = scenes.lattice(16, 12, 16, spacing=1.0, seed=6)
    lo, sp = np.array([8.0, 6.0, 8.0]), 0.35
    blob, bv = scenes.lattice(9, 9, 9, origin=tuple(lo), spacing=sp, jitter=0.02, seed=7)
    inside = np.all((pos[:, :3] > lo - 0.5) & (pos[:, :3] < lo + 8 * sp + 0.5), axis=1)
    pos = np.concatenate([pos[~inside], blob]); vel = np.concatenate([vel[~inside], bv])
    a = _run(pbd, params, pos, vel, 8)
    b = _run(pbd, params, pos, vel, 8, full_walk=True)
    _same(a, b)


@pytest.mark.parametrize("cap", [20, 40])
def test_lists_with_a_small_cap(need_gpu, pbd, scenes, cap):
    """maxNeighboursPerParticle below the ~32 candidates of the 27 cells: every stored list is
    cut at the cap in the cells' order, as the walk cuts it"""
    params = scenes.workload_params(pbd, 32, 1000.0, vorticity=0.0005, viscosity=0.01, max_neighbours=cap)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(20, 16, 20, spacing=0.9, seed=8)
    a = _run(pbd, params, pos, vel, 12)
    b = _run(pbd, params, pos, vel, 12, full_walk=True)
    _same(a, b)


def test_block_size_leaves_results_unchanged(need_gpu, pbd, scenes, tmp_path):
    """pbd_autotune picks the neighbour passes' block size; every size gives the same bits (the
    particles without a list are walked by whichever blocks, each on its own)"""
    import json
    params = scenes.workload_params(pbd, 32, 1000.0, vorticity=0.0005, viscosity=0.01)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(20, 16, 20, spacing=0.9, seed=12)
    probe = tmp_path / "probe.jsonl"
    sim = pbd.Sim(params, len(pos))
    sim.add_particles(pos, vel)
    assert sim.autotune(str(probe)) in (64, 128, 256)
    sim.close()
    sig = json.loads(probe.read_text().splitlines()[0])["signature"]
    states = []
    for block in (64, 128, 256):
        cache = tmp_path / f"b{block}.jsonl"
        cache.write_text(json.dumps({"signature": sig, "block": block}) + "\n")
        sim = pbd.Sim(params, len(pos))
        sim.add_particles(pos, vel)
        assert sim.autotune(str(cache)) == block          # served from the cache: no frames run
        sim.step(10)
        sim.sync()
        states.append(sim.state())
        sim.close()
    for st in states[1:]:
        _same(states[0], st)


@pytest.mark.parametrize("vort,visc", [(0.0, 0.0), (0.0005, 0.01), (0.0005, 0.0), (0.0, 0.01)])
def test_step_readback_matches_step_and_get_state(need_gpu, pbd, scenes, vort, visc):
    """pbd_step_readback (positions, and velocities that viscosity leaves alone, copied beside the
    last passes; velocities that viscosity changes stored into host memory by that pass) returns
    the state pbd_step + pbd_get_state return, and the simulation continues from it identically"""
    params = scenes.workload_params(pbd, 32, 1000.0, vorticity=vort, viscosity=visc)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(20, 16, 20, spacing=0.9, seed=13)
    a = pbd.Sim(params, len(pos)); a.add_particles(pos, vel)
    b = pbd.Sim(params, len(pos)); b.add_particles(pos, vel)
    for n in (1, 3, 1):
        xa, va = a.step_readback(n)
        b.step(n)
        sb = b.state()
        assert np.array_equal(xa, sb["x"]) and np.array_equal(va, sb["v"])
    _same(a.state(), b.state())
    a.close(); b.close()


def test_readback_arrays_fed_back_in(need_gpu, pbd, scenes):
    """A host loop that feeds pbd_step_readback's own arrays back through pbd_clear +
    pbd_add_particles (the copy is queued, not waited for) gives, frame by frame, the bits of a
    loop that restarts from host copies of the same state with the synchronous path"""
    params = scenes.workload_params(pbd, 32, 1000.0, vorticity=0.0005, viscosity=0.01)
    params.lambda_epsilon = 0.1
    pos, vel = scenes.lattice(20, 16, 20, spacing=0.9, seed=13)
    n = len(pos)
    a = pbd.Sim(params, n); a.add_particles(pos, vel)
    b = pbd.Sim(params, n); b.add_particles(pos, vel)
    L = pbd.lib()
    rx, rv = pbd.C.POINTER(pbd.C.c_float)(), pbd.C.POINTER(pbd.C.c_float)()
    pbd.check(L.pbd_step_readback(a.h, 1, None, pbd.C.byref(rx), pbd.C.byref(rv)))
    b.step(1)
    for _ in range(4):
        pbd.check(L.pbd_clear(a.h))
        pbd.check(L.pbd_add_particles(a.h, n, rx, rv, None))
        pbd.check(L.pbd_step_readback(a.h, 1, None, pbd.C.byref(rx), pbd.C.byref(rv)))
        sb = b.state()
        b.clear()
        b.add_particles(sb["x"], sb["v"])
        b.step(1)
        sb = b.state()
        xa = np.ctypeslib.as_array(rx, shape=(n, 4))
        va = np.ctypeslib.as_array(rv, shape=(n, 4))
        assert np.array_equal(xa, sb["x"]) and np.array_equal(va, sb["v"])
    a.close(); b.close()


@pytest.mark.parametrize("shells,cap", [(1, 512), (2, 20), (2, 100), (2, 512), (2, 513), (2, 1500), (3, 300), (3, 512)])
def test_long_rows_bit_identical_to_full_walk(need_gpu, pbd, scenes, shells, cap):
    """16^3 particles around cell 4095 = (15, 15, 15), whose range the cell-end quirk stretches: the
    particles within the shells of it have long lists, stored by a warp (up to 512 entries; longer
    ones walk the cells), cut at the cap inside the 27 cells, inside the shells and beyond"""
    params = scenes.workload_params(pbd, 32, 1995.0, vorticity=0.0005, viscosity=0.00015, max_neighbours=cap)
    params.lambda_epsilon = 0.0001
    params.kernel_width_poly, params.kernel_width_spiky, params.kernel_width_neighbours = 4.1, 3.5, shells
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(16, 16, 16, seed=21)
    a = _run(pbd, params, pos, vel, 3)
    b = _run(pbd, params, pos, vel, 3, full_walk=True)
    _same(a, b)


def test_more_particles_without_a_list_than_rows(need_gpu, pbd, scenes):
    """a blob of 12,167 particles at spacing 0.35, most of them with more than 128 entries: the rows
    (8,192) run out and the rest walk the cells"""
    params = scenes.workload_params(pbd, 32, 1000.0, vorticity=0.0005, viscosity=0.01)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(23, 23, 23, origin=(6.0, 6.0, 6.0), spacing=0.35, jitter=0.02, seed=22)
    a = _run(pbd, params, pos, vel, 2)
    b = _run(pbd, params, pos, vel, 2, full_walk=True)
    _same(a, b)


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("n_scorr,mass", [(4, False), (4, True), (3, False), (0, True)])
def test_delta_pass_variants_bit_identical_to_full_walk(need_gpu, pbd, scenes, dense, n_scorr, mass):
    """the delta pass fixes nSCorr = 4 and the absence of inverse masses at compile time where they
    hold; every variant gives the bits of the pass that looks at them for every entry"""
    params = scenes.workload_params(pbd, 24, 1995.0 if dense else 1000.0)
    params.lambda_epsilon = 0.0001 if dense else 0.1
    params.n_scorr = n_scorr
    if dense:
        params.kernel_width_poly, params.kernel_width_spiky, params.kernel_width_neighbours = 4.1, 3.5, 2
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(13, 11, 15, seed=23, spacing=0.95)
    w = np.where(np.arange(len(pos)) % 7 == 0, 0.0, 1.0).astype(np.float32) if mass else None
    a = _run(pbd, params, pos, vel, 3, inv_mass=w)
    b = _run(pbd, params, pos, vel, 3, inv_mass=w, full_walk=True)
    _same(a, b)


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 3), (3, 5, 7), (16, 32, 16), (19, 19, 23), (24, 25, 27), (16, 32, 32), (25, 27, 29), (24, 32, 32), (27, 29, 32)])
def test_lanes_per_particle_bit_identical_to_full_walk(need_gpu, pbd, scenes, shape, dense):
    """the list passes take 16, 8, 4 or 1 lanes per particle by the number of particles (16 up to 8,192,
    8 up to 16,384, 4 up to 24,576): both sides of every change, partial warps, one particle"""
    params = scenes.workload_params(pbd, 40, 1995.0 if dense else 1000.0, vorticity=0.0005, viscosity=0.00015 if dense else 0.01)
    params.lambda_epsilon = 0.0001 if dense else 0.1
    if dense:
        params.kernel_width_poly, params.kernel_width_spiky, params.kernel_width_neighbours = 4.1, 3.5, 2
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(*shape, seed=24, spacing=0.95)
    vel[:, :3] = np.random.default_rng(24).normal(0, 0.5, size=(len(vel), 3)).astype(np.float32)
    a = _run(pbd, params, pos, vel, 2)
    b = _run(pbd, params, pos, vel, 2, full_walk=True)
    _same(a, b)


@pytest.mark.parametrize("where", ["inside", "walls", "touching"])
def test_coarse_filter_keeps_every_near_pair(need_gpu, pbd, scenes, where):
    """the near lists are filtered by positions in steps of 1/512 cell: pairs at the cut to the last bits,
    positions at the enclosure's limits (1.5 and 126.5, where the coarse position is near its end) and
    particles pressed through one another, against the walk of every cell"""
    params = scenes.workload_params(pbd, 128, 1000.0, vorticity=0.0005, viscosity=0.01)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    rng = np.random.default_rng(25)
    origin = {"inside": (60.0, 60.0, 60.0), "walls": (98.0, 1.6, 98.0), "touching": (30.0, 30.0, 30.0)}[where]
    pos, vel = scenes.lattice(30, 30, 30, origin=origin, spacing={"inside": 1.00005, "walls": 0.98, "touching": 0.7}[where], jitter=1e-6 if where == "inside" else 0.1, seed=25)
    vel[:, :3] = rng.normal(0, 0.0 if where == "inside" else 20.0, size=(len(vel), 3)).astype(np.float32)
    a = _run(pbd, params, pos, vel, 4)
    b = _run(pbd, params, pos, vel, 4, full_walk=True)
    _same(a, b)


@pytest.mark.parametrize("radius,shells", [(0.4, 1), (0.4, 2), (0.63, 2), (0.5, 3), (0.3, 3)])
def test_list_columns_bit_identical_to_full_walk(need_gpu, pbd, scenes, radius, shells):
    """the first lambda pass stores a column's cells as runs of two where their z follow each other; a
    diameter other than 1 repeats or skips cells, positions a rounding below a whole number make
    p + 1 the cell after the next"""
    params = scenes.workload_params(pbd, 64, 1995.0, vorticity=0.0005, viscosity=0.00015)
    params.particle_radius = radius
    params.lambda_epsilon = 0.1
    params.kernel_width_poly, params.kernel_width_spiky, params.kernel_width_neighbours = 2.1, 2.0, shells
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(31, 29, 33, origin=(1.6, 1.6, 1.6), spacing=0.9, seed=26)
    pos[::3, :3] = np.nextafter(np.ceil(pos[::3, :3]), np.float32(0), dtype=np.float32)
    a = _run(pbd, params, pos, vel, 2)
    b = _run(pbd, params, pos, vel, 2, full_walk=True)
    _same(a, b)


@pytest.mark.parametrize("collision_type", [0, 1])
def test_two_entries_at_a_time_bit_identical_to_full_walk(need_gpu, pbd, scenes, collision_type):
    """lambda and delta over full lists take two entries per call and test each kernel's range where its
    term is added: pairs on both sides of every limit, pairs at one place, rows of every remainder"""
    params = scenes.workload_params(pbd, 64, 1995.0, vorticity=0.0005, viscosity=0.00015)
    params.lambda_epsilon = 0.1
    params.collision_type = collision_type
    params.kernel_width_poly, params.kernel_width_spiky, params.kernel_width_neighbours = 2.1, 2.0, 2
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(29, 31, 30, origin=(8.0, 8.0, 8.0), spacing=0.93, seed=27)
    gaps = np.array([0.0, 1e-5, 2e-5, 9.99e-5, 1e-4, 1.01e-4, 9.99e-4, 1e-3, 1.01e-3, 0.5, 1.0, 1.9998, 1.9999, 2.0, 2.0989, 2.099, 2.1, 2.1002], np.float32)
    a = np.arange(0, len(pos) - 1, 3)
    pos[a + 1, :3] = pos[a, :3]
    pos[a + 1, a % 3] += gaps[a // 3 % len(gaps)]
    _same(_run(pbd, params, pos, vel, 2), _run(pbd, params, pos, vel, 2, full_walk=True))


@pytest.mark.parametrize("collision_type", [0, 1])
def test_infinite_positions_in_the_solver(need_gpu, pbd, scenes, collision_type):
    """isolated pairs that s_corr (a reference density close to zero) throws to infinity in the first
    iteration: in the second every entry of a pair's list is out of range, so lambda is 1 / eps for both,
    whichever way the entries are read (lists of one entry, padded to a group of four with the particle
    itself, whose difference is inf - inf)"""
    params = scenes.workload_params(pbd, 128, 1000.0, iterations=2)
    params.lambda_epsilon = 0.1
    params.gravity = 0.0
    params.collision_type = collision_type
    params.kernel_width_poly, params.kernel_width_spiky, params.q_scorr = 1.6, 1.5, 1.598 / 1.5
    params.flags &= ~pbd.FLAG_CELL_END_QUIRK
    g = np.stack(np.meshgrid(*[np.arange(24)] * 3, indexing="ij"), -1).reshape(-1, 3) * 5.0 + 3.0
    pos = np.zeros((2 * len(g), 4), np.float32)
    pos[0::2, :3] = g
    pos[1::2, :3] = g + np.array([0.6, 0.7, 0.75])
    out = []
    for flags in (0, pbd.FLAG_FULL_WALK):
        p = params.copy()
        p.flags |= flags
        with pbd.Sim(p, len(pos)) as sim:
            sim.add_particles(pos, np.zeros_like(pos))
            sim.step(1)
            sim.sync()
            out.append((sim.debug()["lambda"], sim.state()["x"][:, :3]))
    lists, walk = out
    assert np.isinf(walk[1]).all()
    assert np.array_equal(walk[0], np.full(len(pos), np.float32(1) / np.float32(0.1), np.float32))
    assert np.array_equal(lists[0], walk[0]) and np.array_equal(lists[1], walk[1])


def test_near_lists_leave_out_positions_that_are_not_numbers(need_gpu, pbd, scenes):
    """a pair in line with the x axis that s_corr throws to (+-inf, NaN, NaN) in the first iteration, beside a
    particle in the enclosure's far corner, where the coarse position of a NaN lies within the kernels'
    reach (3.2 cells): its lambda in the second iteration, with nothing finite in range, is 1 / eps"""
    params = scenes.workload_params(pbd, 128, 1000.0, iterations=2)
    params.lambda_epsilon = 0.1
    params.gravity = 0.0
    params.kernel_width_poly, params.q_scorr, params.kernel_width_neighbours = 3.2, 3.198, 3
    params.flags &= ~pbd.FLAG_CELL_END_QUIRK
    g = np.stack(np.meshgrid(*[np.arange(30)] * 3, indexing="ij"), -1).reshape(-1, 3) * 4.0 + 3.0   # alone, for their number
    pos = np.zeros((len(g) + 3, 4), np.float32)
    pos[3:, :3] = g
    pos[:3, :3] = [(126.4, 126.4, 126.4), (124.0, 126.0, 126.0), (124.8, 126.0, 126.0)]
    with pbd.Sim(params, len(pos)) as sim:
        sim.add_particles(pos, np.zeros_like(pos))
        sim.step(1)
        sim.sync()
        lam, x = sim.debug()["lambda"], sim.state()["x"][:, :3]
    assert np.isnan(x).any(axis=1).sum() == 2 and np.isinf(x[:, 0]).sum() == 2
    corner = np.where((x > 126).all(axis=1))[0]
    assert len(corner) == 1 and lam[corner[0]] == np.float32(1) / np.float32(0.1)


def _one_lane(pbd, params, pos, vel, frames, kernels, inv_mass=None):
    """lists against the full walk with more than 24,576 particles (a thread per particle), and that the
    frames ran `kernels` (parts of their names)"""
    assert len(pos) > 24576
    got = []
    names = device_events(lambda: got.append(_run(pbd, params, pos, vel, frames, inv_mass=inv_mass)))
    for k in kernels if names else ():
        assert any(k in s for s in names), (k, sorted(set(names)))
    _same(got[0], _run(pbd, params, pos, vel, frames, inv_mass=inv_mass, full_walk=True))


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("n_scorr,mass,known", [(4, False, 1), (4, True, 2), (3, False, 0), (0, True, 0)])
def test_delta_variants_with_one_lane(need_gpu, pbd, scenes, dense, n_scorr, mass, known):
    """delta_list_kernel knows nSCorr = 4 and the absence (1) or presence (2) of inverse masses at compile time,
    or nothing (0): over near lists and over full lists, each against the walk of every cell"""
    params = scenes.workload_params(pbd, 40, 1995.0 if dense else 1000.0)
    params.lambda_epsilon = 0.0001 if dense else 0.1
    params.n_scorr = n_scorr
    if dense:
        params.kernel_width_poly, params.kernel_width_spiky, params.kernel_width_neighbours = 4.1, 3.5, 2
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(31, 29, 30, seed=23, spacing=0.95)
    w = np.where(np.arange(len(pos)) % 7 == 0, 0.0, 1.0).astype(np.float32) if mass else None
    full = "true" if dense else "false"
    _one_lane(pbd, params, pos, vel, 3, [f"delta_list_kernel<{m}u, {full}, {known}u>" for m in (7, 39)], w)


@pytest.mark.parametrize("cap", [20, 40])
def test_small_cap_with_one_lane(need_gpu, pbd, scenes, cap):
    params = scenes.workload_params(pbd, 40, 1000.0, vorticity=0.0005, viscosity=0.01, max_neighbours=cap)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(30, 29, 31, spacing=0.9, seed=8)
    _one_lane(pbd, params, pos, vel, 4, ["lambda_kernel<true>", "lambda_list_kernel<true, true>", "omega_list_kernel<true, true>"])


def test_solids_with_one_lane(need_gpu, pbd, scenes):
    pos, vel, w = scenes.solids_scene(fluid_shape=(30, 30, 30), n_boxes=2, box_shape=(6, 6, 8), box=64, seed=5)
    params = scenes.workload_params(pbd, 64, 1000.0)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    _one_lane(pbd, params, pos, vel, 10, ["delta_list_kernel<7u, false, 2u>"], w)


@pytest.mark.parametrize("vort,visc", [(0.0, 0.0), (0.0005, 0.01), (0.0, 0.01)])
def test_dense_blob_with_one_lane(need_gpu, pbd, scenes, vort, visc):
    """a blob at spacing 0.35 inside a lattice at spacing 1, as above: particles with neither list among
    those with both"""
    params = scenes.workload_params(pbd, 48, 1000.0, vorticity=vort, viscosity=visc)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    params.flags &= ~pbd.FLAG_CELL_END_QUIRK
    pos, vel = scenes.lattice(31, 30, 29, spacing=1.0, seed=6)
    lo, sp = np.array([8.0, 6.0, 8.0]), 0.35
    blob, bv = scenes.lattice(9, 9, 9, origin=tuple(lo), spacing=sp, jitter=0.02, seed=7)
    inside = np.all((pos[:, :3] > lo - 0.5) & (pos[:, :3] < lo + 8 * sp + 0.5), axis=1)
    pos = np.concatenate([pos[~inside], blob]); vel = np.concatenate([vel[~inside], bv])
    _one_lane(pbd, params, pos, vel, 4, ["lambda_list_kernel<true, true>"])


@pytest.mark.parametrize("shells,cap", [(1, 512), (2, 20), (2, 100), (2, 512), (2, 513), (2, 1500), (3, 300), (3, 512)])
def test_long_rows_with_one_lane(need_gpu, pbd, scenes, shells, cap):
    """32^3 particles around cell 32767 = (31, 31, 31), whose range the cell-end quirk stretches"""
    params = scenes.workload_params(pbd, 48, 1995.0, vorticity=0.0005, viscosity=0.00015, max_neighbours=cap)
    params.lambda_epsilon = 0.0001
    params.kernel_width_poly, params.kernel_width_spiky, params.kernel_width_neighbours = 4.1, 3.5, shells
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(32, 32, 32, seed=21)
    _one_lane(pbd, params, pos, vel, 2, ["lambda_kernel<true>", "lambda_long_kernel", "lambda_list_kernel<true, false>"])


def test_more_rows_than_slots_with_one_lane(need_gpu, pbd, scenes):
    """a blob of 29,791 particles at spacing 0.35: more particles without a list than rows (8,192); the first
    lambda pass walks the cells for the rest itself"""
    params = scenes.workload_params(pbd, 32, 1000.0, vorticity=0.0005, viscosity=0.01)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(31, 31, 31, origin=(6.0, 6.0, 6.0), spacing=0.35, jitter=0.02, seed=22)
    _one_lane(pbd, params, pos, vel, 2, ["lambda_kernel<true>", "lambda_long_kernel"])


@pytest.mark.parametrize("collision_type,mass", [(0, False), (0, True), (1, False)])
def test_two_entries_at_a_time_over_full_lists(need_gpu, pbd, scenes, collision_type, mass):
    """lambda and delta over full lists (kernels of 2.6 cells in a list of 5: no near lists) take two entries
    per call and test each kernel's range where its term is added: pairs on both sides of every limit,
    pairs at one place, rows of every remainder"""
    params = scenes.workload_params(pbd, 64, 1995.0, vorticity=0.0005, viscosity=0.00015)
    params.lambda_epsilon = 0.1
    params.collision_type = collision_type
    params.kernel_width_poly, params.kernel_width_spiky, params.kernel_width_neighbours = 2.6, 2.5, 2
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(29, 31, 30, origin=(8.0, 8.0, 8.0), spacing=0.93, seed=27)
    gaps = np.array([0.0, 1e-5, 2e-5, 9.99e-5, 1e-4, 1.01e-4, 9.99e-4, 1e-3, 1.01e-3, 0.5, 1.0, 2.4998, 2.4999, 2.5, 2.5989, 2.599, 2.6, 2.6002], np.float32)
    a = np.arange(0, len(pos) - 1, 3)
    pos[a + 1, :3] = pos[a, :3]
    pos[a + 1, a % 3] += gaps[a // 3 % len(gaps)]
    w = np.where(np.arange(len(pos)) % 7 == 0, 0.0, 1.0).astype(np.float32) if mass else None
    known = 0 if collision_type else (2 if mass else 1)
    unit = "false" if collision_type else "true"
    delta = "delta_list_kernel<0u, true, 0u>" if collision_type else f"delta_list_kernel<7u, true, {known}u>"
    _one_lane(pbd, params, pos, vel, 2, [f"lambda_list_kernel<{unit}, false>", delta], w)


def test_loaded_delta_with_a_w(need_gpu, pbd, scenes):
    """collisionType 1 writes p.w = 0 for some particles, so the corrections it stores have a w; frames that
    then apply them without computing new ones (collisionType 0) move p.w off 1, and the passes after that
    see it in the spiky gradient: lists against the full walk"""
    params = scenes.workload_params(pbd, 64, 1000.0, vorticity=0.0005, viscosity=0.01, iterations=3)
    params.lambda_epsilon = 0.1
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(30, 30, 30, spacing=0.8, seed=31)
    vel[:, :3] = np.random.default_rng(31).normal(0, 1.0, size=(len(vel), 3)).astype(np.float32)
    out = []
    for flags in (0, pbd.FLAG_FULL_WALK):
        p = params.copy()
        p.flags |= flags
        p.collision_type = 1
        with pbd.Sim(p, len(pos)) as sim:
            sim.add_particles(pos, vel)
            sim.step(2)
            p.collision_type = 0
            p.active &= ~pbd.ACTIVE["computeDeltaPositions"]
            sim.set_params(p)
            sim.step(2)
            sim.sync()
            out.append((sim.state(), sim.debug()))
    assert np.ptp(out[1][0]["p"][:, 3]) > 0
    _same(out[0][0], out[1][0])
    for k in ("lambda", "omega"):
        assert np.array_equal(out[0][1][k], out[1][1][k]), k


@pytest.mark.parametrize("shape", [(1, 1, 3), (6, 7, 8), (22, 21, 23), (27, 28, 28)])
@pytest.mark.parametrize("stab", [1, 2])
def test_far_pairs_that_are_not_numbers(need_gpu, pbd, scenes, shape, stab):
    """a negative nSCorr makes s_corr of a pair beyond the kernels infinite and its correction NaN: p* becomes
    NaN, but the contacts alone move x (updatePositions off), which stays a number in the walk of the cells and
    so it must with several lanes per particle"""
    params = scenes.workload_params(pbd, 40, 1000.0, iterations=3)
    params.lambda_epsilon = 0.1
    params.n_scorr = -1
    params.stabilization_iterations = stab
    params.kernel_width_neighbours = 2
    params.active |= pbd.ACTIVE["findNeighbours"]
    params.active &= ~pbd.ACTIVE["updatePositions"]
    params.flags |= pbd.FLAG_TRACK_IDS
    pos, vel = scenes.lattice(*shape, spacing=0.9, seed=33)
    a, b = (_run(pbd, params, pos, vel, 1, full_walk=fw) for fw in (False, True))
    assert np.isfinite(b["x"][:, :3]).all()
    for k in ("x", "v", "p"):
        assert np.array_equal(a[k], b[k], equal_nan=True), k


@pytest.mark.parametrize("numbers", [(20, 20, 20), (30, 30, 30)])
def test_rows_of_positions_that_are_not_numbers(need_gpu, pbd, scenes, numbers):
    """9,000 particles whose positions are not numbers (all in cell 0) beside a fluid at the wall: they and the
    fluid's particles next to them have long rows or, beyond 8,192 of them, walk the cells; what an entry that is
    not a number does to a sum must not depend on which"""
    params = scenes.workload_params(pbd, 40, 1000.0, iterations=1)
    params.lambda_epsilon = 0.1
    pos, vel = scenes.lattice(*numbers, origin=(1.6, 1.6, 1.6), spacing=0.9, seed=34)
    lost = np.full((9000, 4), np.nan, np.float32)
    pos, vel = np.concatenate([pos, lost]), np.concatenate([vel, np.zeros_like(lost)])
    out = []
    for flags in (0, 0, pbd.FLAG_FULL_WALK):
        p = params.copy()
        p.flags |= flags
        with pbd.Sim(p, len(pos)) as sim:
            sim.add_particles(pos, vel)
            sim.step(1)
            sim.sync()
            out.append({**sim.state(), "lambda": sim.debug()["lambda"]})
    for a in out[:2]:
        for k in ("x", "v", "p", "lambda"):
            assert np.array_equal(a[k], out[2][k], equal_nan=True), k
