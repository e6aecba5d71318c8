"""Batched scenes: many independent scenes in one simulation must evolve exactly as each scene
stepped alone (same sort order, same arithmetic), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene_list(scenes):
    out = []
    for k, (shape, box, rho, g, seed) in enumerate([((6, 5, 7), 16, 950.0, -9.0, 41), ((8, 8, 8), 16, 1050.0, -10.5, 42),
                                                      ((4, 9, 3), 20, 1000.0, -8.2, 43), ((10, 6, 10), 24, 900.0, -11.0, 44)]):
        pos, vel = scenes.lattice(*shape, seed=seed)
        rng = np.random.default_rng(seed)
        vel[:, :3] = rng.normal(0, 3, size=(len(vel), 3)).astype(np.float32)
        out.append(dict(pos=pos, vel=vel, box=box, rho=rho, g=g))
    return out


def _shared(pbd, scenes):
    p = scenes.workload_params(pbd, 16, 1000.0, vorticity=0.0005, viscosity=0.01)
    p.lambda_epsilon = 0.1
    return p


def _single(pbd, shared, sc):
    p = shared.copy()
    p.rest_density = sc["rho"]
    p.gravity = sc["g"]
    for a in range(3):
        p.bounds_min[a] = 1.5
        p.bounds_max[a] = sc["box"] - 1.5
    return p


def test_batch_equals_scenes_stepped_alone(need_gpu, pbd, scenes):
    shared = _shared(pbd, scenes)
    sl = _scene_list(scenes)
    descs = [pbd.scene_desc(len(sc["pos"]) + 5, sc["rho"], sc["g"], sc["box"]) for sc in sl]
    with pbd.Batch(shared, descs) as b:
        for k, sc in enumerate(sl):
            b.add_particles(k, sc["pos"], sc["vel"])
        b.step(6)
        b.sync()
        got = [b.state(k) for k in range(len(sl))]
    for k, sc in enumerate(sl):
        with pbd.Sim(_single(pbd, shared, sc), len(sc["pos"])) as s:
            s.add_particles(sc["pos"], sc["vel"])
            s.step(6)
            s.sync()
            ref = s.state()
        assert np.array_equal(got[k]["x"], ref["x"]), k
        assert np.array_equal(got[k]["v"], ref["v"]), k


def test_batch_add_between_frames_and_autotune(need_gpu, pbd, scenes, tmp_path):
    shared = _shared(pbd, scenes)
    sl = _scene_list(scenes)
    descs = [pbd.scene_desc(len(sc["pos"]) + 5, sc["rho"], sc["g"], sc["box"]) for sc in sl]
    cache = tmp_path / "tune.jsonl"
    with pbd.Batch(shared, descs) as b:
        for k, sc in enumerate(sl):
            b.add_particles(k, sc["pos"][:-5], sc["vel"][:-5])
        b.step(2)
        for k, sc in enumerate(sl):
            b.add_particles(k, sc["pos"][-5:], sc["vel"][-5:])
        assert b.count(0) == len(sl[0]["pos"])
        with pytest.raises(pbd.PBDError) as e:
            b.add_particles(0, sl[0]["pos"][:6], sl[0]["vel"][:6])
        assert e.value.code == pbd.ERR_CAPACITY
        blk = b.autotune(str(cache))
        assert blk in (64, 128, 256)
        assert cache.read_text().count("signature") == 1
        assert b.autotune(str(cache)) == blk            # served from the cache
        b.step(3)
        b.sync()
        assert all(np.all(np.isfinite(b.state(k)["x"])) for k in range(len(sl)))


def test_batch_state_with_interleaved_adds(need_gpu, pbd, scenes):
    """a scene's state is its sorted run followed by what was added since: adds in turns, before the
    first frame and after it, in the order they came"""
    shared = _shared(pbd, scenes)
    sl = _scene_list(scenes)
    descs = [pbd.scene_desc(len(sc["pos"]), sc["rho"], sc["g"], sc["box"]) for sc in sl]
    half = [len(sc["pos"]) // 2 for sc in sl]
    with pbd.Batch(shared, descs) as b:
        for k in (2, 0, 3):
            b.add_particles(k, sl[k]["pos"][:half[k]], sl[k]["vel"][:half[k]])
        b.add_particles(2, sl[2]["pos"][half[2]:-3], sl[2]["vel"][half[2]:-3])
        assert len(b.state(1)["x"]) == 0
        assert np.array_equal(b.state(2)["x"], sl[2]["pos"][:-3]) and np.array_equal(b.state(2)["v"], sl[2]["vel"][:-3])
        assert np.array_equal(b.state(3)["x"], sl[3]["pos"][:half[3]])
        b.step(2)
        b.sync()
        before = [b.state(k) for k in range(len(sl))]
        b.add_particles(1, sl[1]["pos"], sl[1]["vel"])
        b.add_particles(0, sl[0]["pos"][half[0]:], sl[0]["vel"][half[0]:])
        after = [b.state(k) for k in range(len(sl))]
    for k, tail in enumerate((sl[0]["pos"][half[0]:], sl[1]["pos"], sl[2]["pos"][:0], sl[3]["pos"][:0])):
        assert np.array_equal(after[k]["x"], np.concatenate([before[k]["x"], tail])), k
    for k, n in ((0, half[0]), (2, len(sl[2]["pos"]) - 3), (3, half[3])):
        with pbd.Sim(_single(pbd, shared, sl[k]), n) as s:
            s.add_particles(sl[k]["pos"][:n], sl[k]["vel"][:n])
            s.step(2)
            s.sync()
            ref = s.state()
        assert np.array_equal(before[k]["x"], ref["x"]) and np.array_equal(before[k]["v"], ref["v"]), k


def test_batch_state_after_many_small_adds(need_gpu, pbd, scenes):
    """a scene filled a particle at a time, alone or in turns with another scene: its state comes in a few
    copies, not two for every add, and in the order of the adds"""
    from helpers import device_events
    shared = _shared(pbd, scenes)
    sl = _scene_list(scenes)
    descs = [pbd.scene_desc(len(sc["pos"]), sc["rho"], sc["g"], sc["box"]) for sc in sl]
    with pbd.Batch(shared, descs) as b:
        for i in range(len(sl[0]["pos"])):
            b.add_particles(0, sl[0]["pos"][i:i + 1], sl[0]["vel"][i:i + 1])
        for i in range(len(sl[1]["pos"])):
            for k in (1, 2):
                b.add_particles(k, sl[k]["pos"][i:i + 1], sl[k]["vel"][i:i + 1])
        for frames in (0, 2):
            b.step(frames)
            for k in (0, 1, 2):
                got = []
                names = device_events(lambda: got.append(b.state(k)))
                assert sum("Memcpy" in s for s in names) <= 16, (frames, k, len(names))
                n = min(len(sl[k]["pos"]), len(sl[1]["pos"])) if k else len(sl[0]["pos"])
                assert len(got[0]["x"]) == n
                if not frames:
                    assert np.array_equal(got[0]["x"], sl[k]["pos"][:n]) and np.array_equal(got[0]["v"], sl[k]["vel"][:n])
