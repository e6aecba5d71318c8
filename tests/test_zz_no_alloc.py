"""The allocation-free sort entry point (pbd_sort_keys_noalloc) against the step's own sort.

Hosts that own all device memory, or frame loops that must not stall on cudaMalloc, sort with
pbd_sort_keys_noalloc, whose working memory is a fixed array inside the library.  Its output
must be the same as the sort the step runs with the memory it allocated at pbd_create
(pbd_debug_front + pbd_debug_dump): integer keys and indices, so bit for bit.  Two calls in a
row with different inputs check that the shared fixed array is cleared between calls.
This file is collected last on purpose: it keeps a fixed array on the GPU for the rest of the
process."""
import ctypes as C

import numpy as np
import pytest

from helpers import workload

pytestmark = pytest.mark.gpu


def _step_sort(pbd, scenes, shape, seed):
    """Keys before the sort, sorted keys and permutation from the step's own sort."""
    params, pos, vel = workload(pbd, scenes, shape=shape, box=max(shape) + 8, seed=seed)
    rng = np.random.default_rng(seed)
    vel[:, :3] = rng.normal(0, 20, size=(len(vel), 3)).astype(np.float32)
    with pbd.Sim(params, len(pos)) as sim:
        sim.add_particles(pos, vel)
        sim.front()
        d = sim.debug()
    keys_sorted, perm = d["keys"], d["perm"]
    keys_in = np.empty_like(keys_sorted)
    keys_in[perm] = keys_sorted
    return keys_in, keys_sorted, perm


def _sort_noalloc(pbd, keys_in, key_bits=24):
    import torch
    d_in = torch.tensor(keys_in.view(np.int32), device="cuda")
    d_keys = torch.full_like(d_in, -1)
    d_perm = torch.full_like(d_in, -1)
    stream = torch.cuda.current_stream()
    rc = pbd.lib().pbd_sort_keys_noalloc(C.c_void_p(d_in.data_ptr()), C.c_void_p(d_keys.data_ptr()),
                                         C.c_void_p(d_perm.data_ptr()), len(keys_in), key_bits,
                                         C.c_void_p(stream.cuda_stream))
    pbd.check(rc)
    stream.synchronize()
    return d_keys.cpu().numpy().view(np.uint32), d_perm.cpu().numpy().view(np.uint32)


def test_noalloc_sort_matches_the_step_sort_twice(need_gpu, pbd, scenes):
    for shape, seed in (((40, 40, 40), 31), ((70, 33, 50), 32)):
        keys_in, keys_sorted, perm = _step_sort(pbd, scenes, shape, seed)
        k, p = _sort_noalloc(pbd, keys_in)
        assert np.array_equal(k, keys_sorted)
        assert np.array_equal(p, perm)


@pytest.mark.parametrize("key_bits", [1, 8, 16, 20, 24, 32])
@pytest.mark.parametrize("n", [1, 100, 4097, 65537, 1 << 20])
def test_noalloc_sort_orders_by_the_low_key_bits(need_gpu, pbd, key_bits, n):
    # every pass count (1 to 4, so both ends of the ping-pong through the fixed array), partial
    # last tiles, one key, the 1,048,576-key limit; keys carry bits above key_bits, which must
    # not take part in the order (a stable sort by the low bits)
    rng = np.random.default_rng(key_bits * 1000003 + n)
    keys = rng.integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32)
    keys[::2] &= np.uint32(0xFFFF003F)   # plenty of equal low bits, so stability is exercised
    mask = np.uint32(0xFFFFFFFF if key_bits == 32 else (1 << key_bits) - 1)
    order = np.argsort(keys & mask, kind="stable")
    k, p = _sort_noalloc(pbd, keys, key_bits=key_bits)
    assert np.array_equal(p, order.astype(np.uint32))
    assert np.array_equal(k, keys[order])
    assert pbd.lib().pbd_sort_noalloc_status(None) == pbd.OK


def test_noalloc_sort_reports_a_wait_that_ran_out(need_gpu, pbd):
    # a short wait limit and a first tile that never publishes its counts: every look-back wait
    # on it gives up (no hang, no trap), the status says so, and the next call is clean again
    L = pbd.lib()
    keys = np.random.default_rng(7).integers(0, 1 << 24, size=50000, dtype=np.uint64).astype(np.uint32)
    try:
        pbd.check(L.pbd_debug_set_wait_limit(None, 2000, 1))
        _sort_noalloc(pbd, keys)
        assert L.pbd_sort_noalloc_status(None) == pbd.ERR_TIMEOUT
        assert b"gave up" in L.pbd_last_error()
    finally:
        pbd.check(L.pbd_debug_set_wait_limit(None, 0, 0))
    k, p = _sort_noalloc(pbd, keys)
    assert L.pbd_sort_noalloc_status(None) == pbd.OK
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(p, order.astype(np.uint32)) and np.array_equal(k, keys[order])


def test_noalloc_sort_rejects_more_keys_than_its_fixed_memory(need_gpu, pbd):
    import torch
    buf = torch.zeros(16, dtype=torch.int32, device="cuda")
    ptr = C.c_void_p(buf.data_ptr())
    rc = pbd.lib().pbd_sort_keys_noalloc(ptr, ptr, ptr, (1 << 20) + 1, 24, None)
    assert rc == pbd.ERR_CAPACITY
    assert b"at most 1048576" in pbd.lib().pbd_last_error()


@pytest.mark.parametrize("n", [1024, 1025, 152 * 1024, 152 * 1024 + 1, 152 * 2048 + 1, 152 * 4096, 152 * 4096 + 1, 6656 * 150 + 1])
def test_noalloc_sort_at_the_edges_of_its_tile_sizes(need_gpu, pbd, n):
    # the tile size follows n (sort_plan): the last n of a size, the first of the next, one key over
    rng = np.random.default_rng(n)
    keys = (rng.integers(0, 1 << 21, size=n, dtype=np.uint64) >> rng.integers(0, 12, size=n, dtype=np.uint64)).astype(np.uint32)
    order = np.argsort(keys, kind="stable")
    k, p = _sort_noalloc(pbd, keys, key_bits=21)
    assert np.array_equal(p, order.astype(np.uint32)) and np.array_equal(k, keys[order])
    assert pbd.lib().pbd_sort_noalloc_status(None) == pbd.OK


@pytest.mark.parametrize("offset,n", [(0, 4099), (1, 4099), (2, 7), (3, 300001)])
def test_noalloc_sort_of_keys_at_any_word(need_gpu, pbd, offset, n):
    # the counting pass reads four keys at a time only from a 16-byte boundary; two sorts in a row, the
    # second finds the counts the first one's last tile left zero
    import torch
    keys = np.random.default_rng(offset).integers(0, 1 << 21, size=n + offset, dtype=np.uint64).astype(np.uint32)
    d = torch.tensor(keys.view(np.int32), device="cuda")[offset:]
    out, perm = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
    order = np.argsort(keys[offset:], kind="stable")
    for _ in range(2):
        pbd.check(pbd.lib().pbd_sort_keys_noalloc(d.data_ptr(), out.data_ptr(), perm.data_ptr(), n, 21, None))
        assert pbd.lib().pbd_sort_noalloc_status(None) == pbd.OK
        assert np.array_equal(perm.cpu().numpy().view(np.uint32), order.astype(np.uint32))


@pytest.mark.parametrize("key_bits", [1, 9, 21, 32])
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 2048, 2049, 4095, 4096, 4097])
def test_noalloc_sort_of_few_keys_by_one_block(need_gpu, pbd, n, key_bits):
    # up to 4,096 keys one block runs all passes, with 1, 2 or 4 keys per thread; bits above key_bits stay out
    rng = np.random.default_rng(n + key_bits)
    keys = (rng.integers(0, 1 << 32, size=n, dtype=np.uint64) & 0xFFFF00FF).astype(np.uint32)
    order = np.argsort(keys & np.uint32((1 << key_bits) - 1), kind="stable")
    k, p = _sort_noalloc(pbd, keys, key_bits=key_bits)
    assert np.array_equal(p, order.astype(np.uint32)) and np.array_equal(k, keys[order])


def test_noalloc_status_is_of_the_last_call_also_for_few_keys(need_gpu, pbd):
    L = pbd.lib()
    many, few = (np.random.default_rng(s).integers(0, 1 << 24, size=s, dtype=np.uint64).astype(np.uint32) for s in (50000, 500))
    try:
        pbd.check(L.pbd_debug_set_wait_limit(None, 2000, 1))
        _sort_noalloc(pbd, many)
        assert L.pbd_sort_noalloc_status(None) == pbd.ERR_TIMEOUT
    finally:
        pbd.check(L.pbd_debug_set_wait_limit(None, 0, 0))
    for keys in (few, many):
        k, _ = _sort_noalloc(pbd, keys)
        assert L.pbd_sort_noalloc_status(None) == pbd.OK
        assert np.array_equal(k, np.sort(keys))


@pytest.mark.parametrize("shape", [(1, 1, 1), (8, 8, 16), (5, 5, 41), (16, 16, 8), (3, 683, 1)])
@pytest.mark.parametrize("forces", [True, False])
def test_step_sort_of_few_particles_by_one_block(need_gpu, pbd, scenes, shape, forces):
    # 1, 1,024, 1,025, 2,048 and 2,049 particles (the last by the tiles' passes), 3 and 4 passes
    params = scenes.workload_params(pbd, 128, 1000.0)
    if not forces:
        params.active &= ~pbd.ACTIVE["applyForces"]
    pos, vel = scenes.lattice(*shape, spacing=0.15 if max(shape) > 100 else 0.9, seed=28)
    pos, vel = pos[::-1].copy(), vel[::-1].copy()
    with pbd.Sim(params, len(pos)) as sim:
        sim.add_particles(pos, vel)
        sim.front()
        d = sim.debug()
    keys, perm = d["keys"], d["perm"].astype(np.int64)
    assert np.array_equal(np.sort(perm), np.arange(len(pos)))
    before = np.empty_like(keys)
    before[perm] = keys
    assert np.array_equal(np.argsort(before, kind="stable"), perm)


def _cut_short(pbd, keys, key_bits):
    """A sort whose last pass never runs: the call recorded as a graph, its last node taken out."""
    import torch
    rt = C.CDLL("libcudart.so.13")
    d = torch.tensor(keys.view(np.int32), device="cuda")
    out, perm = torch.empty_like(d), torch.empty_like(d)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    graph, exe, count = C.c_void_p(), C.c_void_p(), C.c_size_t()
    st = C.c_void_p(stream.cuda_stream)
    assert rt.cudaStreamBeginCapture(st, 1) == 0
    rc = pbd.lib().pbd_sort_keys_noalloc(d.data_ptr(), out.data_ptr(), perm.data_ptr(), len(keys), key_bits, st)
    assert rt.cudaStreamEndCapture(st, C.byref(graph)) == 0 and rc == pbd.OK
    assert rt.cudaGraphGetNodes(graph, None, C.byref(count)) == 0
    nodes = (C.c_void_p * count.value)()
    assert rt.cudaGraphGetNodes(graph, nodes, C.byref(count)) == 0
    last = []
    for node in nodes:
        after = C.c_size_t()
        assert rt.cudaGraphNodeGetDependentNodes(C.c_void_p(node), None, None, C.byref(after)) == 0
        if after.value == 0:
            last.append(node)
    assert len(last) == 1 and count.value > 2
    assert rt.cudaGraphDestroyNode(C.c_void_p(last[0])) == 0
    assert rt.cudaGraphInstantiate(C.byref(exe), graph, C.c_ulonglong(0)) == 0
    assert rt.cudaGraphLaunch(exe, st) == 0
    stream.synchronize()
    rt.cudaGraphExecDestroy(exe)
    rt.cudaGraphDestroy(graph)


@pytest.mark.parametrize("n,after", [(50000, 30000), (30000, 50000), (1 << 20, 5000), (5000, 1 << 20)])
def test_noalloc_sort_after_a_call_that_did_not_finish(need_gpu, pbd, n, after):
    # a call leaves nothing that the next one relies on: when its last pass never ran (a launch that
    # failed), the next sort, of more or of fewer tiles, and the one after it are right all the same
    rng = np.random.default_rng(n)
    first, second = (rng.integers(0, 1 << 21, size=k, dtype=np.uint64).astype(np.uint32) for k in (n, after))
    _sort_noalloc(pbd, first, key_bits=21)
    _cut_short(pbd, first, 21)
    for keys in (second, first):
        k, p = _sort_noalloc(pbd, keys, key_bits=21)
        order = np.argsort(keys, kind="stable")
        assert np.array_equal(p, order.astype(np.uint32)) and np.array_equal(k, keys[order])
        assert pbd.lib().pbd_sort_noalloc_status(None) == pbd.OK
