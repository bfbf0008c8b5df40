"""Edits of cached chunks that run out of device memory: the call either makes the
edit or returns an error with the field as it was, and what the chunk is meshed
from afterwards is the field of a context that had the memory."""
import numpy as np
import pytest

from leven_gb300 import workloads as W

pytestmark = pytest.mark.gpu

CHUNK = ((0, 0, 0), 256)


def same_mesh(a, b):
    assert a.triangles.shape[0] > 0
    assert np.array_equal(a.vertices.view(np.int32), b.vertices.view(np.int32))
    assert np.array_equal(a.triangles, b.triangles)
    assert np.array_equal(a.seams, b.seams)


def brushes(lvn, k, n):
    """n operations, a different set for every k, whose surfaces add to the chunk's edges."""
    rng = np.random.default_rng(k)
    return [lvn.make_op(0, 1, 3 + i % 4, rng.uniform(8.0, 56.0, 3), (6.0, 6.0, 6.0)) for i in range(n)]


@pytest.mark.parametrize("fail", [1, 2])
def test_edit_without_memory_for_its_edges(lvn_gpu, fail):
    """The allocations for the longer edge list fail, which only happens once the
    corners are changed: the edit stands, with its edges."""
    lvn = lvn_gpu
    lvn.set_density(**W.FBM2D)
    lvn.clear_csg_operations()
    mg, ref = lvn.MeshGen(64), lvn.MeshGen(64)
    try:
        same_mesh(mg.generate_chunk_mesh(*CHUNK), ref.generate_chunk_mesh(*CHUNK))
        for k in range(3):
            edges = mg.debug_fetch(lvn.DEBUG_EDGE_KEYS, 0, np.int32).size
            lvn.inject_fault(lvn.LVN_FAULT_DEVICE_ALLOC, fail)
            mg.apply_csg_operations(brushes(lvn, k, 4), *CHUNK)
            lvn.inject_fault(lvn.LVN_FAULT_NONE, 0)
            ref.apply_csg_operations(brushes(lvn, k, 4), *CHUNK)
            keys = mg.debug_fetch(lvn.DEBUG_EDGE_KEYS, 0, np.int32)
            assert keys.size > edges
            assert np.array_equal(keys, ref.debug_fetch(lvn.DEBUG_EDGE_KEYS, 0, np.int32))
            assert np.array_equal(mg.debug_fetch(lvn.DEBUG_MATERIALS, 0, np.uint8),
                                  ref.debug_fetch(lvn.DEBUG_MATERIALS, 0, np.uint8))
            for c in (mg, ref):
                c.free_chunk_octree(*CHUNK)
            same_mesh(mg.generate_chunk_mesh(*CHUNK), ref.generate_chunk_mesh(*CHUNK))
        # the pools, some of whose buffers went to the entry, serve other calls
        far = [((512, 0, 0), 256), ((512, 0, 256), 256)]
        for x, y in zip(mg.generate_chunks(far), ref.generate_chunks(far)):
            assert np.array_equal(x.view(np.int32), y.view(np.int32))
    finally:
        lvn.inject_fault(lvn.LVN_FAULT_NONE, 0)
        mg.close()
        ref.close()
        lvn.set_density(mode=0)


@pytest.mark.parametrize("stored", [True, False])
def test_edit_refused_before_it_starts(lvn_gpu, stored):
    """No memory for the operations themselves: an error, the field unchanged, and
    the same operations (stored ones by replay) are made by the next call."""
    lvn = lvn_gpu
    lvn.set_density(**W.FBM2D)
    lvn.clear_csg_operations()
    ops = brushes(lvn, 9, 12)  # more than the operation buffer was made for
    mg, ref = lvn.MeshGen(64), lvn.MeshGen(64)
    try:
        before = mg.generate_chunk_mesh(*CHUNK)
        ref.generate_chunk_mesh(*CHUNK)
        for c in (mg, ref):
            c.free_chunk_octree(*CHUNK)
        if stored:
            for op in ops:
                lvn.store_csg_operation(op)
        lvn.inject_fault(lvn.LVN_FAULT_DEVICE_ALLOC, 1)
        with pytest.raises(lvn.LvnError) as e:
            mg.generate_chunk_mesh(*CHUNK) if stored else mg.apply_csg_operations(ops, *CHUNK)
        assert e.value.code == lvn.LVN_ERR_OUT_OF_MEMORY
        lvn.inject_fault(lvn.LVN_FAULT_NONE, 0)
        if not stored:
            same_mesh(mg.generate_chunk_mesh(*CHUNK), before)
            mg.free_chunk_octree(*CHUNK)
            for c in (mg, ref):
                c.apply_csg_operations(ops, *CHUNK)
        got, want = mg.generate_chunk_mesh(*CHUNK), ref.generate_chunk_mesh(*CHUNK)
        same_mesh(got, want)
        assert got.vertices.shape != before.vertices.shape
    finally:
        lvn.inject_fault(lvn.LVN_FAULT_NONE, 0)
        mg.close()
        ref.close()
        lvn.clear_csg_operations()
        lvn.set_density(mode=0)
