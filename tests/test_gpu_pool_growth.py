"""Pools that cannot grow and caches that are dropped.  A batch whose pools cannot
grow (a device allocation fails after the first run has found them too small) returns
an error and leaves the context usable: the next batch, one that the pools had already
held, meshes as before."""
import numpy as np
import pytest

from leven_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# a field whose sign changes at most voxels
DENSE = dict(mode=2, octaves2=8, freq2=1 / 256, lacunarity2=2.0, gain2=0.5, amp2=48.0, octaves3=6, freq3=0.25,
             lacunarity3=2.0, gain3=0.5, amp3=4096.0)


@pytest.mark.parametrize("n", [4, 9])
@pytest.mark.parametrize("simplify", [-1.0, 0.05])
def test_context_survives_a_failed_growth(lvn_gpu, n, simplify):
    lvn = lvn_gpu
    lvn.clear_csg_operations()
    chunks = [((256 * i, -128, 0), 256) for i in range(n)]
    mg = lvn.MeshGen(64)
    try:
        mg.set_simplify(simplify)
        lvn.set_density(**W.FBM2D)
        before = mg.generate_chunks(chunks)
        for rep in range(2):
            lvn.set_density(**DENSE)
            lvn.inject_fault(lvn.LVN_FAULT_DEVICE_ALLOC, 1)
            with pytest.raises(lvn.LvnError) as e:
                mg.generate_chunks(chunks)
            assert e.value.code == lvn.LVN_ERR_OUT_OF_MEMORY
            lvn.inject_fault(lvn.LVN_FAULT_NONE, 0)
            with pytest.raises(lvn.LvnError):  # the failed batch is not there to be fetched
                mg.debug_fetch(lvn.DEBUG_EDGE_KEYS, 0, np.int32)
            lvn.set_density(**W.FBM2D)
            after = mg.generate_chunks(chunks)
            assert before[1].shape[0] > 0
            for x, y in zip(before, after):
                assert np.array_equal(x.view(np.int32), y.view(np.int32))
    finally:
        lvn.inject_fault(lvn.LVN_FAULT_NONE, 0)
        mg.close()
        lvn.set_density(mode=0)


def test_dropped_caches_give_their_memory_back(lvn_gpu):
    """Setting a context's surrogate drops its cached fields: 200 rounds of two cached
    64^3 chunks (1.5 MB each) leave the device's free memory where it was."""
    import torch

    lvn = lvn_gpu
    lvn.clear_csg_operations()
    lvn.set_density(**W.FBM2D)
    chunks = [((0, 0, 0), 256), ((256, 0, 0), 256)]
    mg = lvn.MeshGen(64)

    def rounds(n):
        for _ in range(n):
            meshes = [mg.generate_chunk_mesh(*c) for c in chunks]
            assert all(m.triangles.shape[0] > 0 for m in meshes)
            mg.set_surrogate(None)
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    try:
        before = rounds(5)
        assert rounds(200) >= before - (64 << 20)
    finally:
        mg.close()
        lvn.set_density(mode=0)
