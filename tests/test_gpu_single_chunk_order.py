"""A single chunk's mesh and the caller's own pending work on its arrays: what the
legacy default stream still has to do with them comes before the mesh, whether they
lie in device or in pinned host memory."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHUNK = ((0, 128, 0), 256)
CAP = 1 << 15


def mesh_out(lvn, memory, v, t, s):
    return lvn.MeshOut(memory, v.data_ptr(), CAP, 0, t.data_ptr(), 2 * CAP, 0, s.data_ptr(), CAP, 0)


@pytest.mark.parametrize("cache", [0, 1])
@pytest.mark.parametrize("where,host_writes", [("device", 1), ("pinned", 1), ("pinned", 0)])
def test_mesh_comes_after_pending_work(lvn_gpu, cache, where, host_writes):
    import torch

    lvn = lvn_gpu
    lvn.set_density(lvn.LVN_DENSITY_FBM2D)
    lvn.clear_csg_operations()
    mg = lvn.MeshGen(64)
    try:
        mg.set_option(lvn.LVN_OPT_CACHE, cache)
        mg.set_option(lvn.LVN_OPT_HOST_WRITES, host_writes)
        want = mg.generate_chunk_mesh(*CHUNK)
        dev = where == "device"
        make = dict(device="cuda") if dev else dict(pin_memory=True)
        arrays = [torch.full((n, w), -7.0, **make) for n, w in ((CAP, 12), (2 * CAP, 3), (CAP, 12))]
        seen = [torch.zeros(a.shape, device="cuda") for a in arrays]
        torch.cuda.synchronize()
        mg.free_chunk_octree(*CHUNK)
        torch.cuda._sleep(200_000_000)  # a tenth of a second of other work on the default stream
        for a, b in zip(arrays, seen):
            b.copy_(a, non_blocking=True)  # the caller still reads what the arrays hold
            if dev:
                a.fill_(-9.0)  # and writes them
        out = mesh_out(lvn, lvn.LVN_MEMORY_DEVICE if dev else lvn.LVN_MEMORY_HOST, *arrays)
        rc = lvn.lib().lvn_meshgen_generate_chunk_mesh(mg.handle, lvn._ivec3(CHUNK[0]), CHUNK[1], C.byref(out))
        assert rc == 0
        torch.cuda.synchronize()
        got = [a.cpu().numpy().view(np.int32) for a in arrays]
        for b in seen:
            assert bool((b == -7.0).all())
        assert out.num_triangles > 0
        assert np.array_equal(got[0][:out.num_vertices], want.vertices.view(np.int32))
        assert np.array_equal(got[1][:out.num_triangles], want.triangles)
        assert np.array_equal(got[2][:out.num_seams], want.seams)
    finally:
        mg.close()
        lvn.set_density(mode=0)
