"""One chunk's mesh through the single-chunk call: meshes that go through the
context's staging buffer and meshes too large for it match the batch call, cached
and fresh, simplified and not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BASE = dict(mode=2, octaves2=8, freq2=1 / 256, lacunarity2=2.0, gain2=0.5, amp2=48.0, octaves3=6, freq3=1 / 64,
            lacunarity3=2.0, gain3=0.5, amp3=12.0)
# a field whose sign changes at most voxels: more vertices than four to a face voxel
DENSE = dict(BASE, freq3=0.25, amp3=4096.0)


@pytest.mark.parametrize("vpc,density", [(8, BASE), (8, DENSE), (16, DENSE), (64, BASE), (64, DENSE)])
@pytest.mark.parametrize("cache", [0, 1])
@pytest.mark.parametrize("simplify", [-1.0, 0.05])
def test_single_chunk_matches_batch(lvn_gpu, vpc, density, cache, simplify):
    lvn = lvn_gpu
    lvn.clear_csg_operations()
    lvn.set_density(**density)
    size = 4 * vpc
    chunks = [((0, -size // 2, 0), size), ((size, -size // 2, 0), size), ((0, 1 << 16, 0), size)]
    mg, ref = lvn.MeshGen(vpc), lvn.MeshGen(vpc)
    try:
        mg.set_option(lvn.LVN_OPT_CACHE, cache)
        mg.set_simplify(simplify)
        ref.set_simplify(simplify)
        for rep in range(2):
            for mn, sz in chunks:
                v, t, s, _ = ref.generate_chunks([(mn, sz)])
                if density is DENSE and mn[1] < 0 and vpc <= 16 and simplify < 0:
                    assert v.shape[0] > 4 * vpc * vpc
                mesh = mg.generate_chunk_mesh(mn, sz, 1 << 18)
                assert np.array_equal(mesh.vertices.view(np.int32), v.view(np.int32))
                assert np.array_equal(mesh.triangles, t)
                assert np.array_equal(mesh.seams, s)
                mg.free_chunk_octree(mn, sz)  # the next call meshes again, from the cached field if there is one
    finally:
        mg.close()
        ref.close()
        lvn.set_density(mode=0)


@pytest.mark.parametrize("n", [4, 9])
@pytest.mark.parametrize("simplify", [-1.0, 0.05])
def test_overflowing_batch_matches_single(lvn_gpu, n, simplify):
    """Batches of chunks so dense that the first run overflows the edge or the
    leaf pools part of the way: the rerun's meshes are the single chunks'."""
    lvn = lvn_gpu
    lvn.clear_csg_operations()
    lvn.set_density(**DENSE)
    chunks = [((256 * i, -128, 0), 256) for i in range(n)]
    mg, one = lvn.MeshGen(64), lvn.MeshGen(64)
    try:
        one.set_option(lvn.LVN_OPT_CACHE, 0)
        mg.set_simplify(simplify)
        one.set_simplify(simplify)
        for rep in range(2):
            v, t, s, res = mg.generate_chunks(chunks)
            for c, (mn, sz) in enumerate(chunks):
                m = one.generate_chunk_mesh(mn, sz, 1 << 18)
                vo, nv, to, nt, so, ns = res[c, :6]
                assert res[c, 6] > 48 * 1024  # edges, past a chunk's share of the first pools
                assert np.array_equal(v[vo:vo + nv].view(np.int32), m.vertices.view(np.int32))
                assert np.array_equal(t[to:to + nt], m.triangles)
                assert np.array_equal(s[so:so + ns], m.seams)
    finally:
        mg.close()
        one.close()
        lvn.set_density(mode=0)
