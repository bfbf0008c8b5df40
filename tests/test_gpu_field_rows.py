"""Heightfield fields in batches on both sides of the size from which a CTA takes
four rows of z, whose last rows and columns are remainders at every chunk size:
every chunk's materials, edges, leaves and mesh against the same chunk alone."""
import numpy as np
import pytest

from leven_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vpc", [8, 16, 32, 64])
@pytest.mark.parametrize("mode", ["terrain", "fbm2d"])
@pytest.mark.parametrize("n", [31, 32, 45])
def test_batch_field_matches_single(lvn_gpu, vpc, mode, n):
    lvn = lvn_gpu
    lvn.clear_csg_operations()
    lvn.set_density(**(dict(mode=0) if mode == "terrain" else W.FBM2D))
    size = 4 * vpc
    base = 2304 if mode == "terrain" else 128
    y0 = base - base % size
    chunks = [((size * (i % 7), y0 + size * (i % 3 - 1), size * (i // 7)), size) for i in range(n)]
    mg, one = lvn.MeshGen(vpc), lvn.MeshGen(vpc)
    try:
        one.set_option(lvn.LVN_OPT_CACHE, 0)
        v, t, s, res = mg.generate_chunks(chunks)
        fields = [mg.debug_fetch(lvn.DEBUG_MATERIALS, c, np.uint8) for c in range(n)]
        for c, (mn, sz) in enumerate(chunks):
            m = one.generate_chunk_mesh(mn, sz)
            vo, nv, to, nt, so, ns = res[c, :6]
            assert np.array_equal(fields[c], one.debug_fetch(lvn.DEBUG_MATERIALS, 0, np.uint8))
            assert np.array_equal(v[vo:vo + nv].view(np.int32), m.vertices.view(np.int32))
            assert np.array_equal(t[to:to + nt], m.triangles)
            assert np.array_equal(s[so:so + ns], m.seams)
    finally:
        mg.close()
        one.close()
        lvn.set_density(mode=0)
