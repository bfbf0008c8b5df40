"""The crossing search and its forms against the oracle, bit for bit, where its
rules can go wrong: densities whose octaves are odd in number, absent, growing,
negative or not powers of two, coarse chunks whose edges span noise cells, and
coordinates at which a float has few bits left for the noise."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

BASE = dict(mode=2, octaves2=8, freq2=1 / 256, lacunarity2=2.0, gain2=0.5, amp2=48.0, octaves3=6, freq3=1 / 64,
            lacunarity3=2.0, gain3=0.5, amp3=12.0)
CASES = {
    "caves-lod0": ({}, (0, 0, 0), 64),
    "caves-lod5": ({}, (-8192, -2048, 4096), 2048),
    "heightfield": (dict(mode=1), (256, 0, -512), 64),
    "odd-octaves": (dict(octaves2=7, octaves3=5), (64, 0, 64), 64),
    "one-octave": (dict(octaves2=1, octaves3=1), (0, 0, 64), 64),
    "no-cave-octaves": (dict(octaves3=0), (0, 0, 0), 64),
    "no-height-octaves": (dict(octaves2=0), (0, -32, 0), 64),
    "growing-gain": (dict(gain3=1.5, amp3=2.0, octaves3=4), (0, 0, 0), 64),
    "negative": (dict(amp2=-30.0, gain3=-0.7, amp3=-9.0, freq3=-1 / 50), (0, 0, -320), 64),
    "irrational": (dict(freq2=0.0037, lacunarity2=1.93, freq3=0.021, lacunarity3=2.17), (1000, 0, 640), 64),
    "rough": (dict(freq3=0.9, amp3=6.0), (0, 0, 0), 128),
    "far": ({}, (4 * (1 << 20), 0, -4 * (1 << 19)), 64),
    "very-far": ({}, (4 * (1 << 23), 0, 4 * (1 << 22)), 256),
}


@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("name", list(CASES))
def test_search_matches_oracle(lvn_gpu, name, form):
    """form 0 is the default (16 lanes an edge on a batch this small), 1 and 2
    the searching kernel with its tables in shared and in global memory."""
    lvn = lvn_gpu
    change, at, size = CASES[name]
    d = dict(BASE, **change)
    lvn.clear_csg_operations()
    lvn.set_density(**d)
    O.set_seed(1)
    od = {k.replace("lacunarity", "lac"): v for k, v in d.items()}
    mg = lvn.MeshGen(16)
    try:
        mg.set_option(lvn.LVN_OPT_CACHE, 0)
        mg.set_option(lvn.LVN_OPT_HERMITE_FORM, form)
        chunks = [((at[0], at[1] + size * j, at[2]), size) for j in (-2, -1, 0, 1)]
        mg.generate_chunks(chunks)
        edges = 0
        for c, (mn, sz) in enumerate(chunks):
            ref = O.OracleChunk(O.density(**od), mn, sz, vpc=16)
            keys = mg.debug_fetch(lvn.DEBUG_EDGE_KEYS, c, np.int32)
            assert np.array_equal(keys, ref.edge_keys())
            info = mg.debug_fetch(lvn.DEBUG_EDGE_INFO, c, np.float32, 4)
            assert np.array_equal(info.view(np.uint32), ref.edge_info().view(np.uint32))
            edges += keys.size
        assert edges > 0 or name in ("far", "very-far")
    finally:
        mg.close()
