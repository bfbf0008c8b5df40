"""The cave field's coarse grid against the oracle: every field point's material,
for densities and chunk sizes that take each grid stride, the longest one, or
no grid at all."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

BASE = dict(mode=2, octaves2=8, freq2=1 / 256, lacunarity2=2.0, gain2=0.5, amp2=48.0, octaves3=6, freq3=1 / 64,
            lacunarity3=2.0, gain3=0.5, amp3=12.0)
CASES = {
    "stride-4": ({}, (256, -128, 0), 1),
    "stride-2": ({}, (-512, -256, 512), 2),
    "scale-3": ({}, (0, -384, 768), 3),
    "no-grid": ({}, (0, -512, 0), 4),
    "stride-8": (dict(freq3=1 / 160), (0, -128, 512), 1),
    "slow-decay": (dict(gain3=0.8), (0, -128, 256), 1),
    "three-octaves": (dict(octaves3=3), (0, -128, 0), 1),
    "two-octaves": (dict(octaves3=2), (0, -128, 0), 1),
    "irrational": (dict(freq3=0.0131, lacunarity3=1.87, amp3=-15.0), (1024, -128, 256), 1),
    "far": ({}, (4 * (1 << 19), -128, -4 * (1 << 18)), 1),
    "farther": ({}, (4 * (1 << 21), -128, 0), 1),
}


@pytest.mark.parametrize("vpc", [16, 64])
@pytest.mark.parametrize("name", list(CASES))
def test_field_matches_oracle(lvn_gpu, name, vpc):
    lvn = lvn_gpu
    change, at, scale = CASES[name]
    d = dict(BASE, **change)
    lvn.clear_csg_operations()
    lvn.set_density(**d)
    O.set_seed(1)
    od = O.density(**{k.replace("lacunarity", "lac"): v for k, v in d.items()})
    size = 4 * vpc * scale
    mg = lvn.MeshGen(vpc)
    try:
        mg.set_option(lvn.LVN_OPT_CACHE, 0)
        chunks = [((at[0], at[1] + size * j, at[2]), size) for j in range(2)]
        mg.generate_chunks(chunks)
        for c, (mn, sz) in enumerate(chunks):
            ref = O.OracleChunk(od, mn, sz, vpc=vpc)
            mats = mg.debug_fetch(lvn.DEBUG_MATERIALS, c, np.uint8)
            assert np.array_equal(mats, ref.materials().astype(np.uint8)), (c, int((mats != ref.materials()).sum()))
    finally:
        mg.close()
