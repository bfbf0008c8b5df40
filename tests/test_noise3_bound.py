"""kNoise3Bound (leven_gb300/csrc/lvn_types.h), the bound on |snoise3| by which the
cave field's band and octave remainders decide points: the lattice sum that it has
to lie above, the oracle's noise climbed to local maxima, and the oracle's cave term
against the band it gives."""
import ctypes as C
import pathlib
import re

import numpy as np

import oracle_lib as O
from test_search_bounds import G, cell, constant, largest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "leven_gb300" / "csrc"
BOUND = float(re.search(r"\bkNoise3Bound = ([0-9.]+);", (CSRC / "lvn_types.h").read_text()).group(1))


def test_one_constant():
    """The band, the remainders and the crossing search use this constant and no other."""
    api = (CSRC / "lvn_api.cu").read_text()
    assert "kNoise3Bound =" not in api
    assert "*band = cave_band(d, kNoise3Bound);" in api
    assert re.search(r"const double r = .*amp3\) \* kNoise3Bound \* sum", api)
    assert constant("kNoise3Max") == BOUND


def test_lattice_sum_within_bound():
    _, Lu, P = cell(3, 1 / 6, 36)
    value = largest(Lu, P, G, 0.6, 32.0)[0]
    assert 0.95 < value * 1.005 <= BOUND


def test_oracle_snoise3_within_bound():
    """The largest of random points, each climbed by steps of falling length."""
    L = O.lib()
    worst = 0.0
    for seed in (1, 7):
        O.set_seed(seed)
        rng = np.random.default_rng(seed)

        def noise(p):
            return np.array([abs(L.orc_snoise3(float(x), float(y), float(z))) for x, y, z in p.astype(np.float32)])

        pts = rng.uniform(-300.0, 300.0, (20000, 3))
        vals = noise(pts)
        top = np.argsort(vals)[-40:]
        pts, vals = pts[top], vals[top]
        for step in np.repeat([0.1, 0.05, 0.02, 0.01, 0.003], 12):
            trial = pts + rng.normal(0.0, step, pts.shape)
            v = noise(trial)
            better = v > vals
            pts[better], vals[better] = trial[better], v[better]
        worst = max(worst, float(vals.max()))
    O.set_seed(1)
    assert 0.75 < worst <= BOUND, worst


def test_cave_term_within_band():
    """|density - density without the 3D term| against |amp3| BOUND times the sum of the
    octave amplitudes plus 0.1 %, cave_band's value."""
    from leven_gb300 import workloads as W

    O.set_seed(1)
    d = W.CAVES
    dens = [O.density(mode=2, octaves2=d["octaves2"], freq2=d["freq2"], lac2=d["lacunarity2"], gain2=d["gain2"],
                      amp2=d["amp2"], octaves3=d["octaves3"], freq3=d["freq3"], lac3=d["lacunarity3"],
                      gain3=d["gain3"], amp3=a) for a in (d["amp3"], 0.0)]
    band = abs(d["amp3"]) * BOUND * sum(d["gain3"] ** k for k in range(d["octaves3"])) * 1.001
    L = O.lib()
    worst = 0.0
    for x, y, z in np.random.default_rng(11).uniform(-4096.0, 4096.0, (20000, 3)).astype(np.float32):
        a, b = (L.orc_density_at(C.byref(e), float(x), float(y), float(z)) for e in dens)
        worst = max(worst, abs(a - b))
    assert 0.0 < worst <= band, (worst, band)
