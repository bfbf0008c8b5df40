"""The noise bounds behind the crossing search (SearchBound in
leven_gb300/csrc/lvn_kernels.cu) and the cave field: second derivative along an
axis, magnitude, 1-norm of the gradient, and the share of lattice points
outside the evaluated simplex, of the simplex noise summed over all lattice
points.  A lattice point's gradient is any of the table's, independently of
its neighbours', so the sum over the lattice points in reach of each one's
largest contribution bounds the noise everywhere; it is maximised over a grid
of one cell.  The sums are smooth with their maxima inside the cell, so a grid of
this spacing misses them by well under the 5% the constants keep above it."""
import pathlib
import re

import numpy as np

SRC = (pathlib.Path(__file__).resolve().parents[1] / "leven_gb300" / "csrc" / "lvn_kernels.cu").read_text()
GRADS = [(0, 1, 1), (0, 1, -1), (0, -1, 1), (0, -1, -1), (1, 0, 1), (1, 0, -1), (-1, 0, 1), (-1, 0, -1), (1, 1, 0),
         (1, -1, 0), (-1, 1, 0), (-1, -1, 0)]
G = np.array([[int(v * 64 + 64) / 255 * 4 - 1 for v in g] for g in GRADS])


def constant(name):
    return float(re.search(rf"\b{name} = ([0-9.]+)f", SRC).group(1))


def cell(dim, skew, n):
    r = np.arange(-1, 3)
    L = np.stack(np.meshgrid(*[r] * dim, indexing="ij"), -1).reshape(-1, dim).astype(float)
    u = (np.arange(n) + 0.5) / n
    P = np.stack(np.meshgrid(*[u] * dim, indexing="ij"), -1).reshape(-1, dim)
    P = P - P.sum(1, keepdims=True) * skew
    return L, L - L.sum(1, keepdims=True) * skew, P


def largest(Lu, P, grads, radius, scale):
    """max over the points of the sums of |f|, |f_xx| and |f_x| + |f_y| (+ |f_z|)."""
    best = np.zeros(3)
    for c in range(0, len(P), 1 << 12):
        D = P[c:c + (1 << 12), None, :] - Lu[None]
        t = np.clip(radius - (D * D).sum(-1), 0, None)
        f = np.zeros((3,) + t.shape)
        for g in grads:
            gd = D @ g
            u = D[..., 0]
            grad = scale * (-8 * t[..., None] ** 3 * D * gd[..., None] + t[..., None] ** 4 * g)
            f2 = scale * (48 * t ** 2 * u * u * gd - 8 * t ** 3 * gd - 16 * t ** 3 * u * g[0])
            f[0] = np.maximum(f[0], np.abs(scale * t ** 4 * gd))
            f[1] = np.maximum(f[1], np.abs(f2))
            f[2] = np.maximum(f[2], np.abs(grad).sum(-1))
        best = np.maximum(best, f.sum(2).max(1))
    return best


def test_noise3_bounds():
    _, Lu, P = cell(3, 1 / 6, 32)
    value, curve, slope = largest(Lu, P, G, 0.6, 32.0)
    assert value * 1.005 <= constant("kNoise3Max")
    assert curve * 1.05 <= constant("kNoise3Curve")
    assert slope <= constant("kNoise3Slope")


def test_noise2_bounds():
    _, Lu, P = cell(2, 0.211324865405, 300)
    value, curve, slope = largest(Lu, P, G[:, :2], 0.5, 70.0)
    assert value * 1.005 <= constant("kNoise2Max")
    assert curve * 1.05 <= constant("kNoise2Curve")
    assert slope <= constant("kNoise2Slope")


def test_noise3_jump_bound():
    """The corners outside a point's simplex that lie within the kernel's radius."""
    L, Lu, P = cell(3, 1 / 6, 40)
    worst = 0.0
    for c in range(0, len(P), 1 << 13):
        x = P[c:c + (1 << 13)]
        xy, xz, yz = x[:, 0] >= x[:, 1], x[:, 0] >= x[:, 2], x[:, 1] >= x[:, 2]
        o1 = np.stack([xy & xz, ~xy & yz, ~xz & ~yz], 1).astype(int)
        o2 = np.stack([xy | xz, ~xy | yz, ~xz | ~yz], 1).astype(int)
        inside = np.zeros((len(x), len(L)), bool)
        for o in (np.zeros_like(o1), o1, o2, np.ones_like(o1)):
            inside |= (L[None] == o[:, None, :]).all(-1)
        D = x[:, None, :] - Lu[None]
        t = np.clip(0.6 - (D * D).sum(-1), 0, None)
        f = 32 * t ** 4 * np.abs(D @ G.T).max(-1)
        worst = max(worst, float((f * ~inside).sum(1).max()))
    assert worst * 1.03 <= constant("kNoise3Jump")
