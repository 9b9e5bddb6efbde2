"""Models that are hard on the order of a solve. Rectangular blocks, one to six nodes a side, with few and rationally
related velocities: fronts meet at exactly equal traveltimes beside the shocks that the jumps make. And models of high
velocity contrast."""
import numpy as np

VALUES = ((1.0, 2.0, 4.0), (1.0, 1.5, 2.0, 2.5, 3.0))


def block_model(n, seed):
    """Velocities of the grid (n) and a source: on a node, in the middle of a cell or anywhere, by the seed."""
    rng = np.random.default_rng(seed)
    cut = []
    for k in n:
        side = []
        while sum(side) < k:
            side.append(int(rng.integers(1, 7)))
        cut.append(np.repeat(np.arange(len(side)), side)[:k])
    block = rng.choice(np.array(VALUES[seed % 2]), size=[c[-1] + 1 for c in cut])
    vel = np.ascontiguousarray(block[np.ix_(*cut)])
    src = np.random.default_rng(seed + 1000).uniform(4.0, np.array(n) - 4.0)
    if seed % 3 < 2:
        src = np.floor(src) + 0.5 * (seed % 3)
    return vel, src


def contrast_model(kind, n, contrast, seed):
    """Velocities between 1 and contrast: blocks of three values, independent at each node, smooth, or 1 but for
    a corner of three nodes a side."""
    rng = np.random.default_rng(seed)
    if kind == "blocks":
        v, _ = block_model(n, seed)
        u = np.unique(v)
        return np.exp(np.linspace(0.0, np.log(contrast), len(u)))[np.searchsorted(u, v)]
    if kind == "noise":
        return np.exp(np.log(contrast) * rng.random(n))
    if kind == "smooth":
        z = rng.standard_normal(n)
        for a in range(len(n)):
            for _ in range(6):
                z = (np.roll(z, 1, a) + z + np.roll(z, -1, a)) / 3
        return np.exp(np.log(contrast) * (z - z.min()) / (z.max() - z.min()))
    v = np.ones(n)
    v[tuple(slice(0, 3) for _ in n)] = contrast
    return v
