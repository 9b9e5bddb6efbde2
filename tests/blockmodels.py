"""Models of rectangular blocks, one to six nodes a side, with few and rationally related velocities: fronts
meet at exactly equal traveltimes beside the shocks that the jumps make."""
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
