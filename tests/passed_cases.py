"""Cloths on which two neighbouring crossings have passed each other along a
yarn: their Eulerian positions exchanged, so that the edge between them has a
negative Eulerian length (du < 0)."""
import numpy as np

CASES = [(weave, k, kf) for weave in range(3) for k in range(2) for kf in (0.0, 1000.0)]


def kwargs(weave, kf, width=7, length=6, base=(2e-3, 170000.0, 1e-4)):
    rng = np.random.default_rng(weave)
    line = lambda n: np.asarray(base) * rng.uniform(0.8, 1.2, (n, 3))  # noqa: E731
    return dict(width=width, length=length, weave=weave, pose=1, warp=line(length), weft=line(width), kf=kf,
                handles=[(0, 0), (width - 1, 0)])


def state(rest, kw, k, amp=1e-4):
    """The rest state `rest` bent by `amp`, in motion, crossings (2, 2) and its
    neighbour along yarn k (0: warp, 1: weft) exchanged."""
    rng = np.random.default_rng(7)
    W, H = kw["width"], kw["length"]
    v, u = np.divmod(np.arange(W * H), W)
    inside = ((u > 0) & (u < W - 1) & (v > 0) & (v < H - 1))[:, None]
    st = {key: np.array(x, float) for key, x in rest.items()}
    N = W * H
    st["LPos"] = st["LPos"] + amp * rng.standard_normal((N, 3))
    st["LVel"] = 1e-2 * rng.standard_normal((N, 3))
    st["EPos"] = st["EPos"] + inside * 2e-6 * rng.standard_normal((N, 2))
    st["EVel"] = inside * 1e-4 * rng.standard_normal((N, 2))
    a, b = 2 + 2 * W, 2 + 2 * W + (W if k else 1)
    st["EPos"][[a, b], k] = st["EPos"][[b, a], k]
    return st
