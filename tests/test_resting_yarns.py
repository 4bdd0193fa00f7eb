"""A flat cloth at rest without gravity or wind: its yarns are as long as their
Eulerian length to the last bit, so the stretch term must give no force at any
crossing spacing. One rounding of |w| = 1 leaves h ks 1.1e-16, at least 1.4e-25
here; a hundredth of that is allowed (the crimp and shear terms of the pose
leave about 1e-31)."""
import numpy as np
import pytest

from emu_py import EmuCloth

Y, H = 1e3, 1e-3


@pytest.mark.parametrize("weave", [0, 1])
def test_no_stretch_force_at_rest(weave):
    rng = np.random.default_rng(0)
    for L in np.exp(rng.uniform(np.log(2e-4), np.log(1e-2), 60)):
        R = L / 10
        line = lambda n: np.tile([1e-3, Y, 1e-5], (n, 1))  # noqa: E731
        em = EmuCloth(width=6, length=5, weave=weave, pose=1, warp=line(5), weft=line(6), L=L, R=R, G=(0.0, 0.0, 0.0))
        em.assemble(H)
        _, b = em.system()
        assert np.abs(b).max() <= 1e-2 * H * Y * np.pi * R * R * 2.0 ** -53, L
