"""The closed form the edge kernels use for the four-state multidimensional
Riemann solver at symmetrised (LLF) speeds and one E,

    E + s / (2 sin t) ((By_R - By_L) - (Bn_U - Bn_D)),

against the oracle's general solver on seeded inputs (any angle that a mesh's
edge frames show, fields and E of either sign, strong and vanishing speeds).
Tolerance: 64 roundings of the largest term, s |B| / sin^2 t or |E| (the
general form divides by sin t twice)."""
import numpy as np
import pytest

from oracle import twod_rs_ez_4state


@pytest.mark.parametrize("orthogonal", [True, False])
def test_closed_form_matches_the_general_solver(orthogonal):
    rng = np.random.default_rng(5)
    for _ in range(2000):
        t = 0.5 * np.pi if orthogonal else rng.uniform(0.3, np.pi - 0.3)
        c, sn = (0.0, 1.0) if orthogonal else (np.cos(t), np.sqrt(1.0 - np.cos(t) ** 2))
        s = 10.0 ** rng.uniform(-6, 3)
        E = rng.normal() * 10.0 ** rng.uniform(-6, 2)
        bnu, bnd, byr, byl = rng.normal(size=4) * 10.0 ** rng.uniform(-4, 2)
        want = twod_rs_ez_4state(s, -s, s, -s, c, sn, E, E, E, E, bnu, bnd, byr, byl)
        got = E + 0.5 * s * ((byr - byl) - (bnu - bnd)) / sn
        scale = abs(E) + s * max(abs(bnu), abs(bnd), abs(byr), abs(byl)) / sn ** 2
        assert abs(got - want) <= 64 * 2.0 ** -53 * scale
