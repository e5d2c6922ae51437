"""The neighbour build's branches that ordinary scenes seldom take: windows too
crowded for the filter pass, particles scattered one per cell (more runs than a
warp keeps windows for), ragged last tiles and slices, and every number of lanes
per particle, which sets how many slots a warp takes and how rows interleave.
"""
import numpy as np
import pytest

import _gpu_helpers as H
from implicitvelocityprojection_b200 import scenes as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LANES = [(1, 128), (2, 128), (4, 64), (8, 16)]  # lanes per particle, particles per tile


def _scattered(n, seed):
    """Particles far apart: most cells hold one, some none."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.1, 1.5, size=(n, 3)).astype(np.float32)
    return S.assemble([x], [], particle_radius=0.01, domain_size=[1.6, 1.6, 1.6])


def _crowded(n, seed):
    """More than 512 particles around every cell, each with few neighbours: all
    but a thin plate lies outside the domain, where the cells are clamped."""
    rng = np.random.default_rng(seed)
    x = rng.uniform([0.05, 0.05, 0.05], [1.0, 0.09, 0.09], size=(n, 3)).astype(np.float32)
    return S.assemble([x], [], particle_radius=0.005, domain_size=[0.12, 0.12, 0.12])


def _block(n, seed):
    w = max(2, int(round(n ** (1.0 / 3.0))) + 1)
    pts = S.lattice_block([0.1, 0.1, 0.1], (w, w, w), 0.0186, jitter=0.15, seed=seed)[:n]
    return S.assemble([pts], [S.domain_walls([0.9, 0.9, 0.9], 0.02)], particle_radius=0.01, domain_size=[0.9, 0.9, 0.9])


SCENES = {
    "one": lambda: _block(1, 1), "seven": lambda: _block(7, 2), "ragged_33": lambda: _block(33, 3),
    "ragged_65": lambda: _block(65, 4), "block_1001": lambda: _block(1001, 5),
    "scattered_600": lambda: _scattered(600, 6), "crowded_900": lambda: _crowded(900, 7),
}


@pytest.mark.parametrize("build_kernel", [1, 2])
@pytest.mark.parametrize("scene", sorted(SCENES))
def test_sums_are_the_same_bits_at_every_lane_count(scene, build_kernel):
    """Build kernel 1 adds density and k in list order: one lane walking its own
    hits (1 and 2 lanes per particle), eight lanes sharing them (4 and 8), and a
    whole warp on a particle whose window does not fit give the same bits.  Build
    kernel 2 adds them by eight lanes, whatever the number of slots a warp takes."""
    sc = SCENES[scene]()
    out = []
    for lanes, ppb in LANES:
        eng = H.engine([sc], lanes_per_particle=lanes, particles_per_block=ppb, build_kernel=build_kernel)
        eng.build()
        out.append((lanes, eng.get("density"), eng.get("k")))
    for lanes, density, k in out[1:]:
        assert np.array_equal(density, out[0][1]), lanes
        assert np.array_equal(k, out[0][2]), lanes


@pytest.mark.parametrize("lanes,ppb", LANES)
@pytest.mark.parametrize("build_kernel", [1, 2])
def test_neighbour_without_mass_gives_the_reference_k(build_kernel, lanes, ppb):
    """A dynamic neighbour of mass zero adds 0 / 0 to Aii (pressure_base.py:49-87
    multiplies |J|^2 by 1 / m): k is NaN around it, as the oracle's, and nowhere
    else."""
    sc = _block(1001, 8)
    sc.density0 = sc.density0.copy()
    sc.density0[[5, 400]] = 0.0
    eng = H.engine([sc], lanes_per_particle=lanes, particles_per_block=ppb, build_kernel=build_kernel)
    eng.build()
    with np.errstate(divide="ignore", invalid="ignore"):
        st = O.State.from_scene(sc)
    st.rebuild()
    dyn = sc.is_dynamic == 1
    k, want = eng.get("k")[dyn], st.k[dyn]
    assert 10 < np.isnan(want).sum() < 200
    assert np.array_equal(np.isnan(k), np.isnan(want))
    np.testing.assert_allclose(k[~np.isnan(k)], want[~np.isnan(want)], rtol=1e-5)
