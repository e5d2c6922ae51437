"""Several engines in one process: what one engine sets up on the kernels that
they share holds for the others, in whatever order engines are created and used."""
import numpy as np
import pytest
import torch

import _gpu_helpers as H
from implicitvelocityprojection_b200 import scenes as S
from implicitvelocityprojection_b200._lib import IVPError

pytestmark = pytest.mark.gpu


def _scenes(n, first=0):
    return [S.random_column(400 + 60 * k, 2.0, seed=200 + first + k, viscosity_method=1, viscosity_coeff=1e-3)
            for k in range(n)]


def _solve(eng, n):
    """A force on its own, then a step: direct launches and (with graphs) a graph
    that is built at this first use."""
    eng.build()
    eng.viscosity_solve()
    eng.step(1)
    assert all(eng.stats(i).status == 0 for i in range(n))
    return [np.concatenate([eng.get("x", i), eng.get("v", i)]) for i in range(n)]


@pytest.mark.parametrize("use_graphs", [True, False])
@pytest.mark.parametrize("n,others", [(3, (1,)), (4, (5,)), (8, (1, 3)), (256, (1,))])
def test_engines_created_later_leave_earlier_ones_working(n, others, use_graphs):
    """The persistent kernels' shared memory grows with the engine's scenes (and
    four scenes take more than five, whose parameters stay in global memory; 256
    take more than the 48 KB that a kernel may use without asking).  Engines of
    other sizes, created in between and used first, change nothing."""
    scs = _scenes(n)
    alone = _solve(H.engine(scs, use_graphs=use_graphs), n)
    eng = H.engine(scs, use_graphs=use_graphs)
    later = [H.engine(_scenes(k, 500), use_graphs=use_graphs) for k in others]
    for k, e in zip(others, later):
        _solve(e, k)
    for a, b in zip(alone, _solve(eng, n)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("use_graphs", [True, False])
def test_step_stopped_half_way_leaves_the_engine_usable(use_graphs, n):
    """A step whose n-th launch fails (before, between and after its solves, and in the build) leaves
    their grid barriers and the build's counts ready: the next step is the step of a fresh engine from the
    state that the failed one left.  A graph's launch cannot stop half-way, so with
    graphs the failing step is a profiled one."""
    sc = S.random_column(3000, 2.0, seed=230, viscosity_method=1, viscosity_coeff=1e-3)
    eng = H.engine([sc], use_graphs=use_graphs, persistent=True)
    eng.build()
    eng.fail_launch(n)
    with pytest.raises(IVPError, match="ivp_fail_launch"):
        eng.profile_step(1) if use_graphs else eng.step(1)
    torch.cuda.synchronize()
    fresh = H.engine([H.with_state(sc, eng.get("x"), eng.get("v"))], use_graphs=use_graphs, persistent=True)
    for e in (eng, fresh):
        e.build()
        e.step(2)
        assert e.stats(0).status == 0
    assert np.array_equal(eng.get("x"), fresh.get("x")) and np.array_equal(eng.get("v"), fresh.get("v"))


@pytest.mark.parametrize("n", range(1, 13))
def test_build_stopped_half_way_leaves_the_engine_usable(n):
    """A build whose n-th launch fails, from the keys to the corrections of lists
    longer than the cache: the next build and solve are those of a fresh engine."""
    pts = S.lattice_block([0.1, 0.1, 0.1], (9, 9, 9), 0.0135, jitter=0.1, seed=5)
    sc = S.assemble([pts], [], particle_radius=0.01, domain_size=[0.5, 0.5, 0.5], max_outer_iters=2,
                    fixed_outer_iters=True)
    eng, fresh = (H.engine([sc], use_graphs=False) for _ in range(2))
    eng.fail_launch(n)
    with pytest.raises(IVPError, match="ivp_fail_launch"):
        eng.build()
    out = []
    for e in (eng, fresh):
        e.build()
        assert e.raw_stats(0).overflow_particles > 0
        e.solve()
        out.append([*e.neighbours(0), e.get("density"), e.get("k"), e.get("v")])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
