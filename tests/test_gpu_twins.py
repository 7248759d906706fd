"""Exactly coincident solids: a particle's twin is a term of 0 in every sum, so
twins that start alike stay bit for bit together, as in the reference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SUBSTEPS = 6


def _doubled(xp, spacing):
    """A sand body every particle of which is there twice."""
    rng = np.random.default_rng(0)
    h = 0.02
    g = np.stack(np.meshgrid(*[np.arange(12)] * 3), -1).reshape(-1, 3) * (spacing * h) + 0.2
    g = (g + rng.normal(0.0, 0.1 * spacing * h, g.shape)).astype(np.float32)
    order = rng.permutation(2 * len(g))  # others lie between two twins
    return dict(positions=np.concatenate([g, g])[order], matIds=np.zeros(2 * len(g), np.uint32),
                materials=[xp.scenes.SAND(30, 0.0)], states=None, velocities=None, colorSeeds=None, h=h,
                domainMin=[0, 0, 0], domainMax=[1, 1, 1], gravity=[0, -9.81, 0], iterations=6, hasWater=False,
                substeps=4, timeScale=0.5), order % len(g)


# half the spacing: some 130 solid neighbours each, past the lists' 64
@pytest.mark.parametrize("spacing", [1.0, 0.5])
@pytest.mark.parametrize("lanes", [1, 2, 4])
def test_twins_stay_together(xp, oracle, built_lib, lanes, spacing):
    sc, body = _doubled(xp, spacing)
    p = xp.params_for(sc, dt=5e-4)
    n = len(body)
    with xp.Simulation(sc) as sim:
        sim.write_params(p)
        sim.set_lanes(lanes)
        ids = np.arange(n)
        for _ in range(SUBSTEPS):
            pw, mw = sim.uniforms()
            ref = oracle.substep(pw, mw, sim.read_state(), sc["iterations"], False, -1)
            sim.step(1, sc["iterations"], False)
            st = sim.read_state()
            ids = ids[st["sortedIdx"]]
            pairs = np.argsort(body[ids], kind="stable").reshape(-1, 2)
            for state, who in ((ref, "oracle"), (st, "GPU")):
                for f in ("pos", "vel", "F"):
                    a, b = state[f][pairs[:, 0]], state[f][pairs[:, 1]]
                    assert np.array_equal(a, b), (who, f, int((a != b).any(axis=1).sum()))
