"""A substep of particles that are flattened, singular or inverted, for each
plasticity model and every path of the constraint, against the oracle."""
import numpy as np
import pytest

from parity_util import compare, perturbed_runs

pytestmark = pytest.mark.gpu

SIGMAS = (0.2, 1e-3, 1e-4, 0.0, -0.1, -0.9, -1.0)
DIRS = ((1, 0, 0), (1, 1, 0), (1, 1, 1))


def _plant(n):
    """Evenly spread particles with singular values (s, 1, 1), s along each direction."""
    F = np.zeros((n, 12), np.float32)
    F[:, [0, 5, 10]] = 1.0
    grads = []
    for axis in DIRS:
        d = np.array(axis, np.float64) / np.linalg.norm(axis)
        grads += [np.eye(3) + (s - 1.0) * np.outer(d, d) for s in SIGMAS]
    idx = np.linspace(0, n - 1, len(grads) + 2)[1:-1].astype(int)
    for i, g in zip(idx, grads):
        F[i].reshape(3, 4)[:, :3] = g.T
    return F, idx


@pytest.mark.parametrize("path", ["lanes1", "lanes2", "lanes4", "features"])
@pytest.mark.parametrize("model", ["elastic_block", "sand_two_blocks", "snowball_smash", "plasticine", "goo",
                                   "snow_classic"])
def test_flattened_and_inverted_particles(xp, oracle, built_lib, model, path):
    sc = getattr(xp.scenes, model)()
    p = xp.params_for(sc)
    it = 2
    F, idx = _plant(len(sc["positions"]))
    with xp.Simulation(sc) as sim:
        sim.write_params(p)
        if path == "features":
            sim.set_lanes(1)
            sim.set_solver(0, 0.0, False, True)
        else:
            sim.set_lanes(int(path[-1]))
        sim.write_state(0, F=F)
        s0 = sim.read_state()
        pw, mw = sim.uniforms()
        ref = oracle.substep(pw, mw, s0, it, False, -1)
        ref64 = oracle.substep(pw, mw, s0, it, False, -1, f64=True)
        sim.encode_substep(it, False)
        s1 = sim.read_state()
    for k in ("pos", "vel", "F", "L", "aux"):
        assert np.isfinite(s1[k]).all(), k
    compare(s1, ref, ref64,
            perturbed=perturbed_runs(oracle, sc, s0, iterations=it, has_water=False, xp=xp, params=p, positions=True))
    # the map's result is no inverted particle: the smallest singular value is clamped at 1e-3
    planted = np.isin(s1["sortedIdx"], idx)
    assert planted.sum() == len(idx)
    assert np.linalg.det(s1["F"].reshape(-1, 3, 4)[planted][:, :, :3].astype(np.float64)).min() > 0.0


@pytest.mark.parametrize("model", ["sand_two_blocks", "plasticine", "goo", "snow_classic"])
def test_strongly_stretched_particles(xp, oracle, built_lib, model):
    """Gradients of size 300, which the return maps bring back: the result is
    as accurate as its own size, not F's."""
    sc = getattr(xp.scenes, model)()
    p = xp.params_for(sc)
    F, idx = _plant(len(sc["positions"]))
    rng = np.random.default_rng(1)
    for i in idx:
        F[i].reshape(3, 4)[:, :3] = 300.0 * rng.normal(size=(3, 3))
    with xp.Simulation(sc) as sim:
        sim.write_params(p)
        sim.write_state(0, F=F)
        s0 = sim.read_state()
        pw, mw = sim.uniforms()
        ref = oracle.substep(pw, mw, s0, 1, False, -1)
        ref64 = oracle.substep(pw, mw, s0, 1, False, -1, f64=True)
        sim.encode_substep(1, False)
        s1 = sim.read_state()
    compare(s1, ref, ref64,
            perturbed=perturbed_runs(oracle, sc, s0, iterations=1, has_water=False, xp=xp, params=p, positions=True))
    scale = np.abs(ref64["F"]).max(axis=1, keepdims=True)
    far = np.isin(s1["sortedIdx"], idx)
    err = [(np.abs(x["F"] - ref64["F"]) / scale)[far].max() for x in (s1, ref)]
    assert err[0] <= max(1e-5, 4.0 * err[1]), err
