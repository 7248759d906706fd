"""The kernels' variants at the sizes where they change: lanes per particle,
shared PBF walks, the staged state, the network's gradient tiles, the scan's
look-back."""
import ctypes as C
import importlib

import numpy as np
import pytest

from oracle import mlp_ref as M
from parity_util import compare, perturbed_runs

pytestmark = pytest.mark.gpu


def _dam(xp, n_drop=7):
    """A thin dam breach (sand beside water), its particle count not a
    multiple of a warp."""
    sc = dict(xp.scenes.config_dam_breach(scale=0.05))
    for k in ("positions", "matIds", "states", "velocities", "colorSeeds"):
        if sc.get(k) is not None:
            sc[k] = sc[k][:len(sc[k]) - n_drop]
    return sc


def _substep(xp, oracle, sc, lanes, iterations, pbf, change=None, warm=2):
    p = dict(xp.params_for(sc), pbfIterations=pbf)
    with xp.Simulation(sc) as sim:
        sim.write_params(p)
        sim.set_lanes(lanes)
        sim.step(warm, iterations, True)
        if change is not None:
            st = sim.read_state()
            sim.write_state(0, **change(st))
        s0 = sim.read_state()
        pw, mw = sim.uniforms()
        ref = oracle.substep(pw, mw, s0, iterations, True, pbf)
        ref64 = oracle.substep(pw, mw, s0, iterations, True, pbf, f64=True)
        sim.encode_substep(iterations, True)
        s1 = sim.read_state()
    return s0, s1, ref, ref64, p


@pytest.mark.parametrize("lanes", [1, 2, 4])
@pytest.mark.parametrize("n_drop", [1, 31])
def test_lanes_of_every_kernel(xp, oracle, built_lib, lanes, n_drop):
    """Water beside sand, a PBF pass after every iteration: every kernel of
    the substep with one, two and four lanes per particle."""
    sc = _dam(xp, n_drop)
    s0, s1, ref, ref64, p = _substep(xp, oracle, sc, lanes, 4, 4)
    assert len(s1["pos"]) % 32 != 0
    compare(s1, ref, ref64, has_pbf=True, perturbed=perturbed_runs(oracle, sc, s0, xp=xp, params=p, iterations=4))


@pytest.mark.parametrize("lanes", [1, 4])
@pytest.mark.parametrize("spacing", [0.95, 0.9, 0.8])
def test_pbf_lists_of_compressed_water(xp, oracle, built_lib, lanes, spacing):
    """Water pressed together: the first pass's wider lists fit, fit for some
    particles, or for none (exact lists and stencil walks), and the
    corrections move particles past the lists' margin between passes."""
    sc = _dam(xp)
    kinds = np.array([m["kind"] for m in sc["materials"]])

    def change(st):
        pos = st["pos"].copy()
        w = kinds[np.abs(pos[:, 3]).astype(int)] == 6
        c = pos[w, :3].mean(axis=0)
        pos[w, :3] = (c + (pos[w, :3] - c) * spacing).astype(np.float32)
        return {"pos": pos}

    s0, s1, ref, ref64, p = _substep(xp, oracle, sc, lanes, 3, 3, change)
    compare(s1, ref, ref64, has_pbf=True,
            perturbed=perturbed_runs(oracle, sc, s0, xp=xp, params=p, iterations=3, count=6, positions=True))


def test_state_of_each_scene_of_a_batch(xp, built_lib):
    """The staged read-back: what was written comes back bit for bit, in the
    reference layouts, for scenes that start at odd particle offsets."""
    scenes = [xp.scenes.plasticine(), xp.scenes.snowball_smash(), xp.scenes.goo()]
    for k, drop in enumerate((1, 6, 0)):
        sc = scenes[k] = dict(scenes[k])
        for f in ("positions", "matIds", "states", "velocities", "colorSeeds"):
            if sc.get(f) is not None:
                sc[f] = sc[f][:len(sc[f]) - drop]
    rng = np.random.default_rng(3)
    with xp.Simulation(scenes) as sim:
        for k, sc in enumerate(scenes):
            sim.write_params(xp.params_for(sc), scene=k)
            sim.set_schedule(k, 2, sc["hasWater"])
        fresh = [sim.read_state(k) for k in range(3)]
        sim.step(2, -1, False)
        for k in range(3):
            n = sim.scene_sizes[k]
            st = sim.read_state(k)
            assert np.array_equal(np.sort(st["sortedIdx"]), np.arange(n, dtype=np.uint32))
            assert st["cellTab"][0] == 0 and (np.diff(st["cellTab"].astype(np.int64)) >= 0).all()
            assert st["cellTab"][-1] <= n
            assert np.array_equal(st["pos"], sim.read_pos(k))
            assert np.array_equal(st["aux"][:, 0], st["vel"][:, 3])
            assert (fresh[k]["aux"][:, 0] == fresh[k]["aux"][0, 0]).all() and fresh[k]["aux"][0, 0] > 0
            new = {"pos": st["pos"], "vel": rng.normal(size=(n, 4)).astype(np.float32),
                   "F": rng.normal(size=(n, 12)).astype(np.float32)}
            new["F"][:, 3::4] = 0.0
            new["vel"][:, 3] = st["vel"][:, 3]
            sim.write_state(k, **new)
            back = sim.read_state(k)
            for f in ("pos", "vel", "F"):
                assert np.array_equal(back[f], new[f]), (k, f)
            assert np.array_equal(back["L"], st["L"])


# Weights, activations and the derivatives handed to the tensor cores are
# rounded to bf16 (2^-9 relative), and a rounding that falls the other way in f32
# than in f64 moves an entry by 2^-8; three layers of that stay below 2e-2.
@pytest.mark.parametrize("rows", [1, 127, 128, 129, 300, 4099])
def test_gradient_of_ragged_batches(built_lib, rows):
    net = importlib.import_module("xpbi-webgpu_gb300.net")
    rng = np.random.default_rng(rows)
    X = rng.standard_normal((rows, 16)).astype(np.float32)
    T = rng.standard_normal(rows).astype(np.float32)
    p = M.init(5)
    g, loss = net.grad(X, T, p)
    gr, lr = M.grad(X, T, p)
    assert abs(loss - lr) <= 2e-2 * (lr + float((T.astype(np.float64) ** 2).mean()))
    o = 0
    for name, shape in M.SIZES:
        n = int(np.prod(shape))
        e = np.abs(g[o:o + n] - gr[o:o + n]).max() / max(np.abs(gr[o:o + n]).max(), 1e-30)
        assert e < 2e-2, (name, e)
        o += n


@pytest.mark.parametrize("dims", [(1, 1, 1), (16, 16, 16), (64, 64, 33), (128, 128, 64)])
def test_scan_over_many_tiles(built_lib, dims):
    """1, 2, 34 and 257 tiles of 4096 cells: the look-back reads 32 at a time."""
    torch = pytest.importorskip("torch")
    abi = importlib.import_module("xpbi-webgpu_gb300._abi")
    rng = np.random.default_rng(1)
    n, cells = 4999, int(np.prod(dims))
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0, 1, (n, 3)) * np.array(dims)
    cell = np.minimum(np.floor(pos[:, :3]).astype(np.int64), np.array(dims) - 1)
    key = cell[:, 0] + dims[0] * (cell[:, 1] + dims[1] * cell[:, 2])
    want = np.lexsort((-np.arange(n), key)).astype(np.uint32)
    start = np.concatenate([[0], np.cumsum(np.bincount(key, minlength=cells))]).astype(np.uint32)
    p = torch.from_numpy(pos).cuda()
    cs = torch.empty(cells + 1, dtype=torch.int32, device="cuda")
    si = torch.empty(n, dtype=torch.int32, device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        rc = abi.lib().xpbi_sort_cells_noalloc(C.c_void_p(p.data_ptr()), n, (C.c_float * 3)(0, 0, 0), C.c_float(1.0),
                                               (C.c_int32 * 3)(*dims), C.c_void_p(cs.data_ptr()),
                                               C.c_void_p(si.data_ptr()), stream)
        assert rc == 0
        assert abi.lib().xpbi_sort_cells_noalloc_status(stream) == 0
        assert np.array_equal(cs.cpu().numpy().view(np.uint32), start)
        assert np.array_equal(si.cpu().numpy().view(np.uint32), want)
