"""Cells that hold thousands of particles: the sort's permutation is the serial
one, and its cost does not grow with the square of a cell's members."""
import ctypes as C
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (8, 8, 8)


def _positions(cell, rng):
    """Particles at random points of the given cells of a unit grid."""
    pos = np.zeros((len(cell), 4), np.float32)
    pos[:, 0] = cell % DIMS[0]
    pos[:, 1] = cell // DIMS[0] % DIMS[1]
    pos[:, 2] = cell // (DIMS[0] * DIMS[1])
    pos[:, :3] += rng.uniform(0.1, 0.9, (len(cell), 3)).astype(np.float32)
    return pos


class _Sort:
    """The allocation-free sort on device buffers of its own."""

    def __init__(self, pos):
        self.torch = pytest.importorskip("torch")
        self.abi = importlib.import_module("xpbi-webgpu_gb300._abi")
        self.n, self.cells = len(pos), int(np.prod(DIMS))
        self.p = self.torch.from_numpy(pos).cuda()
        self.start = self.torch.empty(self.cells + 1, dtype=self.torch.int32, device="cuda")
        self.idx = self.torch.empty(self.n, dtype=self.torch.int32, device="cuda")
        self.stream = C.c_void_p(self.torch.cuda.current_stream().cuda_stream)

    def __call__(self):
        assert self.abi.lib().xpbi_sort_cells_noalloc(
            C.c_void_p(self.p.data_ptr()), self.n, (C.c_float * 3)(0, 0, 0), C.c_float(1.0), (C.c_int32 * 3)(*DIMS),
            C.c_void_p(self.start.data_ptr()), C.c_void_p(self.idx.data_ptr()), self.stream) == 0

    def results(self):
        self.start.fill_(-1)
        self.idx.fill_(-1)
        self()
        assert self.abi.lib().xpbi_sort_cells_noalloc_status(self.stream) == 0
        return self.start.cpu().numpy().view(np.uint32), self.idx.cpu().numpy().view(np.uint32)

    def best_ms(self):
        self()
        best = np.inf
        for _ in range(5):
            a, b = (self.torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            self()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best


# around the line of 8192 members, a part of a segment of 8192 particles past a
# whole one, and the sort's most particles
@pytest.mark.parametrize("members", [8191, 8192, 8193, 16385, 30011, 262144])
@pytest.mark.parametrize("mix", ["alone", "beside", "two"])
def test_permutation(built_lib, members, mix):
    rng = np.random.default_rng(members)
    n = members if mix == "alone" else min(262144, 2 * members + 777)
    cell = np.full(n, 77, np.int64)
    if mix == "beside":  # the others spread over the grid, in the first and last cells too
        other = rng.permutation(n)[members:]
        cell[other] = rng.integers(0, int(np.prod(DIMS)), len(other))
    elif mix == "two":   # two crowded cells, their particles interleaved at random
        cell[rng.permutation(n)[n - n // 2:]] = 78
    sort = _Sort(_positions(cell, rng))
    for _ in range(2):
        start, idx = sort.results()
        assert np.array_equal(start, np.concatenate([[0], np.cumsum(np.bincount(cell, minlength=sort.cells))]))
        assert np.array_equal(idx, np.lexsort((-np.arange(n), cell)))


def test_cost_of_one_cell(built_lib):
    """Eight times the members of one cell take at most eight times as long, a
    cost in proportion. (Comparing all with all makes every member's chain
    eight times as long, and there are eight times as many of them: 0.96 and
    14.3 ms.)"""
    rng = np.random.default_rng(0)
    small, large = (_Sort(_positions(np.full(n, 77, np.int64), rng)).best_ms() for n in (32768, 262144))
    assert large <= 8.0 * small, (small, large)


def test_substep_of_a_collapsed_scene(xp, built_lib):
    """A whole scene in one cell, and one of NaN positions (the grid clamps
    them into its first cell): the substep's own sort."""
    sc = xp.scenes.config_dam_breach(scale=0.05)
    n = len(sc["positions"])
    rng = np.random.default_rng(3)
    for nan in (False, True):
        with xp.Simulation(sc) as sim:
            sim.write_params(xp.params_for(sc))
            pos = sim.read_state()["pos"].copy()
            words = sim.uniforms()[0]
            origin, cs = words[:3].view(np.float32), words[3:4].view(np.float32)
            dims = words[4:7].astype(np.float32)
            inside = origin + cs * (np.floor(dims / 2) + rng.uniform(0.2, 0.8, (n, 3)).astype(np.float32))
            pos[:, :3] = np.nan if nan else inside
            sim.write_state(0, pos=pos)
            sim.encode_substep(1, False)
            st = sim.read_state()
        assert np.bincount(np.repeat(np.arange(len(st["cellTab"])), np.diff(np.append(st["cellTab"], n)))).max() == n
        assert np.array_equal(st["sortedIdx"], np.arange(n, dtype=np.uint32)[::-1])
