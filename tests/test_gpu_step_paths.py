"""The size-dependent routes of a re-sort: which list build and which sort kernel runs depends
on sizes and density.  Each route at the sizes where it can go wrong (partial warps and tiles,
runs that change row of cells, lists beyond a stage, crowded cells) against the CPU oracle."""
import numpy as np
import pytest

from espressopp_b200 import _abi
from simdriver import Sim, cell_grid, cuda_lib, mb_velocities, oracle_lib

pytestmark = pytest.mark.gpu

RC, SKIN = 2.5, 0.3
SHIFT = 4.0 * (RC ** -12 - RC ** -6)
RHO = 0.8442


def _box_lattice(nx, ny, nz, rho=RHO, jitter=0.05, seed=1):
    a = rho ** (-1.0 / 3.0)
    k = np.arange(nx * ny * nz)
    pos = (np.stack([k % nx, (k // nx) % ny, k // (nx * ny)], 1) + 0.5) * a
    pos += np.random.default_rng(seed).uniform(-jitter, jitter, pos.shape)
    return pos, np.array([nx, ny, nz]) * a


def _fluid(lib, prec, pos, box, types=None, vel=None, rc=RC, excl=None, grid=None):
    s = Sim(lib, box, SKIN, cell_grid(box, rc, SKIN) if grid is None else grid, precision=prec,
            seed=7)
    s.add(np.arange(len(pos)), pos, vel, types)
    s.decompose()
    s.vl(rc, excl=excl)
    for t1, t2, eps, sig in ((0, 0, 1.0, 1.0), (0, 1, 1.5, 0.8), (1, 1, 0.5, 0.88)):
        if types is not None or t2 == 0:
            q = (sig / rc) ** 6
            s.lj(t1, t2, eps, sig, rc, 4.0 * eps * (q * q - q))
    s.integrator(0.005)
    return s


# lattice edges: partial last runs of 32, rows of cells shorter and longer than a run, few and
# wide cells, elongated boxes
@pytest.mark.parametrize("shape", [(11, 11, 11), (13, 13, 12), (9, 40, 11), (61, 9, 9),
                                   (17, 19, 23)])
@pytest.mark.parametrize("excluded", [False, True])
def test_build_pair_set(shape, excluded):
    pos, box = _box_lattice(*shape, jitter=0.2, seed=sum(shape))
    n = len(pos)
    excl = None
    if excluded:
        k = np.arange(0, n - 1, 3)
        excl = np.stack([k, k + 1], 1)
    g = _fluid(cuda_lib(), _abi.PREC_MIXED, pos, box, excl=excl)
    o = _fluid(oracle_lib(), _abi.PREC_FP64, pos, box, excl=excl)
    assert g.digest() == o.digest()
    g.vl_rebuild()  # on the cells of the re-sort: the reference's neighbour cells enforced
    assert g.digest() == o.digest()


@pytest.mark.parametrize("rc", [3.2, 3.6, 5.0])
def test_long_lists(rc):
    """Lists beyond the block form's stages (capacity above 192 entries) take the run form."""
    pos, box = _box_lattice(17, 17, 18, jitter=0.2, seed=4)
    g = _fluid(cuda_lib(), _abi.PREC_MIXED, pos, box, rc=rc)
    o = _fluid(oracle_lib(), _abi.PREC_FP64, pos, box, rc=rc)
    assert g.digest() == o.digest()


def test_narrow_cells():
    """Cells narrower than the list cutoff: partners come from the 27 neighbour cells only."""
    pos, box = _box_lattice(20, 20, 20, jitter=0.2, seed=5)
    grid = [int(b / 1.6) for b in box]
    g = _fluid(cuda_lib(), _abi.PREC_MIXED, pos, box, rc=1.6, grid=grid)
    o = _fluid(oracle_lib(), _abi.PREC_FP64, pos, box, rc=1.6, grid=grid)
    assert g.digest() == o.digest()


@pytest.mark.parametrize("n", [31, 700, 6000])
def test_crowded_cells(n):
    """27 cells of up to 222 particles: a re-sort block holds more rows than its shared memory
    ranks.  Uniform random points, pair set and order-independent state only."""
    rng = np.random.default_rng(n)
    box = np.full(3, 3.3)
    pos = rng.uniform(0.0, 3.3, (n, 3))
    sims = []
    for lib in (cuda_lib(), oracle_lib()):
        s = Sim(lib, box, 0.1, [3, 3, 3], seed=3)
        s.add(np.arange(n), pos, mb_velocities(n, 1.0, 2))
        s.decompose()
        s.vl(0.45)
        sims.append(s)
    g, o = sims
    assert g.digest() == o.digest()
    for a, b in zip(g.particles(np.arange(n)), o.particles(np.arange(n))):
        assert np.array_equal(a, b)
