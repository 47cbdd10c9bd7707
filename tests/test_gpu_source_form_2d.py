"""The source form of a 2-D (D2Q9) state against stepping the stored populations, which reading ``f`` between steps
brings back: the same bits, over extents at the edges of the phi pass's windows of columns (382 inner columns a
block, from 32 columns on) and of its runs of rows; checkpoints of either resume alike."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")


def _solver(grid, theta, init=True):
    from lbm.fe_ac_solver import AllenCahnSolver
    from lbm.fe_config import FEConfig
    nx, ny = grid
    rng = np.random.default_rng(nx * 10000 + ny)
    cfg = FEConfig(nx=nx, ny=ny, nz=1, rho_l=1.0, rho_g=1.0 / 828.0, sigma=0.01424, xi=4.0, tau_l=0.53, tau_g=0.53,
                   theta_eq=theta, device="cuda")
    frac = np.zeros(grid)
    frac[:, 0] = 1.0
    frac[:, 1] = rng.uniform(0.0, 1.0, nx)  # partial nodes, boundary nodes of every orientation
    s = AllenCahnSolver(cfg, dtype=torch.float32, geo_amplification=1.5, geometric_wetting=True)
    s.set_solid(frac >= 0.5, frac)
    if init:
        s.init_fields(rng.uniform(0.0, 1.0, grid).astype(np.float32),
                      rng.uniform(-0.02, 0.02, (2,) + grid).astype(np.float32))
    return s


def _same(a, b):
    for x, y in zip(a.fields("phi", "u", "P") + [a.f, a.g], b.fields("phi", "u", "P") + [b.f, b.g]):
        assert bool(((x == y) | (x.isnan() & y.isnan())).all())
    assert a.scalars() == b.scalars()


@pytest.mark.parametrize("grid,theta", [((41, 31), 120.0), ((3, 32), 150.0), ((2, 33), 120.0), ((64, 382), 162.0),
                                        ((129, 383), 100.0), ((37, 765), 150.0), ((700, 45), 120.0)])
def test_source_form_2d_matches_stored_populations(grid, theta):
    a, b = _solver(grid, theta), _solver(grid, theta)
    for _ in range(5):
        a.run(1)
        b.run(1)
        assert b.f.shape == (9,) + grid  # the state holds populations from here
    c = _solver(grid, theta, init=False)
    a.run(2)
    c.load_state_dict(a.state_dict())
    b.run(2)
    _same(a, b)
    for s in (a, b, c):
        s.run(3)
    _same(a, b)
    _same(a, c)
