"""The source form of the state (tau_f == 1, float compute): phi, u and the
interface source stand for the phase-field populations between steps.  Stepping
it must give the same bits as stepping the stored populations, which reading
``f`` between steps brings back, over grids at the edges of the phi pass's
tiles and plane pairs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")


def _solver(grid, dtype, theta):
    from lbm.fe_ac_solver import AllenCahnSolver
    from lbm.fe_config import FEConfig
    nx, ny, nz = grid
    rng = np.random.default_rng(nx * 10000 + ny * 100 + nz)
    cfg = FEConfig(nx=nx, ny=ny, nz=nz, rho_l=1.0, rho_g=1.0 / 828.0, sigma=0.01424, xi=4.0, tau_l=0.53,
                   tau_g=0.53, theta_eq=theta, device="cuda")
    frac = np.zeros(grid)
    frac[:, :, 0] = 1.0
    if min(grid) > 4:  # a rough wall: partial nodes, boundary nodes of every orientation
        frac[:, :, 1] = rng.uniform(0.0, 1.0, grid[:2])
    phi = rng.uniform(0.0, 1.0, grid).astype(np.float32)
    u = rng.uniform(-0.02, 0.02, (3,) + grid).astype(np.float32)
    s = AllenCahnSolver(cfg, dtype=dtype, geo_amplification=1.5, geometric_wetting=True)
    s.set_solid(frac >= 0.5, frac)
    s.init_fields(phi, u)
    return s


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("grid,theta", [((2, 2, 2), 120.0), ((3, 5, 4), 150.0), ((7, 17, 18), 120.0),
                                        ((8, 33, 19), 162.0), ((17, 14, 106), 150.0), ((5, 9, 211), 100.0),
                                        ((40, 31, 27), 120.0), ((65, 8, 16), 150.0)])
def test_source_form_matches_stored_populations(grid, theta, dtype):
    a, b = _solver(grid, dtype, theta), _solver(grid, dtype, theta)
    for _ in range(5):
        a.run(1)
        b.run(1)
        f = b.f  # the state holds populations from here
        assert f.shape == (19,) + grid
    for x, y in zip(a.fields("phi", "u", "P") + [a.f, a.g], b.fields("phi", "u", "P") + [b.f, b.g]):
        assert torch.equal(x, y) or bool(((x == y) | (x.isnan() & y.isnan())).all())
    assert a.scalars() == b.scalars()
