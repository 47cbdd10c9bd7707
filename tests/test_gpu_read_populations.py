"""Reading f between steps leaves the state as it is, whether it holds the populations or the source form, and may
overlap the next step from another stream; the stored populations (a checkpoint holds them) step on to the same bits as
the source form."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")


def _solver(grid, dtype, theta=120.0, seed=0, **kw):
    from lbm.fe_ac_solver import AllenCahnSolver
    from lbm.fe_config import FEConfig
    nz = grid[2] if len(grid) == 3 else 1
    rng = np.random.default_rng(seed + sum(g * 100 ** i for i, g in enumerate(grid)))
    cfg = FEConfig(nx=grid[0], ny=grid[1], nz=nz, rho_l=1.0, rho_g=1.0 / 828.0, sigma=0.01424, xi=4.0, tau_l=0.53,
                   tau_g=0.53, theta_eq=theta, device="cuda", **kw)
    frac = np.zeros(grid)
    frac[..., 0] = 1.0
    if grid[-1] > 4:  # a rough wall: partial nodes, boundary nodes of every orientation
        frac[..., 1] = rng.uniform(0.0, 1.0, grid[:-1])
    s = AllenCahnSolver(cfg, dtype=dtype, geo_amplification=1.5, geometric_wetting=True)
    s.set_solid(frac >= 0.5, frac)
    s.init_fields(rng.uniform(0.0, 1.0, grid).astype(np.float32),
                  rng.uniform(-0.02, 0.02, (len(grid),) + grid).astype(np.float32))
    return s


def _equal(x, y):
    return bool(((x == y) | (x.isnan() & y.isnan())).all())


def _same(a, b):
    for x, y in zip(a.fields("phi", "u", "P") + [a.f, a.g], b.fields("phi", "u", "P") + [b.f, b.g]):
        assert _equal(x, y)
    assert a.scalars() == b.scalars()


CASES = [((2, 2, 2), torch.float32), ((7, 17, 18), torch.float32), ((40, 31, 27), torch.float16),
         ((5, 9, 107), torch.float16), ((59, 58, 58), torch.float32), ((59, 58, 59), torch.float32),
         ((101, 97, 53), torch.float32), ((101, 97, 53), torch.float16), ((33, 40), torch.float32),
         ((6, 383), torch.float32)]


@pytest.mark.parametrize("grid,dtype", CASES)
def test_stored_populations_step_on_to_the_same_bits(grid, dtype):
    a, b = _solver(grid, dtype), _solver(grid, dtype)
    for _ in range(4):
        a.run(1)
        b.run(1)
        f = a.f
        b.load_state_dict(b.state_dict())  # b holds populations from here
        assert _equal(f, b.f)
    _same(a, b)


@pytest.mark.parametrize("grid,dtype", [((96, 96, 64), torch.float32), ((96, 96, 64), torch.float16),
                                        ((512, 512), torch.float32)])
def test_reading_f_on_another_stream_beside_a_step(grid, dtype):
    a, b = _solver(grid, dtype), _solver(grid, dtype)
    side = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(4):
        a.run(2)
        b.run(2)
        want = b.f
        reads = []
        for st in side:
            st.wait_stream(torch.cuda.current_stream())
            a._cache.clear()  # each stream makes its own read
            with torch.cuda.stream(st):
                reads.append(a.f)
        a.run(1)  # not ordered after the reads by this program
        b.run(1)
        torch.cuda.synchronize()
        for f in reads:
            assert _equal(f, want)
    _same(a, b)
