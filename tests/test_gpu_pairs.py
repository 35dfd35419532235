"""RK4 with its stages in pairs (csrc/kg_pair.cu): the bits of the oracle, on the
sizes where the paired form can go wrong -- one column or row beyond a tile of 28 x
8, tiles narrower than that, two or more chunks in phi, an even Nz (whose pole
partner is not an involution), both outer boundaries and metric forms -- and after
everything that leaves a state no ghost fill has seen."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [dict(Nx=16, Ny=9, Nz=17, xmin=1.8, xmax=12.0),     # one tile, partial rows and columns
         dict(Nx=4, Ny=5, Nz=5, xmin=1.8, xmax=6.0),        # the smallest grid
         dict(Nx=25, Ny=17, Nz=33, xmin=1.8, xmax=14.0),    # exactly 28 interior columns, 16 rows
         dict(Nx=26, Ny=18, Nz=70, xmin=1.8, xmax=15.0),    # one column and one row more, even Nz
         dict(Nx=61, Ny=12, Nz=12, xmin=1.8, xmax=30.0),
         dict(Nx=92, Ny=26, Nz=9, xmin=1.8, xmax=30.0)]


def _pair(g, metric="Kerr_Schild", bc="outflow", pairs=2):
    from kg_b200 import ScalarField
    from kg_b200.initial_data import shell_ylm
    from oracle.oracle import Oracle, KERR_SCHILD, SCHW_EF, OUTFLOW, INFLOW
    dev = ScalarField(g["Nx"], g["Ny"], g["Nz"], g["xmin"], g["xmax"], 0.25, m=0.3, metric=metric,
                      boundary_type_rmax=bc)
    dev._ck(dev._lib.kg_set_rk4_pairs(dev.handle, pairs))
    ora = Oracle(g["Nx"], g["Ny"], g["Nz"], g["xmin"], g["xmax"], CFL=0.25, m=0.3,
                 metric=KERR_SCHILD if metric == "Kerr_Schild" else SCHW_EF,
                 bc_rmax=OUTFLOW if bc == "outflow" else INFLOW)
    u0, _ = shell_ylm(g["Nx"], g["Ny"], g["Nz"], g["xmin"], g["xmax"], seed=4, r0=5.0, sd=1.0)
    dev.u = u0
    ora.set_state(u0)
    return dev, ora, u0


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("metric,bc", [("Kerr_Schild", "outflow"), ("Schw_EF", "inflow"),
                                       ("Kerr_Schild", "inflow")])
def test_paired_rk4_bitexact(grid, metric, bc):
    dev, ora, _ = _pair(grid, metric, bc)
    for n in (1, 2, 4, 1):  # a single step, graph replay, an odd count
        dev.rk4(nsteps=n)
        ora.rk4(n)
        assert np.array_equal(dev.u, ora.get_state())


@pytest.mark.parametrize("pairs", [2, 0])  # 0: the stages that store their own ghost values
@pytest.mark.parametrize("bc", ["outflow", "inflow"])
def test_rk4_after_other_writers_of_u(pairs, bc):
    """states whose seam planes no fill has left: set anew, one face filled alone,
    another stepper in between"""
    dev, ora, u0 = _pair(GRIDS[3], bc=bc, pairs=pairs)
    rng = np.random.default_rng(5)
    dev.rk4(nsteps=5)
    ora.rk4(5)
    rough = u0 + 1e-3 * (rng.normal(size=u0.shape) + 1j * rng.normal(size=u0.shape))  # seams and ghosts included
    dev.u = rough
    ora.set_state(rough)
    dev.rk4(nsteps=4)
    ora.rk4(4)
    assert np.array_equal(dev.u, ora.get_state())
    dev.pirk2(2)
    ora.pirk2(2)
    dev.rk4(nsteps=2)
    ora.rk4(2)
    assert np.array_equal(dev.u, ora.get_state())
    dev.boundary_xL()
    s = dev.u
    ora.set_state(s)
    dev.rk4(nsteps=3)
    ora.rk4(3)
    dev.rk3(nsteps=2)
    ora.rk3(2)
    assert np.array_equal(dev.u, ora.get_state())


def test_paired_mode_is_checked():
    dev, _, _ = _pair(GRIDS[0])
    assert dev._lib.kg_set_rk4_pairs(dev.handle, 3) != 0
    assert dev._lib.kg_set_rk4_pairs(dev.handle, -1) != 0
