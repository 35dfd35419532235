"""The ghost fill (csrc/kg_boundary.cu) on rows one point short of a multiple of its
blocks' columns, at it and one and two beyond -- the outermost column copies its
neighbour, which may be another block's -- and the state exchange with device
buffers that the conversion can and cannot reach in place."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = [127, 128, 129, 130, 257]  # points of a row along r


def _solve(ni, Ny=6, Nz=8, bc="outflow"):
    from kg_b200 import ScalarField
    rng = np.random.default_rng(ni)
    s = ScalarField(ni - 5, Ny, Nz, 1.8, 30.0, 0.25, m=0.3, boundary_type_rmax=bc)
    assert s.NI == ni
    u0 = rng.normal(size=s.state_shape()) + 1j * rng.normal(size=s.state_shape())
    s.u = u0
    return s, u0


def _oracle(ni, u0, Ny=6, Nz=8, bc="outflow"):
    from oracle.oracle import Oracle, INFLOW, KERR_SCHILD, OUTFLOW
    ora = Oracle(ni - 5, Ny, Nz, 1.8, 30.0, CFL=0.25, m=0.3, metric=KERR_SCHILD,
                 bc_rmax=OUTFLOW if bc == "outflow" else INFLOW)
    ora.set_state(u0)
    return ora


@pytest.mark.parametrize("method", ["pirk2", "pirk3", "rk3"])
@pytest.mark.parametrize("Nz", [8, 9])  # the partner of the seam plane differs
@pytest.mark.parametrize("bc", ["outflow", "inflow"])
@pytest.mark.parametrize("ni", ROWS)
def test_fill_bitexact(ni, bc, Nz, method):
    dev, u0 = _solve(ni, Nz=Nz, bc=bc)
    ora = _oracle(ni, u0, Nz=Nz, bc=bc)
    getattr(dev, method)(nsteps=3)
    getattr(ora, method)(3)
    assert np.array_equal(dev.u, ora.get_state())


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batched_fill_matches_solo(precision):
    from kg_b200.batch import Batch
    batch = Batch(precision=precision)
    solos, members = [], []
    for ni in ROWS:
        m, _ = _solve(ni)
        s, _ = _solve(ni)
        s.precision = precision
        batch.add(m)
        members.append(m)
        solos.append(s)
    batch.rk4(3)
    for m, s in zip(members, solos):
        s.rk4(nsteps=3)
        assert np.array_equal(m.u, s.u)


@pytest.mark.parametrize("shift", [0, 8])  # bytes beyond a 16-byte boundary
@pytest.mark.parametrize("which", [0, 1])  # u; u_stage, whose Pi changes places with every step
def test_device_exchange_in_place_and_staged(which, shift):
    import torch
    dev, _ = _solve(37)
    dev.pirk2(nsteps=3)
    n = dev._get(which).size
    buf = torch.zeros(2 * n + 2, dtype=torch.float64, device="cuda")
    base = buf[shift // 8:shift // 8 + 2 * n]
    assert base.data_ptr() % 16 == shift
    torch.cuda.synchronize()
    ptr = C.c_void_p(base.data_ptr())
    want = dev._get(which)
    dev._ck(dev._lib.kg_get_state_device(dev.handle, which, ptr))
    dev._ck(dev._lib.kg_synchronize(dev.handle))
    got = base.cpu().numpy().view(np.complex128).reshape(want.shape)
    assert np.array_equal(got, want)
    rough = want * (1.5 - 0.25j)
    base.copy_(torch.from_numpy(np.ascontiguousarray(rough).view(np.float64).reshape(-1)))
    torch.cuda.synchronize()
    dev._ck(dev._lib.kg_set_state_device(dev.handle, which, ptr))
    assert np.array_equal(dev._get(which), rough)
