"""The nonlocal projection and apply over state counts at the edges of their lane groups, rows and chunks, in
both forms of the operator, against the oracle: 1e-12 (FP64) and 2e-6 (single precision), the bounds of the
parity tests."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nl_bulk", [0, 1, -1])
@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 2e-6)])
@pytest.mark.parametrize("nst", [1, 3, 8, 9, 17, 33, 64, 65, 129, 257, 513])
def test_operator_with_projectors(nst, precision, tol, nl_bulk):
    import inq_b200 as ib
    rng = np.random.default_rng(nst)
    # an odd number of points with an odd count in one grid, an even one in the other
    sizes = (15, 15, 15) if nst in (3, 65) else (16, 18, 14)
    lat = np.diag([6.0, 6.5, 6.2])
    pos = np.array([[1.0, 1.2, 0.4], [2.1, 1.5, 1.0], [5.8, 6.1, 3.0]])
    kb = rng.uniform(-1.0, 1.0, (3, 4, 4))
    kb = kb + np.swapaxes(kb, 1, 2)
    V = rng.standard_normal(sizes)
    A, kp = np.array([0.02, 0.0, -0.01]), (0.1, 0.0, 0.2)
    cell = O.Cell(lat)
    rs = O.RealSpace(cell, sizes)
    pa = O.ProjectorAll.pack([O.build_projector(rs, R, 2.0, 2.0, kb[a]) for a, R in enumerate(pos)])
    oh = O.Hamiltonian(rs, V, pa, A)
    basis = ib.RealSpace(ib.Cell(lat), sizes=sizes)
    ham = ib.KSHamiltonian(basis)
    ham.set_scalar_potential(V)
    ham.update_projectors_gaussian(pos, 2.0, 2.0, kb)
    ham.uniform_vector_potential = A
    ham.set_option("nl_bulk", nl_bulk)
    prec = ib.F64 if precision == "f64" else ib.F32
    x = rng.standard_normal(sizes + (nst,)) + 1j * rng.standard_normal(sizes + (nst,))
    rel = lambda a, b: float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))  # noqa: E731
    phi = ib.OrbitalSet.from_array(basis, x, kpoint=kp, precision=prec)
    assert rel(ham(phi).hypercubic(), oh.apply_real(phi.hypercubic().astype(complex), kp)) < tol
    f = ib.OrbitalSet.from_array(basis, x, kpoint=kp, space=ib.FOURIER_SPACE, precision=prec)
    assert rel(ham(f).hypercubic(), oh.apply_fourier(f.hypercubic().astype(complex), kp)) < tol
    ham.ctx.synchronize()
