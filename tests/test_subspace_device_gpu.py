"""Cholesky, triangular inverse, Jacobi rotations and per-state sums on the device, at state counts around the
edges of their tiles, lane groups and clusters, against numpy and the host routines."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.2e-16


def _set(nst, sizes=(12, 10, 9), seed=0, precision=None):
    import inq_b200 as ib
    rng = np.random.default_rng(seed + nst)
    basis = ib.RealSpace(ib.Cell.orthorhombic(*[0.5 * n for n in sizes]), sizes=sizes)
    x = rng.standard_normal((basis.size(), nst)) + 1j * rng.standard_normal((basis.size(), nst))
    return basis, rng, x, ib.OrbitalSet.from_array(basis, x, precision=ib.F64 if precision is None else precision)


# phi U^-1 against numpy's factor: the overlaps of random sets have condition numbers below 1e3 here (fewer
# states than half the points), which with sums of 1080 terms leaves about 1e3 * 30 * EPS
@pytest.mark.parametrize("nst", [1, 2, 31, 32, 33, 64, 65, 100, 129, 200, 257, 400])
def test_orthogonalize(nst):
    import inq_b200 as ib
    basis, _, x, phi = _set(nst)
    dv = basis.volume_element()
    ref = x @ np.linalg.inv(np.linalg.cholesky(dv * (x.conj().T @ x)).conj().T)
    ib.orthogonalize(phi)
    got = phi.matrix()
    assert np.linalg.norm(got - ref) < 1e-11 * np.linalg.norm(ref)
    S = dv * (got.conj().T @ got)
    assert np.abs(S - np.eye(nst)).max() < 1e-12


@pytest.mark.parametrize("nst", [5, 33, 64, 65])
def test_orthogonalize_single(nst):
    import inq_b200 as ib
    basis, _, x, phi = _set(nst, precision=ib.F32)
    ib.orthogonalize(phi)
    got = phi.matrix().astype(complex)
    S = basis.volume_element() * (got.conj().T @ got)
    assert np.abs(S - np.eye(nst)).max() < 1e-5  # split-BF16 overlaps: 1e-6 per element times the condition number


@pytest.mark.parametrize("nst", [3, 40])
def test_orthogonalize_refuses_dependent_states(nst):
    import inq_b200 as ib
    _, _, x, _ = _set(nst)
    x[:, nst - 1] = 0.0
    basis, _, _, phi = _set(nst)
    phi.upload(x)
    with pytest.raises(ib.InqbError, match="not positive definite"):
        ib.orthogonalize(phi)
    assert np.array_equal(phi.matrix(), x)


# the failing pivot in the first, a middle and the last tile row, at its first and last row, with up to 12 CTAs per
# launch and as many launches after the failing one; the context's next call is not affected
@pytest.mark.parametrize("nst,row", [(400, 0), (400, 31), (400, 32), (129, 63), (129, 100), (129, 127), (129, 128)])
def test_orthogonalize_refuses_at_any_row(nst, row):
    import inq_b200 as ib
    basis, _, x, phi = _set(nst)
    x[:, row] = 0.0
    phi.upload(x)
    for _ in range(3):
        with pytest.raises(ib.InqbError, match="not positive definite"):
            ib.orthogonalize(phi)
    assert np.array_equal(phi.matrix(), x)
    _, _, y, good = _set(65)
    ib.orthogonalize(good)
    got = good.matrix()
    assert np.abs(basis.volume_element() * (got.conj().T @ got) - np.eye(65)).max() < 1e-12


# The device's waves are the host routine's rotations in another order of independent ones: eigenvalues agree
# to rounding, eigenvectors to rounding over the smallest gap, each up to a phase.  The phase of a vector is
# that of the off-diagonal element r of its last rotation by about pi / 2 (which swaps two columns), known to
# EPS * norm / r: dense random matrices still swap columns at r = 1e-10 norm and below, so for them the phases
# hold to 1e-3 only (5e-6 seen at 130 states; the host routine moves as much when a last bit of H changes).
@pytest.mark.parametrize("nst", [1, 2, 13, 14, 15, 64, 97, 130])
def test_subspace_diagonalization_matches_host_rotations(nst):
    import inq_b200 as ib
    basis, rng, x, phi = _set(nst)
    ham = ib.KSHamiltonian(basis)
    ham.set_scalar_potential(rng.standard_normal(basis.sizes))
    ib.orthogonalize(phi)
    H = ib.overlap(phi, ham(phi))
    w, V = ib.hermitian_eigen(H)
    ref = phi.matrix() @ V
    eig = ham.subspace_diagonalization(phi)
    got = phi.matrix()
    norm = np.abs(w).max()
    assert np.all(np.diff(eig) >= 0.0)
    assert np.abs(eig - w).max() < 100 * EPS * norm * max(1, nst) ** 0.5
    gap = np.diff(w).min() if nst > 1 else norm
    z = (ref.conj() * got).sum(0) / (np.abs(ref) ** 2).sum(0)
    assert np.linalg.norm(got - ref * (z / np.abs(z))) < (1e-12 + 200 * EPS * norm / gap) * np.linalg.norm(ref)
    assert np.abs(z - 1.0).max() < 1e-3


# sums of npoints products in double (double of single-precision values): 1e-13 of the norms is 100 roundings
@pytest.mark.parametrize("nst", [1, 7, 8, 9, 33, 128, 200, 256, 257, 300])
@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_state_sums(nst, precision):
    import inq_b200 as ib
    prec = ib.F64 if precision == "f64" else ib.F32
    basis, rng, x, phi = _set(nst, sizes=(9, 7, 5), precision=prec)
    a = phi.matrix().astype(complex)
    b_set = ib.OrbitalSet.from_array(basis, x[::-1].copy(), precision=prec)
    b = b_set.matrix().astype(complex)
    dv = basis.volume_element()
    scale = dv * np.sqrt((np.abs(a) ** 2).sum(0) * (np.abs(b) ** 2).sum(0))
    assert np.all(np.abs(ib.overlap_diagonal(phi, b_set) - dv * (a.conj() * b).sum(0)) < 1e-13 * scale)
    ham = ib.KSHamiltonian(basis)
    ham.set_scalar_potential(rng.standard_normal(basis.sizes))
    h = ham(phi).matrix().astype(complex)
    n2 = (np.abs(a) ** 2).sum(0)
    e = (a.conj() * h).real.sum(0) / n2
    eig, res = ham.eigenvalues(phi)
    assert np.all(np.abs(eig - e) < 1e-12 * np.abs(h).max())
    assert np.allclose(res, dv * (np.abs(h - e * a) ** 2).sum(0), rtol=1e-11)
    occ = rng.uniform(0.0, 2.0, nst)
    dens = ib.density([phi, b_set], [occ, occ])
    assert np.allclose(dens, (np.abs(a) ** 2) @ occ + (np.abs(b) ** 2) @ occ, rtol=1e-13)


# a grid of more than 2^31 points: the coordinates of the last ones need 64-bit indices.  One plane wave e^{iG.r} with
# G = -(1, 2, 3) 2 pi / L; its kinetic energy is one term, so only the rounding of that term is left
def test_kinetic_energy_beyond_32_bit_points():
    import torch

    import inq_b200 as ib
    n = (1296, 1296, 1280)
    assert n[0] * n[1] * n[2] > 2 ** 31
    length = [0.3 * k for k in n]
    basis = ib.RealSpace(ib.Cell.orthorhombic(*length), sizes=n)
    data = torch.zeros(n + (1,), dtype=torch.complex64, device="cuda")
    data[n[0] - 1, n[1] - 2, n[2] - 3, 0] = 2.0
    torch.cuda.synchronize()
    phi = ib.OrbitalSet.from_tensor(basis, data, space=ib.FOURIER_SPACE)
    ham = ib.KSHamiltonian(basis)
    got = ham.kinetic_expectation_value(phi)
    g2 = sum((m * 2.0 * np.pi / l) ** 2 for m, l in zip((1, 2, 3), length))
    want = 0.5 * g2 * 4.0 * np.prod(length) / float(basis.size()) ** 2
    del ham, phi, data
    torch.cuda.empty_cache()
    assert abs(got[0] - want) < 1e-12 * want


# few states: the host forms the factor, and the device runs the overlap's two kernels and one rotation (the chain of
# tiles would add at least three more launches and take longer); more states on either side of the change
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("nst", [1, 2, 16, 49, 50, 51, 52])
def test_orthogonalize_of_few_states(nst, precision):
    import inq_b200 as ib
    basis, _, x, phi = _set(nst, precision=ib.F64 if precision == "f64" else ib.F32)
    x = phi.matrix().astype(complex)
    dv = basis.volume_element()
    ref = x @ np.linalg.inv(np.linalg.cholesky(dv * (x.conj().T @ x)).conj().T)
    before = basis.ctx.launch_count()
    ib.orthogonalize(phi)
    launches = basis.ctx.launch_count() - before
    assert launches <= 3 if nst <= 50 else launches > 3
    assert np.linalg.norm(phi.matrix() - ref) < (1e-11 if precision == "f64" else 1e-5) * np.linalg.norm(ref)


# more rows of 64 points than CTAs are resident (444 or 592 on a B200) and several tiles of states: the triangular
# rotation works in place, each CTA on its own points
@pytest.mark.parametrize("precision,nst,tol", [("f64", 200, 1e-12), ("f32", 200, 2e-5), ("f32", 131, 2e-5)])
def test_orthogonalize_many_points(nst, precision, tol):
    import inq_b200 as ib
    basis, _, x, phi = _set(nst, sizes=(40, 40, 42), precision=ib.F64 if precision == "f64" else ib.F32)
    dv = basis.volume_element()
    x = phi.matrix().astype(complex)
    ref = x @ np.linalg.inv(np.linalg.cholesky(dv * (x.conj().T @ x)).conj().T)
    ib.orthogonalize(phi)
    assert np.linalg.norm(phi.matrix() - ref) < tol * np.linalg.norm(ref)


# the SIMT products: the full rotation, once the host knows that there is a factor
@pytest.mark.parametrize("precision,nst,tol", [("f64", 33, 1e-11), ("f64", 100, 1e-11), ("f32", 33, 1e-5), ("f32", 64, 1e-5)])
def test_orthogonalize_without_fp64_tensor_cores(precision, nst, tol):
    import inq_b200 as ib
    basis, _, x, phi = _set(nst, precision=ib.F64 if precision == "f64" else ib.F32)
    dv = basis.volume_element()
    x = phi.matrix().astype(complex)
    ref = x @ np.linalg.inv(np.linalg.cholesky(dv * (x.conj().T @ x)).conj().T)
    basis.ctx.set_option("fp64_mma", 0)
    try:
        ib.orthogonalize(phi)
        assert np.linalg.norm(phi.matrix() - ref) < tol * np.linalg.norm(ref)
        x[:, nst // 2] = 0.0
        phi.upload(x)
        held = phi.matrix()
        with pytest.raises(ib.InqbError, match="not positive definite"):
            ib.orthogonalize(phi)
        assert np.array_equal(phi.matrix(), held)
    finally:
        basis.ctx.set_option("fp64_mma", 1)


# more than 1024 states: several rounds of a block's threads over a wave's rotations, whose table is larger than the
# 48 KB a kernel may have without asking.  Against numpy: eigenvalues, orthonormal states, a diagonal matrix
def test_subspace_diagonalization_of_many_states():
    import inq_b200 as ib
    nst = 1030
    basis, rng, x, phi = _set(nst, sizes=(12, 10, 12))
    ham = ib.KSHamiltonian(basis)
    ham.set_scalar_potential(rng.standard_normal(basis.sizes))
    ib.orthogonalize(phi)
    w = np.linalg.eigvalsh(ib.overlap(phi, ham(phi)))
    eig = ham.subspace_diagonalization(phi)
    norm = np.abs(w).max()
    assert np.abs(eig - w).max() < 100 * EPS * norm * nst ** 0.5
    H = ib.overlap(phi, ham(phi))
    assert np.linalg.norm(H - np.diag(eig)) < 1e-12 * np.linalg.norm(H)
    assert np.abs(ib.overlap(phi) - np.eye(nst)).max() < 1e-11


# norms (a set with itself, its own sum) against the same set under another address and numpy: all terms are positive,
# so 1e-14 is about 50 roundings of sums that add in groups
@pytest.mark.parametrize("nst", [1, 8, 9, 40, 256, 300, 600])
@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_norms_of_a_set(nst, precision):
    import inq_b200 as ib
    basis, _, _, phi = _set(nst, sizes=(9, 7, 5), precision=ib.F64 if precision == "f64" else ib.F32)
    n = ib.overlap_diagonal(phi)
    want = basis.volume_element() * (np.abs(phi.matrix().astype(complex)) ** 2).sum(0)
    assert np.all(n.imag == 0.0)
    assert np.allclose(n.real, want, rtol=1e-14, atol=0.0)
    assert np.allclose(ib.overlap_diagonal(phi, phi.copy()).real, n.real, rtol=1e-14, atol=0.0)
