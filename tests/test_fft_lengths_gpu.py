"""FFT passes of every specialised line length, and of the state counts at the edges of their tiles: few
states, odd and ragged counts, chunks of z-lines that end short, sets that fall back to the generic kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [16, 18, 20, 21, 24, 25, 27, 28, 30, 32, 35, 36, 40, 42, 45, 48, 49, 50, 54, 56, 60, 63, 64, 70, 72, 75, 80,
           81, 84, 90, 96, 98, 100, 105, 108, 112, 120, 126, 128]
TRIPLES = [tuple(LENGTHS[i::13]) for i in range(13)]


def _rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


# H|psi> against the generic kernel (another factorisation of every line) of the same set: six transforms
# of log2(N) <= 21 rounding steps in all, about sqrt(6 * 21) * 1.1e-16 = 1.2e-15 times the largest kinetic
# energy over the mean one (under 10 here); single precision alike with 6e-8, times 4 for both sides
@pytest.mark.parametrize("precision,tol", [("f64", 2e-14), ("f32", 2e-5)])
@pytest.mark.parametrize("sizes", TRIPLES)
def test_operator_matches_generic_kernel(sizes, precision, tol):
    import inq_b200 as ib
    rng = np.random.default_rng(sum(sizes))
    n = [sizes[k] for k in rng.permutation(3)]
    prec = ib.F64 if precision == "f64" else ib.F32
    basis = ib.RealSpace(ib.Cell.orthorhombic(*[0.3 * x for x in n]), sizes=n)
    ham = ib.KSHamiltonian(basis)
    ham.set_scalar_potential(rng.standard_normal(n))
    ham.uniform_vector_potential = [0.02, 0.0, -0.01]
    for nst in (1, 5, 18):
        x = rng.standard_normal((basis.size(), nst)) + 1j * rng.standard_normal((basis.size(), nst))
        for space in (ib.REAL_SPACE, ib.FOURIER_SPACE):
            phi = ib.OrbitalSet.from_array(basis, x, kpoint=(0.1, 0.0, 0.2), space=space, precision=prec)
            got = ham(phi).matrix()
            ham.set_option("fft_impl", 1)
            ref = ham(phi).matrix()
            ham.set_option("fft_impl", -1)
            assert _rel(got, ref) < tol, (n, nst, space)


# transforms against numpy: forward one third of the above and no energies, so 1e-14 / 2e-6 are wide
@pytest.mark.parametrize("precision,tol", [("f64", 1e-14), ("f32", 2e-6)])
@pytest.mark.parametrize("sizes,nst", [((16, 18, 20), 1), ((20, 21, 45), 16), ((21, 25, 27), 3), ((18, 16, 27), 3),
                                       ((24, 24, 24), 9), ((24, 20, 63), 33), ((16, 20, 105), 63), ((30, 16, 126), 31),
                                       ((16, 16, 128), 97), ((20, 18, 50), 200)])
def test_transforms_against_numpy(sizes, nst, precision, tol):
    import inq_b200 as ib
    rng = np.random.default_rng(nst)
    prec = ib.F64 if precision == "f64" else ib.F32
    basis = ib.RealSpace(ib.Cell.orthorhombic(*[0.3 * x for x in sizes]), sizes=sizes)
    x = rng.standard_normal(tuple(sizes) + (nst,)) + 1j * rng.standard_normal(tuple(sizes) + (nst,))
    phi = ib.OrbitalSet.from_array(basis, x, precision=prec)
    f = ib.to_fourier(phi)
    assert _rel(f.hypercubic(), np.fft.fftn(phi.hypercubic().astype(complex), axes=(0, 1, 2))) < tol
    assert _rel(ib.to_real(f).hypercubic(), phi.hypercubic()) < 2 * tol
    assert _rel(ib.to_real(f, normalize=False).hypercubic() / basis.size(), phi.hypercubic()) < 2 * tol


# x passes over flattened columns with state counts around the tile widths (16 double, 32 single): a column's factors
# are those of its own line, whether a tile's columns lie on one line, on two or on many; the bounds are those above
@pytest.mark.parametrize("precision,tol", [("f64", 2e-14), ("f32", 2e-5)])
@pytest.mark.parametrize("nst", [2, 15, 16, 17, 31, 32, 33, 47, 62])
def test_kinetic_factors_around_tile_widths(nst, precision, tol):
    import inq_b200 as ib
    rng = np.random.default_rng(nst)
    n = (24, 9, 10)
    prec = ib.F64 if precision == "f64" else ib.F32
    basis = ib.RealSpace(ib.Cell.orthorhombic(*[0.3 * x for x in n]), sizes=n)
    ham = ib.KSHamiltonian(basis)
    ham.set_scalar_potential(rng.standard_normal(n))
    x = rng.standard_normal((basis.size(), nst)) + 1j * rng.standard_normal((basis.size(), nst))
    for space in (ib.REAL_SPACE, ib.FOURIER_SPACE):
        phi = ib.OrbitalSet.from_array(basis, x, kpoint=(0.1, 0.0, 0.2), space=space, precision=prec)
        got = ham(phi).matrix()
        ham.set_option("fft_impl", 1)
        ref = ham(phi).matrix()
        ham.set_option("fft_impl", -1)
        assert _rel(got, ref) < tol
        # every state by itself: bounds on the whole set could hide one column's factors
        assert (np.linalg.norm(got - ref, axis=0) < 2 * tol * np.linalg.norm(ref, axis=0)).all()


# single-precision sets beyond L2 (128 MB) whose final pass keeps line tiles while the other z passes take whole lines:
# the operator and its Horner step, with either arithmetic of the final pass, against the generic kernel
@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("sizes,nst", [((48, 64, 96), 62), ((40, 72, 72), 90), ((64, 96, 48), 58)])
def test_final_tiles_of_large_single_sets(sizes, nst, mode):
    import inq_b200 as ib
    rng = np.random.default_rng(nst)
    basis = ib.RealSpace(ib.Cell.orthorhombic(*[0.3 * x for x in sizes]), sizes=sizes)
    assert basis.size() * nst * 8 > 128 << 20
    ham = ib.KSHamiltonian(basis)
    ham.set_scalar_potential(rng.standard_normal(sizes))
    x = rng.standard_normal((basis.size(), nst), dtype=np.float32) + 1j * rng.standard_normal((basis.size(), nst), dtype=np.float32)
    phi = ib.OrbitalSet.from_array(basis, x, kpoint=(0.1, 0.0, 0.2), precision=ib.F32)
    basis.ctx.set_option("mixed_compute", mode)
    try:
        got = ham(phi).matrix(), ib.exponential(ham, -0.002j, phi).matrix()
        ham.set_option("fft_impl", 1)
        ref = ham(phi).matrix(), ib.exponential(ham, -0.002j, phi).matrix()
    finally:
        basis.ctx.set_option("mixed_compute", 0)
    for a, b in zip(got, ref):
        assert _rel(a, b) < 2e-5
