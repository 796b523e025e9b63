"""Options that choose kernel forms: what each asks for is what runs, and no depth or form changes a result or refuses
a set that the other forms take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(nst, natoms, sizes=(20, 20, 20), precision="f64"):
    import inq_b200 as ib
    rng = np.random.default_rng(nst + natoms)
    basis = ib.RealSpace(ib.Cell.orthorhombic(*[0.4 * n for n in sizes]), sizes=sizes)
    ham = ib.KSHamiltonian(basis)
    ham.set_scalar_potential(rng.standard_normal(sizes))
    kb = rng.uniform(-1.0, 1.0, (natoms, 4, 4))
    ham.update_projectors_gaussian(rng.uniform(0.0, 8.0, (natoms, 3)), 2.0, 2.0, kb + np.swapaxes(kb, 1, 2))
    x = rng.standard_normal((basis.size(), nst)) + 1j * rng.standard_normal((basis.size(), nst))
    prec = ib.F64 if precision == "f64" else ib.F32
    return ib, basis, ham, ib.OrbitalSet.from_array(basis, x, kpoint=(0.1, 0.0, 0.2), precision=prec)


# The bulk-copy projection is chosen by its CTAs, projectors x ranges x chunks of 256 states, against two per SM
# (296 on a B200).  The forms add a sphere's points in other groups, so their results tell them apart.
@pytest.mark.parametrize("natoms,ranges,bulk", [(10, 1, False), (10, 16, False), (10, 30, True), (20, 0, True),
                                                (9, 0, False), (40, 1, False), (40, 8, True)])
def test_projection_form_follows_the_ranges_asked_for(natoms, ranges, bulk):
    ib, basis, ham, phi = _system(64, natoms)
    ctx = basis.ctx
    ctx.set_option("nl_project_ranges", ranges)
    try:
        out = {}
        for form in (0, 1, -1):
            ctx.set_option("nl_bulk", form)
            out[form] = ham.non_local(phi).matrix()
    finally:
        ctx.set_option("nl_bulk", 0)
        ctx.set_option("nl_project_ranges", 0)
    assert not np.array_equal(out[1], out[-1])
    assert np.array_equal(out[0], out[1 if bulk else -1])


# ring depths deeper than shared memory holds: line lengths and state counts that only the generic kernel took before
# their specialised passes still take every depth, and a depth changes no result
@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("sizes,nst", [((16, 80, 20), 64), ((100, 20, 16), 64), ((20, 16, 80), 30), ((24, 20, 96), 9),
                                       ((128, 16, 16), 3)])
def test_every_ring_depth_is_taken(sizes, nst, precision):
    ib, basis, ham, phi = _system(nst, 2, sizes, precision)
    ctx = basis.ctx
    run = lambda: (ham(phi).matrix(), ib.to_real(ib.to_fourier(phi)).matrix())  # noqa: E731
    ref = run()
    try:
        for depth in (1, 2, 3, 5, 8):
            ctx.set_option("fft_stages", depth)
            for got, want in zip(run(), ref):
                assert np.array_equal(got, want), depth
    finally:
        ctx.set_option("fft_stages", 0)


# the nine lengths with at least a 256-byte row of states refuse a ring that does not fit, as the option always did
def test_too_deep_ring_is_refused_for_whole_rows():
    ib, basis, ham, phi = _system(64, 1, (16, 96, 16), "f32")
    ctx = basis.ctx
    ctx.set_option("fft_stages", 8)
    try:
        with pytest.raises(ib.InqbError, match="does not fit"):
            ham(phi)
    finally:
        ctx.set_option("fft_stages", 0)
    ham(phi).matrix()


# V + |k|^2 / 2 of the Fourier form at the sphere points, where the nonlocal apply forms it, in the passes' double
# arithmetic (whole 16-byte rows of at least 256 bytes): V = 1 and a shift of 5e-8 that single precision would drop
# (an ulp of 1 is 1.2e-7).  The rounding of the stored sets is random, 1e-7 in each of 24^3 * 34 values, 1e-10 in
# their mean; with the sphere on about half the points (radius 36 in a 72 bohr cell) a dropped shift leaves 2.5e-8.
@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("nst", [34, 64])
def test_fourier_form_keeps_double_arithmetic_at_sphere_points(nst, mode):
    import inq_b200 as ib
    rng = np.random.default_rng(nst)
    n, length = 24, 72.0
    basis = ib.RealSpace(ib.Cell.cubic(length), sizes=(n, n, n))
    ham = ib.KSHamiltonian(basis)
    ham.set_scalar_potential(np.ones((n, n, n)))
    ham.update_projectors_gaussian(np.array([[36.0, 36.0, 36.0]]), 36.0, 2.0, np.zeros((1, 4, 4)))
    k = np.sqrt(2.0 * 5e-8)
    x = rng.standard_normal((n, n, n, nst)) + 1j * rng.standard_normal((n, n, n, nst))
    f = ib.OrbitalSet.from_array(basis, x, kpoint=(k * length, 0.0, 0.0), space=ib.FOURIER_SPACE, precision=ib.F32)
    basis.ctx.set_option("mixed_compute", mode)
    try:
        got = ham(f).hypercubic().astype(complex)
    finally:
        basis.ctx.set_option("mixed_compute", 0)
    x = f.hypercubic().astype(complex)
    g = 2.0 * np.pi / length * np.fft.fftfreq(n, 1.0 / n)
    kin = 0.5 * (g[:, None, None] ** 2 + g[None, :, None] ** 2 + g[None, None, :] ** 2) + g[:, None, None] * k
    want = (kin + 1.0 + float(np.float32(0.5 * k * k)))[..., None] * x
    assert abs((x.conj() * (got - want)).sum().real) < 5e-9 * (np.abs(x) ** 2).sum()


# double-precision arithmetic over single-precision sets with fewer states than a 256-byte row, whose flattened
# tiles lie on several lines: against the generic kernel (single-precision arithmetic; 2e-6 for both, as the parity
# tests take)
@pytest.mark.parametrize("mode", [1, 2, 3])
@pytest.mark.parametrize("sizes,nst", [((24, 24, 24), 1), ((32, 24, 40), 2), ((48, 24, 32), 9), ((24, 40, 64), 16),
                                       ((24, 72, 24), 31)])
def test_wide_arithmetic_of_few_states(sizes, nst, mode):
    ib, basis, ham, phi = _system(nst, 3, sizes, "f32")
    ctx = basis.ctx
    f = ib.to_fourier(phi)
    ctx.set_option("mixed_compute", mode)
    try:
        for s in (phi, f):
            got = ham(s).matrix()
            ham.set_option("fft_impl", 1)
            ref = ham(s).matrix()
            ham.set_option("fft_impl", -1)
            assert np.linalg.norm(got - ref) < 2e-6 * np.linalg.norm(ref)
    finally:
        ctx.set_option("mixed_compute", 0)
