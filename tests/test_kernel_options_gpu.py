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
