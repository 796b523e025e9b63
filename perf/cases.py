"""The work a user of inq_b200 has it do, as cases that can be prepared, run, checked and timed.

Every case goes through the package's public Python interface.  Orbitals, results and operators live on the
device as they do in a program that propagates or minimises: the sets wrap torch storage (the zero-copy form
of the boundary), the Hamiltonian keeps its potential and projector tables, and only what a program reads on
the host (overlap matrices, eigenvalues, dipoles) crosses to it.

Operations:
  apply         H|psi> of a real-space set (ks_hamiltonian::operator())
  fourier       H|psi> of a Fourier-space set, the form the eigensolver uses
  etrs          one real-time step: orbitals, density and dipole; fixed or interacting (Hartree + LDA)
  overlap       <psi_i|H psi_j>, the subspace matrix, of two sets
  orthogonalize Cholesky orthonormalisation of a set
  ground        one ground-state iteration: steepest descent, transform, subspace diagonalisation, density
"""

import math

import numpy as np
import torch

import inq_b200 as ib
from inq_b200 import core

SPACING = 0.21375      # bohr; the grid of the 96^3 / 20.52 bohr system
RADIUS = 2.0           # bohr, projector spheres
RC = 2.0               # bohr, radial Gaussian of the projectors
ECUT = 25.0            # Ha, of the random orbitals
KPOINT = (0.1, 0.0, 0.2)
VECTOR_POTENTIAL = (0.02, 0.0, -0.01)

REAL = {"f64": torch.complex128, "f32": torch.complex64}
SIZE = {"f64": 16, "f32": 8}


def _case(name, op, n, nst, precision, atoms, kpoint=False, interacting=False):
    nx, ny, nz = n
    c = {"op": op, "nx": nx, "ny": ny, "nz": nz, "nst": nst, "precision": precision, "atoms": atoms,
         "kpoint": kpoint, "interacting": interacting}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a few orbitals of a small molecule: the smallest call, where launches and latency count
        _case("apply_molecule_f32", "apply", (24, 24, 24), 9, "f32", 2),
        # the 8-atom unit cell with a k-point and a vector potential, plain double precision
        _case("apply_unit_cell_f64", "apply", (32, 32, 32), 16, "f64", 8, kpoint=True),
        # an orthorhombic cell whose grid follows from its spacing (products of 2, 3, 5 and 7)
        _case("apply_spacing_grid_f64", "apply", (54, 60, 45), 50, "f64", 12),
        # an odd number of orbitals on the largest grid of the batched workload
        _case("apply_odd_states_f32", "apply", (72, 72, 72), 99, "f32", 32),
        # the headline system: 96^3, 256 orbitals, 64 atoms, mixed precision
        _case("apply_large_f32", "apply", (96, 96, 96), 256, "f32", 64),
        # the real-time grid in plain double precision, a slice of its orbitals
        _case("apply_large_f64", "apply", (120, 120, 120), 64, "f64", 128),
        # the operator as the eigensolver calls it
        _case("fourier_f64", "fourier", (48, 48, 48), 40, "f64", 8),
        # one real-time step, fixed Hamiltonian, mixed precision
        _case("etrs_f32", "etrs", (72, 72, 72), 128, "f32", 32),
        # one real-time step with the potential rebuilt from every density, double precision, ragged count
        _case("etrs_interacting_f64", "etrs", (40, 40, 40), 33, "f64", 8, interacting=True),
        # subspace matrix of a mixed-precision set on the tensor cores
        _case("overlap_f32", "overlap", (80, 80, 80), 200, "f32", 0),
        # orthonormalisation, double precision
        _case("orthogonalize_f64", "orthogonalize", (64, 64, 64), 128, "f64", 0),
        # one iteration of the ground-state loop
        _case("ground_f64", "ground", (50, 50, 50), 64, "f64", 8),
    ]


def _smooth(lo, hi):
    def ok(n):
        for f in (2, 3, 5, 7):
            while n % f == 0:
                n //= f
        return n == 1
    return [n for n in range(lo, hi + 1) if ok(n)]


GRIDS = _smooth(20, 100)
# the largest share of the headline system's orbital bytes that a drawn case of an operation may have
LIMIT = {"apply": 1.0, "fourier": 0.5, "etrs": 0.15, "overlap": 0.5, "orthogonalize": 0.25, "ground": 0.06}


def draw(rng):
    op = rng.choice(["apply", "apply", "apply", "apply", "fourier", "etrs", "etrs", "overlap", "orthogonalize", "ground"])
    precision = rng.choice(["f32", "f64"])
    if op == "ground":
        precision = "f64"
    top = LIMIT[op] * 96 ** 3 * 256 * 8
    while True:
        base = 20.0 * (100.0 / 20.0) ** rng.random()
        near = [g for g in GRIDS if 0.8 * base <= g <= 1.25 * base]
        n = [rng.choice(near) for _ in range(3)]
        if rng.random() < 0.4:
            n = [n[0]] * 3  # cubic cells are common
        nst = int(round(4.0 * (256.0 / 4.0) ** rng.random()))
        nst = min(nst, 96) if op == "ground" else nst
        if n[0] * n[1] * n[2] * nst * SIZE[precision] <= top:
            break
    volume = n[0] * n[1] * n[2] * SPACING ** 3
    atoms = 0 if op in ("overlap", "orthogonalize") else max(1, min(128, int(round(volume / 135.0 * (0.5 + rng.random())))))
    return _case(None, op, n, nst, precision, atoms, kpoint=op in ("apply", "fourier", "etrs") and rng.random() < 0.3,
                 interacting=op == "etrs" and rng.random() < 0.5)


# ------------------------------------------------------------------ inputs, made with torch from the seed


def _sizes(case):
    return (case["nx"], case["ny"], case["nz"])


def _lengths(case):
    return [n * SPACING for n in _sizes(case)]


def _gen(seed, stream):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 8 + stream)


def _gvectors(case):
    """2 pi m / L along each axis, broadcastable over [nx, ny, nz]."""
    out = []
    for k, (n, l) in enumerate(zip(_sizes(case), _lengths(case))):
        g = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda") * (2.0 * math.pi / l)
        out.append(g.reshape([n if j == k else 1 for j in range(3)]))
    return out


def _g2(case, k=(0.0, 0.0, 0.0)):
    g = _gvectors(case)
    return sum((gi + ki) ** 2 for gi, ki in zip(g, k))


def _points(case):
    """Fractional coordinates of the grid points along each axis."""
    return [torch.arange(n, dtype=torch.float64, device="cuda") / n for n in _sizes(case)]


def _orbitals(case, seed, orthonormal=True):
    """Normal G-coefficients with |G|^2 / 2 < ECUT, in real space [nx, ny, nz, nst], complex128."""
    n = _sizes(case)
    c = torch.randn(n + (case["nst"],), dtype=torch.complex128, device="cuda", generator=_gen(seed, 1))
    c *= (0.5 * _g2(case) < ECUT)[..., None]
    for axis in range(3):
        c = torch.fft.ifft(c, dim=axis)
    dv = SPACING ** 3
    if orthonormal:
        m = c.reshape(-1, case["nst"])
        u = torch.linalg.cholesky(dv * (m.conj().T @ m)).mH
        c = torch.linalg.solve_triangular(u, m, upper=True, left=False).reshape(c.shape)
    else:
        c /= torch.sqrt(dv * torch.sum(c.abs() ** 2, dim=(0, 1, 2)))
    return c


def _atoms(case, seed):
    """Positions on a jittered lattice filling the cell (fractional), and symmetric KB matrices."""
    m = case["atoms"]
    side = 1
    while side ** 3 < m:
        side += 1
    i = torch.arange(m, device="cuda")
    f = torch.stack([i // (side * side), (i // side) % side, i % side], dim=1).double() / side
    f = f + torch.randn((m, 3), dtype=torch.float64, device="cuda", generator=_gen(seed, 2)) * 0.02 / side
    kb = 2.0 * torch.rand((m, 4, 4), dtype=torch.float64, device="cuda", generator=_gen(seed, 3)) - 1.0
    return torch.remainder(f, 1.0), torch.triu(kb) + torch.triu(kb, 1).mT


def _offsets(case, frac):
    """Per axis the minimum-image fractional offset of every grid point from an atom."""
    out = []
    for k, x in enumerate(_points(case)):
        d = x - frac[k]
        d = d - torch.round(d)
        out.append(d.reshape([len(x) if j == k else 1 for j in range(3)]))
    return out


def _potential(case, frac):
    """Wells of depth 2 Ha and width 1 bohr at the atoms."""
    v = torch.zeros(_sizes(case), dtype=torch.float64, device="cuda")
    for f in frac:
        v -= 2.0 * torch.exp(-sum((d * l) ** 2 for d, l in zip(_offsets(case, f), _lengths(case))))
    return v


def _projectors(case, frac, kb):
    """Kleinman-Bylander tables of one s and three p functions per atom: flat points, float32 fractional
    offsets and values, padded to the largest sphere."""
    n, length = _sizes(case), _lengths(case)
    pts, offs, vals = [], [], []
    for f in frac:
        d = _offsets(case, f)
        r2 = sum((x * l) ** 2 for x, l in zip(d, length))
        p = torch.nonzero((r2 <= RADIUS * RADIUS).reshape(-1)).reshape(-1)
        o = torch.stack([x.expand(n).reshape(-1)[p] for x in d], dim=1)
        x, y, z = (o[:, k] * length[k] for k in range(3))
        r = torch.sqrt(x * x + y * y + z * z)
        safe = torch.where(r > 0.0, r, torch.ones_like(r))
        c0, c1 = 0.5 / math.sqrt(math.pi), math.sqrt(0.75 / math.pi)
        g = torch.exp(-(r / RC) ** 2)
        pts.append(p)
        offs.append(o.float())
        vals.append(torch.stack([c0 * g, c1 * g * y / safe, c1 * g * z / safe, c1 * g * x / safe]))
    most = max(len(p) for p in pts)
    points = torch.full((len(pts), most), -1, dtype=torch.int64, device="cuda")
    offsets = torch.zeros((len(pts), most, 3), dtype=torch.float32, device="cuda")
    values = torch.zeros((len(pts), 4, most), dtype=torch.float64, device="cuda")
    for a, (p, o, m) in enumerate(zip(pts, offs, vals)):
        points[a, :len(p)], offsets[a, :len(p)], values[a, :, :len(p)] = p, o, m
    return {"points": points, "offsets": offsets, "values": values, "kb": kb, "count": [len(p) for p in pts]}


def _occupations(case):
    """Fermi-like occupations, so that every state counts with a weight of its own."""
    s = np.arange(case["nst"])
    return 2.0 / (1.0 + np.exp((s - 0.7 * case["nst"]) / (0.1 * case["nst"])))


def _dt(case):
    """Half the stability bound of the order-4 Taylor propagator on this grid."""
    top = 0.5 * sum((math.pi / SPACING) ** 2 for _ in range(3))
    return 0.5 * 2.0 * math.sqrt(2.0) / top


def _vectors(case):
    """(k, A) as the operator takes them: covariant components."""
    if not case["kpoint"]:
        return (0.0, 0.0, 0.0), (0.0, 0.0, 0.0)
    return KPOINT, VECTOR_POTENTIAL


def _hamiltonian(case, seed, basis):
    frac, kb = _atoms(case, seed)
    ham = core.KSHamiltonian(basis)
    v = _potential(case, frac).cpu().numpy()
    if case["interacting"]:
        ham.set_interaction(v, hartree=True, xc="lda")
    ham.set_scalar_potential(v)
    t = _projectors(case, frac, kb)
    n = _sizes(case)
    p = t["points"]
    grid = torch.stack([p // (n[1] * n[2]), (p // n[2]) % n[1], p % n[2]], dim=2)
    grid[p < 0] = -1
    ham.set_projectors(grid.cpu().numpy(), t["offsets"].cpu().numpy(), t["values"].cpu().numpy(), kb.cpu().numpy(),
                       np.array(t["count"]), np.full(len(t["count"]), 4))
    if case["kpoint"]:
        ham.uniform_vector_potential = VECTOR_POTENTIAL
    return ham


def _fft3(x, inverse=False):
    for axis in range(3):
        x = torch.fft.ifft(x, dim=axis) if inverse else torch.fft.fft(x, dim=axis)
    return x


def prepare(case, seed):
    basis = core.RealSpace(core.Cell.orthorhombic(*_lengths(case)), sizes=_sizes(case))
    op, dtype = case["op"], REAL[case["precision"]]
    k, _ = _vectors(case)
    st = {"op": op, "basis": basis}

    def wrap(t, space=ib.REAL_SPACE):
        return core.OrbitalSet.from_tensor(basis, t, kpoint=k, space=space)

    psi = _orbitals(case, seed, orthonormal=op != "orthogonalize")
    if op in ("overlap", "orthogonalize"):
        st["psi"] = psi.to(dtype).contiguous()
        st["phi"] = wrap(st["psi"])
        if op == "overlap":
            st["chi_data"] = (psi * _mixing(case)[..., None]).to(dtype).contiguous()
            st["chi"] = wrap(st["chi_data"])
        else:
            st["work_data"] = torch.empty_like(st["psi"])
            st["work"] = wrap(st["work_data"])
        torch.cuda.synchronize()
        return st
    st["ham"] = _hamiltonian(case, seed, basis)
    st["occ"] = _occupations(case)
    if op in ("fourier", "ground"):
        psi = _fft3(psi)
    space = ib.FOURIER_SPACE if op in ("fourier", "ground") else ib.REAL_SPACE
    st["psi"] = psi.to(dtype).contiguous()
    st["phi"] = wrap(st["psi"], space)
    if op in ("apply", "fourier"):
        st["out_data"] = torch.empty_like(st["psi"])
        st["out"] = wrap(st["out_data"], space)
    elif op == "etrs":
        st["dt"] = _dt(case)
        st["density"] = torch.empty(basis.size(), dtype=torch.float64, device="cuda")
    else:
        st["work_data"] = torch.empty_like(st["psi"])
        st["work"] = wrap(st["work_data"], ib.FOURIER_SPACE)
        st["rs_data"] = torch.empty_like(st["psi"])
        st["rs"] = wrap(st["rs_data"])
    torch.cuda.synchronize()
    return st


def run(st):
    op = st["op"]
    if op in ("apply", "fourier"):
        st["ham"].apply(st["phi"], st["out"])
        return st["out_data"]
    if op == "etrs":
        # the propagation goes on from where the last step left the orbitals
        dens, dip, _ = core.etrs(st["ham"], [st["phi"]], [st["occ"]], st["dt"], density_out=st["density"])
        return {"orbitals": st["psi"], "density": dens, "dipole": dip}
    if op == "overlap":
        return core.overlap(st["phi"], st["chi"])
    if op == "orthogonalize":
        st["work"].assign(st["phi"])
        core.orthogonalize(st["work"])
        return st["work_data"]
    st["work"].assign(st["phi"])
    st["ham"].steepest_descent(st["work"])
    st["rs"].assign(core.to_real(st["work"]))
    eig = st["ham"].subspace_diagonalization(st["rs"])
    return {"eigenvalues": eig, "orbitals": st["rs_data"], "density": core.density([st["rs"]], [st["occ"]])}


# ------------------------------------------------------------------ what a pass cannot do without


def work(case):
    n, s, c = case["nx"] * case["ny"] * case["nz"], case["nst"], SIZE[case["precision"]]
    sphere = case["atoms"] * 4.0 / 3.0 * math.pi * RADIUS ** 3 / SPACING ** 3
    transform = 5.0 * n * math.log2(n) * s
    h_flops = 2.0 * transform + 10.0 * n * s + 2.0 * sphere * 4 * 8 * s
    h_extra = 8.0 * n + sphere * (4 + 12 + 32)
    op = case["op"]
    if op in ("apply", "fourier"):
        return {"bytes": 2.0 * n * s * c + h_extra, "flops": h_flops}
    if op == "etrs":  # the exponentials of the prediction and of one self-consistency pass, order 4
        return {"bytes": 2.0 * n * s * c + h_extra + 8.0 * n, "flops": 8 * h_flops}
    if op == "overlap":
        return {"bytes": 2.0 * n * s * c + 16.0 * s * s, "flops": 8.0 * n * s * s}
    if op == "orthogonalize":  # half of a Hermitian product and a triangular one
        return {"bytes": 2.0 * n * s * c, "flops": 8.0 * n * s * s}
    # six operators, an orthogonalisation, a transform, the subspace operator, matrix and rotation
    return {"bytes": 2.0 * n * s * c + h_extra + 8.0 * n, "flops": 7 * h_flops + transform + 24.0 * n * s * s}


# About four times the distance from the 64-bit results at these sizes.  The small corrections that a time
# step makes carry less of the single-precision error of H (5.7e-8); a dipole is what remains of large terms
# of both signs.  The eigenvectors of close eigenvalues are fixed by rounding to 1e-16 * |H| / gap.
TOLERANCE = {
    "f32": {"apply": 4e-6, "fourier": 4e-6, "etrs": 4e-7, "overlap": 1e-6, "orthogonalize": 1e-6},
    "f64": {"apply": 1e-14, "fourier": 1e-14, "etrs": 1e-12, "overlap": 1e-14, "orthogonalize": 1e-14, "ground": 1e-10},
}


def tolerance(case):
    return {"rel": TOLERANCE[case["precision"]][case["op"]]}


# ------------------------------------------------------------------ the same in 64 bits with torch


def _mixing(case):
    """A smooth real factor: the second set of an overlap is the first times it."""
    x, y, z = (t.reshape([-1 if j == k else 1 for j in range(3)]) for k, t in enumerate(_points(case)))
    return 1.0 + 0.5 * torch.cos(2.0 * math.pi * x) * torch.sin(2.0 * math.pi * y) + 0.25 * torch.cos(4.0 * math.pi * z)


class _Exact:
    def __init__(self, case, seed):
        self.case = case
        frac, kb = _atoms(case, seed)
        self.vion = _potential(case, frac)
        self.v = self.vion
        self.t = _projectors(case, frac, kb)
        k, a = _vectors(case)
        length = _lengths(case)
        cov = [x + y for x, y in zip(k, a)]
        self.kcart = [x / l for x, l in zip(cov, length)]
        phase = self.t["offsets"].double() @ torch.tensor(cov, dtype=torch.float64, device="cuda")
        self.phase = torch.polar(torch.ones_like(phase), phase)
        self.kinetic = 0.5 * _g2(case, self.kcart)
        self.dv = SPACING ** 3

    def apply(self, psi):
        out = _fft3(_fft3(psi) * self.kinetic[..., None], inverse=True)
        out += self.v[..., None] * psi
        flat, res = psi.reshape(-1, psi.shape[-1]), out.reshape(-1, psi.shape[-1])
        t = self.t
        for a, cnt in enumerate(t["count"]):
            p = t["points"][a, :cnt]
            m = t["values"][a, :, :cnt] * self.phase[a, :cnt]
            proj = t["kb"][a].to(torch.complex128) @ (self.dv * (m @ flat[p]))
            res.index_add_(0, p, m.mH @ proj)
        return out

    def exponential(self, factor, psi, order=4):
        out, term = psi.clone(), psi
        for n in range(1, order + 1):
            term = self.apply(term) * (factor / n)
            out += term
        return out

    def density(self, psi, occ):
        return (psi.abs() ** 2) @ torch.as_tensor(occ, device="cuda")

    def update(self, dens):
        g2 = _g2(self.case)
        kern = torch.where(g2 < 1e-6, torch.zeros_like(g2), 4.0 * math.pi / torch.where(g2 < 1e-6, torch.ones_like(g2), g2))
        vh = torch.fft.ifftn(torch.fft.fftn(dens) * kern).real
        n = torch.clamp(dens, min=1e-300)
        ex = -0.75 * (3.0 / math.pi) ** (1.0 / 3.0) * n ** (1.0 / 3.0)
        rs = (3.0 / (4.0 * math.pi * n)) ** (1.0 / 3.0)
        sq = torch.sqrt(rs)
        den = 1.0 + 1.0529 * sq + 0.3334 * rs
        low = -0.1423 / den * (1.0 + 7.0 / 6.0 * 1.0529 * sq + 4.0 / 3.0 * 0.3334 * rs) / den
        lr = torch.log(rs)
        high = (0.0311 * lr + (-0.048 - 0.0311 / 3.0) + 2.0 / 3.0 * 0.0020 * rs * lr
                + (2.0 * -0.0116 - 0.0020) / 3.0 * rs)
        vxc = torch.where(dens > 1e-15, 4.0 / 3.0 * ex + torch.where(rs >= 1.0, low, high), torch.zeros_like(dens))
        self.v = self.vion + vh + vxc

    def etrs(self, psi, occ, dt, nscf=5, threshold=5e-5):
        half = self.exponential(-0.5j * dt, psi)
        dens = self.density(self.exponential(-1j * dt, psi), occ)
        if self.case["interacting"]:
            self.update(dens)
        for _ in range(nscf):
            psi = self.exponential(-0.5j * dt, half)
            old, dens = dens, self.density(psi, occ)
            delta = float(self.dv * torch.sum((old - dens).abs()))
            if self.case["interacting"]:
                self.update(dens)
            if delta < threshold:
                break
        r = []
        for x, l in zip(_points(self.case), _lengths(self.case)):
            half_n = (len(x) + 1) // 2
            r.append(l * torch.cat([x[:half_n], x[half_n:] - 1.0]))
        dip = [float(self.dv * torch.sum(dens * c.reshape([-1 if j == k else 1 for j in range(3)])))
               for k, c in enumerate(r)]
        return psi, dens.reshape(-1), np.array(dip)

    def steepest_descent(self, f):
        """Five preconditioned line minimisations per state (Teter, Payne, Allan), Fourier space."""
        n = f.shape[0] * f.shape[1] * f.shape[2]
        dvg = self.dv / n

        def h(x):
            return _fft3(self.apply(_fft3(x, inverse=True)))

        def dot(x, y):
            return dvg * torch.sum(x.conj() * y, dim=(0, 1, 2))

        g2 = 0.5 * _g2(self.case)[..., None]
        hf = h(f)
        for _ in range(5):
            ev, nrm = dot(hf, f), dot(f, f)
            res = hf - f * (ev / nrm.real)
            kin = (dot(g2 * res, res) / dot(res, res)).real
            x = g2 / kin
            top = 27.0 + 18.0 * x + 12.0 * x ** 2 + 8.0 * x ** 3
            res = res * (top / (top + 16.0 * x ** 4))
            hres = h(res)
            m0, m1, m2, m3 = dot(res, res), dot(f, res), dot(res, hres), dot(f, hres)
            a, b, c = (m0 * m3 - m2 * m1).real, (nrm * m2 - ev * m0).real, (ev * m1 - m3 * nrm).real
            d = b + torch.sqrt(b * b - 4.0 * a * c)
            step = torch.where(d.abs() < 1e-15, torch.zeros_like(d), 2.0 * c / d)
            f = f + step * res
            hf = hf + step * hres
        return f


def _orthonormal(m, weight):
    u = torch.linalg.cholesky(weight * (m.conj().T @ m)).mH
    return torch.linalg.solve_triangular(u, m, upper=True, left=False)


def exact(case, seed):
    op = case["op"]
    psi = _orbitals(case, seed, orthonormal=op != "orthogonalize")
    wide = lambda x: x.to(REAL[case["precision"]]).to(torch.complex128)  # noqa: E731  (the inputs as run() gets them)
    s, dv = case["nst"], SPACING ** 3
    if op == "overlap":
        chi = wide(psi * _mixing(case)[..., None]).reshape(-1, s)
        return (dv * (wide(psi).reshape(-1, s).conj().T @ chi)).cpu().numpy()
    if op == "orthogonalize":
        return _orthonormal(wide(psi).reshape(-1, s), dv).reshape(psi.shape)
    e = _Exact(case, seed)
    if op == "apply":
        return e.apply(wide(psi))
    if op == "fourier":
        return _fft3(e.apply(_fft3(wide(_fft3(psi)), inverse=True)))
    occ = _occupations(case)
    if op == "etrs":
        phi, dens, dip = e.etrs(wide(psi), occ, _dt(case))
        return {"orbitals": phi, "density": dens, "dipole": dip}
    n = psi[..., 0].numel()
    f = e.steepest_descent(wide(_fft3(psi)))
    f = _orthonormal(f.reshape(-1, s), dv / n).reshape(psi.shape)
    phi = _fft3(f, inverse=True)
    m = phi.reshape(-1, s)
    w, vec = torch.linalg.eigh(dv * (m.conj().T @ e.apply(phi).reshape(-1, s)))
    dens = e.density((m @ vec).reshape(psi.shape), occ).reshape(-1)
    # the phases of the eigenvectors are free: no value for the orbitals
    return {"eigenvalues": w.cpu().numpy(), "orbitals": None, "density": dens.cpu().numpy()}
