"""Performance cases of miepy_gb300: what users of the package have it compute.

Every case goes through public entry points (ClusterBatch, wavelength_sweep,
sphere_cluster and its observables, large.near_field) on inputs made from a seed, and
returns the whole result.  Kinds of case:

  solve      assembly, BiCGSTAB solve and epilogue of one cluster (ClusterBatch), in the
             precision and with the right-hand sides the user asks for
  sweep      a spectrum: one cluster at many wavelengths (wavelength_sweep)
  substrate  a whole sphere_cluster above a planar interface (dense FP64 route)
  lattice    a whole sphere_cluster repeated on a periodic lattice (lattice sums)
  field      E or H of a solved sphere_cluster on a plane (FP64, interior included)
  map        a large near-field map with FP32 exterior sums (large.near_field)
  pattern    the radiation pattern: cluster coefficients, cross-sections per multipole
             and far fields over the sphere of directions

exact() evaluates the same physics in 64 bits with plain torch and numpy: Gaunt
coefficients from the closed form of the 3j symbol, dense operators, direct sums.
"""

import math
import types

import numpy as np
import torch

import miepy_gb300 as gb
from miepy_gb300 import large, sweep

NM = 1e-9


# ------------------------------------------------------------------- cases --
def listed():
    return [
        # a few silver spheres near a resonance at low order: the smallest everyday solve,
        # all launches and latency
        dict(name="pentamer_fp64", kind="solve", N=5, lmax=2, R=1, precision="fp64", tol=1e-5, metal=True,
             tensor=False),
        # the default precision and tolerance on an ordinary cluster of an odd size
        dict(name="cluster61_lmax5_fp64", kind="solve", N=61, lmax=5, R=1, precision="fp64", tol=1e-5, metal=False,
             tensor=False),
        # the benchmark cluster (200 spheres, both polarisations) in mixed precision
        dict(name="cluster200_lmax4_mixed", kind="solve", N=200, lmax=4, R=2, precision="mixed", tol=1e-10, metal=False,
             tensor=False),
        # closely packed larger spheres that need high orders
        dict(name="cluster97_lmax8_mixed", kind="solve", N=97, lmax=8, R=1, precision="mixed", tol=1e-10, metal=False,
             tensor=False),
        # eight excitations of one cluster (two polarisations, four incidences) on the tensor cores
        dict(name="eight_sources_mixed", kind="solve", N=200, lmax=4, R=8, precision="mixed", tol=1e-10, metal=False,
             tensor=True),
        # a metasurface patch: the largest single system
        dict(name="metasurface2000_mixed", kind="solve", N=2000, lmax=3, R=1, precision="mixed", tol=1e-10, metal=False,
             tensor=False),
        # a spectrum of a Drude-metal cluster with lmax by wavelength: a ragged batch
        dict(name="sweep40x24_mixed", kind="sweep", N=40, W=24, precision="mixed", tol=1e-10),
        # nanoparticles on glass: the dense route, as a whole user call
        dict(name="substrate30_lmax3", kind="substrate", N=30, lmax=3),
        # the unit cell of a square lattice: the lattice sums, as a whole user call
        dict(name="lattice6_lmax3", kind="lattice", N=6, lmax=3, square=True),
        # a field picture around and inside a cluster
        dict(name="field25_lmax4", kind="field", N=25, lmax=4, n=97, magnetic=False),
        # a field map over a metasurface patch
        dict(name="map2000_lmax3", kind="map", N=2000, lmax=3, n=512, magnetic=False),
        # a scattering pattern over all directions
        dict(name="pattern50_lmax4", kind="pattern", N=50, lmax=4, lmax_cluster=6, n=60),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "sweep", "substrate", "lattice", "field", "map", "pattern"])
    if kind == "solve":
        precision = rng.choice(["fp64", "mixed", "mixed", "tensor"])
        if precision == "tensor":
            return dict(kind=kind, N=_logint(rng, 20, 240), lmax=rng.randint(2, 5), R=rng.choice([4, 8]),
                        precision="mixed", tol=1e-10, metal=False, tensor=True)
        lmax = rng.randint(1, 8)
        most = 1e8 if precision == "fp64" else 1.5e9    # elements of the packed matrix
        hi = min(400 if lmax > 3 else 1900, int(math.sqrt(2 * most)) // (2 * lmax * (lmax + 2)))
        N = _logint(rng, 2, hi)
        return dict(kind=kind, N=N, lmax=lmax, R=rng.choice([1, 2]), precision=precision,
                    tol=1e-5 if precision == "fp64" else 1e-10, metal=N <= 12 and lmax <= 4 and rng.random() < 0.5,
                    tensor=False)
    if kind == "sweep":
        return dict(kind=kind, N=_logint(rng, 4, 60), W=_logint(rng, 4, 32), precision=rng.choice(["mixed", "fp64"]),
                    tol=1e-10)
    if kind == "substrate":
        return dict(kind=kind, N=_logint(rng, 2, 60), lmax=rng.randint(1, 4))
    if kind == "lattice":
        return dict(kind=kind, N=_logint(rng, 1, 12), lmax=rng.randint(1, 4), square=rng.random() < 0.7)
    if kind == "field":
        return dict(kind=kind, N=_logint(rng, 1, 60), lmax=rng.randint(1, 6), n=_logint(rng, 16, 140),
                    magnetic=rng.random() < 0.5)
    if kind == "map":
        return dict(kind=kind, N=_logint(rng, 50, 1900), lmax=rng.randint(1, 5), n=_logint(rng, 64, 360),
                    magnetic=rng.random() < 0.5)
    return dict(kind=kind, N=_logint(rng, 1, 100), lmax=rng.randint(1, 6), lmax_cluster=rng.randint(2, 8),
                n=_logint(rng, 8, 90))


# ------------------------------------------------------------------ inputs --
WAVELENGTH = 600 * NM


def _spheres(rng, N, lmax):
    """N non-overlapping spheres in a cube at the density of the benchmark cluster,
    their radii growing with the order that they need."""
    scale = 1.0 if lmax <= 5 else 1.5
    rad = rng.uniform(50, 100, N) * NM * scale
    box = 2000 * NM * scale * (N / 200) ** (1 / 3) + 150 * NM
    pos = np.empty((N, 3))
    k = 0
    while k < N:
        c = rng.uniform(-box / 2, box / 2, 3)
        if k == 0 or np.all(np.linalg.norm(pos[:k] - c, axis=1) > rad[:k] + rad[k] + 2 * NM):
            pos[k] = c
            k += 1
        else:
            box *= 1.0005
    return pos, rad


def _sources(rng, R):
    """R plane waves: both polarisations of as many directions as that takes."""
    out = []
    for q in range(R):
        if q % 2 == 0:
            th, ph = (0.0, 0.0) if q == 0 else (float(rng.uniform(0.1, 1.2)), float(rng.uniform(0, 2 * np.pi)))
        out.append(gb.plane_wave([1, 0] if q % 2 == 0 else [0, 1], theta=th, phi=ph))
    return out


def _spec(pos, rad, index, lmax, sources, wavelength=WAVELENGTH):
    md = gb.material_struct([gb.constant_material(index=index)] * len(rad), gb.constant_material(index=1.0),
                            wavelength=wavelength)
    ms, mi = gb.mie_coefficients(rad, md.eps, md.mu, md.eps_b, md.mu_b, md.k_b, lmax)
    k = float(np.real(md.k_b))
    p_src = np.ascontiguousarray(np.stack([s.structure(pos, k, lmax) for s in sources], axis=-1))
    return dict(position=pos, mie_scat=ms, mie_int=mi, k=k, p_src=p_src), md


def _solve_inputs(c, seed):
    rng = np.random.default_rng([11, seed])
    if c["N"] > 400:
        pos = large.hex_lattice(N=c["N"], seed=int(rng.integers(1 << 30)), cells=int(math.sqrt(c["N"])) + 2)
        rad = np.full(c["N"], 80 * NM)
    else:
        pos, rad = _spheres(rng, c["N"], c["lmax"])
    index = 0.06 + 4.0j if c["metal"] else (2.0 if c["N"] > 400 else 1.5 + 0.01j)
    return _spec(pos, rad, index, c["lmax"], _sources(rng, c["R"]))[0]


def _sweep_inputs(c, seed):
    rng = np.random.default_rng([12, seed])
    pos, rad = sweep.drude_cluster(N=c["N"], seed=int(rng.integers(1 << 30)),
                                   box=2e-6 * (c["N"] / 100) ** (1 / 3) + 1e-7)
    wl = np.linspace(400 * NM, 1000 * NM, c["W"]) * (1 + 0.002 * rng.uniform(-1, 1))
    return sweep.sweep_specs(pos, rad, gb.drude_material(9.0, 9.0, 0.07), wl, sweep.adaptive_lmax)


def _plane_cluster(rng, N, rmin, rmax, pitch):
    """N spheres on a jittered square grid in the plane z = 0."""
    side = int(math.ceil(math.sqrt(N)))
    xy = np.array([(i, j) for i in range(side) for j in range(side)][:N], float) * pitch
    xy = xy - xy.mean(axis=0) + rng.uniform(-0.1, 0.1, (N, 2)) * pitch
    return np.column_stack([xy, np.zeros(N)]), rng.uniform(rmin, rmax, N)


def _cluster_args(c, seed):
    """The arguments of the sphere_cluster calls (solver.exact: the fields and patterns
    below are compared to their own accuracy, not to a solver tolerance)."""
    rng = np.random.default_rng([13, seed])
    kind, N = c["kind"], c["N"]
    if kind == "substrate":
        pos, rad = _plane_cluster(rng, N, 50 * NM, 75 * NM, 220 * NM)
        return dict(position=pos + [0, 0, 90 * NM], radius=rad, index=0.06 + 4.0j, wavelength=633 * NM,
                    theta=float(rng.uniform(0, 0.8)), phi=float(rng.uniform(0, 6)), substrate=1.5, cell=None)
    if kind == "lattice":
        pos, rad = _plane_cluster(rng, N, 40 * NM, 70 * NM, 230 * NM)
        return dict(position=pos, radius=rad, index=3.5 + 0.1j, wavelength=700 * NM, theta=float(rng.uniform(0, 0.5)),
                    phi=float(rng.uniform(0, 6)), substrate=None, cell=230 * NM * math.ceil(math.sqrt(N)) + 180 * NM)
    pos, rad = _spheres(rng, N, c["lmax"])
    return dict(position=pos, radius=rad, index=2.0 + 0.02j, wavelength=WAVELENGTH, theta=float(rng.uniform(0, 1)),
                phi=float(rng.uniform(0, 6)), substrate=None, cell=None)


def _make_cluster(c, a):
    sym = None
    if a["cell"] is not None:
        sym = gb.symmetry.square_lattice_2d(a["cell"]) if c["square"] else gb.symmetry.x_translation_1d(a["cell"])
    return gb.sphere_cluster(
        position=a["position"], radius=a["radius"], material=gb.constant_material(index=a["index"]),
        source=gb.plane_wave([1, 0.3j], theta=a["theta"], phi=a["phi"]), wavelength=a["wavelength"], lmax=c["lmax"],
        symmetry=sym, interface=gb.interface(gb.constant_material(index=a["substrate"])) if a["substrate"] else None,
        method=gb.solver.exact)


def _plane(a, n):
    lo, hi = a["position"].min(axis=0) - 300 * NM, a["position"].max(axis=0) + 300 * NM
    x, y = np.meshgrid(np.linspace(lo[0], hi[0], n), np.linspace(lo[1], hi[1], n + 3), indexing="ij")
    return x, y, np.full_like(x, a["position"][0, 2] + 11 * NM)


def _directions(n):
    th, ph = np.meshgrid(np.linspace(0.01, np.pi - 0.01, n), np.linspace(0, 2 * np.pi, 2 * n), indexing="ij")
    return th, ph, 1e-3     # a detector 1 mm away


def _map_inputs(c, seed):
    """A metasurface patch under a plane wave, each sphere excited by the incident wave:
    coefficients of the size and phases that a map meets."""
    rng = np.random.default_rng([14, seed])
    pos = large.hex_lattice(N=c["N"], seed=int(rng.integers(1 << 30)), cells=int(math.sqrt(c["N"])) + 2)
    rad = np.full(c["N"], 80 * NM)
    spec, md = _spec(pos, rad, 2.0, c["lmax"], [gb.plane_wave([1, 0.3], theta=float(rng.uniform(0, 0.8)), phi=1.0)])
    return spec, md, rad, large.plane_grid(pos, n=c["n"], z=float(rng.uniform(20, 120)) * NM)


def prepare(case, seed):
    c = case
    if c["kind"] == "solve":
        b = gb.ClusterBatch([_solve_inputs(c, seed)], R=c["R"], precision=c["precision"], tensor=c["tensor"])
        return c, b
    if c["kind"] == "sweep":
        return c, _sweep_inputs(c, seed)
    a = _cluster_args(c, seed) if c["kind"] != "map" else None
    if c["kind"] in ("substrate", "lattice"):
        return c, a
    if c["kind"] == "field":
        return c, _make_cluster(c, a), _plane(a, c["n"])
    if c["kind"] == "pattern":
        return c, _make_cluster(c, a), _directions(c["n"])
    spec, md, rad, pts = _map_inputs(c, seed)
    b = gb.ClusterBatch([spec], precision="mixed", packed=False)
    b.x.copy_(b.b)
    b.epilogue(1.0)
    return c, b, md, rad, torch.from_numpy(pts).to(b.device)


# --------------------------------------------------------------------- run --
def run(state):
    c = state[0]
    if c["kind"] == "solve":
        b = state[1]
        b.assemble()
        b.solve(tol=c["tol"], maxiter=1000, inner_tol=1e-4, max_refine=8)
        b.epilogue(1.0)
        return dict(p_inc=b.x, p_scat=b.p_scat, p_int=b.p_int, xs=b.xs, force=b.F, torque=b.T)
    if c["kind"] == "sweep":
        r = gb.sweep.wavelength_sweep(None, None, None, None, precision=c["precision"], tol=c["tol"], per_particle=True,
                                      specs=state[1])
        return dict(C=[r.C_sca, r.C_abs, r.C_ext], per_particle=r.per_particle)
    if c["kind"] in ("substrate", "lattice"):
        cl = _make_cluster(c, state[1])
        C = cl.cross_sections()
        return dict(p_inc=cl.p_inc, p_scat=cl.p_scat, p_int=cl.p_int, C=np.array(C),
                    force=cl.force(), torque=cl.torque())
    if c["kind"] == "field":
        cl, (x, y, z) = state[1:]
        return cl.H_field(x, y, z) if c["magnetic"] else cl.E_field(x, y, z)
    if c["kind"] == "pattern":
        cl, (th, ph, radius) = state[1:]
        C = cl.cross_sections_per_multipole(c["lmax_cluster"])
        return dict(p_cluster=cl.p_cluster, C=[C.scattering, C.absorption, C.extinction],
                    E=cl.E_angular(th, ph, radius=radius), H=cl.H_angular(th, ph, radius=radius))
    _, b, md, rad, pts = state
    # kept as complex64, the precision of the map's sums
    return large.near_field(b, 0, md, rad, pts, precision="fp32", magnetic=c["magnetic"]).to(torch.complex64)


# -------------------------------------------------------------------- work --
def work(case):
    """Bytes of the inputs and outputs; operations of the translation operator's products
    (16 real operations per block element, right-hand side and product, for as many
    products as the tolerance takes on such clusters) or of the expansions' terms (about
    40 real operations per point, particle and mode)."""
    c = case
    rmax = lambda L: L * (L + 2)   # noqa: E731
    vec = lambda N, L: 16.0 * 2 * rmax(L) * N   # noqa: E731
    if c["kind"] == "solve":
        N, B = c["N"], 2 * rmax(c["lmax"])
        products = 16 if c["tol"] > 1e-8 else 24
        return dict(bytes=c["R"] * 4 * vec(N, c["lmax"]) + 100 * N,
                    flops=16.0 * products * c["R"] * N * (N - 1) / 2 * B * B + c["R"] * 400 * N * B)
    if c["kind"] == "sweep":
        L = sweep.adaptive_lmax(np.linspace(400 * NM, 1000 * NM, c["W"]))
        return dict(bytes=float(sum(vec(c["N"], int(l)) * 2 for l in L)),
                    flops=float(sum(16.0 * 24 * c["N"] * (c["N"] - 1) / 2 * (2 * rmax(int(l))) ** 2 for l in L)))
    if c["kind"] in ("substrate", "lattice"):
        D = 2 * rmax(c["lmax"]) * c["N"]
        cells = 1 if c["kind"] == "substrate" else 5000
        return dict(bytes=4 * vec(c["N"], c["lmax"]),
                    flops=8.0 * 30 * D * D + 40.0 * cells * c["N"] ** 2 * (2 * c["lmax"] + 1) ** 2)
    if c["kind"] == "pattern":
        points = 2.0 * c["n"] ** 2
        return dict(bytes=2 * 2 * 16 * points + vec(c["N"], c["lmax"]),
                    flops=2 * 40.0 * points * c["N"] * rmax(c["lmax"]))
    points = float(c["n"] * (c["n"] + 3 if c["kind"] == "field" else c["n"]))
    return dict(bytes=(24 + 48) * points + 2 * vec(c["N"], c["lmax"]), flops=40.0 * points * c["N"] * rmax(c["lmax"]))


# ------------------------------------------------------- 64-bit evaluation --
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _modes(L):
    return [(n, m) for n in range(1, L + 1) for m in range(-n, n + 1)]


def _w3j(j1, j2, j3, m1, m2):
    """The 3j symbol (j1 j2 j3; m1 m2 -m1-m2): Racah's sum over integers."""
    m3 = -m1 - m2
    if abs(m1) > j1 or abs(m2) > j2 or abs(m3) > j3 or not abs(j1 - j2) <= j3 <= j1 + j2:
        return 0.0
    f, a, b, d = math.factorial, j1 + j2 - j3, j1 - j2 + j3, -j1 + j2 + j3
    s = 0
    for t in range(a + 1):
        if 0 <= j1 - m1 - t <= b and 0 <= j2 + m2 - t <= d:
            s += (-1) ** t * math.comb(a, t) * math.comb(b, j1 - m1 - t) * math.comb(d, j2 + m2 - t)
    num = f(j1 + m1) * f(j1 - m1) * f(j2 + m2) * f(j2 - m2) * f(j3 + m3) * f(j3 - m3)
    return (-1) ** ((j1 - j2 - m3) % 2) * s * math.sqrt(num / (f(a) * f(b) * f(d) * f(j1 + j2 + j3 + 1)))


_FACTORS = {}


def _translation_factors(Lo, Li):
    """Real matrices (CA, CB) [2L'+.., rmax_o * rmax_i] with A = i^(n+v) CA^T G and
    B = i^(n+v+1) CB^T G for G[p, mu] = P_p^mu(cos theta) z_p(kr) e^(i mu phi) flattened:
    the vector addition theorem for (n, m) <= Lo from (v, u) <= Li."""
    if (Lo, Li) in _FACTORS:
        return _FACTORS[Lo, Li]
    f, S = math.factorial, Lo + Li
    mo, mi = _modes(Lo), _modes(Li)
    CA = np.zeros(((S + 2) * (2 * S + 1), len(mo) * len(mi)))
    CB = np.zeros_like(CA)
    for a, (n, mm) in enumerate(mo):
        m = -mm
        for b, (v, u) in enumerate(mi):
            col, mu = a * len(mi) + b, u + m
            pre = 0.5 * (-1) ** (m % 2) * math.sqrt((2 * v + 1) * (2 * n + 1) / (v * (v + 1) * n * (n + 1)) *
                                                    (f(v - u) * f(n - m)) / (f(v + u) * f(n + m)))
            gaunt = (-1) ** (mu % 2) * math.sqrt((f(n + m) * f(v + u)) / (f(n - m) * f(v - u)))
            for q in range(min(n, v, (n + v - abs(mu)) // 2) + 1):
                p = n + v - 2 * q
                w = _w3j(n, v, p, 0, 0) * _w3j(n, v, p, m, u) * math.sqrt(f(p - mu) / f(p + mu))
                CA[p * (2 * S + 1) + mu + S, col] += pre * gaunt * (2 * p + 1) * w * (-1) ** q * (
                    n * (n + 1) + v * (v + 1) - p * (p + 1))
            for q in range(1, min(n, v, (n + v + 1 - abs(mu)) // 2) + 1):
                p = n + v - 2 * q
                w = _w3j(n, v, p, 0, 0) * _w3j(n, v, p + 1, m, u) * math.sqrt(f(p + 1 - mu) / f(p + 1 + mu))
                CB[(p + 1) * (2 * S + 1) + mu + S, col] -= pre * gaunt * (2 * p + 3) * w * (-1) ** q * math.sqrt(
                    ((p + 1) ** 2 - (n - v) ** 2) * ((n + v + 1) ** 2 - (p + 1) ** 2))
    ip = np.array([1j ** ((n + v) % 4) for n, _ in mo for v, _ in mi])
    _FACTORS[Lo, Li] = (CA, CB, ip)
    return _FACTORS[Lo, Li]


def _sph_bessel_up(x, nmax):
    """j_n and y_n, n = 0..nmax, of real x (tensors): y by the upward recurrence, j by the
    downward one (Miller), normalised at j_0 or j_1."""
    y = [-torch.cos(x) / x, -torch.cos(x) / x ** 2 - torch.sin(x) / x]
    for n in range(2, nmax + 1):
        y.append((2 * n - 1) / x * y[-1] - y[-2])
    return _sph_jn(x, nmax), y[: nmax + 1]


def _sph_jn(x, nmax):
    """j_n, n = 0..nmax, of real or complex x: upward where |x| is large, else downward."""
    j0, j1 = torch.sin(x) / x, torch.sin(x) / x ** 2 - torch.cos(x) / x
    up = [j0, j1]
    for n in range(2, nmax + 1):
        up.append((2 * n - 1) / x * up[-1] - up[-2])
    xs = torch.where(x.abs() > nmax + 1, torch.ones_like(x), x)
    hi, cur, down = torch.zeros_like(x), torch.full_like(x, 1e-290), [None] * (nmax + 2)
    for n in range(nmax + 26, -1, -1):
        if n <= nmax + 1:
            down[n] = cur
        hi, cur = cur, (2 * n + 1) / xs * cur - hi
        big = cur.abs() > 1e250
        if bool(big.any()):
            sc = torch.where(big, torch.full_like(x, 1e-250), torch.ones_like(x))
            hi, cur = hi * sc, cur * sc
            down = [d if d is None else d * sc for d in down]
    use0 = down[0].abs() * j0.abs() >= down[1].abs() * j1.abs()
    s = torch.where(use0, j0 / down[0], j1 / down[1])
    return [torch.where(x.abs() > nmax + 1, up[n], s * down[n]) for n in range(nmax + 1)]


def _legendre(ct, st, L):
    """P[n][m] (no Condon-Shortley phase) and P[n][m] / sin(theta) for m >= 1."""
    P = [[None] * (n + 1) for n in range(L + 1)]
    Q = [[None] * (n + 1) for n in range(L + 1)]
    one = torch.ones_like(ct)
    for T, m0 in ((P, 0), (Q, 1)):
        for m in range(m0, L + 1):
            d = 1.0
            for k in range(1, m + 1):
                d *= 2 * k - 1
            T[m][m] = d * (st ** (m - m0) if m > m0 else one)
            if m + 1 <= L:
                T[m + 1][m] = ct * (2 * m + 1) * T[m][m]
            for n in range(m + 2, L + 1):
                T[n][m] = ((2 * n - 1) * ct * T[n - 1][m] - (n + m - 1) * T[n - 2][m]) / (n - m)
    return P, Q


def _angles(d):
    rho = torch.hypot(d[..., 0], d[..., 1])
    r = torch.hypot(rho, d[..., 2])
    on = rho == 0
    safe = torch.where(on, torch.ones_like(rho), rho)
    cp = torch.where(on, torch.ones_like(rho), d[..., 0] / safe)
    sp = torch.where(on, torch.zeros_like(rho), d[..., 1] / safe)
    return r, d[..., 2] / r, rho / r, torch.complex(cp, sp)


def _translation_G(d, k, S, regular=False):
    """G [P, (S+2) * (2S+1)] of separations d [P, 3]."""
    r, ct, st, e = _angles(d)
    j, y = _sph_bessel_up(k * r, S + 1)
    P, _ = _legendre(ct, st, S + 1)
    G = torch.zeros(d.shape[0], S + 2, 2 * S + 1, dtype=torch.complex128, device=d.device)
    for p in range(S + 2):
        z = torch.complex(j[p], torch.zeros_like(j[p]) if regular else y[p])
        for m in range(0, min(p, S) + 1):
            G[:, p, S + m] = P[p][m] * z * e ** m
            if m:
                G[:, p, S - m] = (-1) ** m * math.factorial(p - m) / math.factorial(p + m) * P[p][m] * z * e.conj() ** m
    return G.reshape(d.shape[0], -1)


def _translation_blocks(G, Lo, Li):
    """[P, 2, rmax_o, 2, rmax_i]: A on equal polarisations, B on opposite ones."""
    CA, CB, ip = (torch.as_tensor(t, device=G.device) for t in _translation_factors(Lo, Li))
    ro, ri = Lo * (Lo + 2), Li * (Li + 2)
    A = ip * torch.complex(G.real @ CA, G.imag @ CA)
    Bm = 1j * ip * torch.complex(G.real @ CB, G.imag @ CB)
    out = torch.stack([torch.stack([A, Bm], 1), torch.stack([Bm, A], 1)], 1).reshape(-1, 2, 2, ro, ri)
    return out.permute(0, 1, 3, 2, 4)


def _mie_rows(mie, L):
    """mie [N, 2, L] -> [N, 2 * rmax]."""
    idx = torch.tensor([n - 1 for n, _ in _modes(L)], device=mie.device)
    return mie[:, :, idx].reshape(mie.shape[0], -1)


def _operator(pos, mie, k, L, mirror=None, cells=None, k_hat=None):
    """Dense I + T [D, D]: sphere aggregate, minus the reflection matrix of an interface
    (mirror = (r0, z)), plus the lattice sums over cells."""
    N, B = pos.shape[0], 2 * L * (L + 2)
    T = torch.zeros(N, B, N, B, dtype=torch.complex128, device=pos.device)
    rows = _mie_rows(mie, L)
    step = max(1, 4_000_000 // (N * B * B) + 1)
    sign = torch.tensor([(-1.0) ** ((m + n + a + 1) % 2) for a in (0, 1) for n, m in _modes(L)], dtype=torch.float64,
                        device=pos.device)
    for i0 in range(0, N, step):
        i1 = min(N, i0 + step)
        ii = torch.arange(i0, i1, device=pos.device)[:, None].expand(-1, N).reshape(-1)
        jj = torch.arange(N, device=pos.device)[None].expand(i1 - i0, -1).reshape(-1)
        off = ii != jj
        d = torch.where(off[:, None], pos[ii] - pos[jj], torch.ones_like(pos[ii]) / k)
        G = _translation_G(d, k, 2 * L)
        G[~off] = 0
        if cells is not None:
            ph = torch.exp(-1j * k * (cells @ k_hat))
            for c0 in range(0, cells.shape[0], 512):
                cc = cells[c0: c0 + 512]
                for q in range(d.shape[0]):
                    G[q] += ph[c0: c0 + 512] @ _translation_G((pos[ii[q]] - pos[jj[q]])[None] - cc, k, 2 * L)
        blk = _translation_blocks(G, L, L).reshape(i1 - i0, N, B, B)
        if mirror is not None:
            image = pos.clone()
            image[:, 2] = 2 * mirror[1] - image[:, 2]
            R = _translation_blocks(_translation_G(image[ii] - pos[jj], k, 2 * L), L, L).reshape(i1 - i0, N, B, B)
            blk = blk + mirror[0] * sign[None, None, :, None] * R
        T[i0:i1] = (blk * rows[None, :, None, :]).permute(0, 2, 1, 3)
    T = T.reshape(N * B, N * B)
    T.diagonal().add_(1.0)
    return T


def _solve(M, b):
    """M x = b by BiCGSTAB with restarts from the true residual, to rounding; LU for
    systems that are small or do not yield."""
    if M.shape[0] <= 3000:
        return torch.linalg.solve(M, b)
    cols = []
    for q in range(b.shape[1]):
        bq, x = b[:, q], torch.zeros_like(b[:, q])
        for _ in range(8):
            r = bq - M @ x
            if r.norm() < 1e-14 * bq.norm():
                break
            r0, p, rho, r_in = r.clone(), r.clone(), torch.vdot(r, r), r.norm()
            for _ in range(60):
                v = M @ p
                al = rho / torch.vdot(r0, v)
                s = r - al * v
                t = M @ s
                om = torch.vdot(t, s) / torch.vdot(t, t)
                x = x + al * p + om * s
                r = s - om * t
                if r.norm() < 1e-9 * r_in or r.norm() < 2e-15 * bq.norm():
                    break
                rho, old = torch.vdot(r0, r), rho
                p = r + rho / old * al / om * (p - om * v)
        if (bq - M @ x).norm() > 1e-12 * bq.norm():
            return torch.linalg.solve(M, b)
        cols.append(x)
    return torch.stack(cols, 1)


def _mie(radius, index, k, L):
    """(a_n, b_n) and (c_n, d_n) [N, 2, L] of spheres of a relative index in vacuum."""
    x = torch.as_tensor(k * radius)
    m = complex(index)
    j, y = _sph_bessel_up(x, L)
    jm = _sph_jn(m * x.to(torch.complex128), L)
    sc, it = [], []
    for n in range(1, L + 1):
        h, h1 = torch.complex(j[n], y[n]), torch.complex(j[n - 1], y[n - 1])
        dj, dh = x * j[n - 1] - n * j[n], x * h1 - n * h           # (x z_n)'
        dm = m * x * jm[n - 1] - n * jm[n]                          # (mx j_n(mx))'
        a = (m * m * jm[n] * dj - j[n] * dm) / (m * m * jm[n] * dh - h * dm)
        b = (jm[n] * dj - j[n] * dm) / (jm[n] * dh - h * dm)
        w = j[n] * dh - h * dj
        sc.append(torch.stack([a, b], 1))
        it.append(torch.stack([w / (jm[n] * dh - h * dm), m * w / (m * m * jm[n] * dh - h * dm)], 1))
    return torch.stack(sc, 2), torch.stack(it, 2)


def _emn(n, m):
    return math.sqrt((2 * n + 1) * math.factorial(n - m) / (n * (n + 1) * math.factorial(n + m)))


def _plane_wave(pos, k, L, theta, phi, pol, amplitude=1.0, phase=0.0):
    """p_src [N, 2, rmax] of a plane wave, and its E and H functions of points."""
    t = lambda v: torch.tensor(v, dtype=torch.float64)   # noqa: E731
    khat = np.array([math.sin(theta) * math.cos(phi), math.sin(theta) * math.sin(phi), math.cos(theta)])
    n_tm = np.array([math.cos(theta) * math.cos(phi), math.cos(theta) * math.sin(phi), -math.sin(theta)])
    n_te = np.array([-math.sin(phi), math.cos(phi), 0.0])
    P, Q = _legendre(t(math.cos(theta)), t(math.sin(theta)), L)
    out = np.zeros((pos.shape[0], 2, L * (L + 2)), complex)
    for r, (n, m) in enumerate(_modes(L)):
        a = abs(m)
        neg = 1.0 if m >= 0 else (-1) ** a * math.factorial(n - a) / math.factorial(n + a)
        pi = neg * m * float(Q[n][a]) if m else 0.0
        up = float(P[n][a + 1]) if a + 1 <= n else 0.0
        tau = -float(P[n][1]) if a == 0 else neg * 0.5 * ((n + a) * (n - a + 1) * float(P[n][a - 1]) - up)
        f = amplitude * np.exp(1j * (k * pos @ khat + phase - m * phi)) * _emn(n, m)
        out[:, 0, r] = f * (tau * pol[0] - 1j * pi * pol[1])
        out[:, 1, r] = f * (pi * pol[0] - 1j * tau * pol[1])
    wave = lambda x: amplitude * np.exp(1j * (np.tensordot(khat, x, 1) * k + phase))   # noqa: E731
    E = lambda x: np.multiply.outer(n_tm * pol[0] + n_te * pol[1], wave(x))   # noqa: E731
    H = lambda x: np.multiply.outer(n_te * pol[0] - n_tm * pol[1], wave(x))   # noqa: E731
    return out, E, H, khat


def _observables(p_inc, p_scat, p_src, k, L):
    """Cross-sections [N, R, 3, 2, L] and force, torque [N, R, 3] from coefficients
    [N, 2, rmax, R] (numpy), in vacuum."""
    N, _, _, R = p_inc.shape
    xs = np.zeros((N, R, 3, 2, L))
    f = 4 * np.pi / k ** 2
    for r, (n, _) in enumerate(_modes(L)):
        i, s, e = p_inc[:, :, r], p_scat[:, :, r], p_src[:, :, r]
        ab = f * (np.real(np.conj(i) * s) - np.abs(s) ** 2)
        ex = f * np.real(np.conj(e) * s)
        for q, v in enumerate((ex - ab, ab, ex)):
            xs[:, :, q, :, n - 1] += np.swapaxes(v, 1, 2)
    at = {nm: r for r, nm in enumerate(_modes(L))}
    eps0 = 8.854187817e-12
    Axy = np.pi / k ** 2 * eps0
    At = -2 * np.pi / k ** 3 * eps0
    F, T = np.zeros((N, R, 3)), np.zeros((N, R, 3))
    Fxy = np.zeros((N, R), complex)
    P, Q, PI, QI = p_scat[:, 0], p_scat[:, 1], p_inc[:, 0], p_inc[:, 1]
    c = np.conj

    def tri(a, b, ai, bi):
        return 2 * a * c(b) - a * c(bi) - ai * c(b)

    for r, (n, m) in enumerate(_modes(L)):
        p, q, pi, qi = P[:, r], Q[:, r], PI[:, r], QI[:, r]
        if m != n:
            s = at[n, m + 1]
            w = math.sqrt((n + m + 1) * (n - m))
            Fxy += Axy * w / (n * (n + 1)) * (tri(p, Q[:, s], pi, QI[:, s]) + tri(q, P[:, s], qi, PI[:, s]))
            base = p * c(P[:, s]) + q * c(Q[:, s])
            u, v = P[:, s] * c(pi) + Q[:, s] * c(qi), p * c(PI[:, s]) + q * c(QI[:, s])
            T[:, :, 0] -= At * w * np.real(base - 0.5 * (u + v))
            T[:, :, 1] -= At * w * np.imag(base + 0.5 * (u - v))
        F[:, :, 2] += np.real(-2 * Axy * m / (n * (n + 1)) * tri(p, q, pi, qi))
        T[:, :, 2] += At * m * (np.abs(p) ** 2 + np.abs(q) ** 2 - np.real(p * c(pi) + q * c(qi)))
        if n < L:
            d = math.sqrt(n * (n + 2) / ((2 * n + 3) * (2 * n + 1))) / (n + 1)
            s = at[n + 1, m + 1]
            Fxy -= Axy * d * math.sqrt((n + m + 2) * (n + m + 1)) * (
                tri(p, P[:, s], pi, PI[:, s]) + tri(q, Q[:, s], qi, QI[:, s]))
            s = at[n + 1, m - 1]
            Fxy += Axy * d * math.sqrt((n - m + 1) * (n - m + 2)) * (
                tri(P[:, s], p, PI[:, s], pi) + tri(Q[:, s], q, QI[:, s], qi))
            s = at[n + 1, m]
            F[:, :, 2] += np.real(-2 * Axy * d * math.sqrt((n - m + 1) * (n + m + 1)) * (
                tri(P[:, s], p, PI[:, s], pi) + tri(Q[:, s], q, QI[:, s], qi)))
    F[:, :, 0], F[:, :, 1] = Fxy.real, Fxy.imag
    return xs, F, T


def _expand(d, c0, c1, k, L, outgoing, far_only=False):
    """Cartesian field [..., 3] of the expansions c0 (N) and c1 (M) [..., rmax] (broadcast)
    at separations d [..., 3]; k real or complex."""
    r, ct, st, e = _angles(d)
    x = k * r
    if outgoing and far_only:   # h_n -> (-i)^(n+1) e^{ix} / x, (x h_n)' / x -> (-i)^n e^{ix} / x
        g = torch.exp(1j * x.to(torch.complex128)) / x
        z = [(-1j) ** (n + 1) * g for n in range(L + 1)]
    elif outgoing:
        j, y = _sph_bessel_up(x, L)
        z = [torch.complex(a, b) for a, b in zip(j, y)]
    else:
        z = _sph_jn(x, L)
    P, Q = _legendre(ct, st, L)
    Er = Et = Ep = 0
    for q, (n, m) in enumerate(_modes(L)):
        a = abs(m)
        neg = 1.0 if m >= 0 else (-1) ** a * math.factorial(n - a) / math.factorial(n + a)
        up = P[n][a + 1] if a + 1 <= n else torch.zeros_like(ct)
        tau = -P[n][1] if a == 0 else neg * 0.5 * ((n + a) * (n - a + 1) * P[n][a - 1] - up)
        pi = neg * m * Q[n][a] if m else torch.zeros_like(ct)
        w = (1j if outgoing else -1j) * 1j ** n * _emn(n, m) * (e ** m if m >= 0 else e.conj() ** a)
        u, v = w * c0[..., q], w * c1[..., q]
        if far_only:
            dz = 1j * z[n]
        else:
            Er = Er + n * (n + 1) * neg * P[n][a] * z[n] / x * u
            dz = z[n - 1] - n * z[n] / x
        Et = Et + tau * dz * u + 1j * pi * z[n] * v
        Ep = Ep + 1j * pi * dz * u - tau * z[n] * v
    cp, sp = e.real, e.imag
    rho_part = Er * st + Et * ct
    return torch.stack([rho_part * cp - Ep * sp, rho_part * sp + Ep * cp, Er * ct - Et * st], -1)


def _field_exact(pos, rad, k, k_int, p_scat, p_int, pts, L, hfac, hint, swap, terms=2_000_000):
    """Sum of the outgoing expansions at pts [P, 3], or the interior one inside a sphere."""
    out = torch.empty(pts.shape[0], 3, dtype=torch.complex128, device=pts.device)
    inside = torch.zeros(pts.shape[0], dtype=torch.bool, device=pts.device)
    o, i = (1, 0) if swap else (0, 1)
    step = max(1, terms // pos.shape[0])
    for a in range(0, pts.shape[0], step):
        d = pts[a: a + step, None] - pos[None]
        out[a: a + step] = hfac * _expand(d, p_scat[None, :, o], p_scat[None, :, i], k, L, True).sum(1)
        hit = (d.square().sum(-1) < rad.square())
        at = torch.nonzero(hit.any(1))[:, 0]
        if at.numel():
            s = hit[at].to(torch.int8).argmax(1)
            f = _expand(d[at, s], p_int[s, o], p_int[s, i], k_int[s], L, False)
            out[a + at] = hint * f
            inside[a + at] = True
    return out, inside


def _cluster_exact(c, a):
    """The solved cluster of the sphere_cluster cases."""
    L, k = c["lmax"], 2 * np.pi / a["wavelength"]
    dev = _dev()
    ms, mi = _mie(a["radius"], a["index"], k, L)
    pol = np.array([1, 0.3j]) / math.sqrt(1.09)
    src, E, H, khat = _plane_wave(a["position"], k, L, a["theta"], a["phi"], pol)
    mirror = cells = kh = None
    if a["substrate"]:
        m, ct = a["substrate"], math.cos(a["theta"])
        tt = math.cos(math.asin(math.sin(a["theta"]) / m))
        rpol = pol * [(m * ct - tt) / (m * ct + tt), (ct - m * tt) / (ct + m * tt)]
        nr = np.linalg.norm(rpol)
        src = src + _plane_wave(a["position"], k, L, np.pi - a["theta"], a["phi"], rpol / nr, nr)[0]
        mirror = ((m - 1) / (m + 1), 0.0)
    if a["cell"] is not None:
        if c["square"]:
            n = 35      # the odd square of up to 5000 cells has 71 a side
            cells = np.array([(i, j, 0) for i in range(-n, n + 1) for j in range(-n, n + 1) if i or j], float)
        else:
            cells = np.array([(i, 0, 0) for i in range(-2500, 2501) if i], float)
        cells, kh = torch.tensor(cells * a["cell"], device=dev), torch.tensor(khat, device=dev)
    pos = torch.tensor(a["position"], device=dev)
    M = _operator(pos, ms.to(dev), k, L, mirror, cells, kh)
    N = pos.shape[0]
    p_inc = _solve(M, torch.tensor(src.reshape(-1, 1), device=dev)).reshape(N, 2, -1)
    scat = p_inc * _mie_rows(ms, L).reshape(N, 2, -1).to(dev)
    pint = p_inc * _mie_rows(mi.flip(1), L).reshape(N, 2, -1).to(dev)
    return types.SimpleNamespace(k=k, L=L, pos=pos, src=src, p_inc=p_inc, p_scat=scat, p_int=pint, E=E, H=H)


def _flat(v):
    return v.reshape(-1)


def exact(case, seed):
    c = case
    dev = _dev()
    n = lambda t: t.cpu().numpy()   # noqa: E731
    T = lambda v: torch.tensor(np.ascontiguousarray(v), device=dev)   # noqa: E731
    if c["kind"] == "solve":
        s = _solve_inputs(c, seed)
        N, L, R = c["N"], c["lmax"], c["R"]
        if 2 * L * (L + 2) * N > 20000:
            return None         # a dense operator of over 6 GB
        p = _solve(_operator(T(s["position"]), T(s["mie_scat"]), s["k"], L), T(s["p_src"].reshape(-1, R)))
        p = n(p).reshape(N, 2, -1, R)
        ps = p * n(_mie_rows(T(s["mie_scat"]), L)).reshape(N, 2, -1, 1)
        pi = p * n(_mie_rows(T(s["mie_int"][:, ::-1]), L)).reshape(N, 2, -1, 1)
        xs, F, Tq = _observables(p, ps, s["p_src"], s["k"], L)
        return dict(p_inc=_flat(p), p_scat=_flat(ps), p_int=_flat(pi), xs=_flat(xs), force=_flat(F), torque=_flat(Tq))
    if c["kind"] == "sweep":
        C, parts = [], []
        for s in _sweep_inputs(c, seed):
            N, L = c["N"], s["lmax"]
            p = _solve(_operator(T(s["position"]), T(s["mie_scat"]), s["k"], L), T(s["p_src"].reshape(-1, 1)))
            p = n(p).reshape(N, 2, -1, 1)
            ps = p * n(_mie_rows(T(s["mie_scat"]), L)).reshape(N, 2, -1, 1)
            parts.append(_observables(p, ps, s["p_src"], s["k"], L)[0])
            C.append(parts[-1].sum(axis=(0, 3, 4)))
        C = np.array(C)
        return dict(C=[C[:, :, 0], C[:, :, 1], C[:, :, 2]], per_particle=parts)
    if c["kind"] == "map":
        spec, md, rad, pts = _map_inputs(c, seed)
        L = c["lmax"]
        p = T(spec["p_src"][..., 0])
        N = p.shape[0]
        scat = p * _mie_rows(T(spec["mie_scat"]), L).reshape(N, 2, -1)
        pint = p * _mie_rows(T(spec["mie_int"][:, ::-1]), L).reshape(N, 2, -1)
        h = (-1j, -1j * 2.0) if c["magnetic"] else (1.0, 1.0)
        return _field_exact(T(spec["position"]), T(rad), spec["k"], T(np.full(N, 2.0 * spec["k"])), scat, pint, T(pts),
                            L, h[0], h[1], c["magnetic"], terms=20_000_000)[0]
    a = _cluster_args(c, seed)
    s = _cluster_exact(c, a)
    if c["kind"] in ("substrate", "lattice"):
        N, L = c["N"], c["lmax"]
        p, ps = n(s.p_inc), n(s.p_scat)
        xs, F, Tq = _observables(p[..., None], ps[..., None], s.src.reshape(N, 2, -1, 1), s.k, L)
        return dict(p_inc=p, p_scat=ps, p_int=n(s.p_int), C=xs.sum(axis=(0, 1, 3, 4)),
                    force=F[:, 0], torque=Tq[:, 0])
    if c["kind"] == "field":
        x = np.stack(_plane(a, c["n"]))
        h = (-1j, -1j * a["index"]) if c["magnetic"] else (1.0, 1.0)
        f, inside = _field_exact(s.pos, T(a["radius"]), s.k, T(np.full(c["N"], a["index"] * s.k)), s.p_scat, s.p_int,
                                 T(x.reshape(3, -1).T), s.L, h[0], h[1], c["magnetic"])
        src = (s.H if c["magnetic"] else s.E)(x)
        return n(f).T.reshape(x.shape) + np.where(n(inside).reshape(x.shape[1:]), 0.0, src)
    # pattern
    Lc, N = c["lmax_cluster"], c["N"]
    G = _translation_G(-s.pos, s.k, Lc + s.L, regular=True)
    pc = n(torch.einsum("parbs,pbs->ar", _translation_blocks(G, Lc, s.L), s.p_scat))
    p0 = _plane_wave(np.zeros((1, 3)), s.k, Lc, a["theta"], a["phi"], np.array([1, 0.3j]) / math.sqrt(1.09))[0][0]
    Cs, Ce = np.zeros((2, Lc)), np.zeros((2, Lc))
    for r, (nn, _) in enumerate(_modes(Lc)):
        Cs[:, nn - 1] += 4 * np.pi / s.k ** 2 * np.abs(pc[:, r]) ** 2
        Ce[:, nn - 1] += 4 * np.pi / s.k ** 2 * np.real(np.conj(p0[:, r]) * pc[:, r])
    th, ph, radius = _directions(c["n"])
    u = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], -1).reshape(-1, 3)
    e_t = np.stack([np.cos(th) * np.cos(ph), np.cos(th) * np.sin(ph), -np.sin(th)], -1).reshape(-1, 3)
    e_p = np.stack([-np.sin(ph), np.cos(ph), 0 * ph], -1).reshape(-1, 3)
    res = {}
    for name, (o, i, f) in (("E", (0, 1, 1.0)), ("H", (1, 0, -1j))):
        v = []
        for b in range(0, u.shape[0], 4096):
            d = T(radius * u[b: b + 4096])[:, None] - s.pos[None]
            e = _expand(d, s.p_scat[None, :, o], s.p_scat[None, :, i], s.k, s.L, True, far_only=True)
            v.append(n(f * e.sum(1)))
        v = np.concatenate(v)
        res[name] = np.stack([(v * e_t).sum(-1), (v * e_p).sum(-1)]).reshape((2,) + th.shape)
    return dict(p_cluster=pc, C=[Cs, Ce - Cs, Ce], E=res["E"], H=res["H"])
