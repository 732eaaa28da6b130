"""Kernel forms against each other at the sizes where tiles, chunks and copies end.

Tolerances: FP32 forms of one update (different summation order and FMA contraction), two steps
from a random state: max |diff| <= 2e-5 x max |ref| per component, as against the oracle. FP64 forms:
equal to double rounding, so their read-back floats differ by one unit in the last place at most:
1.2e-7 x max |ref|. Forms that only cut the work differently: bitwise.
"""
import numpy as np
import pytest

import cgfd_b200
from cgfd_b200 import Simulation, media_layer_gpu, CGFD_MEDIA_ARI, CGFD_MEDIA_HAR, CGFD_PREC_FP64
from cgfd_b200 import CGFD_MEDIA_LOC
from cgfd_b200.abi import Sources, media_layer_any_gpu
from cgfd_b200.formats import LayerMedia, LayerModel
from helpers import small_problem, random_wavefield
from perf import cases

pytestmark = pytest.mark.gpu

# smaller than a tile, one point over a tile in x / y, several tiles with remainders
GRIDS = [(9, 8, 13), (33, 37, 21), (70, 41, 34)]


def _two_steps(p, shots=None, variant=None, setup=None):
    sim = Simulation(p, shots)
    if variant is not None:
        sim.set_bulk_variant(variant)
    if setup:
        setup(sim)
    for s in range(sim.nshot):
        sim.set_wavefield(random_wavefield(p, seed=3 + s), s)
    sim.run(2)
    return [sim.wavefield(s) for s in range(sim.nshot)]


def _close(a, b, tol):
    for c in range(9):
        scale = float(np.abs(b[c]).max())
        assert float(np.abs(a[c] - b[c]).max()) <= tol * scale, f"component {c}"


@pytest.mark.parametrize("medium", ["iso", "vti", "aniso", "ac"])
@pytest.mark.parametrize("grid", GRIDS + [(101, 64, 48)])
def test_default_chunk_changes_no_result(medium, grid):
    p = small_problem(medium, *grid, nsteps=4, npml=3, nsrc=1)
    (a,), (b,) = _two_steps(p), _two_steps(p, setup=lambda s: s.set_zchunk(12))
    np.testing.assert_array_equal(a, b)


# a field below the staged copy's least size, one of a single chunk, one of a chunk and a remainder
@pytest.mark.parametrize("grid", [(40, 36, 30), (120, 100, 70), (300, 280, 210)])
def test_wavefield_readback_equals_box(grid):
    p = small_problem("iso", *grid, nsteps=2, npml=0, nsrc=0, sta_grid=None)
    sim = Simulation(p)
    rng = np.random.default_rng(1)
    w = np.zeros((9,) + tuple(n + 6 for n in grid[::-1]), np.float32)
    w[:, 3:-3, 3:-3, 3:-3] = rng.standard_normal((9,) + grid[::-1], dtype=np.float32)
    sim.set_wavefield(w)
    out = sim.wavefield()
    np.testing.assert_array_equal(out, w)
    np.testing.assert_array_equal(out[:, 3:-3, 3:-3, 3:-3], sim.wavefield_box((0, 0, 0), grid))


@pytest.mark.parametrize("method", [CGFD_MEDIA_HAR, CGFD_MEDIA_ARI])
@pytest.mark.parametrize("dims", [(8, 8, 8), (19, 11, 14)])
def test_layer_averages_at_mixed_points(method, dims):
    """Flat layers on a Cartesian grid: the 9^3 sub-points of a mixed half-grid cell lie on 9
    elevations, those within 1 m of an interface take the mean of both layers (the reference's
    integer test). A float sum of 729 terms is within 729 x 2^-24 = 4.4e-5 of the exact one."""
    ni, nj, nk = dims
    dh = 100.0
    coord = np.zeros((3, nk + 6, nj + 6, ni + 6), np.float32)
    coord[0] = (np.arange(-3, ni + 3) * dh)[None, None, :]
    coord[1] = (np.arange(-3, nj + 3) * dh)[None, :, None]
    coord[2] = (np.arange(-3, nk + 3) * dh - (nk - 1) * dh)[:, None, None]
    tops = [float(coord[2].max()) + 500.0, -233.0, -512.0]
    par = {"vp": [4000.0, 5500.0, 6500.0], "vs": [2300.0, 3200.0, 3750.0], "rho": [2500.0, 2700.0, 2900.0]}
    shape = (3, 4, 5)
    f = {"elevation": np.array(tops, np.float32)[:, None, None] * np.ones(shape, np.float32)}
    for n, v in par.items():
        f[n] = np.array(v, np.float32)[:, None, None] * np.ones(shape, np.float32)
        f[n + "_grad"] = np.zeros(shape, np.float32)
        f[n + "_pow"] = np.ones(shape, np.float32)
    m = LayerModel(float(coord[0].min()) - 50, float(coord[1].min()) - 50, 1000.0, 1000.0, **f)
    got = media_layer_gpu(coord, m, method)

    def values(z):  # (rho, lambda, mu) at elevation z
        n = max(q for q in range(3) if tops[q] >= z)
        layers = [n - 1, n] if n > 0 and int(tops[n] - z) == 0 else [n]
        rho, vp, vs = (np.mean([par[k][q] for q in layers]) for k in ("rho", "vp", "vs"))
        return np.array([rho, rho * vp * vp - 2 * rho * vs * vs, rho * vs * vs])

    mixed = 0
    for k in range(1, nk + 5):
        z = float(coord[2, k, 0, 0])
        lo, hi = z - dh / 2, z + dh / 2
        if max(q for q in range(3) if tops[q] >= lo) == max(q for q in range(3) if tops[q] >= hi):
            want = values(z)
        else:
            mixed += 1
            v = np.array([values(lo + (hi - lo) / 8 * s) for s in range(9)])
            want = v.mean(0)
            if method == CGFD_MEDIA_HAR:
                mu = 1 / np.mean(1 / v[:, 2])
                want = np.array([want[0], 1 / np.mean(1 / (v[:, 1] + 2 / 3 * v[:, 2])) - 2 / 3 * mu, mu])
        np.testing.assert_allclose(got[:, k, 1:-1, 1:-1], want[:, None, None] * np.ones((3, nj + 4, ni + 4)), rtol=5e-5)
    assert mixed >= 2


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("nmax", [1, 3, 4, 5])
@pytest.mark.parametrize("free_top", [0, 1])
def test_visco_fused_equals_separate_passes(nmax, grid, free_top):
    p = small_problem("vis", *grid, nsteps=4, npml=3, free_top=free_top, nsrc=0)
    p.visco["nmaxwell"] = nmax
    (a,), (b,) = _two_steps(p), _two_steps(p, variant=0)
    _close(a, b, 2e-5)


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("medium", ["iso", "vti"])
@pytest.mark.parametrize("free_top", [0, 1])
def test_fp64_tma_equals_direct(medium, grid, free_top):
    p = small_problem(medium, *grid, nsteps=4, npml=3, free_top=free_top, nsrc=0)
    p.precision = CGFD_PREC_FP64
    (a,), (b,) = _two_steps(p), _two_steps(p, variant=0)
    _close(a, b, 1.2e-7)


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("free_top", [0, 1])
@pytest.mark.parametrize("nshot", [1, 3])
def test_acoustic_tiles_equal_direct(grid, free_top, nshot):
    p = small_problem("ac", *grid, nsteps=4, npml=3, free_top=free_top, nsrc=1)
    shots = [p.src] * nshot if nshot > 1 else None
    for a, b in zip(_two_steps(p, shots), _two_steps(p, shots, variant=0)):
        _close(a, b, 2e-5)  # components 4-8 stay 0 in both


# inside a tile; across tile corners in x, y and z chunks; clipped by the grid's edge; reaching into the
# surface slab's planes (then the source kernel runs); two that overlap
@pytest.mark.parametrize("at", [[(40, 17, 9)], [(31, 8, 12)], [(0, 1, 2)], [(40, 17, 26)], [(33, 18, 11), (35, 20, 12)]])
@pytest.mark.parametrize("medium,precision,tol", [("iso", 0, 2e-5), ("vis", 0, 2e-5), ("iso", CGFD_PREC_FP64, 1.2e-7)])
@pytest.mark.parametrize("cmp_type", [1, 2])
def test_sources_in_tiles_equal_source_kernel(at, medium, precision, tol, cmp_type):
    n, steps = len(at), 5
    p = small_problem(medium, 70, 41, 30, nsteps=steps, npml=3, nsrc=0)
    p.precision = precision
    rng = np.random.default_rng(2)
    cmp = rng.uniform(-1, 1, (n, 9)).astype(np.float32) * np.array([1e12] * 3 + [1e16] * 6, np.float32)
    coefs = np.zeros((n, 10), np.float32)
    coefs[:, 0], coefs[:, 1] = 3.0, 0.02
    p.src = Sources(loc=np.array(at, np.float32), t_start=np.zeros(n, np.float32), wavelet=np.zeros(n, np.int32),
                    wavelet_coefs=coefs, cmp=cmp, stf_length=3 * p.dt, cmp_type=cmp_type)
    out = []
    for variant in (None, 0):
        sim = Simulation(p)
        if variant is not None:
            sim.set_bulk_variant(variant)
        sim.run(steps)  # the time function ends before the run does
        out.append(sim.wavefield())
    assert np.abs(out[1]).max() > 0
    _close(out[0], out[1], tol)


@pytest.mark.parametrize("medium", ["iso", "aniso", "ac"])
def test_fp64_batch_equals_its_shots_alone(medium):
    p = small_problem(medium, 40, 37, 30, nsteps=8, npml=4, nsrc=1)
    p.precision = CGFD_PREC_FP64
    waves = [random_wavefield(p, seed=s) for s in (1, 2, 3)]
    if medium == "ac":
        for w in waves:
            w[4:] = 0

    def run(shots, state):
        with Simulation(p, shots) as sim:
            for s, w in enumerate(state):
                sim.set_wavefield(w, s)
            sim.run(4)
            return [sim.wavefield(s) for s in range(sim.nshot)]
    for got, w in zip(run([p.src] * 3, waves), waves):
        np.testing.assert_array_equal(got, run(None, [w])[0])


def _point_sources(p, at, amp=1.0):
    n = len(at)
    rng = np.random.default_rng(2)
    cmp = amp * rng.uniform(-1, 1, (n, 9)).astype(np.float32) * np.array([1e12] * 3 + [1e16] * 6, np.float32)
    coefs = np.zeros((n, 10), np.float32)
    coefs[:, 0], coefs[:, 1] = 3.0, 0.02
    return Sources(loc=np.array(at, np.float32), t_start=np.zeros(n, np.float32), wavelet=np.zeros(n, np.int32),
                   wavelet_coefs=coefs, cmp=cmp, stf_length=6 * p.dt, cmp_type=3)


INSIDE, CORNER = (40, 20, 14), (2, 2, 12)


# shots' sources; launches of the source kernel a step (0: the tiles inject)
@pytest.mark.parametrize("at,launches", [([[INSIDE]], 0), ([[INSIDE, (44, 22, 12)]], 4), ([[CORNER]], 4), ([[(40, 20, 25)]], 4),
                                         ([[INSIDE], [(38, 14, 16)], [(44, 22, 9)]], 0), ([[INSIDE], [CORNER]], 4),
                                         ([[INSIDE]] * 32, 0), ([[INSIDE]] * 33, 4)])
def test_route_of_sources(at, launches):
    p = small_problem("iso", 80, 41, 30, nsteps=2, npml=4, nsrc=0)
    shots = [_point_sources(p, a) for a in at]
    p.src = shots[0]
    sim = Simulation(p, shots if len(shots) > 1 else None)
    sim.set_timing(True)
    sim.run(1)
    assert sim.timing()["source"][1] == launches


@pytest.mark.parametrize("precision", ["CGFD_PREC_FP32", "CGFD_PREC_U16_COEF", "CGFD_PREC_FP64"])
@pytest.mark.parametrize("nshot", [1, 3])
def test_tiles_inject_what_the_source_kernel_does(precision, nshot):
    """A second source of zero moment sends a problem to the source kernel and adds nothing: bitwise."""
    p = small_problem("iso", 80, 41, 30, nsteps=8, npml=4, nsrc=0, sta_grid=None)
    p.precision = getattr(cgfd_b200, precision)
    out = []
    for more in (False, True):
        shots = [_point_sources(p, [(40 + s, 20, 14 - s)]) for s in range(nshot)]
        if more:
            shots[-1] = _point_sources(p, [(39 + nshot, 20, 15 - nshot), (44, 22, 12)])
            shots[-1].cmp[0] = _point_sources(p, [(40, 20, 14)]).cmp[0]
            shots[-1].cmp[1] = 0
        p.src = shots[0]
        with Simulation(p, shots if nshot > 1 else None) as sim:
            sim.run(8)  # the time function ends before the run does
            out.append([sim.wavefield(s) for s in range(nshot)])
            sim.set_timing(True)
            sim.run(1)
            assert sim.timing()["source"][1] == (4 if more else 0)
    for a, b in zip(*out):
        assert np.abs(b).max() > 0
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("shots", [0, 3])
def test_tiles_inject_what_the_source_kernel_does_in_mixed_storage(shots):
    """The same with FP16 stage levels, whose scale the injecting threads feed, from a wavefield and
    sources of the tracked workloads (a source that starts at its full rate in a zero wavefield can
    outgrow the scale's headroom within its first step, by either route)."""
    c = cases._sim("run", "iso", 96, 80, 40, 16, 6, precision="mixed", shots=shots)
    p, sources, waves = cases._inputs(c, 3)
    sources = sources or [p.src]
    out = []
    for more in (False, True):
        if more:
            s = sources[-1]
            sources[-1] = Sources(loc=np.concatenate([s.loc, s.loc + 2]), t_start=np.zeros(2, np.float32), wavelet=np.zeros(2, np.int32),
                                  wavelet_coefs=np.repeat(s.wavelet_coefs, 2, 0), cmp=np.concatenate([s.cmp, 0 * s.cmp]),
                                  stf_length=s.stf_length, cmp_type=s.cmp_type)
        p.src = sources[0]
        with Simulation(p, sources if shots else None) as sim:
            for s, w in enumerate(waves):
                sim.set_wavefield(w, s)
            sim.run(15)
            out.append([sim.wavefield(s) for s in range(sim.nshot)])
            sim.set_timing(True)
            sim.run(1)
            assert sim.timing()["source"][1] == (4 if more else 0)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("method", [CGFD_MEDIA_LOC, CGFD_MEDIA_HAR, CGFD_MEDIA_ARI])
@pytest.mark.parametrize("medium", ["ac", "iso"])
def test_layer_averages_with_gradients_and_powers(method, medium):
    """Flat layers whose parameters rise with depth by powers 0, 1, 2 and between (dz^pow gradient in
    double), on a Cartesian grid, isotropic and acoustic files, against the same sums in 64 bits. An
    interface lies half a metre above a sub-point: the reference's integer test then takes the mean of
    both layers. Tolerance: as above, 729 x 2^-24 of the sum, and a few roundings of the values."""
    ni, nj, nk, dh = 9, 12, 17, 100.0
    coord = np.zeros((3, nk + 6, nj + 6, ni + 6), np.float32)
    coord[0] = (np.arange(-3, ni + 3) * dh)[None, None, :]
    coord[1] = (np.arange(-3, nj + 3) * dh)[None, :, None]
    coord[2] = (np.arange(-3, nk + 3) * dh - (nk - 1) * dh)[:, None, None]
    tops = [float(coord[2].max()) + 500.0, -237.0, -612.0, -1099.5]
    vals = {"rho": ([2500.0, 2600.0, 2700.0, 2900.0], [10.0, 0.02, 1e-5, 0.3], [0.0, 1.0, 2.0, 0.5]),
            "vp": ([4000.0, 4800.0, 5500.0, 6500.0], [0.4, 1.0, 30.0, 1e-4], [0.5, 0.75, 0.0, 2.0]),
            "vs": ([2300.0, 2700.0, 3200.0, 3750.0], [1e-4, 0.02, 0.3, 5.0], [2.0, 1.0, 0.5, 0.0])}
    names = ("rho", "vp") if medium == "ac" else ("rho", "vp", "vs")
    shape = (4, 4, 5)
    flat = lambda v: np.array(v, np.float32)[:, None, None] * np.ones(shape, np.float32)  # noqa: E731
    param = np.stack([np.stack([flat(v) for v in vals[n]]) for n in names])
    m = LayerMedia(10 if medium == "ac" else 21, float(coord[0].min()) - 50, float(coord[1].min()) - 50, 1000.0, 1000.0,
                   flat(tops), param)
    got = media_layer_any_gpu(coord, m, 1 if medium == "ac" else 2, method)

    def at(name, layer, dz):
        v, g, p = (float(np.float32(q[layer])) for q in vals[name])
        return v + dz ** p * g

    def values(z):  # (rho, kappa) or (rho, lambda, mu) at elevation z
        n = max(q for q in range(4) if tops[q] >= z)
        layers = [n - 1, n] if n > 0 and int(tops[n] - z) == 0 else [n]
        # (acoustic files: the layer above at the depth below the lower interface, as the reference does)
        dz = {q: tops[n if medium == "ac" else q] - z for q in layers}
        v = [np.mean([at(name, q, dz[q]) for q in layers]) for name in names]
        if medium == "ac":
            return np.array([v[0], v[0] * v[1] ** 2])
        return np.array([v[0], v[0] * v[1] ** 2 - 2 * v[0] * v[2] ** 2, v[0] * v[2] ** 2])

    mixed = 0
    for k in range(1, nk + 5):
        z = float(coord[2, k, 0, 0])
        lo, hi = z - dh / 2, z + dh / 2
        if method == CGFD_MEDIA_LOC or len({max(q for q in range(4) if tops[q] >= e) for e in (lo, hi)}) == 1:
            want = values(z)
        else:
            mixed += 1
            v = np.array([values(lo + (hi - lo) / 8 * s) for s in range(9)])
            want = v.mean(0)
            if method == CGFD_MEDIA_HAR and medium == "ac":
                want[1] = 1 / np.mean(1 / v[:, 1])
            elif method == CGFD_MEDIA_HAR:
                mu = 1 / np.mean(1 / v[:, 2])
                want = np.array([want[0], 1 / np.mean(1 / (v[:, 1] + 2 / 3 * v[:, 2])) - 2 / 3 * mu, mu])
        np.testing.assert_allclose(got[:, k, 1:-1, 1:-1], want[:, None, None] * np.ones((len(want), nj + 4, ni + 4)),
                                   rtol=5e-5, err_msg=f"plane {k}")
    assert mixed == (0 if method == CGFD_MEDIA_LOC else 3)


@pytest.mark.parametrize("nmax", [1, 3, 4, 5])
@pytest.mark.parametrize("free", [True, False])
def test_visco_against_64_bits(nmax, free):
    """The attenuation of the fused kernel (up to 4 mechanisms) and of the separate pass against a
    restatement in 64 bits that shares no code with them; 1e-5 x max |ref| per component and FP32 step."""
    c = cases._sim("run", "vis", 70, 45, 37, 16, 6, free=free, nmax=nmax)
    p, _, (wave,) = cases._inputs(c, 11)
    ref = cases._Run64(c, p, p.src, wave)
    with Simulation(p) as sim:
        sim.set_wavefield(wave)
        sim.run(5)
        got = sim.wavefield()[:, 3:-3, 3:-3, 3:-3]
    for it in range(5):
        ref.step(it)
    _close(got, ref.pre[:, 3:-3, 3:-3, 3:-3].cpu().numpy(), 5e-5)
