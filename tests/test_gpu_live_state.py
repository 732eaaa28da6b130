"""Calls that change a problem which holds live state, and what runs beside it."""
import numpy as np
import pytest

from cgfd_b200 import Simulation
from perf import cases

pytestmark = pytest.mark.gpu


def _case(medium, shots=0, **kw):
    c = cases._sim("run", medium, 44, 41, 36, 16, 6, shots=shots, **kw)
    return (c,) + cases._inputs(c, 5)


def _close(a, b, tol):
    for c in range(9):
        scale = float(np.abs(b[c]).max())
        assert float(np.abs(a[c] - b[c]).max()) <= tol * scale, f"component {c}"


@pytest.mark.parametrize("medium,kw", [("iso", {}), ("vti", {"free": False}), ("ac", {}), ("vis", {"nmax": 2}),
                                       ("vis", {"nmax": 5}), ("iso", {"precision": "fp64"})])
def test_set_step_to_the_other_parity_keeps_live_state(medium, kw):
    """Steps 0 1 2, then 6 7: the wavefield, the CFS-PML auxiliaries and the memory variables of the
    problem move to the levels of the new parity. Against the same steps in 64 bits; tolerance: 1e-5 x
    max |ref| per component and FP32 step, as of the kernels' forms against each other."""
    c, p, _, (wave,) = _case(medium, **kw)
    ref = cases._Run64(c, p, p.src, wave)
    with Simulation(p) as sim:
        sim.set_wavefield(wave)
        sim.run(3)
        sim.set_step(6)
        sim.run(2)
        got = sim.wavefield()[:, 3:-3, 3:-3, 3:-3]
    for it in (0, 1, 2, 6, 7):
        ref.step(it)
    want = np.zeros(got.shape)
    want[: ref.nf] = ref.pre[:, 3:-3, 3:-3, 3:-3].cpu().numpy()
    _close(got, want, 5e-5)


@pytest.mark.parametrize("medium,shots,kw", [("iso", 3, {}), ("ac", 3, {}), ("vis", 0, {"nmax": 3}), ("iso", 0, {"precision": "fp64"})])
def test_settings_hold_from_the_next_step_on(medium, shots, kw):
    """The tile lists, line receivers and slices of a problem that is running, replaced without a wait
    before or after: every step reads complete ones. Cutting the work differently changes no result."""
    c, p, sources, waves = _case(medium, shots, **kw)
    points = [(i, 7 + i % 30, 20 + i % 16) for i in range(40)]

    def run(change):
        with Simulation(p, sources) as sim:
            for s, w in enumerate(waves):
                sim.set_wavefield(w, s)
            sim.enqueue(2)
            sim.set_line_receivers(points)
            sim.set_slices(iz=[35, 3], ring_steps=16)
            for n, z in enumerate((5, 40, 3, 11)):
                if change:
                    sim.set_zchunk(z)
                    if shots:
                        sim.set_shot_group(1 + n % 3)
                    if medium == "iso" and not kw:
                        sim.set_tile_shape(n % 2)
                sim.enqueue(3)
            sim.synchronize()
            return ([sim.wavefield(s) for s in range(sim.nshot)], sim.seismograms(), sim.line_seismograms(),
                    [sim.slices(it)[2] for it in range(2, 14)])

    def flat(v):
        return sum((flat(q) for q in v), []) if isinstance(v, (list, tuple)) else [v]
    for a, b in zip(flat(run(True)), flat(run(False)), strict=True):
        np.testing.assert_array_equal(a, b)
