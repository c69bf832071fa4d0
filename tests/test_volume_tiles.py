"""The volume kernels' tiles at the sizes where they change shape: interior
boxes whose width leaves 0, 1, 8 (the most that join the x PML slab), 9 or
31 columns beyond whole 32-point tiles, odd strike and depth sizes (a last
block of each plane with one row at work), against the CPU oracle; and the
small grids' schedule, with the boundary kinds in one launch, against the
separate kernels'."""
import numpy as np
import pytest

import inputs
from cgfd import Solver, WAVE_COMPONENTS
from oracle import OracleSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left", [0, 1, 8, 9, 31])
def test_leftover_columns(cgfd_lib, oracle_built, left):
    # 5-layer PML faces take 6 columns at either side; the fault's
    # neighbourhood lies in the first tile
    p = inputs.tpv_planar(ni=12 + 32 + left, nj=61, nk=37, fault_x_index=20, fault_grid=[15, 46, 12, 37], nuc_half=3,
                          pml=5, nt=10, nsta=4, margin=10)
    rng = np.random.default_rng(left)
    g, o = Solver(p), OracleSolver(p)
    wide = 32 if 0 < left <= 8 else 32 + left
    rows = [61 - 12, 37 - 6 - 4]
    assert wide * rows[0] * rows[1] - 7 * rows[0] * rows[1] < g.kernel_timing(1)[2] <= wide * rows[0] * rows[1]
    for c in range(9):
        f = (rng.standard_normal((p.nk, p.nj, p.ni)) * (1e-3 if c < 3 else 1e3)).astype(np.float32)
        g.set_wavefield(c, f)
        o.set_wavefield(c, f)
    g.run(8)
    o.run(8)
    for c in range(9):
        a, b = g.wavefield(c), o.wavefield(c)
        # the float32 bound of the parity tests' random-state steps
        assert np.linalg.norm(a - b) <= 2e-5 * np.linalg.norm(b), WAVE_COMPONENTS[c]


def _cases():
    yield "free", inputs.small_planar(nt=20)
    yield "buried, continuity matrices", inputs.small_planar(nt=20, dynamic_method=1, free_surface=0)
    # split nodes up to the PML: the fault planes that wait for them lie in
    # the PML slab, edge and shell boxes too
    yield "fault in the PML", inputs.small_planar(nt=20, margin=6)
    yield "two faults", inputs.two_faults(nt=20)
    p = inputs.small_planar(nt=20, ni=37, nj=59, nk=33, fault_grid=[9, 48, 9, 33], nuc_center=(27, 22))
    yield "odd sizes", p


@pytest.mark.parametrize("name", [n for n, _ in _cases()])
def test_merged_boundary_launch(cgfd_lib, oracle_built, monkeypatch, name):
    """The kinds' code is the same in both schedules: equal bit for bit, and
    to the oracle within the rupture tests' 1e-4."""
    p = dict(_cases())[name]
    runs = []
    for m in ("0", "1"):
        monkeypatch.setenv("CGFD_MERGED", m)
        g = Solver(p)
        rng = np.random.default_rng(3)
        for c in range(9):
            g.set_wavefield(c, (rng.standard_normal((p.nk, p.nj, p.ni)) * (1e-3 if c < 3 else 1e3)).astype(np.float32))
        g.run(9)
        g.run_noalloc(8)
        runs.append(g)
    apart, together = runs
    assert together.last_launches() < apart.last_launches()
    o = OracleSolver(p)
    rng = np.random.default_rng(3)
    for c in range(9):
        o.set_wavefield(c, (rng.standard_normal((p.nk, p.nj, p.ni)) * (1e-3 if c < 3 else 1e3)).astype(np.float32))
    o.run(17)
    for c in range(9):
        a, b = apart.wavefield(c), together.wavefield(c)
        assert np.array_equal(a, b), WAVE_COMPONENTS[c]
        r = o.wavefield(c)
        assert np.linalg.norm(b - r) <= 1e-4 * np.linalg.norm(r), WAVE_COMPONENTS[c]
    for f in range(p.num_faults):
        assert np.array_equal(apart.fault_all(f), together.fault_all(f)), f
    assert np.array_equal(apart.stations(), together.stations())


@pytest.mark.parametrize("name", ["extruded", "hills", "sheared"])
def test_aligned_grid_kernels(cgfd_lib, oracle_built, monkeypatch, name):
    """Grids whose x and y lines keep to their axis leave the metric's four
    off-axis entries out (extruded planar grid, hills); on a sheared one the
    general kernels run.  What is left out is below 2^-40 of the entries kept,
    so the two agree to rounding: the 1e-6 of the other rounding-only
    variants."""
    if name == "extruded":
        p = inputs.small_planar(nt=20)
    else:
        p = inputs.hills_layered(ni=40, nj=57, nk=33, pml=5, nsta=4, fault_len=36, fault_depth=20, margin=9, nt=20,
                                 nhills=3, nuc_half=2, dip=60.0 if name == "sheared" else None)
    runs = []
    for al in ("0", "1"):
        monkeypatch.setenv("CGFD_ALIGNED", al)
        g = Solver(p)
        rng = np.random.default_rng(5)
        for c in range(9):
            g.set_wavefield(c, (rng.standard_normal((p.nk, p.nj, p.ni)) * (1e-3 if c < 3 else 1e3)).astype(np.float32))
        g.run(17)
        runs.append(g)
    same = True
    for c in range(9):
        a, b = (g.wavefield(c) for g in runs)
        same &= np.array_equal(a, b)
        assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(a), WAVE_COMPONENTS[c]
    # rounding differs where the aligned kernels ran, and only there
    assert same == (name == "sheared")


@pytest.mark.parametrize("pml", [0, 5])
def test_getter_and_setter_leave_the_step_alone(cgfd_lib, pml):
    """Wavefield reads and writes stage a component in a level that is dead
    between steps; its ghost points, which taps at the grid's sides read, must
    be zero again afterwards.  37x59x33 points: rows that fill no tile."""
    p = inputs.small_planar(nt=20, ni=37, nj=59, nk=33, fault_grid=[9, 48, 9, 33], nuc_center=(27, 22), pml=pml)
    rng = np.random.default_rng(1)
    f = [(rng.standard_normal((p.nk, p.nj, p.ni)) * (1e-3 if c < 3 else 1e3)).astype(np.float32) for c in range(9)]
    g, h = Solver(p), Solver(p)
    for s in (g, h):
        for c in range(9):
            s.set_wavefield(c, f[c])
    for c in range(9):
        assert np.array_equal(g.wavefield(c), f[c]), WAVE_COMPONENTS[c]
    g.run(8)
    for _ in range(8):
        h.run(1)
        for c in (0, 8):
            h.set_wavefield(c, h.wavefield(c))
    for c in range(9):
        assert np.array_equal(g.wavefield(c), h.wavefield(c)), WAVE_COMPONENTS[c]
