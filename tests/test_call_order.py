"""What the calls put on which stream, and in which order.

On the CPU: the library's objects linked with a CUDA runtime that records
instead of running (recording_cudart.cpp), so that an ordering that a test run
on an idle GPU would hardly ever break is seen from the calls themselves.  On
the GPU: the same call sequences against their plain counterparts."""
import ctypes
import glob
import os
import re
import subprocess

import numpy as np
import pytest

import inputs
from conftest import PKG, TESTS


def on_recording_runtime(d, kind):
    """The library of the build's *.cu{kind}.o objects on the recording runtime."""
    import cgfd
    obj, lib = str(d / "recording_cudart.o"), str(d / "libcgfd_recording.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-I/usr/local/cuda/include", "-c",
                           os.path.join(TESTS, "recording_cudart.cpp"), "-o", obj])
    built = sorted(glob.glob(os.path.join(PKG, "_build", f"*.cu{kind}.o"))) + [os.path.join(PKG, "_build", "setup.cpp.o")]
    subprocess.check_call(["g++", "-shared", "-Wl,-Bsymbolic", "-o", lib] + built + [obj, "-lgomp"])
    r = cgfd.load_library(lib)
    r.recording_log.restype = ctypes.c_char_p
    return r


@pytest.fixture(scope="module")
def recording(cgfd_lib, tmp_path_factory):
    return on_recording_runtime(tmp_path_factory.mktemp("recording"), "")


@pytest.fixture(scope="module")
def recording64(cgfd_lib, tmp_path_factory):
    return on_recording_runtime(tmp_path_factory.mktemp("recording64"), "64")


def operations(lib, clear=True):
    """The log as (op, stream, rest...) tuples."""
    ops = [tuple(line.split()) for line in lib.recording_log().decode().splitlines()]
    if clear:
        lib.recording_clear()
    return ops


def unordered_before_graphs(ops):
    """(graph launch, earlier device operation on another stream) pairs that
    nothing orders: no event wait, no wait of the host.  What lies inside a
    capture belongs to the graph's own launch."""
    host, after, events, work, found = set(), {}, {}, [], []
    capturing = False
    for n, (op, st, *rest) in enumerate(ops):
        if op in ("begin", "end"):
            capturing = op == "begin"
        if capturing or op == "end":
            continue
        known = after.setdefault(st, set())
        known |= host
        if op == "record":
            events[rest[0]] = set(known)
        elif op == "wait":
            known |= events.get(rest[0], set())
        elif op == "sync":
            host |= known
        else:
            if op == "graph":
                found += [((n, op, st), (w,) + ops[w][:2]) for w in work if w not in known]
            work.append(n)
            known.add(n)
            if op == "blockcopy":
                host.add(n)
    return found


def kernel(name):
    """Short name of a launched kernel; k_volume with its kind."""
    kind = re.search(r"k_volumeI(?:Li\dE){4}Li(\d)E", name)
    return f"k_volume {kind.group(1)}" if kind else re.search(r"k_(?:fault_)?[a-z]+(?:_[a-z]+)?", name).group(0)


def clear_of_the_pml(nt=20):
    """A fault whose neighbourhood (i0 +- 6, split box + 3 nodes) stays clear of
    every PML slab and edge box, as on the large workloads, on a grid small
    enough that the boundary kinds run in one launch by default."""
    p = inputs.tpv_planar(ni=40, nj=80, nk=40, fault_x_index=21, fault_grid=[25, 56, 15, 40], nuc_half=3,
                          pml=5, nt=nt, nsta=4, margin=10)
    i0 = p.fault_x_index[0] - 1
    assert i0 - 6 > 5 and i0 + 6 < p.ni - 6 and p.welded_margin - 3 > 5
    return p


def closed_box(**kw):
    """A small rupture without a free surface (whose steps the recording
    runtime counts)."""
    return inputs.small_planar(nt=20, free_surface=0, **kw)


def test_ensemble_waits_for_its_members_streams(recording, monkeypatch):
    """The wavefield getter leaves a clear on its member's stream; the next
    ensemble steps start on a stream of their own and write what it clears."""
    import cgfd
    monkeypatch.setattr(cgfd, "load_library", lambda *a: recording)
    members = [cgfd.Solver(closed_box(seed=q), lib=recording) for q in (7, 8)]
    ens = cgfd.Ensemble(members)
    operations(recording)
    ens.run(2)
    members[1].wavefield("Vx")
    ens.run(1)
    ops = operations(recording)
    assert [o[0] for o in ops].count("graph") == 3 and any(o[0] == "set" for o in ops)
    assert unordered_before_graphs(ops) == []
    ens.close()


@pytest.mark.gpu
def test_ensemble_after_a_wavefield_read(cgfd_lib):
    """Members read between two runs of their ensemble go on as those that
    are stepped alone and never read."""
    from cgfd import Ensemble, Solver, WAVE_COMPONENTS
    probs = inputs.ensemble_scenarios(3, seed=11, nt=24, size_lo=(36, 60, 36), size_hi=(48, 80, 44), pml=5, margin=6)
    alone, members = [Solver(p) for p in probs], [Solver(p) for p in probs]
    ens = Ensemble(members)
    for n in (5, 1, 6):
        ens.run(n)
        for m in members:
            for c in WAVE_COMPONENTS:
                m.wavefield(c)
    for s, m in zip(alone, members):
        s.run(12)
        for c in WAVE_COMPONENTS:
            assert np.array_equal(s.wavefield(c), m.wavefield(c)), c
        assert np.array_equal(s.fault_all(), m.fault_all())
    ens.close()


def test_which_schedule_a_switch_gives(recording, monkeypatch):
    """Without the one boundary launch of small grids the next stage's first
    fault kernels are issued before a stage's PML kernels (what every large
    grid does), with CGFD_PRE_EARLY=0 after them."""
    from cgfd import Solver
    p = clear_of_the_pml()

    def step(**env):
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        s = Solver(p, lib=recording)
        for k in env:
            monkeypatch.delenv(k)
        ops = operations(recording)
        s.close()
        first = next(n for n, o in enumerate(ops) if o[0] == "begin")
        last = next(n for n, o in enumerate(ops) if o[0] == "end")
        return [(kernel(o[2]), o[1]) for o in ops[first:last] if o[0] == "launch"]

    assert any(k == "k_volume_all" for k, _ in step())
    for env, early in (({"CGFD_MERGED": "0"}, True), ({"CGFD_PRE_EARLY": "0"}, False)):
        launches = step(**env)
        names = [k for k, _ in launches]
        assert "k_volume_all" not in names
        pre = [n for n, k in enumerate(names) if k == "k_fault_pre"]
        face_x = [n for n, k in enumerate(names) if k == "k_volume 2"]
        assert len(pre) == len(face_x) == 4
        assert [pre[n + 1] < face_x[n] for n in range(3)] == [early] * 3
        # three branches, the fault's on a stream of its own
        assert len({st for _, st in launches}) == 3


@pytest.mark.gpu
@pytest.mark.parametrize("serial", [("CGFD_PRE_EARLY", "0"), ("CGFD_BRANCHES", "0")])
def test_early_schedule_is_the_serial_one_bit_for_bit(cgfd_lib, monkeypatch, serial):
    """The schedule that large grids run (three branches, the fault kernels
    beside the interior and ahead of the PML kernels, the slabs right after
    them), here with CGFD_MERGED=0, against the same kernels one after the
    other."""
    from cgfd import Solver, WAVE_COMPONENTS
    p = clear_of_the_pml(nt=60)
    monkeypatch.setenv("CGFD_MERGED", "0")
    early = Solver(p)
    monkeypatch.setenv(*serial)
    other = Solver(p)
    for s in (early, other):
        s.run(60)
    assert early.fault("Vs").max() > 0.1
    for f in ("Vs", "Slip", "Tn", "Ts1"):
        assert np.array_equal(early.fault(f), other.fault(f)), f
    for c in WAVE_COMPONENTS:
        assert np.array_equal(early.wavefield(c), other.wavefield(c)), c
    assert np.array_equal(early.stations(), other.stations())


def test_launch_counts_are_those_of_the_schedule_that_ran(recording, monkeypatch):
    """last_launches is the count of the graph that ran, whatever other
    schedule of the solver was enqueued last: timed graphs, an ensemble's,
    direct launches."""
    import cgfd
    monkeypatch.setattr(cgfd, "load_library", lambda *a: recording)
    a, b = (cgfd.Solver(closed_box(seed=q), lib=recording) for q in (7, 8))
    kernels, inside = {}, None       # kernels of each captured graph

    def launched():
        """Kernels launched since the last look, directly or in graphs."""
        nonlocal inside
        n = 0
        for op, st, *rest in operations(recording):
            if op == "begin":
                inside = 0
            elif op == "end":
                kernels[rest[0]], inside = inside, None
            elif op == "launch" and inside is not None:
                inside += 1
            elif op == "launch":
                n += 1
            elif op == "graph":
                n += kernels[rest[0]]
        return n

    launched()
    ens = cgfd.Ensemble([a, b])

    def check(call, solvers):
        call()
        assert sum(s.last_launches() for s in solvers) == launched()

    for timing in (False, True, False):
        a.set_timing(timing)
        b.set_timing(timing)
        launched()
        check(lambda: a.run(3), [a])
        check(lambda: b.run(3), [b])
        check(lambda: ens.run(2), [a, b])
        check(lambda: a.run(1), [a])
        check(lambda: b.run_noalloc(1), [b])
        check(lambda: a.run(9), [a])
        check(lambda: b.run(9), [b])
    ens.close()


@pytest.mark.parametrize("free_surface", [0, 1])
def test_timing_keeps_the_schedule(recording, free_surface):
    """cgfd_set_timing adds events to a step, no launch and no order: what it
    times is the step that runs without it."""
    from cgfd import Solver
    p = inputs.small_planar(nt=20, free_surface=free_surface)
    s = Solver(p, lib=recording)

    def graphs():
        # a capture's launches with their streams, and its forks and joins
        out, lines = [], None
        external = set()
        for o in operations(recording):
            if o[0] == "begin":
                lines = []
            elif o[0] == "end":
                out.append(lines)
                lines = None
            elif lines is not None and not (o[0] == "record" and o[3] == "1"):
                lines.append(o)
            elif lines is not None:
                external.add(o[2])
        return out, external

    plain, none = graphs()
    s.set_timing(True)
    timed, external = graphs()
    assert len(plain) == len(timed) == 8 and not none
    assert any("k_volume_all" in o[2] for o in plain[0] if o[0] == "launch")
    assert timed == plain
    # four events a stage, of which every step has its own
    assert len(external) == 8 * 4 * 4


@pytest.mark.gpu
@pytest.mark.parametrize("free_surface", [0, 1])
def test_timed_run_is_the_untimed_one(cgfd_lib, free_surface):
    from cgfd import Solver, WAVE_COMPONENTS
    a, b = (Solver(inputs.small_planar(nt=20, free_surface=free_surface)) for _ in range(2))
    b.set_timing(True)
    for s in (a, b):
        s.run(17)
    assert a.last_launches() == b.last_launches()
    run_ms, vol_ms, vol_n = b.last_timing()
    int_ms, int_n, _ = b.kernel_timing(1)
    assert vol_n == int_n == 4 * 17 and 0 < int_ms <= vol_ms <= run_ms
    for c in WAVE_COMPONENTS:
        assert np.array_equal(a.wavefield(c), b.wavefield(c)), c
    assert np.array_equal(a.fault_all(), b.fault_all())


SCHEDULES = [{}, {"CGFD_MERGED": "0"}, {"CGFD_BRANCHES": "0"}, {"CGFD_BRANCHES": "1"}, {"CGFD_BRANCHES": "2"},
             {"CGFD_PRE_OVERLAP": "0"}, {"CGFD_POST_EARLY": "0"}, {"CGFD_PRE_EARLY": "0"},
             {"CGFD_TOP": "0"}]


@pytest.mark.parametrize("env", SCHEDULES, ids=lambda e: ",".join(f"{k}={v}" for k, v in e.items()) or "default")
def test_dependent_launches_follow_their_kernel(recording, monkeypatch, env):
    """A programmatic dependent launch starts beside the operation ahead of it
    in its stream; it is used only where that is the fault kernel it was
    written to run beside, never behind an event wait or a timing event."""
    from cgfd import Solver
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    ahead_of = {"k_fault_split": {"k_fault_pre"}, "k_fault_slab": {"k_fault_split", "k_fault_slab"}}
    for p in (clear_of_the_pml(), closed_box(), inputs.two_faults(nt=20)):
        s = Solver(p, lib=recording)
        s.set_timing(True)
        s.set_timing(False)
        try:
            s.run_noalloc(1)
        except Exception as e:      # free surface: nothing counts the steps here
            assert "counter" in str(e)
        last, dependent = {}, set()
        for op, st, *rest in operations(recording):
            if op == "launch":
                name = kernel(rest[0])
                if rest[-1] == "1":
                    assert last[st] in ahead_of[name], (name, last[st])
                    dependent.add(name)
                last[st] = name
            elif op != "record" or rest[1] == "1":
                last[st] = op
        assert "k_fault_split" in dependent
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("env", SCHEDULES, ids=lambda e: ",".join(f"{k}={v}" for k, v in e.items()) or "default")
def test_timed_schedules_agree(cgfd_lib, monkeypatch, env):
    """Every schedule with timing on (its events lie among the launches) is
    the untimed one bit for bit."""
    from cgfd import Solver, WAVE_COMPONENTS
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    for p in (clear_of_the_pml(), inputs.two_faults(nt=20)):
        a, b = Solver(p), Solver(p)
        b.set_timing(True)
        for s in (a, b):
            s.run(17)
        for c in WAVE_COMPONENTS:
            assert np.array_equal(a.wavefield(c), b.wavefield(c)), c
        for f in range(p.num_faults):
            assert np.array_equal(a.fault_all(f), b.fault_all(f)), f


def test_chunk_choice_is_kept_per_kernel(recording, monkeypatch):
    """The interior kernel's y chunk is timed once per kernel and grid shape: a
    solver that runs the general kernel does not take over what was fastest
    for the aligned one on an interior box of the same extents."""
    from cgfd import Solver
    p = inputs.small_planar(nt=20, ni=38, nj=58)

    def timed():
        operations(recording)
        Solver(p, lib=recording).close()
        ops = operations(recording)
        first = next(n for n, o in enumerate(ops) if o[0] == "begin")
        return sum(o[0] == "launch" and kernel(o[2]) == "k_volume 0" for o in ops[:first])

    assert timed() > 0 and timed() == 0
    monkeypatch.setenv("CGFD_ALIGNED", "0")
    assert timed() > 0 and timed() == 0
    monkeypatch.delenv("CGFD_ALIGNED")
    assert timed() == 0


@pytest.mark.parametrize("n", [1, 2, 100])
def test_chunk_switch_counts_eight_rows(recording, monkeypatch, n):
    """CGFD_INTERIOR_YCHUNK=n asks for chunks of 8 n rows whatever the height
    of the kernel's tiles (so its grid's z extent, which is limited to 65535,
    does not grow when the tiles get lower)."""
    from cgfd import Solver
    p = inputs.small_planar(nt=20, nj=61)
    rows, planes = 61 - 2 * 6, 32 - 6 - 4
    monkeypatch.setenv("CGFD_INTERIOR_YCHUNK", str(n))
    operations(recording)
    Solver(p, lib=recording).close()
    grid = next([int(v) for v in o[3:6]] for o in operations(recording) if o[0] == "launch" and kernel(o[2]) == "k_volume 0")
    tiles = -(-rows // 4)
    chunk = min(2 * n, tiles)
    assert grid[1:] == [chunk, planes * -(-tiles // chunk)]


@pytest.mark.parametrize("double", [False, True])
def test_writes_to_the_device_follow_the_solvers_stream(recording, recording64, double):
    """The blocking copy of pageable memory may return before the device has
    all of it, and orders nothing on the solver's stream: a state or a
    wavefield that is put in place goes by that stream, and is waited for."""
    from cgfd import Solver
    lib = recording64 if double else recording
    operations(lib)
    s = Solver(closed_box(), lib=lib)
    s.run(1)
    calls = [operations(lib)]
    buf = s.checkpoint()
    operations(lib)
    s.restore(buf)
    calls.append(operations(lib))
    s.set_wavefield("Vx", np.zeros((s.prob.nk, s.prob.nj, s.prob.ni), np.float32))
    calls.append(operations(lib))
    for ops in calls:
        assert not any(o[0] == "blockcopy" and o[3] == "in" for o in ops)
        assert any(o[0] == "copy" for o in ops)
    for ops in calls[1:]:
        streams = {o[1] for o in ops if o[0] == "copy"}
        assert len(streams) == 1 and ops[-1] == ("sync", streams.pop())
    s.close()
