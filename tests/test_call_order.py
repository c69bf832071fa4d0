"""What the calls put on which stream, and in which order.

On the CPU: the library's objects linked with a CUDA runtime that records
instead of running (recording_cudart.cpp), so that an ordering that a test run
on an idle GPU would hardly ever break is seen from the calls themselves.  On
the GPU: the same call sequences against their plain counterparts."""
import ctypes
import glob
import os
import subprocess

import numpy as np
import pytest

import inputs
from conftest import PKG, TESTS


@pytest.fixture(scope="module")
def recording(cgfd_lib, tmp_path_factory):
    """The float library on the recording runtime."""
    import cgfd
    d = tmp_path_factory.mktemp("recording")
    obj, lib = str(d / "recording_cudart.o"), str(d / "libcgfd_recording.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-I/usr/local/cuda/include", "-c",
                           os.path.join(TESTS, "recording_cudart.cpp"), "-o", obj])
    built = sorted(glob.glob(os.path.join(PKG, "_build", "*.cu.o"))) + [os.path.join(PKG, "_build", "setup.cpp.o")]
    subprocess.check_call(["g++", "-shared", "-Wl,-Bsymbolic", "-o", lib] + built + [obj, "-lgomp"])
    r = cgfd.load_library(lib)
    r.recording_log.restype = ctypes.c_char_p
    return r


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
