"""Evaluations and runs on streams of the caller's that the library may not capture:
one that the caller is capturing, and the legacy default stream by its handle.  They
give the bits that the system's own stream gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(lib, n_waters=300, edge=21.0):
    from mdpy_gb300 import constraint as C, systems
    from mdpy_gb300.ensemble import Ensemble

    w = systems.water_box(n_waters, edge, seed=4)
    ens = Ensemble(w.topology, w.pbc_matrix)
    ens.add_constraints(C.NonbondedConstraint(w.parameters["nonbonded"], 9.0),
                        C.PMEConstraint(grid_size=24, real_space_cutoff=9.0),
                        C.CharmmBondConstraint(w.parameters["bond"]),
                        C.CharmmAngleConstraint(w.parameters["angle"]))
    ens.state.set_positions(w.positions)
    ens.state.set_velocities(w.velocities)
    ens.system.integrator_config(lib.INTEGRATOR_LANGEVIN, 0.5, 300.0, 1e-3, 9)
    return ens


def _steps(ens, runs):
    for n in runs:
        ens.system.compute_forces(ens.term_mask)
        ens.system.integrate(n, ens.term_mask, want_energy=False)


def _state(ens):
    s = ens.system
    return s.get_positions(), s.get_velocities(), s.get_forces()


RUNS = (3, 9, 9, 9, 9)


@pytest.mark.parametrize("every", [1, 2])
def test_legacy_stream(lib, every):
    out = []
    for legacy in (False, True):
        ens = _system(lib)
        ens.system.set_mts(every)
        if legacy:
            ens.system.set_stream(0x1)
        _steps(ens, RUNS + (45,))
        out.append(_state(ens))
        ens.system.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("warm", [False, True])  # without and with graphs kept from before
def test_under_a_callers_capture(lib, warm):
    import torch

    def prepared():
        ens = _system(lib)
        stream = torch.cuda.Stream()
        ens.system.set_stream(stream.cuda_stream)
        if warm:
            _steps(ens, RUNS)
        else:
            ens.system.compute_forces(ens.term_mask)
        torch.cuda.synchronize()
        return ens, stream

    want, _ = prepared()
    _steps(want, RUNS)
    ens, stream = prepared()
    with torch.cuda.stream(stream):
        g = torch.cuda.CUDAGraph()
        g.capture_begin(capture_error_mode="thread_local")
        _steps(ens, RUNS)
        g.capture_end()
        g.replay()
    torch.cuda.synchronize()
    for a, b in zip(_state(ens), _state(want)):
        assert np.array_equal(a, b)
    for e in (ens, want):
        e.system.close()
