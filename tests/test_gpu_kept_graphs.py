"""Captured steps and evaluations are kept from call to call while nothing
changes: the same program gives the same bits whether its graphs are kept,
dropped before every call, or replaced by one graph per step, through changes
of the integrator, the outer step, the terms, the positions and the box's
re-sort phase."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _program(lib, mode, drop, langevin):
    from mdpy_gb300 import constraint as C, systems
    from mdpy_gb300.ensemble import Ensemble
    from mdpy_gb300.integrator import LangevinIntegrator, VerletIntegrator

    w = systems.water_box(300, 21.0, seed=4)
    ens = Ensemble(w.topology, w.pbc_matrix)
    bond = C.CharmmBondConstraint(w.parameters["bond"])
    ens.add_constraints(C.NonbondedConstraint(w.parameters["nonbonded"], 9.0),
                        C.PMEConstraint(grid_size=24, real_space_cutoff=9.0), bond,
                        C.CharmmAngleConstraint(w.parameters["angle"]))
    ens.system.set_graph_mode(mode)
    ens.state.set_positions(w.positions)
    ens.state.set_velocities(w.velocities)
    out = []

    def go(integ, n):
        if drop:
            ens.system.set_reorder_interval(20)  # drops every graph
        integ.integrate(ens, n)
        out.append((ens.state.positions, ens.state.velocities,
                    np.array([ens.potential_energy, ens.kinetic_energy])))

    def make(temperature, dt, every=1):
        return (LangevinIntegrator(dt, temperature, 1e-3, seed=9, reciprocal_every=every)
                if langevin else VerletIntegrator(dt, reciprocal_every=every))

    a, b, m = make(300.0, 0.5), make(320.0, 0.25), make(300.0, 0.5, every=2)
    for n in (3, 1, 25, 7, 45, 0, 2):
        go(a, n)
    go(b, 8)                      # other settings: the steps are captured anew
    go(a, 21)
    for _ in range(4):            # evaluations of other terms in between
        bond.update()
        ens.update()
        out.append((ens.forces, bond.forces, np.array([ens.potential_energy])))
        go(a, 2)
    go(m, 5)                      # multiple time steps, and back
    go(a, 6)
    for k in range(4):            # new positions, an evaluation of each
        ens.state.set_positions(out[k][0] + 0.01 * k)
        ens.update()
        out.append((ens.forces, np.array([ens.potential_energy])))
        go(a, 3)
    return out


@pytest.mark.parametrize("langevin", [True, False])
def test_kept_graphs_change_nothing(lib, langevin):
    ref = _program(lib, lib.GRAPH_CHUNK, True, langevin)
    for mode, drop in ((lib.GRAPH_CHUNK, False), (lib.GRAPH_STEP, False), (lib.GRAPH_STEP, True)):
        got = _program(lib, mode, drop, langevin)
        assert len(got) == len(ref)
        for k, (g, r) in enumerate(zip(got, ref)):
            for u, v in zip(g, r):
                assert np.array_equal(u, v), (mode, drop, k)
