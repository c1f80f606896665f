"""Bare Coulomb over all pairs: small and ragged systems against the FP64
oracle, with and without energies, and as members of a batch."""
import numpy as np
import pytest

from tests.helpers import half_box_tie_atoms, make_system, rel_rms_excluding

pytestmark = pytest.mark.gpu


def _box(n_waters, seed):
    from mdpy_gb300 import systems

    edge = max(12.0, (3 * n_waters / 0.1) ** (1 / 3))
    w = systems.water_box(n_waters, edge, seed=seed)
    t = w.topology
    return w, dict(charges=t.charges.reshape(-1), lj=np.zeros((w.num_particles, 4)),
                   bonded=t.bonded_particles, scaling=t.scaling_particles, cutoff=5.0,
                   lj_on=False)


# fewer atoms than a warp, one more than a cluster, a last cluster of 30, more
# than a hundred clusters
@pytest.mark.parametrize("n_waters", [2, 11, 234, 1100])
def test_bare_coulomb_vs_oracle_and_in_a_batch(lib, orc, n_waters):
    mask = lib.mask(lib.TERM_COUL_REAL)
    w, kw = _box(n_waters, seed=n_waters)
    s = make_system(lib, w.num_particles, w.box, coulomb=lib.COUL_BARE, positions=w.positions, **kw)
    s.compute_forces(mask)
    f, (e, _) = s.get_forces(), s.get_energies()
    fo, eo = orc.nonbonded(w.positions, w.box, kw["lj"], kw["charges"], kw["bonded"],
                           kw["scaling"], 5.0, lj=False, coulomb="bare")
    ties = half_box_tie_atoms(w.positions, w.box)
    # FP32 pair arithmetic, as every pair term: 1e-5 of the force RMS
    assert rel_rms_excluding(f, fo, ties) <= 1e-5
    scale = np.sum(np.abs(fo)) / max(1, w.num_particles)  # energies cancel: an absolute bar
    assert abs(e[lib.TERM_COUL_REAL] - eo["coulomb"]) <= 1e-4 * abs(eo["coulomb"]) + 1e-5 * scale
    # the variant without energies (an integration step) adds the same forces
    s.integrator_config(lib.INTEGRATOR_VERLET, 1.0)
    s.set_masses(np.ones(w.num_particles))
    s.set_velocities(np.zeros((w.num_particles, 3)))
    s.integrate(1, mask, want_energy=False)
    x1 = s.get_positions()
    # a member of a batch gets the sums it has alone, bit for bit
    o, ko = _box(50, seed=3)
    ws, ks = (o, w), (ko, kw)
    b = lib.System.batch([x.num_particles for x in ws], [x.box for x in ws])
    b.set_charges(np.concatenate([k["charges"] for k in ks]))
    width = max(k["bonded"].shape[1] for k in ks)
    bonded = np.full((o.num_particles + w.num_particles, width), -1)
    bonded[:o.num_particles, :ko["bonded"].shape[1]] = ko["bonded"]
    bonded[o.num_particles:, :kw["bonded"].shape[1]] = np.where(
        kw["bonded"] >= 0, kw["bonded"] + o.num_particles, -1)
    b.set_exclusions(bonded, np.full((len(bonded), 1), -1))
    b.nonbonded_config(5.0, 0.0, False, lib.COUL_BARE, 0.0)
    b.set_positions(np.concatenate([x.positions for x in ws]))
    b.compute_forces(mask)
    assert np.array_equal(b.get_forces()[o.num_particles:], f)
    b.set_masses(np.ones(len(bonded)))
    b.set_velocities(np.zeros((len(bonded), 3)))
    b.integrator_config(lib.INTEGRATOR_VERLET, 1.0)
    b.integrate(1, mask, want_energy=False)
    assert np.array_equal(b.get_positions()[o.num_particles:], x1)
    s.close()
    b.close()
