"""The pair kernel's block form (several warps per work item, small systems):
the sums are cut up as in the one-warp form, so a batch large enough to be
taken by single warps gives each member the forces and energies it has alone,
bit for bit, in both candidate searches and at the sizes where the number of
warps changes."""
import numpy as np
import pytest

from tests.helpers import rel_rms, water_lj_rows

pytestmark = pytest.mark.gpu


def _system(lib, ws, rc, switch, lj):
    s = lib.System.batch([w.num_particles for w in ws], [w.box for w in ws])
    s.set_charges(np.concatenate([w.topology.charges.reshape(-1) for w in ws]))
    s.set_lj(np.concatenate([water_lj_rows(w) for w in ws]))
    off = np.cumsum([0] + [w.num_particles for w in ws])
    ex = [np.where(w.topology.bonded_particles >= 0, w.topology.bonded_particles + o, -1)
          for w, o in zip(ws, off)]
    s.set_exclusions(np.concatenate(ex), np.full((int(off[-1]), 1), -1))
    s.nonbonded_config(rc, switch, lj, lib.COUL_EWALD, 0.3)
    s.set_positions(np.concatenate([w.positions for w in ws]))
    return s


# waters: a box of few clusters; eight warps an item, four, two (full scan, then
# columns), the largest system of the form; four by a full scan, three
@pytest.mark.parametrize("n_waters,rc,switch,lj", [
    (40, 5.0, 0.0, True), (900, 12.0, 10.0, True), (1300, 9.0, 0.0, True), (2000, 10.0, 8.0, True),
    (2600, 8.0, 0.0, False), (1000, 12.0, 10.0, True), (1700, 10.0, 0.0, True)])
def test_block_form_equals_one_warp_form(lib, orc, n_waters, rc, switch, lj):
    from mdpy_gb300 import systems

    edge = max((3 * n_waters / 0.1) ** (1 / 3), 2.02 * rc)
    w = systems.water_box(n_waters, edge, seed=n_waters)
    filler = systems.water_box(2600, 42.8, seed=2)
    mask = lib.mask(lib.TERM_LJ, lib.TERM_COUL_REAL)
    alone = _system(lib, [w], rc, switch, lj)
    alone.compute_forces(mask)
    f, e = alone.get_forces(), alone.get_energies_batch()[0][0]
    many = _system(lib, [filler, w, filler, filler], rc, switch, lj)
    many.compute_forces(mask)
    n0, n = filler.num_particles, w.num_particles
    assert np.array_equal(many.get_forces()[n0:n0 + n], f)
    eb = many.get_energies_batch()[0][1]
    for t in (lib.TERM_LJ, lib.TERM_COUL_REAL):
        assert eb[t] == e[t]
    # and against the FP64 oracle (FP32 pair arithmetic: 1e-5)
    t = w.topology
    fo, _ = orc.nonbonded(w.positions, w.box, water_lj_rows(w), t.charges.reshape(-1),
                          t.bonded_particles, t.scaling_particles, rc, switch=switch or None,
                          lj=lj, coulomb="ewald", beta=0.3)
    assert rel_rms(f, fo) <= 1e-5
    # the variant without energies leaves the same forces: one step of each
    for s, sl in ((alone, slice(0, n)), (many, slice(n0, n0 + n))):
        s.set_masses(np.ones(s.n))
        s.integrator_config(lib.INTEGRATOR_VERLET, 1.0)
        s.set_velocities(np.zeros((s.n, 3)))
        s.integrate(2, mask, want_energy=False)
    assert np.array_equal(many.get_positions()[n0:n0 + n], alone.get_positions())
    alone.close()
    many.close()
