"""The pair dump takes the form of the pair kernel that the system's forces take -- the
block form, single warps in a batch or in a small system without Ewald -- and finds
the all-pairs set there, also after the atoms have drifted far from their sort columns
without a re-sort; the forces of the same form see the same pairs."""
import numpy as np
import pytest

from tests.helpers import (cutoff_band, keys_to_pairs, pair_keys, ref32_keys, rel_rms,
                           water_lj_rows)

pytestmark = pytest.mark.gpu


def _drifted(lib, ws, rc, coulomb):
    """A batch of the boxes, 400 Langevin steps at 900 K on from their start, no re-sort."""
    from mdpy_gb300 import systems

    s = lib.System.batch([w.num_particles for w in ws], [w.box for w in ws])
    n = s.n
    s.set_masses(np.concatenate([w.topology.masses.reshape(-1) for w in ws]))
    s.set_lj(np.concatenate([water_lj_rows(w) for w in ws]))
    s.set_charges(np.zeros(n))
    s.set_exclusions(np.full((n, 1), -1), np.full((n, 1), -1))
    s.nonbonded_config(rc, 0.0, True, lib.COUL_NONE)
    s.set_positions(np.concatenate([w.positions for w in ws]))
    s.set_velocities(np.concatenate([systems.maxwell_boltzmann(np.random.default_rng(3),
                                                               w.topology.masses, 900.0) for w in ws]))
    s.set_reorder_interval(100000)
    s.integrator_config(lib.INTEGRATOR_LANGEVIN, 1.0, 900.0, 0.001, 7)
    s.integrate(400, lib.mask(lib.TERM_LJ), want_energy=False)
    if coulomb:
        s.nonbonded_config(rc, 0.0, True, lib.COUL_EWALD, 0.3)
    return s


def _same(orc, pairs, x, box, rc):
    got, want = pair_keys(pairs), ref32_keys(orc, x, box, rc)
    assert np.array_equal(got, want), (keys_to_pairs(np.setdiff1d(got, want))[:5].tolist(),
                                       keys_to_pairs(np.setdiff1d(want, got))[:5].tolist())
    return len(got)


# 27 images of a full scan and neighbour columns; alone (with Ewald the block form), and
# as a member of a batch that single warps take
@pytest.mark.parametrize("coulomb", [True, False])
@pytest.mark.parametrize("n_waters,edge,rc,many", [(900, 30.0, 12.0, False), (900, 30.0, 12.0, True),
                                                   (2600, 42.8, 8.0, False), (2600, 42.8, 8.0, True)])
def test_pair_set_and_forces_after_drift(lib, orc, n_waters, edge, rc, many, coulomb):
    from mdpy_gb300 import systems

    w = systems.water_box(n_waters, edge, seed=21)
    filler = [systems.water_box(2600, 42.8, seed=k) for k in (2, 3, 4)] if many else []
    ws = filler[:1] + [w] + filler[1:]
    n, n0 = w.num_particles, 7800 if many else 0
    s = _drifted(lib, ws, rc, coulomb)
    x = s.get_positions()[n0:n0 + n]
    pairs = np.asarray(s.pairset())
    mine = pairs[(pairs[:, 0] >= n0) & (pairs[:, 0] < n0 + n)] - n0
    found = _same(orc, mine, x, w.box, rc)
    # the forces: FP32 coordinates of up to 1.25 x 43 A are rounded by 1.1e-6 A rms, which
    # a repulsion as r^-13 at 2.6 A turns into 8e-6 of it
    mask = lib.mask(lib.TERM_LJ, *([lib.TERM_COUL_REAL] if coulomb else []))
    s.compute_forces(mask)
    none = np.full((n, 1), -1)
    fo, _ = orc.nonbonded(x, w.box, water_lj_rows(w), np.zeros(n), none, none, rc,
                          coulomb="ewald" if coulomb else "none", beta=0.3)
    assert rel_rms(s.get_forces()[n0:n0 + n], fo) <= 2e-5
    if coulomb and not many:  # every pair is evaluated, and counted
        band = cutoff_band(orc, x, w.box, rc)
        assert abs(s.nonbonded_stats()["pairs_in_cutoff"] - found) <= len(band)
    s.close()
