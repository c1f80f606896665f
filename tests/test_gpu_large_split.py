"""Work items per cluster by the size of each system: the Ewald pair kernel at 128,000
atoms and more (two items), and a batch with members on both sides of that line, each
cut up as it is alone, also after its launch shape was read and written back."""
import numpy as np
import pytest

from tests.helpers import rel_rms, water_lj_rows

pytestmark = pytest.mark.gpu

RC, BETA = 9.0, 0.35


@pytest.fixture(scope="module")
def boxes():
    from mdpy_gb300 import systems

    return [systems.water_box(n // 3, (n / 0.1) ** (1 / 3), seed=n) for n in (129000, 3000)]


def _system(lib, ws):
    s = lib.System.batch([w.num_particles for w in ws], [w.box for w in ws])
    s.set_charges(np.concatenate([w.topology.charges.reshape(-1) for w in ws]))
    s.set_lj(np.concatenate([water_lj_rows(w) for w in ws]))
    off = np.cumsum([0] + [w.num_particles for w in ws])
    ex = [np.where(w.topology.bonded_particles >= 0, w.topology.bonded_particles + o, -1)
          for w, o in zip(ws, off)]
    s.set_exclusions(np.concatenate(ex), np.full((int(off[-1]), 1), -1))
    s.nonbonded_config(RC, 0.0, True, lib.COUL_EWALD, BETA)
    s.set_positions(np.concatenate([w.positions for w in ws]))
    return s


def _forces(lib, s):
    s.compute_forces(lib.mask(lib.TERM_LJ, lib.TERM_COUL_REAL))
    return s.get_forces(), s.get_energies_batch()[0]


def test_two_items_per_cluster_vs_oracle(lib, orc, boxes):
    w = boxes[0]
    t, n = w.topology, w.num_particles
    rows = np.random.default_rng(0).choice(n, 3000, replace=False)
    fo, _ = orc.nonbonded(w.positions, w.box, water_lj_rows(w), t.charges.reshape(-1),
                          t.bonded_particles, t.scaling_particles, RC, coulomb="ewald", beta=BETA,
                          rows=rows)
    s = _system(lib, [w])
    assert s.launch_shape["split"] == 0
    by_size = _forces(lib, s)
    # 1e-5 as for boxes of up to 64 A; coordinates of 109 A have an ulp twice theirs
    assert rel_rms(by_size[0][rows], fo) <= 2e-5
    s.set_launch_shape(split=2)
    for a, b in zip(_forces(lib, s), by_size):
        assert np.array_equal(a, b)
    s.close()


def test_members_of_a_batch_are_cut_up_as_alone(lib, boxes):
    alone = []
    for w in boxes:
        s = _system(lib, [w])
        alone.append(_forces(lib, s))
        s.close()
    b = _system(lib, boxes)
    n0 = boxes[0].num_particles

    def same():
        f, e = _forces(lib, b)
        for k, sl in enumerate((slice(0, n0), slice(n0, None))):
            assert np.array_equal(f[sl], alone[k][0])
            for t in (lib.TERM_LJ, lib.TERM_COUL_REAL):
                assert e[k, t] == alone[k][1][0, t]

    same()
    b.set_launch_shape(**b.launch_shape)
    same()
    b.set_launch_shape(pme_block=128)  # another field keeps the default split
    same()
    b.set_launch_shape(split=4)
    b.set_launch_shape(split=0)
    same()
    b.close()


def test_the_tuner_keeps_a_split_by_size(lib, boxes):
    """Read back after tuning, the shape gives the forces that it was tuned with."""
    b = _system(lib, boxes)
    r = b.autotune(lib.mask(lib.TERM_LJ, lib.TERM_COUL_REAL), reps=1)
    assert r["split"] in (0, 2, 4, 8)
    f, e = _forces(lib, b)
    b.set_launch_shape(**b.launch_shape)
    f2, e2 = _forces(lib, b)
    assert np.array_equal(f, f2) and np.array_equal(e, e2)
    b.close()
