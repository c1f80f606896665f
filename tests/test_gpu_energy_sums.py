"""The pair kernel's energies are summed in no fewer bits than FP64: small shares are
not lost beside a large one, nor rounded away one by one, in each form of the kernel
that sums Ewald energies (block form, one warp an item in a batch, large systems)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BETA = 0.1


def _energy(lib, systems, index, rc):
    """Real-space Coulomb energy of system `index` of a batch, and the batch's clusters."""
    s = lib.System.batch([len(x) for x, _, _ in systems], [b for _, _, b in systems])
    s.set_charges(np.concatenate([q for _, q, _ in systems]))
    s.nonbonded_config(rc, 0.0, False, lib.COUL_EWALD, BETA)
    s.set_positions(np.concatenate([x for x, _, _ in systems]))
    s.compute_forces(lib.mask(lib.TERM_COUL_REAL))
    e = s.get_energies_batch()[0][index][lib.TERM_COUL_REAL]
    clusters = s.nonbonded_stats()["clusters"]
    s.close()
    return e, clusters


def _lattice(n, edge, seed):
    rng = np.random.default_rng(seed)
    per = int(np.ceil(n ** (1 / 3)))
    site = rng.permutation(per ** 3)[:n]
    x = (np.stack(np.unravel_index(site, (per,) * 3), 1) + 0.5) * (edge / per)
    return x + rng.uniform(-0.1, 0.1, (n, 3))


def _fillers(many):
    """Uncharged systems that leave the system under test to single warps."""
    return [(_lattice(7500, 42.0, k), np.zeros(7500), np.full(3, 42.0)) for k in range(3)] if many else []


FORMS = [(2100, False), (2100, True), (9000, False)]


@pytest.mark.parametrize("n,many", FORMS)
def test_small_shares_add_up(lib, orc, n, many):
    """Energies of 1e-12 a pair: the sum of a lane over 64 j atoms is below half of
    2^-32, an item's is not.  One rounding to 2^-32 an item (four items a cluster)."""
    edge, rc = (n / 0.1) ** (1 / 3), 9.0
    x, q = _lattice(n, edge, 1), np.full(n, 9.5e-6)
    w = (x, q, np.full(3, edge))
    e, clusters = _energy(lib, [w], 0, rc)
    if many:
        e = _energy(lib, [w] + _fillers(many), 0, rc)[0]
    none = np.full((n, 1), -1)
    _, eo = orc.nonbonded(x, np.full(3, edge), np.zeros((n, 4)), q, none, none, rc, lj=False,
                          coulomb="ewald", beta=BETA)
    bar = 4 * clusters * 2.0 ** -33 + 1e-5 * eo["coulomb"]
    assert bar < 0.6 * eo["coulomb"]
    assert abs(e - eo["coulomb"]) <= bar


@pytest.mark.parametrize("n,many", [(3, False), (3, True), (9000, False)])
def test_a_small_share_beside_a_large_one(lib, n, many):
    """An atom with a partner at 0.5 A (an energy of about 2e5) and one at 6 A (9e-3, less
    than a unit in the last place of the former in FP32), which sweeps take in
    different halves of a packed pair: the second counts in full."""
    from mdpy_gb300 import unit

    edge = 40.0 if n == 3 else (n / 0.1) ** (1 / 3)
    x = np.zeros((n, 3))
    if n > 3:
        x[3:] = _lattice(n - 3, edge, 2)
    # one column, one height bin, first by index: neighbours in their cluster
    x[:3] = np.array([[0.3, 0.5, 0.1], [0.8, 0.5, 0.1], [6.3, 0.5, 0.1]])
    energies = []
    for third in (0.0, 1e-3):
        q = np.zeros(n)
        q[:3] = 1000.0, 1000.0, third
        energies.append(_energy(lib, [(x, q, np.full(3, edge))] + _fillers(many), 0, 9.0)[0])
    share = sum(unit.COULOMB_K * 1000.0 * 1e-3 * math.erfc(BETA * r) / r for r in (6.0, 5.5))
    # FP32 pair arithmetic 1e-5, one rounding to 2^-32 an item in each run
    assert abs(energies[1] - energies[0] - share) <= 1e-5 * share + 8 * 2.0 ** -33


@pytest.mark.parametrize("n,many,items", [(64, False, 5), (64, True, 5), (9000, False, 1200)])
def test_an_item_beyond_the_range_is_refused(lib, orc, n, many, items):
    """Like charges whose energies make an item's total pass 1e9 (what int64 fixed point
    holds, with room), although no lane's share and no force does; half of that
    in the whole system is taken, and right."""
    edge = 20.0 if n == 64 else (n / 0.1) ** (1 / 3)
    x, rc = _lattice(n, edge, 3), 9.0
    none = np.full((n, 1), -1)
    unit_energy = orc.nonbonded(x, np.full(3, edge), np.zeros((n, 4)), np.ones(n), none, none, rc,
                                lj=False, coulomb="ewald", beta=BETA)[1]["coulomb"]

    def energy(total):
        q = np.full(n, math.sqrt(total / unit_energy))
        return _energy(lib, [(x, q, np.full(3, edge))] + _fillers(many), 0, rc)[0]

    with pytest.raises(Exception, match="fixed-point range"):
        energy(items * 2.5e9)
    assert energy(5e8) == pytest.approx(5e8, rel=1e-5)
