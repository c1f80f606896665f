"""The PME grids' own transforms against the FP64 PME of the oracle: every
radix, odd lengths, lines of one pair, the largest plane that fits, and a batch
that mixes them with grids that keep the library's plans."""
import numpy as np
import pytest

from tests.helpers import rel_rms

pytestmark = pytest.mark.gpu

GRIDS = [(8, 9, 10), (9, 8, 15), (16, 25, 27), (27, 20, 18), (30, 32, 45), (48, 36, 40), (100, 12, 8),
         (500, 48, 50), (10, 150, 162), (8, 8, 288),
         (22, 24, 26), (13, 16, 20)]


def _random(n, K, seed):
    rng = np.random.default_rng(seed)
    box = np.array(K, float)
    return rng.uniform(0, 1, (n, 3)) * box, box, rng.normal(size=n)


def _expected(orc, x, box, q, beta, K, order):
    f, e = orc.pme(x, box, q, beta, K, order)
    return f, e, orc.ewald_self(q, beta) + orc.ewald_net_charge(q, box, beta)


@pytest.mark.parametrize("order", [4, 5, 6])
def test_transforms_vs_oracle(lib, orc, order):
    grids = [g for g in GRIDS if min(g) >= 2 * order]
    systems = [_random(150 + 7 * k, K, k) for k, K in enumerate(grids)]
    beta = 0.35
    alone = []
    for K, (x, box, q) in zip(grids, systems):
        s = lib.System(len(q), box)
        s.set_charges(q)
        s.nonbonded_config(2.0, 0.0, False, lib.COUL_EWALD, beta)
        s.pme_config(K, order, beta)
        s.set_positions(x)
        for _ in range(2):  # the charge grid is left zeroed
            s.compute_forces(lib.mask(lib.TERM_COUL_RECIP))
        f, (e, _) = s.get_forces(), s.get_energies()
        fo, eo, const = _expected(orc, x, box, q, beta, K, order)
        assert rel_rms(f, fo) <= 2e-5, K
        assert abs(e[lib.TERM_COUL_RECIP] - eo - const) <= 2e-6 * (abs(eo) + abs(const)), K
        alone.append((f, e[lib.TERM_COUL_RECIP]))
        s.close()
    b = lib.System.batch([len(s[2]) for s in systems], [s[1] for s in systems])
    b.set_charges(np.concatenate([s[2] for s in systems]))
    b.nonbonded_config(2.0, 0.0, False, lib.COUL_EWALD, beta)
    b.pme_config_batch(grids, order, beta)
    b.set_positions(np.concatenate([s[0] for s in systems]))
    b.compute_forces(lib.mask(lib.TERM_COUL_RECIP))
    f, (e, _) = b.get_forces(), b.get_energies_batch()
    off = 0
    for k, (x, _, q) in enumerate(systems):
        assert rel_rms(f[off:off + len(q)], alone[k][0]) <= 1e-6, grids[k]
        assert e[k, lib.TERM_COUL_RECIP] == pytest.approx(alone[k][1], rel=1e-6), grids[k]
        off += len(q)
    b.close()


# a cluster and a bit, many clusters of a small system (8 atoms a warp), more
# clusters (a thread per atom gathers), clusters unsplit in spreading
@pytest.mark.parametrize("order", [4, 5, 6])
@pytest.mark.parametrize("n,K", [(37, (12, 13, 18)), (3001, (30, 32, 36)), (45000, (64, 60, 72)),
                                 (160000, (64, 60, 72))])
def test_rows_equal_tiles(lib, order, n, K):
    """Spreading and gathering row by row add the same contributions and read
    the same values in the same order as through tiles (uncharged atoms and
    partly filled clusters among them)."""
    x, box, q = _random(n, K, n)
    q[::5] = 0.0
    s = lib.System(n, box)
    s.set_charges(q)
    s.nonbonded_config(2.0, 0.0, False, lib.COUL_EWALD, 0.35)
    s.pme_config(K, order, 0.35)
    s.set_positions(x)
    out = []
    for tiles in (0, 1, 2, 3):
        s.set_launch_shape(4, 0, 64, 0, 1, tiles)
        s.compute_forces(lib.mask(lib.TERM_COUL_RECIP))
        out.append((s.get_forces(), s.get_energies()[0][lib.TERM_COUL_RECIP]))
    for f, e in out[1:]:
        assert np.array_equal(f, out[0][0]) and e == out[0][1]
    s.close()
