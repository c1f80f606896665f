"""The re-sort's variants -- short and long scans, few and many columns, bins that
hold one atom and bins that hold hundreds -- give the same order: a batch member's
forces are the ones it has alone, bit for bit."""
import numpy as np
import pytest

from tests.helpers import make_system

pytestmark = pytest.mark.gpu


def _lj(lib, x, box, sigma, rc, eps=1e-4):
    n = len(x)
    return make_system(lib, n, box, charges=np.zeros(n), lj=np.tile([eps, sigma] * 2, (n, 1)),
                       cutoff=rc, positions=x)


def _clump(rng, n, apart):
    """n atoms `apart` A apart (0.3: hundreds of them in a few bins)."""
    per = int(np.ceil(n ** (1 / 3)))
    c = np.stack(np.unravel_index(np.arange(n), (per,) * 3), 1) * apart
    return c + rng.uniform(-0.15, 0.15, (n, 3)) * apart


def test_long_scan_equals_short_scan(lib):
    """60,000 atoms alone (one block scans the bins) and twice in a batch (three
    kernels): the same order, hence the same forces."""
    rng = np.random.default_rng(7)
    n, edge = 60000, 84.0
    sites = np.stack(np.unravel_index(np.arange(40 ** 3), (40,) * 3), 1) * (edge / 40)
    xs = [rng.permutation(sites)[:n] + rng.uniform(-0.5, 0.5, (n, 3)) for _ in range(2)]
    b = lib.System.batch([n, n], np.full((2, 3), edge))
    b.set_lj(np.tile([1e-2, 0.4, 1e-2, 0.4], (2 * n, 1)))
    b.set_charges(np.zeros(2 * n))
    b.nonbonded_config(4.0)
    b.set_positions(np.concatenate(xs))
    b.compute_forces(lib.mask(lib.TERM_LJ))
    f = b.get_forces()
    b.compute_forces(lib.mask(lib.TERM_LJ))
    assert np.array_equal(b.get_forces(), f)
    assert np.abs(f).max() > 0
    for q, x in enumerate(xs):
        s = _lj(lib, x, edge, 0.4, 4.0, eps=1e-2)
        s.compute_forces(lib.mask(lib.TERM_LJ))
        assert np.array_equal(s.get_forces(), f[q * n:(q + 1) * n])
        s.close()
    b.close()


def test_batch_of_many_columns_equals_members_alone(lib):
    rng = np.random.default_rng(5)
    counts = rng.integers(40, 400, 300)  # about 900 columns
    boxes = [np.full(3, max(12.0, (c / 0.1) ** (1 / 3))) * [1.0, 1.3, 1.1] for c in counts]
    xs = [_clump(rng, c, 2.0) if k % 4 else _clump(rng, c, 0.3)
          for k, (c, b) in enumerate(zip(counts, boxes))]
    b = lib.System.batch(counts, boxes)
    prm = np.tile([1e-4, 0.3, 1e-4, 0.3], (int(counts.sum()), 1))
    b.set_lj(prm)
    b.set_charges(np.zeros(len(prm)))
    b.nonbonded_config(5.0)
    b.set_positions(np.concatenate(xs))
    b.compute_forces(lib.mask(lib.TERM_LJ))
    f, off = b.get_forces(), 0
    for c, box, x in zip(counts, boxes, xs):
        s = _lj(lib, x, box, 0.3, 5.0)
        s.compute_forces(lib.mask(lib.TERM_LJ))
        assert np.array_equal(f[off:off + c], s.get_forces())
        s.close()
        off += c
    b.close()
