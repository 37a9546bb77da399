"""The largest systems nepx_compute_noalloc takes: the counts that fill its 16 MiB
with every buffer carved by itself and no rows of heads, for rows long and short, many
types, and a long basis.  Each is accepted (the head rows and the descriptor kernel's
outputs share memory with what is spent by then) and equals nepx_compute."""
import numpy as np
import pytest

import workloads
from test_zz_no_alloc import _close, _noalloc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _lattice(n, spacing, types, seed=0):
    """n atoms on the sites of a jittered cubic lattice, random types."""
    m = int(np.ceil(n ** (1.0 / 3.0)))
    rng = np.random.default_rng(seed)
    sites = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    pos = (sites + 0.5) * spacing + rng.normal(0.0, 0.05, (n, 3))
    h = np.diag([m * spacing] * 3).reshape(-1)
    return (rng.integers(0, types, n).astype(np.int32), h,
            np.ascontiguousarray(pos.T % (m * spacing)))


@pytest.mark.parametrize("n,mn,rc,types,n_max,basis,spacing", [
    (1504, (400, 200), (5.0, 4.0), 1, (4, 4), (8, 8), 2.2),
    (592, (800, 640), (4.2, 3.7), 1, (4, 4), (8, 8), 2.2),
    (10532, (16, 10), (4.2, 3.7), 10, (4, 4), (8, 8), 3.3),
    (2697, (200, 100), (5.0, 4.0), 2, (6, 6), (12, 10), 2.2)])
def test_sizes_that_fit(tmp_path, n, mn, rc, types, n_max, basis, spacing):
    import nepx
    symbols = ("C", "H", "O", "Cu", "N", "Si", "Ba", "Ti", "Al", "Fe")[:types]
    path = workloads.write_nep(str(tmp_path / "nep.txt"), symbols=symbols, rc=rc, mn=mn,
                               n_max=n_max, basis=basis, l_max=(4, 2, 1), H=10, seed=3,
                               q_scaler=0.02)
    t, h, p = _lattice(n, spacing, types)
    pot = nepx.Potential(path, max_atoms=n)
    ref = [x.clone() for x in pot.compute(torch.as_tensor(t, device="cuda"), h,
                                          torch.as_tensor(p, device="cuda"), sync_check=True)]
    rc_, out = _noalloc(pot, t, h, p)
    assert rc_ == 0, nepx.lib().nepx_last_error(pot._h)
    _close(ref, out)
    pot.close()
