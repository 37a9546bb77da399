"""Row lengths at the edges of what handles them: the gather finds a neighbour's
slot by blocks of eight entries (seven heads in the first load, 56 entries), and
the rebuild sorts rows in registers up to 128 and 256 entries and in shared
memory above.  Diamond at growing cutoffs, as one system and in a batch with
a small structure, against the FP64 oracle."""
import numpy as np
import pytest

import oracle
import workloads
from test_gpu_force import assert_close

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# (radial, angular) cutoff: angular rows of 4, 16, 34, about 63, 123; Verlet rows of
# 29 to 378 entries
CUTOFFS = [(2.0, 1.8), (3.0, 2.8), (4.2, 3.7), (4.8, 4.4), (6.0, 5.5), (7.0, 3.9)]


@pytest.mark.parametrize("rc", CUTOFFS)
def test_row_lengths(tmp_path, rc):
    import nepx
    path = workloads.write_nep(str(tmp_path / "nep.txt"), rc=rc, mn=(400, 200), seed=6,
                               q_scaler=0.02)
    big = workloads.diamond(ncell=6, jitter=0.08, seed=4)
    small = workloads.diamond(ncell=2, jitter=0.08, seed=5)
    model = oracle.OracleModel(path)
    refs = [model.compute(*s) for s in (big, small)]
    n = [len(s[0]) for s in (big, small)]
    pot = nepx.Potential(path, max_atoms=sum(n))
    dev = [[torch.as_tensor(np.ascontiguousarray(s[0], dtype=np.int32), device="cuda"),
            torch.as_tensor(np.ascontiguousarray(s[2]), device="cuda")] for s in (big, small)]
    for s, (t, p), ref in zip((big, small), dev, refs):
        got = [x.cpu().numpy() for x in pot.compute(t, s[1], p, sync_check=True)]
        assert_close(ref, got, "rc %s, %d atoms" % (rc, len(s[0])))
    got = pot.compute_batch([(n[0], big[1], (1, 1, 1)), (n[1], small[1], (1, 1, 1))],
                            torch.cat([d[0] for d in dev]),
                            torch.cat([d[1] for d in dev], dim=1).contiguous(), sync_check=True)
    at = 0
    for k, ref in enumerate(refs):
        part = [x[..., at:at + n[k]].cpu().numpy() for x in got]
        assert_close(ref, part, "batch, structure %d, rc %s" % (k, rc))
        at += n[k]
    pot.close()
