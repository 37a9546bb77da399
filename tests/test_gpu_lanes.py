"""Lanes per center: the wider groups that small systems take by rule, at the
sizes where the rule changes, and every grouping pinned, on both row paths,
against the FP64 oracle; and the rule gives two handles the same sums."""
import numpy as np
import pytest

import oracle
import workloads
from conftest import potential
from test_gpu_force import assert_close, run_gpu

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
PATH = potential("nep_water.txt")


# 23 molecules: a small box; 510, 513, 1,023, 1,026 atoms: either side of the lines
@pytest.mark.parametrize("molecules", [23, 170, 171, 341, 342])
def test_rule_by_size(molecules):
    t, h, p = workloads.water(n_mol=molecules, density=0.6 if molecules > 100 else 1.0, seed=2)
    ref = oracle.OracleModel(PATH).compute(t, h, p)
    pot, pe, f, w = run_gpu(PATH, t, h, p)
    assert pot.tuning()[0]["gather_group"] == 32
    assert_close(ref, (pe, f, w), "%d molecules" % molecules)
    _, _, f2, _ = run_gpu(PATH, t, h, p)
    assert np.array_equal(f, f2)


@pytest.mark.parametrize("molecules", [30, 250])      # explicit rows, Verlet rows
@pytest.mark.parametrize("lanes", [4, 8, 16, 32])
def test_every_group_matches_oracle(molecules, lanes):
    import nepx
    t, h, p = workloads.water(n_mol=molecules, seed=12)
    ref = oracle.OracleModel(PATH).compute(t, h, p)
    tt = torch.as_tensor(np.asarray(t, dtype=np.int32), device="cuda")
    pp = torch.as_tensor(np.ascontiguousarray(p), device="cuda")
    pot = nepx.Potential(PATH, max_atoms=len(t))
    for fused in (0, 1):
        pot.set_tuning(filter_group=lanes, fused_group=lanes, f12_group=lanes,
                       gather_group=lanes, fused_f12=fused)
        got = [x.cpu().numpy() for x in pot.compute(tt, h, pp, sync_check=True)]
        assert_close(ref, got, "G=%d fused=%d" % (lanes, fused))
    pot.close()
