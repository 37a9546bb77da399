"""Launch choices follow the size of each call, not that of a handle's first one:
a handle that serves a small system and then a large one takes the large one's
lanes for it, and the small one's again afterwards, in direct calls and in an MD
between whose runs the handle served another size.  A batch handle and a server
keep one set for their life (a structure's sums must not depend on what shares
its launch), whose descriptor lanes are not those of a small first step.  Pinned choices stay, and a
call under stream capture times nothing."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
import workloads
from conftest import ROOT, potential
from test_gpu_force import assert_close

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
PATH = potential("nep_water.txt")
LARGE = 6000                     # molecules: 18,000 atoms, past every wide group


def _device(t, p):
    return (torch.as_tensor(np.asarray(t, dtype=np.int32), device="cuda"),
            torch.as_tensor(np.ascontiguousarray(p), device="cuda"))


def _narrow(pot):
    c = pot.tuning()[0]
    return all(c[k] in (4, 8) for k in ("filter_group", "fused_group", "gather_group"))


@pytest.mark.parametrize("small", [20, 250])          # 60 atoms, a small box; 750, Verlet rows
def test_small_call_then_large(small):
    import nepx
    ts, hs, ps = workloads.water(n_mol=small, seed=3)
    tl, hl, pl = workloads.water(n_mol=LARGE, seed=4)
    small_dev, large_dev = _device(ts, ps), _device(tl, pl)
    pot = nepx.Potential(PATH, max_atoms=len(tl))
    first = pot.compute(small_dev[0], hs, small_dev[1], sync_check=True)[1].clone()
    lanes = pot.tuning()[0]
    assert lanes["gather_group"] == 32 and lanes["fused_group"] in (16, 32)
    mixed = pot.compute(large_dev[0], hl, large_dev[1], sync_check=True)[1].clone()
    assert pot.tuning()[1] and _narrow(pot)
    again = pot.compute(small_dev[0], hs, small_dev[1], sync_check=True)[1].clone()
    assert pot.tuning()[0] == lanes and torch.equal(first, again)
    fresh = nepx.Potential(PATH, max_atoms=len(tl))
    alone = fresh.compute(large_dev[0], hl, large_dev[1], sync_check=True)[1]
    assert torch.equal(mixed, alone)                  # the picks of the size, in either order
    fresh.close()
    pinned = dict(filter_group=8, fused_group=4, fused_ctas_per_sm=3, f12_group=8,
                  gather_group=8, fused_f12=1, gather_ctas_per_sm=3)
    pot.set_tuning(**pinned)
    for t, h, p in ((small_dev[0], hs, small_dev[1]), (large_dev[0], hl, large_dev[1])):
        pot.compute(t, h, p, sync_check=True)
        assert pot.tuning() == (pinned, True)
    pot.close()


def test_md_between_calls_of_another_size():
    import nepx
    t, h, p = workloads.water(n_mol=LARGE, seed=5)
    ts, hs, ps = workloads.water(n_mol=20, seed=6)
    m = np.where(np.asarray(t) == 0, 15.999, 1.008)
    pot = nepx.Potential(PATH, max_atoms=len(t))
    small_dev = _device(ts, ps)
    pot.compute(small_dev[0], hs, small_dev[1], sync_check=True)
    md = nepx.MD(pot, t, m, p, workloads.maxwell_boltzmann(m, 300.0, seed=7), h)
    md.set_ensemble("nve")
    md.run(2, 0.5)
    assert _narrow(pot)
    pot.compute(small_dev[0], hs, small_dev[1], sync_check=True)
    assert not _narrow(pot)
    md.run(2, 0.25)                                   # another step size: captured anew
    assert _narrow(pot)
    md.close()
    pot.close()


def test_server_whose_first_step_is_small():
    import nepx
    structs = [workloads.water(n_mol=n, seed=8) for n in (20, 2000, 250)]
    pot = nepx.Potential(PATH, max_atoms=18000)
    srv = nepx.Server(pot, max_atoms=18000, max_struct=8)
    got = [srv.wait(srv.submit(structs[0][0], structs[0][2], structs[0][1]))]
    choices = pot.tuning()
    assert choices[0]["fused_group"] == 8             # not the 32 of 60 atoms
    tickets = [srv.submit(t, p, h) for t, h, p in structs]
    got += [srv.wait(k) for k in tickets]
    assert pot.tuning() == choices
    srv.close()
    # a direct call takes its own lanes; the batch after it the handle's again
    small_dev = _device(structs[0][0], structs[0][2])
    pot.compute(small_dev[0], structs[0][1], small_dev[1], sync_check=True)
    assert not _narrow(pot)
    pe, f, w = pot.compute_batch([(60, structs[0][1], (1, 1, 1))], *small_dev, sync_check=True)
    assert pot.tuning() == choices
    for r in got[:2]:
        assert np.array_equal(r["force"], f.cpu().numpy())
    model = oracle.OracleModel(PATH)
    for (t, h, p), r in zip(structs, got[1:]):
        assert_close(model.compute(t, h, p), (r["pe"], r["force"], r["virial"]), len(t))
    pot.close()


def test_nothing_is_timed_under_capture(tmp_path):
    import nepx
    # a model of its own: no other test of this process has timed it
    path = workloads.write_nep(str(tmp_path / "nep.txt"), symbols=("O", "H"), rc=(6.0, 4.0),
                               mn=(250, 100), H=17, seed=12, q_scaler=0.02)
    ts, hs, ps = workloads.water(n_mol=250, seed=9)
    tl, hl, pl = workloads.water(n_mol=1700, seed=10)           # 5,100 atoms: timed
    pot = nepx.Potential(path, max_atoms=len(tl))
    dev = _device(ts, ps)
    pot.compute(dev[0], hs, dev[1], sync_check=True)
    dev = _device(tl, pl)
    n = len(tl)
    out = [torch.full(shape, float("nan"), dtype=torch.float64, device="cuda")
           for shape in ((n,), (3, n), (9, n))]
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        pot.compute(dev[0], hl, dev[1], out=out)
    assert pot.tuning()[1] is False and _narrow(pot)
    graph.replay()
    torch.cuda.synchronize()
    assert_close(oracle.OracleModel(path).compute(tl, hl, pl), [x.cpu().numpy() for x in out],
                 "captured call")
    del graph
    pot.close()


SCRIPT = r"""
import sys
sys.path.insert(0, %r); sys.path.insert(0, %r)
import numpy as np, torch, workloads, nepx, os, tempfile
from conftest import potential
t, h, p = workloads.water(n_mol=300, seed=11)
wide = workloads.write_nep(os.path.join(tempfile.mkdtemp(), "nep.txt"), symbols=("O", "H"),
                           rc=(5.0, 4.0), mn=(200, 100), n_max=(6, 5), basis=(12, 10), seed=3,
                           q_scaler=0.05)
tt = torch.as_tensor(t, device="cuda"); pp = torch.as_tensor(p, device="cuda")
for path, mode in ((potential("nep_water.txt"), "fp32"), (potential("nep_water.txt"), "mixed"),
                   (wide, "fp32")):
    pot = nepx.Potential(path, max_atoms=len(t))
    pot.set_precision(mode)
    sys.stderr.write("handle\n"); sys.stderr.flush()
    pot.compute(tt, h, pp, sync_check=True)
    assert pot.tuning()[1]
    pot.close()
"""


def test_small_systems_outside_the_rule_are_timed():
    """The rule by size was measured for the usual shape in FP32; a mixed mode and
    another shape below its line are timed (NEPX_VERBOSE names each timing)."""
    code = SCRIPT % (os.path.join(ROOT, "dmg-md_b200"), os.path.join(ROOT, "tests"))
    env = {k: v for k, v in os.environ.items() if k != "NEPX_TUNE_FILE"}
    r = subprocess.run([sys.executable, "-c", code], env=dict(env, NEPX_VERBOSE="1"), cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    usual, mixed, other = r.stderr.split("handle\n")[1:]
    assert "autotune" not in usual
    assert "autotune (N=900)" in mixed and "autotune (N=900)" in other
