"""Batches and servers past the sizes and shapes of test_gpu_batch.py: larger
structures whose candidates come from a cell grid (at least 125 cells) in sheared
boxes and slabs, against the FP64 oracle; and structures that enter and leave a server
between steps that work in place."""
import time

import numpy as np
import pytest

import oracle
import workloads
from conftest import potential
from test_gpu_batch import _pack, _split
from test_gpu_force import assert_close

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
PATH = potential("nep_water.txt")
MASS = np.array([15.999, 1.008])


def _water(molecules, seed, tilt=0.0):
    t, h, p = workloads.water(n_mol=molecules, seed=seed)
    if tilt:
        shear = np.eye(3)
        shear[0, 1], shear[0, 2], shear[1, 2] = tilt, -0.5 * tilt, 0.7 * tilt
        h = (shear @ h.reshape(3, 3)).reshape(-1)
        p = np.ascontiguousarray(shear @ p)
    return t, h, p


# cells of 3 A: 37 A of water is 12 a direction
@pytest.mark.parametrize("molecules,tilt,pbc", [(1000, 0.15, (1, 1, 1)), (1700, 0.0, (1, 1, 0)),
                                                (1700, 0.0, (0, 1, 1)), (1700, 0.1, (1, 1, 0)),
                                                (1300, 0.0, (1, 1, 1))])
def test_cell_grids_match_oracle(molecules, tilt, pbc):
    import nepx
    structs = [_water(60, 3) + ((1, 1, 1),), _water(molecules, 4, tilt) + (pbc,)]
    pot = nepx.Potential(PATH, max_atoms=sum(len(s[0]) for s in structs))
    tt, pp, descs = _pack(structs)
    got = [x.cpu().numpy() for x in pot.compute_batch(descs, tt, pp, sync_check=True)]
    model = oracle.OracleModel(PATH)
    for k, s in enumerate(structs):
        part = [_split(x, structs)[k] for x in got]
        assert_close(model.compute(*s[:3], s[3]), part, "structure %d of %s" % (k, pbc))
    pot.close()


@pytest.mark.parametrize("tilt,pbc", [(0.1, (1, 1, 1)), (0.0, (1, 1, 0))])
def test_kept_candidates_on_a_grid(tilt, pbc):
    """An MD segment whose candidates (cells of 3.5 A) come from such a grid, with
    reuse and with rows built afresh: the same bits."""
    import nepx
    t, h, p = _water(2300 if tilt else 3000, 6, tilt)
    m = MASS[np.asarray(t)]
    v = workloads.maxwell_boltzmann(m, 300.0, seed=7)
    pot = nepx.Potential(PATH, max_atoms=len(t))
    out = []
    for reuse in (True, False):
        srv = nepx.Server(pot, max_atoms=len(t), max_struct=2)
        srv.set_row_reuse(reuse)
        out.append(srv.wait(srv.submit(t, p, h, pbc, md_steps=12, dt_fs=0.5, masses=m, vel=v,
                                       want_state=True)))
        srv.close()
    for key in ("pe", "force", "virial", "pos", "vel"):
        assert np.array_equal(out[0][key], out[1][key]), key
    pot.close()


def test_arrivals_after_steps_in_place():
    """Steps that nothing enters or leaves work with the tables the device holds; a
    structure that arrives after a stretch of them, and one that then leaves, change
    none of the others' results."""
    import nepx
    rng = np.random.default_rng(5)
    segs = []
    for n, steps in ((60, 900), (250, 500), (25, 40), (120, 300)):
        t, h, p = workloads.water(n_mol=n, seed=int(rng.integers(1 << 30)))
        m = MASS[np.asarray(t)]
        segs.append(dict(types=t, pos=p, h=h, md_steps=steps, dt_fs=0.5, masses=m, want_state=True,
                         vel=workloads.maxwell_boltzmann(m, 300.0, seed=n)))
    pot = nepx.Potential(PATH, max_atoms=2000)
    alone = []
    for s in segs:
        srv = nepx.Server(pot, max_atoms=2000, max_struct=8)
        alone.append(srv.wait(srv.submit(**s)))
        srv.close()
    srv = nepx.Server(pot, max_atoms=2000, max_struct=8)
    tickets = []
    for s in segs:
        tickets.append(srv.submit(**s))
        at = srv.stats()["steps"]
        end = time.time() + 60.0
        while srv.stats()["steps"] < at + 12 and time.time() < end:
            time.sleep(0.0005)
    got = [srv.wait(k) for k in tickets]
    assert got[0]["t_done"] > got[2]["t_done"] and got[3]["t_admit"] > got[0]["t_admit"]
    srv.close()
    for a, b in zip(alone, got):
        for key in ("pe", "force", "virial", "pos", "vel"):
            assert np.array_equal(a[key], b[key]), key
    pot.close()
