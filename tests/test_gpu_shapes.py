"""The descriptor kernel has builds of its own for the usual shape (n_max 4 4,
basis 8 8, l_max 4) beside the ones that take any shape up to it; every shape
around that edge, with odd and even l_max (the harmonics are summed in pairs of
components) and one and two types, against the FP64 oracle."""
import numpy as np
import pytest

import oracle
import workloads
from test_gpu_force import assert_close, run_gpu

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [((4, 4), (8, 8), (4, 2, 1)), ((4, 4), (8, 8), (3, 0, 0)), ((4, 4), (8, 8), (1, 0, 0)),
          ((4, 4), (8, 8), (2, 2, 0)), ((4, 3), (8, 8), (4, 2, 1)), ((3, 4), (8, 7), (4, 2, 0)),
          ((2, 0), (5, 3), (3, 2, 0)), ((0, 2), (1, 8), (4, 0, 1)), ((5, 4), (8, 8), (4, 2, 1)),
          ((4, 4), (9, 8), (4, 2, 1)), ((7, 6), (12, 10), (3, 2, 0))]


@pytest.mark.parametrize("n_max,basis,l_max", SHAPES)
def test_shapes_match_oracle(tmp_path, n_max, basis, l_max):
    path = workloads.write_nep(str(tmp_path / "nep.txt"), symbols=("O", "H"), rc=(5.0, 4.0),
                               mn=(200, 100), n_max=n_max, basis=basis, l_max=l_max, H=21,
                               seed=3, q_scaler=0.05)
    t, h, p = workloads.water(n_mol=217, seed=8)      # 18.6 A: Verlet rows
    ref = oracle.OracleModel(path).compute(t, h, p)
    _, pe, f, w = run_gpu(path, t, h, p)
    assert_close(ref, (pe, f, w), "large box")
    t, h, p = workloads.water(n_mol=40, seed=9)       # 10.6 A: explicit rows of images
    ref = oracle.OracleModel(path).compute(t, h, p)
    _, pe, f, w = run_gpu(path, t, h, p)
    assert_close(ref, (pe, f, w), "small box")
