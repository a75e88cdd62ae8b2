"""The plain gain with four 16-byte columns per thread (one FP32 cell, b-rows of 384 states and
more) and just below it, with b-rows that do not fill the last thread, against the FP64 oracle
(relative L-inf 1e-12 and 2e-5, the tolerances of the plain path)."""
import pytest

from test_gpu_gain_pass import _cells_workload, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("p_g,u_g", [(47, 8), (48, 8), (49, 8), (63, 8), (73, 7), (64, 8), (103, 5), (65, 8)])
def test_columns_of_a_pass_match_oracle(cuda, prec, p_g, u_g):
    _check(_cells_workload((4, 2, p_g, u_g), 1, seed=p_g, flux=False), prec)
