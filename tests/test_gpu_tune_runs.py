"""Autotuning on runs of blocks (marked gpu): the mixed HLLC kernels have one
form there, so the tuner times it once; the exact solver's keep their three
candidates.  The shape that was set stays."""
import pytest

from flash5_b200 import abi, setups
from flash5_b200.grid import UniformGrid
from flash5_b200.hydro import Hydro


@pytest.mark.gpu
@pytest.mark.parametrize("rs,forms", [(abi.RS_HLLC, 1), (abi.RS_EXACT, 3)])
def test_one_trial_per_form(rs, forms):
    grid = UniformGrid(3, (8, 8, 8), (4, 4, 4), bc="periodic")
    h = Hydro(abi.default_params(gamma=5.0 / 3.0, precision=abi.PREC_MIXED, riemann_solver=rs), grid)
    h.upload(setups.kelvin_helmholtz(grid))
    dt, _ = h.compute_dt()
    before = h.tuning
    best, trials = h.autotune(dt, steps=2)
    # + the other mx_runs and the other sweep order, + the transverse pass
    assert len(trials) == forms + 2 + len(h.tuning_candidates()["sig_threads"])
    if forms == 1:
        assert best["mx_threads"] == before["mx_threads"]
    h.close()
