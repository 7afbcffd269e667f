"""The FP64 direction kernels (marked gpu): runs of four blocks along the
sweep (full uniform 3D grids whose block counts divide by 4) against one
block per CTA (the block-list step) and against the oracle, bit for bit, on
periodic, outflow and reflecting boundaries and with the options that change
the kernels' branches; the 2D kernels against the oracle with the same
options.  No tolerance: the kernels share one evaluation of each slope,
flattening switch and reciprocal between cells and divisions, which leaves
every bit as the reference's expressions give it.
"""
import numpy as np
import pytest

from flash5_b200 import abi, setups
from flash5_b200.grid import UniformGrid, VAR
from flash5_b200.hydro import Hydro, next_dt
from oracle import orc

OPTIONS = [{}, {"slope_limiter": abi.LIM_MC}, {"slope_limiter": abi.LIM_HYBRID, "char_limiting": 0},
           {"use_flattening": 0, "use_3d_full_ctu": 0}, {"use_steepening": 1, "slope_limiter": abi.LIM_MINMOD},
           {"use_aux_eint": 0}, {"eint_switch": 1e3}]


def _advance(h, o, grid, unk, steps, blocks=None):
    h.upload(unk)
    dt, loc = h.compute_dt()
    t, dt_old, dts = 0.0, dt, []
    for _ in range(steps):
        if blocks is None:
            h(t + dt, dt, dt_old)
        else:
            h.step_blocks(blocks, t + dt, dt, dt_old)
        if o is not None:
            assert o[0].hydro(o[1], t + dt, dt, dt_old) == 0
        t += dt
        new, loc = h.compute_dt()
        dts.append((new, tuple(loc)))
        dt_old, dt = dt, next_dt(new, dt)
    out = grid.new_unk()
    h.download(out)
    return out, dts


def _check_oracle(grid, params, unk, steps):
    ref = unk.copy()
    o = orc.Oracle(params, grid)
    o.eos_init(ref)
    h = Hydro(params, grid)
    out, dts = _advance(h, (o, ref), grid, unk, steps)
    h.close()
    _, dto, loco = o.compute_dt(ref)
    assert dts[-1] == (dto, tuple(loco))
    for v in VAR:
        if v != "shok":
            a, b = grid.interior(out)[..., VAR[v]], grid.interior(ref)[..., VAR[v]]
            assert np.array_equal(a, b), (v, float(np.abs(a - b).max()))
    return out, dts


@pytest.mark.gpu
@pytest.mark.parametrize("opt", OPTIONS, ids=lambda o: "-".join(f"{k}{v}" for k, v in o.items()) or "default")
@pytest.mark.parametrize("bc", ["periodic", "walls"])
def test_runs_equal_oracle_and_one_block(bc, opt):
    b = "periodic" if bc == "periodic" else ["outflow", "reflecting", "reflecting", "outflow", "outflow", "reflecting"]
    grid = UniformGrid(3, (8, 8, 8), (4, 8, 4), bc=b, order="morton" if bc == "walls" else "lex")
    if bc == "periodic":
        unk, gamma = setups.kelvin_helmholtz(grid), 5.0 / 3.0
    else:
        unk, gamma = setups.sod(grid, xangle=30.0, yangle=70.0), 1.4
    params = abi.default_params(gamma=gamma, **opt)
    out, dts = _check_oracle(grid, params, unk, 2)
    h = Hydro(params, grid)
    one, dts1 = _advance(h, None, grid, unk, 2, blocks=range(grid.nblocks))
    h.close()
    assert dts1 == dts
    assert np.array_equal(one, out)


@pytest.mark.gpu
def test_exact_solver_runs_equal_one_block():
    grid = UniformGrid(3, (8, 8, 8), (4, 4, 8), bc=["outflow", "reflecting"] + ["periodic"] * 4)
    unk = setups.sod_axis(grid, axis=0)
    params = abi.default_params(riemann_solver=abi.RS_EXACT)
    h = Hydro(params, grid)
    runs, dts = _advance(h, None, grid, unk, 3)
    one, dts1 = _advance(h, None, grid, unk, 3, blocks=range(grid.nblocks))
    h.close()
    assert dts1 == dts and np.array_equal(runs, one)


@pytest.mark.gpu
@pytest.mark.parametrize("opt", OPTIONS, ids=lambda o: "-".join(f"{k}{v}" for k, v in o.items()) or "default")
@pytest.mark.parametrize("nb", [8, 16])
def test_2d_equals_oracle(nb, opt):
    grid = UniformGrid(2, (nb, nb), (5, 3), bc=["reflecting", "outflow", "outflow", "reflecting"])
    _check_oracle(grid, abi.default_params(**opt), setups.four_quadrant(grid), 3)


@pytest.mark.gpu
@pytest.mark.parametrize("prec,rs", [(abi.PREC_FP64, abi.RS_HLLC), (abi.PREC_MIXED, abi.RS_HLLC),
                                     (abi.PREC_MIXED, abi.RS_EXACT)])
def test_species_on_runs_equal_one_block(prec, rs):
    """The per-line data the run kernels leave for the species pass (mass
    fluxes, flattening, first-order flags, shared at the seams of a run)
    against one block per CTA: bit for bit (FP64), to rounding (mixed)."""
    grid = UniformGrid(3, (8, 8, 8), (8, 4, 4), bc=["outflow", "reflecting"] + ["periodic"] * 4, nspecies=2,
                       nmass_scalars=1)
    unk = setups.add_species(grid, setups.sod_axis(grid, axis=0))
    h = Hydro(abi.default_params(precision=prec, riemann_solver=rs), grid)
    runs, _ = _advance(h, None, grid, unk, 3)
    one, _ = _advance(h, None, grid, unk, 3, blocks=range(grid.nblocks))
    h.close()
    if prec == abi.PREC_FP64:
        assert np.array_equal(runs, one)
    else:
        # FP32 face values of separately compiled kernels: 1e-7 of values of order one
        assert np.abs(grid.interior(runs)[..., grid.species] - grid.interior(one)[..., grid.species]).max() <= 1e-7
