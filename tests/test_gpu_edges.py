"""States at the edges of the branch-free arithmetic (marked gpu).

The FP64 direction kernels divide without branches and repeat a phase with
plain divisions where an operand leaves the range that is proven for them
(hy_core.cuh, ``Arith``); here velocities, densities and pressures leave it
on purpose, on one block per CTA and on runs of blocks, with and without
species: bit for bit the oracle's results, no status raised.  The mixed
path's HLLC hands vanishing densities and pressures to its general form.
"""
import numpy as np
import pytest

from flash5_b200 import abi, setups
from flash5_b200.grid import UniformGrid, VAR
from flash5_b200.hydro import Hydro, next_dt
from oracle import orc
from tests.test_gpu_parity import conserved_l1

GRIDS = {"2d8": (2, (8, 8), (5, 3)), "2d16": (2, (16, 16), (2, 3)), "3d": (3, (8, 8, 8), (3, 2, 2)),
         "3druns": (3, (8, 8, 8), (4, 4, 4))}


def _tiny_velocity(grid, unk, seed=7):
    """the last velocity component: random values between 1e-140 and 5e-324
    in magnitude, a third of them zero"""
    it = grid.interior(unk)
    r = np.random.default_rng(seed)
    shape = it.shape[:-1]
    v = r.choice([-1.0, 1.0], shape) * 10.0 ** r.uniform(-323.3, -140.0, shape) * r.integers(0, 3, shape).clip(0, 1)
    it[..., VAR["velz" if grid.ndim == 3 else "vely"]] = v
    return unk


def _state(name, kind):
    ndim, nb, nblk = GRIDS[name]
    sp = {"nspecies": 2, "nmass_scalars": 1} if kind == "species" else {}
    bc = ["outflow", "reflecting"] + ["periodic"] * (2 * ndim - 2)
    grid = UniformGrid(ndim, nb, nblk, bc=bc, **sp)
    if kind in ("velocity", "species"):
        unk = _tiny_velocity(grid, setups.sod_axis(grid, axis=0))
        return grid, setups.add_species(grid, unk), abi.default_params()
    if kind == "subnormal":  # multiples of 2^-1074 below 2^-1042, the rest of the state as in a Sod tube
        unk = setups.sod_axis(grid, axis=0)
        it = grid.interior(unk)
        r = np.random.default_rng(3)
        it[..., VAR["velz" if ndim == 3 else "vely"]] = r.integers(-(1 << 20), 1 << 20, it.shape[:-1]) * 5e-324
        return grid, unk, abi.default_params()
    if kind == "thin":      # densities and pressures of 1e-170, below 2^-500 and above the floors
        unk = setups.sod_axis(grid, axis=ndim - 1, rho_l=1e-170, rho_r=1.25e-171, p_l=1e-170, p_r=1e-171)
        return grid, unk, abi.default_params(tiny=1e-300, smlrho=1e-300, smallp=1e-300, smalle=1e-10)
    if kind == "vanish":    # pressures below `tiny` on one side: no flux there
        return grid, setups.sod_axis(grid, axis=0), abi.default_params(tiny=0.12)
    if kind == "huge":      # densities above 2^1022, whose reciprocals' seeds flush to zero
        return grid, setups.uniform(grid, rho=6e307, p=0.4 * 6e307 * 1e-10), abi.default_params()
    raise KeyError(kind)


def _run(h, grid, unk, steps, o=None, ref=None):
    h.upload(unk)
    dt, loc = h.compute_dt()
    t, dt_old = 0.0, dt
    for _ in range(steps):
        h(t + dt, dt, dt_old)
        if o is not None:
            assert o.hydro(ref, t + dt, dt, dt_old) == 0
        t += dt
        new, loc = h.compute_dt()                 # raises where a status bit is set
        dt_old, dt = dt, next_dt(new, dt)
    out = grid.new_unk()
    h.download(out)
    return out, new, tuple(loc)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["velocity", "subnormal", "thin", "vanish", "species", "huge"])
@pytest.mark.parametrize("name", sorted(GRIDS))
def test_fp64_equals_oracle(name, kind):
    grid, unk, params = _state(name, kind)
    ref = unk.copy()
    o = orc.Oracle(params, grid)
    o.eos_init(ref)
    h = Hydro(params, grid)
    out, dt, loc = _run(h, grid, unk, 2, o, ref)
    h.close()
    _, dto, loco = o.compute_dt(ref)
    assert (dt, loc) == (dto, tuple(loco))
    a, b = grid.interior(out), grid.interior(ref)
    shok = [v for v in range(grid.nunk) if v != VAR["shok"]]
    assert np.all(np.isfinite(b))
    bad = a[..., shok] != b[..., shok]
    assert not bad.any(), (int(bad.sum()), a[..., shok][bad][:3], b[..., shok][bad][:3])


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(GRIDS))
def test_mixed_vanishing_pressures_close_to_oracle(name):
    grid, unk, params = _state(name, "vanish")
    params.precision = abi.PREC_MIXED
    ref = unk.copy()
    o = orc.Oracle(params, grid)
    o.eos_init(ref)
    h = Hydro(params, grid)
    out, _, _ = _run(h, grid, unk, 2, o, ref)
    h.close()
    for k, l1 in conserved_l1(out, ref, grid).items():
        assert l1 <= 1e-6, (k, l1)


@pytest.mark.gpu
@pytest.mark.parametrize("rs", [abi.RS_HLLC, abi.RS_EXACT])
def test_fma_runs_follow_the_setting(rs):
    """FP64_FMA kernels on runs are compiled (and contracted) apart from the
    one-block ones: with mx_runs = 1 a full step equals the block-list step
    bit for bit, on runs to rounding."""
    grid = UniformGrid(3, (8, 8, 8), (4, 4, 4), bc="periodic")
    unk = setups.kelvin_helmholtz(grid)
    params = abi.default_params(gamma=5.0 / 3.0, precision=abi.PREC_FP64_FMA, riemann_solver=rs)
    out = {}
    for how in ("runs", "one", "list"):
        h = Hydro(params, grid)
        assert h.tuning["mx_runs"] == 4
        if how == "one":
            h.tuning = dict(h.tuning, mx_runs=1)
        h.upload(unk)
        dt, _ = h.compute_dt()
        for _ in range(3):
            if how == "list":
                h.step_blocks(range(grid.nblocks), 0.0, dt, dt)
            else:
                h(0.0, dt, dt)
        out[how] = grid.new_unk()
        h.download(out[how])
        h.close()
    assert np.array_equal(out["one"], out["list"])
    # three steps of a state of order one: a few roundings of 1e-16 each
    assert np.abs(out["runs"] - out["one"])[..., [VAR[v] for v in ("dens", "velx", "vely", "velz", "eint")]].max() <= 1e-13
