"""The exact Riemann solver at the edges of its arithmetic (marked gpu).

* its error against extended precision, over the isolated workload's
  states, is no larger than that of the same formulas in plain IEEE double
  arithmetic (1 % for the scatter between two roundings of one formula);
* pairs with densities and pressures far outside the range of its
  branch-free arithmetic ([2^-300, 2^300)), on either side of that range's
  ends, and with pressure ratios beyond the largest double, solve as the
  oracle does.
"""
import numpy as np
import pytest

from flash5_b200 import abi, setups
from flash5_b200.grid import UniformGrid, VAR
from flash5_b200.hydro import Hydro, next_dt
from oracle import orc
from tests.test_gpu_parity import conserved_l1


@pytest.fixture(scope="module")
def rs():
    from flash5_b200.riemann import ExactRiemann
    r = ExactRiemann(0)
    yield r
    r.close()


def _star(S, T, tol, evals):
    """(p*, u*) of the states S [7, n] in the type T by the solver's formulas
    and stopping rule: Newton on w = p^z from the two-rarefaction guess until
    the step, or the step predicted from the last two, is small."""
    dl, ul, pl, dr, ur, pr, g = (a.astype(T) for a in S)
    one, two, half = T(1), T(2), T(0.5)
    z, n = (g - one) / (two * g), two * g / (g - one)
    k2, a2, g6 = two / (g - one), two / (g + one), (g - one) / (g + one)
    cl, cr, wl, wr = np.sqrt(g * pl / dl), np.sqrt(g * pr / dr), np.exp2(z * np.log2(pl)), np.exp2(z * np.log2(pr))
    kl, kr, du = k2 * cl / wl, k2 * cr / wr, ur - ul
    seven = S[6] == 1.4                                    # n = 7, else 5

    def power(w):
        w2 = w * w
        w4 = w2 * w2
        return w4 * np.where(seven, w2 * w, w)

    def side(w, p, dpdw, wk, pk, dk, k):
        r = one / (g6 * pk + p)
        q = np.sqrt(a2 / dk * r)
        sh = w > wk
        return np.where(sh, (p - pk) * q, k * (w - wk)), np.where(sh, (one - half * (p - pk) * r) * q * dpdw, k)
    w = (cl + cr - half * (g - one) * du) / (half * (g - one) * (kl + kr))
    done, prev, us = np.zeros(w.shape, bool), np.zeros(w.shape, T), np.zeros(w.shape, T)
    for _ in range(evals):
        p = power(w)
        fl, fdl = side(w, p, n * p / w, wl, pl, dl, kl)
        fr, fdr = side(w, p, n * p / w, wr, pr, dr, kr)
        step = np.where(done, T(0), (fl + fr + du) / (fdl + fdr))
        step = np.where(w > step, step, half * w)
        size = np.abs(step)
        # f linearised from the last evaluation to the returned w
        us = np.where(done, us, half * (ul + ur) + half * ((fr - fdr * step) - (fl - fdl * step)))
        new = (size <= z * T(tol) * w) | ((size < prev) & (size ** 3 <= T(0.01) * z * T(tol) * w * prev ** 2))
        w, prev, done = w - step, size, done | new
    return np.stack([power(w), us])


@pytest.mark.gpu
def test_error_no_larger_than_plain_arithmetic(rs):
    S = rs.generate(424242, 400000)
    out, _, flags = rs.solve(S, learned=False)
    assert rs.sync() == 0
    ok = (flags.cpu().numpy() & 2) == 0
    S, out = S.cpu().numpy()[:, ok], out.cpu().numpy()[:, ok]
    true = _star(S, np.longdouble, 1e-30, 40)
    plain = _star(S, np.float64, 1e-12, 40)
    norm = np.sqrt((true ** 2).sum())
    e_gpu, e_plain = (float(np.sqrt(((a - true) ** 2).sum()) / norm) for a in (out, plain))
    assert e_gpu <= 1.01 * e_plain, (e_gpu, e_plain)


PRESSURES = [(1e-160, 1e160), (1e-95, 1e95), (1e-89, 1e89), (1e-300, 1e-290), (1e290, 1e300), (1e-310, 1e-300),
             (1e-100, 1e-101), (2.0 ** -299, 2.0 ** -301), (2.0 ** 299, 2.0 ** 301), (2.0 ** 301, 2.0 ** 302)]


@pytest.mark.gpu
@pytest.mark.parametrize("learned", [False, True])
def test_out_of_range_pairs_match_oracle(rs, learned):
    rows = []
    for g in (1.4, 5.0 / 3.0, 1.3):
        for a, b in PRESSURES:
            for pl, pr in ((a, b), (b, a)):
                for dr in (1.0, 0.125):
                    c = np.sqrt(g * max(a, b))
                    rows += [(1.0, m * c, pl, dr, -m * c, pr, g) for m in (0.0, 0.5, -0.2)]
        for d in (1e-95, 2.0 ** -300, 2.0 ** -301, 2.0 ** 299, 2.0 ** 300):     # densities
            rows += [(d, 0.0, 1.0, 0.5 * d, 0.0, 0.1, g), (0.5 * d, 0.0, 0.1, d, 0.0, 1.0, g)]
    S = np.array(rows).T.copy()
    ps, us, _, st = orc.star_batch(*S, tol=1e-12, max_iter=50)
    ok = st == 0
    assert ok.mean() > 0.9
    o, _, fl = rs.solve(rs.torch.tensor(np.ascontiguousarray(S[:, ok]), device="cuda:0"), learned=learned)
    assert rs.sync() == 0
    o, fl = o.cpu().numpy(), fl.cpu().numpy()
    assert not (fl & 6).any(), np.argwhere(fl & 6)[:4]
    rel = np.abs(o[0] / ps[ok] - 1)
    assert rel.max() <= 1e-11, (rel.max(), S[:, ok][:, rel.argmax()])
    # u* is the difference of velocities as large as the sound speeds
    c = np.sqrt(S[6] * np.maximum(S[2] / S[0], S[5] / S[3]))[ok] + np.abs(S[1][ok])
    assert (np.abs(o[1] - us[ok]) / c).max() <= 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-100, 1e100])
@pytest.mark.parametrize("flip", [False, True])
def test_hydro_out_of_range_matches_oracle(scale, flip):
    """FP64 steps with the exact solver, the pressures (and energies) outside
    the range, the larger one on either side."""
    grid = UniformGrid(2, (8, 8), (4, 2), bc="outflow")
    p = (0.1 * scale, scale) if flip else (scale, 0.1 * scale)
    unk = setups.sod_axis(grid, axis=0, p_l=p[0], p_r=p[1], rho_l=0.125 if flip else 1.0, rho_r=1.0 if flip else 0.125)
    params = abi.default_params(riemann_solver=abi.RS_EXACT, tiny=1e-300, smallp=1e-300, smalle=1e-300)
    ref = unk.copy()
    o = orc.Oracle(params, grid)
    o.eos_init(ref)
    h = Hydro(params, grid)
    h.upload(unk)
    dt, _ = h.compute_dt()
    dt_old, t = dt, 0.0
    for _ in range(3):
        h(t + dt, dt, dt_old)
        assert o.hydro(ref, t + dt, dt, dt_old) == 0
        t += dt
        new, _ = h.compute_dt()
        _, ref_dt, _ = o.compute_dt(ref)
        assert abs(new - ref_dt) <= 1e-10 * ref_dt
        dt_old, dt = dt, new
    out = grid.new_unk()
    h.download(out)
    h.close()
    for k, l1 in conserved_l1(out, ref, grid).items():
        assert l1 <= 1e-10, (k, l1)


@pytest.mark.gpu
def test_a_solver_holds_no_training_memory():
    """Creating a solver takes one small allocation (cudaMalloc hands out
    2 MB); the gradient rows come with the first training."""
    import torch
    from flash5_b200.riemann import ExactRiemann
    first = ExactRiemann(0)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    r = ExactRiemann(0)
    assert free - torch.cuda.mem_get_info()[0] <= 2 << 20
    X, T = torch.randn(64, 8, device="cuda:0"), torch.randn(64, device="cuda:0")
    r.train(X, T, 64, epochs=1, batch=32)
    r.close()
    first.close()
