"""axb_c2p_cells with Noble first on the ideal gas (its own kernel: the common
path per thread, anything else through the whole cascade): recovered cells
against the primitives they were made from, and the cells that leave the
common path against what the cascade makes of them, at block remainders.
Tolerance: the Newton search ends at a relative step of 1e-10 and converges
quadratically, so its error is rounding amplified by the recovery, below
1e-9 for W <= 5 and b^2/rho <= 1."""
import numpy as np
import pytest

from asterx_b200 import abi
from asterx_b200 import workloads as W

GAMMA = 5.0 / 3.0
OUT = ["rho", "eps", "press", "velx", "vely", "velz", "w_lorentz", "Ye", "temperature",
       "entropy"]


def _run(engine, c, n, seeds=None, **over):
    torch = engine.torch
    t = {k: torch.as_tensor(np.ascontiguousarray(c[k]), device=engine.device)
         for k in abi.CELL_INPUTS}
    for k, v in (seeds or {}).items():
        t[k] = torch.as_tensor(np.ascontiguousarray(v), device=engine.device)
    out = {k: torch.full((n,), -7.0, dtype=torch.float64, device=engine.device)
           for k in OUT + ["iters", "flag", "fallback"]}
    p = abi.default_params(**{**dict(c2p_prime="noble", c2p_second="palenzuela", c2p_tol=1e-10,
                                     max_iter=100, vw_lim=60.0, B_lim=1e3, rho_abs_min=1e-14,
                                     t_atmo=1e-12), **over})
    eos = engine.eos_idealgas(GAMMA, rho=(1e-40, 1e10), eps=(0.0, 1e10))
    engine.status_reset()
    engine.c2p_cells(engine.cells(n, {**t, **out}), p, eos)
    st = engine.status()
    return {k: v.cpu().numpy() for k, v in out.items()}, st


def _cells(n, seed):
    return W.c2p_cells(n, seed=seed, gamma=GAMMA, rho_range=(1e-6, 1.0), eps_range=(1e-3, 10.0),
                       w_range=(1.0, 5.0), sigma_range=(1e-4, 1.0))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 128, 129, 1000])
def test_recovered_cells(engine, n):
    c = _cells(n, seed=n)
    got, st = _run(engine, c, n)
    assert (got["flag"] == abi.C2P_PRIME).all() and st["c2p_fail"] == 0
    assert (got["fallback"] == 0).all() and (got["iters"] >= 1).all()
    assert st["iter_hist"].sum() == n
    for k in OUT:
        want = c["W" if k == "w_lorentz" else k]
        scale = np.maximum(np.abs(want), 1e-3 if k.startswith("vel") else 0.0)
        assert np.max(np.abs(got[k] - want) / scale) <= 1e-9, k
    # seeds one step away: the same cells in fewer steps
    seeds = {"seed_" + k: c[k] * 1.01 for k in ("rho", "eps", "Ye")}
    seeds.update({"seed_" + k: c[k] * 0.999 for k in ("velx", "vely", "velz")})
    warm, _ = _run(engine, c, n, seeds)
    assert (warm["flag"] == abi.C2P_PRIME).all()
    assert warm["iters"].mean() < got["iters"].mean()
    assert np.max(np.abs(warm["rho"] - c["rho"]) / c["rho"]) <= 1e-9


@pytest.mark.gpu
def test_cells_off_the_common_path(engine):
    n = 300
    c = _cells(n, seed=3)
    sq = c["dens"] / (c["rho"] * c["W"])
    c["dens"][0:40] = sq[0:40] * 1e-15      # below the atmosphere's cut
    c["tau"][40:60] = np.nan                # neither scheme recovers
    for q in "xyz":
        c["dB" + q][60:80] = 2e3 * sq[60:80]  # above B_lim in both schemes
    c["gxx"][80:90] = -1.0                  # no metric
    got, st = _run(engine, c, n)
    flag = got["flag"]
    assert (flag[:40] == abi.C2P_ATMO).all() and (got["iters"][:40] == -1).all()
    assert (got["rho"][:40] == 1e-14).all() and (got["w_lorentz"][:40] == 1.0).all()
    assert (flag[40:90] == abi.C2P_FAIL).all() and (got["rho"][40:90] == 1e-14).all()
    assert (got["velx"][:90] == 0.0).all()
    assert st["c2p_fail"] == 50 and st["error_word"] & abi.EW_C2P_FAIL
    assert (flag[90:] == abi.C2P_PRIME).all()
    assert np.max(np.abs(got["rho"] - c["rho"])[90:] / c["rho"][90:]) <= 1e-9


@pytest.mark.gpu
def test_cells_floors(engine):
    n = 200
    c = _cells(n, seed=5)
    t_atmo = float(np.median(c["temperature"]))
    got, _ = _run(engine, c, n, t_atmo=t_atmo, vw_lim=3.0)
    cold = c["temperature"] < t_atmo * (1 - 1e-9)
    fast = c["W"] > np.sqrt(10.0) * (1 + 1e-9)
    assert cold.sum() > 20 and fast.sum() > 20
    wlim = np.sqrt(1.0 + 9.0)
    assert np.max(np.abs(got["w_lorentz"][fast] - wlim)) <= 1e-14
    D = c["rho"] * c["W"]
    assert np.max(np.abs(got["rho"][fast] - D[fast] / wlim) / D[fast]) <= 1e-13
    floored = cold & ~fast
    assert np.max(np.abs(got["temperature"][floored] - t_atmo)) <= 1e-15 * t_atmo
    assert np.max(np.abs(got["eps"][floored] - t_atmo / (GAMMA - 1))) <= 1e-14 * t_atmo


@pytest.mark.gpu
@pytest.mark.parametrize("first", ["noble", "palenzuela"])
def test_cells_on_the_atmosphere_cut(engine, first):
    """With atmo_tol = 0 a cell set to the atmosphere (D = sqrt(gamma) rho_atm)
    lies on the cut itself and is atmosphere again, whatever the metric and
    whichever scheme is first; one just above it (1e-12) is not."""
    n = 1000
    c = _cells(n, seed=11)
    rho = 3e-9
    # det gamma as the recovery forms it, so that D is on the cut to the bit
    xx, xy, xz, yy, yz, zz = (c["g" + k] for k in ("xx", "xy", "xz", "yy", "yz", "zz"))
    det = xx * (yy * zz - yz * yz) - xy * (xy * zz - yz * xz) + xz * (xy * yz - yy * xz)
    c["dens"] = np.sqrt(det) * rho
    c["dens"][::2] *= 1.0 + 1e-12
    second = "palenzuela" if first == "noble" else "noble"
    got, _ = _run(engine, c, n, rho_abs_min=rho, atmo_tol=0.0, c2p_prime=first,
                  c2p_second=second)
    assert (got["flag"][1::2] == abi.C2P_ATMO).all()
    assert (got["iters"][1::2] == -1).all() and (got["rho"][1::2] == rho).all()
    assert (got["flag"][::2] != abi.C2P_ATMO).all()


@pytest.mark.gpu
def test_small_and_large_launches_agree(engine):
    """A launch that fills the GPU (8 CTAs per SM) and launches of few blocks
    (the registers the cascade wants) give every cell the same bits, on the
    common path and off it; the failure count is that of the flags."""
    n = (1 << 18) + 77
    c = _cells(n, seed=21)
    u = np.random.default_rng(4).uniform(size=n)
    sq = c["dens"] / (c["rho"] * c["W"])
    c["tau"] = np.where(u < 0.01, np.nan, c["tau"])
    c["dBx"] = np.where((u > 0.01) & (u < 0.03), c["dBx"] * 1e9, c["dBx"])
    c["dens"] = np.where((u > 0.03) & (u < 0.04), sq * 1e-15, c["dens"])
    c["gxx"] = np.where((u > 0.04) & (u < 0.05), -1.0, c["gxx"])
    got, st = _run(engine, c, n, B_lim=1e8)
    flags = np.bincount(got["flag"].astype(int), minlength=7)
    assert flags[abi.C2P_FAIL] == st["c2p_fail"] > 0 and flags[abi.C2P_ATMO] > 0
    assert flags[abi.C2P_PRIME] > 0.9 * n
    for lo, hi in ((0, 1), (1000, 3000), (n // 2, n // 2 + 5000), (n - 100, n)):
        part, _ = _run(engine, {k: v[lo:hi] for k, v in c.items()}, hi - lo, B_lim=1e8)
        for k, v in part.items():
            assert np.array_equal(v, got[k][lo:hi], equal_nan=True), (k, lo)
