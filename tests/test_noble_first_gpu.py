"""The box recovery with Noble first on the ideal gas, alone and as the boxes of
a level: its own kernels, whose common path leaves cells inside the mask,
non-finite ones and those of a failed search to the whole cascade.  Against the
restated reference on rows at the edges of a block: flags identical, failures
counted, values within 1e-9 of their largest value where a search stops at 1e-12
of its unknown (the recovery amplifies that by at most about 1e3 for W <= 3,
b^2/rho <= 0.3 and eps >= 0.1)."""
import numpy as np
import pytest

from asterx_b200 import abi
from asterx_b200 import workloads as W
from oracle.oracle import restatement
from tests.helpers import errors, full_fields, interior

OUT = (["rho", "eps", "press", "velx", "vely", "velz", "temperature", "entropy", "Ye",
        "Bvecx", "Bvecy", "Bvecz"] + abi.CONS + abi.SAVED)
GAMMA = 4.0 / 3.0
EOS = dict(rho=(1e-40, 1e10), eps=(0.0, 1e10))
SHAPES = [(1, 1, 1), (31, 2, 3), (128, 2, 1), (129, 1, 2), (37, 5, 3), (24, 20, 11)]
# (a level's boxes are at least as wide as its ghost layers)
LEVEL = [(24, 20, 11), (5, 5, 5), (37, 6, 5), (5, 31, 7)]


def _params(max_iter):
    return abi.default_params(c2p_prime="noble", c2p_second="palenzuela", c2p_tol=1e-12,
                              max_iter=max_iter, excise=1, alp_thresh=0.5, rho_BH=1e-2,
                              eps_BH=1e-3, vwlim_BH=1.0)


def _box(n, seed, off_path):
    L, f = W.curved_box(n=n, ng=5, seed=seed, wmax=3.0, sigma=(1e-3, 0.3), theta=(0.1, 1.0))
    W.cons_from_prims(L, f)
    W.perturbed_saved(f, seed=3)
    f = full_fields(L, f)
    if off_path:
        u = np.random.default_rng(seed).uniform(size=L.size)
        f["tau"] = np.where(u < 0.05, np.nan, f["tau"])               # nothing recovers it
        f["dens"] = np.where((u > 0.05) & (u < 0.1), 1e-16, f["dens"])  # atmosphere
        # seeds so far off that 46 steps rarely bring the search back
        f["saved_eps"] = np.where((u > 0.1) & (u < 0.2), 1e15, f["saved_eps"])
        i = np.arange(L.size) % L.sy
        f["alp"] = np.where(i > L.ng + (3 * n[0]) // 4, 0.1, f["alp"])  # inside the mask
    return L, f


def _restated(L, f, max_iter):
    host = {k: a.copy() for k, a in f.items()}
    ref = restatement()
    ref.setup(L, _params(max_iter), host)
    ref.eos_idealgas(GAMMA, **EOS)
    ref.con2prim_group()
    return host


def _want(L, f, max_iter):
    """The restated recovery, and the cells it is compared in: not those whose
    first search ends with the last allowed step (in the restatement the flag
    is another with a step more or less), which is a matter of the last ulp.
    The second scheme's never does: 43 bisections of its bracket (below 10 wide)
    reach 1e-12, fewer than 46."""
    host = _restated(L, f, max_iter)
    flag = interior(L, "x", host["con2prim_flag"])
    sure = np.ones(flag.shape, bool)
    for step in (-1, 1):
        other = _restated(L, f, max_iter + step)["con2prim_flag"]
        sure &= interior(L, "x", other) == flag
    assert (~sure).sum() <= (0.01 * flag.size if max_iter == 46 else 0)
    return host, sure


def _check(L, got, want):
    want, sure = want
    flags = interior(L, "x", want["con2prim_flag"])
    mine = interior(L, "x", got["con2prim_flag"])
    assert np.array_equal(mine[sure], flags[sure])
    for k in OUT:
        a, b = interior(L, k, got[k])[sure], interior(L, k, want[k])[sure]
        assert np.array_equal(np.isnan(a), np.isnan(b)), k
        emax, _ = errors(np.nan_to_num(a), np.nan_to_num(b))
        assert emax <= 1e-9, (k, emax)
    return np.bincount(mine.astype(int).ravel(), minlength=7)


# max_iter: 100 (only the broken cells fail) and 46 (the first search from the
# far seeds is cut off, and the second scheme recovers those cells)
@pytest.mark.gpu
@pytest.mark.parametrize("max_iter,off_path", [(100, False), (100, True), (46, True)])
@pytest.mark.parametrize("n", SHAPES)
def test_box(engine, n, max_iter, off_path):
    L, f = _box(n, 7 + n[0], off_path)
    p = _params(max_iter)
    want = _want(L, f, max_iter)
    dev = engine.upload(L, f)
    eos = engine.eos_idealgas(GAMMA, **EOS)
    engine.status_reset()
    engine.con2prim_group(L, dev, p, eos)
    st = engine.status()
    count = _check(L, {k: dev[k].cpu().numpy() for k in OUT + ["con2prim_flag"]}, want)
    assert st["c2p_fail"] == count[abi.C2P_FAIL]
    if off_path and n == SHAPES[-1]:
        assert count[abi.C2P_FAIL] > 0 and count[abi.C2P_ATMO] > 0
        assert (count[abi.C2P_SECOND] > 0) == (max_iter == 46)
    if not off_path:
        assert count[abi.C2P_PRIME] == count.sum()


@pytest.mark.gpu
@pytest.mark.parametrize("max_iter,off_path", [(100, False), (100, True), (46, True)])
def test_level(engine, max_iter, off_path):
    """Boxes as one level: a substep that sets U = U_n and recovers it."""
    p = _params(max_iter)
    boxes = [_box(n, 7 + n[0], off_path) for n in LEVEL]
    wants = [_want(L, f, max_iter) for L, f in boxes]
    devs = [engine.upload(L, f) for L, f in boxes]
    evolved = abi.CONS + ["Avec_x", "Avec_y", "Avec_z", "Psi"]
    devs_n = [{k: d[k].clone() for k in evolved} for d in devs]
    eos = engine.eos_idealgas(GAMMA, **EOS)
    batch = engine.batch_create([L for L, _ in boxes], devs, devs_n, p, eos)
    engine.status_reset()
    engine.batch_substep(batch, 1.0, 0.0, 0.0, 0.0, periodic=False)
    st = engine.status()
    engine.batch_destroy(batch)
    count = sum(_check(L, {k: d[k].cpu().numpy() for k in OUT + ["con2prim_flag"]}, w)
                for (L, _), d, w in zip(boxes, devs, wants))
    assert st["c2p_fail"] == count[abi.C2P_FAIL]
    assert (count[abi.C2P_FAIL] > 0) == off_path
