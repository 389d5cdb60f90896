"""The box recovery with Palenzuela first (the fast pass: tiles of 128 cells
along a row, with the root searches of a tabulated EOS drawn from a block's
pool) against the restated reference, on rows at the edges of a tile: flags
identical, primitives and conserved variables within 1e-10 of their largest
value (Brent's bracket is 1e-12 wide; the last ulps of its root function are
amplified by at most W^2 = 9)."""
import numpy as np
import pytest

from asterx_b200 import abi
from asterx_b200 import workloads as W
from oracle.oracle import restatement
from tests.helpers import errors, full_fields, interior

OUT = (["rho", "eps", "press", "velx", "vely", "velz", "temperature", "entropy", "Ye",
        "Bvecx", "Bvecy", "Bvecz"] + abi.CONS + abi.SAVED)


@pytest.mark.gpu
@pytest.mark.parametrize("table", [False, True])
@pytest.mark.parametrize("n", [(1, 1, 1), (31, 2, 3), (128, 2, 1), (129, 1, 2), (37, 5, 3)])
def test_recovery_tiles(engine, n, table):
    kw = dict(n=n, ng=5, seed=7 + n[0], wmax=3.0)
    if table:
        L, f = W.tabulated_box(**kw)
    else:
        L, f = W.curved_box(sigma=(1e-3, 0.3), theta=(0.1, 1.0), **kw)
    W.cons_from_prims(L, f)
    W.perturbed_saved(f, seed=3)
    f = full_fields(L, f)
    p = abi.default_params(c2p_prime="palenzuela", c2p_second="noble", c2p_tol=1e-12,
                           max_iter=100, reconstruct_with_temperature=int(table),
                           **(dict(t_atmo=0.011) if table else {}))
    host = {k: a.copy() for k, a in f.items()}
    ref = restatement()
    ref.setup(L, p, host)
    if table:
        ref.eos_tabulated(*W.synthetic_table(nrho=60, ntemp=40, nye=12))
        eos = engine.eos_tabulated(*W.synthetic_table(nrho=60, ntemp=40, nye=12))
    else:
        ref.eos_idealgas(4.0 / 3.0, rho=(1e-40, 1e10), eps=(0.0, 1e10))
        eos = engine.eos_idealgas(4.0 / 3.0, rho=(1e-40, 1e10), eps=(0.0, 1e10))
    ref.con2prim_group()
    dev = engine.upload(L, f)
    engine.con2prim_group(L, dev, p, eos)
    got = {k: dev[k].cpu().numpy() for k in OUT + ["con2prim_flag"]}
    flags = interior(L, "x", host["con2prim_flag"])
    assert np.array_equal(interior(L, "x", got["con2prim_flag"]), flags)
    assert (flags == abi.C2P_PRIME).mean() > 0.9
    for k in OUT:
        emax, _ = errors(interior(L, k, got[k]), interior(L, k, host[k]))
        assert emax <= 1e-10, (k, emax)
