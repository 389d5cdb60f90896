"""axb_tmunu against a numpy restatement of AsterX_Tmunu with the same order
of operations (AsterX/src/tmunu.cxx:76-178, AsterUtils/src/
aster_interp.hxx:97-148), on boxes at the edges of the fourth-order kernel's
tiles (29 x 13 x 3 vertices; a box of n cells has n + 1).  Neither side
contracts multiply-adds, so the results are equal to the bit."""
import numpy as np
import pytest

from asterx_b200 import abi
from asterx_b200 import workloads as W
from tests.helpers import full_fields


def _lower(g, v):
    return [g[0] * v[0] + g[1] * v[1] + g[2] * v[2],
            g[1] * v[0] + g[3] * v[1] + g[4] * v[2],
            g[2] * v[0] + g[4] * v[1] + g[5] * v[2]]


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _at(a, axis, by):
    return np.roll(a, -by, axis=2 - axis)


def _c2v(a, order):
    if order == 2:
        s = 0.0
        for k in (0, 1):
            for j in (0, 1):
                for i in (0, 1):
                    s = s + _at(_at(_at(a, 0, -i), 1, -j), 2, -k)
        return s / 8.0
    wt = [-1 / 16, 9 / 16, 9 / 16, -1 / 16]

    def along(f, axis):
        s = 0.0
        for m in range(4):
            s = s + wt[m] * _at(f, axis, m - 2)
        return s

    avg = 0.0
    for i, j, k in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
        g = along(along(a, i), j)
        for m in range(4):
            avg = avg + wt[m] * _at(g, k, m - 2)
    return avg / 3.0


def _tmunu(L, f, order, recvar):
    v = lambda n: _c2v(L.view(f[n]), order)
    rho, eps, press = v("rho"), v("eps"), v("press")
    B = [v("Bvec" + x) for x in "xyz"]
    g = [L.view(f[n]) for n in ("gxx", "gxy", "gxz", "gyy", "gyz", "gzz")]
    sym = lambda p, q: g[{(0, 0): 0, (0, 1): 1, (0, 2): 2, (1, 1): 3, (1, 2): 4,
                          (2, 2): 5}[(p, q)]]
    alp = L.view(f["alp"])
    beta = [L.view(f["beta" + x]) for x in "xyz"]
    bl = _lower(g, beta)
    if recvar == "v":
        vu = [v("vel" + x) for x in "xyz"]
        vl = _lower(g, vu)
        w = 1.0 / np.sqrt(1.0 - _dot(vu, vl))
    else:
        z = [v("zvec_" + x) for x in "xyz"]
        zl = _lower(g, z)
        w = np.sqrt(1.0 + _dot(z, zl))
        vu, vl = [x / w for x in z], [x / w for x in zl]
    rhw2 = (rho * (1.0 + eps) + press) * w * w
    ut = -alp + _dot(bl, vu)
    ui = [vu[d] - beta[d] / alp for d in range(3)]
    bst = w * _dot(B, vl) / alp
    bsi = [(B[d] + alp * bst * w * ui[d]) / w for d in range(3)]
    gtt = -alp * alp + _dot(bl, beta)
    bstl = bst * gtt + _dot(bsi, bl)
    gb = _lower(g, bsi)
    bsl = [bst * bl[d] + gb[d] for d in range(3)]
    bs2 = bst * bstl + _dot(bsi, bsl)
    w2 = w * w
    t = [rhw2 * ut * ut + press * gtt + (w2 * ut * ut + 0.5 * gtt) * bs2 - bstl * bstl]
    for d in range(3):
        t.append(rhw2 * ut * vl[d] + press * bl[d]
                 + (w2 * ut * vl[d] + 0.5 * bl[d]) * bs2 - bstl * bsl[d])
    for p in range(3):
        for q in range(p, 3):
            t.append(rhw2 * vl[p] * vl[q] + press * sym(p, q)
                     + (w2 * vl[p] * vl[q] + 0.5 * sym(p, q)) * bs2 - bsl[p] * bsl[q])
    return t


@pytest.mark.gpu
@pytest.mark.parametrize("n,order,recvar", [
    ((28, 12, 2), 4, "z"), ((29, 13, 3), 4, "v"), ((30, 11, 4), 4, "z"), ((3, 3, 3), 4, "v"),
    ((58, 25, 6), 4, "z"), ((12, 10, 9), 2, "z"), ((127, 3, 4), 2, "v")])
def test_tmunu_tiles(engine, n, order, recvar):
    L, f = W.curved_box(n=n, ng=3, seed=sum(n), wmax=2.0, njumps=1)
    W.cons_from_prims(L, f)
    f = full_fields(L, f)
    rng = np.random.default_rng(5)
    held = [rng.normal(size=L.size) for _ in range(10)]
    dev = engine.upload(L, f)
    eT = [engine.torch.as_tensor(h, device=engine.device) for h in held]
    engine.tmunu(L, dev, abi.default_params(recon_type={"v": 0, "z": 1}[recvar]), eT,
                 interp_order=order)
    engine.torch.cuda.synchronize()
    sl = L.interior((0, 0, 0))
    for h, t, want in zip(held, eT, _tmunu(L, f, order, recvar)):
        full = L.view(h.copy())
        full[sl] = full[sl] + want[sl]
        assert np.isfinite(want[sl]).all()
        assert np.array_equal(t.cpu().numpy(), full.reshape(-1))  # ghosts as they were
