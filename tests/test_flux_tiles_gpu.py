"""The RHS group at the edges of the flux passes' tiles (30-cell chunks along
x, 128 pencils of the transverse plane, pencil segments of one step and of
several) and of the sources' z columns, against the restated reference: largest error over the largest
value <= 1e-12, as the RHS parity tests take it (both sides evaluate the same
formulas in FP64; multiply-add contraction and shared reciprocals move the
last ulps)."""
import numpy as np
import pytest

from asterx_b200 import abi
from asterx_b200 import workloads as W
from oracle.oracle import restatement
from tests.helpers import errors, full_fields, interior

SIZES = [(3, 4, 5), (29, 4, 3), (30, 5, 33), (31, 18, 4), (64, 3, 35), (5, 66, 17)]
# boxes whose pencils and columns take 6 or 7 steps, the last one fewer, on a
# GPU of SMS multiprocessors (test_steps.py holds the split to that; the boxes
# above take one step a thread)
LONG = [(61, 130, 37)]
SMS = 148


def _box(n, seed):
    # (reconstructed velocities stay below 1 on boxes this coarse)
    L, f = W.curved_box(n=n, ng=5, seed=seed, wmax=1.3, sigma=(1e-3, 0.3), theta=(0.1, 1.0),
                        njumps=0)
    # the generator clips rho, and an exactly symmetric stencil of clipped
    # values leaves WENO-Z's weights to rounding
    u = 1.0 + 1e-3 * np.random.default_rng(seed).uniform(size=L.size)
    f["rho"], f["press"] = f["rho"] * u, f["press"] * u
    f["entropy"] = f["entropy"] * u ** (-1.0 / 3.0)
    W.cons_from_prims(L, f)
    return L, full_fields(L, f)


@pytest.mark.gpu
@pytest.mark.parametrize("recon,flux,order", [("wenoz", "hlle", 2), ("mp5", "lxf", 4),
                                              ("ppm", "hlle", 2), ("minmod", "hlle", 4)])
@pytest.mark.parametrize("n", SIZES + LONG)
def test_rhs_tiles(engine, n, recon, flux, order):
    if n in LONG:
        props = engine.torch.cuda.get_device_properties(engine.device)
        assert props.multi_processor_count == SMS
    L, f = _box(n, seed=sum(n))
    p = abi.default_params(reconstruction_method=recon, flux_type=flux,
                           local_spatial_order=order)
    host = {k: a.copy() for k, a in f.items()}
    ref = restatement()
    ref.setup(L, p, host)
    ref.eos_idealgas(4.0 / 3.0, rho=(1e-40, 1e10), eps=(0.0, 1e10))
    ref.rhs_group()
    dev = engine.upload(L, f)
    eos = engine.eos_idealgas(4.0 / 3.0, rho=(1e-40, 1e10), eps=(0.0, 1e10))
    engine.status_reset()
    engine.rhs_group(L, dev, p, eos)
    st = engine.status()
    assert st["error_word"] == 0 and 0.1 < st["max_speed"] < 1.1
    for k in abi.HYDRO_RHS + abi.AVEC_RHS:
        got = dev[k].cpu().numpy()
        emax, _ = errors(interior(L, k, got), interior(L, k, host[k]))
        assert emax <= 1e-12, (k, emax)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(8, 6, 5), (33, 20, 17)])
def test_batch_equals_single_boxes(engine, n):
    """The same box alone and as every box of a level: the passes may take
    other tiles and segments, never other values (to the last ulps of the
    multiply-add contraction, carried by one substep)."""
    p = abi.default_params(reconstruction_method="wenoz", flux_type="hlle",
                           c2p_prime="palenzuela", c2p_second="noble", c2p_tol=1e-12,
                           max_iter=100, recon_type=1)
    eos = engine.eos_idealgas(4.0 / 3.0, rho=(1e-40, 1e10), eps=(0.0, 1e10))
    evolved = abi.CONS + ["Avec_x", "Avec_y", "Avec_z", "Psi"]

    def state(seed):
        L, f = W.curved_box(n=n, ng=3, seed=seed, wmax=2.0, sigma=(1e-3, 0.1), njumps=0)
        W.cons_from_prims(L, f)
        W.perturbed_saved(f, seed=3)
        dev = engine.upload(L, full_fields(L, f))
        return L, dev, {k: dev[k].clone() for k in evolved}

    L, one, one_n = state(4)
    dt = 0.05 * min(L.dx)
    engine.substep(L, one, one_n, p, eos, 0.0, 1.0, 1.0, dt)
    boxes = [state(4) for _ in range(3)]
    batch = engine.batch_create([b[0] for b in boxes], [b[1] for b in boxes],
                                [b[2] for b in boxes], p, eos)
    engine.batch_substep(batch, 0.0, 1.0, 1.0, dt)
    engine.torch.cuda.synchronize()
    for _, dev, _ in boxes:
        for k in evolved + abi.PRIMS:
            a, b = dev[k].cpu().numpy(), one[k].cpu().numpy()
            emax, _ = errors(a, b)
            assert emax <= 1e-10, (k, emax)
    engine.batch_destroy(batch)
