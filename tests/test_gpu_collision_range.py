"""The collision's short form of the reference's operations holds where no
quotient leaves the range of the exact division by FMA; every other cell takes
IEEE divisions. Fields far outside the physical range, over whole planes and
in single cells beside ordinary ones, non-finite ones included, against the
oracle (tolerance 0: both forms round as the reference does)."""
import numpy as np
import pytest

import amrlbm
from amrlbm import AmrLbm
from oracle_lib import Oracle
from parity import copy_state_to_gpu, field_ids, randomize_leaves

pytestmark = pytest.mark.gpu


def scale(orc, every, c=1.0, g=1.0, add=0.0):
    """Multiplies C and g of every `every`-th interior cell of the leaves."""
    for bid in field_ids(orc, leaves_only=True):
        b = orc.download_block(int(bid))
        f = {k: b[k].copy() for k in ("h", "g", "C", "P", "Ux", "Uy")}
        n = b["C"].size
        mask = (np.arange(n) % every == 0).reshape(b["C"].shape)
        f["C"][mask] = f["C"][mask] * c + add
        m = (np.arange(f["g"][0].size) % every == 0).reshape(f["g"][0].shape)
        f["g"][:, m] *= g
        orc.upload_block(int(bid), f["h"], f["g"], f["C"], f["P"], f["Ux"], f["Uy"])


def compare(gpu, orc, fields):
    """Finite values equal, non-finite ones in the same places: where populations
    overflowed, the reference's sums over e_x g(k) hold 0*inf and give NaN, the
    device's, which leave the zero terms out, an infinity."""
    ids = field_ids(orc, leaves_only=True)
    d = gpu.download_fields(ids)
    for i, bid in enumerate(ids):
        o = orc.download_block(int(bid))
        for k in fields:
            a, b = d[k][i].reshape(o[k].shape, order="F"), o[k]
            ok = (a == b) | (~np.isfinite(a) & ~np.isfinite(b))
            assert ok.all(), f"block {bid} field {k}: {np.argwhere(~ok)[:5].tolist()}"


@pytest.mark.parametrize("every", [1, 7])
@pytest.mark.parametrize("name,kw", [
    ("tiny_contrast", dict(c=1e-285)), ("subrange_contrast", dict(c=1e-296)), ("huge_contrast", dict(c=1e90)),
    ("overflowing", dict(c=1e200)), ("fast", dict(g=1e40)), ("faster", dict(g=1e140)), ("slow", dict(g=1e-290)),
    ("constant", dict(c=0.0, add=1.0)), ("infinite", dict(add=np.inf)), ("nan", dict(add=np.nan)),
])
def test_collision_outside_the_usual_range(name, kw, every):
    p = amrlbm.bubble_params(16, 32, 3, radius=10.0, xc=64.0, yc=80.0, rho_ratio=1000.0, visc_ratio=100.0,
                             eo=10.0, mo=1e-5, n=8, regrid_every=1000)
    orc = Oracle(p)
    orc.initialize_rising_bubble()
    randomize_leaves(orc, seed=7)
    scale(orc, every, **kw)
    with AmrLbm(p) as gpu:
        copy_state_to_gpu(orc, gpu)
        for f in ("fill_ghost_cells_c2", "phase_field_lbm_h_g", "macroscopic_values_h",
                  "fill_ghost_cells_c", "macroscopic_values_g"):
            getattr(orc, f)()
            getattr(gpu, f)()
        compare(gpu, orc, ("h", "g", "C", "P", "Ux", "Uy"))
        orc.main_loop(1)  # the collision that evaluates P and U itself
        gpu.main_loop(1)
        gpu.sync()
        compare(gpu, orc, ("h", "g", "C"))
