"""Which path a fill takes, and that path's values, on meshes whose coarse-fine
boundary meets a wall (a coarser neighbour's ghost cells behind the wall become
foreign cells: no level order) and on one whose coarse-to-fine stencils read a
ghost cell that is itself coarse-to-fine (level order). A mesh within the 2:1
balance has no such cell: every block it could lie in touches a refined block and
so is at most one level coarser than the reading leaf. It is made here by
pointing one block's upper neighbours at a coarser block, which a topology given
by a caller may hold; host oracle and device read the same pointers.

Random fields on the leaves, so that a value of the wrong cell or population
shows: neighbouring populations differ by the order of their weight."""
import numpy as np
import pytest

import amrlbm
from amrlbm import F_LEAF, AmrLbm
from oracle_lib import Oracle
from parity import compare_state, copy_state_to_gpu, field_ids, randomize_leaves
from test_gpu_blocks import near_walls

gpu = pytest.mark.gpu
ULP = {"fp16": 2.0 ** -10, "bf16": 2.0 ** -7}  # of a stored deviation, rounded at random
# A population h moves by at most 20 ulp of the largest deviation, the
# weight 1/9 (a uniform draw below the weight): each store errs by 2 ulp (its
# rounding and the one it carries), after the conversion (times the relaxation's
# 0.79), after the collision, behind a wall, and after streaming; in between
# a fine-to-coarse value multiplies by at most 1.25^2, a coarse-to-fine one by
# 1.19^2 (1.19^4 under level order), Lax-Wendroff by 1.25. g has no carried
# rounding: 16 ulp of the largest value, of which its deviations are at most 1.25.
H_ULPS, G_ULPS = 20, 16


def wall_leaves(orc):
    """Leaves at a wall beside a coarser leaf at the same wall."""
    t, nb = orc.topology(), orc.neighbours()
    lv, leaf = t["level"], (t["flags"] & F_LEAF) != 0
    out = []
    for b in orc.leaves():
        for wall in (2, 3):
            for side in (0, 1):
                q = nb[b - 1, side]
                if nb[b - 1, wall] < 0 and q > 0 and leaf[q - 1] and lv[q - 1] == lv[b - 1] - 1 \
                        and nb[q - 1, wall] < 0:
                    out.append(int(b))
    return out


def mild(n, levels):
    """Density ratio 2: the density stays positive where random fields stream."""
    p = near_walls(n, n, levels, 1000)
    p.rho_l, p.visc_ratio = 0.5, 2.0
    return p


def beside_a_wall(n):
    p = mild(n, 2)
    orc = Oracle(p)
    orc.initialize_rising_bubble()
    assert wall_leaves(orc)
    return p, orc


def coarse_behind_coarse(n):
    """Leaves of three levels; of one leaf of the finest, the upper left child,
    the coarser left neighbour's upper neighbours become a block two levels
    coarser than the leaf."""
    p = mild(n, 3)
    orc = Oracle(p)
    orc.initialize_rising_bubble()
    t, nb = orc.topology(), orc.neighbours()
    lv, leaf = t["level"], (t["flags"] & F_LEAF) != 0
    coarsest = [int(b) for b in orc.leaves() if lv[b - 1] == 1]
    pick = [(int(b), int(nb[b - 1, 0])) for b in orc.leaves()
            if lv[b - 1] == 3 and t["bi"][b - 1] % 2 == 0 and t["bj"][b - 1] % 2 == 1
            and nb[b - 1, 0] > 0 and leaf[nb[b - 1, 0] - 1] and lv[nb[b - 1, 0] - 1] == 2
            and nb[nb[b - 1, 0] - 1, 3] > 0]
    assert coarsest and pick
    q = pick[0][1]
    for side in (3, 7):  # above, above right
        t["nbr_owner"][q - 1, side], t["nbr_slot"][q - 1, side] = coarsest[0], 0
    orc.set_topology(t, orc.counts()["kk"])
    return p, orc


def run(p, orc, precision, calls, **change):
    q = amrlbm.Params(**{**p.as_dict(), **change})
    with AmrLbm(q) as sim:
        copy_state_to_gpu(orc, sim)
        sim.set_precision(precision)
        for steps in calls:
            sim.main_loop(steps)
        sim.sync()
        order = sim.fill_order()
        return order, sim.download_fields(field_ids(orc, leaves_only=True))


MESHES = {"wall": (beside_a_wall, False), "coarse_behind_coarse": (coarse_behind_coarse, True)}


@pytest.mark.parametrize("n", [8, 16])
def test_meshes_have_the_cells(n):
    beside_a_wall(n)
    _, orc = coarse_behind_coarse(n)
    orc.main_loop(1)
    assert orc.level_jumps() == 0


@gpu
@pytest.mark.parametrize("n", [8, 16])
@pytest.mark.parametrize("mesh", list(MESHES))
def test_fp64_path_and_values(mesh, n):
    make, ordered = MESHES[mesh]
    p, orc = make(n)
    randomize_leaves(orc, seed=n, c_lo=0.3, c_hi=0.7)
    with AmrLbm(p) as sim:
        copy_state_to_gpu(orc, sim)
        assert list(sim.fill_order().values()) == 3 * [ordered]
        for steps in (1, 3):
            orc.main_loop(steps)
            sim.main_loop(steps)
            sim.sync()
            compare_state(sim, orc)


@gpu
@pytest.mark.parametrize("precision", ["fp16", "bf16"])
@pytest.mark.parametrize("n", [8, 16])
@pytest.mark.parametrize("mesh", list(MESHES))
def test_16_bit_values(mesh, n, precision):
    """One step against the oracle's, population by population."""
    make, ordered = MESHES[mesh]
    p, orc = make(n)
    randomize_leaves(orc, seed=n, c_lo=0.3, c_hi=0.7)
    order, d = run(p, orc, precision, (1,))
    assert list(order.values()) == 3 * [ordered]
    orc.main_loop(1)
    ref = [orc.download_block(int(b)) for b in field_ids(orc, leaves_only=True)]
    g_max = max(np.abs(o["g"]).max() for o in ref)
    for i, o in enumerate(ref):
        for k, tol in (("h", H_ULPS * ULP[precision] / 9.0), ("g", G_ULPS * ULP[precision] * g_max)):
            err = np.abs(d[k][i].reshape(o[k].shape, order="F") - o[k])
            assert err.max() <= tol, (k, i, float(err.max()), tol)


@gpu
@pytest.mark.parametrize("precision", ["fp64", "fp16", "bf16"])
@pytest.mark.parametrize("n", [8, 16])
@pytest.mark.parametrize("mesh", list(MESHES))
def test_whole_rings_and_needed_populations(mesh, n, precision):
    """The last step of a call fills whole rings, the others the populations
    that streaming reads: one call of four steps gives the bits of four calls of
    one. A regrid after every step, whose tolerances change nothing, has every
    step read the P, Ux and Uy that the one before stored, in both."""
    p, orc = MESHES[mesh][0](n)
    randomize_leaves(orc, seed=n, c_lo=0.3, c_hi=0.7)
    still = dict(regrid_every=1, refin_tol=1e30, deref_tol=-1.0)
    _, a = run(p, orc, precision, (4,), **still)
    _, b = run(p, orc, precision, (1, 1, 1, 1), **still)
    for k in a:
        assert np.isfinite(a[k]).all() and np.array_equal(a[k], b[k]), k
