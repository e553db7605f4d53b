"""The block-tree solve, the one-kernel sort and the culled lists at the sizes where they
change form: levels of the tree, the sizes where a warp per particle takes over, particles
with more neighbours than a row, a warp or a block holds, boxes a few supports wide, sets
far from the origin, and the sort's steps of pairs a thread.  Plain results are required to
equal the oracle's, or the list-based loop's (a solve without gradients), bit for bit."""
import numpy as np
import pytest

from cosmosphere_b200 import capi, inputs
from oracle import oracle as O
from test_parity_gpu import FIELDS, FORCE, _vel_acc, assert_same, check_all, run_pair

pytestmark = pytest.mark.gpu
UNIT = [0.0, 1.0, 0.0, 1.0, 0.0, 1.0]


def _box(n, seed=1, hscale=1.2):
    rng = np.random.default_rng(seed)
    x, y, z = rng.random((3, n))
    h = hscale * (1.0 / n) ** (1.0 / 3.0) * rng.uniform(0.8, 1.25, n)
    return inputs.Particles(x=x, y=y, z=z, h=h, pmass=1.0 / n)


# blocks of 8, levels of 8^k blocks, and one particle beyond each; a force, then a Newton
# and gradient pass, of a warp per particle up to 12288 and 32768 particles
@pytest.mark.parametrize("n,periodic", [(200, True), (511, False), (512, True), (513, False), (4096, False),
                                        (4097, True), (12288, False), (12289, True), (32768, True), (32769, False)])
def test_sizes_around_the_levels_and_the_forms(n, periodic):
    c, o = run_pair(_box(n), box=UNIT if periodic else None)
    check_all(c, o)


@pytest.mark.parametrize("case", ["huge", "overflow", "overflow_quintic", "narrow", "dead", "far", "outlier"])
def test_uncommon_sets(case):
    quintic, box = case.endswith("quintic"), None
    if case == "huge":            # a few particles start with most of the set inside their support
        p = inputs.plummer(9000, hfact=1.2, lnsigma=0.2, seed=3)
        p["h"][::700] *= 60.0
    elif case.startswith("overflow"):
        p = inputs.plummer(6000, lnsigma=0.9, seed=12)
    elif case == "narrow":        # the box is under four supports wide
        p, box = _box(300, 4), UNIT
    elif case == "dead":
        p, box = _box(5000, 6), UNIT
        p["h"][::3] = -1.0
        p["pmass"] *= 1.5
    elif case == "far":           # h is 1e-8 of the coordinates
        p = _box(5000, 7)
        for k in "xyz":
            p[k] += 4.0e6
    else:                         # one particle a thousand set sizes away, with a support that reaches
        p = _box(5000, 8)
        p["x"][17] += 1000.0
        p["h"][17] = 700.0
    c, o = run_pair(p, quintic=quintic, box=box)
    check_all(c, o)


def test_no_live_particle():
    p = _box(300)
    p["h"][:] = -1.0
    c = capi.Cosmo()
    c.set_precision(False)
    c.arrays_init(p.n)
    c.upload(capi.POS, np.stack([p["x"], p["y"], p["z"]]))
    c.upload(capi.HSML, p["h"])
    assert c.density_status(p.n, p["pmass"]) == 0
    g = c.download(capi.GRAD_OUT, p.n)
    assert np.all(g[1] == 1.0) and np.all(g[0] == 0.0) and np.all(g[2] == 0.0)


def _solve(p, gradients, box=None, frozen=None):
    c = capi.Cosmo()
    c.set_precision(False)
    c.arrays_init(p.n)
    v, a = _vel_acc(p)
    for slot, data in ((capi.POS, np.stack([p["x"], p["y"], p["z"]])), (capi.HSML, p["h"]), (capi.VEL, v),
                       (capi.ACCEL, a)):
        c.upload(slot, data)
    c.set_frozen(frozen)
    try:
        st = c.density_status(p.n, p["pmass"], periodic_box=box, with_gradients=gradients)
    finally:
        c.set_frozen(None)
    return st, {k: c.array(k) for k in ("order", "h", "activePerIter")}, c.scalar("itersRun")


@pytest.mark.parametrize("case", ["frozen", "all_frozen", "outside", "drifted", "far", "outlier", "plummer"])
def test_block_tree_equals_the_list_loop(case):
    """A solve with gradients runs over the block tree, one without over leaf lists (and
    leaves rho at the h before its last step, where the gradient sweep makes it anew)."""
    box, frozen, p = None, None, _box(6000, 21)
    if case.endswith("frozen"):
        box, frozen = UNIT, (np.arange(p.n) % 3 != 0) | (case == "all_frozen")
    elif case == "outside":       # particles far beyond the periodic box: both over lists
        box = UNIT
        p["x"] += 0.3
        p["y"][::5] -= 0.7
    elif case == "drifted":       # particles that have just left the periodic box
        box = UNIT
        p["x"] += 0.009 * p["h"]
        p["y"] -= 0.009 * p["h"]
    elif case == "far":
        for k in "xyz":
            p[k] -= 3.0e5
    elif case == "outlier":
        p["z"][5] += 1000.0
        p["h"][5] = 700.0
    else:
        p = inputs.plummer(20000, hfact=1.2, lnsigma=0.5, seed=9)
    near, lists = _solve(p, True, box, frozen), _solve(p, False, box, frozen)
    assert near[0] == lists[0] and near[2] == lists[2]
    for k in near[1]:
        np.testing.assert_array_equal(near[1][k], lists[1][k], err_msg=k)


def test_batch_of_many_small_sets():
    """More sets than a block has threads, two of them without a live particle."""
    sets = [dict(_box((200 if k % 2 else 40) + k % 53, 300 + k), box=UNIT if k % 2 else None) for k in range(300)]
    for k in (7, 250):
        sets[k]["h"] = np.full(sets[k]["x"].size, -1.0)
    capi.Cosmo().set_precision(False)
    b = capi.Batch(sets)
    b.upload()
    assert b.density() == 0
    h, rho, gradh = b.download()
    for k in (0, 7, 31, 128, 255, 256, 299):
        s = sets[k]
        if k in (7, 250):
            np.testing.assert_array_equal(h[k], s["h"])
            continue
        o = O.Oracle()
        assert o.density(s["x"], s["y"], s["z"], s["h"], s["pmass"], periodic_box=s["box"],
                         with_gradients=False) == 0
        for got, name in ((h[k], "h"), (rho[k], "rho"), (gradh[k], "gradh")):
            np.testing.assert_array_equal(got, o.unsorted(name), err_msg=f"set {k} {name}")


@pytest.mark.parametrize("lnsigma", [0.3, 0.9])
def test_mixed_force_after_a_plain_solve(lnsigma):
    """The precision may change between the two: the mixed force pass then finds its leaves
    (and, where rows overflowed, its lists) made for it.  1e-5 of each field's norm is the
    mixed form's own bound."""
    p = inputs.plummer(6000, lnsigma=lnsigma, seed=12)
    c, o = run_pair(p)
    ref = {k: c.array(k) for k in FORCE}
    assert_same(c, o, FIELDS + FORCE)
    c.set_precision(True)
    try:
        c.force(p.n, p["pmass"], beta=2.0, alphau=0.1)
        for k in ("fx", "fy", "fz"):
            got = c.array(k)
            assert np.all(np.isfinite(got)), k
            assert np.linalg.norm(got - ref[k]) <= 1e-5 * np.linalg.norm(ref[k]), k
    finally:
        c.set_precision(False)


@pytest.mark.parametrize("case", ["plummer_cut", "plummer_scattered", "box", "narrow", "quintic"])
def test_mixed_groups_of_every_size(case):
    """Leaves' last few particles, cut groups of one, of a few and of more, and a box whose
    groups span half a period: h and rho of a mixed solve, alone and in a batch, within the
    mixed form's 1e-5 of the plain one's."""
    quintic, box = case == "quintic", UNIT if case in ("box", "narrow") else None
    if case == "plummer_cut" or quintic:
        p = inputs.plummer(20000, hfact=1.0 if quintic else 1.2, lnsigma=0.2, seed=31)
    elif case == "plummer_scattered":
        p = inputs.plummer(9000, hfact=1.2, lnsigma=0.7, seed=32)
    else:
        p = _box(300 if case == "narrow" else 8000, 33)
    c = capi.Cosmo(quintic)
    got = []
    for mixed in (False, True):
        c.set_precision(mixed)
        try:
            c.arrays_init(p.n)
            c.upload(capi.POS, np.stack([p["x"], p["y"], p["z"]]))
            c.upload(capi.HSML, p["h"])
            assert c.density_status(p.n, p["pmass"], periodic_box=box, hfact=1.0 if quintic else 1.2) == 0
            got.append((c.download(capi.HSML, p.n)[0], c.download(capi.DENS_OUT, p.n)[0]))
            if not quintic:
                b = capi.Batch([dict(p, box=box)])
                b.upload()
                assert b.density(tolh=1e-4, hfact=1.2, final_rho=True) == 0
                h, rho, _ = b.download()
                got.append((h[0], rho[0]))
        finally:
            c.set_precision(False)
    for h, rho in got[1:]:
        assert np.max(np.abs(h / got[0][0] - 1)) <= 1e-5
        assert np.max(np.abs(rho / got[0][1] - 1)) <= 1e-5


def _sort_sizes():
    import torch
    step = torch.cuda.get_device_properties(0).multi_processor_count * 1024 if torch.cuda.is_available() else 148 * 1024
    return [33, 1024, 1025, 4097, step, step + 1, 4 * step + 1, 8 * step + 1, 16 * step, 16 * step + 1]


@pytest.mark.parametrize("which", range(10))
def test_sort_steps(which):
    """The key order is the stable one, with ties (coincident particles) and dead particles,
    on both sides of every step of pairs a thread and of the one-kernel sort's capacity."""
    n = _sort_sizes()[which]
    rng = np.random.default_rng(n)
    side = int(np.ceil((n / 4) ** (1.0 / 3.0)))      # two particles a lattice point, and as many elsewhere
    pos = rng.integers(0, side, (3, n)).astype(np.float64)
    pos[:, n // 2:] = rng.random((3, n - n // 2)) * side
    h = np.where(rng.random(n) < 0.05, -1.0, 0.3)
    c = capi.Cosmo()
    c.set_precision(False)
    c.arrays_init(n)
    c.upload(capi.POS, pos)
    c.upload(capi.HSML, h)
    c.density_status(n, 1.0 / n, max_iter=1, with_gradients=False)
    keys, order = c.array("keys"), c.array("order")
    caller = np.empty_like(keys)
    caller[order] = keys
    assert np.array_equal(np.bincount(order, minlength=n), np.ones(n, dtype=np.int64))
    np.testing.assert_array_equal(order, np.argsort(caller, kind="stable").astype(order.dtype))
    assert int((keys == np.uint64(2**64 - 1)).sum()) == int((h <= 0).sum())
