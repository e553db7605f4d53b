"""The batched form where it leaves the common path: iterations running out before every h has
converged, and the batches that are solved over lists (many neighbours, rows that do not
fit, a set outside its box, the settings of that loop)."""
import numpy as np
import pytest

from cosmosphere_b200 import autotune as at
from cosmosphere_b200 import capi, inputs

pytestmark = pytest.mark.gpu
UNIT = [0.0, 1.0, 0.0, 1.0, 0.0, 1.0]


def _box(n, seed=1, hscale=1.2):
    rng = np.random.default_rng(seed)
    x, y, z = rng.random((3, n))
    h = hscale * (1.0 / n) ** (1.0 / 3.0) * rng.uniform(0.8, 1.25, n)
    return dict(inputs.Particles(x=x, y=y, z=z, h=h, pmass=1.0 / n), box=UNIT)


def _plummer(n, seed=2, lnsigma=0.8, hfact=1.2):
    return dict(inputs.plummer(n, hfact=hfact, lnsigma=lnsigma, seed=seed))


def _batch(sets, quintic=False, staging=False, tuning=None, mixed=False, **kw):
    capi.Cosmo(quintic).set_precision(mixed)
    b = capi.Batch(sets, quintic=quintic)
    b.set_staging(staging)
    try:
        if tuning is not None:
            b.set_tuning(**tuning)
        b.upload()
        st = b.density(**kw)
        return st, b, b.download()
    finally:
        b.set_staging(False)
        capi.Cosmo(quintic).set_precision(False)


def _kernel(q, quintic):
    if not quintic:
        a, b = np.maximum(2.0 - q, 0.0), np.maximum(1.0 - q, 0.0)
        return 0.25 * (a**3 - 4.0 * b**3), 0.25 * (-3.0 * a**2 + 12.0 * b**2)
    a, b, c = (np.maximum(k - q, 0.0) for k in (3.0, 2.0, 1.0))
    return a**5 - 6.0 * b**5 + 15.0 * c**5, -5.0 * a**4 + 30.0 * b**4 - 75.0 * c**4


def _direct(s, h, quintic):
    """rho and d(rho)/dh of every particle at h by direct summation over all pairs, and the
    sum of the second's terms' sizes, which its rounding is measured against."""
    pos = np.stack([s["x"], s["y"], s["z"]])
    norm = s["pmass"] * (1.0 / (120.0 * np.pi) if quintic else 1.0 / np.pi)
    out = np.empty((3, h.size))
    for a in range(0, h.size, 500):
        d = pos[:, a:a + 500, None] - pos[:, None, :]
        if s.get("box") is not None:
            d -= np.round(d)
        hi = h[a:a + 500, None]
        q = np.sqrt((d * d).sum(axis=0)) / hi
        w, dw = _kernel(q, quintic)
        g = -q * dw - 3.0 * w
        out[:, a:a + 500] = np.stack([w.sum(axis=1), g.sum(axis=1), np.abs(g).sum(axis=1)])
    return out[0] * norm / h**3, out[1] * norm / h**4, out[2] * norm / h**4


@pytest.mark.parametrize("max_iter,graph,quintic", [(1, True, False), (2, True, False), (2, False, False),
                                                    (4, True, True)])
def test_final_rho_of_unconverged_particles(max_iter, graph, quintic):
    """rho and d(rho)/dh are those of the returned h for every particle, also for those whose
    last step outgrew their row or that never had one.  Sums of up to n terms round by n
    2^-53 of the sum of their sizes: 1e-11 is ten times that for 9000."""
    hf = 1.0 if quintic else 1.2
    sets = [_box(3000, 4, hf), _plummer(9000, hfact=hf), _plummer(900, seed=9, hfact=hf)]
    st, b, (h, rho, gradh) = _batch(sets, quintic, max_iter=max_iter, graph=graph, final_rho=True, hfact=hf)
    assert st == 1 and b.scalar("unconverged") > 1000
    for k, s in enumerate(sets):
        r, g, size = _direct(s, h[k], quintic)
        assert np.max(np.abs(rho[k] / r - 1.0)) <= 1e-11, k
        assert np.max(np.abs(gradh[k] - g) / size) <= 1e-11, k


@pytest.mark.parametrize("sizes,hfact,near", [((200000, 200000), 1.6, 1), ((200000, 200001), 1.6, 0),
                                              ((200000, 200001), 1.5, 1)])
def test_large_crowded_batches_are_solved_over_lists(sizes, hfact, near):
    sets = [_box(n, 20 + k, hfact) for k, n in enumerate(sizes)]
    st, b, got = _batch(sets, hfact=hfact, final_rho=True)
    assert st == 0 and b.scalar("blockTree") == near
    if not near:
        _, _, ref = _batch(sets, staging=True, hfact=hfact, final_rho=True)
        for a, r in zip(got, ref):
            for x, y in zip(a, r):
                np.testing.assert_array_equal(x, y)


def test_a_set_outside_its_box_sends_the_batch_over_lists_once():
    """One set of a batch has a particle beyond its periodic box: all are solved over lists, as
    each alone, and nothing is solved twice (launches are a staged batch's, which runs over
    lists by itself)."""
    sets = [_box(5000, 30), _box(3000, 31), _plummer(4000, 32, 0.3), _box(900, 33)]
    sets[1]["x"] = sets[1]["x"].copy()
    sets[1]["x"][7] += 1.7
    c = capi.Cosmo()
    n0 = c.launches()
    st, b, got = _batch(sets, graph=False)
    n1 = c.launches()
    st2, _, ref = _batch(sets, graph=False, staging=True)
    n2 = c.launches()
    assert st == 0 and st2 == 0 and b.scalar("blockTree") == 0
    assert n1 - n0 <= n2 - n1 + 2
    for a, r in zip(got, ref):
        for x, y in zip(a, r):
            np.testing.assert_array_equal(x, y)
    for k, s in enumerate(sets):
        n = s["x"].size
        c.arrays_init(n)
        c.upload(capi.POS, np.stack([s["x"], s["y"], s["z"]]))
        c.upload(capi.HSML, s["h"])
        assert c.density_status(n, s["pmass"], periodic_box=s.get("box"), with_gradients=False) == 0
        np.testing.assert_array_equal(got[0][k], c.download(capi.HSML, n)[0])
        np.testing.assert_array_equal(got[1][k], c.download(capi.DENS_OUT, n)[0])


def test_a_batch_whose_rows_do_not_fit_is_solved_over_lists():
    """Rows take 1 KB a particle: a batch they have no room for takes the lists, which do not
    need it, and gives the same results."""
    sets = [_box(300000, 40), _box(300001, 41)]
    L, c = capi.load(), capi.Cosmo()
    out = []
    assert c.set_option("batch_room_mb", -2) == -1
    for room in (500, -1):
        held = L.cosmo_serve_stat(b"device_bytes")
        assert c.set_option("batch_room_mb", room) == 0
        try:
            st, b, got = _batch(sets)
        finally:
            c.set_option("batch_room_mb", -1)
        assert st == 0 and b.scalar("blockTree") == (room < 0)
        if room >= 0:     # no rows (a batch solved before may hold some already)
            assert L.cosmo_serve_stat(b"device_bytes") - held < 600001 * 128 * 8 // 2
        out.append(got)
    for a, r in zip(*out):
        for x, y in zip(a, r):
            np.testing.assert_array_equal(x, y)


SETTINGS = [dict(bucket=16), dict(bucket=128), dict(bucket=512), dict(list_margin=1.0), dict(list_margin=1.3),
            dict(split_stream=32, split_work=32),
            dict(bucket=[16, 128, 32, 64], list_margin=[1.0, 1.3, 1.05, 1.15],
                 split_stream=[2048, 32, 4096, 8192], split_work=[65536, 64, 262144, 131072])]


@pytest.fixture(scope="module")
def mixture():
    return [_box(4000, 50), _plummer(9000, 51, 0.2), _box(700, 52), _plummer(3000, 53, 0.6)]


@pytest.fixture(scope="module")
def near_results(mixture):
    st, b, got = _batch(mixture, final_rho=True)
    assert st == 0 and b.scalar("blockTree") == 1
    return got


# a staged batch and one with a particle outside its box run over lists, where the settings act
@pytest.mark.parametrize("setting", [{}] + SETTINGS)
@pytest.mark.parametrize("staging", [True, False])
def test_settings_of_the_list_loop_keep_the_plain_results(mixture, near_results, setting, staging):
    sets = mixture
    if not staging:
        out = _box(40, 54)
        out["x"] = out["x"].copy()
        out["x"][3] -= 1.2
        sets = mixture + [out]
        setting = {k: list(v) + [v[0]] if isinstance(v, list) else v for k, v in setting.items()}
    st, b, got = _batch(sets, staging=staging, tuning=setting or None, final_rho=True)
    assert st == 0 and b.scalar("blockTree") == 0
    for a, r in zip(got, near_results):
        for x, y in zip(a, r):
            np.testing.assert_array_equal(x, y)


def test_a_plain_batch_has_nothing_to_tune(mixture):
    """The tuner times a plain class once and keeps the defaults; a mixed one it tunes."""
    cands = {"bucket": (32, 64), "list_margin": (1.05, 1.15), "split_stream": (4096,), "split_work": (131072,)}
    for mixed in (False, True):
        capi.Cosmo().set_precision(mixed)
        try:
            table = at.tune(mixture, repeats=1, candidates=cands)
        finally:
            capi.Cosmo().set_precision(False)
        for c, t in table.entries.items():
            assert table.times[c]["evaluated"] == (3 if mixed else 1)
            assert mixed or t == at.DEFAULT
