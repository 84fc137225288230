"""t9gb_pme_own_fft and t9gb_pme_fft_cluster: every choice can be taken back,
and whatever came before, a choice gives the bits that it gives on a new
context.  On 32^3 all routes exist: the one-cluster transform (the default),
the plane passes, cuFFT, and the plane passes while the learned guess trains."""
import numpy as np
import pytest

from gpu_util import cpu, engine_for

pytestmark = pytest.mark.gpu


def _engine(tg, n):
    e = engine_for(tg.systems.make_config("water648", nfft=n))
    e.pair_lanes(8)  # the default while the learned guess trains
    return e


def _fields(e):
    rng = np.random.default_rng(3)
    u, up = rng.normal(size=(e.n, 3)) * 0.05, rng.normal(size=(e.n, 3)) * 0.05
    return np.concatenate([cpu(x) for x in e.dfield() + e.ufield(u, up)])


def _routes(tg, n):
    default, cufft = _engine(tg, n), _engine(tg, n)
    cufft.pme_own_fft(False)
    r = {"default": _fields(default), "cufft": _fields(cufft)}
    assert not np.array_equal(r["default"], r["cufft"])
    if n == 32:
        planes = _engine(tg, n)
        planes.pme_own_fft(True)
        r["planes"] = _fields(planes)
        assert not any(np.array_equal(r["planes"], r[k]) for k in ("default", "cufft"))
    return r


def test_choices_32(gpu_lib, tg):
    r = _routes(tg, 32)
    e = _engine(tg, 32)
    for step, want in [
        (lambda: e.fft_cluster(0), "default"),
        (lambda: e.pme_own_fft(True), "planes"),
        (lambda: e.fft_cluster(4), "planes"),  # the same bits from the clusters
        (lambda: e.pme_own_fft(-1), "planes"),  # a partition asked for stays
        (lambda: e.fft_cluster(0), "default"),
        (lambda: e.learn_config(1), "planes"),
        (lambda: e.pme_own_fft(False), "cufft"),
        (lambda: e.learn_config(0), "cufft"),
        (lambda: e.pme_own_fft(-1), "default"),
        (lambda: e.fft_cluster(2), "planes"),
        (lambda: e.fft_cluster(0), "default"),
    ]:
        step()
        assert np.array_equal(_fields(e), r[want]), want


def test_choices_24(gpu_lib, tg):
    r = _routes(tg, 24)
    e = _engine(tg, 24)
    for step, want in [(lambda: e.fft_cluster(0), "default"), (lambda: e.pme_own_fft(False), "cufft"),
                       (lambda: e.fft_cluster(0), "cufft"), (lambda: e.pme_own_fft(-1), "default"),
                       (lambda: e.learn_config(1), "cufft"), (lambda: e.learn_config(0), "default")]:
        step()
        assert np.array_equal(_fields(e), r[want]), want
    for bad in (lambda: e.pme_own_fft(True), lambda: e.fft_cluster(4)):
        with pytest.raises(gpu_lib.T9Error):
            bad()
        assert np.array_equal(_fields(e), r["default"])


def test_solves_follow_the_choice(gpu_lib, tg):
    """The captured graph of a solve is rebuilt when the transform changes."""
    e, f = _engine(tg, 32), _engine(tg, 32)
    f.pme_own_fft(True)
    d0, p0 = (cpu(x) for x in e.induce()[:2])
    d1, p1 = (cpu(x) for x in f.induce()[:2])
    for choice, d, p in ((True, d1, p1), (-1, d0, p0), (True, d1, p1)):
        e.pme_own_fft(choice)
        x, y = e.induce()[:2]
        assert np.array_equal(cpu(x), d) and np.array_equal(cpu(y), p)
