"""Several small handles stepping at once.  A launch of the resident kernels
holds its SMs for milliseconds, so handles that fill the GPU alone would take
turns; they step with one launch per kernel while others run, which overlap.
What a handle computes does not depend on the way it took."""

import threading
import time

import numpy as np
import pytest

from test_steps_resident import build, read_all

pytestmark = pytest.mark.gpu


def in_threads(jobs):
    """Seconds from the start of all jobs to the end of the last."""
    failed = []

    def guarded(job):
        try:
            job()
        except Exception as e:  # noqa: BLE001 - reported by the caller's assert
            failed.append(e)

    threads = [threading.Thread(target=guarded, args=(j,)) for j in jobs]
    t0 = time.perf_counter()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    return time.perf_counter() - t0


def handle(pkg, p, pin):
    s = pkg.Simulation(p)
    s.set_particles(pin)
    s.step(10)
    s.particles()
    return s


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("call", [200, 8000])
def test_handles_at_once_overlap(pkg, cases, call, precision):
    """Four handles at 101 x 301 (148 blocks of the resident kernel each): in
    turn they take four times the time of one, overlapped about half of that.
    The smallest of a few attempts, as the host's threads may be held up."""
    p, pin = build(cases, "c1", 101, 301, 1, 24.0, precision)
    p.series_every = 0

    def job(s):
        def run():
            for _ in range(8000 // call):
                s.step(call)
            s.particles()
        return run

    sims = [handle(pkg, p, pin) for _ in range(4)]
    alone = min(in_threads([job(sims[0])]) for _ in range(3))
    ratio = 1e9
    for _ in range(5):
        ratio = min(ratio, in_threads([job(s) for s in sims]) / alone)
        if ratio < 3.4:
            break
    for s in sims:
        assert s.status() == 0
        s.close()
    assert ratio < 3.4


@pytest.mark.parametrize("precision", [0, 1])
def test_handles_at_once_give_the_bits_of_one_alone(pkg, cases, precision):
    """Calls of many lengths, each of which may find the other handles running
    or idle, with a history ring that wraps; one handle of each kind: one that
    fits beside others, ones that do not, and a batch."""
    specs = [("c1", 31, 40, 1, 6.0), ("c1", 101, 301, 1, 24.0), ("c3", 161, 161, 8, 8.0),
             ("c6", 81, 201, 2, 10.0)]
    calls = (1, 700, 1, 1, 300, 1500, 2, 495)

    def make(spec):
        p, pin = build(cases, *spec, precision)
        p.series_every, p.series_capacity, p.series_particles = 5, 64, spec[3]
        return p, pin

    def drive(s, out):
        rec = []
        for n in calls:
            s.step(n)
            if n in (1500, 495):
                rec.append(s.series())
        out.update(read_all(s), series=np.concatenate(rec))

    want = []
    for spec in specs:
        p, pin = make(spec)
        s = pkg.Simulation(p)
        s.set_particles(pin)
        out = {}
        drive(s, out)
        assert s.status() == 0 and s.kk == sum(calls)
        want.append(out)
        s.close()
    sims, got = [], [{} for _ in specs]
    for spec in specs:
        p, pin = make(spec)
        s = pkg.Simulation(p)
        s.set_particles(pin)
        sims.append(s)
    p, pin = make(specs[3])
    p.series_every = 0
    b = pkg.Batch([p, p])
    for s in b.sims:
        s.set_particles(pin)
    jobs = [lambda s=s, o=o: drive(s, o) for s, o in zip(sims, got)]
    in_threads(jobs + [lambda: [b.step(100) for _ in range(10)]])
    b.close()
    for s, g, w in zip(sims, got, want):
        assert s.status() == 0 and s.kk == sum(calls)
        for k, v in w.items():
            assert np.array_equal(g[k], v, equal_nan=True), k
        s.close()


def test_gradients_at_once_overlap(pkg, cases):
    """Two gradients in a row in each of four threads, on fresh handles: the
    gradient of one alone within the kernels' rounding (FP64, 2e-9 as between
    the two ways in test_adjoint_levels), in less than four times its time."""
    p, pin = build(cases, "c1", 101, 301, 1, 24.0, 0)
    p.series_every = 0

    def gradients(n, out=None):
        sims = []
        for _ in range(n):
            s = pkg.Simulation(p)
            s.set_particles(pin)
            sims.append(s)

        def run():
            for s in sims:
                g = s.adjoint(500, 600)
                if out is not None:
                    out.append(g)
        return sims, run

    def timed(threads, outs):
        made = [gradients(2, o) for o in outs]
        t = in_threads([run for _, run in made])
        for sims, _ in made:
            for s in sims:
                s.close()
        return t

    alone = [[]]
    t1 = min(timed(1, alone) for _ in range(3))
    ratio = 1e9
    for _ in range(5):
        outs = [[] for _ in range(4)]
        ratio = min(ratio, timed(4, outs) / t1)
        j0, g0 = alone[0][0]
        for j, g in (x for o in outs for x in o):
            assert j == j0  # the forward kernels share their operations
            for k in g0:
                a, b = np.atleast_1d(g[k]), np.atleast_1d(g0[k])
                scale = np.max(np.abs(b)) if k not in ("x0", "y0") else max(
                    np.max(np.abs(g0["x0"])), np.max(np.abs(g0["y0"])))
                assert np.all(np.abs(a - b) <= 2e-9 * (np.abs(b) + scale)), k
        if ratio < 3.4:
            break
    assert ratio < 3.4


def test_short_calls_beside_a_long_one(pkg, cases):
    """Calls of ten steps and a particle read while another handle makes calls
    of 20,000 steps: the long calls give way, so a short one does not wait for
    launches of 1024 steps (about 7 ms each, two queued) but for its own few
    kernels.  The mean over a stretch of them stays below 2 ms (0.1 to 0.2 on an
    idle host; 7 to 65 ms behind resident launches only)."""
    made = []
    for nx, ny in ((400, 1200), (200, 600)):
        p, pin = build(cases, "c1", nx, ny, 1, 24.0, 0)
        p.series_every = 0
        made.append(handle(pkg, p, pin))
    a, b = made
    stop = threading.Event()

    def long_calls():
        while not stop.is_set():
            b.step(20000)
            b.particles()

    best = 1e9
    t = threading.Thread(target=long_calls)
    t.start()
    try:
        time.sleep(0.02)
        for _ in range(5):
            t0 = time.perf_counter()
            for _ in range(100):
                a.step(10)
                a.particles()
            best = min(best, (time.perf_counter() - t0) / 100)
            if best < 2e-3:
                break
    finally:
        stop.set()
        t.join()
    assert a.status() == 0 and b.status() == 0
    a.close()
    b.close()
    assert best < 2e-3
