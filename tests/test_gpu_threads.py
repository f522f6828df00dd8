"""One context a host thread: threads that resample clouds of different sizes, score
on maps of different layouts and scans of different lengths, and score spread clouds,
all at once, get what each call gives alone.  (What a kernel may take of shared
memory is one setting for the whole process; no call may set it to its own size.)"""
import threading

import numpy as np
import pytest

from oracle import oracle_py as O
from tsdf_localization_gb300 import Context, DeviceMap, ResidualSystematicResampler, TSDFEvaluator, synth

from test_gpu_scoring_kernels import cloud, random_map, scan

pytestmark = pytest.mark.gpu


def run_all(jobs):
    """Each job in a thread of its own, all started together."""
    gate, errors = threading.Barrier(len(jobs)), []

    def body(job):
        try:
            gate.wait()
            job()
        except BaseException as e:   # noqa: BLE001  (reported by the test)
            errors.append(e)

    threads = [threading.Thread(target=body, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def test_residual_resampling_of_different_sizes():
    rng = np.random.default_rng(1)
    jobs, contexts = [], []
    for m in (2561, 100_003, 4096, 23_457, 3000, 60_000):
        w = rng.gamma(0.8, size=m) + 0.02
        w = (w / w.sum()).astype(np.float32)
        want = O.resample_residual_systematic(w, 0.371)
        r = ResidualSystematicResampler(Context(0))
        contexts.append(r.ctx)

        def job(r=r, w=w, want=want):
            for _ in range(60):
                assert np.array_equal(r.resample_indices(w, 0.371), want)

        jobs.append(job)
    run_all(jobs)
    for c in contexts:
        c.close()


def test_scoring_on_different_maps():
    rng = np.random.default_rng(2)
    jobs, contexts = [], []
    # two sizes of map, so bitmaps of two sizes; short and long scans; two spread clouds
    for size, layout, spread, P, n, times in (
            ((21.3, 17.6, 5.2), {"dense": True}, False, 300, 257, 40), ((90.0, 70.0, 5.0), {"dense": True}, False, 40, 9000, 40),
            ((21.3, 17.6, 5.2), {}, False, 64, 14_000, 40), ((90.0, 70.0, 5.0), {"grid": True}, False, 64, 100, 40),
            ((21.3, 17.6, 5.2), {"dense": True}, True, 70_000, 750, 6),
            ((90.0, 70.0, 5.0), {"dense": True}, True, 70_000, 750, 6)):
        coef, occ, codes = random_map(size, 0.25, (0, 0, 0), 7)
        ctx = Context(0)
        contexts.append(ctx)
        dmap = DeviceMap(ctx, coef, occ, codes=codes, **layout)
        parts, pts = cloud(spread, P, size, (0, 0, 0), rng), scan(n, rng)
        want = TSDFEvaluator(dmap, generic=True).evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
        slow = TSDFEvaluator(dmap, generic=True)
        fast = TSDFEvaluator(dmap)

        def job(fast=fast, slow=slow, parts=parts, pts=pts, want=want, times=times):
            for k in range(times):
                ev = slow if k % 8 == 7 else fast
                d = ev.evaluate_debug(parts.copy(), pts, synth.IDENTITY_TF)
                assert np.array_equal(d["raw"], want["raw"]) and np.array_equal(d["hits"], want["hits"])

        jobs.append(job)
    run_all(jobs)
    for c in contexts:
        c.close()
