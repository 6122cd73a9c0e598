"""Server streams whose blocks grow while several are in flight and other
streams are opened: each block's outputs equal those of the same stream served
alone, block by block (bit for bit)."""
import time

import numpy as np
import pytest

from libfalcon_dsp_gb300.serving import ChannelizerServer, random_job

pytestmark = pytest.mark.gpu

SIZES = (5000, 21_000, 21_001, 60_000, 140_000, 139_999, 300_000)


def _caps(job, n):
    return [(n * c["up_rate"] + c["down_rate"] - 1) // c["down_rate"] + 2 for c in job["channels"]]


def _run(jobs, together):
    srv = ChannelizerServer(8 << 30, len(jobs))
    sids, waiting, res = {}, {}, {i: [None] * len(SIZES) for i in range(len(jobs))}

    def finish(keep=0):
        while len(waiting) > keep:
            for t in list(waiting):
                i, k, bufs = waiting[t]
                done, n_out, _ = srv.poll(t, len(bufs))
                if done:
                    res[i][k] = [b[:n].copy() for b, n in zip(bufs, n_out)]
                    del waiting[t]
            time.sleep(0.0005)

    for k, n in enumerate(SIZES):
        for i, j in enumerate(jobs):
            if i > k and together:
                continue  # stream i is opened while the first k blocks of the others are in flight
            for kk in ([k] if together and i < k else range(k + 1) if together else [k]):
                if i not in sids:
                    sids[i] = srv.open(j["fs"], j["channels"], max(SIZES), 1)
                    assert sids[i] is not None
                caps = _caps(j, max(SIZES))
                bufs = [np.empty(c, np.complex64) for c in caps]
                t = srv.submit(sids[i], j["x"][kk].ctypes.data, SIZES[kk], [b.ctypes.data for b in bufs], caps)
                waiting[t] = (i, kk, bufs)
                if not together:
                    finish()
    finish()
    for sid in sids.values():
        srv.close(sid)
    return res


def test_growing_blocks_in_flight():
    rng = np.random.default_rng(12)
    jobs = []
    for _ in range(4):
        j = random_job(rng, max_channels=8)
        j["x"] = [((rng.standard_normal(n) + 1j * rng.standard_normal(n)) * 0.2).astype(np.complex64) for n in SIZES]
        jobs.append(j)
    alone = [_run([j], False)[0] for j in jobs]
    mix = _run(jobs, True)
    for i in range(len(jobs)):
        for k in range(len(SIZES)):
            assert len(mix[i][k]) == len(alone[i][k])
            for a, b in zip(mix[i][k], alone[i][k]):
                assert np.array_equal(a, b), (i, k)
