"""Threads on streams of their own, in the same calls and in different ones at a time: the cached workspaces
are shared between them, results are the oracle's in each."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _jobs(nsgb, oracle, seed):
    """(call, what it has to give), sizes of their own for each thread, so that the buffers grow too."""
    rng = np.random.default_rng(seed)
    h, w = 200 + 61 * seed, 333 - 40 * seed
    image = rng.integers(0, 256, (h, w), dtype=np.uint8)
    mask = np.where(rng.random((h, w)) < 0.45, 255, 0).astype(np.uint8)
    labels = oracle.bwlabel2(mask, 8, True)[0]
    f = rng.random((1, h, w), dtype=np.float32)
    m = f * np.float32(0.75)
    d = {k: torch.from_numpy(v).cuda() for k, v in
         {"image": image, "mask": mask, "labels": labels, "f": f, "m": m}.items()}
    return [
        (lambda: nsgb.imfillHoles(d["image"], False, 4), oracle.imfill_holes(image, False, 4)),
        (lambda: nsgb.bwlabel(d["mask"], 8, True), labels),
        (lambda: nsgb.distanceTransform(d["mask"]), oracle.distance_transform(mask)),
        (lambda: nsgb.morphOpen(d["image"], nsgb.disk19()), oracle.morph_open(image, nsgb.disk19())),
        (lambda: nsgb.bounding_boxes(d["labels"]), oracle.bounding_box(labels)),
        (lambda: nsgb.recon_f32(d["m"], d["f"], 8)[0], oracle.recon_f32_prov(m, f, 8)[0]),
    ]


@pytest.mark.parametrize("together", [True, False])
def test_threads(nsgb, oracle, together):
    work = [_jobs(nsgb, oracle, seed) for seed in range(4)]
    torch.cuda.synchronize()
    wrong, start = [], threading.Barrier(len(work))

    def run(k):
        try:
            jobs = work[k]
            stream = torch.cuda.Stream()
            start.wait(60)
            with torch.cuda.stream(stream):
                for r in range(5):
                    for j in range(len(jobs)):
                        call, want = jobs[j if together else (j + k) % len(jobs)]
                        got = call()
                        stream.synchronize()
                        if not np.array_equal(got.cpu().numpy(), want):
                            wrong.append((k, r, j))
        except Exception as e:  # a thread's exception does not fail the test by itself
            wrong.append((k, repr(e)))

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:4]
