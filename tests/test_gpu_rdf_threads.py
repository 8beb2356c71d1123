"""Pair histograms of different sizes from several threads at once, each with a context, a stream and a plan of its own:
what one launch asks of shared memory does not limit another's."""
import threading

import numpy as np
import pytest
import torch

from trj_analysis_b200 import frames

pytestmark = pytest.mark.gpu


def test_plans_of_different_sizes_from_threads():
    from trj_analysis_b200 import engine
    fr = frames.FCCSpec(cells=(5, 5, 5), sigma=0.1, seed=3).frame(0)
    half = float(min(fr.box)) / 2
    bins = (40, 4000, 12000, 800)  # shared memory per CTA from 25 to 100 KB
    calls, errors, counts = 1500, [], {}
    start = threading.Barrier(len(bins))

    def work(k):
        try:
            ctx, stream = engine.Context(0), torch.cuda.Stream()
            with torch.cuda.stream(stream):
                stage = engine.FrameStage(ctx, fr.n, 1)
                stage.upload_and_pack(fr.xyz, np.zeros(fr.n, np.int32), fr.box)
                plan = engine.RdfPlan(ctx, 1, half / bins[k], 0.0, fr.box, fr.n)
                hist = plan.new_hist()
                stream.synchronize()
                start.wait()
                for _ in range(calls):
                    plan.accumulate(stage.packed, fr.n, fr.box, hist, stream=stream)
                ctx.check(stream)
                counts[k] = int(hist.sum())
            plan.close()
            ctx.close()
        except Exception as e:  # reported by the main thread
            errors.append(e)
            start.abort()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(bins))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert len(counts) == len(bins) and all(c % calls == 0 and c > 0 for c in counts.values())
