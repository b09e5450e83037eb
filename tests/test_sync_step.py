"""The synchronous step waits for events that its context keeps and reads the
error word in host memory: more threads than kept events, and a failed step."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DT = 300.0


def test_more_threads_than_kept_events(gpu_ctx):
    import torch
    import scream_gb300 as p3
    n = 11
    inps = [p3.generate_inputs(0, 40 + i, 5 + i, 24) for i in range(n)]
    want = []
    for inp in inps:
        f = p3.P3Fields.from_inputs(inp)
        assert gpu_ctx.p3_main(f, DT, p3.P3X_FP64) > 0
        want.append(f.to_host())
    got, bad = [None] * n, []
    start = threading.Barrier(n)

    def work(i):
        try:
            stream = torch.cuda.Stream()
            for _ in range(4):
                with torch.cuda.stream(stream):
                    f = p3.P3Fields.from_inputs(inps[i])
                start.wait()
                gpu_ctx.p3_main(f, DT, p3.P3X_FP64, stream=stream)
            with torch.cuda.stream(stream):
                got[i] = f.to_host()
        except Exception as e:  # noqa: BLE001
            bad.append(e)
            start.abort()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
    for g, w in zip(got, want):
        for k in w:
            np.testing.assert_array_equal(g[k], w[k], err_msg=k)


@pytest.mark.parametrize("precision", [0, 1])
def test_a_failed_step_is_reported_once(gpu_ctx, precision):
    import scream_gb300 as p3
    good = p3.generate_inputs(0, 3, 4, 16)
    bad = {k: v.copy() for k, v in good.items()}
    bad["th"][2, 5] = np.nan
    for _ in range(2):
        with pytest.raises(p3.P3Error):
            gpu_ctx.p3_main(p3.P3Fields.from_inputs(bad), DT, precision)
        gpu_ctx.p3_main(p3.P3Fields.from_inputs(good), DT, precision)
