"""Sedimentation of a column by one warp leaves the rime out on 32 levels where
there is none.  A CTA per column (small calls) always takes the whole path, so
both give the same bits whatever the pattern of rime."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DT = 300.0


def rime_columns(n, nlev):
    """Ice on every level of every column; rime on none, on all, or on single
    levels around the 32-level chunks, also below the smallest rime mass."""
    import scream_gb300 as p3
    inp = {k: v.copy() for k, v in p3.generate_inputs(0, 5, n, nlev).items()}
    rng = np.random.default_rng(3)
    inp["qi"][:] = 10.0 ** rng.uniform(-9, -3, (n, nlev))
    inp["ni"][:] = 10.0 ** rng.uniform(2, 6, (n, nlev))
    rime = np.zeros((n, nlev))
    levels = [0, 1, 30, 31, 32, 33, 62, 63, 64, nlev - 2, nlev - 1]
    for c in range(n):
        kind = c % (len(levels) + 4)
        if kind < len(levels):
            rime[c, min(levels[kind], nlev - 1)] = 0.4
        elif kind == len(levels):
            rime[c] = 0.3
        elif kind == len(levels) + 1:
            rime[c, nlev // 2:] = 1.0
        elif kind == len(levels) + 2:
            rime[c] = 1e-12
    inp["qm"][:] = rime * inp["qi"]
    inp["bm"][:] = inp["qm"] / rng.uniform(40.0, 1000.0, (n, nlev))
    for f in ("cld_frac_i", "cld_frac_l", "cld_frac_r"):
        inp[f][:] = 1.0
    return inp


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nlev", [33, 64, 100])
@pytest.mark.parametrize("per_sm", [9, 21])
def test_chunks_without_rime(gpu_ctx, precision, nlev, per_sm):
    import torch
    import scream_gb300 as p3
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = per_sm * sms
    inp = rime_columns(n, nlev)
    whole = p3.P3Fields.from_inputs(inp)
    gpu_ctx.p3_main(whole, DT, precision)
    whole = whole.to_host()
    for a, b in ((0, 45), (n - sms, n)):
        part = p3.P3Fields.from_inputs({k: np.ascontiguousarray(v[a:b]) for k, v in inp.items()})
        gpu_ctx.p3_main(part, DT, precision)
        for k, v in part.to_host().items():
            np.testing.assert_array_equal(v, whole[k][a:b], err_msg=f"{k} {a}")
