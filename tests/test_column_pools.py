"""Part1+2 pools columns per warp, in sizes that depend on the call's columns
and levels; a pool ends at an instance's last column.  Columns are independent,
so whatever the pools every field is bitwise the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DT = 300.0


def step(ctx, inp, prec):
    import scream_gb300 as p3
    f = p3.P3Fields.from_inputs(inp)
    ctx.p3_main(f, DT, prec)
    return f.to_host()


def rows(inp, a, b):
    return {k: np.ascontiguousarray(v[a:b]) for k, v in inp.items()}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nlev", [1, 33, 72, 257, 1030])
def test_pool_sizes_agree(gpu_ctx, nlev, precision):
    """Pools of 1 to 16 columns (more columns than warps; lanes 32, 16, 8) against
    calls with one column per CTA."""
    import torch
    import scream_gb300 as p3
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = (40 if nlev <= 72 else 17) * sms + 5
    inp = p3.generate_inputs(0, 31, n, nlev)
    orig = gpu_ctx.launch_config(precision)
    try:
        whole = step(gpu_ctx, inp, precision)
        for lanes, cols in ((16, 2), (8, 16)):
            gpu_ctx.set_launch_config(precision, lanes=lanes, columns_per_block=cols)
            again = step(gpu_ctx, inp, precision)
            for k in whole:
                np.testing.assert_array_equal(again[k], whole[k], err_msg=f"{lanes} {k}")
    finally:
        gpu_ctx.set_launch_config(precision, lanes=orig["lanes_per_column"],
                                  columns_per_block=orig["columns_per_block"])
    for a in (0, n // 2, n - sms):
        part = step(gpu_ctx, rows(inp, a, a + sms), precision)
        for k, v in part.items():
            np.testing.assert_array_equal(v, whole[k][a:a + sms], err_msg=f"{k} {a}")


@pytest.mark.parametrize("precision", [0, 1])
def test_pools_end_at_an_instance(gpu_ctx, precision):
    """A batch of many small instances of different depths, more columns than
    warps, against one call per instance."""
    import torch
    import scream_gb300 as p3
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sizes = [(5 + i % 9, 3 + i % 41) for i in range(3 * sms)]
    inps = [p3.generate_inputs(0, 100 + i, nc, nl) for i, (nc, nl) in enumerate(sizes)]
    fields = [p3.P3Fields.from_inputs(i) for i in inps]
    b = p3.P3Batch(gpu_ctx, fields, [DT] * len(fields), precision=precision)
    b.run()
    torch.cuda.synchronize()
    got = [f.to_host() for f in fields]
    b.close()
    for i in range(0, len(sizes), 5):
        one = step(gpu_ctx, inps[i], precision)
        for k in one:
            np.testing.assert_array_equal(got[i][k], one[k], err_msg=f"{i} {k}")


@pytest.mark.parametrize("precision,deepest", [(0, 2639), (1, 2903)])
def test_deepest_columns(gpu_ctx, precision, deepest):
    """The deepest accepted column gives the same bits alone and with others; a
    deeper one is refused."""
    import scream_gb300 as p3
    inp = p3.generate_inputs(0, 8, 3, deepest)
    whole = step(gpu_ctx, inp, precision)
    one = step(gpu_ctx, rows(inp, 2, 3), precision)
    for k, v in one.items():
        np.testing.assert_array_equal(v, whole[k][2:3], err_msg=k)
    with pytest.raises(p3.P3Error):
        step(gpu_ctx, p3.generate_inputs(0, 8, 1, deepest + 1), precision)
