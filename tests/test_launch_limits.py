"""Limits of part1+2's launch: blocks_per_sm CTAs an SM and a launch's share of
the GPU hold for every way that it takes its columns (a CTA each, pools of the
warps, CTAs of one warp), and change no bit."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
DT = 300.0


def test_launch_sizes_keep_to_their_limits(tmp_path):
    exe = tmp_path / "plan"
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{ROOT / 'scream_gb300' / 'csrc'}", str(ROOT / "tests" / "plan_check.cpp"),
                    "-o", str(exe)], check=True)
    assert int(subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("per_sm", [0.5, 1.5, 3, 7, 12, 30])
def test_blocks_per_sm_changes_no_bit(gpu_ctx, precision, per_sm):
    import torch
    import scream_gb300 as p3
    n = int(per_sm * torch.cuda.get_device_properties(0).multi_processor_count) + 1
    inp = p3.generate_inputs(0, 41, n, 72)

    def step():
        f = p3.P3Fields.from_inputs(inp)
        gpu_ctx.p3_main(f, DT, precision)
        return f.to_host()

    orig = gpu_ctx.launch_config(precision)
    whole = step()
    try:
        for blocks in (1, 3):
            gpu_ctx.set_launch_config(precision, blocks_per_sm=blocks)
            again = step()
            for k in whole:
                np.testing.assert_array_equal(again[k], whole[k], err_msg=f"{blocks} {k}")
    finally:
        gpu_ctx.set_launch_config(precision, blocks_per_sm=orig["blocks_per_sm"])
